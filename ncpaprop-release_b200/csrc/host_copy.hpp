// Results to host memory.  A copy into pageable memory runs through the
// driver's staging buffer on one thread and synchronises each time (15-20 us a
// copy however small, 8-10 GB/s however large).  Here the parts of a result go
// to a page-locked ring of the context, and the calling thread and up to
// kHelpers others copy the chunks on as they arrive (most of a large result's
// time is the first touch of its pages).  Page-locked destinations are written
// directly.  64 receivers x 20000 ranges (20 MB, 0.35 ms of it the sum): 5.0 -> 1.1 ms; one
// problem of 0.05 Hz with 200 ranges (a few KB in eight parts): 500 -> 336 us a
// call.
#pragma once

#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <condition_variable>
#include <cstring>
#include <exception>
#include <memory>
#include <mutex>
#include <thread>
#include <vector>

namespace ncpa {

class HostCopier {
public:
    struct Part {
        void* dst;
        const void* src;  // device memory
        size_t bytes;
    };

    HostCopier() = default;
    HostCopier(const HostCopier&) = delete;
    HostCopier& operator=(const HostCopier&) = delete;
    ~HostCopier() {
        {
            std::lock_guard<std::mutex> lk(mu_);
            stop_ = true;
        }
        cv_.notify_all();
        for (std::thread& t : helpers_) t.join();
        for (cudaEvent_t e : ev_) cudaEventDestroy(e);
        if (ring_) cudaFreeHost(ring_);
    }

    // Copies the parts after what the stream holds, and waits for all of it
    // (the stream is idle on return, after errors and exceptions too: nothing
    // writes to the caller's memory or the ring any more).
    cudaError_t run(int device, cudaStream_t st, const Part* parts, size_t n) {
        struct Wait {
            cudaStream_t st;
            bool done = false;
            cudaError_t now() {
                done = true;
                return cudaStreamSynchronize(st);
            }
            ~Wait() {
                if (!done) cudaStreamSynchronize(st);
            }
        } wait{st};
        std::vector<Chunk> todo;
        std::vector<const void*> dev;
        for (size_t i = 0; i < n; ++i) {
            const Part& p = parts[i];
            if (!p.bytes) continue;
            cudaPointerAttributes a{};
            const bool pageable =
                cudaPointerGetAttributes(&a, p.dst) == cudaSuccess && a.type == cudaMemoryTypeUnregistered;
            if (!pageable || !ready()) {
                cudaGetLastError();
                const cudaError_t e = cudaMemcpyAsync(p.dst, p.src, p.bytes, cudaMemcpyDeviceToHost, st);
                if (e != cudaSuccess) return e;
                continue;
            }
            for (size_t o = 0; o < p.bytes; o += kChunk)
                todo.push_back({static_cast<char*>(p.dst) + o, static_cast<const char*>(p.src) + o,
                                std::min(kChunk, p.bytes - o), nullptr});
        }
        for (size_t i = 0; i < todo.size();) {
            // as many chunks as the ring holds; few small ones share one wait
            size_t used = 0, e = i;
            dev.clear();
            for (; e < todo.size() && used + todo[e].bytes <= kRing && e - i < kEvents; ++e) {
                dev.push_back(todo[e].src);
                todo[e].src = ring_ + used;
                used += (todo[e].bytes + 63) / 64 * 64;
            }
            const bool shared = used <= kAlone;
            for (size_t k = i; k < e; ++k) {
                cudaError_t rc = cudaMemcpyAsync(const_cast<char*>(todo[k].src), dev[k - i], todo[k].bytes,
                                                 cudaMemcpyDeviceToHost, st);
                if (rc == cudaSuccess && !shared) rc = event(k - i, &todo[k].ev);
                if (rc == cudaSuccess && !shared) rc = cudaEventRecord(todo[k].ev, st);
                if (rc != cudaSuccess) return rc;
            }
            if (shared) {
                const cudaError_t rc = cudaStreamSynchronize(st);
                if (rc != cudaSuccess) return rc;
                for (size_t k = i; k < e; ++k) std::memcpy(todo[k].dst, todo[k].src, todo[k].bytes);
            } else {
                auto job = std::make_shared<Job>();
                job->device = device;
                job->chunks.assign(todo.begin() + i, todo.begin() + e);
                finish(job);
                const cudaError_t rc = static_cast<cudaError_t>(job->err.load());
                if (rc != cudaSuccess) return rc;
            }
            i = e;
        }
        return wait.now();
    }

    // The same between host arrays.
    void host(int device, const Part* parts, size_t n) {
        size_t total = 0;
        for (size_t i = 0; i < n; ++i) total += parts[i].bytes;
        if (total <= kAlone) {
            for (size_t i = 0; i < n; ++i)
                if (parts[i].bytes) std::memcpy(parts[i].dst, parts[i].src, parts[i].bytes);
            return;
        }
        auto job = std::make_shared<Job>();
        job->device = device;
        for (size_t i = 0; i < n; ++i)
            for (size_t o = 0; o < parts[i].bytes; o += kChunk)
                job->chunks.push_back({static_cast<char*>(parts[i].dst) + o, static_cast<const char*>(parts[i].src) + o,
                                       std::min(kChunk, parts[i].bytes - o), nullptr});
        finish(job);
    }

private:
    static constexpr size_t kChunk = 256 << 10, kRing = 16 << 20, kAlone = 128 << 10, kEvents = 128;
    static constexpr int kHelpers = 3;

    struct Chunk {
        char* dst;
        const char* src;  // in the ring, or the host source
        size_t bytes;
        cudaEvent_t ev;  // null: the data is there
    };
    struct Job {
        int device = 0;
        std::vector<Chunk> chunks;
        std::atomic<size_t> next{0}, done{0};
        std::atomic<int> err{0};
        void work() {
            for (size_t i; (i = next.fetch_add(1)) < chunks.size(); done.fetch_add(1, std::memory_order_release)) {
                const cudaError_t rc = chunks[i].ev ? cudaEventSynchronize(chunks[i].ev) : cudaSuccess;
                if (rc == cudaSuccess) std::memcpy(chunks[i].dst, chunks[i].src, chunks[i].bytes);
                else err.store(rc);
            }
        }
    };

    // the ring, allocated with the first pageable copy; without it (no
    // page-locked memory left) copies go the driver's way
    bool ready() {
        if (!ring_ && !failed_ && cudaHostAlloc((void**)&ring_, kRing, cudaHostAllocDefault) != cudaSuccess) {
            cudaGetLastError();
            ring_ = nullptr;
            failed_ = true;
        }
        return ring_ != nullptr;
    }
    cudaError_t event(size_t i, cudaEvent_t* ev) {
        while (ev_.size() <= i) {
            cudaEvent_t e;
            const cudaError_t rc = cudaEventCreateWithFlags(&e, cudaEventDisableTiming);
            if (rc != cudaSuccess) return rc;
            ev_.push_back(e);
        }
        *ev = ev_[i];
        return cudaSuccess;
    }
    // runs the job on this thread and the helpers
    void finish(const std::shared_ptr<Job>& job) {
        post(job);
        job->work();
        while (job->done.load(std::memory_order_acquire) < job->chunks.size()) std::this_thread::yield();
    }
    void post(const std::shared_ptr<Job>& job) {
        if (helpers_.empty()) {
            const int n = std::min<int>(kHelpers, (int)std::thread::hardware_concurrency() - 1);
            try {
                for (int i = 0; i < n; ++i) helpers_.emplace_back([this] { help(); });
            } catch (const std::exception&) {
                // fewer helpers, or none: the caller copies on its own
            }
        }
        {
            std::lock_guard<std::mutex> lk(mu_);
            job_ = job;
            ++turn_;
        }
        cv_.notify_all();
    }
    void help() {
        unsigned long long seen = 0;
        int device = -1;
        for (;;) {
            std::shared_ptr<Job> job;
            {
                std::unique_lock<std::mutex> lk(mu_);
                cv_.wait(lk, [&] { return stop_ || turn_ != seen; });
                if (stop_) return;
                seen = turn_;
                job = job_;
            }
            if (device != job->device && cudaSetDevice(job->device) != cudaSuccess) continue;
            device = job->device;
            job->work();
        }
    }

    char* ring_ = nullptr;
    bool failed_ = false;
    std::vector<cudaEvent_t> ev_;
    std::vector<std::thread> helpers_;
    std::mutex mu_;
    std::condition_variable cv_;
    std::shared_ptr<Job> job_;
    unsigned long long turn_ = 0;
    bool stop_ = false;
};

}  // namespace ncpa
