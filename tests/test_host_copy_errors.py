"""The staged result copies leave the stream idle when a copy fails or memory
runs out half way: nothing may still write to the caller's arrays or the ring.
The header is compiled against a stand-in of the CUDA runtime whose copies fail
at a given call and which knows whether copies are outstanding (no GPU)."""
import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "ncpaprop-release_b200" / "csrc"

RUNTIME = r"""
#pragma once
#include <cstddef>
#include <cstdlib>
#include <cstring>
#include <atomic>
typedef int cudaError_t;
typedef void* cudaStream_t;
typedef void* cudaEvent_t;
enum { cudaSuccess = 0, cudaErrorUnknown = 999 };
enum { cudaMemcpyDeviceToHost = 2, cudaHostAllocDefault = 0, cudaEventDisableTiming = 2 };
enum { cudaMemoryTypeUnregistered = 0, cudaMemoryTypeHost = 1 };
struct cudaPointerAttributes { int type; };
inline int fail_at = -1, n_copy = 0;
inline std::atomic<int> outstanding{0};
inline const void *pinned_lo = nullptr, *pinned_hi = nullptr;
inline cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void* p) {
    a->type = p >= pinned_lo && p < pinned_hi ? cudaMemoryTypeHost : cudaMemoryTypeUnregistered;
    return cudaSuccess;
}
inline cudaError_t cudaGetLastError() { return cudaSuccess; }
inline cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, int, cudaStream_t) {
    if (n_copy++ == fail_at) return cudaErrorUnknown;
    std::memcpy(d, s, n);
    ++outstanding;
    return cudaSuccess;
}
inline cudaError_t cudaStreamSynchronize(cudaStream_t) { outstanding = 0; return cudaSuccess; }
inline cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
inline cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, int) { *e = (void*)1; return cudaSuccess; }
inline cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
inline cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
inline cudaError_t cudaHostAlloc(void** p, size_t n, int) { *p = std::malloc(n); return cudaSuccess; }
inline cudaError_t cudaFreeHost(void* p) { std::free(p); return cudaSuccess; }
inline cudaError_t cudaSetDevice(int) { return cudaSuccess; }
"""

MAIN = r"""
#include <cstdio>
#include <new>
#include "host_copy.hpp"
static long allocs_left = -1;  // allocations before bad_alloc (-1: no limit)
void* operator new(size_t n) {
    if (allocs_left == 0) throw std::bad_alloc();
    if (allocs_left > 0) --allocs_left;
    if (void* p = std::malloc(n)) return p;
    throw std::bad_alloc();
}
void operator delete(void* p) noexcept { std::free(p); }
void operator delete(void* p, size_t) noexcept { std::free(p); }

int main() {
    const size_t big = 20 << 20, small = 1000;
    char *src = (char*)std::malloc(big), *dst = (char*)std::malloc(big), *pin = (char*)std::malloc(2 * small);
    std::memset(src, 7, big);
    pinned_lo = pin;
    pinned_hi = pin + 2 * small;
    int bad = 0, failed = 0, thrown = 0;
    for (size_t bytes : {small, size_t(300000), big}) {
        const ncpa::HostCopier::Part parts[] = {{pin, src, small}, {dst, src, bytes}, {pin + small, src, small}};
        for (int at = -1; at < 90; ++at) {  // the copy that fails
            ncpa::HostCopier c;
            n_copy = 0;
            fail_at = at;
            std::memset(dst, 0, bytes);
            const cudaError_t rc = c.run(0, nullptr, parts, 3);
            if (outstanding != 0) ++bad;
            if (rc == cudaSuccess && std::memcmp(dst, src, bytes) != 0) ++bad;
            if (rc != cudaSuccess) ++failed;
            outstanding = 0;
        }
        fail_at = -1;
        for (long k = 0; k < 60; ++k) {  // the allocation that fails
            ncpa::HostCopier c;
            allocs_left = k;
            try {
                c.run(0, nullptr, parts, 3);
            } catch (const std::bad_alloc&) {
                ++thrown;
            }
            allocs_left = -1;
            if (outstanding != 0) ++bad;
            outstanding = 0;
        }
    }
    std::printf("%d %d %d\n", bad, failed, thrown);
    return 0;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_stream_idle_after_errors(tmp_path):
    (tmp_path / "cuda_runtime.h").write_text(RUNTIME)
    (tmp_path / "main.cpp").write_text(MAIN)
    subprocess.run(["g++", "-O1", "-std=c++17", "-pthread", "-I", str(tmp_path), "-I", str(CSRC), "-o",
                    str(tmp_path / "copies"), str(tmp_path / "main.cpp")], check=True)
    r = subprocess.run([str(tmp_path / "copies")], check=True, capture_output=True, text=True, timeout=120)
    bad, failed, thrown = map(int, r.stdout.split())
    assert failed > 10 and thrown > 5
    assert bad == 0
