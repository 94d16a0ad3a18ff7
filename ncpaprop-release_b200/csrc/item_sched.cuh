// Which warp runs which work item of the eigen-solve kernels.
#pragma once

#include <cuda_runtime.h>

#include "kernels.hpp"

namespace ncpa {

// Item scheduler of the bisection (and of the isolation scan's units, all of
// equal cost).  The bisection's item list is cost-ordered, heaviest first
// (k_make_items with order 1).  On each warp scheduler (SM and sub-partition)
// the first warp to arrive takes items from the heavy end of the list and the
// next workers - 1 from the light end, so a scheduler runs a heavy and a
// light item side by side; later warps run no bisection (in the fused launch
// they exit, or take eigenvector items when ev_workers_only is off).  A worker first draws a ticket
// (n tickets for n items) and then an index from its end of the list: front
// and back indices never meet, so every item runs exactly once.  Where the
// CTAs land only decides the balance: the first warp on every scheduler is a
// worker.  sched: kSchedInts ints zeroed before the launch; null keeps plain
// round-robin (item q to warp q mod (grid x kWarpsPerCta)).
struct ItemSched {
    int* S;
    int role;     // 0: none, 1: heavy end, 2: light end
    bool worker;  // the warp runs bisection items (every warp without sched)
    __device__ ItemSched(int* sched, int workers) : S(sched), role(0), worker(true) {
        if (!S) return;
        const int lane = threadIdx.x & 31;
        if (lane == 0) {
            // the warp's SM and its sub-partition (hardware warp slot mod 4; a
            // CTA's warp index does not determine it)
            unsigned smid, slot;
            asm volatile("mov.u32 %0, %%smid;" : "=r"(smid));
            asm volatile("mov.u32 %0, %%warpid;" : "=r"(slot));
            const int key = smid < (unsigned)kSchedSms ? (int)(smid * 4 + (slot & 3u)) : -1;
            const int k = key >= 0 ? atomicAdd(S + 3 + key, 1) : 0;
            role = k == 0 ? 1 : (k < workers ? 2 : 0);
        }
        role = __shfl_sync(0xffffffffu, role, 0);
        worker = role != 0;
    }
    // next item of this warp (-1: none left); walk = plain round-robin position
    __device__ long long next(int n, long long& walk, long long stride) {
        if (!S) {
            const long long it = walk;
            walk += stride;
            return it < n ? it : -1;
        }
        if (!role) return -1;
        int it = -1;
        if ((threadIdx.x & 31) == 0) {
            if (atomicAdd(S, 1) < n) it = role == 1 ? atomicAdd(S + 1, 1) : n - 1 - atomicAdd(S + 2, 1);
        }
        it = __shfl_sync(0xffffffffu, it, 0);
        if (it < 0) role = 0;
        return it;
    }
};

}  // namespace ncpa
