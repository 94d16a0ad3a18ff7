// Device helpers shared by the sm_100a kernels of the ESS normal-mode path.
//
// Arithmetic conventions: the library is compiled with --fmad=false, so a
// fused multiply-add appears only where fma() is written.  Any CPU code that
// performs the same operations in the same order without contraction
// (-ffp-contract=off) reproduces the profile sampling, matrix build and Sturm
// counts bit-for-bit.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

#include <cuda/std/complex>

#include "kernels.hpp"

namespace ncpa {

constexpr double kPi = 3.141592653589793;  // value of PI in src/common/util.h:13-14


// ---------------------------------------------------------------------------
// Steffen monotone cubic on non-uniform knots (gsl_interp_steffen as used by
// src/atmosphere/AtmosphericProperty1D.cpp:72-136).  coef[4i..4i+3] = a,b,c,d
// with y = d + t (c + t (b + t a)), t = x - x_i.
// ---------------------------------------------------------------------------
__device__ __forceinline__ int knot_search(int n, const double* __restrict__ x, double xq) {
    int lo = 0, hi = n - 1;
    while (hi > lo + 1) {
        int mid = (lo + hi) >> 1;
        if (x[mid] > xq) hi = mid; else lo = mid;
    }
    return lo;
}

__device__ __forceinline__ double spline_get(int n, const double* __restrict__ x,
                                             const double* __restrict__ y,
                                             const double* __restrict__ coef, double xq) {
    if (xq > x[n - 1]) return y[n - 1];
    if (xq < x[0]) return y[0];
    int i = knot_search(n, x, xq);
    const double* c = coef + 4 * i;
    double t = xq - x[i];
    return c[3] + t * (c[2] + t * (c[1] + t * c[0]));
}

// shift t of an isolation scan of n points on an even grid of [lo, hi]
__device__ __forceinline__ double scan_x(double lo, double hi, int t, int n) {
    if (t == 0) return lo;
    if (t == n - 1) return hi;
    return lo + (hi - lo) * ((double)t / (double)(n - 1));
}

// ---------------------------------------------------------------------------
// power-of-two rescaling (exact)
// ---------------------------------------------------------------------------
__device__ __forceinline__ int biased_exp(double v) {
    return (__double2hiint(v) >> 20) & 0x7ff;
}
// shift e such that max(|a|,|b|) * 2^-e is near 1, or 0 when inside 2^+-480
__device__ __forceinline__ int rescale_shift(double a, double b) {
    int e = max(biased_exp(a), biased_exp(b));
    if (e == 0) return 0;
    e -= 1023;
    return (e > 480 || e < -480) ? e : 0;
}
// overflow-only variant for recurrences whose squares are accumulated: keeps
// |a|,|b| below 2^240 so that sums of squares stay finite
__device__ __forceinline__ int grow_shift(double a, double b) {
    int e = max(biased_exp(a), biased_exp(b)) - 1023;
    return e > 240 ? e : 0;
}
// 2^k as a double; 0 below the normal range, +inf above it
__device__ __forceinline__ double pow2(int k) {
    if (k < -1022) return 0.0;
    if (k > 1023) return __longlong_as_double(0x7ff0000000000000ll);
    return __hiloint2double((k + 1023) << 20, 0);
}

// ---------------------------------------------------------------------------
// TMA bulk copies (cp.async.bulk, non-tensor) into shared memory with an
// mbarrier transaction count, and bounded waits.
// ---------------------------------------------------------------------------
__device__ __forceinline__ uint32_t smem_u32(const void* p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ void mbar_init(uint64_t* bar, unsigned count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void fence_mbar_init() {
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void fence_proxy_async() {
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
                 : "memory");
}
// global -> shared bulk copy; dst, src 16-byte aligned, bytes a multiple of 16
__device__ __forceinline__ void tma_load_1d(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
            smem_u32(dst)),
        "l"(src), "r"(bytes), "r"(smem_u32(bar))
        : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}
__device__ __forceinline__ uint64_t global_ns() {
    uint64_t t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}
// Bounded wait: gives up after one second of wall time (or at once when
// another wait of this launch already gave up), records kErrTimeout and
// returns false.
__device__ __forceinline__ bool mbar_wait_bounded(uint64_t* bar, uint32_t parity, unsigned* err) {
    if (mbar_try_wait(bar, parity)) return true;
    const uint64_t t0 = global_ns();
    for (;;) {
        if (mbar_try_wait(bar, parity)) return true;
        if (global_ns() - t0 > 1000000000ull || (*((volatile unsigned*)err) & kErrTimeout)) break;
    }
    atomicOr(err, kErrTimeout);
    return false;
}

// Bounded wait for copies this block issued itself, used on the way out after
// another wait gave up: one second of wall time whatever the error word says.
__device__ __forceinline__ bool mbar_wait_drain(uint64_t* bar, uint32_t parity) {
    const uint64_t t0 = global_ns();
    while (!mbar_try_wait(bar, parity))
        if (global_ns() - t0 > 1000000000ull) return false;
    return true;
}

// One Laguerre step for the degree-n polynomial det(T - x), all of whose
// roots are real, from g = det'/det and h = g^2 - det''/det (Laguerre's method;
// e.g. Li & Zeng, SIAM J. Sci. Comput. 15 (1994), for symmetric tridiagonal
// matrices): x_new = x - n / (g +- sqrt((n - 1)(n h - g^2))).  The two signs
// step to the nearest root above and below x; up selects the root above.
// Returns the correction subtracted from x (not finite when g and h are not).
__device__ __forceinline__ double laguerre_step(double g, double h, double n, bool up) {
    const double disc = fmax((n - 1.0) * fma(n, h, -g * g), 0.0);
    const double sq = sqrt(disc);
    const double dp = n / (g + sq), dm = n / (g - sq);
    // x - dp and x - dm: the one above x has the negative correction
    return up ? (dp < 0.0 ? dp : dm) : (dp > 0.0 ? dp : dm);
}

// principal square root of x + i y
__device__ __forceinline__ cuda::std::complex<double> csqrt_principal(double x, double y) {
    double m = hypot(x, y);
    double t = sqrt(0.5 * (m + fabs(x)));
    if (x >= 0.0) return cuda::std::complex<double>(t, y / (2.0 * t));
    return cuda::std::complex<double>(fabs(y) / (2.0 * t), copysign(t, y));
}

}  // namespace ncpa
