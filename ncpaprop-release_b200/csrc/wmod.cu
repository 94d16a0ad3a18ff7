// Wide-angle (WMod) normal modes: the quadratic eigenproblem
// (M k^2 + C k + D) v = 0 of WModeSolver::solve (WModeSolver.cpp:257-486),
// which the reference linearises to a 2N pencil and hands to SLEPc
// (EigenEngine::doWideAngleCalculation, EigenEngine.cpp:174-395).
//
// Here T(k) h^2 has unit off-diagonal and diagonal
//   t_i = (B_i - U_i kappa)^2 - kappa^2 - 2,  kappa = h k,
//   B_i = h omega / c0_i,  U_i = wc_i / c0_i,
// plus the ground term g0 in row 0: the polynomial a2 k^2 + a1 k + a0 of
// WModeSolver.cpp:544-565 (a2 = (U^2 - 1) h^2, a1 = -2 omega U / c0 h^2,
// a0 = (omega / c0)^2 h^2 - 2; no last-row repeat, EigenEngine.cpp:266-275)
// in factored form, two doubles per row.  For real k inside the propagating
// window dT/dk is negative definite (subsonic winds), so the number of
// negative eigenvalues of T grows by one at each real eigenvalue: the modes
// are found with Sturm counts in kappa and safeguarded Newton steps on det T,
// and each eigenvector is the null vector of T: panel.cu with the WmodPanel
// rows (64 frequencies x 20000 points: 6.5 -> 2.3 ms a call against sweeps of
// the rows themselves).  This file builds the rows.
#include <algorithm>

#include "device_common.cuh"
#include "kernels.hpp"

namespace ncpa {

// Rows (B_i, U_i) of one group's problems (nz_pad rows apart, problem p =
// frequency-major over n_az azimuths) on the sampling grid z_min + i dz_grid
// (WModeSolver.cpp:196-208), with the matrix spacing dz, and the ground term
// g0 = h^2 / (dz^2 (dz admittance + 1)); also (omega/c_eff)^2 for the WKB
// search and the c_eff extrema / ground / top values of getModalTrace
// (WModeSolver.cpp:530-629).  Padding rows are zero.  One thread per
// (azimuth, grid point) and kWbFreqs frequencies: the profile is sampled once.
constexpr int kWbFreqs = 16;

__global__ void __launch_bounds__(256) k_wmod_build(const GroupDesc* __restrict__ desc, int tiles) {
    const GroupDesc& G = desc[blockIdx.z];
    const int az = blockIdx.y;
    const int i = (blockIdx.x % tiles) * blockDim.x + threadIdx.x;
    const int n_f = G.n_f, n_az = G.n_az, nk = G.nk, nz = G.nz, nz_pad = G.nz_pad;
    const int f0 = (blockIdx.x / tiles) * kWbFreqs, f1 = min(n_f, f0 + kWbFreqs);
    if (az >= n_az || f0 >= f1 || (blockIdx.x % tiles) * blockDim.x >= nz_pad) return;
    const double *__restrict__ zk = G.zk, *__restrict__ c0k = G.c0k, *__restrict__ c0c = G.c0c;
    const double *__restrict__ wck = G.wck, *__restrict__ wcc = G.wcc;
    const double *__restrict__ ceffk = G.ceffk, *__restrict__ ceffc = G.ceffc;
    const double z_min = G.z_min, dz_grid = G.dz_grid, dz = G.dz, admittance = G.admittance;
    ProblemInfo* __restrict__ pinfo = G.pinfo;
    double2* __restrict__ rows = reinterpret_cast<double2*>(G.s);
    double* __restrict__ kz2 = G.kz2;
    double cmin = 1e300, cmax = -1e300, c0min = 1e300;
    const int top = nz - (nz / 10);
    const int itop = top + 1 < nz ? top + 1 : nz - 1;
    if (i >= nz && i < nz_pad)
        for (int f = f0; f < f1; ++f) rows[(size_t)(f * n_az + az) * nz_pad + i] = make_double2(0.0, 0.0);
    if (i < nz) {
        const double z = z_min + i * dz_grid;
        const double c0 = spline_get(nk, zk, c0k, c0c, z);
        const double wc = spline_get(nk, zk, wck + (size_t)az * nk, wcc + (size_t)az * 4 * (nk - 1), z);
        const double ce = spline_get(nk, zk, ceffk + (size_t)az * nk, ceffc + (size_t)az * 4 * (nk - 1), z);
        cmin = cmax = ce;
        c0min = c0;
        for (int f = f0; f < f1; ++f) {
            const int p = f * n_az + az;
            const double omega = pinfo[p].omega;
            const size_t o = (size_t)p * nz_pad + i;
            rows[o] = make_double2(dz * (omega / c0), wc / c0);
            if (i == 0) pinfo[p].g0 = 1.0 / (dz * admittance + 1.0);
            if (kz2) {
                const double te = omega / ce;
                kz2[o] = te * te;
            }
            if (i == 0) pinfo[p].ceff_grnd = ce;
            if (i == itop) pinfo[p].ceff_top = ce;
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        cmin = fmin(cmin, __shfl_xor_sync(0xffffffffu, cmin, o));
        cmax = fmax(cmax, __shfl_xor_sync(0xffffffffu, cmax, o));
        c0min = fmin(c0min, __shfl_xor_sync(0xffffffffu, c0min, o));
    }
    __shared__ double smin[8], smax[8], s0min[8];
    const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (lane == 0) {
        smin[wid] = cmin;
        smax[wid] = cmax;
        s0min[wid] = c0min;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int k = 1; k < 8; ++k) {
            cmin = fmin(cmin, smin[k]);
            cmax = fmax(cmax, smax[k]);
            c0min = fmin(c0min, s0min[k]);
        }
        cmin = fmin(cmin, smin[0]);
        cmax = fmax(cmax, smax[0]);
        if (cmin < 1e300) {
            for (int f = f0; f < f1; ++f) {
                const int p = f * n_az + az;
                atomicMin(&pinfo[p].ceffmin_bits, (unsigned long long)__double_as_longlong(cmin));
                atomicMax(&pinfo[p].ceffmax_bits, (unsigned long long)__double_as_longlong(cmax));
                atomicMin(&pinfo[p].c0min_bits, (unsigned long long)__double_as_longlong(c0min));
            }
        }
    }
}

int launch_wmod_build(cudaStream_t st, const GroupDesc* desc, const GroupDims& d) {
    const int tiles = (d.nz_pad + 255) / 256;
    int n = 0;
    for (int g0 = 0; g0 < d.n; g0 += 65535, ++n)
        k_wmod_build<<<dim3(tiles * ((d.n_f + kWbFreqs - 1) / kWbFreqs), d.n_az, std::min(65535, d.n - g0)), 256, 0,
                       st>>>(desc + g0, tiles);
    return n;
}

}  // namespace ncpa
