// sm_100a kernels of the effective-sound-speed (ESS) normal-mode path.
//
//  K0  knot-level fields: Steffen coefficients, c0 / wind speed / direction,
//      c_eff per azimuth, Sutherland-Bass absorption per frequency
//      (src/atmosphere/{AtmosphericProperty1D,Atmosphere1D,AtmosphericModel}.cpp)
//  K1  matrix build on the Nz grid (ESSModeSolver::getModalTrace,
//      ESSModeSolver.cpp:531-559; EigenEngine.cpp:57-83 assembly)
//  K2  WKB window (ESSModeSolver.cpp:561-621)
//  K3, K4  eigenvalues and mode values: panel.cu (here only the mode values of
//      the calls without allocations, K4s)
//  K5  modal sums for 1-D / 2-D transmission loss (ModeSolver.cpp:292-565)
//  K6  ModBB transfer function + pulse synthesis
//      (ModalBroadbandPropagator.cpp:245-277, BroadbandPropagator.cpp:327-662)
#include <algorithm>

#include "device_common.cuh"
#include "kernels.hpp"

#include <cuda/std/complex>

namespace ncpa {

// ===========================================================================
// K0: knot-level fields
// ===========================================================================
__device__ __forceinline__ double sgn1(double v) { return v < 0.0 ? -1.0 : 1.0; }

// Steffen (1990) slope at knot i; one-sided secants at the ends
__device__ double steffen_slope(int n, const double* __restrict__ x, const double* __restrict__ y, int i) {
    if (i == 0) return (y[1] - y[0]) / (x[1] - x[0]);
    if (i == n - 1) return (y[n - 1] - y[n - 2]) / (x[n - 1] - x[n - 2]);
    double hl = x[i] - x[i - 1], hr = x[i + 1] - x[i];
    double sl = (y[i] - y[i - 1]) / hl, sr = (y[i + 1] - y[i]) / hr;
    double pp = (sl * hr + sr * hl) / (hl + hr);
    double m = fabs(sl);
    if (fabs(sr) < m) m = fabs(sr);
    if (0.5 * fabs(pp) < m) m = 0.5 * fabs(pp);
    return (sgn1(sl) + sgn1(sr)) * m;
}

// coefficients of the interval i
__device__ __forceinline__ void steffen_coef(int n, const double* __restrict__ x, const double* __restrict__ y, int i,
                                             double* __restrict__ c) {
    const double y0 = steffen_slope(n, x, y, i), y1 = steffen_slope(n, x, y, i + 1);
    const double h = x[i + 1] - x[i];
    const double s = (y[i + 1] - y[i]) / h;
    c[0] = (y0 + y1 - 2.0 * s) / h / h;
    c[1] = (3.0 * s - 2.0 * y0 - y1) / h;
    c[2] = y0;
    c[3] = y[i];
}

__global__ void k_steffen(int n, const double* __restrict__ x, const double* __restrict__ yall, int batch,
                          int ystride, double* __restrict__ call, int cstride) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    int b = blockIdx.y;
    if (i >= n - 1 || b >= batch) return;
    steffen_coef(n, x, yall + (size_t)b * ystride, i, call + (size_t)b * cstride + 4 * i);
}

int launch_steffen(cudaStream_t st, int n, const double* x, const double* y, int batch, int ystride,
                   double* coef, int cstride) {
    dim3 grid((n - 1 + 255) / 256, batch);
    k_steffen<<<grid, 256, 0, st>>>(n, x, y, batch, ystride, coef, cstride);
    return 1;
}

// c0 = sqrt(1.4 P/rho) with P, rho read through their splines at the knots
// (Atmosphere1D.cpp:821-848); wind speed and direction, degrees clockwise
// from north (Atmosphere1D.cpp:484-544)
__global__ void k_profile_derived(int n, const double* __restrict__ z, const double* __restrict__ u,
                                  const double* __restrict__ v, const double* __restrict__ p,
                                  const double* __restrict__ rho, const double* __restrict__ pcoef,
                                  const double* __restrict__ rcoef, int have_c0, double* __restrict__ c0,
                                  double* __restrict__ ws, double* __restrict__ wd) {
    int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    if (!have_c0) {
        double pv = spline_get(n, z, p, pcoef, z[k]);
        double rv = spline_get(n, z, rho, rcoef, z[k]);
        c0[k] = sqrt(1.4 * pv / rv);
    }
    ws[k] = sqrt(u[k] * u[k] + v[k] * v[k]);
    wd[k] = (kPi / 2.0 - atan2(v[k], u[k])) * 180.0 / kPi;
}

int launch_profile_derived(cudaStream_t st, int n, const double* z, const double* u, const double* v,
                           const double* p, const double* rho, const double* pcoef, const double* rcoef,
                           int have_c0, double* c0, double* ws, double* wd) {
    k_profile_derived<<<(n + 255) / 256, 256, 0, st>>>(n, z, u, v, p, rho, pcoef, rcoef, have_c0, c0, ws, wd);
    return 1;
}

// c_eff = c0 + |w| cos(dir - az) at the knots (Atmosphere1D.cpp:546-610)
__global__ void k_ceff_knots(int n, int n_az, const double* __restrict__ az, const double* __restrict__ c0,
                             const double* __restrict__ ws, const double* __restrict__ wd,
                             double* __restrict__ ceff) {
    int k = blockIdx.x * blockDim.x + threadIdx.x;
    int a = blockIdx.y;
    if (k >= n || a >= n_az) return;
    double az_rad = az[a] * kPi / 180.0;
    double dir = wd[k] * kPi / 180.0;
    double wc = ws[k] * cos(dir - az_rad);
    ceff[(size_t)a * n + k] = wc + c0[k];
}

int launch_ceff_knots(cudaStream_t st, int n, int n_az, const double* az, const double* c0, const double* ws,
                      const double* wd, double* ceff) {
    dim3 grid((n + 255) / 256, n_az);
    k_ceff_knots<<<grid, 256, 0, st>>>(n, n_az, az, c0, ws, wd, ceff);
    return 1;
}

// Sutherland-Bass absorption [Np/m] (AtmosphericModel.cpp:86-219), split into
// its frequency-independent part at a knot (sound speed, viscosity, mole
// fractions, rotational collision number, vibrational relaxation frequencies
// and strengths: every pow / exp of the model) and the per-frequency rational
// part, so a thread evaluates one knot's part once for kSbFreqs frequencies.
struct SbKnot {
    double c;       // sound speed sqrt(1.4 P / rho)
    double nu_f;    // nu / f = 8 pi mu / (3 P)
    double nn;      // (4/5) sqrt(3/7) Z_rot
    double x_on;    // (X_O2 + X_N2) / 0.9903
    double am[4];   // A_max / c of the four vibrational modes
    double fv[4];   // their relaxation frequencies
};

// z in km
__device__ SbKnot sb_knot(double z, double T_z, double P_z, double D_z) {
    const double mu_o = 18.192E-6, T_o = 293.15, P_o = 101325, S = 117.0;
    const double Cv_R[4] = {5.0 / 2.0, 5.0 / 2.0, 3.0, 3.0};
    const double Cp_R[4] = {7.0 / 2.0, 7.0 / 2.0, 4.0, 4.0};
    const double theta[4] = {2239.1, 3352.0, 915.0, 1037.0};
    const double PI = kPi;
    SbKnot K;
    K.c = sqrt(1.4 * P_z / D_z);
    const double mu = mu_o * sqrt(T_z / T_o) * ((1.0 + S / T_o) / (1.0 + S / T_z));
    K.nu_f = (8.0 * PI * mu) / (3.0 * P_z);
    const double z2 = z * z, z3 = z2 * z, z4 = z3 * z, z5 = z4 * z;
    double X[7];
    X[0] = (z > 90.0) ? pow(10.0, 49.296 - (1.5524 * z) + (1.8714E-2 * z2) - (1.1069E-4 * z3) + (3.199E-7 * z4) -
                                      (3.6211E-10 * z5))
                      : pow(10.0, -0.67887);
    X[1] = (z > 76.0) ? pow(10.0, (1.3972E-1) - (5.6269E-3 * z) + (3.9407E-5 * z2) - (1.0737E-7 * z3))
                      : pow(10.0, -0.10744);
    X[2] = pow(10.0, -3.3979);
    X[3] = (z > 80.0) ? pow(10.0, -4.234 - (3.0975E-2 * z))
                      : pow(10.0, -19.027 + (1.3093 * z) - (4.6496E-2 * z2) + (7.8543E-4 * z3) - (6.5169E-6 * z4) +
                                      (2.1343E-8 * z5));
    X[4] = (z > 95.0) ? pow(10.0, -3.2456 + (4.6642E-2 * z) - (2.6894E-4 * z2) + (5.264E-7 * z3))
                      : pow(10.0, -11.195 + (1.5408E-1 * z) - (1.4348E-3 * z2) + (1.0166E-5 * z3));
    X[5] = pow(10.0, -53.746 + (1.5439 * z) - (1.8824E-2 * z2) + (1.1587E-4 * z3) - (3.5399E-7 * z4) +
                         (4.2609E-10 * z5));
    X[6] = (z > 30.0) ? pow(10.0, -4.2563 + (7.6245E-2 * z) - (2.1824E-3 * z2) - (2.3010E-6 * z3) +
                                      (2.4265E-7 * z4) - (1.2500E-09 * z5))
                      : pow(10.0, -1.7491 + (4.4986E-2 * z) - (6.8549E-2 * z2) + (5.4639E-3 * z3) -
                                      (1.5539E-4 * z4) + (1.5063E-06 * z5));
    K.x_on = (X[0] + X[1]) / 0.9903;
    const double tc = pow(T_z, -1.0 / 3.0);
    const double Z_rot_0 = 54.1 * exp(-17.3 * tc);
    const double Z_rot_1 = 63.3 * exp(-16.7 * tc);
    const double Z_rot_ = 1.0 / ((X[1] / Z_rot_1) + (X[0] / Z_rot_0));
    K.nn = (4.0 / 5.0) * sqrt(3.0 / 7.0) * Z_rot_;
    const double Tr = pow(T_z / T_o, -1.0 / 3.0) - 1.0;
    const double A1 = (X[0] + X[1]) * 24.0 * exp(-9.16 * Tr);
    const double A2 = (X[4] + X[5]) * 2400.0;
    const double B = 40400.0 * exp(10.0 * Tr);
    const double C = 0.02 * exp(-11.2 * Tr);
    const double Dd = 0.391 * exp(8.41 * Tr);
    const double E = 9.0 * exp(-19.9 * Tr);
    const double F = 60000.0;
    const double G = 28000.0 * exp(-4.17 * Tr);
    const double H = 22000.0 * exp(-7.68 * Tr);
    const double I_ = 15100.0 * exp(-10.4 * Tr);
    const double J = 11500.0 * exp(-9.17 * Tr);
    const double Kc = (8.48E08) * exp(9.17 * Tr);
    const double L = exp(-7.72 * Tr);
    const double ZZ = H * X[2] + I_ * (X[0] + 0.5 * X[4]) + J * (X[1] + 0.5 * X[5]) + Kc * (X[6] + X[3]);
    const double hu = 100.0 * (X[3] + X[6]);
    const double pf = (P_z / P_o) * (mu_o / mu);
    K.fv[0] = pf * (A1 + A2 + B * hu * (C + hu) * (Dd + hu));
    K.fv[1] = pf * (E + F * X[3] + G * X[6]);
    K.fv[2] = pf * ZZ;
    K.fv[3] = pf * (1.2E5) * L;
#pragma unroll
    for (int m = 0; m < 4; m++) {
        const double et = exp(-theta[m] / T_z);
        const double tt = theta[m] / T_z, om = 1 - et;
        const double C_R = ((tt * tt) * et) / (om * om);
        const double A_max = (X[m] * (PI / 2) * C_R) / (Cp_R[m] * (Cv_R[m] + C_R));
        K.am[m] = A_max / K.c;
    }
    return K;
}

__device__ double sb_alpha(const SbKnot& K, double freq) {
    const double PI = kPi;
    const double sigma = 5.0 / sqrt(21.0);
    const double nu = K.nu_f * freq;
    const double chi = 3.0 * K.nn * nu / 4.0;
    const double cchi = 2.36 * chi;
    const double nu2 = nu * nu, cchi2 = cchi * cchi, sc = sigma * cchi;
    const double r1 = sqrt(1 + nu2);
    const double kf = 2 * PI * freq / K.c;
    const double a_cl = kf * sqrt(0.5 * (r1 - 1) * (1 + cchi2) / ((1 + nu2) * (1 + sc * sc)));
    const double a_rot = kf * K.x_on * ((sigma * sigma - 1) * chi / (2 * sigma)) *
                         sqrt(0.5 * (r1 + 1) / ((1 + nu2) * (1 + cchi2)));
    const double a_diff = 0.003 * a_cl;
    double a_vib = 0.0;
#pragma unroll
    for (int m = 0; m < 4; m++) {
        const double q = freq / K.fv[m];
        a_vib = a_vib + K.am[m] * ((2 * (freq * freq) / K.fv[m]) / (1 + q * q));
    }
    return a_cl + a_rot + a_diff + a_vib;
}

// Knot-level fields of every group and their Steffen coefficients in one
// launch: c_eff per azimuth (and, for wide-angle rows, the wind component and
// c0), absorption per frequency.  A block takes kKnotStep intervals of one
// field, or of kSbFreqs frequencies' absorptions (the knot's part is evaluated
// once), with the knots around them in shared memory.  Bound by launch latency:
// 32 groups of one problem took 128 launches for this (with their uploads and
// allocations 1.9 ms a solve, now 0.1).
constexpr int kSbFreqs = 8;  // frequencies of an absorption block
constexpr int kKnotThreads = 128, kKnotStep = kKnotThreads - 3;

__global__ void __launch_bounds__(kKnotThreads) k_knots(const GroupDesc* __restrict__ desc, int tiles) {
    __shared__ double ys[kKnotThreads];
    const GroupDesc& G = desc[blockIdx.z];
    const int n = G.nk, t = threadIdx.x, k0 = (blockIdx.x % tiles) * kKnotStep - 1;
    if (k0 + 1 >= n - 1) return;
    int row = blockIdx.x / tiles;
    const int k = min(max(k0 + t, 0), n - 1);
    const bool own = k0 + t == k && ((t >= 1 && t <= kKnotStep) || k == n - 1);
    // one field: its value v at this thread's knot, y and coefficients to global
    auto field = [&](double v, double* __restrict__ y, double* __restrict__ coef) {
        ys[t] = v;
        if (own) y[k] = v;
        __syncthreads();
        const int i = k0 + t;
        if (t >= 1 && t <= kKnotStep && i < n - 1) steffen_coef(n, G.zk, ys - k0, i, coef + 4 * i);
        __syncthreads();
    };
    if (row < G.n_az * (G.wide ? 2 : 1)) {
        const int a = row % G.n_az;
        const double az_rad = G.az[a] * kPi / 180.0;
        const double dir = G.wd[k] * kPi / 180.0;
        const double wc = G.ws[k] * cos(dir - az_rad);
        if (row < G.n_az) field(wc + G.c0[k], G.ceffk + (size_t)a * n, G.ceffc + (size_t)a * 4 * (n - 1));
        else field(wc, G.wck + (size_t)a * n, G.wcc + (size_t)a * 4 * (n - 1));
        return;
    }
    row -= G.n_az * (G.wide ? 2 : 1);
    if (G.wide) {
        if (row == 0) {
            field(G.c0[k], G.c0k, G.c0c);
            return;
        }
        --row;
    }
    const int f0 = row * kSbFreqs, f1 = min(G.n_f, f0 + kSbFreqs);
    if (f0 >= f1) return;
    SbKnot K;
    if (!G.attn) K = sb_knot(G.zk[k] * 0.001, G.t[k], G.p[k], G.rho[k]);
    for (int f = f0; f < f1; ++f)
        field(G.attn ? G.attn[k] : sb_alpha(K, G.freqs[f]), G.alpha + (size_t)f * n, G.alphac + (size_t)f * 4 * (n - 1));
}

// rho at the source and receiver rows and the weights w_i = ((omega / c_T)
// alpha_i) 2 of doPerturb, c_T = sqrt(1.4 P / rho), of every group.  A thread
// takes one grid point and kAwFreqs frequencies: one knot search, every value
// by spline_get's expression; padding rows are zero.
constexpr int kAwFreqs = 16;

__global__ void __launch_bounds__(256) k_grid_fields(const GroupDesc* __restrict__ desc) {
    const GroupDesc& G = desc[blockIdx.z];
    const int i = blockIdx.x * blockDim.x + threadIdx.x, nk = G.nk;
    const int f0 = blockIdx.y * kAwFreqs, f1 = min(G.n_f, f0 + kAwFreqs);
    if (i >= G.nz_pad || f0 >= f1) return;
    if (i >= G.nz) {
        for (int f = f0; f < f1; ++f) G.w[(size_t)f * G.nz_pad + i] = 0.0;
        return;
    }
    const double h = G.z_min + i * G.dz_grid;
    int where = 0, kn = 0;  // 0 inside the knots, 1 above, 2 below
    double t = 0.0;
    if (h > G.zk[nk - 1]) {
        where = 1;
    } else if (h < G.zk[0]) {
        where = 2;
    } else {
        kn = knot_search(nk, G.zk, h);
        t = h - G.zk[kn];
    }
    auto at = [&](const double* __restrict__ y, const double* __restrict__ coef) {
        if (where == 1) return y[nk - 1];
        if (where == 2) return y[0];
        const double* c = coef + 4 * kn;
        return c[3] + t * (c[2] + t * (c[1] + t * c[0]));
    };
    const double r = at(G.rho, G.rcoef), pv = at(G.p, G.pcoef);
    if (blockIdx.y == 0) {
        if (i == G.isrc) G.rho_pair[0] = r;
        if (i == G.ircv) G.rho_pair[1] = r;
    }
    const double ct = sqrt(1.4 * pv / r);
    const double *__restrict__ al = G.alpha, *__restrict__ ac = G.alphac, *__restrict__ fr = G.freqs;
    double* __restrict__ w = G.w + i;
    const int wstride = G.nz_pad;
#pragma unroll 4
    for (int f = f0; f < f1; ++f) {
        const double a = at(al + (size_t)f * nk, ac + (size_t)f * 4 * (nk - 1));
        const double omega = 2 * kPi * fr[f];
        w[(size_t)f * wstride] = ((omega / ct) * a) * 2;
    }
}

// ===========================================================================
// K1: matrix build
// ===========================================================================
__device__ __forceinline__ double warp_min(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmin(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}
__device__ __forceinline__ double warp_max(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}

// One thread per (azimuth, grid point) and kBmFreqs frequencies of the group:
// c_eff is sampled once and every problem's entries use the same expressions.
constexpr int kBmFreqs = 16;

__global__ void __launch_bounds__(256) k_build_matrix(const GroupDesc* __restrict__ desc, int tiles) {
    const GroupDesc& G = desc[blockIdx.z];
    const int a = blockIdx.y;
    const int i = (blockIdx.x % tiles) * blockDim.x + threadIdx.x;
    const int n_f = G.n_f, n_az = G.n_az, nk = G.nk, nz = G.nz, nz_pad = G.nz_pad;
    const int f0 = (blockIdx.x / tiles) * kBmFreqs, f1 = min(n_f, f0 + kBmFreqs);
    if (a >= n_az || f0 >= f1 || (blockIdx.x % tiles) * blockDim.x >= nz_pad) return;
    const double* __restrict__ zk = G.zk;
    const double* __restrict__ ck = G.ceffk + (size_t)a * nk;
    const double* __restrict__ cc = G.ceffc + (size_t)a * 4 * (nk - 1);
    const double z_min = G.z_min, dz_grid = G.dz_grid, dz = G.dz, admittance = G.admittance;
    ProblemInfo* __restrict__ pinfo = G.pinfo;
    double *__restrict__ s = G.s, *__restrict__ kz2 = G.kz2, *__restrict__ g = G.gs;
    const double h2 = dz * dz;
    const double bnd = (1. / (dz * admittance + 1)) / (dz * dz);
    double cmin = 1e300, cmax = -1e300;
    const int top = nz - (nz / 10);
    const int itop = top + 1 < nz ? top + 1 : nz - 1;
    if (i < nz) {
        const double c = spline_get(nk, zk, ck, cc, z_min + i * dz_grid);
        // last row of the assembled matrix repeats diag[nz-2] (EigenEngine.cpp:59-71)
        const double c2 = i < nz - 1 ? c : spline_get(nk, zk, ck, cc, z_min + (nz - 2) * dz_grid);
        cmin = cmax = c;
        for (int f = f0; f < f1; ++f) {
            const int p = f * n_az + a;
            const double omega = pinfo[p].omega;
            double t = omega / c;
            double d = t * t;
            if (kz2) kz2[(size_t)p * nz_pad + i] = d;
            if (g) g[(size_t)p * nz_pad + i] = 1.0 / (c * c);
            double sd;
            if (i < nz - 1) {
                sd = (i == 0) ? (bnd + d) : d;
            } else {
                double t2 = omega / c2;
                sd = t2 * t2;
                if (nz - 2 == 0) sd = bnd + sd;
            }
            s[(size_t)p * nz_pad + i] = sd * h2 - 2.0;
            if (i == 0) pinfo[p].ceff_grnd = c;
            if (i == itop) pinfo[p].ceff_top = c;
        }
    } else if (i < nz_pad) {
        for (int f = f0; f < f1; ++f) {
            const int p = f * n_az + a;
            s[(size_t)p * nz_pad + i] = 0.0;
            if (g) g[(size_t)p * nz_pad + i] = 0.0;
        }
    }
    cmin = warp_min(cmin);
    cmax = warp_max(cmax);
    __shared__ double smin[8], smax[8];
    int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (lane == 0) {
        smin[wid] = cmin;
        smax[wid] = cmax;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int k = 1; k < 8; ++k) {
            cmin = fmin(cmin, smin[k]);
            cmax = fmax(cmax, smax[k]);
        }
        cmin = fmin(cmin, smin[0]);
        cmax = fmax(cmax, smax[0]);
        if (cmin < 1e300) {
            for (int f = f0; f < f1; ++f) {
                const int p = f * n_az + a;
                atomicMin(&pinfo[p].ceffmin_bits, (unsigned long long)__double_as_longlong(cmin));
                atomicMax(&pinfo[p].ceffmax_bits, (unsigned long long)__double_as_longlong(cmax));
            }
        }
    }
}

int launch_groups(cudaStream_t st, const GroupDesc* desc, const GroupDims& d) {
    int n = 0;
    for (int g0 = 0; g0 < d.n; g0 += 65535, n += 2) {  // grid.z limit
        const int m = std::min(65535, d.n - g0);
        const int tiles = (d.nk - 1 + kKnotStep - 1) / kKnotStep, rows = d.n_fields + (d.n_f + kSbFreqs - 1) / kSbFreqs;
        k_knots<<<dim3(tiles * rows, 1, m), kKnotThreads, 0, st>>>(desc + g0, tiles);
        k_grid_fields<<<dim3((d.nz_pad + 255) / 256, (d.n_f + kAwFreqs - 1) / kAwFreqs, m), 256, 0, st>>>(desc + g0);
    }
    return n;
}

int launch_build_matrix(cudaStream_t st, const GroupDesc* desc, const GroupDims& d) {
    const int tiles = (d.nz_pad + 255) / 256;
    int n = 0;
    for (int g0 = 0; g0 < d.n; g0 += 65535, ++n)
        k_build_matrix<<<dim3(tiles * ((d.n_f + kBmFreqs - 1) / kBmFreqs), d.n_az, std::min(65535, d.n - g0)), 256, 0,
                         st>>>(desc + g0, tiles);
    return n;
}

// ===========================================================================
// K2: wavenumber window.  The reference walks trial values kk_j = k_gnd^2 + j
// dkk (built by repeated additions) and, for each, adds dz sqrt|kk_j - kz2_i|
// up the grid until a row comes within dkk of kk_j; the first trial whose
// integral reaches 10 sets k_max.
//
// k_wkb: one warp per (problem, trial), 128 rows a step (four coalesced loads
// in flight per lane).  As one thread per trial the walk was a serial chain of
// load, square root and add over up to nz rows: 1500 us on 20000 rows at 0.1 Hz
// (no trial reaches 10 there) and 4700 us on the 360 mixed grids of a 45-azimuth
// sweep.  The lanes' partial sums differ from the row-by-row sum by rounding
// only (< 1e-11 here); a sum within 1e-9 of the threshold is redone row by row,
// so the chosen trial is the sequential walk's.  A warp stops once its sum is
// past the threshold (the terms are not negative) or an earlier trial has hit.
// ===========================================================================
constexpr int kWkbTrials = 128;  // the walk has at most 101 trials
constexpr int kWkbWarps = 4;     // trials per CTA

// the trial grid of one problem; false: the walk is not taken
__device__ __forceinline__ bool wkb_trials(const ProblemInfo& pi, double& kk0, double& dkk, double& kmf2) {
    const double k_max_full = pi.omega / __longlong_as_double((long long)pi.ceffmin_bits);
    const double k_gnd = pi.omega / pi.ceff_grnd;
    kmf2 = k_max_full * k_max_full;
    dkk = (kmf2 - k_gnd * k_gnd) / 100.0;
    kk0 = k_gnd * k_gnd;
    return dkk > 1.0e-10;
}

__global__ void __launch_bounds__(kWkbWarps * 32) k_wkb(ProblemInfo* __restrict__ pinfo,
                                                        const double* __restrict__ kz2) {
    const int p = blockIdx.y, lane = threadIdx.x & 31;
    const int j = blockIdx.x * kWkbWarps + (threadIdx.x >> 5);
    const ProblemInfo& pi = pinfo[p];
    volatile int* hit = &pinfo[p].wkb_trial;
    double kk0, dkk, kmf2;
    if (!wkb_trials(pi, kk0, dkk, kmf2)) return;
    double kk = kk0;
    for (int q = 0; q < j; ++q) kk = kk + dkk;
    if (!(kk < kmf2)) {  // past the last trial: the walk ends here at the latest
        if (lane == 0) atomicMin(&pinfo[p].wkb_trial, j);
        return;
    }
    const double* row = kz2 + pi.s_off;
    const int nz = pi.nz;
    const double dz = pi.dz;
    constexpr double kGoal = 10.0, kSlack = 1.0e-9;
    double part = 0.0;
    int n = nz;  // rows of the integral
    for (int i0 = 0; i0 < nz; i0 += 128) {
        double v[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int i = i0 + 32 * u + lane;
            v[u] = i < nz ? row[i] : kk;
        }
        bool stop = false;
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const double term = fabs(kk - v[u]);
            const unsigned low = __ballot_sync(0xffffffffu, !(term > dkk));
            const int last = low ? __ffs(low) - 1 : 31;  // the first row within dkk still counts
            const int i = i0 + 32 * u + lane;
            if (!stop && lane <= last && i < nz) part = part + dz * sqrt(term);
            if (!stop && low) {
                n = min(nz, i0 + 32 * u + last + 1);
                stop = true;
            }
        }
        if (stop) break;
        if ((i0 & 511) == 384) {  // every 512 rows
            double s = part;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
            if (s >= kGoal + kSlack) {
                part = s;  // decided: the rows above only add
                n = -1;
                break;
            }
            const int h = __shfl_sync(0xffffffffu, *hit, 0);
            if (h <= j) return;
        }
    }
    bool reach = n < 0;
    if (!reach) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) part += __shfl_xor_sync(0xffffffffu, part, o);
        reach = part >= kGoal;
        if (fabs(part - kGoal) <= kSlack) {  // too close to call: the walk row by row
            double integral = 0.0;
            for (int i = 0; i < n; ++i) integral = integral + dz * sqrt(fabs(kk - row[i]));
            reach = integral >= kGoal;
        }
    }
    if (reach && lane == 0) atomicMin(&pinfo[p].wkb_trial, j);
}

__global__ void k_window(int P, ProblemInfo* __restrict__ pinfo, int wkb, int wvnum, double c_min, double c_max,
                         unsigned* err) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= P) return;
    const ProblemInfo& pi = pinfo[p];
    const double dz = pi.dz;
    const double omega = pi.omega;
    const double ceffmin = __longlong_as_double((long long)pi.ceffmin_bits);
    double k_max;
    if (wkb) {
        double kk, dkk, kmf2;
        if (wkb_trials(pi, kk, dkk, kmf2)) {
            int jsel = pi.wkb_trial;
            if (jsel >= kWkbTrials) {
                atomicOr(err, kErrWkb);
                jsel = kWkbTrials - 1;
            }
            for (int q = 0; q < jsel; ++q) kk = kk + dkk;
        }
        k_max = sqrt(kk);
    } else {
        k_max = omega / ceffmin;
    }
    double k_min = omega / pi.ceff_top;
    if (wkb && k_max < k_min) k_max = omega / ceffmin;
    if (wvnum) {
        k_min = 2 * kPi * pi.freq / c_max;
        k_max = 2 * kPi * pi.freq / c_min;
    }
    const double h2 = dz * dz;
    const double lo = (k_min * k_min) * h2, hi = (k_max * k_max) * h2;
    pinfo[p].k_min = k_min;
    pinfo[p].k_max = k_max;
    pinfo[p].lo = lo;
    pinfo[p].hi = hi;
    pinfo[p].used_wkb = wkb ? 1 : 0;
    pinfo[p].n_scan = kScanDefault;
    pinfo[p].m_est = -1.f;
}

int launch_window(cudaStream_t st, int P, ProblemInfo* pinfo, const double* kz2, int wkb, int wvnum,
                  double c_min, double c_max, unsigned* err) {
    int n = 1;
    if (wkb) {
        for (int p0 = 0; p0 < P; p0 += 65535) {  // grid.y limit
            dim3 grid(kWkbTrials / kWkbWarps, P - p0 < 65535 ? P - p0 : 65535);
            k_wkb<<<grid, kWkbWarps * 32, 0, st>>>(pinfo + p0, kz2);
            ++n;
        }
    }
    k_window<<<(P + 63) / 64, 64, 0, st>>>(P, pinfo, wkb, wvnum, c_min, c_max, err);
    return n;
}

// ===========================================================================
// FP64 FMA throughput probe (denominator of the bisection roofline)
// ===========================================================================
__global__ void k_fp64_probe(int n_iter, double* out) {
    double a[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) a[k] = 1.0 + 1e-9 * (threadIdx.x + k);
    const double m = 0.999999999, c = 1e-12;
    for (int it = 0; it < n_iter; ++it) {
#pragma unroll
        for (int k = 0; k < 8; ++k) a[k] = fma(a[k], m, c);
    }
    double t = 0.0;
#pragma unroll
    for (int k = 0; k < 8; ++k) t += a[k];
    if (t == 12345.0) out[0] = t;  // practically never: keeps the chains live
}

int launch_fp64_probe(cudaStream_t st, int grid, int block, int n_iter, double* out) {
    k_fp64_probe<<<grid, block, 0, st>>>(n_iter, out);
    return 1;
}

// ===========================================================================
// K4s: mode values by twisted factorisation on the rows themselves, for the
// calls that keep their memory in the library's image (noalloc.cu; everything
// else runs on panel.cu).  One eigenvalue per lane, one work item (<= 32
// eigenvalues of a problem) per warp.  For S - mu with unit off-diagonals the
// forward solution of rows 0..i-1 is z_i = (-1)^i p_{i-1} and the backward
// solution of rows i+1..n-1 is z_i = (-1)^(n-1-i) q_{i+1} (q_n = 1); with the
// twist r maximising |p_{r-1} q_{r+1}|,
//   z_i = (-1)^i p_{i-1} q_{r+1} (i <= r),  z_i = (-1)^i p_{r-1} q_{i+1} (i >= r)
// solves (S - mu) z = gamma_r e_r: one inverse-iteration step from e_r.  Each
// warp streams the diagonal s and the weights w through its own TMA ring, so
// warps never wait on each other.
// ===========================================================================
constexpr int kEvC = 256;     // doubles per chunk and array
constexpr int kEvB = 3;       // ring slots per warp
constexpr int kEvWarps = 4;   // warps per CTA

struct EvRing {
    double* s;       // [kEvB][kEvC]
    double* w;
    uint64_t* bars;  // [kEvB]
    unsigned loads;
};

// chunk c of the rows and of w
__device__ __forceinline__ void evr_issue(EvRing& r, unsigned k, int c, const double* sp, const double* wp) {
    const int slot = k % kEvB;
    mbar_expect_tx(&r.bars[slot], 2 * kEvC * 8);
    tma_load_1d(r.s + slot * kEvC, sp + (size_t)c * kEvC, kEvC * 8, &r.bars[slot]);
    tma_load_1d(r.w + slot * kEvC, wp + (size_t)c * kEvC, kEvC * 8, &r.bars[slot]);
}

// One item: two passes and a twist chosen among the coarse rows c = 0, kCk, 2 kCk, ...
//  pass 1  backward recurrence q with the sums T = sum_{i > c} q_{i+1}^2 (1, w)
//          over the rows above; at every coarse row c the slot keeps q_{c+1}, its
//          exponent and T;
//  pass 2  forward recurrence p with the sums A = sum_{i <= c} p_{i-1}^2 (1, w);
//          at each coarse row the twist key |p_{c-1} q_{c+1}| (proportional
//          to |z_c|) picks the best twist r so far.
// Then sum z^2 / z_r^2 = A_r / p_{r-1}^2 + T_r / q_{r+1}^2 (each in its own
// recurrence's scale).  Restricting r to the coarse rows costs at most the
// ratio of the largest |z_i| to the largest |z_c| in residual (one
// inverse-iteration step from e_r, residual |gamma_r| / |z|): measured on
// the 20000- to 100000-point grids of 0.05-2 Hz, at most 1.06 for every
// mode with 64-row spacing and 1.8 with 256.
constexpr int kCk = kCkRows;  // rows between coarse twist candidates
static_assert(kEvC % kCk == 0 && kCk % kBlk == 0, "coarse rows start blocks and chunks");

__device__ __forceinline__ void eigvec_item(const EigvecArgs& A, const WorkItem w, EvRing& R, double* ckq, double* ckt,
                                            int* cke) {
    const int lane = threadIdx.x & 31;
    const ProblemInfo pi = A.pinfo[w.problem];
    const int nz = pi.nz;
    const int nch = (nz + kEvC - 1) / kEvC;
    const int isrc = pi.isrc, ircv = pi.ircv;
    const double* sp = A.s + pi.s_off;
    const double* wp = A.w + pi.w_off;
    const bool active = lane < w.m;
    const double mu = active ? A.mu[pi.off + w.j0 + lane] : pi.lo;

    // ---------------- pass 1: backward recurrence, coarse checkpoints ----------
    double qs = 1.0, qrc = 1.0;  // q_{isrc+1}, q_{ircv+1}
    int Eqs = 0, Eqrc = 0;
    {
        const unsigned base = R.loads;
        if (lane == 0)
            for (int o = 0; o < nch && o < kEvB; ++o) evr_issue(R, base + o, nch - 1 - o, sp, wp);
        __syncwarp();
        double q1 = 1.0, q2 = 0.0;  // q_{i+1}, q_{i+2} before row i; q_n = 1, q_{n+1} = 0
        double Tn = 0.0, Tw = 0.0;
        int E = 0;
        for (int o = 0; o < nch; ++o) {
            const int c = nch - 1 - o;
            const unsigned k = base + o;
            const int slot = k % kEvB;
            mbar_wait_bounded(&R.bars[slot], (k / kEvB) & 1u, A.err);
            const double* sb = R.s + slot * kEvC;
            const double* wb = R.w + slot * kEvC;
            const int valid = min(kEvC, nz - c * kEvC);
            auto row = [&](int li) {
                const double qq = q1 * q1;
                Tn = Tn + qq;
                Tw = fma(qq, wb[li], Tw);
                const double qi = fma(sb[li] - mu, q1, -q2);
                q2 = q1;
                q1 = qi;
            };
            auto store = [&](int gbase) {
                const size_t ci = (size_t)(gbase / kCk) * 32 + lane;
                ckq[ci] = q1;
                cke[ci] = E;
                ckt[ci * 2] = Tn;
                ckt[ci * 2 + 1] = Tw;
            };
            for (int lb = ((valid - 1) / kBlk) * kBlk; lb >= 0; lb -= kBlk) {
                const int gbase = c * kEvC + lb;
                const bool coarse = (gbase % kCk) == 0;
                const bool special = lb + kBlk > valid || (isrc >= gbase && isrc < gbase + kBlk) ||
                                     (ircv >= gbase && ircv < gbase + kBlk);
                if (!special) {
#pragma unroll
                    for (int u = kBlk - 1; u >= 0; --u) {
                        if (u == 0 && coarse) store(gbase);
                        row(lb + u);
                    }
                } else {
                    for (int u = min(kBlk, valid - lb) - 1; u >= 0; --u) {
                        const int i = gbase + u;
                        if (i == isrc) {
                            qs = q1;
                            Eqs = E;
                        }
                        if (i == ircv) {
                            qrc = q1;
                            Eqrc = E;
                        }
                        if (u == 0 && coarse) store(gbase);
                        row(lb + u);
                    }
                }
                const int sft = grow_shift(q1, q2);
                if (sft) {
                    const double sc = pow2(-sft), sc2 = pow2(-2 * sft);
                    q1 *= sc;
                    q2 *= sc;
                    Tn *= sc2;
                    Tw *= sc2;
                    E += sft;
                }
            }
            __syncwarp();
            if (lane == 0 && o + kEvB < nch) {
                fence_proxy_async();
                evr_issue(R, base + o + kEvB, nch - 1 - (o + kEvB), sp, wp);
            }
        }
        R.loads = base + nch;
    }
    __syncwarp();  // the slot's checkpoints written by every lane before they are read

    // ---------------- pass 2: forward recurrence, coarse twist ----------------
    double pm2 = 0.0, pm1 = 1.0;  // p_{i-2}, p_{i-1}
    int Ep = 0;
    double An = 0.0, Aw = 0.0;
    double best = -INFINITY;
    int r = 0, Epr = 0, Eqr = 0;
    double Anr = 1.0, Awr = 0.0, pr = 1.0, qr = 1.0, Tnr = 0.0, Twr = 0.0;
    double ps = 1.0, prc = 1.0;  // p_{isrc-1}, p_{ircv-1}
    int Eps = 0, Eprc = 0;
    {
        const unsigned base = R.loads;
        if (lane == 0)
            for (int c = 0; c < nch && c < kEvB; ++c) evr_issue(R, base + c, c, sp, wp);
        __syncwarp();
        // checkpoint of the next coarse row, loaded one candidate ahead
        double nq = ckq[lane], nt0 = ckt[lane * 2], nt1 = ckt[lane * 2 + 1];
        int nE = cke[lane];
        const int n_coarse = (nz + kCk - 1) / kCk;
        for (int c = 0; c < nch; ++c) {
            const unsigned k = base + c;
            const int slot = k % kEvB;
            mbar_wait_bounded(&R.bars[slot], (k / kEvB) & 1u, A.err);
            const double* sb = R.s + slot * kEvC;
            const double* wb = R.w + slot * kEvC;
            const int valid = min(kEvC, nz - c * kEvC);
            auto row = [&](int li) {
                const double sq = pm1 * pm1;
                An = An + sq;
                Aw = fma(sq, wb[li], Aw);
            };
            auto step = [&](int li) {
                const double pn = fma(sb[li] - mu, pm1, -pm2);
                pm2 = pm1;
                pm1 = pn;
            };
            auto candidate = [&](int gbase) {
                // key log2 |p_{c-1} q_{c+1}| with both recurrences' exponents
                const double key = log2(fabs(pm1 * nq)) + (double)(Ep + nE);
                if (key > best) {
                    best = key;
                    r = gbase;
                    Anr = An;
                    Awr = Aw;
                    pr = pm1;
                    Epr = Ep;
                    qr = nq;
                    Eqr = nE;
                    Tnr = nt0;
                    Twr = nt1;
                }
                const int kc = gbase / kCk + 1;
                if (kc < n_coarse) {
                    const size_t ci = (size_t)kc * 32 + lane;
                    nq = ckq[ci];
                    nE = cke[ci];
                    nt0 = ckt[ci * 2];
                    nt1 = ckt[ci * 2 + 1];
                }
            };
            for (int lb = 0; lb < valid; lb += kBlk) {
                const int gbase = c * kEvC + lb;
                const bool coarse = (gbase % kCk) == 0;
                const bool special = lb + kBlk > valid || (isrc >= gbase && isrc < gbase + kBlk) ||
                                     (ircv >= gbase && ircv < gbase + kBlk);
                if (!special) {
#pragma unroll
                    for (int u = 0; u < kBlk; ++u) {
                        row(lb + u);
                        if (u == 0 && coarse) candidate(gbase);
                        step(lb + u);
                    }
                } else {
                    const int nrow = min(kBlk, valid - lb);
                    for (int u = 0; u < nrow; ++u) {
                        const int i = gbase + u;
                        if (i == isrc) {
                            ps = pm1;
                            Eps = Ep;
                        }
                        if (i == ircv) {
                            prc = pm1;
                            Eprc = Ep;
                        }
                        row(lb + u);
                        if (u == 0 && coarse) candidate(gbase);
                        step(lb + u);
                    }
                }
                const int sft = grow_shift(pm1, pm2);
                if (sft) {
                    const double sc = pow2(-sft), sc2 = pow2(-2 * sft);
                    pm1 *= sc;
                    pm2 *= sc;
                    An *= sc2;
                    Aw *= sc2;
                    Ep += sft;
                }
            }
            __syncwarp();
            if (lane == 0 && c + kEvB < nch) {
                fence_proxy_async();
                evr_issue(R, base + c + kEvB, c + kEvB, sp, wp);
            }
        }
        R.loads = base + nch;
    }
    // ---------------- combine ----------------------------------------
    const double ip2 = 1.0 / (pr * pr), iq2 = 1.0 / (qr * qr);
    const double nrm = Anr * ip2 + Tnr * iq2;
    const double scale = 1.0 / sqrt(nrm * pi.dz);
    double zs = (isrc <= r) ? (ps / pr) * pow2(Eps - Epr) : (qs / qr) * pow2(Eqs - Eqr);
    double zr = (ircv <= r) ? (prc / pr) * pow2(Eprc - Epr) : (qrc / qr) * pow2(Eqrc - Eqr);
    if ((isrc - r) & 1) zs = -zs;
    if ((ircv - r) & 1) zr = -zr;
    const double absorption = (Awr * ip2 + Twr * iq2) / nrm;
    const double ks = sqrt(mu / (pi.dz * pi.dz));
    const double kk = ks * ks;
    const auto kp = csqrt_principal(kk, absorption);
    if (active) {
        const int o = pi.off + w.j0 + lane;
        A.kr[o] = kp.real();
        A.ki[o] = kp.imag();
        A.vs[o] = zs * scale;
        A.vr[o] = zr * scale;
        if (A.vg) A.vg[o] = 0.0;
    }
}

__global__ void __launch_bounds__(kEvWarps * 32, 4) k_eigvec(EigvecArgs A) {
    extern __shared__ __align__(128) unsigned char smem_raw[];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    double* wb0 = reinterpret_cast<double*>(smem_raw) + (size_t)wid * kEvB * 2 * kEvC;
    EvRing R;
    R.s = wb0;
    R.w = wb0 + kEvB * kEvC;
    R.bars = reinterpret_cast<uint64_t*>(smem_raw + (size_t)kEvWarps * kEvB * 2 * kEvC * 8) + wid * kEvB;
    R.loads = 0;
    if (lane == 0) {
        for (int k = 0; k < kEvB; ++k) mbar_init(&R.bars[k], 1);
        fence_mbar_init();
    }
    __syncwarp();
    const size_t gw = (size_t)blockIdx.x * kEvWarps + wid;
    double* ck1 = A.ck_q1 + gw * A.ck_slot_stride;
    double* ck2 = A.ck_q2 + gw * A.ck_slot_stride;
    int* cke = A.ck_e + gw * A.ck_slot_stride;
    // static round-robin over the grid's warps
    for (int it = blockIdx.x * kEvWarps + wid; it < A.n_items; it += gridDim.x * kEvWarps)
        eigvec_item(A, A.items[it], R, ck1, ck2, cke);
}

int launch_eigvec(cudaStream_t st, int grid, const EigvecArgs& a) {
    const size_t sm = (size_t)kEvWarps * (kEvB * 2 * kEvC * 8 + kEvB * 8);
    cudaFuncSetAttribute(k_eigvec, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    k_eigvec<<<grid, kEvWarps * 32, sm, st>>>(a);
    return 1;
}

// ===========================================================================
// K5: 1-D transmission loss.  One CTA per (problem, chunk of kTlRanges
// ranges), so a batch's problems (2 to ~300 modes each) spread over many
// small CTAs instead of one CTA per problem.  Modes are staged in shared
// memory in tiles: per mode the amplitude c = V_s V_r / sqrt(k) (principal
// root), V_s^2 V_r^2 / |k| for the incoherent sum, the step w = e^{(i k_r -
// k_i) dr}, the chunk's first phase e^{(i k_r - k_i) r_b} and the powers
// w4^(2^b), w4 = e^{(i k_r - k_i) kTlRun dr} (each from the one before by
// squaring: the relative error grows to about 2^6 ulps).  A thread covers kTlRun
// consecutive ranges: its first phase is the chunk's times the powers of
// its index's set bits, the next ones follow by w.  Each tile is summed apart
// and the tiles in order, so that they can also run on blocks of their own.
// FP64 issue: 11 fused instructions a range and mode (19 when products and sums
// were apart: 45 azimuths x 8 frequencies 434 -> 326 us, 256 frequencies 110 ->
// 93).
// ===========================================================================
constexpr int kTlRun = 4;      // consecutive ranges per thread
constexpr int kTlThreads = 64;
constexpr int kTlBits = 6;     // thread index bits (kTlThreads = 2^kTlBits)
constexpr int kTlRanges = kTlThreads * kTlRun;
constexpr int kTlTile = 64;    // modes per shared-memory tile, summed apart
static_assert(kTlThreads == 1 << kTlBits, "the powers cover every thread index");

// the pressure and the incoherent sum at range i from the sums over modes
__device__ __forceinline__ void tl1d_store(int i, double dr, double sre, double sim, double sinc, size_t o,
                                           double* __restrict__ re, double* __restrict__ im,
                                           double* __restrict__ incoh) {
    // 1000 * 4 pi i e^{-i pi/4} / sqrt(8 pi) / sqrt(r)
    const double ang = kPi * 0.25;
    const double r = (i + 1) * dr;
    const double c0 = 1000.0 * 4 * kPi / sqrt(8.0 * kPi) / sqrt(r);
    const double fr = c0 * sin(ang), fi = c0 * cos(ang);
    re[o] = fr * sre - fi * sim;
    im[o] = fr * sim + fi * sre;
    incoh[o] = 1000.0 * 4 * kPi * sqrt(sinc) * sqrt(1. / 8. / kPi / r);
}

// kSplit: one tile of modes per blockIdx.z, its sums to part [problem][tile][3][nr]
template <bool kSplit>
__global__ void __launch_bounds__(kTlThreads) k_tl1d(const ProblemInfo* __restrict__ pinfo,
                                                     const double* __restrict__ kr, const double* __restrict__ ki,
                                                     const double* __restrict__ vs, const double* __restrict__ vr,
                                                     int nr, double dr, int lossless, double* __restrict__ re,
                                                     double* __restrict__ im, double* __restrict__ incoh,
                                                     double* __restrict__ part) {
    const int p = blockIdx.y;
    const int i0 = blockIdx.x * kTlRanges + threadIdx.x * kTlRun;  // first range of this thread
    const int M = pinfo[p].M, off = pinfo[p].off;
    if (kSplit && (int)blockIdx.z * kTlTile >= M) return;
    __shared__ double2 m_c[kTlTile], m_w[kTlTile], m_b[kTlTile];
    __shared__ double m_inc[kTlTile];
    __shared__ double2 m_pw[kTlBits][kTlTile];
    const double rb = ((double)blockIdx.x * kTlRanges + 1.0) * dr;  // the chunk's first range
    double tre[kTlRun], tim[kTlRun], tinc[kTlRun];  // over the tiles, in order
#pragma unroll
    for (int j = 0; j < kTlRun; ++j) tre[j] = tim[j] = tinc[j] = 0.0;
    for (int m0 = kSplit ? blockIdx.z * kTlTile : 0; m0 < M; m0 += kSplit ? gridDim.z * kTlTile : kTlTile) {
        double sre[kTlRun], sim[kTlRun], sinc[kTlRun];
#pragma unroll
        for (int j = 0; j < kTlRun; ++j) sre[j] = sim[j] = sinc[j] = 0.0;
        __syncthreads();
        for (int t = threadIdx.x; t < kTlTile && m0 + t < M; t += kTlThreads) {
            const int o = off + m0 + t;
            const double a = kr[o], b = lossless ? 0.0 : ki[o];
            // V_s V_r / sqrt(k): principal root of k, then the reciprocal
            const auto sk = csqrt_principal(a, b);
            const double den = sk.real() * sk.real() + sk.imag() * sk.imag();
            const double vv = vs[o] * vr[o];
            m_c[t] = make_double2(vv * sk.real() / den, -vv * sk.imag() / den);
            m_inc[t] = (vv * vv) * (lossless ? 1.0 / a : 1.0 / hypot(a, b));
            double sn, cs;
            sincos(a * dr, &sn, &cs);
            const double w = exp(-b * dr);
            m_w[t] = make_double2(w * cs, w * sn);
            sincos(a * rb, &sn, &cs);
            const double wb = exp(-b * rb);
            m_b[t] = make_double2(wb * cs, wb * sn);
            const double x = (double)kTlRun * dr;
            sincos(a * x, &sn, &cs);
            const double wp = exp(-b * x);
            double qr = wp * cs, qi = wp * sn;
#pragma unroll
            for (int bit = 0; bit < kTlBits; ++bit) {
                m_pw[bit][t] = make_double2(qr, qi);
                const double nq = qr * qr - qi * qi;
                qi = 2.0 * qr * qi;
                qr = nq;
            }
        }
        __syncthreads();
        const int mt = min(kTlTile, M - m0);
        if (i0 < nr) {
            for (int t = 0; t < mt; ++t) {
                // e^{i k r} at this thread's first range: the chunk's phase
                // times the powers of the thread index's set bits
                const double2 b0 = m_b[t];
                double er = b0.x, ei = b0.y;
#pragma unroll
                for (int bit = 0; bit < kTlBits; ++bit) {
                    if ((threadIdx.x >> bit) & 1) {
                        const double2 q = m_pw[bit][t];
                        const double nr_ = fma(er, q.x, -(ei * q.y));
                        ei = fma(er, q.y, ei * q.x);
                        er = nr_;
                    }
                }
                const double2 c = m_c[t], w = m_w[t];
                const double inc = m_inc[t];
#pragma unroll
                for (int j = 0; j < kTlRun; ++j) {
                    sre[j] = fma(er, c.x, fma(-ei, c.y, sre[j]));
                    sim[j] = fma(er, c.y, fma(ei, c.x, sim[j]));
                    sinc[j] = fma(inc, fma(er, er, ei * ei), sinc[j]);
                    const double nr_ = fma(er, w.x, -(ei * w.y));
                    ei = fma(er, w.y, ei * w.x);
                    er = nr_;
                }
            }
        }
#pragma unroll
        for (int j = 0; j < kTlRun; ++j) {
            tre[j] += sre[j];
            tim[j] += sim[j];
            tinc[j] += sinc[j];
        }
    }
#pragma unroll
    for (int j = 0; j < kTlRun; ++j) {
        const int i = i0 + j;
        if (i >= nr) break;
        if (kSplit) {
            double* o = part + ((size_t)p * gridDim.z + blockIdx.z) * 3 * nr + i;
            o[0] = tre[j];
            o[nr] = tim[j];
            o[2 * (size_t)nr] = tinc[j];
        } else {
            tl1d_store(i, dr, tre[j], tim[j], tinc[j], (size_t)p * nr + i, re, im, incoh);
        }
    }
}

// the tiles' sums in order
__global__ void __launch_bounds__(128) k_tl1d_sum(const ProblemInfo* __restrict__ pinfo, int tiles, int nr, double dr,
                                                  const double* __restrict__ part, double* __restrict__ re,
                                                  double* __restrict__ im, double* __restrict__ incoh) {
    const int p = blockIdx.y, i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nr) return;
    const int n = (pinfo[p].M + kTlTile - 1) / kTlTile;
    const double* q = part + (size_t)p * tiles * 3 * nr + i;
    double sre = 0.0, sim = 0.0, sinc = 0.0;
#pragma unroll 4
    for (int t = 0; t < n; ++t, q += 3 * (size_t)nr) {
        sre += q[0];
        sim += q[nr];
        sinc += q[2 * (size_t)nr];
    }
    tl1d_store(i, dr, sre, sim, sinc, (size_t)p * nr + i, re, im, incoh);
}

// Tiles of modes on blocks of their own while problems and ranges fill less
// than two blocks an SM: 1185 modes x 1000 ranges of one problem are 4 blocks
// of 245 us, or 76 of 18 us and 10 us for the sum of their parts.  The order of the
// sums is the same either way.
static size_t tl1d_parts(int P, int nr, int m_max) {
    return (size_t)P * ((m_max + kTlTile - 1) / kTlTile) * 3 * nr * 8;
}
static bool tl1d_split(int P, int nr, int m_max, int num_sms) {
    return m_max > kTlTile && (long long)P * ((nr + kTlRanges - 1) / kTlRanges) < 2ll * num_sms &&
           tl1d_parts(P, nr, m_max) <= (size_t)256 << 20;
}

size_t tl1d_scratch(int P, int nr, int m_max, int num_sms) {
    return tl1d_split(P, nr, m_max, num_sms) ? tl1d_parts(P, nr, m_max) : 0;
}

int launch_tl1d(cudaStream_t st, int P, const ProblemInfo* pinfo, const double* kr, const double* ki,
                const double* vs, const double* vr, int nr, double dr, int lossless, double* re, double* im,
                double* incoh, int m_max, int num_sms, double* scratch) {
    const int chunks = (nr + kTlRanges - 1) / kTlRanges;
    if (!tl1d_split(P, nr, m_max, num_sms)) {
        k_tl1d<false><<<dim3(chunks, P), kTlThreads, 0, st>>>(pinfo, kr, ki, vs, vr, nr, dr, lossless, re, im, incoh,
                                                              nullptr);
        return 1;
    }
    const int tiles = (m_max + kTlTile - 1) / kTlTile;
    k_tl1d<true><<<dim3(chunks, P, tiles), kTlThreads, 0, st>>>(pinfo, kr, ki, vs, vr, nr, dr, lossless, re, im, incoh,
                                                                scratch);
    k_tl1d_sum<<<dim3((nr + 127) / 128, P), 128, 0, st>>>(pinfo, tiles, nr, dr, scratch, re, im, incoh);
    return 2;
}

// ===========================================================================
// K5b: FP64 modal sum at many heights (2-D TL, receiver arrays):
//   P(r_i, z_j) = C(r_i) sum_m v_m(z_j) b_m(r_i),  b_m = v_m(z_s) e^{i k r} / sqrt(k),
// a real matrix product of [heights x modes] and [modes x 2 ranges], bound by
// the FP64 unit: it goes through the FP64 matrix instructions, whose operand
// traffic is a third of that of the same tile in FMAs (shared memory bound the
// latter).  A CTA takes 64 heights x 8 NB ranges and 32 modes a step, two
// buffers deep; its warps take 32 heights x 4 NB ranges of one half of each
// step, the two halves added at the end: with whole steps to four warps the
// last CTAs of a grid ran on their SM at a quarter of its rate.  b is not
// evaluated per point: k_sum_phases tabulates b_m every 32nd tile, e^{i k dr}
// of the 32 tiles up to there and of the ranges of one, and a CTA multiplies
// the three (8 instructions a value instead of sine, cosine and exponential
// each).  64 heights x 20000 ranges x 1185 modes: 3150 us with a thread per
// range walking the modes, 476 us as a 4 x 4 tile of FMAs, 340 us as this
// (165 us at the FP64 peak; the copies and products of a step take the rest).
// ===========================================================================

namespace {

constexpr int kSumJ = 64, kSumK = 32;  // heights of a CTA, modes of a step; it takes 8 NB ranges
constexpr int kSumMid = 32;  // tiles of a coarse phase
constexpr int kSumThreads = 256;
constexpr int kSumLd = 68;  // 4 mod 16 doubles: the fragments' 4 x 4 words of a half warp on different banks
constexpr size_t kSumSmem = 2 * kSumK * 2 * kSumLd * 8;
static_assert(kSumJ + 4 <= kSumLd && 2 * 8 * 4 + 4 <= kSumLd, "tile");
static_assert(kSumSmem / 8 >= 32 * 128, "the partial sums reuse the buffers");

// tab[row][m]: n0 coarse phases, kSumMid middle ones, n1 (ranges of a tile) fine ones
__global__ void __launch_bounds__(128) k_sum_phases(int M, const double* __restrict__ kr,
                                                    const double* __restrict__ ki,
                                                    const double* __restrict__ vs_src, double dr, int lossless,
                                                    int n0, int n1, double2* __restrict__ tab) {
    const int m = blockIdx.y * blockDim.x + threadIdx.x, t = blockIdx.x;
    if (m >= M) return;
    const double a = kr[m], b = lossless ? 0.0 : ki[m];
    double sn, cs;
    double2 v;
    if (t < n0) {
        const double r = ((double)t * (kSumMid * n1) + 1.0) * dr;
        const auto sk = csqrt_principal(a, b);
        const double den = sk.real() * sk.real() + sk.imag() * sk.imag();
        const double isr = sk.real() / den, isi = -sk.imag() / den;
        sincos(a * r, &sn, &cs);
        const double amp = exp(-b * r) * vs_src[m];
        const double er = amp * cs, ei = amp * sn;
        v = make_double2(er * isr - ei * isi, er * isi + ei * isr);
    } else {
        const double r = (double)(t < n0 + kSumMid ? (t - n0) * n1 : t - n0 - kSumMid) * dr;
        sincos(a * r, &sn, &cs);
        const double w = exp(-b * r);
        v = make_double2(w * cs, w * sn);
    }
    tab[(size_t)t * M + m] = v;
}

// C += A B of 16 x 8 by 8 x 8 on the FP64 matrix unit
__device__ __forceinline__ void mma_f64(double (&c)[4], const double (&a)[4], const double (&b)[2]) {
    asm("mma.sync.aligned.m16n8k8.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+d"(c[0]), "+d"(c[1]), "+d"(c[2]), "+d"(c[3])
        : "d"(a[0]), "d"(a[1]), "d"(a[2]), "d"(a[3]), "d"(b[0]), "d"(b[1]));
}

__device__ __forceinline__ double2 cmul(double2 a, double2 b) {
    return make_double2(fma(a.x, b.x, -(a.y * b.y)), fma(a.x, b.y, a.y * b.x));
}

// n bytes (8 or 16) to shared memory, zeros where off
template <int N>
__device__ __forceinline__ void copy_async(double* dst, const void* src, bool on) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;" ::"r"((unsigned)__cvta_generic_to_shared(dst)),
                 "l"(src), "n"(N), "r"(on ? N : 0));
}

template <int NB>
__global__ void __launch_bounds__(kSumThreads, 2) k_modal_sum(int M, const double2* __restrict__ tab, int n0,
                                                              const double* __restrict__ vec,
                                                              const int* __restrict__ rows, int nj, int nr,
                                                              double dr, long long sr, long long sj,
                                                              double* __restrict__ re, double* __restrict__ im) {
    constexpr int kSumR = 8 * NB;
    extern __shared__ __align__(16) double smem[];
    using Buf = double[kSumK][kSumLd];
    Buf* A = reinterpret_cast<Buf*>(smem);  // [2][mode][height]
    Buf* B = A + 2;                         // [2][mode][range, re | im]
    __shared__ long long roff[kSumJ];
    const int tile = blockIdx.x, j0 = blockIdx.y * kSumJ;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, q4 = lane & 3;
    const int jw = (warp & 1) * 32, cw = ((warp >> 1) & 1) * kSumR, kw = (warp >> 2) * (kSumK / 2);
    if (threadIdx.x < kSumJ) {
        const int j = j0 + threadIdx.x;
        roff[threadIdx.x] = j < nj ? (long long)rows[j] * M : -1;
    }
    __syncthreads();
    double acc[2][NB][4];
#pragma unroll
    for (int a = 0; a < 2; ++a)
#pragma unroll
        for (int b = 0; b < NB; ++b)
#pragma unroll
            for (int c = 0; c < 4; ++c) acc[a][b][c] = 0.0;
    // copies: a thread 8 heights and 4 ranges of one mode; 4 modes x 4 rows a
    // half warp, whose words fall on different banks
    const int cm = 8 * (warp & 3) + (lane & 3) + 4 * (lane >> 4), c4 = (lane >> 2) & 3;
    const int cj = (kSumJ / 2) * (warp >> 2) + c4, cr = (kSumR / 2) * (warp >> 2) + c4;
    const double2* coarse = tab + (size_t)(tile / kSumMid) * M;
    const double2* mid = tab + (size_t)(n0 + tile % kSumMid) * M;
    const double2* fine = tab + (size_t)(n0 + kSumMid + cr) * M;
    double2 x0 = make_double2(0.0, 0.0), x1 = x0;
    auto issue = [&](int m0, int s) {
        const int m = m0 + cm;
        const bool on = m < M;
        const int mc = on ? m : 0;
#pragma unroll
        for (int q = 0; q < kSumJ / 8; ++q) {
            const long long o = roff[cj + 4 * q];
            copy_async<8>(&A[s][cm][cj + 4 * q], vec + (o < 0 ? 0 : o) + mc, on && o >= 0);
        }
#pragma unroll
        for (int q = 0; q < kSumR / 8; ++q)
            copy_async<16>(&B[s][cm][2 * (cr + 4 * q)], fine + (size_t)(4 * q) * M + mc, on);
        x0 = coarse[mc];
        x1 = mid[mc];
    };
    if (M > 0) issue(0, 0);
    int s = 0;
    for (int m0 = 0; m0 < M; m0 += kSumK, s ^= 1) {
        asm volatile("cp.async.wait_all;" ::: "memory");
        const double2 x = cmul(x0, x1);
#pragma unroll
        for (int q = 0; q < kSumR / 8; ++q) {  // this thread's own copies
            double2* p = reinterpret_cast<double2*>(&B[s][cm][2 * (cr + 4 * q)]);
            *p = cmul(x, *p);
        }
        __syncthreads();
        if (m0 + kSumK < M) issue(m0 + kSumK, s ^ 1);
#pragma unroll
        for (int kk = 0; kk < kSumK / 2; kk += 8) {
            const int k = kw + kk + q4;
            double fa[2][4], fb[NB][2];
#pragma unroll
            for (int a = 0; a < 2; ++a)
#pragma unroll
                for (int i = 0; i < 4; ++i) fa[a][i] = A[s][k + 4 * (i >> 1)][jw + 16 * a + g + 8 * (i & 1)];
#pragma unroll
            for (int b = 0; b < NB; ++b)
#pragma unroll
                for (int i = 0; i < 2; ++i) fb[b][i] = B[s][k + 4 * i][cw + 8 * b + g];
#pragma unroll
            for (int a = 0; a < 2; ++a)
#pragma unroll
                for (int b = 0; b < NB; ++b) mma_f64(acc[a][b], fa[a], fb[b]);
        }
    }
    // the second halves of the steps to the first warps
    __syncthreads();
    double* part = smem + (threadIdx.x & 127);
    if (warp >= 4) {
#pragma unroll
        for (int a = 0; a < 2; ++a)
#pragma unroll
            for (int b = 0; b < NB; ++b)
#pragma unroll
                for (int c = 0; c < 4; ++c) part[((a * NB + b) * 4 + c) * 128] = acc[a][b][c];
    }
    __syncthreads();
    if (warp >= 4) return;
    const double ang = kPi * 0.25;
    const double sa = sin(ang), ca = cos(ang);
#pragma unroll
    for (int b = 0; b < NB; ++b) {
        const int i = tile * kSumR + (cw >> 1) + 4 * b + q4;
        if (i >= nr) continue;
        const double c0 = 1000.0 * 4 * kPi / sqrt(8.0 * kPi) / sqrt((i + 1) * dr);
        const double fr = c0 * sa, fi = c0 * ca;
#pragma unroll
        for (int a = 0; a < 4; ++a) {
            const int j = j0 + jw + 8 * a + g;
            if (j >= nj) continue;
            const int c = 2 * (a & 1), p = ((a >> 1) * NB + b) * 4 + c;
            const double xr = acc[a >> 1][b][c] + part[p * 128], xi = acc[a >> 1][b][c + 1] + part[(p + 1) * 128];
            const size_t o = (size_t)i * sr + (size_t)j * sj;
            re[o] = fr * xr - fi * xi;
            im[o] = fr * xi + fi * xr;
        }
    }
}

int sum_coarse(int nr, int nb) { return (nr + kSumMid * 8 * nb - 1) / (kSumMid * 8 * nb); }

template <int NB>
int run_modal_sum(cudaStream_t st, int M, const double2* tab, const double* vec, const int* rows, int nj, int nr,
                  double dr, long long sr, long long sj, double* re, double* im) {
    if (cudaFuncSetAttribute(k_modal_sum<NB>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSumSmem) !=
        cudaSuccess)
        return -1;
    const dim3 grid((nr + 8 * NB - 1) / (8 * NB), (nj + kSumJ - 1) / kSumJ);
    k_modal_sum<NB><<<grid, kSumThreads, kSumSmem, st>>>(M, tab, sum_coarse(nr, NB), vec, rows, nj, nr, dr, sr, sj,
                                                        re, im);
    return 1;
}

}  // namespace

size_t modal_sum_scratch(int M, int nr) {
    return (size_t)(sum_coarse(nr, 2) + kSumMid + 32) * (size_t)std::max(M, 1) * sizeof(double2);
}

int launch_modal_sum(cudaStream_t st, int M, const double* kr, const double* ki, const double* vs_src,
                     const double* vec, const int* rows, int nj, int nr, double dr, int lossless, bool range_major,
                     int num_sms, void* scratch, double* re, double* im) {
    // 32, 24 or 16 ranges a CTA: whichever keeps the last round of CTAs (2 on
    // an SM) fullest, a round of one more tile costing as much as a full one
    // (64 heights x 20000 ranges x 1185 modes: 24 ranges 330 us, 32 381 us)
    int nb = 4;
    long long best = 0;
    for (int n = 4; n >= 2; --n) {
        const long long ctas = (long long)((nr + 8 * n - 1) / (8 * n)) * ((nj + kSumJ - 1) / kSumJ);
        const long long cost = (ctas + 2 * num_sms - 1) / (2 * num_sms) * (n + 1);  // + 1: the heights' copies
        if (best == 0 || cost < best) best = cost, nb = n;
    }
    double2* tab = static_cast<double2*>(scratch);
    const int n0 = sum_coarse(nr, nb), n1 = 8 * nb;
    if (M > 0)
        k_sum_phases<<<dim3(n0 + kSumMid + n1, (M + 127) / 128), 128, 0, st>>>(M, kr, ki, vs_src, dr, lossless, n0,
                                                                             n1, tab);
    const long long sr = range_major ? nj : 1, sj = range_major ? 1 : nr;
    const int rc = nb == 4   ? run_modal_sum<4>(st, M, tab, vec, rows, nj, nr, dr, sr, sj, re, im)
                   : nb == 3 ? run_modal_sum<3>(st, M, tab, vec, rows, nj, nr, dr, sr, sj, re, im)
                             : run_modal_sum<2>(st, M, tab, vec, rows, nj, nr, dr, sr, sj, re, im);
    return rc < 0 ? rc : rc + (M > 0);
}

// ===========================================================================
// K6: ModBB synthesis
// ===========================================================================
__global__ void k_twiddle(int nfft, double* __restrict__ tw) {
    int m = blockIdx.x * blockDim.x + threadIdx.x;
    if (m >= nfft) return;
    double ang = -2.0 * kPi * (double)m / (double)nfft;
    double sn, cs;
    sincos(ang, &sn, &cs);
    tw[2 * m] = cs;
    tw[2 * m + 1] = sn;
}

int launch_twiddle(cudaStream_t st, int nfft, double* tw) {
    k_twiddle<<<(nfft + 255) / 256, 256, 0, st>>>(nfft, tw);
    return 1;
}

// per-mode factors of the transfer function: V_s V_r and 1/sqrt(k) (principal)
__global__ void k_bb_prep(int n, const double* __restrict__ re_k, const double* __restrict__ im_k,
                          const double* __restrict__ vs, const double* __restrict__ vr, int zero_attn,
                          double* __restrict__ fac) {
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= n) return;
    const double a = re_k[j], b = zero_attn ? 0.0 : im_k[j];
    const auto sk = csqrt_principal(a, b);
    const double den = sk.real() * sk.real() + sk.imag() * sk.imag();
    fac[4 * j + 0] = vs[j] * vr[j];
    fac[4 * j + 1] = sk.real() / den;
    fac[4 * j + 2] = -sk.imag() / den;
    fac[4 * j + 3] = b;
}

// transfer function H(f, r) = i e^{-i pi/4}/sqrt(8 pi r) sqrt(rho_r/rho_s)
//   sum_j V_s V_r e^{i k r}/sqrt(k), half-Hann over the top 10 % of bins;
// one warp per (frequency, range), lanes over the modes of that frequency
__global__ void k_bb_transfer(int nfreq, const int* __restrict__ off, const double* __restrict__ re_k,
                              const double* __restrict__ fac, double rho_ratio, int nr,
                              const double* __restrict__ ranges, double* __restrict__ h) {
    const int wg = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (wg >= nfreq * nr) return;
    const int f = wg % nfreq, ir = wg / nfreq;
    const double r = ranges[ir];
    double cr = 0.0, ci = 0.0;
    for (int j = off[f] + lane; j < off[f + 1]; j += 32) {
        double sn, cs;
        sincos(r * re_k[j], &sn, &cs);
        const double amp = exp(-r * fac[4 * j + 3]) * fac[4 * j];
        const double er = amp * cs, ei = amp * sn;
        const double isr = fac[4 * j + 1], isi = fac[4 * j + 2];
        cr += er * isr - ei * isi;
        ci += er * isi + ei * isr;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        cr += __shfl_xor_sync(0xffffffffu, cr, o);
        ci += __shfl_xor_sync(0xffffffffu, ci, o);
    }
    if (lane != 0) return;
    // i e^{-i pi/4} = sin(pi/4) + i cos(pi/4)
    const double c0 = sqrt(rho_ratio) / sqrt(8.0 * kPi * r);
    const double ang = kPi * 0.25;
    const double fr = c0 * sin(ang), fi = c0 * cos(ang);
    double hr = fr * cr - fi * ci, hi = fr * ci + fi * cr;
    const int smooth = (int)floor(0.1 * nfreq);
    const int begin = nfreq - smooth, end = nfreq - 1;
    if (smooth > 0 && f >= begin) {
        // one-bin window (end == begin): the limit value 1 instead of the
        // reference's 0/0 (BroadbandPropagator.cpp:654-662)
        const double hh = end == begin ? 1.0 : 0.5 * (cos(kPi * (f - begin) / (end - begin)) + 1.0);
        hr *= hh;
        hi *= hh;
    }
    h[((size_t)ir * nfreq + f) * 2] = hr;
    h[((size_t)ir * nfreq + f) * 2 + 1] = hi;
}

int launch_bb_transfer(cudaStream_t st, int nfreq, const int* off, const double* re_k, const double* im_k,
                       const double* vs, const double* vr, double rho_ratio, int nr, const double* ranges,
                       int zero_attn, int n_modes, double* fac, double* h) {
    int launches = 0;
    if (n_modes > 0) {
        k_bb_prep<<<(n_modes + 255) / 256, 256, 0, st>>>(n_modes, re_k, im_k, vs, vr, zero_attn, fac);
        ++launches;
    }
    const long long threads = (long long)nfreq * nr * 32;
    k_bb_transfer<<<(unsigned)((threads + 255) / 256), 256, 0, st>>>(nfreq, off, re_k, fac, rho_ratio, nr, ranges,
                                                                     h);
    return launches + 1;
}

// built-in source spectra at the dispersion bins (BroadbandPropagator.cpp:
// 260-297, 420-438): 0 impulse e^{2 pi i f Nfreq/2}; 1 pulse1 (analytic fit,
// scale = 1/f_center); the returned spectrum is interleaved (re, im)
__global__ void k_src_builtin(int kind, int nfreq, const double* __restrict__ f, double scale,
                              double* __restrict__ out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nfreq) return;
    const double PI = kPi;
    double re, im;
    if (kind == 0) {
        double sn, cs;
        sincos(2.0 * PI * f[i] * (double)nfreq / 2.0, &sn, &cs);
        re = cs;
        im = sn;
    } else {
        const double fnorm = 0.780776406404415;
        const double x = scale * fnorm * f[i];
        // x e^{(-x - x^2)/2} e^{-i pi/2} scale / 33.4336, times 4 pi 5 e^{2 pi i x 0.01}
        const double mag = 4.0 * PI * 5.0 * (x * exp((-x - x * x) / 2) * scale / 33.4336);
        double ph = -0.5 * PI + 2.0 * PI * x * 0.01 + 2.0 * PI * f[i] * scale;
        double sn, cs;
        sincos(ph, &sn, &cs);
        re = mag * cs / 2.0;
        im = mag * sn / 2.0;
    }
    out[2 * i] = re;
    out[2 * i + 1] = im;
}

// power-law pulse model of source type pulse2, sampled at t = i dt
__global__ void k_src_pulse2(int n, double dt, double scale, double power, double* __restrict__ x) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double xx = 2.094 * (1.0 + power) * (i * dt) / scale;
    x[i] = pow(xx, power) * (1 - xx / (1.0 + power)) * exp(-xx) / 1.387566e+03;
}

int launch_src_builtin(cudaStream_t st, int kind, int nfreq, const double* f, double scale, double* out) {
    k_src_builtin<<<(nfreq + 127) / 128, 128, 0, st>>>(kind, nfreq, f, scale, out);
    return 1;
}

int launch_src_pulse2(cudaStream_t st, int n, double dt, double scale, double* x) {
    k_src_pulse2<<<(n + 255) / 256, 256, 0, st>>>(n, dt, scale, 8.0, x);
    return 1;
}

// p(t_k) = 2 Re( df sum_n e^{-2 pi i f_n t0} S_n H_n e^{-2 pi i k n / nfft} )
constexpr int kPulseMaxFreq = 4096;

constexpr int kPulseBins = 64;  // time bins per CTA of k_bb_pulse (8 warps x 8)

__global__ void __launch_bounds__(256) k_bb_pulse(int nfreq, const double* __restrict__ f,
                                                  const double* __restrict__ s_src, const double* __restrict__ h,
                                                  int nr, const double* __restrict__ t0s, int nfft,
                                                  const double* __restrict__ tw, double* __restrict__ out) {
    extern __shared__ double arg[];  // 2 * nfreq
    const int ir = blockIdx.y;
    const double t0 = t0s[ir];
    for (int n = threadIdx.x; n < nfreq; n += blockDim.x) {
        double sn, cs;
        sincos(((-2.0 * kPi) * f[n]) * t0, &sn, &cs);
        const double sr = s_src[2 * n], si = s_src[2 * n + 1];
        const double hr = h[((size_t)ir * nfreq + n) * 2], hi = h[((size_t)ir * nfreq + n) * 2 + 1];
        const double ar = cs * sr - sn * si, ai = cs * si + sn * sr;
        arg[2 * n] = ar * hr - ai * hi;
        arg[2 * n + 1] = ar * hi + ai * hr;
    }
    __syncthreads();
    const double df = f[2] - f[1];  // f_step of ModalBroadbandPropagator.cpp:65
    // one warp per time bin k: lanes split the frequencies, then a shuffle sum
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int kend = min(nfft, (blockIdx.x + 1) * kPulseBins);
    for (int k = blockIdx.x * kPulseBins + wid; k < kend; k += blockDim.x >> 5) {
        double accr = 0.0;
        for (int n = lane; n < nfreq; n += 32) {
            const int idx = (int)(((long long)n * k) % nfft);
            accr += arg[2 * n] * tw[2 * idx] - arg[2 * n + 1] * tw[2 * idx + 1];
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) accr += __shfl_xor_sync(0xffffffffu, accr, o);
        if (lane == 0) out[(size_t)ir * nfft + k] = 2.0 * (df * accr);
    }
}

int launch_bb_pulse(cudaStream_t st, int nfreq, const double* f, const double* s_src, const double* h, int nr,
                    const double* t0, int nfft, const double* tw, double* out) {
    dim3 grid((nfft + kPulseBins - 1) / kPulseBins, nr);
    size_t sm = (size_t)2 * nfreq * sizeof(double);
    if (sm > 48 * 1024) cudaFuncSetAttribute(k_bb_pulse, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    k_bb_pulse<<<grid, 256, sm, st>>>(nfreq, f, s_src, h, nr, t0, nfft, tw, out);
    return 1;
}

// source spectrum of a sampled waveform: dt sum_n x_n e^{+2 pi i k n/nfft};
// one warp per frequency bin k, lanes split the samples, then a shuffle sum
__global__ void __launch_bounds__(256) k_src_dft(int n, const double* __restrict__ x, double dt, int nfft,
                                                 int nfreq, const double* __restrict__ tw, double* __restrict__ s) {
    const int lane = threadIdx.x & 31;
    const int k = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (k >= nfreq) return;  // warp-uniform
    double ar = 0.0, ai = 0.0;
    const int nn = min(n, nfft);
    for (int j = lane; j < nn; j += 32) {
        const int idx = (int)(((long long)j * k) % nfft);
        ar += x[j] * tw[2 * idx];
        ai -= x[j] * tw[2 * idx + 1];  // conjugate twiddle: e^{+i}
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        ar += __shfl_xor_sync(0xffffffffu, ar, o);
        ai += __shfl_xor_sync(0xffffffffu, ai, o);
    }
    if (lane == 0) {
        s[2 * k] = ar * dt;
        s[2 * k + 1] = ai * dt;
    }
}

// out[i] = (re[i], im[i])
__global__ void __launch_bounds__(256) k_pairs(size_t n, const double* __restrict__ re, const double* __restrict__ im,
                                               double2* __restrict__ out) {
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i] = make_double2(re[i], im[i]);
}

int launch_pairs(cudaStream_t st, size_t n, const double* re, const double* im, double* out) {
    k_pairs<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(n, re, im, reinterpret_cast<double2*>(out));
    return 1;
}

// out[c][r] = in[r][c] for a rows x cols matrix of doubles, 32 x 32 tiles
// staged in shared memory (both sides coalesced)
__global__ void __launch_bounds__(256) k_transpose(int rows, int cols, const double* __restrict__ in,
                                                   double* __restrict__ out) {
    __shared__ double t[32][33];
    const int c0 = blockIdx.x * 32, r0 = blockIdx.y * 32;
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;  // 32 x 8 threads
    for (int k = ty; k < 32; k += 8) {
        const int r = r0 + k, c = c0 + tx;
        if (r < rows && c < cols) t[k][tx] = in[(size_t)r * cols + c];
    }
    __syncthreads();
    for (int k = ty; k < 32; k += 8) {
        const int c = c0 + k, r = r0 + tx;
        if (r < rows && c < cols) out[(size_t)c * rows + r] = t[tx][k];
    }
}

int launch_transpose(cudaStream_t st, int rows, int cols, const double* in, double* out) {
    if (rows < 1 || cols < 1) return 0;
    dim3 grid((cols + 31) / 32, (rows + 31) / 32);
    k_transpose<<<grid, 256, 0, st>>>(rows, cols, in, out);
    return 1;
}

// values of a Steffen spline at m points (clamped outside the knots)
__global__ void k_spline_eval(int n, const double* __restrict__ x, const double* __restrict__ y,
                              const double* __restrict__ coef, int m, const double* __restrict__ xq,
                              double* __restrict__ out) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k < m) out[k] = spline_get(n, x, y, coef, xq[k]);
}

int launch_spline_eval(cudaStream_t st, int n, const double* x, const double* y, const double* coef, int m,
                       const double* xq, double* out) {
    k_spline_eval<<<(m + 255) / 256, 256, 0, st>>>(n, x, y, coef, m, xq, out);
    return 1;
}

// modal starter field (ESSModeSolver::getModalStarter, ESSModeSolver.cpp:
// 670-723): psi(z_j) = pi sqrt(k0) sum_m v_m(z_s) v_m(z_j) / sqrt(Re k_m)
__global__ void k_starter(int M, int nz, int step, int isrc, const double* __restrict__ v,
                          const double* __restrict__ kr, double k0, double* __restrict__ out) {
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    const int zi = j * step;
    if (zi >= nz) return;
    double acc = 0.0;
    for (int m = 0; m < M; ++m) acc += v[(size_t)isrc * M + m] * v[(size_t)zi * M + m] / sqrt(kr[m]);
    out[j] = acc * kPi * sqrt(k0);
}

int launch_starter(cudaStream_t st, int M, int nz, int step, int isrc, const double* v, const double* kr,
                   double k0, double* out) {
    const int nout = (nz + step - 1) / step;
    k_starter<<<(nout + 127) / 128, 128, 0, st>>>(M, nz, step, isrc, v, kr, k0, out);
    return 1;
}

// unit transfer function (complex 1) for [nr x nfreq] bins
__global__ void k_fill_unit(int n, double* __restrict__ h) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k < n) {
        h[2 * k] = 1.0;
        h[2 * k + 1] = 0.0;
    }
}

int launch_fill_unit(cudaStream_t st, int n, double* h) {
    k_fill_unit<<<(n + 255) / 256, 256, 0, st>>>(n, h);
    return 1;
}

int launch_src_dft(cudaStream_t st, int n, const double* x, double dt, int nfft, int nfreq, const double* tw,
                   double* s) {
    k_src_dft<<<(nfreq * 32 + 255) / 256, 256, 0, st>>>(n, x, dt, nfft, nfreq, tw, s);
    return 1;
}

}  // namespace ncpa
