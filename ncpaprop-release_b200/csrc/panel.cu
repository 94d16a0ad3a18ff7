// The eigen-solve on panel expansions of the tridiagonal rows.
//
// The rows S = h^2 A - x (unit off-diagonals) act on the state (u_i, e_i),
// u_i = (-1)^{i+1} p_i of the Sturm recurrence and e_i = u_i - u_{i-1}, as
//   e_i = e_{i-1} - sigma_i u_{i-1},   u_i = u_{i-1} + e_i,
//   sigma_i = s_i + 2 - x:
// a discrete u'' = -sigma u.  The 2 x 2 transfer matrix of a block of B
// consecutive rows is a smooth function of x: with x = x_c + r t, |t| <= 1, its
// entries behave like cos and sin of B sqrt(sigma), whose Taylor series in t
// falls like rho^k / (2k)!, rho = r B^2.  So the shifts of a solve are grouped
// into panels (of scan points, then of work items), as wide as rho <= kRhoMax =
// 10 allows at B = 128 rows a block, or one unit or item each at smaller
// blocks; per panel and block the four entries are expanded once to degree kPD
// (a thread per column, so the work is parallel over the rows), and every sweep
// of the scan, the multisection, Laguerre's iteration and the eigenvector
// passes advances B rows with four Horner evaluations.  The first term left
// out, rho^15 / 30!, is 4e-18.
//
// What it buys (the row recurrence is bound by FP64 issue, 2 instructions a row
// for a count and 6 with two derivatives, plus one for the sign): at B = 128
// a count costs 65 instructions a block (0.5 a row) and a Laguerre chain 190
// (1.5 a row), the serial chain is two FMAs a block instead of one a row, and
// segments of blocks can be taken apart.  0.1 Hz, 20000 rows: eigenvalues 750
// -> 77 us, mode values 647 -> 86; 256 frequencies 3.28 -> 0.88 ms for both.
// Accuracy: the rounding of a block perturbs sigma by about 1e-16 on one row
// in B, and errors relative to u are harmless.  What counts is that the shift is
// taken as doubles see it (Shift: up to 1.1e-16) and that the iteration ends with
// a correction below 1e-15: eigenvalues are within 1.1e-15 (median 6e-17, units
// of h^2 A) of an evaluation of the rows in 80 bits (0.1 and 0.5 Hz, 5000 and
// 20000 rows), mode values within 1e-12.
//
// Counts.  The number of negative pivots is nz minus the sign changes of u.
// In a block, the solution that starts with u = 0 changes sign n2(x) times, and
// any other solution n2 or n2 + 1 times (Sturm separation), so the parity of
// the sign change between the block's ends decides.  n2 is counted at the
// panel's centre.  Elsewhere it is less by the zeros of the entry T12 in between,
// the levels of the block's rows with u = 0 at both ends: at even sigma they are
// 29 / B^2 apart and half a panel is kRhoMax / B^2, so it differs by one at most,
// which the sign of T12 tells; with sigma varying by V over the block they are
// still 29 / B^2 - V apart.  Where V is above kFlat / B^2 the roots of T12 are
// bounded from its coefficients, where these allow more than one the expansion
// counts at the panel's ends too, and a block that differs there by more than one
// (two wells with a barrier between them) is counted by its rows.
//
// Eigenvectors.  u runs up from the ground and b, the solution that meets the
// upper boundary, runs down; they are joined at the twist row r where |u b| is
// largest.  The norm sum z^2, the attenuation integral sum z^2 w and the
// group-speed integral need no sums over rows: for a perturbation sigma_i +
// eps W_i the derivatives (u_eps, e_eps) satisfy
//   u e_eps - e u_eps = - sum over the rows so far of W_i u_{i-1}^2
// (and with the other sign downwards for b), so the derivative chains of the
// same block matrices give them: d/dx (W = -1) from the Horner steps, d/deps
// expanded to degree kPW.  Both directions stop at the twist, where neither
// solution is contaminated by the growing one.  (A single chain carried to the
// far boundary would do at half the cost, but its error is first order in the
// eigenvalue's: 1e-6 of Im k for ducted modes, whose weights aloft are 1e9
// times those in the duct.)
#include <algorithm>
#include <climits>
#include <cmath>

#include "device_common.cuh"
#include "kernels.hpp"

namespace ncpa {

namespace {

constexpr int kTD = kPanelChunk * kRecT;  // doubles of a chunk of T records
constexpr int kWD = kPanelChunk * kRecW;  // doubles of a chunk of one weight's records
constexpr int kPBuf = 3;                  // ring slots per warp
constexpr int kPWarps = 4;                // warps per CTA (two pairs)
// a chunk's growth in bits, at most, and where the mode values' chains are
// rescaled: sums are products of u at kVecBits + kGrowBits and a derivative
// at 130 more
constexpr int kGrowBits = 400, kVecBits = 20;
static_assert(480 + kGrowBits + 130 < 1023 && 2 * (kVecBits + kGrowBits) + 130 < 1023, "the sweeps stay finite");
constexpr int kPanelCtas = 3;             // CTAs per SM
constexpr int kSoloMin = 6;               // items by rows per SM from which on each has a warp
constexpr int kRowsCtas = 4;              // CTAs per SM then
constexpr int kRecZeros = 4 * (kPD + 1), kRecMid = kRecZeros + 1;
static_assert(kRecT == kRecMid + 1 && kRecT % 2 == 0, "T record: coefficients, zero count, split, 16-byte size");
static_assert(kRecW == 4 * (kPW + 1), "W record: coefficients");

struct Panel {
    double xc, r;
    const double* rows;  // raw rows of the problem
    long long rec;       // first block record
    int nblk, blk, nz;   // blk = 0: no records, the sweeps run on the raw rows
    double e0, um0;  // e_{-1} and u_{-2}
};

// the coefficients of -sigma in t: s0 + s1 t + s2 t^2
struct Quad {
    double s0, s1, s2;
};

// ---------------------------------------------------------------------------
// row formats
// ---------------------------------------------------------------------------
// sigma at centre xc and its linear and quadratic coefficients in t
struct EssPanel {
    static constexpr int kW = 1;
    static constexpr bool kUnitNorm = true;  // the norm is -dg/dx: no weight of ones
    static constexpr bool kQuad = false;     // sigma is linear in x
    static constexpr bool kLaguerre = true;  // the determinant has real roots only
    // around the panel's centre, for the expansion
    __device__ static __forceinline__ Quad series(const double* __restrict__ row, int i, double xc, double r) {
        return {-((__ldg(row + i) + 2.0) - xc), r, 0.0};
    }
    // of the row itself at a shift (s_i - x in doubles)
    __device__ static __forceinline__ double sigma(const double* __restrict__ row, int i, double x) {
        return (__ldg(row + i) - x) + 2.0;
    }
    __device__ static __forceinline__ double um_init(const ProblemInfo&) { return 0.0; }  // p_{-2} = 0
    // a row (staged in shared memory) at a shift: 2 - sigma, and d / dx of it over kSlope
    struct At {
        double x;
        __device__ __forceinline__ At() {}
        __device__ __forceinline__ explicit At(double x_) : x(x_) {}
        __device__ __forceinline__ double turn(const double* __restrict__ r) const { return x - r[0]; }
        __device__ __forceinline__ double turn(const double* __restrict__ r, double& slope) const {
            slope = 1.0;
            return x - r[0];
        }
    };
    static constexpr double kSlope = 1.0;
    __device__ static __forceinline__ double lo(const ProblemInfo& pi) { return pi.lo; }
    __device__ static __forceinline__ double hi(const ProblemInfo& pi) { return pi.hi; }
    __device__ static __forceinline__ double tol_scale(const ProblemInfo&) { return 1.0; }
    __device__ static __forceinline__ double steepness(const ProblemInfo&) { return 1.0; }  // of sigma in x
    // a bound of |sigma| = |h^2 omega^2 / c_eff^2 - x| in the window
    __device__ static __forceinline__ float span(const ProblemInfo& pi) {
        const float wh = (float)(pi.omega * pi.dz), lo = (float)pi.lo, hi = (float)pi.hi;
        const float k0 = wh / (float)__longlong_as_double((long long)pi.ceffmax_bits);
        const float k1 = wh / (float)__longlong_as_double((long long)pi.ceffmin_bits);
        return fmaxf(k1 * k1 - fminf(lo, hi), fmaxf(lo, hi) - k0 * k0);
    }
    // The shift that a row sees.  The stored rows are multiples of 2^-52 in (-2,
    // -1] (but for the ground row and very coarse grids).  So in doubles s_i - x
    // is s_i less x rounded to that grid where it lies above -2, and below,
    // where doubles are 2^-51 apart, s_i less the grid point under or over x as
    // s_i is even or odd: halfway, on average.  The block sweeps take their
    // shifts there too (a block counts as below by its middle row): no nearer to
    // the exact eigenvalues, but nearer to those of an evaluation of the rows in
    // doubles, so that pairs of modes closer than 1e-8 or phases k r at 1000 km
    // come out alike whichever way they are computed.  (Where h k is above 1 the
    // rows leave (-2, -1], their spacing is another, and the shift is merely
    // rounded by as much.)
    struct Shift {
        double x, t0, t1;
        __device__ __forceinline__ Shift() {}
        __device__ __forceinline__ Shift(const Panel& P, double x_) : x(x_) {
            const double above = (1.0 + x) - 1.0, below = (floor(x * 4503599627370496.0) + 0.5) * 2.220446049250313e-16;
            const double rinv = 1.0 / P.r;
            t0 = (above - P.xc) * rinv;
            t1 = (below - P.xc) * rinv;
        }
        __device__ __forceinline__ double at(const double* rec) const { return x > rec[kRecMid] ? t1 : t0; }
    };
    // kRecMid of a block with middle row i: rows below this are on the coarser side
    __device__ static __forceinline__ double middle(const double* __restrict__ row, int i, double) {
        return __ldg(row + i) + 2.0;
    }
};

// Wide-angle rows (B_i, U_i) at kappa = h k: sigma_i = (B_i - U_i kappa)^2 -
// kappa^2, plus the ground term in the first state.  det T(kappa) has roots off
// the real axis too: Newton's steps instead of Laguerre's.
struct WmodPanel {
    static constexpr int kW = 2;
    static constexpr bool kUnitNorm = false;  // the norm needs a weight of ones
    static constexpr bool kQuad = true;
    static constexpr bool kLaguerre = false;
    __device__ static __forceinline__ double2 row_at(const double* __restrict__ row, int i) {
        return __ldg(reinterpret_cast<const double2*>(row) + i);
    }
    __device__ static __forceinline__ Quad series(const double* __restrict__ row, int i, double xc, double r) {
        const double2 q = row_at(row, i);
        const double d = fma(-q.y, xc, q.x);
        return {(xc - d) * (xc + d), 2.0 * r * fma(q.y, d, xc), r * r * fma(-q.y, q.y, 1.0)};
    }
    __device__ static __forceinline__ double sigma(const double* __restrict__ row, int i, double x) {
        const double2 q = row_at(row, i);
        const double d = fma(-q.y, x, q.x);
        return fma(d, d, fma(-x, x, -2.0)) + 2.0;
    }
    // -d sigma / dx
    __device__ static __forceinline__ double slope(const double* __restrict__ row, int i, double x) {
        const double2 q = row_at(row, i);
        return 2.0 * fma(q.y, fma(-q.y, x, q.x), x);
    }
    __device__ static __forceinline__ double um_init(const ProblemInfo& pi) { return pi.g0; }
    struct At {
        double x, c;
        __device__ __forceinline__ At() {}
        __device__ __forceinline__ explicit At(double x_) : x(x_), c(fma(-x_, x_, -2.0)) {}
        __device__ __forceinline__ double turn(const double* __restrict__ r) const {
            const double2 q = *reinterpret_cast<const double2*>(r);
            const double d = fma(-q.y, x, q.x);
            return -fma(d, d, c);
        }
        __device__ __forceinline__ double turn(const double* __restrict__ r, double& slope) const {
            const double2 q = *reinterpret_cast<const double2*>(r);
            const double d = fma(-q.y, x, q.x);
            slope = fma(q.y, d, x);
            return -fma(d, d, c);
        }
    };
    static constexpr double kSlope = 2.0;
    __device__ static __forceinline__ double lo(const ProblemInfo& pi) { return pi.k_min * pi.dz; }
    __device__ static __forceinline__ double hi(const ProblemInfo& pi) { return pi.k_max * pi.dz; }
    __device__ static __forceinline__ double tol_scale(const ProblemInfo& pi) { return pi.k_max * pi.dz; }
    // |d sigma / d kappa| = 2 (kappa + U d), U d < kappa / 2 at winds below half
    // the speed of sound
    __device__ static __forceinline__ double steepness(const ProblemInfo& pi) { return 3.0 * (pi.k_max * pi.dz); }
    // A bound of |sigma| = |d^2 - kappa^2|: at phase speed c, d = h omega (1 - w /
    // c) / c_0 is at most h omega / c_0 downwind, and upwind, with c_0 = c_eff -
    // w, at most h omega / min c_eff (for c from there on)
    __device__ static __forceinline__ float span(const ProblemInfo& pi) {
        const float c = fminf((float)__longlong_as_double((long long)pi.ceffmin_bits),
                              (float)__longlong_as_double((long long)pi.c0min_bits));
        const float dz = (float)pi.dz, d = (float)pi.omega * dz / c;
        const float a = (float)pi.k_min * dz, b = (float)pi.k_max * dz, k0 = fminf(a, b), k1 = fmaxf(a, b);
        return fmaxf(fmaxf(d, k1) * fmaxf(d, k1) - k0 * k0, k1 * k1);
    }
    // An evaluation of the rows rounds -kappa^2 - 2 once for all of them, a
    // common shift of sigma by up to 2e-16; the blocks take the kappa that
    // shifts theirs alike (by the middle row's slope).
    struct Shift {
        double t0, dt;
        __device__ __forceinline__ Shift() {}
        __device__ __forceinline__ Shift(const Panel& P, double x) {
            const double rinv = 1.0 / P.r, c = fma(-x, x, -2.0);
            t0 = (x - P.xc) * rinv;
            dt = -fma(x, x, c + 2.0) * rinv;
        }
        __device__ __forceinline__ double at(const double* rec) const { return fma(dt, rec[kRecMid], t0); }
    };
    __device__ static __forceinline__ double middle(const double* __restrict__ row, int i, double xc) {
        return 1.0 / slope(row, i, xc);
    }
};

// ---------------------------------------------------------------------------
// panels
// ---------------------------------------------------------------------------

template <class Row>
__device__ __forceinline__ Panel panel_of(const ProblemInfo& pi, const PanelDesc& d, const double* rows) {
    Panel P;
    P.xc = d.xc;
    P.r = d.blk ? d.r : 1.0;  // raw rows: derivatives in x itself
    P.blk = d.blk;
    P.rows = rows + (size_t)pi.s_off * Row::kW;
    P.nz = pi.nz;
    P.nblk = d.blk ? (pi.nz + d.blk - 1) / d.blk : 0;
    P.rec = d.rec;
    P.um0 = Row::um_init(pi);
    P.e0 = 1.0 - P.um0;
    return P;
}

__device__ __forceinline__ int padded(int nblk) { return (nblk + kPanelChunk - 1) / kPanelChunk * kPanelChunk; }

// The most rows of a block, for the growth of a chain over a chunk of them: with
// |sigma| <= S a row multiplies the state by at most e^lambda, cosh lambda = 1 +
// S / 2 (the comparison recurrence |e'| = |e| + S |u|, |u'| = |u| + |e'|).  The
// sweeps rescale once a chunk, so that a state below 2^480 stays finite, and the
// mode values' chains, whose sums are products of two, one below 2^kVecBits.  (In
// single precision, whose errors the bits to spare cover: in double 3 us a solve.)
__device__ __forceinline__ int most_rows(float S) {
    const float h = 0.5f * S, bits = log1pf(h + sqrtf(h * (h + 2.f))) * 1.4426950f;
    int B = kPanelMaxBlk;
    while (B > 0 && !(bits * (float)(kPanelChunk * B) <= (float)kGrowBits)) B >>= 1;
    return B;
}

// rows per block for shifts within r of the centre: the most (of `most`) that
// keep r B^2 within kRhoMax (0: not even panel_min_blk, the rows as they are)
__device__ __forceinline__ int block_rows(double r, int nz, int most) {
    for (int B = most; B >= panel_min_blk(nz); B >>= 1)
        if (r * (double)B * (double)B <= kRhoMax) return B;
    return 0;
}

// panel q of a problem's isolation scan: pi.upp units of kScanStep points
template <class Row>
__device__ __forceinline__ PanelDesc scan_panel(const ProblemInfo& pi, int q) {
    const int n = pi.n_scan, t0 = q * pi.upp * kScanStep, t1 = min(n, t0 + pi.upp * kScanStep) - 1;
    PanelDesc d;
    const double a = scan_x(Row::lo(pi), Row::hi(pi), t0, n), b = scan_x(Row::lo(pi), Row::hi(pi), t1, n);
    d.xc = 0.5 * (a + b);
    d.r = fmax(0.5 * fabs(b - a), 1e-300);
    d.blk = pi.upp ? pi.sp_blk : 0;
    d.rec = pi.blk_off + (long long)q * padded(d.blk ? (pi.nz + d.blk - 1) / d.blk : 0);
    d.problem = 0;
    return d;
}

// The scan's panels of a problem whose scan size is final: as many units per
// panel as kRhoMax allows at the largest block, or one unit and a smaller one
template <class Row>
__device__ void plan_scan_panels(ProblemInfo& pi, int n) {
    const int units = n / kScanStep;
    const double st = Row::steepness(pi);
    const double d = fabs(Row::hi(pi) - Row::lo(pi)) / (double)(n - 1);
    const int most = most_rows(Row::span(pi));
    int upp = most >= panel_min_blk(pi.nz) ? units : 0, B = 0;
    for (; upp >= 1; --upp) {
        const double r = 0.5 * d * (double)(upp * kScanStep - 1);
        if (st * r * (double)most * (double)most <= kRhoMax) {
            B = most;
            break;
        }
    }
    if (!B) {
        upp = 1;
        B = block_rows(st * (0.5 * d * (double)(kScanStep - 1)), pi.nz, most);
    }
    const long long need = B ? (long long)((units + upp - 1) / upp) * padded((pi.nz + B - 1) / B) : 0;
    const bool fits = B != 0 && need <= pi.blk_cap;
    pi.upp = fits ? upp : 0;
    pi.sp_blk = fits ? B : 0;
}

// ---------------------------------------------------------------------------
// expansion
// ---------------------------------------------------------------------------
constexpr int kExpThreads = 64;
constexpr double kFlat = 16.0;
constexpr int kByRows = 1 << 20;  // (even) added to the n2 of a block that is counted by its rows
static_assert(kRhoMax + kFlat < 27.0, "two levels of a block are further apart than half a panel");

__device__ __forceinline__ unsigned neg(double v) { return static_cast<unsigned>(__double2hiint(v)) >> 31; }

// the upper words of doubles as integers in the same order, and back
__device__ __forceinline__ int order_word(double v) {
    const int h = __double2hiint(v);
    return h ^ ((h >> 31) & 0x7fffffff);
}
__device__ __forceinline__ double word_value(int k) { return __hiloint2double(k ^ ((k >> 31) & 0x7fffffff), 0); }

// whether the sign changes over the rows [a, end) of the solution that starts with
// u = 0 differ by more than one between t = 0, where they are n2, and t = -1 or 1
template <class Row>
__device__ __forceinline__ bool far_zeros(const Panel& P, int a, int end, int n2) {
    double u[2] = {0.0, 0.0}, e[2] = {1.0, 1.0};
    unsigned prev[2] = {0u, 0u};
    int n[2] = {0, 0};
    for (int i = a; i < end; ++i) {
        const Quad q = Row::series(P.rows, i, P.xc, P.r);
        const double even = Row::kQuad ? q.s0 + q.s2 : q.s0;
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            e[k] = fma(k ? even + q.s1 : even - q.s1, u[k], e[k]);
            u[k] += e[k];
            n[k] += static_cast<int>(neg(u[k]) ^ prev[k]);
            prev[k] = neg(u[k]);
        }
    }
    return n[0] > n2 + 1 || n[1] < n2 - 1;
}

// sign changes in the coefficients of a polynomial
__device__ __forceinline__ int variations(const double (&c)[kPD + 1]) {
    int n = 0;
#pragma unroll
    for (int k = 0; k < kPD; ++k) n += static_cast<int>(neg(c[k]) ^ neg(c[k + 1]));
    return n;
}
// By Budan's theorem a polynomial has at most as many roots in (s, t] as its
// Taylor coefficients lose sign changes from s to t: whether that leaves T12 (c)
// more than one root on either side of 0 within [-1, 1]
__device__ __forceinline__ bool may_have_pairs(const double (&c)[kPD + 1]) {
    const int here = variations(c);
    double p[kPD + 1], m[kPD + 1];
#pragma unroll
    for (int k = 0; k <= kPD; ++k) p[k] = m[k] = c[k];
#pragma unroll
    for (int i = 0; i < kPD; ++i)
#pragma unroll
        for (int j = kPD - 1; j >= i; --j) {
            p[j] += p[j + 1];
            m[j] -= m[j + 1];
        }
    return variations(m) - here > 1 || here - variations(p) > 1;
}

// One thread per (panel, block, column of the transfer matrix): it runs the
// block's rows with the power series of u and e in t, and of their derivatives
// with respect to a perturbation eps W_i of sigma.  Bound by FP64 issue: 3
// instructions per row and coefficient (4 for the W series); the B rows of a
// thread are consecutive, so a warp touches 16 lines at a time, each used for
// 16 rows out of L1.
template <class Row, int NW>
__device__ __forceinline__ void expand_block(const Panel& P, int b, int col, const double* __restrict__ wp,
                                             const double* __restrict__ gp, double* __restrict__ T,
                                             double* __restrict__ W0, double* __restrict__ W1) {
    const int a = b * P.blk, end = min(P.nz, a + P.blk);
    constexpr int kNW0 = NW > 0 ? kPW + 1 : 1;
    double u[kPD + 1], e[kPD + 1], v0[kNW0], f0[kNW0];
    double v1[NW > 1 ? kPW + 1 : 1], f1[NW > 1 ? kPW + 1 : 1];
#pragma unroll
    for (int k = 0; k <= kPD; ++k) u[k] = e[k] = 0.0;
#pragma unroll
    for (int k = 0; k < kNW0; ++k) v0[k] = f0[k] = 0.0;
    if (NW > 1) {
#pragma unroll
        for (int k = 0; k <= kPW; ++k) v1[k] = f1[k] = 0.0;
    }
    if (col == 0) u[0] = 1.0;
    else e[0] = 1.0;
    const double r = P.r;
    unsigned prev = 0u;
    int n2 = 0, top = INT_MIN, bot = INT_MAX;
    for (int i = a; i < end; ++i) {
        const Quad sq = Row::series(P.rows, i, P.xc, r);
        const double sg = sq.s0, s1 = sq.s1;
        top = max(top, order_word(sg));
        bot = min(bot, order_word(sg));
        const double wi = NW > 0 ? -__ldg(wp + i) : 0.0;
        const double gi = NW > 1 ? (gp ? -__ldg(gp + i) : -1.0) : 0.0;
#pragma unroll
        for (int k = 0; NW > 0 && k <= kPW; ++k) {
            double x = fma(sg, v0[k], f0[k]);
            if (k > 0) x = fma(s1, v0[k - 1], x);
            if (Row::kQuad && k > 1) x = fma(sq.s2, v0[k - 2], x);
            f0[k] = fma(wi, u[k], x);
            if (NW > 1) {
                double y = fma(sg, v1[k], f1[k]);
                if (k > 0) y = fma(s1, v1[k - 1], y);
                if (Row::kQuad && k > 1) y = fma(sq.s2, v1[k - 2], y);
                f1[k] = fma(gi, u[k], y);
            }
        }
#pragma unroll
        for (int k = 0; k <= kPD; ++k) {
            e[k] = fma(sg, u[k], e[k]);
            if (k > 0) e[k] = fma(s1, u[k - 1], e[k]);
            if (Row::kQuad && k > 1) e[k] = fma(sq.s2, u[k - 2], e[k]);
        }
#pragma unroll
        for (int k = 0; k <= kPD; ++k) u[k] += e[k];
#pragma unroll
        for (int k = 0; NW > 0 && k <= kPW; ++k) {
            v0[k] += f0[k];
            if (NW > 1) v1[k] += f1[k];
        }
        // zeros of the solution that starts with u = 0 (column 1), at t = 0
        const unsigned s = static_cast<unsigned>(__double2hiint(u[0])) >> 31;
        n2 += static_cast<int>(s ^ prev);
        prev = s;
    }
    const size_t rec = (size_t)(P.rec + b);
    double* o = T + rec * kRecT + col;
#pragma unroll
    for (int k = 0; k <= kPD; ++k) {
        o[4 * k] = u[k];
        o[4 * k + 2] = e[k];
    }
    if (col == 1) {
        const double hi = word_value(top), lo = word_value(bot);  // to 2^-20 of themselves
        const bool flat = (hi - lo + 1e-6 * (fabs(hi) + fabs(lo))) * (double)P.blk * (double)P.blk <= kFlat;
        if (!flat && may_have_pairs(u) && far_zeros<Row>(P, a, end, n2)) n2 += kByRows;
        T[rec * kRecT + kRecZeros] = __hiloint2double(0, n2);
        T[rec * kRecT + kRecMid] = Row::middle(P.rows, min(P.nz - 1, a + P.blk / 2), P.xc);
    }
    if (NW > 0) {
        o = W0 + rec * kRecW + col;
#pragma unroll
        for (int k = 0; k <= kPW; ++k) {
            o[4 * k] = v0[k];
            o[4 * k + 2] = f0[k];
        }
    }
    if (NW > 1) {
        o = W1 + rec * kRecW + col;
#pragma unroll
        for (int k = 0; k <= kPW; ++k) {
            o[4 * k] = v1[k];
            o[4 * k + 2] = f1[k];
        }
    }
}

// the panels of the work items, one per blockIdx.y
template <class Row, int NW>
__global__ void __launch_bounds__(kExpThreads) k_expand_items(const ProblemInfo* __restrict__ pinfo,
                                                              const PanelDesc* __restrict__ desc, int d0,
                                                              const double* __restrict__ rows,
                                                              const double* __restrict__ w,
                                                              const double* __restrict__ g, double* __restrict__ T,
                                                              double* __restrict__ W0, double* __restrict__ W1) {
    const PanelDesc d = desc[d0 + blockIdx.y];
    if (d.problem < 0 || !d.blk) return;
    const ProblemInfo& pi = pinfo[d.problem];
    const Panel P = panel_of<Row>(pi, d, rows);
    const double* gp = NW > 1 && g ? g + pi.s_off : nullptr;
    for (int t = blockIdx.x * kExpThreads + threadIdx.x; t < 2 * P.nblk; t += gridDim.x * kExpThreads)
        expand_block<Row, NW>(P, t >> 1, t & 1, w + pi.w_off, gp, T, W0, W1);
}

// the scan's panels: kScanMax / kScanStep slots per problem on blockIdx.y
constexpr int kScanSlots = kScanMax / kScanStep;
template <class Row>
__global__ void __launch_bounds__(kExpThreads) k_expand_scan(const ProblemInfo* __restrict__ pinfo, int p0,
                                                             const double* __restrict__ rows,
                                                             double* __restrict__ T) {
    const ProblemInfo& pi = pinfo[p0 + blockIdx.y / kScanSlots];
    const int q = blockIdx.y % kScanSlots;
    if (!pi.upp || q * pi.upp * kScanStep >= pi.n_scan) return;
    const Panel P = panel_of<Row>(pi, scan_panel<Row>(pi, q), rows);
    for (int t = blockIdx.x * kExpThreads + threadIdx.x; t < 2 * P.nblk; t += gridDim.x * kExpThreads)
        expand_block<Row, 0>(P, t >> 1, t & 1, nullptr, nullptr, T, nullptr, nullptr);
}

// ---------------------------------------------------------------------------
// sweeps
// ---------------------------------------------------------------------------
// A warp's ring of chunks in shared memory (1-D bulk copies), sl doubles per
// slot: T records, then the weights' (eigenvector passes), or raw rows
struct PRing {
    double* buf;
    uint64_t* bars;
    unsigned loads;  // identical in all lanes
    int sl;
};

__device__ __forceinline__ PRing make_ring(unsigned char* smem, int wid, int sl) {
    PRing R;
    R.sl = sl;
    R.buf = reinterpret_cast<double*>(smem) + (size_t)wid * kPBuf * sl;
    R.bars = reinterpret_cast<uint64_t*>(smem + (size_t)kPWarps * kPBuf * sl * 8) + wid * kPBuf;
    R.loads = 0;
    if ((threadIdx.x & 31) == 0) {
        for (int k = 0; k < kPBuf; ++k) mbar_init(&R.bars[k], 1);
        fence_mbar_init();
    }
    __syncwarp();
    return R;
}
template <int kSl>
constexpr size_t kRingBytes = (size_t)kPWarps * kPBuf * (kSl * 8 + 8);

// Streams n chunks through the ring: issue(slot buffer, barrier, c) starts the
// copies of chunk c, use(slot buffer, c) consumes it (all lanes).
template <class Issue, class Use>
__device__ __forceinline__ void ring_stream(PRing& R, int n, unsigned* err, Issue issue, Use use) {
    const int lane = threadIdx.x & 31;
    const unsigned base = R.loads;
    auto start = [&](int c) {
        const int slot = (base + c) % kPBuf;
        issue(R.buf + slot * R.sl, &R.bars[slot], c);
    };
    if (lane == 0) {
        fence_proxy_async();
        for (int c = 0; c < n && c < kPBuf; ++c) start(c);
    }
    __syncwarp();
    for (int c = 0; c < n; ++c) {
        const unsigned k = base + c;
        const int slot = k % kPBuf;
        mbar_wait_bounded(&R.bars[slot], (k / kPBuf) & 1u, err);
        use(R.buf + slot * R.sl, c);
        __syncwarp();
        if (lane == 0 && c + kPBuf < n) {
            fence_proxy_async();
            start(c + kPBuf);
        }
    }
    R.loads = base + n;
}

// n2 at a shift x where the panel's centre does not tell, by the rows of block b
template <class Row>
__device__ __forceinline__ int rows_zeros(const Panel& P, int b, double x) {
    double u = 0.0, e = 1.0;
    unsigned prev = 0u;
    int n = 0;
    const int end = min(P.nz, (b + 1) * P.blk);
#pragma unroll 1
    for (int i = b * P.blk; i < end; ++i) {
        e = fma(-Row::sigma(P.rows, i, x), u, e);
        u += e;
        n += static_cast<int>(neg(u) ^ prev);
        prev = neg(u);
    }
    return n;
}

// n2 at t from that at the panel's centre and the sign of T12 there
__device__ __forceinline__ int zeros_here(double T12, double t, int n2) {
    return neg(T12) != static_cast<unsigned>(n2 & 1) ? n2 + (t > 0.0 ? -1 : 1) : n2;
}
// sign changes of a chain across a block: u before, un after
__device__ __forceinline__ int block_zeros(double u, double un, int n2) {
    return n2 + static_cast<int>((neg(u) ^ neg(un)) ^ static_cast<unsigned>(n2 & 1));
}

__device__ __forceinline__ void scale2(double& a, double& b) {
    const int sh = rescale_shift(a, b);
    if (sh) {
        const double sc = pow2(-sh);
        a *= sc;
        b *= sc;
    }
}

// the four entries of two blocks at NC shifts per lane: 8 NC independent Horner
// chains, so a lone warp keeps the FP64 pipe busy over their latency
template <int NC>
__device__ __forceinline__ void horner_blocks(const double* __restrict__ c0, const double* __restrict__ c1,
                                              const double (&t)[2][NC], double (&p)[2][NC][4]) {
    const double2* q[2] = {reinterpret_cast<const double2*>(c0), reinterpret_cast<const double2*>(c1)};
#pragma unroll
    for (int k = kPD; k >= 0; --k)
#pragma unroll
        for (int b = 0; b < 2; ++b) {
            const double2 v = q[b][2 * k], w = q[b][2 * k + 1];
            const double cf[4] = {v.x, v.y, w.x, w.y};
#pragma unroll
            for (int n = 0; n < NC; ++n)
#pragma unroll
                for (int j = 0; j < 4; ++j) p[b][n][j] = k == kPD ? cf[j] : fma(p[b][n][j], t[b][n], cf[j]);
        }
}

// ---------------------------------------------------------------------------
// Rows as they are, where a panel has no records: the recurrence u_i = (2 -
// sigma_i) u_{i-1} - u_{i-2}, upwards from the ground and, the same with the
// indices reversed, downwards from the upper boundary (b), over half of the
// rows each.  Two instructions a row and shift for a count, six with two
// derivatives, five for a vector with one weight: what blocks of 32 rows cost
// (see panel_min_blk).  The rows run through the warp's ring.
// ---------------------------------------------------------------------------
template <class Row>
constexpr int kStage = 128 / Row::kW;  // rows of a chunk
static_assert(128 <= kTD, "a slot holds a chunk of rows");
constexpr int kRun = 16;  // rows between rescalings
// (the sweeps are functions of their own, so that the code of the block sweeps
// stays what it is; the ring's count comes back with their results)

// Rows [i0, i1), downwards or up, in runs of at most kRun rows that start at
// multiples of it: run(rows, x, lo, n) for the rows lo .. lo + n - 1, with x[k]
// their values of the NX further arrays xs.
template <class Row, int NX, bool kDown, class Run>
__device__ __forceinline__ void rows_sweep(const Panel& P, int i0, int i1, PRing& R, unsigned* err,
                                           const double* const* xs, Run run) {
    constexpr int kS = kStage<Row>;
    const int c0 = i0 / kS, nc = i1 > i0 ? (i1 + kS - 1) / kS - c0 : 0;
    ring_stream(
        R, nc, err,
        [&](double* dst, uint64_t* bar, int o) {
            const size_t c = kDown ? c0 + nc - 1 - o : c0 + o;
            mbar_expect_tx(bar, (128 + NX * kS) * 8);
            tma_load_1d(dst, P.rows + c * 128, 128 * 8, bar);
#pragma unroll
            for (int k = 0; k < NX; ++k) tma_load_1d(dst + kTD + k * kWD, xs[k] + c * kS, kS * 8, bar);
        },
        [&](const double* buf, int o) {
            const int first = (kDown ? c0 + nc - 1 - o : c0 + o) * kS;
            for (int q = 0; q < kS / kRun; ++q) {
                const int a = first + kRun * (kDown ? kS / kRun - 1 - q : q);
                const int lo = max(a, i0), n = min(a + kRun, i1) - lo;
                if (n > 0) run(buf + (lo - first) * Row::kW, buf + kTD + (lo - first), lo, n);
            }
        });
}
// f(j) for the n rows of a run in order
template <bool kDown, class F>
__device__ __forceinline__ void run_rows(int n, F f) {
    if (n == kRun) {
#pragma unroll
        for (int j = 0; j < kRun; ++j) f(kDown ? kRun - 1 - j : j);
    } else {
        for (int j = 0; j < n; ++j) f(kDown ? n - 1 - j : j);
    }
}

// sign changes over the last m rows: their signs in the low bits, the one before
// them above
__device__ __forceinline__ int run_zeros(unsigned bits, int m) {
    return __popc((bits ^ (bits >> 1)) & ((1u << m) - 1u));
}

// Counts of NC shifts per lane by rows: the sign changes z of a chain over rows
// [0, h) upwards, with v = u_h and w = u_{h-1}, or over rows (h, nz) downwards,
// with v = b_h and w = b_{h-1}.
template <int NC>
struct RowCounts {
    static constexpr int kSize = NC > 0 ? NC : 1;
    double v[kSize], w[kSize];
    int z[kSize];
    unsigned loads;
};
template <class Row, int NC, bool kDown>
struct CountRows {
    static constexpr int kSize = NC > 0 ? NC : 1;
    double u[kSize], um[kSize];
    unsigned bits[kSize];
    int z[kSize];
    typename Row::At at[kSize];
    __device__ __forceinline__ CountRows(const Panel& P, double x0, double x1) {
#pragma unroll
        for (int n = 0; n < NC; ++n) {
            u[n] = 1.0;
            um[n] = kDown ? 0.0 : P.um0;
            z[n] = 0;
            bits[n] = 0u;
            at[n] = typename Row::At(n ? x1 : x0);
        }
    }
    __device__ __forceinline__ void row(const double* r) {
#pragma unroll
        for (int n = 0; n < NC; ++n) {
            const double un = fma(at[n].turn(r), u[n], -um[n]);
            um[n] = u[n];
            u[n] = un;
            bits[n] = __funnelshift_l(__double2hiint(un), bits[n], 1);
        }
    }
    __device__ __forceinline__ void fold(int m) {
#pragma unroll
        for (int n = 0; n < NC; ++n) {
            z[n] += run_zeros(bits[n], m);
            scale2(u[n], um[n]);
        }
    }
    __device__ __forceinline__ void end(RowCounts<NC>& out) const {
#pragma unroll
        for (int n = 0; n < NC; ++n) {
            out.v[n] = kDown ? um[n] : u[n];
            out.w[n] = kDown ? u[n] : um[n];
            // row h is the joint's
            out.z[n] = z[n] - (kDown ? 0 : static_cast<int>(neg(u[n]) ^ neg(um[n])));
        }
    }
};
template <class Row, int NC, bool kDown>
__device__ __noinline__ RowCounts<NC> rows_count(const Panel P, double x0, double x1, int h, PRing R, unsigned* err) {
    CountRows<Row, NC, kDown> C(P, x0, x1);
    rows_sweep<Row, 0, kDown>(P, kDown ? h + 1 : 0, kDown ? P.nz : h + 1, R, err, nullptr,
                              [&](const double* r, const double*, int, int m) {
                                  run_rows<kDown>(m, [&](int j) { C.row(r + j * Row::kW); });
                                  C.fold(m);
                              });
    RowCounts<NC> out;
    C.end(out);
    out.loads = R.loads;
    return out;
}

// the count from both ends' chains at row h (values v at h and w at h - 1,
// sign changes z): those of u over all rows are z + z' and one more or none at
// the joint (the inertia of the twisted factorisation), by the sign of u_{nz-1}
// = w b_h - ... , the chains' Wronskian
__device__ __forceinline__ int rows_join(int nz, double u, double um, int zu, double b, double bm, int zb) {
    const int z = zu + zb;
    return nz - z - static_cast<int>(neg(u * bm - um * b) ^ static_cast<unsigned>(z & 1));
}

// ---------------------------------------------------------------------------
// Laguerre sweeps, in four segments of the blocks: the first runs a state
// upwards (u), the last one downwards (b), those between the two columns of
// their transfer matrices, all with first and half second derivatives in t.
// Put together, W = u e^b - e u^b is -u_{nz-1}, the determinant up to sign, and
// its derivatives follow by the product rule.  An isolated eigenvalue needs no
// counts: the sign of the determinant is the parity of the count.
// ---------------------------------------------------------------------------
struct LagChain {
    double u, e, u1, e1, u2, e2;
    __device__ __forceinline__ void rescale() {
        const int sh = rescale_shift(fmax(fmax(fabs(u), fabs(u1)), fabs(u2)), fmax(fmax(fabs(e), fabs(e1)), fabs(e2)));
        if (sh) {
            const double sc = pow2(-sh);
            u *= sc;
            e *= sc;
            u1 *= sc;
            e1 *= sc;
            u2 *= sc;
            e2 *= sc;
        }
    }
};

// two chains by a common factor
__device__ __forceinline__ void rescale_pair(LagChain& A, LagChain& B) {
    const double mu = fmax(fmax(fmax(fabs(A.u), fabs(A.u1)), fabs(A.u2)), fmax(fmax(fabs(B.u), fabs(B.u1)), fabs(B.u2)));
    const double me = fmax(fmax(fmax(fabs(A.e), fabs(A.e1)), fabs(A.e2)), fmax(fmax(fabs(B.e), fabs(B.e1)), fabs(B.e2)));
    const int sh = rescale_shift(mu, me);
    if (sh) {
        const double sc = pow2(-sh);
        for (LagChain* C : {&A, &B}) {
            C->u *= sc;
            C->e *= sc;
            C->u1 *= sc;
            C->e1 *= sc;
            C->u2 *= sc;
            C->e2 *= sc;
        }
    }
}

// entries at t with first (d) and, for k2, half second (s) derivatives
template <bool k2>
__device__ __forceinline__ void horner_der(const double* __restrict__ c, double t, double (&p)[4], double (&d)[4],
                                           double (&s)[4]) {
    const double2* q = reinterpret_cast<const double2*>(c);
#pragma unroll
    for (int k = kPD; k >= 0; --k) {
        const double2 v = q[2 * k], w = q[2 * k + 1];
        const double cf[4] = {v.x, v.y, w.x, w.y};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            if (k2 && k < kPD - 1) s[j] = k == kPD - 2 ? d[j] : fma(s[j], t, d[j]);
            if (k < kPD) d[j] = k == kPD - 1 ? p[j] : fma(d[j], t, p[j]);
            p[j] = k == kPD ? cf[j] : fma(p[j], t, cf[j]);
        }
    }
    if (!k2) s[0] = s[1] = s[2] = s[3] = 0.0;
}

// one block's matrix on a chain: values, first and half second derivatives
template <class Row>
__device__ __forceinline__ void lag_step(const double (&p)[4], const double (&d)[4], const double (&s)[4],
                                         LagChain& C) {
    double u2 = 0.0, e2 = 0.0;
    if (Row::kLaguerre) {
        u2 = fma(p[0], C.u2, p[1] * C.e2) + fma(d[0], C.u1, d[1] * C.e1) + fma(s[0], C.u, s[1] * C.e);
        e2 = fma(p[2], C.u2, p[3] * C.e2) + fma(d[2], C.u1, d[3] * C.e1) + fma(s[2], C.u, s[3] * C.e);
    }
    const double u1 = fma(p[0], C.u1, p[1] * C.e1) + fma(d[0], C.u, d[1] * C.e);
    const double e1 = fma(p[2], C.u1, p[3] * C.e1) + fma(d[2], C.u, d[3] * C.e);
    const double u = fma(p[0], C.u, p[1] * C.e), e = fma(p[2], C.u, p[3] * C.e);
    C = LagChain{u, e, u1, e1, u2, e2};
}

// NC chains through the chunks [c0, c1), upwards or down
template <class Row, int NC>
__device__ __forceinline__ void lag_segment(const Panel& P, const double* __restrict__ Trec, double x, int c0, int c1,
                                            bool down, PRing& R, unsigned* err, LagChain (&C)[NC]) {
    const typename Row::Shift sh(P, x);
    const double* src = Trec + (size_t)P.rec * kRecT;
    ring_stream(
        R, max(c1 - c0, 0), err,
        [&](double* dst, uint64_t* bar, int o) {
            const size_t c = down ? c1 - 1 - o : c0 + o;
            mbar_expect_tx(bar, kTD * 8);
            tma_load_1d(dst, src + c * kTD, kTD * 8, bar);
        },
        [&](const double* buf, int o) {
            const int c = down ? c1 - 1 - o : c0 + o, nb = min(kPanelChunk, P.nblk - c * kPanelChunk);
            for (int i = 0; i < nb; ++i) {
                const double* rec = buf + (down ? nb - 1 - i : i) * kRecT;
                double p[4], d[4], s[4];
                horner_der<Row::kLaguerre>(rec, sh.at(rec), p, d, s);
                if (down) {  // the inverses: (u, e) -> (p3 u - p1 e, p0 e - p2 u)
                    const double m[4] = {p[3], -p[1], -p[2], p[0]}, f[4] = {d[3], -d[1], -d[2], d[0]},
                                 g[4] = {s[3], -s[1], -s[2], s[0]};
#pragma unroll
                    for (int n = 0; n < NC; ++n) lag_step<Row>(m, f, g, C[n]);
                } else {
#pragma unroll
                    for (int n = 0; n < NC; ++n) lag_step<Row>(p, d, s, C[n]);
                }
            }
            if (NC == 1) C[0].rescale();
            else rescale_pair(C[0], C[NC - 1]);
        });
}

// The same by rows, up over [0, nz / 2) or down over the others, with the sign
// changes z as of rows_count (their joint is row nz / 2 - 1).
struct RowLag {
    LagChain C;
    int z;
    unsigned loads;
};
template <class Row, bool kDown>
struct LagRows {
    LagChain U;  // e: the value before
    unsigned bits = 0u;
    int z = 0;
    typename Row::At at;
    __device__ __forceinline__ LagRows(const Panel& P, double x)
        : U{1.0, kDown ? 0.0 : P.um0, 0.0, 0.0, 0.0, 0.0}, at(x) {}
    __device__ __forceinline__ void row(const double* r) {
        double sl;
        const double q = at.turn(r, sl);
        double u2 = 0.0;
        if (Row::kLaguerre) u2 = fma(q, U.u2, U.u1 - U.e2);
        const double u1 = Row::kLaguerre ? fma(q, U.u1, U.u - U.e1) : fma(q, U.u1, fma(sl, U.u, -U.e1));
        const double u = fma(q, U.u, -U.e);
        bits = __funnelshift_l(__double2hiint(u), bits, 1);
        U = LagChain{u, U.u, u1, U.u1, u2, U.u2};
    }
    __device__ __forceinline__ void fold(int m) {
        z += run_zeros(bits, m);
        U.rescale();
    }
    // the state before row nz / 2; the derivative was taken over kSlope
    __device__ __forceinline__ void end(RowLag& out) const {
        constexpr double k = Row::kSlope;
        out.z = z - (kDown ? 0 : static_cast<int>(neg(U.u) ^ neg(U.e)));
        if (kDown) out.C = {U.e, U.e - U.u, k * U.e1, k * (U.e1 - U.u1), U.e2, U.e2 - U.u2};
        else out.C = {U.u, U.u - U.e, k * U.u1, k * (U.u1 - U.e1), U.u2, U.u2 - U.e2};
    }
};
template <class Row, bool kDown>
__device__ __noinline__ RowLag rows_lag(const Panel P, double x, PRing R, unsigned* err) {
    LagRows<Row, kDown> C(P, x);
    const int h = P.nz / 2;
    rows_sweep<Row, 0, kDown>(P, kDown ? h : 0, kDown ? P.nz : h, R, err, nullptr,
                              [&](const double* r, const double*, int, int m) {
                                  run_rows<kDown>(m, [&](int j) { C.row(r + j * Row::kW); });
                                  C.fold(m);
                              });
    RowLag out;
    C.end(out);
    out.loads = R.loads;
    return out;
}

// Both directions in one warp, row by row in turn, so that it has twice the
// chains in flight: the Laguerre chains of xa (kLag) and the counts of NC shifts.
template <int NC>
struct RowBoth {
    RowLag L[2];
    RowCounts<NC> K[2];
    unsigned loads;
};
template <class Row, bool kLag, int NC>
__device__ __noinline__ RowBoth<NC> rows_both(const Panel P, double xa, double x0, double x1, PRing R, unsigned* err) {
    constexpr int kS = kStage<Row>, kW = Row::kW;
    static_assert(kTD + 128 <= kTD + kWD, "a slot with one weight holds two chunks of rows");
    LagRows<Row, false> lu(P, xa);
    LagRows<Row, true> ld(P, xa);
    CountRows<Row, NC, false> cu(P, x0, x1);
    CountRows<Row, NC, true> cd(P, x0, x1);
    // the counts' joint is row h, the Laguerre chains meet before it: row h is taken
    // by the upward counts and by the downward Laguerre chain apart
    const int h = P.nz / 2, top = (P.nz - 1) / kS;
    const int nf = h / kS + 1, nb = top - h / kS + 1;  // chunks with rows [0, h], [h, nz)
    auto up = [&](const double* r, bool last) {
        if (kLag && !last) lu.row(r);
        cu.row(r);
    };
    auto dn = [&](const double* r, bool last) {
        if (kLag) ld.row(r);
        if (!last) cd.row(r);
    };
    auto fold_up = [&](int m, int ml) {
        if (kLag && ml) lu.fold(ml);
        cu.fold(m);
    };
    auto fold_dn = [&](int m, int mc) {
        if (kLag) ld.fold(m);
        if (mc) cd.fold(mc);
    };
    ring_stream(
        R, max(nf, nb), err,
        [&](double* dst, uint64_t* bar, int o) {
            mbar_expect_tx(bar, ((o < nf) + (o < nb)) * 128 * 8);
            if (o < nf) tma_load_1d(dst, P.rows + (size_t)o * 128, 128 * 8, bar);
            if (o < nb) tma_load_1d(dst + kTD, P.rows + (size_t)(top - o) * 128, 128 * 8, bar);
        },
        [&](const double* buf, int o) {
            int f = o * kS, b = o < nb ? min(P.nz, (top - o + 1) * kS) : 0;  // next row up; behind the next one down
            const int f1 = o < nf ? min(h + 1, f + kS) : f, b0 = o < nb ? max(h, (top - o) * kS) : b;
            const double *rf = buf - f * kW, *rb = buf + kTD - (top - o) * kS * kW;
            while (f < f1 || b > b0) {
                const int m = min(kRun, f1 - f), n = b - max(b0, (b - 1) / kRun * kRun);
                if (m == kRun && n == kRun && f + kRun <= h && b - kRun > h) {
                    const double *p = rf + f * kW, *q = rb + (b - kRun) * kW;
#pragma unroll
                    for (int j = 0; j < kRun; ++j) {
                        up(p + j * kW, false);
                        dn(q + (kRun - 1 - j) * kW, false);
                    }
                    fold_up(kRun, kRun);
                    fold_dn(kRun, kRun);
                } else {
                    if (m > 0) {
                        for (int j = 0; j < m; ++j) up(rf + (f + j) * kW, f + j == h);
                        fold_up(m, m - (f + m > h));
                    }
                    if (n > 0) {
                        for (int j = 0; j < n; ++j) dn(rb + (b - 1 - j) * kW, b - 1 - j == h);
                        fold_dn(n, n - (b - n == h));
                    }
                }
                f += max(m, 0);
                b -= max(n, 0);
            }
        });
    RowBoth<NC> out;
    lu.end(out.L[0]);
    ld.end(out.L[1]);
    cu.end(out.K[0]);
    cd.end(out.K[1]);
    out.loads = R.loads;
    return out;
}

// the two columns of NC transfer matrices by a common factor
template <int NC>
__device__ __forceinline__ void rescale_columns(double (&u)[NC], double (&e)[NC], double (&v)[NC], double (&f)[NC]) {
#pragma unroll
    for (int n = 0; n < NC; ++n) {
        const int s = rescale_shift(fmax(fabs(u[n]), fabs(v[n])), fmax(fabs(e[n]), fabs(f[n])));
        if (s) {
            const double sc = pow2(-s);
            u[n] *= sc;
            e[n] *= sc;
            v[n] *= sc;
            f[n] *= sc;
        }
    }
}

// The transfer matrix of the chunks [c0, c1) at NC shifts per lane (its two
// columns u, e and v, f up to a common scale) and the sign changes of the
// column that starts with u = 0 (v), by which those of any state that enters
// follow from the parity.
template <class Row, int NC>
__device__ __forceinline__ void count_segment(const Panel& P, const double* __restrict__ Trec, const double (&x)[NC],
                                              int c0, int c1, PRing& R, unsigned* err, double (&u)[NC],
                                              double (&e)[NC], double (&v)[NC], double (&f)[NC], int (&zeros)[NC]) {
    typename Row::Shift sh[NC];
#pragma unroll
    for (int n = 0; n < NC; ++n) {
        u[n] = f[n] = 1.0;
        e[n] = v[n] = 0.0;
        zeros[n] = 0;
        sh[n] = typename Row::Shift(P, x[n]);
    }
    const double* src = Trec + (size_t)P.rec * kRecT;
    ring_stream(
        R, max(c1 - c0, 0), err,
        [&](double* dst, uint64_t* bar, int o) {
            mbar_expect_tx(bar, kTD * 8);
            tma_load_1d(dst, src + (size_t)(c0 + o) * kTD, kTD * 8, bar);
        },
        [&](const double* rec, int o) {
            const int nb = min(kPanelChunk, P.nblk - (c0 + o) * kPanelChunk);
            for (int q = 0; q < nb; q += 2, rec += 2 * kRecT) {
                double p[2][NC][4], t[2][NC];
#pragma unroll
                for (int n = 0; n < NC; ++n) {
                    t[0][n] = sh[n].at(rec);
                    t[1][n] = sh[n].at(rec + kRecT);
                }
                horner_blocks<NC>(rec, rec + kRecT, t, p);
#pragma unroll
                for (int b = 0; b < 2; ++b) {
                    if (q + b >= nb) break;
                    const int n2 = __double2loint(rec[b * kRecT + kRecZeros]);
#pragma unroll
                    for (int n = 0; n < NC; ++n) {
                        const double(&m)[4] = p[b][n];
                        const double un = fma(m[0], u[n], m[1] * e[n]), vn = fma(m[0], v[n], m[1] * f[n]);
                        e[n] = fma(m[2], u[n], m[3] * e[n]);
                        f[n] = fma(m[2], v[n], m[3] * f[n]);
                        zeros[n] += block_zeros(v[n], vn, zeros_here(m[1], t[b][n], n2));
                        u[n] = un;
                        v[n] = vn;
                    }
                }
            }
            rescale_columns(u, e, v, f);
        });
    if (zeros[0] < kByRows) return;
    // some block has its count from its rows: the sweep again, a block at a time
#pragma unroll
    for (int n = 0; n < NC; ++n) {
        u[n] = f[n] = 1.0;
        e[n] = v[n] = 0.0;
        zeros[n] = 0;
    }
    ring_stream(
        R, c1 - c0, err,
        [&](double* dst, uint64_t* bar, int o) {
            mbar_expect_tx(bar, kTD * 8);
            tma_load_1d(dst, src + (size_t)(c0 + o) * kTD, kTD * 8, bar);
        },
        [&](const double* buf, int o) {
            const int b0 = (c0 + o) * kPanelChunk, nb = min(kPanelChunk, P.nblk - b0);
#pragma unroll 1
            for (int q = 0; q < nb; ++q) {
                const double* rec = buf + q * kRecT;
                const int n2 = __double2loint(rec[kRecZeros]);
#pragma unroll
                for (int n = 0; n < NC; ++n) {
                    const double t = sh[n].at(rec);
                    double m[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll 1
                    for (int k = kPD; k >= 0; --k)
#pragma unroll
                        for (int j = 0; j < 4; ++j) m[j] = fma(m[j], t, rec[4 * k + j]);
                    const int z = n2 >= kByRows ? rows_zeros<Row>(P, b0 + q, x[n]) : zeros_here(m[1], t, n2);
                    const double un = fma(m[0], u[n], m[1] * e[n]), vn = fma(m[0], v[n], m[1] * f[n]);
                    e[n] = fma(m[2], u[n], m[3] * e[n]);
                    f[n] = fma(m[2], v[n], m[3] * f[n]);
                    zeros[n] += block_zeros(v[n], vn, z);
                    u[n] = un;
                    v[n] = vn;
                }
            }
            rescale_columns(u, e, v, f);
        });
}

// ---------------------------------------------------------------------------
// Isolation scan: units of kScanStep shifts, a CTA each, whose four warps take
// a quarter of the blocks: with one warp to a unit a single problem's scan was
// a chain of 157 blocks on 2 to 8 warps (0.1 Hz 49 us, 2 Hz 183 us; now 22 and 73),
// and that of 256 problems ended with half of the chip idle (143 us, now 89).  The
// second column costs 8 more instructions a block next to 120 of Horner's rule.
// ---------------------------------------------------------------------------
template <class Row>
__global__ void __launch_bounds__(kPWarps * 32) k_panel_scan(const ProblemInfo* __restrict__ pinfo,
                                                             const double* __restrict__ rows,
                                                             const double* __restrict__ T, int* __restrict__ counts,
                                                             unsigned* err) {
    extern __shared__ __align__(128) unsigned char smem_raw[];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int p = blockIdx.x / kScanSlots, unit = blockIdx.x % kScanSlots;
    const ProblemInfo& pi = pinfo[p];
    const int n = pi.n_scan;
    if (unit * kScanStep >= n) return;
    PRing R = make_ring(smem_raw, wid, kTD);
    const Panel P = panel_of<Row>(pi, scan_panel<Row>(pi, pi.upp ? unit / pi.upp : 0), rows);
    const int t0 = unit * kScanStep + 2 * lane;
    const double lo = Row::lo(pi), hi = Row::hi(pi);
    const double x[2] = {scan_x(lo, hi, t0, n), scan_x(lo, hi, t0 + 1, n)};
    int c[2];
    struct Seg {
        double m[4][2][32];
        int z[2][32];
    };
    Seg* box = reinterpret_cast<Seg*>(smem_raw + kRingBytes<kTD>);
    if (!P.blk) {  // by rows: a warp takes one of the two shifts over half of them
        const int h = P.nz / 2, k = wid >> 1;
        const double xk = k ? x[1] : x[0];
        const auto o = wid & 1 ? rows_count<Row, 1, true>(P, xk, 0.0, h, R, err)
                               : rows_count<Row, 1, false>(P, xk, 0.0, h, R, err);
        box[wid].m[0][0][lane] = o.v[0];
        box[wid].m[1][0][lane] = o.w[0];
        box[wid].z[0][lane] = o.z[0];
        __syncthreads();
        if (wid) return;
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            const Seg &U = box[2 * k], &B = box[2 * k + 1];
            c[k] = rows_join(P.nz, U.m[0][0][lane], U.m[1][0][lane], U.z[0][lane], B.m[0][0][lane], B.m[1][0][lane],
                             B.z[0][lane]);
        }
    } else {
        const int nch = (P.nblk + kPanelChunk - 1) / kPanelChunk;
        double u[2], e[2], v[2], f[2];
        int z[2];
        count_segment<Row, 2>(P, T, x, nch * wid / kPWarps, nch * (wid + 1) / kPWarps, R, err, u, e, v, f, z);
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            box[wid].m[0][k][lane] = u[k];
            box[wid].m[1][k][lane] = e[k];
            box[wid].m[2][k][lane] = v[k];
            box[wid].m[3][k][lane] = f[k];
            box[wid].z[k][lane] = z[k];
        }
        __syncthreads();
        if (wid) return;
#pragma unroll
        for (int k = 0; k < 2; ++k) {  // the state (1, e0) through the segments
            double a = 1.0, b = P.e0;
            int zeros = 0;
            for (int s = 0; s < kPWarps; ++s) {
                const double an = fma(box[s].m[0][k][lane], a, box[s].m[2][k][lane] * b);
                b = fma(box[s].m[1][k][lane], a, box[s].m[3][k][lane] * b);
                const int n2 = box[s].z[k][lane];
                zeros += n2 + static_cast<int>((neg(a) ^ neg(an)) ^ static_cast<unsigned>(n2 & 1));
                a = an;
                scale2(a, b);
            }
            c[k] = P.nz - zeros;
        }
    }
    *reinterpret_cast<int2*>(counts + (size_t)p * kScanMax + t0) = make_int2(c[0], c[1]);
}

// ---------------------------------------------------------------------------
// work items
// ---------------------------------------------------------------------------
constexpr int kItemThreads = 1024;

__device__ int block_scan(int v, int* sh, int* total) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    int incl = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int a = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += a;
    }
    __syncthreads();  // sh free
    if (lane == 31) sh[wid] = incl;
    __syncthreads();
    if (wid == 0) {
        int w = sh[lane];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int a = __shfl_up_sync(0xffffffffu, w, o);
            if (lane >= o) w += a;
        }
        sh[lane] = w;
    }
    __syncthreads();
    *total = sh[31];
    return incl - v + (wid ? sh[wid - 1] : 0);
}

// One CTA: per problem the mode number, the CSR offset and the place of its
// items in the list.  With order set and P <= kRankMax the problems are listed
// by the cost of an item, nz x m x (1 + M / 512) (m eigenvalues of a problem
// with M: denser windows need more rounds), heaviest first, and
// taken in that order as teams get free.
constexpr int kRankMax = 4096;

__global__ void __launch_bounds__(kItemThreads) k_panel_items(int P, ProblemInfo* __restrict__ pinfo,
                                                              const int* __restrict__ counts, int max_modes,
                                                              int bis_item, int cap, int* __restrict__ tot, bool first,
                                                              unsigned* __restrict__ err, int order) {
    __shared__ int sh[32];
    __shared__ float skey[kRankMax];
    __shared__ int sperm[kRankMax];
    const bool ranked = order != 0 && P <= kRankMax;
    int base_m = first ? 0 : tot[2];
    for (int p0 = 0; p0 < P; p0 += kItemThreads) {
        const int p = p0 + threadIdx.x;
        int M = 0;
        if (p < P) {
            const ProblemInfo& pi = pinfo[p];
            const int c_lo = counts[(size_t)p * kScanMax], c_hi = counts[(size_t)p * kScanMax + pi.n_scan - 1];
            M = max(0, c_hi - c_lo);
            if (M > max_modes) {
                atomicOr(err, kErrTooMany);
                M = max_modes;
            }
            pinfo[p].c_lo = c_lo;
            pinfo[p].c_hi = c_hi;
            pinfo[p].M = M;
            const int nb = (M + bis_item - 1) / bis_item;
            if (ranked)
                skey[p] = nb > 0 ? (float)pi.nz * ((float)M / (float)nb) * (1.0f + (float)M * (1.0f / 512.0f)) : 0.f;
        }
        int tm;
        const int om = block_scan(M, sh, &tm);
        if (p < P) pinfo[p].off = base_m + om;
        base_m += tm;
    }
    __syncthreads();
    if (ranked) {
        for (int p = threadIdx.x; p < P; p += kItemThreads) {
            const float kp = skey[p];
            int r = 0;
            for (int q = 0; q < P; ++q) {
                const float kq = skey[q];
                r += (kq > kp || (kq == kp && q < p)) ? 1 : 0;
            }
            sperm[r] = p;
        }
        __syncthreads();
    }
    int base = 0;
    for (int r0 = 0; r0 < P; r0 += kItemThreads) {
        const int r = r0 + threadIdx.x;
        const int p = r < P ? (ranked ? sperm[r] : r) : 0;
        const int nb = r < P ? (pinfo[p].M + bis_item - 1) / bis_item : 0;
        int tb;
        const int ob = block_scan(nb, sh, &tb);
        if (r < P) pinfo[p].item0 = base + ob;
        base += tb;
    }
    if (threadIdx.x == 0) {
        if (base > cap) atomicOr(err, kErrTooMany);
        tot[0] = min(base, cap);
        tot[1] = min(base, cap);
        tot[2] = base_m;
        tot[5] = first ? 0 : tot[5] + tot[3];
        tot[3] = tot[4] = 0;
    }
}

// index of the last scan point with a count <= J (counts are monotone; a
// rounding slip between neighbours still ends at a valid bracket)
__device__ __forceinline__ int scan_bracket(const int* __restrict__ cnt, int n, int J) {
    int t0 = 0, t1 = n - 1;
    while (t1 - t0 > 1) {
        const int t = (t0 + t1) >> 1;
        if (cnt[t] <= J) t0 = t;
        else t1 = t;
    }
    return t0;
}

// One warp per problem: its items (at most bis_item consecutive eigenvalues,
// balanced) and their panels.  Consecutive items share a panel while their
// brackets fit kRhoMax at the largest block; an item too wide for that gets
// its own panel and a smaller block.  Items beyond the problem's panels or
// records (sized by the host from the profile's sound speeds) keep none and
// sweep the raw rows.
constexpr int kPlanWarps = 2, kPlanItems = 256;
template <class Row>
__global__ void __launch_bounds__(kPlanWarps * 32) k_panel_groups(int P, const ProblemInfo* __restrict__ pinfo,
                                                                  const int* __restrict__ counts, int bis_item,
                                                                  WorkItem* __restrict__ items, int cap,
                                                                  PanelDesc* __restrict__ desc,
                                                                  int* __restrict__ tot) {
    __shared__ double xa[kPlanWarps][kPlanItems], xb[kPlanWarps][kPlanItems];
    __shared__ int grp[kPlanWarps][kPlanItems];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int p = blockIdx.x * kPlanWarps + wid;
    if (p >= P) return;
    const ProblemInfo& pi = pinfo[p];
    const int* cnt = counts + (size_t)p * kScanMax;
    const double lo = Row::lo(pi), hi = Row::hi(pi), st = Row::steepness(pi);
    const int M = pi.M, n = pi.n_scan, nb = (M + bis_item - 1) / bis_item;
    const int most = most_rows(Row::span(pi));
    int ng = 0, used = 0;  // panels and records taken so far (warp-uniform)
    for (int k0 = 0; k0 < nb; k0 += kPlanItems) {
        const int m = min(kPlanItems, nb - k0);
        for (int i = lane; i < m; i += 32) {
            const int k = k0 + i;
            const int j0 = (int)((long long)M * k / nb), j1 = (int)((long long)M * (k + 1) / nb);
            const double a = scan_x(lo, hi, scan_bracket(cnt, n, pi.c_lo + j0), n);
            const double b = scan_x(lo, hi, scan_bracket(cnt, n, pi.c_lo + j1 - 1) + 1, n);
            xa[wid][i] = fmin(a, b);
            xb[wid][i] = fmax(a, b);
        }
        __syncwarp();
        if (lane == 0) {
            for (int i = 0; i < m;) {
                const double a = xa[wid][i];
                double b = xb[wid][i];
                int e = i + 1;
                auto wide = [&](double c) {
                    return !(st * (0.5 * (c - a)) * (double)most * (double)most <= kRhoMax);
                };
                if (!wide(b))
                    while (e < m && !wide(fmax(b, xb[wid][e]))) b = fmax(b, xb[wid][e++]);
                PanelDesc d;
                d.xc = 0.5 * (a + b);
                d.r = fmax(0.5 * (b - a), 1e-300);
                d.blk = block_rows(st * d.r, pi.nz, most);
                d.problem = p;
                d.rec = pi.blk_off + used;
                const int need = d.blk ? padded((pi.nz + d.blk - 1) / d.blk) : 0;
                int id = -1;
                if (d.blk && ng < pi.grp_cap && used + need <= pi.blk_cap) {
                    id = pi.grp_off + ng++;
                    desc[id] = d;
                    used += need;
                }
                for (; i < e; ++i) grp[wid][i] = id;
            }
        }
        __syncwarp();
        for (int i = lane; i < m; i += 32) {
            const int k = k0 + i, q = pi.item0 + k;
            const int j0 = (int)((long long)M * k / nb), j1 = (int)((long long)M * (k + 1) / nb);
            if (q < cap) items[q] = WorkItem{p, j0, j1 - j0, grp[wid][i]};
            if (grp[wid][i] < 0) atomicAdd(&tot[3], 1);  // sweeps its rows
        }
        __syncwarp();
        ng = __shfl_sync(0xffffffffu, ng, 0);
        used = __shfl_sync(0xffffffffu, used, 0);
    }
    for (int i = ng + lane; i < pi.grp_cap; i += 32) {
        PanelDesc d{};
        d.problem = -1;
        desc[pi.grp_off + i] = d;
    }
}

// ---------------------------------------------------------------------------
// A work item runs on a pair of warps or on a team of four: of every sweep of its
// eigenvalues they take two or one of four segments of the blocks (so the sums
// are the same), of the eigenvectors the first two take the upward and the
// downward pass.  All keep the state of every slot and take the same decisions
// from what they exchange.
// ---------------------------------------------------------------------------
struct PairBox {
    double v[2][2][3][32];  // [parity][half][value][lane]: of the eigenvector passes
    int c[2][2][32];        // counts
    int err[2][4];
    int item[2];
};

// The W warps (2 or 4) of an item: warp `half` of W.  The segments' results are
// exchanged through the rings, which are idle between sweeps.
template <int W>
struct Team {
    PairBox* box;
    double* area;  // ring of the team's first warp
    int stride;    // doubles of a warp's ring
    int id, half;
    int turn;  // buffer of the next exchange
    __device__ __forceinline__ void sync() const {
        if (W == 1) __syncwarp();
        else asm volatile("bar.sync %0, %1;" ::"r"(1 + id), "n"(32 * W) : "memory");
    }
    // the first two warps
    __device__ __forceinline__ void sync2() const {
        if (W <= 2) sync();
        else asm volatile("bar.sync 8, 64;" ::: "memory");
    }
    // where segment s puts its results (n doubles a segment of the first kind a warp takes)
    __device__ __forceinline__ double* slot(int s, int n) const {
        if (W == 4) return area + s * stride;
        return area + (s >> 1) * stride + ((s == 1 || s == 2) ? n : 0);
    }
    // and set s of 32 shifts by rows, upwards or down
    __device__ __forceinline__ double* rows(int s, bool down) const {
        constexpr int kR = 7 * 32;
        if (W == 4) return area + (2 * s + down) * stride;
        if (W == 2) return area + down * stride + s * kR;
        return area + (2 * s + down) * kR;
    }
};

// position of the n-th (0-based) set bit of m
__device__ __forceinline__ int nth_set(unsigned m, int n) {
    int pos = 0;
#pragma unroll
    for (int sh = 16; sh >= 1; sh >>= 1) {
        const unsigned low = m & ((1u << sh) - 1u);
        const int c = __popc(low);
        if (n >= c) {
            n -= c;
            m >>= sh;
            pos += sh;
        } else {
            m = low;
        }
    }
    return pos;
}

// A round by rows: the Laguerre chains of the first nN of 32 shifts (xe) and the
// counts of the others and of 32 more (xs), or the counts of 64.  The chains stay
// in pr.rows(0, .), the counts of lane v go to c[v >> 5][v & 31].
template <class Row, int W>
__device__ __forceinline__ void rows_round(const Panel& P, const double (&xs)[2], double xe, int nN, int nB, PRing& R,
                                           unsigned* err, Team<W>& pr, int (&c)[2][32]) {
    const int lane = threadIdx.x & 31, h = P.nz / 2;
    const double xa = lane < nN || nB == 0 ? xe : xs[0];
    constexpr int kNC = W == 4 ? 1 : 2, kDirs = W == 1 ? 2 : 1;
    const bool down = W != 1 && (pr.half & 1);
    const int s0 = W == 4 ? pr.half >> 1 : 0;                        // first set of this warp
    const bool lag = nN > 0 && s0 == 0;                              // has Laguerre chains
    const bool count = nN == 0 || (nB > 0 && s0 + kNC == 2);        // has counts,
    const int n0 = nN > 0 ? kNC - 1 : 0;                             // of its sets from this one on
    // the ring is in use until this warp's last sweep: results go there afterwards
    RowLag L[kDirs];
    RowCounts<kNC> K[kDirs];
    auto last = [&](const RowCounts<1>& r, int d) {
        K[d].v[kNC - 1] = r.v[0];
        K[d].w[kNC - 1] = r.w[0];
        K[d].z[kNC - 1] = r.z[0];
    };
    if constexpr (W == 1) {
        if (nN == 0) {
            const auto r = rows_both<Row, false, 2>(P, xa, xs[0], xs[1], R, err);
            K[0] = r.K[0];
            K[1] = r.K[1];
            R.loads = r.loads;
        } else {
            auto keep = [&](const auto& r) {
                L[0] = r.L[0];
                L[1] = r.L[1];
                R.loads = r.loads;
            };
            if (nB > 0) {
                const auto r = rows_both<Row, true, 1>(P, xa, xs[1], 0.0, R, err);
                keep(r);
                last(r.K[0], 0);
                last(r.K[1], 1);
            } else {
                keep(rows_both<Row, true, 0>(P, xa, 0.0, 0.0, R, err));
            }
        }
    } else {
        if (lag) {
            L[0] = down ? rows_lag<Row, true>(P, xa, R, err) : rows_lag<Row, false>(P, xa, R, err);
            R.loads = L[0].loads;
        }
        if (count && nN > 0) {
            const RowCounts<1> r = down ? rows_count<Row, 1, true>(P, xs[1], 0.0, h, R, err)
                                        : rows_count<Row, 1, false>(P, xs[1], 0.0, h, R, err);
            last(r, 0);
            R.loads = r.loads;
        } else if (count) {
            const double x0 = s0 ? xs[1] : xs[0];
            K[0] = down ? rows_count<Row, kNC, true>(P, x0, xs[1], h, R, err)
                        : rows_count<Row, kNC, false>(P, x0, xs[1], h, R, err);
            R.loads = K[0].loads;
        }
    }
    __syncwarp();
#pragma unroll
    for (int d = 0; d < kDirs; ++d) {
        const bool dn = W == 1 ? d == 1 : down;
        if (lag) {
            double* o = pr.rows(0, dn) + lane;
            o[0] = L[d].C.u;
            o[32] = L[d].C.e;
            o[64] = L[d].C.u1;
            o[96] = L[d].C.e1;
            o[128] = L[d].C.u2;
            o[160] = L[d].C.e2;
            o[192] = __hiloint2double(0, L[d].z);
        }
#pragma unroll
        for (int n = 0; n < kNC; ++n) {
            if (!count || n < n0) continue;
            double* o = pr.rows(s0 + n, dn) + lane;
            o[0] = K[d].v[n];
            o[32] = K[d].w[n];
            o[64] = __hiloint2double(0, K[d].z[n]);
        }
    }
    if (nB == 0) return;
    pr.sync();
#pragma unroll
    for (int s = 0; s < 2; ++s) {
        if (W != 1 && pr.half != s) continue;
        const double *a = pr.rows(s, false) + lane, *b = pr.rows(s, true) + lane;
        if (s == 0 && nN > 0) {
            const int z = __double2loint(a[192]) + __double2loint(b[192]);
            const double w0 = a[0] * b[32] - a[32] * b[0];  // -u_{nz-1}
            c[0][lane] = P.nz - z - static_cast<int>((neg(w0) ^ 1u) ^ static_cast<unsigned>(z & 1));
        } else {
            c[s][lane] = rows_join(P.nz, a[0], a[32], __double2loint(a[64]), b[0], b[32], __double2loint(b[64]));
        }
    }
}

// Eigenvalues of a work item (<= 32), lane l owning slot l, to x.  Every round:
// slots isolated in their bracket (Sturm counts J and J + 1 at its ends) take a
// safeguarded Laguerre step; the other virtual lanes (v = lane + 32 half) are
// dealt over the slots not yet isolated and cut their brackets.  A slot is final
// when the correction is below tol, or when the last two steps stayed inside
// the bracket and the cubic model predicts the next one below tol.
template <class Row, int W, bool kRows>
__device__ __forceinline__ double panel_bisect(const ProblemInfo& pi, const Panel& P, const WorkItem& w,
                                               const double* __restrict__ Trec, const int* __restrict__ counts,
                                               double tol_in, unsigned* err, unsigned long long* steps, PRing& R,
                                               Team<W>& pr) {
    const int lane = threadIdx.x & 31;
    const double lo = Row::lo(pi), hi = Row::hi(pi);
    const int nz = pi.nz, n = pi.n_scan;
    const int* cnt = counts + (size_t)w.problem * kScanMax;
    const double tol = tol_in * Row::tol_scale(pi);
    const int J = pi.c_lo + w.j0 + lane;
    double a = P.xc, b = P.xc, x = P.xc;
    double dprev = 0.0;  // size of the previous accepted correction (0: none yet)
    int ca = 0, cb = 0, mode = 2;
    if (lane < w.m) {  // bracket from the scan
        const int t0 = scan_bracket(cnt, n, J);
        ca = cnt[t0];
        cb = cnt[t0 + 1];
        if (!(ca <= J && cb > J)) atomicOr(err, kErrBracket);
        a = scan_x(lo, hi, t0, n);
        b = scan_x(lo, hi, t0 + 1, n);
        x = 0.5 * (a + b);
        mode = !(b - a > tol) ? 2 : ((ca == J && cb == J + 1) ? 1 : 0);
    }
    for (int round = 0; round < 512; ++round) {
        const unsigned nm = __ballot_sync(0xffffffffu, mode == 1);
        const unsigned bm = __ballot_sync(0xffffffffu, mode == 0);
        const int nN = __popc(nm), nB = __popc(bm);
        if (nN + nB == 0) break;
        const int nlB = 64 - nN;
        PairBox& X = *pr.box;
        const int tb = pr.turn;
        pr.turn ^= 1;
        // segments of this warp: one of four, or an end and its neighbour
        constexpr int kSegs = 4 / W;
        auto seg_of = [&](int i) { return W == 4 ? pr.half : (pr.half ? 3 - i : i); };
        const int nch = (P.nblk + kPanelChunk - 1) / kPanelChunk;
        double xs[2] = {x, x}, xe = x;
        if (nB > 0) {  // counts: virtual lanes v = lane, lane + 32 of every warp
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int v = lane + 32 * h;
                const int t = v >= nN ? v - nN : 0, k = t % nB, g = t / nB, G = (nlB - 1 - k) / nB + 1;
                const int e = nth_set(bm, k);
                const double ae = __shfl_sync(0xffffffffu, a, e);
                const double be = __shfl_sync(0xffffffffu, b, e);
                xs[h] = ae + (be - ae) * ((double)(g + 1) / (double)(G + 1));
            }
        }
        // Laguerre chains of slots nth_set(nm, lane)
        if (nN > 0) xe = __shfl_sync(0xffffffffu, x, lane < nN ? nth_set(nm, lane) : 0);
        constexpr int kL = 6 * 32;  // doubles of a chain
        auto put = [&](double* o, const LagChain& C) {
            o[lane] = C.u;
            o[32 + lane] = C.e;
            o[64 + lane] = C.u1;
            o[96 + lane] = C.e1;
            o[128 + lane] = C.u2;
            o[160 + lane] = C.e2;
        };
        if constexpr (kRows) {
            rows_round<Row, W>(P, xs, xe, nN, nB, R, err, pr, X.c[tb]);
        } else {
            if (nB > 0) {
                constexpr int kN = 5 * 64;  // doubles of a segment
                double su[kSegs][2], se[kSegs][2], sv[kSegs][2], sf[kSegs][2];
                int z[kSegs][2];
#pragma unroll
                for (int i = 0; i < kSegs; ++i) {
                    const int s = seg_of(i);
                    count_segment<Row, 2>(P, Trec, xs, nch * s / 4, nch * (s + 1) / 4, R, err, su[i], se[i], sv[i],
                                          sf[i], z[i]);
                }
#pragma unroll
                for (int i = 0; i < kSegs; ++i) {
                    double* o = pr.slot(seg_of(i), kN);
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        const int v = lane + 32 * h;
                        o[v] = su[i][h];
                        o[64 + v] = se[i][h];
                        o[128 + v] = sv[i][h];
                        o[192 + v] = sf[i][h];
                        o[256 + v] = __hiloint2double(0, z[i][h]);
                    }
                }
                pr.sync();
                if (pr.half < 2) {  // shifts lane + 32 half: the state (1, e0) through the segments
                    const int v = lane + 32 * pr.half;
                    double ua = 1.0, eb = P.e0;
                    int zeros = 0;
#pragma unroll
                    for (int s = 0; s < 4; ++s) {
                        const double* o = pr.slot(s, kN);
                        const double un = fma(o[v], ua, o[128 + v] * eb);
                        eb = fma(o[64 + v], ua, o[192 + v] * eb);
                        const int n2 = __double2loint(o[256 + v]);
                        zeros += n2 + static_cast<int>((neg(ua) ^ neg(un)) ^ static_cast<unsigned>(n2 & 1));
                        ua = un;
                        scale2(ua, eb);
                    }
                    X.c[tb][pr.half][lane] = nz - zeros;
                }
                pr.sync();  // the rings are free again
            }
            if (nN > 0) {
                LagChain S[1], M[2];
                S[0] = pr.half ? LagChain{0.0, -1.0, 0.0, 0.0, 0.0, 0.0} : LagChain{1.0, P.e0, 0.0, 0.0, 0.0, 0.0};
                M[0] = LagChain{1.0, 0.0, 0.0, 0.0, 0.0, 0.0};
                M[1] = LagChain{0.0, 1.0, 0.0, 0.0, 0.0, 0.0};
                if (W == 2 || pr.half == 0 || pr.half == 3) {
                    const int s = pr.half ? 3 : 0;
                    lag_segment<Row, 1>(P, Trec, xe, nch * s / 4, nch * (s + 1) / 4, s == 3, R, err, S);
                }
                if (W == 2 || pr.half == 1 || pr.half == 2) {
                    const int s = W == 4 ? pr.half : 1 + pr.half;
                    lag_segment<Row, 2>(P, Trec, xe, nch * s / 4, nch * (s + 1) / 4, false, R, err, M);
                }
                if (W == 2 || pr.half == 0 || pr.half == 3) put(pr.slot(pr.half ? 3 : 0, kL), S[0]);
                if (W == 2 || pr.half == 1 || pr.half == 2) {
                    double* o = pr.slot(W == 4 ? pr.half : 1 + pr.half, kL);
                    put(o, M[0]);
                    put(o + kL, M[1]);
                }
            }
        }
        if (steps && lane == 0 && pr.half == 0) {
            atomicAdd(steps, (unsigned long long)((nB > 0 ? 64 : 0) + (nN > 0 ? 32 : 0)) * (unsigned long long)nz);
            if (nN > 0) atomicAdd(steps + 1, 32ull * (unsigned long long)nz);
        }
        if (lane == 0) X.err[tb][pr.half] = (*((volatile unsigned*)err) & kErrTimeout) != 0u;
        pr.sync();
        if (mode == 1) {
            const int v = __popc(nm & ((1u << lane) - 1u));
            auto get = [&](const double* o) {
                return LagChain{o[v], o[32 + v], o[64 + v], o[96 + v], o[128 + v], o[160 + v]};
            };
            LagChain U = get(kRows ? pr.rows(0, false) : pr.slot(0, kL));
            const LagChain D = get(kRows ? pr.rows(0, true) : pr.slot(3, kL));
            if (!kRows) {
#pragma unroll
                for (int s = 1; s <= 2; ++s) {  // through the segments between
                    const LagChain A = get(pr.slot(s, kL)), B = get(pr.slot(s, kL) + kL);
                    const double m[4] = {A.u, B.u, A.e, B.e}, d[4] = {A.u1, B.u1, A.e1, B.e1},
                                 q[4] = {A.u2, B.u2, A.e2, B.e2};
                    lag_step<Row>(m, d, q, U);
                    U.rescale();
                }
            }
            const double u = U.u, e = U.e, u1 = U.u1, e1 = U.e1, u2 = U.u2, e2 = U.e2;
            const double y = D.u, z = D.e, y1 = D.u1, z1 = D.e1, y2 = D.u2, z2 = D.e2;
            const double w0 = u * z - e * y;
            const double w1 = u1 * z + u * z1 - (e1 * y + e * y1);
            // below the eigenvalue the count nz - (sign changes of u) is J, above
            // it J + 1; w0 = -u_{nz-1}
            const bool below = ((neg(w0) ^ 1u) ^ static_cast<unsigned>(nz & 1)) == static_cast<unsigned>(J & 1);
            const double xo = x;
            if (below) a = xo;
            else b = xo;
            double corr;
            if (Row::kLaguerre) {
                const double w2 = u2 * z + u1 * z1 + u * z2 - (e2 * y + e1 * y1 + e * y2);  // half W''
                const double rinv = 1.0 / P.r, g = w1 / w0 * rinv, h = fma(g, g, -(2.0 * (w2 / w0) * rinv * rinv));
                corr = laguerre_step(g, h, (double)nz, below);
            } else {
                corr = w0 / w1 * P.r;
            }
            const double ad = fabs(corr);
            if (ad <= tol) {
                x = fmin(fmax(xo - corr, a), b);
                mode = 2;
            } else {
                const double xn = xo - corr;
                const bool ok = isfinite(xn) && xn > a && xn < b;
                x = ok ? xn : 0.5 * (a + b);
                const double ad2 = ad * ad, dp2 = dprev * dprev;
                if (!(b - a > tol)) mode = 2;
                // cubic (Newton: quadratic) convergence: the next correction would be
                // about ad^4 / dprev^3 (ad^3 / dprev^2)
                else if (ok && dprev > 0.0 && ad <= 0.25 * dprev &&
                         (Row::kLaguerre ? ad2 * ad2 <= tol * dp2 * dprev : ad2 * ad <= tol * dp2))
                    mode = 2;
                dprev = ok ? ad : 0.0;
            }
        } else if (mode == 0) {
            const int k = __popc(bm & ((1u << lane) - 1u));
            const int G = (nlB - 1 - k) / nB + 1;
            int gb = -1, cg = ca;
            for (int g = 0; g < G; ++g) {
                const int v = nN + k + g * nB, c = X.c[tb][v >> 5][v & 31];
                if (c <= J) {
                    gb = g;
                    cg = c;
                }
            }
            const double A0 = a, B0 = b;
            const int g1 = gb + 1, v1 = nN + k + g1 * nB;
            if (gb >= 0) {
                ca = cg;
                a = A0 + (B0 - A0) * ((double)(gb + 1) / (double)(G + 1));
            }
            if (g1 < G) {
                cb = X.c[tb][v1 >> 5][v1 & 31];
                b = A0 + (B0 - A0) * ((double)(gb + 2) / (double)(G + 1));
            }
            x = 0.5 * (a + b);
            if (!(b - a > tol) || (a == A0 && b == B0)) mode = 2;
            else if (ca == J && cb == J + 1) mode = 1;
        }
        const bool gave_up = (X.err[tb][0] | (W == 1 ? 0 : X.err[tb][1]) | (W == 4 ? X.err[tb][2] | X.err[tb][3] : 0)) != 0;
        pr.sync();  // the rings are free again
        if (gave_up) break;  // a ring wait ran out: abandon the item
    }
    return x;
}

// ---------------------------------------------------------------------------
// one item: mode values, norm and integrals
// ---------------------------------------------------------------------------
// state (u, e) before row i0 advanced to before row i1 (i1 >= i0) at shift x
template <class Row>
__device__ __forceinline__ void rows_up(const double* __restrict__ rows, int i0, int i1, double x, double& u,
                                        double& e) {
    for (int i = i0; i < i1; ++i) {
        e = fma(-Row::sigma(rows, i, x), u, e);
        u += e;
    }
}
// state after row i0 - 1 taken down to before row i1 (i1 <= i0)
template <class Row>
__device__ __forceinline__ void rows_down(const double* __restrict__ rows, int i0, int i1, double x, double& u,
                                          double& e) {
    for (int i = i0 - 1; i >= i1; --i) {
        u -= e;
        e = fma(Row::sigma(rows, i, x), u, e);
    }
}

// Grids so coarse that a mode can live between two coarse rows: beyond it a chain
// picks up the growing solution, by e^g eps of the mode after a decay of e^-g.
// The coarse twist leaves at most half of kCkRows for that; up to g = 10 it costs
// 2e-12 of the mode's top.  Above, the twist is checked: z solves the rows but for
// gamma at the twist, and |gamma| / |z| is about the eigenvalue's error over
// z_r / |z|.  From kTwist on (the twist a factor of some 1e4 below the top, on
// grids where modes live in a few rows any row at all) the mode is redone with the
// best of all rows (k_twist_modes).
constexpr double kTwist = 1e-9;
__device__ __forceinline__ bool twist_check(const ProblemInfo& pi) {
    const double c0 = __longlong_as_double((long long)pi.ceffmin_bits), c1 = __longlong_as_double((long long)pi.ceffmax_bits);
    const double g = 0.5 * kCkRows * (pi.omega * pi.dz);
    return g * g * (1.0 / (c0 * c0) - 1.0 / (c1 * c1)) > 100.0;
}

// v = m 2^E with |m| in [1, 2)
__device__ __forceinline__ void normalize(double& v, int& E) {
    const int e = biased_exp(v);
    if (e == 0) return;
    v *= pow2(1023 - e);
    E += e - 1023;
}

// the inverse of a transfer matrix (determinant 1) applied to (u, e)
__device__ __forceinline__ void adj_apply(const double (&p)[4], double& u, double& e) {
    const double a = fma(p[3], u, -(p[1] * e)), b = fma(p[0], e, -(p[2] * u));
    u = a;
    e = b;
}
__device__ __forceinline__ void adj_add(const double (&d)[4], double u, double e, double& du, double& de) {
    du += fma(d[3], u, -(d[1] * e));
    de += fma(d[0], e, -(d[2] * u));
}

// sums an item keeps: the norm (from d/dx where -d sigma / dx = 1) and the weights
template <class Row, int NW>
constexpr int kSums = (Row::kUnitNorm ? 1 : 0) + NW;

// What a warp of the mode-value pass carries beside its chain (part 0: all).  A
// team of four splits it: the norm to one warp and the weights to the other, or
// a weight each.
template <class Row, int NW, int kPart>
struct Part {
    static constexpr bool norm = Row::kUnitNorm && kPart != 2;
    static constexpr int lo = kPart == 2 && !Row::kUnitNorm ? 1 : 0;
    static constexpr int hi = kPart == 1 ? (Row::kUnitNorm ? 0 : 1) : NW;  // weights [lo, hi)
};

// a chain (u, e) with its derivatives d/dt and d/deps.  The common exponent
// follows u and e alone (so that it does not depend on the part): the
// derivatives are at most some 2^130 above, where the chain has decayed to its
// rounding while they have grown, and their products stay finite.
template <class Row, int NW, int kPart>
struct VecChain {
    using Q = Part<Row, NW, kPart>;
    double u, e, u1, e1, uw[NW], ew[NW];
    int E;  // common exponent
    __device__ __forceinline__ void start(double u0, double e0) {
        u = u0;
        e = e0;
        u1 = e1 = 0.0;
#pragma unroll
        for (int n = 0; n < NW; ++n) uw[n] = ew[n] = 0.0;
        E = 0;
    }
    __device__ __forceinline__ void rescale() {
        const int x = max(biased_exp(u), biased_exp(e)), sh = x - 1023;
        if (x != 0 && (sh > kVecBits || sh < -240)) {  // products of two stay finite
            const double sc = pow2(-sh);
            u *= sc;
            e *= sc;
            if (Q::norm) {
                u1 *= sc;
                e1 *= sc;
            }
#pragma unroll
            for (int n = Q::lo; n < Q::hi; ++n) {
                uw[n] *= sc;
                ew[n] *= sc;
            }
            E += sh;
        }
    }
    // sum number n of the rows passed so far (sgn = 1 upwards, -1 downwards)
    __device__ __forceinline__ double sum(int n, double rinv, double sgn) const {
        if (Row::kUnitNorm && n == 0) return sgn * ((u * e1 - e * u1) * rinv);
        const int k = n - (kSums<Row, NW> - NW);
        return sgn * (e * uw[k] - u * ew[k]);
    }
};

// matrices of two blocks at t: values, d/dt (Row::kUnitNorm) and the weights'
template <class Row, int NW, int kPart>
struct VecMats {
    using Q = Part<Row, NW, kPart>;
    double p[2][4], d[2][4], w[2][NW][4];
    __device__ __forceinline__ void eval(const double* const (&T)[2], const double* const (&W)[2],
                                         const double (&t)[2]) {
        const double2* q[2] = {reinterpret_cast<const double2*>(T[0]), reinterpret_cast<const double2*>(T[1])};
#pragma unroll
        for (int k = kPD; k >= 0; --k)
#pragma unroll
            for (int b = 0; b < 2; ++b) {
                const double2 v0 = q[b][2 * k], v1 = q[b][2 * k + 1];
                const double cf[4] = {v0.x, v0.y, v1.x, v1.y};
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    if (Q::norm && k < kPD) d[b][j] = k == kPD - 1 ? p[b][j] : fma(d[b][j], t[b], p[b][j]);
                    p[b][j] = k == kPD ? cf[j] : fma(p[b][j], t[b], cf[j]);
                }
                if (k <= kPW) {
#pragma unroll
                    for (int n = Q::lo; n < Q::hi; ++n) {
                        const double2* r = reinterpret_cast<const double2*>(W[b] + n * kWD);
                        const double2 w0 = r[2 * k], w1 = r[2 * k + 1];
                        const double wf[4] = {w0.x, w0.y, w1.x, w1.y};
#pragma unroll
                        for (int j = 0; j < 4; ++j) w[b][n][j] = k == kPW ? wf[j] : fma(w[b][n][j], t[b], wf[j]);
                    }
                }
            }
    }
    __device__ __forceinline__ void up(int b, VecChain<Row, NW, kPart>& C) const {
        const double(&m)[4] = p[b];
        if (Q::norm) {
            const double v = fma(m[0], C.u1, m[1] * C.e1) + fma(d[b][0], C.u, d[b][1] * C.e);
            C.e1 = fma(m[2], C.u1, m[3] * C.e1) + fma(d[b][2], C.u, d[b][3] * C.e);
            C.u1 = v;
        }
#pragma unroll
        for (int n = Q::lo; n < Q::hi; ++n) {
            const double(&g)[4] = w[b][n];
            const double v = fma(m[0], C.uw[n], m[1] * C.ew[n]) + fma(g[0], C.u, g[1] * C.e);
            C.ew[n] = fma(m[2], C.uw[n], m[3] * C.ew[n]) + fma(g[2], C.u, g[3] * C.e);
            C.uw[n] = v;
        }
        const double un = fma(m[0], C.u, m[1] * C.e);
        C.e = fma(m[2], C.u, m[3] * C.e);
        C.u = un;
    }
    __device__ __forceinline__ void down(int b, VecChain<Row, NW, kPart>& C) const {
        if (Q::norm) {
            adj_apply(p[b], C.u1, C.e1);
            adj_add(d[b], C.u, C.e, C.u1, C.e1);
        }
#pragma unroll
        for (int n = Q::lo; n < Q::hi; ++n) {
            adj_apply(p[b], C.uw[n], C.ew[n]);
            adj_add(w[b][n], C.u, C.e, C.uw[n], C.ew[n]);
        }
        adj_apply(p[b], C.u, C.e);
    }
};

// Half of the eigenvector work of an item by rows: the sums of squares as they
// are, five instructions a row (see vector_half for what is kept).
struct RowVals {
    double vs, vr;
    int Es, Er;
    unsigned loads;
};
template <class Row, int NW, bool kV, int kPart, bool kDown>
__device__ __noinline__ RowVals rows_vector(const ModesArgs& A, const ProblemInfo& pi, const Panel P, double mu,
                                            VecState* __restrict__ st, PRing R, double* __restrict__ ck,
                                            int* __restrict__ cke) {
    using Q = Part<Row, NW, kPart>;
    constexpr int kN = kSums<Row, NW>, NX = Q::hi - Q::lo;
    const int lane = threadIdx.x & 31, isrc = pi.isrc, ircv = pi.ircv, M = pi.M;
    // the weights of this part (one without an array: ones, not read)
    const double* const w[2] = {A.w + pi.w_off, NW > 1 && A.g ? A.g + pi.s_off : A.w + pi.w_off};
    const typename Row::At at(mu);
    double u = 1.0, um = kDown ? 0.0 : P.um0, sum[kN];
    int E = 0;
    RowVals out{0.0, 0.0, 0, 0, 0u};
#pragma unroll
    for (int n = 0; n < kN; ++n) sum[n] = 0.0;
    auto row = [&](const double* r, const double* x) {
        const double x2 = u * u;  // of z_i
        if (Q::norm) sum[0] += x2;
#pragma unroll
        for (int n = Q::lo; n < Q::hi; ++n) {
            double& s = sum[kN - NW + n];
            s = n == 1 && !Row::kUnitNorm ? s + x2 : fma(x[(n - Q::lo) * kWD], x2, s);
        }
        const double un = fma(at.turn(r), u, -um);
        um = u;
        u = un;
    };
    // of the state before row i
    auto keep = [&](int i) {
        if (i % kCkRows) return;
        const double v = kDown ? um : u, e = kDown ? um - u : u - um;
        const size_t c = (size_t)(i / kCkRows);
        double* o = ck + c * (2 + kN) * 32 + lane;
        if (kPart != 2) {
            o[0] = v;
            o[32 * (1 + kN)] = e;
            cke[c * 32 + lane] = E;
        }
        if (Q::norm) o[32] = sum[0];
#pragma unroll
        for (int n = Q::lo; n < Q::hi; ++n) o[32 * (1 + kN - NW + n)] = sum[kN - NW + n];
        if (kV && kPart != 2 && st) st[c * M] = VecState{v, e, E, 0};
    };
    auto value = [&](int i) {
        const double v = kDown ? um : u;
        if (i == isrc) out.vs = v, out.Es = E;
        if (i == ircv) out.vr = v, out.Er = E;
    };
    rows_sweep<Row, NX, kDown>(
        P, 0, P.nz, R, A.err, w + (NX > 0 ? Q::lo : 0), [&](const double* r, const double* x, int lo, int m) {
            if (!kDown) keep(lo);
            if (kPart != 2 && ((isrc >= lo && isrc < lo + m) || (ircv >= lo && ircv < lo + m))) {
                for (int k = 0; k < m; ++k) {
                    const int j = kDown ? m - 1 - k : k;
                    if (!kDown) value(lo + j);
                    row(r + j * Row::kW, x + j);
                    if (kDown) value(lo + j);
                }
            } else {
                run_rows<kDown>(m, [&](int j) { row(r + j * Row::kW, x + j); });
            }
            if (kDown) keep(lo);
            // a run grows by 2^368 at most; a chain that decays keeps its sums
            const int big = max(biased_exp(u), biased_exp(um)) - 1023;
            if (big > 100) {
                const double sc = pow2(-big);
                u *= sc;
                um *= sc;
#pragma unroll
                for (int n = 0; n < kN; ++n) sum[n] *= sc * sc;
                E += big;
            }
        });
    out.loads = R.loads;
    return out;
}

// Half of the eigenvector work of an item: the upward chain u (half 0) or the
// downward chain b (half 1); at every coarse row (multiples of kCkRows) its
// value, exponent and sums go to the checkpoints and, for full vectors (kV),
// its state to `st` (stride: modes).  vs, vr: its values at the source and
// receiver rows.
template <class Row, int NW, bool kV, int kPart>
__device__ __forceinline__ void vector_half(const ModesArgs& A, const ProblemInfo& pi, const Panel& P, double mu,
                                            int half, VecState* __restrict__ st, PRing& R, double* __restrict__ ck, int* __restrict__ cke,
                                            double& vs, int& Es, double& vr, int& Er) {
    using Q = Part<Row, NW, kPart>;
    constexpr int kN = kSums<Row, NW>;
    const int lane = threadIdx.x & 31;
    const int nz = P.nz, isrc = pi.isrc, ircv = pi.ircv;
    const bool check = twist_check(pi);
    const double rinv = 1.0 / P.r;
    const typename Row::Shift sh(P, mu);
    VecChain<Row, NW, kPart> C;
    if (half == 0) C.start(1.0, P.e0);
    else C.start(0.0, -1.0);
    vs = vr = 0.0;
    Es = Er = 0;
    auto keep = [&](int a, double sgn) {  // state before row a
        if (a % kCkRows) return;
        const size_t c = (size_t)(a / kCkRows);
        double* o = ck + c * (2 + kN) * 32 + lane;
        if (kPart != 2) {
            o[0] = C.u;
            if (check) o[32 * (1 + kN)] = C.e;
            cke[c * 32 + lane] = C.E;
        }
        if (Q::norm) o[32] = C.sum(0, rinv, sgn);
#pragma unroll
        for (int n = Q::lo; n < Q::hi; ++n) o[32 * (1 + kN - NW + n)] = C.sum(kN - NW + n, rinv, sgn);
        if (kV && kPart != 2 && st) st[c * pi.M] = VecState{C.u, C.e, C.E, 0};
    };
    // the chain at row i of the block [a, end): from below (u) or above (b)
    auto value = [&](int i, int a, int end, double& v, int& E) {
        if (kPart == 2 || i < a || i >= end) return;
        double f = C.e;
        v = C.u;
        E = C.E;
        if (half == 0) rows_up<Row>(P.rows, a, i, mu, v, f);
        else rows_down<Row>(P.rows, end, i, mu, v, f);
    };
    const int nch = (P.nblk + kPanelChunk - 1) / kPanelChunk;
    const double* src = A.T + (size_t)P.rec * kRecT;
    const double* sw[2] = {A.W0 + (size_t)P.rec * kRecW, NW > 1 ? A.W1 + (size_t)P.rec * kRecW : nullptr};
    ring_stream(
        R, nch, A.err,
        [&](double* dst, uint64_t* bar, int o) {
            const size_t c = half ? nch - 1 - o : o;
            mbar_expect_tx(bar, (kTD + (Q::hi - Q::lo) * kWD) * 8);
            tma_load_1d(dst, src + c * kTD, kTD * 8, bar);
#pragma unroll
            for (int n = Q::lo; n < Q::hi; ++n) tma_load_1d(dst + kTD + n * kWD, sw[n] + c * kWD, kWD * 8, bar);
        },
        [&](const double* buf, int o) {
            const int c = half ? nch - 1 - o : o, nb = min(kPanelChunk, P.nblk - c * kPanelChunk);
            for (int q0 = 0; q0 < kPanelChunk; q0 += 2) {
                const int qa = half ? kPanelChunk - 1 - q0 : q0, qb = half ? qa - 1 : qa + 1;
                if (min(qa, qb) >= nb) continue;
                VecMats<Row, NW, kPart> M;
                const double* const Ts[2] = {buf + qa * kRecT, buf + qb * kRecT};
                const double* const Ws[2] = {buf + kTD + qa * kRecW, buf + kTD + qb * kRecW};
                const double t[2] = {sh.at(Ts[0]), sh.at(Ts[1])};
                M.eval(Ts, Ws, t);
#pragma unroll
                for (int b = 0; b < 2; ++b) {
                    const int q = b ? qb : qa;
                    if (q >= nb) continue;
                    const int a = (c * kPanelChunk + q) * P.blk, end = min(nz, a + P.blk);
                    if (half == 0) keep(a, 1.0);
                    value(isrc, a, end, vs, Es);
                    value(ircv, a, end, vr, Er);
                    if (half == 0) {
                        M.up(b, C);
                    } else {
                        M.down(b, C);
                        keep(a, -1.0);
                    }
                }
            }
            C.rescale();
        });
}

// |u b| at a coarse row as m 2^E, m in [1, 2) (m = 0: none yet)
struct TwistKey {
    double m;
    int E, c;
    __device__ __forceinline__ void take(double u, int Eu, double b, int Eb, int at) {
        double v = fabs(u * b);
        int e = Eu + Eb;
        normalize(v, e);
        if (v > 0.0 && (m == 0.0 || e > E || (e == E && v > m))) {
            m = v;
            E = e;
            c = at;
        }
    }
};

// the chains and their sums at the row where they are joined: rows below r in
// su (at u's exponent), rows from r on in sb
template <int kN>
struct TwistAt {
    double u, b, su[kN], sb[kN];
    int Eu, Eb, r;
};

// where a mode's chains end at the source and receiver rows, from below and above
struct ModeEnds {
    double us, ur, bs, br;
    int Eus, Eur, Ebs, Ebr;
};

// the values of mode i from its chains; returns sum z^2 / z_r^2
template <class Row, int NW, bool kV>
__device__ __forceinline__ double finish_mode(const ModesArgs& A, const ProblemInfo& pi, int i, bool write, double mu,
                                              const TwistAt<kSums<Row, NW>>& tw, const ModeEnds& v) {
    constexpr int kN = kSums<Row, NW>;
    double ut = tw.u, bt = tw.b;
    int Eut = tw.Eu, Ebt = tw.Eb;
    normalize(ut, Eut);
    normalize(bt, Ebt);
    const int eut = Eut - tw.Eu, ebt = Ebt - tw.Eb;  // exponents of u and b themselves
    const double iu2 = 1.0 / (ut * ut), ib2 = 1.0 / (bt * bt);
    auto total = [&](int n) {  // sum over all rows in units of z_r^2
        double x = tw.su[n], y = tw.sb[n];
        int ex = 0, ey = 0;
        normalize(x, ex);
        normalize(y, ey);
        // both sums were taken at the exponents of u and b at the twist
        return x * iu2 * pow2(ex - 2 * eut) + y * ib2 * pow2(ey - 2 * ebt);
    };
    const int r = tw.r, isrc = pi.isrc, ircv = pi.ircv;
    const int n1 = Row::kUnitNorm ? 0 : kN - 1, nw = kN - NW;
    const double nrm = total(n1);
    const double f2 = Row::kUnitNorm ? 1.0 : 1.0 / (1.0 + (mu / pi.dz) * (mu / pi.dz));
    const double scale = Row::kUnitNorm ? 1.0 / sqrt(nrm * pi.dz) : sqrt(f2 / (nrm * pi.dz));
    const double zs = (isrc <= r) ? (v.us / ut) * pow2(v.Eus - Eut) : (v.bs / bt) * pow2(v.Ebs - Ebt);
    const double zr = (ircv <= r) ? (v.ur / ut) * pow2(v.Eur - Eut) : (v.br / bt) * pow2(v.Ebr - Ebt);
    const double absorption = total(nw) / nrm * f2;
    const double ks = Row::kUnitNorm ? sqrt(mu / (pi.dz * pi.dz)) : mu / pi.dz;
    const auto kp = csqrt_principal(ks * ks, absorption);
    if (write) {
        A.kr[i] = kp.real();
        A.ki[i] = kp.imag();
        A.vs[i] = zs * scale;
        A.vr[i] = zr * scale;
        if (kV) A.vtwist[i] = VecTwist{mu, scale / ut, scale / bt, Eut, Ebt, r, 0};
        if (Row::kUnitNorm && NW > 1) {
            const double vph = pi.omega / kp.real();
            A.vg[i] = 1.0 / (vph * (total(nw + 1) / nrm));
        } else if (A.vg) {
            A.vg[i] = 0.0;
        }
    }
    return nrm;
}

template <class Row, int NW, bool kV, int W, bool kRows>
__device__ __forceinline__ void panel_vector(const ModesArgs& A, const ProblemInfo& pi, const Panel& P,
                                             const WorkItem& w, int it, double mu, PRing& R, Team<W>& pr,
                                             bool split, double* __restrict__ ck, int* __restrict__ cke) {
    constexpr int kN = kSums<Row, NW>;
    const int lane = threadIdx.x & 31, half = pr.half & 1;
    const int nc = (P.nz + kCkRows - 1) / kCkRows;
    double* cks[2] = {ck, ck + A.ck_stride * (2 + kN)};
    int* ckes[2] = {cke, cke + A.ck_stride};
    double vs, vr;
    int Es, Er;
    RowVals above{};  // W == 1
    VecState* st = nullptr;
    if (kV && lane < w.m) st = A.vstate + A.vstate_off[w.problem] + w.j0 + lane;
    if (kV && st) st += (long long)half * nc * pi.M;
    // a team alone on its SM splits the sums (1185 modes: 403 -> 294 us);
    // two of them fill it, and the transfer matrices evaluated twice cost more
    // than the idle warps (36 azimuths of 0.5 Hz: both stages 286 us, split 300)
    double* c = cks[half];
    int* ce = ckes[half];
    if constexpr (kRows) {
        RowVals o{};
        if (W == 1) {
            o = rows_vector<Row, NW, kV, 0, false>(A, pi, P, mu, st, R, cks[0], ckes[0]);
            R.loads = o.loads;
            VecState* sd = st ? st + (long long)nc * pi.M : st;
            above = rows_vector<Row, NW, kV, 0, true>(A, pi, P, mu, sd, R, cks[1], ckes[1]);
            R.loads = above.loads;
        } else if (W == 4 && split && pr.half >= 2) {
            o = half ? rows_vector<Row, NW, kV, 2, true>(A, pi, P, mu, st, R, c, ce)
                     : rows_vector<Row, NW, kV, 2, false>(A, pi, P, mu, st, R, c, ce);
            R.loads = o.loads;
        } else if (W == 4 && split) {
            o = half ? rows_vector<Row, NW, kV, 1, true>(A, pi, P, mu, st, R, c, ce)
                     : rows_vector<Row, NW, kV, 1, false>(A, pi, P, mu, st, R, c, ce);
            R.loads = o.loads;
        } else if (pr.half < 2) {
            o = half ? rows_vector<Row, NW, kV, 0, true>(A, pi, P, mu, st, R, c, ce)
                     : rows_vector<Row, NW, kV, 0, false>(A, pi, P, mu, st, R, c, ce);
            R.loads = o.loads;
        }
        vs = o.vs;
        vr = o.vr;
        Es = o.Es;
        Er = o.Er;
    } else if (W == 4 && split) {
        if (pr.half < 2) vector_half<Row, NW, kV, 1>(A, pi, P, mu, half, st, R, c, ce, vs, Es, vr, Er);
        else vector_half<Row, NW, kV, 2>(A, pi, P, mu, half, st, R, c, ce, vs, Es, vr, Er);
    } else if (pr.half < 2) {
        vector_half<Row, NW, kV, 0>(A, pi, P, mu, half, st, R, c, ce, vs, Es, vr, Er);
    }
    PairBox& X = *pr.box;
    const int tb = pr.turn, t2 = tb ^ 1;
    if (pr.half == 1) {
        X.v[tb][1][0][lane] = vs;
        X.v[tb][1][1][lane] = vr;
        X.v[tb][1][2][lane] = __hiloint2double(Es, Er);
    }
    pr.sync();  // checkpoints of both halves (and the box) visible to both
    if (pr.half >= 2) return;
    // the twist: the coarse row with the largest |u b|, the lowest of equal ones;
    // each half looks through half of the rows
    TwistKey K{0.0, 0, 0};
    const int c0 = half ? nc / 2 : 0, c1 = half || W == 1 ? nc : nc / 2;
#pragma unroll 4
    for (int c = c0; c < c1; ++c) {
        const size_t o = (size_t)c * (2 + kN) * 32 + lane, i = (size_t)c * 32 + lane;
        K.take(__ldcg(cks[0] + o), __ldcg(ckes[0] + i), __ldcg(cks[1] + o), __ldcg(ckes[1] + i), c);
    }
    if (half) {
        X.v[t2][1][0][lane] = K.m;
        X.v[t2][1][1][lane] = __hiloint2double(K.E, K.c);
    }
    pr.sync2();
    if (half) return;
    if (W != 1) {
        const double m = X.v[t2][1][0][lane], ec = X.v[t2][1][1][lane];
        const int E = __double2hiint(ec);
        if (m > 0.0 && (K.m == 0.0 || E > K.E || (E == K.E && m > K.m))) K.c = __double2loint(ec);
    }
    ModeEnds ends;
    ends.us = vs;
    ends.ur = vr;
    ends.Eus = Es;
    ends.Eur = Er;
    ends.bs = W == 1 ? above.vs : X.v[tb][1][0][lane];
    ends.br = W == 1 ? above.vr : X.v[tb][1][1][lane];
    const double eb = W == 1 ? __hiloint2double(above.Es, above.Er) : X.v[tb][1][2][lane];
    ends.Ebs = __double2hiint(eb);
    ends.Ebr = __double2loint(eb);
    TwistAt<kN> tw;
    tw.r = K.c * kCkRows;
    const size_t o = (size_t)K.c * (2 + kN) * 32 + lane;
    tw.u = __ldcg(cks[0] + o);
    tw.b = __ldcg(cks[1] + o);
    tw.Eu = __ldcg(ckes[0] + (size_t)K.c * 32 + lane);
    tw.Eb = __ldcg(ckes[1] + (size_t)K.c * 32 + lane);
#pragma unroll
    for (int n = 0; n < kN; ++n) {
        tw.su[n] = __ldcg(cks[0] + o + 32 * (1 + n));
        tw.sb[n] = __ldcg(cks[1] + o + 32 * (1 + n));
    }
    const double nrm = finish_mode<Row, NW, kV>(A, pi, pi.off + w.j0 + lane, lane < w.m, mu, tw, ends);
    if (A.redo && twist_check(pi)) {
        const double g = __ldcg(cks[1] + o + 32 * (1 + kN)) / tw.b - __ldcg(cks[0] + o + 32 * (1 + kN)) / tw.u;
        const unsigned bad = __ballot_sync(0xffffffffu, lane < w.m && !(g * g <= kTwist * kTwist * nrm));
        if (bad && lane == 0) A.redo[atomicAdd(A.n_redo, 1)] = make_int2(it, (int)bad);
    }
}

// ---------------------------------------------------------------------------
// eigenvalues and mode values of every item.  kDo: 1 eigenvalues to mu, 2 mode
// values of the eigenvalues in mu, 3 both.  The pairs take items from the
// cost-ordered list as they get free (sched: two zeroed counters), or round-robin.
// ---------------------------------------------------------------------------
// doubles of a ring slot: eigenvalues alone need no weights
template <int NW, int kDo>
constexpr int kModesSl = kTD + (kDo == 1 ? 0 : NW) * kWD;

template <class Row, int NW, int kDo, bool kV, int W>
__global__ void __launch_bounds__(kPWarps * 32, kPanelCtas) k_panel_modes(const __grid_constant__ ModesArgs A) {
    extern __shared__ __align__(128) unsigned char smem_raw[];
    constexpr int kSl = kModesSl<NW, kDo>;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int n_items = *A.n_items_dev;
    if (n_items < A.min_items || n_items > A.max_items) return;  // another launch's
    PRing R = make_ring(smem_raw, wid, kSl);
    constexpr int kTeams = kPWarps / W;
    Team<W> pr;
    pr.id = wid / W;
    pr.half = wid % W;
    pr.box = reinterpret_cast<PairBox*>(smem_raw + kRingBytes<kSl>) + pr.id;
    pr.stride = kPBuf * kSl;
    pr.area = reinterpret_cast<double*>(smem_raw) + (size_t)pr.id * W * pr.stride;
    pr.turn = 0;
    const long long gp = (long long)blockIdx.x * kTeams + pr.id;
    double* ck = A.ck_u + gp * 2 * A.ck_stride * (2 + kSums<Row, NW>);
    int* cke = A.ck_e + gp * 2 * A.ck_stride;
    // first items: one to the first team of as many CTAs as there are SMs (which
    // start on different ones), then to their second teams, then to the next
    // CTAs, so that few items have a scheduler for each warp; later ones as the
    // teams get free (sched), or round-robin
    const int n_pairs = gridDim.x * kTeams, row = blockIdx.x / A.num_sms;
    const int width = min(A.num_sms, (int)gridDim.x - row * A.num_sms);  // CTAs of this row
    long long walk = (long long)row * A.num_sms * kTeams + pr.id * width + blockIdx.x % A.num_sms;
    bool first = true;
    for (int turn = 0;; turn ^= 1) {
        if (pr.half == 0 && lane == 0) {
            long long it = walk;
            if (A.sched && !first) it = n_pairs + atomicAdd(A.sched, 1);
            pr.box->item[turn] = it < n_items ? (int)it : -1;
        }
        walk += n_pairs;
        first = false;
        pr.sync();
        const int it = pr.box->item[turn];
        if (it < 0) break;
        const WorkItem w = A.items[it];
        if (w.pad < 0) continue;  // k_rows_modes'
        const ProblemInfo& pi = A.pinfo[w.problem];
        const Panel P = panel_of<Row>(pi, A.desc[w.pad], A.rows);
        double x = P.xc;
        if (kDo & 1) {
            x = panel_bisect<Row, W, false>(pi, P, w, A.T, A.counts, A.tol, A.err, A.steps, R, pr);
            if (pr.half == 0 && lane < w.m) A.mu[pi.off + w.j0 + lane] = x;
        } else if (lane < w.m) {
            x = A.mu[pi.off + w.j0 + lane];
        }
        if (kDo & 2) panel_vector<Row, NW, kV, W, false>(A, pi, P, w, it, x, R, pr, n_items <= A.num_sms, ck, cke);
    }
}

// The items by rows (what: 1 eigenvalues, 2 mode values, 3 both), on a stream
// beside k_panel_modes, whose code stays smaller without them (2 Hz, 20000 rows:
// 541 us, with the rows' sweeps in the same kernel 578).  Teams of four while the
// items are few: a sweep is a chain over half of the rows.  A warp to an item
// from kSoloMin an SM on, both directions in turn and no exchange: bound by FP64
// issue and, on grids of some hundred rows, by the latency of a sweep's first
// rows, which more items in flight hide (12 on an SM, 3 teams of four; 90
// azimuths of 1 Hz, 2500 rows 1040 -> 730 us).  The values are the same.
template <class Row, int NW, bool kV, int W, int kDo>
__global__ void __launch_bounds__(kPWarps * 32, W == 1 ? kRowsCtas : kPanelCtas)
    k_rows_modes(const __grid_constant__ ModesArgs A) {
    extern __shared__ __align__(128) unsigned char smem_raw[];
    constexpr int kSl = kTD + NW * kWD, kTeams = kPWarps / W;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int n_items = A.n_items_dev[0], n_rows = A.n_items_dev[3];
    if (n_rows == 0 || (n_rows > kSoloMin * A.num_sms) != (W == 1)) return;  // none, or the other launch's
    PRing R = make_ring(smem_raw, wid, kSl);
    Team<W> pr;
    pr.id = wid / W;
    pr.half = wid % W;
    pr.box = reinterpret_cast<PairBox*>(smem_raw + kRingBytes<kSl>) + pr.id;
    pr.stride = kPBuf * kSl;
    pr.area = reinterpret_cast<double*>(smem_raw) + (size_t)pr.id * W * pr.stride;
    pr.turn = 0;
    const long long slot = (long long)blockIdx.x * kTeams + pr.id;
    double* ck = A.ck_u + slot * 2 * A.ck_stride * (2 + kSums<Row, NW>);
    int* cke = A.ck_e + slot * 2 * A.ck_stride;
    const int n_teams = gridDim.x * kTeams;
    int next = pr.id * gridDim.x + blockIdx.x;  // first items on different SMs
    for (int turn = 0;; turn ^= 1) {
        if (pr.half == 0 && lane == 0) {
            while (next < n_items && A.items[next].pad >= 0)  // k_panel_modes'
                next = A.sched ? n_teams + atomicAdd(A.sched, 1) : next + n_teams;
            pr.box->item[turn] = next < n_items ? next : -1;
            next = A.sched ? n_teams + atomicAdd(A.sched, 1) : next + n_teams;
        }
        pr.sync();
        const int it = pr.box->item[turn];
        if (it < 0) break;
        const WorkItem w = A.items[it];
        const ProblemInfo& pi = A.pinfo[w.problem];
        PanelDesc d{};
        d.xc = Row::lo(pi);
        const Panel P = panel_of<Row>(pi, d, A.rows);
        double x = P.xc;
        if (kDo & 1) {
            x = panel_bisect<Row, W, true>(pi, P, w, A.T, A.counts, A.tol, A.err, A.steps, R, pr);
            if (pr.half == 0 && lane < w.m) A.mu[pi.off + w.j0 + lane] = x;
        } else if (lane < w.m) {
            x = A.mu[pi.off + w.j0 + lane];
        }
        if (kDo & 2) panel_vector<Row, NW, kV, W, true>(A, pi, P, w, it, x, R, pr, false, ck, cke);
    }
}

// a chain's state normalised: the larger of |u|, |e| in [1, 2)
struct RowState {
    double u, e;
    int E;
    __device__ __forceinline__ void normal() {
        const int x = max(biased_exp(u), biased_exp(e));
        if (x == 0 || x == 1023) return;
        const double sc = pow2(1023 - x);
        u *= sc;
        e *= sc;
        E += x - 1023;
    }
};

// The modes whose coarse twist was not good enough (redo: item and lanes), a CTA
// to an item: both chains by rows, on a warp each, then |u b| row by row, 32 rows
// of b in shared memory at a time, and the values from the row where it is
// largest.  Rows of the two chunks at the coarse twist while gamma is below 1e-7
// of |z|; from there on the decay to the coarse rows may be past the chains'
// rounding, where |u b| is level and its largest value tells nothing, and the
// four warps go through all chunks.  A serial chain over the rows, some 30 cycles
// each: 100 us for 2500 rows.
template <class Row, int NW, bool kV>
__global__ void __launch_bounds__(kPWarps * 32) k_twist_modes(const __grid_constant__ ModesArgs A) {
    extern __shared__ __align__(128) unsigned char smem_raw[];
    constexpr int kSl = kTD + NW * kWD, kN = kSums<Row, NW>, kSeg = 32, kSegs = kCkRows / kSeg;
    static_assert(kSeg * 32 <= kPBuf * kSl, "a segment fits the ring");
    __shared__ RowVals box[32];
    __shared__ TwistKey keys[kPWarps][32];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int n = *A.n_redo;
    if (blockIdx.x >= n) return;
    PRing R = make_ring(smem_raw, wid, kSl);
    double* cks[2];
    int* ckes[2];
    for (int h = 0; h < 2; ++h) {
        cks[h] = A.ck_u + (2ll * blockIdx.x + h) * A.ck_stride * (2 + kN);
        ckes[h] = A.ck_e + (2ll * blockIdx.x + h) * A.ck_stride;
    }
    for (int k = blockIdx.x; k < n; k += gridDim.x) {
        const int2 job = A.redo[k];
        const WorkItem w = A.items[job.x];
        const ProblemInfo& pi = A.pinfo[w.problem];
        PanelDesc d{};
        d.xc = Row::lo(pi);
        const Panel P = panel_of<Row>(pi, d, A.rows);
        const int nz = P.nz, nc = (nz + kCkRows - 1) / kCkRows, i = pi.off + w.j0 + lane;
        const bool mine = ((unsigned)job.y >> lane) & 1u;
        const double mu = lane < w.m ? A.mu[i] : P.xc;
        VecState* st = nullptr;
        if (kV && mine) st = A.vstate + A.vstate_off[w.problem] + w.j0 + lane + (long long)(wid & 1) * nc * pi.M;
        RowVals below{};
        if (wid == 0) {
            below = rows_vector<Row, NW, kV, 0, false>(A, pi, P, mu, st, R, cks[0], ckes[0]);
            R.loads = below.loads;
        } else if (wid == 1) {
            box[lane] = rows_vector<Row, NW, kV, 0, true>(A, pi, P, mu, st, R, cks[1], ckes[1]);
            R.loads = box[lane].loads;
        }
        __syncthreads();
        auto at = [&](int h, int c) { return cks[h] + (size_t)c * (2 + kN) * 32 + lane; };
        auto state = [&](int h, int c) {
            const double* o = at(h, c);
            return RowState{o[0], o[32 * (1 + kN)], ckes[h][(size_t)c * 32 + lane]};
        };
        auto up = [&](RowState& S, int row) {
            S.e = fma(-Row::sigma(P.rows, row, mu), S.u, S.e);
            S.u += S.e;
        };
        auto down = [&](RowState& S, int row) {
            S.u -= S.e;
            S.e = fma(Row::sigma(P.rows, row, mu), S.u, S.e);
        };
        TwistKey K{0.0, 0, 0};
        for (int c = 0; c < nc; ++c) {
            const RowState U = state(0, c), S = state(1, c);
            K.take(U.u, U.E, S.u, S.E, c);
        }
        const int c0 = K.c;
        bool all;
        {
            const RowState U = state(0, c0), S = state(1, c0);
            const int q = Row::kUnitNorm ? 1 : kN;  // the norm
            const double g = S.e / S.u - U.e / U.u;
            const double nrm = at(0, c0)[32 * q] / (U.u * U.u) + at(1, c0)[32 * q] / (S.u * S.u);
            all = __any_sync(0xffffffffu, mine && !(g * g <= 1e-14 * nrm));
        }
        double* buf = R.buf + lane;
        K = TwistKey{0.0, 0, 0};
        for (int q = wid; q < (all ? nc : 2); q += kPWarps) {
            const int c = all ? q : max(c0 - 1, 0) + min(q, c0);
            const int a = c * kCkRows, end = min(nz, a + kCkRows);
            RowState S = c + 1 < nc ? state(1, c + 1) : RowState{0.0, -1.0, 0}, behind[kSegs];
            S.normal();
#pragma unroll
            for (int s = kSegs - 1; s >= 0; --s) {  // b behind each segment
                behind[s] = S;
#pragma unroll 8
                for (int row = min(end, a + (s + 1) * kSeg) - 1; row >= a + s * kSeg; --row) down(S, row);
                S.normal();
            }
            RowState U = state(0, c);
            U.normal();
#pragma unroll
            for (int s = 0; s < kSegs; ++s) {
                const int lo = a + s * kSeg, hi = min(end, lo + kSeg);
                S = behind[s];
#pragma unroll 8
                for (int row = hi - 1; row >= lo; --row) {
                    down(S, row);
                    buf[(row - lo) * 32] = S.u;
                }
#pragma unroll 4
                for (int row = lo; row < hi; ++row) {
                    K.take(U.u, U.E, buf[(row - lo) * 32], behind[s].E, row);
                    up(U, row);
                }
                U.normal();
            }
        }
        keys[wid][lane] = K;
        __syncthreads();
        if (wid == 0) {
            for (int q = 1; q < kPWarps; ++q) {
                const TwistKey& o = keys[q][lane];
                if (o.m > 0.0 && (K.m == 0.0 || o.E > K.E || (o.E == K.E && (o.m > K.m || (o.m == K.m && o.c < K.c)))))
                    K = o;
            }
        }
        const RowVals above = box[lane];
        __syncthreads();  // the box and the keys are free
        if (wid == 0 && mine && K.m > 0.0) {
            TwistAt<kN> tw;
            const int c = K.c / kCkRows, a = c * kCkRows, end = min(nz, a + kCkRows);
            const double* wp = A.w + pi.w_off;
            const double* gp = NW > 1 && A.g ? A.g + pi.s_off : nullptr;
            auto add = [&](double (&x)[kN], RowState& S, int row) {
                const double z2 = S.u * S.u;
                if (Row::kUnitNorm) x[0] += z2;
                x[kN - NW] = fma(wp[row], z2, x[kN - NW]);
                if (NW > 1) x[kN - 1] = fma(gp ? gp[row] : 1.0, z2, x[kN - 1]);
            };
            auto fold = [&](double (&x)[kN], RowState& S, int row) {  // the squares stay finite
                const int big = max(biased_exp(S.u), biased_exp(S.e)) - 1023;
                if ((row & 7) || big <= 100) return;
                const double sc = pow2(-big);
                S.u *= sc;
                S.e *= sc;
                S.E += big;
                for (int q = 0; q < kN; ++q) x[q] *= sc * sc;
            };
            tw.r = K.c;
            RowState S{0.0, -1.0, 0};
            if (c + 1 < nc) S = state(1, c + 1);
#pragma unroll
            for (int q = 0; q < kN; ++q) {
                tw.su[q] = cks[0][((size_t)c * (2 + kN) + 1 + q) * 32 + lane];
                tw.sb[q] = c + 1 < nc ? cks[1][((size_t)(c + 1) * (2 + kN) + 1 + q) * 32 + lane] : 0.0;
            }
            for (int row = end - 1; row >= tw.r; --row) {
                down(S, row);
                add(tw.sb, S, row);
                if (row > tw.r) fold(tw.sb, S, row);
            }
            tw.b = S.u;
            tw.Eb = S.E;
            S = state(0, c);
            for (int row = a; row < tw.r; ++row) {
                add(tw.su, S, row);
                up(S, row);
                fold(tw.su, S, row);
            }
            tw.u = S.u;
            tw.Eu = S.E;
            const ModeEnds ends{below.vs, below.vr, above.vs, above.vr, below.Es, below.Er, above.Es, above.Er};
            finish_mode<Row, NW, kV>(A, pi, i, true, mu, tw, ends);
        }
        __syncthreads();  // and the checkpoints
    }
}

// ---------------------------------------------------------------------------
// full vectors: every mode at every row, from the states that the mode-value
// pass left at the coarse rows: a warp takes 32 modes x kCkRows rows, up from
// the lower state below the twist and down from the upper one above it (the
// growing direction of either chain).  A first launch finds each mode's largest
// |value|, where modes are positive; computing the values twice (2 FMAs each)
// is cheaper than reading and turning them.  Bound by the writes (8 B a value),
// which run along the modes as the rows are stored; a block of 128 rows is a
// serial chain of about 2 us, with thousands of them in flight.
// 0.3 Hz, 20000 rows: 31 us for both launches after 130 us of states (one kernel
// before,
// whose warps walked 32 modes up and down all rows, 3.8 ms)
// ---------------------------------------------------------------------------
template <class Row, bool kPeak>
__global__ void __launch_bounds__(256) k_panel_fill(int p0, ModesArgs A) {
    const int p = p0 + blockIdx.z;
    const ProblemInfo& pi = A.pinfo[p];
    const int M = pi.M, nz = pi.nz, nc = (nz + kCkRows - 1) / kCkRows;
    const int c = blockIdx.y * 8 + (threadIdx.x >> 5), j = blockIdx.x * 32 + (threadIdx.x & 31);
    if (c >= nc || j >= M) return;
    const double* rows = A.rows + (size_t)pi.s_off * Row::kW;
    const VecTwist t = A.vtwist[pi.off + j];
    const VecState* st = A.vstate + A.vstate_off[p] + j;
    unsigned long long* key = A.vpeak + pi.off + j;
    const int a = c * kCkRows, end = min(nz, a + kCkRows);
    double* out = A.vfull + A.vfull_off[p] + j;
    double sg = 1.0, top = 0.0;  // top: the value of largest magnitude
    if (!kPeak) {
        sg = (*key & 1ull) ? -1.0 : 1.0;
        if (c == 0 && sg < 0.0) {
            A.vs[pi.off + j] = -A.vs[pi.off + j];
            A.vr[pi.off + j] = -A.vr[pi.off + j];
        }
    }
    auto put = [&](int i, double u) {
        if (kPeak) top = fabs(u) > fabs(top) ? u : top;
        else out[(long long)i * M] = u;
    };
    const int mid = min(max(t.r, a), end);  // rows from the twist on come from above
    if (a < mid) {
        const VecState v = st[(long long)c * M];
        const double f = sg * t.fu * pow2(v.E - t.Eu);
        double u = v.u * f, e = v.e * f;
#pragma unroll 16
        for (int i = a; i < mid; ++i) {
            put(i, u);
            e = fma(-Row::sigma(rows, i, t.mu), u, e);
            u += e;
        }
    }
    if (mid < end) {
        VecState v{0.0, -1.0, 0, 0};
        if (c + 1 < nc) v = st[(long long)(nc + c + 1) * M];
        const double f = sg * t.fb * pow2(v.E - t.Eb);
        double u = v.u * f, e = v.e * f;
#pragma unroll 16
        for (int i = end - 1; i >= mid; --i) {
            u -= e;
            e = fma(Row::sigma(rows, i, t.mu), u, e);
            put(i, u);
        }
    }
    if (kPeak) {  // magnitude, with the sign in the last bit
        const unsigned long long b = (unsigned long long)__double_as_longlong(fabs(top));
        atomicMax(key, (b & ~1ull) | (top < 0.0 ? 1ull : 0ull));
    }
}

// checkpoint slots of k_panel_modes: two directions of two pairs a CTA
int panel_slots(int grid) { return 2 * (kPWarps / 2) * grid; }

template <class Row, int NW, int kDo, bool kV, int W>
void modes_run(cudaStream_t st, int grid, const ModesArgs& a) {
    constexpr int kSl = kModesSl<NW, kDo>;
    static_assert(kSl * kPBuf >= 18 * 32 && kSl * kPBuf >= 2 * 5 * 64, "a warp's segments fit its ring");
    const size_t sm = kRingBytes<kSl> + (kPWarps / 2) * sizeof(PairBox);
    auto* f = k_panel_modes<Row, NW, kDo, kV, W>;
    cudaFuncSetAttribute((const void*)f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    f<<<grid, kPWarps * 32, sm, st>>>(a);
}

template <class Row, int NW, bool kV, int W, int kDo>
void rows_run(cudaStream_t st, int ctas, const ModesArgs& a) {
    constexpr int kSl = kTD + NW * kWD;
    static_assert(kSl * kPBuf >= 4 * 7 * 32, "a warp's chains fit its ring");
    const size_t sm = kRingBytes<kSl> + (kPWarps / W) * sizeof(PairBox);
    auto* f = k_rows_modes<Row, NW, kV, W, kDo>;
    cudaFuncSetAttribute((const void*)f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    f<<<ctas, kPWarps * 32, sm, st>>>(a);
}
template <class Row, int NW, bool kV>
int rows_run(cudaStream_t st, int grid, const ModesArgs& a, int what) {
    ModesArgs r = a;
    const long long used = panel_slots(grid);  // behind k_panel_modes' checkpoints
    r.ck_u += used * kCkVals * a.ck_stride;
    r.ck_e += used * a.ck_stride;
    if (r.sched) r.sched += 2;
    const int teams = std::min(grid, a.item_cap);
    if (what == 3) rows_run<Row, NW, kV, 4, 3>(st, teams, r);
    if (what == 1) rows_run<Row, 1, false, 4, 1>(st, teams, r);
    if (what == 2) rows_run<Row, NW, kV, 4, 2>(st, teams, r);
    int n = 1;
    if (a.item_cap > kSoloMin * a.num_sms) {
        const int ctas = std::min(grid / kPanelCtas * kRowsCtas, (a.item_cap + kPWarps - 1) / kPWarps);
        if (what & 1) rows_run<Row, 1, false, 1, 1>(st, ctas, r), ++n;
        if (what == 3 && r.sched) ++r.sched;
        if (what & 2) rows_run<Row, NW, kV, 1, 2>(st, ctas, r), ++n;
    }
    return n;
}

template <class Row, int NW, int kDo, int W>
void modes_run(cudaStream_t st, int grid, const ModesArgs& a) {
    if (kDo != 1 && a.vstate) modes_run<Row, NW, kDo, kDo != 1, W>(st, grid, a);
    else modes_run<Row, NW, kDo, false, W>(st, grid, a);
}

// How many warps an item gets, by the number of items (known on the device: a
// launch that it does not ask for returns at once; those beyond item_cap are
// left out).  The arithmetic is the same.
//  up to two an SM     teams of four, both stages in one launch: an item alone on
//                      its SM has a scheduler for each warp (0.1 Hz: 77 + 86
//                      us as pairs 129 + 107; 32 requests 289 + 205 as pairs 543
//                      + 207)
//  up to 4 x the pairs teams of four for the eigenvalues, pairs for the mode
//  that fit            values: items are finished sooner, so fewer idle at the
//                      end (256 frequencies, 1.3 x: 553 us, as pairs 603; 64
//                      wide-angle ones 408, as pairs 659)
//  more                pairs: 6 % less work than in the transfer matrices of the
//                      inner segments twice over (45-azimuth sweep 1906 us, as
//                      teams 1962)
// The stages apart where SMs are full: in one kernel their code shares the
// instruction cache (256 frequencies: 1118 us in one launch of pairs, 950 in two).
template <class Row, int NW>
int modes_launch(cudaStream_t st, int grid, const ModesArgs& a, int what) {
    ModesArgs few = a, some = a, many = a, rest = a;
    few.min_items = 0;
    few.max_items = std::min(grid, 2 * a.num_sms);
    rest.min_items = some.min_items = few.max_items + 1;
    some.max_items = std::max(4 * (kPWarps / 2) * grid, few.max_items);
    many.min_items = some.max_items + 1;
    rest.max_items = many.max_items = INT_MAX;
    if (what == 1) modes_run<Row, 1, 1, 4>(st, few.max_items, few);
    if (what == 2) modes_run<Row, NW, 2, 4>(st, few.max_items, few);
    if (what == 3) modes_run<Row, NW, 3, 4>(st, few.max_items, few);
    int n = 1;
    if (what & 1) {
        if (a.item_cap >= some.min_items) modes_run<Row, 1, 1, 4>(st, grid, some), ++n;
        if (a.item_cap >= many.min_items) modes_run<Row, 1, 1, 2>(st, grid, many), ++n;
    }
    if (what & 2 && a.item_cap >= rest.min_items) {
        if (what == 3 && rest.sched) ++rest.sched;  // a counter of its own
        modes_run<Row, NW, 2, 2>(st, grid, rest), ++n;
    }
    return n;
}

// CTAs per panel: enough for one thread per column of 128-row blocks, more
// blocks go round the loop
int expand_ctas(int nz_max) {
    return std::max(1, (2 * ((nz_max + kPanelMaxBlk - 1) / kPanelMaxBlk) + kExpThreads - 1) / kExpThreads);
}

template <class Row, int NW>
int expand_launch(cudaStream_t st, int n_desc, int nz_max, const ProblemInfo* pinfo, const PanelDesc* desc,
                  const double* rows, const double* w, const double* g, double* T, double* W0, double* W1) {
    int n = 0;
    for (int d0 = 0; d0 < n_desc; d0 += 65535, ++n) {  // grid.y limit
        dim3 grid(expand_ctas(nz_max), std::min(65535, n_desc - d0));
        k_expand_items<Row, NW><<<grid, kExpThreads, 0, st>>>(pinfo, desc, d0, rows, w, g, T, W0, W1);
    }
    return n;
}

// Scan size of every problem and the scan's panels.  The number of eigenvalues
// of S (diagonal s_i, unit off-diagonals) below x is close to the sum over the
// rows of theta_i / pi with cos theta_i = (s_i - x) / 2 clipped to [-1, 1] (each
// row's local band is [s_i - 2, s_i + 2]); on the 20000-point grids of 0.002-0.5
// Hz it gives the mode count in [lo, hi] within one mode.  The scan takes about
// two shifts per mode plus 32, in units of kScanStep: of the problem alone, so
// that its modes do not depend on the batch to the last bit.  (Batches were once
// trimmed to a multiple of the device's warp schedulers, for units of one warp
// each; units have blocks of four: 45-azimuth sweep 6.86 ms trimmed, 6.69 not,
// 256 frequencies 2.31 and 2.28.)
// The sum over the rows is taken in 256 partial sums (single precision: their
// order fixes the scan's size); 1024 threads evaluate its terms, 2048 rows at a
// time, which the sums then take from shared memory (one problem of 20000 rows
// 31 us with a thread to a partial sum, now 22; a 45-azimuth sweep 88 and 65).
constexpr int kSizeThreads = 1024, kSizeSums = 256, kSizeRows = 2048;

__global__ void __launch_bounds__(kSizeThreads) k_panel_size(int P, ProblemInfo* __restrict__ pinfo,
                                                             const double* __restrict__ s) {
    __shared__ float part[kSizeSums / 32], term[kSizeRows];
    const int p = blockIdx.x;
    const double lo = pinfo[p].lo, hi = pinfo[p].hi;
    const double* __restrict__ row = s + pinfo[p].s_off;
    const int nz = pinfo[p].nz;
    float acc = 0.f;
    for (int r0 = 0; r0 < nz; r0 += kSizeRows) {
#pragma unroll
        for (int j = 0; j < kSizeRows / kSizeThreads; ++j) {
            const int t = threadIdx.x + j * kSizeThreads, i = r0 + t;
            float x = 0.f;
            if (i < nz) {
                const double v = row[i];
                const float ch = fminf(fmaxf((float)((v - hi) * 0.5), -1.f), 1.f);
                const float cl = fminf(fmaxf((float)((v - lo) * 0.5), -1.f), 1.f);
                x = acosf(ch) - acosf(cl);
            }
            term[t] = x;
        }
        __syncthreads();
        if (threadIdx.x < kSizeSums)
            for (int j = 0; j < kSizeRows / kSizeSums; ++j) acc += term[threadIdx.x + j * kSizeSums];
        __syncthreads();
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, off);
    if ((threadIdx.x & 31) == 0 && threadIdx.x < kSizeSums) part[threadIdx.x >> 5] = acc;
    __syncthreads();
    if (threadIdx.x == 0) {
        float t = 0.f;
        for (int w = 0; w < kSizeSums / 32; ++w) t += part[w];
        const float m_est = fmaxf(t * (float)(1.0 / kPi), 0.f);
        const int n = ((int)(2.f * m_est) + 32 + kScanStep - 1) / kScanStep * kScanStep;
        pinfo[p].n_scan = min(max(n, kScanStep), kScanMax);
        pinfo[p].m_est = m_est;
        plan_scan_panels<EssPanel>(pinfo[p], pinfo[p].n_scan);
    }
}

// the scan's panels where its size stands (wide-angle rows: kScanDefault points)
__global__ void k_panel_size_fixed(int P, ProblemInfo* __restrict__ pinfo) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p < P) plan_scan_panels<WmodPanel>(pinfo[p], pinfo[p].n_scan);
}

template <class Row>
int scan_launch(cudaStream_t st, int P, int nz_max, const ProblemInfo* pinfo, const double* rows, double* T,
                int* counts, unsigned* err) {
    int n = 1;
    const int step = 65535 / kScanSlots;
    for (int p0 = 0; p0 < P; p0 += step, ++n) {  // grid.y limit
        dim3 grid(expand_ctas(nz_max), kScanSlots * std::min(step, P - p0));
        k_expand_scan<Row><<<grid, kExpThreads, 0, st>>>(pinfo, p0, rows, T);
    }
    // the warps' rings, then their segments
    const size_t sm = kRingBytes<kTD> + kPWarps * (4 * 2 * 32 * 8 + 2 * 32 * 4);
    cudaFuncSetAttribute(k_panel_scan<Row>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    k_panel_scan<Row><<<P * kScanSlots, kPWarps * 32, sm, st>>>(pinfo, rows, T, counts, err);
    return n;
}

}  // namespace

int launch_panel_scan(cudaStream_t st, bool wide, int P, int nz_max, ProblemInfo* pinfo, const double* rows, double* T,
                      int* counts, unsigned* err) {
    if (wide) {
        k_panel_size_fixed<<<(P + 127) / 128, 128, 0, st>>>(P, pinfo);
        return 1 + scan_launch<WmodPanel>(st, P, nz_max, pinfo, rows, T, counts, err);
    }
    k_panel_size<<<P, kSizeThreads, 0, st>>>(P, pinfo, rows);
    return 1 + scan_launch<EssPanel>(st, P, nz_max, pinfo, rows, T, counts, err);
}

int launch_panel_items(cudaStream_t st, bool wide, int P, ProblemInfo* pinfo, const int* counts, int max_modes,
                       int bis_item, WorkItem* items, int cap, PanelDesc* desc, int* tot, bool first, unsigned* err,
                       int order) {
    if (bis_item < 1 || bis_item > kWItem) return -1;
    k_panel_items<<<1, kItemThreads, 0, st>>>(P, pinfo, counts, max_modes, bis_item, cap, tot, first, err, order);
    auto* f = wide ? k_panel_groups<WmodPanel> : k_panel_groups<EssPanel>;
    f<<<(P + kPlanWarps - 1) / kPlanWarps, kPlanWarps * 32, 0, st>>>(P, pinfo, counts, bis_item, items, cap, desc, tot);
    return 2;
}

int launch_panel_expand(cudaStream_t st, bool wide, int n_desc, int nz_max, const ProblemInfo* pinfo,
                        const PanelDesc* desc, const double* rows, const double* w, const double* g, double* T,
                        double* W0, double* W1) {
    if (wide) return expand_launch<WmodPanel, 2>(st, n_desc, nz_max, pinfo, desc, rows, w, nullptr, T, W0, W1);
    return g ? expand_launch<EssPanel, 2>(st, n_desc, nz_max, pinfo, desc, rows, w, g, T, W0, W1)
             : expand_launch<EssPanel, 1>(st, n_desc, nz_max, pinfo, desc, rows, w, nullptr, T, W0, nullptr);
}

int launch_panel_fill(cudaStream_t st, bool wide, int P, int nz_max, int m_max, const ModesArgs& a) {
    int n = 0;
    const int ny = ((nz_max + kCkRows - 1) / kCkRows + 7) / 8;
    auto* peak = wide ? k_panel_fill<WmodPanel, true> : k_panel_fill<EssPanel, true>;
    auto* fill = wide ? k_panel_fill<WmodPanel, false> : k_panel_fill<EssPanel, false>;
    for (int p0 = 0; p0 < P && m_max > 0; p0 += 32768) {
        const dim3 grid((m_max + 31) / 32, ny, std::min(P - p0, 32768));
        peak<<<grid, 256, 0, st>>>(p0, a);
        fill<<<grid, 256, 0, st>>>(p0, a);
        n += 2;
    }
    return n;
}

namespace {
template <class Row, int NW, bool kV>
int twist_run(cudaStream_t st, int grid, const ModesArgs& a) {
    const size_t sm = kRingBytes<kTD + NW * kWD>;
    auto* f = k_twist_modes<Row, NW, kV>;
    cudaFuncSetAttribute((const void*)f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    f<<<std::min(panel_slots(grid) / 2, a.item_cap), kPWarps * 32, sm, st>>>(a);
    return 1;
}
}  // namespace

int launch_twist_modes(cudaStream_t st, bool wide, int grid, const ModesArgs& a) {
    if (wide) return a.vstate ? twist_run<WmodPanel, 2, true>(st, grid, a) : twist_run<WmodPanel, 2, false>(st, grid, a);
    if (a.g) return a.vstate ? twist_run<EssPanel, 2, true>(st, grid, a) : twist_run<EssPanel, 2, false>(st, grid, a);
    return a.vstate ? twist_run<EssPanel, 1, true>(st, grid, a) : twist_run<EssPanel, 1, false>(st, grid, a);
}

int launch_rows_modes(cudaStream_t st, bool wide, int grid, const ModesArgs& a, int what) {
    if (wide) return a.vstate ? rows_run<WmodPanel, 2, true>(st, grid, a, what) : rows_run<WmodPanel, 2, false>(st, grid, a, what);
    if (a.g) return a.vstate ? rows_run<EssPanel, 2, true>(st, grid, a, what) : rows_run<EssPanel, 2, false>(st, grid, a, what);
    return a.vstate ? rows_run<EssPanel, 1, true>(st, grid, a, what) : rows_run<EssPanel, 1, false>(st, grid, a, what);
}

int launch_panel_modes(cudaStream_t st, bool wide, int grid, const ModesArgs& a, int what) {
    if (wide) return modes_launch<WmodPanel, 2>(st, grid, a, what);
    return a.g ? modes_launch<EssPanel, 2>(st, grid, a, what) : modes_launch<EssPanel, 1>(st, grid, a, what);
}

int panel_ctas_per_sm() { return kPanelCtas; }

int panel_ck_slots(int grid, bool rows) {
    return panel_slots(grid) + (rows ? 2 * kPWarps * (grid / kPanelCtas * kRowsCtas) : 0);
}

}  // namespace ncpa
