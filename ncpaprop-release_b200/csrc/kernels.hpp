// Launchers of the sm_100a kernels of the ESS normal-mode path.  Host code in
// ncpa_api.cu calls these; each returns the number of kernels it launched.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

namespace ncpa {

// error flags written by kernels into the context's device status word
enum : unsigned {
    kErrTimeout = 1u,  // a bounded mbarrier wait gave up
    kErrBracket = 2u,  // bisection bracket inconsistent with the Sturm counts
    kErrWkb = 4u,      // WKB search needed more trial wavenumbers than threads
    kErrTooMany = 8u,  // a problem has more modes than allowed (device-built work items)
};

// Per (frequency, azimuth) problem, device resident.  Every problem carries
// its own solver grid (size, spacing, source/receiver rows and the offsets of
// its rows in the batch arrays), so one batch may mix grid sizes.
struct ProblemInfo {
    double freq, omega, az;
    double k_min, k_max;   // wavenumber window [1/m]
    double lo, hi;         // window in units of the scaled matrix S = h^2 A
    double ceff_grnd, ceff_top;
    double dz;             // grid spacing [m]
    unsigned long long ceffmin_bits, ceffmax_bits;  // positive doubles as ordered bits
    long long s_off;       // offset (doubles) of the problem's row in s, g and kz2 (rows padded to kChunk)
    long long w_off;       // offset (doubles) of its attenuation-weight row in w
    int nz;                // grid points
    int isrc, ircv;        // source / receiver grid rows
    int c_lo, c_hi;        // Sturm counts at lo, hi
    int M, off;            // number of modes and offset into the mode arrays
    int used_wkb;
    int wkb_trial;         // first WKB trial that ends the walk (kWkbNone before it is taken)
    int n_scan;            // shifts of the isolation scan (<= kScanMax)
    float m_est;           // estimated mode count in [lo, hi] (-1: not estimated)
    int upp, sp_blk;       // the scan's panels (panel.cu): scan units per panel and rows per block (0: raw rows)
    int item0;             // first work item
    int grp_off, grp_cap;  // panel descriptors reserved for the work items
    int blk_cap;           // block records reserved (the scan's panels, then the work items')
    long long blk_off;     // the first of them
    double g0;             // wide-angle rows: ground term of row 0, 1 / (dz admittance + 1)
    unsigned long long c0min_bits;  // wide-angle rows: least c_0
};

constexpr int kWkbNone = 1 << 30;

struct WorkItem {
    int problem;  // problem index
    int j0;       // first eigen-index inside the problem (0 = lowest k)
    int m;        // eigenvalues in this item (<= kWItem for bisection)
    int pad;      // its panel (panel.cu; -1: none)
};

// Panel expansions (panel.cu): degrees of the block matrices and of their
// derivatives with respect to a weight, record sizes in doubles, records per
// shared-memory chunk, block sizes and the bound on r B^2
constexpr int kPD = 14, kPW = 11;
constexpr int kRecT = 4 * (kPD + 1) + 2, kRecW = 4 * (kPW + 1);
constexpr int kPanelChunk = 4;
constexpr int kPanelMaxBlk = 128;
// The shortest blocks; a panel that asks for shorter ones sweeps the rows as they
// are.  Blocks of 16 rows cost twice the instructions of the rows, in a quarter
// of the chain: worth it on long grids, whose solves wait for chains more than
// for the FP64 pipe (4 Hz, 20000 rows alone 2.15 -> 1.85 ms; 36 azimuths of 2 Hz,
// 8000 rows, wide 8.8 -> 5.8), not on short ones (90 azimuths of 1 Hz, 2500 rows
// 1.5 -> 2.0).  Blocks of 8 cost four times the rows and were used before (2.4).
#ifdef __CUDACC__
__host__ __device__
#endif
constexpr int panel_min_blk(int nz) { return nz >= 4096 ? 16 : 32; }
constexpr double kRhoMax = 10.0;

struct PanelDesc {
    double xc, r;   // shifts within r of xc
    long long rec;  // first block record
    int blk;        // rows per block
    int problem;    // -1: unused
};

constexpr int kScanMax = 512;      // count slots per problem of the isolation scan
constexpr int kScanStep = 64;      // shifts per scan unit (four warps, each a quarter of the rows, two shifts per lane)
constexpr int kScanDefault = 256;  // shifts per problem unless the scan sizes them (wide-angle rows)
constexpr int kChunk = 1024;      // doubles per TMA chunk of the diagonal
constexpr int kBlk = 16;          // rows between rescalings in k_eigvec
constexpr int kCkRows = 128;      // rows between twist candidates
// elements of each checkpoint array per warp slot of k_eigvec for grids of up
// to nz points (room for the sums of every coarse row)
inline long long ck_slot_elems(long long nz) {
    const long long a = (nz + kBlk - 1) / kBlk, b = 3 * ((nz + kCkRows - 1) / kCkRows);
    return (a > b ? a : b) * 32;
}
// elements per warp slot of the coarse rows of grids of up to nz points
inline long long coarse_slot_elems(long long nz) { return (nz + kCkRows - 1) / kCkRows * 32; }
constexpr int kWItem = 32;        // eigenvalues per warp work item of the bisection
constexpr int kEvItem = 32;       // eigenvalues per warp work item of the eigenvector kernel
constexpr int kEvWarpsPerCta = 4; // warps per eigenvector CTA

// knot-level derived quantities
int launch_steffen(cudaStream_t st, int n, const double* x, const double* y, int batch, int ystride,
                   double* coef, int cstride);
int launch_profile_derived(cudaStream_t st, int n, const double* z, const double* u, const double* v,
                           const double* p, const double* rho, const double* pcoef, const double* rcoef,
                           int have_c0, double* c0, double* ws, double* wd);
int launch_ceff_knots(cudaStream_t st, int n, int n_az, const double* az, const double* c0, const double* ws,
                      const double* wd, double* ceff);
// One group (a profile's frequencies x azimuths on one grid): what the knot-
// and grid-level kernels read and write.  Problem p = frequency n_az + azimuth;
// its rows are nz_pad apart in s (doubles, or (B, U) pairs when wide), gs and
// kz2 (or null), its weights per frequency in w.
struct GroupDesc {
    int nk, nz, nz_pad, n_f, n_az, wide, isrc, ircv;
    double z_min, dz_grid, dz, admittance;
    const double *zk, *c0, *ws, *wd, *t, *p, *rho, *rcoef, *pcoef;
    const double* attn;  // user attenuation at the knots, or null: Sutherland-Bass
    const double *freqs, *az;
    double *ceffk, *ceffc, *alpha, *alphac;  // [n_az | n_f][nk], coefficients [..][4 (nk - 1)]
    double *wck, *wcc, *c0k, *c0c;           // wide: wind component, c0
    double* rho_pair;                        // rho at the source and receiver rows
    ProblemInfo* pinfo;
    double *s, *w, *gs, *kz2;
};
// the largest of the groups' sizes (n groups; n_fields: c_eff and wide fields)
struct GroupDims {
    int n, nk, nz_pad, n_f, n_az, n_fields;
};
// knot- and grid-level fields of every group
int launch_groups(cudaStream_t st, const GroupDesc* desc, const GroupDims& d);
// matrix build (K1): s, optional kz2 = (omega/c)^2 and gs = 1/c^2; fills ceff
// extrema / ground / top in ProblemInfo
int launch_build_matrix(cudaStream_t st, const GroupDesc* desc, const GroupDims& d);
// WKB window and scaled bounds (K2); the records carry wkb_trial = kWkbNone
int launch_window(cudaStream_t st, int P, ProblemInfo* pinfo, const double* kz2, int wkb, int wvnum,
                  double c_min, double c_max, unsigned* err);
// FP64 throughput probe: each thread runs n_iter iterations of 8 independent
// FMA chains; out receives a value that keeps the chains live
int launch_fp64_probe(cudaStream_t st, int grid, int block, int n_iter, double* out);
// mode values by twisted factorisation of the rows (K4s, noalloc.cu)
struct EigvecArgs {
    const ProblemInfo* pinfo;
    const double* s;  // rows at pinfo[p].s_off
    const double* w;  // rows at pinfo[p].w_off
    const WorkItem* items;
    int n_items;
    const double* mu;
    double* kr;
    double* ki;
    double* vs;
    double* vr;
    double* vg;
    double* ck_q1;  // checkpoint scratch, one slot per warp of the grid
    double* ck_q2;
    int* ck_e;
    long long ck_slot_stride;  // elements per warp slot (blocks of the largest grid x 32)
    unsigned* err;
};
int launch_eigvec(cudaStream_t st, int grid, const EigvecArgs& a);
// The eigen-solve on panel expansions (panel.cu) of the ESS rows or, wide, of
// the wide-angle rows (mu = kappa = h k; W1 for a weight of ones).  T: block
// transfer matrices (kRecT doubles a record), W0, W1: their derivatives for the
// weights w and, for group speeds, g (kRecW doubles).
// Isolation scan: sizes, expansions and Sturm counts at pinfo[p].n_scan points,
// counts[p kScanMax + t]
int launch_panel_scan(cudaStream_t st, bool wide, int P, int nz_max, ProblemInfo* pinfo, const double* s, double* T, int* counts,
                      unsigned* err);
// c_lo, c_hi, M and off of every problem, the work items (at most bis_item
// eigenvalues, their panel in WorkItem::pad or -1) and the panels; tot =
// {items, items, modes, items without a panel, 0, 0}, or after the first part of
// a batch the modes and [5], the items without a panel, added to those of the
// parts before; kErrTooMany above max_modes or cap
int launch_panel_items(cudaStream_t st, bool wide, int P, ProblemInfo* pinfo, const int* counts, int max_modes, int bis_item,
                       WorkItem* items, int cap, PanelDesc* desc, int* tot, bool first, unsigned* err, int order);
// expansions of the work items' panels
int launch_panel_expand(cudaStream_t st, bool wide, int n_desc, int nz_max, const ProblemInfo* pinfo, const PanelDesc* desc,
                        const double* s, const double* w, const double* g, double* T, double* W0, double* W1);
constexpr int kCkVals = 5;  // doubles of a coarse row's checkpoint, at most
// full vectors: the state of a chain before a coarse row, times 2^E
struct VecState {
    double u, e;
    int E, pad;
};
// and per mode its shift, the factors of either chain (with exponents) that
// make it the mode function, and the row where they meet
struct VecTwist {
    double mu, fu, fb;
    int Eu, Eb, r, pad;
};
struct ModesArgs {
    const ProblemInfo* pinfo;
    const double* rows;
    const double* w;
    const double* g;  // null: no group speeds
    const double *T, *W0, *W1;
    const PanelDesc* desc;
    const int* counts;
    const WorkItem* items;
    const int* n_items_dev;
    int item_cap;  // at most this many
    double tol;
    double* mu;
    double *kr, *ki, *vs, *vr, *vg;
    double* ck_u;  // panel_ck_slots x kCkVals ck_stride doubles and x ck_stride ints
    int* ck_e;
    long long ck_stride;
    // full vectors (null: none): per problem at vstate_off the upward states
    // [coarse row][mode], then the downward ones
    VecState* vstate;
    const long long* vstate_off;
    VecTwist* vtwist;
    unsigned long long* vpeak;  // zeroed
    double* vfull;              // [row][mode] per problem at vfull_off
    const long long* vfull_off;
    int* sched;  // six item counters (zeroed) or null: round-robin
    int2* redo;   // items and lanes for launch_twist_modes, and their number (zeroed)
    int* n_redo;
    int num_sms;
    int min_items, max_items;  // (set by the launcher) a launch returns for other item counts
    unsigned* err;
    unsigned long long* steps;  // optional counter of row steps
};
// what: 1 eigenvalues, 2 mode values of the eigenvalues in mu, 3 both
int launch_panel_modes(cudaStream_t st, bool wide, int grid, const ModesArgs& a, int what);
// the mode functions at every row from the states that launch_panel_modes
// left; m_max: the most modes of a problem
int launch_panel_fill(cudaStream_t st, bool wide, int P, int nz_max, int m_max, const ModesArgs& a);
int panel_ctas_per_sm();
// the items without panels, which launch_panel_modes leaves out: the same grid and
// arguments, on any stream
int launch_rows_modes(cudaStream_t st, bool wide, int grid, const ModesArgs& a, int what);
// the modes whose twist the launches above found wanting, after them (grids with
// a few rows to a mode; elsewhere there are none)
int launch_twist_modes(cudaStream_t st, bool wide, int grid, const ModesArgs& a);
// checkpoint slots of all on that many CTAs
int panel_ck_slots(int grid, bool rows);

// 1-D TL; m_max: at least the most modes of a problem; scratch of tl1d_scratch
// bytes (0: none)
size_t tl1d_scratch(int P, int nr, int m_max, int num_sms);
int launch_tl1d(cudaStream_t st, int P, const ProblemInfo* pinfo, const double* kr, const double* ki,
                const double* vs, const double* vr, int nr, double dr, int lossless, double* re, double* im,
                double* incoh, int m_max, int num_sms, double* scratch);
// FP64 modal sum at heights rows[j] (rows of vec, M values each):
// re/im [nr x nj] with range_major, else [nj x nr]; scratch of
// modal_sum_scratch bytes
size_t modal_sum_scratch(int M, int nr);
int launch_modal_sum(cudaStream_t st, int M, const double* kr, const double* ki, const double* vs_src,
                     const double* vec, const int* rows, int nj, int nr, double dr, int lossless, bool range_major,
                     int num_sms, void* scratch, double* re, double* im);
// out[2 i], out[2 i + 1] = re[i], im[i]
int launch_pairs(cudaStream_t st, size_t n, const double* re, const double* im, double* out);
// out[c][r] = in[r][c] (rows x cols doubles)
int launch_transpose(cudaStream_t st, int rows, int cols, const double* in, double* out);
// broadband synthesis
int launch_twiddle(cudaStream_t st, int nfft, double* tw);
// fac: scratch of 4 doubles per mode
int launch_bb_transfer(cudaStream_t st, int nfreq, const int* off, const double* re_k, const double* im_k,
                       const double* vs, const double* vr, double rho_ratio, int nr, const double* ranges,
                       int zero_attn, int n_modes, double* fac, double* h);
int launch_src_builtin(cudaStream_t st, int kind, int nfreq, const double* f, double scale, double* out);
int launch_spline_eval(cudaStream_t st, int n, const double* x, const double* y, const double* coef, int m,
                       const double* xq, double* out);
int launch_starter(cudaStream_t st, int M, int nz, int step, int isrc, const double* v, const double* kr,
                   double k0, double* out);
int launch_fill_unit(cudaStream_t st, int n, double* h);
int launch_src_pulse2(cudaStream_t st, int n, double dt, double scale, double* x);
int launch_bb_pulse(cudaStream_t st, int nfreq, const double* f, const double* s_src, const double* h, int nr,
                    const double* t0, int nfft, const double* tw, double* out);
int launch_src_dft(cudaStream_t st, int n, const double* x, double dt, int nfft, int nfreq, const double* tw,
                   double* s);

// Wide-angle (WMod) modes (wmod.cu).  Rows of T(k) h^2: two doubles per row, (B_i, U_i) interleaved, at
// 2 * pinfo[p].s_off (the s layout, rows padded to kChunk); row 0's ground
// term goes to pinfo[p].g0.  The eigen-solve runs in kappa = h k: pinfo
// k_min / k_max bound the window in k, kappa_min = k_min dz.
int launch_wmod_build(cudaStream_t st, const GroupDesc* desc, const GroupDims& d);

// K5 modal sum on the tensor cores (modal_sum.cu)
struct MsPlan {
    int groups, n_chunks, M_pad, n_tiles, n_ctas, n_parts;
    long long n_units;  // (receiver group, range tile, mode chunk) units
    size_t a_img_bytes, q_bytes, tab_bytes, raw_bytes;
    // guarded sum (fmt 2): partial sums of |A'|, FP64 tables, flagged points
    size_t s_part_bytes, b64_bytes, tp64_bytes, a64_bytes, fix_list_bytes;
};
MsPlan ms_plan(int n_rcv, int M, int n_ranges, int num_sms);
// flag threshold of the guarded sum: a point with |P| < tau S is recomputed
double ms_guard_tau(const MsPlan& p);
// the error bound eps behind it: |P_tc - P| <= eps S
double ms_guard_eps(const MsPlan& p);
// fmt: 0 = 3-term split-BF16 (kind::f16), 1 = TF32 (kind::tf32), 2 = guarded
// 6-term split-BF16.  Buffers: a_img = A as complex FP32 per (receiver group,
// mode chunk), q = tile phases, tab = the B' image of each mode chunk
// (tile-independent); b64, tp64, a64 (fmt 2 only, else NULL) = the FP64
// offset phases, tile phases and A the fix-up reads
int launch_ms_prepare(cudaStream_t st, const MsPlan& p, int fmt, int n_rcv, int M, const double* kr,
                      const double* ki, const double* vs, const int* idx, const double* vfull, double dr, int lossless,
                      void* a_img, void* q, void* tab, void* b64, void* tp64, void* a64);
// variant: the schedule (ring depths) of the tensor-core kernel, 0 ..
// ms_tc_variants() - 1 (0: the deepest rings); results do not depend on it
int launch_ms_tc(cudaStream_t st, const MsPlan& p, int fmt, int n_ranges, const void* a_img, const void* q,
                 const void* tab, float* raw, float* s_part, unsigned* err, int variant);
int ms_tc_variants();
// ranges per tile of the tensor-core sums (the UMMA N)
int ms_tile_ranges();
void ms_tc_variant_shape(int fmt, int variant, int* t_stages, int* g_stages);
// s_part non-NULL: flag the points the guarded sum must recompute into
// fix_list / fix_count (zeroed by the caller)
int launch_ms_finish(cudaStream_t st, const MsPlan& p, int n_rcv, int n_ranges, double dr, const float* raw,
                     double* re, double* im, const float* s_part, int* fix_count, void* fix_list);
int launch_ms_fix(cudaStream_t st, int num_sms, int M, int M_pad, int n_ranges, double dr, const int* fix_count,
                  const void* fix_list, const void* a64, const void* tp64, const void* b64, double* re, double* im);

}  // namespace ncpa
