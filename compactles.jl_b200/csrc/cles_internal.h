// Internal declarations shared by the host runtime and the CUDA kernels.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>
#include <atomic>
#include <memory>
#include <stdexcept>
#include <string>
#include <utility>
#include <vector>

#include "../../include/cles.h"

namespace cles {

// ---------------------------------------------------------------- errors ----
struct Error : std::runtime_error {
    int code;
    Error(int c, const std::string& m) : std::runtime_error(m), code(c) {}
};
void set_last_error(const std::string& s);
#define CLES_CUDA(call)                                                                         \
    do {                                                                                        \
        cudaError_t e_ = (call);                                                                \
        if (e_ != cudaSuccess)                                                                  \
            throw ::cles::Error(CLES_ECUDA, std::string(#call) + ": " + cudaGetErrorString(e_)); \
    } while (0)
void count_launch(int n = 1);
int64_t launch_count();   // kernels launched by this library so far
// CUDA-event bracketing of compact launches (cles_profile_enable)
bool profiling();
int prof_begin(cudaStream_t st, int family, double bytes);
void prof_end(int rec, cudaStream_t st);
void check_launch(const char* what);

// -------------------------------------------------- dependent launches ----
// Kernels of a step follow one another on one stream, a few microseconds each on
// small grids.  Inside a DependentLaunches scope (one thread's launches, one
// solver's step) they are launched with programmatic stream serialization: a
// kernel's blocks may start while its predecessor drains, set up what does not
// depend on it (indices, constant tables) and wait in grid_dependency_wait until
// it has completed.  Only kernels that call it are launched so.
// Such a kernel is alive while its predecessor still writes, so its pointer
// parameters carry no __restrict__ (that promises memory nobody else writes for the
// kernel's whole life, and lets reads move above the wait).  The promise is made
// to an inlined body called after the wait; constant plan tables keep it.
struct DependentLaunches {
    explicit DependentLaunches(bool on);
    ~DependentLaunches();
    DependentLaunches(const DependentLaunches&) = delete;
    static bool active();

private:
    bool prev_;
};
#ifdef __CUDACC__
// Until every earlier kernel of the stream has completed (at once when launched
// normally); lets the next kernel's blocks come in behind this one's.
__device__ __forceinline__ void grid_dependency_wait() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
// Launch of a kernel that calls grid_dependency_wait before it touches anything
// another kernel writes.
template <typename... K, typename... A>
inline void launch_dependent(void (*kern)(K...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, A&&... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    if (DependentLaunches::active()) {
        at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        at[0].val.programmaticStreamSerializationAllowed = 1;
        cfg.attrs = at;
        cfg.numAttrs = 1;
    }
    CLES_CUDA(cudaLaunchKernelEx(&cfg, kern, std::forward<A>(args)...));
}
// A launch with more than 48 KB of dynamic shared memory needs the kernel's limit
// raised.  The limit belongs to the kernel and device, not to a launch or a host
// thread: it goes to the device's maximum once (`raised`: the kernel's devices), never
// to one launch's size, which another thread's larger launch may be between its own
// call and its launch.
constexpr size_t kMaxDynamicSmem = 227 * 1024;   // sm_100, kernels without static shared memory
template <typename K>
inline void raise_smem_limit(K* kern, size_t bytes, std::atomic<uint64_t>& raised) {
    if (bytes <= 48 * 1024) return;
    int dev = 0;
    CLES_CUDA(cudaGetDevice(&dev));
    const uint64_t bit = dev < 64 ? (uint64_t)1 << dev : 0;
    if (raised.load(std::memory_order_acquire) & bit) return;
    CLES_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMaxDynamicSmem));
    raised.fetch_or(bit, std::memory_order_release);
}
#endif

// ------------------------------------------------------------ field views ----
// A batch of scalar fields of one grid: element (i, j, k) of field b sits at
// base + b*comp_stride + i + j*sy + k*sz (elements).  `base` points at
// interior element (0, 0, 0).
struct FieldView {
    void* base;
    int64_t comp_stride;
    int64_t sy, sz;
};

// ------------------------------------------------------------ compact plans ---
constexpr int kMaxSeg = 32;        // points per thread (register tile)
constexpr int kMaxClo = CLES_MAX_NC;
constexpr int kMaxCloLen = CLES_MAX_CLO_LEN;

// Kernel parameters of one directional compact operator (passed by value).
struct CompactParams {
    int n;               // line length
    int dim;             // 0, 1, 2
    int nx, ny, nz;      // interior extents of the grid
    int S;               // segments per line
    int seg_base, seg_rem;  // segment s: length seg_base + (s < seg_rem), local_range split
    int LB;              // lines per CTA
    int q, M;
    int symmetric;
    int periodic;
    int lo_closed, hi_closed;
    // an open end is a rank interface of a split line: interior rows whose
    // stencil reads the caller's halo, couplings beyond the end left to the
    // rank-level spikes
    int lo_open, hi_open;
    int nc;
    int hasred;
    double a0;
    double ci[CLES_MAX_M];
    int clo_len[kMaxClo];
    double clo[kMaxClo][kMaxCloLen];
    double chi[kMaxClo][kMaxCloLen];
    // offsets (elements) into the coefficient table
    int64_t off_f0, off_f1, off_f2, off_f3, off_f4;  // q=1: l, dinv, c ; q=2: L1, L2, U1, U2, Uinv0
    int64_t off_V, off_W;                              // V[s][t][i], W[s][t][i]
    int64_t off_G;                                     // reduced inverse, (2qS) x (2qS) row-major
    // Closed tridiagonal lines: the interface system is solved by parallel
    // cyclic reduction with precomputed 2x2 blocks instead of the dense inverse.
    // Level l (distance 2^l), segment s: alpha[4], gamma[4] at off_pcr + (l*S + s)*8,
    // then the final 2x2 inverse of segment s at off_pcr + (pcr_levels*S + s)*8.
    int pcr, pcr_levels;
    int64_t off_pcr;
    int64_t lines;
};

// Warp-per-line form for periodic tridiagonal x lines of n = 32 * XP points
// (XP = 2, 4, 6, 8, 12, 16: n = 64, 128, 192, 256, 384, 512):
// lane s owns the XP contiguous points [s*XP, (s+1)*XP).  Every lane segment
// is the same Toeplitz block, so the local factorisation, the spikes and the
// parallel-cyclic-reduction matrices of the 32-segment interface system are
// line- and lane-independent and travel as kernel parameters.
constexpr int kMaxXP = 16;
struct WarpLineParams {
    int XP;                                   // points per lane: 2, 4, 6, 8, 12 or 16
    double l[kMaxXP], dinv[kMaxXP], c[kMaxXP];  // segment Thomas factors
    double v[kMaxXP], w[kMaxXP];              // spikes: couplings to the previous tail / next head
    double alpha[4][4], gamma[4][4];          // PCR steps at distances 1, 2, 4, 8 (2x2, row-major)
    double alpha_f[4], binv_f[4];             // pairing at distance 16, then the 2x2 solve
    float lf[kMaxXP], dinvf[kMaxXP], cf[kMaxXP], vf[kMaxXP], wf[kMaxXP];
    float alphaf[4][4], gammaf[4][4], alpha_ff[4], binv_ff[4];
};

// TMA-pipelined form for periodic tridiagonal y/z lines with equal segments
// (n = S * m, m <= 32, n <= 256): every segment has the same factorisation and
// spikes, which travel as kernel parameters; the reduced inverse stays in the
// table (copied to shared memory once per persistent CTA).
struct TileLineParams {
    int m;
    double l[kMaxSeg], dinv[kMaxSeg], c[kMaxSeg], v[kMaxSeg], w[kMaxSeg];
    float lf[kMaxSeg], dinvf[kMaxSeg], cf[kMaxSeg], vf[kMaxSeg], wf[kMaxSeg];
};

// Host-side plan: parameters plus the coefficient tables on the device.
// General tile form (closed lines, or the pentadiagonal C10): with equal
// segments only three segment classes exist -- the first (closure rows, no
// left spike), the interior ones (all alike) and the last -- so their
// factorisations and spikes travel as kernel parameters with static indices.
// f: q = 1 -> l, dinv, c; q = 2 -> L1, L2, U1, U2, 1/U0 (same as the table).
struct TileGenParams {
    double f[3][5][kMaxSeg];
    double v[3][2][kMaxSeg], w[3][2][kMaxSeg];
    float ff[3][5][kMaxSeg];
    float vf[3][2][kMaxSeg], wf[3][2][kMaxSeg];
};

// Coefficients of the segment kinds of a LinePlan (0 first, 1 long interior, 2
// short interior, 3 last segment; periodic lines use 1 and 2), kernel
// parameters of k_line.  f: q = 1 -> l, 1/u0, u1/u0; q = 2 -> L1, L2, u1/u0,
// u2/u0, 1/u0, with rows past the segment's end copying the forward values
// upwards and contributing nothing backwards.  v / w: spikes.  tl: what the tail
// needs (see ln_sweep).
template <typename T, int Q, int MS>
struct LineCoef {
    T f[4][Q == 1 ? 3 : 5][MS];
    T v[4][Q][MS], w[4][Q][MS];
    T tl[4][4];
    T clo[kMaxClo][kMaxCloLen], chi[kMaxClo][kMaxCloLen];   // closure rows, as in CompactParams
    T ci[CLES_MAX_M], a0, pad_;
};

// Where element e (of n: [2q rows][Wn segments][2q end values]) of segment s's
// inverse rows sits.  Short tiles run few lines a block, so that the lanes of a
// warp hold neighbouring segments: segment fastest.  The others share a segment
// among 16 or 32 lanes: a segment's elements together, for wide broadcast loads
// (C10 on 201x161x129: 254 us against 299 us segment-fastest).
__host__ __device__ inline size_t line_row_index(int MS, int S, int n, int e, int s) {
    return MS == 16 ? (size_t)e * S + s : (size_t)s * n + e;
}

// Segmented form of a line (k_line; line_segments gives the lengths): S segments, the first `rem`
// of base + 1 points and the others of base, on register tiles of MS points.
struct LinePlan {
    int MS = 32, S = 0, base = 0, rem = 0;
    int mm = 0;                       // longest segment, rounded up to a group of four rows
    int Wn = 0, Kr = 0;               // interface window: segments, radius
    std::vector<unsigned char> coef;  // LineCoef<plan dtype, q, MS>
    std::vector<unsigned char> host_tab;   // reduced inverse rows (line_row_index), until they are on the device
    const void* dcoef = nullptr;      // coef and those rows in the plan's device block
    const void* tab = nullptr;
};
struct LineArgs {
    FieldView in, out;
    // fields split .. are fields 0 .. of a second group under the same operator
    // (strides of the first)
    const void* in2;
    void* out2;
    int split;
    int S, base, rem, mm, Wn, Kr;
    int logL, SC, CL;                 // lines (log2) and segments per block, blocks per cluster
    int pitch;                        // shared row of an x line, elements
    int gstage;                       // the inverse rows are staged in shared memory
    int mode, rk_first;
    struct {
        double *Q, *du;
        double A, B, dt;
        const double* dtp;
    } rk;
};

struct CompactPlan {
    bool has_tl = false;
    TileLineParams TL;
    bool has_tg = false;   // y/z lines fit the general tile kernel (closures, q = 2)
    TileGenParams TG;
    bool has_xw = false;
    WarpLineParams XW;
    CompactParams P;
    int dtype = CLES_F64;
    void* dev = nullptr;     // device block of all tables
    double* tab64 = nullptr; // into dev
    float* tab32 = nullptr;
    size_t tab_elems = 0;
    std::unique_ptr<LinePlan> line;   // k_line form, where the plan has one
    ~CompactPlan();
};

// Launch shape of k_line: lines and segments per block, blocks per cluster.
struct LineShape {
    int L, SC, CL;
};
LineShape line_shape(const CompactParams& P, const LinePlan& lp, int count, int num_sms, size_t el);

// Builds the plan of `scheme` along `dim` (0-based) of a grid with interior
// extents n3[3]; periodic says whether the line wraps.  lo_fold / hi_fold set
// a coordinate-singularity fold at that end of a closed line: the antipodal
// parity (+1 / -1) of the field the plan is applied to, 0 for a closure.
// lo_open / hi_open make that end of a non-periodic line a rank interface.
// pow2_seg_max > 0 (batched plans): S is the fewest power-of-two segments of
// at most pow2_seg_max (8, 16 or 32) points.
// host_only: everything but the device tables (no CUDA call).
void build_compact_plan(CompactPlan& plan, const cles_scheme& scheme, const int n3[3], int dim,
                        bool periodic, double h, int dtype, int lo_fold = 0, int hi_fold = 0,
                        bool lo_open = false, bool hi_open = false, int pow2_seg_max = 0, bool host_only = false);

// The LHS band of one line (or one rank's piece of a split line), row-major
// n x (2q+1): interior band, closure rows at closed ends, parity folds, and
// no couplings beyond a non-periodic end.  Unpivoted banded LU of the whole
// band; solve() applies its inverse in place.
struct LineBand {
    int n = 0, q = 1;
    std::vector<double> a;
    std::vector<double> L, U;
    void factor();
    void solve(double* x) const;
};
LineBand make_line_band(const cles_scheme& s, int n, int lo_fold, int hi_fold, bool lo_open, bool hi_open);

// Output modes of the compact operator.  OUT_RK finishes the flux divergence
// and applies the low-storage RK update in the store (see launch_compact_rk).
enum { OUT_STORE = 0, OUT_NEGATE = 1, OUT_SUBTRACT = 2, OUT_RK = 3 };

// Low-storage RK epilogue: with dq = out - D(f), v = A du + dt dq; du = v;
// Q += B v (src/timestep.jl:86-95).  Q and du share the layout of `out`.
struct RkEpilogue {
    double* Q;
    double* du;
    double A, B, dt;
    const double* dtp;  // when set, dt is read from device memory (graph mode)
    // k_line also stores dq into `out`: the right-hand side of a step's last stage,
    // for cles_get_rhs (the tile kernels consume it)
    int keep;
};

int num_sms();   // multiprocessors of the current device
// Whether a tile kernel can take `count` fields of this plan and view (y / z lines).
bool tma_takes(const CompactPlan& plan, const FieldView& in, int count);
// TMA-pipelined y/z launch; false when the plan or the views do not qualify.
bool try_launch_tma(const CompactPlan& plan, const FieldView& in, const FieldView& out, int count, int mode,
                    cudaStream_t st, const RkEpilogue* rk = nullptr);
// x lines of a plan with the general tile form: persistent kernel, cp.async
// staging into a transposed shared-memory tile; false if the plan does not fit.
bool try_launch_xt(const CompactPlan& plan, const FieldView& in, const FieldView& out, int count, int mode,
                   cudaStream_t st);
// k_line launch; false (and nothing launched) when the plan has no line form.
// rk: the RK update of mode OUT_RK; rk_first: no earlier direction stored into
// `out`, the divergence is this direction's alone.
// in2 / out2 / count2: a second group of fields, views of the same strides.
bool try_launch_line(const CompactPlan& plan, const FieldView& in, const FieldView& out, int count, int mode,
                     cudaStream_t st, const RkEpilogue* rk = nullptr, bool rk_first = false,
                     const void* in2 = nullptr, void* out2 = nullptr, int count2 = 0);
// The operator over two groups of fields (OUT_STORE, views of the same strides):
// one launch where the kernel can take both, else two.
void launch_compact_pair(const CompactPlan& plan, const FieldView& in, const FieldView& out, int count,
                         const FieldView& in2, const FieldView& out2, int count2, cudaStream_t st);
// Flux divergence of the last direction fused with the RK update; false (and
// nothing launched) when the plan takes neither the TMA path nor k_line.  first:
// the only direction, `out` holds nothing yet (and is not written).
bool launch_compact_rk(const CompactPlan& plan, const FieldView& in, const FieldView& out, int count,
                       const RkEpilogue& rk, cudaStream_t st, bool first = false);
// One rank's piece of a line split across `ranks` ranks along `dim`
// (src/decomposition.jl:73-78 local_range; src/tridiag.jl:85-170 and
// src/banded.jl:108-214 with P > 1).  `local` solves the rank's own rows with
// open (interface) ends.  V / W are this rank's spikes: the response of its
// local solve to the couplings of its first q rows to the previous rank's
// last q unknowns and of its last q rows to the next rank's first q.  Gsel
// holds the 2q rows of the inverse of the (2q ranks)^2 reduced system that
// give those 2q unknowns from every rank's local heads and tails.
struct SplitPlan {
    CompactPlan local;
    int ranks = 1, rank = 0, dim = 0, q = 1, M = 1, n = 0;
    int n3[3] = {0, 0, 0};
    int64_t lines = 0;
    bool lo_open = false, hi_open = false;
    int prev = -1, next = -1;   // neighbouring rank coordinates, -1 for none
    int dtype = CLES_F64;
    void* tab = nullptr;        // [V q x n][W q x n][Gsel 2q x 2q*ranks], plan dtype
    ~SplitPlan();
};
void build_split_plan(SplitPlan& sp, const cles_scheme& s, const int n3_local[3], int dim, bool periodic,
                      int n_global, int ranks, int rank, double h, int dtype);
// The M planes at each end of a local interior along `dim` (lines: the
// product of the other two extents, lower dimension fastest).
struct HaloSpec {
    int dim = 0;
    int n3[3] = {0, 0, 0};
    int M = 0;
    int64_t lines = 0;
    bool lo_open = false, hi_open = false;
};
HaloSpec halo_spec(const SplitPlan& sp);
// Copies the M planes next to each open end of the local interior into lo / hi
// ([count][M][lines]) when pack, or those buffers into the halo planes
// beyond each open end when !pack.
void halo_planes(const HaloSpec& hs, const FieldView& f, void* lo, void* hi, int count, bool pack, int dtype,
                 cudaStream_t st);
void split_halo(const SplitPlan& sp, const FieldView& f, void* lo, void* hi, int count, bool pack, cudaStream_t st);
// From every rank's heads and tails ([ranks][count][2q][lines]): the 2q
// neighbouring unknowns per line into zbuf ([count][2q][lines]), then
// out -= V z_prev + W z_next over the local interior.
void split_correct(const SplitPlan& sp, const void* gathered, void* zbuf, const FieldView& out, int count,
                   cudaStream_t st);
// The same with the local solution read from `loc` and the corrected value
// r = loc - V z_prev - W z_next written to `out` by mode: OUT_STORE out = r,
// OUT_NEGATE out = -r, OUT_SUBTRACT out -= r (loc may alias out except for
// OUT_SUBTRACT).
void split_correct(const SplitPlan& sp, const void* gathered, void* zbuf, const FieldView& loc, const FieldView& out,
                   int count, int mode, cudaStream_t st);
// dst = src over an n3 interior of `count` fields (views of equal extents,
// any strides).
void copy_view(const FieldView& src, const FieldView& dst, const int n3[3], int count, int dtype, cudaStream_t st);

// ---- batched line solves over many grids (batch_compact.cu) ----------------
// One grid's directional plan in a batched launch.  Its lines are cut into
// power-of-two segments (build_compact_plan with pow2_segments), and P.LB is
// the launch's threads / P.S, so every CTA of the launch runs LB x S threads.
// The grid's fields start at element `off` of the launch's arena blocks.
struct BatchLinePlan {
    CompactParams P;
    const void* tab;      // the plan's coefficient table (launch dtype)
    int64_t off;          // element offset of the grid's cell (0, 0, 0)
    int64_t sy, sz;       // strides of the grid's fields
    const double* clk;    // graph-mode clock of the grid (dt in slot 1)
};
constexpr int kBatchMaxThreads = 512;   // threads per CTA of a batched line-solve launch (at most)
// Kernel template of a batched launch (shared by all its plans).
struct BatchLaunchKind {
    int dtype;            // CLES_F64 / CLES_F32
    int q, M, xmode;
    int ms;               // register tile: 8, 16 or 32 points (>= every plan's longest segment)
    int threads;          // LB x S of every plan
    size_t smem;          // dynamic shared memory (max over the plans)
};
// Dynamic shared memory one plan needs with LB lines per CTA.
size_t batch_plan_smem(const CompactParams& P, int LB, int dtype);
// blocks[b] = (plan, first line); blockIdx.y = field.  in / out / Q / du are
// arena block starts (fields cells_total elements apart).  mode OUT_RK applies
// the low-storage RK update with coefficients (A, B) and each grid's dt
// (clk[1]); skip_idle leaves out every grid whose dt is 0 (done or failed).
void launch_compact_batch(const BatchLaunchKind& kind, const BatchLinePlan* plans, const int2* blocks, int nblocks,
                          const void* in, void* out, int64_t cells_total, int count, int mode, double* Q, double* du,
                          double A, double B, int skip_idle, cudaStream_t st);

// Bounded-wait timeouts recorded by device kernels since the last call (cleared).
int take_device_timeouts(cudaStream_t st);
// One CTA that waits limit_ns on an mbarrier nothing completes (the expiry
// path of the operators' bounded wait).
void launch_wait_selftest(uint64_t limit_ns, cudaStream_t st);

// Launch the operator over `count` fields of `in` into `out` (may alias).
void launch_compact(const CompactPlan& plan, const FieldView& in, const FieldView& out, int count, int mode,
                    cudaStream_t st);
// y/z lines of a split-line plan in the general tile form, the TMA box
// widened by the M halo rows at each end; false (nothing launched) when the
// plan or the views do not qualify.
bool try_launch_tg_split(const CompactPlan& plan, const FieldView& in, const FieldView& out, int count, void* iface,
                         cudaStream_t st);
// Local solve of a split-line plan (tile or generic kernel, OUT_STORE); the first and
// last q values of every line's local solution also go to iface, laid out
// [count][2q][lines] in the plan's dtype.
void launch_compact_split(const CompactPlan& plan, const FieldView& in, const FieldView& out, int count, void* iface,
                          cudaStream_t st);

}  // namespace cles
