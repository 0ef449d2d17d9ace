// Segmented compact line solve for lines of 18 points and more along any dimension
// (up to 512 segments: 8192 points in short tiles, 16384 in long ones): the kernel
// behind launch_line (line_f64.cu, line_f32.cu).
//
// A thread owns one segment of at most MS points of one line in registers.
// Lines are cut into S segments of base or base + 1 points, so only four kinds
// of segment exist (first, long interior, short interior, last) and the
// coefficients of all four travel as kernel parameters: the unrolled sweeps
// take them as constant operands, without a load per point.  The 2q values at
// the ends of every segment go to shared memory; each thread forms the two
// neighbouring interface values it needs from the rows of the reduced inverse
// cut to a window of Wn segments (the inverse decays like rho^points away from
// the diagonal; what the window leaves out is below 2^-60 of the row's sum, in
// FP32 plans 2^-34).  A value that is not finite therefore reaches its window only,
// where a solve with the whole inverse spreads it over the line.
//
// The segments of one line may be spread over a cluster of CL blocks, which
// exchange end values through distributed shared memory: long lines then need
// neither a wide block nor a second launch, and a store in place is safe since
// every block has read its points before the cluster barrier.
//
// What bounds it: large plans in FP64 the registers (128 a thread, 16 warps an SM:
// load, solve and store phases of the resident blocks cover each other only in
// part), in FP32 instruction issue; small plans latency.  Against the kernels it
// replaced (generic segments with table loads; two launches of pieces for few long
// lines), us a launch on B200:
//   C10, three FP64 201x161x129 fields, walls, x / y / z: 243 / 166 / 136 -> 99 / 80 / 72
//   C6, five FP64 129^3 fields, walls: 154 / 86 / 86 -> 66 / 48 / 49
//   C6, six FP64 2048x1024 fields, walls, x / y: 211 / 120 -> 72 / 68
//   C8 filter, five FP32 256x192x160 fields, walls, x: 130 -> 101
//   C6, six FP64 lines of 5712 points: 18.9 -> 10.8
//
// XM = false (y, z lines): lanes are consecutive x, the window is read straight
// from global memory.  XM = true (x lines): the block's rows are staged by
// cp.async into shared rows of odd pitch, so that both the row-wise copies and
// the threads' walks along their segments are free of bank conflicts.
#pragma once

#include <algorithm>
#include <type_traits>

#include "cles_internal.h"

namespace cles {
namespace {

__device__ __forceinline__ unsigned ln_smem(const void* p) {
    return static_cast<unsigned>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ void ln_cp_async(double* dst, const double* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(ln_smem(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void ln_cp_async(float* dst, const float* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(ln_smem(dst)), "l"(src) : "memory");
}
// release / acquire: both barriers of the kernel order shared-memory accesses
// across blocks
__device__ __forceinline__ void ln_cluster_arrive() { asm volatile("barrier.cluster.arrive.release;" ::: "memory"); }
__device__ __forceinline__ void ln_cluster_wait() { asm volatile("barrier.cluster.wait.acquire;" ::: "memory"); }
// shared-window address of `addr` in block `rank` of the cluster
__device__ __forceinline__ unsigned ln_map(unsigned addr, unsigned rank) {
    unsigned r;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}
__device__ __forceinline__ double ln_remote(unsigned addr, double) {
    double v;
    asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(v) : "r"(addr) : "memory");
    return v;
}
__device__ __forceinline__ float ln_remote(unsigned addr, float) {
    float v;
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(addr) : "memory");
    return v;
}

// The coefficients of one segment kind.  LnConst: kind CLS of the kernel
// parameters, constant operands of the unrolled code.  LnShared: the thread's
// kind in the block's shared copy.
template <typename T, int Q, int MS, int CLS>
struct LnConst {
    const LineCoef<T, Q, MS>& C;
    __device__ __forceinline__ T f(int a, int i) const { return C.f[CLS][a][i]; }
    __device__ __forceinline__ T v(int t, int i) const { return C.v[CLS][t][i]; }
    __device__ __forceinline__ T w(int t, int i) const { return C.w[CLS][t][i]; }
    __device__ __forceinline__ T tl(int e) const { return C.tl[CLS][e]; }
};
template <typename T, int Q, int MS>
struct LnShared {
    const T *pf, *pv, *pw, *pt;
    __device__ __forceinline__ LnShared(const LineCoef<T, Q, MS>& C, int cls)
        : pf(&C.f[cls][0][0]), pv(&C.v[cls][0][0]), pw(&C.w[cls][0][0]), pt(&C.tl[cls][0]) {}
    __device__ __forceinline__ T f(int a, int i) const { return pf[a * MS + i]; }
    __device__ __forceinline__ T v(int t, int i) const { return pv[t * MS + i]; }
    __device__ __forceinline__ T w(int t, int i) const { return pw[t * MS + i]; }
    __device__ __forceinline__ T tl(int e) const { return pt[e]; }
};

// whether group g of four rows holds rows of some segment
template <int MS>
__device__ __forceinline__ bool ln_group(int g, int mm) {
    return 4 * g < MS - 8 || 4 * g < mm;
}

// Local solve of one segment.  Rows past its m points are zero on entry; the
// forward coefficients there copy the last q eliminated values upwards, so the
// tail leaves the loop in a fixed register whatever m is.  The longest segment
// has more than MS - 8 points (the shortest MS - 8 or more): only the last two groups
// of four rows can lie past
// it (mm, rounded up to a group) and are guarded.
template <typename T, int Q, int MS, typename K>
__device__ __forceinline__ void ln_sweep(const K& C, const int mm, T (&y)[MS], T (&tail)[Q]) {
    if constexpr (Q == 1) {
        T carry = y[0];
#pragma unroll
        for (int g = 0; g < MS / 4; ++g) {
            if (ln_group<MS>(g, mm)) {
#pragma unroll
                for (int i = 4 * g; i < 4 * g + 4; ++i)
                    if (i > 0) y[i] -= C.f(0, i) * y[i - 1];
                carry = y[4 * g + 3];
            }
        }
        tail[0] = carry * C.tl(0);
#pragma unroll
        for (int g = MS / 4 - 1; g >= 0; --g) {
            if (ln_group<MS>(g, mm)) {
#pragma unroll
                for (int i = 4 * g + 3; i >= 4 * g; --i) {
                    y[i] *= C.f(1, i);
                    if (i < MS - 1) y[i] -= C.f(2, i) * y[i + 1];
                }
            }
        }
    } else {
        T c0 = y[0], c1 = y[0];
#pragma unroll
        for (int g = 0; g < MS / 4; ++g) {
            if (ln_group<MS>(g, mm)) {
#pragma unroll
                for (int i = 4 * g; i < 4 * g + 4; ++i) {
                    if (i > 1) y[i] -= C.f(1, i - 2) * y[i - 2];
                    if (i > 0) y[i] -= C.f(0, i - 1) * y[i - 1];
                }
                c0 = y[4 * g + 2];
                c1 = y[4 * g + 3];
            }
        }
        // tl: 1/U0 of the last row, U1 / U0 and 1/U0 of the row before it, and
        // whether the copied pair arrives swapped
        const bool sw = C.tl(3) != T(0);
        const T e1 = sw ? c0 : c1, e0 = sw ? c1 : c0;
        tail[Q - 1] = e1 * C.tl(0);
        tail[0] = e0 * C.tl(2) - C.tl(1) * tail[Q - 1];
#pragma unroll
        for (int g = MS / 4 - 1; g >= 0; --g) {
            if (ln_group<MS>(g, mm)) {
#pragma unroll
                for (int i = 4 * g + 3; i >= 4 * g; --i) {
                    y[i] *= C.f(4, i);
                    if (i < MS - 2) y[i] -= C.f(3, i) * y[i + 2];
                    if (i < MS - 1) y[i] -= C.f(2, i) * y[i + 1];
                }
            }
        }
    }
}

template <typename T, int Q, int MS, typename K>
__device__ __forceinline__ void ln_correct(const K& C, const int mm, T (&y)[MS], const T (&zp)[Q],
                                           const T (&zn)[Q]) {
#pragma unroll
    for (int g = 0; g < MS / 4; ++g) {
        if (ln_group<MS>(g, mm)) {
#pragma unroll
            for (int i = 4 * g; i < 4 * g + 4; ++i)
#pragma unroll
                for (int t = 0; t < Q; ++t) y[i] -= C.v(t, i) * zp[t] + C.w(t, i) * zn[t];
        }
    }
}

// Registers a thread: 16 to 24 warps on an SM in FP64, 24 to 32 in FP32.  The FP64
// 24- and 32-point tiles and the FP32 x lines fit; bytes spilled (stores / loads): FP64
// 16-point y / z tiles of C4, C6 and C10 56 / 48, 64 / 72 and 224 / 240 (their x lines up
// to 28 / 44, the filter 12 / 12), FP32 y / z tiles of C10 up to 80 / 72, others 28 / 36.
template <typename T, int M, int MS>
constexpr int ln_regs() {
    return sizeof(T) == 8 ? (MS == 32 ? 128 : MS == 24 ? 104 : M <= 2 ? 80 : 96) : (MS == 32 ? 80 : 64);
}

// Small plans (the short tile) run in a few microseconds, which straight-line
// code over kernel parameters spends on constant-cache misses, one after the
// other: their blocks copy the coefficients and their rows of the reduced
// inverse to shared memory while the points arrive.  Large plans take the
// parameters themselves.
template <int MS>
constexpr bool ln_shared() {
    return MS == 16;
}
template <typename T, int Q, int MS>
using LnParam = typename std::conditional<ln_shared<MS>(), const LineCoef<T, Q, MS>*, LineCoef<T, Q, MS>>::type;

// the coefficients a block uses: its shared copy, or the kernel parameter
template <typename T, int Q, int MS>
__device__ __forceinline__ const LineCoef<T, Q, MS>& ln_coef(const LineCoef<T, Q, MS>* const&, const T* csm) {
    return *reinterpret_cast<const LineCoef<T, Q, MS>*>(csm);
}
template <typename T, int Q, int MS>
__device__ __forceinline__ const LineCoef<T, Q, MS>& ln_coef(const LineCoef<T, Q, MS>& C, const T*) {
    return C;
}

template <typename T>
__device__ __forceinline__ void ln_stage(T* dst, const T* src, int count) {
    for (int i = threadIdx.x; i < count; i += blockDim.x) ln_cp_async(dst + i, src + i);
}

// KEEP: the RK store that also writes dq (RkEpilogue::keep), an instantiation of its
// own: as a run-time branch it added up to 360 bytes of spills to the FP32 forms.
template <typename T, int Q, int M, int MS, bool XM, bool KEEP = false>
__global__ void __maxnreg__((ln_regs<T, M, MS>())) k_line(const __grid_constant__ CompactParams P,
                                                       const __grid_constant__ LnParam<T, Q, MS> C,
                                                       const __grid_constant__ LineArgs A, const T* __restrict__ Gw) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    using Coef = LineCoef<T, Q, MS>;
    constexpr bool CS = ln_shared<MS>();
    const int n = P.n, S = A.S, SC = A.SC, CL = A.CL;
    const int L = 1 << A.logL;
    const int tid = threadIdx.x;
    const int lane = tid & (L - 1);
    const int sl = tid >> A.logL;              // segment within the block
    const int crank = CL > 1 ? (int)(blockIdx.x % CL) : 0;
    const int line0 = (CL > 1 ? (int)(blockIdx.x / CL) : (int)blockIdx.x) * L;
    const int seg0 = crank * SC;               // the block's first segment
    const int seg = seg0 + sl;
    const int comp = blockIdx.y;
    const int line = line0 + lane;
    const bool ok = sl < SC && line < P.lines && seg < S;
    const int base = A.base;
    const int off = seg * base + min(seg, A.rem);
    const int m = base + (seg < A.rem ? 1 : 0);
    const int mm = A.mm;
    const bool periodic = P.periodic != 0;
    const bool second = comp >= A.split;
    const int fc = second ? comp - A.split : comp;
    const T* fin = static_cast<const T*>(second ? A.in2 : A.in.base) + (int64_t)fc * A.in.comp_stride;
    T* fout = static_cast<T*>(second ? A.out2 : A.out.base) + (int64_t)fc * A.out.comp_stride;
    T* tile = reinterpret_cast<T*>(smem_raw);
    T* ht = XM ? tile + (size_t)L * A.pitch : tile;   // [SC][2q][L]
    // shared copies of a small plan: coefficients, inverse rows
    T* csm = ht + (size_t)SC * 2 * Q * L;
    T* gsm = csm + sizeof(Coef) / sizeof(T);
    if constexpr (CS) {
        ln_stage(csm, reinterpret_cast<const T*>(C), (int)(sizeof(Coef) / sizeof(T)));
        if (A.gstage) ln_stage(gsm, Gw, 2 * Q * A.Wn * 2 * Q * S);
    }
    grid_dependency_wait();   // the tables above are constant

    // element offset of point 0 of x line l
    auto line_base = [&](const FieldView& v, int l) -> int64_t {
        if (v.sz == (int64_t)P.ny * v.sy) return (int64_t)l * v.sy;
        return (int64_t)(l % P.ny) * v.sy + (int64_t)(l / P.ny) * v.sz;
    };
    // x rows: points [c0, c1) of the block at row elements M + (g - c0), M
    // points beyond each end around them.  A row belongs to one warp, or to
    // `parts` warps that take runs of 32 k points of it.
    const int c0 = seg0 * base + min(seg0, A.rem);
    const int sE = min(seg0 + SC, S);
    const int len = sE * base + min(sE, A.rem) - c0;
    const int nwarps = blockDim.x >> 5, warp = tid >> 5, wl = tid & 31;
    const int parts = nwarps > L ? nwarps >> A.logL : 1;
    const int r0 = nwarps > L ? warp & (L - 1) : warp, dr = nwarps > L ? L : nwarps;
    const int ppart = nwarps > L ? warp >> A.logL : 0;
    const int run = ((len + parts - 1) / parts + 31) & ~31;
    const int ib = ppart * run, ie = ppart < parts ? min(len, ib + run) : 0;

    T y[MS];
    const bool hi_clo = P.hi_closed && seg == S - 1;
    if (XM) {
        if (len > 0 && ppart < parts) {
            for (int r = r0; r < L && line0 + r < P.lines; r += dr) {
                const T* row = fin + line_base(A.in, line0 + r);
                T* dst = tile + (size_t)r * A.pitch;
                if (ppart == 0 && wl < 2 * M) {
                    int g = wl < M ? c0 - M + wl : c0 + len + wl - M;
                    if (periodic) g = g < 0 ? g + n : (g >= n ? g - n : g);
                    if (g >= 0 && g < n) ln_cp_async(dst + (wl < M ? wl : len + wl), row + g);
                }
                row += c0;
                dst += M;
                int i = ib + wl;
                for (; i + 224 < ie; i += 256)
#pragma unroll
                    for (int k = 0; k < 8; ++k) ln_cp_async(dst + i + 32 * k, row + i + 32 * k);
                for (; i < ie; i += 32) ln_cp_async(dst + i, row + i);
            }
        }
    }
    if (XM) {
        asm volatile("cp.async.wait_all;" ::: "memory");
        __syncthreads();
    }
    const int lo_i = XM ? 0 : (ok ? line % P.nx : 0), lo_o = XM ? 0 : (ok ? line / P.nx : 0);
    const int64_t lb_in = XM ? 0 : lo_i + (int64_t)lo_o * (P.dim == 1 ? A.in.sz : A.in.sy);
    const int64_t st_in = XM ? 1 : (P.dim == 1 ? A.in.sy : A.in.sz);
    const int woff = ok ? off - c0 : 0;   // window element j of this thread: row element woff + j
    const T* trow = tile + (size_t)lane * A.pitch + woff;
    {
        // Window element j is line point off - M + j.  Elements past m + 2M - 1
        // (up to seven: the rounding of mm and of the group of four) are read where
        // they lie, within the line, and masked below.
        T w[MS + 2 * M];
        constexpr int WG = (MS + 2 * M + 3) / 4;
        const int wn = mm + 2 * M;
        if (XM) {
#pragma unroll
            for (int g = 0; g < WG; ++g)
                if (4 * g < MS - 8 + 2 * M || 4 * g < wn) {
#pragma unroll
                    for (int j = 4 * g; j < 4 * g + 4 && j < MS + 2 * M; ++j) w[j] = trow[j];
                }
        } else if (ok) {
            const int stb = (int)st_in * (int)sizeof(T);
            const char* p = reinterpret_cast<const char*>(fin + lb_in + (int64_t)(off - M) * st_in);
            if (off >= M && off - M + ((wn + 3) & ~3) <= n) {
#pragma unroll
                for (int g = 0; g < WG; ++g)
                    if (4 * g < MS - 8 + 2 * M || 4 * g < wn) {
#pragma unroll
                        for (int j = 4 * g; j < 4 * g + 4 && j < MS + 2 * M; ++j)
                            w[j] = *reinterpret_cast<const T*>(p + (int64_t)j * stb);
                    }
            } else {
                const T* fb = fin + lb_in;
#pragma unroll
                for (int g = 0; g < WG; ++g)
                    if (4 * g < MS - 8 + 2 * M || 4 * g < wn) {
#pragma unroll
                        for (int j = 4 * g; j < 4 * g + 4 && j < MS + 2 * M; ++j) {
                            int e = off - M + j;
                            if (periodic) e = e < 0 ? e + n : (e >= n ? e - n : e);
                            else e = e < 0 ? 0 : (e >= n ? n - 1 : e);   // feeds rows that closure rows replace
                            w[j] = fb[(int64_t)e * st_in];
                        }
                    }
            }
        }
        if (CS && !XM) {   // the window's loads are in flight meanwhile
            asm volatile("cp.async.wait_all;" ::: "memory");
            __syncthreads();
        }
        const T a0 = (ln_coef<T, Q, MS>(C, csm)).a0;
        T ci[M];
#pragma unroll
        for (int k = 0; k < M; ++k) ci[k] = (ln_coef<T, Q, MS>(C, csm)).ci[k];
        const bool sym = P.symmetric != 0;
#pragma unroll
        for (int g = 0; g < MS / 4; ++g) {
            if (4 * g >= MS - 8) {
#pragma unroll
                for (int i = 4 * g; i < 4 * g + 4; ++i) y[i] = T(0);
            }
            if (ln_group<MS>(g, mm)) {
                if (sym) {
#pragma unroll
                    for (int i = 4 * g; i < 4 * g + 4; ++i) {
                        T acc = a0 * w[i + M];
#pragma unroll
                        for (int k = 1; k <= M; ++k) acc += ci[k - 1] * (w[i + M + k] + w[i + M - k]);
                        y[i] = acc;
                    }
                } else {
#pragma unroll
                    for (int i = 4 * g; i < 4 * g + 4; ++i) {
                        T acc = T(0);
#pragma unroll
                        for (int k = 1; k <= M; ++k) acc += ci[k - 1] * (w[i + M + k] - w[i + M - k]);
                        y[i] = acc;
                    }
                }
                if (4 * g + 4 > MS - 8 && 4 * g + 4 > base) {   // rows past the segment's end are zero
#pragma unroll
                    for (int i = 4 * g; i < 4 * g + 4; ++i) y[i] = i < m ? y[i] : T(0);
                }
            }
        }
        if (P.lo_closed && seg == 0) {
#pragma unroll
            for (int i = 0; i < kMaxClo; ++i) {
                if (i < P.nc) {
                    T acc = T(0);
#pragma unroll
                    for (int k = 0; k < kMaxCloLen; ++k)
                        if (k < P.clo_len[i] && M + k < MS + 2 * M) acc += (ln_coef<T, Q, MS>(C, csm)).clo[i][k] * w[M + k];
                    y[i] = acc;
                }
            }
        }
    }
    if (hi_clo) {
        T hv[kMaxClo];
#pragma unroll
        for (int jr = 0; jr < kMaxClo; ++jr) {
            T acc = T(0);
            if (jr < P.nc)
#pragma unroll
                for (int k = 0; k < kMaxCloLen; ++k)
                    if (k < P.clo_len[jr] && ok) {
                        const T v = XM ? trow[M + m - 1 - k] : fin[lb_in + (int64_t)(n - 1 - k) * st_in];
                        acc += (ln_coef<T, Q, MS>(C, csm)).chi[jr][k] * v;
                    }
            hv[jr] = acc;
        }
        // the segment has MS - 8 rows or more (see ln_sweep)
#pragma unroll
        for (int i = MS - 8 - kMaxClo; i < MS; ++i)
#pragma unroll
            for (int jr = 0; jr < kMaxClo; ++jr) y[i] = (jr < P.nc && i == m - 1 - jr) ? hv[jr] : y[i];
    }

    // ---- local solve ----
    const int cls = (!periodic && seg == 0) ? 0 : (!periodic && seg == S - 1) ? 3 : (seg < A.rem ? 1 : 2);
    T tail[Q];
    if constexpr (CS) {
        ln_sweep<T, Q, MS>(LnShared<T, Q, MS>((ln_coef<T, Q, MS>(C, csm)), cls), mm, y, tail);
    } else {
        if (cls == 1) ln_sweep<T, Q, MS>(LnConst<T, Q, MS, 1>{C}, mm, y, tail);
        else if (cls == 2) ln_sweep<T, Q, MS>(LnConst<T, Q, MS, 2>{C}, mm, y, tail);
        else if (cls == 0) ln_sweep<T, Q, MS>(LnConst<T, Q, MS, 0>{C}, mm, y, tail);
        else ln_sweep<T, Q, MS>(LnConst<T, Q, MS, 3>{C}, mm, y, tail);
    }

    // ---- interface values ----
    if (sl < SC) {   // the last warp may hold threads past the block's segments
#pragma unroll
        for (int t = 0; t < Q; ++t) {
            ht[(size_t)(sl * 2 * Q + t) * L + lane] = y[t];
            ht[(size_t)(sl * 2 * Q + Q + t) * L + lane] = tail[t];
        }
    }
    if (CL > 1) {
        ln_cluster_arrive();
        ln_cluster_wait();
    } else {
        __syncthreads();
    }
    T zp[Q], zn[Q];
    {
        T ap[Q], an[Q];
#pragma unroll
        for (int t = 0; t < Q; ++t) ap[t] = an[t] = T(0);
        if (ok) {
            const int Wn = A.Wn;
            // this segment's rows (line_row_index)
            const T* g = CS ? (A.gstage ? gsm : Gw) + seg : Gw + (int64_t)seg * (2 * Q) * Wn * (2 * Q);
            const int ge = CS ? S : 1;
            // first segments of the two windows (around seg - 1 and seg + 1)
            int jp = seg - 1 - A.Kr, jn = seg + 1 - A.Kr;
            if (periodic) {
                jp = jp < 0 ? jp + S : jp;
                jp = jp < 0 ? jp + S : jp;
                jn = jn < 0 ? jn + S : (jn >= S ? jn - S : jn);
            } else {
                jp = max(0, min(jp, S - Wn));
                jn = max(0, min(jn, S - Wn));
            }
            if (CL == 1) {
#pragma unroll(CS ? 3 : 1)
                for (int j = 0; j < Wn; ++j) {
#pragma unroll
                    for (int u = 0; u < 2 * Q; ++u) {
                        const T hp = ht[(size_t)(jp * 2 * Q + u) * L + lane];
                        const T hn = ht[(size_t)(jn * 2 * Q + u) * L + lane];
#pragma unroll
                        for (int t = 0; t < Q; ++t) {
                            ap[t] += g[((t * Wn + j) * 2 * Q + u) * ge] * hp;
                            an[t] += g[(((Q + t) * Wn + j) * 2 * Q + u) * ge] * hn;
                        }
                    }
                    jp = jp + 1 == S ? 0 : jp + 1;
                    jn = jn + 1 == S ? 0 : jn + 1;
                }
            } else {
                const unsigned hb = ln_smem(ht) + (unsigned)(lane * sizeof(T));
                const unsigned rowb = (unsigned)(L * sizeof(T));
#pragma unroll(CS ? 3 : 1)
                for (int j = 0; j < Wn; ++j) {
                    const int cp = jp / SC, cn = jn / SC;
                    const unsigned bp = ln_map(hb, cp) + (unsigned)((jp - cp * SC) * 2 * Q) * rowb;
                    const unsigned bn = ln_map(hb, cn) + (unsigned)((jn - cn * SC) * 2 * Q) * rowb;
#pragma unroll
                    for (int u = 0; u < 2 * Q; ++u) {
                        const T hp = ln_remote(bp + u * rowb, T(0));
                        const T hn = ln_remote(bn + u * rowb, T(0));
#pragma unroll
                        for (int t = 0; t < Q; ++t) {
                            ap[t] += g[((t * Wn + j) * 2 * Q + u) * ge] * hp;
                            an[t] += g[(((Q + t) * Wn + j) * 2 * Q + u) * ge] * hn;
                        }
                    }
                    jp = jp + 1 == S ? 0 : jp + 1;
                    jn = jn + 1 == S ? 0 : jn + 1;
                }
            }
        }
#pragma unroll
        for (int t = 0; t < Q; ++t) {
            zp[t] = ap[t];
            zn[t] = an[t];
        }
    }
    // No block leaves while another may still read its end values: the arrival
    // releases this block's remote reads above, the wait at the end of the kernel
    // acquires those of the others.  The correction and the stores come in between.
    if (CL > 1) ln_cluster_arrive();
    if constexpr (CS) {
        ln_correct<T, Q, MS>(LnShared<T, Q, MS>((ln_coef<T, Q, MS>(C, csm)), cls), mm, y, zp, zn);
    } else {
        if (cls == 1) ln_correct<T, Q, MS>(LnConst<T, Q, MS, 1>{C}, mm, y, zp, zn);
        else if (cls == 2) ln_correct<T, Q, MS>(LnConst<T, Q, MS, 2>{C}, mm, y, zp, zn);
        else if (cls == 0) ln_correct<T, Q, MS>(LnConst<T, Q, MS, 0>{C}, mm, y, zp, zn);
        else ln_correct<T, Q, MS>(LnConst<T, Q, MS, 3>{C}, mm, y, zp, zn);
    }

    // ---- store ----
    const int mode = KEEP ? OUT_RK : A.mode;
    const double rdt = mode == OUT_RK ? (A.rk.dtp ? *A.rk.dtp : A.rk.dt) : 0.0;
    if (XM) {
        // every thread has read its window (the barrier above): results go
        // back into the rows, then out in coalesced rows
        if (ok) {
            T* orow = tile + (size_t)lane * A.pitch + woff + M;
#pragma unroll
            for (int g = 0; g < MS / 4; ++g) {
                if (4 * g + 4 <= MS - 8 || 4 * g + 4 <= base) {
#pragma unroll
                    for (int i = 4 * g; i < 4 * g + 4; ++i) orow[i] = y[i];
                } else if (ln_group<MS>(g, mm)) {
#pragma unroll
                    for (int i = 4 * g; i < 4 * g + 4; ++i)
                        if (i < m) orow[i] = y[i];
                }
            }
        }
        __syncthreads();
        if (len > 0 && ppart < parts) {
            for (int r = r0; r < L && line0 + r < P.lines; r += dr) {
                const int64_t rb = line_base(A.out, line0 + r) + c0;
                T* row = fout + rb;
                const T* src = tile + (size_t)r * A.pitch + M;
                int i = ib + wl;
                if (mode == OUT_SUBTRACT) {
                    for (; i < ie; i += 128) {
                        T old[4];
#pragma unroll
                        for (int k = 0; k < 4; ++k)
                            if (i + 32 * k < ie) old[k] = row[i + 32 * k];
#pragma unroll
                        for (int k = 0; k < 4; ++k)
                            if (i + 32 * k < ie) row[i + 32 * k] = old[k] - src[i + 32 * k];
                    }
                } else if (mode == OUT_RK) {
                    double* Qp = A.rk.Q + (int64_t)comp * A.out.comp_stride + rb;
                    double* dp = A.rk.du + (int64_t)comp * A.out.comp_stride + rb;
                    for (; i < ie; i += 128) {
                        T old[4];
                        double dv[4], qv[4];
#pragma unroll
                        for (int k = 0; k < 4; ++k)
                            if (i + 32 * k < ie) {
                                old[k] = A.rk_first ? T(0) : row[i + 32 * k];
                                dv[k] = dp[i + 32 * k];
                                qv[k] = Qp[i + 32 * k];
                            }
#pragma unroll
                        for (int k = 0; k < 4; ++k)
                            if (i + 32 * k < ie) {
                                const T dq = old[k] - src[i + 32 * k];
                                if (KEEP) row[i + 32 * k] = dq;
                                const double v = A.rk.A * dv[k] + rdt * double(dq);
                                dp[i + 32 * k] = v;
                                Qp[i + 32 * k] = qv[k] + A.rk.B * v;
                            }
                    }
                } else {
                    const T sg = mode == OUT_NEGATE ? T(-1) : T(1);
                    for (; i + 224 < ie; i += 256)
#pragma unroll
                        for (int k = 0; k < 8; ++k) row[i + 32 * k] = sg * src[i + 32 * k];
                    for (; i < ie; i += 32) row[i] = sg * src[i];
                }
            }
        }
    } else if (ok) {
        const int64_t st = P.dim == 1 ? A.out.sy : A.out.sz;
        const int stb = (int)st * (int)sizeof(T);
        const int64_t ob = lo_i + (int64_t)lo_o * (P.dim == 1 ? A.out.sz : A.out.sy) + (int64_t)off * st;
        char* o = reinterpret_cast<char*>(fout + ob);
        auto at = [&](int i) -> T& { return *reinterpret_cast<T*>(o + (int64_t)i * stb); };
        if (mode == OUT_SUBTRACT) {
#pragma unroll
            for (int i0 = 0; i0 < MS; i0 += 8) {
                if (i0 >= MS - 8 && i0 >= mm) continue;
                T old[8];
#pragma unroll
                for (int q = 0; q < 8; ++q)
                    if (i0 + q < m) old[q] = at(i0 + q);
#pragma unroll
                for (int q = 0; q < 8; ++q)
                    if (i0 + q < m) at(i0 + q) = old[q] - y[i0 + q];
            }
        } else if (mode == OUT_RK) {
            char* Qp = reinterpret_cast<char*>(A.rk.Q + (int64_t)comp * A.out.comp_stride + ob);
            char* dp = reinterpret_cast<char*>(A.rk.du + (int64_t)comp * A.out.comp_stride + ob);
            const int sd = (int)st * 8;
            auto atd = [&](char* b, int i) -> double& { return *reinterpret_cast<double*>(b + (int64_t)i * sd); };
#pragma unroll
            for (int i0 = 0; i0 < MS; i0 += 4) {
                if (i0 >= MS - 8 && i0 >= mm) continue;
                T old[4];
                double dv[4], qv[4];
#pragma unroll
                for (int q = 0; q < 4; ++q)
                    if (i0 + q < m) {
                        old[q] = A.rk_first ? T(0) : at(i0 + q);
                        dv[q] = atd(dp, i0 + q);
                        qv[q] = atd(Qp, i0 + q);
                    }
#pragma unroll
                for (int q = 0; q < 4; ++q)
                    if (i0 + q < m) {
                        const T dq = old[q] - y[i0 + q];
                        if (KEEP) at(i0 + q) = dq;
                        const double v = A.rk.A * dv[q] + rdt * double(dq);
                        atd(dp, i0 + q) = v;
                        atd(Qp, i0 + q) = qv[q] + A.rk.B * v;
                    }
            }
        } else {
            auto put = [&](auto val) {
#pragma unroll
                for (int g = 0; g < MS / 4; ++g) {
                    if (4 * g + 4 <= MS - 8 || 4 * g + 4 <= base) {
#pragma unroll
                        for (int i = 4 * g; i < 4 * g + 4; ++i) at(i) = val(i);
                    } else if (ln_group<MS>(g, mm)) {
#pragma unroll
                        for (int i = 4 * g; i < 4 * g + 4; ++i)
                            if (i < m) at(i) = val(i);
                    }
                }
            };
            if (mode == OUT_NEGATE) put([&](int i) { return -y[i]; });
            else put([&](int i) { return y[i]; });
        }
    }
    if (CL > 1) ln_cluster_wait();
}

template <typename T, int Q, int M, int MS, bool XM, bool KEEP>
void launch_line_k(const CompactPlan& plan, const FieldView& in, const FieldView& out, int count, int mode,
                   cudaStream_t st, const RkEpilogue& rk, bool rk_first, const void* in2, void* out2, int count2, int num_sms) {
    const CompactParams& P = plan.P;
    const LinePlan& lp = *plan.line;
    const LineShape s = line_shape(P, lp, count + count2, num_sms, sizeof(T));
    LineArgs A;
    A.in = in;
    A.out = out;
    A.in2 = in2;
    A.out2 = out2;
    A.split = count;
    A.S = lp.S;
    A.base = lp.base;
    A.rem = lp.rem;
    A.mm = lp.mm;
    A.Wn = lp.Wn;
    A.Kr = lp.Kr;
    A.SC = s.SC;
    A.CL = s.CL;
    A.logL = 0;
    while ((1 << A.logL) < s.L) ++A.logL;
    A.mode = mode;
    A.rk = {rk.Q, rk.du, rk.A, rk.B, rk.dt, rk.dtp};
    A.rk_first = rk_first ? 1 : 0;
    A.pitch = 0;
    size_t smem = sizeof(T) * (size_t)s.SC * 2 * Q * s.L;
    if (XM) {
        // odd, with room for the masked window elements past the last segment
        A.pitch = (s.SC * (lp.base + (lp.rem ? 1 : 0)) + 2 * M + 8) | 1;
        smem += sizeof(T) * (size_t)s.L * A.pitch;
    }
    A.gstage = 0;
    if (ln_shared<MS>()) {
        smem += sizeof(LineCoef<T, Q, MS>);
        const size_t g = sizeof(T) * (size_t)lp.S * 2 * Q * lp.Wn * 2 * Q;
        if (g <= 16 * 1024) {
            A.gstage = 1;
            smem += g;
        }
    }
    auto kern = k_line<T, Q, M, MS, XM, KEEP>;
    static std::atomic<uint64_t> raised{0};
    raise_smem_limit(kern, smem, raised);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)((P.lines + s.L - 1) / s.L) * s.CL, (unsigned)(count + count2));
    // whole warps for the row copies; threads past SC segments only take part
    // in those and in the barriers
    cfg.blockDim = dim3((unsigned)((s.L * s.SC + 31) / 32 * 32));
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at[2];
    cfg.attrs = at;
    if (s.CL > 1) {
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = (unsigned)s.CL;
        at[0].val.clusterDim.y = 1;
        at[0].val.clusterDim.z = 1;
        cfg.numAttrs = 1;
    }
    if (DependentLaunches::active()) {
        at[cfg.numAttrs].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        at[cfg.numAttrs++].val.programmaticStreamSerializationAllowed = 1;
    }
    const void* tab = lp.tab;
    const void* dcoef = lp.dcoef;
    void* cp = ln_shared<MS>() ? static_cast<void*>(&dcoef) : const_cast<unsigned char*>(lp.coef.data());
    void* args[4] = {const_cast<CompactParams*>(&P), cp, &A, &tab};
    CLES_CUDA(cudaLaunchKernelExC(&cfg, reinterpret_cast<const void*>(kern), args));
    count_launch();
    check_launch("k_line");
}

template <typename T, int Q, int M, int MS, bool XM>
void launch_line_t(const CompactPlan& plan, const FieldView& in, const FieldView& out, int count, int mode,
                   cudaStream_t st, const RkEpilogue& rk, bool rk_first, const void* in2, void* out2, int count2, int num_sms) {
    if (mode == OUT_RK && rk.keep)
        launch_line_k<T, Q, M, MS, XM, true>(plan, in, out, count, mode, st, rk, rk_first, in2, out2, count2, num_sms);
    else
        launch_line_k<T, Q, M, MS, XM, false>(plan, in, out, count, mode, st, rk, rk_first, in2, out2, count2, num_sms);
}

template <typename T, int Q, int M, bool XM>
void launch_line_ms(const CompactPlan& plan, const FieldView& in, const FieldView& out, int count, int mode,
                    cudaStream_t st, const RkEpilogue& rk, bool rk_first, const void* in2, void* out2, int count2, int num_sms) {
    if (plan.line->MS == 16) launch_line_t<T, Q, M, 16, XM>(plan, in, out, count, mode, st, rk, rk_first, in2, out2, count2, num_sms);
    else if (plan.line->MS == 24) launch_line_t<T, Q, M, 24, XM>(plan, in, out, count, mode, st, rk, rk_first, in2, out2, count2, num_sms);
    else launch_line_t<T, Q, M, 32, XM>(plan, in, out, count, mode, st, rk, rk_first, in2, out2, count2, num_sms);
}

template <typename T>
bool launch_line_dtype(const CompactPlan& plan, const FieldView& in, const FieldView& out, int count, int mode,
                       cudaStream_t st, const RkEpilogue& rk, bool rk_first, const void* in2, void* out2, int count2, int num_sms) {
    const CompactParams& P = plan.P;
    auto go = [&](auto q, auto m) {
        constexpr int Q = decltype(q)::value, M = decltype(m)::value;
        if (P.dim == 0) launch_line_ms<T, Q, M, true>(plan, in, out, count, mode, st, rk, rk_first, in2, out2, count2, num_sms);
        else launch_line_ms<T, Q, M, false>(plan, in, out, count, mode, st, rk, rk_first, in2, out2, count2, num_sms);
        return true;
    };
    using I1 = std::integral_constant<int, 1>;
    using I2 = std::integral_constant<int, 2>;
    using I3 = std::integral_constant<int, 3>;
    using I4 = std::integral_constant<int, 4>;
    if (P.q == 1 && P.M == 1) return go(I1{}, I1{});
    if (P.q == 1 && P.M == 2) return go(I1{}, I2{});
    if (P.q == 1 && P.M == 4) return go(I1{}, I4{});
    if (P.q == 2 && P.M == 3) return go(I2{}, I3{});
    return false;
}

}  // namespace
}  // namespace cles
