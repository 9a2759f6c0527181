// The multigrid cycles of poiss_z_ft / poiss_x_ft with a mode's whole problem
// resident in the shared memory of one thread-block cluster.
//
// What bounds a V-cycle of these small 2-D problems is the latency of its
// dependent phases, not bytes or operations.  The cycle of k_mg.cu keeps the
// work arrays in global memory, i fastest: a y line is read one 32-byte sector
// per row, each phase pays an L2 round trip for its loads and another for the
// stores its cluster barrier has to flush, and a defect and a restriction
// pass lie between the relaxations.  Here
//   * every array a phase exchanges is in shared memory, its lines dealt to
//     the blocks of the cluster in pairs (an odd line and the even one above
//     it); a line another block owns is read through distributed shared
//     memory.  A line is stored in the order a warp solves it (rows l R ..
//     l R + R - 1 of lane l, real parts in one half of the warp and imaginary
//     ones in the other), so a warp moves it in contiguous vectors;
//   * a right-hand side is a sum of scaled lines, so the passes between the
//     relaxations disappear.  With no initial guess (oldv = 0) the odd lines
//     solve T g = r exactly, the even ones T g = r - aw g(i-1) - ae g(i+1),
//     so the defect that godown restricts is -(aw g(i-1) + ae g(i+1)) on the
//     odd lines and zero on the even ones: the next level's source is formed
//     from two lines of g where it is used, and neither defect nor restricted
//     residual is stored (poiss_z_ft.f90:438-463; below the top level the
//     post-smoothing solves against that defect, as there).  Prolonged even
//     lines are only read by the odd lines' right-hand sides, so goup's sum
//     folds into them as three scaled coarse lines (:411-435);
//   * the scans of a line solve take their multipliers, products of the LU
//     factors that never change, from a table, and a lane corrects its rows
//     by one multiply-add each instead of running its recurrence again.
//   * a half sweep is one piece of code on a list of tasks, one per line, made
//     once per solve: addresses and weights of the lines to sum, the line
//     written.  A lone warp issues an instruction every few clocks, so at the
//     coarse levels, one or two lines a phase, a phase's time is its
//     instruction count; working the addresses out anew at each phase took
//     two thirds of it.
//   * a warp's solve table for its next line comes in by asynchronous copy
//     while it works on the present one: the tables of a block's lines do
//     not stay in L1 beside its shared memory, and a phase that loads its own
//     waits an L2 round trip, longer than the rest of it.
// A cycle has two barriers per level and direction.  Levels of few lines stay
// on block 0 (block barriers), the larger ones are spread (cluster barriers).
//
// Measured on one GB300, a V-cycle of the slowest mode with k_mg.cu's cycle
// and with this one: 128x96 mixed form 110 and 32 us, 256x192 mixed 410 and
// 68 us, 64x48 FP64 182 and 49 us.  What is left: about 700 clocks a phase in
// FP32 are the two scans of a line solve, 64 clocks an operation of a warp
// are FP64's, and the top level's FP64 residual is bound by that pipe.
#pragma once
#include "k_fft.cuh"
#include <cooperative_groups.h>
#include <type_traits>

namespace lg {

constexpr int kMgMaxLev = 20;
constexpr int kMglMaxPhase = 160;      // half sweeps of a cycle: 4 per level, 2 nbli on level 0

// One level: its lines as pairs, pp pairs per block (solo: all on block 0),
// its first line in a block's store.
struct MgLevel {
    int ibg, n, np, pp, off, solo;
    unsigned inv;               // q / pp = umulhi(q, inv) (pp = 1: inv = 0, the quotient is q)
};

// A mode's solve as the kernel sees it; the tables are per mode unless noted.
struct MgLineArgs {
    int nl, n2m, nld, nlev, nbli, mgitr, xft, prd, cs, bshared;
    int lines;                  // lines of the G store of a block (all levels)
    int top2;                   // top-level lines of a block, 2 pp
    MgLevel lev[kMgMaxLev + 1];
    const double *tab_d, *lc_d, *act, *asl, *anl;   // lc, asl, anl: shared by the modes
    const float *tab_f, *lc_f;
    double2 *ccap;
    double *bt;
    long long *iters;
    DScal *S;
    int ndesc;                  // task descriptors a block may need
    int slot, timing;           // timing: a run of the autotuner (criterion relative to the first residual)
};

constexpr int kLcN = 8;         // line coefficients: aw, ae, s0, s1, w0, w1, w2, unused
// Solve table of a line, entries of one lane of the 16 that hold its rows:
// bet, p = -as bet, g = -gam (R each), the four multipliers of the forward and
// of the backward scan and, on lines short enough for the registers, the
// running products of p and g over the lane's rows.  Stored in 16-byte groups,
// the 16 lanes of a group side by side.
template <int R> constexpr bool mgl_cum() { return R <= 8; }
template <int R> constexpr int mgl_entries() { return (mgl_cum<R>() ? 5 : 3) * R + 8; }
template <int R, class T> constexpr int mgl_groups() { return (mgl_entries<R>() * (int)sizeof(T) + 15) / 16; }
template <int R, class T> constexpr int mgl_tab_len() { return mgl_groups<R, T>() * 16 * (16 / (int)sizeof(T)); }
constexpr int kMglThreads = 256;
// rows per lane of the instance for lines of n2m cells: half a warp holds the
// real parts of a line, the other half the imaginary ones
inline int mgl_r(int n2m) {
    const int m = (n2m + 15) / 16;
    return m <= 4 ? (m < 2 ? 2 : m) : m <= 6 ? 6 : m <= 8 ? 8 : m <= 12 ? 12 : 16;
}
// A line in a block's store: row r of a lane in vectors of W elements, so a
// warp moves a line in R / W conflict-free accesses.
template <int R, class T> constexpr int mgl_w() {
    return sizeof(T) == 4 ? (R % 4 == 0 ? 4 : R % 2 == 0 ? 2 : 1) : (R % 2 == 0 ? 2 : 1);
}
template <int R, class T> LG_HD int mgl_at(int r, int lane) {
    constexpr int W = mgl_w<R, T>();
    return (r / W) * (32 * W) + lane * W + r % W;
}
// the same for one value per row (both halves read it): 16 lanes
template <int R> LG_HD int mgl_row_at(int r, int lane16) {
    constexpr int W = mgl_w<R, double>();
    return (r / W) * (16 * W) + lane16 * W + r % W;
}

// A task of a half sweep: up to five lines of the cluster's shared memory to
// sum with their weights, the line of the solve table, the line to write.
template <class T>
struct alignas(16) MglTask {
    unsigned p[5], out;         // shared-window addresses
    int unused;
    int info;                   // terms | own line l - 2 q0 of the top level << 8 | shift task << 31
    T s[5], sk;                 // weights; the pinned value's
    const T *tab;               // the line's solve table
};
template <class T> constexpr size_t mgl_task_bytes() { return sizeof(MglTask<T>); }
// a block's copies of the warps' next solve tables, and of as, an
template <int R, class T> constexpr int mgl_stage_bytes() { return mgl_groups<R, T>() * 256; }
inline size_t mgl_fixed_bytes(int r, bool mixed) {
    const int e = (r <= 8 ? 5 : 3) * r + 8, groups = (e * (mixed ? 4 : 8) + 15) / 16;
    return (size_t)groups * 256 * (kMglThreads / 32) + 2 * (size_t)r * 16 * sizeof(double);
}

typedef void (*MglKernel)(const MgLineArgs *, int);
MglKernel mgl_kernel_mixed(int r);
MglKernel mgl_kernel_fp64(int r);

// ------------------------------------------------------------- device side
// The phases of a cycle.
enum MglKind {
    MGL_DOWN_ODD, MGL_DOWN_EVEN,        // relax(ilev, 0, 1) of the way down
    MGL_UP_ODD, MGL_UP_EVEN,            // goup onto the level, relax(ilev, 1, 1)
    MGL_SRC0, MGL_C_FIRST, MGL_C_ODD, MGL_C_EVEN,   // level 0: its source, relax(0, 0, nbli)
    MGL_COARSE,                         // the same in one phase, a warp per line
    MGL_TOP_FIRST, MGL_TOP_ODD, MGL_TOP_EVEN,       // toplevel
    MGL_IDLE                            // a barrier only
};
__device__ __forceinline__ bool mgl_even(int kind) {
    return kind == MGL_DOWN_EVEN || kind == MGL_UP_EVEN || kind == MGL_C_EVEN || kind == MGL_TOP_EVEN;
}
// What a phase waits for before it reads what the previous one wrote.  The
// cluster barrier is split: a phase announces its arrival, loads what does
// not depend on the others (its task, the solve table) and waits only then.
enum MglSync { MGL_NONE = 0, MGL_BLOCK = 1, MGL_CLUSTER = 2 };
__device__ __forceinline__ void mgl_arrive(int s) {
    if (s == MGL_CLUSTER) cooperative_groups::this_cluster().barrier_arrive();
}
__device__ __forceinline__ void mgl_wait(int s) {
    if (s == MGL_CLUSTER) cooperative_groups::this_cluster().barrier_wait();
    else if (s == MGL_BLOCK) __syncthreads();
}
// A phase of the schedule: its tasks and what they do.
constexpr int kMglInit = 1;     // the first term is taken as it is
constexpr int kMglB = 2;        // the sum starts from the right-hand side
constexpr int kMglSolve = 4, kMglStore = 8, kMglPut = 16, kMglPin = 32, kMglCoarse = 64;
struct alignas(16) MglPhase { int first, n, flags, sync; };

// what the threads of a block share about their mode
struct MglCtx {
    MgLineArgs a;
    int kv, rank, nph;
    unsigned long long test2;   // bits of the least squared norm that is not below the criterion
    double *x, *b;              // iterate and right-hand side of the own top lines
    unsigned char *g;           // lines of every level: corrections; the top's also the residual
    unsigned char *r0, *zero;   // source of level 0; a line of zeros
    unsigned char *task;
    double *rows;               // as, then an, in the rows' order
    unsigned stage;             // shared-window address of the table copies
    unsigned pin;               // address of the zero wavenumber's pin (of its real part)
    unsigned long long slot[2][16];     // max squared norms of the cluster's blocks (bits)
    MglPhase ph[kMglMaxPhase];
};

// neighbours of line l, -1 outside the level
__device__ __forceinline__ int mgl_im(const MglCtx &c, const MgLevel &L, int l) { return l > 0 ? l - 1 : c.a.prd ? L.n - 1 : -1; }
__device__ __forceinline__ int mgl_ip(const MglCtx &c, const MgLevel &L, int l) { return l + 1 < L.n ? l + 1 : c.a.prd ? 0 : -1; }
// the address of line l of a level as a task holds it: in the shared window
// of the cluster (an own line: the block's own window, part of it)
template <int R, class T>
__device__ __forceinline__ unsigned mgl_addr(const MglCtx &c, T *area, const MgLevel &L, int l) {
    const int q = l >> 1;
    const int own = L.inv ? (int)__umulhi((unsigned)q, L.inv) : q;
    const int home = L.solo ? 0 : own;
    const unsigned at = (unsigned)__cvta_generic_to_shared(area + (L.off + (q - own * L.pp) * 2 + (l & 1)) * (R * 32));
    if (home == c.rank) return at;
    unsigned r;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(at), "r"(home));
    return r;
}

// a warp's line at a shared-window address, R rows a lane
template <int R>
__device__ __forceinline__ void mgl_ld(float (&v)[R], unsigned at, int lane) {
    constexpr int W = mgl_w<R, float>();
    at += lane * W * 4;
#pragma unroll
    for (int r = 0; r < R; r += W) {
        const unsigned q = at + (r / W) * (32 * W * 4);
        if constexpr (W == 4)
            asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v[r]), "=f"(v[r + 1]), "=f"(v[r + 2]), "=f"(v[r + 3]) : "r"(q) : "memory");
        else if constexpr (W == 2)
            asm volatile("ld.shared::cluster.v2.f32 {%0, %1}, [%2];" : "=f"(v[r]), "=f"(v[r + 1]) : "r"(q) : "memory");
        else
            asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v[r]) : "r"(q) : "memory");
    }
}
template <int R>
__device__ __forceinline__ void mgl_ld(double (&v)[R], unsigned at, int lane) {
    constexpr int W = mgl_w<R, double>();
    at += lane * W * 8;
#pragma unroll
    for (int r = 0; r < R; r += W) {
        const unsigned q = at + (r / W) * (32 * W * 8);
        if constexpr (W == 2)
            asm volatile("ld.shared::cluster.v2.f64 {%0, %1}, [%2];" : "=d"(v[r]), "=d"(v[r + 1]) : "r"(q) : "memory");
        else
            asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(v[r]) : "r"(q) : "memory");
    }
}
// own lines are written through the block's window
template <int R>
__device__ __forceinline__ void mgl_st(const float (&v)[R], unsigned at, int lane) {
    constexpr int W = mgl_w<R, float>();
    at += lane * W * 4;
#pragma unroll
    for (int r = 0; r < R; r += W) {
        const unsigned q = at + (r / W) * (32 * W * 4);
        if constexpr (W == 4)
            asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};" :: "r"(q), "f"(v[r]), "f"(v[r + 1]), "f"(v[r + 2]), "f"(v[r + 3]) : "memory");
        else if constexpr (W == 2)
            asm volatile("st.shared.v2.f32 [%0], {%1, %2};" :: "r"(q), "f"(v[r]), "f"(v[r + 1]) : "memory");
        else
            asm volatile("st.shared.f32 [%0], %1;" :: "r"(q), "f"(v[r]) : "memory");
    }
}
template <int R>
__device__ __forceinline__ void mgl_st(const double (&v)[R], unsigned at, int lane) {
    constexpr int W = mgl_w<R, double>();
    at += lane * W * 8;
#pragma unroll
    for (int r = 0; r < R; r += W) {
        const unsigned q = at + (r / W) * (32 * W * 8);
        if constexpr (W == 2)
            asm volatile("st.shared.v2.f64 [%0], {%1, %2};" :: "r"(q), "d"(v[r]), "d"(v[r + 1]) : "memory");
        else
            asm volatile("st.shared.f64 [%0], %1;" :: "r"(q), "d"(v[r]) : "memory");
    }
}

// the FP32 <-> FP64 conversions of the defect correction on the bit patterns
// (exact; to nearest even; below the least normal float: zero): a conversion
// instruction takes the FP64 pipe, which is what bounds these phases
__device__ __forceinline__ double mgl_widen(float f) {
    const unsigned b = __float_as_uint(f), e = b & 0x7f800000u;
    const unsigned hi = ((b & 0x7fffffffu) >> 3) + (e == 0x7f800000u ? 0x70000000u : 0x38000000u);
    return __hiloint2double((int)((b & 0x80000000u) | (e ? hi : 0u)), (int)(e ? b << 29 : 0u));
}
__device__ __forceinline__ float mgl_narrow(double d) {
    const unsigned hi = (unsigned)__double2hiint(d), lo = (unsigned)__double2loint(d), h = hi & 0x7fffffffu;
    const unsigned t = ((h - 0x38000000u) << 3) | (lo >> 29), rem = lo & 0x1fffffffu;
    unsigned r = t + (rem > 0x10000000u || (rem == 0x10000000u && (t & 1u)) ? 1u : 0u);
    if (h < 0x38100000u) r = 0u;
    if (h >= 0x47f00000u) r = h > 0x7ff00000u || (h == 0x7ff00000u && lo) ? 0x7fffffffu : 0x7f800000u;
    return __uint_as_float(r | (hi & 0x80000000u));
}
template <class T> __device__ __forceinline__ T mgl_to(double d);
template <> __device__ __forceinline__ double mgl_to<double>(double d) { return d; }
template <> __device__ __forceinline__ float mgl_to<float>(double d) { return mgl_narrow(d); }
__device__ __forceinline__ double mgl_from(double d) { return d; }
__device__ __forceinline__ double mgl_from(float f) { return mgl_widen(f); }

template <class T> __device__ __forceinline__ const T *mgl_tab(const MgLineArgs &a);
template <> __device__ __forceinline__ const double *mgl_tab<double>(const MgLineArgs &a) { return a.tab_d; }
template <> __device__ __forceinline__ const float *mgl_tab<float>(const MgLineArgs &a) { return a.tab_f; }
template <class T> __device__ __forceinline__ const T *mgl_lc(const MgLineArgs &a);
template <> __device__ __forceinline__ const double *mgl_lc<double>(const MgLineArgs &a) { return a.lc_d; }
template <> __device__ __forceinline__ const float *mgl_lc<float>(const MgLineArgs &a) { return a.lc_f; }

// the solve table of a line: entry e of bet, p, g, forward, backward, products
template <int R, class T>
struct MglOp {
    static constexpr int N = mgl_groups<R, T>(), W = 16 / (int)sizeof(T);
    T e[N * W];
    __device__ __forceinline__ void load(unsigned stage, int lane) {
        asm volatile("cp.async.wait_all;" ::: "memory");
        __syncwarp();
        stage += (lane & 15) * 16;
#pragma unroll
        for (int r = 0; r < N; r++) {
            if constexpr (W == 4)
                asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(e[W * r]), "=f"(e[W * r + 1]), "=f"(e[W * r + 2]), "=f"(e[W * r + 3]) : "r"(stage + r * 256) : "memory");
            else
                asm volatile("ld.shared.v2.f64 {%0, %1}, [%2];" : "=d"(e[W * r]), "=d"(e[W * r + 1]) : "r"(stage + r * 256) : "memory");
        }
        __syncwarp();
    }
    // straight from global memory
    __device__ __forceinline__ void fetch(const T *tab, int lane) {
        using Q = typename std::conditional<sizeof(T) == 4, float4, double2>::type;
        const Q *q = reinterpret_cast<const Q *>(tab) + (lane & 15);
#pragma unroll
        for (int r = 0; r < N; r++) {
            const Q x = __ldg(q + r * 16);
            e[W * r] = x.x;
            e[W * r + 1] = x.y;
            if constexpr (W == 4) { e[W * r + 2] = x.z; e[W * r + 3] = x.w; }
        }
    }
    __device__ __forceinline__ T bt(int r) const { return e[r]; }
    __device__ __forceinline__ T p(int r) const { return e[R + r]; }
    __device__ __forceinline__ T g(int r) const { return e[2 * R + r]; }
    __device__ __forceinline__ T fa(int s) const { return e[3 * R + s]; }
    __device__ __forceinline__ T ba(int s) const { return e[3 * R + 4 + s]; }
    __device__ __forceinline__ T cp(int r) const { return e[3 * R + 8 + r]; }
    __device__ __forceinline__ T cg(int r) const { return e[4 * R + 8 + r]; }
};

// One line's table from its LU factors: rows sj apart in bet and gam, as
// 1-based; by the 16 lanes of `half`, formed in FP64.
template <int R, class T>
__device__ void mgl_table(const double *as, const double *bet, const double *gam, int sj, int n2m, int lane, unsigned half, T *tab) {
    constexpr int W = 16 / (int)sizeof(T);
    auto put = [&](int e, double v) { tab[(e / W) * (16 * W) + lane * W + e % W] = (T)v; };
    double P = 1.0, G = 1.0;
    for (int q = 0; q < R; q++) {
        const int j = lane * R + q, jb = lane * R + R - 1 - q;      // 0-based rows
        const double b = j < n2m ? bet[(size_t)sj * j] : 0.0;
        const double p = j < n2m ? -as[j + 1] * b : 0.0;
        const double g = jb + 1 < n2m ? -gam[(size_t)sj * (jb + 1)] : 0.0;
        P *= p;
        G *= g;
        put(q, b);
        put(R + q, p);
        put(2 * R + R - 1 - q, g);
        if (mgl_cum<R>()) {
            put(3 * R + 8 + q, P);
            put(4 * R + 8 + R - 1 - q, G);
        }
    }
    for (int s = 0; s < 4; s++) {
        const int d = 1 << s;
        put(3 * R + s, lane >= d ? P : 0.0);
        put(3 * R + 4 + s, lane + d < 16 ? G : 0.0);
        const double Po = __shfl_up_sync(half, P, d, 16), Go = __shfl_down_sync(half, G, d, 16);
        if (lane >= d) P *= Po;
        if (lane + d < 16) G *= Go;
    }
}

// start the copy of a line's table into the warp's stage
template <int R, class T>
__device__ __forceinline__ void mgl_fetch(const T *tab, unsigned stage, int lane) {
    constexpr int n = mgl_groups<R, T>() * 16;
    const unsigned char *src = reinterpret_cast<const unsigned char *>(tab) + lane * 16;
    stage += lane * 16;
#pragma unroll
    for (int k = 0; k < n; k += 32)
        if (n % 32 == 0 || k + lane < n)
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" :: "r"(stage + k * 16), "l"(src + k * 16) : "memory");
}

// trdiag1m (poiss_z_ft.f90:383-408) of the two real lines a warp holds, lane l
// of a half with rows l R .. l R + R - 1.  Each lane solves its rows with a
// zero incoming value, the lanes' last (first) values are joined by a shuffle
// scan over the half, and the incoming value is added with the product of the
// rows' multipliers.  Rows past n2m and lanes a scan step does not reach have
// zero table entries.
template <int R, class T>
__device__ __forceinline__ void mgl_solve(T (&v)[R], const MglOp<R, T> &o, int lane) {
    v[0] *= o.bt(0);
#pragma unroll
    for (int r = 1; r < R; r++) v[r] = o.p(r) * v[r - 1] + v[r] * o.bt(r);
    T B = v[R - 1];
#pragma unroll
    for (int s = 0; s < 4; s++) B += o.fa(s) * __shfl_up_sync(0xffffffffu, B, 1 << s, 16);
    T y = __shfl_up_sync(0xffffffffu, B, 1, 16);
    if ((lane & 15) == 0) y = T(0.0);
    if constexpr (mgl_cum<R>()) {
#pragma unroll
        for (int r = 0; r < R; r++) v[r] += o.cp(r) * y;
    } else {
        T m = o.p(0);
#pragma unroll
        for (int r = 0; r < R; r++) {
            v[r] += m * y;
            if (r + 1 < R) m *= o.p(r + 1);
        }
    }
#pragma unroll
    for (int r = R - 2; r >= 0; r--) v[r] += o.g(r) * v[r + 1];
    T D = v[0];
#pragma unroll
    for (int s = 0; s < 4; s++) D += o.ba(s) * __shfl_down_sync(0xffffffffu, D, 1 << s, 16);
    T x = __shfl_down_sync(0xffffffffu, D, 1, 16);
    if ((lane & 15) == 15) x = T(0.0);
    if constexpr (mgl_cum<R>()) {
#pragma unroll
        for (int r = 0; r < R; r++) v[r] += o.cg(r) * x;
    } else {
        T m = o.g(R - 1);
#pragma unroll
        for (int r = R - 1; r >= 0; r--) {
            v[r] += m * x;
            if (r > 0) m *= o.g(r - 1);
        }
    }
}

// own pairs of a level: [q0, q1)
__device__ __forceinline__ void mgl_own(const MglCtx &c, const MgLevel &L, int &q0, int &q1) {
    q0 = L.solo ? (c.rank == 0 ? 0 : L.np) : min(L.np, c.rank * L.pp);
    q1 = L.solo ? L.np : min(L.np, q0 + L.pp);
}

// tasks of a phase on this block
__device__ __forceinline__ int mgl_ntask(const MglCtx &c, int kind, int ilev) {
    if (kind == MGL_IDLE) return 0;
    const MgLevel &L = c.a.lev[ilev];
    int q0, q1;
    mgl_own(c, L, q0, q1);
    if (kind == MGL_SRC0 || kind == MGL_COARSE) return L.n;
    if (ilev == 0) return mgl_even(kind) ? L.n / 2 : (L.n + 1) / 2;
    return kind == MGL_TOP_EVEN && c.kv == 1 ? 2 * (q1 - q0) : q1 - q0;
}

// Task t of a phase.  The zero wavenumber's pin adds tasks to the top level's
// even phase: poiss_z_ft.f90:301-381 shifts the odd lines by g(1, n2m - 1)
// after the even ones have been formed from the shifted values (a periodic
// wrap shifts twice, as there), poiss_x_ft.f90:328-335 by g(1, n2m) before.
template <int R, class T>
__device__ void mgl_make_task(const MglCtx &c, int kind, int ilev, int t, MglTask<T> &d) {
    constexpr bool kMixed = sizeof(T) == 4;
    const MgLineArgs &a = c.a;
    const MgLevel &L = a.lev[ilev];
    T *g = reinterpret_cast<T *>(c.g);
    int q0, q1;
    mgl_own(c, L, q0, q1);
    const bool shift = kind == MGL_TOP_EVEN && t >= q1 - q0;
    const bool all = kind == MGL_SRC0 || kind == MGL_COARSE;
    const int q = all ? t >> 1 : q0 + (shift ? t - (q1 - q0) : t);
    const int l = all ? t : 2 * q + (mgl_even(kind) && !shift ? 1 : 0);
    const T *lc = mgl_lc<T>(a) + (size_t)(L.ibg - 1 + l) * kLcN;
    const int im = mgl_im(c, L, l), ip = mgl_ip(c, L, l);
    const unsigned line = mgl_addr<R, T>(c, g, L, l);
    const unsigned r0 = (unsigned)__cvta_generic_to_shared(reinterpret_cast<T *>(c.r0) + l * (R * 32));
    int n = 0;
    auto term = [&](unsigned p, T s) { d.p[n] = p; d.s[n] = s; n++; };
    // a line outside the level, or one of weight zero, adds nothing
    auto maybe = [&](T *area, const MgLevel &M, int i, T s) { if (i >= 0 && s != T(0.0)) term(mgl_addr<R, T>(c, area, M, i), s); };
    d.out = kind == MGL_SRC0 ? r0 : line;
    d.tab = mgl_tab<T>(a) + ((size_t)a.nld * (c.kv - 1) + (size_t)(L.ibg - 1 + l)) * mgl_tab_len<R, T>();
    d.sk = lc[0] + (!a.xft && ip >= 0 && ip < l ? T(2.0) * lc[1] : lc[1]);
    if (kind == MGL_COARSE) {
        // the source's two lines, then the neighbours, zero lines standing in
        const MgLevel &F = a.lev[1];
        const unsigned zero = (unsigned)__cvta_generic_to_shared(c.zero);
        const int f0 = a.nlev == 1 ? 2 * l : mgl_im(c, F, 2 * l);
        term(f0 < 0 ? zero : mgl_addr<R, T>(c, g, F, f0), f0 < 0 ? T(0.0) : lc[2]);
        term(mgl_addr<R, T>(c, g, F, 2 * l + 1), lc[3]);
        term(im < 0 ? zero : mgl_addr<R, T>(c, g, L, im), im < 0 ? T(0.0) : -lc[0]);
        term(ip < 0 ? zero : mgl_addr<R, T>(c, g, L, ip), ip < 0 ? T(0.0) : -lc[1]);
    } else if (kind <= MGL_DOWN_EVEN || kind == MGL_SRC0) {
        // the source: the restricted top residual, or the finer level's
        // defect, from its even lines
        const MgLevel &F = a.lev[ilev + 1];
        maybe(g, F, ilev == a.nlev - 1 ? 2 * l : mgl_im(c, F, 2 * l), lc[2]);
        maybe(g, F, 2 * l + 1, lc[3]);
    } else if (kind == MGL_C_FIRST || kind == MGL_C_ODD || kind == MGL_C_EVEN) {
        term(r0, T(1.0));
    } else if (ilev == a.nlev && (kMixed || shift)) {
        term(line, T(1.0));             // the residual the line itself holds; a shift's solution
    }
    if (kind == MGL_UP_ODD || kind == MGL_TOP_ODD) {
        // prolonged even neighbours.  On the way up the source is the defect
        // kept from the way down, -(aw g(i-1) + ae g(i+1)): the even lines
        // count twice
        const MgLevel &Cl = a.lev[ilev - 1];
        maybe(g, Cl, mgl_im(c, Cl, q), lc[4]);
        maybe(g, Cl, q, lc[5]);
        maybe(g, Cl, mgl_ip(c, Cl, q), lc[6]);
        if (kind == MGL_UP_ODD) {
            maybe(g, L, im, T(-2.0) * lc[0]);
            maybe(g, L, ip, T(-2.0) * lc[1]);
        } else if constexpr (!kMixed) {
            maybe(c.x, L, im, -lc[0]);
            maybe(c.x, L, ip, -lc[1]);
        }
    } else if (kind != MGL_COARSE && (mgl_even(kind) ? !shift : kind == MGL_C_ODD)) {
        maybe(g, L, im, -lc[0]);
        maybe(g, L, ip, -lc[1]);
    }
    // the unused terms add a line of zeros
    for (int k = n; k < 5; k++) { d.p[k] = (unsigned)__cvta_generic_to_shared(c.zero); d.s[k] = T(0.0); }
    d.info = n | ((l - 2 * q0) << 8) | (shift ? (int)0x80000000 : 0);
}

// a task in registers
template <class T>
struct MglRegs {
    unsigned p[5], out;
    int info;
    T s[5], sk;
    const T *tab;
    __device__ __forceinline__ void read(const MglTask<T> &d) {
        const uint4 d0 = reinterpret_cast<const uint4 *>(&d)[0], d1 = reinterpret_cast<const uint4 *>(&d)[1];
        p[0] = d0.x; p[1] = d0.y; p[2] = d0.z; p[3] = d0.w;
        p[4] = d1.x; out = d1.y; info = (int)d1.w;
        if constexpr (sizeof(T) == 4) {
            const float4 a = reinterpret_cast<const float4 *>(&d)[2];
            const float2 b = reinterpret_cast<const float2 *>(&d)[6];
            s[0] = a.x; s[1] = a.y; s[2] = a.z; s[3] = a.w;
            s[4] = b.x; sk = b.y;
        } else {
            const double2 a = reinterpret_cast<const double2 *>(&d)[2], b = reinterpret_cast<const double2 *>(&d)[3],
                          e = reinterpret_cast<const double2 *>(&d)[4];
            s[0] = a.x; s[1] = a.y; s[2] = b.x; s[3] = b.y;
            s[4] = e.x; sk = e.y;
        }
        tab = d.tab;
    }
};

// A task below the top level: sum, solve, store.  A sum has at most two
// terms or at most five; FP32 sums take their zero terms along, which costs
// less than a branch per term, FP64 ones (64 clocks an operation of a warp)
// leave them out.
template <int R, class T>
__device__ __forceinline__ void mgl_line_task(const MglRegs<T> &d, const MglOp<R, T> &o, int lane) {
    constexpr bool kMixed = sizeof(T) == 4;
    constexpr int B = R <= (kMixed ? 6 : 4) ? 3 : 1;
    const int n = d.info & 255;
    T v[R], w0[R], w1[R];
    mgl_ld<R>(w0, d.p[0], lane);
    mgl_ld<R>(w1, d.p[1], lane);
    if (n > 2) {
        T w[B][R];
#pragma unroll
        for (int k = 0; k < B; k++) mgl_ld<R>(w[k], d.p[2 + k], lane);
#pragma unroll
        for (int r = 0; r < R; r++) v[r] = d.s[0] * w0[r] + d.s[1] * w1[r];
#pragma unroll
        for (int k = 0; k < 3; k++) {
            if (kMixed || k + 2 < n) {
#pragma unroll
                for (int r = 0; r < R; r++) v[r] += d.s[2 + k] * w[k % B][r];
            }
            if (k + B < 3) mgl_ld<R>(w[k % B], d.p[2 + (k + B < 3 ? k + B : 2)], lane);
        }
    } else {
#pragma unroll
        for (int r = 0; r < R; r++) v[r] = d.s[0] * w0[r];
        if (kMixed || n > 1) {
#pragma unroll
            for (int r = 0; r < R; r++) v[r] += d.s[1] * w1[r];
        }
    }
    mgl_solve<R, T>(v, o, lane);
    mgl_st<R>(v, d.out, lane);
}

// A task of a half sweep.  The top level's give the FP64 form's new iterate,
// or the mixed form's FP32 correction, which is added to the FP64 iterate.
template <int R, class T>
__device__ __forceinline__ void mgl_work(const MglCtx &c, const MglRegs<T> &d, const MglOp<R, T> &o, int flags, T tt, int lane) {
    constexpr bool kMixed = sizeof(T) == 4;
    constexpr int LS = R * 32;
    const int n = d.info & 255, l = (d.info >> 8) & 0x7fffff;
    const bool shift = d.info < 0;
    // the lines to sum: all in flight together where the registers hold
    // them, else two at a time
    constexpr int B = R <= (kMixed ? 6 : 3) ? 5 : 2;
    T v[R], w[B][R];
#pragma unroll
    for (int k = 0; k < B; k++)
        if (k < n) mgl_ld<R>(w[k], d.p[k], lane);
    int k0 = 0;
    if (!kMixed && (flags & kMglB) && !shift) {
        const double *b = c.b + l * LS;
#pragma unroll
        for (int r = 0; r < R; r++) v[r] = b[mgl_at<R, double>(r, lane)];
    } else if ((flags & kMglInit) || shift) {
        k0 = 1;
    } else {
#pragma unroll
        for (int r = 0; r < R; r++) v[r] = T(0.0);
    }
#pragma unroll
    for (int k = 0; k < 5; k++)
        if (k < n) {
            if (k == 0 && k0 == 1) {
#pragma unroll
                for (int r = 0; r < R; r++) v[r] = w[0][r];
            } else {
#pragma unroll
                for (int r = 0; r < R; r++) v[r] += d.s[k] * w[k % B][r];
            }
            if (k + B < 5 && k + B < n) mgl_ld<R>(w[k % B], d.p[k + B < 5 ? k + B : 4], lane);
        }
    if (!shift) {
        if (flags & kMglPin) {
#pragma unroll
            for (int r = 0; r < R; r++) v[r] += d.sk * tt;
        }
        if (flags & kMglSolve) mgl_solve<R, T>(v, o, lane);
        if (flags & kMglStore) mgl_st<R>(v, d.out, lane);
    }
    if (flags & kMglPut) {              // the iterate, less a pinned odd line's shift
        double *x = c.x + l * LS;
        if (shift) {
#pragma unroll
            for (int r = 0; r < R; r++) v[r] = (lane & 15) * R + r < c.a.n2m ? v[r] - tt : T(0.0);
        }
#pragma unroll
        for (int r = 0; r < R; r++) {
            double &xr = x[mgl_at<R, double>(r, lane)];
            if constexpr (kMixed) xr += mgl_from(v[r]);
            else xr = v[r];
        }
    }
}

// Level 0 in one phase: the source of the warp's line (l = warp) and the nbli
// zebra sweeps, the line's source, table and neighbours kept in registers.
template <int R, class T>
__device__ __forceinline__ void mgl_coarse(const MglRegs<T> &d, const MglOp<R, T> &o, bool have, int warp, int nsweep, int lane) {
    T src[R];
    if (have) {
        T w0[R], w1[R];
        mgl_ld<R>(w0, d.p[0], lane);
        mgl_ld<R>(w1, d.p[1], lane);
#pragma unroll
        for (int r = 0; r < R; r++) src[r] = d.s[0] * w0[r] + d.s[1] * w1[r];
    }
    for (int it = 0; it < nsweep; it++) {
        if (have && ((warp ^ it) & 1) == 0) {
            T v[R];
#pragma unroll
            for (int r = 0; r < R; r++) v[r] = src[r];
            if (it > 0) {
                T w0[R], w1[R];
                mgl_ld<R>(w0, d.p[2], lane);
                mgl_ld<R>(w1, d.p[3], lane);
#pragma unroll
                for (int r = 0; r < R; r++) v[r] += d.s[2] * w0[r] + d.s[3] * w1[r];
            }
            mgl_solve<R, T>(v, o, lane);
            mgl_st<R>(v, d.out, lane);
        }
        if (it + 1 < nsweep) __syncthreads();
    }
}

__device__ __forceinline__ unsigned long long mgl_warp_max(unsigned long long v) {
    const unsigned hi = __reduce_max_sync(0xffffffffu, (unsigned)(v >> 32));
    const unsigned lo = __reduce_max_sync(0xffffffffu, (unsigned)(v >> 32) == hi ? (unsigned)v : 0u);
    return (unsigned long long)hi << 32 | lo;
}

// Residual b - A x of the own top lines in FP64 -> the top level's lines of
// the G store; the max squared norm over the cluster (its bits).
template <int R, class T>
__device__ __forceinline__ unsigned long long mgl_resid(MglCtx &c, int par, int sync) {
    mgl_arrive(sync);
    constexpr int LS = R * 32;
    __shared__ unsigned long long sh[16];
    const MgLineArgs &a = c.a;
    const MgLevel &L = a.lev[a.nlev];
    T *g = reinterpret_cast<T *>(c.g);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    int q0, q1;
    mgl_own(c, L, q0, q1);
    // squared norms are not negative: their bit patterns order as integers,
    // which keeps the comparisons off the FP64 pipe; a NaN is passed over, as
    // fmax does
    constexpr unsigned long long kInf = 0x7ff0000000000000ULL;
    unsigned long long mx = 0ULL;
    double dg[R];                       // diagonal of the warp's next line
    auto diag = [&](int l) {
        const double *ac = a.act + ((size_t)a.nl * (c.kv - 1) + l) * (R * 16);
#pragma unroll
        for (int r = 0; r < R; r++) dg[r] = __ldg(ac + mgl_row_at<R>(r, lane & 15));
    };
    if (2 * q0 + warp < 2 * q1) diag(2 * q0 + warp);
    mgl_wait(sync);
    for (int l = 2 * q0 + warp; l < 2 * q1; l += nw) {
        const double *lcd = a.lc_d + (size_t)l * kLcN;
        const double aw = __ldg(lcd), ae = __ldg(lcd + 1);
        const double *bl = c.b + (l - 2 * q0) * LS;
        const int im = mgl_im(c, L, l), ip = mgl_ip(c, L, l);
        const unsigned zero = (unsigned)__cvta_generic_to_shared(c.zero);
        double x[R], d[R], m[R], p[R];
        mgl_ld<R>(x, mgl_addr<R, double>(c, c.x, L, l), lane);
        mgl_ld<R>(m, im < 0 ? zero : mgl_addr<R, double>(c, c.x, L, im), lane);
        mgl_ld<R>(p, ip < 0 ? zero : mgl_addr<R, double>(c, c.x, L, ip), lane);
        double lo = __shfl_up_sync(0xffffffffu, x[R - 1], 1, 16), hi = __shfl_down_sync(0xffffffffu, x[0], 1, 16);
        if ((lane & 15) == 0) lo = 0.0;
        if ((lane & 15) == 15) hi = 0.0;
#pragma unroll
        for (int r = 0; r < R; r++) {
            const int t = mgl_row_at<R>(r, lane & 15);
            double e = bl[mgl_at<R, double>(r, lane)];
            e -= aw * m[r];
            e -= ae * p[r];
            e -= c.rows[t] * (r > 0 ? x[r - 1] : lo);
            e -= c.rows[R * 16 + t] * (r + 1 < R ? x[r + 1] : hi);
            d[r] = e - dg[r] * x[r];
        }
        if (l + nw < 2 * q1) diag(l + nw);
        T o[R];
#pragma unroll
        for (int r = 0; r < R; r++) o[r] = mgl_to<T>(d[r]);
        mgl_st<R>(o, (unsigned)__cvta_generic_to_shared(g + (l - 2 * q0) * LS), lane);
        // |d|^2: the halves exchange their parts so that the lower one forms
        // the even rows' norms and the upper one the odd rows'
        const bool up = lane >= 16;
#pragma unroll
        for (int r = 0; r < R; r += 2) {
            const double d1 = r + 1 < R ? d[r + 1 < R ? r + 1 : r] : 0.0;
            const double got = __shfl_xor_sync(0xffffffffu, up ? d[r] : d1, 16), own = up ? d1 : d[r];
            const unsigned long long n = (unsigned long long)__double_as_longlong(own * own + got * got);
            mx = n > mx && n <= kInf ? n : mx;
        }
    }
    mx = mgl_warp_max(mx);
    if (lane == 0) sh[warp] = mx;
    __syncthreads();
    if (warp == 0) {
        mx = mgl_warp_max(lane < nw ? sh[lane] : 0ULL);
        if (lane < a.cs) *cooperative_groups::this_cluster().map_shared_rank(&c.slot[par][c.rank], lane) = mx;
    }
    mgl_arrive(sync);
    mgl_wait(sync);
    return mgl_warp_max(lane < a.cs ? c.slot[par][lane] : 0ULL);
}

// The half sweeps of one cycle as a block runs them, and their tasks.  Levels
// spread over the cluster wait at cluster barriers; block 0 runs the others
// between two of them.  Called by every thread of the block.
template <int R, class T>
__device__ void mgl_schedule(MglCtx &c) {
    const MgLineArgs &a = c.a;
    constexpr bool kMixed = sizeof(T) == 4;
    const int wide = a.cs > 1 ? MGL_CLUSTER : MGL_BLOCK;
    int nph = 0, nd = 0;
    auto add = [&](int kind, int ilev, int sync, int at = -1) {
        const int n = mgl_ntask(c, kind, ilev), first = at >= 0 ? at : nd;
        int f = 0;
        if (kind != MGL_IDLE) f |= kind == MGL_SRC0 ? kMglStore : kMglSolve;
        if (kind == MGL_COARSE) f |= kMglCoarse;
        if (kind < MGL_TOP_FIRST) f |= kMglStore;
        if (ilev == a.nlev) {
            const bool even = kind == MGL_TOP_EVEN;
            f |= kMixed ? kMglInit : kMglB;
            if (!even) f |= kMglStore;
            if (even || c.kv != 1) f |= kMglPut;
            if (even && c.kv == 1) f |= kMglPin;
        } else if (kind == MGL_C_FIRST || kind == MGL_C_ODD || kind == MGL_C_EVEN) {
            f |= kMglInit;
        }
        if (threadIdx.x == 0) c.ph[nph] = MglPhase{first, n, f, sync};
        nph++;
        if (at < 0) {
            for (int t = threadIdx.x; t < n; t += blockDim.x)
                mgl_make_task<R, T>(c, kind, ilev, t, reinterpret_cast<MglTask<T> *>(c.task)[first + t]);
            nd += n;
        }
        return first;
    };
    add(MGL_TOP_FIRST, a.nlev, MGL_BLOCK);
    const int even = add(MGL_TOP_EVEN, a.nlev, wide);
    // the residual's exchange is a barrier: the first phase after it needs none
    int sync = MGL_NONE, l = a.nlev - 1;
    for (; l >= 1 && !a.lev[l].solo; l--) {
        add(MGL_DOWN_ODD, l, sync);
        add(MGL_DOWN_EVEN, l, wide);
        sync = wide;
    }
    const int first = l;                // the first level of block 0 alone
    if (c.rank != 0) {
        if (sync == MGL_CLUSTER) add(MGL_IDLE, 0, sync);        // block 0 waits here for the last spread level
    } else {
        for (; l >= 1; l--) {
            add(MGL_DOWN_ODD, l, sync);
            add(MGL_DOWN_EVEN, l, MGL_BLOCK);
            sync = MGL_BLOCK;
        }
        const bool one = a.lev[0].n <= kMglThreads / 32;
        add(one ? MGL_COARSE : MGL_SRC0, 0, sync);
        int odd = -1, ev = -1;
        for (int it = 0; it < a.nbli && !one; it++) {
            if (it == 0) add(MGL_C_FIRST, 0, MGL_BLOCK);
            else odd = add(MGL_C_ODD, 0, MGL_BLOCK, odd);
            ev = add(MGL_C_EVEN, 0, MGL_BLOCK, ev);
        }
        for (l = 1; l <= first; l++) {
            add(MGL_UP_ODD, l, MGL_BLOCK);
            add(MGL_UP_EVEN, l, MGL_BLOCK);
        }
    }
    for (l = first + 1; l <= a.nlev - 1; l++) {
        add(MGL_UP_ODD, l, wide);
        add(MGL_UP_EVEN, l, wide);
    }
    add(MGL_TOP_ODD, a.nlev, wide);
    add(MGL_TOP_EVEN, a.nlev, wide, even);
    if (threadIdx.x == 0) {
        c.nph = nph;
        const int jr = a.xft ? a.n2m - 1 : a.n2m - 2;           // 0-based row of the pin
        const unsigned line = mgl_addr<R, T>(c, reinterpret_cast<T *>(c.g), a.lev[a.nlev], 0);
        c.pin = line + mgl_at<R, T>(jr % R, jr / R) * (int)sizeof(T);
    }
}

// mg2d (poiss_z_ft.f90:239-299): the cycles of one mode; returns their number
template <int R, class T>
__device__ __forceinline__ int mgl_cycles(MglCtx &c, bool &unconv) {
    const MgLineArgs &a = c.a;
    const int wide = a.cs > 1 ? MGL_CLUSTER : MGL_BLOCK, nph = c.nph;
    unsigned long long limit = c.test2;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = kMglThreads >> 5;
    const unsigned stage = c.stage + warp * mgl_stage_bytes<R, T>();
    const MglTask<T> *task = reinterpret_cast<const MglTask<T> *>(c.task);
    // the phase and the warp's task at hand; the next ones are read, and the
    // next line's table sent for, before the phase waits for the others
    MglPhase P = c.ph[0];
    MglRegs<T> d;
    bool have = warp < P.n;
    if (have) {
        d.read(task[P.first + warp]);
        mgl_fetch<R, T>(d.tab, stage, lane);
    }
    int kk = 0;
    for (int ph = 0;;) {
        mgl_arrive(P.sync);
        const MglPhase N = c.ph[ph + 1 < nph ? ph + 1 : 2];
        bool waiting = true;
        T tt = T(0.0);
        int t = warp;
        do {
            MglOp<R, T> o;
            if (have && (P.flags & kMglSolve)) o.load(stage, lane);
            const int tn = t + nw, at = tn < P.n ? P.first + tn : warp < N.n ? N.first + warp : -1;
            MglRegs<T> e;
            if (at >= 0) {
                e.read(task[at]);
                if ((tn < P.n ? P.flags : N.flags) & kMglSolve) mgl_fetch<R, T>(e.tab, stage, lane);
            }
            if (waiting) {
                mgl_wait(P.sync);
                waiting = false;
                if (P.flags & kMglPin) {
                    if constexpr (sizeof(T) == 4)
                        asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(tt) : "r"(c.pin + (lane & 16) * mgl_w<R, T>() * 4) : "memory");
                    else
                        asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(tt) : "r"(c.pin + (lane & 16) * mgl_w<R, T>() * 8) : "memory");
                }
            }
            if (P.flags & kMglCoarse) mgl_coarse<R, T>(d, o, have, warp, 2 * a.nbli, lane);
            else if (have && P.flags == (kMglSolve | kMglStore)) mgl_line_task<R, T>(d, o, lane);
            else if (have) mgl_work<R, T>(c, d, o, P.flags, tt, lane);
            have = at >= 0;
            if (have) d = e;
            t = tn;
        } while (t < P.n);
        P = N;
        ph++;
        if (ph != 2 && ph != nph) continue;
        const unsigned long long res = mgl_resid<R, T>(c, kk & 1, wide);
        // a timing run stops at a thousandth of its first residual
        if (a.timing && kk == 0) limit = (unsigned long long)__double_as_longlong(1.0e-6 * __longlong_as_double((long long)res));
        if (res < limit) return kk;
        if (kk == a.mgitr) break;
        kk++;
        ph = 2;
    }
    unconv = true;
    return a.xft ? a.mgitr : a.mgitr + 1;
}

// Cluster b of the launch solves mode b % nmodes + 1 of the case described by
// as[b / nmodes]; its right-hand side in ccap is replaced by the solution.
template <int R, bool MIXED>
__global__ void __launch_bounds__(kMglThreads, 1) k_mgl_modes(const MgLineArgs *as, int nmodes) {
    using T = typename std::conditional<MIXED, float, double>::type;
    constexpr int LS = R * 32;
    extern __shared__ __align__(16) unsigned char smraw[];
    __shared__ MglCtx c;
    namespace cg = cooperative_groups;
    const int cs = (int)cg::this_cluster().num_blocks(), rank = (int)cg::this_cluster().block_rank();
    const int b = blockIdx.x / cs, kv = b % nmodes + 1;
    {
        const int *src = reinterpret_cast<const int *>(as + b / nmodes);
        int *dst = reinterpret_cast<int *>(&c.a);
        for (int t = threadIdx.x; t < (int)(sizeof(MgLineArgs) / sizeof(int)); t += blockDim.x) dst[t] = src[t];
    }
    __syncthreads();
    const MgLineArgs &a = c.a;
    const int ntop = a.top2 * LS;
    if (threadIdx.x == 0) {
        c.kv = kv;
        c.rank = rank;
        unsigned char *p = smraw;
        c.x = reinterpret_cast<double *>(p); p += ntop * sizeof(double);
        if (a.bshared) { c.b = reinterpret_cast<double *>(p); p += ntop * sizeof(double); }
        else c.b = a.bt + ((size_t)(kv - 1) * cs + rank) * ntop;
        c.zero = p; p += LS * sizeof(double);
        c.rows = reinterpret_cast<double *>(p); p += 2 * R * 16 * sizeof(double);
        c.stage = (unsigned)__cvta_generic_to_shared(p); p += mgl_stage_bytes<R, T>() * (kMglThreads / 32);
        c.task = p; p += a.ndesc * sizeof(MglTask<T>);
        c.g = p; p += a.lines * LS * sizeof(T);
        c.r0 = p;
        // sqrt(n) < test as an integer test of n: the least n whose root is
        // not below the criterion
        const double test = a.S->mg_test;
        double t2 = test > 0.0 ? test * test : 0.0;     // 0 too where the square underflows: a zero residual passes
        if (test > 0.0 && t2 <= 1.0e300) {
            while (t2 > 0.0 && sqrt(t2) >= test) t2 = __longlong_as_double(__double_as_longlong(t2) - 1);
            while (sqrt(t2) < test) t2 = __longlong_as_double(__double_as_longlong(t2) + 1);
        }
        c.test2 = (unsigned long long)__double_as_longlong(t2);
    }
    __syncthreads();
    mgl_schedule<R, T>(c);
    const MgLevel &L = a.lev[a.nlev];
    int q0, q1;
    mgl_own(c, L, q0, q1);
    const int own = 2 * (q1 - q0);
    // b and the FP32 source start as the mode's right-hand side, everything else as zero
    for (int t = threadIdx.x; t < ntop; t += blockDim.x) {
        c.x[t] = 0.0;
        c.b[t] = 0.0;
    }
    for (int t = threadIdx.x; t < LS; t += blockDim.x) reinterpret_cast<double *>(c.zero)[t] = 0.0;
    for (int t = threadIdx.x; t < R * 16; t += blockDim.x) { c.rows[t] = a.asl[t]; c.rows[R * 16 + t] = a.anl[t]; }
    for (int t = threadIdx.x; t < (a.lines + a.lev[0].n) * LS; t += blockDim.x) reinterpret_cast<T *>(c.g)[t] = T(0.0);
    __syncthreads();
    double2 *plane = a.ccap + (size_t)a.nl * a.n2m * (kv - 1);
    for (int t = threadIdx.x; t < own * a.n2m; t += blockDim.x) {
        const int l = t % own, j = t / own, r = j % R, n = j / R;
        const double2 v = plane[(2 * q0 + l) + (size_t)a.nl * j];
        c.b[l * LS + mgl_at<R, double>(r, n)] = v.x;
        c.b[l * LS + mgl_at<R, double>(r, n + 16)] = v.y;
        if constexpr (MIXED) {
            T *g = reinterpret_cast<T *>(c.g) + l * LS;
            g[mgl_at<R, T>(r, n)] = (T)v.x;
            g[mgl_at<R, T>(r, n + 16)] = (T)v.y;
        }
    }
    __syncthreads();
    bool unconv = false;
    const int it = mgl_cycles<R, T>(c, unconv);
    asm volatile("cp.async.wait_all;" ::: "memory");
    for (int t = threadIdx.x; t < own * a.n2m; t += blockDim.x) {
        const int l = t % own, j = t / own, r = j % R, n = j / R;
        plane[(2 * q0 + l) + (size_t)a.nl * j] =
            make_double2(c.x[l * LS + mgl_at<R, double>(r, n)], c.x[l * LS + mgl_at<R, double>(r, n + 16)]);
    }
    if (rank == 0 && threadIdx.x == 0) {
        a.iters[kv - 1] = it;
        atomicMax((unsigned long long *)&a.S->poisson_iters[a.slot], (unsigned long long)it);
        // not counted in the autotuner's timing runs
        if (unconv && !a.timing) atomicAdd((unsigned long long *)&a.S->poisson_unconv, 1ULL);
    }
    // every block has passed the last norm exchange, after which no block
    // reads another's shared memory
}

}  // namespace lg
