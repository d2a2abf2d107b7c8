// fx_reference.cu -- the reference hierarchy's smoothers and transfers (multigrid.rs:188-473) as
// fused passes.  Every point value is the expression of the backend ops they replace, in the same
// order, so the cycle built from them equals the op-by-op one bit for bit.
#include <algorithm>
#include <atomic>

#include <cooperative_groups.h>

#include "fx_reference.cuh"
#include "fx_wcycle.cuh"

using namespace fx;
namespace cg = cooperative_groups;

FX_CHECK_FILE(reference);

namespace {

// ---------------------------------------------------------------- lexicographic sweep
//
// An in-place lexicographic sweep of a five-point stencil: a point needs its new north and west
// neighbours and its old south and east ones, so all points of a diagonal r + c = t are independent
// and a sweep is a chain of rows + cols dependent steps.  What bounds it is the latency of one
// step -- the new north value arrives by a shuffle and is followed by seven dependent operations
// in the reference's order: about 90 cycles in FP64 -- so the work is laid out to keep everything
// else off that chain:
//
//  - a warp owns 32 rows, lane l the column t - l of its row at step t: the new west value is the
//    lane's own last result, the new north value the lane above's (a shuffle); the old values it
//    needs are read from shared memory eight steps ahead;
//  - x and b pass through a 64-column window per row in shared memory.  A partner warp refills it
//    16 columns at a time by cp.async and stores finished columns, coalesced, while the sweeping
//    warp runs (in one warp the copies took as long as the sweep: 136 us for a 256 x 256 sweep);
//  - a phase is 16 steps.  The warp below starts three phases later (its first row needs the last
//    row of this warp, 31 columns behind lane 0) and receives that row through its own shared
//    memory, in the next block of the cluster where needed.  Phases are joined by a barrier of the
//    cluster, so nothing spins;
//  - consecutive sweeps run in the same launch, each 8 phases behind the one before: the first
//    load of a column block by sweep k + 1 comes after sweep k stored it (and the row below it).
//
// The form any radius-1 stencil needs -- one block of 1024 threads stepping over the hyperplanes
// 2 r + c with x in global memory, a barrier and dependent loads per step -- takes 1400 us for two
// 256 x 256 sweeps in FP64, this one 88 us: 48 phases of 2000 cycles of sweeping and 1000 of barrier
// (the release of the row and column stores is 700 of them).  Grids of up to 34 rows and 66
// columns run in one warp without any phase (k_lex5_small).
constexpr int kLexK = 16;              // steps per phase, columns per block
constexpr int kLexGroup = 8;           // steps whose operands are read together, ahead of the chain
constexpr int kLexWin = 64;            // window columns
constexpr int kLexPitch = kLexWin + 2; // row pitch: lane l's column t - l falls in its own bank
constexpr int kLexMaxCta = 8;          // blocks per cluster (the portable size)
constexpr int kLexLag = 3;             // phases between a warp and the one below it
constexpr int kLexSweepLag = 8;        // phases between a sweep and the next

template <typename T>
struct LexArgs {
    T *x;
    const T *b;
    int rows, cols;
    T w[5];
    T om, id;
    int nwr;      // warps over the rows of one sweep
    int nsweeps;  // sweeps in this launch
    int nsuper;   // row blocks of 32 nwr rows, one after the other (nsweeps = 1 when > 1)
};

template <typename T>
struct LexWarpSmem {
    T x[33 * kLexPitch];
    T b[32 * kLexPitch];
    T n[kLexWin];  // the row above: new values
};

// fma(om, id (b - A x), x) with A x accumulated in entry order (k_lex_jacobi)
template <typename T>
__device__ __forceinline__ T lex_point(const T (&w)[5], T om, T id, T b, T c, T n, T s, T we, T e) {
    T ax = fx_fma(w[0], c, (T)0);
    ax = fx_fma(w[1], n, ax);
    ax = fx_fma(w[2], s, ax);
    ax = fx_fma(w[3], we, ax);
    ax = fx_fma(w[4], e, ax);
    return fx_fma(om, id * (b - ax), c);
}

// NW: sweeping warps per block, each with a copying partner.
template <typename T, int NW>
__global__ void __launch_bounds__(NW * 64) k_lex5(LexArgs<T> A) {
    grid_dep_enter();
    extern __shared__ __align__(16) unsigned char lex_smem[];
    cg::cluster_group cluster = cg::this_cluster();
    const int ncta = (int)cluster.num_blocks(), rank = (int)cluster.block_rank();
    const int lane = threadIdx.x & 31;
    const bool io = threadIdx.x >= NW * 32;  // the copying partner of a sweeping warp
    const int wid = (threadIdx.x >> 5) & (NW - 1);
    LexWarpSmem<T> *const all = reinterpret_cast<LexWarpSmem<T> *>(lex_smem);
    LexWarpSmem<T> &W = all[wid];
    const int wt = rank * NW + wid;
    const int sweep = wt / A.nwr, gw = wt - sweep * A.nwr;
    const int rows = A.rows, cols = A.cols, R = rows - 2, C = cols - 2;
    const long long n = (long long)rows * cols;
    (void)n;
    // the next warp's copy of the row above it (this warp's last row)
    LexWarpSmem<T> *next = nullptr;
    if (gw + 1 < A.nwr && sweep < A.nsweeps)
        next = wid + 1 < NW ? all + wid + 1 : (rank + 1 < ncta ? cluster.map_shared_rank(all, rank + 1) : nullptr);
    const int P = (C - 1 + kLexK - 1) / kLexK + 3;  // phases: the last one stores column C - 1's block
    const int G = kLexLag * (A.nwr - 1) + kLexSweepLag * (A.nsweeps - 1) + P;
    const int off = sweep * kLexSweepLag + gw * kLexLag;
    constexpr int WM = kLexWin - 1;

    for (int sb = 0; sb < A.nsuper; sb++) {
        const int base = (sb * A.nwr + gw) * 32;  // interior row of lane 0
        const int nl = sweep < A.nsweeps ? min(32, R - base) : 0;
        const bool on = nl > 0;
        if (io) {
            // Column block q: columns u = (q - 1) K + 1 .. q K (u = grid column - 1); lane halves take
            // alternate rows, so a half warp moves 16 consecutive columns.  Row 32 is the row below
            // the warp's; the other half then takes the row above it for the first warp.
            const int half = lane >> 4, cq = lane & 15;
            const int r0 = 1 + base + half;
            const int nx = (rows - r0 + 1) >> 1, nb = (rows - 1 - r0 + 1) >> 1, ns = (nl - half + 1) >> 1;  // rows r0, r0 + 2, ..
            const T *const any = A.b;
            auto copy_in = [&](int q) {
                const int u = (q - 1) * kLexK + 1 + cq, k = u & WM;
                const bool ux = u >= 0 && u <= C, ub = u >= 0 && u < C;
                long long o = (long long)r0 * cols + u + 1;
                T *sx = W.x + half * kLexPitch + k, *sB = W.b + half * kLexPitch + k;
#pragma unroll 4
                for (int i = 0; i < 16; i++) {
                    cp_async_elem(sx, A.x + o, ux && i < nx && FX_IN(o, n), any);
                    cp_async_elem(sB, A.b + o, ub && i < nb && FX_IN(o, n), any);
                    o += 2 * cols;
                    sx += 2 * kLexPitch;
                    sB += 2 * kLexPitch;
                }
                const int gr = half ? base : 1 + base + 32;
                o = (long long)gr * cols + u + 1;
                if (!half || gw == 0)
                    cp_async_elem(half ? W.n + k : W.x + 32 * kLexPitch + k, A.x + o, ux && gr < rows && FX_IN(o, n), any);
            };
            auto copy_out = [&](int q) {
                const int u = (q - 1) * kLexK + 1 + cq;
                if (u < 0 || u >= C) return;
                const T *sx = W.x + half * kLexPitch + (u & WM);
                long long o = (long long)r0 * cols + u + 1;
                T v[16];
#pragma unroll
                for (int i = 0; i < 16; i++) v[i] = sx[i * 2 * kLexPitch];
#pragma unroll
                for (int i = 0; i < 16; i++) {
                    if (i < ns && FX_IN(o, n)) A.x[o] = v[i];
                    o += 2 * cols;
                }
            };
            for (int g = -1; g < G; g++) {
                const int p = g - off;
                if (on && p >= -1 && p < P) {
                    if (p < 0) copy_in(0);
                    else copy_out(p - 2);  // finished in every lane when phase p - 1 ended
                    copy_in(p + 2);        // into the slots of block p - 2 (block 1 before the first phase)
                    cp_async_commit();
                    cp_async_wait<0>();
                }
                if (ncta > 1) cluster.sync();
                else __syncthreads();
            }
            continue;
        }
        const unsigned Cm = lane < nl ? (unsigned)C : 0u;  // this lane's columns
        T prev = (T)0, cur = (T)0;
        const T *const bx = W.x + lane * kLexPitch;
        for (int g = -1; g < G; g++) {
            const int p = g - off;
            if (p == -1) {
                const long long o = (long long)(1 + base + lane) * cols;
                if (lane < nl && FX_IN(o, n)) prev = A.x[o];  // west of the first column
            } else if (on && p >= 0 && p * kLexK < C + nl - 1) {
                if (p == 0) cur = bx[0];  // the first lane's first centre value
                // The old values a step reads (b, east, south; the first lane's north) do not change
                // before the lane reaches them: they are read a group of steps ahead of the chain.
                // Groups are short so that the loop stays in the instruction cache of its scheduler.
                struct Old {
                    T b, s, e, n;
                };
                Old o[2][kLexGroup];
                auto read = [&](Old (&d)[kLexGroup], int s0) {
#pragma unroll
                    for (int k = 0; k < kLexGroup; k++) {
                        const int j = (s0 + k - lane) & WM;
                        d[k].b = W.b[lane * kLexPitch + j];
                        d[k].s = bx[kLexPitch + j];
                        d[k].e = bx[(j + 1) & WM];
                        d[k].n = W.n[j];
                    }
                };
                auto sweep_group = [&](const Old (&d)[kLexGroup], int s0) {
#pragma unroll
                    for (int k = 0; k < kLexGroup; k++) {
                        const int u = s0 + k - lane;
                        const T up = __shfl_up_sync(0xffffffffu, prev, 1);
                        const T v = lex_point(A.w, A.om, A.id, d[k].b, cur, lane ? up : d[k].n, d[k].s, prev, d[k].e);
                        if ((unsigned)u < Cm) {
                            prev = v;
                            W.x[lane * kLexPitch + (u & WM)] = v;
                        }
                        cur = d[k].e;
                    }
                };
                const int s0 = p * kLexK;
                read(o[0], s0);
#pragma unroll 1
                for (int k = 0; k < kLexK; k += 2 * kLexGroup) {
                    read(o[1], s0 + k + kLexGroup);
                    __syncwarp();
                    sweep_group(o[0], s0 + k);
                    if (k + 2 * kLexGroup < kLexK) read(o[0], s0 + k + 2 * kLexGroup);
                    __syncwarp();
                    sweep_group(o[1], s0 + k + kLexGroup);
                }
                __syncwarp();
                // the columns the last row finished in this phase: the next warp's row above
                const int u = s0 - 31 + lane;
                if (next && lane < kLexK && u >= 0 && u < C) next->n[u & WM] = W.x[31 * kLexPitch + (u & WM)];
            }
            if (ncta > 1) cluster.sync();
            else __syncthreads();
        }
    }
}

// The whole grid in shared memory, one warp: at most 32 interior rows and 64 interior columns.  The
// sweeps follow each other without a gap: lane l starts the next sweep as soon as it has finished
// its row (the lane below is one column behind in the same sweep, the lane above one ahead).
constexpr int kLexSmallRows = 34, kLexSmallCols = 66;

// The old values of the next point are read a step ahead of the chain (AHEAD), which needs three
// interior columns: with fewer, the row below finishes the point a wrapped step reads in that step.
template <typename T, bool AHEAD>
__global__ void __launch_bounds__(32) k_lex5_small(LexArgs<T> A) {
    grid_dep_enter();
    __shared__ T xs[kLexSmallRows * kLexSmallCols], bs[kLexSmallRows * kLexSmallCols];
    const int lane = threadIdx.x;
    const int rows = A.rows, cols = A.cols, R = rows - 2, C = cols - 2, n = rows * cols;
    if (!FX_IN(n - 1, kLexSmallRows * kLexSmallCols)) return;
    for (int i = lane; i < n; i += 32) {
        cp_async_elem(xs + i, A.x + i, true, A.x);
        cp_async_elem(bs + i, A.b + i, true, A.b);
    }
    cp_async_commit();
    cp_async_wait<0>();
    __syncwarp();
    const bool mine = lane < R;
    const int row = (mine ? 1 + lane : 1) * cols + 1;  // this lane's first interior point
    const T *bp = bs + row;
    const T west0 = xs[row - 1];
    T prev = (T)0;
    struct Old {
        T b, c, n, s, e;
    };
    auto read = [&](int u) {
        const int i = row + u;
        return Old{bp[u], xs[i], xs[i - cols], xs[i + cols], xs[i + 1]};
    };
    // lane l is at point t = s - l of its row's sweeps: column t mod C
    const int total = A.nsweeps * C;
    Old o = read(0);
    int u = 0;
    for (int s = 0; s < total + min(R, 32) - 1; s++) {
        const int t = s - lane;
        const bool act = mine && t >= 0 && t < total;
        const int un = u + 1 < C ? u + 1 : 0;  // the column after this one
        if (!AHEAD) o = read(u);
        const Old nx = AHEAD ? read(act ? un : u) : o;
        const T up = __shfl_up_sync(0xffffffffu, prev, 1);
        if (act) {
            const T v = lex_point(A.w, A.om, A.id, o.b, o.c, lane ? up : o.n, o.s, u == 0 ? west0 : prev, o.e);
            xs[row + u] = v;
            prev = v;
            u = un;
            o = nx;
        }
        __syncwarp();
    }
    for (int i = lane; i < n; i += 32) A.x[i] = xs[i];
}

template <typename K, typename... Args>
int launch_cluster(fx_ctx *ctx, K kernel, int blocks, int threads, size_t smem, const char *what, Args... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)blocks);
    cfg.blockDim = dim3((unsigned)threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = ctx->stream;
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = (unsigned)blocks;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = ctx->pdl ? 2 : 1;
    (void)cudaLaunchKernelEx(&cfg, kernel, args...);  // errors surface in check_launch
    return check_launch(ctx, what);
}

// ---------------------------------------------------------------- Chebyshev and residual passes
//
// One point per thread, a row of blocks per grid row (no division).  A step reads the iterate's
// five points, the rhs and at most one further vector and writes one: the op-by-op form made
// eight launches of it (apply_stencil and its ring, copy, axpy, scale, axpy, axpy,
// zero_boundaries), 1.8 us each at any size up to 1024 x 768, where the vectors stay in L2 and a
// launch's latency is the cost.

template <typename F>
__global__ void __launch_bounds__(256) k_rows(int rows, int cols, F f) {
    grid_dep_enter();
    const int c = blockIdx.x * 256 + threadIdx.x;
    if (c >= cols) return;
    for (int r = blockIdx.y; r < rows; r += gridDim.y)
        if (FX_IN((long long)r * cols + c, (long long)rows * cols)) f(r, c, (size_t)r * cols + c);
}

template <typename F>
int launch_rows(fx_ctx *ctx, size_t rows, size_t cols, F f, const char *what) {
    const dim3 grid((unsigned)((cols + 255) / 256), (unsigned)std::min<size_t>(rows, 65535));
    timing_pre(ctx, what);
    launch_pdl(ctx, k_rows<F>, grid, dim3(256), 0, (int)rows, (int)cols, f);
    timing_post(ctx, (double)rows * (double)cols);
    return check_launch(ctx, what);
}

// the iterate (zero when u is null), corrected by the piecewise-constant prolongation of `e` when
// that is not null
struct ChebIn {
    const double *u, *e;
    int cols, ccols;
    __device__ __forceinline__ double at(int r, int c, size_t i) const {
        const double v = u ? u[i] : 0.0;
        return e ? v + e[(size_t)(r >> 1) * ccols + (c >> 1)] : v;
    }
    __device__ __forceinline__ Nb<double> nb(int r, int c, size_t i) const {
        Nb<double> v;
        v.c = at(r, c, i);
        v.n = at(r - 1, c, i - cols);
        v.s = at(r + 1, c, i + cols);
        v.w = at(r, c - 1, i - 1);
        v.e = at(r, c + 1, i + 1);
        v.nw = v.ne = v.sw = v.se = 0.0;
        return v;
    }
};

struct ChebFirst {  // w0 = u + (scale / diag) (rhs - S u), ring 0
    ChebIn in;
    const double *rhs;
    double *out;
    StencilP P;
    double f;
    int rows, cols;
    __device__ __forceinline__ void operator()(int r, int c, size_t i) const {
        if (r == 0 || c == 0 || r == rows - 1 || c == cols - 1) {
            out[i] = 0.0;
            return;
        }
        const Nb<double> v = in.nb(r, c, i);
        const double d = fma(-1.0, stencil_eval<double, 5>(P, v), rhs[i]) * f;
        out[i] = fma(1.0, v.c, d);
    }
};

struct ChebNext {  // out = omega (scale / diag) (rhs - S x_k) + omega x_k + (1 - omega) x_{k-1}, ring 0
    const double *xk;
    ChebIn km1;
    const double *rhs;
    double *out;  // may be the buffer of x_{k-1}
    StencilP P;
    double inv_diag, os, om, om1;
    int rows, cols;
    __device__ __forceinline__ void operator()(int r, int c, size_t i) const {
        if (r == 0 || c == 0 || r == rows - 1 || c == cols - 1) {
            out[i] = 0.0;
            return;
        }
        const Nb<double> v = ChebIn{xk, nullptr, cols, 0}.nb(r, c, i);
        double d = fma(-1.0, stencil_eval<double, 5>(P, v), rhs[i]);
        d = d * inv_diag;
        d = d * os;
        d = fma(om, v.c, d);
        out[i] = fma(om1, km1.at(r, c, i), d);
    }
};

// One coarse point: the residual at its four fine points (ring points by the boundary values) and
// their average.
struct RefRestrict {
    const double *u, *rhs;
    double *crhs, *cu;
    StencilP P;
    BcP B;
    int rows, cols, ccols;
    __device__ __forceinline__ double resid(int r, int c) const {
        const size_t i = (size_t)r * cols + c;
        double t;
        if (r == 0) t = bc_value(B, 0, u[i], u[i + cols], B.dy);
        else if (r == rows - 1) t = bc_value(B, 1, u[i], u[i - cols], B.dy);
        else if (c == 0) t = bc_value(B, 2, u[i], u[i + 1], B.dx);
        else if (c == cols - 1) t = bc_value(B, 3, u[i], u[i - 1], B.dx);
        else t = stencil_eval<double, 5>(P, ChebIn{u, nullptr, cols, 0}.nb(r, c, i));
        return fma(1.0, rhs[i], t * -1.0);
    }
    __device__ __forceinline__ void operator()(int r, int c, size_t i) const {
        const int fr = 2 * r, fc = 2 * c;
        const int fr1 = fr + 1 < rows - 1 ? fr + 1 : rows - 1, fc1 = fc + 1 < cols - 1 ? fc + 1 : cols - 1;
        crhs[i] = 0.25 * (((resid(fr, fc) + resid(fr1, fc)) + resid(fr, fc1)) + resid(fr1, fc1));
        if (cu) cu[i] = 0.0;
    }
};

// ---------------------------------------------------------------- the Chebyshev hierarchy's tail
//
// The coarse levels in one block, every vector in shared memory.  A launch of a small level costs
// 1.9 us whatever it computes, and a cycle from 64 x 48 down makes 34 of them; in one block a step
// is a barrier, a shared round trip and the point's chain of ten dependent operations.  What then
// bounds it is instruction issue and that chain, so: a level is worked on by the warps it has points
// for and the others sleep at a barrier (all warps through every step: 36 us), the residual is taken
// once per fine point and not four times around the average, and the ring's four sides share one
// code path (those two: 32 -> 25 us).  MG-PCG on 1024 x 768, 33 cycles: 5.07 -> 3.96 ms.
// A level's three iterates rotate: after n steps the iterate is buffer n mod 3, so nothing is copied.
// The tail starts at the first level whose vectors, with those below it, fit in 200 KB (4800 points
// or so); a larger level has work for more than one SM.

constexpr int kChebTailLevels = 10;
constexpr int kChebTailSteps = 32;
constexpr int kChebTailThreads = 512;  // 1024: level
constexpr size_t kChebTailSmem = 200 * 1024;

struct ChebTailLevel {
    int rows, cols;
    unsigned magic;  // 2^32 / cols, rounded up: i / cols = umulhi(i, magic) for i * cols < 2^32
    double w[5];     // centre, north, south, west, east
    double f, inv_diag;
    BcP B;
};

struct ChebTailArgs {
    const double *u_in;  // null: zero
    const double *rhs;
    double *u_out;
    int nlev, n_pre, n_post, n_coarse;
    ChebTailLevel L[kChebTailLevels];
    double os[kChebTailSteps], om[kChebTailSteps];  // of the steps after the first
};

__global__ void __launch_bounds__(kChebTailThreads) k_cheb_tail(const __grid_constant__ ChebTailArgs A_in) {
    // the arguments in shared memory: read a level at a time they would miss the constant cache in
    // every one of the short steps
    __shared__ ChebTailArgs A;
    static_assert(sizeof(ChebTailArgs) % sizeof(long long) == 0, "copied by words");
    for (int i = threadIdx.x; i < (int)(sizeof(ChebTailArgs) / sizeof(long long)); i += blockDim.x)
        reinterpret_cast<long long *>(&A)[i] = reinterpret_cast<const long long *>(&A_in)[i];
    grid_dep_enter();
    __syncthreads();
    extern __shared__ double ct_smem[];  // level l: iterates 0, 1, 2 and the rhs, n values each
    double *const sm = ct_smem;
    // a level is worked on by as many warps as it has points for; the others wait at the barrier of
    // the level above until the cycle comes back up (barrier 1 + l: level l's warps)
    auto warps = [&](int l) { return min((int)blockDim.x >> 5, (A.L[l].rows * A.L[l].cols + 31) >> 5); };
    auto sync = [](int l, int w) { asm volatile("barrier.sync %0, %1;" ::"r"(1 + l), "r"(w * 32) : "memory"); };
    const int wid = threadIdx.x >> 5, last = A.nlev - 1;
    {
        const int n0 = A.L[0].rows * A.L[0].cols;
        for (int i = threadIdx.x; i < n0; i += blockDim.x) {
            sm[i] = A.u_in ? A.u_in[i] : 0.0;
            sm[3 * n0 + i] = A.rhs[i];
        }
        __syncthreads();
    }
    int off = 0, e = 0;  // of the level; of the correction to add
    int k = 0;           // the iterate
    for (int v = 0; v <= 2 * last; v++) {  // down to the coarsest level and up again
        const bool down = v < last;
        const int l = v <= last ? v : 2 * last - v;
        const ChebTailLevel &L = A.L[l];
        const int rows = L.rows, cols = L.cols, np = rows * cols, nw = warps(l);
        const unsigned magic = L.magic;
        if (wid < nw) {
            auto points = [&](int pc, int n, unsigned mg, auto f) {
#pragma unroll 1
                for (int i = threadIdx.x; i < n; i += nw * 32) {
                    const int r = (int)__umulhi((unsigned)i, mg);
                    f(r, i - r * pc, i);
                }
                sync(l, nw);
            };
            const double *const rhs = sm + (off + 3 * np);
            const double wc = L.w[0], wn = L.w[1], ws = L.w[2], ww = L.w[3], we = L.w[4], f = L.f, inv_diag = L.inv_diag;
            auto ring = [&](int r, int c) { return r == 0 || c == 0 || r == rows - 1 || c == cols - 1; };
            auto apply = [&](const double *u) {  // stencil_eval<double, 5>
                StencilP P;
                P.c = wc, P.n = wn, P.s = ws, P.w = ww, P.e = we;
                Nb<double> nb;
                nb.c = u[0], nb.n = u[-cols], nb.s = u[cols], nb.w = u[-1], nb.e = u[1];
                nb.nw = nb.ne = nb.sw = nb.se = 0.0;
                return stencil_eval<double, 5>(P, nb);
            };
            const int n = down ? A.n_pre : (v == last ? A.n_coarse : A.n_post);
            k = v <= last ? 0 : A.n_pre % 3;
            if (v > last) {
                sync(l, nw);  // the level below is done
                const int cc = A.L[l + 1].cols, u = off + k * np;
                points(cols, np, magic, [&](int r, int c, int i) { sm[u + i] += sm[e + (r >> 1) * cc + (c >> 1)]; });
            }
            for (int i = 0; i < n; i++) {  // ChebFirst, ChebNext
                const int k1 = k == 2 ? 0 : k + 1, km = k == 0 ? 2 : k - 1;
                const double *const u = sm + (off + k * np), *const um = sm + (off + km * np);
                double *const out = sm + (off + k1 * np);
                if (i == 0) {
                    points(cols, np, magic, [&](int r, int c, int p) {
                        out[p] = ring(r, c) ? 0.0 : fma(1.0, u[p], fma(-1.0, apply(u + p), rhs[p]) * f);
                    });
                } else {
                    const double om = A.om[i], os = A.os[i], om1 = 1.0 - om;
                    points(cols, np, magic, [&](int r, int c, int p) {
                        double d = 0.0;
                        if (!ring(r, c)) {
                            d = fma(-1.0, apply(u + p), rhs[p]) * inv_diag;
                            d = fma(om1, um[p], fma(om, u[p], d * os));
                        }
                        out[p] = d;
                    });
                }
                k = k1;
            }
            if (down) {  // RefRestrict: the residual once per point into the free iterate, then the averages
                const ChebTailLevel &C = A.L[l + 1];
                const int nc = C.rows * C.cols, cc = C.cols;
                const double *const u = sm + (off + k * np);
                double *const res = sm + (off + (k == 2 ? 0 : k + 1) * np), *const cu = sm + (off + 4 * np);
                points(cols, np, magic, [&](int r, int c, int p) {
                    double t;
                    if (ring(r, c)) {
                        const int side = r == 0 ? 0 : (r == rows - 1 ? 1 : (c == 0 ? 2 : 3));
                        const int d = side == 0 ? cols : (side == 1 ? -cols : (side == 2 ? 1 : -1));
                        t = bc_value(L.B, side, u[p], u[p + d], side < 2 ? L.B.dy : L.B.dx);
                    } else {
                        t = apply(u + p);
                    }
                    res[p] = fma(1.0, rhs[p], t * -1.0);
                });
                points(cc, nc, C.magic, [&](int r, int c, int p) {
                    const int fr1 = min(2 * r + 1, rows - 1), fc1 = min(2 * c + 1, cols - 1);
                    const double *const r0 = res + 2 * r * cols, *const r1 = res + fr1 * cols;
                    cu[3 * nc + p] = 0.25 * (((r0[2 * c] + r1[2 * c]) + r0[fc1]) + r1[fc1]);
                    cu[p] = 0.0;
                });
            }
        }
        if (down) {
            off += 4 * np;
        } else if (l > 0) {
            e = off + (v == last ? A.n_coarse : A.n_pre + A.n_post) % 3 * np;
            off -= 4 * A.L[l - 1].rows * A.L[l - 1].cols;
        }
    }
    const int n0 = A.L[0].rows * A.L[0].cols;
    if (wid < warps(0))
        for (int i = threadIdx.x; i < n0; i += warps(0) * 32) A.u_out[i] = sm[k * n0 + i];
}

// the Chebyshev recurrence over the fixed spectrum [0.2, 2] (multigrid.rs:308-473)
struct ChebSeq {
    double scale, mu, omegaprod, c_km1, c_k;
    ChebSeq() {
        const double emax = 2.0, emin = 0.1 * emax;
        scale = 2.0 / (emax + emin);
        const double alpha = 1.0 - scale * emin;
        mu = 1.0 / alpha;
        omegaprod = 2.0 / alpha;
        c_km1 = 1.0;
        c_k = mu;
    }
    double next() {  // omega of the next step
        const double c_kp1 = 2.0 * mu * c_k - c_km1;
        const double omega = omegaprod * c_k / c_kp1;
        c_km1 = c_k;
        c_k = c_kp1;
        return omega;
    }
};

double cheb_inv_diag(double dx, double dy) {
    const double inv_dx2 = 1.0 / (dx * dx), inv_dy2 = 1.0 / (dy * dy);
    return -1.0 / (2.0 * inv_dx2 + 2.0 * inv_dy2);
}

template <typename T, int NW>
int lex5_launch(fx_ctx *ctx, const LexArgs<T> &A, int warps) {
    constexpr size_t smem = NW * sizeof(LexWarpSmem<T>);
    static std::atomic<unsigned long long> attr_done{0};  // one bit per device
    const unsigned long long bit = 1ull << (ctx->device & 63);
    if (!(attr_done.load() & bit)) {
        FX_CUDA(cudaFuncSetAttribute(k_lex5<T, NW>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        attr_done.fetch_or(bit);
    }
    int blocks = 1;  // a power of two covering the warps
    while (blocks * NW < warps) blocks *= 2;
    timing_pre(ctx, "weighted_jacobi");
    const int st = launch_cluster(ctx, k_lex5<T, NW>, blocks, NW * 64, smem, "weighted_jacobi", A);
    timing_post(ctx, (double)A.rows * (double)A.cols);
    return st;
}

}  // namespace

namespace fx {

bool lex5_order(const fx_stencil *s) {
    static const int dr[5] = {0, -1, 1, 0, 0}, dc[5] = {0, 0, 0, -1, 1};
    if (!s || s->n != 5) return false;
    for (int k = 0; k < 5; k++)
        if (s->dr[k] != dr[k] || s->dc[k] != dc[k]) return false;
    return true;
}

template <typename T>
int lex5_sweeps(fx_ctx *ctx, T *x, const T *b, size_t rows, size_t cols, const double (&w)[5], double omega,
                double inv_diag, size_t nsweeps) {
    LexArgs<T> A;
    A.x = x;
    A.b = b;
    A.rows = (int)rows;
    A.cols = (int)cols;
    for (int k = 0; k < 5; k++) A.w[k] = (T)w[k];
    A.om = (T)omega;
    A.id = (T)inv_diag;
    A.nwr = A.nsuper = 1;
    if (nsweeps == 0) return FX_OK;
    if (rows <= (size_t)kLexSmallRows && cols <= (size_t)kLexSmallCols) {
        while (nsweeps) {
            // a single interior column: the lane below would still be at the point this lane's next sweep reads
            A.nsweeps = cols == 3 ? 1 : (int)std::min<size_t>(nsweeps, 1u << 16);
            nsweeps -= (size_t)A.nsweeps;
            timing_pre(ctx, "weighted_jacobi");
            if (cols >= 5) launch_pdl(ctx, k_lex5_small<T, true>, dim3(1), dim3(32), 0, A);
            else launch_pdl(ctx, k_lex5_small<T, false>, dim3(1), dim3(32), 0, A);
            timing_post(ctx, (double)rows * (double)cols);
            FX_TRY(check_launch(ctx, "weighted_jacobi"));
        }
        return FX_OK;
    }
    const int R = (int)rows - 2, need = (R + 31) / 32, max_warps = kLexMaxCta * 4;
    A.nwr = std::min(need, max_warps);
    A.nsuper = (need + A.nwr - 1) / A.nwr;
    while (nsweeps) {
        A.nsweeps = A.nsuper > 1 ? 1 : (int)std::min<size_t>(nsweeps, (size_t)(max_warps / A.nwr));
        nsweeps -= (size_t)A.nsweeps;
        // two sweeping warps per block while the cluster has the blocks for it: the copies of four
        // slow each other and the sweeps down.  One FP64 sweep with four a block and with two: 192 x 192
        // 55 and 52 us, 256 x 256 74 and 69, 512 x 512 157 and 138; 128 x 128, whose four warps would share
        // one block and its barrier, 29 and 34.  FP32: 54 and 52, 73 and 70, 149 and 142, 27 and 34.
        const int warps = A.nwr * A.nsweeps;
        if (warps <= kLexMaxCta * 2) FX_TRY((lex5_launch<T, 2>(ctx, A, warps)));
        else FX_TRY((lex5_launch<T, 4>(ctx, A, warps)));
    }
    return FX_OK;
}
template int lex5_sweeps<float>(fx_ctx *, float *, const float *, size_t, size_t, const double (&)[5], double, double,
                                size_t);
template int lex5_sweeps<double>(fx_ctx *, double *, const double *, size_t, size_t, const double (&)[5], double, double,
                                 size_t);

int cheb_smooth(fx_ctx *ctx, const ChebLevel &L, const double *coarse, size_t ccols, size_t n, bool u_zero) {
    if (n == 0) return FX_OK;
    ChebSeq seq;
    const double inv_diag = cheb_inv_diag(L.dx, L.dy), scale = seq.scale;
    const int rows = (int)L.rows, cols = (int)L.cols;
    const ChebIn in{u_zero ? nullptr : L.u, coarse, cols, (int)ccols};
    FX_TRY(launch_rows(ctx, L.rows, L.cols, ChebFirst{in, L.rhs, L.w0, L.P, scale * inv_diag, rows, cols}, "cheb_step"));
    double *buf[3] = {L.u, L.w0, L.w1};
    int km1 = 0, k = 1, kp1 = 2;
    for (size_t i = 1; i < n; i++) {
        const double omega = seq.next();
        // the last step writes u itself where it may: x_{k-1} is read at the point alone, x_k around it
        double *out = i + 1 == n && k != 0 ? L.u : buf[kp1];
        const ChebIn prev = i == 1 ? in : ChebIn{buf[km1], nullptr, cols, 0};
        FX_TRY(launch_rows(ctx, L.rows, L.cols,
                           ChebNext{buf[k], prev, L.rhs, out, L.P, inv_diag, omega * scale, omega, 1.0 - omega, rows, cols},
                           "cheb_step"));
        if (i + 1 == n && out == L.u) return FX_OK;
        const int t = km1;
        km1 = k;
        k = kp1;
        kp1 = t;
    }
    if (buf[k] != L.u)
        FX_CUDA(cudaMemcpyAsync(L.u, buf[k], L.rows * L.cols * sizeof(double), cudaMemcpyDeviceToDevice, ctx->stream));
    return FX_OK;
}

int cheb_tail_top(const ChebLevel *L, int nl, size_t n_pre, size_t n_post, size_t n_coarse) {
    if (n_post == 0 || std::max(n_coarse, n_pre) > (size_t)kChebTailSteps) return nl;
    int top = nl;
    size_t bytes = 0;
    for (int l = nl - 1; l >= 0 && nl - l <= kChebTailLevels; l--) {
        if (L[l].rows < 2 || L[l].cols < 2 || L[l].rows > kChebTailSmem || L[l].cols > kChebTailSmem) break;
        bytes += 4 * sizeof(double) * L[l].rows * L[l].cols;
        if (bytes > kChebTailSmem) break;
        top = l;
    }
    return top;
}

int cheb_tail(fx_ctx *ctx, const ChebLevel *L, const BcP *B, int nlev, bool u_zero, size_t n_pre, size_t n_post,
              size_t n_coarse) {
    ChebTailArgs A;
    A.u_in = u_zero ? nullptr : L[0].u;
    A.rhs = L[0].rhs;
    A.u_out = L[0].u;
    A.nlev = nlev;
    A.n_pre = (int)n_pre;
    A.n_post = (int)n_post;
    A.n_coarse = (int)n_coarse;
    ChebSeq seq;
    const double scale = seq.scale;
    A.os[0] = A.om[0] = 0.0;
    for (int i = 1; i < kChebTailSteps; i++) {
        A.om[i] = seq.next();
        A.os[i] = A.om[i] * scale;
    }
    size_t bytes = 0;
    for (int l = 0; l < nlev; l++) {
        ChebTailLevel &T = A.L[l];
        T.rows = (int)L[l].rows;
        T.cols = (int)L[l].cols;
        T.magic = (unsigned)((1ull << 32) / L[l].cols + 1);
        const StencilP &P = L[l].P;
        T.w[0] = P.c, T.w[1] = P.n, T.w[2] = P.s, T.w[3] = P.w, T.w[4] = P.e;
        T.inv_diag = cheb_inv_diag(L[l].dx, L[l].dy);
        T.f = scale * T.inv_diag;
        T.B = B[l];
        bytes += 4 * sizeof(double) * L[l].rows * L[l].cols;
    }
    FX_TRY(strip_smem_optin(k_cheb_tail, kChebTailSmem));
    const size_t n0 = L[0].rows * L[0].cols;
    timing_pre(ctx, "cheb_tail");
    launch_pdl(ctx, k_cheb_tail, dim3(1), dim3((unsigned)std::min<size_t>(kChebTailThreads, (n0 + 31) / 32 * 32)), bytes, A);
    timing_post(ctx, (double)n0);
    return check_launch(ctx, "cheb_tail");
}

int ref_restrict_residual(fx_ctx *ctx, const double *u, const double *rhs, size_t rows, size_t cols, const StencilP &P,
                          const BcP &B, double *coarse_rhs, double *coarse_u, size_t crows, size_t ccols) {
    return launch_rows(ctx, crows, ccols,
                       RefRestrict{u, rhs, coarse_rhs, coarse_u, P, B, (int)rows, (int)cols, (int)ccols},
                       "ref_restrict_residual");
}

}  // namespace fx
