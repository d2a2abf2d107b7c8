// fx_explicit.cu -- explicit diffusion steps (solver.rs:344-495) as fused passes: forward Euler, Heun
// and classical RK4 of du/dt = alpha Lap u with homogeneous Dirichlet sides.
//
// The reference's step is a sequence of field operations (a Runge-Kutta 4 step: 22 launches that
// move about 400 B/point).  Here a pass reads u once and writes the result of up to four stencil
// stages -- one RK4 step, two Heun steps or four Euler steps -- 16 B/point: a warp marches a strip of
// 64 columns (56 of its own, a halo of one per stage) with two columns per lane, as the multigrid's
// level passes do (fx_wcycle.cuh), stage s working s rows behind the row that arrives.  A stage's last
// rows stay in registers (the march is unrolled by six, so every window is a constant), outer
// neighbours come by shuffle, the rows ahead by cp.async.  Every value is the expression of the field
// operations, so a step equals theirs bit for bit.
//
// u and a scratch field take turns; an odd number of passes ends with a copy.
//
// Measured at 1537 x 2050, ten RK4 steps: 1902 us as field operations, 224 us in passes, bound by the
// FP64 latency of the four stages (12 warps per SM); the vectors are in L2.
#include "fx_cdcycle.cuh"

using namespace fx;

FX_CHECK_FILE(explicit);

namespace {

constexpr int kExWarps = 4;
constexpr int kExOwn = 56;   // own columns: lanes 2 .. 29 (a halo of up to 4)
constexpr int kExRing = 6, kExAhead = 5;

enum { kEuler = 0, kHeun = 1, kRk4 = 2 };

struct ExCoef {
    double c, n, s, w, e;       // stencil weights
    double h1, h2, c1, c2;      // Euler / Heun: h1 = dt alpha; RK4: h1 = dt alpha / 2, h2 = dt alpha, c1 = dt alpha / 6, c2 = 2 c1
};

__device__ __forceinline__ double ex_stencil(const ExCoef &P, double c, double n, double s, double w, double e) {
    return fma(P.c, c, fma(P.n, n, fma(P.s, s, fma(P.w, w, P.e * e))));
}

// ST stencil stages of the scheme (RK4: 4, Heun: 2 per step, Euler: 1 per step)
template <int SCHEME, int ST>
__global__ void __launch_bounds__(kExWarps * 32, 3) k_explicit(StripGeom G, ExCoef P, const double *__restrict__ u,
                                                               double *__restrict__ out) {
    grid_dep_enter();
    __shared__ __align__(16) double ring[kExWarps][kExRing * 64];
    constexpr int R = kExRing;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int item = blockIdx.x * kExWarps + wid;
    if (item >= G.nitems) return;  // whole warps
    const int strip = item % G.nstrips;
    const int rows = G.rows, cols = G.cols;
    const int r0 = item / G.nstrips * G.chunk_rows, r1 = min(r0 + G.chunk_rows, rows);
    const int ca = strip * kExOwn - 4 + 2 * lane, cb = ca + 1;
    const bool ga = ca >= 0 && ca < cols, gb = cb >= 0 && cb < cols;                      // in the grid
    const bool ina = ca >= 1 && ca <= cols - 2, inb = cb >= 1 && cb <= cols - 2;          // inside its ring
    const bool own = lane >= 2 && lane < 30;
    const long long nf = (long long)rows * cols;
    (void)nf;
    // step q: row q of u arrives, stage s is computed on row q - s; rows [r0, r1) of the last are written
    const int q_first = r0 - ST, q_last = r1 - 1 + ST;
    const double *const su = ring[wid] + 2 * lane;
    long long og = (long long)q_first * cols + ca;
    const double *pu = u + og;
    double *const ru = ring[wid] + 2 * lane;
    auto put = [&](int slot, int q) {
        const bool rv = q >= 0 && q < rows && q <= q_last;
        cp_async_elem(ru + slot * 64, pu, rv && ga && FX_IN(og, nf), u);
        cp_async_elem(ru + slot * 64 + 1, pu + 1, rv && gb && FX_IN(og + 1, nf), u);
        cp_async_commit();
        pu += cols;
        og += cols;
    };
#pragma unroll
    for (int k = 0; k < kExAhead; k++) put(k, q_first + k);
    // v[s]: the field stage s + 1 reads (v[0] = u); d[s]: RK4's stage derivative k_s
    double va[ST][R] = {}, vb[ST][R] = {}, da[4][R] = {}, db[4][R] = {};
    long long oo = (long long)(q_first - ST) * cols + ca;
    double *po = out + oo;
    auto step = [&](int k, int q, auto fast) {
        constexpr bool F = decltype(fast)::value;  // every stage's row is inside the grid's ring
        {
            cp_async_wait<kExAhead - 1>();
            const Pair<double> x = lds2(su + k * 64);
            va[0][k] = x.a;
            vb[0][k] = x.b;
            put((k + kExAhead) % R, q + kExAhead);
        }
#pragma unroll
        for (int s = 1; s <= ST; s++) {
            const int r = q - s;  // this stage's row
            const int m = (k + 2 * R - s) % R, mn = (m + R - 1) % R, ms = (m + 1) % R;  // slots of rows r, r - 1, r + 1
            const double xa = va[s - 1][m], xb = vb[s - 1][m];
            const double wa = shfl_w(xb), eb = shfl_e(xa);
            const bool rin = F || (r >= 1 && r <= rows - 2);
            const bool pa = rin && ina, pb = rin && inb;
            const double ka = ex_stencil(P, xa, va[s - 1][mn], va[s - 1][ms], wa, xb);
            const double kb = ex_stencil(P, xb, vb[s - 1][mn], vb[s - 1][ms], xa, eb);
            double ra, rb;  // the field after this stage
            if constexpr (SCHEME == kEuler) {
                ra = pa ? fma(P.h1, ka, xa) : xa;
                rb = pb ? fma(P.h1, kb, xb) : xb;
            } else if constexpr (SCHEME == kHeun) {
                ra = pa ? fma(P.h1, ka, xa) : xa;
                rb = pb ? fma(P.h1, kb, xb) : xb;
                if ((s & 1) == 0) {  // the second Euler step averaged with the step's start
                    constexpr int kZero = 0;
                    const int b0 = s >= 2 ? s - 2 : kZero;
                    ra = fma(1.0, va[b0][m], ra) * 0.5;
                    rb = fma(1.0, vb[b0][m], rb) * 0.5;
                }
            } else {
                const double ua = va[0][m], ub = vb[0][m];  // u at the row
                const double za = pa ? ka : 0.0, zb = pb ? kb : 0.0;  // the derivative, 0 on the ring
                if (s < 4) {
                    da[s - 1][m] = za;
                    db[s - 1][m] = zb;
                    // u + h k inside; the first stage keeps the ring, the later ones zero it
                    const double h = s == 3 ? P.h2 : P.h1;
                    ra = pa ? fma(h, ka, ua) : (s == 1 ? ua : 0.0);
                    rb = pb ? fma(h, kb, ub) : (s == 1 ? ub : 0.0);
                } else {
                    ra = fma(P.c1, za, fma(P.c2, da[2][m], fma(P.c2, da[1][m], fma(P.c1, da[0][m], ua))));
                    rb = fma(P.c1, zb, fma(P.c2, db[2][m], fma(P.c2, db[1][m], fma(P.c1, db[0][m], ub))));
                }
            }
            if (s < ST) {
                va[s][m] = ra;
                vb[s][m] = rb;
            } else {
                if (r >= r0 && r < r1) {  // uniform over the warp
                    if (own && ga && FX_IN(oo, nf)) po[0] = ra;
                    if (own && gb && FX_IN(oo + 1, nf)) po[1] = rb;
                }
                po += cols;
                oo += cols;
            }
        }
    };
    for (int qb = q_first; qb <= q_last; qb += R) {
        if (qb - ST >= 1 && min(qb + R - 1, q_last) <= rows - 2) {
#pragma unroll
            for (int k = 0; k < R; k++) {
                if (qb + k > q_last) break;  // uniform over the warp
                step(k, qb + k, fast_t<true>{});
            }
        } else {
#pragma unroll
            for (int k = 0; k < R; k++) {
                if (qb + k > q_last) break;
                step(k, qb + k, fast_t<false>{});
            }
        }
    }
    cp_async_wait<0>();  // no copy outlives the warp
}

template <int SCHEME, int ST>
int launch_explicit(fx_ctx *ctx, size_t rows, size_t cols, const ExCoef &P, const double *u, double *out) {
    static std::atomic<int> occ{0};
    const long cap = (long)band_capacity(ctx, k_explicit<SCHEME, ST>, occ, kExWarps * 32) * kExWarps;
    const StripGeom G = strip_geom(rows, cols + 1, kExOwn, cap);  // own ranges tile all columns
    StripGeom H = G;
    H.cols = (int)cols;
    timing_pre(ctx, "explicit_step");
    launch_pdl(ctx, k_explicit<SCHEME, ST>, (G.nitems + kExWarps - 1) / kExWarps, kExWarps * 32, 0, H, P, u, out);
    timing_post(ctx, (double)rows * (double)cols, (double)rows * (double)cols * 16.0);
    return check_launch(ctx, "explicit_step");
}

// `steps` steps of the scheme in one pass
int explicit_pass(fx_ctx *ctx, int scheme, int steps, size_t rows, size_t cols, const ExCoef &P, const double *u, double *out) {
    if (scheme == kRk4) return launch_explicit<kRk4, 4>(ctx, rows, cols, P, u, out);
    if (scheme == kHeun)
        return steps == 1 ? launch_explicit<kHeun, 2>(ctx, rows, cols, P, u, out)
                          : launch_explicit<kHeun, 4>(ctx, rows, cols, P, u, out);
    switch (steps) {
        case 1: return launch_explicit<kEuler, 1>(ctx, rows, cols, P, u, out);
        case 2: return launch_explicit<kEuler, 2>(ctx, rows, cols, P, u, out);
        case 3: return launch_explicit<kEuler, 3>(ctx, rows, cols, P, u, out);
        default: return launch_explicit<kEuler, 4>(ctx, rows, cols, P, u, out);
    }
}

}  // namespace

extern "C" {

int fx_diffusion_steps(fx_ctx *ctx, fx_buf *u, fx_buf *scratch, const fx_grid *g, const fx_stencil *s, double alpha,
                       double dt, int scheme, size_t nsteps) {
    if (!ctx) return fail(FX_ERR_INVALID_ARGUMENT, "null context");
    FX_TRY(check_grid(g));
    FX_TRY(check_buf(u, "u"));
    FX_TRY(check_buf(scratch, "scratch"));
    FX_TRY(check_grid_len(g, u));
    FX_TRY(check_same(u, scratch));
    if (u->ptr == scratch->ptr) return fail(FX_ERR_INVALID_ARGUMENT, "u and scratch must be distinct buffers");
    if (u->dtype != FX_F64) return fail(FX_ERR_UNSUPPORTED, "explicit steps need F64 fields");
    if (scheme < kEuler || scheme > kRk4) return fail(FX_ERR_INVALID_ARGUMENT, "unknown time scheme");
    StencilP S;
    FX_TRY(make_stencil(s, &S));
    if (S.mode != 5) return fail(FX_ERR_UNSUPPORTED, "explicit steps need a five-point stencil");
    ExCoef P{S.c, S.n, S.s, S.w, S.e, 0, 0, 0, 0};
    if (scheme == kRk4) {
        P.h1 = 0.5 * dt * alpha;
        P.h2 = dt * alpha;
        P.c1 = dt * alpha / 6.0;
        P.c2 = 2.0 * P.c1;
    } else {
        P.h1 = dt * alpha;
    }
    const size_t most = scheme == kEuler ? 4 : (scheme == kHeun ? 2 : 1);  // steps a pass can hold
    double *buf[2] = {(double *)u->ptr, (double *)scratch->ptr};
    size_t passes = (nsteps + most - 1) / most;
    if ((passes & 1) && passes < nsteps) passes++;  // end in u where the steps can be split so
    for (size_t p = 0; p < passes; p++) {
        const size_t a = nsteps * p / passes, b = nsteps * (p + 1) / passes;
        FX_TRY(explicit_pass(ctx, scheme, (int)(b - a), g->rows, g->cols, P, buf[p & 1], buf[(p + 1) & 1]));
    }
    if (passes & 1) return fx_copy(ctx, scratch, u);
    return FX_OK;
}

}  // extern "C"
