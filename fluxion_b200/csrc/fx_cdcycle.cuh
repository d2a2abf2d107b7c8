// fx_cdcycle.cuh -- fused level passes of the convection-diffusion V(2,2)-cycle (scalar kappa), one
// warp per strip, for the single-problem cycle (fx_solvers.cu) and the batch (fx_batch.cu).
//
// With a zero initial guess and two sweeps on each leg a level is two passes instead of seven:
//
//   down: from the rhs b alone, x1 = omega b / d, x2 = x1 + omega (b - A x1) / d, the residual
//         b - A x2 and its full weighting -- reads b, vx, vy, writes x2 and a quarter of a coarse
//         rhs (34 B/point in FP64; the sweep pair, residual, restriction and zero-fills it
//         replaces moved 98);
//   up:   f = x2 + bilinear(e), x3 = f + omega (b - A f) / d, z = x3 + omega (b - A x3) / d --
//         reads x2, b, vx, vy and a quarter of e, writes z (42 B/point, from 66).
//
// Both march strips as k_wdown / k_wup do (fx_wcycle.cuh): a lane holds two adjacent columns' last
// three rows of every stage in registers, the outer west / east neighbours come by shuffle.  The
// coefficients would not fit beside them: b, vx and vy of a row are needed at up to three stages,
// so their rows stay in a six-row ring of shared memory per warp -- three rows in flight by
// cp.async ahead of the march, three behind -- and each stage reads its row from there (16 bytes a
// lane).  The march is unrolled by six rows, so every ring slot is a constant.  1 / d is computed
// once per point and pass (an IEEE division) and kept in registers for the next row's stage.
//
// An FP32 cycle reads the FP64 vector r and writes the FP64 vector z at level 0 directly (TB, TZ).
// Every point value is the expression of FlatCdSweep / FlatCdResid and the transfers, so the cycle
// equals the unfused one bit for bit.
//
// Measured on a whole cycle, FP64 / FP32, levels of up to 300000 points by tiles (below): 4097 x 4097
// 448 / 354 us (separate passes: 1066 / 861), 1025 x 1025 98 / 75 (206 / 185), 65 x 65 46 / 30 (90 / 77).  The
// level-0 passes of 4097 x 4097 move 76 B/point in FP64, down at 0.63 and up at 0.79 of the copy rate;
// they are bound by the latency of a step (three dependent stages of ten FP64 operations after a
// division) at 16 and 12 warps per SM.
#pragma once

#include "fx_points.cuh"
#include "fx_wcycle.cuh"

FX_CHECK_FILE(cdcycle);

namespace fx {

__device__ __forceinline__ bool sign_bit(double v) { return __double2hiint(v) < 0; }
__device__ __forceinline__ bool sign_bit(float v) { return __float_as_int(v) < 0; }
__device__ __forceinline__ double fx_abs(double v) { return fabs(v); }
__device__ __forceinline__ float fx_abs(float v) { return fabsf(v); }

// The operator of a level with scalar kappa: A v = sigma v + coeff (kappa Lap v + v.grad v).
template <typename T>
struct CdOp {
    ConvDiffC<T> K;
    T sigma, coeff, kap;
    // conv_diff_at's value with fewer instructions: the upwind difference of either sign of v enters
    // as |v| times (c - upwind neighbour) / h, since (e - c) = -(c - e) and every rounding is
    // symmetric in sign; the side is picked by the sign bit (at v = -0 it may be the other side,
    // whose term is a zero as well).
    __device__ __forceinline__ T apply(T c, T n, T s, T w, T e, T vx, T vy) const {
        const T lap = fx_fma(w + e, K.inv_dx2, (n + s) * K.inv_dy2) - K.k2 * c;
        const T dx = (c - (sign_bit(vx) ? e : w)) * K.inv_dx;
        const T dy = (c - (sign_bit(vy) ? s : n)) * K.inv_dy;
        const T conv = fx_fma(fx_abs(vx), dx, fx_abs(vy) * dy);
        return fx_fma(coeff, kap * lap + conv, sigma * c);
    }
    __device__ __forceinline__ T inv_diag(T vx, T vy) const {
        return (T)1 / fx_fma(coeff, fx_fma(-kap, K.k2, fx_fma(fabs(vx), K.inv_dx, fabs(vy) * K.inv_dy)), sigma);
    }
};

// One level of one problem.
template <typename T, typename TB, typename TZ>
struct CdLevelArgs {
    int rows, cols, ccols;
    CdOp<T> A;
    T omega;
    const TB *b;
    const T *vx, *vy;
    T *x2;       // down writes, up reads
    T *crhs;     // down: the coarse rhs (interior)
    const T *e;  // up: the coarse correction
    TZ *z;       // up
};

constexpr int kCdRing = 6;               // ring rows: 3 ahead, the row, 2 behind
constexpr int kCdAhead = 3;
constexpr int kCdOwnDown = kDownOwn;     // 56 own columns of 64: halo 4
constexpr int kCdOwnUp = kUpOwn;         // 60: halo 2
static_assert(kStripUnroll == kCdRing, "ring slots are unroll positions");

// cp.async of a lane's two adjacent elements, `na` / `nb` bytes of each read (0: zero-filled, nothing
// read); the second one's offsets are immediates.
template <typename E>
__device__ __forceinline__ void cp_async_pair(unsigned dst, const E *src, int na, int nb) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;\n" ::"r"(dst), "l"(src), "n"((int)sizeof(E)), "r"(na) : "memory");
    asm volatile("cp.async.ca.shared.global [%0+%2], [%1+%2], %2, %3;\n" ::"r"(dst), "l"(src), "n"((int)sizeof(E)), "r"(nb)
                 : "memory");
}

// A strip's rows of one array on their way to the ring: the address of this lane's column pair in
// the row being fetched (clamped into the row, so that it is valid where nothing is read), and the
// lane's place in ring slot 0.
template <typename E>
struct RingSrc {
    const E *p, *any;
    unsigned dst;
    int na, nb;  // bytes read of each column
    __device__ __forceinline__ void init(const E *base, int cols, int q, int ca, bool ina, bool inb, E *slot0) {
        const int cc = min(max(ca, 0), cols - 2);
        p = base + ((long long)q * cols + cc);
        any = base;
        dst = (unsigned)__cvta_generic_to_shared(slot0);
        na = ina ? (int)sizeof(E) : 0;
        nb = inb ? (int)sizeof(E) : 0;
    }
    // the row into ring slot `slot`; rv: it is one to read (oa, ob: its columns' checks)
    template <bool FAST>
    __device__ __forceinline__ void put(int slot, bool rv, bool oa, bool ob, int cols) {
        const unsigned d = dst + slot * 64 * (unsigned)sizeof(E);
        if constexpr (FAST) cp_async_pair(d, p, oa ? na : 0, ob ? nb : 0);
        else cp_async_pair(d, rv ? p : any, rv && oa ? na : 0, rv && ob ? nb : 0);
        p += cols;
    }
};

template <typename T>
struct Pair {
    T a, b;
};
template <typename T>
__device__ __forceinline__ Pair<T> lds2(const T *p) {  // p: an even element
    if constexpr (sizeof(T) == 8) {
        const double2 v = *reinterpret_cast<const double2 *>(p);
        return Pair<T>{v.x, v.y};
    } else {
        const float2 v = *reinterpret_cast<const float2 *>(p);
        return Pair<T>{v.x, v.y};
    }
}

// shared memory per warp
template <typename T, typename TB>
__host__ __device__ constexpr size_t cd_down_warp_smem() { return kCdRing * 64 * (sizeof(TB) + 2 * sizeof(T)); }
template <typename T, typename TB>
__host__ __device__ constexpr size_t cd_up_warp_smem() { return kCdRing * 64 * (sizeof(TB) + 3 * sizeof(T)); }

// Warp over strip `strip`, fine rows [r0, r1), r0 even.
template <typename T, typename TB, typename TZ>
__device__ __forceinline__ void cd_down_strip(const CdLevelArgs<T, TB, TZ> &L, int strip, int r0, int r1,
                                              unsigned char *smem) {
    constexpr int R = kCdRing;
    const int lane = threadIdx.x & 31;
    const int rows = L.rows, cols = L.cols;
    const int ca = strip * kCdOwnDown - 4 + 2 * lane, cb = ca + 1;
    const bool ina = ca >= 1 && ca <= cols - 2, inb = cb >= 1 && cb <= cols - 2;
    const bool own = lane >= 2 && lane < 30;
    const bool sta = own && ina, stb = own && inb;
    const bool cpt = own && ca >= 2 && ca <= cols - 3;  // coarse point (fr, ca) for even fr
    const long long nf = (long long)rows * cols, nc = (long long)((rows - 1) / 2 + 1) * L.ccols;
    (void)nf;
    (void)nc;
    TB *const sb = reinterpret_cast<TB *>(smem) + 2 * lane;
    T *const sx = reinterpret_cast<T *>(smem + R * 64 * sizeof(TB)) + 2 * lane;
    T *const sy = sx + R * 64;
    // step q: b, vx, vy row q arrive, x1 row q; x2 row q-1; residual row q-2; full weighting of fine
    // row q-3 (even q-3 only)
    const int q_first = r0 - 3, q_last = r1 + 2;
    auto row_in = [&](int r) { return r >= 1 && r <= rows - 2; };
    // steps with every row test true
    const int q_lo = max(r0, 2) + 3, q_hi = min(rows - 2, q_last) - kCdAhead;
    RingSrc<TB> gb;
    RingSrc<T> gx, gy;
    gb.init(L.b, cols, q_first, ca, ina, inb, sb);
    gx.init(L.vx, cols, q_first, ca, ina, inb, sx);
    gy.init(L.vy, cols, q_first, ca, ina, inb, sy);
    long long og = (long long)q_first * cols + ca;  // the row being fetched
    auto put = [&](int slot, int q, auto fast) {
        constexpr bool F = decltype(fast)::value;
        const bool rv = F || (row_in(q) && q <= q_last);
        const bool oa = !(rv && ina) || FX_IN(og, nf), ok = !(rv && inb) || FX_IN(og + 1, nf);
        gb.template put<F>(slot, rv, oa, ok, cols);
        gx.template put<F>(slot, rv, oa, ok, cols);
        gy.template put<F>(slot, rv, oa, ok, cols);
        cp_async_commit();
        og += cols;
    };
#pragma unroll
    for (int k = 0; k < kCdAhead; k++) put(k, q_first + k, fast_t<false>{});

    T x1a[3] = {}, x1b[3] = {}, x2a[3] = {}, x2b[3] = {};
    T rsa[3] = {}, rsb[3] = {}, rwa[3] = {};
    T ida = (T)0, idb = (T)0;  // 1 / d of row q - 1
    long long ox = (long long)(q_first - 1) * cols + ca;         // the x2 row being stored
    long long oc = (long long)((q_first - 3) >> 1) * L.ccols + (ca >> 1);  // q_first - 3 even
    auto step = [&](int k, int q, auto fast) {
        constexpr bool F = decltype(fast)::value;
        const int s0 = k % 3, s1 = (k + 2) % 3, s2 = (k + 1) % 3;  // register slots of rows q, q-1, q-2
        const int m0 = k, m1 = (k + R - 1) % R, m2 = (k + R - 2) % R;  // ring slots of rows q, q-1, q-2
        T ca_id, cb_id;
        // row q: x1 = omega b / d (0 on the ring); refill with row q + 3 (over row q - 3)
        {
            cp_async_wait<kCdAhead - 1>();
            const Pair<TB> b = lds2(sb + m0 * 64);
            const Pair<T> vx = lds2(sx + m0 * 64), vy = lds2(sy + m0 * 64);
            const bool rin = F || row_in(q);
            ca_id = L.A.inv_diag(vx.a, vy.a);
            cb_id = L.A.inv_diag(vx.b, vy.b);
            x1a[s0] = (rin && ina) ? fx_fma(L.omega, (T)b.a * ca_id, (T)0) : (T)0;
            x1b[s0] = (rin && inb) ? fx_fma(L.omega, (T)b.b * cb_id, (T)0) : (T)0;
            put((k + kCdAhead) % R, q + kCdAhead, fast_t<F>{});
        }
        // row q-1: x2
        {
            const T xa = x1a[s1], xb = x1b[s1];
            const T wa = shfl_w(xb), eb = shfl_e(xa);
            const bool rin = F || row_in(q - 1);
            const Pair<TB> b = lds2(sb + m1 * 64);
            const Pair<T> vx = lds2(sx + m1 * 64), vy = lds2(sy + m1 * 64);
            T va = (T)0, vb = (T)0;
            if (rin && ina) va = fx_fma(L.omega, ((T)b.a - L.A.apply(xa, x1a[s2], x1a[s0], wa, xb, vx.a, vy.a)) * ida, xa);
            if (rin && inb) vb = fx_fma(L.omega, ((T)b.b - L.A.apply(xb, x1b[s2], x1b[s0], xa, eb, vx.b, vy.b)) * idb, xb);
            x2a[s1] = va;
            x2b[s1] = vb;
            if (F || (rin && q - 1 >= r0 && q - 1 < r1)) {
                if (sta && FX_IN(ox, nf)) L.x2[ox] = va;
                if (stb && FX_IN(ox + 1, nf)) L.x2[ox + 1] = vb;
            }
            ox += cols;
            ida = ca_id;
            idb = cb_id;
        }
        // row q-2: residual, and the residual west of ca for the restriction
        {
            const T xa = x2a[s2], xb = x2b[s2];
            const T wa = shfl_w(xb), eb = shfl_e(xa);
            const bool rin = F || row_in(q - 2);
            const Pair<TB> b = lds2(sb + m2 * 64);
            const Pair<T> vx = lds2(sx + m2 * 64), vy = lds2(sy + m2 * 64);
            T va = (T)0, vb = (T)0;
            if (rin && ina) va = (T)b.a - L.A.apply(xa, x2a[s0], x2a[s1], wa, xb, vx.a, vy.a);
            if (rin && inb) vb = (T)b.b - L.A.apply(xb, x2b[s0], x2b[s1], xa, eb, vx.b, vy.b);
            rsa[s2] = va;
            rsb[s2] = vb;
            rwa[s2] = shfl_w(vb);
        }
        // fine row q-3: full weighting onto coarse row (q-3) / 2 at coarse column ca / 2
        if (!(k & 1)) {  // q - 3 even (r0 even, so q_first odd)
            const int fr = q - 3;
            if (cpt && (F || (fr >= r0 && fr < r1 && fr >= 2 && fr <= rows - 3)) && FX_IN(oc, nc)) {
                const T e = (rsa[s1] + rsa[s2]) + (rwa[s0] + rsb[s0]);
                const T d = (rwa[s1] + rsb[s1]) + (rwa[s2] + rsb[s2]);
                L.crhs[oc] = ((T)4 * rsa[s0] + ((T)2 * e + d)) * (T)0.0625;
            }
            oc += L.ccols;
        }
    };
    for (int qb = q_first; qb <= q_last; qb += R) {
        if (qb >= q_lo && qb + R - 1 <= q_hi) {
#pragma unroll
            for (int k = 0; k < R; k++) step(k, qb + k, fast_t<true>{});
        } else {
#pragma unroll
            for (int k = 0; k < R; k++) {
                if (qb + k > q_last) break;  // uniform over the warp
                step(k, qb + k, fast_t<false>{});
            }
        }
    }
    cp_async_wait<0>();  // no copy outlives the warp
}

template <typename T, typename TB, typename TZ>
__device__ __forceinline__ void cd_up_strip(const CdLevelArgs<T, TB, TZ> &L, int strip, int nstrips, int r0, int r1,
                                            bool zero_ring, unsigned char *smem) {
    constexpr int R = kCdRing;
    const int lane = threadIdx.x & 31;
    const int rows = L.rows, cols = L.cols, ccols = L.ccols, crows = (rows - 1) / 2 + 1;
    const int ca = strip * kCdOwnUp - 2 + 2 * lane, cb = ca + 1;
    const bool ina = ca >= 1 && ca <= cols - 2, inb = cb >= 1 && cb <= cols - 2;
    const bool own = lane >= 1 && lane < 31;
    const bool sta = own && ina, stb = own && inb;
    const int kc = ca >> 1;  // coarse column of ca; cb interpolates between kc and kc + 1
    const bool ce0 = kc >= 0 && kc < ccols && (ina || inb), ce1 = kc + 1 < ccols && inb;
    const long long nf = (long long)rows * cols, nc = (long long)crows * ccols;
    (void)nf;
    (void)nc;
    TB *const sb = reinterpret_cast<TB *>(smem) + 2 * lane;
    T *const sx = reinterpret_cast<T *>(smem + R * 64 * sizeof(TB)) + 2 * lane;
    T *const sy = sx + R * 64, *const su = sy + R * 64;
    // step q: f row q = x2 + P e; x3 row q-1; z row q-2
    const int q_first = r0 - 2, q_last = r1 + 1;  // q_first even
    const int q_lo = max(r0, 1) + 2, q_hi = min(rows - 2, q_last) - kCdAhead;
    const int m_last = (q_last >> 1) + 1;  // last coarse row any step reads
    auto row_in = [&](int r) { return r >= 1 && r <= rows - 2; };
    RingSrc<TB> gb;
    RingSrc<T> gu, gx, gy;
    gu.init(L.x2, cols, q_first, ca, ina, inb, su);
    gb.init(L.b, cols, q_first, ca, ina, inb, sb);
    gx.init(L.vx, cols, q_first, ca, ina, inb, sx);
    gy.init(L.vy, cols, q_first, ca, ina, inb, sy);
    long long og = (long long)q_first * cols + ca;  // the row being fetched
    auto put = [&](int slot, int q, auto fast) {
        constexpr bool F = decltype(fast)::value;
        const bool rv = F || (row_in(q) && q <= q_last);
        const bool oa = !(rv && ina) || FX_IN(og, nf), ok = !(rv && inb) || FX_IN(og + 1, nf);
        gu.template put<F>(slot, rv, oa, ok, cols);
        gb.template put<F>(slot, rv, oa, ok, cols);
        gx.template put<F>(slot, rv, oa, ok, cols);
        gy.template put<F>(slot, rv, oa, ok, cols);
        cp_async_commit();
        og += cols;
    };
    // coarse rows of the unrolled step's row pairs, R rows ahead
    T ea_[R / 2], eb_[R / 2];
    auto load_coarse = [&](int m, T &v0, T &v1, long long o) {
        v0 = (T)0;
        v1 = (T)0;
        if (m >= 0 && m < crows && m <= m_last) {
            if (ce0 && FX_IN(o, nc)) v0 = L.e[o];
            if (ce1 && FX_IN(o + 1, nc)) v1 = L.e[o + 1];
        }
    };
    T c0a, c0b;  // coarse row q >> 1 of the current pair, columns kc, kc + 1
#pragma unroll
    for (int k = 0; k < kCdAhead; k++) put(k, q_first + k, fast_t<false>{});
    load_coarse(q_first >> 1, c0a, c0b, (long long)(q_first >> 1) * ccols + kc);
#pragma unroll
    for (int k = 0; k < R; k += 2) {
        const int m = ((q_first + k) >> 1) + 1;
        load_coarse(m, ea_[k / 2], eb_[k / 2], (long long)m * ccols + kc);
    }
    long long oe = (long long)((q_first + R + 2) >> 1) * ccols + kc;
    long long oz = (long long)(q_first - 2) * cols + ca;
    T fa[3] = {}, fb[3] = {}, x3a[3] = {}, x3b[3] = {};
    T ida = (T)0, idb = (T)0;  // 1 / d of row q - 2
    auto step = [&](int k, int q, auto fast) {
        constexpr bool F = decltype(fast)::value;
        const int s0 = k % 3, s1 = (k + 2) % 3, s2 = (k + 1) % 3;
        const int m0 = k, m1 = (k + R - 1) % R, m2 = (k + R - 2) % R;
        // row q: f = x2 + bilinear(e); the parities are fixed: ca even, cb odd, q odd <=> k odd
        {
            const bool ro = k & 1;
            const T e00 = c0a, e01 = c0b;                // coarse row q >> 1
            const T e10 = ea_[k / 2], e11 = eb_[k / 2];  // coarse row (q >> 1) + 1
            T pa, pb;
            if (ro) {
                pa = (T)0.5 * (e00 + e10);
                pb = (T)0.25 * ((e00 + e10) + (e01 + e11));
            } else {
                pa = e00;
                pb = (T)0.5 * (e00 + e01);
            }
            const bool rin = F || row_in(q);
            cp_async_wait<kCdAhead - 1>();
            const Pair<T> u = lds2(su + m0 * 64);
            fa[s0] = (rin && ina) ? u.a + pa : (T)0;
            fb[s0] = (rin && inb) ? u.b + pb : (T)0;
            if (ro) {  // the pair is done: its lower coarse row becomes the upper one
                c0a = e10;
                c0b = e11;
                load_coarse((q + R + 1) >> 1, ea_[k / 2], eb_[k / 2], oe);
                oe += ccols;
            }
            put((k + kCdAhead) % R, q + kCdAhead, fast_t<F>{});
        }
        // row q-2's 1 / d is kept in ida / idb; row q-1's is computed here for both of its stages
        T na, nb_;
        // row q-1: x3
        {
            const T xa = fa[s1], xb = fb[s1];
            const T wa = shfl_w(xb), eb = shfl_e(xa);
            const bool rin = F || row_in(q - 1);
            const Pair<TB> b = lds2(sb + m1 * 64);
            const Pair<T> vx = lds2(sx + m1 * 64), vy = lds2(sy + m1 * 64);
            na = L.A.inv_diag(vx.a, vy.a);
            nb_ = L.A.inv_diag(vx.b, vy.b);
            T va = (T)0, vb = (T)0;
            if (rin && ina) va = fx_fma(L.omega, ((T)b.a - L.A.apply(xa, fa[s2], fa[s0], wa, xb, vx.a, vy.a)) * na, xa);
            if (rin && inb) vb = fx_fma(L.omega, ((T)b.b - L.A.apply(xb, fb[s2], fb[s0], xa, eb, vx.b, vy.b)) * nb_, xb);
            x3a[s1] = va;
            x3b[s1] = vb;
        }
        // row q-2: z
        {
            const T xa = x3a[s2], xb = x3b[s2];
            const T wa = shfl_w(xb), eb = shfl_e(xa);
            const int r = q - 2;
            if (F || (row_in(r) && r >= r0 && r < r1)) {
                const Pair<TB> b = lds2(sb + m2 * 64);
                const Pair<T> vx = lds2(sx + m2 * 64), vy = lds2(sy + m2 * 64);
                const T va = fx_fma(L.omega, ((T)b.a - L.A.apply(xa, x3a[s0], x3a[s1], wa, xb, vx.a, vy.a)) * ida, xa);
                const T vb = fx_fma(L.omega, ((T)b.b - L.A.apply(xb, x3b[s0], x3b[s1], xa, eb, vx.b, vy.b)) * idb, xb);
                if (sta && FX_IN(oz, nf)) L.z[oz] = (TZ)va;
                if (stb && FX_IN(oz + 1, nf)) L.z[oz + 1] = (TZ)vb;
            }
            oz += cols;
            ida = na;
            idb = nb_;
        }
    };
    for (int qb = q_first; qb <= q_last; qb += R) {
        if (qb >= q_lo && qb + R - 1 <= q_hi) {
#pragma unroll
            for (int k = 0; k < R; k++) step(k, qb + k, fast_t<true>{});
        } else {
#pragma unroll
            for (int k = 0; k < R; k++) {
                if (qb + k > q_last) break;
                step(k, qb + k, fast_t<false>{});
            }
        }
    }
    cp_async_wait<0>();  // no copy outlives the warp
    if (zero_ring) {  // this warp's part of z's ring
        if (strip == 0)
            for (int r = r0 + lane; r < r1; r += 32)
                if (FX_IN((long long)r * cols, nf)) L.z[(size_t)r * cols] = (TZ)0;
        if (strip == nstrips - 1)
            for (int r = r0 + lane; r < r1; r += 32)
                if (FX_IN((long long)r * cols + cols - 1, nf)) L.z[(size_t)r * cols + cols - 1] = (TZ)0;
        for (int r = r0 == 0 ? 0 : rows - 1; r < r1; r += rows - 1) {
            const long long o = (long long)r * cols + ca;
            if (own && ca >= 0 && ca < cols && FX_IN(o, nf)) L.z[o] = (TZ)0;
            if (own && cb >= 0 && cb < cols && FX_IN(o + 1, nf)) L.z[o + 1] = (TZ)0;
        }
    }
}

// ---------------------------------------------------------------- one problem

// resident blocks per SM asked of the compiler.  More of them is slower (FP64 cycle at 4097 x 4097 by
// strips: 489 us with 3, 500 with 4 at 128 registers): the chunks get shorter, and the unrolled march is
// larger than a scheduler's instruction cache, so warps at different rows evict each other's
// instructions.  For the same reason there is no third variant of the step without column masks
// (528 us).
template <typename T>
__host__ __device__ constexpr int cd_minb() { return sizeof(T) == 8 ? 3 : 5; }
constexpr int kCdWarps = 4;

template <typename T, typename TB, typename TZ>
__global__ void __launch_bounds__(kCdWarps * 32, cd_minb<T>()) k_cd_down(StripGeom G, CdLevelArgs<T, TB, TZ> L,
                                                                         const int *skip) {
    grid_dep_enter();
    if (skip && *(volatile const int *)skip) return;
    extern __shared__ __align__(16) unsigned char cd_smem[];
    const int item = blockIdx.x * kCdWarps + (threadIdx.x >> 5);
    if (item >= G.nitems) return;  // whole warps
    const int strip = item % G.nstrips, r0 = item / G.nstrips * G.chunk_rows;
    cd_down_strip(L, strip, r0, min(r0 + G.chunk_rows, G.rows), cd_smem + (threadIdx.x >> 5) * cd_down_warp_smem<T, TB>());
}

template <typename T, typename TB, typename TZ>
__global__ void __launch_bounds__(kCdWarps * 32, cd_minb<T>()) k_cd_up(StripGeom G, CdLevelArgs<T, TB, TZ> L,
                                                                       int zero_ring, const int *skip) {
    grid_dep_enter();
    if (skip && *(volatile const int *)skip) return;
    extern __shared__ __align__(16) unsigned char cd_smem[];
    const int item = blockIdx.x * kCdWarps + (threadIdx.x >> 5);
    if (item >= G.nitems) return;
    const int strip = item % G.nstrips, r0 = item / G.nstrips * G.chunk_rows;
    cd_up_strip(L, strip, G.nstrips, r0, min(r0 + G.chunk_rows, G.rows), zero_ring != 0,
                cd_smem + (threadIdx.x >> 5) * cd_up_warp_smem<T, TB>());
}

// ---------------------------------------------------------------- small levels
//
// A level with fewer strip chunks than the GPU has warps is pure latency: a march takes seven or
// more steps of some 1400 cycles (a copy that arrives, two shuffles and three chains of dependent
// operations each).  Here a block of 16 x 16 own points holds its halo too, one point per thread:
// one load of everything, then a barrier per stage.  The halo is recomputed (22^2 points down, 20^2
// up, for 256), which a level that leaves SMs idle gets for nothing.  By strips a level of 33^2 to
// 129^2 took 7.8 us down and 6.2 us up.
// Every value is the strip passes' expression.

constexpr int kCdTile = 16;                        // own points per side (even)
constexpr int kCdTileDown = kCdTile + 6;           // halo 3: x1 -> x2 -> residual -> restriction
constexpr int kCdTileUp = kCdTile + 4;             // halo 2: f -> x3 -> z
constexpr int kCdTileDownThreads = (kCdTileDown * kCdTileDown + 31) / 32 * 32;
constexpr int kCdTileUpThreads = (kCdTileUp * kCdTileUp + 31) / 32 * 32;
// Levels up to this size go by tiles.  BiCGSTAB on 1025^2 (20 cycles) with the line at 129^2, 257^2,
// 513^2 and 1025^2: 2967, 2836, 2759 and 3010 us; by strips alone 3490.  One cycle with the finest level
// by strips and by tiles, FP64 / FP32 in us: 321^2 62 / 47 and 52 / 38, 449^2 69 / 52 and 59 / 43, 513^2 76 / 55
// and 66 / 47.  The crossover is between 769^2 (80 / 62 and 75 / 57) and 1025^2; the line is under it, where
// the levels of 2^k + 1 grids leave it.
constexpr long long kCdTilePoints = 300000;

template <typename T, typename TB, typename TZ>
__global__ void __launch_bounds__(kCdTileDownThreads) k_cd_down_tile(CdLevelArgs<T, TB, TZ> L, const int *skip) {
    grid_dep_enter();
    if (skip && *(volatile const int *)skip) return;
    constexpr int W = kCdTileDown;
    __shared__ T s0[kCdTileDownThreads], s1[kCdTileDownThreads];
    const int t = threadIdx.x, ty = t / W, tx = t - ty * W;
    const int r = (int)blockIdx.y * kCdTile - 3 + ty, c = (int)blockIdx.x * kCdTile - 3 + tx;
    const int rows = L.rows, cols = L.cols;
    const long long o = (long long)r * cols + c, nf = (long long)rows * cols;
    const bool in = t < W * W && r >= 1 && r <= rows - 2 && c >= 1 && c <= cols - 2 && FX_IN(o, nf);
    auto within = [&](int h) { return tx >= h && ty >= h && tx < W - h && ty < W - h; };
    T b = (T)0, vx = (T)0, vy = (T)0, id = (T)0, x1 = (T)0;
    if (in) {
        b = (T)L.b[o];
        vx = L.vx[o];
        vy = L.vy[o];
        id = L.A.inv_diag(vx, vy);
        x1 = fx_fma(L.omega, b * id, (T)0);
    }
    s0[t] = x1;
    __syncthreads();
    T x2 = (T)0;
    if (in && within(1)) {
        x2 = fx_fma(L.omega, (b - L.A.apply(x1, s0[t - W], s0[t + W], s0[t - 1], s0[t + 1], vx, vy)) * id, x1);
        if (within(3)) L.x2[o] = x2;
    }
    s1[t] = x2;
    __syncthreads();
    s0[t] = in && within(2) ? b - L.A.apply(x2, s1[t - W], s1[t + W], s1[t - 1], s1[t + 1], vx, vy) : (T)0;
    __syncthreads();
    constexpr int H = kCdTile / 2;
    if (t < H * H) {
        const int cy = t / H, cx = t - cy * H;
        const int fr = (int)blockIdx.y * kCdTile + 2 * cy, fc = (int)blockIdx.x * kCdTile + 2 * cx;
        const long long oc = (long long)(fr >> 1) * L.ccols + (fc >> 1);
        if (fr >= 2 && fr <= rows - 3 && fc >= 2 && fc <= cols - 3 && FX_IN(oc, (long long)((rows - 1) / 2 + 1) * L.ccols)) {
            const T *const q = s0 + (3 + 2 * cy) * W + 3 + 2 * cx;
            const T e = (q[-W] + q[W]) + (q[-1] + q[1]);
            const T d = (q[-W - 1] + q[-W + 1]) + (q[W - 1] + q[W + 1]);
            L.crhs[oc] = ((T)4 * q[0] + ((T)2 * e + d)) * (T)0.0625;
        }
    }
}

template <typename T, typename TB, typename TZ>
__global__ void __launch_bounds__(kCdTileUpThreads) k_cd_up_tile(CdLevelArgs<T, TB, TZ> L, int zero_ring, const int *skip) {
    grid_dep_enter();
    if (skip && *(volatile const int *)skip) return;
    constexpr int W = kCdTileUp;
    __shared__ T s0[kCdTileUpThreads], s1[kCdTileUpThreads];
    const int t = threadIdx.x, ty = t / W, tx = t - ty * W;
    const int r = (int)blockIdx.y * kCdTile - 2 + ty, c = (int)blockIdx.x * kCdTile - 2 + tx;
    const int rows = L.rows, cols = L.cols, ccols = L.ccols;
    const long long o = (long long)r * cols + c, nf = (long long)rows * cols;
    const bool grid = t < W * W && r >= 0 && r < rows && c >= 0 && c < cols && FX_IN(o, nf);
    const bool in = grid && r >= 1 && r <= rows - 2 && c >= 1 && c <= cols - 2;
    auto within = [&](int h) { return tx >= h && ty >= h && tx < W - h && ty < W - h; };
    T b = (T)0, vx = (T)0, vy = (T)0, id = (T)0, f = (T)0;
    if (in) {
        const int crows = (rows - 1) / 2 + 1, m = r >> 1, k = c >> 1;
        const bool ro = r & 1, co = c & 1;
        auto at = [&](bool need, int cr, int cc) {
            const long long oc = (long long)cr * ccols + cc;
            return need && cr < crows && cc < ccols && FX_IN(oc, (long long)crows * ccols) ? L.e[oc] : (T)0;
        };
        const T e00 = at(true, m, k), e01 = at(co, m, k + 1), e10 = at(ro, m + 1, k), e11 = at(ro && co, m + 1, k + 1);
        const T x2 = L.x2[o];
        b = (T)L.b[o];
        vx = L.vx[o];
        vy = L.vy[o];
        const T p = ro ? (co ? (T)0.25 * ((e00 + e10) + (e01 + e11)) : (T)0.5 * (e00 + e10))
                       : (co ? (T)0.5 * (e00 + e01) : e00);
        f = x2 + p;
        id = L.A.inv_diag(vx, vy);
    }
    s0[t] = f;
    __syncthreads();
    T x3 = (T)0;
    if (in && within(1))
        x3 = fx_fma(L.omega, (b - L.A.apply(f, s0[t - W], s0[t + W], s0[t - 1], s0[t + 1], vx, vy)) * id, f);
    s1[t] = x3;
    __syncthreads();
    if (!within(2) || !grid) return;
    if (in)
        L.z[o] = (TZ)fx_fma(L.omega, (b - L.A.apply(x3, s1[t - W], s1[t + W], s1[t - 1], s1[t + 1], vx, vy)) * id, x3);
    else if (zero_ring)
        L.z[o] = (TZ)0;
}

inline dim3 cd_tiles(int rows, int cols) {
    return dim3((unsigned)((cols + kCdTile - 1) / kCdTile), (unsigned)((rows + kCdTile - 1) / kCdTile));
}

template <typename T, typename TB, typename TZ>
int launch_cd_down(fx_ctx *ctx, const CdLevelArgs<T, TB, TZ> &L, const int *skip) {
    static std::atomic<int> occ{0};
    constexpr size_t smem = kCdWarps * cd_down_warp_smem<T, TB>();
    static_assert(smem <= 48 * 1024, "no opt-in needed");
    const double pts = (double)L.rows * (double)L.cols;
    if ((long long)L.rows * L.cols <= kCdTilePoints) {
        timing_pre(ctx, "cdmg_down");
        launch_pdl(ctx, k_cd_down_tile<T, TB, TZ>, cd_tiles(L.rows, L.cols), dim3(kCdTileDownThreads), 0, L, skip);
        timing_post(ctx, pts, pts * (sizeof(TB) + 3.25 * sizeof(T)));
        return check_launch(ctx, "cdmg_down");
    }
    const long cap = (long)band_capacity(ctx, k_cd_down<T, TB, TZ>, occ, kCdWarps * 32, smem) * kCdWarps;
    const StripGeom G = strip_geom(L.rows, L.cols, kCdOwnDown, cap);
    timing_pre(ctx, "cdmg_down");
    launch_pdl(ctx, k_cd_down<T, TB, TZ>, (G.nitems + kCdWarps - 1) / kCdWarps, kCdWarps * 32, smem, G, L, skip);
    timing_post(ctx, pts, pts * (sizeof(TB) + 3.25 * sizeof(T)));
    return check_launch(ctx, "cdmg_down");
}

template <typename T, typename TB, typename TZ>
int launch_cd_up(fx_ctx *ctx, const CdLevelArgs<T, TB, TZ> &L, bool zero_ring, const int *skip) {
    static std::atomic<int> occ{0};
    constexpr size_t smem = kCdWarps * cd_up_warp_smem<T, TB>();
    const double pts = (double)L.rows * (double)L.cols;
    if ((long long)L.rows * L.cols <= kCdTilePoints) {
        timing_pre(ctx, "cdmg_up");
        launch_pdl(ctx, k_cd_up_tile<T, TB, TZ>, cd_tiles(L.rows, L.cols), dim3(kCdTileUpThreads), 0, L, zero_ring ? 1 : 0,
                   skip);
        timing_post(ctx, pts, pts * (sizeof(TB) + 3.25 * sizeof(T) + sizeof(TZ)));
        return check_launch(ctx, "cdmg_up");
    }
    if (smem > 48 * 1024) FX_TRY(strip_smem_optin(k_cd_up<T, TB, TZ>, smem));
    const long cap = (long)band_capacity(ctx, k_cd_up<T, TB, TZ>, occ, kCdWarps * 32, smem) * kCdWarps;
    const StripGeom G = strip_geom(L.rows, L.cols, kCdOwnUp, cap);
    timing_pre(ctx, "cdmg_up");
    launch_pdl(ctx, k_cd_up<T, TB, TZ>, (G.nitems + kCdWarps - 1) / kCdWarps, kCdWarps * 32, smem, G, L, zero_ring ? 1 : 0,
               skip);
    timing_post(ctx, pts, pts * (sizeof(TB) + 3.25 * sizeof(T) + sizeof(TZ)));
    return check_launch(ctx, "cdmg_up");
}

}  // namespace fx
