// fx_reference.cuh -- the reference hierarchy's smoothers and transfers as fused passes
// (fx_reference.cu): the lexicographic weighted-Jacobi sweep, the Chebyshev step, and the
// residual with its restriction.
#pragma once

#include "fx_points.cuh"

namespace fx {

// `nsweeps` in-place lexicographic weighted-Jacobi sweeps (ops.rs:425-473) of the five-point
// stencil with weights w = {centre, north, south, west, east}, applied in that order.
template <typename T>
int lex5_sweeps(fx_ctx *ctx, T *x, const T *b, size_t rows, size_t cols, const double (&w)[5], double omega,
                double inv_diag, size_t nsweeps);

// Whether a stencil's entry list is exactly centre, north, south, west, east.
bool lex5_order(const fx_stencil *s);

// One level of the reference hierarchy (FP64) as the Chebyshev smoother sees it.
struct ChebLevel {
    size_t rows, cols;
    double dx, dy;
    StencilP P;  // the level Laplacian, five-point form
    double *u, *w0, *w1;
    const double *rhs;
};

// `n` Chebyshev steps (multigrid.rs:308-473) on u.  coarse non-null: u is first corrected by the
// piecewise-constant prolongation of it (ccols its columns), ring included, in the same passes.
// u_zero: u stands for zeros, whatever it holds; it is written only.
int cheb_smooth(fx_ctx *ctx, const ChebLevel &L, const double *coarse, size_t ccols, size_t n, bool u_zero);

// The first of the levels that one block can take, with all that lie below it (nl: none).
int cheb_tail_top(const ChebLevel *L, int nl, size_t n_pre, size_t n_post, size_t n_coarse);

// The cycle over levels L[0 .. nlev), in one block: L[0].u and .rhs as given (u_zero as above), the
// other levels' vectors in shared memory.
int cheb_tail(fx_ctx *ctx, const ChebLevel *L, const BcP *B, int nlev, bool u_zero, size_t n_pre, size_t n_post,
              size_t n_coarse);

// coarse rhs = the clamped 2 x 2 average of rhs - S u (ring values by the boundary conditions), and
// coarse u = 0 unless it is null (multigrid.rs:205-215: apply_stencil, scale(-1), axpy, restrict, fill).
int ref_restrict_residual(fx_ctx *ctx, const double *u, const double *rhs, size_t rows, size_t cols, const StencilP &P,
                          const BcP &B, double *coarse_rhs, double *coarse_u, size_t crows, size_t ccols);

}  // namespace fx
