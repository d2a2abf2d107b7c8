"""The reference hierarchy's fused passes on the GPU: the lexicographic sweep by diagonals (one warp
for small grids, a cluster of warps with 16-column phases above) and the cycles built from it and
from the Chebyshev steps, bit for bit against the oracle.  Sizes sit at the edges of a warp's 32
rows, of a 16-column block, of the 64-column window, of the small kernel and of a cluster's rows."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def dev():
    from fluxion_b200 import Device
    return Device.best()


def _up(dev, a):
    return dev.backend().upload_f64(a)


@pytest.mark.parametrize("rows,cols", [(3, 67), (34, 66), (34, 67), (35, 3), (35, 18), (35, 19), (66, 66), (67, 83),
                                       (131, 258), (290, 97), (1026, 20), (1027, 70), (2060, 37)])
def test_lexicographic_sweep_sizes(dev, rows, cols):
    from fluxion_b200 import Boundaries, Grid, Stencil
    h = 1.0 / (cols - 1)
    g = Grid.new(rows, cols, h, h)
    rng = np.random.default_rng(rows * 7 + cols)
    x, b = rng.uniform(-1, 1, rows * cols), rng.uniform(-1, 1, rows * cols) / h
    st = Stencil.laplacian_2d_5pt(h, 1.5 * h)
    X, B = _up(dev, x), _up(dev, b)
    for _ in range(2):
        dev.backend().weighted_jacobi(X, B, 2.0 / 3.0, g, st, Boundaries.zero_dirichlet())
        O.weighted_jacobi(x, b, 2.0 / 3.0, rows, cols, st.as_triples())
    assert np.array_equal(X.to_numpy(), x)


def test_lexicographic_sweep_f32(dev):
    """FP32: each operation of the sequential sweep rounded to single precision (an fma's product and
    sum are exact in FP64 up to its one rounding here: 24 + 24 bits, then rounded to 24)."""
    from fluxion_b200 import Boundaries, Grid, Stencil
    rows, cols = 37, 70
    h = 0.5
    g = Grid.new(rows, cols, h, h)
    rng = np.random.default_rng(5)
    x = rng.integers(-64, 64, (rows, cols)).astype(np.float32) / 64
    b = rng.integers(-64, 64, (rows, cols)).astype(np.float32) / 64
    st = Stencil.laplacian_2d_5pt(h, h)
    X, B = dev.backend().upload_f32(x), dev.backend().upload_f32(b)
    dev.backend().weighted_jacobi(X, B, 2.0 / 3.0, g, st, Boundaries.zero_dirichlet())
    f = np.float32
    w = [f(t[2]) for t in st.as_triples()]
    om, idg = f(2.0 / 3.0), f(1.0 / st.as_triples()[0][2])
    for r in range(1, rows - 1):
        for c in range(1, cols - 1):
            ax = f(0)
            for wk, v in zip(w, (x[r, c], x[r - 1, c], x[r + 1, c], x[r, c - 1], x[r, c + 1])):
                ax = f(np.float64(wk) * np.float64(v) + np.float64(ax))
            x[r, c] = f(np.float64(om) * np.float64(f(idg * f(b[r, c] - ax))) + np.float64(x[r, c]))
    got = X.to_numpy().reshape(rows, cols)
    # the FP64 sum may round twice: one FP32 step of the largest value, carried through the sweep
    assert np.abs(got - x).max() <= 4 * np.finfo(f).eps * np.abs(x).max()


@pytest.mark.parametrize("smoother", [0, 1])
@pytest.mark.parametrize("rows,cols,pre,post", [(64, 64, 2, 2), (128, 96, 1, 3), (80, 160, 3, 2), (48, 64, 4, 1),
                                                (320, 256, 2, 2)])
def test_reference_cycle_matches_oracle(dev, smoother, rows, cols, pre, post):
    """v_cycle from a nonzero guess and as a preconditioner from zero, also with x and b in one buffer."""
    from fluxion_b200 import Boundaries, DType, Field, Grid, Multigrid, SmootherKind
    h = 1.0 / (cols - 1)
    g = Grid.new(rows, cols, h, h)
    mg = Multigrid.build(g, Boundaries.zero_dirichlet(), dev, pre, post, 2.0 / 3.0, SmootherKind(smoother))
    om = O.Multigrid(rows, cols, h, h, pre, post, 2.0 / 3.0, mode=0, smoother=smoother)
    rng = np.random.default_rng(rows + cols)
    x, b = rng.uniform(-1, 1, rows * cols), rng.uniform(-1, 1, rows * cols)
    X, B = Field.from_f64(g, x, dev), Field.from_f64(g, b, dev)
    mg.v_cycle(X, B)
    xo = x.copy()
    om.v_cycle(xo, b)
    assert np.array_equal(X.to_vec_f64(), xo)
    Z = Field.zeros(g, DType.F64, dev)
    mg.precondition(Z, B)
    zo = np.zeros_like(b)
    om.v_cycle(zo, b)
    assert np.array_equal(Z.to_vec_f64(), zo)
    mg.v_cycle(B, B)
    bo = b.copy()
    om.v_cycle(bo, b.copy())
    assert np.array_equal(B.to_vec_f64(), bo)


def test_reference_cycle_boundary_values_reach_the_coarse_grid(dev):
    """Neumann and Robin sides: the residual of the ring points enters the restriction."""
    from fluxion_b200 import Boundaries, BoundaryCondition, Field, Grid, Multigrid, SmootherKind
    rows, cols = 64, 48
    h = 1.0 / (cols - 1)
    g = Grid.new(rows, cols, h, h)
    bc = Boundaries(BoundaryCondition.Neumann(0.5), BoundaryCondition.Robin(1.0, 2.0, 0.3),
                    BoundaryCondition.Dirichlet(0.7), BoundaryCondition.Neumann(-0.2))
    rng = np.random.default_rng(8)
    x, b = rng.uniform(-1, 1, rows * cols), rng.uniform(-1, 1, rows * cols)
    for sm in (0, 1):
        mg = Multigrid.build(g, bc, dev, 2, 2, 2.0 / 3.0, SmootherKind(sm))
        om = O.Multigrid(rows, cols, h, h, 2, 2, 2.0 / 3.0, mode=0, smoother=sm, bcs=bc.as_tuples())
        X, xo = Field.from_f64(g, x, dev), x.copy()
        mg.v_cycle(X, Field.from_f64(g, b, dev))
        om.v_cycle(xo, b)
        assert np.array_equal(X.to_vec_f64(), xo)
