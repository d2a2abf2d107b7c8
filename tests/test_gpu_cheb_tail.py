"""The Chebyshev hierarchy's coarse levels in one block, bit for bit against the oracle: hierarchies that
fit whole, that just do not, long thin ones, step counts at the ends of the step table and without
pre-smoothing, and boundary values that reach the coarse grids."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def dev():
    from fluxion_b200 import Device
    return Device.best()


@pytest.mark.parametrize("rows,cols,pre,post", [
    (4, 4, 2, 2),       # a single level
    (8, 6, 1, 1),
    (96, 48, 2, 2),     # 4608 points: all levels in the block
    (64, 80, 2, 2),     # 5120: the finest level by launches
    (4, 1024, 3, 1),
    (512, 8, 2, 3),
    (96, 64, 0, 2),     # no pre-smoothing: the coarse iterate is read as zeros
    (96, 64, 11, 11),   # 32 steps on the coarsest level: the last that fits
    (96, 64, 12, 11),   # 33: every level by launches
    (192, 160, 0, 1),
    (192, 160, 2, 0),   # no post-smoothing: the plain prolongation
])
@pytest.mark.parametrize("mixed_bc", [False, True])
def test_chebyshev_cycle_sizes(dev, rows, cols, pre, post, mixed_bc):
    from fluxion_b200 import Boundaries, BoundaryCondition, DType, Field, Grid, Multigrid, SmootherKind
    h = 1.0 / (cols - 1)
    g = Grid.new(rows, cols, h, 1.25 * h)
    bc = Boundaries.zero_dirichlet()
    if mixed_bc:
        bc = Boundaries(BoundaryCondition.Neumann(0.5), BoundaryCondition.Robin(1.0, 2.0, 0.3),
                        BoundaryCondition.Dirichlet(0.7), BoundaryCondition.Neumann(-0.2))
    mg = Multigrid.build(g, bc, dev, pre, post, 2.0 / 3.0, SmootherKind(1))
    om = O.Multigrid(rows, cols, h, 1.25 * h, pre, post, 2.0 / 3.0, mode=0, smoother=1,
                     **({"bcs": bc.as_tuples()} if mixed_bc else {}))
    rng = np.random.default_rng(rows * 3 + cols + pre)
    x, b = rng.uniform(-1, 1, rows * cols), rng.uniform(-1, 1, rows * cols)
    X, B = Field.from_f64(g, x, dev), Field.from_f64(g, b, dev)
    xo = x.copy()
    for _ in range(2):  # the second from a nonzero iterate of the first
        mg.v_cycle(X, B)
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
