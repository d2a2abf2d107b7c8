"""The reference hierarchy's cycle on arguments at the edge of what it takes."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def dev():
    from fluxion_b200 import Device
    return Device.best()


@pytest.mark.parametrize("smoother", [0, 1])
@pytest.mark.parametrize("n", [17, 18, 34, 130])
def test_refused_cycle_leaves_x(dev, smoother, n):
    """A side that halves to an odd number on the way down has a point outside the coarse grid's
    prolongation: the cycle is refused and x keeps its values."""
    from fluxion_b200 import Boundaries, DimensionMismatch, Field, Grid, Multigrid, SmootherKind
    g = Grid.square(n, 1.0 / (n - 1))
    rng = np.random.default_rng(n)
    x, b = rng.uniform(-1, 1, n * n), rng.uniform(-1, 1, n * n)
    mg = Multigrid.build(g, Boundaries.zero_dirichlet(), dev, 2, 2, 2.0 / 3.0, SmootherKind(smoother))
    X = Field.from_f64(g, x, dev)
    with pytest.raises(DimensionMismatch):
        mg.v_cycle(X, Field.from_f64(g, b, dev))
    assert np.array_equal(X.to_vec_f64(), x)


@pytest.mark.parametrize("smoother", [0, 1])
@pytest.mark.parametrize("shift", [5, 64, 640])
def test_overlapping_vectors(dev, smoother, shift):
    """x and b that share a part of their memory: the cycle is that of b as it was passed."""
    import torch
    from fluxion_b200 import Boundaries, DType, Field, Grid, Multigrid, SmootherKind
    n = 128
    g = Grid.square(n, 1.0 / (n - 1))
    mg = Multigrid.build(g, Boundaries.zero_dirichlet(), dev, 2, 2, 2.0 / 3.0, SmootherKind(smoother))
    om = O.Multigrid(n, n, g.dx, g.dx, 2, 2, 2.0 / 3.0, mode=0, smoother=smoother)
    data = np.random.default_rng(shift).uniform(-1, 1, n * n + shift)
    for xs, bs in ((0, shift), (shift, 0)):
        t = torch.from_numpy(data).cuda()
        torch.cuda.synchronize()
        X, B = (Field(dev.backend().wrap(t[o:].data_ptr(), n * n, DType.F64), g, dev) for o in (xs, bs))
        mg.v_cycle(X, B)
        xo = data[xs:xs + n * n].copy()
        om.v_cycle(xo, data[bs:bs + n * n].copy())
        assert np.array_equal(X.to_vec_f64(), xo)


@pytest.mark.parametrize("smoother", [0, 1])
def test_hierarchy_keeps_the_vectors_its_cycle_uses(dev, smoother):
    """u and rhs on every level, and the Chebyshev smoother's two iterates: no vector more."""
    import torch
    from fluxion_b200 import Boundaries, Grid, Multigrid, SmootherKind
    n = 4096
    g = Grid.square(n, 1.0 / (n - 1))
    dev.backend().synchronize()
    free = torch.cuda.mem_get_info()[0]
    mg = Multigrid.build(g, Boundaries.zero_dirichlet(), dev, 2, 2, 2.0 / 3.0, SmootherKind(smoother))
    dev.backend().synchronize()
    taken = free - torch.cuda.mem_get_info()[0]
    del mg
    levels = n * n * 8 * 4 / 3
    assert taken < ((4 if smoother else 2) + 0.5) * levels
