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
