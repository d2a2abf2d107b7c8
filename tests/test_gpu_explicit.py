"""Fused explicit diffusion passes against the sequence of field operations they replace, bit for bit:
grids at the edges of a strip's 56 own and 64 total columns and of short row chunks, step counts that
split into an even number of passes and that do not, a nonzero ring (kept by every scheme)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def dev():
    from fluxion_b200 import Device
    return Device.best()


def _sequence(solver, u, n):
    """n steps as the field operations (what a step with other boundaries or a source runs)."""
    for _ in range(n):
        solver._record(u, None)


@pytest.mark.parametrize("scheme", ["Euler", "Rk2", "Rk4"])
@pytest.mark.parametrize("rows,cols", [(3, 3), (4, 57), (9, 56), (65, 58), (33, 113), (130, 61), (257, 64), (100, 345)])
def test_passes_equal_field_operations(dev, scheme, rows, cols):
    from fluxion_b200 import Boundaries, Field, Grid
    from fluxion_b200.steppers import DiffusionSolver, TimeScheme
    h = 1.0 / (max(rows, cols) - 1)
    g = Grid.new(rows, cols, h, 1.5 * h)
    data = np.random.default_rng(rows * cols).uniform(-1, 1, rows * cols)
    for n in (1, 2, 3, 5, 8):
        a, b = (DiffusionSolver.build(g, 0.7, None, Boundaries.zero_dirichlet(), TimeScheme[scheme], dev) for _ in range(2))
        ua, ub = Field.from_f64(g, data, dev), Field.from_f64(g, data, dev)
        a.step_n(ua, n)
        _sequence(b, ub, n)
        assert a.steps_done() == n
        assert np.array_equal(ua.to_vec_f64(), ub.to_vec_f64())


def test_graph_solver_stays_with_its_field(dev):
    from fluxion_b200 import Boundaries, Field, Grid
    from fluxion_b200.steppers import DiffusionSolver, TimeScheme
    g = Grid.square(40, 1.0 / 39)
    data = np.random.default_rng(1).uniform(-1, 1, 1600)
    u, v = Field.from_f64(g, data, dev), Field.from_f64(g, data, dev)
    s = DiffusionSolver.build(g, 1.0, None, Boundaries.zero_dirichlet(), TimeScheme.Rk4, dev)
    s.enable_graph()
    s.step_n(u, 3)
    with pytest.raises(ValueError):
        s.step_n(v, 1)
