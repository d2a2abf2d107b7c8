"""Options of the explicit stepper around its fused passes: what the passes do not hold runs as the
sequence of field operations, with the same results as ever."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def dev():
    from fluxion_b200 import Device
    return Device.best()


def _solver(g, scheme, dev, boundaries=None, stencil=None):
    from fluxion_b200 import Boundaries
    from fluxion_b200.steppers import DiffusionSolver, TimeScheme
    s = DiffusionSolver.build(g, 0.7, None, boundaries or Boundaries.zero_dirichlet(), TimeScheme[scheme], dev)
    if stencil is not None:
        s.stencil = stencil
    return s


def _grid_and_data(rows=37, cols=50):
    from fluxion_b200 import Grid
    h = 1.0 / (max(rows, cols) - 1)
    return Grid.new(rows, cols, h, 1.5 * h), np.random.default_rng(rows * cols).uniform(-1, 1, rows * cols)


@pytest.mark.parametrize("scheme", ["Euler", "Rk2", "Rk4"])
@pytest.mark.parametrize("entries", ["nine", "three", "five, another order"])
def test_other_stencils(dev, scheme, entries):
    """A solver whose stencil is not the five-point form steps by the field operations; five entries in
    any order are the five-point form."""
    from fluxion_b200 import Field, Stencil
    g, data = _grid_and_data()
    five = Stencil.laplacian_2d_5pt(g.dx, g.dy)
    stencil = {"nine": Stencil.laplacian_2d_9pt(g.dx, g.dy), "three": Stencil(five.as_triples()[:3]),
               "five, another order": Stencil(five.as_triples()[::-1])}[entries]
    a, b = (_solver(g, scheme, dev, stencil=stencil) for _ in range(2))
    ua, ub = Field.from_f64(g, data, dev), Field.from_f64(g, data, dev)
    a.step_n(ua, 3)
    a.step(ua)
    for _ in range(4):
        b._record(ub, None)
    assert a.steps_done() == 4
    assert np.array_equal(ua.to_vec_f64(), ub.to_vec_f64())


def _boundaries(kind):
    from fluxion_b200 import BoundaryCondition, Boundaries
    return {"zero Dirichlet": Boundaries.zero_dirichlet(),
            "Dirichlet": Boundaries(*[BoundaryCondition.Dirichlet(v) for v in (0.3, -0.2, 0.0, 0.7)]),
            "mixed": Boundaries(BoundaryCondition.Neumann(0.5), BoundaryCondition.Robin(1.0, 2.0, 0.3),
                                BoundaryCondition.Dirichlet(0.7), BoundaryCondition.Neumann(-0.2))}[kind]


@pytest.mark.parametrize("scheme", ["Euler", "Rk2", "Rk4"])
@pytest.mark.parametrize("kind", ["zero Dirichlet", "Dirichlet", "mixed"])
def test_graph_solver_repeats_its_first_step(dev, scheme, kind):
    """With the graph enabled the first step_n fixes the step: later calls repeat it on the same field,
    whatever the solver's attributes are by then, and the result is that of the field operations."""
    from fluxion_b200 import Field, Stencil
    g, data = _grid_and_data()
    a, b = (_solver(g, scheme, dev, _boundaries(kind)) for _ in range(2))
    ua, ub = Field.from_f64(g, data, dev), Field.from_f64(g, data, dev)
    a.enable_graph()
    a.step_n(ua, 10)
    with pytest.raises(ValueError):
        a.step_n(Field.from_f64(g, data, dev), 1)
    a.boundaries = _boundaries("Dirichlet" if kind == "mixed" else "mixed")
    a.step_n(ua, 6)
    a.step_n(ua, 1)
    a.boundaries = _boundaries("zero Dirichlet")
    a.alpha, a.stencil = 0.3, Stencil.laplacian_2d_9pt(g.dx, g.dy)
    a.step_n(ua, 7)
    a.step_n(ua, 1)
    for _ in range(25):
        b._record(ub, None)
    assert a.steps_done() == 25
    assert np.array_equal(ua.to_vec_f64(), ub.to_vec_f64())


@pytest.mark.parametrize("graph", [False, True])
@pytest.mark.parametrize("kind", ["zero Dirichlet", "mixed"])
def test_step_counts(dev, graph, kind):
    """A step count is an integer: another number is refused and a negative one makes no step."""
    from fluxion_b200 import Field
    g, data = _grid_and_data()
    s, u = _solver(g, "Euler", dev, _boundaries(kind)), Field.from_f64(g, data, dev)
    if graph:
        s.enable_graph()
    with pytest.raises(TypeError):
        s.step_n(u, 2.5)
    s.step_n(u, -3)
    s.step_n(u, 0)
    assert s.steps_done() == 0 and np.array_equal(u.to_vec_f64(), data)
    s.step_n(u, np.int64(2))
    assert s.steps_done() == 2
