"""The vertex V-cycle's level passes by tiles (small levels) and by strips (large ones) on the GPU:
grids that end inside, at and just past a 16 x 16 tile, long thin ones, just under and over the size
where strips take over, and both in one hierarchy, bit for bit against the oracle in FP64 and its FP32
restatement."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def dev():
    from fluxion_b200 import Device
    return Device.best()


@pytest.mark.parametrize("rows,cols", [(81, 113), (129, 65), (97, 161), (161, 97), (209, 177), (65, 1025), (1025, 81),
                                       (385, 385), (401, 385), (545, 561), (257, 1185), (1185, 273)])
def test_vertex_cycle(dev, rows, cols):
    from fluxion_b200 import DType, Field, Grid, Multigrid, Stencil
    dx, dy = 1.0 / (cols - 1), 1.25 / (rows - 1)
    g = Grid.new(rows, cols, dx, dy)
    st = Stencil.poisson_neg_laplacian(dx, dy)
    rng = np.random.default_rng(rows * 11 + cols)
    b = np.zeros((rows, cols))
    b[1:-1, 1:-1] = rng.uniform(-1, 1, (rows - 2, cols - 2))
    b = b.ravel()
    B = Field.from_f64(g, b, dev)
    om = O.Multigrid(rows, cols, dx, dy, 2, 2, 0.8, mode=1, op_coeff=1.0, entries=st.as_triples(), coarse_max=7,
                     coarse_sweeps=40)
    for dtype, cycle in ((DType.F64, om.v_cycle), (DType.F32, om.v_cycle_f32)):
        mg = Multigrid.vertex(g, None, dev, 2, 2, 0.8, 7, 40, dtype)
        assert mg.depth() == om.depth() >= 3
        z, zo = Field.zeros(g, DType.F64, dev), np.zeros(rows * cols)
        mg.precondition(z, B)
        cycle(zo, b)
        assert np.array_equal(z.to_vec_f64(), zo)
