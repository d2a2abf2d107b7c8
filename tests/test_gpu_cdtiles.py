"""The convection-diffusion cycle's level passes by tiles (small levels) and by strips (large ones) on
the GPU, bit for bit against the oracle: grids at the edges of a 16 x 16 tile and its halo, just
under and over the size where strips take over, and both in one hierarchy."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def dev():
    from fluxion_b200 import Device
    return Device.best()


@pytest.mark.parametrize("rows,cols", [(9, 9), (13, 45), (17, 17), (29, 33), (31, 35), (37, 17), (49, 97), (65, 261),
                                       (257, 257), (269, 265), (301, 293), (57, 1301), (1301, 63), (517, 533),
                                       (541, 553), (549, 553), (57, 5301)])
@pytest.mark.parametrize("f32", [False, True])
def test_level_passes(dev, rows, cols, f32):
    from fluxion_b200 import ConvDiffMultigrid, ConvDiffOperator, DType, Field, Grid
    h = 1.0 / (max(rows, cols) - 1)
    g = Grid.new(rows, cols, h, 1.25 * h)
    rng = np.random.default_rng(rows * 5 + cols)
    n = rows * cols
    vx, vy, r = (rng.uniform(-1, 1, n) for _ in range(3))
    vx[::7], vy[::5] = 0.0, -0.0
    V = [Field.from_f64(g, v, dev) for v in (vx, vy)]

    def apply(kappa):
        op = ConvDiffOperator(g, V[0], V[1], kappa, sigma=0.5, coeff=0.75)
        mg = ConvDiffMultigrid(op, coarse_max=7, dtype=DType.F32 if f32 else DType.F64)
        # FP64: what z holds does not matter, ring included; the separate FP32 passes keep its ring
        z = Field.from_f64(g, np.full(n, 0.0 if f32 else 3.0), dev)
        mg.apply(z, Field.from_f64(g, r, dev))
        return z.to_vec_f64()

    got = apply(-1e-2)
    if f32:  # a kappa field of one value takes the separate passes
        want = apply(Field.from_f64(g, np.full(n, -1e-2), dev))
    else:
        want = O.CdMultigrid(O.cd_op(rows, cols, h, 1.25 * h, vx, vy, kappa=None, kappa_s=-1e-2, sigma=0.5, coeff=0.75),
                             coarse_max=7).apply(r)
    assert np.array_equal(got, want)
