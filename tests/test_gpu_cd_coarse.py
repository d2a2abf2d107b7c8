"""The convection-diffusion cycle's one-block coarsest solve with several points a thread: coarsest grids
of 34 x 34 to 64 x 64 (more than 1024 points, the most a block holds is 4096).  FP64 bit for bit
against the oracle; FP32 with a scalar kappa and a kappa field of that value bit for bit alike, and within
1e-4 of FP64 (some 200 sweeps, each rounding at 6e-8)."""
import numpy as np
import pytest

from oracle import oracle as O
from tests.helpers import rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("side", [33, 34, 45, 46, 64])
@pytest.mark.parametrize("pre,post", [(1, 1), (2, 2)])
def test_coarse_grids_beyond_a_block(side, pre, post):
    from fluxion_b200 import ConvDiffMultigrid, ConvDiffOperator, Device, DType, Field, Grid
    dev = Device.best()
    n = 2 * side - 1
    h = 1.0 / (n - 1)
    g = Grid.square(n, h)
    vx, vy, r = np.random.default_rng(side).uniform(-1, 1, (3, n * n))
    VX, VY = Field.from_f64(g, vx, dev), Field.from_f64(g, vy, dev)

    def cycle(kappa, dtype):
        mg = ConvDiffMultigrid(ConvDiffOperator(g, VX, VY, kappa, sigma=0.0), pre, post, coarse_max=side - 2, dtype=dtype)
        assert mg.depth() == 2
        z = Field.from_f64(g, np.full(n * n, 3.0), dev)
        mg.apply(z, Field.from_f64(g, r, dev))
        return z.to_vec_f64()

    field = Field.from_f64(g, np.full(n * n, -1e-2), dev)
    want = O.CdMultigrid(O.cd_op(n, n, h, h, vx, vy, kappa=None, kappa_s=-1e-2, sigma=0.0, coeff=1.0), pre, post,
                         coarse_max=side - 2).apply(r)
    assert np.array_equal(cycle(-1e-2, DType.F64), want)
    assert np.array_equal(cycle(field, DType.F64), want)
    single = cycle(-1e-2, DType.F32)
    assert np.array_equal(single, cycle(field, DType.F32))
    assert rel_err(single, want) < 1e-4
