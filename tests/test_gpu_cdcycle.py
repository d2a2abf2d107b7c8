"""The fused level passes of the convection-diffusion cycle on the GPU: grids at the edges of a strip's
own columns (56 down, 60 up), of its 64 columns and of short row chunks, square and rectangular,
velocities of both signs, zero and negative zero.  FP64 bit for bit against the oracle; FP32 bit for
bit against the separate passes (a kappa field of one value takes them); the whole result vector is
written, ring included."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def dev():
    from fluxion_b200 import Device
    return Device.best()


def _op(dev, rows, cols, sigma, coeff, nu, seed, kappa_field=False):
    from fluxion_b200 import ConvDiffOperator, Field, Grid
    h = 1.0 / (max(rows, cols) - 1)
    g = Grid.new(rows, cols, h, 1.25 * h)
    rng = np.random.default_rng(seed)
    vx, vy = rng.uniform(-1, 1, rows * cols), rng.uniform(-1, 1, rows * cols)
    vx[::7], vy[::5] = 0.0, -0.0
    kap = Field.from_f64(g, np.full(rows * cols, -nu), dev) if kappa_field else -nu
    op = ConvDiffOperator(g, Field.from_f64(g, vx, dev), Field.from_f64(g, vy, dev), kap, sigma=sigma, coeff=coeff)
    oop = O.cd_op(rows, cols, h, 1.25 * h, vx, vy, kappa=None, kappa_s=-nu, sigma=sigma, coeff=coeff)
    return g, op, oop, rng.uniform(-1, 1, rows * cols)


SHAPES = [(19, 19), (33, 57), (57, 33), (61, 63), (37, 65), (113, 117), (69, 121), (129, 181), (257, 41), (41, 241),
          (389, 125)]


@pytest.mark.parametrize("rows,cols", SHAPES)
@pytest.mark.parametrize("sigma,coeff", [(0.0, 1.0), (1.0, 5e-3)])
def test_fused_cycle_matches_oracle(dev, rows, cols, sigma, coeff):
    from fluxion_b200 import ConvDiffMultigrid, Field
    g, op, oop, r = _op(dev, rows, cols, sigma, coeff, 1e-2, rows + cols)
    mg, omg = ConvDiffMultigrid(op, coarse_max=7), O.CdMultigrid(oop, coarse_max=7)
    assert mg.depth() == omg.depth() >= 2
    z = Field.from_f64(g, np.full(rows * cols, 3.0), dev)  # overwritten, ring included
    for _ in range(2):
        mg.apply(z, Field.from_f64(g, r, dev))
        assert np.array_equal(z.to_vec_f64(), omg.apply(r))


@pytest.mark.parametrize("rows,cols", SHAPES)
def test_fused_f32_cycle_equals_separate_passes(dev, rows, cols):
    from fluxion_b200 import ConvDiffMultigrid, DType, Field
    out = []
    for kf in (False, True):
        g, op, _, r = _op(dev, rows, cols, 0.5, 0.75, 1e-2, rows * cols, kf)
        mg = ConvDiffMultigrid(op, coarse_max=7, dtype=DType.F32)
        z = Field.zeros(g, DType.F64, dev)
        mg.apply(z, Field.from_f64(g, r, dev))
        out.append(z.to_vec_f64())
    assert np.array_equal(out[0], out[1])


def test_batch_of_mixed_depths(dev):
    """A problem whose coarsest level is its only one beside deeper ones, both precisions, against the
    single-problem cycle."""
    from fluxion_b200 import ConvDiffMultigrid, ConvDiffOperator, DType, Field, Grid
    from fluxion_b200.batch import BatchSolver
    for sides in ([17, 33, 129], [65, 129, 33, 257]):
        rng = np.random.default_rng(len(sides))
        parts = [[rng.uniform(-1, 1, n * n) for n in sides] for _ in range(3)]
        be = dev.backend()
        vx, vy, r = (be.upload_f64(np.concatenate(p)) for p in parts)
        for dt in (DType.F64, DType.F32):
            b = BatchSolver(dev, sides, 1e-2, vx, vy, cycle_dtype=dt)
            z = be.upload_f64(np.full(b.offsets[-1], 5.0))
            if dt == DType.F32 and 17 in sides:
                z = be.allocate(b.offsets[-1])
            b.precondition(z, r)
            z = z.to_numpy()
            for i, n in enumerate(sides):
                g = Grid.square(n, 1.0 / (n - 1))
                op = ConvDiffOperator(g, Field.from_f64(g, parts[0][i], dev), Field.from_f64(g, parts[1][i], dev), -1e-2,
                                      sigma=0.0)
                zs = Field.zeros(g, DType.F64, dev)
                ConvDiffMultigrid(op, dtype=dt).apply(zs, Field.from_f64(g, parts[2][i], dev))
                assert np.array_equal(z[b.offsets[i]:b.offsets[i + 1]], zs.to_vec_f64())
