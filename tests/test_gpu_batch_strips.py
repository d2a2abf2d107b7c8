"""The batch's strip items: few problems (short chunks), as many as fill the GPU with chunks in between,
more than it holds (64 rows), mixed sides.  The batched cycle equals the single-problem
cycle bit for bit in each."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def dev():
    from fluxion_b200 import Device
    return Device.best()


@pytest.mark.parametrize("cycle", ["F64", "F32"])
@pytest.mark.parametrize("sides", [[33], [65, 65], [257, 33, 9, 1025], [129] * 100, [65] * 1500, [513] * 40])
def test_batched_cycle_equals_single_problem_cycle(dev, cycle, sides):
    from fluxion_b200 import ConvDiffMultigrid, ConvDiffOperator, DType, Field, Grid
    from fluxion_b200.batch import BatchSolver
    be = dev.backend()
    kinds = 3  # distinct problems of a side, repeated
    data = {n: [np.random.default_rng(n + k).uniform(-1, 1, (3, n * n)) for k in range(kinds)] for n in set(sides)}
    vx, vy, r = (np.concatenate([data[n][p % kinds][i] for p, n in enumerate(sides)]) for i in range(3))
    B = BatchSolver(dev, sides, 1e-2, be.upload_f64(vx), be.upload_f64(vy), cycle_dtype=DType[cycle])
    z = be.upload_f64(np.ones(r.size))
    B.precondition(z, be.upload_f64(r))
    got = z.to_numpy()
    want = {}
    for n in data:
        g = Grid.square(n, 1.0 / (n - 1))
        for k in range(kinds):
            VX, VY, R = (Field.from_f64(g, a, dev) for a in data[n][k])
            Z = Field.zeros(g, DType.F64, dev)
            ConvDiffMultigrid(ConvDiffOperator(g, VX, VY, -1e-2, sigma=0.0), dtype=DType[cycle]).apply(Z, R)
            want[n, k] = Z.to_vec_f64()
    for p, n in enumerate(sides):
        assert np.array_equal(got[B.offsets[p]:B.offsets[p + 1]], want[n, p % kinds]), p
