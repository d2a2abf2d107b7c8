"""The convection-diffusion hierarchy's replay option where nothing is replayed: the application is the
one of a hierarchy without the option."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def dev():
    from fluxion_b200 import Device
    return Device.best()


@pytest.mark.parametrize("cycle", ["F64", "F32"])
@pytest.mark.parametrize("n", [41, 65, 129])
def test_direct_applications_do_not_depend_on_the_option(dev, cycle, n):
    """Launches and values of an application inside a caller's own capture, and of one beyond the
    vector pairs that the hierarchy keeps recordings for."""
    from fluxion_b200 import ConvDiffMultigrid, ConvDiffOperator, DType, Field, Grid
    g = Grid.square(n, 1.0 / (n - 1))
    rng = np.random.default_rng(n)
    vx, vy, r = (Field.from_f64(g, rng.uniform(-1, 1, n * n), dev) for _ in range(3))
    op = ConvDiffOperator(g, vx, vy, -1e-2, sigma=0.0)
    be = dev.backend()
    plain, mg = ConvDiffMultigrid(op, dtype=DType[cycle]), ConvDiffMultigrid(op, dtype=DType[cycle])
    mg.set_replay(True)
    z = [Field.from_f64(g, rng.uniform(-1, 1, n * n), dev) for _ in range(18)]

    def count(m, out, recorded=False):
        c0 = be.launch_count()
        if recorded:
            be.graph_begin()
            m.apply(out, r)
            graph = be.graph_end()
            c = be.launch_count() - c0
            graph.launch()
            return c
        m.apply(out, r)
        return be.launch_count() - c0

    want = count(plain, z[0])
    values = z[0].to_vec_f64()
    assert count(mg, z[1], recorded=True) == want
    assert np.array_equal(z[1].to_vec_f64(), values)
    for k in range(16):
        mg.apply(z[k], r)
        assert np.array_equal(z[k].to_vec_f64(), values)
    assert count(mg, z[17]) == want
    assert np.array_equal(z[17].to_vec_f64(), values)


@pytest.mark.parametrize("n", [65, 1025])
@pytest.mark.parametrize("shift", [1, -64, -5125])
def test_overlapping_vectors_of_an_f32_cycle(dev, n, shift):
    """z and r that share a part of their memory: an F32 cycle works on F32 copies of them."""
    import torch
    from fluxion_b200 import ConvDiffMultigrid, ConvDiffOperator, DType, Field, Grid
    g = Grid.square(n, 1.0 / (n - 1))
    rng = np.random.default_rng(n)
    vx, vy = (Field.from_f64(g, rng.uniform(-1, 1, n * n), dev) for _ in range(2))
    mg = ConvDiffMultigrid(ConvDiffOperator(g, vx, vy, -1e-2, sigma=0.0), dtype=DType.F32)
    r, z = Field.from_f64(g, rng.uniform(-1, 1, n * n), dev), Field.zeros(g, DType.F64, dev)
    mg.apply(z, r)
    t = torch.zeros(n * n + abs(shift), dtype=torch.float64, device="cuda")
    at = max(shift, 0), max(-shift, 0)  # of r and z
    t[at[0]:at[0] + n * n] = torch.from_numpy(r.to_vec_f64())
    torch.cuda.synchronize()
    R, Z = (Field(dev.backend().wrap(t[o:].data_ptr(), n * n, DType.F64), g, dev) for o in at)
    mg.apply(Z, R)
    assert np.array_equal(Z.to_vec_f64(), z.to_vec_f64())
