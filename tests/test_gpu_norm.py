"""The FP32 2-norm on the GPU by four-element loads: lengths about the size where they begin and with
every remainder, against the sum in FP64.  A product of two FP32 values is exact in FP64, and a
thread's plain partial has at most a few hundred terms of one sign: 1e-13 covers their roundings."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 4095, 4096, 4097, 4098, 4099, 1 << 20, (1 << 22) + 3])
def test_norm_f32(n):
    from fluxion_b200 import Device
    be = Device.best().backend()
    x = np.random.default_rng(n).standard_normal(n).astype(np.float32)
    want = np.sqrt(np.sum(x.astype(np.longdouble) ** 2))
    assert abs(be.norm_l2(be.upload_f32(x)) - want) <= 1e-13 * want
