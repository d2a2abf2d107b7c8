"""The training gradient over batches below, at and above one sample per resident block (two blocks
per SM) against the mean of the single samples' gradients.  Each gradient entry is an FP32 sum over
the batch; with n terms its error is within n u sum|terms|, u = 6e-8, so the bar is n u times the sum
of the singles' norms over n, that is n u times their mean norm."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("count", [1, 7, 296, 297, 700])
@pytest.mark.parametrize("lam", [0.0, 0.4])
def test_batch_gradient_is_the_mean(count, lam):
    from fluxion_b200 import ConvDiffOperator, Device, Field, Grid
    from fluxion_b200.learned import LearnedSmoother, SmootherSamples
    dev = Device.best()
    n = 97
    g = Grid.square(n, 1.0 / (n - 1))
    rng = np.random.default_rng(3)
    f = [Field.from_f64(g, rng.uniform(-1, 1, n * n), dev) for _ in range(5)]
    op = ConvDiffOperator(g, f[0], f[1], -1e-2, sigma=0.0)
    S = SmootherSamples(dev, 5)
    S.add_patches(op, f[2], f[3], f[4], 0.8, [(4, 4), (10, 20), (60, 44), (30, 6), (44, 76)])
    net = LearnedSmoother(dev, 5)
    p = net.params
    p[-145:-1] = rng.normal(0.0, 0.2, 144)
    p[432:448], p[2752:2768] = rng.normal(0.0, 0.05, 16), rng.normal(0.0, 0.05, 16)
    net.params = p
    one = [net.loss_grad(S, [i], True, lam) for i in range(5)]
    idx = rng.integers(0, 5, count)
    loss, grad = net.loss_grad(S, idx, True, lam)
    want = sum(one[i][1].astype(np.float64) for i in idx) / count
    norm = sum(np.linalg.norm(one[i][1].astype(np.float64)) for i in idx) / count
    u = 2.0 ** -24
    assert np.linalg.norm(grad - want) <= (count + 500) * u * norm  # 500: a single gradient's own terms per partial sum
    assert abs(loss - sum(one[i][0] for i in idx) / count) <= (count + 500) * u * loss
    assert np.array_equal(grad, net.loss_grad(S, idx, True, lam)[1])  # the same bits again
