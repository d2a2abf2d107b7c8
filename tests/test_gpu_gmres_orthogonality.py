"""Two-pass modified Gram-Schmidt where orthogonality decides: ill-conditioned operators, on which GMRES
with one-pass classical Gram-Schmidt fails.

The operator is a random diffusion field (kappa over eight decades) without velocities on a patch of 9
to 40 points.  GMRES runs as many iterations as the patch has points, up to 32.  With modified
Gram-Schmidt it is backward stable (Paige, Rozloznik, Strakos 2006): ||b - A x|| <= C u (||A|| ||x|| +
||b||) with a small multiple of the number of iterations m for C; the bar is C = 4 m.  Classical
Gram-Schmidt, and the two passes with a Gram matrix that is left out, transposed or one row late,
end a hundred times above the bar or more; the CPU test below holds each of them to that.

On the larger grids the operator is zero outside the patch, so the vectors are too: the dots' partial
sums then come from blocks that the patch's rows are spread over."""
import numpy as np
import pytest

U = 2.0 ** -53
PATCHES = [(3, 3, 9), (4, 4, 16), (5, 5, 25), (5, 6, 30), (4, 8, 32)]  # interior rows, columns, iterations


def _kappa(pr, pc, rows, cols, seed=0):
    """The patch's field on a rows x cols grid (zero outside), its first interior point at (1, 1) of the
    smallest grid and somewhere inside a larger one."""
    k = np.zeros((rows, cols))
    r0, c0 = (rows - pr) // 2, (cols - pc) // 2
    k[r0:r0 + pr, c0:c0 + pc] = -10.0 ** np.random.default_rng(seed).uniform(-8, 0, (pr, pc))
    return k, (slice(r0, r0 + pr), slice(c0, c0 + pc))


def _dense(kappa, h):
    """The operator kappa Lap v (zero ring) on the points of the field's support, row by row."""
    rows, cols = kappa.shape
    idx = {p: i for i, p in enumerate(zip(*np.nonzero(kappa)))}
    A = np.zeros((len(idx), len(idx)))
    for (r, c), i in idx.items():
        A[i, i] = -4.0 * kappa[r, c] / h ** 2
        for q in ((r - 1, c), (r + 1, c), (r, c - 1), (r, c + 1)):
            if q in idx:
                A[i, idx[q]] = kappa[r, c] / h ** 2
    return A


def _gmres(A, b, m, gram):
    """m iterations of GMRES in NumPy, the projections by modified Gram-Schmidt (gram None) or from one
    set of dots and the Gram rows as `gram` passes them on."""
    beta = np.linalg.norm(b)
    V, H, L = np.zeros((m + 1, b.size)), np.zeros((m + 1, m)), np.zeros((m + 1, m + 1))
    V[0] = b / beta
    for k in range(m):
        w = A @ V[k]
        if gram is None:
            for j in range(k + 1):
                H[j, k] = V[j] @ w
                w = w - H[j, k] * V[j]
        else:
            L[k, :k] = V[:k] @ V[k]
            H[:k + 1, k] = np.linalg.solve(np.eye(k + 1) + gram(L[:k + 1, :k + 1]), V[:k + 1] @ w)
            for j in range(k + 1):
                w = w - H[j, k] * V[j]
        H[k + 1, k] = np.linalg.norm(w)
        V[k + 1] = w / H[k + 1, k]
    e = np.zeros(m + 1)
    e[0] = beta
    return V[:m].T @ np.linalg.lstsq(H, e, rcond=None)[0]


def _late(L):
    out = L.copy()
    out[-1] = 0.0
    return out


def _over_bar(A, x, b, m):
    bar = 4 * m * U * (np.linalg.norm(A, 2) * np.linalg.norm(x) + np.linalg.norm(b))
    return np.linalg.norm(b - A @ x) / bar


@pytest.mark.parametrize("pr,pc,m", PATCHES)
def test_the_operators_tell_the_methods_apart(pr, pc, m):
    kappa, _ = _kappa(pr, pc, pr + 2, pc + 2)
    A = _dense(kappa, 1.0 / (max(pr, pc) + 1))
    b = np.random.default_rng(m).uniform(-1, 1, pr * pc)
    assert _over_bar(A, _gmres(A, b, m, None), b, m) < 1.0
    assert _over_bar(A, _gmres(A, b, m, lambda L: L), b, m) < 1.0
    for gram in (lambda L: 0.0 * L, lambda L: L.T, _late):
        assert _over_bar(A, _gmres(A, b, m, gram), b, m) > 100.0


@pytest.mark.gpu
@pytest.mark.parametrize("pr,pc,m", PATCHES)
@pytest.mark.parametrize("grid", ["patch", (64, 97), (129, 513)])
def test_attained_residual(pr, pc, m, grid):
    from fluxion_b200 import ConvDiffOperator, Device, DType, FgmresSolver, Field, GmresSolver, Grid
    dev = Device.best()
    rows, cols = (pr + 2, pc + 2) if grid == "patch" else grid
    h = 1.0 / (max(pr, pc) + 1)
    kappa, at = _kappa(pr, pc, rows, cols)
    A = _dense(kappa, h)
    b = np.zeros((rows, cols))
    b[at] = np.random.default_rng(m).uniform(-1, 1, (pr, pc))
    g = Grid.new(rows, cols, h, h)
    zero = [Field.zeros(g, DType.F64, dev) for _ in range(2)]
    op = ConvDiffOperator(g, *zero, Field.from_f64(g, kappa.ravel(), dev), sigma=0.0)
    outs = []
    for cls in (GmresSolver, FgmresSolver):
        x = Field.zeros(g, DType.F64, dev)
        cls(g, dev, m, 1e-300, m).solve_op(x, Field.from_f64(g, b.ravel(), dev), op, None)
        outs.append(x.to_vec_f64().reshape(rows, cols))
        assert np.count_nonzero(outs[-1]) <= pr * pc
        assert _over_bar(A, outs[-1][at].ravel(), b[at].ravel(), m) < 1.0
    assert np.array_equal(outs[0], outs[1])
