"""Two-pass modified Gram-Schmidt in GMRES and FGMRES: restart lengths at the edges of a group of basis
vectors (8), of the pass (32 vectors) and beyond it, grids of odd sizes down to fewer elements than a
block, against the oracle's vector-by-vector method after the same number of iterations.

The operator's condition number is about 200 (coeff = -25 h^2: eigenvalues 1 to 201), so a rounding
difference of u = 1.1e-16 per coefficient moves an iterate by at most about m kappa u = 1e-12
relative; the bar is 1e-10."""
import numpy as np
import pytest

from oracle import oracle as O
from tests.helpers import rel_err

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def dev():
    from fluxion_b200 import Device
    return Device.best()


@pytest.mark.parametrize("rows,cols", [(9, 11), (67, 45), (131, 258)])
@pytest.mark.parametrize("restart,its", [(2, 5), (9, 9), (17, 20), (32, 32), (33, 33), (40, 45)])
def test_iterates_match_oracle(dev, rows, cols, restart, its):
    from fluxion_b200 import Boundaries, DType, FgmresSolver, Field, GmresSolver, Grid, Stencil
    its = min(its, (rows - 2) * (cols - 2) // 4)
    h = 1.0 / (max(rows, cols) - 1)
    g = Grid.new(rows, cols, h, h)
    b = np.zeros((rows, cols))
    b[1:-1, 1:-1] = np.random.default_rng(rows * restart).uniform(-1, 1, (rows - 2, cols - 2))
    b = b.ravel()
    st, coeff = Stencil.laplacian_2d_5pt(h, h), -25.0 * h * h
    xo = np.zeros(rows * cols)
    it, res, _ = O.gmres_solve(xo, b, rows, cols, coeff, O.laplacian_5pt(h, h), restart, 1e-13, its)
    outs = []
    for cls in (GmresSolver, FgmresSolver):
        x = Field.zeros(g, DType.F64, dev)
        s = cls(g, dev, restart, 1e-13, its).solve(x, Field.from_f64(g, b, dev), coeff, st, Boundaries.zero_dirichlet())
        assert s.iterations == it
        outs.append(x.to_vec_f64())
        assert rel_err(outs[-1], xo) < 1e-10
    assert np.array_equal(outs[0], outs[1])  # without a preconditioner FGMRES is GMRES
