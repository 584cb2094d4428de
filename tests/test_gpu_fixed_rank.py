"""Fixed-rank bases (pivoted Cholesky of the Gram matrix or pivoted QR, then the
orthogonal completion) where their kernels change: empty boxes, box sizes
around the limits of the panels in registers and shared memory, ranks that are
no multiple of a panel."""
import numpy as np
import pytest

import h2_oracle as O
import mxc_b200 as m

pytestmark = pytest.mark.gpu


def _solve(M, x):
    z = x.copy()
    M.solvePrecondition(z)
    return z


@pytest.mark.parametrize("precision", [m.FP64, m.FP32])
def test_empty_box_beside_full_ones(handle, precision):
    """A caller's own tree with a leaf of no bodies, its neighbours taking 64
    pivots.  d^2 has ranks of at most 6 and so no fill to drop: the solve is
    that of the dense matrix (FP32: to 1e-3)."""
    b = np.random.default_rng(0).random((600, 3))
    b[:, 0] += np.repeat([0., 2., 3.], 200)
    child = np.array([[1, 3], [3, 5], [5, 7]] + [[-1, -1]] * 4)
    body = np.array([[0, 600], [0, 200], [200, 600], [0, 200], [200, 200], [200, 400], [400, 600]])
    R, C = np.zeros((7, 3)), np.zeros((7, 3))
    for i, (b0, b1) in enumerate(body):
        if b1 > b0:
            lo, hi = b[b0:b1].min(axis=0), b[b0:b1].max(axis=0)
            R[i], C[i] = (hi - lo) / 2 + 1e-8, (hi + lo) / 2
    t = m.Tree(2, child, body, R, C)
    M = m.H2MatrixSolver(handle, m.Quadratic(1e-3, 1.0), 0.0, 64, 0, t, 1.0, b, samples=0, precision=precision)
    dims, ranks = M.level_dims(2)
    assert list(dims) == [200, 0, 200, 200] and list(ranks) == [64, 0, 64, 64]
    assert sum(M.factorizeM()) == 0
    x = np.random.default_rng(1).random(len(b))
    ref = np.linalg.solve(O.gen_matrix(O.Kernel(O.QUADRATIC, 1e-3, 1.0), b, b), x)
    assert np.linalg.norm(_solve(M, x) - ref) < (1e-9 if precision == m.FP64 else 1e-3) * np.linalg.norm(ref)
