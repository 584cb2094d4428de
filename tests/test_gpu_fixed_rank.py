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


def _row_of_cubes(box, seed):
    """Four leaves of `box` bodies in a row of unit cubes."""
    b = np.random.default_rng(seed).random((4 * box, 3))
    b[:, 0] += np.repeat(np.arange(4.), box)
    return b, m.build_tree(b, 2)


SIZES = [(256, 100), (257, 100), (512, 129), (513, 129), (726, 161), (727, 161), (800, 70), (801, 70), (1100, 301)]
CASES = [(box, rank, precision, mode) for box, rank in SIZES for precision in (m.FP64, m.FP32)
         for mode in (m._lib.BASIS_GRAM, m._lib.BASIS_HOUSEHOLDER)
         if mode == m._lib.BASIS_GRAM or box in (257, 513, 801)]


@pytest.mark.parametrize("box,rank,precision,mode", CASES)
def test_fixed_rank_box_sizes(handle, box, rank, precision, mode):
    """Leaf bases: Q orthogonal, the points a permutation of the box's, and the
    first `rank` columns span the far field (every other body: a preconditioner's
    far lists are those of weak admissibility) to the larger of a hundred times
    the best rank's error and the Gram matrix's 1e-7 (FP32: 1e-5)."""
    b, t = _row_of_cubes(box, box)
    handle.set_basis_mode(mode)
    try:
        M = m.H2MatrixSolver(handle, m.Laplace3D(1e-3), 0.0, rank, 0, t, 1.0, b, samples=0, precision=precision)
    finally:
        handle.set_basis_mode(m._lib.BASIS_GRAM)
    dims, ranks = M.level_dims(2)
    assert np.all(dims == box) and np.all(ranks == rank)
    S = M.export(2, m._lib.EXPORT_S).reshape(4, box, 3)
    Q = M.export(2, m._lib.EXPORT_Q).reshape(4, box, box)  # rows: columns of Q
    eps = 2.2e-16 if precision == m.FP64 else 1.2e-7
    # Entries of Q^T Q: products over FP64 sums (Gram mode rounds to FP32 at the end only), or a sum of `box`
    # FP32 products in sequence, up to box eps.
    orth = box * eps if (precision, mode) == (m.FP32, m._lib.BASIS_HOUSEHOLDER) else 4 * eps * (np.sqrt(box) + 10)
    for i in (0, 3):
        own, got = b[i * box:(i + 1) * box], S[i]
        assert np.array_equal(got[np.lexsort(got.T)], own[np.lexsort(own.T)])
        assert np.abs(Q[i] @ Q[i].T - np.eye(box)).max() < orth
        X = O.gen_matrix(O.Kernel(O.LAPLACE, 1e-3), own, np.concatenate([b[:i * box], b[(i + 1) * box:]]))
        U = Q[i][:rank]
        best = np.linalg.svd(X, compute_uv=False)
        err = np.linalg.norm(X - U.T @ (U @ X), 2)
        assert err < max(100 * best[rank], (1e-7 if precision == m.FP64 else 1e-5) * best[0])
    M.close()


@pytest.mark.parametrize("box,rank,precision", [(256, 40, m.FP64), (513, 40, m.FP64), (801, 33, m.FP64),
                                                (1100, 70, m.FP64), (513, 40, m.FP32), (801, 33, m.FP32)])
def test_fixed_rank_solve_of_exact_ranks(handle, box, rank, precision):
    """d^2 has ranks of at most 6 and so no fill to drop, and pivots below the
    noise floor beyond: the solve is that of the dense matrix."""
    b, t = _row_of_cubes(box, box)
    M = m.H2MatrixSolver(handle, m.Quadratic(1e-4, 1.0), 0.0, rank, 0, t, 1.0, b, samples=0, precision=precision)
    assert sum(M.factorizeM()) == 0
    x = np.random.default_rng(1).random(4 * box)
    ref = np.linalg.solve(O.gen_matrix(O.Kernel(O.QUADRATIC, 1e-4, 1.0), b, b), x)
    assert np.linalg.norm(_solve(M, x) - ref) < (1e-9 if precision == m.FP64 else 1e-3) * np.linalg.norm(ref)
