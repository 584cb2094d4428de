"""The pivoted factorizations of a box at the sizes where their kernels change:
the LU of a redundant block (panel, register-row and shared-memory limits) and
the column-pivoted QR of an operator box (cluster sizes, rows per lane, the
kernel for boxes beyond a cluster)."""
import numpy as np
import pytest

import h2_oracle as O
import mxc_b200 as m

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [m.FP64, m.FP32])
@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 64, 95, 146, 147, 203, 204, 256, 257, 512, 513, 1024, 1025])
def test_single_box_solve_is_backward_stable(handle, n, precision):
    """A tree of one box has rank 0: factorize is the partial-pivot LU of the
    dense matrix and solvePrecondition its solve.  The small diagonal makes the
    rows move.  The residual is within the LU's backward error, about
    eps n growth ||K|| ||x|| (growth at most about n^(2/3) in practice)."""
    b = np.random.default_rng(n).random((n, 3))
    t = m.build_tree(b, 0)
    M = m.H2MatrixSolver(handle, m.Laplace3D(10.0), 0.0, 8, 0, t, 2.0, b, precision=precision)
    assert M.factorizeM() == [0]
    rhs = np.asfortranarray(np.random.default_rng(1).random((n, 3)))
    x = rhs.copy(order="F")
    M.solvePrecondition(x)
    K = O.gen_matrix(O.Kernel(O.LAPLACE, 10.0), b, b)
    eps = np.finfo(np.float64 if precision == m.FP64 else np.float32).eps
    bound = eps * n ** (2.0 / 3.0) * 10 * np.linalg.norm(K) * np.linalg.norm(x) + eps * np.linalg.norm(rhs)
    assert np.linalg.norm(K @ x - rhs) < bound


@pytest.mark.parametrize("precision", [m.FP64, m.FP32])
@pytest.mark.parametrize("n", [128, 1024])
def test_factorization_memory(n, precision):
    """The LU factors of the redundant blocks need no memory of their own: a
    box takes A U and B beside what the solver holds (powers of two, the size
    classes of the handle's cache), and the plans."""
    b = np.random.default_rng(n).random((n, 3))
    h = m.Handle(0)
    M = m.H2MatrixSolver(h, m.Laplace3D(1e-2), 0.0, 8, 0, m.build_tree(b, 0), 2.0, b, precision=precision)
    h.synchronize()
    live = h.memory()[0]
    h.memory_peak(reset=True)
    M.factorizeM()
    block = n * n * (8 if precision == m.FP64 else 4)
    assert h.memory_peak() - live <= 2 * block + 32768
    M.close()
    h.close()


def _fma32(c, x, y):
    """c - x y rounded once to float32 (twice where the double lies on a tie: about 1 in 2^29)."""
    return (c.astype(float) - x.astype(float) * y.astype(float)).astype(np.float32)


def _inverse_fp32(K, panel):
    """The inverse by a float32 LU with partial pivoting that subtracts `panel` products from an element of
    the trailing block as one sum, and the solve's order of operations (32 rows at a time)."""
    a, n = K.astype(np.float32), len(K)
    p = np.arange(n)
    for k0 in range(0, n, panel):
        j0 = min(k0 + panel, n)
        for k in range(k0, j0):
            q = k + int(np.argmax(abs(a[k:, k])))
            a[[k, q]], p[[k, q]] = a[[q, k]], p[[q, k]]
            a[k + 1:, k] /= a[k, k]
            a[k + 1:, k + 1:j0] = _fma32(a[k + 1:, k + 1:j0], a[k + 1:, k:k + 1], a[k:k + 1, k + 1:j0])
        for i in range(k0, j0):
            a[i + 1:j0, j0:] = _fma32(a[i + 1:j0, j0:], a[i + 1:j0, i:i + 1], a[i:i + 1, j0:])
        s = np.zeros_like(a[j0:, j0:])
        for i in range(k0, j0):
            s = _fma32(s, a[j0:, i:i + 1], a[i:i + 1, j0:])
        a[j0:, j0:] += s
    X = np.eye(n, dtype=np.float32)[p]
    for j in range(n):
        X[j + 1:] = _fma32(X[j + 1:], a[j + 1:, j:j + 1], X[j:j + 1])
    for b0 in range((n - 1) // 32 * 32, -1, -32):
        e = min(b0 + 32, n)
        for j in range(e, n):
            X[b0:e] = _fma32(X[b0:e], a[b0:e, j:j + 1], X[j:j + 1])
        for j in range(e - 1, b0 - 1, -1):
            X[j] /= a[j, j]
            X[b0:j] = _fma32(X[b0:j], a[b0:j, j:j + 1], X[j:j + 1])
    return X


@pytest.mark.parametrize("n", [257, 320, 513, 700])
def test_fp32_factor_in_scratch_sums_by_panels(handle, n):
    """FP32 blocks beyond shared memory: the inverse is that of an LU whose
    trailing updates are sums of 32 products, operation for operation (the
    margin is for a double rounding of the restatement; updates one product at
    a time move it by 1e-6 and more)."""
    b = np.random.default_rng(n).random((n, 3))
    M = m.H2MatrixSolver(handle, m.Laplace3D(1e-4), 0.0, 8, 0, m.build_tree(b, 0), 2.0, b, precision=m.FP32)
    K = M.export(0, m._lib.EXPORT_A).reshape(n, n).T
    assert M.factorizeM() == [0]
    got = M.export(0, m._lib.EXPORT_R).reshape(n, n)
    ref = _inverse_fp32(K, 32)
    assert np.linalg.norm(got - ref) < 1e-7 * np.linalg.norm(ref)


@pytest.mark.parametrize("box", [20, 33, 156, 157, 256, 257, 312, 480, 513, 650, 769])
@pytest.mark.parametrize("eps", [1e-3, 1e-9])
def test_operator_box_sizes(handle, box, eps):
    """Operators whose leaves hold `box` bodies: the product is within ten
    times the bases' threshold of the dense one, and the interpolation keeps
    every body (the skeleton order is a permutation)."""
    n = 8 * box
    b = np.random.default_rng(box).random((n, 3))
    t = m.build_tree(b, 3)
    k = m.Laplace3D(1e-2)
    A = m.H2MatrixSolver(handle, k, eps, 100, 0, t, 1.0, b)
    dims, ranks = A.level_dims(3)
    assert np.all(ranks > 0) and np.all(ranks <= dims)
    S = A.export(3, m._lib.EXPORT_S).reshape(-1, 3)
    for i in range(8):
        own = b[i * box:(i + 1) * box]
        got = S[i * box:(i + 1) * box]
        assert np.array_equal(got[np.lexsort(got.T)], own[np.lexsort(own.T)])
    x = np.random.default_rng(2).random(n)
    y = x.copy()
    A.matVecMul(y)
    d = m.dense_matvec(handle, k, b, x)
    assert np.linalg.norm(y - d) < 10 * eps * np.linalg.norm(d)


def test_operator_boxes_smaller_than_their_cluster(handle):
    """A level of boxes of 3 to 256 bodies runs its pivoted QRs on clusters
    sized for the largest: CTAs of the small ones start late and own no column.
    The product is within ten times the threshold of the dense one, the points
    stay a permutation and repeated builds give the same bits."""
    rng = np.random.default_rng(0)
    b = np.concatenate([0.1 * rng.random((900, 3)), rng.random((60, 3))])
    t = m.build_tree(b, 4, 3, 256)
    k, eps, first = m.Laplace3D(1e-2), 1e-9, None
    x = np.random.default_rng(2).random(len(b))
    for _ in range(5):
        A = m.H2MatrixSolver(handle, k, eps, 100, 0, t, 1.0, b)
        dims, ranks = A.level_dims(4)
        assert dims.min() == 3 and dims.max() == 256 and np.all(ranks <= dims)
        S = A.export(4, m._lib.EXPORT_S).reshape(-1, 3)
        assert np.array_equal(S[np.lexsort(S.T)], b[np.lexsort(b.T)])
        y = x.copy()
        A.matVecMul(y)
        A.close()
        if first is None:
            d = m.dense_matvec(handle, k, b, x)
            assert np.linalg.norm(y - d) < 10 * eps * np.linalg.norm(d)
            first = y, S
        assert np.array_equal(y, first[0]) and np.array_equal(S, first[1])


@pytest.mark.parametrize("box,seed", [(20, 1), (64, 2), (130, 3), (321, 4)])
@pytest.mark.parametrize("precision", [m.FP64, m.FP32])
def test_sketched_operator_box_sizes(box, seed, precision):
    """Sketched bases at row-tile counts, far lists cut into parts and boxes that
    take their whole far block: the product is within a hundred times the
    threshold of the dense one (the sketch's distortion, FP32 rounding)."""
    n = 16 * box
    b = np.random.default_rng(seed).random((n, 3))
    t = m.build_tree(b, 4)
    h = m.Handle(0)
    h.set_option(m._lib.OPT_SAMPLING, m._lib.SAMPLING_SKETCH)
    eps = 1e-9 if precision == m.FP64 else 1e-4
    A = m.H2MatrixSolver(h, m.Laplace3D(1e-2), eps, 100, 0, t, 1.0, b, precision=precision)
    x = np.random.default_rng(2).random(n)
    y = x.copy()
    A.matVecMul(y)
    d = m.dense_matvec(h, m.Laplace3D(1e-2), b, x)
    assert np.linalg.norm(y - d) < 100 * eps * np.linalg.norm(d)
    A.close()
    h.close()
