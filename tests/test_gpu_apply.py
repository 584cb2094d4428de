"""The by-rows block apply (plans with at most 16 output columns): rows around
a CTA's 32 and 64, sums around its chunks of 16, column counts between its
widths, odd leading dimensions (element loads), more entries per task than one
staging of them, and accumulation.  Elementwise within the forward bound of a
sum of k * nterms products in its own precision, (k nterms + 8) eps times the
magnitudes."""
import ctypes as C

import numpy as np
import pytest

import mxc_b200 as m
from mxc_b200 import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [m.FP64, m.FP32])
@pytest.mark.parametrize("rows,k,n,nterms,pad,beta", [
    (1, 1, 1, 1, 0, 0.0), (31, 15, 2, 1, 1, 0.0), (32, 16, 3, 2, 0, 1.0), (33, 17, 4, 3, 1, -0.5),
    (64, 128, 1, 8, 0, 1.0), (65, 100, 1, 70, 0, 0.0), (200, 33, 2, 129, 3, 2.0), (156, 312, 1, 9, 0, 1.0),
    (128, 256, 16, 1, 0, 0.0), (100, 212, 16, 2, 0, 1.0), (101, 156, 12, 3, 1, 0.0), (45, 500, 7, 1, 0, 1.0)])
def test_apply_by_rows(handle, rows, k, n, nterms, pad, beta, precision):
    import torch

    dt = np.float64 if precision == m.FP64 else np.float32
    rng = np.random.default_rng(rows + k)
    batch, lda, ldb, ldc = 3, rows + pad, k + pad, rows + pad
    A = rng.standard_normal((batch, nterms, k, lda)).astype(dt)
    B = rng.standard_normal((batch, nterms, n, ldb)).astype(dt)
    C0 = rng.standard_normal((batch, n, ldc)).astype(dt)
    dA, dB, dC = (torch.from_numpy(x.copy()).cuda() for x in (A, B, C0))
    torch.cuda.synchronize()
    _lib.check(_lib.lib().h2dev_batched_gemm_device(
        handle.h, precision, batch, nterms, rows, n, k, 0, 0, -1.0, C.c_void_p(dA.data_ptr()), lda, lda * k,
        C.c_void_p(dB.data_ptr()), ldb, ldb * n, beta, C.c_void_p(dC.data_ptr()), ldc, ldc * n), "gemm")
    handle.synchronize()
    got = dC.cpu().numpy()
    A64, B64, C64 = A[..., :rows].astype(float), B[..., :k].astype(float), C0[..., :rows].astype(float)
    ref = beta * C64 - np.einsum("btkr,btnk->bnr", A64, B64)
    mag = abs(beta) * abs(C64) + np.einsum("btkr,btnk->bnr", abs(A64), abs(B64))
    assert np.all(abs(got[..., :rows] - ref) <= (k * nterms + 8) * np.finfo(dt).eps * mag)
    if pad:
        assert np.array_equal(got[..., rows:], C0[..., rows:])
