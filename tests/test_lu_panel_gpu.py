"""LU panels and triangular blocks (csrc/dense_z.cu) through scw_zgesv: pivots that tie, zero, denormal, huge and
infinite pivots, NaN, panels of every remainder, few and many columns per CTA, against numpy."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    from scwatter_gb300 import evaluator as ev
    return ev.Context(0)


def _solve(ctx, A, B):
    import torch
    from scwatter_gb300 import _lib
    batch, n, _ = A.shape
    dA, dB = torch.from_numpy(A.copy()).cuda(), torch.from_numpy(B.copy()).cuda()
    torch.cuda.synchronize()
    info = (ctypes.c_int * batch)()
    st = _lib.load().scw_zgesv(ctx.handle, n, B.shape[2], ctypes.c_void_p(dA.data_ptr()), ctypes.c_void_p(dB.data_ptr()),
                               batch, info)
    ctx.synchronize()
    return st, dB.cpu().numpy(), list(info)


@pytest.mark.parametrize("scale", [1.0, 1e-290, 1e290])
@pytest.mark.parametrize("n,nrhs,batch", [(1, 1, 1), (2, 3, 2), (31, 7, 1), (32, 8, 3), (33, 9, 1), (65, 40, 2), (97, 300, 20),
                                          (260, 33, 2)])
def test_solve(ctx, n, nrhs, batch, scale):
    rng = np.random.default_rng(n)
    A = rng.standard_normal((batch, n, n)) + 1j * rng.standard_normal((batch, n, n))
    A[:, :, 0] = 1.0                              # a column of equal candidates
    A = A * scale
    X = rng.standard_normal((batch, n, nrhs)) + 1j * rng.standard_normal((batch, n, nrhs))
    st, got, info = _solve(ctx, A, A @ X if scale == 1.0 else (A / scale @ X) * scale)
    assert st == 0 and not any(info)
    eps = np.finfo(float).eps
    for a, x, g in zip(A / scale, X, got):
        # backward stable elimination: growth times n eps times the condition number
        assert np.linalg.norm(g - x) <= 50 * n * eps * np.linalg.cond(a) * np.linalg.norm(x)


@pytest.mark.parametrize("n", [5, 40])
def test_zero_column_and_nan(ctx, n):
    rng = np.random.default_rng(n)
    A = rng.standard_normal((3, n, n)) + 0j
    A[0, :, 2] = 0.0                              # no pivot in column 3
    A[2, :, 1] = np.nan
    st, got, info = _solve(ctx, A, np.ones((3, n, 2), complex))
    assert st != 0 and info[0] == 3 and info[1] == 0
    assert np.isfinite(got[1]).all() and np.allclose(A[1] @ got[1], 1.0, atol=1e-9)
    assert not np.isfinite(got[2]).any()
