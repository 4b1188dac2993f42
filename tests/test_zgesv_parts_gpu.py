"""LU of matrices with entries of very different size: every entry's error is small against |L| |U|, as with FP64 sums."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    from scwatter_gb300 import evaluator as ev
    return ev.Context(0)


@pytest.mark.parametrize("n", [40, 70, 150])
def test_factors_entry_by_entry(ctx, n):
    import torch
    from scwatter_gb300 import _lib
    rng = np.random.default_rng(n)
    A = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))
    # row 0 meets the odd columns right of the first panel only, rows 1 .. 31 all of them; below the panel column 0
    # is strong and the others weak, and so are the even columns: those entries are sums of weak terms alone
    A[0, 1:32] = 0
    A[0, 32::2] = 0
    A[32:, 1:32] *= 1e-12
    A[32:, 32::2] *= 1e-12
    A[np.arange(n), np.arange(n)] += 40                            # no interchanges
    dA, dB = torch.from_numpy(A).cuda(), torch.ones((n, 1), dtype=torch.complex128, device="cuda")
    torch.cuda.synchronize()
    _lib.call("scw_zgesv", ctx.handle, n, 1, ctypes.c_void_p(dA.data_ptr()), ctypes.c_void_p(dB.data_ptr()), 1, None)
    LU = dA.cpu().numpy()
    L, U = np.tril(LU, -1) + np.eye(n), np.triu(LU)
    err = abs(L.astype(np.clongdouble) @ U.astype(np.clongdouble) - A)
    # |L U - A| <= gamma_n |L| |U|, complex operations within a factor of 4
    assert (err <= 4 * n * 2.0 ** -53 * (abs(L) @ abs(U))).all()
