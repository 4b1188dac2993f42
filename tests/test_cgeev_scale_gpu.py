"""scw_cgeev on matrices far from unit scale: shifts and reflectors neither overflow nor vanish."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    from scwatter_gb300 import evaluator as ev
    return ev.Context(0)


@pytest.mark.parametrize("scale", [1e-14, 1e-11, 1e-6, 1.0, 1e6, 1e11, 1e15, 1e18])
@pytest.mark.parametrize("n,batch", [(2, 1), (5, 2), (33, 1), (90, 2), (300, 1)])
def test_scaled(ctx, n, batch, scale):
    import torch
    from scwatter_gb300 import _lib
    rng = np.random.default_rng(n)
    A = ((rng.standard_normal((batch, n, n)) + 1j * rng.standard_normal((batch, n, n))) * (scale / np.sqrt(2 * n))).astype(np.complex64)
    dA = torch.from_numpy(A).cuda()
    W = torch.zeros((batch, n), dtype=torch.complex64, device="cuda")
    V = torch.zeros_like(dA)
    torch.cuda.synchronize()
    _lib.call("scw_cgeev", ctx.handle, n, *(ctypes.c_void_p(t.data_ptr()) for t in (dA, W, V)), batch, None)
    W, V = W.cpu().numpy().astype(complex) / scale, V.cpu().numpy().astype(complex)
    eps = np.finfo(np.float32).eps
    for b in range(batch):
        a = A[b].astype(complex) / scale
        norm = np.linalg.norm(a)
        # backward error of a Schur form: a modest multiple of n eps, as LAPACK's cgeev
        res = np.linalg.norm(a @ V[b] - V[b] * W[b], axis=0) / np.linalg.norm(V[b], axis=0)
        assert res.max() <= 20 * np.sqrt(n) * eps * norm
        assert abs(W[b].sum() - np.trace(a)) <= 20 * n * eps * norm
