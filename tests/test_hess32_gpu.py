"""FP32 Hessenberg panels (csrc/hess32.cu) through scw_cgeev, where their storage changes: rows of A in
shared memory in full, in part, and V, Y and b in global memory (orders above 2480); panels of every remainder."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,batch", [(3, 1), (4, 3), (34, 2), (35, 1), (66, 2), (99, 1), (161, 40), (300, 150), (520, 24),
                                     (1100, 2), (2500, 1)])
def test_panels(n, batch):
    import torch
    from scwatter_gb300 import _lib, evaluator as ev
    ctx = ev.Context(0)
    g = torch.Generator().manual_seed(n)
    A = torch.randn((batch, n, n), dtype=torch.complex64, generator=g)
    i = torch.arange(n)
    A = 0.2 * A * torch.exp(-abs(i[:, None] - i[None]) / 6.0) + torch.diag(1.0 - 0.9 * (i / n) ** 2)
    A = A.to(torch.complex64).cuda()
    dA, W, V = A.clone(), torch.zeros((batch, n), dtype=torch.complex64, device="cuda"), torch.zeros_like(A)
    torch.cuda.synchronize()
    _lib.call("scw_cgeev", ctx.handle, n, *(ctypes.c_void_p(t.data_ptr()) for t in (dA, W, V)), batch, None)
    eps = np.finfo(np.float32).eps
    for b in range(batch):
        a, v, w = A[b].to(torch.complex128), V[b].to(torch.complex128), W[b].to(torch.complex128)
        norm = torch.linalg.norm(a)
        # backward error of a Schur form: a modest multiple of n eps, as LAPACK's cgeev
        res = torch.linalg.norm(a @ v - v * w, dim=0) / torch.linalg.norm(v, dim=0)
        assert res.max() <= 20 * np.sqrt(n) * eps * norm
        assert abs(w.sum() - torch.trace(a)) <= 20 * n * eps * norm
