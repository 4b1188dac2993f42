"""Eigenvectors of triangular matrices whose entries differ by many decades: every entry is as exact as substitution
makes it, small ones too."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    from scwatter_gb300 import evaluator as ev
    return ev.Context(0)


@pytest.mark.parametrize("entry,real,decades", [("scw_zgeev", np.float64, 24), ("scw_cgeev", np.float32, 9)])
@pytest.mark.parametrize("n,batch", [(2, 1), (33, 2), (70, 1), (130, 2)])
def test_triangular(ctx, entry, real, decades, n, batch):
    import torch
    from scwatter_gb300 import _lib
    rng = np.random.default_rng(n)
    ct = np.result_type(real, np.complex64)
    d = np.linspace(1.0, 2.0, n)
    A = np.zeros((batch, n, n), complex)
    # couplings to the last column only, of every size: x_i = a_i / (d_n - d_i), x_n = 1
    A[:, :-1, -1] = (rng.standard_normal((batch, n - 1)) + 1j * rng.standard_normal((batch, n - 1))) * \
        10.0 ** rng.uniform(-decades, 0, (batch, n - 1))
    A[:, 0, -1] = 1.0
    A += np.diag(d)
    A = A.astype(ct)
    dA = torch.from_numpy(A).cuda()
    W = torch.zeros((batch, n), dtype=dA.dtype, device="cuda")
    V = torch.zeros_like(dA)
    torch.cuda.synchronize()
    _lib.call(entry, ctx.handle, n, *(ctypes.c_void_p(t.data_ptr()) for t in (dA, W, V)), batch, None)
    W, V = W.cpu().numpy(), V.cpu().numpy().astype(complex)
    eps = np.finfo(real).eps
    for b in range(batch):
        a = A[b].astype(complex)
        k = int(np.argmax(W[b].real))
        x = V[b][:, k] / V[b][-1, k]
        ref = np.append(a[:-1, -1] / (a[-1, -1] - np.diag(a)[:-1]), 1.0)
        # one difference of the diagonal entries, one division, one product with a unitary diagonal
        assert (abs(x - ref) <= 16 * n * eps * abs(ref)).all()
