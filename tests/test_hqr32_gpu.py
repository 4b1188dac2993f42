"""FP32 Schur stage (multishift QR with aggressive early deflation, csrc/hqr32.cu) through scw_cgeev:
sizes around its deflation window (32), its chase window (64) and several windows per sweep, one and
several CTAs per matrix, against LAPACK's double-precision eigenvalues."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    from scwatter_gb300 import evaluator as ev
    return ev.Context(0)


def _cgeev(ctx, A):
    import torch
    from scwatter_gb300 import _lib
    batch, n, _ = A.shape
    dA = torch.from_numpy(A.astype(np.complex64)).cuda()
    W = torch.zeros((batch, n), dtype=torch.complex64, device="cuda")
    V = torch.zeros((batch, n, n), dtype=torch.complex64, device="cuda")
    torch.cuda.synchronize()
    _lib.call("scw_cgeev", ctx.handle, n, *(ctypes.c_void_p(t.data_ptr()) for t in (dA, W, V)), batch, None)
    return W.cpu().numpy().astype(complex), V.cpu().numpy().astype(complex)


def _matrices(kind, rng, batch, n):
    A = (rng.standard_normal((batch, n, n)) + 1j * rng.standard_normal((batch, n, n))) / np.sqrt(2 * n)
    if kind == "normal":
        return A
    if kind == "layer":            # a smooth layer's reduced matrix: a graded diagonal, decaying couplings
        i = np.arange(n)
        return 0.2 * A * np.exp(-abs(i[:, None] - i[None]) / 6.0) + np.diag(1.0 - 0.9 * (i / n) ** 2)
    if kind == "clusters":         # eightfold eigenvalues up to rounding
        d = np.repeat(np.linspace(-1, 1, (n + 7) // 8), 8)[:n]
        return np.diag(d)[None] + 1e-9 * A
    raise ValueError(kind)


@pytest.mark.parametrize("kind", ["normal", "layer", "clusters"])
@pytest.mark.parametrize("ctas", [0, 1, 2, 5])
@pytest.mark.parametrize("n,batch", [(1, 2), (2, 1), (31, 1), (32, 2), (33, 2), (47, 1), (64, 1), (65, 3), (96, 2), (130, 1),
                                     (257, 2)])
def test_cgeev_sizes(ctx, kind, ctas, n, batch):
    from scwatter_gb300 import _lib
    rng = np.random.default_rng(n + batch)
    A = _matrices(kind, rng, batch, n).astype(np.complex64).astype(complex)
    _lib.call("scw_set_qr_cluster", ctas)
    try:
        W, V = _cgeev(ctx, A)
    finally:
        _lib.call("scw_set_qr_cluster", 0)
    eps = np.finfo(np.float32).eps
    for b in range(batch):
        norm = np.linalg.norm(A[b])
        # backward error of a Schur form: a modest multiple of n eps, as LAPACK's cgeev
        R = A[b] @ V[b] - V[b] * W[b]
        res = np.linalg.norm(R, axis=0) / np.linalg.norm(V[b], axis=0)
        assert res.max() <= 20 * np.sqrt(n) * eps * norm
        if kind != "clusters":
            # every eigenvalue once: matched one to one within the conditioning of the spectrum
            w = np.linalg.eigvals(A[b])
            cost = abs(w[:, None] - W[b][None])
            from scipy.optimize import linear_sum_assignment
            i, j = linear_sum_assignment(cost)
            assert cost[i, j].max() <= 2e-2 * norm / np.sqrt(n)
            assert abs(W[b].sum() - np.trace(A[b])) <= 20 * n * eps * norm
