"""Real and imaginary parts of an FP64 product that are far smaller than the largest of their row and column keep the
accuracy of an FP64 sum."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    from scwatter_gb300 import evaluator as ev
    return ev.Context(0)


def _zgemm(ctx, A, B, C=None, alpha=1.0, beta=0.0):
    import torch
    from scwatter_gb300 import _lib
    batch, M, K = A.shape
    N = B.shape[2]
    dA, dB = (torch.from_numpy(np.ascontiguousarray(v, np.complex128)).cuda() for v in (A, B))
    dC = torch.zeros((batch, M, N), dtype=torch.complex128, device="cuda") if C is None else torch.from_numpy(C).cuda()
    torch.cuda.synchronize()
    al, be = ((ctypes.c_double * 2)(complex(v).real, complex(v).imag) for v in (alpha, beta))
    _lib.call("scw_zgemm", ctx.handle, M, N, K, al, ctypes.c_void_p(dA.data_ptr()), ctypes.c_void_p(dB.data_ptr()), be,
              ctypes.c_void_p(dC.data_ptr()), batch)
    ctx.synchronize()
    return dC.cpu().numpy()


def _operands(kind, rng, batch, M, N, K):
    A = rng.standard_normal((batch, M, K)) + 1j * rng.standard_normal((batch, M, K))
    B = rng.standard_normal((batch, K, N)) + 1j * rng.standard_normal((batch, K, N))
    if kind == "identity":         # rows over 24 decades times the identity
        A *= 10.0 ** rng.uniform(-12, 12, (M, K))
        B = np.broadcast_to(np.eye(K, N) + 0j, B.shape).copy()
    if kind == "triangular":       # a strong column that half of B's columns do not meet
        A[:, :, 0] *= 1e12
        B[:, 0, ::2] = 0
    if kind == "absorbing":        # imaginary parts 1e-9 of the real ones
        A.imag *= 1e-9
        B.imag *= 1e-9
    if kind == "real":
        A, B = A.real + 0j, B.real + 0j
    if kind == "one":              # one weak row, one weak column among ordinary ones
        A[:, M // 2] *= 10.0 ** rng.uniform(-15, 0, K)
        B[:, :, N // 2] *= 10.0 ** rng.uniform(-15, 0, K)
        B[:, :, N // 2] *= rng.integers(0, 2, K)
    return A, B


@pytest.mark.parametrize("kind", ["random", "identity", "triangular", "absorbing", "real", "one"])
@pytest.mark.parametrize("M,N,K,batch", [(1, 2, 2, 1), (64, 64, 16, 2), (65, 33, 17, 1), (129, 63, 128, 1), (50, 50, 50, 4),
                                         (200, 130, 300, 1)])
def test_parts(ctx, kind, M, N, K, batch):
    rng = np.random.default_rng([M, N, K])
    A, B = _operands(kind, rng, batch, M, N, K)
    got = _zgemm(ctx, A, B)
    Al, Bl = A.astype(np.clongdouble), B.astype(np.clongdouble)
    for b in range(batch):
        ref = Al[b] @ Bl[b]
        ar, ai, br, bi = (abs(v) for v in (A[b].real, A[b].imag, B[b].real, B[b].imag))
        # an FP64 sum of 2 K products, each rounded, in any order
        gamma = (2 * K + 1) * 2.0 ** -53
        assert (abs(got[b].real - ref.real) <= gamma * (ar @ br + ai @ bi)).all()
        assert (abs(got[b].imag - ref.imag) <= gamma * (ar @ bi + ai @ br)).all()


def test_row_times_identity(ctx):
    A = np.array([[[1e10, 1 / 3]]], complex)
    assert np.array_equal(_zgemm(ctx, A, np.eye(2)[None] + 0j), A)


@pytest.mark.parametrize("alpha,beta", [(1.0, 1.0), (-0.5 + 2j, 0.25 - 1j)])
def test_parts_added_to_c(ctx, alpha, beta):
    rng = np.random.default_rng(9)
    A, B = _operands("one", rng, 2, 70, 70, 90)
    C = 1e-6 * (rng.standard_normal((2, 70, 70)) + 1j * rng.standard_normal((2, 70, 70)))
    got = _zgemm(ctx, A, B, C.copy(), alpha, beta)
    Al, Bl = A.astype(np.clongdouble), B.astype(np.clongdouble)
    for b in range(2):
        ref = alpha * (Al[b] @ Bl[b]) + beta * C[b]
        S = abs(A[b]) @ abs(B[b])
        assert (abs(got[b] - ref) <= (2 * 90 + 8) * 2.0 ** -52 * (abs(alpha) * S + abs(beta) * abs(C[b]))).all()
