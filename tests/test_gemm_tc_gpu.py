"""FP64 complex GEMM on the tensor cores (scw_zgemm) against extended-precision products, at the edges
of its tiles (128 rows, 32 columns, 16 inner indices a stage, 128 a drain) and on operands whose
digits are extreme, graded or not finite."""
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
    if K == 0:                 # no element, but the entry point wants addresses
        dA = dB = torch.zeros(1, dtype=torch.complex128, device="cuda")
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
    if kind == "extreme":      # every digit at its largest magnitude, all products of one sign
        v = sum(127.0 * 256.0 ** -i for i in range(1, 9))
        A = np.full_like(A, v * (1 + 1j))
        B = np.full_like(B, v * (1 - 1j))
    if kind == "graded":       # inner rows over 60 decades; A's columns the other way
        g = 10.0 ** rng.uniform(-30, 30, K)
        A, B = A / g, B * g[:, None]
    if kind == "diagonal":     # a strong diagonal among small couplings
        A = 1e-7 * A
        A[:, np.arange(min(M, K)), np.arange(min(M, K))] += 1.5
    return A, B


@pytest.mark.parametrize("kind", ["random", "extreme", "graded", "diagonal"])
@pytest.mark.parametrize("M,N,K,batch", [(1, 2, 1, 1), (128, 32, 16, 2), (129, 33, 17, 1), (127, 31, 128, 1),
                                         (50, 50, 50, 4), (40, 300, 129, 1), (260, 66, 400, 1)])
def test_zgemm_against_extended_precision(ctx, kind, M, N, K, batch):
    rng = np.random.default_rng(M + N + K)
    A, B = _operands(kind, rng, batch, M, N, K)
    got = _zgemm(ctx, A, B)
    Al, Bl = A.astype(np.clongdouble), B.astype(np.clongdouble)
    for b in range(batch):
        ref = np.zeros((M, N), np.clongdouble)
        for k in range(K):
            ref += Al[b][:, k:k + 1] * Bl[b][k:k + 1]
        part = lambda z: np.maximum(abs(z.real), abs(z.imag))  # noqa: E731
        f = part(B[b]).max(1)                                  # inner scaling, within a factor of two
        R, S = (part(A[b]) * f).max(1), (part(B[b]) / f[:, None]).max(0)
        # per inner index and part: 2^-61 of the largest value for each operand's cut to 62 bits, 2^-57
        # for the dropped diagonals, two products; the scales are powers of two; then one rounding
        bound = K * 2.0 ** -54 * R[:, None] * S[None] + 2.0 ** -52 * abs(ref)
        assert (abs(got[b] - ref) <= bound).all()


def test_zgemm_alpha_beta_and_empty_inner(ctx):
    rng = np.random.default_rng(5)
    A, B = _operands("random", rng, 2, 70, 45, 33)
    C = rng.standard_normal((2, 70, 45)) + 1j * rng.standard_normal((2, 70, 45))
    for alpha, beta in [(-1.0, 1.0), (0.5 - 2j, 0.0), (1.0, -0.25 + 1j)]:
        got = _zgemm(ctx, A, B, C.copy(), alpha, beta)
        ref = alpha * (A @ B) + beta * C
        assert abs(got - ref).max() < 1e-13 * abs(ref).max()
    got = _zgemm(ctx, A[:, :, :0], B[:, :0], C.copy(), 1.0, 2.0)
    assert np.array_equal(got, 2.0 * C)


def test_zgemm_zero_and_non_finite_operands(ctx):
    rng = np.random.default_rng(6)
    A, B = _operands("random", rng, 1, 140, 40, 50)
    A[0, 3] = 0
    B[0, 7] = 0
    B[0, :, 11] = 0
    clean = _zgemm(ctx, A, B)[0]
    assert (clean[3] == 0).all() and (clean[:, 11] == 0).all()
    A[0, 130, 4] = np.nan
    B[0, 9, 33] = np.inf
    got = _zgemm(ctx, A, B)[0]
    keep_r, keep_c = np.arange(140) != 130, np.arange(40) != 33
    assert np.isnan(got[130]).all() and np.isnan(got[keep_r][:, 33]).all()
    other = np.ix_(keep_r, keep_c)
    # the infinite entry leaves its inner row's scale to the finite ones
    assert abs(got[other] - clean[other]).max() < 1e-13 * abs(clean).max()


def test_zgemm_scale_limits(ctx):
    rng = np.random.default_rng(7)
    A, B = _operands("random", rng, 1, 33, 35, 20)
    for sa, sb in [(1e-300, 1e300), (1e-160, 1e-155), (1e-310, 1.0)]:
        got = _zgemm(ctx, A * sa, B * sb)[0]
        ref = (A[0] * sa).astype(np.clongdouble) @ (B[0] * sb).astype(np.clongdouble)
        tol = 1e-13 * abs(ref).max() if abs(ref).max() > 1e-290 else 1e-12 * abs(ref).max() + 1e-321
        assert abs(got - ref).max() <= tol
