"""The dense steps of the solve that run on products and on the cluster LU: LU sizes around its panel
(32 columns, narrower where a cluster's shared memory asks for it), singular matrices, and the
boundary system of order 6 MF that a grazing harmonic needs."""
import ctypes

import numpy as np
import pytest

from oracle import solve_oracle as so
from scwatter_gb300 import samples

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    from scwatter_gb300 import evaluator as ev
    return ev.Context(0)


@pytest.mark.parametrize("n,nrhs,batch", [(2, 1, 1), (31, 2, 1), (32, 33, 2), (33, 1, 3), (64, 40, 1), (255, 1, 1),
                                          (256, 3, 2), (700, 65, 1), (3500, 2, 1)])
def test_zgesv_panels(ctx, n, nrhs, batch):
    import torch
    from scwatter_gb300 import _lib
    g = torch.Generator(device="cuda").manual_seed(n)
    A = torch.randn((batch, n, n), dtype=torch.complex128, device="cuda", generator=g)
    A[:, :, : n // 2] *= 1e-3                       # rows whose pivots move
    B = torch.randn((batch, n, nrhs), dtype=torch.complex128, device="cuda", generator=g)
    LU, X = A.clone(), B.clone()
    torch.cuda.synchronize()
    info = np.zeros(batch, np.int32)
    _lib.call("scw_zgesv", ctx.handle, n, nrhs, ctypes.c_void_p(LU.data_ptr()), ctypes.c_void_p(X.data_ptr()), batch,
              ctypes.c_void_p(info.ctypes.data))
    assert not info.any()
    for b in range(batch):
        r = torch.linalg.norm(A[b] @ X[b] - B[b]) / (torch.linalg.norm(A[b]) * torch.linalg.norm(X[b]))
        assert r.item() < 1e-14 * np.sqrt(n) + 1e-15          # backward error of LU with partial pivoting
        assert LU[b].tril(-1).abs().max().item() <= 1.0 * np.sqrt(2) + 1e-12   # |Re| + |Im| pivoting


def test_zgesv_singular(ctx):
    import torch
    from scwatter_gb300 import _lib
    A = np.eye(70, dtype=complex)[None].repeat(2, 0)
    A[1, :, 40] = 0
    dA, dB = torch.from_numpy(A).cuda(), torch.ones((2, 70, 1), dtype=torch.complex128, device="cuda")
    torch.cuda.synchronize()
    info = np.zeros(2, np.int32)
    with pytest.raises(_lib.ScwError):
        _lib.call("scw_zgesv", ctx.handle, 70, 1, ctypes.c_void_p(dA.data_ptr()), ctypes.c_void_p(dB.data_ptr()), 2,
                  ctypes.c_void_p(info.ctypes.data))
    assert list(info) == [0, 41]


@pytest.mark.parametrize("sz,n1", [(0.01, 1.0), (0.3, 1.0), (0.01, 1.3)])
def test_boundary_system_near_grazing(ctx, sz, n1):
    # one row of harmonics; the p = 2 harmonic leaves the upper medium at Sz = sz
    from scwatter_gb300 import solver
    sx = np.sqrt(1.0 - sz * sz) - 2.0 / 16.0
    s = samples.spheres((2, 16, 16), n_spheres=2, radius=(3, 5), seed=3)
    kw = dict(lam=1.0, direction=(sx, 0.0, np.sqrt(1 - sx * sx)), ex=(0, 0), ey=(1, 0), size=(16.0, 16.0, 2.0), coef=(5, 1))
    r = so.solve(s, so.SolveParams(n=(1.0, n1), kappa=(0.0,), **kw))
    g = solver.solve(s, n=(1.0, n1), ctx=ctx, **kw)
    assert g.M == (5, 1) and min(abs(r.Sz0)) == pytest.approx(sz, rel=1e-3)
    # the solve's tolerance, times the conditioning a small Sz brings
    assert np.linalg.norm(g.x - r.x) <= 1e-11 / sz * np.linalg.norm(r.x)
