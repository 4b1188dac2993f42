"""The plain summation adds at most 1024 waves in FP32: longer sums lose nothing to their partial sums."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    from scwatter_gb300 import evaluator as ev
    return ev.Context(0)


@pytest.mark.parametrize("n", [1000, 4096, 9000, 20001])
def test_partial_sums_cancel(ctx, n):
    """Waves of k = 0, whose amplitudes are multiples of 2^-13 below 2: 1024 of them add up to less than 2^11, exactly in
    FP32.  All of them reach thousands before they cancel."""
    import torch
    from scwatter_gb300 import evaluator as ev
    r = np.random.default_rng(n)
    a = r.integers(2 ** 13, 2 ** 14, (n, 3, 2)) * 2.0 ** -13
    a[n // 2:] *= -1
    W = np.zeros((n, 6), np.complex64)
    W[:, :3] = a[..., 0] + 1j * a[..., 1]
    f = np.float32
    ws = ev.WaveSet.from_unpacked(ctx, 1, np.array([-10.0], f), np.array([0, 0]), np.array([0, n]), W)
    Nx, Ny, Nz = 200, 320, 40             # 1000 tiles: no tile's waves are dealt to several CTAs below 4096 waves
    out = torch.zeros((Nz, Ny, Nx, 3), dtype=torch.complex64, device="cuda")
    torch.cuda.synchronize()
    ws.eval_volume_device(f(0), f(0), f(0), f(0.1), f(0.1), f(0.1), Nx, Ny, Nz, out.data_ptr())
    ctx.synchronize()
    s = a.sum(0)
    exact = (s[:, 0] + 1j * s[:, 1]).astype(np.complex64)
    assert (out == torch.from_numpy(exact).cuda()).all()
