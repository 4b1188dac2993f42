"""The plain summation's error on grids from a small part of a wavelength to many: no more than sums of FP32 operands have."""
import numpy as np
import pytest

from oracle import oracle_lib as ol

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("seed", range(3))
@pytest.mark.parametrize("extent", [1e-4, 1e-2, 0.3, 3.0, 20.0])
def test_error_of_a_term(extent, seed):
    import torch
    from scwatter_gb300 import evaluator as ev
    ctx = ev.Context(0)
    r = np.random.default_rng(seed)
    n, f = 600, np.float32
    k = r.uniform(-6, 6, (n, 3)) + 0j
    E = r.standard_normal((n, 3)) + 1j * r.standard_normal((n, 3))
    W = np.concatenate([E, k], 1).astype(np.complex64)
    zl, begin, end = np.array([-50.0], f), np.array([0, 0]), np.array([0, n])
    ws = ev.WaveSet.from_unpacked(ctx, 1, zl, begin, end, W)
    Nx, Ny, Nz = 60, 64, 2
    d, s, z0, dz = f(extent / 60), f(-extent / 2), f(-extent / 3), f(extent / 5)
    out = torch.zeros((Nz, Ny, Nx, 3), dtype=torch.complex64, device="cuda")
    torch.cuda.synchronize()
    ws.eval_volume_device(s, s, z0, d, d, dz, Nx, Ny, Nz, out.data_ptr())
    ctx.synchronize()
    ax = [(a + q * np.arange(m, dtype=f)).astype(f) for a, q, m in ((s, d, Nx), (s, d, Ny), (z0, dz, Nz))]
    P = np.transpose(np.stack(np.meshgrid(*ax, indexing="xy"), -1), (2, 0, 1, 3)).reshape(-1, 3)
    ref = ol.eval_points_f64(W.astype(np.complex128), begin, end, ol.thresholds(zl), P)
    got = out.cpu().numpy().reshape(-1, 3)
    # amplitude, phase factor, their product and the sum in 24 bits: 2^-24 each, added up
    assert np.linalg.norm(got - ref) <= 2.0 ** -22 * np.linalg.norm(ref)
