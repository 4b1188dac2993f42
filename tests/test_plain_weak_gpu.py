"""A component far weaker than the others keeps its own accuracy in the plain summation."""
import numpy as np
import pytest

from oracle import oracle_lib as ol

pytestmark = pytest.mark.gpu

# a term's error: operands in 22 bits (2^-22 each, 2^-22 for the product of the lows), phases and steps about 4e-7
TOL = 4e-6


@pytest.fixture(scope="module")
def ctx():
    from scwatter_gb300 import evaluator as ev
    return ev.Context(0)


@pytest.mark.parametrize("weak", range(3))
@pytest.mark.parametrize("bits", [15, 24, 32, 60])
def test_weak_component(ctx, weak, bits):
    import torch
    from scwatter_gb300 import evaluator as ev
    r = np.random.default_rng([weak, bits])
    n, shape, f = 300, (45, 70, 2), np.float32
    k = r.uniform(-6, 6, (n, 3)) + 0j
    k[::3, 2] += 0.2j
    E = r.standard_normal((n, 3)) + 1j * r.standard_normal((n, 3))
    E[:, weak] *= 2.0 ** -bits
    W = np.concatenate([E, k], 1).astype(np.complex64)
    zl, begin, end = np.zeros(1, f), np.array([0, 200]), np.array([200, n])
    ws = ev.WaveSet.from_unpacked(ctx, 1, zl, begin, end, W)
    start, d = [f(v) for v in (-2.1, -1.7, -0.4)], [f(v) for v in (0.11, 0.07, 0.83)]
    Nx, Ny, Nz = shape
    out = torch.zeros((Nz, Ny, Nx, 3), dtype=torch.complex64, device="cuda")
    torch.cuda.synchronize()
    ws.eval_volume_device(*start, *d, Nx, Ny, Nz, out.data_ptr())
    ctx.synchronize()
    ax = [(s + q * np.arange(m, dtype=f)).astype(f) for s, q, m in zip(start, d, shape)]
    P = np.transpose(np.stack(np.meshgrid(*ax, indexing="xy"), -1), (2, 0, 1, 3)).reshape(-1, 3)
    ref = ol.eval_points_f64(W.astype(np.complex128), begin, end, ol.thresholds(zl), P)
    got = out.cpu().numpy().reshape(-1, 3).astype(complex)
    for c in range(3):
        assert np.linalg.norm(got[:, c] - ref[:, c]) <= TOL * np.linalg.norm(ref[:, c])
