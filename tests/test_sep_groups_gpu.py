"""The contraction's kernels for 1 to 8 planes per pass (and regions of more, split evenly): a volume
equals its planes evaluated one at a time, bit for bit, since a plane's sums do not depend on the
planes beside it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("paired", [True, False])
@pytest.mark.parametrize("shape", [0, 1])
@pytest.mark.parametrize("per", [1, 2, 3, 4, 5, 6, 7, 8, 9, 17])
def test_volume_equals_its_planes(paired, shape, per):
    import torch
    from scwatter_gb300 import evaluator as ev
    from scwatter_gb300 import separable as sp
    from scwatter_gb300 import synthetic as syn
    ctx = ev.Context(0)
    M0, M1, Z = 5, 7, 2                       # 35 harmonics: the last warp's rows run past the end
    if paired:
        s = sp.SeparableSet.from_paired(ctx, syn.make_paired(M0, M1, Z, size=(16.0, 16.0, float(Z)), seed=per))
    else:
        s = sp.SeparableSet.from_factored(ctx, syn.make_factored(M0, M1, Z, size=(16.0, 16.0, float(Z)), seed=per,
                                                                 dtype=np.complex64))
    s.set_tiles(shape)
    N, Nz = 12, per * Z + 2                   # and one plane in each outer medium
    z0, dz = np.float32(-Z / 2 - 0.5 / per), np.float32(1.0 / per)
    whole = torch.zeros((Nz, N, N, 3), dtype=torch.complex64, device="cuda")
    s.eval_volume_device(-2.0, -1.0, z0, 0.3, 0.2, dz, N, N, Nz, whole.data_ptr())
    ctx.synchronize()
    one = torch.zeros((N, N, 3), dtype=torch.complex64, device="cuda")
    for k in range(Nz):
        z = np.float32(z0 + np.float32(dz * np.float32(k)))
        s.eval_volume_device(-2.0, -1.0, z, 0.3, 0.2, dz, N, N, 1, one.data_ptr())
        ctx.synchronize()
        assert torch.equal(whole[k], one), k
