"""The QR's deflation test looks at both parts of a complex subdiagonal entry: an imaginary one far above rounding,
with a tiny entry across the diagonal, is not dropped (csrc/scw_complex.cuh, csrc/hqr32.cu)."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("entry,dtype,size", [("scw_zgeev", np.complex128, 1e-11), ("scw_cgeev", np.complex64, 1e-4)])
@pytest.mark.parametrize("phase", [1.0, 1j, 1j * (1 + 1e-9j)])
def test_imaginary_subdiagonal(entry, dtype, size, phase):
    import torch
    from scwatter_gb300 import _lib, evaluator as ev
    ctx = ev.Context(0)
    eps = np.finfo(dtype).eps
    A = np.array([[[1.0, eps * 1e-6], [size * phase, 1.0 + 10 * eps]]], dtype)
    dA = torch.from_numpy(A.copy()).cuda()
    W, V = torch.zeros((1, 2), dtype=dA.dtype, device="cuda"), torch.zeros_like(dA)
    torch.cuda.synchronize()
    _lib.call(entry, ctx.handle, 2, *(ctypes.c_void_p(t.data_ptr()) for t in (dA, W, V)), 1, None)
    w, v = W.cpu().numpy()[0].astype(complex), V.cpu().numpy()[0].astype(complex)
    a = A[0].astype(complex)
    # backward error of a few roundings per operation, 2 x 2; dropped, the entry itself remains
    assert (np.linalg.norm(a @ v - v * w, axis=0) <= 50 * eps * np.linalg.norm(v, axis=0)).all()
