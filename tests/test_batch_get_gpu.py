"""A batch's results into memory that is not pageable: the copy takes it or refuses it, the process goes on."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CODE = """
import ctypes, os, sys
import numpy as np
import torch
sys.path.insert(0, %r)
from scwatter_gb300 import _lib, evaluator as ev, samples, batch as bt
ctx = ev.Context(0)
s = samples.spheres((2, 12, 12), n_spheres=2, radius=(2, 4), seed=1)
it = bt.BatchItem(sample=s, grid=(-6, -6, -3, 1.0, 1.0, 0.9, 12, 11, 7), lam=1.0, direction=(0, 0, 1), ex=(1, 0), ey=(0, 0),
                  size=(12.0, 12.0, 2.0), coef=(3, 3))
b = bt.Batch(ctx, [it], lanes=1, method=2)
b.run()
assert not b.wait().any()
x, g, f = b.result(0)
pinned = torch.zeros(f.shape, dtype=torch.complex64).pin_memory()
device = torch.zeros(f.shape, dtype=torch.complex64, device="cuda")
torch.cuda.synchronize()
get = _lib.load().scw_batch_get
assert get(b.handle, 0, None, None, ctypes.c_void_p(pinned.data_ptr()), None) == 0
assert np.array_equal(pinned.numpy(), f)
st = get(b.handle, 0, None, None, ctypes.c_void_p(device.data_ptr()), None)
assert st in (0, 4)
assert np.array_equal(b.result(0)[2], f)
print("ok", flush=True)
os._exit(0)
"""


def test_pinned_and_device_addresses():
    r = subprocess.run([sys.executable, "-c", CODE % ROOT], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.strip().endswith("ok"), r.stdout + r.stderr
