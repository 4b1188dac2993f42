"""Objects freed after their context, as a garbage collector may order it: their memory goes back and no error is left behind."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CODE = """
import os, sys
import numpy as np
import torch
sys.path.insert(0, %r)
from scwatter_gb300 import batch as bt, evaluator as ev, samples, separable as sp, solver, synthetic as syn
torch.zeros(1, device="cuda")
kw = dict(lam=1.0, direction=(0, 0, 1), ex=(1, 0), ey=(0, 0), size=(12.0, 12.0, 2.0), coef=(3, 3))
vol = samples.spheres((2, 12, 12), n_spheres=2, radius=(2, 4), seed=1)
fs = syn.make_factored(4, 5, 2, size=(16.0, 16.0, 2.0), seed=1, dtype=np.complex64)
make = {
    "waves": lambda c: ev.WaveSet.from_cw(c, syn.to_structure(fs)),
    "sep": lambda c: sp.SeparableSet.from_factored(c, fs),
    "solution": lambda c: solver.solve(vol, ctx=c, **kw),
    "batch": lambda c: bt.Batch(c, [bt.BatchItem(sample=vol, grid=(-6, -6, -3, 1.0, 1.0, 0.9, 12, 11, 7), **kw)], lanes=1, method=2),
}[sys.argv[1]]
ctx = ev.Context(0)
o = make(ctx)
ctx.close()
o.close()
assert torch.zeros(3, device="cuda").sum().item() == 0        # (raises where an error was left)
c2 = ev.Context(0)
make(c2).close()
c2.synchronize()
print("ok", flush=True)
os._exit(0)
"""


@pytest.mark.parametrize("kind", ["waves", "sep", "solution", "batch"])
def test_after_the_context(kind):
    # freed host memory is overwritten, so that a look at the freed context shows
    r = subprocess.run([sys.executable, "-c", CODE % ROOT, kind], env=dict(os.environ, MALLOC_PERTURB_="85"), capture_output=True,
                       text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.strip().endswith("ok"), r.stdout + r.stderr
