"""Separable sets: the viewer's three planes side by side equal planes evaluated one at a time, and descriptors that
go with the launches (up to 3584 bytes) give what uploaded ones give, bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def sets():
    from scwatter_gb300 import evaluator as ev
    from scwatter_gb300 import separable as sp
    from scwatter_gb300 import synthetic as syn
    ctx = ev.Context(0)
    size = (12.0, 12.0, 3.0)
    return ctx, [sp.SeparableSet.from_paired(ctx, syn.make_paired(7, 6, 3, size=size, seed=2)),
                 sp.SeparableSet.from_factored(ctx, syn.make_factored(7, 6, 3, size=size, seed=2, dtype=np.complex64))]


@pytest.mark.parametrize("method", ["FP32", "TF32X3", "BF16X3"])
@pytest.mark.parametrize("N", [1, 33, 200, 700])
def test_three_planes(sets, N, method):
    import torch
    from scwatter_gb300 import separable as sp
    ctx, both = sets
    m = getattr(sp, method)
    d = np.float32(10.0 / max(1, N - 1))
    for s in both:
        for shift in (0.0, 0.37):
            xs, ys, zs, x, y, z = -5.0 + shift, -4.5, -2.9, 0.7, -1.3, 0.4 + shift
            got = s.evaluate_planes_host(xs, ys, zs, x, y, z, d, N, method=m)
            one = torch.zeros((N, N, 3), dtype=torch.complex64, device="cuda")
            for g, (axis, a, b, c) in zip(got, [(0, xs, ys, z), (2, xs, zs, y), (1, ys, zs, x)]):
                s.eval_plane_device(axis, a, b, c, d, N, one.data_ptr(), method=m)
                ctx.synchronize()
                assert np.array_equal(one.cpu().numpy().view(np.uint32), g.view(np.uint32))


@pytest.mark.parametrize("planes", [60, 900])
def test_volume_in_slabs(sets, planes):
    import torch
    from scwatter_gb300 import separable as sp
    ctx, both = sets
    grid = (-2.0, -1.0, -1.7, 0.3, 0.2, 3.4 / planes)
    for s in both:
        whole = torch.zeros((planes, 5, 9, 3), dtype=torch.complex64, device="cuda")
        part = torch.zeros_like(whole)
        torch.cuda.synchronize()
        s.eval_volume_device(*grid, 9, 5, planes, whole.data_ptr(), method=sp.FP32)
        for k in range(0, planes, 20):
            s.eval_slab_device(*grid, 9, 5, k, min(planes, k + 20), part[k:].data_ptr(), method=sp.FP32)
        ctx.synchronize()
        assert torch.equal(whole, part)


@pytest.mark.parametrize("method", ["FP32", "TF32X3", "BF16X3"])
@pytest.mark.parametrize("n,planes,z0", [(1, 1, 0.1), (65, 33, -1.6), (300, 9, -1.4), (70, 12, 40.0), (70, 12, -60.0), (33, 40, -4.0)])
def test_queued_evaluations(sets, n, planes, z0, method):
    """Evaluations queued one behind the other (their kernels' ends and starts overlap; planes inside the sample,
    outside only, both) equal the same ones with the stream drained in between."""
    import torch
    from scwatter_gb300 import separable as sp
    ctx, both = sets
    m = getattr(sp, method)
    jobs = []
    for s in both:
        for shift in (0.0, 0.21):
            jobs.append(lambda o, s=s, f=shift: s.eval_volume_device(-2.0 + f, -1.0, z0, 0.03, 0.2, 0.1, n, 5, planes, o, method=m))
            for axis in (1, 2):
                jobs.append(lambda o, s=s, f=shift, a=axis: s.eval_plane_device(a, -2.0, z0, f, 0.1, n, o, method=m))
    size = max(planes * 5 * n, n * n) * 3
    one = torch.zeros((len(jobs), size), dtype=torch.complex64, device="cuda")
    for o, job in zip(one, jobs):
        ctx.synchronize()
        torch.cuda.synchronize()
        job(o.data_ptr())
    ctx.synchronize()
    for _ in range(3):
        queued = torch.zeros_like(one)
        torch.cuda.synchronize()
        for o, job in zip(queued, jobs):
            job(o.data_ptr())
        ctx.synchronize()
        assert torch.equal(queued, one)
    assert int((one != 0).sum()) > 0
