"""Plain summation on the tensor cores, at the edges of its tiles, runs and rules, vs the FP64 sum."""
import numpy as np
import pytest

from oracle import oracle_lib as ol
from tests._util import rel_l2

pytestmark = pytest.mark.gpu

# a term's error: operands in 22 bits (2^-22 each, 2^-22 for the product of the lows), phases and steps
# about 4e-7, FP32 sums of 4096 waves about 1e-6 of their size
TOL = 4e-6
TOL_SUM = 2e-5          # the summation kernel, for what the operands cannot hold


def _waves(n, seed, decay):
    r = np.random.default_rng([n, seed])
    k = r.uniform(-9, 9, (n, 3)) + 0j
    if decay:
        k[:, 2] += 1j * r.uniform(-decay, decay, n)
        k[::3, 0] += 0.2j * decay
    E = (r.standard_normal((n, 3)) + 1j * r.standard_normal((n, 3))) * 2.0 ** r.integers(-6, 6, (n, 1))
    return np.concatenate([E, k], 1).astype(np.complex64)


def _volume(ctx, counts, zl, start, d, shape, seed=0, decay=0.0, edit=None):
    import torch
    from scwatter_gb300 import evaluator as ev
    W = _waves(sum(counts), seed, decay)
    if edit:
        edit(W)
    end = np.cumsum(counts)
    begin = end - np.array(counts)
    zl = np.asarray(zl, np.float32)
    ws = ev.WaveSet.from_unpacked(ctx, len(zl), zl, begin, end, W)
    f = np.float32
    x0, y0, z0 = map(f, start)
    dx, dy, dz = map(f, d)
    Nx, Ny, Nz = shape
    out = torch.zeros((Nz, Ny, Nx, 3), dtype=torch.complex64, device="cuda")
    torch.cuda.synchronize()
    ws.eval_volume_device(x0, y0, z0, dx, dy, dz, Nx, Ny, Nz, out.data_ptr())
    ctx.synchronize()
    ax = [(s + q * np.arange(n, dtype=f)).astype(f) for s, q, n in ((x0, dx, Nx), (y0, dy, Ny), (z0, dz, Nz))]
    P = np.transpose(np.stack(np.meshgrid(*ax, indexing="xy"), -1), (2, 0, 1, 3))
    with np.errstate(all="ignore"):
        ref = ol.eval_points_f64(W.astype(np.complex128), begin, end, ol.thresholds(zl), P.reshape(-1, 3))
    return out.cpu().numpy(), ref.reshape(Nz, Ny, Nx, 3)


@pytest.fixture(scope="module")
def ctx():
    from scwatter_gb300 import evaluator as ev
    return ev.Context(0)


@pytest.mark.parametrize("decay", [0.0, 0.3])
@pytest.mark.parametrize("counts,shape", [
    ((1, 1), (1, 1, 2)), ((31, 33), (8, 9, 2)), ((32, 0), (7, 1, 3)), ((100, 64), (39, 63, 2)), ((129, 5), (40, 64, 2)),
    ((257, 97), (41, 65, 2)), ((40, 4096), (16, 15, 2)), ((4097, 33), (17, 128, 1)), ((9000, 300), (81, 17, 2))])
def test_volume(ctx, counts, shape, decay):
    got, ref = _volume(ctx, counts, [0.0], (-3.1, 1.7, -0.4), (0.11, 0.07, 0.83), shape, decay=decay)
    assert max(rel_l2(got, ref)) < TOL


@pytest.mark.parametrize("N", [16, 33, 65, 120])
def test_planes_through_regions(ctx, N):
    """Rows of a region from one to the whole plane, and empty regions."""
    from scwatter_gb300 import evaluator as ev
    counts = (120, 70, 0, 500, 33)
    W = _waves(sum(counts), 3, 0.2)
    end = np.cumsum(counts)
    begin = end - np.array(counts)
    zl = np.array([-1.9, -1.85, 0.1, 1.2], np.float32)
    ws = ev.WaveSet.from_unpacked(ctx, 4, zl, begin, end, W)
    d = np.float32(5.0 / (N - 1))
    xs, ys, zs, x, y, z = -2.5, -2.4, -2.6, 0.7, -1.3, 0.6
    got = ws.evaluate_planes_host(xs, ys, zs, x, y, z, d, N)
    for g, (axis, a0, b0, c) in zip(got, [(ol.AXIS_XY, xs, ys, z), (ol.AXIS_XZ, xs, zs, y), (ol.AXIS_YZ, ys, zs, x)]):
        P = ol.plane_points(axis, a0, b0, c, d, N)
        ref = ol.eval_points_f64(W.astype(np.complex128), begin, end, ol.thresholds(zl), P.reshape(-1, 3))
        assert max(rel_l2(g, ref)) < TOL


@pytest.mark.parametrize("start,d,decay", [
    ((9.0e4, -3.0, 0.5), (0.11, 0.07, 0.8), 0.0),        # coordinates rounded to 0.008
    ((0.0, 0.0, 0.5), (4.0e4, 0.07, 0.8), 0.0),          # a million turns in a tile
    ((-3.0, 1.7, 0.5), (1.9, 0.4, 0.8), 0.5),            # growth along x beyond the operands' scale
])
def test_hard_grids(ctx, start, d, decay):
    got, ref = _volume(ctx, (20, 90), [0.0], start, d, (45, 20, 1), seed=5, decay=decay)
    assert max(rel_l2(got, ref)) < TOL_SUM


def test_not_finite(ctx):
    """An infinite amplitude spoils its own component only; a NaN wave vector everything in its region."""
    def amplitude(W):
        W[7, 0] = np.inf

    def vector(W):
        W[7, 3] = np.nan
    got, ref = _volume(ctx, (20, 90), [0.0], (-3.1, 1.7, -0.4), (0.11, 0.07, 0.83), (41, 20, 2), edit=amplitude)
    assert not np.isfinite(got[0, ..., 0]).any()
    assert max(rel_l2(got[0, ..., 1:].repeat(2, -1)[..., :3], ref[0, ..., 1:].repeat(2, -1)[..., :3])) < TOL
    assert max(rel_l2(got[1], ref[1])) < TOL
    got, ref = _volume(ctx, (20, 90), [0.0], (-3.1, 1.7, -0.4), (0.11, 0.07, 0.83), (41, 20, 2), edit=vector)
    assert np.isnan(got[0]).all()
    assert max(rel_l2(got[1], ref[1])) < TOL_SUM


def test_more_tiles_than_one_launch(ctx):
    got, ref = _volume(ctx, (10, 4100), [-1.0], (0.3, 0.2, -0.9), (0.1, 0.1, 1e-3), (1, 1, 2100), decay=0.2)
    assert max(rel_l2(got, ref)) < TOL
