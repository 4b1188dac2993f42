"""The work that users of this package have it do, as measurable cases.

Three programs use the package: the viewer (three planes of a structure into host arrays), the
field evaluation of whole volumes (device buffers, or streamed from host amplitudes), and the
volume solver (a refractive-index sample in, boundary amplitudes and the field out; one sample
at a time or many in one batch graph).  A case is a dict of plain values; ``kind`` selects the
program, the other keys are its sizes and options.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from scwatter_gb300 import batch as bt
from scwatter_gb300 import evaluator as ev
from scwatter_gb300 import samples
from scwatter_gb300 import separable as sp
from scwatter_gb300 import solver as sv
from scwatter_gb300 import synthetic as syn

_ctx = None


def context():
    """One context per process, as a program keeps it."""
    global _ctx
    if _ctx is None:
        _ctx = ev.Context(0)
    return _ctx


METHODS = {"fp32": sp.FP32, "tf32x3": sp.TF32X3, "bf16x3": sp.BF16X3}


def listed():
    return [
        # the viewer on a small structure (3 x 3 harmonics, 2 slices): launch and copy latency
        dict(name="planes_small", kind="planes", M0=3, M1=3, Z=2, N=64),
        # the viewer at a size between its resolutions on a 16 x 20 structure, plain summation
        dict(name="planes_large", kind="planes", M0=16, M1=20, Z=2, N=200),
        # a volume by plain summation: the drop-in for structures that do not factor
        dict(name="volume_plain", kind="volume_plain", M0=8, M1=9, Z=4, Nx=101, Ny=77, Nz=50),
        # the viewer with the separable evaluator on a structure read from a .cw file (two halves)
        dict(name="planes_sep", kind="planes_sep", M0=20, M1=20, Z=3, N=256, method="fp32"),
        # a small separable volume: one item of an uneven set
        dict(name="volume_small", kind="volume", M0=8, M1=13, Z=5, Nx=65, Ny=71, Nz=33, method="bf16x3"),
        # the [20, 64, 64] sphere workload on its 128 x 128 x 64 grid
        dict(name="volume_mid", kind="volume", M0=20, M1=20, Z=20, Nx=128, Ny=128, Nz=64, method="tf32x3"),
        # the [64, 128, 128] sphere workload at 40 x 40 harmonics on its 512 x 512 x 256 grid
        dict(name="volume_full", kind="volume", M0=40, M1=40, Z=64, Nx=512, Ny=512, Nz=256, method="tf32x3"),
        # a volume from host amplitudes to host planes, page-locked on both sides
        dict(name="volume_host", kind="volume_host", M0=20, M1=20, Z=20, Nx=160, Ny=144, Nz=64, method="tf32x3"),
        # a first look at a small sample: 5 x 5 harmonics, 4 layers
        dict(name="solve_small", kind="solve", sample="spheres", Z=4, Y=16, X=16, c0=5, c1=5, lam=1.0, angle=0.0,
             Nx=32, Ny=32, Nz=16),
        # a smoothly varying sample under oblique incidence
        dict(name="solve_mid", kind="solve", sample="grf", Z=10, Y=64, X=64, c0=12, c1=9, lam=0.9, angle=20.0,
             Nx=96, Ny=80, Nz=40),
        # the [20, 64, 64] sphere sample at 18 x 18 harmonics
        dict(name="solve_large", kind="solve", sample="spheres", Z=20, Y=64, X=64, c0=18, c1=18, lam=1.0, angle=0.0,
             Nx=128, Ny=128, Nz=64),
        # several samples of uneven sizes in one graph
        dict(name="batch_uneven", kind="batch", count=6, m_lo=6, m_hi=12, z_lo=4, z_hi=10, pixels=64, n_xy=64, n_z=32),
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["planes", "volume_plain", "planes_sep", "volume", "volume", "volume_host", "solve", "solve",
                       "batch"])
    if kind == "planes":
        return dict(kind=kind, M0=rng.randint(2, 16), M1=rng.randint(2, 16), Z=rng.randint(1, 3),
                    N=_logint(rng, 33, 256))
    if kind == "volume_plain":
        return dict(kind=kind, M0=rng.randint(2, 9), M1=rng.randint(2, 9), Z=rng.randint(1, 6),
                    Nx=_logint(rng, 17, 120), Ny=_logint(rng, 17, 120), Nz=_logint(rng, 5, 50))
    if kind == "planes_sep":
        return dict(kind=kind, M0=rng.randint(3, 20), M1=rng.randint(3, 20), Z=rng.randint(1, 4),
                    N=_logint(rng, 32, 512), method=rng.choice(sorted(METHODS)))
    if kind in ("volume", "volume_host"):
        host = kind == "volume_host"
        return dict(kind=kind, M0=rng.randint(4, 20 if host else 32), M1=rng.randint(4, 20 if host else 32),
                    Z=rng.randint(2, 20), Nx=_logint(rng, 33, 200 if host else 512),
                    Ny=_logint(rng, 33, 200 if host else 512), Nz=_logint(rng, 9, 64 if host else 128),
                    method=rng.choice(["tf32x3", "tf32x3", "bf16x3"]))
    if kind == "solve":
        pix = rng.choice([16, 32, 64])
        return dict(kind=kind, sample=rng.choice(["spheres", "grf"]), Z=rng.randint(1, 20), Y=pix, X=pix,
                    c0=rng.randint(3, min(16, pix // 2)), c1=rng.randint(3, min(16, pix // 2)),
                    lam=round(rng.uniform(0.8, 1.2), 3), angle=round(rng.choice([0.0, rng.uniform(1.0, 30.0)]), 2),
                    Nx=_logint(rng, 24, 128), Ny=_logint(rng, 24, 128), Nz=_logint(rng, 8, 64))
    lo = rng.randint(3, 7)
    return dict(kind=kind, count=rng.randint(2, 6), m_lo=lo, m_hi=lo + rng.randint(1, 5), z_lo=rng.randint(1, 4),
                z_hi=rng.randint(5, 10), pixels=rng.choice([32, 64]), n_xy=rng.randint(33, 80), n_z=rng.randint(9, 32))


# ------------------------------------------------------------------------------------------
# inputs
# ------------------------------------------------------------------------------------------
def _size(c):
    """Extent of a coefficient set's sample: 3.2 wavelengths per harmonic, 1 per slice."""
    return 3.2 * max(c["M0"], c["M1"]), 3.2 * max(c["M0"], c["M1"]), float(c["Z"])


def _factored(c, seed):
    return syn.make_factored(c["M0"], c["M1"], c["Z"], size=_size(c), seed=seed, dtype=np.complex64)


def _paired(c, seed):
    return syn.device_paired(c["M0"], c["M1"], c["Z"], size=_size(c), seed=seed)


def _volume_grid(c, seed):
    """x0, y0, z0, dx, dy, dz (float32 values): the sample's x, y extent and its depth."""
    r = np.random.default_rng([seed, 7])
    sx, sy, sz = _size(c)
    f = lambda v: float(np.float32(v))  # noqa: E731
    off = float(r.uniform(0.01, 0.04))
    span = 0.96 if c["kind"] != "volume_plain" else 1.3      # the plain volume also sees both outer media
    return (f(-sx / 2 + off), f(-sy / 2 + off), f(-span * sz / 2 + off), f(sx / max(1, c["Nx"] - 1)),
            f(sy / max(1, c["Ny"] - 1)), f(span * sz / max(1, c["Nz"])))


def _plane_grid(c, seed):
    """x_start, y_start, z_start, x, y, z, d of the viewer's three planes."""
    r = np.random.default_rng([seed, 8])
    sx = _size(c)[0]
    f = lambda v: float(np.float32(v))  # noqa: E731
    ext = sx
    z = (int(r.integers(0, c["Z"])) + float(r.uniform(0.2, 0.8))) - c["Z"] / 2.0
    return (f(-ext / 2), f(-ext / 2), f(-ext / 2 + 0.013), f(r.uniform(-1, 1)), f(r.uniform(-1, 1)), f(z),
            f(ext / (c["N"] - 1)))


def _sample(c, seed):
    shape = (c["Z"], c["Y"], c["X"])
    if c["sample"] == "grf":
        return samples.gaussian_random_field(shape, corr_px=8.0, seed=seed)
    return samples.spheres(shape, n_spheres=max(2, c["Z"] // 3), radius=(c["X"] / 16, c["X"] / 6), seed=seed)


def _solve_options(c, seed):
    th, ph = math.radians(c["angle"]), 0.4 + 0.1 * (seed % 7)
    d = (math.sin(th) * math.cos(ph), math.sin(th) * math.sin(ph), math.cos(th))
    return dict(lam=c["lam"], direction=d, ex=(1.0, 0.0), ey=(0.0, 0.0), size=(float(c["X"]), float(c["Y"]),
                                                                               float(c["Z"])), coef=(c["c0"], c["c1"]))


def _solve_grid(c):
    f = lambda v: float(np.float32(v))  # noqa: E731
    return (f(-c["X"] / 2), f(-c["Y"] / 2), f(-0.97 * c["Z"]), f(c["X"] / (c["Nx"] - 1)), f(c["Y"] / (c["Ny"] - 1)),
            f(1.94 * c["Z"] / (c["Nz"] - 1)))


def _batch_items(c, seed):
    items = bt.uneven_items(c["count"], seed=seed % 100000, m_range=(c["m_lo"], c["m_hi"]),
                            z_range=(c["z_lo"], c["z_hi"]), grid_xy=(c["n_xy"] // 2, c["n_xy"]),
                            grid_z=(max(4, c["n_z"] // 2), c["n_z"]), lam_range=(0.8, 1.2), pixels=c["pixels"])
    return items


def _batch_sizes(c):
    """Harmonics, slices and grids are the case's, not the seed's: the items of every seed have the
    sizes of seed 0 and samples, directions and wavelengths of their own."""
    return [(it.coef, it.sample.shape[0], it.grid) for it in _batch_items(c, 0)]


def _batch(c, seed):
    out = []
    for i, (coef, Z, grid) in enumerate(_batch_sizes(c)):
        it = _batch_items(dict(c, z_lo=Z, z_hi=Z), seed)[i]
        it.coef, it.grid = coef, grid
        it.size = (float(c["pixels"]), float(c["pixels"]), float(Z))
        out.append(it)
    return out


def prepare(case, seed):
    c, ctx = case, context()
    k = c["kind"]
    st = dict(case=c)
    if k in ("planes", "volume_plain"):
        fs = _factored(c, seed)
        st["set"] = ev.WaveSet.from_cw(ctx, syn.to_structure(fs))
    elif k == "planes_sep":
        st["set"] = sp.SeparableSet.from_factored(ctx, _factored(c, seed))
    elif k in ("volume", "volume_host"):
        ps, V = _paired(c, seed)
        torch.cuda.synchronize()
        st["set"] = sp.SeparableSet.from_paired(ctx, ps, V)
        if k == "volume_host":
            st["amplitudes"] = V.cpu().pin_memory()
            st["out"] = torch.empty((c["Nz"], c["Ny"], c["Nx"], 3), dtype=torch.complex64).pin_memory()
        del V
    elif k == "solve":
        st["sample"], st["options"], st["grid"] = _sample(c, seed), _solve_options(c, seed), _solve_grid(c)
    elif k == "batch":
        st["batch"] = bt.Batch(ctx, _batch(c, seed), lanes=4, method=sp.TF32X3)
    if k in ("planes", "planes_sep"):
        st["grid"] = _plane_grid(c, seed)
    if k in ("volume_plain", "volume", "volume_host"):
        st["grid"] = _volume_grid(c, seed)
    if k in ("volume_plain", "volume", "solve"):
        st["out"] = torch.empty((c["Nz"], c["Ny"], c["Nx"], 3), dtype=torch.complex64, device="cuda")
    torch.cuda.synchronize()
    return st


def run(state):
    c = state["case"]
    k = c["kind"]
    if k == "planes":
        return state["set"].evaluate_planes_host(*state["grid"], c["N"])
    if k == "planes_sep":
        return state["set"].evaluate_planes_host(*state["grid"], c["N"], method=METHODS[c["method"]])
    if k == "volume_plain":
        state["set"].eval_volume_device(*state["grid"], c["Nx"], c["Ny"], c["Nz"], state["out"].data_ptr())
        return state["out"]
    if k == "volume":
        state["set"].eval_volume_device(*state["grid"], c["Nx"], c["Ny"], c["Nz"], state["out"].data_ptr(),
                                        method=METHODS[c["method"]])
        return state["out"]
    if k == "volume_host":
        return state["set"].eval_volume_host(state["amplitudes"], *state["grid"], c["Nx"], c["Ny"], c["Nz"],
                                             out=state["out"], method=METHODS[c["method"]])
    if k == "solve":
        # boundary amplitudes, spectrum (the order in which the modes come has no meaning: by real
        # part here) and the field of the solved sample
        sol = sv.solve(state["sample"], ctx=context(), **state["options"])
        sep = sol.to_sep()
        sep.eval_volume_device(*state["grid"], c["Nx"], c["Ny"], c["Nz"], state["out"].data_ptr(), method=sp.TF32X3)
        context().synchronize()
        return {"x": sol.x, "gamma2": np.sort(sol.gamma ** 2, axis=1), "field": state["out"]}
    b = state["batch"]
    b.run()
    if b.wait().any():
        raise RuntimeError("an item of the batch failed")
    out = []
    for i in range(c["count"]):
        x, g, f = b.result(i)
        out.append({"x": x, "gamma2": np.sort(g ** 2, axis=1), "field": f})
    return out


# ------------------------------------------------------------------------------------------
# work: the operations and bytes of the separable forms, which any evaluation can use, and the
# operation counts of the dense algebra of a solve
# ------------------------------------------------------------------------------------------
def _volume_work(M0, M1, planes, Nx, Ny, Z, halves):
    MF = M0 * M1
    coef = Z * halves * 3 * MF * 2 * MF * 8
    macs = planes * 3 * (MF * 2 * MF * halves + M0 * M1 * Ny + M0 * Nx * Ny)
    return coef + planes * Nx * Ny * 24, 8 * macs


def _solve_work(Z, c0, c1, Y, X, Nx, Ny, Nz):
    MF = c0 * c1
    n = 2 * MF
    # per slice: P Q, eigenpairs (25 n^3 complex operations), Q U, two factorisations, four products
    # with 3 MF columns, Ez rows; then the 6 MF boundary system
    cmacs = Z * (n ** 3 * (1 + 12.5 + 1 + 2 / 3 + 6) + MF * MF * n) + (6 * MF) ** 3 / 3
    b, f = _volume_work(c0, c1, Nz, Nx, Ny, Z, 1)
    return Z * Y * X * 16 + b, 8 * cmacs + f


def work(case):
    c = case
    k = c["kind"]
    if k in ("planes", "planes_sep"):
        MF, N = c["M0"] * c["M1"], c["N"]
        # xy: one z; xz and yz: N values of z, one row of points each
        macs = 3 * ((1 + 2 * N) * MF * 4 * MF + 3 * MF * N + 3 * c["M0"] * N * N)
        b, f = c["Z"] * 2 * 3 * MF * 2 * MF * 8 + 3 * N * N * 24, 8 * macs
    elif k in ("volume_plain", "volume", "volume_host"):
        b, f = _volume_work(c["M0"], c["M1"], c["Nz"], c["Nx"], c["Ny"], c["Z"], 2 if k == "volume_plain" else 1)
    elif k == "solve":
        b, f = _solve_work(c["Z"], c["c0"], c["c1"], c["Y"], c["X"], c["Nx"], c["Ny"], c["Nz"])
    else:
        b = f = 0
        for coef, Z, g in _batch_sizes(c):
            w = _solve_work(Z, coef[0], coef[1], c["pixels"], c["pixels"], *g[6:9])
            b, f = b + w[0], f + w[1]
    return {"bytes": float(b), "flops": float(f)}


# ------------------------------------------------------------------------------------------
# 64-bit results
# ------------------------------------------------------------------------------------------
_C = torch.complex128


def _t(a):
    return torch.as_tensor(a).to("cuda", _C)


def _axis(start, d, n):
    """start + d i, product and sum each rounded to float32."""
    return (np.float32(start) + np.float32(d) * np.arange(n, dtype=np.float32)).astype(np.float64)


def _region(z, zb):
    """The last boundary with z >= z_l - 0.001: -1 above the sample, Z below it."""
    r = -1
    for l, b in enumerate(np.asarray(zb, np.float32).astype(np.float64)):
        if float(np.float32(z)) >= b - 0.001:
            r = l
    return r


class _Exact:
    """Field of a set of modes: block(l) gives (Q_dn, Q_up) [3, MF, J] of slice l."""

    def __init__(self, kx, ky, zb, kz_dn, kz_up, block, ext):
        self.kx, self.ky = torch.as_tensor(kx).cuda(), torch.as_tensor(ky).cuda()
        self.zb, self.kz_dn, self.kz_up, self.block, self.ext = zb, kz_dn, kz_up, block, ext

    def coefficients(self, zs):
        """[len(zs), 3, MF]"""
        Z = len(self.zb) - 1
        reg = [_region(z, self.zb) for z in zs]
        MF = len(self.kx) * len(self.ky)
        C = torch.zeros((len(zs), 3, MF), dtype=_C, device="cuda")
        inc, kzi, refl, kzr, trans, kzt = [_t(a) for a in self.ext]
        z = torch.as_tensor(np.asarray(zs, np.float64)).cuda()
        for l in sorted(set(reg)):
            at = torch.as_tensor([i for i, r in enumerate(reg) if r == l], device="cuda")
            zz = z[at][:, None]
            if l < 0:
                C[at] = (inc[None] * torch.exp(1j * kzi[None] * zz)[:, None]
                         + refl[None] * torch.exp(1j * kzr[None] * (zz - float(self.zb[0])))[:, None])
            elif l >= Z:
                C[at] = trans[None] * torch.exp(1j * kzt[None] * (zz - float(self.zb[Z])))[:, None]
            else:
                dn, up = self.block(l)
                pd = torch.exp(1j * _t(self.kz_dn[l])[None] * (zz - float(self.zb[l])))
                pu = torch.exp(1j * _t(self.kz_up[l])[None] * (zz - float(self.zb[l + 1])))
                J = pd.shape[1]
                C[at] = (dn.reshape(-1, J) @ pd.T + up.reshape(-1, J) @ pu.T).T.reshape(-1, 3, MF)
        return C

    def grid(self, xs, ys, zs):
        """[z, y, x, 3]"""
        C = self.coefficients(zs).reshape(len(zs), 3, len(self.kx), len(self.ky))
        ex = torch.exp(1j * torch.as_tensor(xs).cuda()[:, None] * self.kx[None])
        ey = torch.exp(1j * torch.as_tensor(ys).cuda()[:, None] * self.ky[None])
        out = torch.empty((len(zs), len(ys), len(xs), 3), dtype=_C, device="cuda")
        for i in range(len(zs)):
            out[i] = (ey @ C[i].transpose(1, 2) @ ex.T).permute(1, 2, 0)
        return out


def _exact_factored(c, seed):
    fs = _factored(c, seed)
    return _Exact(fs.kx, fs.ky, fs.z, fs.gamma_dn * fs.k, fs.gamma_up * fs.k,
                  lambda l: (_t(fs.Q_dn[l]), _t(fs.Q_up[l])),
                  (fs.inc, fs.kz_inc, fs.refl, fs.kz_refl, fs.trans, fs.kz_trans))


def _exact_paired(c, seed):
    ps, V = _paired(c, seed)
    b = ps.base
    flip = torch.tensor([1.0, 1.0, -1.0], dtype=torch.float64, device="cuda")[:, None, None]

    def block(l):
        v = V[l].to(_C)
        return v * _t(ps.beta_dn[l]), flip * v * _t(ps.beta_up[l])

    return _Exact(b.kx, b.ky, b.z, b.gamma_dn * b.k, b.gamma_up * b.k, block,
                  (b.inc, b.kz_inc, b.refl, b.kz_refl, b.trans, b.kz_trans))


def _crop(a, M1, M0):
    Y, X = a.shape
    s = np.fft.fftshift(np.fft.fft2(a) / (Y * X))
    r, q = Y // 2 - M1 // 2, X // 2 - M0 // 2
    return s[r:r + M1, q:q + M0]


def _exact_solve(sample, lam, direction, ex, ey, size, coef, grid, shape):
    """The coupled-wave solve in numpy, on the reduced problem of order 2 MF."""
    PI = 3.141592653                                     # the value the reference's grids use
    M0, M1 = coef
    MF, Z = M0 * M1, sample.shape[0]
    n = 2 * MF
    k = 2 * PI / lam
    d = np.asarray(direction) / np.linalg.norm(direction)
    e = np.array([complex(*ex), complex(*ey), 0j])
    e = e / np.sqrt(np.sum(e * e))
    e = np.cross(d, np.cross(e, d))
    ps, qs = np.arange(M0) - M0 // 2, np.arange(M1) - M1 // 2
    up, wq = 2 * PI * ps / size[0] + d[0] * k, 2 * PI * qs / size[1] + d[1] * k
    zb = -size[2] / 2 + np.concatenate([[0.0], np.cumsum(np.full(Z, size[2] / Z))])
    Sx, Sy = np.repeat(up / k, M1), np.tile(wq / k, M0)
    Sz = np.sqrt(1.0 + 0j - Sx ** 2 - Sy ** 2)
    EF = np.zeros((3, M0, M1), complex)
    EF[:, M0 // 2, M1 // 2] = e
    EF = EF.reshape(3, MF)
    upm, wqm = np.tile(up, M1), np.repeat(wq, M0)        # harmonic m = q M0 + p
    qm, pm = np.repeat(np.arange(M1), M0), np.tile(np.arange(M0), M1)
    R = ((np.fmod(qs[qm][:, None], M1) - np.fmod(qs[qm][None], M1) + M1) % M1 + M1 // 2) % M1
    Cc = ((np.fmod(ps[pm][:, None], M0) - np.fmod(ps[pm][None], M0) + M0) % M0 + M0 // 2) % M0
    I = np.eye(MF)
    U, W, G, E, KN = [], [], [], [], []
    for l in range(Z):
        S = sample[l].reshape(-1).reshape(sample.shape[2], sample.shape[1]).T
        nf, ni = _crop(S ** 2, M1, M0), _crop(S ** -2.0, M1, M0)
        NF, NI = nf[R, Cc], ni[R, Cc]
        u, w = upm[:, None], wqm[:, None]
        P = np.block([[u * NI * wqm, I * k * k - u * NI * upm], [w * NI * wqm - I * k * k, -w * NI * upm]]) / k ** 2
        Q = np.block([[-I * u * w / k ** 2, I * u * u / k ** 2 - NF], [NF - I * w * w / k ** 2, I * u * w / k ** 2]])
        lamb, v = np.linalg.eig(P @ Q)
        g = np.sqrt(lamb)
        g = np.where((g.imag < 0) | ((g.imag == 0) & (g.real < 0)), -g, g)
        U.append(v)
        W.append(Q @ v / g)
        G.append(g)
        E.append(np.exp(1j * k * g * (zb[l + 1] - zb[l])))
        lin = ((qm[:, None] - qm[None] + M1) % M1 + M1 // 2) % M1 * M0 + ((pm[:, None] - pm[None] + M0) % M0
                                                                          + M0 // 2) % M0
        KN.append(-ni.flatten(order="F")[lin] / k)
    O, D = np.zeros((MF, MF), complex), np.diag
    f2 = np.block([[I, O, O], [O, I, O], [O, D(Sz), D(Sy)], [-D(Sz), O, -D(Sx)]])
    f3 = np.block([[-I, O, O], [O, -I, O], [O, D(Sz), -D(Sy)], [-D(Sz), O, D(Sx)]])
    ph = np.exp(1j * k * zb[0] * Sz)
    f1 = np.concatenate([ph * EF[0], ph * EF[1], ph * (Sy * EF[2] - Sz * EF[1]), ph * (Sz * EF[0] - Sx * EF[2])])
    T = f3
    for l in range(Z - 1, -1, -1):
        a1, a2 = np.linalg.solve(U[l], T[:n]), np.linalg.solve(W[l], T[n:])
        yt, yb = (a1 + a2) / 2 / E[l][:, None], E[l][:, None] * (a1 - a2) / 2
        T = np.concatenate([U[l] @ (yt + yb), W[l] @ (yt - yb)])
    A = np.zeros((6 * MF, 6 * MF), complex)
    A[:MF, :3 * MF] = np.block([D(Sx), D(Sy), -D(Sz)])
    A[MF:2 * MF, 3 * MF:] = np.block([D(Sx), D(Sy), D(Sz)])
    A[2 * MF:, :3 * MF], A[2 * MF:, 3 * MF:] = f2, T
    x = np.linalg.solve(A, np.concatenate([np.zeros(2 * MF), -f1]))
    v = f1 + f2 @ x[:3 * MF]
    upz = np.tile(2 * ps * math.pi / size[0] + d[0] * k, M1)[:, None]
    wqz = np.repeat(2 * qs * math.pi / size[1] + d[1] * k, M0)[:, None]
    dn, upw = [], []
    for l in range(Z):
        b1, b2 = np.linalg.solve(U[l], v[:n]), np.linalg.solve(W[l], v[n:])
        bd, bu = (b1 + b2) / 2, (b1 - b2) / 2 / E[l]
        ez = KN[l] @ (upz * W[l][MF:] - wqz * W[l][:MF])
        dn.append(np.concatenate([U[l] * bd, ez * bd]).reshape(3, MF, n))
        upw.append(np.concatenate([U[l] * bu, -ez * bu]).reshape(3, MF, n))
        v = np.concatenate([U[l] @ (E[l] * bd + bu), W[l] @ (E[l] * bd - bu)])
    G = np.stack(G)
    f = _Exact(up, wq, zb, G * k, -G * k, lambda l: (_t(dn[l]), _t(upw[l])),
               (EF, Sz * k, x[:3 * MF].reshape(3, MF), -Sz * k, x[3 * MF:].reshape(3, MF), Sz * k))
    x0, y0, z0, dx, dy, dz = grid
    field = f.grid(_axis(x0, dx, shape[0]), _axis(y0, dy, shape[1]), _axis(z0, dz, shape[2]))
    return {"x": x, "gamma2": np.sort(G ** 2, axis=1), "field": field}


def exact(case, seed):
    c = case
    k = c["kind"]
    if k in ("planes", "planes_sep"):
        f = _exact_factored(c, seed)
        xs, ys, zs, x, y, z, d = _plane_grid(c, seed)
        X, Y, Zs = _axis(xs, d, c["N"]), _axis(ys, d, c["N"]), _axis(zs, d, c["N"])
        one = lambda v: np.array([np.float32(v)], np.float64)  # noqa: E731
        return (f.grid(X, Y, one(z))[0], f.grid(X, one(y), Zs)[:, 0], f.grid(one(x), Y, Zs)[:, :, 0])
    if k in ("volume_plain", "volume", "volume_host"):
        f = _exact_factored(c, seed) if k == "volume_plain" else _exact_paired(c, seed)
        x0, y0, z0, dx, dy, dz = _volume_grid(c, seed)
        return f.grid(_axis(x0, dx, c["Nx"]), _axis(y0, dy, c["Ny"]), _axis(z0, dz, c["Nz"]))
    if k == "solve":
        if c["Z"] * (2 * c["c0"] * c["c1"] / 250) ** 3 > 12:
            return None                                  # minutes of LAPACK
        o = _solve_options(c, seed)
        return _exact_solve(_sample(c, seed), o["lam"], o["direction"], o["ex"], o["ey"], o["size"], o["coef"],
                            _solve_grid(c), (c["Nx"], c["Ny"], c["Nz"]))
    items = _batch(c, seed)
    out, left = [], 12.0
    for it in items:
        left -= it.sample.shape[0] * (2 * it.coef[0] * it.coef[1] / 250) ** 3
        if left < 0:
            out.append({"x": None, "gamma2": None, "field": None})
        else:
            out.append(_exact_solve(it.sample, it.lam, it.direction, it.ex, it.ey, it.size, it.coef, it.grid[:6],
                                    it.grid[6:9]))
    return out
