"""The pairs of components in which a solve's boundary system is written (host code): no division by a small Sz where a harmonic
grazes an outer medium, and the solution of the full system of order 6 MF in extended precision."""
import glob
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG = os.path.join(ROOT, "scwatter_gb300")
MAIN = r"""
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include "solve_plan.h"
static void put(double2 v) { std::printf("%.17g %.17g ", v.x, v.y); }
int main(int, char** a) {
    scw_solve_params q{};
    const double sx = std::atof(a[1]), sy = std::atof(a[2]);
    q.lambda = 1.0;
    q.direction[0] = sx;
    q.direction[1] = sy;
    q.direction[2] = std::sqrt(1 - sx * sx - sy * sy);
    q.ex[0] = 1.0;
    q.n[0] = 1.0;
    q.n[1] = std::atof(a[3]);
    q.size[0] = q.size[1] = 16.0;
    q.size[2] = 1.0;
    q.coef[0] = 5;
    q.coef[1] = std::atoi(a[4]);
    q.pz = 1;
    scw::sv::SolvePlan p;
    if (scw::sv::plan_solve(&q, 1, 16, 16, p) != SCW_OK) return 1;
    for (int m = 0; m < p.MF; m++) {
        const scw::sv::BcPair& h = p.bc[m];
        std::printf("%.17g %.17g ", p.Sx[m], p.Sy[m]);
        put(make_double2(p.Sz0[m].real(), p.Sz0[m].imag()));
        put(make_double2(p.Sz1[m].real(), p.Sz1[m].imag()));
        for (const double2& v : h.L) put(v);
        for (const double2& v : h.M) put(v);
        for (const double2& v : h.Fi) put(v);
        for (const double2& v : h.r1) put(v);
        for (const double2& v : h.r0) put(v);
        std::printf("%d %d %d %d %d %d\n", h.c1, h.c0, h.p[0], h.p[1], h.q[0], h.q[1]);
    }
    return 0;
}
"""


@pytest.fixture(scope="module")
def pairs(tmp_path_factory):
    from scwatter_gb300 import build
    build.build()
    d = tmp_path_factory.mktemp("pairs")
    (d / "main.cpp").write_text(MAIN)
    exe = str(d / "pairs")
    objs = sorted(glob.glob(os.path.join(PKG, "_obj", "*.o")))
    subprocess.run([build.NVCC, "-std=c++17", "-I", os.path.join(PKG, "csrc"), "-o", exe, str(d / "main.cpp"), *objs, "-lcudart", "-ldl"],
                   check=True)

    def run(*args):
        out = subprocess.run([exe, *map(repr, args)], check=True, capture_output=True, text=True).stdout
        v = np.array([[float(t) for t in line.split()] for line in out.splitlines()])
        cplx = lambda a: a[:, ::2] + 1j * a[:, 1::2]  # noqa: E731
        return v[:, 0], v[:, 1], cplx(v[:, 2:6]), cplx(v[:, 6:46]), v[:, 46:].astype(int)
    return run


def _solve(A, b):
    """Gaussian elimination with partial pivoting in extended precision."""
    A, x = A.astype(np.clongdouble), b.astype(np.clongdouble)
    n = len(x)
    for k in range(n):
        p = k + int(np.argmax(abs(A[k:, k])))
        A[[k, p]], x[[k, p]] = A[[p, k]], x[[p, k]]
        f = A[k + 1:, k] / A[k, k]
        A[k + 1:] -= f[:, None] * A[k]
        x[k + 1:] -= f * x[k]
    for k in range(n - 1, -1, -1):
        x[k] = (x[k] - A[k, k + 1:] @ x[k + 1:]) / A[k, k]
    return x


@pytest.mark.parametrize("sz", [0.3, 0.05, 0.0201, 0.0199, 1e-4, 1e-7])
@pytest.mark.parametrize("n1,c1", [(1.0, 1), (1.3, 1), (1.3, 3)])
def test_pairs(pairs, sz, n1, c1):
    Sx, Sy, Sz, v, idx = pairs(float(np.sqrt(1 - sz * sz) - 2 / 16), 0.0, n1, c1)   # the p = 2 harmonic leaves at Sz = sz
    MF = len(Sx)
    assert min(abs(Sz[:, 0])) < 1.01 * sz + 1e-7
    L, M, Fi, r1, r0 = v[:, :8].reshape(MF, 4, 2), v[:, 8:12].reshape(MF, 2, 2), v[:, 12:16].reshape(MF, 2, 2), v[:, 16:18], v[:, 18:20]
    # nothing is magnified: ratios at most 1, the rows' inverse bounded by their determinant's choice
    assert abs(r1).max() <= 1 + 1e-15 and abs(r0).max() <= 1 + 1e-15
    assert abs(Fi).max() <= 4 and abs(M).max() <= 4
    rng = np.random.default_rng(MF)
    cn = lambda *s: rng.standard_normal(s) + 1j * rng.standard_normal(s)  # noqa: E731
    G = np.eye(4 * MF) + 0.3 * cn(4 * MF, 4 * MF) / np.sqrt(4 * MF)      # Gd_0 Gc_static^-1
    f = cn(4 * MF)
    D, O, E = np.diag, np.zeros((MF, MF)), np.eye(MF)
    S0, S1 = Sz[:, 0], Sz[:, 1]
    f3 = np.block([[-E, O, O], [O, -E, O], [O, D(S1), -D(Sy)], [-D(S1), O, D(Sx)]])
    f2 = np.block([[E, O, O], [O, E, O], [O, D(S0), D(Sy)], [-D(S0), O, -D(Sx)]])
    Z3 = np.zeros((MF, 3 * MF))
    full = np.block([[np.hstack([D(Sx), D(Sy), -D(S0)]), Z3], [Z3, np.hstack([D(Sx), D(Sy), D(S1)])], [f2, G @ f3]])
    ref = _solve(full, np.concatenate([np.zeros(2 * MF), -f]))
    # by the pairs
    F3 = np.zeros((4 * MF, 2 * MF), complex)
    for m in range(MF):
        for q in range(4):
            F3[q * MF + m, [m, MF + m]] = L[m, q]
    t = np.hstack([G @ F3, -f[:, None]])
    A = np.zeros((2 * MF, 2 * MF + 1), complex)
    for m in range(MF):
        _, _, p0, p1, q0, q1 = idx[m]
        for k, q in enumerate((q0, q1)):
            A[k * MF + m] = t[q * MF + m] - M[m, k, 0] * t[p0 * MF + m] - M[m, k, 1] * t[p1 * MF + m]
    tau = np.linalg.solve(A[:, :-1], A[:, -1])
    r = t[:, :-1] @ tau
    x = np.zeros(6 * MF, complex)

    def put(base, m, c, ratio, u):
        a, b = [i for i in range(3) if i != c]
        x[base + a * MF + m], x[base + b * MF + m], x[base + c * MF + m] = u[0], u[1], ratio @ u
    for m in range(MF):
        put(3 * MF, m, idx[m][0], r1[m], tau[[m, MF + m]])
        put(0, m, idx[m][1], r0[m], Fi[m] @ np.array([-f[p * MF + m] - r[p * MF + m] for p in idx[m][2:4]]))
    # an LU of order 2 MF with a condition of a few
    assert np.linalg.norm((x - ref).astype(complex)) <= 2 * MF * 10 * 2.0 ** -53 * np.linalg.norm(ref.astype(complex))
