"""The plan of a solve, host code only: which eigen-solver it chooses."""
import glob
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG = os.path.join(ROOT, "scwatter_gb300")
MAIN = r"""
#include <cstdio>
#include <cstdlib>
#include "solve_plan.h"
int main(int, char** a) {
    scw_solve_params q{};
    q.lambda = 1.0;
    q.direction[2] = 1.0;
    q.ex[0] = 1.0;
    q.n[0] = q.n[1] = 1.0;
    const int c0 = std::atoi(a[1]), c1 = std::atoi(a[2]);
    q.size[0] = q.size[1] = 400.0;
    q.size[2] = 1.0;
    q.coef[0] = c0;
    q.coef[1] = c1;
    q.pz = 1;
    q.eig_fp64 = std::atoi(a[3]);
    scw::sv::SolvePlan p;
    if (scw::sv::plan_solve(&q, 1, c1, c0, p) != SCW_OK) return 1;
    std::printf("%d %d\n", p.n, p.eig_mixed ? 1 : 0);
    return 0;
}
"""


@pytest.fixture(scope="module")
def plan(tmp_path_factory):
    from scwatter_gb300 import build
    build.build()
    d = tmp_path_factory.mktemp("plan")
    (d / "main.cpp").write_text(MAIN)
    exe = str(d / "plan")
    objs = sorted(glob.glob(os.path.join(PKG, "_obj", "*.o")))
    subprocess.run([build.NVCC, "-std=c++17", "-I", os.path.join(PKG, "csrc"), "-o", exe, str(d / "main.cpp"), *objs, "-lcudart", "-ldl"],
                   check=True)
    return lambda *args: [int(v) for v in subprocess.run([exe, *map(str, args)], check=True, capture_output=True, text=True).stdout.split()]


@pytest.mark.parametrize("c0,c1,fp64,n,mixed", [(3, 5, 0, 30, 1), (3, 5, 1, 30, 0), (64, 32, 0, 4096, 1), (89, 23, 0, 4094, 1),
                                                (683, 3, 0, 4098, 0), (50, 50, 0, 5000, 0)])
def test_eigen_solver(plan, c0, c1, fp64, n, mixed):
    """Orders above 4096 go to the FP64 solver: the mixed one refuses them."""
    assert plan(c0, c1, fp64) == [n, mixed]
