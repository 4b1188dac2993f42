"""CUDA calls that fail, made to by a library loaded before the runtime (host side only: an allocation that cannot be had, an
error code in place of a call, little memory left): what can go on without it does, and an error leaves the context as it was."""
import os
import subprocess
import sys
import textwrap

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SHIM = r"""
#define _GNU_SOURCE
#include <dlfcn.h>
#include <stddef.h>
static int malloc_at = -1, wait_at = -1;          /* calls until the one that fails */
static size_t free_bytes;                         /* what cudaMemGetInfo says, unless zero */
void shim_malloc(int at) { malloc_at = at; }
void shim_wait(int at) { wait_at = at; }
void shim_free(size_t n) { free_bytes = n; }
static void* runtime(const char* name) { return dlsym(dlopen("libcudart.so.13", RTLD_LAZY | RTLD_NOLOAD), name); }
int cudaMalloc(void** p, size_t n) {
    static int (*next)(void**, size_t);
    if (!next) next = (int (*)(void**, size_t))runtime("cudaMalloc");
    return next(p, malloc_at >= 0 && malloc_at-- == 0 ? (size_t)1 << 50 : n);
}
int cudaMemGetInfo(size_t* f, size_t* t) {
    int r = ((int (*)(size_t*, size_t*))runtime("cudaMemGetInfo"))(f, t);
    if (free_bytes) *f = free_bytes;
    return r;
}
int cudaStreamWaitEvent(void* s, void* e, unsigned f) {
    static int (*next)(void*, void*, unsigned);
    if (!next) next = (int (*)(void*, void*, unsigned))runtime("cudaStreamWaitEvent");
    return wait_at >= 0 && wait_at-- == 0 ? 999 : next(s, e, f);
}
"""


@pytest.fixture(scope="module")
def shim(tmp_path_factory):
    d = tmp_path_factory.mktemp("shim")
    (d / "shim.c").write_text(SHIM)
    subprocess.run(["gcc", "-shared", "-fPIC", "-o", str(d / "shim.so"), str(d / "shim.c"), "-ldl"], check=True)
    return str(d / "shim.so")


def _child(shim, body):
    head = """
    import ctypes, os, sys
    import numpy as np
    sys.path.insert(0, %r)
    shim = ctypes.CDLL(%r)
    from scwatter_gb300 import _lib, evaluator as ev, separable as sp, synthetic as syn
    ctx = ev.Context(0)
    def stream():
        s = ctypes.c_void_p()
        _lib.call("scw_ctx_stream", ctx.handle, ctypes.byref(s))
        return s.value
    def new_set():
        return sp.SeparableSet.from_factored(ctx, syn.make_factored(5, 6, 3, size=(18.0, 18.0, 3.0), seed=1, dtype=np.complex64))
    def planes(s):
        f = np.float32
        return s.evaluate_planes_host(f(-9), f(-9), f(-2), f(0.3), f(-0.4), f(0.2), f(0.4), 45)
    def same(a, b):
        return all(np.array_equal(x, y) for x, y in zip(a, b))
    """ % (ROOT, shim)
    code = textwrap.dedent(head) + textwrap.dedent(body) + "\nprint('ok', flush=True)\nos._exit(0)\n"
    r = subprocess.run([sys.executable, "-c", code], env=dict(os.environ, LD_PRELOAD=shim), capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.strip().endswith("ok"), r.stdout + r.stderr


def test_planes_in_turn_where_three_do_not_fit(shim):
    _child(shim, """
    ref = planes(new_set())
    ctx = ev.Context(0)
    s = new_set()
    shim.shim_malloc(1)                # the planes' output is allocated, then the scratch of all three
    assert same(planes(s), ref)
    """)


def test_product_without_room_for_its_digits(shim):
    _child(shim, """
    import torch
    A, B = (torch.randn(1, 70, 70, dtype=torch.complex128, device="cuda") for _ in range(2))
    C = torch.zeros_like(A)
    torch.cuda.synchronize()
    one, zero = (ctypes.c_double * 2)(1, 0), (ctypes.c_double * 2)(0, 0)
    shim.shim_malloc(0)
    _lib.call("scw_zgemm", ctx.handle, 70, 70, 70, one, *(ctypes.c_void_p(t.data_ptr()) for t in (A, B)), zero,
              ctypes.c_void_p(C.data_ptr()), 1)
    ctx.synchronize()
    assert (C - A @ B).abs().max().item() < 1e-12
    """)


@pytest.mark.parametrize("at", range(3))
def test_planes_leave_the_context_on_its_stream(shim, at):
    _child(shim, """
    ref = planes(new_set())
    s = new_set()
    planes(s)
    mine = stream()
    shim.shim_wait(%d)                 # of the waits of the second and third plane
    try:
        planes(s)
        raise SystemExit("no error")
    except _lib.ScwError as e:
        assert e.status == 4
    assert stream() == mine
    del s
    assert same(planes(new_set()), ref)
    """ % at)


def test_batch_lanes_where_memory_is_short(shim):
    """Digits of whole batches of slices give way to lanes.  30 slices of order 98: arenas of about 40 MB, 65 with them."""
    _child(shim, """
    from scwatter_gb300 import batch as bt, samples
    def batch(lanes):
        items = [bt.BatchItem(sample=samples.spheres((30, 16, 16), n_spheres=3, radius=(2, 5), seed=i),
                              grid=(-8, -8, -20, 1.0, 1.0, 4.0, 16, 15, 10), lam=1.0, direction=(0, 0, 1), ex=(1, 0), ey=(0, 0),
                              size=(16.0, 16.0, 30.0), coef=(7, 7)) for i in range(4)]
        return bt.Batch(ctx, items, lanes=lanes, method=2)
    shim.shim_free(ctypes.c_size_t(210 << 20))
    b = batch(4)
    shim.shim_free(ctypes.c_size_t(0))
    assert b.info()["lanes"] == 4, b.info()["lanes"]
    b.run()
    assert not b.wait().any()
    ref = batch(4)
    ref.run()
    assert not ref.wait().any()
    for i in range(4):
        for u, v in zip(b.result(i), ref.result(i)):
            assert np.abs(u - v).max() <= 1e-5 * np.abs(v).max()
    """)


def test_solve_without_room_for_a_batch_of_digits(shim):
    _child(shim, """
    from scwatter_gb300 import solver, samples
    kw = dict(lam=1.0, direction=(0, 0, 1), ex=(1, 0), ey=(0, 0), size=(16.0, 16.0, 6.0), coef=(5, 5))
    s = samples.spheres((6, 16, 16), n_spheres=3, radius=(2, 5), seed=1)
    ref = solver.solve(s, ctx=ctx, **kw).x
    shim.shim_malloc(0)                # the solve's arena
    x = solver.solve(s, ctx=ctx, **kw).x
    assert np.abs(x - ref).max() <= 1e-11 * np.abs(ref).max()
    """)


def test_eigen_solvers_without_room_for_digits(shim):
    _child(shim, """
    import torch
    A0 = torch.randn(3, 40, 40, dtype=torch.complex128, device="cuda")
    for name, at in (("scw_zgeev_mixed", 2), ("scw_zgeev", 2)):        # work, status, digits
        A, V = A0.clone(), torch.zeros_like(A0)
        W = torch.zeros(3, 40, dtype=torch.complex128, device="cuda")
        torch.cuda.synchronize()
        shim.shim_malloc(at)
        more = (None, None, None) if name == "scw_zgeev_mixed" else (None,)
        _lib.call(name, ctx.handle, 40, *(ctypes.c_void_p(t.data_ptr()) for t in (A, W, V)), 3, *more)
        R = A0 @ V - V * W[:, None, :]
        assert (torch.linalg.norm(R) / torch.linalg.norm(A0) / torch.linalg.norm(V)).item() < 1e-12
    """)
