"""CUDA calls that fail, made to by a library loaded before the runtime (host side only: an allocation that cannot be had, an
error code in place of a call): what can go on without it does, and an error leaves the context as it was."""
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
void shim_malloc(int at) { malloc_at = at; }
void shim_wait(int at) { wait_at = at; }
static void* runtime(const char* name) { return dlsym(dlopen("libcudart.so.13", RTLD_LAZY | RTLD_NOLOAD), name); }
int cudaMalloc(void** p, size_t n) {
    static int (*next)(void**, size_t);
    if (!next) next = (int (*)(void**, size_t))runtime("cudaMalloc");
    return next(p, malloc_at >= 0 && malloc_at-- == 0 ? (size_t)1 << 50 : n);
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
