"""Calls without a context (allocation-free gravity, the MLP) after a cudaDeviceReset, which ends the process's own device
context: the library's kernels come back with their default limits, and every device pointer and pool of before is gone.
Each case runs in a process of its own, with buffers from the CUDA runtime, since a reset would take torch's along."""
import subprocess
import sys
import textwrap

import pytest

pytestmark = pytest.mark.gpu

PROLOGUE = """
    import ctypes as C
    import numpy as np
    from cuda.bindings import runtime as rt
    from botheadstudios_b200 import _lib

    L = _lib.load()

    def ok(r):
        assert r[0] == rt.cudaError_t.cudaSuccess, r
        return r[1] if len(r) > 1 else None

    def ptr(a):
        return a.ctypes.data_as(C.c_void_p)
"""

GRAVITY = """
    def call(leaf):
        rng = np.random.default_rng(5)
        n = 5000
        body = np.concatenate([rng.normal(size=(n, 3)), rng.uniform(0.5, 1.5, (n, 1))], 1).astype(np.float32)
        out = np.full((n, 4), np.nan, np.float32)
        a, b = ok(rt.cudaMalloc(body.nbytes)), ok(rt.cudaMalloc(out.nbytes))
        ok(rt.cudaMemcpy(a, body.ctypes.data, body.nbytes, rt.cudaMemcpyKind.cudaMemcpyHostToDevice))
        st = L.sph_gravity_tree_noalloc(C.c_void_p(a), n, 1.0, 0.05, 0.5, leaf, 1, C.c_void_p(b), None)
        assert st == _lib.SPH_OK, st
        ok(rt.cudaDeviceSynchronize())
        ok(rt.cudaMemcpy(out.ctypes.data, b, out.nbytes, rt.cudaMemcpyKind.cudaMemcpyDeviceToHost))
        ok(rt.cudaFree(a))
        ok(rt.cudaFree(b))
        return out

    for leaf in (8, 32):
        want = call(leaf)
        assert np.isfinite(want).all()
        for _ in range(2):
            ok(rt.cudaDeviceReset())
            assert np.array_equal(call(leaf), want)
"""

MLP = """
    def call():
        rng = np.random.default_rng(6)
        n = 700
        p = rng.normal(scale=0.1, size=_lib.MLP_PARAMS).astype(np.float32)
        p[-1], p[-10:-2] = 1.0, 1.0  # scales of the target and of the inputs
        x, t = rng.normal(size=(n, 8)).astype(np.float32), rng.normal(size=n).astype(np.float32)
        y, g, loss = np.empty(n, np.float32), np.empty(_lib.MLP_TRAINABLE, np.float32), np.empty(2, np.float32)
        assert L.sph_mlp_forward(ptr(p), ptr(x), n, ptr(y)) == _lib.SPH_OK
        assert L.sph_mlp_grad(ptr(p), ptr(x), ptr(t), n, ptr(g), ptr(loss)) == _lib.SPH_OK
        cfg = _lib.MlpTrainCfg(epochs=2, batch=256, lr=1e-3, seed=3)
        assert L.sph_mlp_train(ptr(p), ptr(x), ptr(t), n, C.byref(cfg), ptr(loss)) == _lib.SPH_OK
        assert np.isfinite(y).all() and np.isfinite(g).all() and np.isfinite(p).all()
        return y, g, p

    want = call()
    for _ in range(2):
        ok(rt.cudaDeviceReset())
        for a, b in zip(call(), want):
            assert np.array_equal(a, b)
"""


def _run(case):
    r = subprocess.run([sys.executable, "-c", textwrap.dedent(PROLOGUE) + textwrap.dedent(case)], capture_output=True,
                       text=True, timeout=240)
    assert r.returncode == 0, r.stderr[-2000:]


def test_allocation_free_gravity_after_a_reset():
    _run(GRAVITY)


def test_mlp_calls_after_a_reset():
    _run(MLP)
