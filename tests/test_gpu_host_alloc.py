"""Pinned results (g5b_host_alloc) from a thread that has not used CUDA: it must not be left with a context of the default device, which
another process may own. (With one GPU that is the engine's device too; what shows is whether the thread keeps a context.)"""
import ctypes
import threading

import numpy as np
import pytest

import common
import synth

pytestmark = pytest.mark.gpu


def test_a_fresh_thread_gets_no_context(gpu_lib):
    c = synth.tiny_spec().cfg.copy()
    c.n_layers, c.vocab = 1, 64
    spec = synth.Spec(c, [0], [1], with_head=True)
    eng, _ = common.build_models(spec, synth.make_model(spec, seed=41, recipe="spread"), 32, oracle=False)
    driver = ctypes.CDLL("libcuda.so.1")
    found = []

    def work():
        ctx = ctypes.c_void_p()
        p = gpu_lib.g5b_host_alloc(1 << 20)
        found.append(bool(p))
        ctypes.memset(p, 7, 1 << 20)
        assert driver.cuCtxGetCurrent(ctypes.byref(ctx)) == 0
        found.append(ctx.value)
        gpu_lib.g5b_host_free(p)
        assert driver.cuCtxGetCurrent(ctypes.byref(ctx)) == 0
        found.append(ctx.value)

    t = threading.Thread(target=work)
    t.start(); t.join()
    assert found == [True, None, None]
    a = eng._pool.array((1 << 17,))                         # and from this thread, which has one
    a[:] = 1.0
    logits, _ = eng.forward(np.array([1, 2], np.int32))
    assert np.isfinite(logits).all()
    eng.close()
