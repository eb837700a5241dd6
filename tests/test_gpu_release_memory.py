"""gg_release_memory gives back what the potentials keep between calls (some
400 Y functions of 5,026 points with the six arrays they are built from:
over 100 MB, more than the pool's blocks), and the next call works."""
import ctypes as C

import numpy as np
import pytest

from tests.test_gpu_potential_functions import _lists, _setup

pytestmark = pytest.mark.gpu


def _free_bytes():
    rt = next(C.CDLL(n) for n in ("libcudart.so.13", "libcudart.so") if _loads(n))
    free, total = C.c_size_t(), C.c_size_t()
    assert rt.cudaMemGetInfo(C.byref(free), C.byref(total)) == 0
    return free.value


def _loads(name):
    try:
        C.CDLL(name)
        return True
    except OSError:
        return False


def test_potential_buffers_are_given_back(gpu_ready, oracle_mod):
    from grasp_gb300 import _lib
    lib = _lib.gpu()
    _, ctx, nw = _setup(5000, 0.005)
    nya, nxa, co = _lists(nw, 400, 20, 1)
    small = ctx.xpot(nxa[:1], co[:1])  # modules loaded, the pool in place
    assert lib.gg_release_memory(0) == 0
    before = _free_bytes()
    x = ctx.xpot(nxa, co)
    held = before - _free_bytes()
    assert held > 64 << 20  # the call's buffers are the context's
    assert lib.gg_release_memory(0) == 0
    assert _free_bytes() >= before - (8 << 20)  # (kernels loaded meanwhile take some)
    for a, b in zip(ctx.xpot(nxa, co) + ctx.xpot(nxa[:1], co[:1]), x + small):
        np.testing.assert_array_equal(a, b)
