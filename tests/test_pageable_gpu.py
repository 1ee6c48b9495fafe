"""F dumps (and the gradient in their layout) into host memory that is neither
page-locked nor touched before, what Lattice.f() makes, take about as long as
touching that memory and the copy take one after the other, whatever handles
came before."""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def best(f, n=4):
    t = []
    for _ in range(n):
        t0 = time.perf_counter()
        keep = f()
        t.append(time.perf_counter() - t0)
        del keep
    return min(t)


def touched(n, dtype):
    a = np.empty(n, dtype)
    a.view(np.uint8)[::4096] = 0  # every page
    return a


def test_dump_into_untouched_memory(capi):
    for dim, prec in ((64, "fp32"), (100, "fp32"), (200, "fp16"), (136, "fp64"), (200, "bf16"), (256, "fp32")):
        with capi.Lattice(dim, precision=prec, noise_sigma=1e-4, seed=2) as L:
            like = 19 * dim ** 3, L.fdtype
            buf = touched(*like)
            copy, touch, fresh = best(lambda: L.f(buf)), best(lambda: touched(*like)), best(lambda: L.f())
            assert np.array_equal(buf, L.f(), equal_nan=True)
        # factors of two, and half a millisecond
        assert fresh <= 2 * copy + 2 * touch + 5e-4, (dim, prec, copy, touch, fresh)


def test_gradient_into_untouched_memory(capi):
    dim = 200
    with capi.Lattice(64) as small:
        small.f()
    with capi.Lattice(dim, velocity=0.05, precision="fp16", tau=0.53) as L:
        L.adjoint_set_loss(dim // 2, None)
        L.adjoint_forward(2, 2)
        like = 19 * dim ** 3, np.float32
        buf = touched(*like)
        sweep = best(lambda: L.adjoint_backward(1.0, want_f0=False))
        copy, touch = best(lambda: L.f(buf)), best(lambda: touched(*like))
        fresh = best(lambda: L.adjoint_backward(1.0, want_f0=True))
    assert fresh <= 2 * sweep + 4 * copy + 2 * touch + 5e-4, (sweep, copy, touch, fresh)
