"""F dumps and loads beyond two pieces of 2^22 elements overlap their copies with
their kernels: two orders of the same state hold the same values, and a state
that has gone through the host goes on as the one it came from, through pinned
and pageable memory, with a last piece that is nearly empty or nearly full, and
more pieces than the staging buffer holds."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def sites_first(f, dim, stride):
    n = dim ** 3
    s = stride or n
    return f.reshape(n // s, 19, s).transpose(1, 0, 2).reshape(19, n)


@pytest.mark.parametrize("pinned", [False, True])
@pytest.mark.parametrize("prec,dim,stride", [("fp32", 72, 1), ("fp32", 76, 0), ("fp64", 80, 4), ("fp16", 96, 32),
                                             ("bf16", 128, 8), ("fp32", 136, 2), ("fp16", 160, 0)])
def test_pieces(capi, prec, dim, stride, pinned):
    torch = pytest.importorskip("torch")
    wide = prec == "fp64"
    word = np.uint64 if wide else np.uint32
    kw = dict(precision=prec, noise_sigma=1e-4)
    with capi.Lattice(dim, 0.0089, 0.05, stride=stride, seed=5, **kw) as a, \
            capi.Lattice(dim, 0.0089, 0.05, stride=16 if stride == 0 else 0, seed=5, **kw) as other, \
            capi.Lattice(dim, 0.0089, 0.05, stride=stride, seed=6, **kw) as b:
        host = torch.empty(19 * dim ** 3, dtype=torch.float64 if wide else torch.float32, pin_memory=pinned).numpy()
        for steps in (3, 2):  # the second time reuses the slots and the events
            a.step(steps)
            other.step(steps)
            host[:] = -1
            a.f(host)
            want = sites_first(other.f().view(word), dim, 16 if stride == 0 else 0)
            assert np.array_equal(sites_first(host.view(word), dim, stride), want)
            b.load_f(host)
            assert np.array_equal(b.f().view(word), host.view(word))
        if prec in ("fp16", "bf16"):
            a.load_f(host)  # the sum w + deviation in FP32 does not give every deviation back
        a.step(2)
        b.step(2)
        assert np.array_equal(a.f().view(word), b.f().view(word))
