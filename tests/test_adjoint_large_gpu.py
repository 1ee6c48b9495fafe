"""Gradients beyond 192^3, where a 16-bit forward iteration is two launches forked
over a second stream, its recorded points come from a one-launch kernel with
other vectors, the FP32 adjoint takes two steps per launch, and a captured
segment may hold a programmatic dependent behind a fork and join: the same bits
with and without graphs, recomputed or recorded, and the FP64 adjoint's values
within the roundings of T iterations (three of 2^-24 each, all alike)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

DIM, T, EVERY = 200, 12, 5


def gradient(capi, prec, tau, **kw):
    rng = np.random.default_rng(DIM)
    lid, target = 0.05 + 0.005 * rng.standard_normal(DIM * DIM), 0.02 * rng.standard_normal(DIM * DIM)
    with capi.Lattice(DIM, velocity=0.0, precision=prec, lid=lid, tau=0.53, seed=3, noise_sigma=1e-4, **kw) as L:
        L.adjoint_set_loss(DIM // 2, target)
        J = L.adjoint_forward(T, EVERY)
        g_tau, g_lid, g_f0 = L.adjoint_backward(1.0, want_tau=tau)
        return J, g_tau, g_lid, g_f0, L.raw()


def same(a, b):
    assert a[0] == b[0] and a[1] == b[1]
    for x, y in zip(a[2:4], b[2:4]):
        np.testing.assert_array_equal(x, y)
    shape = (19, DIM, DIM, DIM, -1)  # (the walls' slots hold unspecified values)
    assert np.array_equal(a[4].reshape(shape)[:, 1:-1, 1:-1, 1:-1], b[4].reshape(shape)[:, 1:-1, 1:-1, 1:-1])


@pytest.mark.parametrize("tau", [False, True])
@pytest.mark.parametrize("prec", ["fp32", "fp16", "bf16"])
@pytest.mark.parametrize("how", [dict(), dict(adjoint_steps=1), dict(adjoint_fp64=True)], ids=["two", "one", "wide"])
def test_large_gradient(capi, prec, tau, how):
    base = gradient(capi, prec, tau, graph_iterations=1, adjoint_tail_segments=-1, **how)
    same(base, gradient(capi, prec, tau, adjoint_tail_segments=-1, **how))        # captured segments
    for tail in (0, 1):                                                           # recorded points
        same(base, gradient(capi, prec, tau, adjoint_tail_segments=tail, **how))
    for tail in (-1, 0, 2):                                                       # states, recomputed and recorded
        full = gradient(capi, prec, tau, adjoint_full_states=True, adjoint_tail_segments=tail, **how)
        if tau:
            same(base, full)
        elif tail < 0:
            states = full
        else:
            same(states, full)
    if not how:
        wide = gradient(capi, prec, tau, adjoint_fp64=True)
        for a, b in zip(base[2:4], wide[2:4]):
            a, b = a.astype(np.float64), b.astype(np.float64)
            assert np.linalg.norm(a - b) <= 3 * T * 2.0 ** -24 * np.linalg.norm(b)


@pytest.mark.parametrize("tau", [False, True])
@pytest.mark.parametrize("graphs", [0, 1])
def test_direct_fp32_gradient(capi, tau, graphs):
    """FP32 DIRECT iterations are two forked launches at every size; their points
    come from the one-launch kernel: the gradient of the default variant."""
    dim, got = 40, []
    lid = 0.05 + 0.005 * np.random.default_rng(4).standard_normal(dim * dim)
    for kernel in (0, "direct"):
        for tail in (-1, 0):
            with capi.Lattice(dim, velocity=0.0, precision="fp32", lid=lid, tau=0.53, seed=3, noise_sigma=1e-4,
                              kernel=kernel, graph_iterations=graphs, adjoint_tail_segments=tail) as L:
                L.adjoint_set_loss(dim // 2, None)
                J = L.adjoint_forward(23, 6)
                got.append((J,) + L.adjoint_backward(1.0, want_tau=tau) + (L.f(),))
    for other in got[1:]:
        assert got[0][0] == other[0] and got[0][1] == other[1]
        for a, b in zip(got[0][2:], other[2:]):
            np.testing.assert_array_equal(a, b)
