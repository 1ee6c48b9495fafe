"""The default iteration kernel at the sizes where its shape changes (vector
width, one launch or two) against the in-place variant, which shares neither
its launches nor its data movement: the same bits after plain, macro and
graph-replayed iterations."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", ["fp32", "fp64", "fp16", "bf16"])
@pytest.mark.parametrize("dim,block", [(8, 0), (40, 0), (48, 32), (104, 0), (112, 256), (192, 0), (200, 0)])
def test_step_shapes_agree(capi, prec, dim, block):
    if prec == "fp64" and dim > 104:
        pytest.skip("one shape for FP64")
    outs = []
    for kernel in ("auto", "aa"):
        with capi.Lattice(dim, 0.005, 0.08, precision=prec, seed=21, noise_sigma=1e-4, kernel=kernel,
                          block_threads=block) as L:
            L.step(3)
            L.step(21, every=21)  # sixteen of them one graph
            L.sync()
            outs.append([a.view(np.uint8) for a in (L.f(), L.rho(), L.u())])
    for a, b in zip(*outs):
        np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("dim", [4, 12, 20])
def test_step_shapes_of_sizes_that_are_no_multiple_of_eight(capi, dim):
    outs = []
    for kernel in ("auto", "narrow", "direct", "aa"):
        with capi.Lattice(dim, 0.005, 0.08, precision="fp32", seed=2, noise_sigma=1e-4, kernel=kernel) as L:
            L.step(5, every=5)
            outs.append([a.view(np.uint8) for a in (L.f(), L.rho(), L.u())])
    for other in outs[1:]:
        for a, b in zip(outs[0], other):
            np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("prec", ["fp32", "fp16", "bf16"])
@pytest.mark.parametrize("dim,iters,every", [(8, 5, 2), (24, 9, 4), (104, 3, 3)])
def test_one_step_adjoint_against_two_steps_per_launch(capi, prec, dim, iters, every):
    """Gradients of the one-launch adjoint step (rows shorter and longer than
    a block, both sweeps) against the two-step kernel's.  Tolerance: FP32
    rounding of 19-term sums over the iterations, 1e-5 of the largest value."""
    rng = np.random.default_rng(dim)
    lid, target = 0.05 + 0.01 * rng.standard_normal(dim * dim), 0.02 * rng.standard_normal(dim * dim)
    res = []
    for steps in (1, 2):
        for tau in (False, True):
            with capi.Lattice(dim, velocity=0.0, precision=prec, lid=lid, tau=0.53, adjoint_steps=steps) as L:
                L.adjoint_set_loss(dim // 2, target)
                L.adjoint_forward(iters, every)
                res.append(L.adjoint_backward(1.0, want_f0=False, want_tau=tau))
    for one, two in zip(res[:2], res[2:]):
        assert np.abs(one[1] - two[1]).max() <= 1e-5 * np.abs(two[1]).max()
        if two[0] is not None:
            assert abs(one[0] - two[0]) <= 1e-5 * abs(two[0])


@pytest.mark.parametrize("kernel,steps", [("auto", 3), ("aa", 3), ("aa", 4)])
@pytest.mark.parametrize("prec,dim", [("fp32", 4), ("fp32", 12), ("fp64", 20), ("fp16", 24), ("bf16", 8)])
def test_dump_and_load_agree_over_strides(capi, prec, dim, kernel, steps):
    """The F dump of one state in every stride that divides dim^3 (elements one
    by one and four at a time) re-indexed to SoA, and loading each into a
    fresh handle gives that state back."""
    want = None
    strides = [0] + [1 << k for k in range(16) if dim ** 3 % (1 << k) == 0]
    for st in strides:
        with capi.Lattice(dim, 0.005, 0.08, precision=prec, seed=6, noise_sigma=1e-3, kernel=kernel,
                          stride=st) as L:
            L.step(steps)
            f = L.f()
            soa = f.reshape(19, -1) if st == 0 else f.reshape(-1, 19, st).transpose(1, 0, 2).reshape(19, -1)
            soa = np.ascontiguousarray(soa)
            want = soa if want is None else want
            np.testing.assert_array_equal(soa.view(np.uint8), want.view(np.uint8))
            L.step(2)
            L.load_f(f)
            # 16-bit storage rounds the dumped floats' deviations once more
            got, tol = L.f(), (0 if prec in ("fp32", "fp64") else 1e-6)
            assert np.array_equal(np.isnan(got), np.isnan(f))
            assert np.nanmax(np.abs(got.astype(np.float64) - f)) <= tol
