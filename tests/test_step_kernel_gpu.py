"""The default iteration kernel at the sizes where its shape changes (vector
width, one launch or two) against the in-place variant, which shares neither
its launches nor its data movement: the same bits after plain, macro and
graph-replayed iterations."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", ["fp32", "fp64", "fp16", "bf16"])
@pytest.mark.parametrize("dim,block", [(8, 0), (40, 0), (48, 32), (72, 0), (80, 256), (192, 0), (200, 0)])
def test_step_shapes_agree(capi, prec, dim, block):
    if prec == "fp64" and dim > 80:
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
