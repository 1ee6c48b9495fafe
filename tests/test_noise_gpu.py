"""The seeded noise of the initial state against the oracle's, bit for bit, over
most of the 2^23 values a draw's radius can take (20 million draws)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec,dim,seed", [("f32", 128, 11), ("f64", 64, 2 ** 40 + 7)])
def test_noise_bits(capi, oracle, prec, dim, seed):
    o = oracle.OracleLattice(dim, 0.0089, 0.05, prec, 32, seed=seed, noise_sigma=1e-4)
    with capi.Lattice(dim, 0.0089, 0.05, precision={"f32": "fp32", "f64": "fp64"}[prec], stride=32, seed=seed,
                      noise_sigma=1e-4) as L:
        f = L.f()
    u = np.uint32 if prec == "f32" else np.uint64
    assert np.array_equal(f.view(u), o.state.view(u))
