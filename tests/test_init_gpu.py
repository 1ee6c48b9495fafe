"""The initial state where sites within three of a wall are written by a kernel
of their own: the smallest lattices, those where rows have no other site, and
ones of several blocks, against the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def lid_of(dim):
    return 0.05 + 0.01 * np.random.default_rng(dim).standard_normal(dim * dim)


@pytest.mark.parametrize("kernel", ["auto", "aa"])
@pytest.mark.parametrize("sigma", [0.0, 1e-4])
@pytest.mark.parametrize("dim", [4, 8, 12, 20, 68])
@pytest.mark.parametrize("prec", ["f32", "f64"])
def test_initial_state_bits(capi, oracle, prec, dim, sigma, kernel):
    lid, u = lid_of(dim), {"f32": np.uint32, "f64": np.uint64}[prec]
    o = oracle.OracleLattice(dim, 0.0089, 0.05, prec, 4, seed=9, noise_sigma=sigma, lid=lid)
    with capi.Lattice(dim, 0.0089, 0.05, precision={"f32": "fp32", "f64": "fp64"}[prec], stride=4, seed=9,
                      noise_sigma=sigma, lid=lid, kernel=kernel) as L:
        f = L.f()
    assert np.array_equal(f.view(u), o.state.view(u))


@pytest.mark.parametrize("sigma", [0.0, 1e-4])
@pytest.mark.parametrize("dim", [8, 16, 72])
@pytest.mark.parametrize("prec,eps", [("fp16", 2.0 ** -11), ("bf16", 2.0 ** -8)])
def test_initial_state_16_bit(capi, prec, eps, dim, sigma):
    """Stored as rounded deviations from the weights: one rounding of the
    deviation, and FP32 roundings of values below 1/2 in the sums on both sides."""
    lid, out = lid_of(dim), []
    for p in ("fp32", prec):
        with capi.Lattice(dim, 0.0089, 0.05, precision=p, stride=0, seed=9, noise_sigma=sigma, lid=lid) as L:
            out.append(L.f().astype(np.float64).reshape(19, -1))
    want, got = out
    assert np.array_equal(np.isnan(want), np.isnan(got))
    w = np.array([1 / 3] + [1 / 18] * 6 + [1 / 36] * 12)[:, None]
    err = np.nan_to_num(np.abs(got - want) - eps * np.abs(want - w))
    assert err.max() <= 4 * 2.0 ** -25
