"""The FP64 update with its additions in 64-bit integers against the oracle's
IEEE operations, bit for bit, where it can go wrong: states at rest (zero
velocities, exact ties), tiny and large deviations, velocities and densities at
and beyond the windows it is valid in (those sites take the IEEE path), and
relaxation times across their range."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

W = np.array([1 / 3] + [1 / 18] * 6 + [1 / 36] * 12)


def state(dim, kind, rng):
    n = dim ** 3
    f = np.tile(W[:, None], (1, n))
    if kind == "rest":
        return f
    if kind == "ulps":       # a few units in the last place about rest
        return f + rng.integers(-3, 4, f.shape) * np.spacing(f)
    if kind == "powers":     # values on and next to powers of two
        return f * (1 + np.ldexp(rng.choice([-1.0, 1.0], f.shape), -rng.integers(3, 53, f.shape)))
    if kind == "tiny":
        return f * (1 + 1e-13 * rng.standard_normal(f.shape))
    if kind == "flow":       # velocities up to and beyond 1/8
        e = np.array([(0, 0, 0), (1, 0, 0), (0, 1, 0), (-1, 0, 0), (0, -1, 0), (0, 0, -1), (0, 0, 1), (1, 1, 0),
                      (-1, 1, 0), (-1, -1, 0), (1, -1, 0), (1, 0, -1), (0, 1, -1), (-1, 0, -1), (0, -1, -1),
                      (1, 0, 1), (0, 1, 1), (-1, 0, 1), (0, -1, 1)], float)
        eu = e @ rng.uniform(-0.13, 0.13, (3, n))
        return f * (1 + 3 * eu) * rng.uniform(0.8, 1.3, n)
    return f * (1 + 0.1 * rng.standard_normal(f.shape).clip(-3, 3))  # rough: many sites outside


@pytest.mark.parametrize("tau", [0.50005, 0.5267, 1.0, 7.3, 900.0])
@pytest.mark.parametrize("kind", ["rest", "ulps", "powers", "tiny", "flow", "rough"])
def test_fp64_update_bits(capi, oracle, kind, tau):
    dim = 16
    rng = np.random.default_rng(len(kind) * 100 + int(tau * 10))
    o = oracle.OracleLattice(dim, (tau - 0.5) / 3, 0.05, "f64", 8)
    with capi.Lattice(dim, (tau - 0.5) / 3, 0.05, precision="fp64", stride=8) as L:
        f = state(dim, kind, rng).reshape(19, -1, 8).transpose(1, 0, 2).reshape(-1)
        L.load_f(f)
        o.state[:] = L.f()  # the loaded state with its walls' constants
        for _ in range(3):
            o.step(1, every=1)
            L.step(1, every=1)
            assert np.array_equal(L.f().view(np.uint64), o.state.view(np.uint64))
            np.testing.assert_array_equal(L.rho().view(np.uint64), o.rho.view(np.uint64))
            np.testing.assert_array_equal(L.u().view(np.uint64), o.u.view(np.uint64))
