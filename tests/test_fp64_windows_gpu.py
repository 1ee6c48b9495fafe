"""FP64 sites outside the windows of the integer update: velocities of 1/8 and
more, densities beyond [7/8, 2), populations of 1 and more, equilibria further
than a factor of two from their populations, and the Sailfish summation order.
They are relaxed by IEEE operations: the bits of the kernel that has only
those (DIRECT), and no more time than it takes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

W = np.array([1 / 3] + [1 / 18] * 6 + [1 / 36] * 12)
E = np.array([(0, 0, 0), (1, 0, 0), (0, 1, 0), (-1, 0, 0), (0, -1, 0), (0, 0, -1), (0, 0, 1), (1, 1, 0), (-1, 1, 0),
              (-1, -1, 0), (1, -1, 0), (1, 0, -1), (0, 1, -1), (-1, 0, -1), (0, -1, -1), (1, 0, 1), (0, 1, 1),
              (-1, 0, 1), (0, -1, 1)], float)


def equilibrium(n, rho, u):
    eu = E @ u
    return np.repeat(rho * W * (1 + 3 * eu + 4.5 * eu * eu - 1.5 * (u @ u)), n)


def state(n, kind):
    if kind == "fast":
        return equilibrium(n, 1.0, np.array([0.15, 0.0, 0.0]))
    if kind == "dense":
        return equilibrium(n, 2.5, np.array([0.03, 0.01, 0.0]))
    if kind == "denser":
        return equilibrium(n, 4.0, np.zeros(3))
    f = equilibrium(n, 1.0, np.array([0.02, 0.0, 0.01]))
    if kind == "mixed":  # every third site fast, every fifth dense
        g = f.reshape(19, n)
        g[:, ::3] = equilibrium(n, 1.0, np.array([0.2, -0.1, 0.0])).reshape(19, n)[:, ::3]
        g[:, ::5] *= 2.2
    if kind == "far":
        f *= np.random.default_rng(1).uniform(0.3, 2.5, f.shape)
    return f


@pytest.mark.parametrize("order", ["reference", "sailfish"])
@pytest.mark.parametrize("kind", ["rest", "fast", "dense", "denser", "mixed", "far"])
@pytest.mark.parametrize("dim", [8, 36])
def test_outside_the_windows_bits(capi, kind, order, dim):
    got = []
    for kernel in ("direct", 0):
        with capi.Lattice(dim, 0.02, 0.2, precision="fp64", kernel=kernel, order=order) as L:
            L.load_f(state(dim ** 3, kind))
            L.step(1, every=1)
            a = [L.f(), L.rho(), L.u()]
            L.step(2)
            got.append([v.view(np.uint64) for v in a + [L.f()]])
    for a, b in zip(*got):
        np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("kind,order", [("fast", "reference"), ("dense", "reference"), ("denser", "reference"),
                                        ("far", "reference"), ("rest", "sailfish")])
def test_outside_the_windows_time(capi, kind, order):
    torch = pytest.importorskip("torch")
    dim = 128
    f = state(dim ** 3, kind)
    pair = [capi.Lattice(dim, 0.02, 0.05, precision="fp64", kernel=k, order=order) for k in ("direct", 0)]
    t = [[], []]
    for _ in range(8):
        for k, L in enumerate(pair):
            L.load_f(f)
            s = torch.cuda.ExternalStream(L.stream)
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record(s)
            L.step(2)
            b.record(s)
            b.synchronize()
            t[k].append(a.elapsed_time(b))
    for L in pair:
        L.close()
    ieee, auto = (float(np.median(v[1:])) for v in t)
    assert auto <= 1.03 * ieee, (ieee, auto)
