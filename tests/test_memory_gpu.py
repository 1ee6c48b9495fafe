"""Handles share one device memory pool: handles made and destroyed in several
threads at once, on recycled buffers, give the bits of a handle alone, and a
gradient evaluated over and over keeps its value."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def run(capi, dim, prec, seed):
    with capi.Lattice(dim, 0.005, 0.08, precision=prec, seed=seed, noise_sigma=1e-4) as L:
        L.step(9, every=9)
        return [a.view(np.uint8).copy() for a in (L.f(), L.rho(), L.u())] + [L.raw()]


def test_threads_on_recycled_memory(capi):
    jobs = [(24, "fp32", 1), (40, "fp16", 2), (32, "bf16", 3), (16, "fp64", 4)]
    want = [run(capi, *j) for j in jobs]
    bad = []

    def work(k):
        for r in range(6):
            j = (k + r) % len(jobs)
            for a, b in zip(run(capi, *jobs[j]), want[j]):
                if not np.array_equal(a, b):
                    bad.append((k, jobs[j]))

    threads = [threading.Thread(target=work, args=(k,)) for k in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad


@pytest.mark.parametrize("tau", [False, True])
def test_gradients_on_recycled_memory(capi, tau):
    got = []
    for dim in (24, 40, 24, 32, 24):
        lid = 0.05 + 0.01 * np.random.default_rng(dim).standard_normal(dim * dim)
        with capi.Lattice(dim, velocity=0.0, precision="fp32", lid=lid, tau=0.53) as L:
            L.adjoint_set_loss(dim // 2, None)
            J = L.adjoint_forward(12, 5)
            g = L.adjoint_backward(1.0, want_tau=tau)
        if dim == 24:
            got.append((J, g[0], g[1], g[2]))
    for other in got[1:]:
        assert got[0][0] == other[0] and got[0][1] == other[1]
        np.testing.assert_array_equal(got[0][2], other[2])
        np.testing.assert_array_equal(got[0][3], other[3])


@pytest.mark.parametrize("prec,steps", [("fp32", 2), ("fp16", 1), ("bf16", 2), ("fp64", 1)])
@pytest.mark.parametrize("dim,iters,every", [(24, 37, 8), (40, 20, 10), (16, 5, 7)])
def test_recorded_states_are_exact(capi, prec, steps, dim, iters, every):
    """With adjoint_full_states the forward records the states of its last
    segments (all, two, one): the loss, the state it ends in and the gradients
    of sweeps with and without a tau gradient are those of recomputing."""
    rng = np.random.default_rng(dim + iters)
    lid, target = 0.05 + 0.01 * rng.standard_normal(dim * dim), 0.02 * rng.standard_normal(dim * dim)
    res = []
    for tail in (-1, 0, 2, 1):
        for tau in (True, False):
            with capi.Lattice(dim, velocity=0.0, precision=prec, lid=lid, tau=0.53, seed=3, noise_sigma=1e-4,
                              adjoint_steps=steps, adjoint_full_states=True, adjoint_tail_segments=tail) as L:
                L.adjoint_set_loss(dim // 2, target)
                out = []
                for _ in range(2):  # the second run starts from the first one's end
                    J = L.adjoint_forward(iters, every)
                    out.append((J, L.f()) + tuple(L.adjoint_backward(1.0, want_tau=tau)))
            res.append(out)
    for k in (2, 4, 6):
        for tau in (0, 1):
            for a, b in zip(res[tau], res[k + tau]):
                assert a[0] == b[0] and a[2] == b[2]
                np.testing.assert_array_equal(a[1], b[1])
                np.testing.assert_array_equal(a[3], b[3])
                np.testing.assert_array_equal(a[4], b[4])


@pytest.mark.parametrize("first_out", [0, 1])
def test_blocks_beyond_what_the_pool_keeps(capi, first_out):
    """Two handles of 46 GB pass the quarter of the device's memory that the
    pool keeps: a lattice of the second one has its own allocation, gives the
    same state, and goes back when its handle does."""
    torch = pytest.importorskip("torch")
    free, total = torch.cuda.mem_get_info(0)
    if total / 4 > 90e9 or free < 120e9:
        pytest.skip("sized for a 280 GB device")
    pair = [capi.Lattice(512, 0.005, 0.08, precision="fp64", seed=3, noise_sigma=1e-4) for _ in range(2)]
    for L in pair:
        L.step(2, every=2)
    a, b = (L.reduce() for L in pair)
    assert a == b
    np.testing.assert_array_equal(pair[0].rho().view(np.uint64), pair[1].rho().view(np.uint64))
    pair[first_out].close()
    left = pair[1 - first_out]
    left.step(1)
    assert left.reduce() != a
    left.close()
    torch.cuda.synchronize()
    assert free - torch.cuda.mem_get_info(0)[0] <= total / 4 + 2e9
