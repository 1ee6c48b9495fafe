"""The noise's quotient and square root are correctly rounded for every argument
they can have: all 2^23 values of u1, on the GPU against its IEEE operations.
And the samples themselves against the oracle's with a sigma so large that the
populations hold them alone."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))


def test_every_radius(capi, tmp_path):
    from lbmcl_gb300 import build
    so = str(tmp_path / "noise_roundings.so")
    r = subprocess.run([build.nvcc(), *build.NVCC_FLAGS, "-shared", "-o", so, os.path.join(HERE, "noise_roundings.cu")],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    out = (ctypes.c_ulonglong * 3)()
    assert ctypes.CDLL(so).noise_roundings(out) == 0
    assert list(out) == [0, 0, 1 << 23]


@pytest.mark.parametrize("prec", ["f32", "f64"])
def test_samples_alone(capi, oracle, prec):
    """sigma = 2^20: a population's last bits are its sample's."""
    dim, seed, sigma = 128, 23, 2.0 ** 20
    o = oracle.OracleLattice(dim, 0.0089, 0.05, prec, 32, seed=seed, noise_sigma=sigma)
    with capi.Lattice(dim, 0.0089, 0.05, precision={"f32": "fp32", "f64": "fp64"}[prec], stride=32, seed=seed,
                      noise_sigma=sigma) as L:
        f = L.f()
    u = np.uint32 if prec == "f32" else np.uint64
    assert np.array_equal(f.view(u), o.state.view(u))
