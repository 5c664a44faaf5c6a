"""Pair windows against the FP64 form beyond the usual ranges of the parameters.

Tolerance 1e-9 for carriers of either sign up to 0.3 Hz: the form's sines are
good to 1e-11 absolute, and the link functions sin(a)/a and the TDI factors fall
to 0.05 of their low-frequency size there.
"""

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def binaries(B, seed, f0=4e-3, fdot=1e-17):
    rng = np.random.default_rng(seed)
    return np.array([10 ** rng.uniform(-23, -21, B), f0 * rng.uniform(1, 1.01, B),
                     np.full(B, fdot), np.zeros(B), rng.uniform(0, 6, B),
                     np.arccos(rng.uniform(-1, 1, B)), rng.uniform(0, 3, B), rng.uniform(0, 6, B),
                     np.arcsin(rng.uniform(-1, 1, B))])


def worst(p, N, T):
    from gbgpu_gb300 import GBGPU
    gb = GBGPU()
    gb.run_wave(*p, N=N, T=T, dt=10.0)
    want = gb.XYZf.clone()
    gb.run_wave(*p, N=N, T=T, dt=10.0, precision="pair")
    err = (gb.XYZf - want).abs().square().sum((1, 2)).sqrt() / want.abs().square().sum((1, 2)).sqrt()
    return err.max().item()


@pytest.mark.parametrize("f0", [1e-4, 3e-3, 0.02, 0.1, 0.29])
@pytest.mark.parametrize("sign", [1, -1])
def test_carrier_of_either_sign(f0, sign):
    assert worst(binaries(64, 1, sign * f0), 128, 31557600.0) < 1e-9


@pytest.mark.parametrize("row", [5, 6, 7, 8])           # iota, psi, lam, beta
@pytest.mark.parametrize("size", [1e5, 1e7, 1e14, 1e17, 1e20, -1e16])
def test_large_angles(row, size):
    """Both forms reduce the same FP64 angle, however large."""
    p = binaries(64, 2)
    p[row] += size
    assert worst(p, 128, 31557600.0) < 1e-10


@pytest.mark.parametrize("f0", [1e-3, 6e-3, 0.02])
@pytest.mark.parametrize("fdot", [1e-15, 2e-14, 1e-12, 1e-11, -1e-11, 1e-10])
def test_chirps(f0, fdot):
    """A month of a strong chirp: the phase pi fdot T^2 is 2e3 rad at most, which
    pairs hold to 2^-48 of it, 8e-12, so that 1e-10 holds as for slow sources."""
    assert worst(binaries(64, 3, f0, fdot), 128, 2629800.0) < 1e-10
