"""FP64 slow part against the oracle over the ranges its branches tell apart:
the link angle a = omL (1 +- k.r)/2 in each series of sin(a)/a and beyond it,
with and without the error terms of a strong chirp, and a chirp so strong that
the two links of an arm differ by more than the FP32 correction covers; the
smallest and largest transforms.

Tolerance: both sides round a carrier phase of at most
phi = 2 pi f0 510 s + pi fdot T^2 + pi/3 fddot T^3 + 30 rad a handful of times,
so their windows agree to 8 eps phi (eps = 1.2e-16).
"""

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

T = 4 * 31557600.0


@pytest.mark.parametrize("N", [32, 64, 512, 4096])
@pytest.mark.parametrize("f0", [1.3e-4, 2.9e-3, 9.1e-3, 2.4e-2, 7.3e-2])
@pytest.mark.parametrize("fdot", [1e-19, 3e-15, -2e-11])
def test_fp64_windows(N, f0, fdot):
    import fastgb_oracle as O
    from gbgpu_gb300 import GBGPU
    rng = np.random.default_rng(int(N + 1e6 * f0))
    B = 5
    p = np.array([np.full(B, 1e-22), f0 * (1 + 1e-3 * rng.uniform(-1, 1, B)), np.full(B, fdot),
                  np.full(B, 11 / 3 * fdot ** 2 / f0), rng.uniform(-9, 9, B),
                  np.arccos(rng.uniform(-1, 1, B)), rng.uniform(0, np.pi, B),
                  rng.uniform(0, 2 * np.pi, B), np.arcsin(rng.uniform(-1, 1, B))])
    gb = GBGPU()
    gb.run_wave(*p, N=N, T=T, dt=5.0)
    w = O.waveform(p, N, T=T, dt=5.0)
    tol = 8 * 1.2e-16 * (2 * np.pi * f0 * 510 + np.pi * abs(fdot) * T * T +
                         np.pi / 3 * p[3].max() * T ** 3 + 30)
    for got, ref in ((gb.XYZf, w["XYZf"]), (gb.AETf[:, :2], w["AETf"][:, :2])):
        got = got.cpu().numpy()
        err = np.sqrt((np.abs(got - ref) ** 2).sum((1, 2)) / (np.abs(ref) ** 2).sum((1, 2)))
        assert err.max() < tol, (err.max(), tol)
    assert np.array_equal(gb.start_inds.cpu().numpy(), w["start_inds"])
