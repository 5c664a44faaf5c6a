"""Pair slow part against the oracle where its branches change: the joint
sin(a)/a series with its fourth term in FP32 (q < 0.4), as a pair (to
|a| = 1.6) and the separate series and sincos beyond; sin(omL/2) from the series
(omL < 0.32) and from the table; weak and strong chirps, whose delays enter in
FP32; A and E (likelihood) and X, Y, Z (windows); smallest and largest sizes.

Tolerance: 1e-10 normwise, the form's stated bound, plus 8 roundings of 2^-46 of
the carrier phase phi = 2 pi f0 510 s + pi |fdot| T^2 + pi/3 |fddot| T^3 + 30;
above 61 mHz (|a| > 1.6) the separate series' FP32 tail, 3e-10 at |a| = 1.6,
times up to 10 near the nulls of sin(omL).
"""

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

T = 4 * 31557600.0


@pytest.mark.parametrize("N", [32, 128, 1024, 4096])
@pytest.mark.parametrize("f0", [3e-4, 7.4e-3, 1.1e-2, 2.4e-2, 7.3e-2])
@pytest.mark.parametrize("fdot", [1e-18, -3e-15, 1e-13])
def test_pair_windows_and_terms(N, f0, fdot):
    import fastgb_oracle as O
    from gbgpu_gb300 import GBGPU
    rng = np.random.default_rng(int(N + 1e6 * f0))
    B = 5
    p = np.array([np.full(B, 1e-22), f0 * (1 + 1e-5 * rng.uniform(-1, 1, B)), np.full(B, fdot),
                  np.full(B, 11 / 3 * fdot ** 2 / f0), rng.uniform(0, 6, B),
                  np.arccos(rng.uniform(-1, 1, B)), rng.uniform(0, np.pi, B),
                  rng.uniform(0, 2 * np.pi, B), np.arcsin(rng.uniform(-1, 1, B))])
    w = O.waveform(p, N, T=T, dt=5.0)
    phi = 2 * np.pi * f0 * 510 + np.pi * abs(fdot) * T * T + np.pi / 3 * p[3].max() * T ** 3 + 30
    tol = (1e-10 if f0 < 0.05 else 3e-9) + 8 * 2.0 ** -46 * phi
    gb = GBGPU()
    gb.d_d = 0.0
    gb.run_wave(*p, N=N, T=T, dt=5.0, precision="pair")
    got = gb.XYZf.cpu().numpy()
    err = np.sqrt((np.abs(got - w["XYZf"]) ** 2).sum((1, 2)) / (np.abs(w["XYZf"]) ** 2).sum((1, 2)))
    assert err.max() < tol, (err.max(), tol)
    # <h|h> of the A and E windows against white noise
    lo = int(w["start_inds"].min())
    L = int(w["start_inds"].max()) + N - lo
    S = np.full(L, 1e-40)
    gb.get_ll(p, [np.zeros(L, complex)] * 2, [S, S], N=N, T=T, dt=5.0, precision="pair",
              start_freq_ind=lo)
    ref = 4 * w["df"] * (np.abs(w["AETf"][:, :2]) ** 2).sum((1, 2)) / 1e-40
    assert np.max(np.abs(gb.h_h.real.cpu().numpy() / ref - 1)) < 2 * tol
