"""FP64 third-body windows against the oracle for periods of an hour and
eccentricities close to 1, where the three spacecraft see the inner binary at
anomalies on either side of periapsis.

Tolerance, as for the longer periods: 8 eps times the carrier phase, plus the
Doppler phase's share: both sides round the mean anomaly M and the anomaly's
solution by a few eps (|M| + 4), which moves v_LOS by at most A2 / (1 - e)^2 of
that and the phase by 2 pi f T / c times the change.
"""

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

YR = 31558149.763545603


@pytest.mark.parametrize("e2", [0.9, 0.99, 0.999])
@pytest.mark.parametrize("P2", [1e-4, 1e-3])
def test_windows_across_periapsis(e2, P2):
    import fastgb_oracle as O
    from gbgpu_gb300 import GBGPUThirdBody
    rng = np.random.default_rng(int(1e4 * e2 + 1e5 * P2))
    B, N, f0, A2, T = 200, 256, 4.1e-3, 3e3, 2629800.0
    p = np.array([np.full(B, 1e-22), f0 * (1 + 1e-3 * rng.uniform(-1, 1, B)), np.full(B, 2e-16),
                  np.zeros(B), rng.uniform(0, 6, B), np.arccos(rng.uniform(-1, 1, B)),
                  rng.uniform(0, np.pi, B), rng.uniform(0, 2 * np.pi, B),
                  np.arcsin(rng.uniform(-1, 1, B)), np.full(B, A2), rng.uniform(0, 2 * np.pi, B),
                  np.full(B, e2), np.full(B, P2), rng.uniform(0, 1, B) * P2])
    gb = GBGPUThirdBody()
    gb.run_wave(*p, N=N, T=T, dt=5.0)
    w = O.waveform(p[:9], N, T=T, dt=5.0, third=p[9:])
    eps = 1.2e-16
    M = 2 * np.pi / (P2 * YR) * (T + P2 * YR)
    phi = 2 * np.pi * f0 * 510 + np.pi * 2e-16 * T * T + 30
    tol = 8 * eps * phi + 4 * eps * (M + 4) * A2 / (1 - e2) ** 2 * 2 * np.pi * f0 * T / 299792458.0
    got = gb.XYZf.cpu().numpy()
    err = np.sqrt((np.abs(got - w["XYZf"]) ** 2).sum((1, 2)) / (np.abs(w["XYZf"]) ** 2).sum((1, 2)))
    assert err.max() < tol, (err.max(), tol)
