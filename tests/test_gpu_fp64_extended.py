"""FP64 windows against extended precision (numpy.longdouble), over the bands that
they are used in.

Bound: the error of the published formulas evaluated in plain FP64, six sines
and cosines a sample and every operation rounded (numpy, the slow part alone).
Both start from the same FP64 angular frequency and its difference from the
carrier bin's, so that what the inputs themselves lose does not enter.
"""

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

LD = np.longdouble
PI = LD("3.14159265358979323846264338327950288")
B, N, T = 120, 128, 4 * 31557600.0
LINKS = (("12", "12", 0, 1), ("23", "23", 1, 1), ("31", "31", 2, 1),
         ("21", "12", 1, -1), ("32", "23", 2, -1), ("13", "31", 0, -1))


def slow_part(p, F):
    """X, Y, Z (B, 3, N) before the transform, in type F (gbgpu.py:399-540, 348-375)."""
    import fastgb_oracle as O
    orbits, pi, dot = O.OracleOrbits(), F(PI), lambda a, b: sum(a[:, c, None] * b[:, c] for c in range(3))
    om = 2.0 * np.pi * p[1]
    dom = F(om - 2.0 * np.pi * (np.rint(p[1] * T) / T))[:, None]
    om = F(om)[:, None]
    f0, fdot, fddot, phi0, iota, psi, lam, beta = (x.astype(F)[:, None] for x in p[1:])
    L, c = F(orbits.armlength), F(O.C_SI)
    fstar, th = c / (L * 2 * pi), pi / 2 - beta
    st, ct, sl, cl = np.sin(th), np.cos(th), np.sin(lam), np.cos(lam)
    u, v, k = (np.concatenate(x, 1) for x in ((ct * cl, ct * sl, -st), (sl, -cl, 0 * sl), (-st * cl, -st * sl, -ct)))
    ci, c2, s2 = np.cos(iota), np.cos(2 * psi), np.sin(2 * psi)
    DP, DC = (1 + ci * ci) * c2 + 2j * ci * s2, -(1 + ci * ci) * s2 + 2j * ci * c2
    t = np.linspace(0, T, num=N, endpoint=False)
    P = [orbits.get_pos(t, np.full(N, s)).astype(F) for s in (1, 2, 3)]
    r = {"12": (P[1] - P[0]) / L, "23": (P[2] - P[1]) / L, "31": (P[0] - P[2]) / L}
    t = t.astype(F)
    f_fstar, phase = [], []
    for s in range(3):
        kP = dot(k, P[s] / c)
        xi = t - kP
        f_fstar.append((f0 + fdot * xi + fddot * xi * xi / 2) / fstar)
        phase.append(om * kP - (phi0 + dom * t + pi * fdot * xi * xi + pi / 3 * fddot * xi ** 3))
    G = {}
    for ij, arm, s, sign in LINKS:
        ru, rv = dot(u, r[arm]), dot(v, r[arm])
        x = F(0.5) * f_fstar[s] * (1 + sign * dot(k, r[arm]))
        ph = x + phase[s]
        G[ij] = F(0.25) * np.sin(x) / x * (np.cos(ph) - 1j * np.sin(ph)) * ((rv * rv - ru * ru) * DP + 2 * ru * rv * DC)
    w = (f0 + fdot * t + fddot * t * t / 2) / fstar
    fc = np.cos(w) - 1j * np.sin(w)
    X = [G["21"] - G["31"] + (G["12"] - G["13"]) * fc, G["32"] - G["12"] + (G["23"] - G["21"]) * fc,
         G["13"] - G["23"] + (G["31"] - G["32"]) * fc]
    return np.stack([4 * w * np.sin(w) * fc * x for x in X], 1)


@pytest.mark.parametrize("band", [(1e-4, 5e-4), (1e-3, 5e-3), (2e-3, 8e-3), (1.2e-2, 2.5e-2)])
def test_no_further_off_than_plain_fp64(band):
    from gbgpu_gb300 import GBGPU
    rng = np.random.default_rng(int(1e5 * band[0]))
    f0, fdot = rng.uniform(*band, B), 10 ** rng.uniform(-18, -15, B)
    p = np.array([np.ones(B), f0, fdot, 11 / 3 * fdot ** 2 / f0, rng.uniform(0, 2 * np.pi, B),
                  np.arccos(rng.uniform(-1, 1, B)), rng.uniform(0, np.pi, B), rng.uniform(0, 2 * np.pi, B),
                  np.arcsin(rng.uniform(-1, 1, B))])
    gb = GBGPU()
    gb.run_wave(*p, N=N, T=T, dt=10.0)
    n = np.arange(N)
    turn = -2 * PI * ((n[:, None] * n) % N).astype(LD) / N
    dft = np.cos(turn) + 1j * np.sin(turn)
    exact = slow_part(p, LD)
    plain = slow_part(p, np.float64)
    window = np.fft.fftshift(exact @ dft, axes=-1) * LD(0.5 * T / N)
    norm = lambda x: float(np.sqrt((np.abs(x) ** 2).sum()))
    here = norm(gb.XYZf.cpu().numpy() - window) / norm(window)
    there = norm(plain - exact) / norm(exact)
    assert here <= there, (here, there)
