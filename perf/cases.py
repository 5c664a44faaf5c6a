"""Performance cases of the FastGB path.

Each case is one call that a user of the package makes, through the class
API (``GBGPU`` / ``GBGPUThirdBody``) or the backend's method table, with the
inputs that such a program has in hand.  ``listed()`` is the fixed list,
``draw(rng)`` another case of the same ranges, ``prepare`` the inputs and the
object, ``run`` one call, ``work`` the bytes and operations the call cannot
do without, and ``exact`` the same outputs from the published formulas in
FP64 torch (no code of this package).

Parameter distributions are the benchmark's: amplitudes log-uniform on
[1e-23, 1e-21], frequencies by band with the N that goes with them, fdot
log-uniform on [1e-18, 1e-15], isotropic angles; the data are Gaussian noise
from the analytic A/E PSD plus a Galactic foreground that is louder than the
noise below 6 mHz.
"""

import math

import numpy as np
import torch

from gbgpu_gb300 import GBGPU, GBGPUThirdBody
from gbgpu_gb300.utility import flops_per_binary

YEAR = 31557600.0                 # observation times are multiples of this
YRSID = 31558149.763545603        # years of the third-body parameters
C = 299792458.0
ARM = 2.5e9
AU = 149597870700.0

# carrier bands (Hz) and the window length that resolves a source there
BANDS = [(1e-4, 5e-4, 64), (5e-4, 1e-3, 128), (1e-3, 3e-3, 256), (3e-3, 6e-3, 512),
         (6e-3, 1.2e-2, 1024), (1.2e-2, 2.5e-2, 2048)]
# single-N batches: the band of f0 for each N
BAND_OF_N = {32: (1e-4, 5e-4), 64: (1e-4, 1e-3), 128: (1e-3, 5e-3), 256: (1e-3, 5e-3),
             512: (2e-3, 8e-3), 1024: (5e-3, 1.2e-2), 2048: (8e-3, 2.5e-2),
             4096: (1e-2, 3e-2)}
SWAP_BAND = 32_768                # bins of a sampler's band


def _case(name, kind, B, N, precision, **kw):
    c = {"name": name, "kind": kind, "B": B, "N": N, "precision": precision, "tdi2": False,
         "years": 4, "dt": 5.0, "rows": 1, "third": False, "host": False, "groups": 1}
    c.update(kw)
    return c


def listed():
    return [
        # a global-fit likelihood over a whole catalogue: every source its own
        # N, the form that holds 1e-6 accuracy in crowded data, parameters on
        # the device, the full 4-yr grid
        _case("catalogue_ll_pair", "ll", 200_000, 0, "pair"),
        # the same catalogue call in the class's default precision, as a
        # check of a smaller batch would make it
        _case("catalogue_ll_fp64", "ll", 10_001, 0, "fp64"),
        # population studies at one N with second-generation TDI and one data
        # row per segment, in the single-precision form
        _case("segments_ll_mixed", "ll", 50_000, 256, "mixed", tdi2=True, rows=8),
        # the plain workload of the reference's tutorial: 1,000 binaries,
        # defaults throughout
        _case("tutorial_ll_fp64", "ll", 1_000, 128, "fp64", dt=10.0),
        # one step of a small sampler: a dozen walkers with their parameters
        # in host arrays, where latency counts
        _case("walkers_ll_pair", "ll", 12, 256, "pair", dt=10.0, years=2, host=True),
        # windows for a waveform library: X/Y/Z and A/E/T in the default form
        _case("library_wave_fp64", "wave", 2_003, 512, "fp64"),
        # one source for an injection or a plot
        _case("single_wave_fp64", "wave", 1, 1024, "fp64", dt=15.0),
        # a galaxy summed into a few templates (one per realisation)
        _case("galaxy_fill_pair", "fill", 60_000, 512, "pair", groups=4),
        # templates from stored windows, the reference's two-call path
        _case("stored_fill_fp64", "fill_stored", 50_000, 256, "fp64", groups=8),
        # the native likelihood entry on stored point-major templates
        _case("stored_ll_fp64", "ll_stored", 50_000, 256, "fp64"),
        # likelihood gradients for a Hamiltonian sampler
        _case("hmc_grad_mixed", "grad", 8_191, 512, "mixed"),
        # third-body search: swap proposals of an ensemble, 14 parameters,
        # the class's default precision
        _case("third_body_swap_fp64", "swap", 1_024, 512, "fp64", third=True, rows=1_024),
    ]


# most samples (sum of N) of a drawn case, by kind and precision: none costs
# more than the largest listed case
_SAMPLES = {("ll", "pair"): 2 ** 24, ("ll", "mixed"): 2 ** 24, ("ll", "fp64"): 2 ** 21,
            ("wave", "pair"): 2 ** 21, ("wave", "fp64"): 2 ** 20, ("fill", "pair"): 2 ** 24,
            ("fill", "mixed"): 2 ** 24, ("fill", "fp64"): 2 ** 21, ("fill_stored", "fp64"): 2 ** 23,
            ("ll_stored", "fp64"): 2 ** 23, ("grad", "mixed"): 2 ** 22, ("swap", "mixed"): 2 ** 20,
            ("swap", "pair"): 2 ** 20, ("swap", "fp64"): 2 ** 18}


def draw(rng):
    kind, precision = rng.choice(sorted(_SAMPLES))
    years = rng.choice([1, 2, 4])
    dt = rng.choice([5.0, 10.0, 15.0])
    third = kind in ("ll", "swap", "grad") and precision != "pair" and rng.random() < 0.3
    uneven = kind == "ll" and not third and rng.random() < 0.4
    top = 9 if third and precision == "fp64" else 10 if third else \
        11 if precision == "fp64" or kind in ("swap", "grad") else 12
    N = 0 if uneven else 2 ** rng.randint(5 if kind in ("ll", "fill") else 6, top)
    most = _SAMPLES[(kind, precision)] // (512 if uneven else N) // (8 if third else 1)
    B = int(round(math.exp(rng.uniform(0.0, math.log(max(2, most))))))
    rows = 1
    if kind == "swap" or (kind in ("ll", "grad") and rng.random() < 0.3):
        rows = rng.choice([1, 3, 16])
    return {"kind": kind, "B": B, "N": N, "precision": precision, "years": years, "dt": dt,
            "tdi2": rng.random() < 0.4, "rows": rows, "third": third, "host": rng.random() < 0.3,
            "groups": rng.choice([1, 2, 7]) if kind.startswith("fill") else 1}


# ------------------------------------------------------------------ inputs
def _T(case):
    return int(case["years"] * YEAR / case["dt"]) * case["dt"]


def _params(case, rng):
    """(9 or 14, B) parameters and the per-binary N."""
    B, N = case["B"], case["N"]
    if N:
        f0 = rng.uniform(*_f_range(case), B)
        Ns = np.full(B, N, np.int64)
    else:
        f0 = 10 ** rng.uniform(-4, np.log10(2.5e-2), B)
        Ns = np.zeros(B, np.int64)
        for lo, hi, n in BANDS:
            Ns[(f0 >= lo) & (f0 <= hi)] = n
    fdot = 10 ** rng.uniform(-18, -15, B)
    p = [10 ** rng.uniform(-23, -21, B), f0, fdot, 11.0 / 3.0 * fdot ** 2 / f0,
         rng.uniform(0, 2 * np.pi, B), np.arccos(rng.uniform(-1, 1, B)), rng.uniform(0, np.pi, B),
         rng.uniform(0, 2 * np.pi, B), np.arcsin(rng.uniform(-1, 1, B))]
    if case["third"]:
        P2 = 10 ** rng.uniform(0, np.log10(40), B)
        p += [10 ** rng.uniform(0, 4, B), rng.uniform(0, 2 * np.pi, B), rng.uniform(0, 0.9, B),
              P2, rng.uniform(0, 1, B) * P2]
    return np.array(p), Ns


def _psd(k, T):
    """Analytic TDI-1.5 PSD of A and E (arXiv:2108.01167) at grid bins k."""
    f = k / T
    x = 2 * math.pi * f * ARM / C
    oms = (15e-12) ** 2 * (1 + (2e-3 / f) ** 4) * (2 * math.pi * f / C) ** 2
    acc = ((3e-15) ** 2 * (1 + (4e-4 / f) ** 2) * (1 + (f / 8e-3) ** 4)
           / (2 * math.pi * f * C) ** 2)
    cx = torch.cos(x)
    return 8 * torch.sin(x) ** 2 * ((2 + cx) * oms + 2 * (3 + 2 * cx + torch.cos(2 * x)) * acc)


def _f_range(case):
    """Lowest and highest carrier frequency of a single-N case."""
    lo, hi = BAND_OF_N[case["N"]]
    # a sampler works band by band: its residual rows hold one band
    return lo, (lo + SWAP_BAND / _T(case) if case["kind"] == "swap" else hi)


def _band(case):
    """[first, last) bins of the grid that the case's data hold: everything
    for a catalogue, else the sources' band."""
    T = _T(case)
    if not case["N"]:
        return 1, int(round(T / case["dt"])) // 2 + 1
    lo, hi = _f_range(case)
    return max(1, int(lo * T) - 2 * case["N"]), int(hi * T) + 2 * case["N"] + 1


def _data(case, seed, first, last):
    """rows x bins of A and E noise plus foreground, and the PSD (device)."""
    T = _T(case)
    gen = torch.Generator(device="cuda").manual_seed(seed)
    k = torch.arange(first, last, dtype=torch.float64, device="cuda")
    S = _psd(k, T)
    sig = torch.sqrt(S * (T / 4)) * torch.where(k / T < 6e-3, 10.0, 1.0)
    shape = (case["rows"], last - first) if case["rows"] > 1 else (last - first,)
    d = [torch.complex(torch.randn(shape, generator=gen, dtype=torch.float64, device="cuda"),
                       torch.randn(shape, generator=gen, dtype=torch.float64, device="cuda")) * sig
         for _ in range(2)]
    return d, S


def _inputs(case, seed):
    """Everything drawn from the seed: parameters, N, data, PSD, indices."""
    rng = np.random.default_rng(seed)
    p, Ns = _params(case, rng)
    s = {"p": p, "Ns": Ns, "T": _T(case)}
    s["first"], s["last"] = first, last = _band(case)
    if case["kind"] == "swap":
        new = p.copy()
        new[0] *= 1 + 0.1 * rng.standard_normal(p.shape[1])
        new[1] += rng.choice([1e-9, 1e-8, 1e-7], p.shape[1]) * rng.standard_normal(p.shape[1])
        new[4:9] += 0.1 * rng.standard_normal((5, p.shape[1]))
        s["new"] = new
    if case["kind"] in ("ll", "ll_stored", "grad", "swap"):
        s["data"], s["S"] = _data(case, seed, first, last)
    s["di"] = (torch.as_tensor(rng.integers(0, case["rows"], case["B"]), dtype=torch.int32,
                               device="cuda") if case["rows"] > 1 else None)
    s["group"] = torch.as_tensor(rng.integers(0, case["groups"], case["B"]), dtype=torch.int32,
                                 device="cuda")
    if case["kind"] in ("ll_stored", "fill_stored"):
        # stored windows as a library file gives them: smooth lines of the
        # sources' amplitude around their carrier, (B, N) each
        gen = torch.Generator(device="cuda").manual_seed(seed + 1)
        B, N = case["B"], case["N"]
        env = torch.exp(-((torch.arange(N, device="cuda") - N / 2) / (N / 16)) ** 2)
        amp = torch.as_tensor(p[0] * s["T"], device="cuda")[:, None] * (env + 1e-6)
        s["tmpl"] = [torch.polar(amp, 2 * math.pi * torch.rand(
            (B, N), generator=gen, dtype=torch.float64, device="cuda")) for _ in range(2)]
        s["start"] = np.rint(p[1] * s["T"]).astype(np.int64) - N // 2
    return s


def prepare(case, seed):
    s = _inputs(case, seed)
    cls = GBGPUThirdBody if case["third"] else GBGPU
    gb = s["gb"] = cls(precision=case["precision"])
    gb.d_d = 0.0
    s["case"] = case
    s["kw"] = {"T": case["years"] * YEAR, "dt": case["dt"], "tdi2": case["tdi2"]}
    s["N"] = case["N"] or s["Ns"]
    s["prm"] = s["p"] if case["host"] else torch.as_tensor(s["p"], device="cuda").contiguous()
    kind, nb = case["kind"], s["last"] - s["first"]
    if kind == "swap":
        s["prm_new"] = s["new"] if case["host"] else \
            torch.as_tensor(s["new"], device="cuda").contiguous()
    if kind == "fill":
        s["prm"] = s["p"].T.copy() if case["host"] else \
            torch.as_tensor(s["p"].T.copy(), device="cuda")
    if kind in ("fill", "fill_stored"):
        s["out"] = torch.zeros((case["groups"], 2, nb), dtype=torch.complex128, device="cuda")
    if kind == "fill_stored":
        s["start"] = torch.as_tensor(s["start"], device="cuda")
    if kind == "ll_stored":
        B = case["B"]
        s["flat"] = [t.T.contiguous().reshape(-1) for t in s.pop("tmpl")]
        s["start"] = torch.as_tensor(s["start"] - s["first"], dtype=torch.int32, device="cuda")
        s["zeros"] = torch.zeros(B, dtype=torch.int32, device="cuda")
        s["terms"] = [torch.zeros(B, dtype=torch.complex128, device="cuda") for _ in range(2)]
    return s


def run(s):
    case, gb, kw = s["case"], s["gb"], s["kw"]
    kind = case["kind"]
    if kind == "ll":
        like = gb.get_ll(s["prm"], s["data"], [s["S"], s["S"]], N=s["N"], data_index=s["di"],
                         start_freq_ind=s["first"], **kw)
        return {"like": like, "d_h": gb.d_h, "h_h": gb.h_h}
    if kind == "grad":
        like, grad = gb.get_ll_grad(s["prm"], s["data"], [s["S"], s["S"]], N=s["N"],
                                    data_index=s["di"], start_freq_ind=s["first"], **kw)
        return {"like": like, "grad": grad}
    if kind == "swap":
        return gb.swap_likelihood(s["prm"], s["prm_new"], s["data"], [s["S"], s["S"]], N=s["N"],
                                  data_index=s["di"], start_freq_ind=s["first"], **kw)
    if kind == "wave":
        gb.run_wave(*s["prm"], N=s["N"], precision=case["precision"], **kw)
        return {"XYZ": gb.XYZf, "AET": gb.AETf, "start": gb.start_inds}
    if kind == "fill":
        gb.generate_global_template(s["prm"], s["group"], s["out"], N=s["N"],
                                    start_freq_ind=s["first"], **kw)
        return s["out"]
    if kind == "fill_stored":
        gb.fill_global_template(s["group"], s["out"], s["tmpl"][0], s["tmpl"][1], s["start"],
                                start_freq_ind=s["first"])
        return s["out"]
    d_h, h_h = s["terms"]
    gb.backend.get_ll(d_h, h_h, *s["flat"], *s["data"], s["S"], s["S"], 1.0 / s["T"], s["start"],
                      case["N"], case["B"], s["zeros"], s["zeros"], s["last"] - s["first"])
    return {"d_h": d_h, "h_h": h_h}


def work(case):
    B, kind = case["B"], case["kind"]
    if case["N"]:
        total = float(B) * case["N"]
        lo, hi = _f_range(case)
        flops = B * float(flops_per_binary(case["N"], case["tdi2"], case["third"], kind != "wave"))
    else:
        lo, hi = 1e-4, 2.5e-2
        span = math.log(hi / lo)
        total = B * sum(n * math.log(b / a) / span for a, b, n in BANDS)
        flops = B * sum(math.log(b / a) / span *
                        float(flops_per_binary(n, case["tdi2"], False, True)) for a, b, n in BANDS)
    T = _T(case)
    npar = 14 if case["third"] else 9
    bins = (hi - lo) * T                       # bins of the sources' band
    # data rows, one PSD, parameters and outputs, each once
    seen = min(total, bins * case["rows"]) * 32 + min(total, bins) * 8
    if kind == "ll":
        return {"bytes": seen + B * (8 * npar + 40), "flops": flops}
    if kind == "grad":
        return {"bytes": seen + B * 8 * (2 * npar + 1), "flops": 2 * flops}
    if kind == "swap":
        return {"bytes": seen + B * 8 * (2 * npar + 1), "flops": 2 * flops}
    if kind == "wave":
        return {"bytes": 96 * total + B * (8 * npar + 8), "flops": flops}
    out = case["groups"] * bins * 32
    if kind == "fill":
        return {"bytes": out + B * (8 * npar + 4), "flops": flops}
    if kind == "fill_stored":
        return {"bytes": 32 * total + out + 12 * B, "flops": 4 * total}
    return {"bytes": 32 * total + min(total, bins) * 40 + 44 * B, "flops": 24 * total}


# ------------------------------------------------------------------ exact
def _orbit(tm):
    """Spacecraft positions (3, N, 3), Cornish & Rubbo (2003)."""
    ecc = ARM / (2 * math.sqrt(3) * AU)
    a = 2 * math.pi / YRSID * tm
    eR = ecc * AU
    out = []
    for i in range(3):
        b = 2 * math.pi * i / 3
        out.append(torch.stack([
            AU * torch.cos(a) + 0.5 * eR * (torch.cos(2 * a - b) - 3 * math.cos(b)),
            AU * torch.sin(a) + 0.5 * eR * (torch.sin(2 * a - b) - 3 * math.sin(b)),
            -math.sqrt(3) * eR * torch.cos(a - b)], -1))
    return torch.stack(out)


def _v_los(t, A2, varpi, e, n2, T2):
    """Line-of-sight velocity of the inner binary on its Kepler orbit."""
    M = n2 * (t - T2)
    M = M - 2 * math.pi * torch.floor(M / (2 * math.pi))
    u = M + 0.85 * e * torch.where(torch.sin(M) >= 0, 1.0, -1.0)
    with torch.no_grad():
        for _ in range(12):
            f, f1 = u - e * torch.sin(u) - M, 1 - e * torch.cos(u)
            f2, f3 = e * torch.sin(u), e * torch.cos(u)
            d = -f / f1
            d = -f / (f1 + 0.5 * d * f2)
            u = u - f / (f1 + 0.5 * d * f2 + d * d * f3 / 6)
    u = u - (u - e * torch.sin(u) - M) / (1 - e * torch.cos(u))     # carries derivatives
    den = 1 - e * torch.cos(u)
    sphi, cphi = torch.sqrt(1 - e * e) * torch.sin(u) / den, (torch.cos(u) - e) / den
    return A2 * (sphi * torch.cos(varpi) + cphi * torch.sin(varpi) + e * torch.sin(varpi))


def _wave(p, N, T, tdi2):
    """X, Y, Z windows (b, 3, N) of parameters p (9 or 14, b), FP64 torch."""
    amp, f0, fdot, fddot, phi0, iota, psi, lam, beta = p[:9, :, None]
    fstar = C / (2 * math.pi * ARM)
    tm = torch.arange(N, dtype=torch.float64, device=p.device) * (T / N)
    P = _orbit(tm)
    r = {"12": (P[1] - P[0]) / ARM, "23": (P[2] - P[1]) / ARM, "31": (P[0] - P[2]) / ARM}
    theta = math.pi / 2 - beta
    st, ct, sl, cl = torch.sin(theta), torch.cos(theta), torch.sin(lam), torch.cos(lam)
    zero = torch.zeros_like(sl)
    u, v = torch.cat([ct * cl, ct * sl, -st], 1), torch.cat([sl, -cl, zero], 1)
    k = torch.cat([-st * cl, -st * sl, -ct], 1)
    ci = torch.cos(iota)
    Ap, Ac = 1 + ci * ci, -2 * ci
    c2, s2 = torch.cos(2 * psi), torch.sin(2 * psi)
    DP, DC = torch.complex(Ap * c2, -Ac * s2), torch.complex(-Ap * s2, -Ac * c2)
    kP = [k @ (x.T / C) for x in P]
    q = torch.round(f0.detach() * T)
    om = 2 * math.pi * f0
    domega = om - 2 * math.pi * (q / torch.full_like(q, T))
    fonfs, phase = [], []
    for s in range(3):
        xi = tm - kP[s]
        f = f0 + fdot * xi + 0.5 * fddot * xi * xi
        arg = phi0 + domega * tm + math.pi * fdot * xi * xi + math.pi / 3 * fddot * xi ** 3
        if p.shape[0] == 14:
            A2, varpi, e2, P2, T2 = p[9:, :, None]
            vl = _v_los(xi, A2, varpi, e2, 2 * math.pi / (P2 * YRSID), T2 * YRSID)
            g = vl * f
            step = (xi[:, 1:] - xi[:, :-1]) * (g[:, 1:] + g[:, :-1]) * (math.pi / C)
            arg = arg + torch.cat([torch.zeros_like(arg[:, :1]), torch.cumsum(step, 1)], 1)
            f = f * (1 + vl / C)
        fonfs.append(f / fstar)
        phase.append(om * kP[s] - arg)
    kr = {a: k @ x.T for a, x in r.items()}
    pol = {}
    for a, x in r.items():
        ru, rv = u @ x.T, v @ x.T
        pol[a] = (rv * rv - ru * ru) * DP + 2 * ru * rv * DC
    G = {}
    for ij, arm, s, sg in (("12", "12", 0, 1), ("23", "23", 1, 1), ("31", "31", 2, 1),
                           ("21", "12", 1, -1), ("32", "23", 2, -1), ("13", "31", 0, -1)):
        a = 0.5 * fonfs[s] * (1 + sg * kr[arm])
        ph = a + phase[s]
        G[ij] = 0.25 * torch.sin(a) / a * torch.complex(torch.cos(ph), -torch.sin(ph)) * pol[arm]
    omL = (f0 + fdot * tm + 0.5 * fddot * tm * tm) / fstar
    fc = torch.complex(torch.cos(omL), -torch.sin(omL))
    fc2 = 4 * omL * torch.sin(omL) * fc
    X = torch.stack([fc2 * (G["21"] - G["31"] + (G["12"] - G["13"]) * fc),
                     fc2 * (G["32"] - G["12"] + (G["23"] - G["21"]) * fc),
                     fc2 * (G["13"] - G["23"] + (G["31"] - G["32"]) * fc)], 1)
    scale = torch.complex(amp * (0.5 * T / N), zero)
    if tdi2:
        w = 2 * om * ARM / C
        scale = scale * torch.complex(2 * torch.sin(w) ** 2, 2 * torch.sin(w) * torch.cos(w))
    return torch.fft.fftshift(torch.fft.fft(X, dim=-1), dim=-1) * scale[:, None]


def _ae(X):
    return torch.stack([(X[:, 2] - X[:, 0]) / math.sqrt(2),
                        (X[:, 0] - 2 * X[:, 1] + X[:, 2]) / math.sqrt(6)], 1)


def _start(f0, N, T):
    return np.round(((np.rint(f0 * T) - N / 2) / T) / (1 / T)).astype(np.int64)


def _gather(rows, di, start, N):
    """(b, 2, N) windows of [A, E] rows."""
    j = start[:, None] + torch.arange(N, device=start.device)
    flat = [x.reshape(-1, x.shape[-1]) for x in rows]
    return torch.stack([x[di[:, None], j] for x in flat], 1)


def _terms(d, h, S, T):
    w = 4 / T / S[:, None]
    return (d.conj() * h * w).sum((1, 2)), ((h.real ** 2 + h.imag ** 2) * w).sum((1, 2))


def _chunks(Ns, samples):
    """Index arrays of binaries of one N, about `samples` samples each."""
    for n in np.unique(Ns):
        idx = np.nonzero(Ns == n)[0]
        step = max(1, samples // int(n))
        for i in range(0, len(idx), step):
            yield int(n), idx[i:i + step]


def exact(case, seed):
    s = _inputs(case, seed)
    kind, B, T, first = case["kind"], case["B"], s["T"], s["first"]
    dev = "cuda"
    p = torch.as_tensor(s["p"], device=dev)
    di = s["di"].long() if s["di"] is not None else torch.zeros(B, dtype=torch.long, device=dev)
    start = torch.as_tensor(_start(s["p"][1], s["Ns"], T), device=dev)
    S = s["S"][None] if s.get("S") is not None else None
    cz = lambda *n: torch.zeros(n, dtype=torch.complex128, device=dev)
    zi = torch.zeros(B, dtype=torch.long, device=dev)
    if kind == "wave":
        X, A = cz(B, 3, case["N"]), cz(B, 3, case["N"])
        for n, ix in _chunks(s["Ns"], 2 ** 20):
            X[ix] = _wave(p[:, ix], n, T, case["tdi2"])
        A[:, :2] = _ae(X)
        A[:, 2] = X.sum(1) / math.sqrt(3)
        return {"XYZ": X, "AET": A, "start": start}
    if kind in ("ll", "grad"):
        d_h, h_h = cz(B), cz(B)
        grad = torch.zeros((p.shape[0], B), dtype=torch.float64, device=dev)
        for n, ix in _chunks(s["Ns"], 2 ** 19 if kind == "grad" else 2 ** 21):
            q = p[:, ix].clone().requires_grad_(kind == "grad")
            h = _ae(_wave(q, n, T, case["tdi2"]))
            a, b = _terms(_gather(s["data"], di[ix], start[ix] - first, n), h,
                          _gather([S, S], zi[ix], start[ix] - first, n)[:, 0], T)
            if kind == "grad":
                grad[:, ix] = torch.autograd.grad((a.real - 0.5 * b).sum(), q)[0]
            d_h[ix], h_h[ix] = a.detach(), b.detach().to(torch.complex128)
        like = (d_h - 0.5 * h_h).real.cpu().numpy()
        if kind == "grad":
            return {"like": like, "grad": grad.cpu().numpy()}
        return {"like": like, "d_h": d_h, "h_h": h_h}
    if kind == "swap":
        new = torch.as_tensor(s["new"], device=dev)
        sn = torch.as_tensor(_start(s["new"][1], s["Ns"], T), device=dev)
        out = torch.zeros(B, dtype=torch.float64, device=dev)
        for n, ix in _chunks(s["Ns"], 2 ** 18):
            ho, hn = (_ae(_wave(x[:, ix], n, T, case["tdi2"])) for x in (p, new))
            sides = []
            for h, st in ((hn, sn[ix]), (ho, start[ix])):
                Sw = _gather([S, S], zi[ix], st - first, n)[:, 0]
                sides.append(_terms(_gather(s["data"], di[ix], st - first, n), h, Sw, T))
            # the old window on the new one's bins, for the cross term
            src = torch.arange(n, device=dev) + (sn[ix] - start[ix])[:, None]
            ok = (src >= 0) & (src < n)
            old = torch.gather(ho, 2, src.clamp(0, n - 1)[:, None, :].expand(-1, 2, -1)) * ok[:, None]
            Sw = _gather([S, S], zi[ix], sn[ix] - first, n)[:, 0]
            cross = _terms(old, hn, Sw, T)[0].real
            out[ix] = (sides[0][0].real - sides[1][0].real
                       - 0.5 * (sides[0][1] + sides[1][1]) + cross)
        return out.cpu().numpy()
    if kind == "ll_stored":
        d_h, h_h = cz(B), cz(B)
        for n, ix in _chunks(s["Ns"], 2 ** 21):
            a, b = _terms(_gather(s["data"], di[ix], start[ix] - first, n),
                          torch.stack([t[ix] for t in s["tmpl"]], 1),
                          _gather([S, S], zi[ix], start[ix] - first, n)[:, 0], T)
            d_h[ix], h_h[ix] = a, b.to(torch.complex128)
        return {"d_h": d_h, "h_h": h_h}
    nb = s["last"] - first
    out = torch.zeros((case["groups"], 2, nb, 2), dtype=torch.float64, device=dev)
    flat = out.view(-1, 2)
    for n, ix in _chunks(s["Ns"], 2 ** 20):
        h = _ae(_wave(p[:, ix], n, T, case["tdi2"])) if kind == "fill" else \
            torch.stack([t[ix] for t in s["tmpl"]], 1)
        j = start[ix][:, None] - first + torch.arange(n, device=dev)
        ok = (j >= 0) & (j < nb)
        for c in range(2):
            to = (s["group"].long()[ix][:, None] * 2 + c) * nb + j
            flat.index_add_(0, to[ok], torch.view_as_real(h[:, c])[ok])
    return torch.view_as_complex(out)
