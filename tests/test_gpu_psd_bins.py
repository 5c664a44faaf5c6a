"""Bins of infinite, zero and undefined PSD in the fused FP64 likelihood, as the
reference's d / S gives them: no weight, an infinite sum, NaN.  On one block per
binary and on clusters, the first binary's window with the bin and the others'
without it.

Tolerance of the finite ones: 1e-12 of the terms (FP64 sums of N bins).
"""

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

T = 31557600.0


@pytest.mark.parametrize("N,B", [(64, 5), (256, 5), (256, 200)])
@pytest.mark.parametrize("psds", [1, 2])
def test_psd_bins(N, B, psds):
    from gbgpu_gb300 import GBGPU
    rng = np.random.default_rng(N + B)
    f0 = np.full(B, 2e-3)
    f0[1:] += 2 * N / T                            # windows that miss the first one's
    p = np.array([np.full(B, 1e-22), f0, np.full(B, 1e-17), np.zeros(B), rng.uniform(0, 6, B),
                  np.arccos(rng.uniform(-1, 1, B)), rng.uniform(0, 3, B), rng.uniform(0, 6, B),
                  np.arcsin(rng.uniform(-1, 1, B))])
    first, L = int(2e-3 * T) - N, 4 * N
    d = [1e-18 * (rng.standard_normal(L) + 1j * rng.standard_normal(L)) for _ in range(2)]
    gb, kw = GBGPU(), dict(N=N, T=T, dt=10.0)
    gb.d_d = 0.0
    gb.run_wave(*p, **kw)
    h, at = gb.AETf[0, :2].cpu().numpy(), int(gb.start_inds[0]) - first
    bin_ = at + N // 2 + 3
    for value in (np.inf, 0.0, np.nan):
        S = np.full(L, 1e-40)
        S[bin_] = value
        S = torch.as_tensor(S, device="cuda")
        like = gb.get_ll(p, [torch.as_tensor(x, device="cuda") for x in d], [S, S if psds == 1 else S.clone()],
                         start_freq_ind=first, **kw)
        dh, hh = gb.d_h.cpu().numpy(), gb.h_h.cpu().numpy().real
        assert np.isfinite(dh[1:]).all() and np.isfinite(hh[1:]).all() and np.isfinite(like[1:]).all()
        if np.isinf(value):
            k = np.arange(N) != bin_ - at
            w = [x[at:at + N][k] for x in d]
            want = 4 / T / 1e-40 * sum((x.conj() * y[k]).sum() for x, y in zip(w, h))
            size = 4 / T / 1e-40 * sum(np.abs(x * y[k]).sum() for x, y in zip(w, h))
            norm = 4 / T / 1e-40 * sum((np.abs(y[k]) ** 2).sum() for y in h)
            assert abs(dh[0] - want) < 1e-12 * size and abs(hh[0] - norm) < 1e-12 * norm
        elif value == 0.0:
            assert hh[0] == np.inf
            # (two PSDs weight the channels apart: infinities of both signs may meet)
            assert psds == 2 or (np.isinf(dh[0].real) and np.isinf(dh[0].imag))
        else:
            assert np.isnan(dh[0].real) and np.isnan(hh[0]) and np.isnan(like[0])
