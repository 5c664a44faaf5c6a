"""The end of get_ll on the device (gbx_log_likelihood): logL in the reference's
order of operations from the call's own terms, bit for bit, around the sizes of
the kernel's blocks, and the kernels' flags raised from the same copy."""

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

T = 2 * 31557600.0


def setup(B, precision):
    from gbgpu_gb300 import GBGPU
    rng = np.random.default_rng(B)
    f0 = 2e-3 + rng.uniform(0, 200, B) / T
    p = np.array([10 ** rng.uniform(-23, -21, B), f0, np.full(B, 1e-17), np.zeros(B),
                  rng.uniform(0, 6, B), np.arccos(rng.uniform(-1, 1, B)), rng.uniform(0, 3, B),
                  rng.uniform(0, 6, B), np.arcsin(rng.uniform(-1, 1, B))])
    lo, L = int(2e-3 * T) - 128, 600
    data = [torch.as_tensor(1e-17 * (rng.standard_normal(L) + 1j * rng.standard_normal(L)),
                            device="cuda") for _ in range(2)]
    S = torch.full((L,), 1e-41, dtype=torch.float64, device="cuda")
    return GBGPU(precision=precision), p, data, [S, S], dict(N=64, T=T, dt=10.0, start_freq_ind=lo)


@pytest.mark.parametrize("B", [1, 255, 256, 257])
@pytest.mark.parametrize("precision", ["fp64", "pair", "mixed"])
def test_value(B, precision):
    gb, p, data, psd, kw = setup(B, precision)
    gb.d_d = 123.456789
    like = gb.get_ll(p, data, psd, **kw)
    dh, hh = gb.d_h.cpu().numpy().real, gb.h_h.cpu().numpy().real
    assert like.shape == (B,)
    np.testing.assert_array_equal(like, -0.5 * (gb.d_d + hh - 2 * dh))
    gb.d_d = np.full(B, 123.456789)                     # one d_d per binary
    np.testing.assert_array_equal(gb.get_ll(p, data, psd, **kw), like)


def test_flags():
    gb, p, data, psd, kw = setup(5, "pair")
    gb.d_d = 0.0
    rows = [torch.stack([d, d]) for d in data]
    prow = [torch.stack([s, s]) for s in psd]
    with pytest.raises(ValueError, match="out of range"):
        gb.get_ll(p, rows, prow, data_index=np.array([0, 1, 2, 0, 0], np.int32), **kw)
    gb.get_ll(p, rows, prow, data_index=np.array([0, 1, 1, 0, 0], np.int32), **kw)   # cleared
    p[1, 0] -= 300 / T               # first bin at most 2e-3 T - 132, before lo
    with pytest.warns(UserWarning, match="past the data"):
        gb.get_ll(p, data, psd, **kw)
