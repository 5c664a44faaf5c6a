"""A NaN parameter: NaN through the set-up's FP64 -> FP32 conversion (which
otherwise is the cast, with zero below FP32's normal range), NaN likelihoods and
gradients for its binary in every form, and the other binaries untouched."""

import ctypes

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

T = 31557600.0


def test_conversion():
    from gbgpu_gb300 import _native as nat
    rng = np.random.default_rng(9)
    x = np.concatenate([rng.standard_normal(100_000) * 10.0 ** rng.uniform(-50, 50, 100_000),
                        [np.nan, -np.nan, np.inf, -np.inf, 0.0, -0.0, 1e39, -1e39, 1 + 2.0 ** -24, 1 + 3 * 2.0 ** -24],
                        np.array([0x7ff0000000000001, 0xfff0000000000001], np.uint64).view(np.float64)])
    with np.errstate(over="ignore", invalid="ignore"):
        want = x.astype(np.float32)
    keep = ~((np.abs(x) < 2.0 ** -126 * (1 + 1e-6)))              # zero below the normal range
    xd = torch.as_tensor(x, device="cuda")
    out = torch.empty(x.size, dtype=torch.float32, device="cuda")
    nat.check(nat.lib().gbx_math_selftest(ctypes.c_void_p(xd.data_ptr()), ctypes.c_void_p(out.data_ptr()),
                                          x.size, 4, 0, nat.stream_handle()), "gbx_math_selftest")
    got = out.cpu().numpy()
    np.testing.assert_array_equal(got[keep], want[keep])
    assert (got[np.abs(x) < 2.0 ** -127] == 0).all()


@pytest.mark.parametrize("precision", ["fp64", "pair", "mixed"])
@pytest.mark.parametrize("row", [0, 2, 3, 4, 5, 6, 7, 8])          # (a NaN carrier has no window)
def test_likelihood(precision, row):
    from gbgpu_gb300 import GBGPU
    rng = np.random.default_rng(row)
    B, N = 3, 64
    p = np.array([np.full(B, 1e-22), 2e-3 + rng.uniform(0, 50, B) / T, np.full(B, 1e-17), np.full(B, 1e-27),
                  rng.uniform(0, 6, B), np.arccos(rng.uniform(-1, 1, B)), rng.uniform(0, 3, B),
                  rng.uniform(0, 6, B), np.arcsin(rng.uniform(-1, 1, B))])
    d = [torch.as_tensor(1e-18 * (rng.standard_normal(512) + 1j * rng.standard_normal(512)), device="cuda")
         for _ in range(2)]
    S = torch.full((512,), 1e-40, dtype=torch.float64, device="cuda")
    gb, kw = GBGPU(precision=precision), dict(N=N, T=T, dt=10.0, start_freq_ind=int(2e-3 * T) - N)
    gb.d_d = 0.0
    want = gb.get_ll(p, d, [S, S], **kw)
    p[row, 1] = np.nan
    like = gb.get_ll(p, d, [S, S], **kw)
    assert np.isnan(like[1]) and like[0] == want[0] and like[2] == want[2]
    if precision == "mixed":
        like, grad = gb.get_ll_grad(p, d, [S, S], **kw)
        assert np.isnan(like[1]) and np.isnan(grad[:, 1]).all() and np.isfinite(grad[:, [0, 2]]).all()
