"""A few FP64 binaries, each on a cluster of blocks, against the same binaries in
a batch large enough for one block each: both cluster sizes, the smallest and
largest windows, chirps, second-generation TDI, one and two PSDs, rows chosen by
index, a bad index and a window beyond the data; and a captured launch.

Tolerance: both sides round a carrier phase of at most phi = 2 pi f0 510 s +
pi fdot T^2 + 30 rad a handful of times and transform in log2 N stages: windows
agree to eps (8 phi + 4 log2 N), eps = 1.2e-16.
"""

import ctypes

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

T = int(2 * 31557600.0 / 10.0) * 10.0
F0, FDOT, MANY = 4e-3, 2e-14, 160


def binaries():
    rng = np.random.default_rng(7)
    f0 = F0 + rng.uniform(0, 100, MANY) / T
    return np.array([10 ** rng.uniform(-23, -21, MANY), f0, FDOT * rng.uniform(-1, 1, MANY),
                     np.full(MANY, 1e-26), rng.uniform(0, 6, MANY), np.arccos(rng.uniform(-1, 1, MANY)),
                     rng.uniform(0, 3, MANY), rng.uniform(0, 6, MANY), np.arcsin(rng.uniform(-1, 1, MANY))])


def tolerance(N):
    return 1.2e-16 * (8 * (2 * np.pi * F0 * 510 + np.pi * FDOT * T * T + 30) + 4 * np.log2(N))


def few():
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    return [1, sms // 8, sms // 8 + 1, 3 * sms // 8]


@pytest.mark.parametrize("N", [256, 512, 2048, 4096])
@pytest.mark.parametrize("tdi2", [False, True])
def test_windows(N, tdi2):
    from gbgpu_gb300 import GBGPU
    p, gb = binaries(), GBGPU()
    gb.run_wave(*p, N=N, T=T, dt=10.0, tdi2=tdi2)
    ref = gb.XYZf.clone(), gb.AETf.clone(), gb.start_inds.clone()
    for B in few():
        gb.run_wave(*p[:, MANY - B:], N=N, T=T, dt=10.0, tdi2=tdi2)
        for got, want in ((gb.XYZf, ref[0]), (gb.AETf[:, :2], ref[1][:, :2])):
            want = want[MANY - B:]
            err = (got - want).abs().square().sum((1, 2)).sqrt() / want.abs().square().sum((1, 2)).sqrt()
            assert err.max().item() < tolerance(N), (B, err.max().item())
        assert torch.equal(gb.start_inds, ref[2][MANY - B:])


@pytest.mark.parametrize("N", [256, 1024, 4096])
@pytest.mark.parametrize("psds", [1, 2])
def test_likelihood(N, psds):
    from gbgpu_gb300 import GBGPU
    rng = np.random.default_rng(N)
    p, gb, L = binaries(), GBGPU(precision="fp64"), N + 300
    start = int(F0 * T) - N // 2 - 60
    data = [torch.as_tensor(1e-18 * (rng.standard_normal((3, L)) + 1j * rng.standard_normal((3, L))),
                            device="cuda") for _ in range(2)]
    S = [torch.as_tensor(10 ** rng.uniform(-41, -40, (2, L)), device="cuda") for _ in range(psds)]
    S = [S[0], S[-1]]
    di, ni = rng.integers(0, 3, MANY).astype(np.int32), rng.integers(0, 2, MANY).astype(np.int32)
    gb.d_d = 0.0
    kw = dict(N=N, T=T, dt=10.0, start_freq_ind=start)
    gb.get_ll(p, data, S, data_index=di, noise_index=ni, **kw)
    dh, hh = gb.d_h.clone(), gb.h_h.real.clone()
    dd = 4 / T * max(sum((d[i].abs() ** 2 / s[j]).sum().item() for d, s in zip(data, S))
                     for i in range(3) for j in range(2))
    tol = tolerance(N)
    for B in few():
        k = slice(MANY - B, MANY)
        gb.get_ll(p[:, k], data, S, data_index=di[k], noise_index=ni[k], **kw)
        assert torch.all((gb.h_h.real - hh[k]).abs() <= 2 * tol * hh[k])
        assert torch.all((gb.d_h - dh[k]).abs() <= tol * (dd * hh[k]).sqrt())
    bad = di[:5].copy()
    bad[2] = 3
    with pytest.raises(ValueError, match="out of range"):
        gb.get_ll(p[:, :5], data, S, data_index=bad, noise_index=ni[:5], **kw)
    with pytest.warns(UserWarning, match="past the data"):       # windows begin below this row
        gb.get_ll(p[:, :5], data, S, **{**kw, "start_freq_ind": int(F0 * T) + 60})


def test_captured():
    from gbgpu_gb300 import GBGPU
    from gbgpu_gb300 import _native as nat
    N, B, gb = 512, 4, GBGPU()
    p = binaries()[:, :B]
    gb.run_wave(*p, N=N, T=T, dt=10.0)
    prm = torch.as_tensor(p, device="cuda")
    a = gb._plan(N, T, "fp64", False, 9, 0, 0).args(prm)
    out = torch.zeros((2, B, 3, N), dtype=torch.complex128, device="cuda")
    start = torch.zeros(B, dtype=torch.int32, device="cuda")
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        rc = nat.lib().gbx_waveform(ctypes.byref(a), nat.ptr(out[0]), nat.ptr(out[1]), nat.ptr(start),
                                    nat.stream_handle())
    assert rc == 0
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(out[0], gb.XYZf) and torch.equal(out[1], gb.AETf)


@pytest.mark.parametrize("N", [256, 1024, 4096])
def test_fills(N):
    """Templates against sums of the large batch's windows; some windows leave
    the templates at either end."""
    from gbgpu_gb300 import GBGPU
    rng = np.random.default_rng(N)
    p, gb, G, L = binaries(), GBGPU(), 3, N + 20
    start = int(F0 * T) - N // 2 + 30
    gb.run_wave(*p, N=N, T=T, dt=10.0)
    win, first = gb.AETf[:, :2].clone(), gb.start_inds.cpu().numpy() - start
    assert first.min() < 0 and first.max() + N > L
    prm = torch.as_tensor(p, device="cuda")
    group = rng.integers(0, G, MANY).astype(np.int32)
    for B in few():
        want = torch.zeros((G, 2, L), dtype=torch.complex128, device="cuda")
        size = 0.0
        for b in range(MANY - B, MANY):
            lo, hi = max(first[b], 0), min(first[b] + N, L)
            want[group[b], :, lo:hi] += win[b, :, lo - first[b]:hi - first[b]]
            size += win[b].abs().square().sum().sqrt().item()
        got = torch.zeros_like(want)
        gb.add_to_templates(prm[:, MANY - B:].contiguous(), torch.as_tensor(group[MANY - B:], device="cuda"),
                            got, start_freq_ind=start, N=N, T=T, dt=10.0, precision="fp64")
        assert (got - want).abs().square().sum().sqrt().item() < tolerance(N) * size
