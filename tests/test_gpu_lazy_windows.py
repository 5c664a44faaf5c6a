"""The windows read after generate_global_template are those of the parameters
the call was given, whatever layout they came in and whatever the caller does
with the array afterwards."""

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

T = 31557600.0


@pytest.mark.parametrize("layout", ["rows", "columns"])
@pytest.mark.parametrize("fill_mode", ["atomic", "deterministic"])
def test_input_changed_after_the_call(layout, fill_mode):
    from gbgpu_gb300 import GBGPU
    B, N, rng = 5, 64, np.random.default_rng(3)
    p = np.array([np.full(B, 1e-22), 2e-3 + rng.uniform(0, 100, B) / T, np.full(B, 1e-17), np.zeros(B),
                  rng.uniform(0, 6, B), np.arccos(rng.uniform(-1, 1, B)), rng.uniform(0, 3, B),
                  rng.uniform(0, 6, B), np.arcsin(rng.uniform(-1, 1, B))])
    gb, kw = GBGPU(), dict(N=N, T=T, dt=10.0)
    gb.run_wave(*p, **kw)
    want = gb.XYZf.clone(), gb.start_inds.clone()
    # (B, 9): its own rows, or the transposed view of a (9, B) array
    x = torch.as_tensor(p.T.copy(), device="cuda") if layout == "rows" else \
        torch.as_tensor(p, device="cuda").T
    out = torch.zeros((1, 2, 2048), dtype=torch.complex128, device="cuda")
    gb.generate_global_template(x, torch.zeros(B, dtype=torch.int32, device="cuda"), out,
                                start_freq_ind=int(2e-3 * T) - N, fill_mode=fill_mode, **kw)
    x[:, 0] *= 3.0
    x[:, 1] += 50 / T
    assert torch.equal(gb.XYZf, want[0]) and torch.equal(gb.start_inds, want[1])
