"""Fill from row-major windows (bulk copies and reductions) against NumPy sums:
chunks' edges, windows that stick out of the data on either side or miss it,
few and odd numbers of binaries, gaps between rows, an index out of range.

Tolerance: at most 40 windows of |values| <= 2 meet in a bin; sums of 40 terms
in any order agree to 40 * 40 * 2 * 2^-53 < 4e-13.
"""

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M", [7, 8, 255, 256, 257, 700])
@pytest.mark.parametrize("B", [1, 5, 1237])
def test_row_major_fill(M, B):
    from gbgpu_gb300 import GBGPU
    rng = np.random.default_rng(M + B)
    L, G, gap = max(40, M * B // 20), 3, 2 * (M % 3)
    start = rng.integers(-M - 3, L + 3, B)
    start[0] = -M + 1                              # one bin inside
    group = rng.integers(0, G, B).astype(np.int32)
    w = rng.uniform(-1, 1, (2, B, M + gap)) + 1j * rng.uniform(-1, 1, (2, B, M + gap))
    ref = np.zeros((G, 2, L), complex)
    for b in range(B):
        lo, hi = max(0, -start[b]), min(M, L - start[b])
        if hi > lo:
            ref[group[b], :, start[b] + lo:start[b] + hi] += w[:, b, lo:hi]
    t = torch.full((G, 2, L), 7.0, dtype=torch.complex128, device="cuda")
    d = [torch.as_tensor(x, device="cuda")[:, :M] for x in w]
    gb = GBGPU()
    gb.fill_global_template(torch.as_tensor(group, device="cuda"), t, d[0], d[1],
                            torch.as_tensor(start, device="cuda"))
    assert np.abs(t.cpu().numpy() - ref).max() < 4e-13
    if B > 1:
        group[1] = G
        with pytest.raises(ValueError, match="out of range"):
            gb.fill_global_template(torch.as_tensor(group, device="cuda"), t, d[0], d[1],
                                    torch.as_tensor(start, device="cuda"))
