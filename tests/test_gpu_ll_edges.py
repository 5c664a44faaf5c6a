"""Drop-in likelihood around its warps and loops: windows inside the data (loads
a bin ahead) and sticking out on either side, window lengths around the 16-bin
stride, odd numbers of binaries, one PSD or two; against NumPy.

Tolerance: the entry's stated 1e-12 of the sum of |terms|.
"""

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M", [1, 15, 16, 17, 33, 300])
@pytest.mark.parametrize("B", [1, 2, 9])
@pytest.mark.parametrize("two", [False, True])
@pytest.mark.parametrize("fp64", [False, True])
def test_windows(M, B, two, fp64):
    from gbgpu_gb300.backend import get_backend
    rng = np.random.default_rng(M * B + two)
    L = 2 * M + 5
    start = rng.integers(0, L - M + 1, B)
    if B > 1:
        start[0], start[-1] = -(M // 2) - 1, L - M // 2
    c = lambda *n: rng.standard_normal(n) + 1j * rng.standard_normal(n)
    A, E, dA, dE = c(B, M) * 1e-20, c(B, M) * 1e-20, c(L) * 1e-19, c(L) * 1e-19
    A[0, 0] = 0.0
    S = 1e-40 * rng.uniform(0.5, 2, (2, L))
    SE = S[1] if two else S[0]
    dev = lambda x, t=None: torch.as_tensor(np.ascontiguousarray(x), dtype=t, device="cuda")
    out = [torch.zeros(B, dtype=torch.complex128, device="cuda") for _ in range(2)]
    sA = dev(S[0])
    z = torch.zeros(B, dtype=torch.int32, device="cuda")
    get_backend().get_ll(*out, dev(A.T).reshape(-1), dev(E.T).reshape(-1), dev(dA), dev(dE), sA,
                         dev(SE) if two else sA, 0.25, dev(start, torch.int32), M, B, z, z, L,
                         fp64=fp64)
    for b in range(B):
        i = np.arange(max(0, -start[b]), min(M, L - start[b]))
        j = start[b] + i
        t = np.conj(dA[j]) * A[b, i] / S[0, j] + np.conj(dE[j]) * E[b, i] / SE[j]
        h = np.abs(A[b, i]) ** 2 / S[0, j] + np.abs(E[b, i]) ** 2 / SE[j]
        size = (np.abs(dA[j] * A[b, i]) / S[0, j] + np.abs(dE[j] * E[b, i]) / SE[j]).sum()
        assert abs(out[0][b].item() - t.sum()) <= 1e-12 * size
        assert abs(out[1][b].item() - h.sum()) <= 1e-12 * h.sum()
