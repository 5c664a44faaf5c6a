"""The FP64 form's sin(a)/a against extended precision over the arguments of its
links, up to |a| = 1.6 (30 mHz): across the series' ranges and beside their ends.

Bound: 1.4e-16.  The last addition rounds by half a unit in the last place of 1
at most, 1.1e-16 of a result above 0.5; below |a| = 1.1 the rounding of a^2 and of
the term before add at most a^2/6 (1.1e-16 + 0.4e-16).  (A correctly rounded sine and a
division may be off by 2.2e-16.)
"""

import ctypes

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def test_sinc_fp64():
    from gbgpu_gb300 import _native as nat
    rng = np.random.default_rng(4)
    edges = np.sqrt([0.0256, 0.25, 1.21])
    a = np.concatenate([rng.uniform(1e-9, 1.6, 400_000), rng.uniform(1.0, 1.6, 400_000),
                        np.concatenate([e * (1 + np.arange(-50, 50) * 2.0 ** -52) for e in edges])])
    a = np.concatenate([a, -a[::7]])
    x = torch.as_tensor(a, device="cuda")
    out = torch.empty_like(x)
    nat.check(nat.lib().gbx_math_selftest(ctypes.c_void_p(x.data_ptr()), ctypes.c_void_p(out.data_ptr()),
                                          a.size, 3, 0, nat.stream_handle()), "gbx_math_selftest")
    al = a.astype(np.longdouble)
    want = np.sin(al) / al
    err = np.abs((out.cpu().numpy() - want) / want)
    assert err.max() < 1.4e-16, (float(err.max()), a[err.argmax()])
