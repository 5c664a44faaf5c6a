"""The launch-shape rule without the autotuner: tiles the kernels accept, never
beyond the shared memory of their blocks, small where a batch is small."""

import pytest

from gbgpu_gb300.gbgpu import default_tile

SMS = 152


@pytest.mark.parametrize("kind", ["ll", "wave", "fill", "swap", "grad"])
@pytest.mark.parametrize("precision", ["fp64", "pair", "mixed"])
@pytest.mark.parametrize("nparams", [9, 14])
@pytest.mark.parametrize("counts", [((32, 1),), ((256, 12),), ((256, 1000),), ((64, 10 ** 6),),
                                    ((2048, 3),), ((64, 5), (512, 400), (2048, 90000))])
def test_rule(kind, precision, nparams, counts):
    t = default_tile(kind, precision, nparams, counts, SMS)
    assert 64 <= t <= 4096 and t & (t - 1) == 0
    if kind == "grad" and nparams == 14:
        assert t == 512
        return
    per = 40 if kind == "grad" else \
        60 if nparams == 14 else (3 if kind == "wave" else 2) * (16 if precision == "pair" else 8)
    if precision == "fp64":
        assert t <= 512
    else:
        assert t <= 512 or t * per <= 113 * 1024
    if sum(c for _, c in counts) < 100:
        assert t == 256


def test_rule_grows_with_the_batch():
    sizes = [default_tile("ll", "pair", 9, ((256, b),), SMS) for b in (12, 600, 1000, 50000)]
    assert sizes == sorted(sizes) and sizes[0] == 256 and sizes[-1] == 2048
