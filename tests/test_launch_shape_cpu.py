"""Launch shapes of a batch with one N per binary: the rule's with autotuning
off, the tuner's with it on, whichever came first."""

import numpy as np

from gbgpu_gb300 import autotune
from gbgpu_gb300.gbgpu import GBGPU


class Tuner:
    calls = 0

    def tune(self, key, run):
        self.calls += 1
        return 1024, 2


def test_switching_the_autotuner(monkeypatch):
    tuner = Tuner()
    monkeypatch.setattr(autotune, "default_tuner", lambda: tuner)
    gb = object.__new__(GBGPU)                 # host logic only: no device
    gb._shapes, gb._tiles, gb._sms, gb.autotune = {}, {}, 152, False
    N = np.array([64, 512, 512, 2048] * 50)

    def shape():
        return gb._launch_shape("ll", N, N.size, "pair", False, 9, run=None)

    rule = shape()
    assert rule != (1024, 2) and rule[1] == 0 and tuner.calls == 0
    gb.autotune = True
    assert shape() == (1024, 2) and shape() == (1024, 2) and tuner.calls == 1
    gb.autotune = False
    assert shape() == rule and tuner.calls == 1


def test_tile_of_an_array_is_found_once(monkeypatch):
    from gbgpu_gb300 import gbgpu as G
    rng = np.random.default_rng(1)
    N = 2 ** rng.integers(5, 14, 3000)
    n, c = np.unique(N, return_counts=True)
    want = list(zip(n.tolist(), c.tolist()))
    assert G._counts(N) == want
    assert G._counts(np.array([-64, 64, 64, 2 ** 40])) == [(-64, 1), (64, 2), (2 ** 40, 1)]
    assert G._counts(np.zeros(0, np.int64)) == []
    gb = object.__new__(GBGPU)
    gb._tiles, gb._sms, calls = {}, 152, []
    monkeypatch.setattr(G, "_counts", lambda x: calls.append(1) or want)
    for _ in range(3):
        assert gb._tile("fill", "pair", 9, N, N.size, nkey=(1, 2)) == \
            G.default_tile("fill", "pair", 9, want, 152)
    assert len(calls) == 1
