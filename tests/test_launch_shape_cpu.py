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
