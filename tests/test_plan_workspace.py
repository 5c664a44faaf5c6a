"""A batch description owns the workspace it points to: a larger batch on the same
plan brings a new one, and the first (which a captured graph may still use) stays."""

import gc
import types
import weakref

import pytest

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("grad", [False, True])
def test_arguments_keep_their_workspace(grad):
    from gbgpu_gb300.gbgpu import WavePlan
    owner = types.SimpleNamespace(device=torch.device("cpu"),
                                  orbits=types.SimpleNamespace(armlength=2.5e9),
                                  _orbit_table=lambda n, T: torch.zeros(8))
    plan = WavePlan(owner, 256, 1e7, "fp64")
    small = plan.args(torch.zeros((9, 3), dtype=torch.float64), grad=grad)
    ws = weakref.ref(plan._ws)
    assert small.workspace == ws().data_ptr()
    large = plan.args(torch.zeros((9, 3000), dtype=torch.float64), grad=grad)
    gc.collect()
    assert large.workspace == plan._ws.data_ptr() != small.workspace
    assert ws() is not None and ws().data_ptr() == small.workspace
    assert small.workspace_bytes == ws().numel() * 16
    del small
    gc.collect()
    assert ws() is None
