"""The view of a simulator's state keeps the simulator, and with it the memory, alive."""

import gc
import types
import weakref

import pytest
import torch

from cvdv_b200 import CudaCvdv, cudaCvdv


def test_the_viewed_object_holds_the_simulator(monkeypatch):
    """What torch is handed (and keeps) refers to the simulator; without a GPU."""
    destroyed = []
    sim = object.__new__(CudaCvdv)
    sim._L = types.SimpleNamespace(cvdvGetStateDevicePtr=lambda ctx: 512, cvdvSynchronize=lambda ctx: None,
                                   cvdvDestroy=destroyed.append)
    sim.ctx, sim.check_errors, sim.precision, sim.total_size = 7, False, "complex64", 4
    monkeypatch.setattr(cudaCvdv.torch, "as_tensor", lambda v, device: v)
    view = sim.stateTensor()
    del sim
    gc.collect()
    assert destroyed == []
    del view
    assert destroyed == [7]  # (at once: no cycle holds device memory)


@pytest.mark.gpu
def test_a_state_tensor_outlives_the_name_of_its_simulator():
    sim = CudaCvdv([1, 2], check_errors=True)
    sim.initFromArray(torch.tensor([1.0] + [0.0] * 7, dtype=torch.complex128).numpy())
    t, ref = sim.stateTensor(), weakref.ref(sim)
    del sim
    gc.collect()
    assert ref() is not None
    assert float(t.abs().sum()) == 1.0
    del t
    assert ref() is None
