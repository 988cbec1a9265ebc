"""How a batch launches and tunes its stages, without a GPU: tensors stay on the host and
the library records the stage launches."""

import types

import pytest
import torch

from cvdv_b200 import batch
from cvdv_b200.batch import MAX_CTAS, BatchedCircuits


@pytest.fixture(autouse=True)
def launches(monkeypatch):
    log, zeros = [], torch.zeros

    def run_stage(states, prec, tasks, nt, progs, grid, stream):
        log.append((nt, grid))
        return 0

    monkeypatch.setattr(torch, "zeros", lambda *a, device=None, **k: zeros(*a, **k))
    monkeypatch.setattr(torch.Tensor, "cuda", lambda self: self)
    monkeypatch.setattr(torch.cuda, "current_stream", lambda: types.SimpleNamespace(cuda_stream=0))
    monkeypatch.setattr(batch._lib, "load", lambda: types.SimpleNamespace(cvdvBatchRunStage=run_stage))
    monkeypatch.setattr(batch, "struct_sizes", lambda: (batch.PHASE_DTYPE.itemsize, batch.PROGRAM_DTYPE.itemsize,
                                                        batch.TASK_DTYPE.itemsize))
    return log


def circuits(count, m=8, gates=(("d", (1, 0.3 + 0.1j)), ("h", (0, 0)))):
    return [dict(qubits=[1, m], gates=list(gates)) for _ in range(count)]


@pytest.mark.parametrize("grid,limit", [(None, MAX_CTAS), (148, 148), (2000, 2000)])
@pytest.mark.parametrize("count", [3, 200, 1500])
def test_the_grid_limits_the_ctas(launches, grid, limit, count):
    b = BatchedCircuits(circuits(count), grid=grid) if grid else BatchedCircuits(circuits(count))
    b.run()
    assert launches == [(count, min(count, limit))] * 2


def test_tuning_the_chunk_keeps_the_row_shapes(launches, monkeypatch):
    """Every trial of grids and chunks has the row shapes the batch was made with, and the
    shapes that the row trials keep are those of the best time."""
    # 150 tasks a stage as made, 450 with chunks of 1024 pairs: on both sides of a shape's line
    b = BatchedCircuits(circuits(100, m=13, gates=[("h", (0, 0)), ("d", (1, 0.3 + 0.1j))]))
    shapes, trials = {13: b._loge(13)}, []

    def clock(self, reps):
        trials.append((self.grid, self.pair_chunk, self._loge(13)))
        return 1.0 + (self._loge(13) != shapes[13])  # the first trial's settings are the fastest

    monkeypatch.setattr(BatchedCircuits, "_time", clock)
    best = b.autotune(grids=(148, 296), chunks=(1024, 8192))
    assert [t[2] for t in trials[:4]] == [shapes[13]] * 4
    assert best == (148, 1024) and b.row_loge == shapes
