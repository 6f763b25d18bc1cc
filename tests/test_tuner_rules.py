"""CPU tests of the schedule search: what it times, keeps and is asked for. The device is made up."""

import types

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from jno_b200 import _lib, batch as batch_module, tuner  # noqa: E402


class Event:
    clock = 0.0

    def __init__(self, enable_timing=True):
        self.at = 0.0

    def record(self):
        self.at = Event.clock

    def elapsed_time(self, end):
        return end.at - self.at


class Plan:
    """Batched solves that take made-up times: grid says which form FP64 runs in, mixed maps a schedule to a status."""

    n, nnz, device = 100, 1000, None

    def __init__(self, grid, mixed=None, options=None):
        self.grid, self.mixed, self.options, self.calls = grid, mixed or {}, options or {}, []
        self.batch_graph = False

    def jacobi(self, vals):
        return vals

    def pcg_batched(self, off, vals, b, x, inv, tol, atol, maxiter, tile_rows=2048, bps=2):
        self.calls.append(("fp64", tile_rows, bps))
        self.batch_graph = self.grid
        Event.clock += 10.0 / bps
        return np.zeros(self.n), np.ones(2), np.zeros(2), np.zeros(2), 0

    def pcg_batched_mixed(self, off, vals, b, inv, x, tol, atol, maxiter, tile_rows=2048, bps=2):
        self.calls.append(("mixed", tile_rows, bps))
        status = self.mixed.get((tile_rows, bps), 0)
        Event.clock += 1.0 if status else 10.0 / bps
        if status:
            raise _lib.FemkError(status, "made up")
        self.batch_graph = True
        return np.zeros(self.n), np.ones(2), np.ones(2), np.zeros(2), np.zeros(2), 0


@pytest.fixture
def device(monkeypatch, tmp_path):
    monkeypatch.setattr(torch.cuda, "Event", Event)
    monkeypatch.setattr(torch.cuda, "synchronize", lambda *a: None)
    monkeypatch.setattr(torch.cuda, "get_device_name", lambda *a: "made up")
    monkeypatch.setenv("JNO_B200_TUNE_CACHE", str(tmp_path / "tune.json"))
    monkeypatch.setattr(tuner, "CANDIDATES", [(64, 1), (64, 2), (128, 2)])


def _batch(plan, off=(0, 40, 100)):
    b = batch_module.BatchedPoisson.__new__(batch_module.BatchedPoisson)
    b.plan, b.row_off, b.nprob = plan, np.asarray(off, dtype=np.int64), len(off) - 1
    return b


@pytest.mark.parametrize("status,goes_on", [(_lib.FEMK_BREAKDOWN, True), (_lib.FEMK_NONFINITE, True),
                                            (_lib.FEMK_TIMEOUT, False), (_lib.FEMK_ECUDA, False),
                                            (_lib.FEMK_EBOUNDS, False), (_lib.FEMK_EINVAL, False)])
def test_a_candidate_that_does_not_run_is_no_fast_one(device, status, goes_on):
    """Problems that FP32 steps break down on still give a time; a wait that ran out, a CUDA error or a refused call
    ends at once and would be the fastest of all."""
    b = _batch(Plan(False, {(64, 2): status}))
    if goes_on:
        tuner.tune(b, None, None, None, 1e-8)
        return
    with pytest.raises(_lib.FemkError) as err:
        tuner.batched_schedule(b, None, None, None, 1e-8)
    assert err.value.status == status and tuner.cached_schedule(b) is None


def test_entries_are_of_one_form(device):
    """What decides the form that is timed (the largest problem, the plan's options) is in the key."""
    keys = {tuner.signature(_batch(Plan(True, options=o), off))
            for o in ({}, {"ring64": 14}, {"ring64": 14, "cols16": 0}) for off in ((0, 40, 100), (0, 50, 100))}
    assert len(keys) == 6
    assert _lib.load().femk_version() > 10300  # entries timed on the FP64 batches of that version are not this one's


def test_only_solves_with_a_schedule_search_for_one(device):
    """FP64 batches that run a problem at a time have no schedule: one solve. In the grid form the first solve searches
    and the second uses what it found; mixed solves have a schedule in any case."""
    plan = Plan(False)
    for _ in range(2):
        _batch(plan).solve(np.ones(1), None)
    assert len(plan.calls) == 2
    _batch(plan).solve(np.ones(1), None, precision="mixed")
    assert {c[0] for c in plan.calls[3:]} == {"mixed"} and len(plan.calls) > 6
    plan = Plan(True, options={"ring64": 14})
    _batch(plan).solve(np.ones(1), None)
    searched = len(plan.calls)
    assert searched > 6 and plan.calls[-1] in [("fp64", 64, 2), ("fp64", 128, 2)]
    _batch(plan).solve(np.ones(1), None)
    assert len(plan.calls) == searched + 1 and plan.calls[-1] == plan.calls[-2]
