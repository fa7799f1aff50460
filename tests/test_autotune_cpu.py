"""CPU: what the batch autotuner times and what it takes from its cache (the
timings are stand-ins; nothing runs on a GPU)."""

import json

import pytest
import torch

import serinv_gb300.batched as bm


@pytest.fixture
def tuner(tmp_path, monkeypatch):
    monkeypatch.setattr(bm, "CACHE", str(tmp_path / "tune.json"))
    monkeypatch.setattr(torch.cuda, "get_device_name", lambda *a: "GPU")
    timed = []

    def install(cost):
        def time_plan(mats, rhs, scratch, srhs, ops, precisions, ns, panel, reps, split=False):
            timed.append((ns, panel, split))
            return cost(ns, panel, split)
        monkeypatch.setattr(bm, "_time_plan", time_plan)
        return timed
    return install


def _mats(b, dtype=torch.float64):
    z = lambda *s: torch.zeros(s, dtype=dtype)
    return [(z(2, b, b), z(1, b, b), z(2, 0, b), z(0, 0))] * 2


def test_every_panel_candidate_is_timed(tuner):
    timed = tuner(lambda ns, panel, split: {0: 3.0, 18: 2.5, 24: 1.0}[panel] + split)
    assert bm.autotune(_mats(96), None, candidates=(1, 2), panel_candidates=(18, 24)) == (1, 24, False)
    assert {(1, 18, False), (1, 24, False)} <= set(timed)


@pytest.mark.parametrize("b,dtype,searched", [(64, torch.float64, False), (33, torch.complex128, True),
                                              (32, torch.complex64, False), (65, torch.float32, True)])
def test_panel_counts_are_searched_where_there_are_column_blocks(tuner, b, dtype, searched):
    timed = tuner(lambda ns, panel, split: 1.0)
    bm.autotune(_mats(b, dtype), None, candidates=(1,), panel_candidates=(18, 24))
    assert any(p for _, p, _ in timed) == searched


def test_choices_of_an_earlier_schedule_are_not_used(tuner, monkeypatch):
    tuner(lambda ns, panel, split: 1.0 + ns + panel)
    with monkeypatch.context() as m:
        m.setattr(bm, "SCHEDULE", bm.SCHEDULE - 1)
        old = bm._signature(_mats(96), None, 7, ["fp64"] * 2)
    with open(bm.CACHE, "w") as f:
        json.dump({old: [2, 24, True]}, f)
    assert bm.autotune(_mats(96), None, candidates=(1, 2)) == (1, 0, False)
    with open(bm.CACHE) as f:
        assert json.load(f)[old] == [2, 24, True]  # kept, not taken
    assert bm.autotune(_mats(96), None, candidates=(2,)) == (1, 0, False)  # its own choice is
