"""Whether a fresh batch of the compacting forward's sizes runs it: timed against the one-launch forward
on that batch, per field, precision and power of two of the size (engine._compaction_pays, CPU, with
faked timings)."""
from __future__ import annotations

import pytest
import torch

from gradsolve_b200 import engine
from gradsolve_b200.fields import field_spec


@pytest.fixture
def fake(monkeypatch):
    """cost[compact] is what a forward takes; ran lists the forwards."""
    cost, ran = {}, []

    def forward(method, spec, y0, p, t1v, saveat_ts, cap, ws, kw, compact=False):
        assert engine._IN_TUNER[0]
        ran.append(compact)
        return ws

    def time_ms(fn, reps):
        for _ in range(reps):
            fn()
        return cost[ran[-1]] * (5.0 if len(set(ran)) < 2 or reps == 1 else 1.0)  # (cold at first)

    monkeypatch.setattr(engine, "_COMPACT", {})
    monkeypatch.setattr(engine, "_forward_one", forward)
    monkeypatch.setattr(engine, "_time_ms", time_ms)
    return cost, ran


def pays(n, precision="float64"):
    y0, p = torch.zeros(n, 2, dtype=torch.float64), torch.zeros(n, 4, dtype=torch.float64)
    return engine._compaction_pays("tsit5", field_spec("lv"), y0, p, 1024, {"precision": precision})


@pytest.mark.parametrize("compact,want", [(0.9, True), (0.995, False), (1.0, False), (1.1, False)])
def test_the_faster_one(fake, compact, want):
    cost, ran = fake
    cost.update({False: 1.0, True: compact})
    assert pays(1 << 10) is want
    assert ran.count(True) == ran.count(False) > 2


def test_once_per_size_and_precision(fake):
    cost, ran = fake
    cost.update({False: 1.0, True: 0.5})
    assert pays(1 << 10) and pays((1 << 11) - 1)
    timed = len(ran)
    assert pays(1 << 10) and len(ran) == timed
    cost[True] = 2.0
    assert not pays(1 << 11) and pays(1 << 10) and not pays(1 << 10, "mixed")


def test_memory_that_does_not_fit_is_one_launch(fake, monkeypatch):
    def none(*a, **kw):
        raise torch.OutOfMemoryError

    with monkeypatch.context() as m:
        m.setattr(engine, "_forward_one", none)
        assert not pays(1 << 10)
    assert engine._COMPACT == {}  # (asked again by the next batch)
