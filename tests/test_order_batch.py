"""Which lane order an even batch's one-thread reverse pass takes, windows or the whole batch: timed once
per field and size (engine._tune_order; CPU, with faked timings); the gradients are the same bits (GPU)."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from gradsolve_b200 import engine
from gradsolve_b200.fields import field_spec

LEAST, PAST = engine.ORDER_TUNE


@pytest.fixture
def fake(monkeypatch):
    cost, ran = {}, []
    monkeypatch.setattr(engine, "_ORDER_BATCH", {})
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: False)
    monkeypatch.setattr(engine, "_sorted_lanes", lambda r, whole: ran.append(whole) or
                        torch.tensor([int(whole)]))
    monkeypatch.setattr(engine, "_time_ms",
                        lambda fn, reps: fn() or cost[ran[-1]] * (3.0 if reps == 1 else 1.0))
    return cost, ran


def record(n, uneven=False):
    e, i = torch.empty(0, dtype=torch.float64), torch.zeros(n, dtype=torch.int32)
    return engine.Record("tsit5", field_spec("vdp"), n, 0.0, 1024, 2, e, e, torch.zeros(n, 2), i, i, i,
                         uneven=uneven)


@pytest.mark.parametrize("whole,want", [(0.5, 1), (0.98, 0), (1.5, 0)])
def test_the_faster_order(fake, whole, want):
    cost, ran = fake
    cost.update({False: 1.0, True: whole})
    r, runs = record(LEAST), []
    engine._tune_order(r, "auto", lambda: runs.append(1))
    assert int(r.lane_order) == want and len(runs) > 4
    timed = len(runs)
    other = record(2 * LEAST - 1)  # later records of the size take it as they are prepared
    engine._tune_order(other, "auto", lambda: runs.append(1))
    assert int(engine.prepare_lane_order(other)) == want and len(runs) == timed
    assert int(engine.prepare_lane_order(record(LEAST, uneven=True))) == 0
    plan = engine.RecordSet("tsit5", field_spec("vdp"), LEAST, 0.0, [(None, r)], None, r.y_final,
                            torch.arange(LEAST, dtype=torch.int32) % 5000, r.n_rej, r.status,
                            uneven=False, streams=[None])
    rows = plan.plan_rows()[0]
    assert torch.equal(rows.sort().values, torch.arange(LEAST))
    assert bool((plan.n_acc[rows].diff() <= 0).all())  # (off the GPU the windows are one)


def test_what_is_not_timed(fake):
    _cost, ran = fake
    for r, schedule in ((record(LEAST - 1), "auto"), (record(PAST), "auto"), (record(LEAST), "refill"),
                        (record(LEAST, uneven=True), "auto")):
        engine._tune_order(r, schedule, lambda: ran.append(2))
    assert not ran and engine._ORDER_BATCH == {}


@pytest.mark.gpu
@pytest.mark.parametrize("method,field", [("tsit5", "vdp"), ("rosenbrock23", "vdp")])
def test_same_bits(gslib, cuda, monkeypatch, method, field):
    monkeypatch.setattr(engine, "_ORDER_BATCH", {})
    n, rng = LEAST + 77, np.random.default_rng(5)
    t = lambda a: torch.tensor(a, device=cuda)  # noqa: E731
    y0, p = t(rng.uniform(-2, 2, (n, 2))), t(rng.uniform(0.5, 6.0, (n, 1)))
    kw = dict(t0=0.0, t1=2.0, rtol=1e-5, atol=1e-8, checkpoint=2)
    r = engine.forward_record(method, field_spec(field), y0, p, **kw)
    bar = torch.ones_like(r.y_final)
    first = engine.adjoint(r, p, bar)
    assert list(engine._ORDER_BATCH) == [engine._order_key(r, n)]
    for whole in (False, True):
        engine._ORDER_BATCH[engine._order_key(r, n)] = whole
        order = engine.prepare_lane_order(r)
        assert torch.equal(order.sort().values, torch.arange(n, device=cuda))
        counts = r.n_acc[order].diff()
        assert bool((counts <= 0).all()) is whole
        for a, b in zip(engine.adjoint(r, p, bar), first):
            assert torch.equal(a, b)
        again = engine.forward_record(method, field_spec(field), y0, p, workspace=engine.forward_record(
            method, field_spec(field), y0, p, **kw), **kw)
        for a, b in zip(engine.adjoint(again, p, bar), first):
            assert torch.equal(a, b)
