"""Whether a batch with its own end times takes the split reverse pass: timed against the unsplit one
from SPLIT_TUNE_MIN trajectories up (engine._split_pays; CPU, with faked timings), and the gradient by
either choice (GPU)."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from gradsolve_b200 import engine
from gradsolve_b200.fields import field_spec


@pytest.fixture
def fake(monkeypatch):
    cost, ran = {}, []
    monkeypatch.setattr(engine, "_SPLIT_PAYS", {})
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: False)
    monkeypatch.setattr(engine, "_time_ms",
                        lambda fn, reps: fn() or cost[ran[-1]] * (3.0 if reps == 1 else 1.0))
    return cost, ran


def record(n, uneven=True):
    e, i = torch.empty(0), torch.zeros(n, dtype=torch.int32)
    return engine.Record("tsit5", field_spec("vdp"), n, 0.0, 1024, 4, e, e, torch.zeros(n, 2), i, i, i,
                         uneven=uneven)


@pytest.mark.parametrize("split,want", [(0.5, True), (0.98, False), (1.5, False)])
def test_the_faster_pass(fake, split, want):
    cost, ran = fake
    cost.update({False: 1.0, True: split})
    assert engine._split_pays(record(4096), 64, ran.append) is want
    assert ran.count(True) == ran.count(False) > 2
    timed = len(ran)
    assert engine._split_pays(record(8191), 64, ran.append) is want and len(ran) == timed
    cost.update({False: split, True: 1.0})
    for r, times in ((record(8192), 64), (record(4096), 0)):
        assert engine._split_pays(r, times, ran.append) is (split > 1.1)


def test_what_is_not_timed(fake, monkeypatch):
    _cost, ran = fake
    assert engine._split_pays(record(4095), 64, ran.append)
    assert engine._split_pays(record(4096, uneven=False), 64, ran.append)
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: True)
    assert engine._split_pays(record(4096), 64, ran.append)
    assert not ran and engine._SPLIT_PAYS == {}


@pytest.mark.gpu
@pytest.mark.parametrize("dense", [False, True])
def test_gradient_of_either_choice(gslib, cuda, monkeypatch, dense):
    n, rng = 5000, np.random.default_rng(3)
    t = lambda a: torch.tensor(a, device=cuda)  # noqa: E731
    y0, p, t1v = t(rng.uniform(-2, 2, (n, 2))), t(rng.uniform(0.5, 5.0, (n, 1))), t(rng.uniform(0.1, 5, n))
    ts = t1v[:, None] * torch.linspace(0.0, 1.0, 9, device=cuda, dtype=torch.float64) if dense else None
    r = engine.forward_record("tsit5", field_spec("vdp"), y0, p, t0=0.0, t1=5.0, t1v=t1v, rtol=1e-6,
                              atol=1e-9, saveat_ts=ts)
    bar = torch.ones_like(r.ys if dense else r.y_final)
    split, real = [], engine._adjoint_split
    monkeypatch.setattr(engine, "_adjoint_split", lambda *a, **kw: split.append(1) or real(*a, **kw))
    got = {}
    for pays in (True, False):
        monkeypatch.setattr(engine, "_split_pays", lambda *a, pays=pays: pays)
        before = len(split)
        got[pays] = engine.adjoint_saveat(r, p, ts, bar) if dense else engine.adjoint(r, p, bar)
        assert (len(split) > before) is pays
    for a, b in zip(got[True], got[False]):
        assert float(((a - b).abs().amax(1) / b.abs().amax(1)).max()) <= 1e-9
    ref = (engine.adjoint_saveat(r, p, ts, bar, schedule="refill") if dense else
           engine.adjoint(r, p, bar, schedule="refill"))
    for a, b in zip(got[False], ref):
        assert torch.equal(a, b)
