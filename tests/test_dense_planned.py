"""How a planned batch (ordered by an earlier solve's counts) takes its dense output
(engine._planned_dense): timed where it is one tier, by size where it is several (CPU, faked timings);
and both routes of the entry point against the replay of the recorded mesh (GPU)."""
from __future__ import annotations

from types import SimpleNamespace

import numpy as np
import pytest
import torch

from gradsolve_b200 import engine
from gradsolve_b200.fields import field_spec


@pytest.fixture
def fake(monkeypatch):
    cost, ran = {}, []
    monkeypatch.setattr(engine, "_DENSE_PLANNED", {})
    monkeypatch.setattr(engine, "_forward_one", lambda *a, dense: ran.append(dense))
    monkeypatch.setattr(engine, "_time_ms",
                        lambda fn, reps: fn() or cost[ran[-1]] * (3.0 if reps == 1 else 1.0))
    return cost, ran


def ask(n, K=4, alone=True, precision="float64", uneven=True, times=64):
    y0, p = torch.zeros(n, 2), torch.zeros(n, 1)
    ts = torch.zeros(n, times) if times else None
    return engine._planned_dense(("tsit5", field_spec("vdp"), y0, p, p[:, 0] if uneven else None, ts,
                                  1024, SimpleNamespace(ckpt_every=K), {"precision": precision}),
                                 alone)


@pytest.mark.parametrize("apart,want", [(0.5, "apart"), (0.995, "within"), (1.5, "within")])
def test_one_tier_is_timed(fake, apart, want):
    cost, ran = fake
    cost.update(within=1.0, apart=apart)
    assert ask(4096) == want and ran.count("apart") == ran.count("within") > 2
    timed = len(ran)
    assert ask(8191) == want and len(ran) == timed  # once per power of two ...
    cost.update(within=apart, apart=1.0)
    other = "within" if apart < 1 else "apart"
    for kw in (dict(n=8192), dict(n=4096, K=8), dict(n=4096, uneven=False), dict(n=4096, times=8)):
        assert ask(**kw) == other or apart == 0.995  # ... and interval, kind and number of times
    assert ask(4096) == want


def test_what_is_not_timed(fake):
    _cost, ran = fake
    assert ask(4095) == ask(4096, precision="mixed") == ask(4096, times=0) == "auto"
    assert ask(1 << 17, alone=False) == "auto" and ask((1 << 17) + 1, alone=False) == "within"
    assert not ran


@pytest.mark.gpu
@pytest.mark.parametrize("schedule", ["auto", "static", "strided"])
@pytest.mark.parametrize("method,field", [("tsit5", "vdp"), ("rosenbrock23", "vdp"),
                                          ("tsit5", "lorenz96_8")])
def test_routes_agree_with_the_replay(gslib, cuda, method, field, schedule):
    rng, n, D = np.random.default_rng(4), 4133, field_spec(field).dim
    t = lambda a: torch.tensor(a, device=cuda)  # noqa: E731
    y0, p = t(rng.uniform(1.0, 2.0, (n, D))), t(rng.uniform(4.0, 8.0, (n, 1)))
    t1v = t(rng.uniform(0.2, 2.0, n))
    ts = t1v[:, None] * torch.linspace(0.0, 1.0, 9, device=cuda, dtype=torch.float64)
    kw = dict(t0=0.0, t1=2.0, rtol=1e-6, atol=1e-9, dt0=None, max_steps=20000, checkpoint=4,
              budget_bytes=1 << 40, precision="float64", schedule=schedule)
    spec, ys = field_spec(field), {}
    for route in ("within", "apart"):
        r = engine._forward_one(method, spec, y0, p, t1v, ts, 1024, None, kw, dense=route)
        assert int(r.status.max()) == 0
        ref = engine.replay_saveat(r, y0, p, ts, write_ckpt=False)[1]
        assert float(((r.ys - ref).abs().amax(2) / ref.abs().amax(2)).max()) <= 1e-10
        assert torch.equal(r.ys[:, -1], r.y_final) and torch.equal(r.ys[:, 0], y0)
        ys[route] = r.ys
    # a planned solve takes one of the two
    full = dict(kw, workspace=None, t1v=t1v, saveat_ts=ts)
    first = engine.forward_record(method, spec, y0, p, **full)
    counts = first.n_acc.clone()  # (the workspace's buffers become the plan's)
    again = engine.forward_record(method, spec, y0, p, **dict(full, workspace=first))
    assert float(((again.ys - ys["apart"]).abs().amax(2) / ys["apart"].abs().amax(2)).max()) <= 1e-10
    assert torch.equal(again.n_acc, counts)
