"""Which reverse passes are split over lanes: Tsit5 up to SPLIT_TSIT5_STEPS steps taken, with and
without per-trajectory end times and dense output, whatever the record's capacity."""
from __future__ import annotations

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture
def splits(monkeypatch):
    from gradsolve_b200 import engine
    calls, real = [], engine._adjoint_split

    def spy(r, lanes, *args, **kw):
        calls.append(lanes)
        return real(r, lanes, *args, **kw)

    monkeypatch.setattr(engine, "_adjoint_split", spy)
    return calls


def _solve(cuda, t1, uneven, dense, **kw):
    from gradsolve_b200 import engine
    from gradsolve_b200.fields import field_spec
    n = 24
    rng = np.random.default_rng(2)
    y0 = torch.tensor(np.array([1.0, 0.0, 0.0]) + rng.normal(0, 0.1, (n, 3)), device=cuda)
    p = torch.tensor(rng.uniform(24, 30, (n, 1)), device=cuda)
    t1v = torch.linspace(0.5 * t1, t1, n, device=cuda, dtype=torch.float64) if uneven else None
    ts = torch.linspace(0.0, 0.5 * t1, 5, device=cuda, dtype=torch.float64) if dense else None
    r = engine.forward_record("tsit5", field_spec("lorenz"), y0, p, t0=0.0, t1=t1, t1v=t1v,
                              rtol=1e-8, atol=1e-8, saveat_ts=ts, **kw)
    bar = torch.ones_like(r.ys if dense else r.y_final)

    def gradient(schedule):
        if dense:
            return engine.adjoint_saveat(r, p, ts, bar, schedule=schedule)
        return engine.adjoint(r, p, bar, schedule=schedule)

    return r, gradient


@pytest.mark.parametrize("dense", [False, True])
@pytest.mark.parametrize("uneven", [False, True])
def test_long_trajectories_are_not_split(gslib, cuda, splits, uneven, dense):
    from gradsolve_b200 import engine
    for kw in ({}, {"cap0": 8192}):  # in tiers, and in one record
        r, gradient = _solve(cuda, 70.0, uneven, dense, **kw)
        assert int(r.n_acc.max()) > engine.SPLIT_TSIT5_STEPS
        got = gradient("auto")
        assert all(lanes == engine.PAIRED for lanes in splits)
        for a, b in zip(got, gradient("refill" if uneven else "static")):
            assert torch.equal(a, b)


@pytest.mark.parametrize("dense", [False, True])
@pytest.mark.parametrize("uneven", [False, True])
def test_short_trajectories_are_split_at_any_capacity(gslib, cuda, splits, uneven, dense):
    _r, gradient = _solve(cuda, 1.0, uneven, dense, cap0=20000)
    gradient("auto")
    assert splits and splits[0] >= 1
