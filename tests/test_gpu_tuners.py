"""What the autotuners time, and which batches take what they chose: the one-thread passes whose
parameter is being chosen, whatever pass the sample's own size would take, and a small even batch's
interval is the two-warp pass's own."""
from __future__ import annotations

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture
def tables(monkeypatch):
    from gradsolve_b200 import engine
    for name in ("_TUNED", "_OCC", "_OCC_REV", "_OCC_TUNED"):
        monkeypatch.setattr(engine, name, {})
    calls, real = [], engine._adjoint_split

    def spy(r, lanes, *args, **kw):
        calls.append(lanes)
        return real(r, lanes, *args, **kw)

    monkeypatch.setattr(engine, "_adjoint_split", spy)
    return calls


def _batch(cuda, field, n):
    rng = np.random.default_rng(n)
    if field == "lorenz":
        y0, p = rng.uniform(-1, 2, (n, 3)), rng.uniform(20, 30, (n, 1))
    else:
        y0 = np.tile([1.0, 0.0, 0.0], (n, 1))
        p = np.array([0.04, 3e7, 1e4]) * 10 ** rng.uniform(-0.5, 0.5, (n, 3))
    return torch.tensor(y0, device=cuda), torch.tensor(p, device=cuda)


@pytest.mark.parametrize("method,field", [("tsit5", "lorenz"), ("rosenbrock23", "robertson")])
@pytest.mark.parametrize("uneven", [False, True])
def test_tuners_time_the_passes_they_choose_for(gslib, cuda, tables, method, field, uneven):
    from gradsolve_b200 import engine
    from gradsolve_b200.fields import field_spec
    spec = field_spec(field)
    y0, p = _batch(cuda, field, 8192)
    t1v = torch.linspace(0.1, 1.0, 8192, device=cuda, dtype=torch.float64) if uneven else None
    kw = dict(t0=0.0, t1=1.0, rtol=1e-6, atol=1e-9, t1v=t1v)
    engine.autotune_ckpt_every(method, spec, y0, p, **kw)
    if not uneven:
        engine.autotune_occupancy(spec, y0, p, checkpoint=2, method=method, **kw)
    assert tables == []


@pytest.mark.parametrize("method,field", [("tsit5", "lorenz"), ("rosenbrock23", "robertson")])
def test_small_even_batches_have_their_own_interval(gslib, cuda, tables, method, field):
    from gradsolve_b200 import engine
    from gradsolve_b200.fields import field_spec
    spec = field_spec(field)
    key = (method, spec.key, "float64")
    kw = dict(t0=0.0, t1=1.0, rtol=1e-6, atol=1e-9)
    y0, p = _batch(cuda, field, 1 << 14)
    r = engine.forward_record(method, spec, y0, p, **kw)
    assert r.ckpt_every == 2 and key not in engine._TUNED  # nothing tuned on them
    engine.adjoint(r, p, torch.ones_like(y0))
    assert tables == [engine.PAIRED]
    engine._TUNED[key] = 12  # as a large batch of the field may have chosen
    assert engine.forward_record(method, spec, y0, p, **kw).ckpt_every == 2
    y0, p = _batch(cuda, field, (1 << 14) + 1)
    assert engine.forward_record(method, spec, y0, p, **kw).ckpt_every == 12


@pytest.mark.parametrize("dense", [False, True])
@pytest.mark.parametrize("method,field,want", [("tsit5", "lorenz", 4),
                                               ("rosenbrock23", "robertson", 8)])
def test_uneven_split_batches_have_their_own_interval(gslib, cuda, tables, method, field, want,
                                                      dense):
    from gradsolve_b200 import engine
    from gradsolve_b200.fields import field_spec
    spec, n = field_spec(field), 5000
    key = (method, spec.key, "float64")
    y0, p = _batch(cuda, field, n)
    t1v = torch.linspace(0.1, 1.0, n, device=cuda, dtype=torch.float64)
    kw = dict(t0=0.0, t1=1.0, rtol=1e-6, atol=1e-9, t1v=t1v,
              saveat_ts=t1v[:, None] * 0.5 if dense else None)
    assert engine.forward_record(method, spec, y0, p, **kw).ckpt_every == want
    assert key not in engine._TUNED
    engine._TUNED[key] = 16
    assert engine.forward_record(method, spec, y0, p, **kw).ckpt_every == want
