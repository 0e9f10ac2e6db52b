"""The float32-stage interval's tuner (engine.autotune_ckpt_every, CPU, timings faked): TUNE_MIXED unless
another interval is faster by the margin in two measurements."""
from __future__ import annotations

from types import SimpleNamespace

import pytest
import torch

from gradsolve_b200 import engine
from gradsolve_b200.fields import field_spec


@pytest.mark.parametrize("first,second,want", [
    ({2: 1.0, 4: 1.03, 8: 1.2}, None, 4),                  # within the margin
    ({2: 1.0, 4: 1.10, 8: 1.2}, {2: 1.0, 4: 1.02}, 4),     # a disturbed first measurement
    ({2: 1.0, 4: 1.10, 8: 1.2}, {2: 1.0, 4: 1.09}, 2),     # slower both times
])
def test_another_interval_wins_twice(monkeypatch, first, second, want):
    now, runs = {}, []

    def forward(method, spec, y0, p, checkpoint, workspace=None, **kw):
        if workspace is None:
            runs.append(checkpoint)
        again = runs.count(checkpoint) > 1
        now["ms"] = (second if again else first)[checkpoint]
        return SimpleNamespace(y_final=y0)

    class Event:
        def __init__(self, enable_timing):
            pass

        def record(self):
            pass

        def synchronize(self):
            pass

        def elapsed_time(self, other):
            return now["ms"]

    monkeypatch.setattr(engine, "forward_record", forward)
    monkeypatch.setattr(engine, "adjoint", lambda *a, **k: None)
    monkeypatch.setattr(engine, "_checkpoint_budget", lambda: 1 << 40)
    monkeypatch.setattr(engine, "_TUNED", {})
    monkeypatch.setattr(torch.cuda, "Event", Event)
    y0 = torch.zeros(5000, 2, dtype=torch.float64)
    got = engine.autotune_ckpt_every("tsit5", field_spec("lv"), y0, y0, t0=0.0, t1=1.0, rtol=1e-6,
                                     atol=1e-8, precision="mixed", candidates=(2, 4, 8))
    assert got == want
    assert runs == [2, 4, 8] + ([] if second is None else [4, 2])
