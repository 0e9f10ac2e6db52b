"""A record's status codes and, where its reverse pass asks for it, its longest step count, in one
read (engine._read_status, CPU)."""
from __future__ import annotations

import pytest
import torch

from gradsolve_b200 import engine
from gradsolve_b200.fields import field_spec


def record(method="tsit5", field="lorenz", n=5, cap=8192, dtype=torch.float64, uneven=False):
    i32 = lambda *v: torch.tensor((v * n)[:n], dtype=torch.int32)  # noqa: E731
    e = torch.empty(0, dtype=dtype)
    return engine.Record(method, field_spec(field), n, 0.0, cap, 2, e, e, torch.zeros(n, 3),
                         i32(3, 5000, 7), i32(0), i32(0, 3, 1), uneven=uneven)


@pytest.mark.parametrize("kw,counts", [
    (dict(), True), (dict(n=1), True), (dict(uneven=True, n=1 << 14), True),
    (dict(cap=4096), False), (dict(method="rosenbrock23"), False), (dict(field="hires"), False),
    (dict(dtype=torch.float32), False), (dict(n=4097), False),
    (dict(uneven=True, n=(1 << 14) + 1), False)])
def test_one_read(kw, counts):
    r = record(**kw)
    assert engine._read_status(r) == int(r.status.max())
    assert r.steps_max == (int(r.n_acc.max()) if counts else None)


def test_row_moves_out_of_range(monkeypatch):
    """The row-move counter is read with them, and still raises."""
    r, c = record(), torch.zeros(1, dtype=torch.int64)
    monkeypatch.setitem(engine._BAD_MOVES, r.status.device.index, c)
    assert engine._read_status(r) == 3 and r.steps_max == 5000
    c += 2
    r.steps_max = None
    with pytest.raises(Exception, match="2"):
        engine._read_status(r)
