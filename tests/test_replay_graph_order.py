"""A captured replay keeps the lane order its reverse pass was captured with, whatever order the record
is given afterwards."""
from __future__ import annotations

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def test_order_outlives_the_records(gslib, cuda, monkeypatch):
    from gradsolve_b200 import engine
    from gradsolve_b200.fields import field_spec
    monkeypatch.setattr(engine, "_ORDER_BATCH", {})
    n, rng = engine.ORDER_TUNE[0] + 5, np.random.default_rng(6)
    t = lambda a: torch.tensor(a, device=cuda)  # noqa: E731
    y0, p = t(rng.uniform(-2, 2, (n, 2))), t(rng.uniform(0.5, 6.0, (n, 1)))
    r = engine.forward_record("tsit5", field_spec("vdp"), y0, p, t0=0.0, t1=2.0, rtol=1e-6, atol=1e-9,
                              checkpoint=2)
    graph = engine.ReplayGraph(r, y0, p, lambda y: 2.0 * y)
    assert graph.order is r.lane_order  # held by the graph, made on the caller's stream
    first = [x.clone() for x in graph()]
    ptr = graph.order.data_ptr()
    r.lane_order = None
    junk = [torch.full((n,), -1, dtype=torch.int64, device=cuda) for _ in range(64)]
    assert all(x.data_ptr() != ptr for x in junk)
    for a, b in zip(graph(), first):
        assert torch.equal(a, b)
