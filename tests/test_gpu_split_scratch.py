"""Dense output's split reverse pass where its workspace does not fit: the unsplit pass, which needs
none, answers instead."""
from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu


def test_gradient_without_room_for_the_workspace(gslib, cuda):
    from gradsolve_b200 import engine
    from gradsolve_b200.fields import field_spec
    n, K, spec = 4096, 2048, field_spec("vdp")
    g = torch.Generator(device=cuda)
    g.manual_seed(0)
    y0 = torch.rand(n, 2, generator=g, device=cuda, dtype=torch.float64)
    p = 0.5 + torch.rand(n, 1, generator=g, device=cuda, dtype=torch.float64)
    ts = torch.linspace(0.0, 1.0, K, device=cuda, dtype=torch.float64)
    r = engine.forward_record("tsit5", spec, y0, p, t0=0.0, t1=1.0, rtol=1e-6, atol=1e-9,
                              saveat_ts=ts)
    bar = torch.ones_like(r.ys)
    ref = engine.adjoint_saveat(r, p, ts, bar, schedule="static")
    assert engine._lanes_for(r, True) > 0
    work = 8 * n * K * (2 + 1)  # 201 MB
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    total = torch.cuda.get_device_properties(0).total_memory
    try:
        torch.cuda.set_per_process_memory_fraction(
            (torch.cuda.memory_reserved() + work // 2) / total)
        got = engine.adjoint_saveat(r, p, ts, bar)
    finally:
        torch.cuda.set_per_process_memory_fraction(1.0)
    for a, b in zip(got, ref):
        assert torch.equal(a, b)
    # with room, the split pass: the same to rounding
    for a, b in zip(engine.adjoint_saveat(r, p, ts, bar), ref):
        assert float((a - b).abs().max() / b.abs().max()) <= 1e-10
