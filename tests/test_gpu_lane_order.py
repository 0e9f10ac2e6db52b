"""gs_lane_order: a permutation ordered by count within each window, equal counts in batch order,
at the edges of the windows; and the reverse pass in that order, bit for bit the batch-order one."""
from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("window", [512, 4096])
@pytest.mark.parametrize("n", [1, 2, 511, 512, 513, 4095, 4097, 12_345])
def test_windows_are_sorted_permutations(gslib, cuda, n, window):
    from gradsolve_b200 import engine
    g = torch.Generator(device=cuda)
    g.manual_seed(n)
    a = torch.randint(0, 50, (n,), generator=g, device=cuda, dtype=torch.int32)
    a[n // 2] = 2 ** 31 - 1
    b = torch.randint(0, 3, (n,), generator=g, device=cuda, dtype=torch.int32)
    for second in (None, b):
        order = engine._window_order(a, second, window).cpu()
        cost = a.cpu().long() + (0 if second is None else b.cpu().long())
        cost = cost.clamp_max(2 ** 31 - 2)
        want = torch.cat([w0 + torch.argsort(cost[w0:w0 + window], descending=True, stable=True)
                          for w0 in range(0, n, window)])
        assert torch.equal(order, want)


def test_reverse_pass_in_window_order(gslib, cuda):
    from gradsolve_b200 import engine
    from gradsolve_b200.fields import field_spec
    g = torch.Generator(device=cuda)
    g.manual_seed(0)
    n = 5000  # above ORDER_LANES_MIN, a partial last window
    y0 = 0.5 + 1.5 * torch.rand(n, 2, generator=g, device=cuda, dtype=torch.float64)
    p = 0.5 + torch.rand(n, 4, generator=g, device=cuda, dtype=torch.float64)
    r = engine.forward_record("tsit5", field_spec("lv"), y0, p, t0=0.0, t1=10.0, rtol=1e-6,
                              atol=1e-8, checkpoint=2)
    got = engine.adjoint(r, p, r.y_final)
    assert r.lane_order is not None
    r.lane_order = torch.arange(n, device=cuda)
    for a, b in zip(got, engine.adjoint(r, p, r.y_final)):
        assert torch.equal(a, b)
