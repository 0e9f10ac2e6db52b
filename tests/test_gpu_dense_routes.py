"""The dense output of a float64 forward by each of its routes -- the forward's own re-steps under each
schedule, and the pass over the checkpoints -- against the replay of the recorded mesh, on both sides
of the sizes and intervals at which the route changes (gs_abi.cu, states_apart)."""
from __future__ import annotations

import ctypes

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def rowrel(a, b):
    a, b = a.reshape(a.shape[0], -1), b.reshape(b.shape[0], -1)
    return float(((a - b).abs().max(1).values / b.abs().max(1).values.clamp_min(1e-12)).max())


def _batch(cuda, field, n):
    g = torch.Generator(device=cuda)
    g.manual_seed(n)
    u = lambda lo, hi, d: lo + (hi - lo) * torch.rand(n, d, generator=g, device=cuda,  # noqa: E731
                                                      dtype=torch.float64)
    start = lambda *v: torch.tensor([v], device=cuda, dtype=torch.float64).repeat(n, 1)  # noqa: E731
    return {"lorenz": lambda: (u(-1, 2, 3), u(20, 30, 1), 0.5),
            "lv": lambda: (u(0.5, 2, 2), u(0.5, 1.5, 4), 3.0),
            "vdp": lambda: (u(-2, 2, 2), u(1.0, 8.0, 1), 2.0),
            "lorenz96_8": lambda: (u(8, 9, 8), u(7.5, 8.5, 1), 0.5),
            "robertson": lambda: (start(1.0, 0, 0), start(0.04, 3e7, 1e4) * u(0.5, 2.0, 3), 10.0),
            "hires": lambda: (start(1.0, 0, 0, 0, 0, 0, 0, 0.0057) * u(0.9, 1.1, 1), start(0.0),
                              5.0)}[field]()


ROW = (0.0, 0.1, 0.37, 0.37, 0.9, 1.0)

# (method, field, uneven, interval, the last size of the pass over the checkpoints)
LINES = [("tsit5", "lorenz", False, 4, 1 << 14), ("tsit5", "lv", False, 32, 1 << 11),
         ("tsit5", "lorenz96_8", False, 2, 1 << 13), ("tsit5", "lorenz96_8", False, 32, 1 << 11),
         ("rosenbrock23", "robertson", False, 32, 1 << 14),
         ("rosenbrock23", "hires", False, 2, 1 << 12), ("rosenbrock23", "hires", False, 32, 1 << 10),
         ("tsit5", "vdp", True, 32, 1 << 15), ("tsit5", "lorenz96_8", True, 32, 1 << 13),
         ("rosenbrock23", "robertson", True, 32, 1 << 15),
         ("rosenbrock23", "hires", True, 8, 1 << 13), ("rosenbrock23", "hires", True, 2, 1 << 15)]


@pytest.mark.parametrize("method,field,uneven,K,most", LINES)
def test_both_sides_of_the_line(gslib, cuda, method, field, uneven, K, most):
    from gradsolve_b200 import engine
    from gradsolve_b200.fields import field_spec
    row = torch.tensor(ROW, device=cuda, dtype=torch.float64)
    for n in (3, most, most + 1):
        y0, p, t1 = _batch(cuda, field, n)
        t1v = torch.linspace(0.2 * t1, t1, n, device=cuda, dtype=torch.float64) if uneven else None
        ts = t1v[:, None] * row if uneven else t1 * row
        r = engine.forward_record(method, field_spec(field), y0, p, t0=0.0, t1=t1, t1v=t1v,
                                  rtol=1e-5, atol=1e-8, checkpoint=K, saveat_ts=ts)
        # (at these tolerances a Robertson trajectory in some thousands leaves the positive octant
        # and ends with status 2, whatever the route)
        ok = r.status == 0
        assert int(ok.sum()) >= n - n // 10000
        _yf, ys = engine.replay_saveat(r, y0, p, ts, write_ckpt=False)
        assert rowrel(r.ys[ok], ys[ok]) <= 1e-10, n
        assert torch.equal(r.ys[ok][:, -1], r.y_final[ok]) and torch.equal(r.ys[:, 0], y0), n


@pytest.mark.parametrize("schedule", ["static", "refill", "strided"])
@pytest.mark.parametrize("method,field", [("tsit5", "lorenz"), ("tsit5", "lorenz96_8"),
                                          ("rosenbrock23", "robertson"), ("rosenbrock23", "hires")])
def test_in_the_forward(gslib, cuda, method, field, schedule):
    """The entry point without a record keeps no mesh to walk: the forward re-steps its times."""
    from gradsolve_b200 import engine
    from gradsolve_b200.fields import field_spec
    spec, n = field_spec(field), 700
    y0, p, t1 = _batch(cuda, field, n)
    t1v = torch.linspace(0.2 * t1, t1, n, device=cuda, dtype=torch.float64)
    ts = t1v[:, None] * torch.tensor(ROW, device=cuda, dtype=torch.float64)
    r = engine.forward_record(method, spec, y0, p, t0=0.0, t1=t1, t1v=t1v, rtol=1e-5, atol=1e-8,
                              checkpoint=4, saveat_ts=ts)
    ys, yf = torch.empty_like(r.ys), torch.empty_like(y0)
    n_acc, n_rej, status = (torch.empty(n, dtype=torch.int32, device=cuda) for _ in range(3))
    _rec, ckpt = engine._alloc_record(n, r.cap, spec.dim, 4, cuda)
    ptr = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
    rc = gslib.lib().gs_fwd_record_saveat(
        engine._METHOD_CODE[method], spec.code, engine._SCHED[schedule], n, ptr(y0), ptr(p), 0.0,
        ptr(t1v), t1, 1e-5, 1e-8, -1.0, 100000, r.cap, 4, None, ptr(ckpt), ptr(yf), ptr(n_acc),
        ptr(n_rej), ptr(status), ptr(ts), len(ROW), len(ROW), ptr(ys), None)
    assert rc == 0, gslib.lib().gs_last_error()
    torch.cuda.synchronize()
    assert torch.equal(n_acc, r.n_acc) and torch.equal(status, r.status)
    assert rowrel(ys, r.ys) <= 1e-10 and rowrel(yf, r.y_final) <= 1e-10


def test_solve_with_saved_times(gslib, cuda, oracle):
    """solve(saveat=) at a size past the line and one below, against the oracle's replay."""
    from types import SimpleNamespace
    import gradsolve_b200 as gs
    problem = SimpleNamespace(name="diffeqgpu_lorenz", dim=3, t0=0.0, t1=1.0, is_stiff=False)
    for n in (64, (1 << 14) + 1):
        y0, p, _t1 = _batch(cuda, "lorenz", n)
        ts = np.linspace(0.0, 1.0, 9)
        r = gs.solve(problem, y0, p, saveat=ts, rtol=1e-8, atol=1e-8)
        rows = np.arange(0, n, max(1, n // 32))
        for k, t in enumerate(ts[1:], 1):  # the state at t is a solve that ends there, to tolerance
            ref = oracle.record("tsit5", "lorenz", y0.cpu().numpy()[rows], p.cpu().numpy()[rows], 0.0,
                                float(t), 1e-10, 1e-10)["y_final"]
            assert np.abs(r.y_saved[rows, k] - ref).max() <= 1e-4
        assert (r.y_saved[:, -1] == r.y_final).all() and (r.y_saved[:, 0] == y0.cpu().numpy()).all()
