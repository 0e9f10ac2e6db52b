"""The reverse pass split over lanes and the dense output from the checkpoints (gs_split.cuh)
against one thread per trajectory: fields of 1 to 3 components, both methods, lanes from 1 to 32,
trajectories with fewer steps than lanes, none at all, partial last segments, repeated and end
times.  Two float64 evaluation orders of the same sums: 1e-10 of the row, the bar this
repository holds the Rosenbrock23 schedules to."""
from __future__ import annotations

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def rowrel(a, b):
    a, b = a.reshape(a.shape[0], -1).cpu().numpy(), b.reshape(b.shape[0], -1).cpu().numpy()
    return float(np.max(np.abs(a - b).max(1) / np.maximum(np.abs(b).max(1), 1e-12)))


def _batch(cuda, field, n, seed=0):
    rng = np.random.default_rng(seed)
    y0, p, t1 = {
        "linear_1": (rng.uniform(0.5, 2.0, (n, 1)), np.zeros((n, 1)), 1.0),
        "vdp": (rng.uniform(-2, 2, (n, 2)), 10 ** rng.uniform(0.0, 1.2, (n, 1)), 2.0),
        "lv": (rng.uniform(0.5, 2, (n, 2)), rng.uniform(0.5, 1.5, (n, 4)), 5.0),
        "lorenz": (rng.uniform(-1, 2, (n, 3)), rng.uniform(20, 30, (n, 1)), 1.0),
        "lorenz3": (rng.uniform(-1, 2, (n, 3)),
                    np.stack([rng.uniform(9, 11, n), rng.uniform(2, 3, n),
                              rng.uniform(20, 30, n)], 1), 1.0),
        "robertson": (np.tile([1.0, 0.0, 0.0], (n, 1)),
                      np.array([0.04, 3e7, 1e4]) * 10 ** rng.uniform(-0.5, 0.5, (n, 3)), 10.0),
    }[field]
    t1v = t1 * rng.uniform(0.05, 1.0, n)
    t1v[n // 2] = 0.0  # a trajectory without steps
    return [torch.tensor(x, device=cuda) for x in (y0, p, t1v)]


# (Robertson is stiff: on an explicit method's stability limit the frozen replay itself loses
# every digit in float64 -- 1e-4 to 1e9 relative against 80-bit arithmetic, split or not)
CASES = [("tsit5", f) for f in ("linear_1", "vdp", "lv", "lorenz", "lorenz3")] + \
        [("rosenbrock23", f) for f in ("linear_1", "vdp", "robertson")]


@pytest.mark.parametrize("method,field", CASES)
def test_split_matches_one_thread(gslib, cuda, method, field):
    from gradsolve_b200 import engine
    from gradsolve_b200.fields import field_spec
    spec = field_spec(field)
    for n in (1, 3, 37):
        y0, p, t1v = _batch(cuda, field, n)
        for K in (1, 3, 64):
            r = engine.forward_record(method, spec, y0, p, t0=0.0, t1=10.0, t1v=t1v, rtol=1e-6,
                                      atol=1e-9, checkpoint=K, max_steps=50000, cap0=50000)
            assert int(r.status.max()) == 0
            ybar = torch.cos(torch.arange(r.y_final.numel(), device=cuda,
                                          dtype=torch.float64)).reshape(r.y_final.shape)
            ref = engine.adjoint(r, p, ybar, schedule="static")
            back = torch.arange(n - 1, -1, -1, device=cuda)
            first = {}
            for lanes in (1, 2, 8, 32):
                got = engine._adjoint_split(r, lanes, p, ybar, None, None, True, True, None)
                for a, b in zip(got, ref):
                    assert rowrel(a, b) <= 1e-10, (n, K, lanes)
                perm = engine._adjoint_split(r, lanes, p, ybar, None, None, True, True, back)
                for a, b in zip(got, perm):  # whichever warp takes which trajectory
                    assert torch.equal(a, b), (n, K, lanes)
                first[lanes] = got
            auto = engine.adjoint(r, p, ybar)
            lanes = engine.split_lanes(n, spec.dim, False, False, method)
            if engine._split_applies(r, "float64", "auto"):
                assert all(torch.equal(a, b) for a, b in zip(auto, first[lanes]))


@pytest.mark.parametrize("method,field", CASES)
def test_split_dense_output(gslib, cuda, method, field):
    from gradsolve_b200 import engine
    from gradsolve_b200.fields import field_spec
    spec = field_spec(field)
    n = 37
    y0, p, t1v = _batch(cuda, field, n, seed=1)
    row = torch.tensor([0.0, 0.0, 0.01, 0.3, 0.3, 0.77, 0.999, 1.0, 1.0], device=cuda,
                       dtype=torch.float64)
    for shared in (False, True):
        tv = None if shared else t1v
        t1 = float(t1v.max())
        ts = t1 * row if shared else t1v[:, None] * row[None, :]
        for K in (1, 3, 64):
            kw = dict(t0=0.0, t1=t1, t1v=tv, rtol=1e-6, atol=1e-9, checkpoint=K,
                      max_steps=50000, cap0=50000)
            r = engine.forward_record(method, spec, y0, p, saveat_ts=ts, **kw)
            yf, ys = engine.replay_saveat(r, y0, p, ts, write_ckpt=False)
            assert rowrel(r.ys, ys) <= 1e-10
            assert torch.equal(r.ys[:, -1], r.y_final) and torch.equal(r.ys[:, 0], y0)
            ysbar = torch.sin(1.0 + torch.arange(ys.numel(), device=cuda,
                                                 dtype=torch.float64)).reshape(ys.shape)
            ybar = torch.ones_like(yf)
            for yb in (None, ybar):
                ref = engine.adjoint_saveat(r, p, ts, ysbar, yb, schedule="static")
                for lanes in (1, 4, 32):
                    got = engine._adjoint_split(r, lanes, p, yb, ts, ysbar, True, True, None)
                    for a, b in zip(got, ref):
                        assert rowrel(a, b) <= 1e-10, (shared, K, lanes)


PAIRED = CASES + [("tsit5", "lorenz96_8"), ("rosenbrock23", "hires")]


@pytest.mark.parametrize("method,field", PAIRED)
def test_two_warps_match_one_thread(gslib, cuda, method, field):
    """Two warps per 32 trajectories: the one-thread pass's arithmetic, with batches below, at and
    past a block, trajectories without steps and idle lanes (an order with entries outside)."""
    from gradsolve_b200 import engine
    from gradsolve_b200.fields import field_spec
    spec = field_spec(field)
    for n in (1, 32, 33, 70):
        if field == "hires":
            y0 = torch.tensor([1.0, 0, 0, 0, 0, 0, 0, 0.0057], device=cuda,
                              dtype=torch.float64).repeat(n, 1)
            p = torch.zeros(n, 1, device=cuda, dtype=torch.float64)
            t1v = torch.linspace(0.0, 5.0, n, device=cuda, dtype=torch.float64)
        elif field == "lorenz96_8":
            g = torch.Generator(device=cuda)
            g.manual_seed(n)
            p = torch.full((n, 1), 8.0, device=cuda, dtype=torch.float64)
            y0 = p + torch.rand(n, 8, generator=g, device=cuda, dtype=torch.float64)
            t1v = torch.linspace(0.0, 1.0, n, device=cuda, dtype=torch.float64)
        else:
            y0, p, t1v = _batch(cuda, field, n)
        for K in (1, 2):
            r = engine.forward_record(method, spec, y0, p, t0=0.0, t1=10.0, t1v=t1v, rtol=1e-6,
                                      atol=1e-9, checkpoint=K, max_steps=50000, cap0=50000)
            ybar = torch.cos(torch.arange(r.y_final.numel(), device=cuda,
                                          dtype=torch.float64)).reshape(r.y_final.shape)
            ref = engine.adjoint(r, p, ybar, schedule="static")
            got = engine._adjoint_split(r, 0, p, ybar, None, None, True, True, None)
            for a, b in zip(got, ref):
                assert rowrel(a, b) <= 1e-10, (n, K)
            order = torch.arange(n - 1, -1, -1, device=cuda)
            if n > 1:
                order[0] = n + 5  # an idle lane: trajectory n - 1 is not written
            part = engine._adjoint_split(r, 0, p, ybar, None, None, True, True, order)
            for a, b in zip(part, got):
                m = n - 1 if n > 1 else n
                assert torch.equal(a[:m], b[:m]), (n, K)


def test_split_refuses(gslib, cuda):
    from gradsolve_b200 import engine
    from gradsolve_b200._lib import GsolveError
    from gradsolve_b200.fields import field_spec
    y0, p, t1v = _batch(cuda, "lorenz", 5)
    r = engine.forward_record("tsit5", field_spec("lorenz"), y0, p, t0=0.0, t1=1.0, rtol=1e-6,
                              atol=1e-9, checkpoint=2)
    with pytest.raises(GsolveError, match="power of two"):
        engine._adjoint_split(r, 3, p, r.y_final, None, None, True, True, None)
    with pytest.raises(GsolveError, match="do not fit"):
        r64 = engine.forward_record("tsit5", field_spec("lorenz"), y0, p, t0=0.0, t1=1.0,
                                    rtol=1e-6, atol=1e-9, checkpoint=64)
        engine._adjoint_split(r64, 0, p, r64.y_final, None, None, True, True, None)
    with pytest.raises(GsolveError, match="cotangent"):
        engine._adjoint_split(r, 2, p, None, None, None, True, True, None)
    spec = field_spec("hires")
    y8 = torch.rand(4, 8, device=cuda, dtype=torch.float64)
    p8 = torch.zeros(4, 1, device=cuda, dtype=torch.float64)
    r8 = engine.forward_record("tsit5", spec, y8, p8, t0=0.0, t1=0.1, rtol=1e-6, atol=1e-9,
                               checkpoint=2)
    with pytest.raises(GsolveError, match="up to 3 components"):
        engine._adjoint_split(r8, 2, p8, r8.y_final, None, None, True, True, None)


def test_split_dense_output_takes_one_workspace(gslib, cuda):
    """adjoint_saveat's scratch is one word per requested time and gradient component, once."""
    from gradsolve_b200 import engine
    from gradsolve_b200.fields import field_spec
    n, K, spec = 4096, 64, field_spec("vdp")
    rng = np.random.default_rng(5)
    y0 = torch.tensor(rng.uniform(-2, 2, (n, 2)), device=cuda)
    p = torch.tensor(rng.uniform(0.1, 5.0, (n, 1)), device=cuda)
    ts = torch.linspace(0.0, 2.0, K, device=cuda, dtype=torch.float64)
    r = engine.forward_record("tsit5", spec, y0, p, t0=0.0, t1=2.0, rtol=1e-6, atol=1e-9,
                              saveat_ts=ts)
    bar = torch.ones_like(r.ys)
    engine.adjoint_saveat(r, p, ts, bar)
    torch.cuda.synchronize()
    before = torch.cuda.memory_allocated()
    torch.cuda.reset_peak_memory_stats()
    engine.adjoint_saveat(r, p, ts, bar)
    work = 8 * n * K * (2 + 1)
    assert torch.cuda.max_memory_allocated() - before < 1.5 * work


@pytest.mark.parametrize("method,field", [("tsit5", "lorenz"), ("tsit5", "vdp"),
                                          ("rosenbrock23", "vdp")])
def test_split_takes_the_replays_steps(gslib, cuda, method, field):
    """A caller's mesh may step backwards or hold a NaN step: the replay takes those steps, and so
    does the reverse pass on both sides of the size from which one thread takes a trajectory."""
    from gradsolve_b200 import engine
    from gradsolve_b200.fields import field_spec
    spec = field_spec(field)
    most = engine.SPLIT_EVEN_MAX[method]
    for n in (37, most, most + 1):
        y0, p, _t1v = _batch(cuda, field, n)
        dts = torch.full((n, 40), 0.02, device=cuda, dtype=torch.float64)
        dts[:, 7::9] = -1e-4
        for K in (1, 3):
            r = engine.record_from_padded(method, spec, dts, 0.0, checkpoint=K)
            yf = engine.replay(r, y0, p)
            ybar = 1.0 + torch.cos(torch.arange(yf.numel(), device=cuda,
                                                dtype=torch.float64)).reshape(yf.shape)
            ref = engine.adjoint(r, p, ybar, schedule="static")
            for a, b in zip(engine.adjoint(r, p, ybar), ref):
                assert rowrel(a, b) <= 1e-10, (n, K)
        dts[1, 5] = float("nan")
        r = engine.record_from_padded(method, spec, dts, 0.0, checkpoint=3)
        yf = engine.replay(r, y0, p)
        gy0, gp = engine.adjoint(r, p, ybar)
        assert bool(gy0[1].isnan().all()) and bool(gp[1].isnan().any()), n
        keep = torch.arange(n, device=cuda) != 1  # the other trajectories are as they were
        for a, b in zip((gy0, gp), ref):
            assert rowrel(a[keep], b[keep]) <= 1e-10, n
