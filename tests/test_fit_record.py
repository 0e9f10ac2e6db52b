"""What a record holds beyond its batch's steps (engine.fit_record): kept and counted while the
records alive hold little enough together, copied away otherwise (CPU); and on the device what
closures hold, and that one whose first capacity does not fit is built all the same."""
from __future__ import annotations

import gc
from types import SimpleNamespace

import pytest
import torch

from gradsolve_b200 import engine
from gradsolve_b200.fields import field_spec


def _record(n, cap, steps, K=2, precision="float64"):
    rec, ckpt = engine._alloc_record(n, cap, 3, K, torch.device("cpu"), precision)
    rec.copy_(torch.arange(rec.numel()))
    ckpt.copy_(-torch.arange(ckpt.numel()).to(ckpt.dtype))
    acc = torch.full((n,), steps, dtype=torch.int32)
    return engine.Record("tsit5", field_spec("lorenz"), n, 0.0, cap, K, rec, ckpt,
                         torch.zeros(n, 3, dtype=torch.float64), acc, acc * 0, acc * 0)


@pytest.mark.parametrize("precision", ["float64", "float32"])
@pytest.mark.parametrize("steps", [0, 1, 7, 8, 95, 1500, 2048])
@pytest.mark.parametrize("K", [1, 2, 5])
def test_copy_is_the_start_of_the_record(gslib, K, steps, precision):
    r = _record(3, 2048, steps, K, precision)
    f = engine.fit_record(r, 0)  # no share at all: every excess is copied away
    cap = max(4, -(-steps // 4) * 4)
    if cap >= 2048:
        assert f is r
        return
    assert f.cap == cap and f.n_acc is r.n_acc and f.ckpt_every == K
    rec, ckpt = engine._alloc_record(3, cap, 3, K, torch.device("cpu"), precision)
    assert f.rec.shape == rec.shape and f.ckpt.shape == ckpt.shape
    assert torch.equal(f.rec, r.rec[:rec.numel()])
    slots = gslib.lib().gs_ckpt_slots(cap, K)
    assert slots * K >= steps + 1  # every written slot is kept
    rows = slots * 3 * 4
    assert torch.equal(f.ckpt[:rows], r.ckpt[:rows])


def test_default_records_are_not_counted(gslib, monkeypatch):
    monkeypatch.setattr(engine, "_EXCESS", {})
    r = _record(3, engine.DEFAULT_CAP0, 7)
    assert engine.fit_record(r, 0) is r and engine._EXCESS == {}


def test_excess_is_bounded_over_the_records_alive(gslib, monkeypatch):
    monkeypatch.setattr(engine, "_EXCESS", {})
    r = _record(64, 4096, 1500)
    excess = r.nbytes - _record(64, engine.DEFAULT_CAP0, 0).nbytes
    budget = engine.CAP_SHARE * (excess + excess // 2)  # room for one record's excess, not two
    assert engine.fit_record(r, budget) is r
    assert engine._EXCESS[None] == excess
    other = _record(64, 4096, 1500)
    fitted = engine.fit_record(other, budget)
    assert fitted is not other and fitted.cap == 1500 and engine._EXCESS[None] == excess
    del r
    gc.collect()
    assert engine._EXCESS[None] == 0
    assert engine.fit_record(other, budget) is other


def _robertson(n, cuda):
    g = torch.Generator(device=cuda)
    g.manual_seed(n)
    y0 = torch.tensor([[1.0, 0.0, 0.0]], device=cuda, dtype=torch.float64).repeat(n, 1)
    p = torch.tensor([[0.04, 3e7, 1e4]], device=cuda, dtype=torch.float64) * (
        0.5 + torch.rand(n, 3, generator=g, device=cuda, dtype=torch.float64))
    problem = SimpleNamespace(name="robertson", dim=3, t0=0.0, t1=1e4, is_stiff=True)
    return problem, y0, p


def _gradient(f, y0, p):
    y0, p = y0.clone().requires_grad_(), p.clone().requires_grad_()
    return torch.autograd.grad(f(y0, p).square().sum(), (y0, p))


@pytest.mark.gpu
def test_closures_alive_share_one_excess(gslib, cuda, monkeypatch):
    import gradsolve_b200 as gs
    monkeypatch.setattr(engine, "_EXCESS", {})
    monkeypatch.setattr(engine, "_checkpoint_budget", lambda: 8 << 30)
    problem, y0, p = _robertson(1000, cuda)
    kw = dict(wrt=("y0", "params"), rtol=1e-6, atol=1e-10)
    ref = _gradient(gs.grad_closure(problem, y0, p, max_steps=1000, **kw), y0, p)
    torch.cuda.synchronize()
    before = torch.cuda.memory_allocated()
    alive = [gs.grad_closure(problem, y0, p, **kw) for _ in range(6)]
    # (50,000 steps were 1.2 GB each; some 600 are 15 MB)
    held = torch.cuda.memory_allocated() - before
    assert held < (8 << 30) // engine.CAP_SHARE + 6 * (32 << 20)
    for f in alive:
        for a, b in zip(_gradient(f, y0, p), ref):
            assert torch.equal(a, b)
    del alive, f
    gc.collect()
    assert engine._EXCESS[0] == 0


@pytest.mark.gpu
def test_closure_whose_first_capacity_does_not_fit(gslib, cuda, monkeypatch):
    import gradsolve_b200 as gs
    problem, y0, p = _robertson(300, cuda)
    kw = dict(wrt=("y0", "params"), rtol=1e-6, atol=1e-10)
    ref = _gradient(gs.grad_closure(problem, y0, p, **kw), y0, p)
    alloc, refused = engine._alloc_record, []

    def short(n, cap, *args):
        if cap > engine.DEFAULT_CAP0:
            refused.append(cap)
            raise torch.OutOfMemoryError("CUDA out of memory")
        return alloc(n, cap, *args)

    monkeypatch.setattr(engine, "_alloc_record", short)
    f = gs.grad_closure(problem, y0, p, **kw)
    assert refused and f.state.record.cap == engine.DEFAULT_CAP0
    for a, b in zip(_gradient(f, y0, p), ref):
        assert torch.equal(a, b)


@pytest.mark.gpu
@pytest.mark.parametrize("checkpoint", [0, -3, 10 ** 6])
def test_refused_intervals(gslib, cuda, checkpoint):
    import gradsolve_b200 as gs
    problem, y0, p = _robertson(3, cuda)
    with pytest.raises(ValueError, match="checkpoint interval"):
        gs.grad_closure(problem, y0, p, checkpoint=checkpoint)
