"""The compacting forward (gs_compact.cuh) against the one-launch forward: the same arithmetic per
trajectory, whatever list it passes through, so everything is bit for bit equal -- below, at and
past a warp and the lists' sizes, with trajectories of one step, full records and max_steps."""
from __future__ import annotations

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

CASES = [("tsit5", "lorenz", "float64"), ("tsit5", "lv", "float64"), ("tsit5", "lv", "mixed"),
         ("tsit5", "lorenz96_4", "float64"), ("rosenbrock23", "robertson", "float64"),
         ("rosenbrock23", "vdp", "float64")]


def _batch(field, n, cuda):
    rng = np.random.default_rng(n)
    y0, p, t1 = {
        "lorenz": (rng.uniform(-1, 2, (n, 3)), rng.uniform(20, 30, (n, 1)), 2.0),
        "lv": (rng.uniform(0.5, 2, (n, 2)), rng.uniform(0.5, 1.5, (n, 4)), 10.0),
        "lorenz96_4": (rng.uniform(6, 9, (n, 4)), rng.uniform(7.5, 8.5, (n, 1)), 2.0),
        "robertson": (np.tile([1.0, 0.0, 0.0], (n, 1)),
                      np.array([0.04, 3e7, 1e4]) * 10 ** rng.uniform(-0.5, 0.5, (n, 3)), 100.0),
        "vdp": (rng.uniform(-2, 2, (n, 2)), 10 ** rng.uniform(0.5, 1.5, (n, 1)), 2.0),
    }[field]
    return torch.tensor(y0, device=cuda), torch.tensor(p, device=cuda), t1


@pytest.mark.parametrize("method,field,precision", CASES)
@pytest.mark.parametrize("n", [1, 31, 33, 1000, 5000])
def test_compacting_forward_is_the_forward(gslib, cuda, method, field, precision, n):
    from gradsolve_b200 import engine
    from gradsolve_b200.fields import field_spec
    spec = field_spec(field)
    y0, p, t1 = _batch(field, n, cuda)
    t1v = t1 * torch.rand(n, device=cuda, dtype=torch.float64)
    t1v[0] = 0.0  # no step at all
    for end, max_steps, cap in ((None, 20000, 4096), (t1v, 20000, 4096), (None, 37, 4096),
                                (None, 20000, 20)):
        kw = dict(t0=0.0, t1=t1, rtol=1e-6, atol=1e-9, dt0=None, max_steps=max_steps,
                  checkpoint=3, budget_bytes=1 << 40, precision=precision, schedule="static")
        a = engine._forward_one(method, spec, y0, p, end, None, cap, None, kw)
        b = engine._forward_one(method, spec, y0, p, end, None, cap, None, kw, compact=True)
        for u, v in ((a.y_final, b.y_final), (a.n_acc, b.n_acc), (a.n_rej, b.n_rej),
                     (a.status, b.status), (a.padded_dts(), b.padded_dts())):
            assert torch.equal(u, v), (end is None, max_steps, cap)
        if cap == 4096 and max_steps > 37:  # the checkpoints too, through the reverse pass
            ybar = torch.ones_like(a.y_final)
            for u, v in zip(engine.adjoint(a, p, ybar, precision=precision),
                            engine.adjoint(b, p, ybar, precision=precision)):
                assert torch.equal(u, v)


def test_compacting_forward_refuses(gslib, cuda):
    import ctypes
    from gradsolve_b200.fields import field_spec

    lib = gslib.lib()

    def call(field, dim, precision, bytes_):
        y0 = torch.rand(4, dim, device=cuda, dtype=torch.float64)
        p = torch.ones(4, 1, device=cuda, dtype=torch.float64)
        buf = torch.zeros(1 << 16, device=cuda, dtype=torch.float64)
        ints = torch.zeros(3, 4, device=cuda, dtype=torch.int32)
        ptr = lambda x: ctypes.c_void_p(x.data_ptr())
        return lib.gs_fwd_record_compact(
            0, field_spec(field).code, precision, 4, ptr(y0), ptr(p), 0.0, None, 0.1, 1e-6, 1e-9,
            -1.0, 100, 64, 2, ptr(buf), ptr(buf[1 << 14:]), ptr(torch.empty_like(y0)),
            ptr(ints[0]), ptr(ints[1]), ptr(ints[2]), ptr(buf[1 << 15:]), bytes_, None)

    assert lib.gs_fwd_compact_bytes(0, field_spec("lorenz96_8").code, 0, 4) == 0
    assert call("lorenz96_8", 8, 0, 1 << 17) != 0      # states of more than 4 components
    assert call("lorenz", 3, 2, 1 << 17) != 0          # float32
    assert call("lorenz", 3, 0, 256) != 0              # scratch too small
    torch.cuda.synchronize()
