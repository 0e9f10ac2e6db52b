"""Which batches run two warps per 32 trajectories: those that are resident at once with room to
spare, by the kernel's own occupancy (gs_adjoint_paired_room); a dense W of 8 components leaves one
block per SM, a sparse one and Tsit5 several."""
from __future__ import annotations

import ctypes

import numpy as np
import pytest
import torch

from conftest import load_golden

pytestmark = pytest.mark.gpu


def test_room(gslib, cuda):
    from gradsolve_b200 import engine
    from gradsolve_b200.fields import field_spec
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    for method, field, most in (("tsit5", "lorenz", 1 << 14), ("tsit5", "lorenz96_8", 1 << 13),
                                ("rosenbrock23", "robertson", 1 << 14),
                                ("rosenbrock23", "hires", 1 << 13)):
        spec = field_spec(field)
        for K in (1, 2):
            room = engine._pair_room(method, spec, K)
            assert room % (32 * sms) == 0 and 8 * most <= 7 * room, (method, field, K)
            assert engine._pairs(method, spec, most, K)
            assert not engine._pairs(method, spec, most + 1, K)
        assert not engine._pairs(method, spec, 64, 3)
    # states the pass is not built for, and intervals that are none
    assert engine._pair_room("tsit5", field_spec("lorenz96_32"), 2) == 0
    room = ctypes.c_longlong(7)
    L = gslib.lib()
    code = field_spec("lorenz").code
    assert L.gs_adjoint_paired_room(0, code, 0, ctypes.addressof(room)) != 0
    assert L.gs_adjoint_paired_room(0, code, 65, ctypes.addressof(room)) != 0
    assert L.gs_adjoint_paired_room(0, code, 2, None) != 0


def test_dense_w(gslib, cuda, monkeypatch):
    import gradsolve_b200 as gsb
    from gradsolve_b200 import engine
    A = load_golden("linstiff_8")["A"]
    assert (A != 0.0).sum() * 8 > A.size * 5  # its W is not eliminated over a sparse pattern
    spec = gsb.register_linstiff(f"linstiff_test_{A.shape[0]}", A)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    assert engine._pair_room("rosenbrock23", spec, 1) == 0
    room = engine._pair_room("rosenbrock23", spec, 2)
    assert room == 32 * sms  # one block of 128,000 bytes per SM
    calls, real = [], engine._adjoint_split
    monkeypatch.setattr(engine, "_adjoint_split",
                        lambda r, lanes, *a: (calls.append(lanes), real(r, lanes, *a))[1])
    rng = np.random.default_rng(0)
    for n, paired in ((64, True), (7 * room // 8, True), (7 * room // 8 + 1, False),
                      (8192, False)):
        y0 = torch.tensor(rng.uniform(-1, 1, (n, 8)), device=cuda)
        p = torch.zeros((n, spec.nparam), dtype=torch.float64, device=cuda)
        r = engine.forward_record("rosenbrock23", spec, y0, p, t0=0.0, t1=0.1, rtol=1e-4,
                                  atol=1e-7, checkpoint=2)
        ybar = torch.ones_like(y0)
        del calls[:]
        got = engine.adjoint(r, p, ybar)[0]
        assert calls == ([engine.PAIRED] if paired else []), n
        ref = engine.adjoint(r, p, ybar, schedule="static")[0]
        # two evaluations of the same expressions, as in test_gpu_split.py
        assert float(((got - ref).abs().max(1).values / ref.abs().max(1).values).max()) <= 1e-10
