"""Rosenbrock23 with W eliminated over its nonzero entries (gs_ros23.cuh kSparseW): constant
matrices with a sparse pattern, with and without steps where partial pivoting takes another row
(those run the pivoted elimination out of line), against the C oracle's dense elimination; and the
branch-free reciprocal the kernels' pivots and error norms use against the division."""
from __future__ import annotations

import ctypes

import numpy as np
import pytest
import torch

from conftest import ROOT

pytestmark = pytest.mark.gpu

D_ROS = 1.0 / (2.0 + np.sqrt(2.0))


def _matrix(kind, D):
    """Upper and lower bidiagonal parts and one corner entry: at most 5/8 of the entries after
    elimination for D >= 5."""
    A = np.diag(-np.linspace(1.0, 6.0, D))
    for i in range(D - 1):
        A[i, i + 1] = 0.3 + 0.1 * i
        A[i + 1, i] = 0.2 * (-1.0) ** i
    A[0, 2] = 0.25
    if kind == "pivots":  # d h |A| above the diagonal's 1 + d h |A| once h exceeds about 0.06
        A[D - 1, D - 2] = 60.0
    return A


def _exchanges(A, dts):
    """Steps (of all rows) whose partial pivoting takes a row other than the diagonal's."""
    k = 0
    for h in dts[dts > 0.0]:
        W = np.eye(A.shape[0]) - D_ROS * h * A
        for c in range(A.shape[0] - 1):
            if np.abs(W[c + 1:, c]).max() > abs(W[c, c]):
                k += 1
                break
            W[c + 1:] -= np.outer(W[c + 1:, c] / W[c, c], W[c])
    return k


@pytest.mark.parametrize("D", [5, 8])
@pytest.mark.parametrize("kind", ["diagonal", "pivots"])
def test_sparse_elimination_matches_dense(gslib, cuda, oracle, kind, D):
    import gradsolve_b200 as gsb
    from gradsolve_b200 import engine
    A = _matrix(kind, D)
    spec = gsb.register_linstiff(f"linstiff_sparse_{kind}_{D}", A)
    name = oracle.set_linstiff(A)
    rng = np.random.default_rng(D)
    y0 = rng.uniform(-1.0, 1.0, (3, D))
    p = np.zeros((3, 1))
    ref = oracle.record("rosenbrock23", name, y0, p, 0.0, 4.0, 1e-3, 1e-5)
    assert (ref["status"] == 0).all()
    k = _exchanges(A, ref["dts"])
    assert k > 0 if kind == "pivots" else k == 0
    y0_d = torch.tensor(y0, device=cuda)
    p_d = torch.zeros((3, spec.nparam), dtype=torch.float64, device=cuda)
    r = engine.forward_record("rosenbrock23", spec, y0_d, p_d, t0=0.0, t1=4.0, rtol=1e-3,
                              atol=1e-5, checkpoint=2)
    np.testing.assert_array_equal(r.n_acc.cpu().numpy(), ref["n_acc"])
    np.testing.assert_array_equal(r.n_rej.cpu().numpy(), ref["n_rej"])
    # the reference's own mesh: values to 1e-10, gradients to 1e-9 (relative, per row)
    ybar = 2.0 * ref["y_final"]
    gy, _ = oracle.replay_vjp("rosenbrock23", name, y0, p, ref["dts"], ybar)
    rowrel = lambda a, b: np.max(np.abs(a - b).max(1) / np.abs(b).max(1))  # noqa: E731
    for K in (1, 2, 7):
        m = engine.record_from_padded("rosenbrock23", spec, torch.tensor(ref["dts"], device=cuda),
                                      0.0, checkpoint=K)
        yf = engine.replay(m, y0_d, p_d)
        assert rowrel(yf.cpu().numpy(), ref["y_final"]) <= 1e-10
        for schedule in ("static", "refill"):
            got, _ = engine.adjoint(m, p_d, torch.tensor(ybar, device=cuda), schedule=schedule)
            assert rowrel(got.cpu().numpy(), gy) <= 1e-9, (K, schedule)


def test_reciprocal_matches_division(gslib, cuda):
    L = ctypes.CDLL(str(ROOT / "gradsolve_b200" / "libgsprobe.so"))
    rng = np.random.default_rng(0)
    tiny, huge = np.finfo(np.float64).tiny, np.finfo(np.float64).max
    x = np.concatenate([
        rng.uniform(0.5, 2.0, 200000), 10.0 ** rng.uniform(-300.0, 300.0, 200000),
        np.nextafter(1.0, [0.0, 2.0]), 2.0 ** np.arange(-1020.0, 1021.0),
        [1.0, 3.0, tiny, 2.0 * tiny]])
    edges = np.array([0.0, -0.0, np.inf, -np.inf, np.nan])
    x = np.concatenate([x, -x, edges])
    xd = torch.tensor(x, device=cuda)
    r, ref = torch.empty_like(xd), torch.empty_like(xd)
    P = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
    assert L.gs_probe_reciprocal(P(xd), ctypes.c_longlong(x.size), P(r), P(ref), None) == 0
    torch.cuda.synchronize()
    r, ref = r.cpu().numpy(), ref.cpu().numpy()
    # the series is truncated below 2^-58 and rounds three times: within 2 ulp
    n = x.size - edges.size
    assert (np.abs(r[:n] - ref[:n]) <= 2.0 * np.spacing(np.abs(ref[:n]))).all()
    np.testing.assert_array_equal(r[n:], ref[n:])


def test_reciprocal_at_the_ends_of_the_range(gslib, cuda):
    """The hardware's approximation flushes to zero: a subnormal operand gives infinity and one
    above 2^1022 zero, with its sign (the error norm divides there, test_tiny_scales).  It reads
    the operand's upper 32 bits, so just above 2^1022 it is still refined."""
    L = ctypes.CDLL(str(ROOT / "gradsolve_b200" / "libgsprobe.so"))
    x = np.array([5e-324, 1e-309, 2.2e-308, np.nextafter(np.finfo(np.float64).tiny, 0.0),
                  np.nextafter(2.0 ** 1022, np.inf), 1e308, np.finfo(np.float64).max])
    x = np.concatenate([x, -x])
    xd = torch.tensor(x, device=cuda)
    r, ref = torch.empty_like(xd), torch.empty_like(xd)
    P = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
    assert L.gs_probe_reciprocal(P(xd), ctypes.c_longlong(x.size), P(r), P(ref), None) == 0
    r, ref = r.cpu().numpy(), ref.cpu().numpy()
    edge = np.abs(x) == np.nextafter(2.0 ** 1022, np.inf)
    assert (np.abs(r[edge] - ref[edge]) <= 2.0 * np.spacing(np.abs(ref[edge]))).all()
    want = np.copysign(np.where(np.abs(x) < 1.0, np.inf, 0.0), x)
    np.testing.assert_array_equal(r[~edge], want[~edge])


@pytest.mark.parametrize("schedule", ["static", "refill"])
@pytest.mark.parametrize("method,field", [("tsit5", "linear_1"), ("tsit5", "linear_8"),
                                          ("tsit5", "linear_32"), ("rosenbrock23", "linear_1"),
                                          ("rosenbrock23", "linear_3")])
def test_tiny_scales(gslib, cuda, method, field, schedule):
    """Without an absolute tolerance a linear field's attempts do not depend on its state's size,
    subnormal scales of the error included (rtol 0.5: the route for scales above 2^1022)."""
    from gradsolve_b200 import engine
    from gradsolve_b200.fields import field_spec
    spec = field_spec(field)
    p = torch.zeros(3, max(spec.nparam, 1), dtype=torch.float64, device=cuda)
    t1v = None if schedule == "static" else torch.full((3,), 1.0, dtype=torch.float64,
                                                       device=cuda)
    for rtol in (1e-6, 0.5):
        y0 = torch.tensor([[1.0], [1e-303], [3e-304]], dtype=torch.float64,
                          device=cuda).repeat(1, spec.dim)
        r = engine.forward_record(method, spec, y0, p, t0=0.0, t1=1.0, t1v=t1v, rtol=rtol,
                                  atol=0.0, schedule=schedule)
        assert r.status.tolist() == [0, 0, 0], (rtol, r.status)
        assert r.n_acc.tolist() == [int(r.n_acc[0])] * 3 and \
            r.n_rej.tolist() == [int(r.n_rej[0])] * 3
        scaled = r.y_final / y0
        assert float((scaled / scaled[0] - 1.0).abs().max()) <= 1e-9


def test_two_warps_with_exchanged_pivots(gslib, cuda):
    """The two-warp reverse pass over a sparse W whose pivots do not hold on some steps: those run
    the pivoted elimination out of line in both warps."""
    import gradsolve_b200 as gsb
    from gradsolve_b200 import engine
    D = 8
    A = _matrix("pivots", D)
    spec = gsb.register_linstiff(f"linstiff_sparse_pivots_{D}", A)
    rng = np.random.default_rng(3)
    n = 70
    y0 = torch.tensor(rng.uniform(-1.0, 1.0, (n, D)), device=cuda)
    p = torch.zeros((n, spec.nparam), dtype=torch.float64, device=cuda)
    for K in (1, 2):
        r = engine.forward_record("rosenbrock23", spec, y0, p, t0=0.0, t1=4.0, rtol=1e-3,
                                  atol=1e-5, checkpoint=K)
        assert _exchanges(A, r.padded_dts().cpu().numpy()) > 0
        ybar = 2.0 * r.y_final
        ref = engine.adjoint(r, p, ybar, schedule="static")[0]
        got = engine._adjoint_split(r, engine.PAIRED, p, ybar, None, None, True, True, None)[0]
        # two float64 evaluation orders of the same sums, as in test_gpu_split.py
        rel = ((got - ref).abs().max(1).values / ref.abs().max(1).values).max()
        assert float(rel) <= 1e-10, K
