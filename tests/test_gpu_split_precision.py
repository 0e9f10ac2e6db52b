"""The split reverse pass of stiff trajectories against 80-bit arithmetic on the same float64 states:
no further from it than one thread per trajectory (Rosenbrock23, Van der Pol, mu = 10 to 100; some
thousand steps, most of them in the jumps, where the columns of a part are nearly parallel)."""
from __future__ import annotations

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

LD = np.longdouble
D_ROS = 1.0 / (2.0 + np.sqrt(2.0))


def _rhs(y, p):
    return np.stack((y[1], p * ((1 - y[0] ** 2) * y[1] - y[0])))


def _vjp(y, p, w):
    return (np.stack((p * (-2 * y[0] * y[1] - 1) * w[1], w[0] + p * (1 - y[0] ** 2) * w[1])),
            ((1 - y[0] ** 2) * y[1] - y[0]) * w[1])


def _solve(W, b):
    det = W[0, 0] * W[1, 1] - W[0, 1] * W[1, 0]
    return np.stack(((W[1, 1] * b[0] - W[0, 1] * b[1]) / det,
                     (W[0, 0] * b[1] - W[1, 0] * b[0]) / det))


def _step_vjp(y, p, h, lam):
    """(dy'/dy)^T lam and (dy'/dp)^T lam of one Rosenbrock23 step, for all trajectories at once."""
    d = y.dtype.type(D_ROS)
    one = np.ones_like(h)
    J = np.array([[0 * h, one], [p * (-2 * y[0] * y[1] - 1), p * (1 - y[0] ** 2)]])
    W = -d * h * J
    W[0, 0] += 1
    W[1, 1] += 1
    k1 = _solve(W, _rhs(y, p))
    s1 = y + h / 2 * k1
    k2p = _solve(W, _rhs(s1, p) - k1)
    WT = np.swapaxes(W, 0, 1)
    k2b = h * lam
    r2 = _solve(WT, k2b)
    k1b = k2b - r2
    s, gp = _vjp(s1, p, r2)
    yb = lam + s
    r1 = _solve(WT, k1b + h / 2 * s)
    G = d * h * (r2[:, None] * k2p[None] + r1[:, None] * k1[None])
    s, g = _vjp(y, p, r1)
    yb, gp = yb + s, gp + g
    yb = yb + np.stack((-2 * p * (G[1, 0] * y[1] + G[1, 1] * y[0]), -2 * p * G[1, 0] * y[0]))
    return yb, gp + G[1, 0] * (-2 * y[0] * y[1] - 1) + G[1, 1] * (1 - y[0] ** 2)


def test_split_error_is_one_threads(gslib, cuda):
    from gradsolve_b200 import engine
    from gradsolve_b200.fields import field_spec
    n, steps = 48, 12000
    rng = np.random.default_rng(4)
    y0 = torch.tensor(rng.uniform(-2, 2, (n, 2)), device=cuda)
    p = torch.tensor(10 ** rng.uniform(1, 2, (n, 1)), device=cuda)
    r = engine.forward_record("rosenbrock23", field_spec("vdp"), y0, p, t0=0.0, t1=10.0,
                              rtol=1e-6, atol=1e-9, cap0=steps, max_steps=steps, checkpoint=1)
    assert int(r.status.max()) == 0
    N = int(r.n_acc.max())
    assert N > 4000
    states = r.ckpt[:(steps + 1) * n * 4].view(steps + 1, n, 4)[:N, :, :2].cpu().numpy()
    dts = r.padded_dts().cpu().numpy().T
    ybar = 2.0 * r.y_final
    lam, gp = ybar.cpu().numpy().T.astype(LD), np.zeros(n, LD)
    q = p[:, 0].cpu().numpy().astype(LD)
    for i in range(N - 1, -1, -1):
        a, b = _step_vjp(states[i].T.astype(LD), q, dts[i].astype(LD), lam)
        live = dts[i] != 0.0
        lam, gp = np.where(live, a, lam), np.where(live, gp + b, gp)

    def error(g):
        y = np.abs(g[0].cpu().numpy().T - lam).max(0) / np.abs(lam).max(0)
        return np.maximum(y, np.abs(g[1].cpu().numpy()[:, 0] - gp) / np.abs(gp))

    one = error(engine.adjoint(r, p, ybar, schedule="static"))
    # rounding of two evaluation orders: a factor in either direction; the split's columns alone
    # were 10 times further off at the median and 20 times at most
    for lanes in (2, 8, 32):
        split = error(engine._adjoint_split(r, lanes, p, ybar, None, None, True, True, None))
        assert np.median(split) <= 4 * np.median(one), lanes
        assert split.max() <= 6 * one.max(), lanes
    # with dense output, whose last time is the end: the same cotangent, by the saved states' pass
    ts = torch.tensor([10.0], device=cuda, dtype=torch.float64)
    split = error(engine._adjoint_split(r, 8, p, None, ts, ybar[:, None].contiguous(), True, True,
                                        None))
    assert np.median(split) <= 4 * np.median(one) and split.max() <= 6 * one.max()
