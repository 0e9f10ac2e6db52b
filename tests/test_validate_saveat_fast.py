"""validate_saveat's single pass accepts and refuses what the checks one by one do (CPU)."""
from __future__ import annotations

import numpy as np
import pytest

from gradsolve_b200 import api


def _rules(ts, t0, t1, t1v):
    """The checks as stated: finite, sorted, first >= t0, last <= its end time."""
    hi = t1v if t1v is not None else t1
    return (np.isfinite(ts).all() and not (np.diff(ts, axis=-1) < 0).any()
            and not (ts[..., 0] < t0).any()
            and not (ts[..., -1] > (hi if ts.ndim == 2 else np.min(hi))).any())


@pytest.mark.parametrize("seed", range(8))
def test_single_pass_equals_the_rules(seed):
    rng = np.random.default_rng(seed)
    seen = set()
    for _ in range(200):
        n, k = int(rng.integers(1, 4)), int(rng.integers(1, 5))
        ts = np.sort(rng.uniform(0.0, 1.0, (n, k)), axis=-1)
        t1v = np.ones(n) if rng.random() < 0.5 else None
        if t1v is not None and rng.random() < 0.2:
            t1v[rng.integers(n)] = np.inf
        if rng.random() < 0.6:
            ts[rng.integers(n), rng.integers(k)] = rng.choice([np.nan, np.inf, -np.inf, -0.5, 1.5])
        ts = ts[0] if rng.random() < 0.3 else ts
        ok = _rules(ts, 0.0, 1.0, t1v)
        seen.add(ok)
        if ok:
            assert api.validate_saveat(ts, 0.0, 1.0, t1v) is not None
        else:
            with pytest.raises(ValueError):
                api.validate_saveat(ts, 0.0, 1.0, t1v)
    assert seen == {True, False}
