"""The capacity of a fresh record (engine.first_capacity): within its share of the memory budget,
never below the default or above max_steps, and what a closure passes on (CPU)."""
from __future__ import annotations

import pytest

from gradsolve_b200 import engine


@pytest.mark.parametrize("precision,word,row", [("float64", 8, 32), ("float32", 4, 16)])
@pytest.mark.parametrize("n", [1, 1000, 20_011, 1 << 20])
@pytest.mark.parametrize("K", [1, 2, 16])
def test_capacity_stays_in_its_share(n, K, precision, word, row):
    budget = 40 << 30
    cap = engine.first_capacity(n, 3, 50_000, K, precision, budget_bytes=budget)
    assert engine.DEFAULT_CAP0 <= cap <= 50_000
    if cap > engine.DEFAULT_CAP0:  # record chunks of 4 steps, cap // K + 2 checkpoint slots
        used = n * ((cap + 3) // 4 * 4 * word + (cap // K + 2) * row)
        assert used <= budget // engine.CAP_SHARE + n * 4 * (word + row)
    if n <= 1000:
        assert cap == 50_000  # the whole of max_steps fits: nothing can overflow


@pytest.mark.parametrize("max_steps", [1, 7, 1024, 1025, 4096])
def test_capacity_never_exceeds_max_steps(max_steps):
    for budget in (0, 1 << 40):
        cap = engine.first_capacity(64, 3, max_steps, 2, "float64", budget_bytes=budget)
        assert min(engine.DEFAULT_CAP0, max_steps) <= cap <= max_steps
    assert engine.first_capacity(0, 3, max_steps, 2, "float64", budget_bytes=1 << 40) == \
        min(engine.DEFAULT_CAP0, max_steps)
