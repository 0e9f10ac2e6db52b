"""Which fresh batches run the compacting forward (engine._compacts, CPU): the sizes from which its
further launches cost less than idle lanes, for both methods."""
from __future__ import annotations

import pytest

from gradsolve_b200 import engine
from gradsolve_b200.fields import field_spec


@pytest.mark.parametrize("method,field,least", [("tsit5", "lv", 1 << 18),
                                                ("rosenbrock23", "vdp", 1 << 17),
                                                ("rosenbrock23", "robertson", 1 << 17)])
def test_sizes(method, field, least):
    spec = field_spec(field)
    for n in (1, least // 2, least - 1, least, 4 * least):
        got = engine._compacts(method, spec, n, "float64", "auto", None, None)
        assert got == (n >= least), n
    assert not engine._compacts(method, spec, least, "float64", "static", None, None)
    assert not engine._compacts(method, spec, least, "float32", "auto", None, None)
