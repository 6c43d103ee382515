"""A buffer that cannot be allocated is an error of that call alone: the harvest is off afterwards (it must not
write to the buffers it gave back, nor from a captured step), and the steps that follow are the plain ones."""
import numpy as np
import pytest

import cases
from imex_sflow2d_v2_b200.solver import ImexError, ImexSolver

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("graph", [False, True])
def test_harvest_that_does_not_fit(graph):
    p, st, q = cases.fractal_small()
    a, b = ImexSolver(p, st), ImexSolver(p, st)
    for g in (a, b):
        g.set_state(q, 0.0)
        g.set_clock(0.0, 1e-2)
    a.harvest_start(capacity=1 << 14, stride=1)
    a.advance(2, use_graph=graph)
    assert a.harvest_data()[2] > 0
    with pytest.raises(ImexError):
        a.harvest_start(capacity=1 << 40, stride=1)        # 48 TB
    assert a.harvest_data()[2] == 0
    a.advance(2, use_graph=graph)                           # raises if the failure were reported again
    assert a.harvest_data()[2] == 0
    a.harvest_start(capacity=1 << 14, stride=1)
    a.advance(1, use_graph=graph)
    assert a.harvest_data()[2] == a.stats().newton_cells
    b.advance(5, use_graph=graph)
    np.testing.assert_array_equal(a.get_state(), b.get_state())
    a.close()
    b.close()


def test_capacity_beyond_any_memory_is_refused():
    p, st, q = cases.fractal_small()
    g = ImexSolver(p, st)
    with pytest.raises(ImexError):
        g.harvest_start(capacity=1 << 60, stride=1)
    g.close()
