"""The contracted build takes the same short paths as the exact one.  The Newton solve's shared evaluation
holds where sums equal one of their terms; a cell for which a contracted product breaks such an equality
goes to the list of large steps, whose kernel time shows how many did (nine times the exact build's
before the products were rounded by themselves)."""
import numpy as np
import pytest

from imex_sflow2d_v2_b200 import configs
from imex_sflow2d_v2_b200.solver import ImexSolver

pytestmark = pytest.mark.gpu


def test_contracted_build_lists_no_more_cells():
    p, st, q = configs.fractal_inlet(n=1024, initial_layer=2.0)
    ms = {}
    for fast in (False, True):
        g = ImexSolver(p, st, fast=fast)
        g.set_state(q, 0.0)
        g.set_clock(0.0, 1e-2)
        g.advance(3)
        g.profile(True)
        part = []
        for _ in range(7):
            g.advance(1)
            part.append(g.kernel_times()["stage2_iter"][0])
        assert g.stats().solve_cells >= 1 << 18
        ms[fast] = float(np.median(part))
        g.close()
    assert 0.0 < ms[True] < 3.0 * ms[False], ms
