"""Harvested training pairs belong to the solves of the harvested steps: cells that an earlier step
solved, or left half solved to the list of large steps, and that are dry now give none."""
import numpy as np
import pytest

from imex_sflow2d_v2_b200 import configs
from imex_sflow2d_v2_b200.solver import ImexSolver

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [64, 640])   # below and above the 262144 solve cells that use the list
@pytest.mark.parametrize("harvest_first", [False, True])
def test_pairs_after_a_wetter_state(n, harvest_first):
    p, st, q = configs.fractal_inlet(n=n, relief=2.0 * n, r_source=25.0, mfr=2e5, initial_layer=2.0)
    g = ImexSolver(p, st)
    g.set_state(q, 0.0)
    g.set_clock(0.0, 1e-2)
    if harvest_first:                      # the earlier solves from the harvest's own passes
        g.harvest_start(capacity=1 << 20, stride=1)
    g.advance(2)
    dry = np.zeros_like(q)
    dry[:, : n // 4, : n // 4] = q[:, : n // 4, : n // 4]
    g.set_state(dry, 0.0)
    g.set_clock(0.0, 1e-2)
    g.harvest_start(capacity=1 << 20, stride=1)
    cells = 0
    for _ in range(3):
        g.advance(1)
        cells += g.stats().newton_cells
    assert 0 < cells < 3 * n * n // 8
    assert g.harvest_data()[2] == cells
    g.close()
