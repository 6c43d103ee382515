"""The Newton solves of the learned start and the harvest (stage 2 cut before the solve): with the harvest,
and with a network whose guess is the plain start, every bit and every count of a plain step."""
import numpy as np
import pytest

from imex_sflow2d_v2_b200 import configs
from imex_sflow2d_v2_b200.solver import ImexMLP, ImexSolver
from test_gpu_stage2_dense import _partly_wet, _wet

pytestmark = pytest.mark.gpu


def _zero_network():
    """Guesses q_si: all outputs 0, unit normalisation."""
    net = ImexMLP(seed=1)
    net.set_params(np.zeros_like(net.params()))
    net.set_norm(np.zeros(12), np.ones(12), np.zeros(2), np.ones(2))
    return net


def _run(p, st, q, mode, steps=3):
    g = ImexSolver(p, st)
    net = _zero_network() if mode == "network" else None
    if net is not None:
        g.set_warmstart(net)
    if mode == "harvest":
        g.harvest_start(capacity=1 << 18, stride=3)
    g.set_state(q, 0.0)
    g.set_clock(0.0, 1e-2)
    rec = []
    for _ in range(steps):
        g.advance(1)
        s = g.stats()
        rec.append((s.newton_cells, s.newton_iters, s.lnsrch_trials, list(s.newton_hist), s.error_mask,
                    s.warm_fallback_cells))
    out = g.get_state(), rec
    g.close()
    if net is not None:
        net.close()
    return out


@pytest.mark.parametrize("ns,rheology", [(1, 1), (2, 6), (3, 1), (4, 6)])
@pytest.mark.parametrize("nx,ny,kind", [(12, 11, "disk"), (43, 97, "above_half"), (301, 257, "stripes")])
def test_cut_solve_equals_plain_step(ns, rheology, nx, ny, kind):
    p, st, q = _partly_wet(ns, nx, ny, _wet(nx, ny, kind), rheology)
    q0, r0 = _run(p, st, q, "plain")
    for mode in ("harvest", "network"):
        q1, r1 = _run(p, st, q, mode)
        np.testing.assert_array_equal(q0, q1, err_msg=mode)
        assert r0 == r1, mode


def test_cut_solve_costs_like_the_plain_one():
    """On 512 x 512 wet cells the cut stage 2 took 1.23 times the plain one while its iterations ran lane by
    lane; the planes between its kernels alone cost a few percent."""
    p, st, q = configs.fractal_inlet(n=512, initial_layer=2.0)
    ms = {}
    for mode in ("plain", "harvest"):
        g = ImexSolver(p, st)
        if mode == "harvest":
            g.harvest_start(capacity=1 << 18, stride=8)
        g.set_state(q, 0.0)
        g.set_clock(0.0, 1e-2)
        g.advance(3)
        g.profile(True)
        part = []
        for _ in range(9):
            g.advance(1)
            part.append(sum(v[0] for k, v in g.kernel_times().items() if k.startswith("stage2")))
        ms[mode] = float(np.median(part))
        g.close()
    assert ms["harvest"] < 1.12 * ms["plain"], ms
