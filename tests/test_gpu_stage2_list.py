"""Steps of 262144 solve cells and more that solve half of the grid: stage 2 leaves the cells its lean Jacobian
does not cover, and a warp's last ones, to a list.  Single grids, row bands of host-state steps and
ensembles, bit for bit against the oracle (or the same step taken otherwise)."""
import numpy as np
import pytest

import cases
from imex_sflow2d_v2_b200 import configs
from imex_sflow2d_v2_b200.solver import ImexEnsemble, ImexSolver
from oracle import Oracle

pytestmark = pytest.mark.gpu

LIST_MIN = 1 << 18


def _mixed(p, q, seed):
    """Half of the cells next to rest, the others moving."""
    rng = np.random.default_rng(seed)
    q = np.array(q, order="F")
    slow = rng.random(q[0].shape) < 0.5
    for i in (1, 2):
        creep = 10.0 ** rng.uniform(-200, -3, q[0].shape) * (q[0] > 0.0)
        q[i] = np.where(slow, creep, q[0] * rng.normal(0.0, 5.0, q[0].shape))
    return q


def _tilted(n, rheology):
    """A wet slab over the whole rough incline, slope and curvature corrections on."""
    p, st, _ = cases.sloped(n=n, rheology=rheology)
    rng = np.random.default_rng(4)
    qp = np.zeros((8, n, n))
    qp[0] = 1.0 + 0.3 * rng.random((n, n))
    qp[6], qp[7] = rng.normal(1.0, 2.0, (2, n, n))
    qp[1], qp[2] = qp[0] * qp[6], qp[0] * qp[7]
    qp[3] = 600.0 + 50.0 * rng.random((n, n))
    qp[4], qp[5] = 0.01 * qp[0], 0.005 * qp[0]
    return p, st, configs.qp_to_qc_grid(p, qp)


@pytest.mark.parametrize("kind", ["n1_voellmy", "n2_quadratic", "n3_voellmy", "n4_quadratic", "tilted_voellmy",
                                  "tilted_quadratic"])
def test_list_form_bitexact(kind):
    rheology = 1 if kind.endswith("voellmy") else 6
    if kind.startswith("tilted"):
        p, st, q = _tilted(541, rheology)
    else:
        p, st, q = cases.dambreak_ns(int(kind[1]), nx=643, ny=517, rheology=rheology)
        q = _mixed(p, q, 6)
    o, g = Oracle(p, st, threads=8), ImexSolver(p, st)
    for s in (o, g):
        s.set_state(q, 0.0)
    t = 0.0
    for step in range(3):
        n = o.check_solve(t)
        assert n == g.check_solve(t) and n >= LIST_MIN and 2 * n >= p.nx * p.ny
        dt = o.timestep()
        assert dt == g.timestep()
        o.rk_step(t, dt)
        g.imex_RK_solver(t, dt)
        o.post_step()
        so, sg = o.stats(), g.stats()
        np.testing.assert_array_equal(o.get_state(), g.get_state(), err_msg="step %d" % step)
        assert (so.newton_cells, so.newton_iters, so.lnsrch_trials, list(so.newton_hist), so.error_mask) == \
            (sg.newton_cells, sg.newton_iters, sg.lnsrch_trials, list(sg.newton_hist), sg.error_mask)
        t += dt
    g.close()


def test_list_in_row_bands():
    p, st, q = cases.dambreak_ns(3, nx=643, ny=517, rheology=1)
    q = _mixed(p, q, 8)
    a, b = ImexSolver(p, st), ImexSolver(p, st)
    for g in (a, b):
        g.set_clock(0.0, 1e-2)
    qa = qb = q.ravel(order="F").copy()
    t = 0.0
    for step in range(3):
        a.set_state(qa, t)
        a.advance(1)
        qa = a.get_state(out=np.empty(q.size))
        _, qb, tb = b.advance_host(qb, t, out=np.empty(q.size))
        sa, sb = a.stats(), b.stats()
        assert sa.t == tb and sa.solve_cells == sb.solve_cells >= LIST_MIN
        np.testing.assert_array_equal(qa, qb, err_msg="step %d" % step)
        assert (sa.newton_iters, sa.lnsrch_trials, list(sa.newton_hist), sa.error_mask, sa.first_error_code) == \
            (sb.newton_iters, sb.lnsrch_trials, list(sb.newton_hist), sb.error_mask, sb.first_error_code)
        t = tb
    a.close()
    b.close()


@pytest.mark.parametrize("ns,rheology", [(1, 6), (3, 1)])
def test_list_in_an_ensemble(ns, rheology):
    mem = []
    for m, (nx, ny) in enumerate(((331, 402), (290, 333), (257, 311))):      # 310 thousand cells together
        p, st, q = cases.dambreak_ns(ns, nx=nx, ny=ny, rheology=rheology)
        mem.append((p, st, _mixed(p, q, m)))
    assert sum(p.nx * p.ny for p, _, _ in mem) >= LIST_MIN
    ens = ImexEnsemble([(p, st) for p, st, _ in mem])
    for m, (p, st, q) in enumerate(mem):
        ens.member(m).set_state(q, 0.0)
        ens.member(m).set_clock(0.0, 1e-2)
    ens.advance(8)                              # six steps try the tile shapes
    assert ens.tile_shape()[0] != (0, 0)        # the batched kernels
    for m, (p, st, q) in enumerate(mem):
        o = Oracle(p, st, threads=8)
        o.set_state(q, 0.0)
        o.set_clock(0.0, 1e-2)
        o.advance(8)
        so, sg = o.stats(), ens.member(m).stats()
        np.testing.assert_array_equal(o.get_state(), ens.member(m).get_state(), err_msg="member %d" % m)
        assert (so.newton_cells, so.newton_iters, so.lnsrch_trials) == \
            (sg.newton_cells, sg.newton_iters, sg.lnsrch_trials)
    ens.close()
