"""Edges of the kernels' shortened arithmetic, bit for bit against the oracle
or IEEE arithmetic (imex_gpu_point_eval): inputs on both sides of each range
that decides between a short path and the general one."""
import numpy as np
import pytest

from imex_sflow2d_v2_b200.solver import point_eval
from oracle import ipow_n

pytestmark = pytest.mark.gpu


def _around(values, steps=200):
    """Each value with its `steps` nearest doubles on either side."""
    v = np.abs(np.asarray(values, np.float64)).view(np.int64)
    return (v[:, None] + np.arange(-steps, steps + 1)[None, :]).ravel().view(np.float64)


@pytest.mark.parametrize("y", [0.5, 0.687, 1.5, 2.4, 4.65, 5.0, np.nextafter(5.0, 6.0), 1e-300])
def test_ipow_common_range_edges(y):
    rng = np.random.default_rng(3)
    # the ends of the common range, the window around 1 that it leaves out,
    # every table row's ends in the binades beside 1 and at the far ones
    edges = [2.0 ** -200, 2.0 ** 200, 1.0 - 2.0 ** -8, 1.0 + 2.0 ** -7, 1.0]
    rows = (1.0 + np.arange(129) / 128.0)[:, None] * 2.0 ** np.array([-199, -30, -2, -1, 0, 1, 9, 198])
    x = np.concatenate([_around(edges), _around(rows.ravel(), 3),
                        np.exp(rng.uniform(np.log(1e-60), np.log(1e60), 200000))])
    g, o = point_eval("ipow", x, np.full(x.size, y)), ipow_n(x, np.full(x.size, y))
    bad = np.flatnonzero(g.view(np.uint64) != o.view(np.uint64))
    assert bad.size == 0, [(x[i], y, g[i], o[i]) for i in bad[:5]]


def _edge_state(kind):
    """Small runs whose faces and interfaces leave the flux kernel's short
    paths: see each branch."""
    import cases
    from imex_sflow2d_v2_b200 import configs
    if kind == "tiny_momentum":        # quotients below the exact-remainder range
        p, st, q = cases.dambreak_ns(3, nx=45, ny=19)
        rng = np.random.default_rng(1)
        q = np.array(q)
        q[1] = 10.0 ** rng.uniform(-320, -150, q[1].shape) * rng.choice([-1.0, 0.0, 1.0], q[1].shape)
        q[2] = 10.0 ** rng.uniform(-320, -150, q[2].shape)
    elif kind == "caps":               # almost all solid: face and interface flux caps
        p, st, q = cases.dambreak_ns(2, nx=70, ny=33)
        rng = np.random.default_rng(2)
        q = np.array(q)
        share = 1.0 - 10.0 ** rng.uniform(-17, -1, q[0].shape)
        q[4], q[5] = 0.6 * share * q[0], 0.4 * share * q[0]
        q[1] = q[0] * rng.normal(0.0, 3.0, q[0].shape)
        q[2] = q[0] * rng.normal(0.0, 3.0, q[0].shape)
        q[3] = q[0] * (1617.0 * 400.0 + 20.0)
    elif kind == "mixed_limiters":     # each variable its own limiter, unequal rounded spacings
        p, st, q = cases.dambreak_ns(3, nx=67, ny=41, dx=0.05)
        p.x0, p.y0, p.theta = 123.4, -7.7, 1.3
        for i in range(9):
            p.limiter[i] = i % 8
    elif kind == "inlet_corner":       # inlet ring two cells from a corner, across tile edges
        p, st, q = configs.radial_current(nx=41, ny=37, dx=2.0, r_source=4.6, mfr=2e5)
        st = dict(st)
        xs = configs.grid(p)[1]
        st.update(configs.init_radial_source(p, xs[5] + 0.6, xs[8] + 0.3, 4.6))
    else:                              # non-finite and huge cells
        p, st, q = cases.dambreak_ns(1, nx=64, ny=24)
        q = np.array(q)
        q[1, 20, 9], q[3, 40, 8], q[0, 33, 15], q[2, 10, 3] = np.inf, np.nan, 1e200, 1e190
    return p, st, q


@pytest.mark.parametrize("kind", ["tiny_momentum", "caps", "mixed_limiters", "inlet_corner", "non_finite"])
def test_flux_edges_bitexact(kind):
    from imex_sflow2d_v2_b200.solver import ImexSolver
    from oracle import Oracle
    p, st, q = _edge_state(kind)
    o, g = Oracle(p, st, threads=4), ImexSolver(p, st)
    for s in (o, g):
        s.set_state(q, 0.0)
    t = 0.0
    for step in range(6):
        assert o.check_solve(t) == g.check_solve(t), step
        dto, dtg = o.timestep(), g.timestep()
        assert dto == dtg or (np.isnan(dto) and np.isnan(dtg)), (step, dto, dtg)
        o.rk_step(t, dto)
        g.imex_RK_solver(t, dto)
        o.post_step()
        np.testing.assert_array_equal(o.get_state(), g.get_state(), err_msg="%s step %d" % (kind, step))
        t += dto


@pytest.mark.parametrize("rheology", [1, 6])
@pytest.mark.parametrize("kind", ["still", "creeping", "small_loads", "ambient", "no_energy", "tilted"])
def test_newton_edges_bitexact(kind, rheology):
    """States at and beyond the edges of the Newton solve's shared
    evaluation: cells at rest, speeds whose squares underflow, components below the
    scaling floor of 1e-3 (where (q/q_org)*q_org need not be q), densities next to
    the ambient one, no kinetic energy in T, slope correction."""
    import cases
    from imex_sflow2d_v2_b200 import configs
    from imex_sflow2d_v2_b200.solver import ImexSolver
    from oracle import Oracle
    p, st, q = cases.sloped(n=40, rheology=rheology) if kind == "tilted" else \
        cases.dambreak_ns(3, nx=40, ny=21, rheology=rheology)
    q = np.array(q)
    rng = np.random.default_rng(5)
    shape = q[0].shape
    wet = q[0] > 0.0
    if kind == "still":
        q[1:3] = 0.0
        q[1, ::3] = 1e-9
    elif kind == "creeping":
        q[1] = np.where(wet, 10.0 ** rng.uniform(-200, -3, shape), 0.0)
        q[2] = np.where(wet, -10.0 ** rng.uniform(-200, -3, shape), 0.0)
    elif kind == "small_loads":
        f = 10.0 ** rng.uniform(-9, 0, shape)
        q = q * f
        q[1], q[2] = q[0] * rng.normal(0.0, 2.0, shape), q[0] * rng.normal(0.0, 2.0, shape)
    elif kind == "ambient":
        q[4:] *= 10.0 ** rng.uniform(-14, 0, shape)
        q[1] = q[0] * rng.normal(0.0, 1.0, shape)
    elif kind == "no_energy":
        p.energy_flag = 0
        q[1] = q[0] * rng.normal(0.0, 5.0, shape)
    o, g = Oracle(p, st, threads=4), ImexSolver(p, st)
    for s in (o, g):
        s.set_state(q, 0.0)
    t = 0.0
    for step in range(5):
        o.check_solve(t)
        g.check_solve(t)
        dt = o.timestep()
        assert dt == g.timestep()
        o.rk_step(t, dt)
        g.imex_RK_solver(t, dt)
        o.post_step()
        so, sg = o.stats(), g.stats()
        np.testing.assert_array_equal(o.get_state(), g.get_state(), err_msg="%s step %d" % (kind, step))
        assert (so.newton_cells, so.newton_iters, so.lnsrch_trials, list(so.newton_hist)) == \
            (sg.newton_cells, sg.newton_iters, sg.lnsrch_trials, list(sg.newton_hist))
        t += dt
