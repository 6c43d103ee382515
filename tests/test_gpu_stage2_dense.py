"""Stage 2 over the list of solve cells (steps of grids of 75776 cells or more that solve less than half
of them) against the oracle, and its cost where every grid block holds a few solve cells."""
import numpy as np
import pytest

import cases
from imex_sflow2d_v2_b200.solver import ImexSolver
from oracle import Oracle

pytestmark = pytest.mark.gpu


def _partly_wet(ns, nx, ny, wet, rheology=1):
    """Moving water and solids where `wet`, dry elsewhere (mostly slow cells, some next to rest)."""
    p, st, q = cases.dambreak_ns(ns, nx=nx, ny=ny, rheology=rheology)
    q = np.array(q, order="F")
    rng = np.random.default_rng(9)
    speed = rng.normal(0.0, 2.0, (2,) + q[0].shape) * np.where(rng.random(q[0].shape) < 0.1, 1e-12, 1.0)
    q[1], q[2] = q[0] * speed[0], q[0] * speed[1]
    q *= wet
    return p, st, q


def _wet(nx, ny, kind):
    x, y = np.arange(nx)[:, None] / nx, np.arange(ny)[None, :] / ny
    if kind == "stripes":                       # a few cells of every grid block
        return np.broadcast_to((np.arange(nx) % 61 < 3)[:, None], (nx, ny)).astype(float)
    if kind == "below_half":
        return ((x < 0.46) & (y > -1)).astype(float)
    if kind == "above_half":
        return ((x < 0.52) & (y > -1)).astype(float)
    return ((x - 0.4) ** 2 + (y - 0.5) ** 2 < 0.04).astype(float)


def _lockstep(p, st, q, steps):
    o, g = Oracle(p, st, threads=8), ImexSolver(p, st)
    for s in (o, g):
        s.set_state(q, 0.0)
    t = 0.0
    for step in range(steps):
        n = o.check_solve(t)
        assert n == g.check_solve(t)
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


@pytest.mark.parametrize("ns,rheology", [(1, 6), (2, 1), (3, 6), (4, 1)])
@pytest.mark.parametrize("kind", ["stripes", "disk", "below_half", "above_half"])
def test_partly_wet_grid_bitexact(kind, ns, rheology):
    nx, ny = 301, 257                           # 77357 cells, ragged tiles and blocks, padded rows
    _lockstep(*_partly_wet(ns, nx, ny, _wet(nx, ny, kind), rheology), 3)


@pytest.mark.parametrize("nx,ny", [(275, 275), (296, 256), (75776, 1), (9, 8500)])
def test_grid_sizes_at_the_limit_bitexact(nx, ny):
    p, st, q = _partly_wet(2, nx, ny, _wet(nx, ny, "disk" if nx < 1000 else "stripes"))
    _lockstep(p, st, q, 2)


def test_graph_across_the_half():
    """One captured step replayed on states of which less and more than half is solved."""
    nx, ny = 320, 270
    p, st, _ = _partly_wet(2, nx, ny, _wet(nx, ny, "disk"))
    g = ImexSolver(p, st)
    for kind in ("disk", "above_half", "stripes"):
        q = _partly_wet(2, nx, ny, _wet(nx, ny, kind))[2]
        o = Oracle(p, st, threads=8)        # set_state leaves values of earlier steps in cells it never solves
        for s in (g, o):
            s.set_state(q, 0.0)
            s.set_clock(0.0, 1e-2)
        g.advance(4, use_graph=True)
        o.advance(4)
        np.testing.assert_array_equal(o.get_state(), g.get_state(), err_msg=kind)
    g.close()


def test_mask_of_a_banded_host_step_is_not_the_listed_one():
    """A host-state step leaves a mask without a list; a stage 2 called after it must take that mask, not
    the list of an earlier check_solve."""
    nx, ny = 320, 270
    p, st, q1 = _partly_wet(2, nx, ny, _wet(nx, ny, "disk"))
    q2 = _partly_wet(2, nx, ny, _wet(nx, ny, "stripes"))[2]
    out = []
    for banded in (False, True):
        g = ImexSolver(p, st)
        g.set_state(q1, 0.0)
        g.check_solve(0.0)                      # lists the disk
        g.set_clock(0.0, 1e-2)
        if banded:
            g.advance_host(q2, 0.0)
        else:
            g.set_state(q2, 0.0)
            g.advance(1)
        g.imex_RK_solver(g.stats().t, 1e-4)
        out.append(g.get_state())
        g.close()
    np.testing.assert_array_equal(out[0], out[1])


def test_thinly_spread_cells_cost_like_packed_ones():
    """65536 wet cells of a 1024 x 1024 grid in stripes that touch every grid block, and in one square: the
    stripes' solve cells (their margins included) are twice the square's."""
    n = 1024
    stripes = np.broadcast_to((np.arange(n) % 64 < 4)[:, None], (n, n)).astype(float)
    square = np.zeros((n, n))
    square[300:556, 300:556] = 1.0
    ms = {}
    for name, wet in (("stripes", stripes), ("square", square)):
        p, st, q = _partly_wet(2, n, n, wet)
        g = ImexSolver(p, st)
        g.profile(True)
        part = []
        for _ in range(7):
            g.set_state(q, 0.0)
            g.set_clock(0.0, 1e-2)
            g.advance(1)
            part.append(sum(v[0] for k, v in g.kernel_times().items() if k.startswith("stage2")))
        ms[name] = float(np.median(part))
        g.close()
    assert ms["stripes"] < 3.0 * ms["square"], ms
