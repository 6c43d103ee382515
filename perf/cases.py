"""Performance cases: what users of this library have it do, through its public entry points.

A case is a dict of plain values; `prepare` builds what a program holds before the call (the solver context, the
initial state, host buffers), `run` makes one pass and `exact` restates the same pass in plain torch float64.

Kinds of pass
  run       a whole small run: state in from the host, n driver steps replayed from the step's graph, state out
  routines  the reference driver's own calls, step by step, on a host-held clock: check_solve, timestep,
            imex_RK_solver, update_erosion_deposition_cell; state and physical variables out
  steps     n driver steps on a state that stays in device memory (put back to its start on the device before)
  host      one driver step from a host state to a host state (a driver that keeps its arrays on the host)
  ensemble  n steps of independent members advanced together
  network   the Newton warm-start network: one loss and gradient, one prediction, on host batches
  setup     a run's set-up: DEM sampling, source cell fractions, restart regridding, on host arrays
"""
import functools
import math

import numpy as np
import torch

from imex_sflow2d_v2_b200 import configs, grid_setup
from imex_sflow2d_v2_b200.solver import ImexEnsemble, ImexMLP, ImexSolver

EPS = 2.220446049250313e-16
F64 = torch.float64


def _steps_case(name, kind, nx, ny, ns, steps, dx, state, **opt):
    """Options: rheology 0 none, 1 Voellmy, 6 quadratic; limiter 1 minmod, 2 superbee, 3 and 4 the theta forms;
    corrections = slope correction and curvature; exchange 0 none, 1 settling and entrainment, 2 settling and
    erosion; moving_bed with the output sweep after each step; inlet a radial source."""
    c = {"name": name, "kind": kind, "nx": nx, "ny": ny, "ns": ns, "steps": steps, "dx": dx, "state": state,
         "rheology": 1, "limiter": 1, "corrections": False, "exchange": 0, "moving_bed": False, "inlet": False,
         "graph": True}
    c.update(opt)
    return c


def listed():
    return [
        # the reference's one-row tests (400 x 1 cells): launch latency is all there is
        _steps_case("row_400", "run", 400, 1, 1, 50, 0.25, "dam", rheology=6),
        # the 200 x 200 dam break, 100 steps from state in to state out: small kernels from a graph
        _steps_case("dambreak_200", "run", 200, 200, 1, 100, 0.05, "dam", rheology=0),
        # a driver that calls the routines one by one, at the reference TEST_2D's size and physics (100 x 68,
        # quadratic friction, settling and entrainment)
        _steps_case("routines_100x68", "routines", 100, 68, 1, 10, 50.0, "layer", rheology=6, exchange=1),
        # rough slope with slope correction and curvature, ragged tiles, superbee, four solid classes
        _steps_case("slope_301x517", "steps", 301, 517, 4, 8, 4.0, "blob", corrections=True, limiter=2),
        # radial current of the 1024 x 1024 workload: two classes, an inlet, mostly dry cells
        _steps_case("radial_1024", "steps", 1024, 1024, 2, 10, 2.0, "blob", inlet=True),
        # moving bed: erosion changes the topography, geometry rebuilt and outputs swept after each step
        _steps_case("moving_bed_765x500", "steps", 765, 500, 3, 4, 10.0, "layer", exchange=2, corrections=True,
                    moving_bed=True),
        # the throughput workload's physics (three classes, settling, erosion, every cell wet) at an odd middle size
        _steps_case("layer_1021x1003", "steps", 1021, 1003, 3, 2, 10.0, "layer", exchange=2, inlet=True,
                    graph=False),
        # and at its own size
        _steps_case("layer_4096", "steps", 4096, 4096, 3, 1, 10.0, "layer", exchange=2, inlet=True, graph=False),
        # a host driver's step: the state goes up and comes back each step
        _steps_case("host_2048", "host", 2048, 2048, 3, 1, 10.0, "layer", exchange=2, inlet=True),
        # ensemble of radial currents on their own grids
        {"name": "ensemble_24", "kind": "ensemble", "members": 24, "side_min": 256, "side_max": 512, "steps": 10},
        # warm-start network: a batch's gradient and predictions
        {"name": "network_65536", "kind": "network", "n": 65536},
        # set-up of a 1024 x 1024 run
        {"name": "setup_1024", "kind": "setup", "nx": 1024, "ny": 1024, "dem": 1100, "radius": 80.0},
    ]


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    kind = rng.choice(["row", "dam", "routines", "slope", "radial", "moving", "layer", "layer", "host", "ensemble",
                       "network", "setup"])
    ns = rng.choice([1, 2, 3, 3, 4])
    rheology = rng.choice([1, 1, 6])
    limiter = rng.choice([1, 1, 2, 3, 4])
    if kind == "row":
        c = _steps_case("", "run", size(60, 4000), 1, 1, rng.randint(20, 80), 0.25, "dam", rheology=rheology)
    elif kind == "dam":
        c = _steps_case("", "run", size(40, 400), size(40, 400), rng.choice([1, 2]), rng.randint(20, 100), 0.05, "dam",
                        rheology=rng.choice([0, 1, 6]), limiter=limiter)
    elif kind == "routines":
        c = _steps_case("", "routines", size(40, 300), size(40, 300), ns, rng.randint(4, 12), 50.0, "layer",
                        rheology=rheology, exchange=rng.choice([0, 1, 2]))
    elif kind == "slope":
        c = _steps_case("", "steps", size(100, 1000), size(100, 1000), ns, rng.randint(2, 8), 4.0, "blob",
                        rheology=rheology, corrections=True, limiter=limiter)
    elif kind == "radial":
        n = size(200, 1600)
        c = _steps_case("", "steps", n, n, ns, rng.randint(4, 12), 2.0, "blob", inlet=True, rheology=rheology)
    elif kind == "moving":
        c = _steps_case("", "steps", size(150, 900), size(150, 900), ns, rng.randint(2, 6), 10.0, "layer", exchange=2,
                        corrections=True, moving_bed=True)
    elif kind == "layer":
        c = _steps_case("", "steps", size(150, 2500), size(150, 2500), ns, rng.randint(1, 2), 10.0, "layer",
                        exchange=rng.choice([0, 1, 2]), inlet=True, graph=False)
    elif kind == "host":
        c = _steps_case("", "host", size(100, 2048), size(100, 2048), ns, 1, 10.0, "layer",
                        exchange=rng.choice([0, 2]), inlet=True)
    elif kind == "ensemble":
        lo = rng.randint(100, 400)
        c = {"kind": kind, "members": rng.randint(3, 24), "side_min": lo, "side_max": lo + rng.randint(20, 150),
             "steps": rng.randint(4, 12)}
    elif kind == "network":
        c = {"kind": kind, "n": size(500, 260000)}
    else:
        c = {"kind": kind, "nx": size(100, 1200), "ny": size(100, 1200), "dem": size(300, 2000),
             "radius": rng.uniform(2.0, 90.0)}
    c.pop("name", None)
    return c


# ------------------------------------------------------------------ inputs

def _gen(seed, salt=0):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed * 1000003 + salt)
    return g


def _smooth(g, ny, nx):
    """A smooth random field of unit size on the grid."""
    f = torch.randn((1, 1, 9, 9), generator=g, device="cuda", dtype=torch.float32)
    f = torch.nn.functional.interpolate(f, size=(ny, nx), mode="bicubic", align_corners=True)[0, 0].to(F64)
    return f / f.abs().max()


@functools.lru_cache(maxsize=1)
def _site(key):
    """Parameters and static planes of a stepping case (the bed and the inlet do not depend on the seed)."""
    c = dict(key)
    nx, ny, ns, dx = c["nx"], c["ny"], c["ns"], c["dx"]
    p = configs.default_params(nx, ny, ns, dx)
    for i in range(ns):
        p.rho_s[i] = 2500.0 - 200.0 * i
        p.diam_s[i] = 10.0 ** (-5.0 + 2.0 * (i + 0.5) / ns) if ns != 3 else (1e-5, 1e-4, 1e-3)[i]
        p.sp_heat_s[i] = 1617.0
    if c["rheology"]:
        p.rheology_flag, p.rheology_model = 1, c["rheology"]
        p.mu, p.xi, p.friction_factor = 0.1, 500.0, 1.0e-3
    p.theta = 1.3
    for i in range(6 + ns):
        p.limiter[i] = c["limiter"]
    (configs.transmissive_bcs if c["state"] == "dam" else configs.zero_gradient_bcs)(p)
    n = max(nx, ny)
    if c["state"] == "dam":
        p.max_dt = 1.0e-2
        B = np.zeros((nx, ny))
    else:
        p.max_dt = 1.0
        B = np.asfortranarray(configs.fractal_dem(n, dx, 0.8, 0.02 * n * dx, 8.0, 20261203)[:nx, :ny])
    st = {"B_cent": B, "solve_mask_time": np.zeros((nx, ny))}
    st.update(configs.topography_geom(B, dx if nx > 1 else 1.0, dx if ny > 1 else 1.0))
    if c["corrections"]:
        p.slope_correction_flag = p.curvature_term_flag = 1
        st.update(configs.slope_correction_planes(st))
    if c["inlet"]:
        _, xc, _, yc = configs.grid(p)
        # centred a fraction of a cell off the cell centres, so that no cell centre lies on the circle
        src = (xc[nx // 4] + 0.31 * dx, yc[ny // 2] + 0.17 * dx)
        st.update(configs.init_radial_source(p, src[0], src[1], 5.3 * dx))
        configs.set_radial_source_state(p, 5.3 * dx, 5000.0 * dx, 10.0, 900.0, [0.95 / ns] * ns)
    if c["exchange"]:
        p.settling_flag = 1
        p.T_erodible = 300.0
        p.rho_c_sub = p.pres / (p.sp_gas_const_a * p.T_erodible)
        st.update(erodible=np.zeros((ns, nx, ny)), deposit=np.zeros((nx, ny, ns)), erosion=np.zeros((nx, ny, ns)))
        if c["exchange"] == 1:
            p.entrainment_flag = 1
        else:
            p.erosion_coeff, p.erodible_porosity = 1.0e-4, 0.4
            p.coeff_porosity = p.erodible_porosity / (1.0 - p.erodible_porosity)
            er = np.empty((ns, nx, ny), order="F")
            er[:] = (1.0 - p.erodible_porosity) / ns
            st["erodible"] = er
        if c["moving_bed"]:
            p.topo_change_flag = 1
    return p, st


def _state(c, p, st, seed):
    """The seeded initial state q as torch planes (n_vars, ny, nx)."""
    g = _gen(seed)
    nx, ny, ns = c["nx"], c["ny"], c["ns"]
    f = [_smooth(g, ny, nx) for _ in range(5)]
    x = (torch.arange(nx, device="cuda", dtype=F64) + 0.5) / nx
    y = (torch.arange(ny, device="cuda", dtype=F64) + 0.5) / ny
    W = torch.zeros((6 + ns, ny, nx), device="cuda", dtype=F64)
    if c["state"] == "dam":         # still water either side of a dam across the longer axis
        s = x[None, :] if nx >= ny else y[:, None]
        W[0] = torch.where(s < 0.5, 1.0, 0.1) * (1.0 + 0.02 * f[0])
        W[3] = 300.0
        a = 0.01
    elif c["state"] == "layer":     # a wet layer over the whole grid, in motion
        W[0] = 2.0 * (1.0 + 0.3 * f[0])
        W[4 + ns] = 4.0 + 3.0 * f[1]
        W[5 + ns] = 3.0 * f[2]
        W[3] = 900.0 + 60.0 * f[3]
        a = 0.02
    else:                           # a spreading current on dry ground
        r = torch.sqrt(((x[None, :] - 0.4) * nx) ** 2 + ((y[:, None] - 0.5) * ny) ** 2) / (0.21 * min(nx, ny))
        W[0] = torch.where(r < 1.0, 1.0 + 4.0 * (1.0 - r * r), 0.0) * (1.0 + 0.2 * f[0])
        W[4 + ns] = 6.0 * (x[None, :] - 0.4) / 0.21 + 2.0 * f[1]
        W[5 + ns] = 6.0 * (y[:, None] - 0.5) / 0.21 + 2.0 * f[2]
        W[3] = 700.0 + 60.0 * f[3]
        a = 0.02
    W[1], W[2] = W[0] * W[4 + ns], W[0] * W[5 + ns]
    for i in range(ns):
        W[4 + i] = a / ns * (1.0 + 0.2 * f[4]) * W[0]
    q = _Plain(p, None).cons(W)
    if c["inlet"]:
        q[:, torch.as_tensor(np.ascontiguousarray(st["source_cell"].T)).cuda() == 1] = 0.0
    return q


def _key(c):
    return tuple(sorted((k, v) for k, v in c.items() if k not in ("name", "steps", "graph")))


class _DevicePlanes:
    """The solver's q planes in device memory; keeps the owner of that memory (the solver, or the ensemble it is a
    member of) alive while a tensor views them."""

    def __init__(self, solver, owner):
        ptr, pitch = solver.device_state()
        self.solver, self.owner = solver, owner
        self.__cuda_array_interface__ = {"shape": (solver.nv, solver.ny, pitch), "typestr": "<f8",
                                         "data": (ptr, False), "version": 3}


def _flat(q):
    """torch planes -> the reference's element order q(n_vars, nx, ny), flat on the host."""
    return np.ascontiguousarray(q.permute(1, 2, 0).contiguous().cpu().numpy().reshape(-1))


class _State:
    pass


def prepare(case, seed):
    s = _State()
    s.case = c = dict(case)
    if c["kind"] == "network":
        x, y, prm = _network_inputs(c, seed)
        s.net, s.x, s.y = ImexMLP(seed=3), x, y
        s.net.set_params(prm)
        return s
    if c["kind"] == "setup":
        s.dem, s.source, s.restart = _setup_inputs(c, seed)
        return s
    if c["kind"] == "ensemble":
        mem = _ensemble_inputs(_key(c))
        s.ens = ImexEnsemble([(p, st) for p, st in mem])
        s.q, s.q0 = [], []
        for m, (p, st) in enumerate(mem):
            g = s.ens.member(m)
            g.set_state(_flat(_state(_member_case(p), p, st, seed * 100 + m)), 0.0)
            s.q.append(torch.as_tensor(_DevicePlanes(g, s.ens), device="cuda"))
            s.q0.append(s.q[-1].clone())
        s.ens.advance(8)          # the tile-shape trials and the step graph of the chosen shape
        return s
    p, st = _site(_key(c))
    q = _state(c, p, st, seed)
    s.solver = ImexSolver(p, st)
    s.dt0 = p.max_dt
    if c["kind"] == "host":
        n = q.numel()
        s.pinned = [torch.empty(n, dtype=F64, pin_memory=True) for _ in range(2)]
        s.q_in, s.q_out = (b.numpy() for b in s.pinned)
        s.q_in[:] = _flat(q)
        s.solver.set_state(s.q_in, 0.0)
        s.solver.set_clock(0.0, s.dt0)
        return s
    host = _flat(q)
    del q
    s.solver.set_state(host, 0.0)
    if c["kind"] == "steps":
        s.stream = torch.cuda.Stream()
        s.solver.set_stream(s.stream.cuda_stream)
        s.q = torch.as_tensor(_DevicePlanes(s.solver, s.solver), device="cuda")
        s.q0 = s.q.clone()
        torch.cuda.synchronize()
        if c["moving_bed"]:
            s.solver.post_init((0.5, 1.0, 2.0), (500.0, 5000.0))
    else:
        s.q_in, s.q_out = host, np.empty_like(host)
    return s


def run(s):
    c = s.case
    kind = c["kind"]
    if kind == "steps":
        with torch.cuda.stream(s.stream):
            s.q.copy_(s.q0)
        s.solver.set_clock(0.0, s.dt0)
        _, t = s.solver.advance(c["steps"], use_graph=c["graph"])
        out = {"q": s.q[:, :, :c["nx"]], "t": t}
        if c["moving_bed"]:
            out["print"] = list(s.solver.post_diag())
        return out
    if kind == "run":
        s.solver.set_state(s.q_in, 0.0)
        s.solver.set_clock(0.0, s.dt0)
        _, t = s.solver.advance(c["steps"], use_graph=c["graph"])
        return {"q": s.solver.get_state(out=s.q_out), "t": t}
    if kind == "routines":
        g, t, cells = s.solver, 0.0, 0
        g.set_state(s.q_in, 0.0)
        for _ in range(c["steps"]):
            cells += g.check_solve(t)
            dt = g.timestep()
            g.imex_RK_solver(t, dt)
            if c["exchange"]:
                g.update_erosion_deposition_cell(dt)
            t += dt
        q, qp = g.get_state(with_qp=True)
        return {"q": q, "qp": qp, "t": t, "cells": cells}
    if kind == "host":
        _, q, t = s.solver.advance_host(s.q_in, 0.0, out=s.q_out)
        return {"q": q, "t": t}
    if kind == "ensemble":
        torch._foreach_copy_(s.q, s.q0)
        torch.cuda.current_stream().synchronize()
        for m in range(len(s.ens)):
            s.ens.member(m).set_clock(0.0, 1.0)
        s.ens.advance(c["steps"])
        return {"q%02d" % m: s.q[m][:, :, :s.ens.member(m).nx] for m in range(len(s.ens))}
    if kind == "network":
        loss, grad = s.net.loss_grad(s.x, s.y)
        return {"loss": loss, "grad": grad, "y": s.net.predict(s.x)}
    (dem, nx, ny, x0, y0, cell), src, rst = s.dem, s.source, s.restart
    B, nod = grid_setup.init_grid_topography(dem, nx, ny, x0, y0, cell)
    frac = grid_setup.compute_cell_fract(nx, ny, x0, y0, cell, *src)
    return {"B": B, "nodata": nod, "fract": frac, "restart": grid_setup.regrid_scalar(rst, nx, ny, x0, y0, cell)}


def work(case):
    """Bytes: each input read once and each output written once.  Flops: the operations of the method's own
    expressions per cell and step (a division, square root or power counts as one), on the cells that are wet."""
    c = dict(case)
    if c["kind"] == "network":
        w = 16 * 64 + 2 * 64 * 64 + 64 * 8
        return {"bytes": c["n"] * (12 + 2 + 12 + 2) * 4 + 3 * w * 4, "flops": 2.0 * w * c["n"] * 4}
    if c["kind"] == "setup":
        n, cells = c["nx"] * c["ny"], math.pi * c["radius"] ** 2
        return {"bytes": 8 * (2 * c["dem"] ** 2 + 3 * n) + n, "flops": cells * 40000 * 13 + 60 * n}
    if c["kind"] == "ensemble":
        n = c["members"] * ((c["side_min"] + c["side_max"]) / 2) ** 2
        ns, wet, exchange, steps = 1, 0.14, 0, c["steps"]
        rheology, corrections = 1, False
    else:
        n, ns, steps, exchange = c["nx"] * c["ny"], c["ns"], c["steps"], c["exchange"]
        wet = 0.14 if c["state"] == "blob" else 1.0
        rheology, corrections = c["rheology"], c["corrections"]
    state = 2 * 8 * (4 + ns) + 16 + (8 * 7 if corrections else 0) + (8 * 6 * ns if exchange else 0)
    flops = 2 * (170 + 60 * ns) + 90 + 20 * ns + (2.3 * (170 + 25 * ns) if rheology else 60 + 10 * ns)
    if exchange:
        flops += 130 + 30 * ns + 15 * 45 * ns
    return {"bytes": n * state, "flops": flops * n * wet * steps}


# ------------------------------------------- ensemble, network and set-up inputs

@functools.lru_cache(maxsize=1)
def _ensemble_inputs(key):
    c = dict(key)
    mem = configs.ensemble_members(n_members=c["members"], side_min=c["side_min"], side_max=c["side_max"],
                                   mfr=(1.0e5, 1.0e6), seed=20261204)
    return [(p, st) for p, st, _, _ in mem]


def _member_case(p):
    return {"nx": p.nx, "ny": p.ny, "ns": 1, "state": "blob", "inlet": True}


def _network_inputs(c, seed):
    g = _gen(seed, 7)
    x = torch.randn((c["n"], 12), generator=g, device="cuda")
    y = torch.stack([torch.tanh(x[:, 1] - x[:, 3]) + 0.1 * x[:, 5], 0.5 * x[:, 2] * x[:, 8]], 1)
    prm = ImexMLP.NPARAM
    w = torch.randn(prm, generator=g, device="cuda") * 0.12
    return x.cpu().numpy(), y.cpu().numpy(), w.cpu().numpy()


def _setup_inputs(c, seed):
    g = _gen(seed, 9)
    nx, ny, n, cell = c["nx"], c["ny"], c["dem"], 10.0
    cs = 1.02 * max(nx, ny) * cell / (n - 2)      # the DEM covers the grid
    x0 = y0 = 0.75 * cs

    def raster(z, nodata_share):
        z = torch.where(torch.rand((n, n), generator=g, device="cuda") < nodata_share, -9999.0, z)
        return grid_setup.Raster(n, n, 0.0, 0.0, cs, -9999.0, np.asfortranarray(z.cpu().numpy()))
    dem = raster(500.0 + 400.0 * _smooth(g, n, n) + torch.randn((n, n), generator=g, device="cuda", dtype=F64), 1e-4)
    rst = raster(torch.relu(3.0 * _smooth(g, n, n)), 1e-4)
    r = c["radius"] * cell
    u = torch.rand(3, generator=g, device="cuda", dtype=F64).tolist()
    src = (x0 + (0.45 + 0.1 * u[0]) * nx * cell, y0 + (0.45 + 0.1 * u[1]) * ny * cell, r, 0.6 * r, 180.0 * u[2])
    return (dem, nx, ny, x0, y0, cell), src, rst


# ------------------------------------------------------- exact: plain float64

class _Plain:
    """The time step of a stepping case in plain torch float64, on planes (ny, nx)."""

    def __init__(self, p, st):
        self.p, self.ns, self.nv = p, p.n_solid, 4 + p.n_solid
        ns = self.ns

        def vec(a):
            return torch.tensor([a[i] for i in range(ns)], device="cuda", dtype=F64)[:, None, None]
        self.rho, self.cps, self.al_src = vec(p.rho_s), vec(p.sp_heat_s), vec(p.alphas_source)
        self.rho_amb = p.pres / (p.sp_gas_const_a * p.T_ambient)
        self.lim = p.limiter[0]
        if st is None:
            return

        def plane(a):
            return torch.as_tensor(np.ascontiguousarray(np.asarray(a).T)).cuda()
        self.dx = p.cell_size if p.nx > 1 else 1.0
        self.dy = p.cell_size if p.ny > 1 else 1.0
        self.B = plane(st["B_cent"])
        zero = torch.zeros_like(self.B)
        self.bx, self.by = plane(st["B_prime_x_geom"]), plane(st["B_prime_y_geom"])
        self.bxx = self.bxy = self.byy = self.dgc = zero
        self.gc, self.gsx, self.gsy = zero + 1.0, 1.0, 1.0
        if p.slope_correction_flag:
            self.bxx, self.bxy, self.byy = (plane(st["B_second_%s_geom" % k]) for k in ("xx", "xy", "yy"))
            self.gc, self.dgc = plane(st["grav_coeff"]), plane(st["d_grav_coeff_dx"])
            self.gsx, self.gsy = plane(st["grav_coeff_stag_x"]), plane(st["grav_coeff_stag_y"])
        self.src = plane(st["source_cell"]) if p.radial_source_flag else None
        if self.src is not None:
            self.side = {k: plane(st["source" + k]) != 0 for k in "EWSN"}
            vx, vy = zero, zero
            for k in "NSWE":          # the last one written wins: E, then W, S, N
                vx = torch.where(self.side[k], plane(st["source%s_vect_x" % k]), vx)
                vy = torch.where(self.side[k], plane(st["source%s_vect_y" % k]), vy)
            h, u = p.h_source, p.vel_source
            self.inlet = [zero + h, h * u * vx, h * u * vy, zero + p.T_source] + \
                [zero + h * p.alphas_source[i] for i in range(ns)] + [u * vx, u * vy]
        if st.get("erodible") is not None:
            self.erodible = torch.stack([plane(st["erodible"][i]) for i in range(ns)])

    # ---- point functions
    def prim(self, q):
        p, ns = self.p, self.ns
        wet = q[0] > EPS
        m = torch.where(wet, q[0], 1.0)
        xs = q[4:] / m
        xc = 1.0 - xs.sum(0)
        cpm = (xs * self.cps).sum(0) + xc * p.sp_heat_a
        T = (q[3] - (0.5 * (q[1] ** 2 + q[2] ** 2) / m if p.energy_flag else 0.0)) / (m * cpm)
        T = torch.where((T <= 0.0) | (m <= p.eps_sing), p.T_ambient, T)
        inv_rho = (xs / self.rho).sum(0) + xc * p.sp_gas_const_a * T / p.pres
        big = m > p.eps_sing
        den = torch.sqrt(m ** 4 + p.eps_sing ** 4)
        u, v = (torch.where(big, a / m, math.sqrt(2.0) * m * a / den) for a in (q[1], q[2]))
        h = m * inv_rho
        W = torch.stack([h, h * u, h * v, T] + [xs[i] / inv_rho / self.rho[i] * h for i in range(ns)] + [u, v])
        dry = torch.zeros_like(W)
        dry[3] = p.T_ambient
        return torch.where(wet, W, dry)

    def mixture(self, W):
        """rho_m, rho_c, reduced gravity, alphas, wet."""
        p, ns = self.p, self.ns
        wet = W[0] > EPS
        al = W[4:4 + ns] / torch.where(wet, W[0], 1.0)
        rho_c = p.pres / (p.sp_gas_const_a * torch.where(wet, W[3], p.T_ambient))
        rho_m = (1.0 - al.sum(0)) * rho_c + (al * self.rho).sum(0)
        rho_m, rho_c = (torch.where(wet, r, self.rho_amb) for r in (rho_m, rho_c))
        return rho_m, rho_c, torch.where(wet, (rho_m - self.rho_amb) / rho_m * p.grav, 0.0), al, wet

    def cons(self, W):
        p, ns = self.p, self.ns
        rho_m, rho_c, _, al, wet = self.mixture(W)
        xs = al * self.rho / rho_m
        cpm = (xs * self.cps).sum(0) + (1.0 - al.sum(0)) * rho_c / rho_m * p.sp_heat_a
        ke = 0.5 * (W[4 + ns] ** 2 + W[5 + ns] ** 2) if p.energy_flag else 0.0
        m = rho_m * W[0]
        q = torch.cat([torch.stack([m, rho_m * W[1], rho_m * W[2], m * (cpm * W[3] + ke)]), xs * m])
        return torch.where(wet, q, 0.0)

    def limit(self, v1, v2, v3, d1, d3):
        def minmod(a, b):
            return torch.where(torch.sign(a) == torch.sign(b), torch.sign(a) * torch.minimum(a.abs(), b.abs()), 0.0)
        a, b, c = (v3 - v2) / d3, (v2 - v1) / d1, (v3 - v1) / (d1 + d3)
        if self.lim == 1:
            return minmod(a, b)
        if self.lim == 2:
            s, t = minmod(a, 2.0 * b), minmod(2.0 * a, b)
            return torch.where(torch.sign(s) == torch.sign(t), torch.sign(s) * torch.maximum(s.abs(), t.abs()), 0.0)
        return minmod(c, (self.p.theta if self.lim == 3 else 2.0) * minmod(a, b))

    # ---- reconstruction and fluxes along x (dir 1) or y (dir 2); the direction is the last axis
    def faces(self, W, dir):
        p, nv = self.p, self.nv
        along = (lambda a: a) if dir == 1 else (lambda a: a.transpose(-1, -2))
        W, n = along(W), W.shape[-1 if dir == 1 else -2]
        d = self.dx if dir == 1 else self.dy
        lo, hi = (p.bcW, p.bcE) if dir == 1 else (p.bcS, p.bcN)
        d1 = torch.full((n,), d, device="cuda", dtype=F64)
        d3 = d1.clone()
        d1[0] = d3[-1] = d / 2.0
        rm = rp = None
        if self.src is not None:
            E, Wd, S, N = (along(self.side[k] & (self.src == 2)) for k in "EWSN")
            rm, rp = ((~E & Wd), E) if dir == 1 else (S, (~S & N))
            d1, d3 = torch.where(rm, d / 2.0, d1), torch.where(rp, d / 2.0, d3)
            inlet = [along(a) for a in self.inlet]
        Fm, Fp = [], []
        for i in range(nv + 2):
            v, e3 = W[i], d3
            flag = (lo[i].flag, hi[i].flag) if i < nv else (0, 0)
            if i < nv:
                g = [torch.full_like(v[..., :1], b[i].value) for b in (lo, hi)]
            else:
                g = [torch.where(F[0][..., s] > 0.0, F[1 + i - nv][..., s] / F[0][..., s], 0.0)
                     for F, s in ((Fm, slice(0, 1)), (Fp, slice(n - 1, n)))]
            v1, v3 = torch.cat([g[0], v[..., :-1]], -1), torch.cat([v[..., 1:], g[1]], -1)
            if rm is not None:
                v1, v3 = torch.where(rm, inlet[i], v1), torch.where(rp, inlet[i], v3)
                if dir == 1 and i == nv + 1:   # the reference's y abscissa in this one x stencil
                    J, K = torch.arange(n, device="cuda", dtype=F64), torch.arange(p.ny, device="cuda", dtype=F64)
                    odd = ~E & N & ~S
                    odd[:, 0] = odd[:, -1] = odd[0] = odd[-1] = False
                    e3 = torch.where(odd, (p.y0 + (K[:, None] + 1) * self.dy) - (p.x0 + (J + 0.5) * self.dx), d3)
            slope = self.limit(v1, v, v3, d1, e3)
            if flag[0]:
                slope[..., 0] = lo[i].value if flag[0] == 1 else (v[..., 1] - v[..., 0]) / d
            if flag[1]:
                slope[..., -1] = hi[i].value if flag[1] == 1 else (v[..., -1] - v[..., -2]) / d
            dq = p.reconstr_coeff * d / 2.0 * slope
            fm, fp = v - dq, v + dq
            if not flag[0]:
                fm[..., 0] = g[0][..., 0]
            elif i == dir:
                fm[..., 0] = fm[..., 0].clamp(max=0.0)
            if not flag[1]:
                fp[..., -1] = g[1][..., 0]
            elif i == dir:
                fp[..., -1] = fp[..., -1].clamp(min=0.0)
            Fm.append(fm)
            Fp.append(fp)
        if rm is not None:
            for i in range(nv + 2):
                Fp[i] = torch.where(rp, inlet[i], Fp[i])
                Fm[i] = torch.where(rm & ~rp, inlet[i], Fm[i])
        Fm, Fp = torch.stack(Fm), torch.stack(Fp)
        QL, QR = torch.cat([Fm[..., :1], Fp], -1), torch.cat([Fm, Fp[..., -1:]], -1)
        if rm is not None:
            one = along(self.src) == 1
            none = torch.zeros_like(one[..., :1])
            cp_a = torch.cat([rm, none], -1)              # the ring cell b gives its minus face to the inlet side
            cp_b = torch.cat([none, rp], -1)
            a_int, b_int = torch.cat([none, one], -1), torch.cat([one, none], -1)
            QL0 = QL
            QL = torch.where(a_int, torch.where(cp_a, QR, 0.0), QL)
            QR = torch.where(b_int, torch.where(cp_b, QL0, 0.0), QR)
        return QL, QR

    def fluxes(self, W, dir, active):
        """Kurganov-Tadmor fluxes and the largest speed at every interface."""
        p, ns, nv = self.p, self.ns, self.nv
        QL, QR = self.faces(W, dir)
        g = self.gsx if dir == 1 else (self.gsy.transpose(-1, -2) if torch.is_tensor(self.gsy) else self.gsy)

        def half(Q):
            rho_m, _, rg, _, wet = self.mixture(Q)
            c = self.cons(Q)
            vel = Q[nv + dir - 1]
            cel = torch.where(rg * Q[0] < 0.0, 0.0, torch.sqrt((rg * Q[0] * g).clamp(min=0.0)))
            pr = 0.5 * rho_m * g * rg * Q[0] ** 2
            f = vel * c
            f[dir] = f[dir] + pr
            f[3] = vel * (c[3] + pr) if p.energy_flag else vel * c[3]
            s = f[4:].sum(0)
            f[4:] = torch.where((f[0] > 0.0) & (s / f[0] > 1.0), f[4:] / s * f[0], f[4:])
            return c, torch.where(wet, f, 0.0), vel - cel, vel + cel
        cL, fL, l0, l1 = half(QL)
        cR, fR, r0, r1 = half(QR)
        aN, aP = torch.minimum(l0, r0).clamp(max=0.0), torch.maximum(l1, r1).clamp(min=0.0)
        gap = torch.where(aP == aN, 1.0, aP - aN)
        H = torch.where(aP == aN, 0.0, (aP * fL - aN * fR) / gap + aP * aN / gap * (cR - cL))
        r = H[4:].sum(0) / H[0]
        H[4:] = torch.where((r >= 1.0) if dir == 1 else (r > 1.0), H[4:] / r, H[4:])
        still = ((QL[1] == 0.0) & (QR[1] == 0.0)) if dir == 1 else ((cL[2] == 0.0) & (cR[2] == 0.0))
        for i in [0] + list(range(3, nv)):
            H[i] = torch.where(still, 0.0, H[i])
        return torch.where(active, H, 0.0), torch.where(active, torch.maximum(aP, -aN), 0.0)

    def stage1(self, q, solve):
        """X = flux divergence - explicit terms, and the CFL time step."""
        p, nv = self.p, self.nv
        W = Wt = self.prim(q)
        if self.src is not None:
            inner = self.src == 1
            Wt = torch.where(inner, 0.0, W)
            W = Wt.clone()
            Wt[3] = torch.where(inner, p.T_ambient, Wt[3])
        X, dt = torch.zeros_like(q), torch.tensor(p.max_dt, device="cuda", dtype=F64)
        for dir, n, d in ((1, p.nx, self.dx), (2, p.ny, self.dy)):
            if n == 1:
                continue
            along = (lambda a: a) if dir == 1 else (lambda a: a.transpose(-1, -2))
            m = along(solve)
            no = torch.zeros_like(m[..., :1])
            active = torch.cat([no, m], -1) | torch.cat([m, no], -1)
            H, amax = self.fluxes(W, dir, active)
            if self.src is not None:
                amax = self.fluxes(Wt, dir, active)[1]
            X = X + along((H[..., 1:] - H[..., :-1]) / d)
            del H
            a = along(torch.maximum(amax[..., 1:], amax[..., :-1]))
            a = a[solve & (a > 0.0)]
            if a.numel():
                dt = torch.minimum(dt, p.cfl * d / a.max())
        W = self.prim(q) if self.src is None else Wt
        rho, _, rg, _, wet = self.mixture(W)
        u, v, h = W[nv], W[nv + 1], W[0]
        centr = self.centrifugal(u, v)
        e = [-(self.gc * rho * (rg + centr) * h * b) + 0.5 * rho * rg * h * h * self.dgc for b in (self.bx, self.by)]
        e = [torch.where(wet, a, 0.0) for a in e]
        X[1] -= e[0]
        X[2] -= e[1]
        if p.energy_flag:
            X[3] -= e[0] * u + e[1] * v
        return X, float(dt)

    def centrifugal(self, u, v):
        return self.bxx * u * u + 2.0 * self.bxy * u * v + self.byy * v * v if self.p.curvature_term_flag else 0.0

    def friction(self, q1, q2, fixed):
        """The implicit friction of momentum (q1, q2), for real or complex values."""
        p = self.p
        m, q3, xs, xc, big = fixed
        u = torch.where(big, q1 / m, math.sqrt(2.0) * m * q1 / torch.sqrt(m ** 4 + p.eps_sing ** 4))
        v = torch.where(big, q2 / m, math.sqrt(2.0) * m * q2 / torch.sqrt(m ** 4 + p.eps_sing ** 4))
        T = (q3 - (0.5 * (q1 * q1 + q2 * q2) / m if p.energy_flag else 0.0)) / \
            (m * ((xs * self.cps).sum(0) + xc * p.sp_heat_a))
        T = torch.where((T.real <= 0.0) | ~big, torch.full_like(T, p.T_ambient), T)
        rho = 1.0 / ((xs / self.rho).sum(0) + xc * p.sp_gas_const_a * T / p.pres)
        w = u * self.bx + v * self.by if p.slope_correction_flag else 0.0 * u
        m2, plane2 = u * u + v * v + w * w, u * u + v * v
        moving = m2.real > 0.0
        s = torch.sqrt(torch.where(moving, m2, torch.ones_like(m2)))
        if p.rheology_model == 1:
            f = rho * ((rho - self.rho_amb) / rho * p.grav) / p.xi * m2 / s
        else:
            f = rho * p.friction_factor * m2 / torch.sqrt(torch.where(moving, plane2, torch.ones_like(m2)))
        return [torch.where(moving, -f * a, torch.zeros_like(f)) for a in (u, v)]

    def stage2(self, q0, X, dt, solve):
        p, nv = self.p, self.nv
        q = q0 - dt * X
        on = solve & (q[0] > 0.0)
        f1, f2 = q[1].clone(), q[2].clone()
        s1, s2 = f1, f2
        if p.rheology_flag:
            W = self.prim(q)
            rho, _, rg, _, _ = self.mixture(W)
            u, v = W[nv], W[nv + 1]
            w = u * self.bx + v * self.by if p.slope_correction_flag else 0.0
            speed = torch.sqrt(u * u + v * v + w * w)
            if p.rheology_model == 1:
                drag = (p.mu * rho * (rg + self.centrifugal(u, v)) * W[0] * torch.sqrt(self.gc)).clamp(min=0.0)
                drag = torch.where(speed > 0.0, drag / torch.where(speed > 0.0, speed, 1.0), 0.0)
                s1, s2 = f1 - dt * drag * u, f2 - dt * drag * v
        F = torch.hypot(f1, f2)
        stop = (F == 0.0) | (s1 * f1 < 0.0) | (s2 * f2 < 0.0)
        r = torch.where(stop, 0.0, torch.hypot(s1, s2) / torch.where(F > 0.0, F, 1.0))
        s1, s2 = r * f1, r * f2
        # q_i = s_i + dt*friction_i(q1, q2): the fully converged Newton solution
        a, b = s1.clone(), s2.clone()
        if p.rheology_flag:
            m = torch.where(on, q[0], 1.0)
            xs = torch.where(on, q[4:] / m, 0.0)
            fixed = (m, q[3], xs, 1.0 - xs.sum(0), m > p.eps_sing)
            step = 1e-30
            for _ in range(12):
                d1 = self.friction(torch.complex(a, torch.full_like(a, step)), torch.complex(b, torch.zeros_like(b)),
                                   fixed)
                r1, r2 = a - s1 - dt * d1[0].real, b - s2 - dt * d1[1].real
                j11, j21 = 1.0 - dt * d1[0].imag / step, -dt * d1[1].imag / step
                d2 = self.friction(torch.complex(a, torch.zeros_like(a)), torch.complex(b, torch.full_like(b, step)),
                                   fixed)
                j12, j22 = -dt * d2[0].imag / step, 1.0 - dt * d2[1].imag / step
                del d1, d2
                det = j11 * j22 - j12 * j21
                a, b = a - (r1 * j22 - r2 * j12) / det, b - (r2 * j11 - r1 * j21) / det
        if p.ny == 1:
            b = torch.zeros_like(b)
        if p.nx == 1:
            a = torch.zeros_like(a)
        S = torch.hypot(s1, s2)
        r = torch.where((S == 0.0) | ((a * s1 <= 0.0) & (b * s2 <= 0.0)), 0.0,
                        torch.hypot(a, b) / torch.where(S > 0.0, S, 1.0))
        q[1], q[2] = torch.where(on, r * s1, q[1]), torch.where(on, r * s2, q[2])
        q = torch.where((q[0] < EPS) & (q[0] > -1.0e-7), 0.0, q)
        neg = (q[4:] < 0.0).any(0) & (q[4:] > -1.0e-7).all(0)
        q[4:] = torch.where(neg, q[4:].clamp(min=0.0), q[4:])
        s = q[4:].sum(0)
        over = (s > q[0]) & (((s - q[0]) / q[0] < 1.0e-10) | (q[0] < EPS))
        q[4:] = torch.where(over, q[4:] / s * q[0], q[4:])
        return torch.where(solve, q, q0)

    def settling(self, i, rho_c):
        p = self.p
        d = p.diam_s[i]
        heavy = p.rho_s[i] > rho_c
        const = torch.sqrt((0.75 * (p.rho_s[i] / rho_c - 1.0) * d * p.grav).clamp(min=0.0))
        v = const.clone()
        go = heavy & (d * v / p.kin_visc_c <= 1000.0)
        for _ in range(20):
            re = d * v / p.kin_visc_c
            new = const * torch.sqrt(re / (24.0 * (1.0 + 0.15 * re ** 0.687)))
            done = go & ((v - new).abs() / v < 1.0e-6)
            v = torch.where(go, new, v)
            go = go & ~done
        return torch.where(heavy, v, 0.0)

    def exchange(self, q0, dt, solve):
        p, ns, nv = self.p, self.ns, self.nv
        W = self.prim(q0)
        rho_m, rho_c, rg, al, wet = self.mixture(W)
        u, v, h, T, at = W[nv], W[nv + 1], W[0], W[3], al.sum(0)
        w = u * self.bx + v * self.by if p.slope_correction_flag else 0.0
        m2 = u * u + v * v + w * w
        por = p.erodible_porosity
        fr = torch.tensor([p.erodible_fract[i] for i in range(ns)], device="cuda", dtype=F64)[:, None, None]
        ers = fr * (p.erosion_coeff * torch.sqrt(m2) * h * (1.0 - at) * (1.0 - por))
        ers = torch.where(wet, torch.minimum(ers, self.erodible / dt).clamp(min=0.0), 0.0)
        full = wet & (at > p.alphastot_min)
        hind = (1.0 - (at / 0.6).clamp(max=1.0)) ** 4.65
        dep = torch.zeros_like(ers)
        for i in range(ns):
            if p.settling_flag:
                x = torch.minimum(al[i] * self.settling(i, rho_c) * hind, h * al[i] / dt)
                dep[i] = torch.where(full & (al[i] > 0.0), x, 0.0)
        sdep = dep.sum(0)
        pe = ers.sum(0) / (1.0 - por) * por
        pl = torch.minimum(p.coeff_porosity * sdep, h * (p.maximum_solid_packing - at).clamp(min=0.0) / dt)
        pl = torch.minimum(pl, (h * (1.0 - at) - p.coeff_porosity * (h * at - dt * sdep)) / dt)
        Ri = torch.where(m2 > 0.0, (rg * h / torch.where(m2 > 0.0, m2, 1.0)).clamp(max=1.0e15), 0.0)
        air = torch.zeros_like(h)
        if p.entrainment_flag:
            air = torch.where(Ri > 0.0, 0.075 / torch.sqrt(1.0 + 718.0 * Ri.clamp(min=0.0) ** 2.4), 0.0) * torch.sqrt(m2)
        lost, gained = (self.rho * dep).sum(0) + rho_c * pl, (self.rho * ers).sum(0) + p.rho_c_sub * pe
        hd, he = (self.rho * self.cps * dep).sum(0), (self.rho * self.cps * ers).sum(0)
        cpc = p.sp_heat_a
        e = [self.rho_amb * air + gained - lost, -u * lost, -v * lost,
             -T * (hd + rho_c * cpc * pl) - (0.5 * m2 * lost if p.energy_flag else 0.0)
             + (T if p.erodible_deposit_flag else p.T_erodible) * (he + p.rho_c_sub * cpc * pe)
             + p.T_ambient * cpc * self.rho_amb * air]
        eq = torch.cat([torch.stack(e), self.rho * (ers - dep)])
        q = q0 + dt * torch.where(full, eq, 0.0)
        q[4:] = q[4:].clamp(min=0.0)
        q = torch.where((q[0] <= 0.0) & (q[0] > -1.0e-10), 0.0, q)
        s = q[4:].sum(0)
        q[4:] = torch.where((s > q[0]) & (q[0] < 1.0e-10), q[4:] / s * q[0], q[4:])
        light = torch.where(q[0] > 0.0, self.mixture(self.prim(q))[2], 0.0) <= 0.0
        q = torch.where(light, 0.0, q)
        self.erodible = torch.where(solve, self.erodible - dt * ers, self.erodible)
        if p.topo_change_flag:
            rise = torch.where(full, (sdep - ers.sum(0)) / (1.0 - por), 0.0)
            self.B = torch.where(solve, self.B + dt * rise, self.B)
        return torch.where(solve, q, q0)

    def geometry(self):
        """The bed's derivatives by the 5-point stencils, the two border cells copying the nearest inner ones."""
        B, ny, nx = self.B, self.p.ny, self.p.nx
        J = torch.arange(nx, device="cuda").clamp(2, nx - 3)
        K = torch.arange(ny, device="cuda").clamp(2, ny - 3)
        c1, c2 = (-2.0, -1.0, 0.0, 1.0, 2.0), (2.0, -1.0, -2.0, -1.0, 2.0)

        def at(dj, dk):
            return B[(K + dk)[:, None], (J + dj)[None, :]]
        dx, dy = self.dx, self.dy
        self.bx = sum(c1[t] * at(t - 2, 0) for t in range(5)) / (10.0 * dx)
        self.by = sum(c1[t] * at(0, t - 2) for t in range(5)) / (10.0 * dy)
        self.bxx = sum(c2[t] * at(t - 2, 0) for t in range(5)) / (7.0 * dx * dx)
        self.byy = sum(c2[t] * at(0, t - 2) for t in range(5)) / (7.0 * dy * dy)
        self.bxy = sum(c1[t] * c1[r] * at(t - 2, r - 2) for t in range(5) for r in range(5)) / (100.0 * dx * dy)
        if self.p.slope_correction_flag:
            g = self.gc = 1.0 / (1.0 + self.bx ** 2 + self.by ** 2)
            self.dgc = -(2.0 * g * g * (self.bx * self.bxx + self.by * self.bxy))
            self.gsx = torch.cat([g[:, :1], 0.5 * (g[:, :-1] + g[:, 1:]), g[:, -1:]], 1)
            self.gsy = torch.cat([g[:1], 0.5 * (g[:-1] + g[1:]), g[-1:]], 0)

    def solve_cells(self, q):
        m = q[0] > 0.0
        if self.src is not None:
            m = m | (self.src == 2)
        m[0] = m[-1] = m[:, 0] = m[:, -1] = True
        for _ in range(2):
            w = m.clone()
            w[1:-1, 1:-1] |= m[1:-1, :-2] | m[1:-1, 2:] | m[:-2, 1:-1] | m[2:, 1:-1]
            m = w
        return m if self.src is None else m & (self.src != 1)

    def advance(self, q, steps, dt0=None):
        """`steps` driver steps (dt0: the clock's first step, None: the routine-by-routine driver, no clipping);
        the state, the time and the solved cells counted over the steps."""
        p, t, cells, old = self.p, 0.0, 0, (dt0, dt0)
        act = p.erosion_coeff != 0.0 or p.settling_flag or p.entrainment_flag
        for _ in range(steps):
            solve = self.solve_cells(q)
            cells += int(solve.sum())
            X, dt = self.stage1(q, solve)
            if dt0 is not None:
                dt = min(dt, 1.1 * 0.5 * (old[0] + old[1]))
                old = (dt, old[0])
            q = self.stage2(q, X, dt, solve)
            del X
            if act:
                q = self.exchange(q, dt, solve)
            if p.topo_change_flag:
                self.geometry()
            t += dt
        return q, t, cells


def _order(q):
    """Planes (n, ny, nx) as an (n, nx, ny) array, as the library hands states out."""
    return q.permute(0, 2, 1).contiguous()


def exact(case, seed):
    c = dict(case)
    kind = c["kind"]
    if kind == "network":
        return _exact_network(c, seed)
    if kind == "setup":
        return _exact_setup(c, seed)
    if kind == "ensemble":
        out = {}
        for m, (p, st) in enumerate(_ensemble_inputs(_key(c))):
            q = _state(_member_case(p), p, st, seed * 100 + m)
            out["q%02d" % m] = _Plain(p, st).advance(q, c["steps"], 1.0)[0]
        return out
    p, st = _site(_key(c))
    q = _state(c, p, st, seed)
    ref = _Plain(p, st)
    q, t, cells = ref.advance(q, c["steps"], None if kind == "routines" else p.max_dt)
    if kind == "steps":
        out = {"q": q, "t": t}
        if c["moving_bed"]:
            d = ref.dx * ref.dy
            out["print"] = [float(d * q[0].sum()), float(d * ref.prim(q)[0].sum()),
                            float(d * (q[0] > 1.0e-7).sum()), float(d * q[4:].sum())]
        return out
    if kind == "routines":
        return {"q": _order(q), "qp": _order(ref.prim(q)), "t": t, "cells": cells}
    return {"q": q.permute(1, 2, 0).reshape(-1).cpu().numpy(), "t": t}


def _exact_network(c, seed):
    x, y, w = (torch.as_tensor(a).cuda().to(F64) for a in _network_inputs(c, seed))
    w.requires_grad_(True)
    a, o = torch.nn.functional.pad(x, (0, 4)), 0
    for n_in, n_out in ((16, 64), (64, 64), (64, 64), (64, 8)):
        a = a @ w[o:o + n_in * n_out].view(n_in, n_out) + w[o + n_in * n_out:o + (n_in + 1) * n_out]
        o += (n_in + 1) * n_out
        if n_out == 64:
            a = torch.nn.functional.silu(a)
    loss = (a[:, :2] - y).square().mean()
    loss.backward()
    return {"loss": float(loss.detach()), "grad": w.grad.cpu().numpy(), "y": a[:, :2].detach().cpu().numpy()}


def _exact_setup(c, seed):
    (dem, nx, ny, x0, y0, cell), (xs, ys, rs, r2s, angle), rst = _setup_inputs(c, seed)
    n, cs = dem.ncols, dem.cellsize

    def centre(o, m):
        return o + (torch.arange(m, device="cuda", dtype=F64) + 0.5) * cell
    z = torch.as_tensor(np.asarray(dem.z)).cuda()
    node = [(torch.arange(n, device="cuda", dtype=F64) + 0.5) * cs] * 2
    at = []
    for v, nd in ((centre(x0, nx), node[0]), (centre(y0, ny), node[1])):
        i = torch.floor((v - nd[0]) / cs).long().clamp(max=n - 2)
        at.append((i, (nd[i + 1] - v) / cs))
    (i, a), (k, b) = at
    i, a, k, b = i[:, None], a[:, None], k[None, :], b[None, :]
    zc = z.clamp(min=0.0)
    B = a * (b * zc[i, k] + (1.0 - b) * zc[i, k + 1]) + (1.0 - a) * (b * zc[i + 1, k] + (1.0 - b) * zc[i + 1, k + 1])
    nod = (z[i, k] == dem.nodata) | (z[i + 1, k] == dem.nodata) | (z[i, k + 1] == dem.nodata) | \
        (z[i + 1, k + 1] == dem.nodata)
    # cell fractions: the share of 200 x 200 points of each cell inside the ellipse
    ang = math.radians(angle)
    sub = ((torch.arange(200, device="cuda", dtype=F64) + 0.5) / 200.0 - 0.5) * cell
    X0, Y0 = centre(x0, nx), centre(y0, ny)
    R = max(rs, r2s)
    js, ks = ((v - s).abs() <= R + cell for v, s in ((X0, xs), (Y0, ys)))
    frac = torch.zeros((nx, ny), device="cuda", dtype=F64)
    kk = torch.nonzero(ks).flatten()
    Y = Y0[kk][:, None, None] + sub[None, :, None] - ys
    for j in torch.nonzero(js).flatten().tolist():
        X = X0[j] + sub[None, None, :] - xs
        u, v = X * math.cos(ang) + Y * math.sin(ang), -X * math.sin(ang) + Y * math.cos(ang)
        inside = ((u / rs) ** 2 + (v / r2s) ** 2 <= 1.0).sum((1, 2))
        frac[j, kk] = (inside.float() / 40000.0).double()
    # regridding: overlap lengths along each axis times the raster (the raster's last column is not read)
    f = torch.as_tensor(np.asarray(rst.z)).cuda()
    f = torch.where(f == rst.nodata, 0.0, f)
    edge = torch.arange(n + 1, device="cuda", dtype=F64) * cs

    def overlap(o, m, last):
        lo = o + torch.arange(m, device="cuda", dtype=F64)[:, None] * cell
        w = (torch.minimum(lo + cell, edge[None, 1:]) - torch.maximum(lo, edge[None, :-1])).clamp(min=0.0) / cell
        w[:, last:] = 0.0
        return w
    back = overlap(x0, nx, n - 1) @ f @ overlap(y0, ny, n).T
    return {"B": B.cpu().numpy(), "nodata": nod.to(torch.int8).cpu().numpy(), "fract": frac.cpu().numpy(),
            "restart": back.cpu().numpy()}
