"""The timed cases: what a wind solve has this library do, from one line
relaxation of a small system to one outer iteration on the largest mesh.

A case is a dict of plain values; `prepare` makes a caller's inputs and kept
objects on the GPU, `run` is one pass through the public entry points,
`work` the bytes and operations the pass cannot do without, and `exact` the
line relaxations' values from plain torch in 64 bits. Meshes and states are
the benchmark workloads' (ablsteadyrans_b200.workloads); the sizes are those
of the workloads, the tests and sizes between them.

Kinds:
  sweep       z-line Jacobi sweeps of one system (gb.zline_jacobi)
  batch       z-line Jacobi sweeps of a batch of uneven tiles' systems
              (gb.zline_jacobi_batch)
  project     a mass-consistent projection by the Poisson solver: new face
              coefficients, the solve and the face fluxes (gb.PoissonSolver)
  residual    the steady residual of a state (SimplecStage.residual)
  initialize  the mass-consistent initial state (SimplecStage.initialize)
  iterate     the local time step and one SIMPLEC outer iteration
              (SimplecStage.local_dtau, SimplecStage.iterate)
"""
import math

import numpy as np
import torch

import ablsteadyrans_b200 as gb
from ablsteadyrans_b200 import abi, batch, workloads
from ablsteadyrans_b200.simplec import FIELDS, DeviceCase, SimplecStage

LOCS = {"cell": gb.LOC_CELL, "x": gb.LOC_XFACE, "y": gb.LOC_YFACE, "z": gb.LOC_ZFACE}
DTYPES = {"f64": torch.float64, "f32": torch.float32}
#: Iterations taken before the kept state of an `iterate` or `residual` case
#: (the state a solve is in after its start; the graphs are recorded too).
SPIN_UP = 6


def listed():
    return [
        # the smallest call: a few sweeps of a small cell system on a host that calls one system at a time
        {"name": "sweep_small", "kind": "sweep", "nx": 33, "ny": 17, "nz": 12, "loc": "cell", "periodic_y": False,
         "dtype": "f64", "sweeps": 2},
        # the u system of the 128 x 128 x 64 hill with the workload's sweep count, periodic in y
        {"name": "sweep_u_128", "kind": "sweep", "nx": 128, "ny": 128, "nz": 64, "loc": "x", "periodic_y": True,
         "dtype": "f64", "sweeps": 4},
        # a ragged w system in FP32, the inner precision of the mixed solves
        {"name": "sweep_w_f32_ragged", "kind": "sweep", "nx": 181, "ny": 150, "nz": 70, "loc": "z", "periodic_y": False,
         "dtype": "f32", "sweeps": 4},
        # the u, v and w systems of twelve uneven tiles in one work-list
        {"name": "batch_12_tiles", "kind": "batch", "tiles": 12, "dtype": "f64", "sweeps": 4},
        # a projection on the Askervein mesh's size: every multigrid level is small
        {"name": "project_30", "kind": "project", "nx": 30, "ny": 30, "nz": 18, "precision": 0},
        # a projection of a ragged mid-size domain with the FP32 inner multigrid
        {"name": "project_ragged_f32", "kind": "project", "nx": 152, "ny": 88, "nz": 57, "precision": 1},
        # the mass-consistent wind of a served tile
        {"name": "initialize_tile_96", "kind": "initialize", "nx": 96, "nz": 64, "precision": 0},
        # the residual of the hill (a norm, a Newton step or a check of a restart)
        {"name": "residual_hill_128", "kind": "residual", "mesh": "hill", "nx": 128, "ny": 128, "nz": 64},
        # the flat neutral boundary layer: every launch is short
        {"name": "iterate_flat_32", "kind": "iterate", "mesh": "flat", "nx": 32, "ny": 32, "nz": 48},
        # a batch member: fractal terrain, inflow on two sides
        {"name": "iterate_tile_96", "kind": "iterate", "mesh": "tile", "nx": 96, "ny": 96, "nz": 48},
        # the headline workload: the 128 x 128 x 64 hill
        {"name": "iterate_hill_128", "kind": "iterate", "mesh": "hill", "nx": 128, "ny": 128, "nz": 64},
        # the largest domain: fractal terrain with a roughness map
        {"name": "iterate_fractal_256", "kind": "iterate", "mesh": "fractal", "nx": 256, "ny": 256, "nz": 96},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case. The FP32 inner precision is drawn where a pass ends at a tight
    tolerance or is itself an FP32 result; an outer iteration is drawn in FP64, where
    its outputs are defined to FP64 rounding."""
    kind = rng.choice(("sweep", "sweep", "batch", "project", "initialize", "residual", "iterate", "iterate", "iterate"))
    if kind == "sweep":
        return {"kind": kind, "nx": _log_int(rng, 16, 256), "ny": _log_int(rng, 16, 256), "nz": _log_int(rng, 12, 96),
                "loc": rng.choice(sorted(LOCS)), "periodic_y": rng.random() < 0.5, "dtype": rng.choice(("f64", "f64", "f32")),
                "sweeps": rng.randint(2, 4)}
    if kind == "batch":
        return {"kind": kind, "tiles": rng.randint(3, 16), "dtype": rng.choice(("f64", "f32")), "sweeps": rng.randint(2, 4)}
    if kind == "project":
        return {"kind": kind, "nx": 8 * _log_int(rng, 4, 24), "ny": 8 * _log_int(rng, 4, 24), "nz": _log_int(rng, 16, 96),
                "precision": rng.randint(0, 1)}
    if kind == "initialize":
        return {"kind": kind, "nx": 8 * _log_int(rng, 6, 24), "nz": rng.randint(40, 96), "precision": rng.randint(0, 1)}
    mesh = rng.choice(("flat", "tile", "hill", "fractal"))
    nx = 8 * _log_int(rng, 4, 24)
    ny = nx if mesh in ("tile", "fractal") else 8 * _log_int(rng, 4, 24)
    return {"kind": kind, "mesh": mesh, "nx": nx, "ny": ny, "nz": rng.randint(40, 96)}


# ------------------------------------------------------------------ sweeps ---

def _system(grid, loc, dtype, rng):
    """A system as the implicit rows give it: six neighbour coefficients, the
    vertical ones the largest (thin layers), the diagonal their sum plus 1 / dtau."""
    v = grid.valid(loc)

    def uniform(lo, hi):
        a = torch.zeros(grid.shape, dtype=torch.float64, device="cuda")
        a[v] = torch.empty(a[v].shape, dtype=torch.float64, device="cuda").uniform_(lo, hi, generator=rng)
        if loc & 1 and grid.periodic_x:
            a[:, :, grid.ng + grid.nx] = a[:, :, grid.ng]
        if loc & 2 and grid.periodic_y:
            a[:, grid.ng + grid.ny, :] = a[:, grid.ng, :]
        return a

    A = torch.zeros((gb.N_COEFS,) + grid.shape, dtype=torch.float64, device="cuda")
    for n in range(1, 7):
        A[n] = uniform(0.1, 1.0) if n < 5 else uniform(1.0, 10.0)
    A[0] = A[1:].sum(0)
    ap = torch.where(A[0] != 0, A[0] + uniform(0.3, 3.0), 0.0)
    return A.to(dtype), ap.to(dtype), uniform(-1.0, 1.0).to(dtype)


def _sweep_grid(case):
    return gb.Grid(case["nx"], case["ny"], case["nz"], 25.0, 25.0, 1500.0 / case["nz"], False, case["periodic_y"])


def _tile_sizes(tiles):
    """The grids of a batch: the batched workload's horizontal sizes and layer counts in a fixed mix."""
    rng = np.random.default_rng(tiles)
    return [(int(rng.choice(batch.CONFIG3_SIZES)), int(rng.choice(batch.CONFIG3_LAYERS))) for _ in range(tiles)]


def _generator(seed):
    rng = torch.Generator(device="cuda")
    rng.manual_seed(seed)
    return rng


def _sweep_systems(case, seed):
    """[(grid, loc, A, ap, rhs)] of a sweep or batch case."""
    rng = _generator(seed)
    dtype = DTYPES[case["dtype"]]
    if case["kind"] == "sweep":
        grid, loc = _sweep_grid(case), LOCS[case["loc"]]
        return [(grid, loc) + _system(grid, loc, dtype, rng)]
    out = []
    for n, nz in _tile_sizes(case["tiles"]):
        grid = gb.Grid(n, n, nz, 30.0, 30.0, 1500.0 / nz, False, False)
        out += [(grid, loc) + _system(grid, loc, dtype, rng) for loc in (gb.LOC_XFACE, gb.LOC_YFACE, gb.LOC_ZFACE)]
    return out


def _exact_sweeps(grid, loc, A, ap, rhs, sweeps):
    """z-line Jacobi in 64 bits: every column's tridiagonal solved by Thomas with
    the neighbours of the iterate before, from zero; (delta, max |last change|)."""
    v = grid.valid(loc)
    c = [A[n].double()[v] for n in range(7)]
    a, b = ap.double()[v], rhs.double()[v]
    nk, nj, ni = b.shape

    def shifted(x, d, dim, n, periodic):
        """The neighbour's value in direction d along dim: zero outside, the periodic image across a seam."""
        y = torch.zeros_like(x)
        m = x.shape[dim]
        if d > 0:
            y.narrow(dim, 0, m - 1).copy_(x.narrow(dim, 1, m - 1))
            if periodic:
                y.narrow(dim, m - 1, 1).copy_(x.narrow(dim, m - n, 1))
        else:
            y.narrow(dim, 1, m - 1).copy_(x.narrow(dim, 0, m - 1))
            if periodic:
                y.narrow(dim, 0, 1).copy_(x.narrow(dim, n - 1, 1))
        return y

    x = torch.zeros_like(b)
    change = 0.0
    for _ in range(sweeps):
        r = (b + c[1] * shifted(x, -1, 2, grid.nx, grid.periodic_x) + c[2] * shifted(x, 1, 2, grid.nx, grid.periodic_x)
             + c[3] * shifted(x, -1, 1, grid.ny, grid.periodic_y) + c[4] * shifted(x, 1, 1, grid.ny, grid.periodic_y))
        cp, e = torch.empty_like(b), torch.empty_like(b)
        for k in range(nk):
            m = a[k] + (c[5][k] * cp[k - 1] if k else 0.0)
            cp[k] = -c[6][k] / m
            e[k] = (r[k] + (c[5][k] * e[k - 1] if k else 0.0)) / m
        new = e
        for k in range(nk - 2, -1, -1):
            new[k] -= cp[k] * new[k + 1]
        change = float((new - x).abs().max())
        x = new
    out = torch.zeros(grid.shape, dtype=torch.float64, device=b.device)
    out[v] = x
    return out, change


# ------------------------------------------------------------------ stages ---

def _instance(case, seed, precision=0):
    """A workload instance: the mesh of the case, the wind of the seed."""
    rng = np.random.default_rng(seed)
    mesh = case.get("mesh", "tile")
    if mesh == "tile":
        inst = workloads.tile(case["nx"], case["nz"], seed % 100000, precision=precision)
    elif mesh == "fractal":
        inst = workloads.config2(precision=precision, n=case["nx"], nz=case["nz"], seed=seed % 100000)
    else:
        make = workloads.config0 if mesh == "flat" else workloads.config1
        inst = make(nx=case["nx"], ny=case["ny"], nz=case["nz"], precision=precision)
    # the seed's wind speed: the log law and its k scale with u* and u*^2
    s = rng.uniform(0.8, 1.2)
    inst.bc.inflow_ustar *= s
    for f, e in (("u", 1), ("v", 1), ("tke", 2)):
        inst.q[f] *= s ** e
    return inst


def _stage(inst):
    ctx = gb.Context()
    z = torch.from_numpy(inst.z).cuda()
    J, ax, ay, az, _ = gb.mesh_metrics(ctx, inst.grid, z)
    case = DeviceCase(inst.grid, z, J, ax, ay, az, inst.nu, inst.gamma_theta, inst.gamma_tke, inst.q, inst.z0map)
    inst.options.poisson.restart = 8  # the correction's relative tolerance of 1e-3 needs few Krylov vectors
    stage = SimplecStage(ctx, case, inst.bc, inst.physics, inst.options)
    return {"ctx": ctx, "dcase": case, "stage": stage, "inst": inst}


def _project_state(case, seed):
    inst = _instance({"mesh": "hill", "nx": case["nx"], "ny": case["ny"], "nz": case["nz"]}, seed)
    g = inst.grid
    rng = _generator(seed)
    ctx = gb.Context()
    z = torch.from_numpy(inst.z).cuda()
    J, ax, ay, az, _ = gb.mesh_metrics(ctx, g, z)
    # inflow west, outflow east, periodic in y: the correction's conditions
    bc = (gb.POISSON_NEUMANN, gb.POISSON_PERIODIC, gb.POISSON_NEUMANN, gb.POISSON_DIRICHLET, gb.POISSON_PERIODIC,
          gb.POISSON_NEUMANN)
    opt = gb.PoissonOptions.default(precision=case["precision"])
    solver = gb.PoissonSolver(ctx, g, z, J, bc, opt)
    # positive face coefficients that vary smoothly (a correction's denominators)
    kk, jj, ii = (torch.arange(n, dtype=torch.float64, device="cuda") for n in g.shape)
    ph = torch.rand(3, dtype=torch.float64, device="cuda", generator=rng) * 2 * math.pi
    # periodic in y: the seam's faces carry one coefficient
    wave = (torch.sin(2 * math.pi * (ii - g.ng) / g.nx + ph[0])[None, None, :]
            * torch.sin(2 * math.pi * (jj - g.ng) / g.ny + ph[1])[None, :, None]
            * torch.cos(math.pi * (kk - g.ng) / g.nz + ph[2])[:, None, None])
    beta = [1.0 + 0.4 * wave, 1.0 - 0.3 * wave, 1.0 + 0.2 * wave]
    # the divergence the projection removes: a few broad features and cell noise
    v = g.valid(gb.LOC_CELL)
    rhs = torch.zeros(g.shape, dtype=torch.float64, device="cuda")
    noise = torch.empty(rhs[v].shape, dtype=torch.float64, device="cuda").uniform_(-1.0, 1.0, generator=rng)
    rhs[v] = 1e-2 * (wave[v] + 0.3 * noise)
    return {"ctx": ctx, "solver": solver, "areas": (ax, ay, az), "beta": beta, "rhs": rhs, "work": rhs.clone(),
            "phi": torch.zeros_like(rhs), "fluxes": [torch.zeros_like(rhs) for _ in range(3)]}


# --------------------------------------------------------------- interface ---

def prepare(case, seed):
    kind = case["kind"]
    if kind in ("sweep", "batch"):
        systems = [s + (torch.zeros_like(s[4]),) for s in _sweep_systems(case, seed)]
        return {"kind": kind, "ctx": gb.Context(), "systems": systems, "sweeps": case["sweeps"]}
    if kind == "project":
        return {"kind": kind, **_project_state(case, seed)}
    s = {"kind": kind, **_stage(_instance(case, seed, case.get("precision", 0)))}
    if kind == "initialize":
        s["options"] = abi.InitOptions.make()
        s["options"].poisson.precision = case["precision"]
        return s
    stage, q = s["stage"], s["dcase"].q
    stage.initialize()
    s["dtau"] = None
    for _ in range(SPIN_UP):
        s["dtau"] = stage.local_dtau(1.0, out=s["dtau"])
        stage.iterate(s["dtau"])
    stage.fill_ghosts()
    s["start"] = {f: q[f].clone() for f in FIELDS}
    if kind == "residual":
        s["R"] = [torch.zeros_like(q["u"]) for _ in range(6)]
    return s


def run(state):
    kind = state["kind"]
    if kind == "sweep":
        grid, loc, A, ap, rhs, delta = state["systems"][0]
        change = gb.zline_jacobi(state["ctx"], grid, loc, A, ap, rhs, state["sweeps"], delta)
        return delta, change
    if kind == "batch":
        change = gb.zline_jacobi_batch(state["ctx"], state["systems"], state["sweeps"])
        return [s[5] for s in state["systems"]], np.array(change)
    if kind == "project":
        # a singular solve would change its right-hand side: the solver gets a copy
        state["work"].copy_(state["rhs"])
        solver = state["solver"]
        solver.set_coeffs(*state["areas"], *state["beta"])
        res = solver.solve(state["work"], state["phi"])
        return state["phi"], solver.fluxes(state["phi"], *state["beta"], out=state["fluxes"]), res.iterations
    stage, q = state["stage"], state["dcase"].q
    if kind == "initialize":
        res = stage.initialize(state["options"])
        return [q[f] for f in FIELDS], res.poisson_iterations
    if kind == "residual":
        return stage.residual(out=state["R"])
    # one step from the kept state (a driver that tries a step keeps the state it started from)
    for f in FIELDS:
        q[f].copy_(state["start"][f])
    dtau = stage.local_dtau(2.0, out=state["dtau"])
    info = stage.iterate(dtau)
    return [q[f] for f in FIELDS], dtau, list(info.residual_norms), info.max_speed, info.poisson_iterations


def exact(case, seed):
    if case["kind"] not in ("sweep", "batch"):
        # the others end in a Krylov solve to a tolerance or are the whole
        # discretisation: no value of theirs follows from a few plain lines
        return None
    done = [_exact_sweeps(*s, case["sweeps"]) for s in _sweep_systems(case, seed)]
    if case["kind"] == "sweep":
        return done[0]
    return [d[0] for d in done], np.array([d[1] for d in done])


def work(case):
    kind = case["kind"]
    if kind in ("sweep", "batch"):
        # six neighbours, the diagonal and the right-hand side in, the increment out;
        # a sweep: the lateral terms (8), the elimination (3) and the back substitution (2), the factors (4) once
        if kind == "sweep":
            points = [int(np.prod(_sweep_grid(case).extents(LOCS[case["loc"]])))]
        else:
            points = [n * n * nz + d for n, nz in _tile_sizes(case["tiles"]) for d in (n * nz, n * nz, n * n)]
        n = float(sum(points))
        return {"bytes": n * 9 * (8 if case["dtype"] == "f64" else 4), "flops": n * (13 * case["sweeps"] + 4)}
    cells = float(case["nx"] * case.get("ny", case["nx"]) * case["nz"])
    vcycle, krylov = 900.0, 140.0  # operations a cell: five operators and four column solves on all levels; one step's rest
    if kind == "project":
        # areas, coefficients, node heights, J and the right-hand side in; the potential and three fluxes out
        return {"bytes": cells * 13 * 8, "flops": cells * (12 * (vcycle + krylov) + 100)}
    if kind == "initialize":
        # node heights, J and areas in; the state out
        return {"bytes": cells * 11 * 8, "flops": cells * (12 * (vcycle + krylov) + 300)}
    if kind == "residual":
        # the state, node heights, J and areas in; six residuals out
        return {"bytes": cells * 16 * 8, "flops": cells * 3000}
    # the state in and out, node heights, J and areas; the residual, the rows and sweeps of five systems, the correction
    return {"bytes": cells * 17 * 8, "flops": cells * (3000 + 5 * 120 + 4 * (vcycle + krylov) + 600)}
