"""The work a user of this framework has it do, as timed cases.

Each case is one call (or one short solver loop) through the public Python
mirror of the C ABI, on meshes and states shaped like the five benchmark
configurations (two-fluid shock tube, AMR shock-bubble with and without THINC,
batched droplets, 3D triple point) in the middle of a run: interfaces a few
cells wide, waves around them and undisturbed gas elsewhere.  The refinement
follows the nominal geometry, so that a mesh depends on the sizes alone and the
state on the seed.

``exact`` restates one step in plain torch, 64 bits, whole mesh at a time,
from the block table a caller hands to the framework.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from godunov_five_eq_gb300 import GodunovImplemGB300
from godunov_five_eq_gb300.configs import EOS, HydroParams
from godunov_five_eq_gb300.mesh import BC_PERIODIC, BC_WALL, BC_ZERO_GRADIENT, BlockMesh, concat_tables

F64 = torch.float64
JWL = (1905.0, 0.8938, 6.321e13, -4.472e9, 11.3, 1.13, 0.0, 0.0)  # LX-17-like products


def _case(name, **kw):
    c = dict(kind="step", problem="tube", mode="fp64", bsize=16, nx=32, ny=2, lmin=0, lmax=0, n_inst=1, steps=1,
             thinc=False, gas="water", source=0, slope=1.0, cfl=0.4)
    c.update(kw)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # the smallest call: 32 blocks of 8x8 cells, one step; launch and latency only
        _case("tube8_mixed", mode="mixed", bsize=8, nx=16, ny=2),
        # the 1D-like two-fluid validation deck (512x32 cells), reference arithmetic
        _case("tube_fp64", nx=32, ny=2),
        # Mie-Grueneisen products against air: the general equation of state, odd block counts
        _case("jwl_fp64", nx=37, ny=5, gas="jwl"),
        # the benchmark's AMR mesh (three levels, coarse/fine records, walls), reference arithmetic
        _case("bubble_fp64", problem="bubble", gas="helium", lmin=4, lmax=6),
        # the same with the sharp-interface reconstruction and a heavy bubble
        _case("bubble_thinc_fp64", problem="bubble", lmin=4, lmax=6, thinc=True, gas="r22"),
        # the solver loop of the benchmark: ten steps with the time step kept on the device
        _case("bubble_run_mixed", kind="run", problem="bubble", mode="mixed", gas="helium", lmin=4, lmax=6, steps=10),
        # one step of a host-resident solver: the state crosses the host link both ways
        _case("bubble_host_mixed", kind="host", problem="bubble", mode="mixed", gas="helium", lmin=4, lmax=6),
        # a parameter study: many independent runs of uneven sizes, a time step each, in one call
        _case("droplets_mixed", problem="droplets", mode="mixed", n_inst=64),
        # 3D AMR with THINC, both precision forms
        _case("triple_mixed", problem="triple", mode="mixed", bsize=8, lmin=0, lmax=2, thinc=True, gas="air"),
        _case("triple_fp64", problem="triple", bsize=8, lmin=0, lmax=2, thinc=True, gas="air"),
        # the device side of a mesh adaptation: flags, remap, the new block table, boundary fill
        _case("adapt_3d", kind="adapt", problem="triple", bsize=8, lmin=0, lmax=2, gas="air"),
        # the datasets of one output file
        _case("fields_2d", kind="fields", problem="bubble", gas="helium", lmin=4, lmax=6),
    ]


def draw(rng):
    def odd_log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    problem = rng.choice(["tube", "bubble", "droplets", "triple"])
    mode = rng.choice(["fp64", "mixed"])
    kind = rng.choice(["step", "step", "step", "run", "host", "adapt", "fields"])
    slope = rng.choice([1.0, 1.0, 2.0])
    source = rng.choice([0, 0, 1])
    cfl = rng.choice([0.4, 0.3, 0.25])
    steps = rng.randint(2, 10) if kind == "run" else 1
    if kind == "adapt" and problem in ("tube", "droplets"):
        problem = "bubble"
    c = dict(kind=kind, mode=mode, steps=steps, slope=slope, source=source, cfl=cfl)
    if problem == "tube":
        b = rng.choice([8, 16, 16])
        return _case(None, problem=problem, bsize=b, nx=odd_log(4, 300 if b == 8 else 150), ny=odd_log(1, 12), gas=rng.choice(["water", "water", "jwl"]), **c)
    if problem == "bubble":
        b = rng.choice([8, 16, 16])
        lmin = rng.randint(3, 4)
        return _case(None, problem=problem, bsize=b, lmin=lmin, lmax=lmin + rng.randint(1, 2), thinc=rng.random() < 0.4, gas=rng.choice(["helium", "r22"]), **c)
    if problem == "droplets":
        return _case(None, problem=problem, n_inst=odd_log(2, 48), bsize=16, **c)
    c["steps"] = min(c["steps"], 3)
    return _case(None, problem=problem, bsize=8, lmin=0, lmax=2 if kind == "adapt" else rng.randint(0, 1 if mode == "fp64" else 2), thinc=rng.random() < 0.6, gas="air", **c)


# --------------------------------------------------------------------------- inputs
def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _centers(mesh, table):
    """Cell centres [n_owned, ncell, dim] of the owned blocks."""
    dev, b, dim, n = _device(), table.bsize, table.dim, table.n_owned
    dx = torch.as_tensor(mesh.level_dx(), device=dev)[torch.as_tensor(table.level[:n], device=dev).long()]
    c = torch.as_tensor(table.coord[:n], device=dev).to(F64)
    i = torch.arange(table.ncell, device=dev)
    cell = torch.stack([(i // b**e) % b for e in range(dim)], -1).to(F64)
    return (c[:, None, :dim] * b + cell[None] + 0.5) * dx[:, None, None]


def _refine(mesh, lmin, lmax, near):
    """Refine every block whose centre is within reach of the geometry: `near`
    gives the distance of points [n, dim] from it."""
    table = mesh.build()
    for level in range(lmin, lmax):
        w = mesh.cell_length(level) * table.bsize
        n = table.n_owned
        at = table.level[:n] == level
        pos = (table.coord[:n, : table.dim] + 0.5) * w
        pick = at & (near(pos) < 1.1 * w)
        mesh.refine([(level,) + tuple(int(v) for v in c) for c in table.coord[:n][pick]])
        mesh.balance()
        table = mesh.build()
    return table


def _bubble_distance(q):
    """Distance from the bubble's edge and the shock."""
    return np.minimum(np.abs(np.hypot(q[:, 0] - 1.0, q[:, 1] - 0.5) - 0.25), np.abs(q[:, 0] - 0.6))


def _triple_distance(q):
    """Distance from the planes between the three regions."""
    right = np.where(q[:, 0] > 1.0, np.abs(q[:, 1] - 1.5), np.hypot(q[:, 0] - 1.0, q[:, 1] - 1.5))
    return np.minimum(np.abs(q[:, 0] - 1.0), right)


def _mixture(P, a0, r0, r1):
    """S, PI, C1, C0 of the pressure-equilibrium mixture: p S = rho e - PI and
    rho c^2 S = p C1 + C0."""
    if P.eos == (0, 0):
        xi = [1.0 / (g - 1.0) for g in P.gamma]
        gp = [P.gamma[k] * P.pinf[k] * xi[k] for k in range(2)]
        S = a0 * xi[0] + (1.0 - a0) * xi[1]
        PI = a0 * gp[0] + (1.0 - a0) * gp[1]
        return S, PI, S + 1.0, PI
    out = [0.0, 0.0, 0.0, 0.0]
    for k, (a, ar) in enumerate(((a0, r0), (1.0 - a0, r1))):
        G, dG, f, df, rho = _law(P, k, a, ar)
        xi = 1.0 / G
        h = xi * (1.0 + rho * dG * xi)
        for j, t in enumerate((xi, -xi * f, h + 1.0, xi * rho * df - h * f)):
            out[j] = out[j] + a * t
    return out


def _law(P, k, a, ar):
    """G, dG/drho, f, df/drho of material k (p = G rho e + f) and its density."""
    if P.eos[k] == EOS["JWL"]:
        rho0, w, A1, A2, R1, R2, e0 = P.mg[k][:7]
        rho = torch.where(a > 0.0, (ar / torch.where(a > 0.0, a, torch.ones_like(a))).clamp_min(P.smallr), torch.full_like(a, rho0))
        x1, x2 = R1 * rho0 / rho, R2 * rho0 / rho
        E1, E2 = torch.exp(-x1), torch.exp(-x2)
        f = A1 * (1.0 - w / x1) * E1 + A2 * (1.0 - w / x2) * E2 - w * rho * e0
        df = (A1 * E1 * (x1 - w - w / x1) + A2 * E2 * (x2 - w - w / x2)) / rho - w * e0
        return torch.full_like(a, w), torch.zeros_like(a), f, df, rho
    rho = torch.where(a > 0.0, (ar / torch.where(a > 0.0, a, torch.ones_like(a))).clamp_min(P.smallr), torch.ones_like(a))
    return torch.full_like(a, P.gamma[k] - 1.0), torch.zeros_like(a), torch.full_like(a, -P.gamma[k] * P.pinf[k]), torch.zeros_like(a), rho


def _conservative(P, a0, r0, r1, p, vel):
    """[n, nv, ncell] from primitive fields [n, ncell]."""
    S, PI, _, _ = _mixture(P, a0, r0, r1)
    rho = r0 + r1
    ek = sum(v * v for v in vel)
    return torch.stack([rho, p * S + PI + 0.5 * rho * ek, *[rho * v for v in vel], a0, r0, 1.0 - a0, r1], 1)


def _waves(x, gen, dim, amp, env):
    """A few long waves under the envelope `env` (zero outside the disturbed region)."""
    out = torch.zeros_like(env)
    for _ in range(3):
        k = [float(gen.uniform(-25.0, 25.0)) for _ in range(dim)]
        ph = float(gen.uniform(0.0, 2.0 * math.pi))
        out = out + torch.sin(sum(k[e] * x[..., e] for e in range(dim)) + ph)
    return 1.0 + amp / 3.0 * out * env


def _bump(s):
    return (1.0 - s * s).clamp_min(0.0) ** 2


def _sigmoid(d, w):
    return 0.5 * (1.0 - torch.tanh(d / w))


EPS = 1e-6


def _problem(case, seed):
    """(mesh, table, params, U with its outside blocks filled) of a case."""
    gen = np.random.default_rng(seed)
    b, prob = case["bsize"], case["problem"]
    # THINC's exponents and thresholds are HydroParams' defaults
    base = dict(bsize=b, slope_type=case["slope"], cfl=case["cfl"], source_term=case["source"], thinc=int(case["thinc"]))
    if prob == "tube":
        mesh = BlockMesh(2, b, (case["nx"], case["ny"]), (False, True), 0, 0, scaling=1.0 / case["nx"])
        table = mesh.build()
        jwl = case["gas"] == "jwl"
        P = HydroParams(dim=2, gamma=(3.0, 1.4) if jwl else (4.4, 1.4), pinf=(0.0, 0.0) if jwl else (6e8, 0.0),
                        eos=(EOS["JWL"], 0) if jwl else (0, 0), mg=(JWL, (0.0,) * 8),
                        bc=(BC_ZERO_GRADIENT, BC_ZERO_GRADIENT) + (BC_PERIODIC,) * 4, level_dx=table.level_dx, **base)
        x = _centers(mesh, table)
        h = float(mesh.cell_length(0))
        xi = 0.5 + 2.0 * h * torch.sin(2.0 * math.pi * x[..., 1] / (case["ny"] * b * h) + gen.uniform(0, 6.28))
        d = x[..., 0] - xi
        a0 = EPS + (1.0 - 2.0 * EPS) * _sigmoid(d, 1.5 * h)
        env = _bump((x[..., 0] - 0.45) / 0.3)
        rho = (1.6 * JWL[0], 1.0) if jwl else (1000.0, 50.0)
        p = torch.where(d < 0, 2e10 if jwl else 1e9, 1e5) * _waves(x, gen, 2, 0.1, env)
        r0, r1 = a0 * rho[0] * _waves(x, gen, 2, 0.05, env), (1.0 - a0) * rho[1] * _waves(x, gen, 2, 0.05, env)
        vel = [gen.uniform(20.0, 60.0) * env * _waves(x, gen, 2, 0.5, env), 10.0 * (_waves(x, gen, 2, 1.0, env) - 1.0)]
    elif prob == "bubble":
        mesh = BlockMesh(2, b, (4, 1), (False, False), case["lmin"], case["lmax"], scaling=1.0)
        xc, rad, xs = 1.0 + gen.uniform(-0.01, 0.01), 0.25 * gen.uniform(0.97, 1.03), 0.6 + gen.uniform(-0.01, 0.01)
        table = _refine(mesh, case["lmin"], case["lmax"], _bubble_distance)
        gb, rb = {"helium": (1.648, 0.138), "r22": (1.249, 3.1538)}[case["gas"]]
        P = HydroParams(dim=2, gamma=(1.4, gb), bc=(BC_ZERO_GRADIENT,) * 2 + (BC_WALL,) * 2 + (BC_PERIODIC,) * 2, level_dx=table.level_dx, **base)
        x = _centers(mesh, table)
        h = float(mesh.cell_length(case["lmax"]))
        dr = torch.sqrt((x[..., 0] - xc) ** 2 + (x[..., 1] - 0.5) ** 2) - rad
        a0 = 1.0 - (EPS + (1.0 - 2.0 * EPS) * _sigmoid(dr, 2.0 * h))
        # the gas behind a Mach 1.22 shock at xs, disturbed; the gas ahead of it at rest but for the bubble
        m2 = 1.22**2
        p2, rho2 = 1.0 + 2.8 / 2.4 * (m2 - 1.0), 2.4 * m2 / (0.4 * m2 + 2.0)
        u2 = math.sqrt(1.4) * 2.0 * (m2 - 1.0) / (2.4 * 1.22)
        post = _sigmoid(x[..., 0] - xs, 1.0 * h)
        env = post * _bump((x[..., 0] - xs + 0.1) / 0.6) + 0.3 * _bump(dr / 0.15)
        comp = (1.0 + (rho2 - 1.0) * post) * _waves(x, gen, 2, 0.1, env)
        p = (1.0 + (p2 - 1.0) * post) * _waves(x, gen, 2, 0.1, env)
        r0, r1 = a0 * comp, (1.0 - a0) * rb * comp
        vel = [u2 * post * _waves(x, gen, 2, 0.3, env), 0.2 * (_waves(x, gen, 2, 1.0, env) - 1.0)]
    elif prob == "triple":
        mesh = BlockMesh(3, b, (14, 6, 3), (False,) * 3, case["lmin"], case["lmax"], scaling=0.5)
        xs, ys = 1.0 + gen.uniform(0.0, 0.06), 1.5 + gen.uniform(0.0, 0.06)
        table = _refine(mesh, case["lmin"], case["lmax"], _triple_distance)
        P = HydroParams(dim=3, gamma=(1.5, 1.4), bc=(BC_ZERO_GRADIENT,) * 6, level_dx=table.level_dx, **base)
        x = _centers(mesh, table)
        h = float(mesh.cell_length(case["lmax"]))
        left = _sigmoid(x[..., 0] - xs, 1.5 * h)
        top = (1.0 - left) * (1.0 - _sigmoid(x[..., 1] - ys, 1.5 * h))
        a0 = EPS + (1.0 - 2.0 * EPS) * (1.0 - top)
        env = _bump((x[..., 0] - xs) / 1.5)
        rho = (1.0 - 0.875 * top) * _waves(x, gen, 3, 0.1, env)
        p = (0.1 + 0.9 * left) * _waves(x, gen, 3, 0.1, env)
        r0, r1 = a0 * rho, (1.0 - a0) * rho
        vel = [0.4 * env * _waves(x, gen, 3, 0.5, env)] + [0.1 * (_waves(x, gen, 3, 1.0, env) - 1.0) for _ in range(2)]
    else:
        return _droplets(case, gen, base)
    U = torch.zeros((table.n_total, table.nv, table.ncell), dtype=F64, device=_device())
    U[: table.n_owned] = _conservative(P, a0, r0, r1, p, vel)
    _fill(table, P, U)
    return mesh, table, P, U


def _droplets(case, gen, base):
    """Independent periodic droplet runs of sides 64 to 512 in one block table."""
    tables, parts, P = [], [], None
    meshes = {}
    sides = np.random.default_rng(case["n_inst"])
    for _ in range(case["n_inst"]):
        level = int(sides.integers(2, 6))
        if level not in meshes:
            m = BlockMesh(2, 16, (1, 1), (True, True), level, level, scaling=1.0)
            t = m.build()
            meshes[level] = (m, t, _centers(m, t))
        mesh, table, x = meshes[level]
        P = P or HydroParams(dim=2, gamma=(4.4, 1.4), pinf=(6e8, 0.0), bc=(BC_PERIODIC,) * 6, level_dx=table.level_dx, **base)
        h = float(mesh.cell_length(level))
        r = torch.sqrt(((x - 0.5) ** 2).sum(-1))
        rad = gen.uniform(0.15, 0.3)
        a0 = EPS + (1.0 - 2.0 * EPS) * _sigmoid(r - rad, 2.0 * h)
        env = _bump((r - rad) / 0.2)
        r0, r1 = a0 * 1000.0 * _waves(x, gen, 2, 1e-3, env), (1.0 - a0) * _waves(x, gen, 2, 0.05, env)
        p = 1e5 * _waves(x, gen, 2, 0.1, env)
        vel = [gen.uniform(-1.0, 1.0) * _waves(x, gen, 2, 0.2, env) for _ in range(2)]
        tables.append(table)
        parts.append(_conservative(P, a0, r0, r1, p, vel))
    table = concat_tables(tables)
    return None, table, P, torch.cat(parts).contiguous()


# fields of an output file: the state's variables, then pressure, sound speed, velocity
FIELDS = [0, 1, 2, 3, 4, 5, 6, 7, 65, 66, 69, 70]


def _names(table):
    mom = ["rho_u", "rho_v", "rho_w"][: table.dim]
    return ["rho", "rho_E", *mom, "alpha0", "alpha0_rho0", "alpha1", "alpha1_rho1"]


def _views(table, U, n):
    return {k: U[:n, v] for v, k in enumerate(_names(table))}


def prepare(case, seed):
    mesh, table, P, U = _problem(case, seed)
    s = {"case": case, "table": table, "U": U}
    kind = case["kind"]
    if kind == "adapt":
        s["old"] = GodunovImplemGB300(P, table)
        rt, new = _adapted(case, mesh, table)
        s["rt"], s["new_table"] = rt, new
        s["new"] = GodunovImplemGB300(P, new)
        s["U_new"] = torch.zeros((new.n_total, new.nv, new.ncell), dtype=F64, device=U.device)
        s["out"] = _views(new, s["U_new"], new.n_total)
        return s
    s["impl"] = GodunovImplemGB300(P, table)
    n = table.n_owned
    if kind == "fields":
        s["out"] = torch.zeros((len(FIELDS), n, table.ncell), dtype=F64, device=U.device)
        return s
    dt = P.cfl / _inv_dt(table, P, U)
    if kind == "host":
        s["U"] = U.cpu().pin_memory()
        s["U2"] = torch.zeros(U.shape, dtype=F64).pin_memory()
        s["dt"] = dt.cpu().numpy()
        s["inv"] = torch.zeros(table.n_inst, dtype=F64).pin_memory()
    else:
        s["U2"] = torch.zeros_like(U)
        s["dt"] = dt
        s["inv"] = torch.zeros(table.n_inst, dtype=F64, device=U.device)
    if kind == "run":
        s["work"] = U.clone()
        s["hist"] = torch.zeros((case["steps"], table.n_inst), dtype=F64, device=U.device)
        s["out"] = {**_views(table, s["work"], n), "dt": s["hist"]}
    else:
        s["out"] = {**_views(table, s["U2"], n), "inv_dt": s["inv"]}
    return s


def run(s):
    case = s["case"]
    kind, mode = case["kind"], case["mode"]
    if kind == "step":
        s["impl"].do_time_step_dev(s["U"], s["U2"], s["dt"], mode=mode, inv_dt_out=s["inv"])
        return s["out"]
    if kind == "run":
        s["work"].copy_(s["U"])
        s["impl"].run(s["work"], s["U2"], case["steps"], mode=mode, dt_hist=s["hist"])
        return s["out"]
    if kind == "host":
        s["impl"].do_time_step_host(s["U"], s["U2"], s["dt"], mode=mode, inv_dt_out=s["inv"])
        return s["out"]
    if kind == "fields":
        s["impl"].pack_fields(s["U"], FIELDS, num_octs=s["table"].n_owned, out=s["out"])
        return {"fields": s["out"]}
    old, new = s["old"], s["new"]
    old.fill_outside_quadrants(s["U"])
    flags = old.refine_flags(s["U"], level_min=case["lmin"], level_max=case["lmax"])
    old.remap(s["rt"], s["U"], s["U_new"])
    new.resize_auxiliary_data(s["new_table"])
    new.fill_outside_quadrants(s["U_new"])
    return {**s["out"], "flags": flags}


def _adapted(case, mesh, table):
    """One adaptation: blocks the interface has left coarsen, some ahead of it refine."""
    n = table.n_owned
    c, lev = table.coord[:n], table.level[:n]
    w = np.array([mesh.cell_length(int(k)) * table.bsize for k in lev])
    near = (_bubble_distance if case["problem"] == "bubble" else _triple_distance)((c[:, : table.dim] + 0.5) * w[:, None])
    flags = np.where(near < 0.6 * w, 2, 1)
    flags[(near > 0.6 * w) & (c[:, 0] // 2 % 4 >= 2)] = 0
    flags[(near < 4.0 * w) & (c[:, 0] % 8 >= 6) & (c[:, 1] % 4 >= 2)] = 2
    flags[(flags == 2) & (lev >= mesh.level_max)] = 1
    flags[(flags == 0) & (lev <= mesh.level_min)] = 1
    rt = mesh.adapt(flags.astype(np.int8))
    return rt, mesh.build()


def work(case):
    """One read of the state and one write of the result; the arithmetic of a
    step counted from the scheme's formulas (per cell and step)."""
    table = _sizes(case)
    cells, dim = table["cells"], table["dim"]
    nv = 8 if dim == 2 else 9
    if case["kind"] == "fields":
        return {"bytes": cells * 8 * (nv + len(FIELDS)), "flops": cells * 60}
    if case["kind"] == "adapt":
        return {"bytes": cells * 8 * (3 * nv), "flops": cells * 30 * dim}
    per_step = 600 if dim == 2 else 1000
    return {"bytes": cells * 16 * nv * case["steps"], "flops": cells * per_step * case["steps"]}


_SIZES = {}


def _sizes(case):
    key = tuple(sorted((k, v) for k, v in case.items() if k != "name"))
    if key not in _SIZES:
        if case["problem"] == "tube":
            _SIZES[key] = {"cells": case["nx"] * case["ny"] * case["bsize"] ** 2, "dim": 2}
        else:
            table = _problem(case, 1)[1]
            _SIZES[key] = {"cells": table.owned_cells(), "dim": table.dim}
    return _SIZES[key]


# --------------------------------------------------------------------------- exact
def _fill(table, P, U):
    """Boundary values of the outside blocks: the last face that applies copies
    its boundary layer (zero gradient) or mirrors the block (wall)."""
    b, dim, n = table.bsize, table.dim, table.n_owned
    if not table.n_outside:
        return
    i = np.arange(table.ncell)
    cell = [(i // b**e) % b for e in range(3)]
    last = np.full(table.n_outside, -1)
    for f in range(2 * dim):
        if P.bc[f] in (BC_ZERO_GRADIENT, BC_WALL):
            last[(table.out_border[:, f] != 0) & (table.out_normal[:, f >> 1] != 0)] = f
    for f in range(2 * dim):
        o = np.nonzero(last == f)[0]
        if not o.size:
            continue
        d = f >> 1
        c = list(cell)
        c[d] = np.full_like(i, b - 1 if f & 1 else 0) if P.bc[f] == BC_ZERO_GRADIENT else b - 1 - cell[d]
        at = torch.as_tensor(c[0] + b * (c[1] + (b * c[2] if dim == 3 else 0)), device=U.device)
        v = U[torch.as_tensor(table.out_src[o], device=U.device).long()][:, :, at]
        if P.bc[f] == BC_WALL:
            v[:, 2 + d] = -v[:, 2 + d]
        U[torch.as_tensor(n + o, device=U.device)] = v


def _ghosted(table, U):
    """Conservative states of the owned blocks with two ghost layers,
    [n, nv, (z,) y, x]: a copy of a same-level or coarser cell, the mean of the
    2^dim finer ones."""
    b, dim, n, dev = table.bsize, table.dim, table.n_owned, U.device
    g = b + 4
    nv = table.nv
    V = U.view(table.n_total, nv, *([b] * dim))
    W = torch.zeros((n, nv) + (g,) * dim, dtype=F64, device=dev)
    W[(slice(None), slice(None)) + (slice(2, b + 2),) * dim] = V[:n]
    rel_all = torch.as_tensor(table.nbr_rel, device=dev).long()
    nbr_all = torch.as_tensor(table.nbr, device=dev).long()
    coord = torch.as_tensor(table.coord[:n], device=dev).long()
    for s in range(3**dim):
        d = [(s // 3**e) % 3 - 1 for e in range(dim)]
        if not any(d):
            continue
        rng = [torch.arange(-2, 0) if k < 0 else torch.arange(b, b + 2) if k > 0 else torch.arange(b) for k in d]
        rng = [r.to(dev) for r in rng]

        def along(e, t):  # t: [m or 1, len_e] on axis e of an [m, (z,) y, x] grid
            shape = [t.shape[0]] + [1] * dim
            shape[dim - e] = t.shape[1]
            return t.view(shape)

        for rel in (-1, 0, 1):
            blk = torch.nonzero(rel_all[:, s] == rel)[:, 0]
            if not blk.numel():
                continue
            v = [(rng[e] - d[e] * b)[None] for e in range(dim)]
            one = (slice(None),) + (None,) * dim
            if rel <= 0:
                if rel < 0:
                    v = [((coord[blk, e] + d[e]) & 1)[:, None] * (b // 2) + (v[e] >> 1) for e in range(dim)]
                ix = [along(e, v[e]) for e in range(dim)]
                val = V[(nbr_all[blk, s, 0][one], slice(None)) + tuple(ix[e] for e in reversed(range(dim)))]
            else:
                ch = [along(e, 2 * v[e] // b) for e in range(dim)]
                f0 = [along(e, 2 * v[e] % b) for e in range(dim)]
                src = nbr_all[blk, s][one + (slice(None),)].expand(blk.numel(), *[r.numel() for r in reversed(rng)], 2**dim)
                kid = sum(ch[e] << e for e in range(dim)).expand(src.shape[:-1])
                src = torch.gather(src, -1, kid[..., None])[..., 0]
                val = 0.0
                for o in range(2**dim):
                    val = val + V[(src, slice(None)) + tuple(f0[e] + ((o >> e) & 1) for e in reversed(range(dim)))]
                val = val / 2**dim
                val[..., dim + 4] = 1.0 - val[..., dim + 2]
                val[..., 0] = val[..., dim + 3] + val[..., dim + 5]
            # (advanced indices split by a slice come first: val is [m, (z,) y, x, nv])
            sl = tuple(slice(int(rng[e][0]) + 2, int(rng[e][-1]) + 3) for e in reversed(range(dim)))
            W[(blk, slice(None)) + sl] = torch.movedim(val, -1, 1)
    return W


def _primitive(P, W, dim):
    """r0 r1 p vel... [n, 3 + dim, ...], clipped volume fraction, and sound speed."""
    d = W[:, 0].clamp_min(P.smallr)
    vel = [W[:, 2 + e] / d for e in range(dim)]
    a0, r0, r1 = W[:, dim + 2], W[:, dim + 3], W[:, dim + 5]
    S, PI, _, _ = _mixture(P, a0, r0, r1)
    p = (W[:, 1] - 0.5 * d * sum(v * v for v in vel) - PI) / S
    z = torch.zeros_like(r0)
    r0, r1 = torch.where(r0 < 1e-12, z, r0), torch.where(r1 < 1e-12, z, r1)
    a = a0.clamp(0.0, 1.0)
    a = torch.where(a < 1e-12, z, torch.where(a > 1.0 - 1e-12, z + 1.0, a))
    S, _, C1, C0 = _mixture(P, a, r0, r1)
    c = torch.sqrt(((p * C1 + C0) / (d * S)).clamp_min(0.0))
    return torch.stack([r0, r1, p, *vel], 1), a, c


def _per_block(table, values):
    dev = _device()
    return torch.as_tensor(np.asarray(values)[table.level[: table.n_owned]], device=dev)


def _inv_dt(table, P, U, blocks=None):
    n, dim = table.n_owned, table.dim
    q, _, c = _primitive(P, U[:n], dim)
    dx = _per_block(table, P.level_dx)[:, None]
    rate = sum(c + q[:, 3 + e].abs() for e in range(dim)) / dx
    inst = torch.as_tensor(table.inst[:n], device=U.device).long()
    return torch.zeros(table.n_inst, dtype=F64, device=U.device).scatter_reduce(0, inst, rate.amax(1), "amax")


def _limited(P, q, m, p):
    """Minmod (slope_type 1) or monotonised central (2) slope from the two neighbours."""
    l, r, c = P.slope_type * (q - m), P.slope_type * (p - q), 0.5 * (p - m)
    lim = torch.where(l * r <= 0.0, torch.zeros_like(c), torch.minimum(l.abs(), r.abs()))
    return torch.where(c >= 0.0, 1.0, -1.0) * torch.minimum(lim, c.abs())


def _thinc(P, q, A, a0, ring, ax, dim, side, hs):
    """THINC reconstruction of one side along an axis (see Shyue & Xiao 2014)."""
    aP, aM = ring(A, {ax: 1}), ring(A, {ax: -1})
    req = (a0 > P.thinc_eps) & (a0 < 1.0 - P.thinc_eps) & ((aP - a0) * (a0 - aM) > 0.0)
    grad = []
    for e in range(dim):
        t = 0.0
        others = [o for o in range(dim) if o != e]
        for k in range(3 ** len(others)):
            off = {o: (k // 3**j) % 3 - 1 for j, o in enumerate(others)}
            w = math.prod(2.0 - abs(v) for v in off.values())
            t = t + w * (ring(A, {**off, e: 1}) - ring(A, {**off, e: -1}))
        grad.append(t)
    nrm = torch.sqrt(sum(t * t for t in grad))
    nd = torch.where(nrm > 0.0, (grad[ax] / torch.where(nrm > 0.0, nrm, torch.ones_like(nrm))).abs(), torch.zeros_like(nrm))
    beta = P.thinc_beta * nd + 0.01
    Aa, Bb = 0.5 * (aP + aM), 0.5 * (aP - aM)
    B1 = torch.where(req, Bb, torch.ones_like(Bb))
    C = torch.tanh(0.5 * beta)
    D = torch.tanh(torch.where(req, 0.5 * beta * (a0 - Aa) / B1, torch.zeros_like(beta)))
    af = Aa + side * Bb * (C + side * D / C) / (1.0 + side * D)
    a_s = torch.where(req, a0, torch.full_like(a0, 0.5))
    r0 = ring(q[:, 0]) * (1.0 + (af - a0) / a_s) + hs[:, 0]
    r1 = ring(q[:, 1]) * (1.0 + (a0 - af) / (1.0 - a_s)) + hs[:, 1]
    return req, af, r0, r1


def _hllc(P, L, al, R, ar, ax, dim):
    """HLLC fluxes r0 r1 a0 a1 e mom... u* of the states L, R [n, 3 + dim, ...]."""
    side = []
    for q, a in ((L, al), (R, ar)):
        S, PI, C1, C0 = _mixture(P, a, q[:, 0], q[:, 1])
        rho = (q[:, 0] + q[:, 1]).clamp_min(P.smallr)
        p = torch.maximum(q[:, 2], rho * P.smallc**2)
        c = torch.sqrt(((p * C1 + C0) / (rho * S)).clamp_min(0.0)).clamp_min(P.smallc)
        E = p * S + PI + 0.5 * rho * sum(q[:, 3 + e] ** 2 for e in range(dim))
        side.append((rho, p, q[:, 3 + ax], c, E))
    (rl, pl, ul, cl, El), (rr, pr, ur, cr, Er) = side
    cm = torch.maximum(cl, cr)
    SL, SR = torch.minimum(ul, ur) - cm, torch.maximum(ul, ur) + cm
    kl, kr = rl * (ul - SL), rr * (SR - ur)
    us = (kr * ur + kl * ul + (pl - pr)) / (kr + kl)
    ps = (kr * pl + kl * pr + kl * kr * (ul - ur)) / (kr + kl)
    w = torch.where

    def star(q, rho, p, u, E, S):
        f = (S - u) / (S - us)
        return q[:, 0] * f, q[:, 1] * f, rho * f, us, ps, ((S - u) * E - p * u + ps * us) / (S - us)

    opts = [(L[:, 0], L[:, 1], rl, ul, pl, El), star(L, rl, pl, ul, El, SL), star(R, rr, pr, ur, Er, SR), (R[:, 0], R[:, 1], rr, ur, pr, Er)]
    r0, r1, ro, u, p, E = (w(SL > 0, a, w(us > 0, b, w(SR > 0, c, d))) for a, b, c, d in zip(*opts))
    m = (r0 + r1) * u
    up = m > 0
    a = w(up, al, ar)
    mom = [ro * u * u + p if e == ax else m * w(up, L[:, 3 + e], R[:, 3 + e]) for e in range(dim)]
    return torch.stack([r0 * u, r1 * u, u * a, u * (1.0 - a), (E + p) * u, *mom, u], 1)


def _reflux(table, F, ax):
    """Coarse faces next to finer blocks take the fine faces' fluxes (scaled by
    the fine dt/dx, hence / 2 after the mean)."""
    b, dim = table.bsize, table.dim
    dev = F.device
    tang = [e for e in reversed(range(dim)) if e != ax]  # array order
    axis = 2 + (dim - 1 - ax)
    new = F.clone()
    for side in (0, 1):
        s = sum((1 if e != ax else 2 * side) * 3**e for e in range(dim))
        blk = np.nonzero(table.nbr_rel[:, s] == 1)[0]
        if not blk.size:
            continue
        big = torch.zeros((blk.size, F.shape[1]) + (2 * b,) * len(tang), dtype=F64, device=dev)
        for k in range(2 ** len(tang)):
            kid = (1 - side) << ax
            sl = []
            for j, e in enumerate(tang):
                c = (k >> j) & 1
                kid |= c << e
                sl.append(slice(c * b, (c + 1) * b))
            fine = torch.as_tensor(table.nbr[blk, s, kid], device=dev).long()
            big[(slice(None), slice(None)) + tuple(sl)] = F[fine].select(axis, b if side == 0 else 0)
        mean = big.view(*big.shape[:2], *[n for _ in tang for n in (b, 2)])
        for j in reversed(range(len(tang))):
            mean = mean.mean(3 + 2 * j)
        at = torch.as_tensor(blk, device=dev)
        part = new[at]
        part.select(axis, b if side else 0).copy_(0.5 * mean)
        new[at] = part
    return new


def _step(table, P, U, dt):
    """One timestep of every owned block, and the CFL rate of the new state."""
    b, dim, n, dev = table.bsize, table.dim, table.n_owned, U.device
    W = _ghosted(table, U)
    q, A, _ = _primitive(P, W, dim)
    del W
    inst = torch.as_tensor(table.inst[:n], device=dev).long()
    lam = (dt[inst] / _per_block(table, P.level_dx)).view(n, *([1] * dim))

    def ring(T, off={}, lo=1, hi=b + 3):
        """The ring (one ghost layer) of T's ghosted trailing axes, shifted."""
        sl = tuple(slice(lo + off.get(e, 0), hi + off.get(e, 0)) for e in reversed(range(dim)))
        return T[(Ellipsis,) + sl]

    c_ = ring(q)
    a0 = ring(A)
    dq = [_limited(P, c_, ring(q, {e: -1}), ring(q, {e: 1})) for e in range(dim)]
    hs = torch.zeros_like(c_)
    if P.integrator == 0:
        r0, r1, p = c_[:, 0], c_[:, 1], c_[:, 2]
        rho = r0 + r1
        S, _, C1, C0 = _mixture(P, a0, r0, r1)
        rc2 = rho * ((p * C1 + C0) / (rho * S)).clamp_min(0.0)
        sr = sp = 0.0
        sv = [0.0] * dim
        for e in range(dim):
            u, dqe = c_[:, 3 + e], dq[e]
            sr = sr - u * (dqe[:, 0] + dqe[:, 1]) - dqe[:, 3 + e] * rho
            sp = sp - u * dqe[:, 2] - dqe[:, 3 + e] * rc2
            for f in range(dim):
                sv[f] = sv[f] - u * dqe[:, 3 + f] - (dqe[:, 2] / rho if f == e else 0.0)
        hs = 0.5 * lam[:, None] * torch.stack([sr * a0, sr * (1.0 - a0), sp, *sv], 1)
    flux = []
    for ax in range(dim):
        states = []
        for side in (1.0, -1.0):
            s = c_ + 0.5 * side * dq[ax] + hs
            a = a0
            if P.thinc:
                req, af, t0, t1 = _thinc(P, q, A, a0, ring, ax, dim, side, hs)
                s = torch.stack([torch.where(req, t0, s[:, 0]), torch.where(req, t1, s[:, 1]), *s[:, 2:].unbind(1)], 1)
                a = torch.where(req, af, a0)
            else:
                s = torch.cat([s[:, :2].clamp_min(P.smallr), s[:, 2:]], 1)
            states.append((s, a))

        def cut(T, lo):
            sl = tuple(slice(lo, lo + b + 1) if e == ax else slice(1, b + 1) for e in reversed(range(dim)))
            return T[(Ellipsis,) + sl]

        (sl_, al), (sr_, ar) = states
        F = _hllc(P, cut(sl_, 0), cut(al, 0), cut(sr_, 1), cut(ar, 1), ax, dim) * lam[:, None]
        flux.append(_reflux(table, F, ax))
    V = U[:n].view(n, table.nv, *([b] * dim))
    new = V.clone()
    iA0, iR0, iA1, iR1 = dim + 2, dim + 3, dim + 4, dim + 5
    k0, k1 = _source(P, V, dim)
    for ax in range(dim):
        axis = 2 + (dim - 1 - ax)
        lo, hi = flux[ax].narrow(axis, 0, b), flux[ax].narrow(axis, 1, b)
        d = lo - hi
        dus = lo[:, -1] - hi[:, -1]
        new[:, iR0] += d[:, 0]
        new[:, iR1] += d[:, 1]
        new[:, iA0] += d[:, 2] - k0 * V[:, iA0] * dus
        new[:, iA1] += d[:, 3] - k1 * V[:, iA1] * dus
        for v in (iR0, iR1, iA0, iA1):
            new[:, v] = torch.where(new[:, v] < 1e-12, torch.zeros_like(dus), new[:, v])
        for v in (iA0, iA1):
            new[:, v] = torch.where(new[:, v] > 1.0 - 1e-12, torch.ones_like(dus), new[:, v])
        new[:, 1 : 2 + dim] += d[:, 4 : 5 + dim]
    tot = new[:, iA0] + new[:, iA1]
    new[:, iA0] /= tot
    new[:, iA1] /= tot
    new[:, 0] = new[:, iR0] + new[:, iR1]
    out = new.reshape(n, table.nv, table.ncell)
    return out, _inv_dt(table, P, out)


def _pressure(P, V, dim):
    """Pressure with the density of the partial densities in the internal energy."""
    dd, d = V[:, 0].clamp_min(P.smallr), (V[:, dim + 3] + V[:, dim + 5]).clamp_min(P.smallr)
    S, PI, _, _ = _mixture(P, V[:, dim + 2], V[:, dim + 3], V[:, dim + 5])
    return (V[:, 1] - d * 0.5 * sum((V[:, 2 + e] / dd) ** 2 for e in range(dim)) - PI) / S


def _source(P, V, dim):
    """Volume-fraction source factors: 1, or 1 - Kbar/K_k (Miller & Puckett)."""
    if P.source_term != 1:
        return 1.0, 1.0
    p, K = _pressure(P, V, dim), []
    for k in range(2):
        a, ar = V[:, dim + 2 + 2 * k], V[:, dim + 3 + 2 * k]
        G, dG, f, df, rho = _law(P, k, a, ar)
        K.append((1.0 + rho * dG / G) * (p - f) + rho * df + G * p)
    kbar = 1.0 / (V[:, dim + 2] / K[0] + V[:, dim + 4] / K[1])
    return 1.0 - kbar / K[0], 1.0 - kbar / K[1]


def exact(case, seed):
    mesh, table, P, U = _problem(case, seed)
    kind, n, dim = case["kind"], table.n_owned, table.dim
    if kind == "fields":
        V = U[:n]
        q, _, c = _primitive(P, V, dim)
        return {"fields": torch.stack([V[:, v] for v in range(8)] + [_pressure(P, V, dim), c, q[:, 3], q[:, 4]])}
    if kind == "adapt":
        rt, new = _adapted(case, mesh, table)
        return {**_views(new, _remapped(table, new, rt, P, U), new.n_total), "flags": None}
    if kind == "run":
        hist = []
        inv = _inv_dt(table, P, U)
        for _ in range(case["steps"]):
            dt = P.cfl / inv
            hist.append(dt)
            U[:n], inv = _step(table, P, U, dt)
            _fill(table, P, U)
        return {**_views(table, U, n), "dt": torch.stack(hist)}
    out, inv = _step(table, P, U, P.cfl / _inv_dt(table, P, U))
    return {**_views(table, out, n), "inv_dt": inv}


def _remapped(table, new, rt, P, U):
    """The state on the adapted mesh: copied, child of a parent cell, or mean of the children."""
    b, dim, dev = table.bsize, table.dim, U.device
    V = U.view(table.n_total, table.nv, *([b] * dim))
    kind, src = torch.as_tensor(rt.kind, device=dev), torch.as_tensor(rt.src, device=dev).long()
    out = torch.zeros((new.n_total, new.nv) + (b,) * dim, dtype=F64, device=dev)
    at = torch.nonzero(kind == 0)[:, 0]
    out[at] = V[src[at, 0]]
    for ch in range(2**dim):
        at = torch.nonzero((kind == 1) & (src[:, 1] == ch))[:, 0]
        part = V[src[at, 0]]
        for e in range(dim):
            axis = 2 + (dim - 1 - e)
            part = part.narrow(axis, ((ch >> e) & 1) * (b // 2), b // 2).repeat_interleave(2, axis)
        out[at] = part
        at = torch.nonzero(kind == 2)[:, 0]
        part = V[src[at, ch]]
        for e in range(dim):
            part = part.unfold(2 + (dim - 1 - e), 2, 2).mean(-1)
        sl = tuple(slice(((ch >> e) & 1) * (b // 2), ((ch >> e) & 1) * (b // 2) + b // 2) for e in reversed(range(dim)))
        out[(at, slice(None)) + sl] = part
    at = torch.nonzero(kind == 2)[:, 0]
    out[at, dim + 4] = 1.0 - out[at, dim + 2]
    out[at, 0] = out[at, dim + 3] + out[at, dim + 5]
    out = out.view(new.n_total, new.nv, new.ncell)
    _fill(new, P, out)
    return out
