"""Performance cases: what a program that uses this package has it do.

Every case goes through the public host interface (``FvmSolverCuda``,
``BatchSolver``, ``AdjointSolver``).  ``listed`` names fixed cases, ``draw``
gives one more of the same ranges, ``prepare`` builds what a program holds
before the call, ``run`` makes one pass, ``work`` states the bytes and
operations one pass cannot do without, and ``exact`` restates the pass in
64-bit torch operations, written from the discretisation alone.

Inputs are synthetic and seeded: box buildings on a street lattice, a
logarithmic inflow with a 5 % Gaussian perturbation, and a velocity with the
same turbulence intensity.
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch
from torch.utils.checkpoint import checkpoint

from unitywindsimulation_b200 import FvmSolverCuda, _lib, cases
from unitywindsimulation_b200.adjoint import AdjointSolver, Objective
from unitywindsimulation_b200.config import default_config
from unitywindsimulation_b200.soft_mask import SoftBuildings
from unitywindsimulation_b200.solver import BatchSolver

KAPPA = 0.41
FIXED, ZERO_GRAD, SYMMETRY = _lib.BND_FIXED_VALUE, _lib.BND_ZERO_GRAD, _lib.BND_SYMMETRY


# --------------------------------------------------------------- the cases
def _step(name, nx, ny, nz, **over):
    c = dict(name=name, kind="step", nx=nx, ny=ny, nz=nz, dx=0.5, ustar=0.5, z0=0.1, cs=0.1, nv=50, np=30, nc=2,
             piso=True, les=True, monitor=False, buildings=8, mu=1.5e-5, cfl=0.25)
    c.update(over)
    return c


def listed():
    return [
        # an interactive host steps a small courtyard scene, one cube: the
        # lowest latency a caller sees
        _step("cube_step", 64, 32, 48, buildings=1),
        # the wind-engineering validation building: few cells, a deeply
        # converged pressure (SIMPLE, 1000 sweeps)
        _step("building_step", 80, 40, 40, dx=1.0, ustar=1.67, z0=1.0, cs=0.18, nv=100, np=1000, nc=0, piso=False,
              buildings=1, cfl=0.5),
        # the default configuration's grid and sweep counts, no turbulence model
        _step("default_step", 100, 50, 100, nc=0, piso=False, les=False, np=400, mu=0.05, buildings=4),
        # the same, with the residual monitoring a user switches on to judge convergence
        _step("monitored_step", 100, 50, 100, nc=0, piso=False, les=False, np=400, mu=0.05, buildings=4,
              monitor=True),
        # a district voxelised at an odd size: no extent is a multiple of four
        _step("ragged_step", 149, 61, 103),
        # a visualiser that feeds measured inflow planes and draws every
        # frame: upload, step, velocity and pressure back in host memory
        dict(_step("frames_step", 128, 64, 96), kind="frames"),
        # the urban block of the benchmark
        _step("urban_step", 256, 96, 192, ustar=0.6, z0=0.3, cs=0.12, np=40, buildings=48, cfl=0.15),
        # the wind tunnel on a stretched mesh: 800 momentum, 2000 pressure sweeps
        dict(name="tunnel_step", kind="tunnel", nx=100, ny=50, nz=100, nv=800, np=2000, les=False),
        # many small scenes (one per wind direction) stepped together
        dict(name="small_batch", kind="batch", cases=16, nx0=48, nx1=72, ny0=24, ny1=40, nz0=48, nz1=72, grid_seed=5),
        # sixteen wind directions over a district, re-meshed per direction
        dict(name="directions_batch", kind="batch", cases=16, nx0=96, nx1=192, ny0=48, ny1=80, nz0=96, nz1=160,
             grid_seed=3),
        # forward and backward: gradient of the pedestrian wind objective
        # with respect to inflow and building heights over a short window
        dict(name="street_gradient", kind="gradient", nx=128, ny=64, nz=96, nv=50, np=30, steps=4, buildings=12),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step", "step", "step", "frames", "tunnel", "batch", "gradient"])
    if kind in ("step", "frames"):
        while True:
            nx, ny, nz = _log_int(rng, 40, 256), _log_int(rng, 20, 96), _log_int(rng, 40, 192)
            piso = rng.random() < 0.6
            c = _step("", nx, ny, nz, piso=piso, nc=2 if piso else 0, les=rng.random() < 0.7, nv=rng.randint(20, 100),
                      np=_log_int(rng, 20, 60) if piso else _log_int(rng, 40, 1000), buildings=rng.randint(1, 32))
            if not c["les"]:
                c["mu"] = 0.05
            c["kind"] = kind
            if work(c)["flops"] <= 1.8e10:
                break
    elif kind == "tunnel":
        c = dict(kind="tunnel", nx=2 * rng.randint(30, 52), ny=rng.randint(30, 50), nz=2 * rng.randint(30, 52),
                 nv=rng.randint(100, 700), np=rng.randint(300, 1700), les=rng.random() < 0.3)
    elif kind == "batch":
        small = rng.random() < 0.5
        lo, hi = (44, 72) if small else (90, 150)
        a, b = rng.randint(lo, hi - 10), rng.randint(20 if small else 40, 30 if small else 56)
        c = dict(kind="batch", cases=rng.randint(3, 16 if small else 10), nx0=a, nx1=a + rng.randint(0, hi - a), ny0=b,
                 ny1=b + rng.randint(0, 10), nz0=lo, nz1=lo + rng.randint(0, hi - lo), grid_seed=rng.randint(0, 10**6))
    else:
        c = dict(kind="gradient", nx=_log_int(rng, 40, 128), ny=_log_int(rng, 24, 64), nz=_log_int(rng, 40, 96),
                 nv=rng.randint(20, 50), np=rng.randint(20, 30), steps=rng.randint(2, 4), buildings=rng.randint(1, 8))
    c.pop("name", None)
    return c


# ------------------------------------------------------------------ inputs
def _log_u(y, ustar, z0):
    return ustar / KAPPA * np.log((y + z0) / z0)


def _lots(nx, nz, count, rng, margin):
    """Footprints (x0, x1, z0, z1), one per lot of a lattice of 16-cell
    blocks and 2-cell streets; a grid too small for one takes one box in its middle."""
    lx, lz = (nx - 2 * margin - 2) // 18, (nz - 2 * margin - 2) // 18
    if lx < 1 or lz < 1:
        return [(nx // 3, nx // 3 + 6, nz // 2 - 3, nz // 2 + 3)]
    out = []
    for k in rng.choice(lx * lz, size=min(count, lx * lz), replace=False):
        i, j = int(k) // lz, int(k) % lz
        wx, wz = int(rng.integers(6, 15)), int(rng.integers(6, 15))
        x0 = margin + 2 + 18 * i + int(rng.integers(0, 17 - wx))
        z0 = margin + 2 + 18 * j + int(rng.integers(0, 17 - wz))
        out.append((x0, x0 + wx, z0, z0 + wz))
    return out


def _margin(nx, nz):
    return 10 if min(nx, nz) >= 96 else 6


def _scene(c, seed):
    """Flags, inlet plane, velocity and pressure of a uniform-grid case."""
    rng = np.random.default_rng([seed, 17])
    nx, ny, nz, dx = c["nx"], c["ny"], c["nz"], c["dx"]
    flags = np.zeros((nz, ny, nx), dtype=np.int32)
    for x0, x1, z0, z1 in _lots(nx, nz, c["buildings"], rng, _margin(nx, nz)):
        flags[z0:z1, :int(rng.integers(4, max(6, min(41, ny // 2)))), x0:x1] = 1
    u = _log_u((np.arange(ny) + 0.5) * dx, c["ustar"], c["z0"]).astype(np.float32)
    inlet = np.zeros((nz, ny, 3), dtype=np.float32)
    inlet[:, :, 0] = u * (1 + 0.05 * rng.standard_normal((nz, ny), dtype=np.float32))
    vel = rng.standard_normal((3, nz, ny, nx), dtype=np.float32)
    vel *= np.float32(0.05) * u[None, None, :, None]
    vel[0] += u[None, :, None]
    vel[:, flags == 1] = 0.0
    pres = np.float32(0.05) * rng.standard_normal((nz, ny, nx), dtype=np.float32)
    pres[flags == 1] = 0.0
    return dict(flags=flags, inlet=inlet, vel=vel, pres=pres, dt=float(np.float32(c["cfl"] * dx / float(u.max()))))


def _uniform_config(c, dt):
    return default_config(
        nx=c["nx"], ny=c["ny"], nz=c["nz"], dx=c["dx"], dt=dt, mu=c["mu"],
        solver_type=_lib.SOLVER_PISO if c["piso"] else _lib.SOLVER_SIMPLE, piso_correctors=c["nc"],
        turbulence=_lib.TURB_SMAGORINSKY if c["les"] else _lib.TURB_NONE, cs=c["cs"], vel_iters=c["nv"],
        pres_iters=c["np"], inflow_type=_lib.INFLOW_LOG, inflow_ustar=c["ustar"], inflow_z0=c["z0"],
        inflow_kappa=KAPPA, wind_speed=0.0, calc_residual=int(c["monitor"]), vel_tol=1e-15, pres_tol=1e-15)


def _members(c):
    """The scenes of a batch: extents spread over the case's ranges, LES + PISO."""
    rng = np.random.default_rng(c["grid_seed"])
    pick = lambda a, b: int(rng.integers(a // 8, b // 8 + 1)) * 8 if a % 8 == 0 and b % 8 == 0 else int(rng.integers(a, b + 1))  # noqa: E731
    return [_step("", pick(c["nx0"], c["nx1"]), pick(c["ny0"], c["ny1"]), pick(c["nz0"], c["nz1"]),
                  buildings=int(rng.integers(1, 24))) for _ in range(c["cases"])]


def _tunnel(c, seed):
    """Wind tunnel on the stretched mesh: constant inflow, one seeded box."""
    rng = np.random.default_rng([seed, 23])
    nx, ny, nz = c["nx"], c["ny"], c["nz"]
    flags = np.zeros((nz, ny, nx), dtype=np.int32)
    w, h = int(rng.integers(4, 8)), int(rng.integers(6, 12))
    x0, z0 = nx // 3 + int(rng.integers(0, 6)), nz // 2 - 2 + int(rng.integers(-3, 4))
    flags[z0:z0 + w, :h, x0:x0 + w] = 1
    side = lambda n: n // 4  # noqa: E731
    faces = [cases.stretched_faces(nx, 1.0, nx - 2 * side(nx), side(nx)), cases.stretched_faces(ny, 1.0, ny, 0),
             cases.stretched_faces(nz, 1.0, nz - 2 * side(nz), side(nz))]
    vel = np.float32(0.5) * rng.standard_normal((3, nz, ny, nx), dtype=np.float32)
    vel[0] += 10.0
    vel[:, flags == 1] = 0.0
    pres = np.float32(0.05) * rng.standard_normal((nz, ny, nx), dtype=np.float32)
    pres[flags == 1] = 0.0
    return dict(flags=flags, faces=faces, vel=vel, pres=pres)


_TUNNEL_VBC = (FIXED, ZERO_GRAD, SYMMETRY, SYMMETRY, SYMMETRY, SYMMETRY)
_TUNNEL_PBC = (ZERO_GRAD, FIXED, SYMMETRY, SYMMETRY, SYMMETRY, SYMMETRY)
_URBAN_VBC = (FIXED, ZERO_GRAD, FIXED, SYMMETRY, SYMMETRY, SYMMETRY)
_URBAN_PBC = (ZERO_GRAD, FIXED, ZERO_GRAD, SYMMETRY, SYMMETRY, SYMMETRY)


def _street(c, seed):
    """Soft buildings and inflow parameters of a gradient case."""
    rng = np.random.default_rng([seed, 31])
    nx, ny, nz, dx = c["nx"], c["ny"], c["nz"], 0.5
    ustar, z0 = float(np.float32(rng.uniform(0.4, 0.6))), float(np.float32(rng.uniform(0.08, 0.15)))
    dt = float(np.float32(0.25 * dx / _log_u((ny - 0.5) * dx, ustar, z0)))
    feet = _lots(nx, nz, c["buildings"], rng, _margin(nx, nz))
    soft = SoftBuildings(feet, rng.uniform(4.0, ny / 2, size=len(feet)), chi_max=50.0 / dt, width=1.0)
    w, d = min(32, nx // 3), min(32, nz // 3)
    obj = dict(x0=nx // 3, x1=nx // 3 + w, z0=nz // 3, z1=nz // 3 + d, y=3, window=c["steps"] // 2)
    return dict(ustar=ustar, z0=z0, dt=dt, soft=soft, obj=obj, dx=dx)


# ------------------------------------------------------- prepare, run, work
class _Cuda:
    """A device pointer torch can view; a tensor made of it keeps its owner alive."""

    def __init__(self, owner, ptr, shape):
        self.owner = owner
        self.__cuda_array_interface__ = dict(shape=shape, typestr="<f4", data=(ptr, False), version=3)


def _views(solver):
    """The solver's current velocity and pressure on the device, not copied."""
    d = solver.device_fields()
    addr = lambda p: ctypes.cast(p, ctypes.c_void_p).value  # noqa: E731
    return (torch.as_tensor(_Cuda(solver, addr(d.vel[0]), (3,) + solver.shape), device="cuda"),
            torch.as_tensor(_Cuda(solver, addr(d.pres), solver.shape), device="cuda"))


def _uniform_solver(c, seed):
    s = _scene(c, seed)
    g = FvmSolverCuda(_uniform_config(c, s["dt"]))
    g.InitFlags(s["flags"])
    g.set_inflow_plane(s["inlet"])
    g.set_state(s["vel"], s["pres"])
    return g, s


def prepare(case, seed):
    kind = case["kind"]
    if kind == "step":
        g, _ = _uniform_solver(case, seed)
        return dict(kind=kind, solver=g, monitor=case["monitor"])
    if kind == "frames":
        g, s = _uniform_solver(case, seed)
        pin = lambda *shape: torch.empty(shape, dtype=torch.float32, pin_memory=True).numpy()  # noqa: E731
        return dict(kind=kind, solver=g, inlet=s["inlet"], vel=pin(*g.shape, 4), pres=pin(*g.shape))
    if kind == "tunnel":
        s = _tunnel(case, seed)
        cfg = default_config(nx=case["nx"], ny=case["ny"], nz=case["nz"], dx=1.0, dt=0.02, mu=1.0, wind_speed=10.0,
                             turbulence=_lib.TURB_SMAGORINSKY if case["les"] else _lib.TURB_NONE,
                             vel_iters=case["nv"], pres_iters=case["np"], vel_bc=_TUNNEL_VBC, pres_bc=_TUNNEL_PBC)
        g = FvmSolverCuda(cfg)
        g.set_face_positions(*s["faces"])
        g.InitVelPresFields()
        g.SetFixedValueVelBndCond()
        g.InitFlags(s["flags"])
        g.set_state(s["vel"], s["pres"])
        return dict(kind=kind, solver=g, monitor=False)
    if kind == "batch":
        solvers = [_uniform_solver(m, seed * 64 + i)[0] for i, m in enumerate(_members(case))]
        return dict(kind=kind, solvers=solvers, batch=BatchSolver(solvers))
    s = _street(case, seed)
    cfg = _uniform_config(_step("", case["nx"], case["ny"], case["nz"], les=False, ustar=s["ustar"], z0=s["z0"],
                                nv=case["nv"], np=case["np"]), s["dt"])
    g = FvmSolverCuda(cfg)
    g.InitFlags(np.zeros((case["nz"], case["ny"], case["nx"]), dtype=np.int32))
    g.set_field(_lib.FIELD_DRAG, s["soft"].drag(case["nx"], case["ny"], case["nz"]).reshape(-1))
    return dict(kind="gradient", solver=g, adjoint=AdjointSolver(g), objective=Objective(**s["obj"]), soft=s["soft"],
                steps=case["steps"])


def run(state):
    kind = state["kind"]
    if kind == "batch":
        state["batch"].step(1)
        return [_views(s) for s in state["solvers"]]
    g = state["solver"]
    if kind == "gradient":
        # from the initial profile, as the gradient's inflow parameters set it
        g.InitVelPresFields()
        r = state["adjoint"].gradient(state["objective"], state["steps"], checkpoint_every=20, soft=state["soft"])
        return {k: r[k] for k in ("J", "dJ_dustar", "dJ_dz0", "dJ_ddrag", "dJ_dheights")}
    if kind == "frames":
        g.set_inflow_plane(state["inlet"])
        g.step_async(1)
        g.readback_begin(state["vel"], state["pres"], _lib.LAYOUT_XYZW)
        g.readback_wait()
        return state["vel"], state["pres"]
    g.Step(1)
    return _views(g) + (g.residuals(),) if state["monitor"] else _views(g)


def _step_flops(n, nv, np_, nc, les):
    # per cell and sweep: momentum 3 x (6 multiply-adds, add, multiply),
    # pressure 6 multiply-adds, add, multiply; assembly and corrections once
    return n * (42.0 * nv + 14.0 * np_ * (1 + nc) + 250.0 + 150.0 * nc + (350.0 if les else 0.0))


def work(case):
    kind = case["kind"]
    if kind == "batch":
        parts = [work(m) for m in _members(case)]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    n = case["nx"] * case["ny"] * case["nz"]
    plane = 12.0 * case["ny"] * case["nz"]
    if kind == "tunnel":
        # velocity, pressure and face fluxes in and out, flags in
        return {"bytes": n * (16.0 * 2 + 12.0 * 2 + 1) + plane,
                "flops": _step_flops(n, case["nv"], case["np"], 0, case["les"])}
    if kind == "gradient":
        # the profile and the drag field in, the drag gradient out; forward,
        # transposed sweeps and one accumulation pass over the sweeps: three times a step's operations
        return {"bytes": n * 8.0 + plane, "flops": 3 * case["steps"] * _step_flops(n, case["nv"], case["np"], 2, False)}
    b = n * (16.0 * 2 + 1) + plane + (n * 4.0 if kind == "frames" else 0.0)
    return {"bytes": b, "flops": _step_flops(n, case["nv"], case["np"], case["nc"], case["les"])}


# ---------------------------------------------- the same in 64-bit torch
# Faces in the order E, W, N, S, U, D; fields are (..., nz, ny, nx).
_DIM = (-1, -1, -2, -2, -3, -3)


def _nb(a, f):
    """Value across face f; outside the domain the cell's own."""
    d = _DIM[f]
    n = a.shape[d]
    if f % 2 == 0:
        return torch.cat([a.narrow(d, 1, n - 1), a.narrow(d, n - 1, 1)], d)
    return torch.cat([a.narrow(d, 0, 1), a.narrow(d, 0, n - 1)], d)


class _Grid:
    """Masks, constants and boundary values of one case."""

    def __init__(self, flags, dx, dt, nu, cs, les, vbc, pbc, device):
        self.fluid = torch.as_tensor(flags, device=device) == 0
        nz, ny, nx = self.fluid.shape
        one = torch.ones_like(self.fluid)
        self.inside, self.nf = [], []
        for f in range(6):
            m = one.clone()
            m.select(_DIM[f], -1 if f % 2 == 0 else 0).fill_(False)
            self.inside.append(m)
            self.nf.append(m & _nb(self.fluid, f))
        self.dx, self.dt, self.nu, self.cs, self.les = dx, dt, nu, cs, les
        # faces' boundary conditions in the order of the faces here
        self.vbc = [vbc[i] for i in (1, 0, 3, 2, 5, 4)]
        self.pbc = [pbc[i] for i in (1, 0, 3, 2, 5, 4)]
        self.bnd = [torch.zeros(3, 1, 1, 1, dtype=torch.float64, device=device) for _ in range(6)]
        self.drag = None
        self.fixed_pressure = FIXED in self.pbc


def _log_law(u, dx, nu):
    """Wall eddy viscosity of the log law by ten Newton steps."""
    big, k = float(np.float32(9.8)) * (dx / 2) / nu, float(np.float32(0.41))
    tau = torch.ones_like(u)
    live = u >= float(np.float32(1e-5))
    for _ in range(10):
        lg = torch.log(big * tau)
        df = lg + 1
        live = live & (df.abs() >= float(np.float32(1e-6)))
        tau = torch.where(live, (tau - (tau * lg - k * u) / df).clamp(min=float(np.float32(1e-5))), tau)
    e = (tau * tau * (dx / 2) / u.clamp(min=1e-30) - nu).clamp(min=0)
    return torch.where(u >= float(np.float32(1e-5)), e, torch.zeros_like(e))


def _wall(G, u):
    """Wall viscosity on the W, S, D faces of every cell."""
    out = []
    for a in range(3):
        f = 2 * a + 1
        j, k = [i for i in range(3) if i != a]
        own = _log_law(torch.hypot(u[j], u[k]), G.dx, G.nu)
        wall = G.inside[f] & ~G.nf[f]
        if a == 1 and G.vbc[3] == FIXED:
            wall = wall | ~G.inside[f]
        zero = torch.zeros_like(own)
        out.append(torch.where(G.fluid, torch.where(wall, own, zero), torch.where(G.nf[f], _nb(own, f), zero)))
    return out


def _les(G, u):
    """Eddy viscosity, wall viscosities and the explicit LES term."""
    wall = _wall(G, u)
    fv = []
    for f in range(6):
        v = torch.where(G.nf[f], 0.5 * (u + _nb(u, f)), torch.zeros_like(u))
        if G.vbc[f] == FIXED:
            o = G.bnd[f].expand_as(u)
        else:
            o = u.clone()
            if G.vbc[f] == SYMMETRY:
                o[f // 2] = 0
        fv.append(torch.where(G.inside[f], v, o))
    g = [[(fv[2 * j][i] - fv[2 * j + 1][i]) / G.dx for j in range(3)] for i in range(3)]
    sym = [0.5 * (g[i][j] + g[j][i]) for i, j in ((0, 1), (1, 2), (2, 0))]
    s2 = g[0][0] ** 2 + g[1][1] ** 2 + g[2][2] ** 2 + 2 * (sym[0] ** 2 + sym[1] ** 2 + sym[2] ** 2)
    eddy = torch.where(G.fluid, G.cs ** 2 * G.dx ** 2 * torch.sqrt(2 * s2), torch.zeros_like(s2))
    vis = _vis(G, eddy, wall)
    term = torch.zeros_like(u)
    for f in range(6):
        a, s = f // 2, 1 if f % 2 == 0 else -1
        row = torch.stack(g[a])
        q = 0.5 * (row + _nb(row, f))
        solid = torch.zeros_like(row)
        solid[a] = -s * u[a] * 2 / G.dx
        if G.vbc[f] == FIXED:
            out = torch.zeros_like(row)
            out[a] = s * (G.bnd[f][a] - u[a]) * 2 / G.dx
        else:
            out = row.clone()
            out[a] = 0
        fg = torch.where(G.inside[f], torch.where(G.nf[f], q, solid), out)
        term = term + s * vis[f] * fg
    return eddy, vis, G.dx ** 2 * term


def _vis(G, eddy, wall):
    vis = []
    for f in range(6):
        a = f // 2
        w = _nb(wall[a], f) if f % 2 == 0 else wall[a]
        v = torch.where(G.nf[f], 0.5 * (eddy + _nb(eddy, f)), w)
        out = wall[1] if f == 3 and G.vbc[3] == FIXED else eddy
        vis.append(G.nu + torch.where(G.inside[f], v, out))
    return vis


def _vel_sweeps(G, A, iD, b, u, n):
    for _ in range(n):
        s = b
        for f in range(6):
            s = s + A[f] * _nb(u, f)
        u = torch.where(G.fluid, iD * s, u)
    return u


def _pres_sweeps(c, inv, rhs, n):
    p = torch.zeros_like(rhs)
    for _ in range(n):
        s = rhs
        for f in range(6):
            s = s - c[f] * _nb(p, f)
        p = inv * s
    return p


def _uniform_step(G, u, p, nv, np_, nc):
    dx, nu = G.dx, G.nu
    ds, dv = dx * dx, dx ** 3
    zero = torch.zeros_like(p)
    uT = u
    if G.les:
        eddy, vis, term = _les(G, u)
    else:
        vis, term = [torch.full_like(p, nu)] * 6, 0.0
    # momentum: D u = sum A_f u_f + b
    D = torch.full_like(u, dv / G.dt)
    b = torch.zeros_like(u)
    A, pf = [], []
    for f in range(6):
        a, s = f // 2, 1 if f % 2 == 0 else -1
        nf, ins = G.nf[f], G.inside[f]
        conv = ds * 0.25 * (u[a] + _nb(u[a], f))
        dif = vis[f] * ds / dx
        A.append(torch.where(nf, dif - s * conv, zero))
        D = D + torch.where(nf, s * conv + dif, torch.where(ins, 2 * dif, zero))
        o = ~ins
        if G.vbc[f] == FIXED:
            b = b + torch.where(o, (2 * dif - s * ds * G.bnd[f][a]) * G.bnd[f], torch.zeros_like(b))
            D = D + torch.where(o, 2 * dif, zero)
        elif G.vbc[f] == ZERO_GRAD:
            D = D + torch.where(o, s * ds * u[a], zero)
        else:
            e = [zero, zero, zero]
            e[a] = torch.where(o, 2 * dif, zero)
            D = D + torch.stack(e)
        pf.append(torch.where(nf, 0.5 * (p + _nb(p, f)),
                              p if G.pbc[f] != FIXED else torch.where(ins, p, zero)))
    b = b - ds * torch.stack([pf[2 * a] - pf[2 * a + 1] for a in range(3)]) + dv / G.dt * u + term
    if G.drag is not None:
        D = D + dv * G.drag
    iD = torch.where(G.fluid, 1 / torch.where(G.fluid, D, torch.ones_like(D)), torch.zeros_like(D))
    A = [torch.where(G.fluid, x, zero) for x in A]
    u = _vel_sweeps(G, A, iD, b, u, nv)
    # pressure correction with Rhie-Chow face fluxes
    Dp, bp, c = zero, zero, []
    for f in range(6):
        a, s = f // 2, 1 if f % 2 == 0 else -1
        nf, o = G.nf[f], ~G.inside[f]
        DI = 0.5 * (iD[a] + _nb(iD[a], f))
        cf = torch.where(nf & G.fluid, dv * DI / dx, zero)
        c.append(cf)
        Dp = Dp - cf
        pQ, pR = _nb(p, f), _nb(p, f ^ 1)
        pQQ = _nb(pQ, f)
        far, back = _nb(G.nf[f], f), G.nf[f ^ 1]
        grad = s * (pQ - p) / dx
        half = s * (pQ - p) / (2 * dx)
        gQ = torch.where(far, s * (pQQ - p) / (2 * dx), half)
        gP = torch.where(back, s * (pQ - pR) / (2 * dx), half)
        ave = torch.where(far | back, 0.5 * (gQ + gP), grad)
        flux = torch.where(nf, 0.5 * (u[a] + _nb(u[a], f)) - dv * DI * (grad - ave), zero)
        if G.vbc[f] == FIXED:
            flux = torch.where(o, G.bnd[f][a], flux)
        elif G.vbc[f] == ZERO_GRAD:
            flux = torch.where(o, u[a], flux)
        bp = bp + s * flux
        if G.pbc[f] == FIXED:
            Dp = Dp - torch.where(o, 2 * dv * iD[a] / dx, zero)
    live = G.fluid & (Dp != 0)
    inv = torch.where(live, 1 / torch.where(live, Dp, torch.ones_like(Dp)), zero)
    pc = _pres_sweeps(c, inv, bp, np_)
    p = p + torch.where(G.fluid, pc, zero)
    if not G.fixed_pressure:
        p = torch.where(G.fluid, p - p[2, p.shape[1] // 2, 2], p)
    uc = []
    for a in range(3):
        q = []
        for f in (2 * a, 2 * a + 1):
            out = zero if G.pbc[f] == FIXED else pc
            q.append(torch.where(G.inside[f], torch.where(G.nf[f], 0.5 * (pc + _nb(pc, f)), pc), out))
        uc.append(-dv * iD[a] * (q[0] - q[1]) / dx)
    uc = torch.stack(uc)
    u = u + uc
    # PISO correctors
    for _ in range(nc):
        ao = torch.zeros_like(u)
        for f in range(6):
            a, s = f // 2, 1 if f % 2 == 0 else -1
            w = s * ds * 0.25 * (uT[a] + _nb(uT[a], f)) - nu * ds / dx
            ao = ao + torch.where(G.nf[f] & G.fluid, w * _nb(uc, f), torch.zeros_like(u))
        co, rhs, cs = zero, zero, []
        for f in range(6):
            a, s = f // 2, 1 if f % 2 == 0 else -1
            m = G.nf[f] & G.fluid
            AI = torch.where(m, 0.5 * (iD[a] + _nb(iD[a], f)), zero)
            cs.append(dv * AI / dx)
            co = co - cs[-1]
            rhs = rhs - s * AI * 0.5 * (ao[a] + _nb(ao[a], f))
        live = G.fluid & (co != 0)
        inv = torch.where(live, 1 / torch.where(live, co, torch.ones_like(co)), zero)
        pc = _pres_sweeps(cs, inv, rhs, np_)
        p = p + pc
        grad = []
        for a in range(3):
            q = [torch.where(G.nf[f], 0.5 * (pc + _nb(pc, f)), pc) for f in (2 * a, 2 * a + 1)]
            grad.append((q[0] - q[1]) / dx)
        uc = -iD * (ao + dv * torch.stack(grad))
        u = u + uc
    return u, p


def _axis(v, a):
    return v.reshape([-1 if d == 2 - a else 1 for d in range(3)])


def _tunnel_step(G, faces, u, p, nv, np_):
    """One SIMPLE step on the stretched mesh; the face fluxes of the first
    step's momentum equation are zero."""
    zero = torch.zeros_like(p)
    d = [_axis(torch.as_tensor(np.diff(np.asarray(x, dtype=np.float64)), device=p.device), a)
         for a, x in enumerate(faces)]
    ds = [d[1] * d[2], d[0] * d[2], d[0] * d[1]]
    dv = d[0] * d[1] * d[2]
    dq = [_nb_axis(d[f // 2], f) for f in range(6)]
    wP = [dq[f] / (d[f // 2] + dq[f]) for f in range(6)]
    h = [0.5 * (d[f // 2] + dq[f]) for f in range(6)]
    if G.les:
        eddy, _, term = _les(G, u)
        vis = [G.nu + torch.where(G.nf[f], wP[f] * eddy + (1 - wP[f]) * _nb(eddy, f), eddy) for f in range(6)]
    else:
        vis, term = [torch.full_like(p, G.nu)] * 6, 0.0
    D = (dv / G.dt).expand_as(u).clone()
    b = torch.zeros_like(u)
    A, pf = [], []
    for f in range(6):
        a = f // 2
        nf, ins = G.nf[f], G.inside[f]
        dif = vis[f] * ds[a] / h[f]
        edge = vis[f] * ds[a] / (0.5 * d[a])
        A.append(torch.where(nf & G.fluid, dif, zero))
        D = D + torch.where(nf, dif, torch.where(ins, edge, zero))
        if G.vbc[f] == FIXED:
            b = b + torch.where(ins, torch.zeros_like(b), edge * G.bnd[f])
            D = D + torch.where(ins, zero, edge)
        elif G.vbc[f] == SYMMETRY:
            e = [zero, zero, zero]
            e[a] = torch.where(ins, zero, edge)
            D = D + torch.stack(e)
        pf.append(torch.where(nf, wP[f] * p + (1 - wP[f]) * _nb(p, f),
                              p if G.pbc[f] != FIXED else torch.where(ins, p, zero)))
    b = b - torch.stack([ds[a] * (pf[2 * a] - pf[2 * a + 1]) for a in range(3)]) + dv / G.dt * u + term
    iD = torch.where(G.fluid, 1 / D, torch.zeros_like(D))
    u = _vel_sweeps(G, A, iD, b, u, nv)
    Dp, bp, c = zero, zero, []
    for f in range(6):
        a, s = f // 2, 1 if f % 2 == 0 else -1
        nf, o = G.nf[f] & G.fluid, ~G.inside[f]
        DI = wP[f] * iD[a] + (1 - wP[f]) * _nb(iD[a], f)
        cf = torch.where(nf, dv * DI / h[f], zero)
        c.append(cf)
        Dp = Dp - cf
        pQ, pR = _nb(p, f), _nb(p, f ^ 1)
        pQQ = _nb(pQ, f)
        hP, hQ, hR = d[a], dq[f], dq[f ^ 1]
        hQQ = _nb_axis(dq[f], f)
        far, back = _nb(G.nf[f], f), G.nf[f ^ 1]
        grad = s * (pQ - p) / h[f]
        gQ = torch.where(far, s * (pQQ - p) / (0.5 * hQQ + hQ + 0.5 * hP), s * (pQ - p) / (1.5 * hQ + 0.5 * hP))
        gP = torch.where(back, s * (pQ - pR) / (0.5 * hQ + hP + 0.5 * hR), s * (pQ - p) / (0.5 * hQ + 1.5 * hP))
        ave = torch.where(far | back, 0.5 * (gQ + gP), grad)
        v = wP[f] * u[a] + (1 - wP[f]) * _nb(u[a], f) - dv * DI * (grad - ave)
        flux = torch.where(nf, v, zero)
        if G.vbc[f] == FIXED:
            flux = torch.where(o, G.bnd[f][a], flux)
        elif G.vbc[f] == ZERO_GRAD:
            flux = torch.where(o, u[a], flux)
        bp = bp + s * flux
        if G.pbc[f] == FIXED:
            Dp = Dp - torch.where(o, dv * iD[a] / (0.5 * d[a]), zero)
    live = G.fluid & (Dp != 0)
    inv = torch.where(live, 1 / torch.where(live, Dp, torch.ones_like(Dp)), zero)
    pc = _pres_sweeps(c, inv, bp, np_)
    p = p + pc
    uc = []
    for a in range(3):
        q = []
        for f in (2 * a, 2 * a + 1):
            out = zero if G.pbc[f] == FIXED else pc
            q.append(torch.where(G.inside[f], torch.where(G.nf[f], wP[f] * pc + (1 - wP[f]) * _nb(pc, f), pc), out))
        uc.append(-dv * iD[a] * (q[0] - q[1]) / d[a])
    return u + torch.stack(uc), p


def _nb_axis(v, f):
    """_nb of an axis' spacings (extent 1 along the others)."""
    return _nb(v, f) if v.shape[_DIM[f]] > 1 else v


def _f32(v):
    return float(np.float32(v))


def _exact_uniform(c, seed, device):
    s = _scene(c, seed)
    G = _Grid(s["flags"], _f32(c["dx"]), s["dt"], _f32(c["mu"]), _f32(c["cs"]), c["les"], _URBAN_VBC, _URBAN_PBC, device)
    t = lambda a: torch.as_tensor(a, device=device).double()  # noqa: E731
    G.bnd[1] = t(s["inlet"]).permute(2, 0, 1).unsqueeze(-1)
    return _uniform_step(G, t(s["vel"]), t(s["pres"]), c["nv"], c["np"], c["nc"])


def exact(case, seed):
    device = "cuda" if torch.cuda.is_available() else "cpu"
    kind = case["kind"]
    if kind == "gradient":
        return _exact_gradient(case, seed, device)
    with torch.no_grad():
        if kind == "batch":
            return [_exact_uniform(m, seed * 64 + i, device) for i, m in enumerate(_members(case))]
        if kind == "tunnel":
            s = _tunnel(case, seed)
            G = _Grid(s["flags"], 1.0, _f32(0.02), 1.0, _f32(0.15), case["les"], _TUNNEL_VBC, _TUNNEL_PBC, device)
            G.bnd[1][0] = 10.0
            return _tunnel_step(G, s["faces"], torch.as_tensor(s["vel"], device=device).double(),
                                torch.as_tensor(s["pres"], device=device).double(), case["nv"], case["np"])
        u, p = _exact_uniform(case, seed, device)
        if kind == "frames":
            return torch.cat([u, torch.zeros_like(u[:1])]).permute(1, 2, 3, 0).contiguous(), p
        return (u, p, None) if case["monitor"] else (u, p)


def _exact_gradient(c, seed, device):
    s = _street(c, seed)
    nx, ny, nz, dx, obj, soft = c["nx"], c["ny"], c["nz"], s["dx"], s["obj"], s["soft"]
    G = _Grid(np.zeros((nz, ny, nx), dtype=np.int32), dx, s["dt"], _f32(1.5e-5), 0.0, False, _URBAN_VBC, _URBAN_PBC,
              device)
    new = lambda v: torch.tensor(v, dtype=torch.float64, device=device, requires_grad=True)  # noqa: E731
    ustar, z0 = new(s["ustar"]), new(s["z0"])
    drag = torch.as_tensor(soft.drag(nx, ny, nz), device=device).double().requires_grad_(True)
    G.drag = drag
    y = torch.arange(ny, dtype=torch.float64, device=device)
    prof = lambda h: ustar / _f32(KAPPA) * torch.log((h + z0) / z0)  # noqa: E731
    zero = torch.zeros(nz, ny, 1, dtype=torch.float64, device=device)
    inlet = torch.stack([prof((y + 0.5) * dx).view(1, ny, 1).expand(nz, ny, 1), zero, zero])
    G.bnd[1] = inlet
    z3 = torch.zeros(nz, ny, nx, dtype=torch.float64, device=device)
    # the interior profile is placed at y = j dx, the inlet at (j + 0.5) dx
    u, p = torch.stack([prof(y * dx).view(1, ny, 1).expand(nz, ny, nx), z3, z3]), z3

    def one(u, p, inlet, drag):
        G.bnd[1], G.drag = inlet, drag
        return _uniform_step(G, u, p, c["nv"], c["np"], 2)

    J = 0.0
    for k in range(c["steps"]):
        u, p = checkpoint(one, u, p, inlet, drag, use_reentrant=False)
        if k >= c["steps"] - obj["window"]:
            patch = u[:, obj["z0"]:obj["z1"], obj["y"], obj["x0"]:obj["x1"]]
            J = J + (patch ** 2).sum() / ((obj["x1"] - obj["x0"]) * (obj["z1"] - obj["z0"]) * obj["window"])
    gu, gz, gd = torch.autograd.grad(J, [ustar, z0, drag])
    # each building's height through its column's solid fraction
    rows = torch.arange(ny, dtype=torch.float64, device=device) + 0.5
    heights = []
    for (x0, x1, a0, a1), hgt in zip(soft.footprints, soft.heights):
        sg = torch.sigmoid((float(hgt) - rows) / soft.width)
        col = gd[a0:a1, :, x0:x1].sum(dim=(0, 2))
        heights.append((col * soft.chi_max * sg * (1 - sg) / soft.width).sum())
    return {"J": float(J.detach()), "dJ_dustar": float(gu), "dJ_dz0": float(gz), "dJ_ddrag": gd.reshape(-1),
            "dJ_dheights": torch.stack(heights)}
