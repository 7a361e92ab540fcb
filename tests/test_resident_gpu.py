"""Loops that keep the grid on chip against the pass kernels.

Both run the same arithmetic in the same order on the same values, so every
field must agree bit for bit: grids of one box and of many, boxes that
overhang the domain on every axis, every count of cells a thread owns, odd
extents, few sweeps, passes that also write iterate n - 1, the stretched mesh
and the adjoint's kept iterates."""
import numpy as np
import pytest

from unitywindsimulation_b200 import FvmSolverCuda, _lib, cases
from unitywindsimulation_b200.adjoint import AdjointSolver

from helpers import ALL_FIELDS

pytestmark = pytest.mark.gpu


def _pair(case):
    out = []
    for mode in (_lib.LOOPS_AUTO, _lib.LOOPS_PASSES):
        s = FvmSolverCuda(case.cfg)
        s.set_loops(mode)
        cases.apply_case(s, case)
        out.append(s)
    return out


def _same(a, b):
    for f in ALL_FIELDS:
        assert np.array_equal(a.get_field(f), b.get_field(f)), _lib.FIELD_NAMES[f]


# extents chosen for 2, 3, 4, 6, 8, 10, 12, 14 and 16 cells a thread on 148
# multiprocessors, with ragged last boxes
GRIDS = [(24, 12, 16), (53, 31, 37), (12, 9, 13), (72, 40, 72), (88, 41, 77), (100, 50, 75), (104, 50, 97),
         (103, 53, 104), (126, 63, 95), (130, 61, 110), (149, 61, 103)]


@pytest.mark.parametrize("grid", GRIDS, ids=lambda g: "%dx%dx%d" % g)
def test_steps_bit_identical(built, grid):
    nx, ny, nz = grid
    case = cases.small_case(nx=nx, ny=ny, nz=nz, seed=nx, nv=5, np_=7, les=nx % 2 == 0)
    a, b = _pair(case)
    for s in (a, b):
        s.Step(2)
    _same(a, b)


@pytest.mark.parametrize("n", [1, 2, 3, 8])
def test_loops_outside_a_step(built, n):
    """The operations also leave iterate n - 1, and start from the last iterate."""
    case = cases.small_case(nx=45, ny=22, nz=31, seed=3)
    a, b = _pair(case)
    for s in (a, b):
        s.Step(1)
        s.op("vel_precompute"); s.op("vel_sweeps", n); s.op("pres_precompute")
        s.op("pres_sweeps", n); s.op("pres_sweeps", n + 1)
    _same(a, b)


# two sweeps a halo trip with 2, 3 and 4 cells a thread, boxes of two cells, and
# boxes that overhang the domain on every axis; odd and even sweep counts
@pytest.mark.parametrize("grid", [(64, 32, 48), (53, 31, 37), (61, 31, 59), (72, 36, 60), (6, 5, 7)],
                         ids=lambda g: "%dx%dx%d" % g)
def test_two_sweeps_a_trip(built, grid):
    nx, ny, nz = grid
    case = cases.small_case(nx=nx, ny=ny, nz=nz, seed=nz)
    a, b = _pair(case)
    for s in (a, b):
        s.Step(1)
        s.op("vel_precompute"); s.op("vel_sweeps", 2); s.op("pres_precompute")
        for n in (2, 3, 4, 7, 12):
            s.op("pres_sweeps", n)
    _same(a, b)


@pytest.mark.parametrize("kw", [dict(), dict(log_inflow=True, les=True), dict(nx=15, x_split=(7, 4))],
                         ids=["tunnel", "urban_les", "odd"])
def test_stretched_mesh_bit_identical(built, kw):
    a, b = _pair(cases.small_nonuniform_case(**kw))
    for s in (a, b):
        s.Step(3)
        s.op("pres_sweeps", 4)
    _same(a, b)
    assert np.array_equal(a.get_face_flux(), b.get_face_flux())


# the adjoint's momentum iterates, forward and transposed, in the other splits (4
# to 15 cells a thread)
@pytest.mark.parametrize("grid", [(72, 40, 72), (88, 41, 77), (100, 50, 75), (103, 53, 104), (128, 64, 96), (130, 61, 110),
                                  (149, 61, 103)], ids=lambda g: "%dx%dx%d" % g)
def test_adjoint_momentum_iterates(built, grid):
    test_adjoint_iterates(built, grid)


@pytest.mark.parametrize("grid", [(24, 12, 16), (41, 21, 30)], ids=lambda g: "%dx%dx%d" % g)
def test_adjoint_iterates(built, grid):
    """Recorded forward step bit for bit; the reversed step to the rounding
    of its float atomics."""
    case = cases.small_soft_case(*grid, nv=5, np_=6)
    rng = np.random.default_rng(1)
    n = case.n_cells
    ub, pb = rng.standard_normal((3, n), dtype=np.float32), rng.standard_normal(n, dtype=np.float32)
    got = []
    for s in _pair(case):
        s.Step(1)
        with AdjointSolver(s) as adj:
            got.append((adj.step_forward(), adj.step_vjp(ub, pb)))
    (fa, va), (fb, vb) = got
    for x, y in zip(fa, fb):
        assert np.array_equal(x, y)
    for x, y in ((va[0], vb[0]), (va[1], vb[1]), (va[3], vb[3])):
        assert np.linalg.norm(x - y) <= 1e-5 * np.linalg.norm(y)


def test_loops_of_several_handles_at_once(built):
    """Handles stepped side by side on their own streams (each loop is one
    cooperative launch of up to every multiprocessor) and from their own
    threads: the fields of stepping them one after another."""
    import threading
    grids = [(24, 12, 16), (64, 32, 48), (53, 31, 37), (104, 50, 97), (72, 40, 72), (48, 20, 28)]
    cs = [cases.small_case(nx=x, ny=y, nz=z, seed=x, nv=4, np_=20) for x, y, z in grids]
    got = []
    for together in (False, True):
        solvers = [FvmSolverCuda(c.cfg) for c in cs]
        for s, c in zip(solvers, cs):
            cases.apply_case(s, c)
            s.Step(1)
        if together:
            for _ in range(6):
                for s in solvers:
                    s.step_async(1)
            threads = [threading.Thread(target=s.Step, args=(4,)) for s in solvers]
            for t in threads:
                t.start()
            for t in threads:
                t.join()
        else:
            for s in solvers:
                s.Step(10)
        for s in solvers:
            s.sync()
        got.append([(s.GetVelField(), s.GetPresField()) for s in solvers])
        for s in solvers:
            s.close()
    for (va, pa), (vb, pb) in zip(*got):
        assert np.array_equal(va, vb) and np.array_equal(pa, pb)


@pytest.mark.parametrize("tols", [(1e-15, 1e-15), (1e-15, None), (None, 1e-15)], ids=["never", "pressure", "momentum"])
@pytest.mark.parametrize("stretched", [False, True], ids=["uniform", "stretched"])
def test_residual_checks_between_fast_loops(built, tols, stretched):
    """With residual checks the pressure loop runs on chip from check to
    check; the sweep at which a tolerance ends a loop, the buffer roles the
    reference's break leaves, the residuals and the fields are the oracle's
    (whose loop checks sweep by sweep)."""
    from helpers import REL_TOL, rel_l2
    from oracle import OracleSolver
    case = cases.small_nonuniform_case(nv=13, np_=23) if stretched else \
        cases.small_case(nx=45, ny=22, nz=31, seed=2, piso=False, nv=13, np_=23)
    case.cfg.calc_residual, case.cfg.vel_res_interval, case.cfg.pres_res_interval = 1, 4, 5
    case.cfg.vel_tol = case.cfg.pres_tol = 1e-15
    if None in tols:  # a tolerance between the residuals of two checked sweeps of the first step
        o = OracleSolver(case.cfg, 32)
        cases.apply_case(o, case)
        o.op("vel_precompute")
        name, sweeps = ("vel", 8) if tols[0] is None else ("pres", 10)
        if name == "pres":
            o.op("vel_sweeps", 13); o.op("pres_precompute")
        o.op(name + "_sweeps", sweeps)
        setattr(case.cfg, name + "_tol", 0.999 * o.op_residual(name))
    got = []
    for make in (FvmSolverCuda, lambda c: OracleSolver(c, 32)):
        s = make(case.cfg)
        cases.apply_case(s, case)
        s.Step(1)
        got.append((s, s.residuals()))
    (g, rg), (o, ro) = got
    # a residual is a difference of two iterates: each carries the rounding of
    # its last sum of eight terms, so the norm is known to 8 eps of D u (Dp p')
    rms = lambda a: float(np.sqrt(np.mean(np.square(a, dtype=np.float64))))  # noqa: E731
    floors = [8 * 2.0 ** -24 * rms(o.get_field(d) * o.get_field(v))
              for d, v in ((_lib.FIELD_D, _lib.FIELD_VEL), (_lib.FIELD_DP, _lib.FIELD_PRES_CORRECT))]
    for a, b, floor in zip(rg, ro, floors):
        assert abs(a - b) <= 1e-3 * abs(b) + floor
    for f in (_lib.FIELD_VEL_LAST_TIME, _lib.FIELD_PRES):
        assert rel_l2(g.get_field(f), o.get_field(f)) <= REL_TOL, _lib.FIELD_NAMES[f]


@pytest.mark.parametrize("stretched", [False, True], ids=["uniform", "stretched"])
def test_checked_steps_bit_identical(built, stretched):
    """Residual checks: on chip between the checks against one sweep a launch."""
    case = cases.small_nonuniform_case(nv=9, np_=23) if stretched else \
        cases.small_case(nx=45, ny=22, nz=31, seed=2, piso=False, nv=9, np_=23)
    case.cfg.calc_residual, case.cfg.vel_res_interval, case.cfg.pres_res_interval = 1, 4, 5
    case.cfg.vel_tol = case.cfg.pres_tol = 1e-15
    a, b = _pair(case)
    for s in (a, b):
        s.Step(2)
    _same(a, b)
    assert a.residuals() == b.residuals()
