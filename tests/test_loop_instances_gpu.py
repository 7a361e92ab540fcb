"""Every kernel instance of the loops on chip against the pass kernels, bit for bit.

The grids are chosen by the split that they get on 148 multiprocessors: the cells a thread
owns and the sweeps a halo exchange are asserted, and that the step then has fewer launches
than in passes, so that no case passes by running the pass kernels on both sides."""
import numpy as np
import pytest

from unitywindsimulation_b200 import FvmSolverCuda, _lib, cases
from unitywindsimulation_b200.adjoint import AdjointSolver

from helpers import ALL_FIELDS

pytestmark = pytest.mark.gpu

P, V = _lib.KERNEL_PRES_SWEEP, _lib.KERNEL_VEL_SWEEP
# grid -> (cells a thread, sweeps a halo exchange) of the pressure loop, cells a thread of
# the momentum loop; ragged last boxes
GRIDS = {(25, 12, 16): ((2, 2), 2), (61, 31, 59): ((3, 2), 2), (72, 36, 60): ((4, 2), 3), (72, 40, 72): ((3, 1), 3),
         (77, 41, 70): ((4, 1), 4), (88, 41, 77): ((6, 1), 6), (97, 49, 99): ((8, 1), 8), (100, 50, 100): ((8, 1), 8),
         (103, 53, 104): ((10, 1), 10), (126, 63, 95): ((12, 1), 12), (130, 61, 110): ((14, 1), 14),
         (149, 61, 103): ((16, 1), 15)}
STRETCHED = [g for g, (p, _) in GRIDS.items() if p[0] <= 8]  # six coefficients a cell


def ids(g):
    return "%dx%dx%d" % g


def _faces(n):
    side = n // 4
    return cases.stretched_faces(n, 0.5, n - 2 * side, side, ratio=1.02)


def _case(grid, stretched=False, **kw):
    nx, ny, nz = grid
    if not stretched:
        return cases.small_case(nx=nx, ny=ny, nz=nz, seed=nx, **kw)
    case = cases.small_nonuniform_case(**kw)
    box = case.flags
    case.cfg.nx, case.cfg.ny, case.cfg.nz = grid
    case.faces = tuple(_faces(n) for n in grid)
    case.flags = np.zeros((nz, ny, nx), np.int32)
    case.flags[:box.shape[0], :box.shape[1], :box.shape[2]] = box
    case.flags[nz // 2:nz // 2 + 5, :ny // 2, nx // 2:nx // 2 + 7] = 1
    return case


def _pair(case, momentum=True):
    """(on chip, in passes), with the splits of the first asserted."""
    grid = (case.cfg.nx, case.cfg.ny, case.cfg.nz)
    (cells, sweeps), vel = GRIDS[grid]
    out = []
    for mode in (_lib.LOOPS_AUTO, _lib.LOOPS_PASSES):
        s = FvmSolverCuda(case.cfg)
        s.set_loops(mode)
        cases.apply_case(s, case)
        out.append(s)
    a, b = out
    assert a.loop_plan(P)[1:] == (cells, sweeps) and a.loop_plan(P)[0] > 1
    assert a.loop_plan(V)[1] == (vel if momentum else 0)
    assert b.loop_plan(P) == b.loop_plan(V) == (0, 0, 0)
    return a, b


def _step(a, b, steps):
    n = []
    for s in (a, b):
        k = s.kernel_launches()
        s.Step(steps)
        n.append(s.kernel_launches() - k)
    assert n[0] < n[1]


def _same(a, b):
    for f in ALL_FIELDS:
        assert np.array_equal(a.get_field(f), b.get_field(f)), _lib.FIELD_NAMES[f]


@pytest.mark.parametrize("grid", GRIDS, ids=ids)
def test_steps(built, grid):
    a, b = _pair(_case(grid, nv=20, np_=20, les=grid[2] % 2 == 0, piso=grid[1] % 2 == 0))
    _step(a, b, 2)
    _same(a, b)


@pytest.mark.parametrize("grid", GRIDS, ids=ids)
def test_checked_steps(built, grid):
    case = _case(grid, nv=5, np_=20, piso=False)
    case.cfg.calc_residual, case.cfg.vel_res_interval, case.cfg.pres_res_interval = 1, 4, 5
    case.cfg.vel_tol = case.cfg.pres_tol = 1e-30
    a, b = _pair(case, momentum=False)
    _step(a, b, 2)
    _same(a, b)
    assert a.residuals() == b.residuals()


@pytest.mark.parametrize("grid", STRETCHED, ids=ids)
def test_stretched_steps(built, grid):
    a, b = _pair(_case(grid, stretched=True, nv=20, np_=20, log_inflow=grid[2] % 2 == 0))
    _step(a, b, 2)
    a.op("pres_sweeps", 17)
    b.op("pres_sweeps", 17)
    _same(a, b)
    assert np.array_equal(a.get_face_flux(), b.get_face_flux())


@pytest.mark.parametrize("grid", STRETCHED, ids=ids)
def test_stretched_checked_steps(built, grid):
    case = _case(grid, stretched=True, nv=5, np_=20)
    case.cfg.calc_residual, case.cfg.vel_res_interval, case.cfg.pres_res_interval = 1, 4, 5
    case.cfg.vel_tol = case.cfg.pres_tol = 1e-30
    a, b = _pair(case, momentum=False)
    _step(a, b, 2)
    _same(a, b)
    assert a.residuals() == b.residuals()


@pytest.mark.parametrize("grid", GRIDS, ids=ids)
def test_last_iterates(built, grid):
    """Outside a step the loops also leave iterate n - 1, and start from the last one."""
    a, b = _pair(_case(grid, nv=20, np_=20))
    for s in (a, b):
        s.Step(1)
        s.op("vel_precompute"); s.op("vel_sweeps", 20); s.op("vel_sweeps", 21); s.op("pres_precompute")
        for n in (5, 6, 9):
            s.op("pres_sweeps", n)
    _same(a, b)


@pytest.mark.parametrize("grid", [(77, 41, 70), (97, 49, 99)], ids=ids)
def test_adjoint_iterates(built, grid):
    """The kept iterates with 4 and 8 cells a thread: the recorded step bit for bit, the
    reversed one to the rounding of its float atomics."""
    case = cases.small_soft_case(*grid, nv=20, np_=20)
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


# batches of two cases: the shared splits, 16 and 12 cells a thread, on half the GPU at most
@pytest.mark.parametrize("grid", [(25, 12, 16), (61, 31, 59), (72, 40, 72), (88, 41, 77)], ids=ids)
def test_batches(built, grid):
    from unitywindsimulation_b200.solver import BatchSolver
    alone, batched, passes = ([], [], [])
    for seed in (0, 1):
        case = cases.small_case(nx=grid[0], ny=grid[1], nz=grid[2], seed=seed, nv=20, np_=20)
        for group, mode in ((alone, _lib.LOOPS_AUTO), (batched, _lib.LOOPS_AUTO), (passes, _lib.LOOPS_PASSES)):
            s = FvmSolverCuda(case.cfg)
            s.set_loops(mode)
            cases.apply_case(s, case)
            group.append(s)
    b, c = BatchSolver(batched), BatchSolver(passes)
    b.step(3)
    c.step(3)
    assert b.kernel_launches() < c.kernel_launches()
    for s in alone:
        s.Step(3)
    for x, y, z in zip(alone, batched, passes):
        for f in (_lib.FIELD_VEL_LAST_TIME, _lib.FIELD_PRES):
            assert np.array_equal(x.get_field(f), y.get_field(f)) and np.array_equal(x.get_field(f), z.get_field(f))
    b.close()
    c.close()
