"""Fluid cells cut off by buildings, on chip.

A fluid cell with no fluid neighbour has Dp = 0 and b = 0: its pressure correction is
0/0, in the reference's kernels too (FvmColl.compute:2790-2848 skips non-fluid neighbours,
so the value stays in the cell).  No loop may carry a cell's NaN through a wall, where
its coefficients are zero."""
import numpy as np
import pytest

from unitywindsimulation_b200 import FvmSolverCuda, _lib, cases

from helpers import ALL_FIELDS

pytestmark = pytest.mark.gpu

WALL = 4  # cells of building on every side: more than a four-sweep pass reaches


def _block(shape, room=1):
    """Flags of one building with a closed room of room^3 cells in its middle."""
    nz, ny, nx = shape
    w = 2 * WALL + room
    x, z = (nx - w) // 2, (nz - w) // 2
    f = np.zeros(shape, np.int32)
    f[z:z + w, 0:w, x:x + w] = 1
    f[z + WALL:z + WALL + room, WALL:WALL + room, x + WALL:x + WALL + room] = 0
    return f


def _faces(n):
    side = n // 4
    return cases.stretched_faces(n, 0.5, n - 2 * side, side, ratio=1.02)


def _case(grid, kind):
    nx, ny, nz = grid
    if kind == "stretched":
        case = cases.small_nonuniform_case(nv=24, np_=19)
        case.cfg.nx, case.cfg.ny, case.cfg.nz = grid
        case.faces = tuple(_faces(n) for n in grid)
    else:
        case = cases.small_case(nx=nx, ny=ny, nz=nz, seed=1, nv=24, np_=19, piso=kind == "piso")
    if kind == "checked":
        case.cfg.calc_residual, case.cfg.vel_res_interval, case.cfg.pres_res_interval = 1, 4, 9
        case.cfg.vel_tol = case.cfg.pres_tol = 1e-30
    return case


def _run(case, mode, before=None, steps=2):
    s = FvmSolverCuda(case.cfg)
    s.set_loops(mode)
    cases.apply_case(s, case)
    if before:
        before(s)
    s.Step(steps)
    return s


# two sweeps a halo trip; 3, 8 and (uniform mesh only) 12 cells a thread
GRIDS = [(24, 16, 24), (72, 40, 72), (100, 50, 100), (128, 64, 96)]


@pytest.mark.parametrize("kind", ["stretched", "checked", "simple", "piso"])
@pytest.mark.parametrize("grid", GRIDS, ids=lambda g: "%dx%dx%d" % g)
def test_pocket_stays_closed(built, grid, kind):
    case = _case(grid, kind)
    case.flags = _block((grid[2], grid[1], grid[0]))
    pocket = np.zeros(case.flags.shape, bool)
    pocket[tuple(n[0] + WALL if a != 1 else WALL for a, n in enumerate(np.nonzero(case.flags == 1)))] = True
    assert case.flags[pocket] == 0 and pocket.sum() == 1
    a, b = _run(case, _lib.LOOPS_AUTO), _run(case, _lib.LOOPS_PASSES)
    p = a.get_field(_lib.FIELD_PRES).reshape(case.flags.shape)
    assert np.isnan(p[pocket]).all() and np.isfinite(p[~pocket]).all()
    for f in ALL_FIELDS:
        assert np.array_equal(a.get_field(f), b.get_field(f), equal_nan=True), _lib.FIELD_NAMES[f]


@pytest.mark.parametrize("grid", GRIDS, ids=lambda g: "%dx%dx%d" % g)
def test_velocities_stay_in_their_room(built, grid):
    """An overflowed velocity in a closed room does not reach the street."""
    case = _case(grid, "simple")
    case.flags = _block((grid[2], grid[1], grid[0]), room=3)
    room = np.zeros(case.flags.shape, bool)
    z, y, x = (n.min() for n in np.nonzero(case.flags == 1))
    room[z + WALL:z + WALL + 3, WALL:WALL + 3, x + WALL:x + WALL + 3] = True
    assert (case.flags[room] == 0).all()

    def spoil(s):
        for f in (_lib.FIELD_VEL_LAST_TIME, _lib.FIELD_VEL_LAST_ITER, _lib.FIELD_VEL):
            u = np.array(s.get_field(f)).reshape((3,) + room.shape)
            u[:, z + WALL + 1, WALL + 1, x + WALL + 1] = np.inf
            s.set_field(f, u.reshape(3, -1))

    a, b = (_run(case, m, spoil) for m in (_lib.LOOPS_AUTO, _lib.LOOPS_PASSES))
    u = a.get_field(_lib.FIELD_VEL_LAST_TIME).reshape((3,) + room.shape)
    assert not np.isfinite(u[:, room]).any() and np.isfinite(u[:, ~room]).all()
    for f in (_lib.FIELD_VEL_LAST_TIME, _lib.FIELD_PRES):
        assert np.array_equal(a.get_field(f), b.get_field(f), equal_nan=True), _lib.FIELD_NAMES[f]


@pytest.mark.parametrize("grid", [(24, 16, 24), (72, 40, 72)], ids=lambda g: "%dx%dx%d" % g)
def test_pocket_that_becomes_building(built, grid):
    """What a former pocket left in the pressure-correction buffers is not read."""
    case = _case(grid, "checked")
    case.flags = _block((grid[2], grid[1], grid[0]))
    solid = case.flags.copy()
    z, y, x = (n.min() for n in np.nonzero(solid == 1))
    solid[z + WALL, WALL, x + WALL] = 1
    got = []
    for mode in (_lib.LOOPS_AUTO, _lib.LOOPS_PASSES):
        s = _run(case, mode)
        p = np.array(s.get_field(_lib.FIELD_PRES))
        s.InitFlags(solid)
        s.set_field(_lib.FIELD_PRES, np.nan_to_num(p))
        s.Step(1)
        got.append(s)
    for f in (_lib.FIELD_VEL_LAST_TIME, _lib.FIELD_PRES):
        v = got[0].get_field(f)
        assert np.isfinite(v).all() and np.array_equal(v, got[1].get_field(f)), _lib.FIELD_NAMES[f]
