"""Block shapes chosen by the grid's extents: every shape of the rule, for one
cell and for four cells a thread, with ragged last blocks, against the oracle,
and the same bits as the wide block."""
import numpy as np
import pytest

from unitywindsimulation_b200 import FvmSolverCuda, _lib, cases
from oracle import OracleSolver

from helpers import ALL_FIELDS, REL_TOL, rel_l2

pytestmark = pytest.mark.gpu

# cells -> block of the four-cell kernels; the one-cell kernels get 32 x 4 x 2,
# 16 x 8 x 2 (44 and 45 cells a row, 8 | ny) and 16 x 4 x 4 (ny = 20)
SHAPES = [((124, 12, 9), (32, 4, 2)), ((44, 24, 10), (16, 8, 2)), ((44, 20, 12), (16, 4, 4)), ((68, 16, 8), (8, 8, 4)),
          ((45, 24, 11), None), ((141, 20, 12), None)]


@pytest.mark.parametrize("grid,block", SHAPES, ids=lambda g: "x".join(map(str, g)) if g else "cells")
def test_blocks_by_extents(built, grid, block):
    nx, ny, nz = grid
    case = cases.small_case(nx=nx, ny=ny, nz=nz, seed=ny)
    a, b, o = FvmSolverCuda(case.cfg), FvmSolverCuda(case.cfg), OracleSolver(case.cfg, 32)
    if block:
        assert a.get_tiles()[1] == block
    for s in (a, b):
        s.set_loops(_lib.LOOPS_PASSES)
    b.set_tiles(b.get_tiles()[0], (32, 4, 2))
    for s in (a, b, o):
        cases.apply_case(s, case)
        s.Step(2)
    for f in ALL_FIELDS:
        assert np.array_equal(a.get_field(f), b.get_field(f)), _lib.FIELD_NAMES[f]
    for f in (_lib.FIELD_VEL_LAST_TIME, _lib.FIELD_PRES):
        assert rel_l2(a.get_field(f), o.get_field(f)) <= REL_TOL, _lib.FIELD_NAMES[f]


@pytest.mark.parametrize("nx", [24, 27])
def test_step_equals_its_operations(built, nx):
    """Inside a step the pre-computes also store the sweeps' reciprocals; the
    operations one by one compute them apart."""
    case = cases.small_case(nx=nx, piso=False, les=False)
    a, b = FvmSolverCuda(case.cfg), FvmSolverCuda(case.cfg)
    for s in (a, b):
        cases.apply_case(s, case)
    a.Step(1)
    b.op("vel_precompute"); b.op("vel_sweeps", case.cfg.vel_iters); b.op("pres_precompute")
    b.op("pres_sweeps", case.cfg.pres_iters); b.op("apply_pres"); b.op("apply_vel"); b.op("end_step")
    f = _lib.FIELD_VEL_LAST_TIME
    assert np.array_equal(a.get_field(f), b.get_field(f))
