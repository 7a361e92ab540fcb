"""A batch of one chain runs its cases one after another, as stepping them does."""
import numpy as np
import pytest

from unitywindsimulation_b200 import FvmSolverCuda, _lib, cases
from unitywindsimulation_b200.solver import BatchSolver

pytestmark = pytest.mark.gpu

GRIDS = [(64, 32, 48), (24, 12, 16), (72, 40, 72), (64, 32, 48)]


def _handles():
    out = []
    for i, (x, y, z) in enumerate(GRIDS):
        c = cases.small_case(nx=x, ny=y, nz=z, seed=i, nv=30, np_=30)
        s = FvmSolverCuda(c.cfg)
        cases.apply_case(s, c)
        s.Step(1)
        out.append(s)
    return out


def test_one_chain_is_as_fast_as_stepping(built):
    """(With the splits for company it took 2.6 times as long.)"""
    alone, batched = _handles(), _handles()
    b = BatchSolver(batched)
    b.set_width(1)
    b.step(3)
    b.prepare_graphs()
    for s in alone:
        s.prepare_graphs()
        s.Step(3)
    one, chain = [], []
    for _ in range(7):
        ms = 0.0
        for s in alone:
            s.Step(2)
            ms += s.last_step_ms()
        one.append(ms)
        b.step(2)
        chain.append(b.last_step_ms())
    assert sorted(chain)[3] <= 1.25 * sorted(one)[3]
    for s, t in zip(alone, batched):
        for f in (_lib.FIELD_VEL_LAST_TIME, _lib.FIELD_PRES):
            assert np.array_equal(s.get_field(f), t.get_field(f)), _lib.FIELD_NAMES[f]
    # and back to all cases at once
    b.set_width(0)
    b.step(2)
    for s, t in zip(alone, batched):
        s.Step(2)
        assert np.array_equal(s.get_field(_lib.FIELD_PRES), t.get_field(_lib.FIELD_PRES))
    b.close()
