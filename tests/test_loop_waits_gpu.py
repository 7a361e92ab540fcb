"""The bounded packet waits of the loops on chip: one that runs out ends its loop with a
status, and the next loops on the same packets run as ever."""
import ctypes

import numpy as np
import pytest

from unitywindsimulation_b200 import FvmSolverCuda, _lib, cases

pytestmark = pytest.mark.gpu

P, V = _lib.KERNEL_PRES_SWEEP, _lib.KERNEL_VEL_SWEEP
SHORT = 2000  # polls: about a millisecond


def _faces(n):
    side = n // 4
    return cases.stretched_faces(n, 0.5, n - 2 * side, side, ratio=1.02)


def _solver(grid, stretched):
    nx, ny, nz = grid
    if stretched:
        case = cases.small_nonuniform_case(nv=20, np_=20)
        box = case.flags
        case.cfg.nx, case.cfg.ny, case.cfg.nz = grid
        case.faces = tuple(_faces(n) for n in grid)
        case.flags = np.zeros((nz, ny, nx), np.int32)
        case.flags[:box.shape[0], :box.shape[1], :box.shape[2]] = box
    else:
        case = cases.small_case(nx=nx, ny=ny, nz=nz, seed=4, nv=20, np_=20)
    s = FvmSolverCuda(case.cfg)
    cases.apply_case(s, case)
    s.Step(2)
    return s


def _selftest(s, kernel, silent, rounds=SHORT):
    st = ctypes.c_int(-1)
    code = s._lib.wf_loop_wait_selftest(s._h, kernel, silent, rounds, ctypes.byref(st))
    return code, st.value


# two sweeps a halo trip; one, with rim threads that fetch (3 cells a thread) and with
# 1/Dp in shared memory (12), whose momentum loop streams its words
@pytest.mark.parametrize("grid,stretched", [((61, 31, 59), False), ((72, 40, 72), False), ((126, 63, 95), False),
                                            ((61, 31, 59), True), ((72, 40, 72), True)],
                         ids=lambda v: "%dx%dx%d" % v if isinstance(v, tuple) else "stretched" if v else "uniform")
@pytest.mark.parametrize("kernel", [P, V], ids=["pressure", "momentum"])
def test_a_wait_that_runs_out(built, grid, stretched, kernel):
    s, ref = _solver(grid, stretched), _solver(grid, stretched)
    blocks = s.loop_plan(kernel)[0]
    assert blocks > 2
    assert _selftest(s, kernel, -1, 1 << 22) == (_lib.WF_OK, _lib.WF_OK)
    for silent in (0, blocks // 2, blocks - 1):
        assert _selftest(s, kernel, silent) == (_lib.WF_OK, _lib.WF_ERR_TIMEOUT)
        # the same slots in the next loop: complete again, and the fields untouched
        assert _selftest(s, kernel, -1, 1 << 22) == (_lib.WF_OK, _lib.WF_OK)
        assert _selftest(s, kernel, silent) == (_lib.WF_OK, _lib.WF_ERR_TIMEOUT)
        s.Step(1)
        ref.Step(1)
        for f in (_lib.FIELD_VEL_LAST_TIME, _lib.FIELD_PRES):
            assert np.array_equal(s.get_field(f), ref.get_field(f)), _lib.FIELD_NAMES[f]


def test_arguments(built):
    s = _solver((61, 31, 59), False)
    blocks = s.loop_plan(P)[0]
    for kernel, silent, rounds in ((2, 0, SHORT), (P, blocks, SHORT), (P, -2, SHORT), (P, 0, 0), (P, 0, (1 << 22) + 1)):
        assert _selftest(s, kernel, silent, rounds)[0] == _lib.WF_ERR_INVALID_ARG
    s.set_loops(_lib.LOOPS_PASSES)
    assert _selftest(s, P, 0)[0] == _lib.WF_ERR_UNSUPPORTED
