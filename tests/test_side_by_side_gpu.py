"""Handles stepped at the same time on their own streams: beside others a handle's loops
take splits that leave room for theirs."""
import threading
import time

import numpy as np
import pytest

from unitywindsimulation_b200 import FvmSolverCuda, _lib, cases

pytestmark = pytest.mark.gpu


def _faces(n):
    side = n // 4
    return cases.stretched_faces(n, 0.5, n - 2 * side, side, ratio=1.02)


def _case(grid, stretched, seed, nv=50, np_=60):
    nx, ny, nz = grid
    if not stretched:
        return cases.small_case(nx=nx, ny=ny, nz=nz, seed=seed, nv=nv, np_=np_)
    case = cases.small_nonuniform_case(nv=nv, np_=np_, seed=seed)
    box = case.flags
    case.cfg.nx, case.cfg.ny, case.cfg.nz = grid
    case.faces = tuple(_faces(n) for n in grid)
    case.flags = np.zeros((nz, ny, nx), np.int32)
    case.flags[:box.shape[0], :box.shape[1], :box.shape[2]] = box[:nz, :ny, :nx]
    return case


def _handles(cs, mode=_lib.LOOPS_AUTO):
    out = []
    for c in cs:
        s = FvmSolverCuda(c.cfg)
        s.set_loops(mode)
        cases.apply_case(s, c)
        s.Step(1)
        out.append(s)
    return out


@pytest.mark.parametrize("stretched", [False, True], ids=["uniform", "stretched"])
@pytest.mark.parametrize("n", [4, 16])
def test_many_small_handles_are_no_slower_than_the_passes(built, stretched, n):
    """Loops that hold the whole GPU run one after another; the passes of small grids
    run side by side.  (With the lone splits alone, 16 handles took 3.5 and 4.5 times
    as long as in passes.)"""
    ms = {}
    for mode in (_lib.LOOPS_AUTO, _lib.LOOPS_PASSES):
        hs = _handles([_case((24, 12, 16), stretched, s) for s in range(n)], mode)
        for h in hs:
            h.prepare_graphs()

        def round_of_steps():
            t = time.perf_counter()
            for _ in range(6):
                for h in hs:
                    h.step_async(1)
            for h in hs:
                h.sync()
            return time.perf_counter() - t

        round_of_steps()
        ms[mode] = sorted(round_of_steps() for _ in range(9))[4]
        for h in hs:
            h.close()
    assert ms[_lib.LOOPS_AUTO] <= 1.25 * ms[_lib.LOOPS_PASSES]


# grids whose splits beside others hold 12 to 54 multiprocessors, with one and two
# sweeps a trip, and one that keeps its lone splits
GRIDS = [(6, 5, 7), (16, 10, 12), (24, 12, 16), (40, 20, 30), (53, 31, 37), (64, 32, 48), (72, 40, 72), (88, 41, 77)]


@pytest.mark.parametrize("stretched", [False, True], ids=["uniform", "stretched"])
def test_fields_do_not_depend_on_company(built, stretched):
    """Round robin, one thread a handle, and with readbacks instead of waits, against
    stepping one after another."""
    grids = [g for g in GRIDS if not stretched or min(g) >= 10]
    cs = [_case(g, stretched, i, nv=20, np_=23) for i, g in enumerate(grids)]
    alone, beside = _handles(cs), _handles(cs)
    for s in alone:
        s.Step(15)
    for s in beside:
        s.prepare_graphs()
    for _ in range(5):
        for s in beside:
            s.step_async(1)
    for s in beside:
        s.sync()
    threads = [threading.Thread(target=s.Step, args=(5,)) for s in beside]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for _ in range(5):
        got = []
        for s in beside:
            s.step_async(1)
            v, p = np.empty((s.n_cells, 3), np.float32), np.empty(s.n_cells, np.float32)
            s.readback_begin(v, p)
            got.append((v, p))
        for s in beside:
            s.readback_wait()
    for a, b, (_, p) in zip(alone, beside, got):
        assert np.array_equal(p, a.GetPresField().ravel())
        for f in (_lib.FIELD_VEL_LAST_TIME, _lib.FIELD_PRES):
            assert np.array_equal(a.get_field(f), b.get_field(f)), (a.shape, _lib.FIELD_NAMES[f])
