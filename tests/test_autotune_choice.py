"""What the autotuner chooses from the times it is given (no GPU: a stand-in solver with
fixed times)."""
import pytest

from unitywindsimulation_b200 import _lib, autotune
from unitywindsimulation_b200.config import default_config

P, V = _lib.KERNEL_PRES_SWEEP, _lib.KERNEL_VEL_SWEEP


class Fake:
    """Passes take `passes[kernel]` us a sweep, loops on chip `chip[kernel]` (absent: the
    grid does not fit)."""

    def __init__(self, passes, chip, vel_iters=50, pres_iters=30, piso=False):
        self.cfg = default_config(nx=32, ny=16, nz=24, vel_iters=vel_iters, pres_iters=pres_iters, piso_correctors=2,
                                  solver_type=_lib.SOLVER_PISO if piso else _lib.SOLVER_SIMPLE)
        self.passes, self.chip = passes, chip
        self.loops, self.blocking, self.tiles, self.timed = _lib.LOOPS_AUTO, (4, 1), (32, (32, 4, 2)), 0

    def _iters(self, kernel):
        return self.cfg.pres_iters if kernel == P else self.cfg.vel_iters

    def set_loops(self, mode):
        self.loops = mode

    def set_blocking(self, p, v):
        self.blocking, self.loops = (p, v), _lib.LOOPS_PASSES

    def get_blocking(self):
        return self.blocking

    def set_tiles(self, rows, block):
        self.tiles, self.loops = (rows, tuple(block)), _lib.LOOPS_PASSES

    def get_tiles(self):
        return self.tiles

    def loop_plan(self, kernel, beside=False):
        on = self.loops == _lib.LOOPS_AUTO and kernel in self.chip and self._iters(kernel) >= 2
        return (100, 4, 1) if on else (0, 0, 0)

    def time_kernel(self, kernel, reps=20, flush_l2=True):
        self.timed += 1
        if self.loop_plan(kernel)[0]:
            n = self._iters(kernel)
            return self.chip[kernel] * n * 1e-3, 0.0, n
        k = self.blocking[0 if kernel == P else 1]
        return self.passes[kernel] * k * 1e-3, 0.0, k


def _tune(solver, path=None):
    return autotune.tune(solver, path, reps=1, device_name="stand-in")


@pytest.mark.parametrize("pres_iters", [2, 3, 4, 5, 30])
def test_few_pressure_sweeps(pres_iters):
    s = Fake({P: 4.0, V: 3.0}, {P: 1.0, V: 1.5}, pres_iters=pres_iters)
    e = _tune(s)
    assert e["loops"] == s.loops == _lib.LOOPS_AUTO
    assert (e["pres_us_per_sweep"], e["vel_us_per_sweep"]) == pytest.approx((1.0, 1.5))


def test_both_loops_decide():
    # pressure loses 0.5 us a sweep on chip, momentum gains 3
    assert _tune(Fake({P: 1.0, V: 5.0}, {P: 1.5, V: 2.0}))["loops"] == _lib.LOOPS_AUTO
    # with two correctors three times the pressure sweeps count, and the gain is smaller
    assert _tune(Fake({P: 1.0, V: 2.5}, {P: 1.5, V: 2.0}, piso=True))["loops"] == _lib.LOOPS_PASSES
    # pressure gains a little, momentum loses more
    e = _tune(Fake({P: 1.0, V: 1.0}, {P: 0.9, V: 2.0}))
    assert e["loops"] == _lib.LOOPS_PASSES
    assert (e["pres_us_per_sweep"], e["vel_us_per_sweep"]) == pytest.approx((1.0, 1.0))


def test_one_loop_on_chip():
    e = _tune(Fake({P: 4.0, V: 3.0}, {P: 1.0}))
    assert e["loops"] == _lib.LOOPS_AUTO
    assert (e["pres_us_per_sweep"], e["vel_us_per_sweep"]) == pytest.approx((1.0, 3.0))
    assert _tune(Fake({P: 4.0, V: 3.0}, {}))["loops"] == _lib.LOOPS_PASSES


def test_cache_tells_sweep_counts_apart(tmp_path):
    path = str(tmp_path / "tune.json")
    times = {P: 1.0, V: 2.5}, {P: 1.5, V: 2.0}
    first, other, again = Fake(*times), Fake(*times, pres_iters=300), Fake(*times)
    assert _tune(first, path)["loops"] == _lib.LOOPS_AUTO
    e = _tune(other, path)
    assert not e["cached"] and e["loops"] == _lib.LOOPS_PASSES
    e = _tune(again, path)
    assert e["cached"] and e["loops"] == again.loops == _lib.LOOPS_AUTO and again.timed == 0
