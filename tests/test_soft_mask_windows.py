"""The height chain rule looks only at a window around each footprint; it is the sum over
the whole grid for every footprint that the mask itself accepts."""
import numpy as np
import pytest

from unitywindsimulation_b200.soft_mask import SoftBuildings

NX, NY, NZ = 23, 9, 17
INF, NAN = float("inf"), float("nan")


def _whole_grid(sb, dchi):
    out = []
    yc = np.arange(NY) + 0.5
    for i, h in enumerate(sb.heights):
        s = 0.5 * (1.0 + np.tanh(0.5 * (h - yc) / sb.width))
        cols = np.asarray(dchi, dtype=np.float64).transpose(1, 0, 2)[:, sb.footprint_mask(i, NX, NZ)]
        out.append((cols.sum(axis=1) * sb.chi_max * s * (1.0 - s) / sb.width).sum())
    return np.array(out)


FOOTPRINTS = {
    "inside": (3, 8, 2, 9), "fractions": (2.3, 7.9, 1.5, 1.6), "over the edge": (-5, 4, 12, 40), "outside": (60, 70, 2, 5),
    "empty": (8, 3, 2, 9), "half a plane": (-INF, 6, 3, 11), "a whole strip": (-INF, INF, 3, 5), "everything": (-INF, INF, -INF, INF),
    "not a number": (NAN, 5, 2, 9), "huge": (-1e300, 1e300, 2, 9), "largest float": (-1.7e308, 1.7e308, -1.7e308, 9),
}


@pytest.mark.parametrize("angle", [0.0, 30.0, 90.0, 211.0])
@pytest.mark.parametrize("name", FOOTPRINTS)
def test_window_holds_the_footprint(name, angle):
    rng = np.random.default_rng(5)
    sb = SoftBuildings([FOOTPRINTS[name]], [4.4], chi_max=50.0, angle_deg=angle, margin=int(angle == 30.0))
    dchi = rng.standard_normal((NZ, NY, NX))
    with np.errstate(invalid="ignore", over="ignore"):
        want = _whole_grid(sb, dchi)
        for g in (dchi, dchi.astype(np.float32), dchi.reshape(-1)):
            got = sb.height_gradient(g, NX, NY, NZ)
            # float32 input: the rounding of the input, 2^-24 of each term
            tol = 1e-12 if g.dtype == np.float64 else 2.0 ** -24 * np.abs(dchi).sum() * 50.0
            assert np.abs(got - want).max() <= tol


def test_window_holds_random_footprints():
    rng = np.random.default_rng(6)
    for _ in range(300):
        x, z = np.sort(rng.uniform(-10, 35, 2)), np.sort(rng.uniform(-10, 30, 2))
        sb = SoftBuildings([(*x, *z)], [rng.uniform(0, NY)], chi_max=1.0, angle_deg=float(rng.uniform(-360, 360)))
        dchi = rng.standard_normal((NZ, NY, NX))
        assert np.abs(sb.height_gradient(dchi, NX, NY, NZ) - _whole_grid(sb, dchi)).max() <= 1e-12
