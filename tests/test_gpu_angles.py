"""Grids whose rows are at angles beyond the poles: accepted like any others
(the functions are those of the angle's sine and cosine), on and off the
sphere, either side of the degrees from which the two-degree recurrence serves
(the angles are in its order of latitudes).

Tolerance: both sides evaluate the same rounded angles, and their functions of
degree n are off by about n 2^-53 of their size (next to a pole n 2^-53 /
cos); 4 n 2^-53 in relative RMS, as for latitudes, times 4 off the sphere."""
import numpy as np
import pytest

from charm_b200.workloads import GM, R_EARTH, kaula, rel_rms
from oracle import orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [60, 410])
@pytest.mark.parametrize("ratio", [1.0, 1.01])
@pytest.mark.parametrize("top", [2.0, 9.0, 60.0, -60.0])
def test_angles_beyond_the_poles(n, ratio, top):
    import charm_b200 as cb
    lat = top * np.linspace(1.0, 0.83, 37)
    lat = lat[np.abs(np.cos(lat)) > 0.05]
    lon = np.arange(2 * n + 2) * (np.pi / (n + 1))
    r = np.full(lat.size, R_EARTH * ratio)
    c, s = kaula(n, 3)
    c[0] = 0.0
    f = cb.shs_point(cb.PointGrid(lat, lon, r), cb.Shc(n, GM, R_EARTH, c, s),
                     n)
    ref = orc.shs_point(orc.Point(orc.GRID, lat, lon, r),
                        orc.Shc(n, GM, R_EARTH, c, s), n)[0]
    tol = 4.0 * n * 2.0 ** -53 * (1 if ratio == 1.0 else 4)
    assert rel_rms(f, ref) <= tol
