"""Grids of few latitudes either side of the lines from which the potential of
one set takes the two-degree recurrence (33 pairs, 129 where some lie next to
the equator, as they do here) and folds the rows' radius into the coefficients
(degree times pairs 70000: 167 pairs), against the CPU oracle.

Tolerance: both sides' functions of degree n carry about n 2^-53 of their size
from the rounded latitude; 4 n 2^-53 in relative RMS over the rows, times 4 off
the sphere (the powers of the radius ratio)."""
import numpy as np
import pytest

from charm_b200.workloads import GM, R_EARTH, kaula, rel_rms
from oracle import orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pairs", [1, 32, 33, 128, 129, 166, 167])
@pytest.mark.parametrize("last", [0.02, 0.2])
@pytest.mark.parametrize("mirror", [False, True])
@pytest.mark.parametrize("ratio", [1.0, 1.02])
@pytest.mark.parametrize("kind", [None, (1, 0, 0), (0, 0, 1)])
def test_few_latitudes(pairs, last, mirror, ratio, kind):
    import charm_b200 as cb
    n = 421
    lat = np.linspace(1.3, last, pairs)
    if mirror:
        lat = np.concatenate([lat, -lat[::-1]])
    lon = np.arange(2 * n + 2) * (np.pi / (n + 1))
    r = np.full(lat.size, R_EARTH * ratio)
    c, s = kaula(n, 12)
    c[0] = 0.0
    p = cb.PointGrid(lat, lon, r)
    shc = cb.Shc(n, GM, R_EARTH, c, s)
    f = cb.shs_point(p, shc, n) if kind is None else cb.shs_point_guru(
        p, shc, n, *kind)
    g, o = orc.Point(orc.GRID, lat, lon, r), orc.Shc(n, GM, R_EARTH, c, s)
    ref = orc.shs_point(g, o, n) if kind is None else orc.shs_point(g, o, n,
                                                                    kind)
    tol = 4.0 * n * 2.0 ** -53 * (1 if ratio == 1.0 else 4)
    assert rel_rms(np.ravel(f), np.ravel(ref[0])) <= tol
