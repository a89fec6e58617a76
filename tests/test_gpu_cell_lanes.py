"""Cell grids with one and with two pairs of cell rows per lane: row counts
at both sides of the lines the transforms draw (320 pairs in analysis, 600 in
synthesis), odd counts, a degree that ends inside a 64-degree stage, against
the oracle's restatement of CHarm's cell kernels.

The tolerance is that of the other cell tests: a relative RMS error of 1e-13
between double-precision evaluations of one recurrence in a different
summation order."""
import numpy as np
import pytest

from charm_b200.workloads import GM, R_EARTH, coef_rel_rms, kaula, rel_rms
from oracle import orc

pytestmark = pytest.mark.gpu

TOL = 1e-13


@pytest.mark.parametrize("nlat", [638, 639, 641, 1023, 1198, 1199, 1201])
@pytest.mark.parametrize("N", [5, 70])
def test_row_counts(N, nlat):
    import charm_b200 as cb
    c, s = kaula(N, 9500 + nlat)
    lat = np.linspace(np.pi / 2, -np.pi / 2, nlat + 1)
    lon = np.linspace(0.0, 2.0 * np.pi, 2 * N + 3)
    args = (lat[1:].copy(), lat[:-1].copy(), lon[:-1].copy(),
            lon[1:].copy(), np.full(nlat, R_EARTH))
    cl = cb.CellGrid(*args)
    co = orc.Cell(orc.CELL_GRID, *args)
    f = cb.shs_cell(cl, cb.Shc(N, GM, R_EARTH, c, s), N)
    ref = np.ravel(orc.shs_cell(co, orc.Shc(N, GM, R_EARTH, c, s), N))
    assert rel_rms(np.ravel(f), ref) <= TOL
    out = cb.sha_cell(cl, f, N, mu=GM, r=R_EARTH)
    back = orc.sha_cell(co, f, N, GM, R_EARTH)
    assert coef_rel_rms(out.c, out.s, back.c, back.s) <= TOL
