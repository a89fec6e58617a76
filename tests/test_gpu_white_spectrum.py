"""Analysis by the two-degree recurrence, every degree and order on its own
scale: grids of white noise, whose coefficients are of one size in all degrees,
against the CPU oracle degree by degree and order by order.

Tolerance: the functions of degree n at a rounded latitude are off by about n
2^-53 of their size on either side, independently from latitude to latitude, so
a coefficient is off by that fraction of the coefficients' size; 4 nmax 2^-53
in RMS over the coefficients of a degree or of an order, and eight times that
for one coefficient."""
import numpy as np
import pytest

from charm_b200.workloads import GM, R_EARTH
from oracle import orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name,grid_nmax,nmax", [
    ("gl", 766, 766), ("gl", 767, 767), ("gl", 800, 651), ("dh1", 511, 511),
    ("dh1", 513, 513), ("dh2", 514, 514)])
def test_analysis(name, grid_nmax, nmax):
    import charm_b200 as cb
    ctor, kind = {"gl": (cb.PointGridGL, None),
                  "dh1": (cb.PointGridDH1, orc.DH1),
                  "dh2": (cb.PointGridDH2, orc.DH2)}[name]
    p = ctor(grid_nmax, R_EARTH)
    g = (orc.gl(grid_nmax, R_EARTH) if kind is None else
         orc.dh(grid_nmax, R_EARTH, kind))
    rng = np.random.default_rng(grid_nmax + nmax)
    f = rng.standard_normal((p.lat.size, p.lon.size))
    out = cb.sha_point(p, f, nmax, GM, R_EARTH)
    ref = orc.sha_point(g, f, nmax, GM, R_EARTH)
    n = np.concatenate([np.arange(m, nmax + 1) for m in range(nmax + 1)])
    m = np.repeat(np.arange(nmax + 1), nmax + 1 - np.arange(nmax + 1))
    size = np.sqrt(np.mean(ref.c ** 2))
    err2 = (out.c - ref.c) ** 2 + (out.s - ref.s) ** 2
    tol = 4.0 * nmax * 2.0 ** -53
    # (C and S together)
    assert np.sqrt(err2.max()) <= 8 * tol * size
    for k in (n, m):
        rms = np.sqrt(np.bincount(k, err2) / np.bincount(k))
        assert rms.max() <= np.sqrt(2.0) * tol * size
