"""Scattered synthesis cut into ranges of orders (sctr.cu): point counts and
degrees with one range, several and the most, tiles of every width, points
from pole to pole on and off the sphere, against the CPU oracle.

Tolerance: both sides' Legendre values of degree n carry about n 2^-53 / cos or
sin(lat) of their size from the rounded latitude and the recurrence; averaged
over points that is a small multiple of n 2^-53 (4 taken), and at least the
rounding of the sums over up to (n + 1)^2 / 2 terms, 1e-15."""
import numpy as np
import pytest

from charm_b200.workloads import GM, R_EARTH, kaula, rel_rms
from oracle import orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nmax,npoint", [
    (0, 5), (1, 33), (20, 31), (31, 32), (45, 129), (90, 4095), (61, 4097),
    (150, 300), (24, 16400)])
@pytest.mark.parametrize("off", [False, True])
@pytest.mark.parametrize("kind", ["pot", "grad1", "grad2"])
def test_order_ranges(nmax, npoint, off, kind):
    import charm_b200 as cb
    rng = np.random.default_rng(npoint)
    lat = np.arcsin(rng.uniform(-1.0, 1.0, npoint))
    lon = rng.uniform(0.0, 2.0 * np.pi, npoint)
    r = R_EARTH + (rng.uniform(-2e4, 2e5, npoint) if off else
                   np.zeros(npoint))
    c, s = kaula(nmax, 3)
    if nmax > 1:
        c[0] = 0.0
    p = cb.PointSctr(lat, lon, r)
    shc = cb.Shc(nmax, GM, R_EARTH, c, s)
    out = {"pot": lambda: [cb.shs_point(p, shc, nmax)],
           "grad1": lambda: cb.shs_point_grad1(p, shc, nmax),
           "grad2": lambda: cb.shs_point_grad2(p, shc, nmax)}[kind]()
    g = orc.Point(orc.SCATTERED, lat, lon, r)
    o = orc.Shc(nmax, GM, R_EARTH, c, s)
    ref = (orc.shs_point(g, o, nmax) if kind == "pot"
           else orc.shs_point(g, o, nmax, kind))
    tol = 4.0 * nmax * 2.0 ** -53 + 1e-15
    keep = np.cos(lat) > 0.1
    for f, e in zip(out, ref):
        f, e = np.asarray(f).ravel(), np.asarray(e).ravel()
        if not np.any(e[keep]):
            continue
        # (derivatives: differences of terms up to 1 / cos(lat)^2 = 100 larger)
        assert rel_rms(f[keep], e[keep]) <= tol * (1 if kind == "pot" else 100)


def test_high_orders_start_below_the_double_range():
    """Ranges that begin at orders whose sectorial values underflow (down to
    1e-2000), and points on the equator, where they do not."""
    import charm_b200 as cb
    n = 700
    lat = np.deg2rad(np.concatenate([np.linspace(89.95, 60.0, 40),
                                     np.linspace(-3.0, 3.0, 21)]))
    lon = np.linspace(0.0, 6.0, lat.size)
    r = np.full(lat.size, R_EARTH + 3e3)
    c, s = kaula(n, 4)
    c[0] = 0.0
    f = cb.shs_point(cb.PointSctr(lat, lon, r), cb.Shc(n, GM, R_EARTH, c, s),
                     n)
    ref = orc.shs_point(orc.Point(orc.SCATTERED, lat, lon, r),
                        orc.Shc(n, GM, R_EARTH, c, s), n)[0]
    rms = np.sqrt(np.mean(ref ** 2))
    amp = 1.0 / np.maximum(np.cos(lat), 1e-3)
    assert np.all(np.abs(f - ref) <= 4.0 * n * 2.0 ** -53 * amp * rms)
