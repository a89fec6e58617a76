"""The two-degree recurrence (two.cuh) and the rules that choose it, against
the CPU oracle: degrees around the rules' lower ends, whole and partial
32-pair groups, latitudes either side of its equatorial band, every radius
rule and latitude orders it must leave to the one-degree kernels.

Tolerance.  Either side's functions of degree n at a rounded latitude are off
by about n 2^-53 / sin or cos(lat) relative to their size (the latitude's
rounding acts as a phase n dlat); over a grid that averages to a small
multiple of n 2^-53, and two independent sides with sums of random
coefficients stay below 4 n 2^-53 in relative RMS.  The model has no degree-0
term, so nothing hides in it."""
import numpy as np
import pytest

from charm_b200.workloads import GM, R_EARTH, coef_rel_rms, kaula, rel_rms
from oracle import orc

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def cb():
    import charm_b200
    return charm_b200


def tol(n):
    return 4.0 * n * 2.0 ** -53


def model(n, seed):
    c, s = kaula(n, seed)
    c[0] = 0.0
    return c, s


def both(cb, p, g, n, kind=None, seed=7):
    c, s = model(n, seed)
    shc = cb.Shc(n, GM, R_EARTH, c, s)
    f = cb.shs_point(p, shc, n) if kind is None else cb.shs_point_guru(
        p, shc, n, *kind)
    o = orc.Shc(n, GM, R_EARTH, c, s)
    ref = orc.shs_point(g, o, n) if kind is None else orc.shs_point(g, o, n,
                                                                    kind)
    return np.asarray(f).ravel(), np.asarray(ref[0]).ravel()


def grids(cb, name, n, r):
    if name == "gl":
        return cb.PointGridGL(n, r), orc.gl(n, r)
    kind = orc.DH1 if name == "dh1" else orc.DH2
    ctor = cb.PointGridDH1 if name == "dh1" else cb.PointGridDH2
    return ctor(n, r), orc.dh(n, r, kind)


@pytest.mark.parametrize("name", ["gl", "dh1", "dh2"])
@pytest.mark.parametrize("nmax", [191, 399, 400, 401, 447])
def test_synthesis(cb, name, nmax):
    p, g = grids(cb, name, nmax, R_EARTH)
    f, ref = both(cb, p, g, nmax)
    assert rel_rms(f, ref) <= tol(nmax)


# one radius above and below the sphere (folded into the coefficients), and
# one so far that the powers would leave the range (general path)
@pytest.mark.parametrize("ratio", [1.04, 0.98, 8.0])
@pytest.mark.parametrize("kind", [None, (1, 0, 0), (2, 0, 0), (0, 0, 1),
                                  (0, 0, 2), (1, 0, 1)])
def test_radii_and_radial_derivatives(cb, ratio, kind):
    n = 410
    p, g = grids(cb, "gl", n, R_EARTH * ratio)
    f, ref = both(cb, p, g, n, kind)
    keep = np.repeat(np.abs(p.lat) < np.deg2rad(89.0), p.lon.size)
    assert rel_rms(f[keep], ref[keep]) <= 4 * tol(n)


@pytest.mark.parametrize("case", ["ascending", "regional", "shuffled",
                                  "radii", "equator", "polar"])
def test_custom_latitudes(cb, case):
    """Orders and spans of latitudes: those that the two-degree kernel takes
    (symmetric, towards the equator) and those that it must not."""
    n = 405
    rng = np.random.default_rng(3)
    half = np.sort(rng.uniform(0.003, 1.56, 75))[::-1]
    lat = np.concatenate([half, -half[::-1]])
    r = np.full(lat.size, R_EARTH)
    if case == "ascending":
        lat = lat[::-1].copy()
    elif case == "regional":
        lat = np.linspace(1.1, -0.4, 71)
        r = np.full(lat.size, R_EARTH)
    elif case == "shuffled":
        lat = rng.permutation(lat)
    elif case == "radii":
        r = R_EARTH + 1e4 * np.abs(lat)
    elif case == "equator":
        lat = np.linspace(0.04, -0.04, 9)
        r = np.full(lat.size, R_EARTH)
    elif case == "polar":
        half = np.linspace(1.5706, 1.2, 70)
        lat = np.concatenate([half, -half[::-1]])
        r = np.full(lat.size, R_EARTH)
    lon = np.arange(2 * n + 2) * (np.pi / (n + 1))
    f, ref = both(cb, cb.PointGrid(lat, lon, r),
                  orc.Point(orc.GRID, lat, lon, r), n)
    assert rel_rms(f, ref) <= tol(n)


def test_columns_that_start_below_the_double_range(cb):
    """nmax 1500 at latitudes whose sectorial values underflow for most
    orders (down to 1e-4800), against the oracle's X-numbers; every row."""
    n = 1500
    half = np.deg2rad(np.concatenate([np.linspace(89.9, 80.0, 40),
                                      np.linspace(79.0, 5.0, 30)]))
    lat = np.concatenate([half, -half[::-1]])
    lon = np.arange(3) * 0.7
    r = np.full(lat.size, R_EARTH)
    f, ref = both(cb, cb.PointGrid(lat, lon, r),
                  orc.Point(orc.GRID, lat, lon, r), n)
    f, ref = f.reshape(lat.size, 3), ref.reshape(lat.size, 3)
    rms = np.sqrt(np.mean(ref ** 2))
    # next to the pole a rounding of the latitude is a phase n / cos(lat)
    amp = 1.0 / np.cos(lat)
    assert np.all(np.abs(f - ref).max(1) <= tol(n) * amp * rms)


# gradients and latitudinal derivatives (families, shs_two.cu) around their
# smallest degree; the rows next to the poles apart, where a rounding of the
# latitude alone is 1 / cos(lat)^2 of the result
@pytest.mark.parametrize("nmax", [127, 128, 163])
@pytest.mark.parametrize("height", [0.0, 2e5])
@pytest.mark.parametrize("kind", ["grad1", "grad2", (0, 1, 0), (0, 2, 0),
                                  (1, 1, 0), (0, 1, 1)])
def test_latitudinal_derivatives(cb, nmax, height, kind):
    p, g = grids(cb, "gl", nmax, R_EARTH + height)
    c, s = model(nmax, 5)
    shc = cb.Shc(nmax, GM, R_EARTH, c, s)
    if kind == "grad1":
        out = cb.shs_point_grad1(p, shc, nmax)
    elif kind == "grad2":
        out = cb.shs_point_grad2(p, shc, nmax)
    else:
        out = [cb.shs_point_guru(p, shc, nmax, *kind)]
    ref = orc.shs_point(g, orc.Shc(nmax, GM, R_EARTH, c, s), nmax, kind)
    u = np.cos(p.lat)
    for f, o in zip(out, ref):
        f = np.asarray(f).reshape(p.lat.size, -1)
        o = np.asarray(o).reshape(p.lat.size, -1)
        rms = np.sqrt(np.mean(o ** 2))
        assert np.all(np.sqrt(np.mean((f - o) ** 2, axis=1))
                      <= 8 * tol(nmax) / u ** 2 * rms)
        keep = u > 0.2
        assert rel_rms(f[keep], o[keep]) <= 16 * tol(nmax)


def test_batch_equals_single_calls(cb):
    """All ten quantities in one pass and three single calls form the same
    sums: the potential, grad1 and grad2 of a set agree bit for bit."""
    import ctypes as ct
    import torch
    from charm_b200._lib import _libcharm as L
    n = 402
    p = cb.PointGridGL(n, R_EARTH + 1e4)
    c, s = kaula(n, 9)
    d = torch.from_numpy(np.stack([c, s])).cuda()
    f = torch.empty((10, p.lat.size, p.lon.size), dtype=torch.float64,
                    device="cuda")
    P = ct.c_void_p
    L.charm_b200_shs_point_batch_dev.argtypes = [
        P, ct.c_size_t, ct.POINTER(ct.c_ulong), ct.POINTER(ct.c_ulong),
        ct.POINTER(ct.c_double), ct.c_double, ct.POINTER(P), ct.POINTER(P),
        ct.c_int, ct.POINTER(P), P]
    nm, mu = (ct.c_ulong * 1)(n), (ct.c_double * 1)(GM)
    err = L.charm_err_init()
    L.charm_b200_shs_point_batch_dev(
        ct.cast(p._Point, P), 1, nm, nm, mu, R_EARTH,
        (P * 1)(d[0].data_ptr()), (P * 1)(d[1].data_ptr()), 3,
        (P * 1)(f.data_ptr()), ct.cast(err, P))
    assert L.charm_err_isempty(err)
    L.charm_err_free(err)
    shc = cb.Shc(n, GM, R_EARTH, c, s)
    one = ([cb.shs_point(p, shc, n)] + list(cb.shs_point_grad1(p, shc, n))
           + list(cb.shs_point_grad2(p, shc, n)))
    for q in range(10):
        assert np.array_equal(f[q].cpu().numpy(), np.asarray(one[q])), q


# either side of the rule's smallest grid (384 pairs, degree 512), whole and
# partial tiles, degrees below the grid's, a triangle larger than the degree
@pytest.mark.parametrize("name,grid_nmax,nmax", [
    ("gl", 765, 765), ("gl", 766, 766), ("gl", 767, 511), ("gl", 800, 700),
    ("dh1", 511, 511), ("dh1", 513, 513), ("dh2", 512, 512)])
@pytest.mark.parametrize("height", [0.0, 5e3])
def test_analysis(cb, name, grid_nmax, nmax, height):
    r = R_EARTH + height
    p, g = grids(cb, name, grid_nmax, r)
    c, s = model(nmax, 11)
    f = np.asarray(cb.shs_point(p, cb.Shc(nmax, GM, R_EARTH, c, s), nmax))
    out = cb.sha_point(p, f, nmax, GM, r)
    ref = orc.sha_point(g, f, nmax, GM, r)
    assert coef_rel_rms(out.c, out.s, ref.c, ref.s) <= tol(nmax)
    # every degree and order on its own scale: a wrong weight of one column
    # or parity would hide in the whole
    n = np.concatenate([np.arange(m, nmax + 1) for m in range(nmax + 1)])
    size = np.sqrt(np.bincount(n, c ** 2 + s ** 2)) / np.sqrt(2.0 * np.arange(
        nmax + 1) + 1.0)
    size[:2] = size[2]
    err = np.hypot(out.c - ref.c, out.s - ref.s)
    assert np.all(err <= 200 * tol(nmax) * size[2])
    high = (n > nmax // 2)
    assert np.sqrt(np.mean(err[high] ** 2)) <= tol(nmax) * size[2]
