"""Workloads of the transforms, from the smallest calls to the largest grids,
through the public entry points a program uses: the device-array calls of the
C ABI, the PyHarm-style calls on numpy arrays and the differentiable
scattered synthesis.

Operations (`op` of a case):

roundtrip  synthesis of a grid and analysis of that grid, device arrays, FP64
           (charm_b200_shs_point_dev, charm_b200_sha_point_dev) or single
           precision (..._dev_f32); `height` in metres above the
           coefficients' sphere
sets       many coefficient sets on one grid (charm_b200_shs_point_batch_dev,
           or the split-precision ..._batch_i8_dev): the potential (kgrad 0)
           or the potential with grad1 and grad2 (kgrad 3)
gradient   grad1 or grad2 of one set (charm_b200_shs_point_dev)
points     potential at scattered points and its gradient with respect to
           the coefficients (charm_b200.autograd, forward and backward)
cells      block means in the cells of a grid and their analysis
           (charm_b200_shs_cell_dev, charm_b200_sha_cell_dev)
forward    global gravity forward modelling (gfm_global_density_3d)
host       synthesis and analysis of numpy arrays (shs_point, sha_point)
"""
import ctypes as ct
import math

import numpy as np
import torch

import charm_b200 as cb
from charm_b200._lib import _libcharm as _L
from charm_b200.autograd import shs_point_sctr
from charm_b200.workloads import GM, R_EARTH

_P, _D, _U = ct.c_void_p, ct.c_double, ct.c_ulong
_PU, _PD, _PP = ct.POINTER(_U), ct.POINTER(_D), ct.POINTER(_P)
_L.charm_b200_shs_point_dev.argtypes = [
    _P, _U, _D, _D, _P, _P, _U, ct.c_int, ct.c_uint, ct.c_uint, ct.c_uint, _P,
    _P]
_L.charm_b200_sha_point_dev.argtypes = [_P, _P, _U, _D, _D, _U, _P, _P, _P]
_L.charm_b200_shs_point_dev_f32.argtypes = [_P, _U, _D, _D, _P, _P, _U, _P, _P]
_L.charm_b200_sha_point_dev_f32.argtypes = [_P, _P, _U, _D, _D, _U, _P, _P, _P]
for _n in ("charm_b200_shs_point_batch_dev",
           "charm_b200_shs_point_batch_i8_dev"):
    getattr(_L, _n).argtypes = [_P, ct.c_size_t, _PU, _PU, _PD, _D, _PP, _PP,
                                ct.c_int, _PP, _P]
_L.charm_b200_shs_cell_dev.argtypes = [_P, _U, _D, _D, _P, _P, _U, _P, _P]
_L.charm_b200_sha_cell_dev.argtypes = [_P, _P, _U, _D, _D, _U, _P, _P, _P]

_GRIDS = {"gl": cb.PointGridGL, "dh1": cb.PointGridDH1, "dh2": cb.PointGridDH2}
_NCOMP = {0: 1, 1: 3, 2: 6, 3: 10}

# the body of the forward modelling: mean radius, constant of gravitation, mass
_R_BODY, _G, _MASS = 1728000.0, 6.67430e-11, 7.346e22


def listed():
    return [
        # a regional or teaching-size model, called many times: latency
        {"name": "roundtrip_gl_47", "op": "roundtrip", "grid": "gl",
         "nmax": 47, "height": 0.0, "f32": False},
        # the degree of the classical global gravity models
        {"name": "roundtrip_gl_360", "op": "roundtrip", "grid": "gl",
         "nmax": 360, "height": 0.0, "f32": False},
        # equiangular grid at flight height, continued down to the sphere
        {"name": "roundtrip_dh2_719_high", "op": "roundtrip", "grid": "dh2",
         "nmax": 719, "height": 10000.0, "f32": False},
        # high-degree global gravity models
        {"name": "roundtrip_gl_2190", "op": "roundtrip", "grid": "gl",
         "nmax": 2190, "height": 0.0, "f32": False},
        # ultra-high-degree topographic potential models
        {"name": "roundtrip_gl_10800", "op": "roundtrip", "grid": "gl",
         "nmax": 10800, "height": 0.0, "f32": False},
        # the same transforms for callers content with single precision
        {"name": "roundtrip_f32_gl_1441", "op": "roundtrip", "grid": "gl",
         "nmax": 1441, "height": 0.0, "f32": True},
        # an ensemble of models, the potential and its derivatives up to the
        # second order at satellite height
        {"name": "ten_quantities_gl_540", "op": "sets", "grid": "gl",
         "nmax": 540, "height": 250000.0, "nsets": 8, "kgrad": 3,
         "split": False},
        # a larger ensemble, the potential alone on the tensor cores
        {"name": "split_sets_gl_1000", "op": "sets", "grid": "gl",
         "nmax": 1000, "height": 0.0, "nsets": 20, "kgrad": 0, "split": True},
        # one iteration of a least-squares fit to scattered observations
        {"name": "points_360", "op": "points", "nmax": 360, "npoint": 60001},
        # block means (the usual form of terrestrial gravity anomalies)
        {"name": "cells_719", "op": "cells", "nmax": 719, "nlat": 720},
        # potential of a body from its shape and density
        {"name": "forward_360", "op": "forward", "nmax": 360, "density": 180,
         "powers": 5, "potential": 720},
        # a PyHarm script on numpy arrays
        {"name": "host_gl_1000", "op": "host", "grid": "gl", "nmax": 1000},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["roundtrip"] * 5 + ["sets"] * 2 + ["gradient", "points",
                                                        "cells", "forward",
                                                        "host"])
    grid = rng.choice(["gl", "gl", "dh1", "dh2"])
    height = rng.choice([0.0, 0.0, float(rng.randrange(1000, 500000))])
    if op == "roundtrip":
        f32 = rng.random() < 0.15
        nmax = _log_int(rng, 24, 2200 if f32 or grid == "dh2" else 5400)
        # downward continuation multiplies degree n by (r / R)^n: e^3 at most
        height = 0.0 if f32 else min(height, 3.0 * R_EARTH / nmax)
        return {"op": op, "grid": grid, "height": height, "nmax": nmax,
                "f32": f32}
    if op == "sets":
        kgrad = rng.choice([0, 3])
        return {"op": op, "grid": "gl" if kgrad else grid, "height": height,
                "nmax": _log_int(rng, 60, 800 if kgrad else 1300),
                "nsets": rng.randrange(2, 9 if kgrad else 25),
                "kgrad": kgrad, "split": rng.random() < 0.4}
    if op == "gradient":
        return {"op": op, "grid": "gl", "height": height,
                "nmax": _log_int(rng, 60, 2190), "kgrad": rng.choice([1, 2])}
    if op == "points":
        nmax = _log_int(rng, 60, 720)
        return {"op": op, "nmax": nmax,
                "npoint": _log_int(rng, 1000, 60000 * 360 ** 2 // nmax ** 2
                                   + 2000)}
    if op == "cells":
        nmax = _log_int(rng, 60, 1500)
        return {"op": op, "nmax": nmax, "nlat": nmax + rng.randrange(1, 40)}
    if op == "forward":
        nmax = _log_int(rng, 40, 360)
        return {"op": op, "nmax": nmax, "density": rng.randrange(10, nmax),
                "powers": rng.randrange(2, 6),
                "potential": nmax + rng.randrange(0, nmax + 1)}
    return {"op": op, "grid": grid, "nmax": _log_int(rng, 30, 1800)}


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------
def _dev():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _tri(nmax):
    return (nmax + 1) * (nmax + 2) // 2


def _degrees_orders(nmax):
    """Degree and order of every entry of the order-major triangle."""
    dev = _dev()
    m = torch.arange(nmax + 1, device=dev)
    count = nmax + 1 - m
    start = torch.cumsum(count, 0) - count
    om = torch.repeat_interleave(m, count)
    return torch.arange(_tri(nmax), device=dev) - start[om] + om, om


def _model(nmax, seed, c00=1.0):
    """Triangles C, S ([2][T]) with Kaula's degree variances and C_00."""
    n, m = _degrees_orders(nmax)
    g = torch.Generator(device=_dev())
    g.manual_seed(seed)
    sig = 1e-5 / n.double().clamp(min=1).square() / (2.0 * n + 1.0).sqrt()
    sig[n < 2] = 0.0
    cs = torch.randn((2, n.numel()), generator=g, device=_dev(),
                     dtype=torch.float64) * sig
    cs[1, m == 0] = 0.0
    cs[0, 0] = c00
    return cs


def _body(nmax, seed, relief, c00):
    rng = np.random.default_rng(seed)
    n = np.concatenate([np.arange(m, nmax + 1) for m in range(nmax + 1)])
    sig = relief / (1.0 + n) ** 2
    c, s = rng.standard_normal(n.size) * sig, rng.standard_normal(n.size) * sig
    s[:nmax + 1] = 0.0
    c[0] = c00
    return c, s


def _set_degrees(case):
    """Degrees of an ensemble: from the largest down to a third of it."""
    N, k = case["nmax"], case["nsets"]
    return [max(2, N - (2 * N // 3) * j // max(1, k - 1)) for j in range(k)]


def _scattered(case, seed):
    rng = np.random.default_rng(seed + 1)
    npt = case["npoint"]
    return (np.arcsin(rng.uniform(-1.0, 1.0, npt)),
            rng.uniform(0.0, 2.0 * np.pi, npt),
            R_EARTH + rng.uniform(0.0, 9000.0, npt), rng.standard_normal(npt))


def _cell_bounds(case):
    nlat, nlon = case["nlat"], 2 * case["nlat"]
    lat = np.pi / 2 - np.arange(nlat + 1) / nlat * np.pi
    lon = np.arange(nlon + 1) / nlon * 2.0 * np.pi
    return lat[1:].copy(), lat[:-1].copy(), lon[:-1].copy(), lon[1:].copy()


def prepare(case, seed):
    op = case["op"]
    st = {"op": op, "case": case}
    if op in ("roundtrip", "sets", "gradient", "host"):
        st["pnt"] = p = _GRIDS[case["grid"]](
            case["nmax"], R_EARTH + case.get("height", 0.0))
        shape = (p.lat.size, p.lon.size)
    if op in ("roundtrip", "gradient"):
        dt = torch.float32 if case.get("f32") else torch.float64
        st["cs"] = _model(case["nmax"], seed).to(dt)
        nq = _NCOMP[case.get("kgrad", 0)]
        st["f"] = torch.empty((nq,) + shape, dtype=dt, device="cuda")
        if op == "roundtrip":
            st["out"] = torch.empty_like(st["cs"])
    elif op == "sets":
        nm = _set_degrees(case)
        k = len(nm)
        st["models"] = [_model(n, 1000 * seed + j) for j, n in enumerate(nm)]
        st["f"] = [torch.empty((_NCOMP[case["kgrad"]],) + shape,
                               dtype=torch.float64, device="cuda")
                   for _ in range(k)]
        st["nm"] = (_U * k)(*nm)
        st["mu"] = (_D * k)(*[GM] * k)
        st["pc"] = (_P * k)(*[m[0].data_ptr() for m in st["models"]])
        st["ps"] = (_P * k)(*[m[1].data_ptr() for m in st["models"]])
        st["pf"] = (_P * k)(*[f.data_ptr() for f in st["f"]])
    elif op == "points":
        lat, lon, r, w = _scattered(case, seed)
        st["pnt"] = cb.PointSctr(lat, lon, r)
        st["w"] = torch.from_numpy(w).cuda()
        st["cs"] = _model(case["nmax"], seed)
    elif op == "cells":
        st["cell"] = cb.CellGrid(*_cell_bounds(case),
                                 np.full(case["nlat"], R_EARTH))
        st["cs"] = _model(case["nmax"], seed)
        st["f"] = torch.empty((case["nlat"], 2 * case["nlat"]),
                              dtype=torch.float64, device="cuda")
        st["out"] = torch.empty_like(st["cs"])
    elif op == "forward":
        nd = [case["density"], case["density"] // 2]
        st["nd"] = nd
        st["shape"] = cb.Shc(case["nmax"], 1.0, 1.0, *_body(
            case["nmax"], seed, 3000.0, _R_BODY + 1700.0))
        st["dens"] = [cb.Shc(nd[0], 1.0, 1.0,
                             *_body(nd[0], seed + 1, 80.0, 2500.0)),
                      cb.Shc(nd[1], 1.0, 1.0,
                             *_body(nd[1], seed + 2, 1e-6, -2e-5))]
    else:
        # a disturbing potential: no degree-0 term
        c, s = _model(case["nmax"], seed, 0.0).cpu().numpy()
        st["shc"] = cb.Shc(case["nmax"], GM, R_EARTH, c, s)
    return st


# ---------------------------------------------------------------------------
# One pass
# ---------------------------------------------------------------------------
def _call(fn, *args):
    err = _L.charm_err_init()
    try:
        fn(*args, ct.cast(err, _P))
        if not _L.charm_err_isempty(err):
            raise RuntimeError(ct.string_at(err.contents.msg).decode())
    finally:
        _L.charm_err_free(err)


def run(st):
    op, case = st["op"], st["case"]
    N = case["nmax"]
    if op == "roundtrip":
        pnt = ct.cast(st["pnt"]._Point, _P)
        f = st["f"].data_ptr()
        (c, s), (oc, os) = ([t.data_ptr() for t in st[k]]
                            for k in ("cs", "out"))
        if case["f32"]:
            _call(_L.charm_b200_shs_point_dev_f32, pnt, N, GM, R_EARTH, c, s,
                  N, f)
            _call(_L.charm_b200_sha_point_dev_f32, pnt, f, N, GM, R_EARTH, N,
                  oc, os)
        else:
            _call(_L.charm_b200_shs_point_dev, pnt, N, GM, R_EARTH, c, s, N,
                  0, 0, 0, 0, f)
            _call(_L.charm_b200_sha_point_dev, pnt, f, N, GM, R_EARTH, N, oc,
                  os)
        return [st["f"], st["out"]]
    if op == "gradient":
        _call(_L.charm_b200_shs_point_dev, ct.cast(st["pnt"]._Point, _P), N,
              GM, R_EARTH, st["cs"][0].data_ptr(), st["cs"][1].data_ptr(), N,
              case["kgrad"], 0, 0, 0, st["f"].data_ptr())
        return st["f"]
    if op == "sets":
        fn = (_L.charm_b200_shs_point_batch_i8_dev if case["split"]
              else _L.charm_b200_shs_point_batch_dev)
        _call(fn, ct.cast(st["pnt"]._Point, _P), len(st["nm"]), st["nm"],
              st["nm"], st["mu"], R_EARTH, st["pc"], st["ps"], case["kgrad"],
              st["pf"])
        return st["f"]
    if op == "points":
        c, s = (t.detach().requires_grad_() for t in st["cs"])
        f = shs_point_sctr(c, s, st["pnt"], N, GM, R_EARTH)
        f.backward(st["w"])
        return [f.detach(), c.grad, s.grad]
    if op == "cells":
        cell = ct.cast(st["cell"]._Cell, _P)
        f = st["f"].data_ptr()
        (c, s), (oc, os) = ([t.data_ptr() for t in st[k]]
                            for k in ("cs", "out"))
        _call(_L.charm_b200_shs_cell_dev, cell, N, GM, R_EARTH, c, s, N, f)
        _call(_L.charm_b200_sha_cell_dev, cell, f, N, GM, R_EARTH, N, oc, os)
        return [st["f"], st["out"]]
    if op == "forward":
        pot = cb.gfm_global_density_3d(
            st["shape"], N, _R_BODY, st["dens"], st["nd"], 1, _G, _MASS, 1,
            case["powers"], case["potential"])
        return [pot.c, pot.s]
    f = cb.shs_point(st["pnt"], st["shc"], N)
    out = cb.sha_point(st["pnt"], f, N, GM, R_EARTH)
    return [f, out.c, out.s]


# ---------------------------------------------------------------------------
# What a pass cannot do without: inputs read and outputs written once; per
# (degree, order, latitude pair) two fused sums and one for the Legendre
# value; the rows' transforms
# ---------------------------------------------------------------------------
def _rows(case):
    N = case["nmax"]
    return {"gl": (N + 1, 2 * N + 2), "dh1": (2 * N + 2, 2 * N + 2),
            "dh2": (2 * N + 2, 4 * N + 4)}[case["grid"]]


def work(case):
    op, N = case["op"], case["nmax"]
    T = _tri(N)

    def grid(nlat, nlon, terms, quantities=1):
        fft = 2.5 * nlon * math.log2(nlon) * nlat * quantities
        return 6.0 * terms * ((nlat + 1) // 2) + fft

    if op in ("roundtrip", "host", "gradient"):
        nlat, nlon = _rows(case)
        size = 4 if case.get("f32") else 8
        nq = _NCOMP[case.get("kgrad", 0)]
        ways = 1 if op == "gradient" else 2
        return {"bytes": ways * size * (2 * T + nq * nlat * nlon),
                "flops": ways * grid(nlat, nlon, T, nq)}
    if op == "sets":
        nlat, nlon = _rows(case)
        nq = _NCOMP[case["kgrad"]]
        nm = _set_degrees(case)
        return {"bytes": sum(8 * (2 * _tri(n) + nq * nlat * nlon) for n in nm),
                "flops": sum(grid(nlat, nlon, _tri(n), nq) for n in nm)}
    if op == "points":
        return {"bytes": 2 * 8 * (2 * T + 4 * case["npoint"]),
                "flops": 2 * 6.0 * T * case["npoint"]}
    if op == "cells":
        nlat, nlon = case["nlat"], 2 * case["nlat"]
        return {"bytes": 2 * 8 * (2 * T + nlat * nlon),
                "flops": 2 * grid(nlat, nlon, 2 * T)}
    flops = 0.0
    for p in range(1, case["powers"] + 1):
        n = p * N + case["density"]
        flops += 2 * grid(n + 1, 2 * n + 2, _tri(min(n, case["potential"])))
        flops += grid(n + 1, 2 * n + 2, T)
    return {"bytes": 16 * (T + 2 * _tri(case["density"])
                           + _tri(case["potential"])), "flops": flops}


# ---------------------------------------------------------------------------
# The same in plain 64-bit torch and numpy: dense sums over degrees for all
# orders and latitudes at once
# ---------------------------------------------------------------------------
def _dense(tri, nmax, top):
    """[n][m] array of degree `top` from an order-major triangle."""
    n, m = _degrees_orders(nmax)
    out = torch.zeros((top + 1, top + 1), dtype=torch.float64, device=_dev())
    out[n, m] = tri.double()
    return out


def _triangle(dense, nmax):
    n, m = _degrees_orders(nmax)
    return dense[n, m]


def _legendre(nmax, lat):
    """Yields (n, P_n, P_n-1, e_n): fully normalised Legendre functions
    [order m <= n][latitude] for n = 0..nmax and e with
    cos(lat) dP_n = e_n P_n-1 - n sin(lat) P_n.  Values whose sectorial seed
    underflows carry an exponent until they have grown back."""
    lat = np.asarray(lat, np.float64)
    lo = lat.astype(np.longdouble)
    u = np.cos(lo)
    seeds = np.ones((nmax + 1, lat.size), np.longdouble)
    f = np.ones(nmax + 1, np.longdouble)
    k = np.arange(1, nmax + 1, dtype=np.longdouble)
    f[1:] = np.sqrt((2 * k + 1) / (2 * k))
    if nmax >= 1:
        f[1] = np.sqrt(np.longdouble(3))
    np.cumprod(f[1:, None] * u[None, :], axis=0, out=seeds[1:])
    mant, expo = np.frexp(seeds)
    dev = _dev()
    x = torch.from_numpy(mant.astype(np.float64)).to(dev)
    E = torch.from_numpy(expo.astype(np.int32)).to(dev)
    small = E < -900
    x = torch.where(small, x, torch.ldexp(x, torch.where(small, 0, E)))
    E = torch.where(small, E, 0)
    live = (~small).double()
    y = torch.zeros_like(x)
    t = torch.from_numpy(np.sin(lo).astype(np.float64)).to(dev)[None, :]
    m = torch.arange(nmax + 1, device=dev, dtype=torch.float64)[:, None]
    for n in range(nmax + 1):
        a = slice(0, n + 1)
        if n > 0:
            b = slice(0, n)
            mm = m[b]
            w = torch.sqrt((2.0 * n + 1.0) / ((n - mm) * (n + mm)))
            bb = torch.sqrt(((n - 1.0) ** 2 - mm * mm).clamp(min=0.0)
                            / max(2.0 * n - 3.0, 1.0))
            z = w * (math.sqrt(2.0 * n - 1.0) * t * x[b] - bb * y[b])
            y[b] = x[b]
            x[b] = z
            if n % 16 == 0 and bool(small.any()):
                big = torch.maximum(x.abs(), y.abs())
                ex = torch.frexp(big)[1]
                started = (torch.arange(nmax + 1, device=dev) < n)[:, None]
                work_ = small & started & (big > 0)
                tot = E + ex
                back = work_ & (tot >= -900)
                shift = torch.where(back, E, torch.where(work_, -ex, 0))
                x, y = torch.ldexp(x, shift), torch.ldexp(y, shift)
                E = torch.where(back, 0, torch.where(work_, tot, E))
                small = small & ~back
                live = (~small).double()
        mm = m[a]
        e = torch.sqrt((n * n - mm * mm) * (2.0 * n + 1.0)
                       / max(2.0 * n - 1.0, 1.0))
        yield n, x[a] * live[a], y[a] * live[a], e


def _rows_from(a, b, nlon):
    """Grid rows sum_m a cos(m lon) + b sin(m lon), [m][lat] inputs."""
    X = torch.zeros((a.shape[1], nlon // 2 + 1), dtype=torch.complex128,
                    device=a.device)
    k = min(a.shape[0], nlon // 2 + 1)
    X[:, :k] = torch.complex(a[:k].T.contiguous(), -b[:k].T.contiguous())
    X[:, 1:] *= 0.5
    return torch.fft.irfft(X, n=nlon, dim=1) * nlon


def _lumped(c, s, nmax, lat, rho, powers):
    """sum_n w(n) rho^(n+1) (C, S) P for the weights named by `powers`:
    functions of (n, P, dP, ddP, weight) -> value."""
    C, S = _dense(c, nmax, nmax), _dense(s, nmax, nmax)
    out = [[torch.zeros((nmax + 1, len(lat)), dtype=torch.float64,
                        device=_dev()) for _ in range(2)] for _ in powers]
    lo = np.asarray(lat, np.longdouble)
    dev = _dev()
    t = torch.from_numpy(np.sin(lo).astype(np.float64)).to(dev)[None]
    u = torch.from_numpy(np.cos(lo).astype(np.float64)).to(dev)[None]
    deriv = len(powers) > 1
    for n, P, Q, e in _legendre(nmax, lat):
        dP = ddP = None
        if deriv:
            m = torch.arange(n + 1, device=dev, dtype=torch.float64)[:, None]
            dP = (e * Q - n * t * P) / u
            ddP = (t / u) * dP + ((m / u) ** 2 - n * (n + 1.0)) * P
        for (A, B), fn in zip(out, powers):
            v = fn(n, P, dP, ddP) * rho ** (n + 1)
            A[:n + 1] += C[n, :n + 1, None] * v
            B[:n + 1] += S[n, :n + 1, None] * v
    return out


def _potential(c, s, nmax, lat, nlon, r):
    (A, B), = _lumped(c, s, nmax, lat, R_EARTH / r,
                      [lambda n, P, dP, ddP: P])
    return _rows_from(A, B, nlon) * (GM / R_EARTH)


def _ten(c, s, nmax, lat, nlon, r):
    """V; x, y, z; xx, xy, xz, yy, yz, zz in the local north-oriented frame
    (x north, y west, z up)."""
    rho = R_EARTH / r
    P, P1, P2, D, D1, DD = _lumped(c, s, nmax, lat, rho, [
        lambda n, p, d, dd: p, lambda n, p, d, dd: (n + 1) * p,
        lambda n, p, d, dd: (n + 1) * (n + 2) * p, lambda n, p, d, dd: d,
        lambda n, p, d, dd: (n + 1) * d, lambda n, p, d, dd: dd])
    lo = np.asarray(lat, np.longdouble)
    dev = _dev()
    u = torch.from_numpy(np.cos(lo).astype(np.float64)).to(dev)[None]
    t = torch.from_numpy(np.sin(lo).astype(np.float64)).to(dev)[None]
    m = torch.arange(nmax + 1, device=dev, dtype=torch.float64)[:, None]

    def lon(q):             # derivative along the parallel
        return m * q[1], -m * q[0]

    def comb(*terms):
        return tuple(sum(w * q[i] for w, q in terms) for i in (0, 1))

    k0, k1, k2 = GM / R_EARTH, GM / R_EARTH ** 2 * rho, \
        GM / R_EARTH ** 3 * rho ** 2
    q = [(k0, P), (k1, D), (k1, comb((-1.0 / u, lon(P)))),
         (k1, comb((-1.0, P1))),
         (k2, comb((1.0, DD), (-1.0, P1))),
         (k2, comb((-1.0 / u, lon(D)), (-t / u / u, lon(P)))),
         (k2, comb((-1.0, D1), (-1.0, D))),
         (k2, comb((-(m / u) ** 2, P), (-t / u, D), (-1.0, P1))),
         (k2, comb((1.0 / u, lon(P)), (1.0 / u, lon(P1)))),
         (k2, P2)]
    return torch.stack([k * _rows_from(a, b, nlon) for k, (a, b) in q])


def _gl_nodes(nmax):
    """Latitudes (north to south) and weights of the Gauss--Legendre grid."""
    L = nmax + 1
    x = np.cos(np.pi * (np.arange(L) + 0.75) / (L + 0.5)).astype(np.longdouble)
    for _ in range(5):
        p0, p1 = np.ones_like(x), x.copy()
        for n in range(2, L + 1):
            p0, p1 = p1, ((2 * n - 1) * x * p1 - (n - 1) * p0) / n
        dp = L * (x * p1 - p0) / (x * x - 1)
        x = x - p1 / dp
    return np.arcsin(x).astype(np.float64), (2 / ((1 - x * x) * dp * dp)
                                             ).astype(np.float64)


def _analyse(f, lat, w, nmax):
    """C, S ([n][m]) of the grid f by quadrature with the latitude weights."""
    nlon = f.shape[1]
    X = torch.fft.rfft(f, dim=1)[:, :nmax + 1].T * (2.0 * math.pi / nlon)
    X = X * torch.from_numpy(w).to(f.device)[None] / (4.0 * math.pi)
    C = torch.zeros((nmax + 1, nmax + 1), dtype=torch.float64, device=f.device)
    S = torch.zeros_like(C)
    re, im = X.real.contiguous(), X.imag.contiguous()
    for n, P, _, _ in _legendre(nmax, lat):
        C[n, :n + 1] = (P * re[:n + 1]).sum(1)
        S[n, :n + 1] = -(P * im[:n + 1]).sum(1)
    return C, S


def _grid_lats(case):
    N = case["nmax"]
    if case["grid"] == "gl":
        return _gl_nodes(N)[0]
    return math.pi / 2 - np.pi * np.arange(2 * N + 2) / (2 * N + 2)


def _exact_points(case, seed):
    N = case["nmax"]
    lat, lon, r, w = _scattered(case, seed)
    c, s = _model(N, seed)
    C, S = _dense(c, N, N), _dense(s, N, N)
    gC, gS = torch.zeros_like(C), torch.zeros_like(S)
    out = []
    for i in range(0, lat.size, 1 << 16):
        k = slice(i, i + (1 << 16))
        rho = torch.from_numpy(R_EARTH / r[k]).to(c.device)
        g = torch.from_numpy(w[k]).to(c.device)
        m = torch.arange(N + 1, device=c.device, dtype=torch.float64)[:, None]
        ang = m * torch.from_numpy(lon[k]).to(c.device)[None]
        cm, sm = torch.cos(ang), torch.sin(ang)
        f, pw = torch.zeros_like(rho), rho.clone()
        for n, P, _, _ in _legendre(N, lat[k]):
            a = slice(0, n + 1)
            vc, vs = P * cm[a] * pw, P * sm[a] * pw
            f += C[n, a] @ vc + S[n, a] @ vs
            gC[n, a] += vc @ g
            gS[n, a] += vs @ g
            pw = pw * rho
        out.append(f)
    k = GM / R_EARTH
    return [k * torch.cat(out), k * _triangle(gC, N), k * _triangle(gS, N)]


def _exact_cells(case, seed):
    N, nlat, nlon = case["nmax"], case["nlat"], 2 * case["nlat"]
    c, s = _model(N, seed)
    lo, hi, west, east = (b.astype(np.longdouble) for b in _cell_bounds(case))
    x, w = np.polynomial.legendre.leggauss(12)
    nodes = (0.5 * (lo + hi))[:, None] + (0.5 * (hi - lo))[:, None] * x[None]
    wt = (0.5 * (hi - lo))[:, None] * w[None] * np.cos(nodes)
    wt = torch.from_numpy(wt.astype(np.float64)).to(c.device)
    m = torch.arange(N + 1, device=c.device, dtype=torch.float64)[:, None]
    d = 2.0 * math.pi / nlon
    width = torch.where(m > 0, 2.0 / m.clamp(min=1.0)
                        * torch.sin(0.5 * m * d), torch.full_like(m, d))
    mid = torch.from_numpy((0.5 * (west + east)).astype(np.float64)).to(
        c.device)[None]
    cm, sm = width * torch.cos(m * mid), width * torch.sin(m * mid)
    area = torch.from_numpy(((np.sin(hi) - np.sin(lo)) * d).astype(
        np.float64)).to(c.device)
    C, S = _dense(c, N, N), _dense(s, N, N)
    A, B = (torch.zeros((N + 1, nlat), dtype=torch.float64, device=c.device)
            for _ in range(2))
    lat = nodes.astype(np.float64).ravel()
    for n, P, _, _ in _legendre(N, lat):
        I = (P.view(n + 1, nlat, 12) * wt[None]).sum(2)
        A[:n + 1] += C[n, :n + 1, None] * I
        B[:n + 1] += S[n, :n + 1, None] * I
    f = GM / R_EARTH * (A.T @ cm + B.T @ sm) / area[:, None]
    Fc, Fs = cm @ f.T, sm @ f.T
    oC, oS = torch.zeros_like(C), torch.zeros_like(S)
    for n, P, _, _ in _legendre(N, lat):
        I = (P.view(n + 1, nlat, 12) * wt[None]).sum(2)
        oC[n, :n + 1] = (I * Fc[:n + 1]).sum(1)
        oS[n, :n + 1] = (I * Fs[:n + 1]).sum(1)
    k = R_EARTH / (4.0 * math.pi * GM)
    return [f, k * torch.stack([_triangle(oC, N), _triangle(oS, N)])]


def _exact_forward(case, seed):
    N, nd = case["nmax"], [case["density"], case["density"] // 2]
    top = case["potential"]
    sets = [(N, _body(N, seed, 3000.0, _R_BODY + 1700.0)),
            (nd[0], _body(nd[0], seed + 1, 80.0, 2500.0)),
            (nd[1], _body(nd[1], seed + 2, 1e-6, -2e-5))]
    sets = [(n, torch.from_numpy(c).to(_dev()), torch.from_numpy(s).to(_dev()))
            for n, (c, s) in sets]
    pot = [torch.zeros((top + 1, top + 1), dtype=torch.float64, device=_dev())
           for _ in range(2)]
    for p in range(1, case["powers"] + 1):
        ng = p * N + nd[0]
        lat, w = _gl_nodes(ng)
        fields = []
        for n, c, s in sets:
            (A, B), = _lumped(c, s, n, lat, 1.0, [lambda n, P, d, dd: P])
            fields.append(_rows_from(A, B, 2 * ng + 2))
        rel = ((fields[0] - _R_BODY) / _R_BODY) ** p
        na = min(ng, top)
        for i in (0, 1):
            C, S = _analyse(fields[1 + i] * rel * _R_BODY ** i, lat, w, na)
            n = torch.arange(na + 1, device=_dev(), dtype=torch.float64)
            k = 2.0 * math.pi * _R_BODY ** 3 / _MASS * 2.0 / (
                (2.0 * n + 1.0) * (n + i + 3.0)) * (n + i + 3.0) / p
            for q in range(1, p):
                k = k * (n + i + 3.0 - q) / (p - q)
            pot[0][:na + 1, :na + 1] += C * k[:, None]
            pot[1][:na + 1, :na + 1] += S * k[:, None]
    return [_triangle(pot[0], top), _triangle(pot[1], top)]


def exact(case, seed):
    op, N = case["op"], case["nmax"]
    if N > 3000:
        return None
    if op in ("roundtrip", "host"):
        cs = _model(N, seed, 0.0 if op == "host" else 1.0)
        if case.get("f32"):
            cs = cs.float().double()
        f = _potential(cs[0], cs[1], N, _grid_lats(case), _rows(case)[1],
                       R_EARTH + case.get("height", 0.0))
        return [f[None], cs] if op == "roundtrip" else [f, cs[0], cs[1]]
    if op == "gradient":
        c, s = _model(N, seed)
        ten = _ten(c, s, N, _grid_lats(case), _rows(case)[1],
                   R_EARTH + case["height"])
        x, y, z, xx, xy, xz, yy, yz, zz = ten[1:]
        # the device call's order: l, r, p and ll, lr, lp, rr, rp, pp
        return torch.stack([y, z, x] if case["kgrad"] == 1
                           else [yy, yz, xy, zz, xz, xx])
    if op == "sets":
        lat, nlon = _grid_lats(case), _rows(case)[1]
        r = R_EARTH + case["height"]
        out = []
        for j, n in enumerate(_set_degrees(case)):
            c, s = _model(n, 1000 * seed + j)
            out.append(_ten(c, s, n, lat, nlon, r) if case["kgrad"] == 3
                       else _potential(c, s, n, lat, nlon, r)[None])
        return out
    if op == "points":
        return _exact_points(case, seed)
    if op == "cells":
        return _exact_cells(case, seed)
    return _exact_forward(case, seed)
