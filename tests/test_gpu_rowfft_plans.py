"""The longitude transforms of every one-CTA plan (transform lengths M = 2^a 3^b
from 64 to 9216): the shortest and the longest rows that a plan serves by
Bluestein's algorithm, fewer rows than share a CTA and one more than they, both
directions and both widths; and rows of several blocks in one launch against
one block alone for the plans that are not fixed at compile time.

The tolerances are those of the other tests of these transforms: 1e-13 against
numpy's inverse transform of the oracle's spectra, 1e-12 for the coefficients
back from a grid, 1e-6 and 1e-4 in single precision.  Blocks of one launch and
a block alone run the same operations, compiled twice: 1e-14."""
import ctypes as ct

import numpy as np
import pytest

from charm_b200.workloads import GM, R_EARTH, coef_rel_rms, kaula, rel_rms
from test_gpu_batch import batch, env  # noqa: F401 (a fixture)
from test_gpu_f32 import sha32, shs32
from test_gpu_rowfft import TOL, oracle_rows

pytestmark = pytest.mark.gpu

LENGTHS = sorted(m for a in range(6, 14) for b in range(5)
                 for m in [2 ** a * 3 ** b] if m <= 9216)


def direct(H):
    a = b = 0
    while H % 2 == 0:
        H, a = H // 2, a + 1
    while H % 3 == 0:
        H, b = H // 3, b + 1
    return H == 1 and a >= 6


def halves(M):
    """The least and the largest half length that Bluestein's algorithm takes
    to length M."""
    k = LENGTHS.index(M)
    lo = (LENGTHS[k - 1] + 1) // 2 + 1 if k else 9
    fit = [H for H in range(lo, (M + 1) // 2 + 1) if not direct(H)]
    return fit[0], fit[-1]


@pytest.mark.parametrize("M", LENGTHS)
def test_synthesis(M):
    import charm_b200 as cb
    for H in set(halves(M)):
        nlon, N = 2 * H, min(H - 1, 300)
        c, s = kaula(N, M + H)
        lon = 2.0 * np.pi * np.arange(nlon) / nlon
        for nlat in (3, 17):
            lat = np.linspace(1.3, -1.2, nlat)
            p = cb.PointGrid(lat, lon, np.full(nlat, R_EARTH))
            f = cb.shs_point(p, cb.Shc(N, GM, R_EARTH, c, s), N)
            assert rel_rms(f, oracle_rows(lat, nlon, N, c, s)) <= TOL, H


@pytest.mark.parametrize("M", [m for m in LENGTHS if m <= 8192])
def test_analysis(M):
    import charm_b200 as cb
    N = halves(M)[1] - 1
    c, s = kaula(N, M)
    p = cb.PointGridGL(N, R_EARTH)
    f = cb.shs_point(p, cb.Shc(N, GM, R_EARTH, c, s), N)
    out = cb.sha_point(p, f, N, GM, R_EARTH)
    assert coef_rel_rms(out.c, out.s, c, s) <= 1e-12


@pytest.mark.parametrize("M", [m for m in LENGTHS if m <= 768])
def test_single_precision(env, M):      # noqa: F811
    cb = env[1]
    N = halves(M)[1] - 1
    c, s = (x.astype(np.float32).astype(np.float64) for x in kaula(N, M))
    p = cb.PointGridGL(N, R_EARTH)
    ref = cb.shs_point(p, cb.Shc(N, GM, R_EARTH, c, s), N)
    f, msg = shs32(env, p, c, s, N)
    assert msg is None, msg
    assert rel_rms(f.cpu().numpy().astype(np.float64).reshape(ref.shape),
                   ref) <= 1e-6
    oc, os_, msg = sha32(env, p, f, N)
    assert msg is None, msg
    assert coef_rel_rms(oc, os_, c, s) <= 1e-4


# direct rows, odd rows, the run-time plan of M = 6144, clusters of CTAs (even
# and odd rows), quarter-length rows; a plan of compile time beside them
@pytest.mark.parametrize("nlon", [384, 301, 5402, 9218, 9999, 21602, 8764, 722])
def test_blocks_of_one_launch(env, nlon):   # noqa: F811
    cb = env[1]
    N = min((nlon - 1) // 2, 60)
    lat = np.linspace(1.3, -1.2, 6)
    lon = 2.0 * np.pi * np.arange(nlon) / nlon
    p = cb.PointGrid(lat, lon, np.full(lat.size, R_EARTH))
    sets = [(n,) + tuple(kaula(n, 50 + n)) + (GM,) for n in (N, N // 2, N)]
    got = batch(env, p, sets, R_EARTH, 0)
    for st, g in zip(sets, got):
        # (alone beside a set of the full degree's tables: its own)
        one, = batch(env, p, [st], R_EARTH, 0)
        assert rel_rms(g[0], one[0]) <= 1e-14 if st[0] == N else \
            rel_rms(g[0], one[0]) <= TOL
    for st, g in zip(sets, got):
        f = oracle_rows(lat, nlon, st[0], st[1], st[2])
        assert rel_rms(g[0], f) <= TOL
