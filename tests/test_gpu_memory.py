"""Grid calls where the device memory holds what the one-degree recurrence
needs and not the tables and coefficient forms of the two-degree one: they run
all the same, with the same results to rounding.  And batches of more sets than
one pass of the kernels takes.

The children hold the device memory down to a limit between the two needs, by
the sizes of the buffers: with T = (n + 1)(n + 2) / 2 and L = (n + 1)^2, tables
24 T, coefficients 16 T, spectra 16 L per quantity, partial sums 16 T per group
(four at these sizes), beside which the two-degree recurrence takes 28 T for
its tables and 16 T for its coefficients (5 x 32 T in their place for the ten
quantities) or for the sums next to the equator."""
import ctypes as ct
import os
import subprocess
import sys

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CHILD = r"""
import ctypes as ct, sys
import numpy as np, torch
import charm_b200 as cb
from charm_b200._lib import _libcharm as L
from charm_b200.workloads import GM, R_EARTH, kaula
op, n, leave, out = sys.argv[1], int(sys.argv[2]), int(sys.argv[3]), sys.argv[4]
P = ct.c_void_p
L.charm_b200_shs_point_dev.argtypes = [
    P, ct.c_ulong, ct.c_double, ct.c_double, P, P, ct.c_ulong, ct.c_int,
    ct.c_uint, ct.c_uint, ct.c_uint, P, P]
L.charm_b200_sha_point_dev.argtypes = [
    P, P, ct.c_ulong, ct.c_double, ct.c_double, ct.c_ulong, P, P, P]
L.charm_b200_shs_point_batch_dev.argtypes = [
    P, ct.c_size_t, ct.POINTER(ct.c_ulong), ct.POINTER(ct.c_ulong),
    ct.POINTER(ct.c_double), ct.c_double, ct.POINTER(P), ct.POINTER(P),
    ct.c_int, ct.POINTER(P), P]

def call(fn, *args):
    err = L.charm_err_init()
    fn(*args, ct.cast(err, P))
    if not L.charm_err_isempty(err):
        sys.exit(ct.string_at(err.contents.msg).decode())
    L.charm_err_free(err)

def run(p, n, cs, f, oc):
    pp = ct.cast(p._Point, P)
    a, b = cs[0].data_ptr(), cs[1].data_ptr()
    if op == "synthesis":
        call(L.charm_b200_shs_point_dev, pp, n, GM, R_EARTH, a, b, n, 0, 0, 0,
             0, f.data_ptr())
        return f
    if op == "analysis":
        call(L.charm_b200_sha_point_dev, pp, f.data_ptr(), n, GM, R_EARTH, n,
             oc[0].data_ptr(), oc[1].data_ptr())
        return oc
    nm = (ct.c_ulong * 1)(n)
    call(L.charm_b200_shs_point_batch_dev, pp, 1, nm, nm,
         (ct.c_double * 1)(GM), R_EARTH, (P * 1)(a), (P * 1)(b), 3,
         (P * 1)(f.data_ptr()))
    return f

def arrays(p, n):
    c, s = kaula(n, 5)
    c[0] = 0.0
    cs = torch.from_numpy(np.stack([c, s])).cuda()
    nq = 10 if op == "ten" else 1
    g = torch.Generator(device="cuda")
    g.manual_seed(1)
    f = torch.randn((nq, p.lat.size, p.lon.size), generator=g, device="cuda",
                    dtype=torch.float64)
    return cs, f, torch.zeros_like(cs)

# the library's kernels of these calls loaded by a smaller one
q = cb.PointGridGL(560 if op != "analysis" else 800, R_EARTH)
run(q, q.lat.size - 1, *arrays(q, q.lat.size - 1))
p = cb.PointGridGL(n, R_EARTH)
args = arrays(p, n)
torch.cuda.synchronize()
hold = []
if leave:
    torch.cuda.empty_cache()
    free = torch.cuda.mem_get_info()[0]
    hold.append(torch.empty(free - (leave << 20), dtype=torch.uint8,
                            device="cuda"))
res = run(p, n, *args)
np.save(out, res.flatten()[::211].cpu().numpy())
"""


# bytes per T of the one-degree call, of the two-degree one beside it, spectra
@pytest.mark.parametrize("op,n,one,more,spectra", [
    ("synthesis", 3000, 24 + 16, 28 + 16, 1),
    ("analysis", 3000, 24 + 4 * 16, 28 + 16, 1),
    ("ten", 1500, 24 + 16, 28 + 5 * 32 - 16, 10)])
def test_without_room_for_the_two_degree_tables(tmp_path, op, n, one, more,
                                                spectra):
    T = (n + 1) * (n + 2) // 2
    # (allocations are rounded up)
    leave = int((one + 0.4 * more) * T + 16 * (n + 1) ** 2 * spectra) >> 20
    got = []
    for k, mib in enumerate((0, leave)):
        out = str(tmp_path / ("%d.npy" % k))
        r = subprocess.run([sys.executable, "-c", CHILD, op, str(n), str(mib),
                            out], cwd=ROOT, capture_output=True, text=True,
                           timeout=300)
        assert r.returncode == 0, r.stderr[-2000:]
        got.append(np.load(out))
    ref, f = got
    # functions of degree n carry n 2^-53 of their size from the rounded
    # latitude (the potential carries the norm of the ten quantities)
    assert np.linalg.norm(f - ref) <= 8.0 * n * 2.0 ** -53 * np.linalg.norm(ref)


def test_more_sets_than_a_pass():
    """Two hundred and forty sets of ten quantities at degree 400 (their
    buffers beyond one pass's 8 GB), three models in turn: equal inputs, equal
    bits."""
    import torch
    import charm_b200 as cb
    from charm_b200._lib import _libcharm as L
    from charm_b200.workloads import GM, R_EARTH, kaula
    n, k = 400, 240
    p = cb.PointGridGL(n, R_EARTH + 1e4)
    models = [torch.from_numpy(np.stack(kaula(n, 30 + j))).cuda()
              for j in range(3)]
    f = torch.full((k, 10, p.lat.size, p.lon.size), np.nan,
                   dtype=torch.float64, device="cuda")
    P = ct.c_void_p
    L.charm_b200_shs_point_batch_dev.argtypes = [
        P, ct.c_size_t, ct.POINTER(ct.c_ulong), ct.POINTER(ct.c_ulong),
        ct.POINTER(ct.c_double), ct.c_double, ct.POINTER(P), ct.POINTER(P),
        ct.c_int, ct.POINTER(P), P]
    nm, mu = (ct.c_ulong * k)(*[n] * k), (ct.c_double * k)(*[GM] * k)
    err = L.charm_err_init()
    L.charm_b200_shs_point_batch_dev(
        ct.cast(p._Point, P), k, nm, nm, mu, R_EARTH,
        (P * k)(*[models[j % 3][0].data_ptr() for j in range(k)]),
        (P * k)(*[models[j % 3][1].data_ptr() for j in range(k)]), 3,
        (P * k)(*[f[j].data_ptr() for j in range(k)]), ct.cast(err, P))
    assert L.charm_err_isempty(err)
    L.charm_err_free(err)
    assert bool(torch.isfinite(f[:3]).all())
    for j in range(3, k):
        assert torch.equal(f[j], f[j % 3]), j
