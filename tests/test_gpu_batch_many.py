"""Batched synthesis of more sets than one launch of the row transforms holds
(their blocks are the y dimension of a launch, 65535 at most): every set
against the sum of its coefficients times the fields of single coefficients.

Tolerance: both sides are sums of at most twelve products, in another order,
followed by rows of six points; each operation rounds to 2^-53 of the largest
partial result, so the relative RMS stays below 1e-14."""
import ctypes as ct

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

NMAX = 2
T = (NMAX + 1) * (NMAX + 2) // 2


def run(torch, L, p, c, s, kgrad):
    """[set][quantity][grid] of the coefficients c, s ([set][T])."""
    n, nq = c.shape[0], {0: 1, 2: 6}[kgrad]
    f = torch.full((n, nq, p.lat.size * p.lon.size), np.nan,
                   dtype=torch.float64, device="cuda")
    P = ct.c_void_p

    def pointers(t):
        step = t.stride(0) * 8
        return (P * n)(*[t.data_ptr() + j * step for j in range(n)])

    L.charm_b200_shs_point_batch_dev.argtypes = [
        P, ct.c_size_t, ct.POINTER(ct.c_ulong), ct.POINTER(ct.c_ulong),
        ct.POINTER(ct.c_double), ct.c_double, ct.POINTER(P), ct.POINTER(P),
        ct.c_int, ct.POINTER(P), P]
    nm, mu = (ct.c_ulong * n)(*[NMAX] * n), (ct.c_double * n)(*[1.0] * n)
    err = L.charm_err_init()
    L.charm_b200_shs_point_batch_dev(
        ct.cast(p._Point, P), n, nm, nm, mu, 1.0, pointers(c), pointers(s),
        kgrad, pointers(f), ct.cast(err, P))
    ok = L.charm_err_isempty(err)
    msg = None if ok else ct.string_at(err.contents.msg).decode()
    L.charm_err_free(err)
    assert ok, msg
    return f


@pytest.mark.parametrize("nsets,kgrad", [(65535, 0), (65536, 0), (131080, 0),
                                         (10923, 2)])
def test_more_blocks_than_a_launch(nsets, kgrad):
    import torch
    import charm_b200 as cb
    from charm_b200._lib import _libcharm as L
    p = cb.PointGridGL(NMAX, 1.0)
    one = torch.eye(2 * T, dtype=torch.float64, device="cuda")
    one[T:T + NMAX + 1] = 0.0           # S_n0 does not exist
    basis = run(torch, L, p, one[:, :T].contiguous(),
                one[:, T:].contiguous(), kgrad)
    g = torch.Generator(device="cuda")
    g.manual_seed(nsets)
    x = torch.randn((nsets, 2 * T), generator=g, device="cuda",
                    dtype=torch.float64)
    f = run(torch, L, p, x[:, :T].contiguous(), x[:, T:].contiguous(), kgrad)
    ref = torch.einsum("jk,kqi->jqi", x, basis)
    err = ((f - ref).norm(dim=(0, 2)) / ref.norm(dim=(0, 2))).max().item()
    assert err <= 1e-14
    # and no set apart from the others
    worst = ((f - ref).norm(dim=2) / ref.norm(dim=2).mean(0)).max().item()
    assert worst <= 1e-13
