"""Rows at the poles, where derivatives along the meridian are rounding noise
over cos(lat): every entry point forms the same noise, because one kernel forms
it.  Grids whose other rows take the two-degree recurrence against the same
rows in an order of latitudes that it does not take, and the single derivative
against the gradient's component: equal bits."""
import numpy as np
import pytest

from charm_b200.workloads import GM, R_EARTH, kaula

pytestmark = pytest.mark.gpu

KINDS = ["grad1", "grad2", (0, 1, 0), (0, 2, 0), (1, 1, 0), (0, 1, 1)]


def rows(cb, n, ratio, order, kind):
    lat = np.pi / 2 - np.pi * np.arange(2 * n + 2) / (2 * n + 2)
    half = lat[:n + 1][order]
    lat = np.concatenate([half, -half[::-1]])     # both poles, mirror rows
    lon = np.arange(2 * n + 2) * (np.pi / (n + 1))
    p = cb.PointGrid(lat, lon, np.full(lat.size, R_EARTH * ratio))
    c, s = kaula(n, 21)
    shc = cb.Shc(n, GM, R_EARTH, c, s)
    if kind == "grad1":
        out = cb.shs_point_grad1(p, shc, n)
    elif kind == "grad2":
        out = cb.shs_point_grad2(p, shc, n)
    else:
        out = [cb.shs_point_guru(p, shc, n, *kind)]
    return np.stack([np.asarray(f).reshape(lat.size, -1) for f in out])


@pytest.mark.parametrize("n", [127, 128, 150])
@pytest.mark.parametrize("ratio", [1.0, 1.01])
@pytest.mark.parametrize("kind", KINDS)
def test_pole_rows_do_not_depend_on_the_other_rows(n, ratio, kind):
    import charm_b200 as cb
    order = np.arange(n + 1)
    a = rows(cb, n, ratio, order, kind)
    other = order.copy()
    other[[40, 50]] = other[[50, 40]]
    b = rows(cb, n, ratio, other, kind)
    assert np.array_equal(a[:, [0, -1]], b[:, [0, -1]])


@pytest.mark.parametrize("n", [127, 150])
@pytest.mark.parametrize("ratio", [1.0, 1.01])
def test_latitudinal_derivative_is_the_gradients(n, ratio):
    import charm_b200 as cb
    order = np.arange(n + 1)
    x = rows(cb, n, ratio, order, "grad1")[0]
    d = rows(cb, n, ratio, order, (0, 1, 0))[0]
    assert np.array_equal(x[[0, -1]], d[[0, -1]])
