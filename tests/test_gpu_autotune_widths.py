"""What the first call of a grid's shape times: one launch per width of the
two-degree synthesis that can be the fastest at its number of latitude pairs,
none where that is one; the result is that of the later calls."""
import numpy as np
import pytest

from charm_b200.workloads import GM, R_EARTH, kaula
from test_gpu_autotune import report

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("np_,widths", [
    (33, []), (64, []), (65, [1, 2]), (699, [1, 2]), (700, [3, 4, 5])])
def test_widths(np_, widths):
    import charm_b200 as cb
    from charm_b200._lib import _libcharm as L
    n = 403
    lat = np.linspace(1.4, 0.1, np_)
    p = cb.PointGrid(lat, np.arange(2 * n + 2) * (np.pi / (n + 1)),
                     np.full(np_, R_EARTH))
    shc = cb.Shc(n, GM, R_EARTH, *kaula(n, 8))
    f1 = np.array(cb.shs_point(p, shc, n))
    line, = [x for x in report(L) if "kgrad=0" in x and
             "nmax=%d pairs=%d " % (n, np_) in x]
    timed = [int(w.split(":")[0]) for w in line.split("ms:")[1].split()]
    assert timed == widths
    assert np.array_equal(f1, np.array(cb.shs_point(p, shc, n)))
