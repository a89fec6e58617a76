"""Forward modelling as one sequence of transforms whose status is read at its
end: a Gauss--Legendre grid that fails in the middle (the limit of the Newton
iterations lowered to one) is reported and not kept for later calls; and a
sequence of more stagings than there are slots."""
import numpy as np
import pytest

from charm_b200.workloads import coef_rel_rms
from oracle import orc
from test_gpu_gfm import GRAV_CONST, MOON_MASS, random_body

pytestmark = pytest.mark.gpu


def test_failed_grid_is_reported_and_not_kept(monkeypatch):
    import charm_b200 as cb
    R, N, top = 1728000.0, 37, 60     # grids of degree 37 and 74
    c, s = random_body(N, 3, R, 3000.0)
    shape = cb.Shc(N, 1.0, 1.0, c, s)
    args = (shape, N, R, 2600.0, GRAV_CONST, MOON_MASS, 1, 2, top)
    monkeypatch.setenv("CHARM_B200_GL_MAXIT", "1")
    with pytest.raises(cb.CHarmError, match="Gauss--Legendre grid"):
        cb.gfm_global_density_const(*args)
    monkeypatch.delenv("CHARM_B200_GL_MAXIT")
    for n in (N, 2 * N):
        grid = cb.PointGridGL(n, R)
        # (a rounding of the node is one of the latitude times 1 / cos(lat))
        assert np.max(np.abs(grid.lat - orc.gl(n, R).lat)) <= 1e-13
    pot = cb.gfm_global_density_const(*args)
    # (the tolerance of the other forward-modelling tests)
    ref = orc.gfm_global(orc.Shc(N, 1.0, 1.0, c, s), N, R, None, None,
                         GRAV_CONST, MOON_MASS, 1, 2, top,
                         const_density=2600.0)
    assert coef_rel_rms(pot.c, pot.s, ref.c, ref.s) <= 1e-12


def test_more_transforms_than_staging_slots():
    """Eighteen powers with three densities: 72 stagings (a synthesis of the
    sets and three analyses a power) in one sequence of 64 slots."""
    import charm_b200 as cb
    R, N, top, powers = 1728000.0, 6, 20, 18
    c, s = random_body(N, 5, R, 2000.0)
    dens = []
    for k in range(3):
        dc, ds = random_body(4, 40 + k, 0.0, 30.0)
        dc[0] = (2600.0, -2e-4, 1e-10)[k]
        dens.append((4, dc, ds))
    pot = cb.gfm_global_density_3d(
        cb.Shc(N, 1.0, 1.0, c, s), N, R,
        [cb.Shc(n, 1.0, 1.0, a, b) for n, a, b in dens], [4, 4, 4], 2,
        GRAV_CONST, MOON_MASS, 1, powers, top)
    ref = orc.gfm_global(
        orc.Shc(N, 1.0, 1.0, c, s), N, R,
        [orc.Shc(n, 1.0, 1.0, a, b) for n, a, b in dens], [4, 4, 4],
        GRAV_CONST, MOON_MASS, 1, powers, top)
    assert coef_rel_rms(pot.c, pot.s, ref.c, ref.s) <= 1e-12
