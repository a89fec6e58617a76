"""What a kernel now finds prepared: the constants of scattered points in the
adjoint, on, above and below the reference sphere, against explicit columns
of the oracle's synthesis; and the digit tiles of the split batch where an
order has as many 64-degree chunks as blocks that share them, and more,
against the FP64 batch.

The tolerance is that of the tests of the same entry points: 1e-13 between
double-precision evaluations in a different order."""
import numpy as np
import pytest

from charm_b200.workloads import GM, R_EARTH
from oracle import orc
from test_gpu_batch_i8 import compare, env, make_sets

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("npt", [1, 33, 257])
@pytest.mark.parametrize("height", [0.0, 9000.0, -9000.0])
def test_adjoint_point_constants(npt, height):
    import torch
    import charm_b200 as cb
    from charm_b200 import autograd as ag
    N = 12
    rng = np.random.default_rng(9700 + npt)
    lat = np.arcsin(rng.uniform(-1.0, 1.0, npt))
    lon = rng.uniform(0.0, 2.0 * np.pi, npt)
    r = R_EARTH + height * rng.uniform(0.1, 1.0, npt)
    T = (N + 1) * (N + 2) // 2
    op = orc.Point(orc.SCATTERED, lat, lon, r)
    y = rng.standard_normal(npt)
    ref = np.zeros(2 * T)
    for k in range(2 * T):
        c, s = np.zeros(T), np.zeros(T)
        (c if k < T else s)[k % T] = 1.0
        ref[k] = y @ np.ravel(
            orc.shs_point(op, orc.Shc(N, GM, R_EARTH, c, s), N)[0])
    gc, gs = ag._adjoint(torch.from_numpy(y).cuda(),
                         cb.PointSctr(lat, lon, r), N, GM, R_EARTH)
    got = np.concatenate([gc.cpu().numpy(), gs.cpu().numpy()])
    assert np.linalg.norm(got - ref) <= 1e-13 * np.linalg.norm(ref)


@pytest.mark.parametrize("N", [63, 511, 512, 640])
def test_split_batch_chunks(env, N):
    torch, cb, L = env
    compare(env, cb.PointGridGL(N, R_EARTH), make_sets(960, [N, N // 2, 3]),
            R_EARTH)
