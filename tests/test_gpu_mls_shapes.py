"""The MLS kernels where their launch shapes can go wrong, against the oracle: one point, lists
around a warp and a CTA, neighbourhoods around the listed length (128) and far above it, and
more points than one launch pair takes."""
import numpy as np
import pytest

from test_mls import NORMAL_TOL_DEG, POINT_TOL_REL, chord_deg

pytestmark = pytest.mark.gpu


def _wavy(n, rng):
    xy = rng.uniform(-20, 20, (n, 2))
    z = 0.02 * xy[:, 0] ** 2 - 0.01 * xy[:, 0] * xy[:, 1] + 0.05 * rng.normal(size=n)
    return np.concatenate([xy, z[:, None]], 1).astype(np.float32)


@pytest.mark.parametrize("n, m, radius, order", [
    (4000, 1, 3.0, 2), (4000, 31, 3.0, 1), (4000, 33, 3.0, 3), (4000, 65, 3.0, 4),
    (16000, 200, 1.99, 2),   # 100-160 neighbours: lists just below and above 128
    (16000, 100, 8.0, 2), (16000, 40, 12.0, 4)])
def test_mls_launch_shapes(n, m, radius, order):
    from oracle import pyoracle as po
    from surface_match_gb300 import PointCloud, estimateNormalMLS
    rng = np.random.default_rng(n + m)
    P = _wavy(n, rng)
    ids = rng.permutation(n)[:m].astype(np.int64)
    op, on, st = po.mls(P, None, ids, radius=radius, order=order)
    pc = estimateNormalMLS(PointCloud(P.copy()), ids, radius, order)
    assert (st == 2).all()
    assert np.linalg.norm(pc.point[ids] - op[ids], axis=1).max() < POINT_TOL_REL * radius
    # the normals' tolerance is for whole neighbourhoods, as in test_mls: at the sheet's rim a
    # one-sided fit of order 4 extrapolates its slope, and FP32 coordinates alone move it by
    # several 1e-3 degrees
    whole = ids[np.all(np.abs(P[ids, :2]) <= 20.0 - radius, axis=1)]
    if len(whole):
        assert chord_deg(pc.normal[whole], on[whole]).max() < NORMAL_TOL_DEG
    assert chord_deg(pc.normal[ids], on[ids]).max() < 0.1


def test_mls_more_points_than_one_launch():
    from surface_match_gb300 import PointCloud, estimateNormalMLS
    rng = np.random.default_rng(9)
    P = _wavy((1 << 18) + 45, rng)
    tail = np.arange((1 << 18) - 7, len(P))
    every = estimateNormalMLS(PointCloud(P.copy()), None, 0.4, 2)
    some = estimateNormalMLS(PointCloud(P.copy()), tail, 0.4, 2)
    ok = np.isfinite(some.normal[tail]).all(1)
    assert ok.mean() > 0.9
    np.testing.assert_array_equal(np.isfinite(every.normal[tail]).all(1), ok)
    d = np.einsum("ij,ij->i", every.normal[tail][ok], some.normal[tail][ok])
    assert np.abs(np.abs(d) - 1.0).max() < 1e-5
    assert np.abs(every.point[tail] - some.point[tail]).max() < POINT_TOL_REL * 0.4
