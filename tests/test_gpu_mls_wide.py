"""Points with more neighbours than the smoothing lists (128): by a warp each where they are few, all
points of a small call by warps, by a thread each where they are many. Values against the oracle at
the edges of that rule, and no longer for a few such points than a warp takes for one."""
import time

import numpy as np
import pytest

from test_gpu_mls_shapes import _wavy
from test_mls import NORMAL_TOL_DEG, POINT_TOL_REL, chord_deg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m, radius, order", [
    (2048, 4.4, 1),    # all by warps, among them points with fewer neighbours (1000 on average)
    (2048, 2.2, 3),    # the same around the listed number
    (2049, 4.4, 2),    # the wide ones by warps, the rest by threads
    (9000, 2.4, 4),    # more wide ones than warps take at this order: threads
    (16000, 2.4, 2)])  # the same at order 2
def test_wide_points(m, radius, order):
    from oracle import pyoracle as po
    from surface_match_gb300 import PointCloud, estimateNormalMLS
    rng = np.random.default_rng(m)
    # (three points by themselves: too few neighbours for a plane)
    P = np.concatenate([[[60, 60, 0], [61, 60, 0], [-70, 0, 5]], _wavy(16000, rng)]).astype(np.float32)
    ids = np.concatenate([[0, 1, 2], 3 + rng.permutation(16000)[:m - 3]]).astype(np.int64)
    op, on, st = po.mls(P, None, ids, radius=radius, order=order)
    pc = estimateNormalMLS(PointCloud(P.copy()), ids, radius, order)
    ok = ids[3:]
    assert (st[3:] == 2).all()
    assert np.linalg.norm(pc.point[ok] - op[ok], axis=1).max() < POINT_TOL_REL * radius
    whole = ok[np.all(np.abs(P[ok, :2]) <= 20.0 - radius, axis=1)]
    assert chord_deg(pc.normal[whole], on[whole]).max() < NORMAL_TOL_DEG
    np.testing.assert_array_equal(pc.point[:3], P[:3])
    np.testing.assert_array_equal(np.isfinite(pc.normal[:3]), np.isfinite(on[:3]))


def test_a_few_wide_points_take_no_thread_chain():
    # 40 points of 1000 neighbours at order 2: 0.6 ms a call (0.6 with a warp for every point), 2.4 by
    # a thread each
    from surface_match_gb300 import PointCloud, estimateNormalMLS
    from surface_match_gb300.detector import Context
    rng = np.random.default_rng(1)
    P = _wavy(16000, rng)
    ids = rng.permutation(16000)[:40].astype(np.int64)
    ctx = Context()
    try:
        best = 1.0
        for _ in range(10):
            pc = PointCloud(P.copy())
            t = time.perf_counter()
            estimateNormalMLS(pc, ids, 5.64, 2, context=ctx)
            best = min(best, time.perf_counter() - t)
    finally:
        ctx.close()
    assert best < 1.4e-3
