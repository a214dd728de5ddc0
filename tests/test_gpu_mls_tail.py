"""Points with a few more neighbours than the smoothing lists (128), by threads or warps: values against
the oracle on both sides of the line between them, and a handful of such points in a whole cloud does
not make the call wait for warps."""
import time

import numpy as np
import pytest

from test_gpu_mls_shapes import _wavy
from test_mls import NORMAL_TOL_DEG, POINT_TOL_REL, chord_deg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n, m, near, order", [
    (16000, 16000, 100, 3), (16000, 2500, 115, 2), (16000, 2500, 145, 2), (16000, 2500, 200, 3),
    (6000, 1500, 130, 4), (6000, 1500, 250, 4), (6000, 300, 118, 1)])
def test_both_sides_of_the_line(n, m, near, order):
    from oracle import pyoracle as po
    from surface_match_gb300 import PointCloud, estimateNormalMLS
    rng = np.random.default_rng(n + m)
    P = _wavy(n, rng)
    radius = float(np.sqrt(near * 1600 / (n * np.pi)))
    ids = rng.permutation(n)[:m].astype(np.int64)
    op, on, st = po.mls(P, None, ids, radius=radius, order=order)
    pc = estimateNormalMLS(PointCloud(P.copy()), ids, radius, order)
    assert (st == 2).all()
    assert np.linalg.norm(pc.point[ids] - op[ids], axis=1).max() < POINT_TOL_REL * radius
    whole = ids[np.all(np.abs(P[ids, :2]) <= 20.0 - radius, axis=1)]
    assert chord_deg(pc.normal[whole], on[whole]).max() < NORMAL_TOL_DEG


def test_a_few_points_just_above_the_list():
    # 16,000 points at order 4, 80 neighbours and 100 (four points with more than 128): 318 and 425 us;
    # 655 with those four by warps
    from surface_match_gb300 import PointCloud, estimateNormalMLS
    from surface_match_gb300.detector import Context
    P = _wavy(16000, np.random.default_rng(1))
    ctx = Context()

    def best(near):
        t = []
        for _ in range(12):
            pc = PointCloud(P)
            t0 = time.perf_counter()
            estimateNormalMLS(pc, None, float(np.sqrt(near * 1600 / (16000 * np.pi))), 4, context=ctx)
            t.append(time.perf_counter() - t0)
        return min(t)

    try:
        assert best(100) < 1.7 * best(80)
    finally:
        ctx.close()
