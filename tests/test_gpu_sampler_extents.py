"""The tree-order sampler over extents that a dense table of cells just above the step does not
cover: stray points, groups as many cells apart as the hashed cells' coordinates wrap at, coordinates
beyond what they count exactly, a step far below the points' spacing. The kept points are the
sequential order's, and take no longer for a stray point."""
import time

import numpy as np
import pytest

from test_gpu_kdtree import _probe

pytestmark = pytest.mark.gpu


def _spheres(n, rng):
    d = rng.normal(size=(n, 3))
    cen = rng.uniform(-150, 150, (10, 3))
    return cen[rng.integers(0, 10, n)] + 60 * d / np.linalg.norm(d, axis=1, keepdims=True)


@pytest.mark.parametrize("n, step, away", [
    (1, 1.4, 1e6), (33, 1.4, 1e4), (5000, 1.4, 1e3), (5000, 1.4, 1e4), (5000, 1.4, 1e9),
    (5000, 1.4, 1e17), (5000, 9.0, 1e12), (3000, 1e-6, 1e5), (3000, 1e-20, 0.0)])
def test_stray_points(n, step, away):
    from oracle.pyoracle import kd_reference
    xyz = np.concatenate([_spheres(n, np.random.default_rng(n)), [[away] * 3, [-away, away, 0.0]]])
    xyz = np.ascontiguousarray(xyz, np.float32)
    _, s, _, _ = _probe(xyz, np.float32(step))
    _, ref, _, _ = kd_reference(xyz, np.float32(step))
    np.testing.assert_array_equal(s, ref)


@pytest.mark.parametrize("groups", [[0.0, 2.0 ** 21], [-2.0 ** 21, 0.0, 2.0 ** 22], [2.0 ** 40, 2.0 ** 52]])
def test_groups_where_cells_wrap(groups):
    from oracle.pyoracle import kd_reference
    rng = np.random.default_rng(5)
    step = np.float32(1.0)
    side = float(step * np.float32(1.0 + 1.0 / 1024.0))  # of a cell
    xyz = np.concatenate([rng.uniform(-8, 8, (1500, 3)) + [g * side, 0, -g * side] for g in groups])
    xyz = np.ascontiguousarray(xyz, np.float32)
    _, s, _, _ = _probe(xyz, step)
    _, ref, _, _ = kd_reference(xyz, step)
    np.testing.assert_array_equal(s, ref)


def test_stray_points_cost_nothing():
    # 10,000 points at 1.4 mm: 0.2 ms; with two points 100 m away, in cells grown with the extent, 842
    xyz = np.concatenate([_spheres(10000, np.random.default_rng(1)), [[1e5] * 3, [-1e5] * 3]])
    xyz = np.ascontiguousarray(xyz, np.float32)

    def best(step):
        t = []
        for _ in range(4):
            t0 = time.perf_counter()
            _probe(xyz, np.float32(step))
            t.append(time.perf_counter() - t0)
        return min(t)

    assert best(1.4) - best(0.0) < 0.1
