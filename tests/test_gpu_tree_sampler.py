"""The tree-order sampler's cell queue against the oracle's sequential greedy thinning where it
can go wrong: one point, cells and neighbourhoods around a warp and around the unrolled rounds,
a step above the extent (one cell), no two points within the step, duplicates, a long chain of
points each blocked by the one before, and a thin cloud whose cells are coarser than the step."""
import numpy as np
import pytest

from test_gpu_kdtree import _probe

pytestmark = pytest.mark.gpu


def _cloud(kind, n, rng):
    if kind == "uniform":
        return rng.uniform(-10, 10, (n, 3))
    if kind == "plane":
        return np.concatenate([rng.uniform(-10, 10, (n, 2)), rng.normal(0, 0.01, (n, 1))], 1)
    if kind == "same":
        return np.full((n, 3), 1.5)
    if kind == "line":  # spaced just below the step: a chain through all of them
        return np.stack([np.arange(n) * 0.99, np.zeros(n), np.zeros(n)], 1)
    if kind == "thin":  # an extent of many cells along one axis
        return np.concatenate([rng.uniform(0, 40000, (n, 1)), rng.uniform(0, 3, (n, 2))], 1)
    clump = rng.normal(0, 0.3, (n // 2, 3))  # half the points in one cell
    return np.concatenate([clump, rng.uniform(-10, 10, (n - n // 2, 3))])


@pytest.mark.parametrize("kind, n, step", [
    ("uniform", 1, 1.0), ("uniform", 2, 100.0), ("uniform", 31, 4.0), ("uniform", 33, 40.0),
    ("uniform", 129, 2.0), ("uniform", 5000, 1e-4), ("uniform", 20000, 1.0),
    ("uniform", 3000, 60.0), ("plane", 30000, 0.7), ("plane", 30000, 5.0), ("same", 1500, 1.0),
    ("line", 3000, 1.0), ("thin", 20000, 0.9), ("clump", 9000, 1.1), ("clump", 9000, 0.05)])
def test_sample_matches_the_sequential_order(kind, n, step):
    from oracle.pyoracle import kd_reference
    xyz = _cloud(kind, n, np.random.default_rng(n)).astype(np.float32)
    _, s, _, _ = _probe(xyz, np.float32(step))
    _, ref, _, _ = kd_reference(xyz, np.float32(step))
    np.testing.assert_array_equal(s, ref)
