"""The grid-order sampler's cell classes and table kinds where they can go wrong, sampled,
keypoint and resampled sets against the oracle: cells around 8, 32 and 128 points, hundreds in
one cell, many kept points around a small cell (more than its staged 32), a dense and a hashed
table, a scene below a warp, all points in one cell."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _scene(kind, n, rng):
    if kind == "uniform":
        return rng.uniform(-60, 60, (n, 3))
    if kind == "sheet":  # cells hold n * step^2 / area points
        return np.concatenate([rng.uniform(-60, 60, (n, 2)), rng.normal(0, 0.05, (n, 1))], 1)
    if kind == "far":  # two far points stretch the box: the table is hashed
        p = rng.uniform(-60, 60, (n, 3))
        p[:2] = [[30000, 0, 0], [0, -30000, 20000]]
        return p
    if kind == "clumps":  # a few cells with hundreds of points among light ones
        c = rng.uniform(-50, 50, (6, 3))
        return np.concatenate([c[rng.integers(0, 6, n // 2)] + rng.normal(0, 0.4, (n // 2, 3)),
                               rng.uniform(-60, 60, (n - n // 2, 3))])
    return np.full((n, 3), 7.0) + rng.normal(0, 1e-4, (n, 3))


@pytest.mark.parametrize("kind, n, sd", [
    ("uniform", 5, 0.05), ("uniform", 30000, 0.03), ("uniform", 60000, 0.15),
    ("sheet", 30000, 0.02), ("sheet", 30000, 0.05), ("sheet", 60000, 0.12), ("sheet", 60000, 0.5),
    ("far", 20000, 0.04), ("clumps", 20000, 0.04), ("same", 3000, 0.05)])
def test_sampled_sets(kind, n, sd):
    from oracle import MODE_GRID, MatchParam as OMP, Oracle
    from surface_match_gb300 import Detector, MatchParam, PointCloud, synth
    mc, _, _ = synth.gear_model(3000, seed=5)
    xyz = _scene(kind, n, np.random.default_rng(n)).astype(np.float32)
    nrm = np.tile(np.array([[0, 0, 1]], np.float32), (n, 1))
    o = Oracle(mode=MODE_GRID, threads=8)
    om = o.train(mc.xyz, mc.normal, 0.08)
    r = o.match(om, xyz, nrm, None, sd, 0.15, 0.9, OMP())
    det = Detector()
    det.trainModel(PointCloud(mc.xyz, mc.normal), 0.08)
    det.matchScene(PointCloud(xyz, nrm, None), sd, 0.15, 0.9, MatchParam())
    for field, ref in ((0, r.sampled), (1, r.keypoints), (2, r.resampled)):
        np.testing.assert_array_equal(det.debug(field), ref)
