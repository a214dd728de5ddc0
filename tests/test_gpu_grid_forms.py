"""The search grid's forms - a direct cell table, a hashed one with occupancy bits, a hashed one
without - and their edges: cell boxes just below and above the direct table's limit, boxes beyond
the bits', point counts at one and around a pass's run of entries. A match's positions, normals and
refinement use the grid, and give the oracle's bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("extent", [0.0, 600.0, 1200.0, 4000.0, 60000.0])
@pytest.mark.parametrize("points", [1500, 5461])
def test_grid_forms(extent, points):
    from oracle import MODE_GRID, MatchParam as OMP, Oracle
    from surface_match_gb300 import Detector, MatchParam, PointCloud, synth
    mc, s, c = synth.gear_model(2600, seed=5)
    sc = synth.make_scene(13, {"gear": s}, 2, ((-100, -100, 40), (100, 100, 140)),
                          points_per_instance=points, clutter_frac=0.1, clutter="shapes", noise=0.2,
                          model_centers={"gear": c})
    xyz = sc.cloud.xyz
    if extent > 0.0:  # two far points stretch the cell box
        far = np.array([[-1, -1, -1], [1, 1, 1]], np.float32) * np.float32(extent / 2)
        xyz = np.concatenate([xyz, far + xyz.mean(0)]).astype(np.float32)
    kw = dict(numMatches=4, poseRefDistThresholdRel=0.2)
    o = Oracle(mode=MODE_GRID, threads=8)
    om = o.train(mc.xyz, mc.normal, 0.06)
    r = o.match(om, xyz, None, sc.viewpoint, 0.06, 0.2, 0.02, OMP(**kw))
    det = Detector()
    det.trainModel(PointCloud(mc.xyz, mc.normal), 0.06)
    poses, scores = det.matchScene(PointCloud(xyz, None, sc.viewpoint), 0.06, 0.2, 0.02,
                                   MatchParam(**kw))
    n = len(r.cand_status)
    assert n > 0
    np.testing.assert_array_equal(det.debug(12)[:n], r.cand_status)
    np.testing.assert_array_equal(det.debug(15)[:n], r.cand_trace, err_msg="ICP traces")
    np.testing.assert_array_equal(scores, r.scores)
    np.testing.assert_array_equal(poses[:, :3, :].reshape(-1, 12), r.results[:, :12])


@pytest.mark.parametrize("far", [0.0, 3e5])
@pytest.mark.parametrize("n", [1, 2, 2047, 2049])
def test_smoothing_over_few_points(n, far):
    """The smallest grids, direct and (with a far point) hashed: no point is lost or met twice."""
    from oracle import pyoracle as po
    from surface_match_gb300 import PointCloud, estimateNormalMLS
    from test_mls import POINT_TOL_REL
    rng = np.random.default_rng(n)
    xy = rng.uniform(-20, 20, (n, 2))
    z = 0.02 * xy[:, 0] ** 2 - 0.01 * xy[:, 0] * xy[:, 1]
    P = np.concatenate([xy, z[:, None]], 1).astype(np.float32)
    if far:
        P[-1] += np.float32(far)
    ids = np.arange(n, dtype=np.int64)
    op, on, st = po.mls(P, None, ids, radius=4.0, order=2)
    pc = estimateNormalMLS(PointCloud(P.copy()), ids, 4.0, 2)
    ok = st == 2
    assert ok.sum() >= (n - 1 if n > 2 else 0)
    assert n <= 2 or np.linalg.norm(pc.point[ok] - op[ok], axis=1).max() < POINT_TOL_REL * 4.0
    np.testing.assert_array_equal(np.isfinite(pc.normal).all(1), np.isfinite(on).all(1))
