"""Reference-order refinement searches started from a bound (sm_kdtree.cuh nn_bound) against the
oracle's reference-order pipeline, whose searches start from the largest float: refinement
traces, statuses and scores bit-exact where the bound could go wrong - no and wide rejection
distances, points that normal estimation moved far out of their leaves (sparse clutter), given
normals (nothing moves), and no dense stage."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("reject, scoring, clutter, normals, dense", [
    (0.1, 0.01, "uniform", False, True),
    (0.1, 0.01, "uniform", False, False),
    (0.0, 0.01, "shapes", False, True),
    (1e-4, 0.05, "shapes", False, True),
    (0.6, 0.0, "uniform", False, True),
    (0.1, 0.02, "shapes", True, True),
])
def test_bounded_searches_match_unbounded(reject, scoring, clutter, normals, dense):
    from oracle import MODE_REF, MatchParam as OMP, Oracle
    from surface_match_gb300 import Detector, MatchParam, PointCloud, synth
    mc, s, c = synth.gear_model(6000, seed=5)
    sc = synth.make_scene(11, {"gear": s}, 2, ((-70, -70, 40), (70, 70, 100)),
                          points_per_instance=5000, clutter_frac=0.15, clutter=clutter, noise=0.2,
                          model_centers={"gear": c})
    xyz = sc.cloud.xyz
    nrm = None
    if normals:  # any finite normals will do for the searches: towards the viewpoint
        nrm = sc.viewpoint - xyz
        nrm = (nrm / np.linalg.norm(nrm, axis=1, keepdims=True)).astype(np.float32)
    kw = dict(numMatches=4, poseRefDistThresholdRel=reject, poseRefScoringDistRel=scoring,
              densePoseRefinement=dense)
    o = Oracle(mode=MODE_REF, threads=8)
    om = o.train(mc.xyz, mc.normal, 0.05)
    r = o.match(om, xyz, nrm, sc.viewpoint, 0.05, 0.2, 0.1, OMP(**kw))
    det = Detector(search_order="reference")
    det.trainModel(PointCloud(mc.xyz, mc.normal), 0.05)
    poses, scores = det.matchScene(PointCloud(xyz, nrm, sc.viewpoint), 0.05, 0.2, 0.1,
                                   MatchParam(**kw))
    n = len(r.cand_status)
    if not normals:
        assert n > 0
    np.testing.assert_array_equal(det.debug(15)[:n], r.cand_trace, err_msg="ICP traces")
    np.testing.assert_array_equal(det.debug(12)[:n], r.cand_status)
    np.testing.assert_array_equal(scores, r.scores)
    np.testing.assert_array_equal(poses[:, :3, :].reshape(-1, 12), r.results[:, :12])


@pytest.mark.parametrize("grid, knn", [(0.0, 10), (0.0, 32), (0.5, 10), (1.5, 31), (1.5, 32),
                                       (4.0, 10)])
def test_searches_with_ties_match_the_tree(grid, knn):
    """Scenes on a lattice of `grid` mm (equally distant neighbours and duplicate points; many
    more than 32 at one distance on the coarsest) and neighbourhoods up to the largest k: which
    of equally distant points a search keeps, and in which order, decides the moved points, the
    normals and everything after them."""
    from oracle import MODE_REF, MatchParam as OMP, Oracle
    from surface_match_gb300 import Detector, MatchParam, PointCloud, synth
    mc, s, c = synth.gear_model(6000, seed=5)
    sc = synth.make_scene(12, {"gear": s}, 2, ((-70, -70, 40), (70, 70, 100)),
                          points_per_instance=5000, clutter_frac=0.1, clutter="shapes", noise=0.2,
                          model_centers={"gear": c})
    xyz = sc.cloud.xyz
    if grid:
        xyz = (np.round(xyz / grid) * grid).astype(np.float32)
    kw = dict(numMatches=4, knnNormal=knn)
    o = Oracle(mode=MODE_REF, threads=8)
    om = o.train(mc.xyz, mc.normal, 0.05)
    r = o.match(om, xyz, None, sc.viewpoint, 0.05, 0.2, 0.1, OMP(**kw))
    det = Detector(search_order="reference")
    det.trainModel(PointCloud(mc.xyz, mc.normal), 0.05)
    poses, scores = det.matchScene(PointCloud(xyz, None, sc.viewpoint), 0.05, 0.2, 0.1,
                                   MatchParam(**kw))
    np.testing.assert_array_equal(det.debug(0), r.sampled)
    np.testing.assert_array_equal(det.debug(2), r.resampled)
    np.testing.assert_array_equal(det.debug(3).view(np.uint32), r.positions.view(np.uint32))
    ok = np.isfinite(r.normals).all(1)
    nrm = det.debug(4)
    np.testing.assert_array_equal(np.isfinite(nrm).all(1), ok)
    np.testing.assert_array_equal(nrm[ok].view(np.uint32), r.normals[ok].view(np.uint32))
    n = len(r.cand_status)
    np.testing.assert_array_equal(det.debug(15)[:n], r.cand_trace, err_msg="ICP traces")
    np.testing.assert_array_equal(scores, r.scores)
    np.testing.assert_array_equal(poses[:, :3, :].reshape(-1, 12), r.results[:, :12])
