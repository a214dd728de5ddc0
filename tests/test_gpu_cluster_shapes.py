"""Pose clustering where its chunks can go wrong - no pose, a few, lists below and above a chunk of
1024, several chunks, more clusters than a chunk - bit-exact against the oracle's sequential walk."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("points, instances, min_score, sd, poses, clusters", [
    (3000, 3, 0.9, 0.05, (0, 0), (0, 0)),
    (1500, 2, 0.1, 0.06, (2, 31), (1, 31)),
    (3000, 3, 0.02, 0.06, (500, 1024), (200, 1024)),
    (4000, 4, 0.02, 0.05, (1025, 2047), (200, 1024)),
    (12000, 8, 0.01, 0.04, (3073, 8192), (500, 1024)),
    (16000, 10, 0.003, 0.03, (4097, 16384), (1025, 8192))])
def test_cluster_shapes(points, instances, min_score, sd, poses, clusters):
    from oracle import MODE_GRID, MatchParam as OMP, Oracle
    from surface_match_gb300 import Detector, MatchParam, PointCloud, synth
    mc, s, c = synth.gear_model(2600, seed=5)
    sc = synth.make_scene(13, {"gear": s}, instances, ((-180, -180, 40), (180, 180, 140)),
                          points_per_instance=points, clutter_frac=0.4, clutter="shapes", noise=0.2,
                          model_centers={"gear": c})
    kw = dict(numMatches=4, densePoseRefinement=False)
    o = Oracle(mode=MODE_GRID, threads=8)
    om = o.train(mc.xyz, mc.normal, sd)
    r = o.match(om, sc.cloud.xyz, None, sc.viewpoint, sd, 1.0, min_score, OMP(**kw))
    assert poses[0] <= len(r.pose_list) <= poses[1]
    assert clusters[0] <= len(r.cluster_sizes) <= clusters[1]
    det = Detector()
    det.trainModel(PointCloud(mc.xyz, mc.normal), sd)
    det.matchScene(PointCloud(sc.cloud.xyz, None, sc.viewpoint), sd, 1.0, min_score, MatchParam(**kw))
    np.testing.assert_array_equal(det.debug(9).view(np.uint32), r.pose_list.view(np.uint32))
    np.testing.assert_array_equal(det.debug(10).view(np.uint32), r.clustered.view(np.uint32))
