"""Lone points far from everything else in the reference's search order, whose searches are answered
on a grid of cells as fine as the scene: stray returns tens to thousands of cells away, alone and as
a group closer together than the neighbourhoods are large, with equally distant and duplicate points
among their neighbours, and clouds of fewer points than a neighbourhood. Sampled points, moved
positions, normals, refinement and poses are the oracle's (the k-d tree throughout), bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _match(xyz, viewpoint, mc, knn):
    from oracle import MODE_REF, MatchParam as OMP, Oracle
    from surface_match_gb300 import Detector, MatchParam, PointCloud
    kw = dict(numMatches=4, knnNormal=knn)
    o = Oracle(mode=MODE_REF, threads=8)
    r = o.match(o.train(mc.xyz, mc.normal, 0.05), xyz, None, viewpoint, 0.05, 0.2, 0.1, OMP(**kw))
    det = Detector(search_order="reference")
    det.trainModel(PointCloud(mc.xyz, mc.normal), 0.05)
    poses, scores = det.matchScene(PointCloud(xyz, None, viewpoint), 0.05, 0.2, 0.1,
                                   MatchParam(**kw))
    np.testing.assert_array_equal(det.debug(0), r.sampled)
    np.testing.assert_array_equal(det.debug(3).view(np.uint32), r.positions.view(np.uint32))
    ok = np.isfinite(r.normals).all(1)
    nrm = det.debug(4)
    np.testing.assert_array_equal(np.isfinite(nrm).all(1), ok)
    np.testing.assert_array_equal(nrm[ok].view(np.uint32), r.normals[ok].view(np.uint32))
    np.testing.assert_array_equal(scores, r.scores)
    np.testing.assert_array_equal(poses[:, :3, :].reshape(-1, 12), r.results[:, :12])
    return det, r, ok


@pytest.mark.parametrize("away, knn, lattice, group", [
    (60.0, 10, 0.0, 1), (60.0, 32, 0.5, 1), (400.0, 10, 0.5, 2), (400.0, 32, 0.0, 12),
    (4000.0, 10, 0.0, 1), (4000.0, 10, 0.5, 12), (4000.0, 32, 0.5, 3), (1e6, 10, 0.5, 2)])
def test_stray_points(away, knn, lattice, group):
    from surface_match_gb300 import synth
    mc, s, c = synth.gear_model(6000, seed=5)
    sc = synth.make_scene(12, {"gear": s}, 2, ((-70, -70, 40), (70, 70, 100)),
                          points_per_instance=5000, clutter_frac=0.1, clutter="shapes", noise=0.2,
                          model_centers={"gear": c})
    xyz = sc.cloud.xyz
    if lattice:
        xyz = (np.round(xyz / lattice) * lattice).astype(np.float32)
    # strays in three directions, each a group of points within 3 mm (sampled as one or two)
    rng = np.random.default_rng(7)
    dirs = np.array([[1.0, 0.9, 0.2], [-1.0, 0.1, 0.3], [0.0, 0.0, 1.0]])
    far = np.concatenate([d * away + np.array([0, 0, 70.0]) + rng.uniform(0, 3, (group, 3)) * (group > 1)
                          for d in dirs * (1.0 + 150.0 / away)]).astype(np.float32)
    xyz = np.concatenate([xyz, far, far[:2]]).astype(np.float32)
    det, r, ok = _match(xyz, sc.viewpoint, mc, knn)
    n = len(r.cand_status)
    np.testing.assert_array_equal(det.debug(2), r.resampled)
    np.testing.assert_array_equal(det.debug(15)[:n], r.cand_trace, err_msg="ICP traces")
    first = len(sc.cloud.xyz)
    assert n > 0 and (r.sampled >= first).sum() >= 3  # the strays are sampled,
    assert ok[r.sampled[r.sampled >= first]].all()    # and have normals


@pytest.mark.parametrize("n, knn, away", [(3, 10, 5.0), (9, 10, 5.0), (9, 32, 3000.0), (31, 32, 900.0),
                                          (7, 10, 1e5)])
def test_fewer_points_than_a_neighbourhood(n, knn, away):
    from surface_match_gb300 import synth
    mc, _, _ = synth.gear_model(6000, seed=5)
    rng = np.random.default_rng(n)
    xyz = (np.round(rng.uniform(0, 4, (n, 3))) * (away / 4)).astype(np.float32)
    xyz[n // 2] = xyz[0]  # a duplicate, and lattice distances: ties
    _match(xyz, np.array([620.0, 100.0, 500.0], np.float32), mc, knn)
