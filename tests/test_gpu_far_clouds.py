"""Whole clouds far from zero (coordinates of a site's own system, say), so that one axis is rounded to
many cells: samples, moved positions, normals, refinement and poses are the oracle's, bit for bit, in
both search orders, and the searches look at a few rings of cells only."""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("order", ["grid", "reference"])
@pytest.mark.parametrize("off", [3e6, 1e8, 2e8])
def test_cloud_far_from_zero(order, off):
    from oracle import MODE_GRID, MODE_REF, MatchParam as OMP, Oracle
    from surface_match_gb300 import Detector, MatchParam, PointCloud, synth
    mc, s, c = synth.gear_model(6000, seed=5)
    sc = synth.make_scene(14, {"gear": s}, 3, ((-120, -120, 40), (120, 120, 140)),
                          points_per_instance=30000, clutter_frac=0.1, clutter="shapes", noise=0.2,
                          model_centers={"gear": c})
    xyz = (sc.cloud.xyz.astype(np.float64) + [off, 0, 0]).astype(np.float32)
    kw = dict(numMatches=8, poseRefDistThresholdRel=0.2)
    o = Oracle(mode=MODE_GRID if order == "grid" else MODE_REF, threads=8)
    r = o.match(o.train(mc.xyz, mc.normal, 0.05), xyz, None, None, 0.05, 0.2, 0.0, OMP(**kw))
    det = Detector(search_order=order)
    det.trainModel(PointCloud(mc.xyz, mc.normal), 0.05)
    best = 1e9
    for _ in range(3):
        t = time.perf_counter()
        poses, scores = det.matchScene(PointCloud(xyz, None, None), 0.05, 0.2, 0.0, MatchParam(**kw))
        best = min(best, time.perf_counter() - t)
    np.testing.assert_array_equal(det.debug(0), r.sampled)
    np.testing.assert_array_equal(det.debug(2), r.resampled)
    np.testing.assert_array_equal(det.debug(3).view(np.uint32), r.positions.view(np.uint32))
    ok = np.isfinite(r.normals).all(1)
    nrm = det.debug(4)
    np.testing.assert_array_equal(np.isfinite(nrm).all(1), ok)
    np.testing.assert_array_equal(nrm[ok].view(np.uint32), r.normals[ok].view(np.uint32))
    assert (r.cand_status == 0).any()  # candidates are refined and scored
    np.testing.assert_array_equal(scores, r.scores)
    np.testing.assert_array_equal(poses[:, :3, :].reshape(-1, 12), r.results[:, :12])
    assert best < 0.1  # some milliseconds; rings out to a margin of 60 cells would take seconds
