"""The voting stage's row packing and splits where they can go wrong, per-keypoint counts, hits,
votes and candidates against the oracle: one keypoint and odd numbers of them, candidate lists
below a word, around a round (1024) and over many parts, in both search orders (candidate masks
and neighbour lists)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("order", ["grid", "reference"])
@pytest.mark.parametrize("n, sd, kp", [(20, 0.05, 1.0), (900, 0.05, 0.02), (1500, 0.02, 0.3),
                                       (9000, 0.03, 0.003), (12000, 0.015, 0.05),
                                       (12000, 0.04, 1.0)])
def test_vote_rows(order, n, sd, kp, monkeypatch):
    from oracle import MODE_GRID, MODE_REF, MatchParam as OMP, Oracle
    from surface_match_gb300 import Detector, MatchParam, PointCloud, synth
    monkeypatch.setenv("SM_VOTE_FINGERPRINT", "1")
    mc, s, c = synth.gear_model(4000, seed=5)
    sc = synth.make_scene(31, {"gear": s}, 2, ((-70, -70, 40), (70, 70, 100)),
                          points_per_instance=12000, clutter_frac=0.1, noise=0.1,
                          model_centers={"gear": c})
    xyz = sc.cloud.xyz[:n].copy()
    assert len(xyz) == n
    o = Oracle(mode=MODE_GRID if order == "grid" else MODE_REF, threads=8)
    om = o.train(mc.xyz, mc.normal, 0.06)
    r = o.match(om, xyz, None, sc.viewpoint, sd, kp, 0.05, OMP(numMatches=2))
    det = Detector(search_order=order)
    det.trainModel(PointCloud(mc.xyz, mc.normal), 0.06)
    poses, scores = det.matchScene(PointCloud(xyz, None, sc.viewpoint), sd, kp, 0.05,
                                   MatchParam(numMatches=2))
    np.testing.assert_array_equal(det.debug(1), r.keypoints)
    np.testing.assert_array_equal(det.debug(7), r.kp_stats)
    np.testing.assert_array_equal(det.debug(8), r.kp_cands)
    np.testing.assert_array_equal(scores, r.scores)
