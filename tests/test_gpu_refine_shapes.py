"""The refinement's launches where their shapes can go wrong, traces and results bit-exact against
the oracle: no iteration, one, more than the trace holds; models whose sampled and resampled
clouds fall below a slot group (32), a CTA (512) and the slots (2048) and above them; one candidate
and many; candidates that stop at different iterations."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("model_points, train_sd, resample, steps, matches", [
    (300, 0.2, 0.1, 5, 1),       # 11 sampled and 53 resampled model points
    (700, 0.12, 0.05, 1, 4),     # 37 and 180, one dense iteration
    (2600, 0.06, 0.01, 0, 4),    # no dense iteration: every candidate fails its stage
    (2600, 0.06, 0.01, 33, 4),   # 181 and 1931, more iterations than the trace holds
    (9000, 0.04, 0.01, 9, 16)])  # 433 and 4116
def test_refinement_shapes(model_points, train_sd, resample, steps, matches):
    from oracle import MODE_GRID, MatchParam as OMP, Oracle, TrainParam as OTP
    from surface_match_gb300 import Detector, MatchParam, PointCloud, TrainParam, synth
    mc, s, c = synth.gear_model(model_points, seed=5)
    sc = synth.make_scene(13, {"gear": s}, 3, ((-100, -100, 40), (100, 100, 140)),
                          points_per_instance=5000, clutter_frac=0.1, clutter="shapes", noise=0.2,
                          model_centers={"gear": c})
    kw = dict(numMatches=matches, poseRefNumSteps=steps, poseRefDistThresholdRel=0.2)
    o = Oracle(mode=MODE_GRID, threads=8)
    om = o.train(mc.xyz, mc.normal, train_sd, OTP(poseRefRelSamplingDistance=resample))
    r = o.match(om, sc.cloud.xyz, None, sc.viewpoint, 0.04, 0.2, 0.02, OMP(**kw))
    det = Detector()
    det.trainModel(PointCloud(mc.xyz, mc.normal), train_sd,
                   TrainParam(poseRefRelSamplingDistance=resample))
    poses, scores = det.matchScene(PointCloud(sc.cloud.xyz, None, sc.viewpoint), 0.04, 0.2, 0.02,
                                   MatchParam(**kw))
    n = len(r.cand_status)
    assert n > 0
    np.testing.assert_array_equal(det.debug(12)[:n], r.cand_status)
    np.testing.assert_array_equal(det.debug(15)[:n], r.cand_trace, err_msg="ICP traces")
    np.testing.assert_array_equal(scores, r.scores)
    np.testing.assert_array_equal(poses[:, :3, :].reshape(-1, 12), r.results[:, :12])
