"""A refinement's step limit set as "until it converges" - a million, or the largest int - takes no
more workspace than a small one and gives the same poses as a limit beyond the last step taken."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("order", ["grid", "reference"])
def test_any_step_limit(order):
    from surface_match_gb300 import Detector, MatchParam, PointCloud, synth
    mc, s, c = synth.gear_model(6000, seed=5)
    sc = synth.make_scene(12, {"gear": s}, 2, ((-70, -70, 40), (70, 70, 100)),
                          points_per_instance=5000, clutter_frac=0.1, clutter="shapes", noise=0.2,
                          model_centers={"gear": c})
    det = Detector(search_order=order)
    det.trainModel(PointCloud(mc.xyz, mc.normal), 0.05)
    got = [det.matchScene(PointCloud(sc.cloud.xyz, None, sc.viewpoint), 0.05, 0.2, 0.02,
                          MatchParam(numMatches=8, poseRefNumSteps=steps))
           for steps in (200, 1000000, 2 ** 31 - 1)]
    assert len(got[0][1]) > 0
    for poses, scores in got[1:]:
        np.testing.assert_array_equal(scores, got[0][1])
        np.testing.assert_array_equal(poses, got[0][0])
