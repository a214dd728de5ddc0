"""The refinement's step loop, which launches a step while the one before it runs and none after one
without candidates: limits of one, two and many steps, from one candidate and from several, give the
oracle's traces, and raising a limit that no candidate reaches launches nothing more."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("order", ["grid", "reference"])
@pytest.mark.parametrize("matches", [1, 6])
def test_step_limits(matches, order):
    from oracle import MODE_GRID, MODE_REF, MatchParam as OMP, Oracle
    from surface_match_gb300 import Detector, MatchParam, PointCloud, _lib, synth
    mc, s, c = synth.gear_model(2600, seed=5)
    sc = synth.make_scene(13, {"gear": s}, 3, ((-100, -100, 40), (100, 100, 140)),
                          points_per_instance=5000, clutter_frac=0.1, clutter="shapes", noise=0.2,
                          model_centers={"gear": c})
    o = Oracle(mode=MODE_REF if order == "reference" else MODE_GRID, threads=8)
    om = o.train(mc.xyz, mc.normal, 0.06)
    det = Detector(search_order=order)
    det.trainModel(PointCloud(mc.xyz, mc.normal), 0.06)
    lib, launches = _lib.load(), {}
    for steps in (1, 2, 3, 30, 60):
        kw = dict(numMatches=matches, poseRefNumSteps=steps, poseRefDistThresholdRel=0.2)
        r = o.match(om, sc.cloud.xyz, None, sc.viewpoint, 0.06, 0.2, 0.02, OMP(**kw))
        cloud = PointCloud(sc.cloud.xyz, None, sc.viewpoint)
        for _ in range(2):  # (the first call of a shape may allocate and clear)
            before = lib.sm_launch_count()
            det.matchScene(cloud, 0.06, 0.2, 0.02, MatchParam(**kw))
            launches[steps] = lib.sm_launch_count() - before
        n = len(r.cand_status)
        assert n > 0
        np.testing.assert_array_equal(det.debug(12)[:n], r.cand_status)
        np.testing.assert_array_equal(det.debug(15)[:n], r.cand_trace, err_msg="ICP traces")
    # no candidate takes 30 steps here (5 % less residual a step): the limits cost the same
    taken = (r.cand_trace[:, 128:256].reshape(n, 32, 4)[:, :, 0] >= 0).sum(axis=1).max()
    assert taken < 29
    assert launches[60] == launches[30]
