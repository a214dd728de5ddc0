"""The trained model's slot table against the one built on the host from the same buckets
(upload): per-keypoint hits, votes and counter bounds of a match agree for models from a few
points (buckets of one entry) to planar ones (buckets of many warps' length)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name, n, sd", [("gear", 300, 0.3), ("gear", 4000, 0.05),
                                         ("bracket", 9000, 0.04), ("torus", 3000, 0.1)])
def test_trained_table_equals_the_uploaded_one(name, n, sd):
    from surface_match_gb300 import Detector, MatchParam, PointCloud, synth
    mc, s, c = synth.model_cloud(name, n, 3)
    sc = synth.make_scene(4, {name: s}, 2, ((-70, -70, 40), (70, 70, 100)), points_per_instance=3000,
                          clutter_frac=0.05, noise=0.1, model_centers={name: c})
    trained = Detector()
    trained.trainModel(PointCloud(mc.xyz, mc.normal), sd)
    d = trained.download()
    assert np.diff(d["offsets"].astype(np.int64)).max() >= 1
    sent = Detector()
    sent.upload(d["sampled"], d["sampled_normal"], d["resampled"], d["resampled_normal"], d["box"],
                d["keys"], d["offsets"], d["refs"], d["alphas"], sd)
    out = []
    for det in (trained, sent):
        det.matchScene(PointCloud(sc.cloud.xyz, None, sc.viewpoint), 0.04, 0.3, 0.1,
                       MatchParam(numMatches=2))
        out.append(det.debug(7))
    np.testing.assert_array_equal(out[0], out[1])
    assert out[0][:, 2].max() >= 1  # there are hits
