"""Reference order counts a call's voting rows (keypoint, neighbour pairs) in 32 bits: a scene with
more of them is refused, as grid order refuses it, and the context goes on working. 47,000 points,
every one a keypoint, all within the model's diameter of each other, have 2.2e9."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("order", ["reference", "grid"])
def test_more_rows_than_an_int_counts(order):
    from surface_match_gb300 import Detector, MatchParam, PointCloud, synth
    mc, s, c = synth.gear_model(6000, seed=5)
    det = Detector(search_order=order)
    det.trainModel(PointCloud(mc.xyz, mc.normal), 0.05)
    rng = np.random.default_rng(3)
    # (0.05 mm steps: the cloud's points are farther apart)
    xyz = np.stack(np.meshgrid(*[np.arange(37)] * 3, indexing="ij"), -1).reshape(-1, 3)[:47000]
    xyz = (xyz * 2.0 + rng.uniform(0, 1, xyz.shape)).astype(np.float32)
    nrm = rng.normal(size=xyz.shape)
    nrm = (nrm / np.linalg.norm(nrm, axis=1, keepdims=True)).astype(np.float32)
    assert len(xyz) ** 2 > 2 ** 31
    with pytest.raises(RuntimeError, match="too many keypoint"):
        det.matchScene(PointCloud(xyz, nrm, None), 0.05 / 142.0, 1.0, 0.0, MatchParam())
    sc = synth.make_scene(12, {"gear": s}, 2, ((-70, -70, 40), (70, 70, 100)),
                          points_per_instance=5000, clutter_frac=0.1, noise=0.2,
                          model_centers={"gear": c})
    _, scores = det.matchScene(PointCloud(sc.cloud.xyz, None, sc.viewpoint), 0.05, 0.2, 0.1,
                               MatchParam(numMatches=2))
    assert len(scores) > 0
