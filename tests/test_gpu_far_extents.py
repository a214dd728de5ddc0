"""Scenes with stray points so far away that the cells between them and the rest are more than an
int counts, in both search orders: samples, moved positions, normals and poses are the oracle's, bit
for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("order", ["grid", "reference"])
@pytest.mark.parametrize("away", [1e10, 1e13, 1e18])
def test_cells_beyond_an_int(order, away):
    from oracle import MODE_GRID, MODE_REF, MatchParam as OMP, Oracle
    from surface_match_gb300 import Detector, MatchParam, PointCloud, synth
    mc, s, c = synth.gear_model(6000, seed=5)
    sc = synth.make_scene(12, {"gear": s}, 2, ((-70, -70, 40), (70, 70, 100)),
                          points_per_instance=5000, clutter_frac=0.1, clutter="shapes", noise=0.2,
                          model_centers={"gear": c})
    far = np.zeros((2, 3), np.float32)
    far[0] = away
    far[1] = -0.5 * away
    xyz = np.concatenate([sc.cloud.xyz, far]).astype(np.float32)
    kw = dict(numMatches=4)
    o = Oracle(mode=MODE_GRID if order == "grid" else MODE_REF, threads=8)
    r = o.match(o.train(mc.xyz, mc.normal, 0.05), xyz, None, sc.viewpoint, 0.05, 0.2, 0.02,
                OMP(**kw))
    det = Detector(search_order=order)
    det.trainModel(PointCloud(mc.xyz, mc.normal), 0.05)
    poses, scores = det.matchScene(PointCloud(xyz, None, sc.viewpoint), 0.05, 0.2, 0.02,
                                   MatchParam(**kw))
    np.testing.assert_array_equal(det.debug(0), r.sampled)
    np.testing.assert_array_equal(det.debug(2), r.resampled)
    np.testing.assert_array_equal(det.debug(3).view(np.uint32), r.positions.view(np.uint32))
    ok = np.isfinite(r.normals).all(1)
    nrm = det.debug(4)
    np.testing.assert_array_equal(np.isfinite(nrm).all(1), ok)
    np.testing.assert_array_equal(nrm[ok].view(np.uint32), r.normals[ok].view(np.uint32))
    assert len(r.cand_status) > 0
    np.testing.assert_array_equal(scores, r.scores)
    np.testing.assert_array_equal(poses[:, :3, :].reshape(-1, 12), r.results[:, :12])
