"""Point preparation, selection and the scans where their vector loads can go wrong, against the
oracle: sizes around four points, a thread's eight values and a tile of 4096; scene arrays that
are not 16-byte aligned; every point finite or some not; given normals."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n, shift, bad, normals", [
    (1, 0, 0, False), (3, 1, 0, False), (5, 2, 1, True), (4095, 3, 0, False), (4096, 1, 7, True),
    (4097, 0, 7, False), (9001, 2, 0, True), (17003, 3, 2000, False)])
def test_prepared_points(n, shift, bad, normals):
    import torch
    from oracle import MODE_GRID, MatchParam as OMP, Oracle
    from surface_match_gb300 import Detector, MatchParam, PointCloud, synth
    mc, s, c = synth.gear_model(3000, seed=5)
    sc = synth.make_scene(21, {"gear": s}, 2, ((-70, -70, 40), (70, 70, 100)),
                          points_per_instance=16000, clutter_frac=0.1, noise=0.2,
                          model_centers={"gear": c})
    rng = np.random.default_rng(n)
    xyz = sc.cloud.xyz[:n].copy()
    assert len(xyz) == n
    nrm = None
    if normals:
        nrm = sc.viewpoint - xyz
    if bad:
        ids = rng.permutation(n)[:bad]
        (xyz if nrm is None else nrm)[ids, rng.integers(0, 3, bad)] = np.nan

    def put(a):  # a device array that starts `shift` floats after a 16-byte boundary
        if a is None:
            return None
        t = torch.zeros(3 * n + shift, dtype=torch.float32, device="cuda")
        t[shift:] = torch.from_numpy(np.ascontiguousarray(a, np.float32).reshape(-1)).cuda()
        v = t[shift:].view(n, 3)
        assert v.data_ptr() % 16 == 4 * shift
        return v

    o = Oracle(mode=MODE_GRID, threads=4)
    om = o.train(mc.xyz, mc.normal, 0.06)
    r = o.match(om, xyz, nrm, sc.viewpoint, 0.06, 0.3, 0.1, OMP(numMatches=2))
    det = Detector()
    det.trainModel(PointCloud(mc.xyz, mc.normal), 0.06)
    p, q = put(xyz), put(nrm)
    torch.cuda.synchronize()
    poses, scores = det.matchScene(PointCloud(p, q, sc.viewpoint), 0.06, 0.3, 0.1,
                                   MatchParam(numMatches=2))
    np.testing.assert_array_equal(det.debug(0), r.sampled)
    np.testing.assert_array_equal(det.debug(1), r.keypoints)
    np.testing.assert_array_equal(det.debug(7), r.kp_stats)
    np.testing.assert_array_equal(scores, r.scores)
