"""Search grids of up to 2^20 cells an axis: a point's cell coordinate is then rounded by up to an
eighth of a cell, which the searches' bounds have to allow for. Moved positions and normals of a
scene beside a point far off on every axis are the oracle's, bit for bit, in both search orders."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("order", ["grid", "reference"])
@pytest.mark.parametrize("away", [-2.1e6, -7e5, 5e4])
def test_rounded_cells(order, away):
    from oracle import MODE_GRID, MODE_REF, MatchParam as OMP, Oracle
    from surface_match_gb300 import Detector, MatchParam, PointCloud, synth
    mc, s, c = synth.gear_model(6000, seed=5)
    sc = synth.make_scene(14, {"gear": s}, 3, ((-120, -120, 40), (120, 120, 140)),
                          points_per_instance=30000, clutter_frac=0.1, clutter="shapes", noise=0.2,
                          model_centers={"gear": c})
    xyz = np.concatenate([sc.cloud.xyz, [[away] * 3]]).astype(np.float32)
    kw = dict(sparsePoseRefinement=False, densePoseRefinement=False)
    o = Oracle(mode=MODE_GRID if order == "grid" else MODE_REF, threads=8)
    r = o.match(o.train(mc.xyz, mc.normal, 0.05), xyz, None, sc.viewpoint, 0.015, 0.01, 0.5,
                OMP(**kw))
    det = Detector(search_order=order)
    det.trainModel(PointCloud(mc.xyz, mc.normal), 0.05)
    det.matchScene(PointCloud(xyz, None, sc.viewpoint), 0.015, 0.01, 0.5, MatchParam(**kw))
    np.testing.assert_array_equal(det.debug(0), r.sampled)
    assert len(r.sampled) > 5000
    np.testing.assert_array_equal(det.debug(3).view(np.uint32), r.positions.view(np.uint32))
    ok = np.isfinite(r.normals).all(1)
    nrm = det.debug(4)
    np.testing.assert_array_equal(np.isfinite(nrm).all(1), ok)
    np.testing.assert_array_equal(nrm[ok].view(np.uint32), r.normals[ok].view(np.uint32))


def test_smoothing_over_rounded_cells():
    from oracle import pyoracle as po
    from surface_match_gb300 import PointCloud, estimateNormalMLS
    from test_gpu_mls_shapes import _wavy
    from test_mls import POINT_TOL_REL
    rng = np.random.default_rng(4)
    P = np.concatenate([_wavy(16000, rng), [[-1.2e6] * 3]]).astype(np.float32)
    ids = rng.permutation(16000)[:2000].astype(np.int64)
    op, on, st = po.mls(P, None, ids, radius=1.5, order=2)
    pc = estimateNormalMLS(PointCloud(P.copy()), ids, 1.5, 2)
    assert (st == 2).all()
    # a neighbour more or less at the rim of some 70 moves a point by several of these tolerances
    assert np.linalg.norm(pc.point[ids] - op[ids], axis=1).max() < POINT_TOL_REL * 1.5
