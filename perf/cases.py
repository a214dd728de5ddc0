"""Performance cases: the calls that a user of this framework makes, over their real range.

Every case goes through the Python API of the package (`Detector.trainModel`,
`Detector.matchScene`, `match_batch`, `estimateNormalMLS`). Scenes and models are the
procedural ones of `surface_match_gb300.synth` (gear, L-bracket, torus) with the instance
counts, noise, clutter and sampling distances of the configured workloads and tests; sizes run
from the scene of a parity test to the largest scenes of the batching workload.

`listed()` gives the cases, `draw(rng)` one more of the same ranges, `prepare(case, seed)` what
a program holds before the call, `run(state)` one pass, `work(case)` its necessary bytes and
operations, `exact(case, seed)` 64-bit results where the outputs have such a value.
"""
import functools
import math

import numpy as np
import torch

from surface_match_gb300 import (Detector, MatchParam, MatchResult, PointCloud,
                                 estimateNormalMLS, match_batch, pinned_empty, synth)

# matchScene's arguments and the scene's make-up; a case overrides what it is about
MATCH = {
    "kind": "match", "model": "gear", "model_points": 20000, "train_sd": 0.04,
    "points": 100000, "instances": 3, "noise": 0.2, "clutter": 0.10, "clutter_kind": "shapes",
    "plane": 0.0, "box": 400.0, "source": "device", "normals": False, "viewpoint": True,
    "order": "grid", "sd": 0.04, "kp": 0.2, "min_score": 0.2, "matches": 16, "knn": 10,
    "smooth": True, "dense": True, "steps": 5, "reject": 0.1, "result": False,
}
TRAIN = {"kind": "train", "model": "gear", "points": 20000, "sd": 0.04, "normals": True,
         "order": "grid"}
BATCH = {"kind": "batch", "scenes": 12, "n_min": 50000, "n_max": 1000000, "sd": 0.04, "kp": 0.2,
         "min_score": 0.2, "matches": 16, "workers": 8, "order": "grid", "shape": 1}
MLS = {"kind": "mls", "model": "gear", "points": 50000, "near": 30.0, "degree": 2, "noise": 0.1}
MODELS = ("gear", "bracket", "torus")
BATCH_MODEL_POINTS = 24000


def listed():
    return [
        # the smallest call: two parts on a table, 13 k points. Launches and latency count.
        dict(MATCH, name="match_tiny", points=13001, instances=2, plane=0.33, box=220.0,
             clutter=0.05, clutter_kind="uniform", train_sd=0.05, sd=0.05, matches=4),
        # an ordinary range image: three parts on a table, points on the GPU already
        dict(MATCH, name="match_small", points=108117, plane=0.25, clutter_kind="uniform",
             kp=0.1),
        # a sensor that delivers normals, in host memory, coarse matching only (no dense
        # refinement), with the sampled scene and key points returned to the caller
        dict(MATCH, name="match_host_normals", model="torus", points=150003, instances=5,
             noise=0.3, clutter=0.25, source="host", normals=True, dense=False, result=True),
        # the large single scene: ten parts, 30% clutter, finer sampling
        dict(MATCH, name="match_large", points=918402, instances=10, noise=0.3, clutter=0.30,
             train_sd=0.03, sd=0.03),
        # the largest scene, from page-locked host memory as a camera driver fills it; so dense a
        # cloud takes more neighbours per normal
        dict(MATCH, name="match_xl_pinned", model="bracket", model_points=30011, points=2600007,
             instances=12, noise=0.2, clutter=0.25, source="pinned", knn=24),
        # the reference's example call: a finer model, many matches, a long refinement with a
        # wide search radius
        dict(MATCH, name="match_long_refine", points=350001, instances=6, clutter=0.2,
             train_sd=0.025, sd=0.025, min_score=0.3, matches=55, steps=15, reject=0.3),
        # the reference's own search order (bit-identical results), ordinary and large
        dict(MATCH, name="match_reference_small", points=108117, plane=0.25,
             clutter_kind="uniform", kp=0.1, order="reference"),
        dict(MATCH, name="match_reference_large", points=918402, instances=10, noise=0.3,
             clutter=0.30, train_sd=0.03, sd=0.03, order="reference"),
        # a model trained and its table taken: exact normals, ordinary sampling
        dict(TRAIN, name="train_gear"),
        # a scanned model without normals at a finer sampling
        dict(TRAIN, name="train_bracket_fine", model="bracket", points=39997, sd=0.03,
             normals=False),
        # scenes of uneven size together (a bin-picking cell's cameras, or a serving queue: the
        # server's slots run the same workers)
        dict(BATCH, name="batch_uneven"),
        # smoothed normals and surface projection of a scan
        dict(MLS, name="mls_scan"),
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["match", "match", "match", "reference", "train", "batch", "mls"])
    if kind in ("match", "reference"):
        # clutter without a surface comes with small scenes: every point of it is sampled
        haze = rng.random() < 0.3
        n = _log_uniform(rng, 8000, 120000 if haze else 2500000 if kind == "match" else 450000)
        sd = rng.choice([0.03, 0.035, 0.04, 0.05])
        return dict(
            MATCH, order="grid" if kind == "match" else "reference", points=n,
            model=rng.choice(MODELS), model_points=_log_uniform(rng, 10000, 40000),
            instances=rng.randint(1, 2) if n < 30000 else rng.randint(1, 10),
            noise=rng.uniform(0.1, 0.4), clutter=rng.uniform(0.05, 0.1 if haze else 0.4),
            clutter_kind="uniform" if haze else "shapes",
            plane=rng.choice([0.0, 0.25]), box=250.0 if n < 30000 else 400.0,
            source=rng.choice(["device", "device", "host", "pinned"]),
            normals=rng.random() < 0.25, viewpoint=rng.random() < 0.8, train_sd=sd, sd=sd,
            kp=rng.choice([0.1, 0.1, 0.2] if haze else [0.1, 0.2, 0.2, 0.3]), min_score=rng.choice([0.2, 0.25, 0.3]),
            matches=rng.choice([1, 4, 16, 16]), knn=rng.choice([8, 10, 10, 16, 24]),
            smooth=rng.random() < 0.8, dense=rng.random() < 0.8, steps=rng.choice([5, 5, 9, 15]),
            reject=rng.choice([0.1, 0.1, 0.2, 0.3] if kind == "match" else [0.1, 0.1, 0.2]))
    if kind == "train":
        return dict(TRAIN, model=rng.choice(MODELS), points=_log_uniform(rng, 5000, 40000),
                    sd=rng.choice([0.03, 0.04, 0.05]), normals=rng.random() < 0.6,
                    order=rng.choice(["grid", "grid", "reference"]))
    if kind == "batch":
        return dict(BATCH, scenes=rng.randint(3, 12), n_max=_log_uniform(rng, 100000, 1000000),
                    workers=rng.choice([4, 8]), shape=rng.randint(1, 1000))
    near = rng.uniform(20.0, 80.0)
    return dict(MLS, model=rng.choice(MODELS), points=_log_uniform(rng, 3000, 50000), near=near,
                degree=rng.randint(1, 3 if near > 45.0 else 2), noise=rng.uniform(0.02, 0.15))


# ---------------------------------------------------------------------------- inputs
@functools.lru_cache(maxsize=None)
def _pool(name):
    """100 k surface points and normals of a model, which scenes draw their instances from."""
    cloud, _, _ = synth.model_cloud(name, 100000, seed=5)
    radius = float(np.linalg.norm(cloud.xyz, axis=1).max())
    return torch.from_numpy(cloud.xyz).cuda(), torch.from_numpy(cloud.normal).cuda(), radius


def _uniform(gen, lo, hi, *shape):
    return torch.rand(*shape, generator=gen, device="cuda") * (hi - lo) + lo


def _rotation(rng):
    return torch.from_numpy(synth.random_rotation(rng).astype(np.float32)).cuda()


def _clutter(gen, rng, n, box, kind):
    """n clutter points and normals: uniform in the box, or on random boxes and spheres."""
    hi = torch.tensor([box / 2, box / 2, box / 2], device="cuda")
    if kind == "uniform":
        p = (torch.rand(n, 3, generator=gen, device="cuda") * 2 - 1) * hi
        p[:, 2] = p[:, 2].abs()
        return p, None
    shapes = int(rng.integers(6, 16))
    cuts = np.linspace(0, n, shapes + 1).astype(int)
    pts, nrm = [], []
    for s in range(shapes):
        m = int(cuts[s + 1] - cuts[s])
        c = rng.uniform([-box / 2, -box / 2, 0], [box / 2, box / 2, box / 2])
        c = torch.from_numpy(c.astype(np.float32)).cuda()
        d = torch.randn(m, 3, generator=gen, device="cuda")
        if rng.random() < 0.5:
            half = torch.from_numpy(rng.uniform(7.5, 30, 3).astype(np.float32)).cuda()
            axis = torch.randint(0, 3, (m, 1), generator=gen, device="cuda")
            sign = torch.where(d[:, :1] > 0, 1.0, -1.0)
            u = _uniform(gen, -1, 1, m, 3).scatter(1, axis, sign)
            nn = torch.zeros(m, 3, device="cuda").scatter(1, axis, sign)
            r = _rotation(rng)
            pts.append((u * half) @ r.T + c)
            nrm.append(nn @ r.T)
        else:
            nn = d / d.norm(dim=1, keepdim=True)
            pts.append(nn * float(rng.uniform(8, 30)) + c)
            nrm.append(nn)
    return torch.cat(pts), torch.cat(nrm)


VIEW = (620.0, 100.0, 500.0)


def _scene(seed, model, n, instances, noise, clutter, clutter_kind, plane, box):
    """n noisy points (and normals) that face the viewpoint: instances without overlap, a ground
    plane holding the share `plane`, and clutter, in random order."""
    rng = np.random.default_rng(seed)
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    pool, pool_n, radius = _pool(model)
    placed = []
    for _ in range(20000):
        if len(placed) == instances:
            break
        t = rng.uniform([-box / 2, -box / 2, 0.6 * radius], [box / 2, box / 2, box / 2])
        if all(np.linalg.norm(t - q) >= 2 * radius for q in placed):
            placed.append(t)
    total = int(2.6 * n) + 64  # about half of the surface faces away
    n_clutter = int(total * clutter)
    n_plane = int(n * plane)
    per = (total - n_clutter - n_plane) // max(1, len(placed))
    pts, nrm = [], []
    for t in placed:
        ids = torch.randint(0, pool.shape[0], (per,), generator=gen, device="cuda")
        r = _rotation(rng)
        pts.append(pool[ids] @ r.T + torch.from_numpy(t.astype(np.float32)).cuda())
        nrm.append(pool_n[ids] @ r.T)
    vp = torch.tensor(VIEW, device="cuda")
    if n_plane:
        p = torch.zeros(n_plane, 3, device="cuda")
        p[:, :2] = _uniform(gen, -box / 2, box / 2, n_plane, 2)
        up = torch.zeros(n_plane, 3, device="cuda")
        up[:, 2] = 1.0
        pts.append(p)
        nrm.append(up)
    p, nn = _clutter(gen, rng, n_clutter, box, clutter_kind)
    pts.append(p)
    if nn is None:  # uniform clutter has no surface: it faces the viewer
        nn = vp - p
        nn = nn / nn.norm(dim=1, keepdim=True)
    nrm.append(nn)
    p, nn = torch.cat(pts), torch.cat(nrm)
    p = p + noise * torch.randn(p.shape, generator=gen, device="cuda")
    seen = ((vp - p) * nn).sum(1) > 0
    p, nn = p[seen], nn[seen]
    order = torch.randperm(p.shape[0], generator=gen, device="cuda")[:n]
    return p[order].contiguous(), nn[order].contiguous()


def _placed(t, source):
    if source == "device":
        return t
    host = t.cpu().numpy()
    if source == "host":
        return host
    pinned = pinned_empty(host.shape)
    pinned[:] = host
    return pinned


def _model(name, n, seed):
    cloud, _, _ = synth.model_cloud(name, n, seed=7 + seed % 1000)
    return cloud


def _match_param(case):
    return MatchParam(numMatches=case["matches"], knnNormal=case.get("knn", 10),
                      smoothNormal=case.get("smooth", True),
                      densePoseRefinement=case.get("dense", True),
                      poseRefNumSteps=case.get("steps", 5),
                      poseRefDistThresholdRel=case.get("reject", 0.1))


def _trained(name, n, seed, sd, order):
    cloud = _model(name, n, seed)
    det = Detector(search_order=order)
    det.trainModel(PointCloud(cloud.xyz, cloud.normal), sd)
    return det


def _mls_input(case, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    pool, _, _ = _pool(case["model"])
    ids = torch.randperm(pool.shape[0], generator=gen, device="cuda")[:case["points"]]
    p = pool[ids]
    p = p + case["noise"] * torch.randn(p.shape, generator=gen, device="cuda")
    return p.cpu().numpy()


def _radius(case):
    """The radius that holds `near` points of the scan on average."""
    return math.sqrt(case["near"] * AREA[case["model"]] / (math.pi * case["points"]))


def prepare(case, seed):
    if case["kind"] == "match":
        p, nn = _scene(seed, case["model"], case["points"], case["instances"], case["noise"],
                       case["clutter"], case["clutter_kind"], case["plane"], case["box"])
        scene = PointCloud(_placed(p, case["source"]),
                           _placed(nn, case["source"]) if case["normals"] else None,
                           np.array(VIEW, np.float32) if case["viewpoint"] else None)
        torch.cuda.synchronize()  # the library runs on its own stream
        rows = SAMPLED_ROWS if case["result"] else 0
        return {"case": case, "scene": scene, "param": _match_param(case),
                "clouds": {k: np.zeros((rows, 3), np.float32) for k in CLOUDS} if rows else None,
                "det": _trained(case["model"], case["model_points"], seed, case["train_sd"],
                                case["order"])}
    if case["kind"] == "train":
        cloud = _model(case["model"], case["points"], seed)
        return {"case": case, "det": Detector(search_order=case["order"]),
                "tables": _tables(case),
                "cloud": PointCloud(cloud.xyz, cloud.normal if case["normals"] else None)}
    if case["kind"] == "batch":
        dets = {m: _trained(m, BATCH_MODEL_POINTS, seed, case["sd"], case["order"])
                for m in MODELS}
        jobs = []
        for j, (m, n, inst, noise, clutter) in enumerate(_batch_scenes(case)):
            p, _ = _scene(seed + 7919 * j, m, n, inst, noise, clutter, "shapes", 0.0, 400.0)
            jobs.append((dets[m], PointCloud(p, None, np.array(VIEW, np.float32))))
        torch.cuda.synchronize()
        return {"case": case, "jobs": jobs, "param": _match_param(case)}
    return {"case": case, "points": _mls_input(case, seed), "radius": _radius(case)}


def _batch_scenes(case):
    """(model, points, instances, noise, clutter) of a batch's scenes: log-uniform sizes."""
    rng = np.random.default_rng(case["shape"])
    out = []
    for _ in range(case["scenes"]):
        n = int(math.exp(rng.uniform(math.log(case["n_min"]), math.log(case["n_max"]))))
        out.append((MODELS[int(rng.integers(3))], n, int(rng.integers(1, 11)),
                    float(rng.uniform(0.2, 0.4)), float(rng.uniform(0.1, 0.4))))
    return out


# ---------------------------------------------------------------------------- one pass
# Results vary in length with the inputs; they are filed in arrays of a fixed one, as a program
# with its own buffers does.
COUNTS = ("n_valid", "n_sampled", "n_keypoints", "n_poses", "n_clusters", "n_pairs", "n_hits",
          "n_votes")
CLOUDS = ("sampled", "sampled_normal", "keypoints")
SAMPLED_ROWS = 65536


def _tables(case):
    """Buffers for a trained model's arrays."""
    n = int(1.8 * _sampled(case["model"], case["sd"])) + 256
    m = min(case["points"], int(1.8 * _sampled(case["model"], 0.01)) + 256)
    return {"sampled": np.zeros((n, 3), np.float32), "sampled_normal": np.zeros((n, 3), np.float32),
            "resampled": np.zeros((m, 3), np.float32),
            "resampled_normal": np.zeros((m, 3), np.float32), "box": np.zeros(6, np.float32),
            "keys": np.zeros(n * n, np.int32), "offsets": np.zeros(n * n + 1, np.int32),
            "refs": np.zeros(n * n, np.int32), "alphas": np.zeros(n * n, np.float32)}


def _filed(buffer, rows):
    buffer[:len(rows)] = rows.view(buffer.dtype)  # (32-bit words stay as they are)
    return buffer


def _results(poses, scores, stats, matches):
    return {"poses": _filed(np.zeros((matches, 4, 4), np.float32), poses),
            "scores": _filed(np.zeros(matches, np.float32), scores),
            "counts": np.array([len(scores)] + [stats[k] for k in COUNTS], np.int64)}


def run(state):
    case = state["case"]
    if case["kind"] == "match":
        det = state["det"]
        res = MatchResult() if case["result"] else None
        poses, scores = det.matchScene(state["scene"], case["sd"], case["kp"],
                                       case["min_score"], state["param"], res)
        out = _results(poses, scores, det.last_stats, case["matches"])
        if res is not None:
            for k, a in zip(CLOUDS, (res.sampledScene.point, res.sampledScene.normal,
                                     res.keyPoint.point)):
                out[k] = _filed(state["clouds"][k], a)
        return out
    if case["kind"] == "train":
        state["det"].trainModel(state["cloud"], case["sd"])
        model = state["det"].download()
        return {k: _filed(b, model[k]) for k, b in state["tables"].items()}
    if case["kind"] == "batch":
        results, stats = match_batch(state["jobs"], case["sd"], case["kp"], case["min_score"],
                                     state["param"], concurrency=case["workers"])
        return [_results(p, s, st, case["matches"]) for (p, s), st in zip(results, stats)]
    pc = PointCloud(state["points"])
    estimateNormalMLS(pc, None, state["radius"], case["degree"])
    return {"points": pc.point, "normals": pc.normal}


# ---------------------------------------------------------------------------- work
# surface (mm^2), diameter (mm) of the models: their sampled sizes follow from them
AREA = {"gear": 25318.0, "bracket": 11129.0, "torus": 9475.0}
DIAMETER = {"gear": 142.8, "bracket": 82.5, "torus": 108.6}


def _sampled(model, sd):
    return 0.7 * AREA[model] / (sd * DIAMETER[model]) ** 2


def work(case):
    """Inputs read once and outputs written once; operations: about 30 per scene point (its cell,
    the distance test that keeps or drops it) and, per model point pair of a training, the pair
    feature and its angle (about 120)."""
    if case["kind"] == "match":
        n = case["points"]
        b = n * (24 if case["normals"] else 12)
        b += 12 * case["model_points"]  # the model's table and clouds, of this order at least
        return {"bytes": b + 68 * case["matches"], "flops": 30 * n}
    if case["kind"] == "train":
        pairs = _sampled(case["model"], case["sd"]) ** 2
        return {"bytes": int(case["points"] * (24 if case["normals"] else 12) + 8 * pairs),
                "flops": int(30 * case["points"] + 120 * pairs)}
    if case["kind"] == "batch":
        n = sum(s[1] for s in _batch_scenes(case))
        return {"bytes": n * 12 + 12 * 3 * BATCH_MODEL_POINTS, "flops": 30 * n}
    n, d = case["points"], case["degree"]
    nc = (d + 1) * (d + 2) // 2
    return {"bytes": n * 36, "flops": int(n * case["near"] * (30 + 3 * nc * (nc + 3) / 2))}


# ---------------------------------------------------------------------------- 64 bits
def exact(case, seed):
    """The moving-least-squares fit in 64 bits. matchScene and trainModel have no such value:
    their outputs hang on which points a greedy sampling keeps and which candidate wins."""
    if case["kind"] != "mls":
        return None
    pts = torch.from_numpy(_mls_input(case, seed)).cuda()
    x = pts.double()
    n, r, deg = len(x), _radius(case), case["degree"]
    out_p, out_n = x.clone(), torch.full_like(x, math.nan)
    mono = [(a, b) for a in range(deg + 1) for b in range(deg + 1 - a)]
    eye = torch.eye(len(mono), dtype=torch.float64, device="cuda")
    for i0 in range(0, n, 512):
        f = pts[i0:i0 + 512]
        dx = f[:, None, 0] - pts[None, :, 0]
        dy = f[:, None, 1] - pts[None, :, 1]
        dz = f[:, None, 2] - pts[None, :, 2]
        near = dx * dx + dy * dy + dz * dz < np.float32(r) * np.float32(r)
        most = int(near.sum(1).max())
        val, idx = torch.topk(near.float(), most, dim=1)
        m = val.double()
        nb = x[idx]
        cnt = m.sum(1)
        c = (nb * m[..., None]).sum(1) / cnt[:, None].clamp(min=1)
        e = (nb - c[:, None]) * m[..., None]
        _, vec = torch.linalg.eigh(e.transpose(1, 2) @ e)
        nv = vec[:, :, 0]
        q = x[i0:i0 + 512]
        mid = q - ((q - c) * nv).sum(1, keepdim=True) * nv
        u, v = vec[:, :, 2], vec[:, :, 1]
        d = nb - mid[:, None]
        w = torch.exp(-(d * d).sum(2) / r ** 2) * m
        uc = (d * u[:, None]).sum(2) / r
        vc = (d * v[:, None]).sum(2) / r
        h = (d * nv[:, None]).sum(2) / r
        basis = torch.stack([uc ** a * vc ** b for a, b in mono], 2)
        gram = (basis * w[..., None]).transpose(1, 2) @ basis
        rhs = (basis * (w * h)[..., None]).sum(1)
        chol, info = torch.linalg.cholesky_ex(gram)
        fit = (info == 0) & (cnt >= 3)
        if deg <= 1:
            fit &= cnt >= len(mono)
        chol = torch.where(fit[:, None, None], chol, eye)
        co = torch.cholesky_solve(rhs[..., None], chol)[..., 0]
        p = mid + (co[:, :1] * r) * nv
        nn = nv - co[:, mono.index((1, 0)), None] * u - co[:, mono.index((0, 1)), None] * v
        nn = nn / nn.norm(dim=1, keepdim=True)
        nn = torch.where(nn[:, 2:] < 0, -nn, nn)
        # where the system is not positive definite (a few neighbours) the fit has no value
        some = cnt >= 3
        out_p[i0:i0 + 512] = torch.where(fit[:, None], p, q)
        out_n[i0:i0 + 512] = torch.where(fit[:, None], nn,
                                         torch.where(some[:, None], nv, math.nan))
    return {"points": out_p, "normals": out_n}
