"""Timed cases of the registration path, through its Python entry points.

A case is a dict of plain values; `prepare` makes what a program holds before
the call (device clouds, prepared models, a context) from a seed, `run` is one
pass, `work` the bytes and operations the pass cannot do without, and `exact`
the same outputs computed in 64 bits by plain torch and numpy.  Clouds are the
package's synthetic furniture and rooms at the sizes of the benchmark and the
tests; every cloud depends on the seed.  Stages whose output count depends on
the cloud are called through the C ABI with output buffers that the program
keeps, sized for the cloud and returned whole (zero past the count).
"""
import ctypes
import math

import numpy as np
import torch

import realtime_robot_gb300 as R

CAM = (0.0, -2.5, 1.5)  # the room's camera
SHAPES = {"chair": R.CHAIR, "desk": R.DESK, "sofa": R.SOFA}
LEAF, KEY_R, SHOT_R = 0.01, 0.02, 0.04


def listed():
    return [
        # The reference's own GPU call, once per keypoint: host arrays in and
        # out, one keypoint's occupied voxels.  The smallest call there is.
        {"name": "tdf_one_keypoint", "kind": "tdf", "dim": 30, "occupied": 180},
        # Plain ICP of two 20,000-point chairs, 50 iterations within 5 cm.
        {"name": "icp_chair_20k", "kind": "icp", "shape": "chair", "source": 20000, "target": 20000,
         "iterations": 50, "max_dist": 0.05},
        # One step of camera tracking: a depth frame back-projected, thinned
        # to 2 cm and registered to the previous frame's full cloud.
        {"name": "odometry_640x480", "kind": "odometry", "width": 640, "height": 480, "iterations": 30},
        # The scene side of main (ScanPoint::getKeypoint), stage by stage, on
        # a cloud whose size is no multiple of anything.
        {"name": "scan_keypoints_123k", "kind": "scan", "points": 123457},
        # Descriptor matching of a whole room against one model.
        {"name": "match_room_111k", "kind": "match", "queries": 111111, "rows": 3001},
        # Grouping of all the correspondences of a room's matching.
        {"name": "group_room_300k", "kind": "group", "points": 300000, "model": 20000},
        # One training batch of the credibility network: forward and backward.
        {"name": "mlp_gradient_4096", "kind": "mlp", "rows": 4096, "backward": True},
        # The reference's descriptor route: occupancy and distance fields, then
        # get_Distance for every pair of keypoints; clouds and keypoints as
        # many as main's own two have.
        {"name": "ref_route_main", "kind": "ref_route", "model": 1818, "scan": 3218, "model_keys": 340,
         "scan_keys": 573},
        # What main's ModelPoint finds in a cloud: Harris keypoints, planes
        # with their areas, and the keypoints' plane-area vectors.
        {"name": "harris_planes_20k", "kind": "harris", "shape": "chair", "points": 20000},
        # Recognition of one segmented object: small, latency counts.
        {"name": "recognize_segment_12k", "kind": "recognize", "scene": "segment", "shape": "chair",
         "points": 12000, "model": 20000},
        # Recognition of the chair in a 300,000-point room: the benchmark's
        # headline.
        {"name": "recognize_room_300k", "kind": "recognize", "scene": "room", "shape": "chair",
         "points": 300000, "model": 20000},
        # 64 model/segment pairs of 2,000 to 60,000 points with learned
        # pruning: registration in bulk.
        {"name": "recognize_batch_64", "kind": "batch", "pairs": 64, "learned": True},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["tdf", "icp", "odometry", "scan", "match", "group", "mlp", "ref_route", "harris",
                       "segment", "room", "batch"])
    shape = rng.choice(sorted(SHAPES))
    if kind == "tdf":
        return {"kind": kind, "dim": rng.randint(8, 30), "occupied": _log(rng, 1, 2000)}
    if kind == "icp":
        return {"kind": kind, "shape": shape, "source": _log(rng, 2000, 60000), "target": _log(rng, 2000, 60000),
                "iterations": rng.randint(10, 50), "max_dist": round(rng.uniform(0.02, 0.1), 3)}
    if kind == "odometry":
        w = rng.randint(160, 640)
        return {"kind": kind, "width": w, "height": max(120, w * 3 // 4), "iterations": rng.randint(10, 30)}
    if kind == "scan":
        return {"kind": kind, "points": _log(rng, 20000, 300000)}
    if kind == "match":
        return {"kind": kind, "queries": _log(rng, 1000, 111111), "rows": _log(rng, 300, 3001)}
    if kind == "group":
        return {"kind": kind, "points": _log(rng, 20000, 300000), "model": _log(rng, 5000, 20000)}
    if kind == "mlp":
        return {"kind": kind, "rows": _log(rng, 200, 30000), "backward": rng.random() < 0.5}
    if kind == "ref_route":
        return {"kind": kind, "model": _log(rng, 600, 3000), "scan": _log(rng, 600, 3218),
                "model_keys": _log(rng, 1, 340), "scan_keys": _log(rng, 10, 573)}
    if kind == "harris":
        return {"kind": kind, "shape": shape, "points": _log(rng, 5000, 30000)}
    if kind == "segment":
        return {"kind": "recognize", "scene": "segment", "shape": shape, "points": _log(rng, 2000, 60000),
                "model": _log(rng, 2000, 60000)}
    if kind == "room":
        return {"kind": "recognize", "scene": "room", "shape": shape, "points": _log(rng, 50000, 300000),
                "model": _log(rng, 5000, 20000)}
    return {"kind": kind, "pairs": rng.randint(4, 40), "learned": rng.random() < 0.5}


# -- inputs -------------------------------------------------------------------
def _dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def _room(n, seed):
    p = R.room_default_params()
    p.n_points = n
    return R.synth_room(seed, p)[0]


def _moved(shape, n, seed, crop):
    """A copy of the shape under a rigid motion with 2 mm noise, partly cut off."""
    T = R.synth_rigid(seed, 30.0, 0.3)
    pts = R.synth_transform_noise(R.synth_shape(SHAPES[shape], n, 7 * seed + 1), T, 0.002, seed + 11)
    return R.synth_crop(pts, crop, seed + 13) if crop > 0 else pts


def _described(ctx, pts, outward):
    """(keypoints, descriptors) of a cloud, the stages of a recognition."""
    vox = ctx.voxel_downsample(pts, LEAF).contiguous()
    nrm = ctx.normals(vox, 10, (0.0, 0.0, 0.0) if outward else CAM, 2.0 * LEAF)
    if outward:
        ctx.orient_outward(vox, nrm)
    keys = ctx.uniform_sample(vox, KEY_R).contiguous()
    return vox[keys.long()].contiguous(), ctx.shot352(vox, nrm, keys, SHOT_R)


def _rows(t, n):
    """n rows of t, the first ones again where it has fewer."""
    return t[torch.arange(n, device=t.device) % t.shape[0]].contiguous()


def _zeros(*shape, dtype=torch.float32):
    return torch.zeros(shape, dtype=dtype, device="cuda")


def _network(rng):
    """He-uniform weights of the 352-128-64-1 network, small biases."""
    parts = []
    for rows, cols in ((128, 352), (64, 128), (1, 64)):
        b = math.sqrt(6.0 / cols)
        parts += [rng.uniform(-b, b, rows * cols), rng.uniform(-0.05, 0.05, rows)]
    return np.concatenate(parts).astype(np.float32)


def _frames(ctx, width, height, seed):
    """Two consecutive depth frames of a furnished room along a camera path,
    and the motion of the step before them."""
    p = R.room_default_params()
    p.n_chairs, p.n_desks, p.n_sofas = 6, 2, 1
    boxes = R.synth_room_boxes(seed, p)[0]
    first = 1 + seed % 200
    poses = R.synth_trajectory(seed, first + 2)
    fx = 525.0 * width / 640.0
    cam = {"fx": fx, "fy": fx, "cx": 0.5 * (width - 1), "cy": 0.5 * (height - 1)}
    depth = ctx.synth_depth_frames(boxes, poses[first:first + 2], width, height, seed=seed, **cam)
    return depth, cam, np.linalg.inv(poses[first - 1]) @ poses[first]


def prepare(case, seed):
    kind = case["kind"]
    rng = np.random.default_rng(seed)
    if kind == "tdf":
        # voxels of a surface patch through the keypoint, as an occupancy grid holds
        d, n = case["dim"], case["occupied"]
        uv = rng.uniform(0, d, (n, 2))
        tilt = rng.uniform(-0.5, 0.5, 2)
        z = d / 2 + (uv - d / 2) @ tilt + rng.normal(0, 0.7, n)
        occ = np.clip(np.floor(np.column_stack([uv, z])), 0, d - 1).astype(np.int32)
        return {"case": case, "occ": occ, "out": np.zeros(27000, np.float32)}
    ctx = R.Context(0)
    s = {"case": case, "ctx": ctx}
    if kind == "icp":
        shape = SHAPES[case["shape"]]
        src = R.synth_shape(shape, case["source"], seed)
        same = case["source"] == case["target"]  # the target is then the source, moved
        tgt = R.synth_transform_noise(src if same else R.synth_shape(shape, case["target"], seed + 1),
                                      R.synth_rigid(seed, 15.0, 0.1), 0.002, seed + 7)
        s["src"], s["tgt"] = _dev(src), _dev(tgt)
    elif kind == "odometry":
        depth, cam, vel = _frames(ctx, case["width"], case["height"], seed)
        pts, cnt = ctx.depth_to_points(depth[0], **cam)
        n = case["width"] * case["height"]
        s.update(depth=depth[1].contiguous(), prev=pts[:int(cnt.item())].contiguous(), cam=cam, vel=vel,
                 cloud=_zeros(n, 4), thin=_zeros(n, 4), count=_zeros(1, dtype=torch.int32))
    elif kind == "scan":
        n = case["points"]
        s.update(pts=_dev(_room(n, seed)), vox=_zeros(n, 4), nrm=_zeros(n, 4), keys=_zeros(n, dtype=torch.int32),
                 shot=_zeros(n, 352), count=_zeros(1, dtype=torch.int32), cam=np.array(CAM, np.float32))
    elif kind == "match":
        room = _dev(_room(min(300000, 20000 + 3 * case["queries"]), seed))
        model = _dev(R.synth_shape(R.CHAIR, min(20000, 2000 + 7 * case["rows"]), seed + 3))
        s["query"] = _rows(_described(ctx, room, False)[1], case["queries"])
        s["db"] = _rows(_described(ctx, model, True)[1], case["rows"])
    elif kind == "group":
        sk, sd = _described(ctx, _dev(_room(case["points"], seed)), False)
        mk, md = _described(ctx, _dev(R.synth_shape(R.CHAIR, case["model"], seed + 3)), True)
        idx, d2 = ctx.match(sd, md)
        kept = torch.nonzero(d2 < 0.25).reshape(-1)
        s.update(mk=mk, sk=sk, cm=idx[kept].contiguous(), cs=kept.to(torch.int32).contiguous(),
                 cd=d2[kept].contiguous(), members=_zeros(256, 128, dtype=torch.int32),
                 sizes=_zeros(256, dtype=torch.int32), poses=_zeros(256, 16, dtype=torch.float64))
    elif kind == "mlp":
        # rows like SHOT descriptors: sparse, non-negative, of unit length; a tenth of them positive
        g = torch.Generator(device="cuda").manual_seed(seed)
        x = torch.relu(torch.randn(case["rows"], 352, device="cuda", generator=g) - 1.0)
        s["x"] = x / x.norm(dim=1, keepdim=True).clamp_min(1e-6)
        s["y"] = (torch.rand(case["rows"], device="cuda", generator=g) < 0.1).float()
        s["theta"] = _network(rng)
        s["mlp"] = R.Mlp(ctx, s["theta"])
    elif kind == "ref_route":
        m = _dev(R.synth_shape(R.CHAIR, case["model"], seed))
        c = _dev(_moved("chair", case["scan"], seed, 0.0))
        s.update(m=m, c=c, mk=_rows(m[ctx.uniform_sample(m, 0.05).long()], case["model_keys"]),
                 ck=_rows(c[ctx.uniform_sample(c, 0.05).long()], case["scan_keys"]))
        s["cap"] = case["model_keys"] * min(case["model"], 512) + 4096
        s["indices"] = _zeros(s["cap"], dtype=torch.int32)
    elif kind == "harris":
        n = case["points"]
        s.update(pts=_dev(R.synth_shape(SHAPES[case["shape"]], n, seed)), keys=_zeros(n, 4),
                 src=_zeros(n, dtype=torch.int32), v3=_zeros(n, 3, dtype=torch.float64),
                 count=_zeros(1, dtype=torch.int32), planes=(R.Surface * 64)())
    elif kind == "recognize":
        room = case["scene"] == "room"
        s["prm"] = R.recog_default_params(viewpoint=CAM) if room else R.recog_default_params(scene_outward=1)
        s["model"] = R.Model(ctx, _dev(R.synth_shape(SHAPES[case["shape"]], case["model"], seed + 3)), s["prm"])
        s["scene"] = _dev(_room(case["points"], seed) if room else _moved(case["shape"], case["points"], seed, 0.4))
        s["result"] = torch.zeros(ctypes.sizeof(R.RecogResult), dtype=torch.uint8, device="cuda")
    elif kind == "batch":
        s["prm"] = R.recog_default_params(viewpoint=(0.0, 0.0, 0.0))
        s["models"], s["scenes"] = [], []
        for i in range(case["pairs"]):
            shape = sorted(SHAPES)[i % 3]
            nm, ns = (int(round(math.exp(rng.uniform(math.log(2000), math.log(60000))))) for _ in range(2))
            s["models"].append(R.Model(ctx, _dev(R.synth_shape(SHAPES[shape], nm, seed + 1000 * i)), s["prm"]))
            s["scenes"].append(_dev(_moved(shape, ns, seed + i, 0.4)))
        s["mlp"] = R.Mlp(ctx, _network(rng)) if case["learned"] else None
        s["results"] = torch.zeros((case["pairs"], ctypes.sizeof(R.RecogResult)), dtype=torch.uint8, device="cuda")
    else:
        raise ValueError(kind)
    return s


# -- one pass -----------------------------------------------------------------
def _recognitions(raw):
    """Views of rtr_recog_result records: counts, then 16 instances each."""
    raw = raw.reshape(-1, raw.shape[-1])
    n = raw.shape[0]
    ints, reals = raw.view(torch.int32), raw.view(torch.float64)
    return {"counts": ints[:, :6],
            "poses": reals[:, 4:].reshape(n, 16, 18)[:, :, :16],
            "scores": raw.view(torch.float32)[:, 8:].reshape(n, 16, 36)[:, :, 32],
            "clusters": ints[:, 8:].reshape(n, 16, 36)[:, :, 33:35]}


def run(s):
    case, kind = s["case"], s["case"]["kind"]
    if kind == "tdf":
        R.compute_tdf_with_cuda(s["occ"], s["out"], case["dim"])
        return s["out"][:case["dim"] ** 3]
    ctx = s["ctx"]
    if kind == "icp":
        r, _, _ = ctx.icp(s["src"], s["tgt"], case["iterations"], case["max_dist"])
        f = r.view(torch.float64)
        return {"pose": f[:16], "fitness": f[16:17], "iterations": r.view(torch.int32)[34:37]}
    lib, h, st = R.lib(), ctx.h, torch.cuda.current_stream().cuda_stream
    if kind == "odometry":
        ctx.depth_to_points(s["depth"], out=s["cloud"], count=s["count"], **s["cam"])
        n = int(s["count"].item())
        R.check(lib.rtr_voxel_downsample(h, s["cloud"].data_ptr(), n, 0.02, s["thin"].data_ptr(),
                                         s["count"].data_ptr(), st))
        r, _, _ = ctx.icp(s["thin"][:int(s["count"].item())], s["prev"], case["iterations"], 0.02, init=s["vel"])
        r = ctx.parse_icp_result(r)
        return {"cloud": s["cloud"], "thin": s["thin"], "pose": r["pose"], "fitness": r["fitness"],
                "n_corr": r["n_corr"]}
    if kind == "scan":
        vox, nrm, keys, shot, count = (s[k] for k in ("vox", "nrm", "keys", "shot", "count"))
        R.check(lib.rtr_voxel_downsample(h, s["pts"].data_ptr(), s["pts"].shape[0], LEAF, vox.data_ptr(),
                                         count.data_ptr(), st))
        n = int(count.item())
        R.check(lib.rtr_normals(h, vox.data_ptr(), n, 10, s["cam"].ctypes.data, 2.0 * LEAF, nrm.data_ptr(), st))
        R.check(lib.rtr_uniform_sample(h, vox.data_ptr(), n, KEY_R, keys.data_ptr(), count.data_ptr(), st))
        R.check(lib.rtr_shot352(h, vox.data_ptr(), nrm.data_ptr(), n, keys.data_ptr(), int(count.item()), SHOT_R,
                                shot.data_ptr(), None, st))
        return {"voxels": vox, "normals": nrm, "keys": keys, "shot": shot}
    if kind == "match":
        idx, d2 = ctx.match(s["query"], s["db"])
        return {"idx": idx, "d2": d2}
    if kind == "group":
        found = ctypes.c_int(0)
        R.check(lib.rtr_gc_group(h, s["mk"].data_ptr(), s["sk"].data_ptr(), s["cm"].data_ptr(), s["cs"].data_ptr(),
                                 s["cd"].data_ptr(), s["cm"].shape[0], 0.01, 5, 256, 128, s["members"].data_ptr(),
                                 s["sizes"].data_ptr(), s["poses"].data_ptr(), ctypes.byref(found), st))
        return {"members": s["members"], "sizes": s["sizes"], "poses": s["poses"], "found": found.value}
    if kind == "mlp":
        if not case["backward"]:
            return {"score": s["mlp"].score(s["x"])}
        loss, grad = s["mlp"].loss_grad(s["x"], s["y"])
        return {"loss": loss, "grad": grad}
    if kind == "ref_route":
        keys, total = s["mk"].shape[0], ctypes.c_longlong(0)
        number, offsets = (torch.empty(k, dtype=torch.int32, device="cuda") for k in (keys, keys + 1))
        R.check(lib.rtr_ref_occupancy(h, s["m"].data_ptr(), s["m"].shape[0], s["mk"].data_ptr(), keys, 0.01, 0.1,
                                      number.data_ptr(), offsets.data_ptr(), s["indices"].data_ptr(), s["cap"],
                                      ctypes.byref(total), st))
        scan_number, _, _ = ctx.ref_occupancy(s["c"], s["ck"])
        tdf = ctx.ref_tdf(s["m"], s["mk"], offsets, s["indices"])
        score, T = ctx.ref_distance(s["m"], s["mk"], offsets, s["indices"], tdf, s["ck"])
        return {"number": number, "offsets": offsets, "indices": s["indices"], "scan_number": scan_number,
                "tdf": tdf, "score": score, "T": T}
    if kind == "harris":
        n, pts, found = s["pts"].shape[0], s["pts"].data_ptr(), ctypes.c_int(0)
        prm, plane_prm = R.harris_default_params(), R.plane_default_params()
        R.check(lib.rtr_harris3d(h, pts, n, ctypes.byref(prm), s["keys"].data_ptr(), s["src"].data_ptr(),
                                 s["count"].data_ptr(), st))
        R.check(lib.rtr_plane_segment(h, pts, n, ctypes.byref(plane_prm), s["planes"], 64, ctypes.byref(found), st))
        R.check(lib.rtr_vector3d(h, s["keys"].data_ptr(), int(s["count"].item()), s["planes"], found.value,
                                 s["v3"].data_ptr(), st))
        p = np.ctypeslib.as_array(s["planes"])
        return {"keys": s["keys"], "src": s["src"], "v3": s["v3"], "found": found.value, "area": p["area"],
                "perimeter": p["perimeter"], "coeffs": p["coeffs"], "inliers": p["n_inliers"],
                "vertices": p["hull_vertices"], "class": p["is_vertical"], "kept": p["kept"]}
    if kind == "recognize":
        return _recognitions(R.recognize(ctx, s["model"], s["scene"], s["prm"], result=s["result"]))
    R.recognize_batch(ctx, s["models"], s["scenes"], s["prm"], mlp=s["mlp"], keep=0.25 if s["mlp"] else 1.0,
                      results=s["results"])
    return _recognitions(s["results"])


# -- the least a pass has to do -------------------------------------------------
def _recognition_work(scene, model):
    """A recognition's inputs and its largest product, keypoints against
    keypoints (about a third of a scene's and a seventh of a model's points)."""
    return 16.0 * scene + 32.0 * model + 2336.0, 2.0 * 352 * (0.38 * scene) * (0.15 * model)


def work(case):
    kind = case["kind"]
    if kind == "tdf":
        b, f = 12.0 * case["occupied"] + 4.0 * case["dim"] ** 3, 0.0
    elif kind == "icp":
        # per iteration a source point is moved, compared with a few target points and summed up
        b, f = 16.0 * (case["source"] + case["target"]) + 152, 100.0 * case["source"] * case["iterations"]
    elif kind == "odometry":
        n = case["width"] * case["height"]
        b, f = 4.0 * n + 16.0 * n + 16.0 * n, 100.0 * 0.05 * n * case["iterations"]
    elif kind == "scan":
        n = case["points"]
        b, f = 16.0 * n + 16.0 * 0.8 * n * 2 + 4.0 * 352 * 0.45 * n, 200.0 * n + 5000.0 * 0.45 * n
    elif kind == "match":
        q, d = case["queries"], case["rows"]
        b, f = 4.0 * 352 * (q + d) + 8.0 * q, 2.0 * 352 * q * d
    elif kind == "group":
        q = 0.37 * case["points"]
        b, f = 16.0 * q + 12.0 * q + 4.0 * 256 * 128, 20.0 * q * 3000
    elif kind == "mlp":
        n, w = case["rows"], 352 * 128 + 128 * 64 + 64
        b = 4.0 * 352 * n + 4.0 * n + 4.0 * 53505 * (2 if case["backward"] else 1)
        f = 2.0 * n * w * (3 if case["backward"] else 1) - (2.0 * n * 352 * 128 if case["backward"] else 0)
    elif kind == "ref_route":
        # 36 turns of some 150 occupied points a pair, a score and a transform out
        pairs = case["model_keys"] * case["scan_keys"]
        b, f = 68.0 * pairs + 4.0 * 27000 * case["model_keys"], 36.0 * 150 * 20 * pairs
    elif kind == "harris":
        b, f = 16.0 * case["points"] * 2, 300.0 * 30 * case["points"]
    elif kind == "recognize":
        b, f = _recognition_work(case["points"], case["model"])
    else:
        b, f = (case["pairs"] * x for x in _recognition_work(14000, 14000))
    return {"bytes": b, "flops": f}


# -- the same outputs in 64 bits -------------------------------------------------
def _nearest(q, t, chunk=1 << 27):
    """Squared distance and index of each q's nearest t (float64, brute force)."""
    t2 = (t * t).sum(1)
    step = max(1, chunk // t.shape[0])
    d, j = [], []
    for a in range(0, q.shape[0], step):
        m = torch.addmm(t2[None, :], q[a:a + step], t.T, alpha=-2.0).min(1)
        j.append(m.indices)
        d.append(((q[a:a + step] - t[m.indices]) ** 2).sum(1))
    return torch.cat(d), torch.cat(j)


def _icp64(src, tgt, iterations, max_dist, init):
    """Point-to-point ICP in float64: pose and the last mean squared distance."""
    src, tgt = src[:, :3].double(), tgt[:, :3].double()
    P = torch.as_tensor(init, dtype=torch.float64, device=src.device).clone()
    fit = 0.0
    for _ in range(iterations):
        p = src @ P[:3, :3].T + P[:3, 3]
        d2, j = _nearest(p, tgt)
        ok = d2 <= max_dist * max_dist
        a, b = p[ok], tgt[j[ok]]
        ma, mb = a.mean(0), b.mean(0)
        U, _, Vt = torch.linalg.svd(((a - ma).T @ (b - mb)).cpu())
        S = torch.diag(torch.tensor([1.0, 1.0, float(torch.sign(torch.det(U @ Vt)))], dtype=torch.float64))
        D = torch.eye(4, dtype=torch.float64)
        D[:3, :3] = Vt.T @ S @ U.T
        D = D.to(src.device)
        D[:3, 3] = mb - D[:3, :3] @ ma
        P = D @ P
        fit = d2[ok].mean()
    return P, fit


def _centroids(pts, leaf):
    """Mean of the points of each voxel, voxels in key order.  The voxel of a
    point is a whole number, found as the filter defines it, in 32 bits."""
    c = torch.floor(pts[:, :3] * torch.tensor(1.0, dtype=torch.float32).div(leaf).to(pts)).long()
    c = c - c.min(0).values
    ext = c.max(0).values + 1
    key = (c[:, 2] * ext[1] + c[:, 1]) * ext[0] + c[:, 0]
    _, inv, num = torch.unique(key, return_inverse=True, return_counts=True)
    out = torch.zeros((num.shape[0], 4), dtype=torch.float64, device=pts.device)
    out.index_add_(0, inv, torch.nn.functional.pad(pts[:, :3].double(), (0, 1)))
    return out / num[:, None]


def _normals64(v, vp, k):
    """Normals and curvature of the k nearest points' covariance."""
    x = v[:, :3]
    x2 = (x * x).sum(1)
    step = max(1, (1 << 27) // x.shape[0])
    near = torch.cat([torch.addmm(x2[None, :], x[a:a + step], x.T, alpha=-2.0).topk(k, 1, largest=False).indices
                      for a in range(0, x.shape[0], step)])
    d = x[near] - x[near].mean(1, keepdim=True)
    w, V = np.linalg.eigh((d.transpose(1, 2) @ d).cpu().numpy())
    n = torch.from_numpy(np.ascontiguousarray(V[:, :, 0])).to(x.device)
    w = torch.from_numpy(w).to(x.device)
    to = torch.tensor(vp, dtype=torch.float64, device=x.device) - x
    n = torch.where(((to * n).sum(1) < 0)[:, None], -n, n)
    return torch.cat([n, (w[:, 0] / w.sum(1))[:, None]], 1)


def exact(case, seed):
    kind = case["kind"]
    if kind in ("group", "ref_route", "harris", "recognize", "batch"):
        # numbers that follow from long chains of whole-number choices (members
        # of consensus sets, octree leaves, samples of a plane)
        return None
    s = prepare(case, seed)
    if kind == "tdf":
        d = case["dim"]
        occ = torch.from_numpy(s["occ"]).cuda().double()
        a = torch.arange(d, device="cuda", dtype=torch.float64)
        z, y, x = torch.meshgrid(a, a, a, indexing="ij")
        v = torch.stack([x, y, z], -1).reshape(-1, 3)
        out = torch.full((v.shape[0],), 900.0, dtype=torch.float64, device="cuda")
        for b in range(0, occ.shape[0], 256):
            out = torch.minimum(out, ((v[:, None] - occ[None, b:b + 256]) ** 2).sum(-1).min(1).values)
        return out.cpu().numpy()
    if kind == "icp":
        P, fit = _icp64(s["src"], s["tgt"], case["iterations"], case["max_dist"], np.eye(4))
        return {"pose": P.reshape(-1), "fitness": fit.reshape(1), "iterations": None}
    if kind == "odometry":
        d, cam = s["depth"].double(), s["cam"]
        v, u = torch.meshgrid(torch.arange(d.shape[0], device="cuda").double(),
                              torch.arange(d.shape[1], device="cuda").double(), indexing="ij")
        pts = torch.stack([(u - cam["cx"]) * d / cam["fx"], (v - cam["cy"]) * d / cam["fy"], d,
                           torch.zeros_like(d)], -1)
        cloud = pts[(s["depth"] > 0.05) & (s["depth"] < 8.0)]
        thin = _centroids(cloud.float(), 0.02)
        P, fit = _icp64(thin, s["prev"], case["iterations"], 0.02, s["vel"])
        cloud, thin = (torch.nn.functional.pad(t, (0, 0, 0, d.numel() - t.shape[0])) for t in (cloud, thin))
        return {"cloud": cloud, "thin": thin, "pose": P.cpu().numpy(), "fitness": float(fit), "n_corr": None}
    if kind == "scan":
        vox = _centroids(s["pts"], LEAF)
        vox, nrm = (torch.nn.functional.pad(t, (0, 0, 0, case["points"] - t.shape[0]))
                    for t in (vox, _normals64(vox, CAM, 10)))
        return {"voxels": vox, "normals": nrm, "keys": None, "shot": None}
    if kind == "match":
        return {"idx": None, "d2": _nearest(s["query"].double(), s["db"].double())[0]}
    # mlp: the forward pass multiplies by the weights rounded to bfloat16
    th = torch.from_numpy(s["theta"]).cuda()
    parts = torch.split(th, [128 * 352, 128, 64 * 128, 64, 64, 1])
    W1, W2, w3 = (parts[i].to(torch.bfloat16).double() for i in (0, 2, 4))
    W1, W2 = W1.reshape(128, 352), W2.reshape(64, 128)
    b1, b2, b3 = (parts[i].double() for i in (1, 3, 5))
    x, y = s["x"].double(), s["y"].double()
    h1 = torch.relu(x @ W1.T + b1)
    h2 = torch.relu(h1 @ W2.T + b2)
    z = h2 @ w3 + b3
    if not case["backward"]:
        return {"score": torch.sigmoid(z)}
    loss = (z.clamp_min(0) - y * z + torch.log1p(torch.exp(-z.abs()))).mean()
    dz = (torch.sigmoid(z) - y) / x.shape[0]
    dh2 = dz[:, None] * w3[None, :] * (h2 > 0)
    dh1 = (dh2 @ W2) * (h1 > 0)
    grad = torch.cat([(dh1.T @ x).reshape(-1), dh1.sum(0), (dh2.T @ h1).reshape(-1), dh2.sum(0), h2.T @ dz,
                      dz.sum().reshape(1)])
    return {"loss": loss.reshape(1), "grad": grad}
