"""GPU parity of the persistent ICP kernel.

Per iteration the FP64 oracle is replayed on the GPU's own pose: the
correspondences must be bit-exact and the oracle's FP64 pose update (on those
same correspondences) must agree with the GPU's to <= 1e-5 m and <= 1e-5 rad."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu

TOL_T = 1e-5  # metres
TOL_R = 1e-5  # radians


def _dev(a):
    import torch
    return torch.from_numpy(np.ascontiguousarray(a, np.float32)).cuda()


def _replay_check(ctx, src, tgt, iters, max_dist, init=None):
    res, tp, tc = ctx.icp(_dev(src), _dev(tgt), iters, max_dist, init=init, trace=True)
    r = ctx.parse_icp_result(res)
    assert r["status"] == 0
    n_it = r["iterations"]
    poses = tp.cpu().numpy()[: n_it + 1]
    corr = tc.cpu().numpy()[:n_it]
    ocorr, opose, ncorr = O.icp_replay(src, tgt, max_dist, poses)
    worst_t = worst_r = 0.0
    for k in range(n_it):
        assert np.array_equal(corr[k], ocorr[k]), f"iteration {k}: correspondences differ"
        if ncorr[k] >= 3:
            dt, dr = O.pose_error(poses[k + 1].reshape(4, 4), opose[k + 1])
            worst_t, worst_r = max(worst_t, dt), max(worst_r, dr)
    assert worst_t <= TOL_T and worst_r <= TOL_R, (worst_t, worst_r)
    return r


@pytest.mark.parametrize("seed", [0, 1, 2])
def test_icp_config0_per_iteration_parity(ctx, rtr, seed):
    src, tgt, T = rtr.config0_pair(seed)
    r = _replay_check(ctx, src, tgt, 50, 0.05)
    assert r["iterations"] == 50 and r["converged"] == 1
    dt, dr = O.pose_error(r["pose"], T)
    assert dt < 2e-3 and dr < np.deg2rad(0.5)


def test_icp_matches_full_oracle_run(ctx, rtr):
    src, tgt, _ = rtr.config0_pair(4, 8000)
    res, _, _ = ctx.icp(_dev(src), _dev(tgt), 30, 0.05)
    g = ctx.parse_icp_result(res)
    o = O.icp(src, tgt, 30, 0.05)
    dt, dr = O.pose_error(g["pose"], o["pose"])
    assert dt < 1e-4 and dr < 1e-4
    assert abs(g["n_corr"] - o["n_corr"]) <= 2


def test_icp_known_answer_pairs(ctx, golden):
    E = np.eye(4)
    E[:3, 3] = golden["t5"]
    r = _replay_check(ctx, golden["p5"], golden["mcloud"], 50, 0.0)
    dt, dr = O.pose_error(r["pose"], E)
    assert dt < 1e-5 and dr < 1e-5
    a, b = golden["p70761"], golden["p70761_c"]
    init = np.eye(4)
    init[:3, 3] = b[:, :3].astype(np.float64).mean(0) - a[:, :3].astype(np.float64).mean(0) + 0.01
    E[:3, 3] = golden["t70761"]
    r = _replay_check(ctx, a, b, 30, 0.0, init=init)
    dt, dr = O.pose_error(r["pose"], E)
    assert dt < 1e-5 and dr < 1e-5


def test_icp_host_entry_point(ctx, rtr):
    src, tgt, T = rtr.config0_pair(6, 5000)
    r = ctx.icp_host(src, tgt, 40, 0.05)
    assert r["status"] == 0 and r["iterations"] == 40
    dt, dr = O.pose_error(r["pose"], T)
    assert dt < 3e-3 and dr < np.deg2rad(0.5)


def test_icp_too_few_correspondences_keeps_pose(ctx, rtr):
    src, _, _ = rtr.config0_pair(7, 2000)
    far = src.copy()
    far[:, 0] += 10.0  # 10 m away: nothing within 5 cm
    res, _, _ = ctx.icp(_dev(src), _dev(far), 20, 0.05)
    r = ctx.parse_icp_result(res)
    assert r["converged"] == 0 and r["iterations"] == 1 and r["n_corr"] == 0
    assert np.array_equal(r["pose"], np.eye(4))
    assert np.all(np.isfinite(r["pose"]))


def test_icp_early_stop_criteria(ctx, rtr):
    src, tgt, _ = rtr.config0_pair(8, 5000)
    # stop once an update moves the source by less than 1e-6 m (|dt|^2 < 1e-12)
    res, _, _ = ctx.icp(_dev(src), _dev(tgt), 200, 0.05, transformation_epsilon=1e-12)
    r = ctx.parse_icp_result(res)
    assert 1 <= r["iterations"] < 200
    o = O.icp(src, tgt, 200, 0.05, eps_t=1e-12)
    assert abs(o["iterations"] - r["iterations"]) <= 2
    dt, dr = O.pose_error(r["pose"], o["pose"])
    assert dt < 1e-4 and dr < 1e-4


@pytest.mark.parametrize("seed", [0, 3])
def test_icp_near_cell_search_same_correspondences(ctx, rtr, seed):
    """With a grid cell wider than the correspondence distance, every match
    lies in the 27 cells around a query and the kernel takes the shorter
    search (no rings).  Its correspondences are those of the ring search and
    of the oracle, iteration by iteration."""
    src, tgt, _ = rtr.config0_pair(seed)
    for d in (0.02, 0.05):
        ring, tp_r, tc_r = ctx.icp(_dev(src), _dev(tgt), 20, d, trace=True)
        near, tp_n, tc_n = ctx.icp(_dev(src), _dev(tgt), 20, d, cell_size=1.5 * d, trace=True)
        assert np.array_equal(tc_r.cpu().numpy(), tc_n.cpu().numpy())
        # the source is sorted by target cell, so another cell size changes the
        # order of the compensated sums: poses agree to rounding
        np.testing.assert_allclose(tp_r.cpu().numpy(), tp_n.cpu().numpy(), rtol=0, atol=1e-9)
        r = ctx.parse_icp_result(near)
        poses = tp_n.cpu().numpy()[: r["iterations"] + 1]
        ocorr, _, _ = O.icp_replay(src, tgt, d, poses)
        corr = tc_n.cpu().numpy()[: r["iterations"]]
        for k in range(r["iterations"]):
            assert np.array_equal(corr[k], ocorr[k]), k


def test_icp_multi_equals_oracle_refinement(ctx, rtr):
    """rtr_icp_multi: independent problems from several initial poses over one
    target grid, against the oracle's multi-problem ICP (the recognition's
    refinement) and against one-problem runs of the same kernel."""
    src, tgt, T = rtr.config0_pair(5, 6000)
    inits = []
    for k in range(6):
        E = np.eye(4)
        E[:3, 3] = T[:3, 3] + np.float64(0.01) * np.array([k % 3 - 1, (k // 3) - 0.5, 0.2 * k])
        E[:3, :3] = T[:3, :3]
        inits.append(E)
    inits = np.array(inits)
    got = ctx.icp_multi(_dev(src), _dev(tgt), inits, 30, 0.02, cell_size=0.03)
    g = O.Grid(tgt, 0.03)
    ref = g.icp_multi(src, 30, 0.02, inits)
    g.close()
    for a, b in zip(got, ref):
        assert a["status"] == 0 and a["iterations"] == 30
        dt, dr = O.pose_error(a["pose"], b["pose"])
        assert dt < 1e-5 and dr < 1e-5, (dt, dr)
        assert abs(a["n_corr"] - b["n_corr"]) <= 2


def test_pose_inliers_equals_oracle(ctx, rtr):
    """rtr_pose_inliers: per pose, the model points within r of a scene point,
    as the oracle's grid counts them."""
    src, tgt, T = rtr.config0_pair(6, 5000)
    poses = np.array([T, np.eye(4), T @ np.diag([1.0, 1.0, 1.0, 1.0])])
    poses[2][:3, 3] += 0.015
    import torch
    for r in (0.005, 0.02):
        cnt = ctx.pose_inliers(_dev(src), _dev(tgt), torch.from_numpy(poses), r).cpu().numpy()
        g = O.Grid(tgt, 1.5 * r)
        frac = g.inlier_fraction(src, 1, poses.reshape(-1, 16), r)
        g.close()
        assert np.array_equal(cnt, np.rint(frac * src.shape[0]).astype(np.int32)), (cnt, frac)


@pytest.mark.parametrize("n_src,n_tgt,max_dist,cell,shift", [
    (7, 50, 0.05, 0.0, 0.0),        # few points: most blocks idle
    (4099, 3001, 0.02, 0.03, 0.03),  # most points without a neighbour at first
    (4099, 3001, 0.3, 0.0, 0.1),    # a bound far beyond the neighbours' distance
    (2500, 2500, 0.0, 0.0, 0.0),    # no bound
    (2500, 2500, 0.0, 0.0, 40.0),   # no bound, and the clouds far apart
    (5000, 5000, 0.05, 0.004, 0.02),  # boxes of many cells
])
def test_icp_kept_neighbours_equal_a_search_from_scratch(ctx, rtr, n_src, n_tgt, max_dist, cell, shift):
    """Every iteration's correspondences, whether the point was searched or
    its last answer kept, equal the oracle's search; two points of the source
    and one of the target are not finite."""
    src, tgt, _ = rtr.config0_pair(n_src, max(n_src, n_tgt))
    src, tgt = src[:n_src].copy(), tgt[:n_tgt].copy()
    src[:, 0] += np.float32(shift)
    if n_src > 100:
        src[5, 1], src[17, 2], tgt[9, 0] = np.nan, np.inf, np.nan
    import torch
    res, tp, tc = ctx.icp(_dev(src), _dev(tgt), 25, max_dist, cell_size=cell, trace=True)
    r = ctx.parse_icp_result(res)
    n_it = r["iterations"]
    poses, corr = tp.cpu().numpy(), tc.cpu().numpy()
    for k in range(n_it):
        q = O.transform_f32(poses[k].reshape(4, 4), src)
        ri, _ = O.nn1(q, tgt, max_dist, "brute")
        assert np.array_equal(corr[k], ri), k


def test_icp_many_problems_share_a_block_each(ctx, rtr):
    """More points per block than one chunk of the matching (2,048): 300
    problems on the GPU's blocks give what one problem alone gives."""
    src, tgt, T = rtr.config0_pair(8, 9001)
    inits = np.array([T, np.eye(4), T])
    inits[2][:3, 3] += 0.01
    alone = [ctx.parse_icp_result(ctx.icp(_dev(src), _dev(tgt), 12, 0.03, init=i, cell_size=0.02)[0]) for i in inits]
    many = ctx.icp_multi(_dev(src), _dev(tgt), inits[np.arange(300) % 3], 12, 0.03, cell_size=0.02)
    for k, m in enumerate(many):
        a = alone[k % 3]
        assert m["status"] == 0 and m["n_corr"] == a["n_corr"]
        np.testing.assert_allclose(m["pose"], a["pose"], rtol=0, atol=1e-9)


def test_recognition_refines_alike_without_room_for_the_matching_state(rtr):
    """A scene of a few points and a large model: the recognition's scratch
    need not hold the refinement's matching state, which then searches every
    point in every iteration.  Same instances and poses as with a larger
    arena."""
    prm = rtr.recog_default_params(scene_outward=1)
    model = rtr.synth_shape(rtr.SOFA, 60000, 3)
    scene = rtr.synth_transform_noise(rtr.synth_shape(rtr.SOFA, 2000, 4), rtr.synth_rigid(5, 20.0, 0.2), 0.002, 6)
    out = []
    for reserve in (0, 1 << 30):
        c = rtr.Context(0)
        m = rtr.Model(c, _dev(model), prm)
        if reserve:
            c.reserve(reserve)
        out.append(rtr.parse_recog_result(rtr.recognize(c, m, _dev(scene), prm)))
        c.check()
        m.close()
        c.close()
    a, b = out
    assert a["n_clusters"] == b["n_clusters"] and len(a["instances"]) == len(b["instances"])
    for x, y in zip(a["instances"], b["instances"]):
        assert x["hypothesis"] == y["hypothesis"] and x["score"] == y["score"]
        np.testing.assert_allclose(x["pose"], y["pose"], rtol=0, atol=1e-9)


@pytest.mark.parametrize("n_src,group", [(3, 0), (31, 0), (33, 8), (257, 2), (20000, 4), (20001, 0), (60007, 0),
                                         (90011, 0), (700001, 0)])
def test_icp_sums_keep_every_point_once(ctx, rtr, n_src, group):
    """The sums' lanes (8, 4 or 2 a point, by the points a block has or by the
    tuning), ragged last passes and blocks of more than one chunk (2,048
    points): the first pose equals the FP64 solve of the same FP32 terms to
    1e-12 (compensated sums hold 2^-45 of the terms' magnitudes, the
    covariance's condition is below 100)."""
    src, tgt, _ = rtr.config0_pair(n_src, 20000)
    rng = np.random.default_rng(n_src)
    src = src[rng.integers(0, src.shape[0], n_src)].copy()
    src[:, :3] += rng.normal(0, 0.01, (n_src, 3)).astype(np.float32)
    ctx.set_tuning("icp_group", group)
    try:
        res, tp, tc = ctx.icp(_dev(src), _dev(tgt), 1, 0.0, trace=True)
        r = ctx.parse_icp_result(res)
    finally:
        ctx.set_tuning("icp_group", 0)
    assert r["status"] == 0 and r["n_corr"] == n_src
    q = tgt[tc.cpu().numpy()[0], :3]
    half = np.float32(0.5)
    cp = half * (src[:, :3].min(0) + src[:, :3].max(0))
    cq = half * (tgt[:, :3].min(0) + tgt[:, :3].max(0))
    dp, dq = src[:, :3] - cp, q - cq
    prod = (dp[:, :, None] * dq[:, None, :]).astype(np.float64)
    mp, mq = dp.astype(np.float64).mean(0), dq.astype(np.float64).mean(0)
    U, _, Vt = np.linalg.svd(prod.sum(0) - n_src * np.outer(mp, mq))
    R = Vt.T @ np.diag([1.0, 1.0, np.sign(np.linalg.det(U @ Vt))]) @ U.T
    want = np.eye(4)
    want[:3, :3] = R
    want[:3, 3] = (mq + cq) - R @ (mp + cp)
    tol = 1e-12 if n_src > 100 else 1e-9  # a few points: worse conditioned
    np.testing.assert_allclose(tp.cpu().numpy()[1].reshape(4, 4), want, rtol=0, atol=tol)


def test_icp_without_its_matching_state(rtr):
    """Under a scratch limit that leaves no room for the matching state of a
    large source (8 MB), every point is searched in every iteration: the same
    correspondences, poses and result, bit for bit."""
    src, tgt, _ = rtr.config0_pair(4, 400000)
    tgt = tgt[:3000].copy()
    out = []
    for mb in (0, 19):
        c = rtr.Context(0)
        try:
            c.set_tuning("scratch_limit_mb", mb)
            res, tp, tc = c.icp(_dev(src), _dev(tgt), 12, 0.05, trace=True)
            out.append((c.parse_icp_result(res), tp.cpu().numpy(), tc.cpu().numpy(), c.scratch_bytes()))
        finally:
            c.close()
    (ra, pa, ca, na), (rb, pb, cb, nb) = out
    assert na >= nb + 4000000 and nb <= 19 << 20  # with the state, and without it
    assert ra["n_corr"] == rb["n_corr"] and ra["iterations"] == rb["iterations"] == 12
    assert np.array_equal(pa, pb) and np.array_equal(ca, cb)


def test_icp_multi_with_the_state_of_some_problems(rtr):
    """64 problems of 20,000 points under a limit that holds the matching state
    of a few: the same results as with all of it, bit for bit."""
    src, tgt, _ = rtr.config0_pair(5, 20000)
    inits = np.repeat(np.eye(4)[None], 64, 0)
    inits[:, 0, 3] = np.linspace(-0.02, 0.02, 64)
    out = []
    for mb in (0, 5):
        c = rtr.Context(0)
        try:
            c.set_tuning("scratch_limit_mb", mb)
            out.append((c.icp_multi(_dev(src), _dev(tgt), inits, 12, 0.05), c.scratch_bytes()))
        finally:
            c.close()
    (a, na), (b, nb) = out
    assert na >= 64 * 20000 * 20 and nb <= 5 << 20
    for x, y in zip(a, b):
        assert np.array_equal(x["pose"], y["pose"]) and x["n_corr"] == y["n_corr"] and x["fitness"] == y["fitness"]


def test_icp_multi_bounds_its_scratch_and_leaves_batch_graphs_alone(rtr):
    """The matching state is asked for up to a gigabyte (300 problems of 300,000
    points would take 1.8); and not at all while a batch graph holds the arena's
    address and the call can do without: the graph stays good."""
    src, tgt, _ = rtr.config0_pair(3, 300000)
    tgt = tgt[:3000].copy()
    inits = np.repeat(np.eye(4)[None], 300, 0)
    c = rtr.Context(0)
    try:
        r = c.icp_multi(_dev(src), _dev(tgt), inits, 1, 0.05)
        assert len(r) == 300 and all(x["status"] == 0 and x["n_corr"] == r[0]["n_corr"] for x in r)
        assert c.scratch_bytes() < 1500000000
    finally:
        c.close()
    prm = rtr.recog_default_params(scene_outward=1)
    c = rtr.Context(0)
    try:
        m = rtr.Model(c, _dev(rtr.synth_shape(rtr.CHAIR, 20000, 3)), prm)
        scene = rtr.synth_transform_noise(rtr.synth_shape(rtr.CHAIR, 6000, 4), rtr.synth_rigid(5, 20.0, 0.2), 0.002, 6)
        scenes = [_dev(scene), _dev(scene)]
        ref = [rtr.parse_recog_result(x) for x in rtr.recognize_batch(c, [m, m], scenes, prm)]
        g = rtr.BatchGraph(c, [m, m], scenes, prm)
        held = c.scratch_bytes()
        n = 2 * held // (64 * 20) + 1000  # points whose state the arena cannot hold
        big = np.repeat(src, -(-n // src.shape[0]), 0)[:n]
        assert len(c.icp_multi(_dev(big), _dev(tgt), inits[:64], 2, 0.05)) == 64
        assert c.scratch_bytes() == held
        got = [rtr.parse_recog_result(x) for x in g.launch()]
        assert [len(x["instances"]) for x in got] == [len(x["instances"]) for x in ref]
        g.close()
        m.close()
    finally:
        c.close()


@pytest.mark.parametrize("group", [2, 4])
@pytest.mark.parametrize("n_tgt,max_dist,cell,shift", [
    (6000, 0.3, 0.06, 0.1),    # boxes of many rows over cells of some 30 points
    (6000, 0.3, 0.2, 0.15),    # hundreds of points a cell
    (6000, 0.0, 0.1, 0.3),     # no bound
    (3000, 0.05, 0.3, 0.02),   # everything in a few cells
])
def test_icp_in_dense_cells_equals_a_search_from_scratch(ctx, rtr, group, n_tgt, max_dist, cell, shift):
    """Targets with many points a cell, whose larger boxes are walked from the
    query outwards and cut by what has been seen: every iteration's
    correspondences equal the oracle's search.  Duplicates tie to the lowest
    index, and one point is not finite."""
    src, tgt, _ = rtr.config0_pair(6, 8000)
    src, tgt = src[:3001].copy(), tgt[:n_tgt].copy()
    src[:, 0] += np.float32(shift)
    tgt[100:140] = tgt[:40]
    tgt[9, 0] = np.nan
    ctx.set_tuning("icp_group", group)
    try:
        res, tp, tc = ctx.icp(_dev(src), _dev(tgt), 15, max_dist, cell_size=cell, trace=True)
        n_it = ctx.parse_icp_result(res)["iterations"]
    finally:
        ctx.set_tuning("icp_group", 0)
    poses, corr = tp.cpu().numpy(), tc.cpu().numpy()
    for k in range(n_it):
        ri, _ = O.nn1(O.transform_f32(poses[k].reshape(4, 4), src), tgt, max_dist, "brute")
        assert np.array_equal(corr[k], ri), k


def test_icp_of_dense_clouds_costs_what_its_neighbours_do(ctx, rtr):
    """Two iterations of two 400,000-point chairs: a bound of 5 cells may cost
    up to three times one of 2 (6.0 with every box scanned whole, 1.8 walked
    outwards)."""
    import torch
    src, tgt, _ = rtr.config0_pair(4, 400000)
    s, t = _dev(src), _dev(tgt)

    def time(max_dist):
        best = float("inf")
        for k in range(6):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            ctx.icp(s, t, 2, max_dist, cell_size=0.01)
            b.record()
            b.synchronize()
            best = min(best, a.elapsed_time(b)) if k else best
        return best
    assert time(0.05) < 3.0 * time(0.02)
