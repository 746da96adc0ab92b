"""GPU parity: exact 1-NN / k-NN through the C ABI vs the CPU oracle.
Indices and squared distances must be bit-exact (ties -> lowest index)."""
import numpy as np
import pytest

import oracle as O

from pathlib import Path

GOLDEN = Path(__file__).resolve().parent / "golden"

pytestmark = pytest.mark.gpu


def _dev(a):
    import torch
    return torch.from_numpy(np.ascontiguousarray(a, np.float32)).cuda()


def _rand(rng, n, scale=1.0):
    p = np.zeros((n, 4), np.float32)
    p[:, :3] = rng.uniform(-scale, scale, (n, 3))
    return p


@pytest.mark.parametrize("max_dist", [0.0, 0.01, 0.05, 0.3])
def test_knn1_bit_exact_random(ctx, max_dist):
    rng = np.random.default_rng(10)
    t = _rand(rng, 20000, 0.5)
    q = _rand(rng, 15000, 0.6)
    idx, d2 = ctx.knn1(_dev(q), _dev(t), max_dist)
    ri, rd = O.nn1(q, t, max_dist, "brute")
    assert np.array_equal(idx.cpu().numpy(), ri)
    got = d2.cpu().numpy()
    ok = ri >= 0
    assert np.array_equal(got[ok], rd[ok]) and np.all(np.isinf(got[~ok]))


def test_knn1_ties_go_to_lowest_index(ctx):
    rng = np.random.default_rng(11)
    t = _rand(rng, 2000)
    t[1000:1100] = t[7]       # 101 copies of point 7
    t[1500] = t[1200]          # a later duplicate
    q = np.concatenate([t[[7, 1050, 1200, 1500]], _rand(rng, 100)])
    idx, _ = ctx.knn1(_dev(q), _dev(t), 0.0)
    idx = idx.cpu().numpy()
    assert list(idx[:4]) == [7, 7, 1200, 1200]
    ri, _ = O.nn1(q, t, 0.0, "brute")
    assert np.array_equal(idx, ri)


def test_knn1_surface_clouds_config0(ctx, rtr):
    src, tgt, T = rtr.config0_pair(5)
    q = O.transform_f32(T, src)
    for md in (0.05, 0.0):
        idx, d2 = ctx.knn1(_dev(q), _dev(tgt), md)
        ri, rd = O.nn1(q, tgt, md, "grid")
        assert np.array_equal(idx.cpu().numpy(), ri)


def test_knn1_edge_cases(ctx):
    rng = np.random.default_rng(12)
    t = _rand(rng, 1)
    q = _rand(rng, 50, 10.0)  # far outside a one-point grid
    idx, _ = ctx.knn1(_dev(q), _dev(t), 0.0)
    assert np.all(idx.cpu().numpy() == 0)
    idx, _ = ctx.knn1(_dev(q), _dev(t), 0.001)
    ri, _ = O.nn1(q, t, 0.001, "brute")
    assert np.array_equal(idx.cpu().numpy(), ri)
    # empty target: every index is -1
    import torch
    e = torch.zeros((0, 4), dtype=torch.float32, device="cuda")
    idx, _ = ctx.knn1(_dev(q), e, 0.0)
    assert np.all(idx.cpu().numpy() == -1)
    # all points identical (one cell, every distance ties)
    t = np.zeros((3000, 4), np.float32)
    idx, d2 = ctx.knn1(_dev(q[:10]), _dev(t), 0.0)
    assert np.all(idx.cpu().numpy() == 0)


@pytest.mark.parametrize("k", [1, 10, 16, 32])
def test_knn_bit_exact(ctx, k):
    rng = np.random.default_rng(13)
    t = _rand(rng, 6000, 0.5)
    t[100:120] = t[5]
    q = np.concatenate([_rand(rng, 3000, 0.55), t[[5, 110]]])
    idx, d2 = ctx.knn(_dev(q), _dev(t), k)
    ri, rd = O.knn(q, t, k)
    assert np.array_equal(idx.cpu().numpy(), ri)
    assert np.array_equal(d2.cpu().numpy(), rd)


@pytest.mark.parametrize("box", [False, True])
def test_range_search_equals_oracle(ctx, box):
    """rtr_radius_search / rtr_box_search against the oracle's brute force:
    the same indices in the same (ascending) order and the same counts, with
    cuts at max_per_query, non-finite points and an empty target set."""
    import torch
    rng = np.random.default_rng(5 + box)
    q = rng.uniform(-1, 1, (3000, 4)).astype(np.float32)
    t = rng.uniform(-1, 1, (50000, 4)).astype(np.float32)
    q[[5, 77], 0] = np.nan
    t[[3, 999], 1] = np.inf
    dq, dt = torch.from_numpy(q).cuda(), torch.from_numpy(t).cuda()
    for r, m in ((0.05, 64), (0.12, 16), (0.3, 0), (3.0, 8)):
        idx, cnt = ctx.radius_search(dq, dt, r, m, box=box)
        oidx, ocnt = O.range_search(q, t, r, box, m)
        assert np.array_equal(cnt.cpu().numpy(), ocnt)
        assert np.array_equal(idx.cpu().numpy(), oidx)
    e = torch.zeros((0, 4), dtype=torch.float32, device="cuda")
    idx, cnt = ctx.radius_search(dq, e, 0.1, 4, box=box)
    assert int(cnt.sum()) == 0 and bool((idx == -1).all())


def test_box_search_at_keypoints_of_main_scan(ctx):
    """The reference's use: the +-10 cm box around each keypoint of the scan
    main registers (KeyPoint::getOccupiedGrid, key_point.h:118-140)."""
    import torch
    d = np.load(GOLDEN / "main_clouds.npz")
    scan = np.ascontiguousarray(d["T0_m8111"], np.float32)
    keys = scan[O.uniform_sample(scan, 0.05)]
    idx, cnt = ctx.radius_search(torch.from_numpy(keys).cuda(), torch.from_numpy(scan).cuda(), 0.1, 4096, box=True)
    oidx, ocnt = O.range_search(keys, scan, 0.1, True, 4096)
    assert np.array_equal(cnt.cpu().numpy(), ocnt) and ocnt.max() < 4096
    assert np.array_equal(idx.cpu().numpy(), oidx)


@pytest.mark.parametrize("kind", ["one_cell", "one_point", "line", "clusters"])
def test_grid_counted_into_place_on_uneven_clouds(ctx, kind):
    """Cells holding the whole cloud, duplicates, a degenerate box and a few
    dense clusters, with points that are not finite: 1-NN and k-NN as brute
    force finds them."""
    rng = np.random.default_rng(3)
    n = 5003
    t = _rand(rng, n, 0.001)
    if kind == "one_point":
        t[:, :3] = 0.25
    elif kind == "line":
        t[:, 1:3] = 0.5
    elif kind == "clusters":
        t[:, :3] += rng.integers(0, 3, (n, 1)).astype(np.float32) * 5
    t[11, 0], t[12, 1] = np.nan, np.inf
    q = np.concatenate([t[:400] + np.float32(1e-4), _rand(rng, 300, 1.0)])
    q[:, 3] = 0
    for md in (0.0, 0.004, 2.0):
        idx, _ = ctx.knn1(_dev(q), _dev(t), md)
        ri, _ = O.nn1(q, t, md, "brute")
        assert np.array_equal(idx.cpu().numpy(), ri), md
    ki, _ = ctx.knn(_dev(q[:50]), _dev(t), 8)
    first = O.nn1(q[:50], t, 0.0, "brute")[0]
    assert np.array_equal(ki.cpu().numpy()[:, 0], first)


@pytest.mark.parametrize("k", [1, 5, 8, 16, 32])
def test_knn_in_dense_cells_equals_brute_force(ctx, k):
    """Clouds whose automatic cells hold dozens of points, lattices (ties) and
    single points: every entry by (FP32 distance, index)."""
    rng = np.random.default_rng(k)
    n = 4000
    t = _rand(rng, n, 1.0)
    t[:2000, :3] = t[:2000, :3] * 0.02
    t[2000:3000, :3] = np.float32(0.25) + np.float32(0.015625) * rng.integers(0, 8, (1000, 3)).astype(np.float32)
    t[11, 0], t[12, 1] = np.nan, np.inf
    q = np.concatenate([t[:300], t[2000:2300] + np.float32(0.0078125), t[3000:3200], _rand(rng, 50, 3.0)])
    q = q[np.isfinite(q[:, :3]).all(1)].copy()
    q[:, 3] = 0
    idx, d2 = ctx.knn(_dev(q), _dev(t), k)
    with np.errstate(all="ignore"):
        d = q[:, None, :3] - t[None, :, :3]
        d = d * d
        ref = (d[..., 0] + d[..., 1]) + d[..., 2]
    ref = np.where(np.isfinite(ref), ref, np.float32(np.inf))
    o = np.argsort(ref, axis=1, kind="stable")[:, :k]
    assert np.array_equal(idx.cpu().numpy(), o)
    assert np.array_equal(d2.cpu().numpy(), np.take_along_axis(ref, o, 1))


def test_pose_inliers_cost_follows_the_hits_not_the_cells(ctx):
    """A wall of a million points: with a radius of 10 cm a cell holds
    thousands, and every query has a hit in its own; no more than 2.5 times the
    2 cm count (5 with the box's corner first, 1.5 with the own cell first)."""
    import torch
    rng = np.random.default_rng(1)
    w = np.zeros((1000000, 4), np.float32)
    w[:, :2] = rng.uniform(0, 4, (1000000, 2))
    w[:, 2] = rng.uniform(0, 0.004, 1000000)
    scene, model = _dev(w), _dev(w[::50])
    poses = np.repeat(np.eye(4)[None], 8, 0)
    poses[:, 0, 3] = np.linspace(0, 0.05, 8)

    def time(radius):
        best = float("inf")
        for k in range(8):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            ctx.pose_inliers(model, scene, poses, radius)
            b.record()
            b.synchronize()
            best = min(best, a.elapsed_time(b)) if k else best
        return best
    assert time(0.1) < 2.5 * time(0.02)
