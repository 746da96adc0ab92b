"""The reference's own descriptor route on the GPU (rtr_ref_*: getOccupiedGrid,
get_TSDF, get_Distance, the gated all-pairs loop, Ransac) against the CPU
oracle (oracle/refmatch.c), bit for bit: integer outputs equal, float scores
and transforms equal, NaN where the oracle has NaN."""
from pathlib import Path

import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu
GOLDEN = Path(__file__).resolve().parent / "golden"


def _dev(a):
    import torch
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def _route(ctx, model, scan, km, ks):
    """Every stage on the GPU and in the oracle; asserts equality, returns
    the oracle's (scores, transforms)."""
    dm, ds, dkm, dks = _dev(model), _dev(scan), _dev(km), _dev(ks)
    mn, mo, mi = ctx.ref_occupancy(dm, dkm)
    sn, so, si = ctx.ref_occupancy(ds, dks)
    rmn, rmo, rmi = O.ref_occupancy(model, km)
    rsn, rso, rsi = O.ref_occupancy(scan, ks)
    assert np.array_equal(mn.cpu().numpy(), rmn) and np.array_equal(mo.cpu().numpy(), rmo)
    assert np.array_equal(mi.cpu().numpy(), rmi)
    assert np.array_equal(sn.cpu().numpy(), rsn) and np.array_equal(so.cpu().numpy(), rso)
    assert np.array_equal(si.cpu().numpy(), rsi)
    tdf = ctx.ref_tdf(dm, dkm, mo, mi)
    rtdf = O.ref_tdf(model, km, rmo, rmi)
    assert np.array_equal(tdf.cpu().numpy(), rtdf)
    sc, T = ctx.ref_distance(dm, dkm, mo, mi, tdf, dks)
    rsc, rT = O.ref_distance(model, km, rmo, rmi, rtdf, ks)
    g = sc.cpu().numpy()
    assert np.array_equal(np.isnan(g), np.isnan(rsc))
    ok = ~np.isnan(rsc)
    bad = np.nonzero(g[ok] != rsc[ok])[0]
    assert bad.size == 0, (bad[:5], g[ok][bad[:5]], rsc[ok][bad[:5]])
    assert np.array_equal(T.cpu().numpy(), rT, equal_nan=True)
    pi = ctx.ref_correspond(dkm, mn, dks, sn, sc)
    rpi = O.ref_correspond(km, rmn, ks, rsn, rsc)
    assert np.array_equal(pi.cpu().numpy(), rpi)
    if rpi.size:
        Tb, inl, best = ctx.ref_ransac(dkm, dks, pi, sc, T)
        rTb, rinl, rbest = O.ref_ransac(km, ks, rpi, rsc, rT)
        assert (inl, best) == (rinl, rbest) and np.array_equal(Tb, rTb)
    return rsc, rT, rpi


def test_route_on_the_reference_clouds(ctx):
    """main's inputs (chair1.pcd model, T0_m8111.pcd scan), keypoints every
    5 cm: 340 x 573 pairs, every stage equal to the oracle."""
    d = np.load(GOLDEN / "main_clouds.npz")
    model, scan = d["chair1"], d["T0_m8111"]
    km = model[O.uniform_sample(model, 0.05)]
    ks = scan[O.uniform_sample(scan, 0.05)]
    sc, _, pi = _route(ctx, model, scan, km, ks)
    assert np.isfinite(sc).all() and pi.size > 0


def test_route_on_a_synthetic_chair(ctx, rtr):
    """A 20k-point chair (occupancy clouds of up to ~2.5k points: the
    512-thread pair kernel) against a cropped, turned copy."""
    model = rtr.synth_shape(rtr.CHAIR, 20000, 2024)
    th = np.radians(20.0)
    T = np.eye(4)
    T[:3, :3] = [[np.cos(th), -np.sin(th), 0], [np.sin(th), np.cos(th), 0], [0, 0, 1]]
    T[:3, 3] = [0.05, -0.03, 0.0]
    scan = rtr.synth_transform_noise(rtr.synth_crop(rtr.synth_shape(rtr.CHAIR, 20000, 501), 0.3, 1), T, 0.002, 10)
    km = model[O.uniform_sample(model, 0.1)]
    ks = scan[O.uniform_sample(scan, 0.1)]
    _route(ctx, model, scan, km, ks)


def test_dense_occupancy_and_explicit_pairs(ctx, rtr):
    """60k points on the chair: occupancy clouds above 4096 points (the
    1024-thread pair kernel), the index buffer regrown past its first
    capacity; explicit pair lists equal the all-pairs result."""
    model = rtr.synth_shape(rtr.CHAIR, 60000, 11)
    scan = rtr.synth_shape(rtr.CHAIR, 30000, 12)
    rng = np.random.default_rng(5)
    km = model[rng.choice(model.shape[0], 24, replace=False)]
    ks = scan[rng.choice(scan.shape[0], 5, replace=False)]
    dm, dkm, dks = _dev(model), _dev(km), _dev(ks)
    mn, mo, mi = ctx.ref_occupancy(dm, dkm)
    rmn, rmo, rmi = O.ref_occupancy(model, km)
    assert np.array_equal(mo.cpu().numpy(), rmo) and np.array_equal(mi.cpu().numpy(), rmi)
    assert np.diff(rmo).max() > 4096 and rmo[-1] > (1 << 16)
    tdf = ctx.ref_tdf(dm, dkm, mo, mi)
    rtdf = O.ref_tdf(model, km, rmo, rmi)
    assert np.array_equal(tdf.cpu().numpy(), rtdf)
    pm = np.array([20, 5, 13, 13, 7, 2], np.int32)  # 20: the largest occupancy cloud (5,589 points)
    ps = np.array([4, 0, 2, 1, 1, 3], np.int32)
    sc, T = ctx.ref_distance(dm, dkm, mo, mi, tdf, dks, _dev(pm), _dev(ps))
    rsc, rT = O.ref_distance(model, km, rmo, rmi, rtdf, ks, pm, ps)
    assert np.array_equal(sc.cpu().numpy(), rsc) and np.array_equal(T.cpu().numpy(), rT)


def test_edge_cases(ctx, rtr):
    """A keypoint with an empty box (Number 0, field all 900, score 0 as in
    the reference), a non-finite scan keypoint (NaN, identity), a scan
    keypoint 40 m away (the octree grows 8 levels)."""
    model = rtr.synth_shape(rtr.CHAIR, 4000, 3)
    km = np.concatenate([model[:3], np.array([[30.0, 30.0, 30.0, 0.0]], np.float32)])
    ks = np.array([[0.1, 0.2, 0.4, 0], [np.nan, 0.0, 0.3, 0], [40.0, -3.0, 1.0, 0], [0.0, 0.0, 0.0, 0]],
                  np.float32)
    dm, dkm, dks = _dev(model), _dev(km), _dev(ks)
    mn, mo, mi = ctx.ref_occupancy(dm, dkm)
    assert mn.cpu().numpy()[3] == 0
    tdf = ctx.ref_tdf(dm, dkm, mo, mi)
    assert np.all(tdf.cpu().numpy()[3] == 900.0)
    sc, T = ctx.ref_distance(dm, dkm, mo, mi, tdf, dks)
    rmn, rmo, rmi = O.ref_occupancy(model, km)
    rsc, rT = O.ref_distance(model, km, rmo, rmi, O.ref_tdf(model, km, rmo, rmi), ks)
    g = sc.cpu().numpy()
    assert np.array_equal(np.isnan(g), np.isnan(rsc)) and np.isnan(g[1::4]).all()
    assert np.array_equal(g[~np.isnan(g)], rsc[~np.isnan(rsc)])
    # the scan keypoint at z = 0 scales by kz / 0: inf and NaN entries, equal too
    assert np.array_equal(T.cpu().numpy(), rT, equal_nan=True)
    assert np.array_equal(T.cpu().numpy()[1], np.eye(4, dtype=np.float32))


def test_bad_arguments_are_refused(ctx, rtr):
    model = _dev(rtr.synth_shape(rtr.CHAIR, 2000, 3))
    keys = model[:4].contiguous()
    with pytest.raises(rtr.RtrError):
        ctx.ref_occupancy(model, keys, 0.01, 0.5)  # 100 leaves across: beyond the 32^3 bitmap
    _, mo, mi = ctx.ref_occupancy(model, keys)
    with pytest.raises(rtr.RtrError):
        ctx.ref_tdf(model, keys, mo, mi, 0.01, 0.2)  # dim 40 > 30
    tdf = ctx.ref_tdf(model, keys, mo, mi)
    import torch
    bad_m = torch.tensor([0, 7], dtype=torch.int32, device="cuda")
    bad_s = torch.tensor([0, 0], dtype=torch.int32, device="cuda")
    with pytest.raises(rtr.RtrError):
        ctx.ref_distance(model, keys, mo, mi, tdf, keys, bad_m, bad_s)  # model index 7 of 4
    ctx.check()


@pytest.mark.parametrize("res,half", [(0.01, 0.15), (0.01, 0.1525), (0.004, 0.0601)])
def test_distance_by_cloud_size_and_position(ctx, res, half):
    """get_Distance over the pair kernel's cases, each equal to the oracle:
    clouds at the edges of its size classes (rows of 32 points up to 512,
    beyond that a CTA per pair), points and offsets on whole leaves (keys
    decided exactly), tiny coordinates, field cubes whose leaves do not meet
    the field's voxels in their middles (half 0.1525, 0.0601), scan keypoints
    near, far and beyond the range of the fixed-point form.  Field values are
    random, so the order of the sums shows."""
    rng = np.random.default_rng(int(res * 1e4) + int(half * 1e5))
    sizes = [0, 1, 31, 32, 33, 64, 65, 96, 97, 128, 129, 160, 161, 192, 193, 256, 257, 384, 385, 512, 513, 700]
    box = np.float32(half * 2 / 3 * 0.98)
    keys, clouds = [], []
    for i, n in enumerate(sizes):
        k = np.zeros(4, np.float32) if i % 4 == 1 else np.append(rng.uniform(-1, 1, 3), 0).astype(np.float32)
        c = np.zeros((n, 4), np.float32)
        c[:, :3] = k[:3] + rng.uniform(-box, box, (n, 3)).astype(np.float32)
        if i % 3 == 0 and n:  # whole leaves about the key
            c[:, :3] = k[:3] + (np.float32(res) * rng.integers(-9, 10, (n, 3))).astype(np.float32)
        if i % 4 == 1 and n:
            c[:, :3] *= 10.0 ** rng.uniform(-9, 0, (n, 3)).astype(np.float32)
        keys.append(k)
        clouds.append(c)
    km = np.stack(keys)
    model = np.concatenate(clouds)
    mo = np.concatenate([[0], np.cumsum(sizes)]).astype(np.int32)
    mi = np.arange(model.shape[0], dtype=np.int32)
    tdf = rng.uniform(0, 900, (len(sizes), 27000)).astype(np.float32)
    off = np.array([[0, 0, 0], [3 * res, -2 * res, res], [0.013, 0.002, -0.02], [0.31, -0.2, 0.05], [-7.3, 4.1, 0.6],
                    [0.0, 0.0, 0.2], [400.0, 0.0, 0.0]], np.float32)
    ks = np.zeros((len(off) * 3, 4), np.float32)
    for j, b in enumerate((1, 4, 7)):
        ks[j * len(off):(j + 1) * len(off), :3] = km[b, :3] + off
    rsc, rT = O.ref_distance(model, km, mo, mi, tdf, ks, res=res, half=half)
    args = (_dev(model), _dev(km), _dev(mo), _dev(mi), _dev(tdf), _dev(ks))
    sc, T = ctx.ref_distance(*args, resolution=res, half_tdf=half)
    assert np.array_equal(sc.cpu().numpy(), rsc, equal_nan=True)
    assert np.array_equal(T.cpu().numpy(), rT, equal_nan=True)
    # the same as a pair list, shuffled
    pm, ps = [x.ravel().astype(np.int32) for x in np.meshgrid(np.arange(len(sizes)), np.arange(len(ks)), indexing="ij")]
    o = rng.permutation(pm.size)
    sc, T = ctx.ref_distance(*args, _dev(pm[o]), _dev(ps[o]), resolution=res, half_tdf=half)
    assert np.array_equal(sc.cpu().numpy(), rsc[o], equal_nan=True)
    assert np.array_equal(T.cpu().numpy(), rT[o], equal_nan=True)


def test_distance_without_room_for_its_tables(rtr):
    """8,000 model keypoints under a 1 MiB scratch limit: the tables of the
    warp form do not fit, every pair takes a CTA, same results."""
    rng = np.random.default_rng(2)
    nk = 8000
    km = np.zeros((nk, 4), np.float32)
    km[:, :3] = rng.uniform(-1, 1, (nk, 3))
    cnt = rng.integers(0, 40, nk)
    mo = np.concatenate([[0], np.cumsum(cnt)]).astype(np.int32)
    cloud = np.zeros((mo[-1], 4), np.float32)
    cloud[:, :3] = np.repeat(km[:, :3], cnt, 0) + rng.uniform(-0.1, 0.1, (mo[-1], 3))
    mi = np.arange(mo[-1], dtype=np.int32)
    tdf = rng.uniform(0, 900, (nk, 27000)).astype(np.float32)
    ks = km[:2] + np.float32(0.05)
    ks[:, 3] = 0
    import torch
    args = (_dev(cloud), _dev(km), _dev(mo), _dev(mi), torch.from_numpy(tdf).cuda(), _dev(ks))
    res = []
    for mb in (0, 1):
        c = rtr.Context(0)
        try:
            c.set_tuning("scratch_limit_mb", mb)
            sc, T = c.ref_distance(*args)
            res.append((sc.cpu().numpy(), T.cpu().numpy()))
        finally:
            c.close()
    assert np.array_equal(res[0][0], res[1][0], equal_nan=True)
    assert np.array_equal(res[0][1], res[1][1], equal_nan=True)


def _unit_case(scale, seed=11):
    """Keypoints up to 1 (metre) of the origin, clouds about them; scaled."""
    rng = np.random.default_rng(seed)
    sizes = [0, 1, 40, 90, 120, 200, 300]
    km = np.zeros((len(sizes), 4), np.float32)
    km[:, :3] = rng.uniform(-1, 1, (len(sizes), 3))
    clouds = []
    for k, n in zip(km, sizes):
        c = np.zeros((n, 4), np.float32)
        c[:, :3] = k[:3] + rng.uniform(-0.1, 0.1, (n, 3))
        c[: n // 3, :3] = k[:3] + 0.01 * rng.integers(-9, 10, (n // 3, 3))
        clouds.append(c)
    ks = np.zeros((12, 4), np.float32)
    ks[:, :3] = rng.uniform(-1, 1, (12, 3))
    ks[:6, :3] = km[1:, :3] + np.float32([0.03, -0.02, 0.01])
    mo = np.concatenate([[0], np.cumsum(sizes)]).astype(np.int32)
    tdf = rng.uniform(0, 900, (len(sizes), 27000)).astype(np.float32)
    sc = np.float32(scale)
    return np.concatenate(clouds) * sc, km * sc, mo, np.arange(mo[-1], dtype=np.int32), tdf, ks * sc


def _launches(ctx, rtr, case, res, half, off=0.0):
    model, km, mo, mi, tdf, ks = case
    model, km, ks = model.copy(), km.copy(), ks.copy()
    for a in (model, km, ks):
        a[:, 0] += np.float32(off)
    ref = O.ref_distance(model, km, mo, mi, tdf, ks, res=res, half=half)
    args = [_dev(x) for x in (model, km, mo, mi, tdf, ks)]
    n0 = rtr.launch_count()
    got = ctx.ref_distance(*args, resolution=res, half_tdf=half)
    n1 = rtr.launch_count()
    for g, r in zip(got, ref):
        assert np.array_equal(g.cpu().numpy(), r, equal_nan=True), (res, off)
    return n1 - n0


@pytest.mark.parametrize("scale", [100.0, 1000.0, 0.001, 1.0e6, 3.7])
def test_distance_in_other_units_takes_the_same_route(ctx, rtr, scale):
    """Clouds in centimetres, millimetres, kilometres and micrometres: the
    pair kernel takes them as it takes metres (no pair left to a CTA of its
    own, which is a launch more), same scores and transforms as the oracle."""
    metres = _launches(ctx, rtr, _unit_case(1.0), 0.01, 0.1525)
    assert _launches(ctx, rtr, _unit_case(scale), 0.01 * scale, 0.1525 * scale) == metres


def test_distance_far_from_the_origin(ctx, rtr):
    """Up to 2^17 leaves from the origin the pair kernel takes every pair;
    beyond, pairs are left to a CTA each; same results as the oracle at both."""
    near = _launches(ctx, rtr, _unit_case(1.0), 0.01, 0.1525)
    for off in (200.0, 1300.0):
        assert _launches(ctx, rtr, _unit_case(1.0), 0.01, 0.1525, off) == near
    assert _launches(ctx, rtr, _unit_case(1.0), 0.01, 0.1525, 1320.0) == near + 1
    assert _launches(ctx, rtr, _unit_case(1.0e6), 1.0e4, 0.1525e6, 3.0e8) == near + 1
