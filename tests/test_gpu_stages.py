"""GPU parity of the recognition stages against the CPU oracle.

Voxel filter, uniform sampling, normals and the outward orientation are
integer/rounding-exact restatements: bit-exact.  SHOT sums its support in
64-bit fixed point (order-free) with the same IEEE operations per term as
the oracle: descriptors and LRFs bit-exact.  The descriptor matcher is
bit-exact (sequential FP32 sums, lowest-index ties)."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


def _dev(a):
    import torch
    return torch.from_numpy(np.ascontiguousarray(a, np.float32)).cuda()


def _host(t):
    return t.cpu().numpy()


@pytest.fixture(scope="module")
def clouds(rtr):
    model = rtr.synth_shape(rtr.CHAIR, 20000, 2024)
    p = rtr.room_default_params()
    p.n_points = 60000
    scene, _, _ = rtr.synth_room(3, p)
    return model, scene


@pytest.mark.parametrize("leaf", [0.01, 0.02, 0.0037])
def test_voxel_downsample_bit_exact(ctx, clouds, leaf):
    for pts in clouds:
        got = _host(ctx.voxel_downsample(_dev(pts), leaf))
        ref = O.voxel_downsample(pts, leaf)
        assert got.shape == ref.shape
        assert np.array_equal(got[:, :3], ref[:, :3])


def test_voxel_downsample_edge_cases(ctx, rtr):
    import torch
    one = np.array([[0.5, -0.25, 3.0, 0.0]], np.float32)
    assert np.array_equal(_host(ctx.voxel_downsample(_dev(one), 0.01))[:, :3], one[:, :3])
    dup = np.repeat(one, 100, axis=0)
    got = _host(ctx.voxel_downsample(_dev(dup), 0.01))
    assert got.shape[0] == 1 and np.array_equal(got[:, :3], O.voxel_downsample(dup, 0.01)[:, :3])
    e = torch.zeros((0, 4), dtype=torch.float32, device="cuda")
    assert ctx.voxel_downsample(e, 0.01).shape[0] == 0
    # a key space beyond 2^32 is reported, not wrapped
    far = np.array([[0, 0, 0, 0], [1e6, 1e6, 1e6, 0]], np.float32)
    with pytest.raises(rtr.RtrError):
        ctx.voxel_downsample(_dev(far), 0.001)


@pytest.mark.parametrize("r", [0.02, 0.05])
def test_uniform_sample_exact(ctx, clouds, r):
    for pts in clouds:
        v = O.voxel_downsample(pts, 0.01)
        got = _host(ctx.uniform_sample(_dev(v), r))
        assert np.array_equal(got, O.uniform_sample(v, r))


@pytest.mark.parametrize("k", [10, 16])
def test_normals_bit_exact(ctx, clouds, k):
    vp = (0.0, -2.5, 1.5)
    for pts in clouds:
        v = O.voxel_downsample(pts, 0.01)
        got = _host(ctx.normals(_dev(v), k, vp, 0.02))
        ref = O.normals(v, k, vp)
        assert np.array_equal(got, ref), np.abs(got - ref).max()


def test_orient_outward_exact(ctx, clouds):
    v = O.voxel_downsample(clouds[0], 0.01)
    n = O.normals(v, 10, (0.0, 0.0, 0.0))
    d_n = _dev(n)
    ctx.orient_outward(_dev(v), d_n)
    assert np.array_equal(_host(d_n), O.orient_outward(v, n))


def test_shot352_matches_oracle(ctx, clouds):
    for pts, vp in ((clouds[0], (0, 0, 0)), (clouds[1], (0.0, -2.5, 1.5))):
        v = O.voxel_downsample(pts, 0.01)
        n = O.normals(v, 10, vp)
        keys = O.uniform_sample(v, 0.02)
        import torch
        got, glrf = ctx.shot352(_dev(v), _dev(n), torch.from_numpy(keys).cuda(), 0.04, lrf=True)
        got = _host(got)
        ref, rlrf = O.shot352(v, n, keys, 0.04)
        assert np.array_equal(got, ref), (np.abs(got - ref).max(axis=1) > 0).sum()
        assert np.array_equal(_host(glrf), rlrf)
        # unit-norm histograms, or all-zero for a keypoint with an empty support
        nrm = np.linalg.norm(got, axis=1)
        assert np.all((np.abs(nrm - 1.0) < 1e-5) | (nrm == 0.0))


def test_shot352_independent_of_point_order(ctx, clouds):
    """The same voxels in a shuffled order (so the grid cells hold them in
    another order and the lanes meet them in another order) give the same
    descriptor and LRF bits per keypoint."""
    import torch
    v = O.voxel_downsample(clouds[1], 0.01)
    n = O.normals(v, 10, (0.0, -2.5, 1.5))
    keys = O.uniform_sample(v, 0.02)
    perm = np.random.default_rng(9).permutation(len(v))
    inv = np.argsort(perm).astype(np.int32)
    a, la = ctx.shot352(_dev(v), _dev(n), torch.from_numpy(keys).cuda(), 0.04, lrf=True)
    b, lb = ctx.shot352(_dev(v[perm]), _dev(n[perm]), torch.from_numpy(inv[keys]).cuda(), 0.04, lrf=True)
    assert torch.equal(a, b) and torch.equal(la, lb)


def test_match_exact_bit_exact(ctx, clouds):
    v = O.voxel_downsample(clouds[0], 0.01)
    n = O.normals(v, 10, (0, 0, 0))
    km = O.uniform_sample(v, 0.01)
    ks = O.uniform_sample(v, 0.02)
    md, _ = O.shot352(v, n, km, 0.04)
    sd, _ = O.shot352(v, n, ks, 0.04)
    sd = sd[:3000]
    idx, d2 = ctx.match_exact(_dev(sd), _dev(md))
    ri, rd = O.match(sd, md)
    assert np.array_equal(_host(idx), ri)
    assert np.array_equal(_host(d2), rd)
    # duplicates in the database: ties go to the lowest index
    md2 = np.concatenate([md[:100], md[:100]])
    idx, _ = ctx.match_exact(_dev(md[:100]), _dev(md2))
    assert np.array_equal(_host(idx), np.arange(100))


@pytest.mark.parametrize("n", [1, 31, 1024, 1025, 8193, 16385, 131072, 131073])
@pytest.mark.parametrize("half,leaf", [(0.02, 0.01), (0.5, 0.01), (3.0, 0.01), (5.0, 0.0065)])
def test_voxels_by_size_and_key_width(ctx, n, half, leaf):
    """The segmentation at the edges of its forms: one CTA to a cluster of
    sixteen, beyond that a grid; keys of one to four bytes (64 voxels to just
    under 2^32); points without a voxel among the others, and alone."""
    rng = np.random.default_rng(n + int(1e4 * leaf))
    pts = np.zeros((n, 4), np.float32)
    pts[:, :3] = rng.uniform(-half, half, (n, 3))
    if n > 1:
        pts[:2, :3] = [[-half] * 3, [half] * 3]
    if n > 30:
        pts[rng.choice(np.arange(2, n), n // 10, replace=False), rng.integers(0, 3)] = np.nan
        pts[n // 2:n // 2 + 5] = pts[2:7]
    got = _host(ctx.voxel_downsample(_dev(pts), leaf))
    assert np.array_equal(got, O.voxel_downsample(pts, leaf))
    assert np.array_equal(_host(ctx.uniform_sample(_dev(pts), leaf)), O.uniform_sample(pts, leaf))
    pts[:, 1] = np.inf
    assert ctx.voxel_downsample(_dev(pts), leaf).shape[0] == 0


@pytest.mark.parametrize("k", [8, 10, 16])
@pytest.mark.parametrize("cell", [0.003, 0.02, 0.2])
def test_normals_sparse_dense_and_odd_points(ctx, k, cell):
    """Neighbour searches at the edges of their forms: dense patches (own cell
    first), single points far from others (boxes grown several times), fewer
    points than k, lattice points (ties), coordinates that are not finite."""
    rng = np.random.default_rng(5)
    a = rng.uniform(-0.1, 0.1, (1500, 3))
    a[:, 2] *= 0.05
    lattice = np.stack(np.meshgrid(*[np.arange(7) * 0.01] * 3), -1).reshape(-1, 3) + [1.0, 0.0, 0.0]
    far = rng.uniform(-3, 3, (40, 3))
    pts = np.zeros((1500 + 343 + 40, 4), np.float32)
    pts[:, :3] = np.concatenate([a, lattice, far])
    pts = pts[rng.permutation(len(pts))]
    for n in (len(pts), 129, 4, 1):
        q = pts[:n]
        got = _host(ctx.normals(_dev(q), k, (0.3, -1.0, 2.0), cell))
        assert np.array_equal(got, O.normals(q, k, (0.3, -1.0, 2.0)), equal_nan=True), n
    q = pts.copy()
    q[7, 0] = np.nan
    q[9, 2] = np.inf
    got = _host(ctx.normals(_dev(q), k, (0.3, -1.0, 2.0), cell))
    keep = np.isfinite(q[:, :3]).all(1)
    assert np.array_equal(got[keep], O.normals(q[keep], k, (0.3, -1.0, 2.0)), equal_nan=True)


@pytest.mark.parametrize("n", [199999, 200000, 260001])
def test_normals_of_large_clouds_even_and_uneven(ctx, n):
    """On both sides of the size from which warps of evenly spread points
    search side by side: an even sheet, a dense patch, points far from others
    and coordinates that are not finite, mixed; each point as the oracle has it
    (a sample of every kind, with its neighbours taken from the whole cloud)."""
    rng = np.random.default_rng(n)
    pts = np.zeros((n, 4), np.float32)
    pts[:, :2] = rng.uniform(0, 4.0, (n, 2))
    pts[:, 2] = rng.normal(0, 0.002, n)
    m = n // 8
    pts[:m, :3] = rng.normal(0, 0.05, (m, 3)) + [6.0, 1.0, 0.0]
    pts[m:m + 50, :3] = rng.uniform(20, 40, (50, 3))
    pts[m + 60, 0], pts[m + 61, 2] = np.nan, np.inf
    pts = pts[rng.permutation(n)]
    keep = np.isfinite(pts[:, :3]).all(1)
    for k, cell in ((10, 0.02), (8, 0.0), (16, 0.0)):
        got = _host(ctx.normals(_dev(pts), k, (0.3, -1.0, 2.0), cell))
        assert np.array_equal(got[keep], O.normals(pts[keep], k, (0.3, -1.0, 2.0)), equal_nan=True), (k, cell)


def test_normals_of_an_even_volume_cost_no_more_with_the_automatic_cell(ctx):
    """300,000 points spread evenly in a volume: the automatic cell holds 27
    cells of 200 candidates, which threads take side by side; within 1.45 of the
    time with a cell fitted to the cloud (1.67 with a warp a point, 1.2 so)."""
    import torch
    n = 300000
    pts = np.zeros((n, 4), np.float32)
    pts[:, :3] = np.random.default_rng(1).uniform(0, 4.0, (n, 3))
    p = _dev(pts)

    def time(cell):
        best = float("inf")
        for k in range(12):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            ctx.normals(p, 8, (0.0, 0.0, 0.0), cell)
            b.record()
            b.synchronize()
            best = min(best, a.elapsed_time(b)) if k > 1 else best
        return best
    assert time(0.0) < 1.45 * time(1.25 * 4.0 / n ** (1 / 3))


@pytest.mark.parametrize("n", [5000, 200000])
def test_launches_that_fail_are_reported(rtr, n):
    """Voxels and keypoints on a stream whose capture has been invalidated (by
    a synchronisation): no kernel can be launched there, by a cluster or a
    grid, and the calls say so; the context stays usable."""
    import ctypes

    import torch
    cu = ctypes.CDLL("libcuda.so.1")
    pts = np.zeros((n, 4), np.float32)
    pts[:, :3] = np.random.default_rng(n).uniform(-1, 1, (n, 3))
    p, out = _dev(pts), torch.zeros((n, 4), dtype=torch.float32, device="cuda")
    cnt = torch.zeros(1, dtype=torch.int32, device="cuda")
    c = rtr.Context(0)
    try:
        ref = _host(c.voxel_downsample(p, 0.05))  # (sizes the scratch)
        c.uniform_sample(p, 0.05)
        torch.cuda.synchronize()
        s, g = ctypes.c_void_p(), ctypes.c_void_p()
        assert cu.cuStreamCreate(ctypes.byref(s), 1) == 0
        assert cu.cuStreamBeginCapture_v2(s, 2) == 0
        assert cu.cuStreamSynchronize(s) != 0
        args = (c.h, p.data_ptr(), n, ctypes.c_float(0.05), out.data_ptr(), cnt.data_ptr(), s)
        rv, ru = rtr.lib().rtr_voxel_downsample(*args), rtr.lib().rtr_uniform_sample(*args)
        assert cu.cuStreamEndCapture(s, ctypes.byref(g)) != 0
        assert cu.cuStreamDestroy_v2(s) == 0
        assert rv != 0 and ru != 0, (rv, ru)
        assert np.array_equal(_host(c.voxel_downsample(p, 0.05)), ref)
    finally:
        c.close()
