"""GPU parity of the tensor-core descriptor matcher: indices and distances
bit-identical to the exact FP32 oracle, and the BF16(hi+lo) GEMM accurate
enough that almost every query is certified by its top-8 (so the tensor-core
path, not the exact fallback, produces the answer)."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


def _dev(a):
    import torch
    return torch.from_numpy(np.ascontiguousarray(a, np.float32)).cuda()


@pytest.fixture(scope="module")
def descs(rtr):
    model = rtr.synth_shape(rtr.CHAIR, 20000, 2024)
    v = O.voxel_downsample(model, 0.01)
    n = O.orient_outward(v, O.normals(v, 10, (0, 0, 0)))
    md, _ = O.shot352(v, n, O.uniform_sample(v, 0.01), 0.04)
    p = rtr.room_default_params()
    p.n_points = 80000
    scene, _, _ = rtr.synth_room(4, p)
    sv = O.voxel_downsample(scene, 0.01)
    sn = O.normals(sv, 10, (0.0, -2.5, 1.5))
    sd, _ = O.shot352(sv, sn, O.uniform_sample(sv, 0.02), 0.04)
    return md, sd


def test_match_tc_bit_exact(ctx, descs):
    md, sd = descs
    idx, d2 = ctx.match(_dev(sd), _dev(md))
    unc = ctx.match_uncertified()
    ri, rd = O.match(sd, md)
    assert np.array_equal(idx.cpu().numpy(), ri)
    assert np.array_equal(d2.cpu().numpy(), rd)
    # the GEMM, not the fallback, decides: nearly every query certified
    assert unc <= 0.02 * len(sd), (unc, len(sd))


def test_match_tc_ragged_sizes(ctx, descs):
    md, sd = descs
    for nq, ndb in ((1, 1), (5, 3), (129, 257), (300, 1000), (1000, 9)):
        q, db = sd[:nq], md[:ndb]
        idx, d2 = ctx.match(_dev(q), _dev(db))
        ri, rd = O.match(q, db)
        assert np.array_equal(idx.cpu().numpy(), ri), (nq, ndb)
        assert np.array_equal(d2.cpu().numpy(), rd), (nq, ndb)


def test_match_tc_duplicates_tie_to_lowest(ctx, descs):
    md, sd = descs
    db = np.concatenate([md[:50]] * 12)  # every descriptor 12 times
    idx, _ = ctx.match(_dev(md[:50]), _dev(db))
    assert np.array_equal(idx.cpu().numpy(), np.arange(50))


@pytest.mark.parametrize("scale", [1e-3, 37.0, 1e3])
def test_match_tc_scaled_descriptors(ctx, descs, scale):
    # the certification bound scales with the descriptor norms
    md, sd = descs
    q = (sd[:3000] * np.float32(scale)).astype(np.float32)
    db = (md * np.float32(scale)).astype(np.float32)
    idx, d2 = ctx.match(_dev(q), _dev(db))
    ri, rd = O.match(q, db)
    assert np.array_equal(idx.cpu().numpy(), ri)
    assert np.array_equal(d2.cpu().numpy(), rd)


def test_match_tc_general_vectors(ctx):
    # signed, non-normalised vectors whose distances crowd together: most
    # queries cannot be certified and go through the exact re-scan
    rng = np.random.default_rng(12)
    q = rng.standard_normal((1500, 352)).astype(np.float32)
    db = rng.standard_normal((2500, 352)).astype(np.float32)
    idx, d2 = ctx.match(_dev(q), _dev(db))
    ri, rd = O.match(q, db)
    assert np.array_equal(idx.cpu().numpy(), ri)
    assert np.array_equal(d2.cpu().numpy(), rd)


def _near_tie_db(md, group, n_groups, seed):
    """n_groups clusters of `group` rows each, equal to a model descriptor up
    to a 1e-6 perturbation: their distances to a query differ far below the
    certification margin, so every query near a cluster is uncertified."""
    rng = np.random.default_rng(seed)
    base = []
    for i in rng.permutation(len(md)):  # well-separated cluster centres (d^2 > 0.05)
        if all(float(((md[i] - b) ** 2).sum()) > 0.05 for b in base):
            base.append(md[i])
        if len(base) == n_groups:
            break
    base = np.asarray(base, np.float32)
    db = np.repeat(base, group, axis=0)
    db = db + np.float32(1e-6) * rng.standard_normal(db.shape).astype(np.float32)
    perm = rng.permutation(len(db))  # cluster members spread over the database
    return base, np.ascontiguousarray(db[perm], np.float32)


@pytest.mark.parametrize("group,expect_full", [(100, False), (400, True)])
def test_match_tc_near_tie_bands(ctx, descs, group, expect_full):
    # clusters up to 256 rows are settled by the band pass; larger ones by
    # the exact scan of the whole database
    md, _ = descs
    base, db = _near_tie_db(md, group, 8, 5 + group)
    rng = np.random.default_rng(group)
    q = np.repeat(base, 40, axis=0) + np.float32(1e-3) * rng.standard_normal((320, 352)).astype(np.float32)
    q = q.astype(np.float32)
    idx, d2 = ctx.match(_dev(q), _dev(db))
    unc, full = ctx.match_uncertified(), ctx.match_full_scans()
    ri, rd = O.match(q, db)
    assert np.array_equal(idx.cpu().numpy(), ri)
    assert np.array_equal(d2.cpu().numpy(), rd)
    assert unc == len(q)
    assert (full == unc) if expect_full else (full == 0), (unc, full)


def test_match_tc_more_uncertified_than_band_rows(ctx, descs):
    # past 16384 uncertified queries the rest take the full scan
    md, _ = descs
    base, db = _near_tie_db(md, 64, 4, 77)
    rng = np.random.default_rng(3)
    q = (np.repeat(base, 4200, axis=0) + np.float32(1e-3) * rng.standard_normal((16800, 352))).astype(np.float32)
    idx, d2 = ctx.match(_dev(q), _dev(db))
    unc, full = ctx.match_uncertified(), ctx.match_full_scans()
    ri, rd = O.match(q, db)
    assert np.array_equal(idx.cpu().numpy(), ri)
    assert np.array_equal(d2.cpu().numpy(), rd)
    assert unc == len(q) and full == len(q) - 16384, (unc, full)


def test_match_tc_zero_and_nonfinite_queries(ctx, descs):
    # a zero query ties with every unit-norm row (band = whole database);
    # Inf or NaN values make the threshold non-finite: both take the full scan
    md, sd = descs
    q = sd[:64].copy()
    q[:8] = 0.0
    q[8, 5] = np.inf
    q[9, 7] = np.nan
    q[10, :] = -np.inf
    idx, d2 = ctx.match(_dev(q), _dev(md))
    ri, rd = O.match(q, md)
    assert np.array_equal(idx.cpu().numpy(), ri)
    assert np.array_equal(d2.cpu().numpy(), rd, equal_nan=True)
    assert ctx.match_full_scans() >= 3


@pytest.mark.parametrize("nq", [1, 127, 129, 2500])
@pytest.mark.parametrize("ndb", [7, 255, 257, 513, 2049, 2300])
@pytest.mark.parametrize("aligned", [True, False])
def test_match_tc_database_ranges(ctx, descs, nq, ndb, aligned):
    """Few queries take the database in up to eight ranges, each with its own
    list of 8: a last range of a row or a few, rows of the first tiles repeated
    at the end (ties across ranges go to the lowest index), rows that do not
    start on 16 bytes, a zero query among them."""
    import torch
    md, sd = descs
    db = np.concatenate([md, md])[:ndb].copy()
    db[-(ndb // 3):] = db[: ndb // 3]
    q = np.concatenate([sd, md])[:nq].copy()
    q[nq // 2] = 0.0
    if nq > 100:
        q[50:100] = md[:50]  # exact hits and ties
    dev = []
    for a in (q, db):
        flat = torch.empty(a.size + 4, dtype=torch.float32, device="cuda")
        v = flat[0 if aligned else 1:][: a.size].view(a.shape)
        v.copy_(torch.from_numpy(a))
        dev.append(v)
    idx, d2 = ctx.match(*dev)
    ri, rd = O.match(q, db)
    assert np.array_equal(idx.cpu().numpy(), ri)
    assert np.array_equal(d2.cpu().numpy(), rd)


@pytest.mark.parametrize("bad", [0, 1, 3])
@pytest.mark.parametrize("nq", [40, 700])
def test_match_tc_nan_rows_leave_the_error_bound_alone(ctx, nq, bad):
    """A database row with a NaN never wins, and must not take the error
    bound's scale (the largest norm) with it: queries of norm 1 against rows
    of norm 1,000 whose distances differ by parts in a million, far below the
    16-bit products' error, which only the large norms' bound covers."""
    import torch
    rng = np.random.default_rng(nq + bad)
    u = rng.normal(size=352)
    u /= np.linalg.norm(u)

    def high(norm):  # how much the two 16-bit parts of -|b|^2 / 2 put a distance too high
        t = torch.tensor([-0.5 * norm * norm], dtype=torch.float32)
        h = t.bfloat16().float()
        return float(2 * (t - h - (t - h).bfloat16().float()))
    norm = max(np.linspace(1000, 1010, 401), key=high)
    db = (norm * u + 0.0001 * rng.normal(size=(300, 352))).astype(np.float32)
    q = rng.normal(size=(nq, 352)).astype(np.float32)
    q /= np.linalg.norm(q, axis=1, keepdims=True)
    big = q[: nq // 2] * np.float32(1000)  # and queries of the rows' norm
    q[: nq // 2] = big
    for k in range(bad):
        db[17 + 90 * k, 5 + k] = np.nan
    idx, d2 = ctx.match(_dev(q), _dev(db))
    ri, rd = O.match(q, db)
    assert np.array_equal(idx.cpu().numpy(), ri)
    assert np.array_equal(d2.cpu().numpy(), rd)
    assert not np.isin(ri, [17, 107, 197][:bad]).any()


@pytest.mark.parametrize("nq", [3, 5, 4001, 8000, 8001, 16001])
def test_match_tc_rerank_shares_and_ties(ctx, descs, nq):
    """Queries dealt to the re-rank's warps by 4, 8 and 16, ragged at the end,
    with every database row nine times (eight candidates a query in doubt, ties
    to the lowest index) and zero queries among them."""
    md, sd = descs
    db = np.concatenate([md[:60]] * 9)
    q = np.concatenate([sd] * (nq // len(sd) + 1))[:nq].copy()
    q[::101] = 0.0
    q[1::7] = md[np.arange(len(q[1::7])) % 60]
    idx, d2 = ctx.match(_dev(q), _dev(db))
    ri, rd = O.match(q, db)
    assert np.array_equal(idx.cpu().numpy(), ri)
    assert np.array_equal(d2.cpu().numpy(), rd)
    assert ri.max() < 60
