"""rtr_harris3d (the keypoint detector of ModelPoint / ScanPoint::
getKeypoint, model_point.h:127-136, scan_point.h:85-94) against the oracle
(oracle/harris.c), bit for bit: the same keypoints (point indices), refined
positions and responses, with suppression and refinement on and off."""
from pathlib import Path

import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu
GOLDEN = Path(__file__).resolve().parent / "golden"


def _dev(a):
    import torch
    return torch.from_numpy(np.ascontiguousarray(a, np.float32)).cuda()


def _check(ctx, rtr, pts, **kw):
    k, s = ctx.harris3d(_dev(pts), rtr.harris_default_params(**{a: int(b) for a, b in kw.items()}))
    rk, rs = O.harris3d(pts, **kw)
    assert np.array_equal(s.cpu().numpy(), rs)
    assert np.array_equal(k.cpu().numpy(), rk)
    return len(rs)


@pytest.mark.parametrize("flags", [dict(), dict(refine=False), dict(non_max=False, refine=False)])
def test_harris_on_shapes_and_main_clouds(ctx, rtr, flags):
    d = np.load(GOLDEN / "main_clouds.npz")
    clouds = [rtr.synth_shape(rtr.CHAIR, 20000, 2024), rtr.synth_shape(rtr.DESK, 20000, 3),
              rtr.synth_shape(rtr.SOFA, 30000, 4), d["chair1"], d["T0_m8111"]]
    found = [_check(ctx, rtr, c, **flags) for c in clouds]
    assert all(f > 0 for f in found), found


def test_harris_on_the_room(ctx, rtr):
    scene, _, _ = rtr.synth_room(1)
    assert _check(ctx, rtr, scene) > 0


@pytest.mark.parametrize("n,tile", [(1, 1), (33, 1), (1023, 1), (1025, 1), (131072, 45), (131073, 45)])
def test_harris_bitmap_edges(ctx, rtr, n, tile):
    """Clouds at the edges of the bitmap's words and of its largest size (the
    next size lists and sorts instead): a chair, or a lattice of chairs far
    apart so that no neighbourhood overflows."""
    if tile == 1:
        pts = rtr.synth_shape(rtr.CHAIR, n, 5)
    else:
        pts = np.concatenate([rtr.synth_shape(rtr.CHAIR, -(-n // tile), 5 + k) for k in range(tile)])[:n].copy()
        k = np.arange(n) // -(-n // tile)
        pts[:, 0] += (2 * (k % 7)).astype(np.float32)
        pts[:, 1] += (2 * (k // 7)).astype(np.float32)
        pts = pts[np.random.default_rng(1).permutation(n)]
    _check(ctx, rtr, pts)


def _lattice(rtr, n):
    """Chairs of 3,000 points far apart."""
    pts = np.concatenate([rtr.synth_shape(rtr.CHAIR, 3000, 5 + j) for j in range(-(-n // 3000))])[:n].copy()
    j = np.arange(n) // 3000
    pts[:, 0] += (2 * (j % 10)).astype(np.float32)
    pts[:, 1] += (2 * (j // 10)).astype(np.float32)
    return pts


@pytest.mark.parametrize("n", [40960, 40961])
def test_harris_on_both_sides_of_the_bitmap(ctx, rtr, n):
    assert _check(ctx, rtr, _lattice(rtr, n)) > 0


def test_harris_time_follows_the_cloud(ctx, rtr):
    """No size of cloud is much slower than a larger one: the bitmap's cost is
    its length, read out for every point."""
    import torch

    def time(n):
        p, best = _dev(_lattice(rtr, n)), float("inf")
        for k in range(6):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            ctx.harris3d(p)
            b.record()
            b.synchronize()
            best = min(best, a.elapsed_time(b)) if k else best
        return best
    assert max(time(n) for n in (100000, 131072)) < 2.0 * time(140000)
