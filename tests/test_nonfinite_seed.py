"""Seeded lookups whose stored distances are +inf or NaN (an ann_prev with such distances, query pixels
that are NaN): a neighbour without a finite distance offers its offset to nobody, and every pull --
lists shared by four warps, every tile width, capped lists, descriptor mode sorted and unsorted -- gives
the field of a plain numpy pull.  Distances of the numpy pull are float64: the returned ones lie within
1e-5 relative of them, the bar every NNF_DIST has."""
import numpy as np
import pytest

import patchtable_b200 as ptb
from oracle.oracle import recompute_dists
from patchtable_b200 import synth
from tests.conftest import srand_all

pytestmark = pytest.mark.gpu
RTOL = 1e-5
ONE_PASS = " -do_table_lookup 0 -kcoherence 0 -coherence_temporal 0 -recalc_dist_temporal 0 -spatial 0 -do_rs 0"


def _seed_field(eh, ew, beh, bew, dist, seed):
    """Random matches with their distances, a third of them +inf or NaN, one corner all NaN."""
    rng = np.random.default_rng(seed)
    prev = np.empty((eh, ew, 3))
    # few distinct offsets, so that neighbours' offsets coincide
    prev[..., 0] = np.clip(np.arange(ew)[None, :] + rng.integers(0, 3, (eh, ew)), 0, bew - 1)
    prev[..., 1] = np.clip(np.arange(eh)[:, None] + rng.integers(0, 3, (eh, ew)), 0, beh - 1)
    prev[..., 2] = dist(prev).astype(np.float32)
    kind = rng.integers(0, 6, (eh, ew))
    prev[..., 2][kind == 0] = np.inf
    prev[..., 2][kind == 1] = np.nan
    prev[:4, :4, 2] = np.nan
    return prev


def _numpy_pull(prev, dist, beh, bew, R, cap):
    """One pull from the field prev: the distance it keeps, per patch."""
    eh, ew = prev.shape[:2]
    out = prev[..., 2].copy()
    lists = [[[] for _ in range(ew)] for _ in range(eh)]
    most = 0
    for y in range(eh):
        for x in range(ew):
            own = (int(prev[y, x, 0]), int(prev[y, x, 1]))
            for dy in range(-R, R + 1):
                for dx in range(-R, R + 1):
                    ny, nx = y + dy, x + dx
                    if (dx == 0 and dy == 0) or not (0 <= ny < eh and 0 <= nx < ew):
                        continue
                    c = (int(prev[ny, nx, 0]) - dx, int(prev[ny, nx, 1]) - dy)
                    key = prev[ny, nx, 2]
                    if not (0 <= c[0] < bew and 0 <= c[1] < beh) or not key < np.inf:
                        continue
                    if c == own or c in [q for q, _ in lists[y][x]]:
                        continue
                    lists[y][x].append((c, key))
            lists[y][x].sort(key=lambda q: q[1])
            lists[y][x] = lists[y][x][:cap or None]
            most = max(most, len(lists[y][x]))
    for k in range(most):
        ann = np.zeros((eh, ew, 3))
        have = np.zeros((eh, ew), bool)
        for y in range(eh):
            for x in range(ew):
                if k < len(lists[y][x]):
                    ann[y, x, :2] = lists[y][x][k][0]
                    have[y, x] = True
        d = dist(ann)
        take = have & (d < out)
        out[take] = d[take]
    return out


def _check(got, prev, want, dist):
    assert np.array_equal(np.isnan(got[..., 2]), np.isnan(want))
    assert np.array_equal(np.isinf(got[..., 2]), np.isinf(want))
    ok = np.isfinite(want)
    np.testing.assert_allclose(got[..., 2][ok], want[ok], rtol=RTOL)
    kept = ~ok
    assert np.array_equal(got[kept][:, :2], prev[kept][:, :2])
    np.testing.assert_allclose(dist(got)[ok], want[ok], rtol=RTOL)


@pytest.mark.parametrize("h,w", [(24, 33), (9, 40), (40, 8)])
@pytest.mark.parametrize("tile", [0, 32, 64, 128, 256])
@pytest.mark.parametrize("dist_param,cap", [(0, 0), (0, 3), (1, 0)])
def test_image_mode_pull(gpu, libc, h, w, tile, dist_param, cap):
    a, _ = synth.pair(h, w, 91)
    _, b = synth.pair(48, 56, 92)
    p = ptb.PatchTableParams("-limit 0.05 -coherence_spatial 4" + ONE_PASS)
    p.prop_dist = p.prop_dist + dist_param
    p.set_schedule((1, 1, cap))
    p.gpu_tile = tile
    R = min(2, p.query_step + p.prop_dist)
    srand_all(libc, 1)
    t = ptb.PatchTable(p, b)

    def dist(ann):
        return recompute_dists(a, b, ann)
    prev = _seed_field(h - 7, w - 7, b.shape[0] - 7, b.shape[1] - 7, dist, 93)
    got = t.lookup(a, ann_prev=prev)
    _check(got, prev, _numpy_pull(prev, dist, b.shape[0] - 7, b.shape[1] - 7, R, cap), dist)
    t.close()


@pytest.mark.parametrize("c", [3, 8, 13])
@pytest.mark.parametrize("dist_param,cap", [(0, 0), (0, 23), (0, 3), (1, 0), (1, 23)])
def test_descriptor_mode_pull(gpu, libc, c, dist_param, cap):
    a, b = synth.descriptor_pair(40, 50, c, 94)
    a = np.ascontiguousarray(a[:17, :30])
    p = ptb.PatchTableParams("-is_descriptor 1 -limit 0.02 -grid_ndims 3 -coherence_spatial 4" + ONE_PASS)
    p.prop_dist = p.prop_dist + dist_param
    p.set_schedule((1, 1, cap))
    R = min(2, p.query_step + p.prop_dist)
    srand_all(libc, 1)
    t = ptb.PatchTable(p, b)
    # three dimensions read a fourth float, the next pixel's first (zero beyond the row: padding)
    pad = lambda x: np.concatenate([x, np.pad(x[:, 1:, :1], ((0, 0), (0, 1), (0, 0)))], 2) if c == 3 else x
    A, B = pad(a).astype(np.float64), pad(b).astype(np.float64)

    def dist(ann):
        d = A - B[ann[..., 1].astype(int), ann[..., 0].astype(int)]
        return (d * d).sum(-1)
    prev = _seed_field(17, 30, 40, 50, dist, 95)
    got = t.lookup(a, ann_prev=prev)
    _check(got, prev, _numpy_pull(prev, dist, 40, 50, R, cap), dist)
    t.close()


@pytest.mark.parametrize("sw", ["", " -speed 1", " -init_random 1"])
def test_nan_pixels_give_every_route_the_same_field(gpu, libc, sw):
    """The default schedule over a query with NaN pixels, seeded with recomputed distances: the patches
    over those pixels stay NaN, and no route reads or returns a match outside b."""
    a, b = synth.pair(61, 83, 96)
    p = ptb.PatchTableParams("-limit 0.05 -coherence_spatial 4 -coherence_temporal 0" + sw)
    srand_all(libc, 1)
    t = ptb.PatchTable(p, b)
    prev = t.lookup(a)
    bad = a.copy()
    bad[20, 30] = np.nan
    bad[50:53, 3, 1] = np.nan
    out = []
    for tile in (0, 32, 64, 128, 256):
        p.gpu_tile = tile
        out.append(t.lookup(bad, ann_prev=prev))
    over = np.zeros(prev.shape[:2], bool)
    for y, x in [(20, 30), (50, 3), (51, 3), (52, 3)]:
        over[max(0, y - 7):y + 1, max(0, x - 7):x + 1] = True
    for o in out:
        assert np.array_equal(o, out[0], equal_nan=True)
    assert np.array_equal(np.isnan(out[0][..., 2]), over)
    assert (out[0][..., 0] >= 0).all() and (out[0][..., 0] < b.shape[1] - 7).all()
    assert (out[0][..., 1] >= 0).all() and (out[0][..., 1] < b.shape[0] - 7).all()
    clean = np.where(np.isnan(bad), 0, bad)
    ok = ~over
    np.testing.assert_allclose(recompute_dists(clean, b, out[0])[ok], out[0][..., 2][ok], rtol=RTOL, atol=1e-9)
    t.close()
