"""Work splits that the launches run (FLETCHER_PlanShot, FLETCHER_PlanBatch;
host code): grids whose last tile row holds few rows of the updated region, both
memory models, every form, and batches of which some shots keep their own plans
and the columns of others are one pool.  Every tile plane of every running shot
is covered exactly once."""
import ctypes as C

import numpy as np
import pytest

from fletcher_petrobras_gb300 import _lib

FP32, FP16, FP16X = 0, 1, 2
FAST, D1D1 = 0, 1
CTAS = 152


def plan_shot(sx, sy, sz, bord=4, rows=16, zchunks=0, form=FP32, numerics=FAST, media=0, ctas=CTAS):
    lib = _lib.load()
    first = np.zeros(ctas + 1, np.int32)
    cost = C.c_long(0)
    args = (ctas, sx, sy, sz, bord, rows, zchunks, form, numerics, media)
    n = lib.FLETCHER_PlanShot(*args, None, 0, _lib.iptr(first), C.byref(cost))
    assert n > 0
    seg = np.zeros((n, 4), np.int32)
    assert lib.FLETCHER_PlanShot(*args, _lib.iptr(seg), n, _lib.iptr(first), C.byref(cost)) == n
    assert first[0] == 0 and first[-1] == n and np.all(np.diff(first) >= 0)
    return seg, first, cost.value


def tiles(sx, sy, bord, rows):
    return -(-(sx - bord - 4) // 32), -(-(sy - bord - 4) // rows)


def covered_once(seg, sx, sy, sz, bord, rows):
    """seg: {tile x index, y0, z0, z1}."""
    ntx, nty = tiles(sx, sy, bord, rows)
    cover = np.zeros((nty, ntx, sz - 2 * bord), np.int32)
    for tx, y0, z0, z1 in seg:
        ty, r = divmod(int(y0) - 4, rows)
        assert r == 0 and 0 <= ty < nty and 0 <= tx < ntx and bord <= z0 < z1 <= sz - bord
        cover[ty, tx, z0 - bord:z1 - bord] += 1
    return bool(np.all(cover == 1))


def by_tile(seg):
    out = seg.copy()
    assert np.all((out[:, 0] - 4) % 32 == 0)
    out[:, 0] = (out[:, 0] - 4) // 32
    return out


MODES = [dict(), dict(media=1), dict(form=FP16), dict(form=FP16X), dict(numerics=D1D1), dict(rows=12), dict(rows=8),
         dict(zchunks=3), dict(zchunks=-5), dict(bord=7)]


@pytest.mark.parametrize("mode", MODES, ids=str)
@pytest.mark.parametrize("size", [(213, 137, 181), (306, 257, 223), (136, 136, 136), (64, 64, 64), (44, 40, 36),
                                  (408, 68, 88), (48, 58, 338), (165, 105, 268), (20, 25, 16), (600, 21, 400)])
def test_shot_covers_every_tile_plane_once(size, mode):
    kw = dict(mode)
    seg, first, cost = plan_shot(*size, **kw)
    rows, bord = kw.get("rows", 16), kw.get("bord", 4)
    assert covered_once(by_tile(seg), *size, bord, rows)
    # The busiest CTA's cost: whole tiles at a plane a plane and 4 a segment, a
    # tile with fewer rows between 4 / 5 of that and all of it.
    last = (size[1] - bord - 4) - (tiles(*size[:2], bord, rows)[1] - 1) * rows
    share = max(last / rows, 0.8)
    full = per = 0.0
    for b in range(CTAS):
        p = seg[first[b]:first[b + 1]]
        w = np.where(p[:, 1] + rows > size[1] - bord, share, 1.0)
        full = max(full, float(np.sum(p[:, 3] - p[:, 2] + 4)))
        per = max(per, float(np.sum(w * (p[:, 3] - p[:, 2] + 4))))
    assert per - 1 <= cost <= full + 1


def test_few_row_tiles_are_counted_apart_where_that_is_cheaper():
    """213 x 137 x 181: the last of nine tile rows holds one row of the updated
    region.  The launch's split is cheaper than that of nine whole rows."""
    lib = _lib.load()
    ntx, nty = tiles(213, 137, 4, 16)
    assert (ntx, nty) == (7, 9) and 137 - 8 - 8 * 16 == 1
    first = np.zeros(CTAS + 1, np.int32)
    whole = C.c_long(0)
    assert lib.FLETCHER_PlanSegments(CTAS, ntx, nty, 16, 4, 173, 0, None, 0, _lib.iptr(first), C.byref(whole)) > 0
    assert plan_shot(213, 137, 181)[2] < whole.value
    # The Der1-Der1 kernel computes every row: the split of whole tile rows.
    assert plan_shot(213, 137, 181, numerics=D1D1)[2] <= whole.value


def test_random_shots_are_covered_once():
    g = np.random.default_rng(3)
    for _ in range(150):
        bord = int(g.integers(4, 9))
        size = [int(v) for v in 2 * bord + np.exp(g.uniform(0, np.log([400, 400, 300]))).astype(int)]
        kw = dict(MODES[g.integers(len(MODES))], ctas=int(g.integers(1, 320)))
        kw["bord"] = bord
        kw.setdefault("zchunks", int(g.integers(-4, 5)))
        seg, _, _ = plan_shot(*size, **kw)
        assert covered_once(by_tile(seg), *size, bord, kw.get("rows", 16)), (size, kw)


@pytest.mark.parametrize("form", [FP32, FP16X])
@pytest.mark.parametrize("rows", [16, 8])
def test_batch_covers_every_tile_plane_of_every_running_shot_once(form, rows):
    lib = _lib.load()
    g = np.random.default_rng(7)
    shots = [(328, 300, 290, 50), (40, 33, 47, 90), (64, 70, 56, 90), (165, 105, 268, 50), (21, 25, 17, 200),
             (213, 137, 181, 300), (96, 41, 88, 10)]
    shots += [tuple(int(v) for v in g.integers(12, 120, 3)) + (int(g.integers(1, 6)),) for _ in range(12)]
    dims = np.array(shots, np.int32)
    ns, bord = len(shots), 4
    steps = sorted({s[3] for s in shots})
    for t in steps:
        running = sum(s[3] >= t for s in shots)
        first = np.zeros(CTAS + 1, np.int32)
        args = (CTAS, ns, _lib.iptr(dims), bord, rows, form, running)
        n = lib.FLETCHER_PlanBatch(*args, None, 0, _lib.iptr(first))
        assert n > 0
        seg = np.zeros((n, 4), np.int32)
        assert lib.FLETCHER_PlanBatch(*args, _lib.iptr(seg), n, _lib.iptr(first)) == n
        assert first[0] == 0 and first[-1] == n and np.all(np.diff(first) >= 0)
        shot = seg[:, 0] >> 16
        seg[:, 0] &= 0xffff
        for i, (sx, sy, sz, k) in enumerate(shots):
            mine = seg[shot == i]
            if k < t:
                assert len(mine) == 0
            else:
                assert covered_once(mine, sx, sy, sz, bord, rows), (t, i)
