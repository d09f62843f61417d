"""Top-k of calls whose rows are scored as a whole (topk_rows_kernel): rows at the edges of what a thread, a sample and the candidates' slots hold, scores that a
sample does not tell apart, absent and non-finite ones, against an exact selection of the same scores."""
import numpy as np
import pytest

import slhav2_b200 as S
from oracle import pyoracle as ora
from tests import helpers as H

pytestmark = pytest.mark.gpu
F = np.float32
TAKEN = S.last_score_stats  # (a whole-row plan has as many slots as the longest row has scores, in multiples of 32)


def _check(tiles, rows, nq, k, qc, qs, state_cold=None):
    """The dense call scores the same rows with the same kernels: the winners are its k largest, ties towards the lower index, bit for bit."""
    dt, seg = S.to_device(tiles), S.make_segments(rows)
    longest = max(r[1] for r in rows)
    idx, sc, cnt = S.score_topk(dt, seg, qc, qs, nq, k)
    assert TAKEN()["buffer_slots"] == (longest + 31) // 32 * 32
    assert S.debug_last_score_kernel() in (S.KERNEL_ROWS, S.KERNEL_ROWS_WIDE) and S.debug_last_score_set() == 0
    flat = S.make_segments([(t, n, q, m, 0) for t, n, q, m, _ in rows])
    dense = S.score_segments(dt, flat, qc, qs, nq, np.zeros((nq, longest), F), np.arange(nq, dtype=np.uint64) * longest, longest, fill=0.0)
    for t, n, q0, m, base in rows:
        for q in range(q0, q0 + m):
            want = dense[q, :n]
            key = np.where(np.isnan(want), F(-0.0), want).view(np.int32).astype(np.int64)
            key = np.where(key < 0, -2**31 - 1 - key, key)  # total order: -0 below 0
            order = np.lexsort((np.arange(n), -key))[:k]
            have = min(n, k)
            assert cnt[q] == have and np.all(idx[q, have:] == 0xFFFFFFFF) and np.all(sc[q, have:] == -np.inf)
            assert np.array_equal(idx[q, :have], order + base)
            assert np.array_equal(sc[q, :have].view(np.uint32), np.where(np.isnan(want), F(-0.0), want)[order].view(np.uint32))
    return idx, sc


@pytest.mark.parametrize("n", [1, 3, 127, 1025, 2047, 2048, 2049, 4095, 4097, 8191, 8193, 16383, 16385, 20011, 32767, 32768])
@pytest.mark.parametrize("k", [1, 17, 256, 1000, 4096])
def test_rows_of_every_length(n, k):
    # around the scores a thread holds (1024, 2048, .. 16 384 a block's round) and the candidates' slots (from n = cap / 2 on a sample gives the bound)
    codec = [0, 3, 4, 5][n % 4]
    base = H.random_tiles(2000, codec, seed=n, warm_every=9, nocorr_every=5)
    tiles = base[np.random.default_rng(n + k).integers(0, len(base), 2 * n)]  # (with equal scores)
    qc, qs = H.random_queries(5, 900 + k)
    _check(tiles, [(0, n, 0, 3, 5), (n, n, 3, 2, 1000)], 5, k, qc, qs)


@pytest.mark.parametrize("n", [900, 9000, 30000])
@pytest.mark.parametrize("shape", ["equal", "few values", "outlier", "rising", "last", "zero query", "infinite", "huge"])
def test_scores_that_a_sample_does_not_tell_apart(n, shape):
    rng = np.random.default_rng(7)
    tiles = np.tile(H.random_tiles(1000, 1, seed=31), n // 1000 + 1)[:n].copy()
    tiles["dynamic_lambda"] = 0
    qc, qs = H.random_queries(2, 32)
    if shape == "equal":
        tiles[:] = tiles[0]
    elif shape == "few values":
        tiles = tiles[rng.integers(0, 3, n)]
    elif shape == "outlier":
        tiles["scale"][n // 3] *= F(1e6)
    elif shape == "rising":
        tiles["scale"] *= np.linspace(0.01, 3.0, n).astype(F)
    elif shape == "last":
        tiles["scale"][:-300] *= F(1e-3)
    elif shape == "zero query":
        qc[:] = 0
    elif shape == "infinite":
        tiles["scale"][::7] = np.inf
        tiles["scale"][3::11] = np.nan
    elif shape == "huge":
        tiles["scale"][:] = rng.choice(np.array([1e37, 1.0, 1e-30], F), n)
    for k in (1, 200, 2000):
        _check(tiles, [(0, n, 0, 2, 0)], 2, k, qc, qs)


@pytest.mark.parametrize("nq,codec", [(16, 1), (40, 2), (64, 4), (70, 5)])
def test_rows_of_many_queries(nq, codec):
    # the 64-row kernel's scores, of NF4 tiles the four-row kernel's; a segment without rows and one without tiles
    n = 2500
    tiles = H.random_tiles(2 * n, codec, seed=60 + nq, warm_every=8, nocorr_every=3)
    qc, qs = H.random_queries(2 * nq + 20, 61)
    _check(tiles, [(0, n, 0, nq, 3), (n, n - 77, nq, nq, 0), (5, 0, 2 * nq, 20, 9), (9, 400, 0, 0, 0)], 2 * nq + 20, 100, qc, qs)


def test_cold_slots_are_no_candidates():
    n, k = 3000, 500
    tiles = H.random_tiles(n, 3, seed=70)
    pool = S.TilePool(n, 2**40)
    pool.insert(tiles)
    rng = np.random.default_rng(71)
    gone = rng.permutation(n)[:2700]
    for s in gone:
        pool.evict(int(s))
    qc, qs = H.random_queries(4, 72)
    idx, sc, cnt = pool.score_topk(qc, qs, 4, k)
    assert np.all(cnt == 300) and np.all(idx[:, 300:] == 0xFFFFFFFF)
    want = S.score_tiles(S.to_device(tiles), n, qc, qs, 4)
    left = np.setdiff1d(np.arange(n), gone)
    for j in range(4):
        order = left[np.lexsort((left, -want[j, left]))]
        assert np.array_equal(np.sort(idx[j, :300]), left) and np.all(np.abs(sc[j, :300] - want[j, order]) <= 1e-3)


@pytest.mark.parametrize("n,k,live", [(16384, 64, lambda s: s // 4 % 512 == 3), (32768, 100, lambda s: s // 4 % 512 == 511), (16384, 2048, lambda s: s // 4 % 512 < 60), (30000, 4096, lambda s: s // 4 % 512 < 64)])
def test_fewer_slots_than_winners_that_few_threads_hold(n, k, live):
    # what is left of a pool lies where a thread holds more candidates than its own list has room for, fewer than k in all
    tiles = np.tile(H.random_tiles(2000, 3, seed=73), n // 2000 + 1)[:n]
    left = np.flatnonzero(live(np.arange(n)))
    pool = S.TilePool(n, 2**40)
    pool.insert(tiles)
    for s in np.setdiff1d(np.arange(n), left):
        pool.evict(int(s))
    qc, qs = H.random_queries(4, 74)
    idx, sc, cnt = pool.score_topk(qc, qs, 4, k)
    m = min(k, len(left))
    assert np.all(cnt == m) and np.all(idx[:, m:] == 0xFFFFFFFF) and np.all(np.isneginf(sc[:, m:]))
    want = S.score_tiles(S.to_device(tiles), n, qc, qs, 4)
    for j in range(4):
        order = left[np.lexsort((left, -want[j, left]))][:m]
        assert len(set(idx[j, :m])) == m and set(idx[j, :m]) <= set(left)
        assert np.all(np.abs(sc[j, :m] - want[j, order]) <= 1e-3 * (1 + np.abs(want[j, order])))


@pytest.mark.parametrize("codec,n_seg", [(0, 100), (4, 100), (2, 60)])
def test_many_rows_whose_segments_end_inside_a_block(codec, n_seg):
    # above what every call's rows are scored as a whole for: the rule's side of them; shares that are cut in blocks of 128 tiles
    n, nq = 16_000, 4
    tiles = H.random_tiles(n + 600, codec, seed=80 + codec)
    qc, qs = H.random_queries(nq * n_seg, 81)
    rows = [(5 * i, n + i, nq * i, nq, 7 * i) for i in range(n_seg)]
    assert sum(r[1] for r in rows) > 640_000
    _check(tiles, rows, nq * n_seg, 300, qc, qs)



def test_rows_handed_on_for_different_reasons():
    # A segment of three blocks, the first of which begins on an NF4 tile and the others meet one, scored with 16 rows behind 49 short NF4 segments in shares of 50
    # blocks (on 148 SMs, one share of others before them), where the CTA that hands its rows on for the first block does so last: the generic arithmetic, bit for bit.
    n, nq, k = 384, 16, 384
    mixed = H.random_tiles(n, 0, seed=85)
    nf4 = H.random_tiles(60, 2, seed=86)
    mixed[0], mixed[130:140], mixed[300] = nf4[59], nf4[49:59], nf4[58]
    rest = np.tile(H.random_tiles(2560, 0, seed=87), 2)
    tiles = np.concatenate([nf4[:49], mixed, rest])
    at = 49 + n
    rows = [(at + i, 512 if i < 12 else 256) for i in range(13)] + [(i, 1) for i in range(49)] + [(49, n)] + [(at + i, 512) for i in range((148 * 50 - 50 - 52) // 4)]
    rows = [(tb, m, nq * i, nq, 0) for i, (tb, m) in enumerate(rows)]
    total = nq * len(rows)
    qc, qs = H.random_queries(total, 88)
    own = slice(62 * nq, 63 * nq)
    dt = S.to_device(tiles)
    S.debug_force_generic_score(True)
    try:
        alone = S.score_topk(dt, S.make_segments([(49, n, 0, nq, 0)]), qc[own], qs[own], nq, k)
    finally:
        S.debug_force_generic_score(False)
    want = ora.score_tiles(mixed, qc[own][3], qs[own][3])
    assert np.all(np.abs(alone[1][3] - want[alone[0][3]]) <= 1e-3)
    for _ in range(5):
        idx, sc, cnt = S.score_topk(dt, S.make_segments(rows), qc, qs, total, k)
        assert S.debug_last_score_kernel() == S.KERNEL_ROWS_WIDE and S.last_score_stats()["rows_handed_to_generic_kernel"] == nq
        assert np.all(cnt[own] == k) and np.array_equal(idx[own], alone[0]) and np.array_equal(sc[own].view(np.uint32), alone[1].view(np.uint32))


@pytest.mark.parametrize("n,k", [(3000, 512), (4096, 2048), (6000, 4096), (30000, 1024)])
def test_equal_scores_and_one_far_from_the_rest_cost_no_multiple(n, k):
    # the selection's device time beside that of scores that differ: within ten times (comparing equal scores with one another took 30 to 60 times as long)
    base = H.random_tiles(1000, 0, seed=31)
    rng = np.random.default_rng(n)
    nq = 128
    qc, qs = H.random_queries(nq, 90)
    seg = S.make_segments([(0, n, 4 * i, 4, 0) for i in range(nq // 4)])
    took = {}
    for shape in ("differ", "equal", "far"):
        tiles = base[rng.integers(0, 1000, n)] if shape != "equal" else np.repeat(base[:1], n)
        tiles["scale"] *= rng.uniform(0.9, 1.1, n).astype(F) if shape != "equal" else F(1)
        if shape == "far":
            tiles["scale"][n // 3] *= F(1e4)
        dt = S.to_device(tiles)
        args = dt, seg, S.to_device(qc), S.to_device(qs), nq, k, S.DeviceBuffer(nq * k * 4), S.DeviceBuffer(nq * k * 4), S.DeviceBuffer(nq * 4)
        S.score_topk(*args)
        S.timing_begin(9)
        for _ in range(9):
            S.score_topk(*args)
        took[shape] = float(np.median(S.timing_end(9)[1]))
        _check(tiles, [(0, n, 0, 2, 0)], 2, k, qc[:2], qs[:2])
    assert max(took["equal"], took["far"]) < 10 * took["differ"], took


@pytest.mark.parametrize("n_seg,kernel", [(8190, S.KERNEL_ROWS_WIDE), (8200, S.KERNEL_WIDE)])
def test_many_short_rows_of_the_64_row_kernel_stay_within_the_plan_s_memory(n_seg, kernel):
    # 16 rows of 17 tiles a segment, which that kernel pads to 128 scores: 64 MB on either side
    n, nq, k = 17, 16, 4
    assert (n_seg * nq * 128 <= 16 << 20) == (kernel == S.KERNEL_ROWS_WIDE) and n_seg * nq * 32 < 16 << 20
    tiles = H.random_tiles(3000, 1, seed=91)
    qc, qs = (np.resize(x, (n_seg * nq,) + x.shape[1:]) for x in H.random_queries(61, 92))
    rows = [(i % 2900, n, nq * i, nq, i) for i in range(n_seg)]
    idx, sc, cnt = S.score_topk(S.to_device(tiles), S.make_segments(rows), qc, qs, n_seg * nq, k)
    assert S.debug_last_score_kernel() == kernel and np.all(cnt == k)
    for i in (0, 1, 4000, n_seg - 1):
        want = ora.score_tiles(tiles[rows[i][0]:rows[i][0] + n], qc[nq * i + 3], qs[nq * i + 3])
        assert np.all(np.abs(sc[nq * i + 3] - np.sort(want)[::-1][:k]) <= 2e-3) and np.all(np.abs(sc[nq * i + 3] - want[idx[nq * i + 3] - i]) <= 1e-3)


@pytest.mark.parametrize("n,k,among", [(30000, 64, 20), (30000, 64, 64), (16384, 64, 25), (30000, 1024, 130), (5000, 64, 40)])
def test_rows_whose_best_lie_where_the_sample_looks(n, k, among):
    # `among` of the k best scores lie at places that are sampled (every fourth to sixteenth score), so that fewer than k reach the first bound; the lower one, or none, is enough
    step = 4 if n > 16384 else 2 if n > 8192 else 1
    place = np.arange(n)
    sampled = np.flatnonzero((place % 4 == 0) & ((place // 4 % 512 + place // 2048) % step == 0))
    rng = np.random.default_rng(n + k)
    tiles = np.resize(H.random_tiles(1, 0, seed=93), n)
    tiles["dynamic_lambda"] = 0
    qc, qs = H.random_queries(1, 94)
    sign = 1 if ora.score_tiles(tiles[:1], qc[0], qs[0])[0] > 0 else -1
    qc = np.repeat(sign * qc, 128, 0)
    best = np.concatenate([rng.choice(sampled, among, replace=False), rng.choice(np.setdiff1d(place, sampled), k - among, replace=False)])
    scale = tiles["scale"] * rng.uniform(0.1, 1.0, n).astype(F)
    scale[best] = tiles["scale"][0] * rng.uniform(1.5, 2.0, k).astype(F)
    tiles["scale"] = scale
    _check(tiles, [(0, n, 0, 2, 0)], 2, k, qc[:2], qs[[0, 0]])
    if among < k:
        seg, nq = S.make_segments([(0, n, 4 * i, 4, 0) for i in range(32)]), 128
        args = S.to_device(qc), S.to_device(np.repeat(qs, nq, 0)), nq, k, S.DeviceBuffer(nq * k * 4), S.DeviceBuffer(nq * k * 4), S.DeviceBuffer(nq * 4)
        took = {}
        for name, t in (("placed", tiles), ("anywhere", tiles[rng.permutation(n)])):
            dt = S.to_device(t)
            S.score_topk(dt, seg, *args)
            S.timing_begin(9)
            for _ in range(9):
                S.score_topk(dt, seg, *args)
            took[name] = float(np.median(S.timing_end(9)[1]))
        assert took["placed"] < 2.5 * took["anywhere"], took


@pytest.mark.parametrize("n,nq,k,kernel", [(3000, 64, 100, S.KERNEL_ROWS_WIDE), (20000, 40, 500, S.KERNEL_ROWS_WIDE), (32768, 250, 16, S.KERNEL_STREAM), (20000, 250, 100, S.KERNEL_STREAM), (1000, 16, 16, S.KERNEL_ROWS_WIDE)])
def test_nf4_rows_of_many_queries(n, nq, k, kernel):
    # the 64-row kernel does not decode NF4: it hands few on, many are streamed (all of them as its own short items took twice as long)
    tiles = H.random_tiles(n, 2, seed=95, warm_every=9)
    qc, qs = H.random_queries(nq, 96)
    dt, seg = S.to_device(tiles), S.make_segments([(0, n, 0, nq, 7)])
    for _ in range(2):
        idx, sc, cnt = S.score_topk(dt, seg, qc, qs, nq, k)
        assert S.debug_last_score_kernel() == kernel and S.last_score_stats()["rows_handed_to_generic_kernel"] == 0
    assert np.all(cnt == k)
    for j in range(0, nq, 13):
        want = ora.score_tiles(tiles, qc[j], qs[j])
        assert np.all(np.abs(sc[j] - want[idx[j] - 7]) <= 1e-3 * (1 + np.abs(sc[j]))) and np.all(np.abs(sc[j] - np.sort(want)[::-1][:k]) <= 2e-3 * (1 + np.abs(sc[j])))


@pytest.mark.parametrize("n,k", [(1, 1), (127, 64), (255, 255), (256, 300), (257, 64), (1000, 64), (1024, 17), (1025, 17), (900, 65)])
def test_many_short_rows(n, k):
    # from 1024 rows on, short ones of which little is selected take half as many threads each
    rng = np.random.default_rng(n + k)
    tiles = H.random_tiles(500, 4, seed=97, warm_every=9)[rng.integers(0, 500, 2 * n)]
    qc, qs = H.random_queries(1030, 98)
    _check(tiles, [(0, n, 0, 515, 3), (n, n - n // 5, 515, 515, 90)], 1030, k, qc, qs)
