"""The tcgen05 scoring kernels at the edges of their blocks: a warp holds 32 tiles, a warpgroup's block 128, a round of a CTA
384 or 512; up to four query rows go through score_stream_kernel (MIX3: score_mix3_kernel), sixteen or more through
score_wide_kernel, any number through the dense kernels.  Oracle: compute_score_scalar.  Bound: the reference's own 1e-3 (1 + |s|)."""
import numpy as np
import pytest

from oracle import pyoracle as ora
from tests import helpers as H

pytestmark = pytest.mark.gpu
S = pytest.importorskip("slhav2_b200")
F = np.float32
LENS = [1, 31, 32, 33, 0, 127, 128, 129, 383, 385, 511, 513, 1025, 2111]


def _layout(nq):
    rows, tb = [], 0
    for i, n in enumerate(LENS):
        rows.append((tb, n, i * nq, nq, 5 * i))
        tb += n
    return rows, tb, nq * len(LENS)


def _inputs(codec, nq, seed):
    rows, n, total = _layout(nq)
    tiles = H.random_tiles(n, codec, seed=seed + codec, warm_every=7, nocorr_every=5)
    qc, qs = H.random_queries(total, seed + 50 + codec)
    return rows, tiles, qc, qs, total


@pytest.mark.parametrize("codec", range(7))
@pytest.mark.parametrize("nq", [1, 4, 6, 17, 64])
def test_top_k_of_segments_around_the_block_sizes(codec, nq):
    rows, tiles, qc, qs, total = _inputs(codec, nq, 900)
    k = 24
    idx, sc, cnt = S.score_topk(S.to_device(tiles), S.make_segments(rows), qc, qs, total, k)
    for tb, n, qb, _, base in rows:
        for j in range(qb, qb + nq):
            m = min(n, k)
            assert cnt[j] == m
            assert np.all(idx[j, m:] == 0xFFFFFFFF) and np.all(np.isneginf(sc[j, m:]))
            if not n:
                continue
            want = ora.score_tiles(tiles[tb:tb + n], qc[j], qs[j])
            got = idx[j, :m].astype(np.int64) - base
            assert len(set(got)) == m and got.min() >= 0 and got.max() < n
            assert np.all(np.abs(sc[j, :m] - want[got]) <= 1e-3)
            assert np.all(np.diff(sc[j, :m]) <= 0)
            # whatever is missing from the winners ties with the last of them
            rest = np.delete(want, got)
            assert not len(rest) or rest.max() <= want[got].min() + 2e-3


@pytest.mark.parametrize("codec", range(7))
@pytest.mark.parametrize("nq", [1, 4, 17, 64])
def test_dense_scores_of_segments_around_the_block_sizes(codec, nq):
    rows, tiles, qc, qs, total = _inputs(codec, nq, 950)
    row_len = max(LENS) + 100
    out = np.full((total, row_len), 9.0, F)
    S.score_segments(S.to_device(tiles), S.make_segments(rows), qc, qs, total, out, np.arange(total, dtype=np.uint64) * row_len, row_len, fill=-3.0)
    for tb, n, qb, _, base in rows:
        for j in range(qb, qb + nq):
            if n:
                want = ora.score_tiles(tiles[tb:tb + n], qc[j], qs[j])
                err = np.abs(out[j, base:base + n] - want)
                assert np.all(err <= 1e-3) and np.all(err <= 1e-3 * (1 + np.abs(want)))
            assert np.all(out[j, base + n:] == -3.0)


@pytest.mark.parametrize("nq", [3, 16])
def test_segments_of_different_codecs_in_one_call(nq):
    # a CTA decodes the kind of its first tile: the rows of the other segments take another pass, the results stay the same
    parts = [H.random_tiles(n, c, seed=70 + c, warm_every=9, nocorr_every=4) for c, n in zip((2, 5, 0, 3, 4), (700, 513, 129, 2049, 40))]
    tiles = np.concatenate(parts)
    qc, qs = H.random_queries(5 * nq, 71)
    rows, tb = [], 0
    for i, p in enumerate(parts):
        rows.append((tb, len(p), i * nq, nq, 0))
        tb += len(p)
    row_len = 2049
    out = np.zeros((5 * nq, row_len), F)
    dt, seg = S.to_device(tiles), S.make_segments(rows)
    S.score_segments(dt, seg, qc, qs, 5 * nq, out, np.arange(5 * nq, dtype=np.uint64) * row_len, row_len)
    idx, sc, _ = S.score_topk(dt, seg, qc, qs, 5 * nq, 32)
    for tb, n, qb, _, _ in rows:
        for j in range(qb, qb + nq):
            want = ora.score_tiles(tiles[tb:tb + n], qc[j], qs[j])
            assert np.all(np.abs(out[j, :n] - want) <= 1e-3 * (1 + np.abs(want)))
            m = min(n, 32)
            assert np.all(np.abs(sc[j, :m] - want[idx[j, :m]]) <= 1e-3)
            assert np.all(np.abs(sc[j, :m] - np.sort(want)[::-1][:m]) <= 2e-3)


def _check_rows(tiles, rows, qc, qs, idx, sc, cnt, k, every=1):
    for i, (tb, n, qb, q, base) in enumerate(rows):
        if i % every:
            continue
        for j in range(qb, qb + q):
            m = min(n, k)
            assert cnt[j] == m and np.all(idx[j, m:] == 0xFFFFFFFF)
            if not n:
                continue
            want = ora.score_tiles(tiles[tb:tb + n], qc[j], qs[j])
            got = idx[j, :m].astype(np.int64) - base
            assert len(set(got)) == m and got.min() >= 0 and got.max() < n
            assert np.all(np.abs(sc[j, :m] - want[got]) <= 1e-3) and np.all(np.abs(sc[j, :m] - np.sort(want)[::-1][:m]) <= 2e-3)


@pytest.mark.parametrize("codec", [3, 5])
@pytest.mark.parametrize("n_seg,longest,nq,k", [(100, 3000, 3, 40), (90, 2500, 6, 300), (3000, 20, 2, 7), (160, 9000, 4, 16), (1, 700, 5, 64), (8, 20011, 4, 512)])
def test_top_k_of_many_ragged_segments(codec, n_seg, longest, nq, k):
    # more streams than half the CTAs: equal shares instead of interleaved ones, several items per CTA, thresholds carried from one
    # item to the next; thousands of short segments; and a few long ones, interleaved
    rng = np.random.default_rng(n_seg + k + 1000 * codec)  # (plans are kept by shape, each for one codec)
    base = H.random_tiles(4000, codec, seed=800 + codec, warm_every=7, nocorr_every=5)
    rows, tb = [], 0
    for i in range(n_seg):
        n = int(rng.integers(0 if i % 3 else 1, longest + 1))
        rows.append((tb, n, i * nq, nq, 3 * i))
        tb += n
    tiles = base[rng.integers(0, len(base), tb)]
    qc, qs = H.random_queries(n_seg * nq, 801)
    idx, sc, cnt = S.score_topk(S.to_device(tiles), S.make_segments(rows), qc, qs, n_seg * nq, k)
    assert S.last_score_stats()["rows_handed_to_generic_kernel"] == 0
    _check_rows(tiles, rows, qc, qs, idx, sc, cnt, k, every=max(1, n_seg // 60))


@pytest.mark.parametrize("seed", range(6))
def test_mix3_top_k_of_random_shapes(seed):
    rng = np.random.default_rng(900 + seed)
    n_seg = int(rng.integers(1, 12))
    base = H.random_tiles(3000, 5, seed=810 + seed, warm_every=9, nocorr_every=4)
    rows, tb, qb = [], 0, 0
    for i in range(n_seg):
        n, nq = int(rng.choice([0, 1, 33, int(rng.integers(2, 2000)), int(rng.integers(2000, 30000))])), int(rng.choice([1, 2, 4, 5, 9]))
        rows.append((tb, n, qb, nq, int(rng.integers(0, 1000))))
        tb, qb = tb + n, qb + nq
    tiles = base[rng.integers(0, len(base), max(tb, 1))]
    qc, qs = H.random_queries(qb, 820 + seed)
    k = int(rng.choice([1, 17, 256, 1500]))
    dt, seg = S.to_device(tiles), S.make_segments(rows)
    for _ in range(2):
        idx, sc, cnt = S.score_topk(dt, seg, qc, qs, qb, k)
        _check_rows(tiles, rows, qc, qs, idx, sc, cnt, k)


@pytest.mark.parametrize("nq,n_seg,n", [(2, 1, 5000), (4, 100, 900), (20, 3, 2000)])
def test_mix3_rows_that_are_handed_back(nq, n_seg, n):
    # a stretch of another codec in one segment, an element beyond the split in another: the rows of those, and no others
    tiles = np.tile(H.random_tiles(n, 5, seed=830, nocorr_every=4), n_seg)
    other = n_seg - 1
    tiles[other * n + n // 2:other * n + n // 2 + 70] = H.random_tiles(70, 4, seed=831)
    rows = [(i * n, n, i * nq, nq, 0) for i in range(n_seg)]
    qc, qs = H.random_queries(n_seg * nq, 832)
    handed = nq
    if n_seg > 1:
        qc[nq + 1, 100] = 1e30
        handed = 2 * nq
    k = 25
    idx, sc, cnt = S.score_topk(S.to_device(tiles), S.make_segments(rows), qc, qs, n_seg * nq, k)
    assert S.last_score_stats()["rows_handed_to_generic_kernel"] == handed
    if n_seg > 1:
        qc[nq + 1] = 0  # (a row of 1e30: its winners are those of one element)
        rows = rows[:1] + rows[2:]
    _check_rows(tiles, rows, qc, qs, idx, sc, cnt, k, every=7 if n_seg > 9 else 1)


@pytest.mark.parametrize("codec", [0, 2, 3, 4, 6])
@pytest.mark.parametrize("nq", [1, 3, 4])
def test_plain_shares_around_the_sets_of_sixteen_and_thirty_two(codec, nq):
    # more than 74 streams: CTAs take contiguous shares, in sets of 16 tiles (items are short), several segments in turn, some of them with WARM
    # tiles, tiles without their correction plane and, in one segment, tiles of another codec (handed to the generic kernel)
    lens = [1, 15, 16, 17, 31, 32, 33, 47, 63, 65, 767, 768, 769, 800, 1537, 0, 5, 24, 49, 2000] * 4
    n, k = sum(lens), 40 + codec  # (plans are kept by shape, each for one codec)
    tiles = H.random_tiles(3000, codec, seed=970 + codec, warm_every=9, nocorr_every=6)
    tiles = np.tile(tiles, n // 3000 + 1)[:n].copy()
    rng = np.random.default_rng(codec)
    rng.shuffle(tiles)
    rows, tb = [], 0
    for i, m in enumerate(lens):
        rows.append((tb, m, i * nq, nq, i))
        tb += m
    odd = rows[12]
    tiles[odd[0] + 400:odd[0] + 403] = H.random_tiles(3, 3 if codec != 3 else 4, seed=5)
    qc, qs = H.random_queries(nq * len(lens), 971)
    S.debug_stream_all_rows(True)  # (such rows are scored as a whole otherwise)
    try:
        idx, sc, cnt = S.score_topk(S.to_device(tiles), S.make_segments(rows), qc, qs, nq * len(lens), k)
        assert S.debug_last_score_set() == 16
    finally:
        S.debug_stream_all_rows(False)
    for tb, m, qb, _, base in rows:
        for j in range(qb, qb + nq):
            have = min(m, k)
            assert cnt[j] == have
            if not have:
                continue
            want = ora.score_tiles(tiles[tb:tb + m], qc[j], qs[j])
            got = idx[j, :have].astype(np.int64) - base
            assert len(set(got)) == have and got.min() >= 0 and got.max() < m
            assert np.all(np.abs(sc[j, :have] - want[got]) <= 1e-3)
            rest = np.delete(want, got)
            assert not len(rest) or rest.max() <= want[got].min() + 2e-3


def _planned_items(lens, sms=148):
    """Work items of a plain plan for four query rows or fewer a segment on `sms` CTAs, as the planner cuts them: at equal shares, and nowhere that leaves a sliver."""
    share = -(-max(768, -(-sum(lens) // sms)) // 16) * 16
    snap, spare, filled, items = min(share // 16, 2048), max(0, share * sms - sum(lens)), 0, []
    for n in lens:
        at = 0
        while at < n:
            if at == 0 and 0 < share - filled < snap and filled and spare >= share - filled:
                spare, filled = spare - (share - filled), 0
            take = min(n - at, share - filled)
            rest = n - at - take
            if 0 < rest < snap:
                take, spare = take + rest, spare + rest
            filled, at = filled + take, at + take
            items.append(take)
            if filled >= share:
                filled = 0
    return items


# Segments that share one buffer of tiles.  INT4 takes sets of 32 from items of 6400 tiles on the average, mixed 8/4 and TQ3 from 18 000, or
# 10 000 where rows have 1000 k tiles, NF4 never.
LONG = [40_000 + 617 * i for i in range(33)] + [65_536, 40_001, 59_999] + [48_000 + 5 * i for i in range(44)]
MIDDLE = [12_000 + 3 * i for i in range(150)]
BETWEEN = [30_000 + 7 * i for i in range(99)]


@pytest.mark.parametrize("codec,nq,k,lens,sets", [(0, 4, 60, LONG, 32), (1, 1, 1024, LONG, 32), (3, 3, 61, LONG, 32), (4, 2, 62, LONG, 32), (2, 4, 63, LONG, 16), (2, 3, 301, LONG, 16),
                                                  (6, 2, 64, MIDDLE, 32), (3, 2, 65, MIDDLE, 16), (4, 3, 20, BETWEEN, 32), (3, 1, 66, BETWEEN, 16)])
def test_plain_shares_of_long_segments_end_inside_a_set_of_thirty_two(codec, nq, k, lens, sets):
    # segments end at every place of a set; some tiles are WARM or without their correction plane; the last segment ends in tiles of another codec
    # and is handed to the generic kernel
    items = _planned_items(lens)
    assert (np.mean(items) >= 18_000) == (lens is LONG) and (np.mean(items) >= 10_000) == (lens is not MIDDLE) and np.mean(items) >= 6400 and len({m % 32 for m in lens}) > 16
    base = np.tile(H.random_tiles(4000, codec, seed=960 + codec, warm_every=9, nocorr_every=6), 17)
    rng = np.random.default_rng(codec)
    rng.shuffle(base)
    base[-5:] = H.random_tiles(5, 3 if codec != 3 else 4, seed=6)
    free = len(base) - 5
    rows = [(int(rng.integers(0, free - m + 1)), m, i * nq, nq, 2 * i) for i, m in enumerate(lens)]
    rows[-1] = (len(base) - lens[-1], lens[-1]) + rows[-1][2:]
    qc, qs = H.random_queries(nq * len(lens), 961)
    idx, sc, cnt = S.score_topk(S.to_device(base), S.make_segments(rows), qc, qs, nq * len(lens), k)
    assert S.debug_last_score_set() == sets
    assert S.last_score_stats()["rows_handed_to_generic_kernel"] == nq
    _check_rows(base, rows[:33] + rows[-1:], qc, qs, idx, sc, cnt, k, every=3)


@pytest.mark.parametrize("codec", [1, 3])
def test_a_pool_of_three_million_slots_skips_its_cold_tiles_in_sets_of_thirty_two(codec):
    # one stream so long that its CTAs take contiguous shares; the slots' states are looked at for both halves of a set
    n, k = 3_000_017, 48 + codec  # (plans are kept by shape, each for one codec)
    base = H.random_tiles(5000, codec, seed=57)
    pool = S.TilePool(n, 2**40, S.PAGE_OLDEST_FIRST, S.EVICT_CAUSAL)
    rng = np.random.default_rng(codec)
    pick = rng.integers(0, len(base), n)
    for b in range(0, n, 500_000):
        pool.insert(base[pick[b:b + 500_000]])
    qc, qs = H.random_queries(2, 58)
    scores = [ora.score_tiles(base, qc[j], qs[j])[pick] for j in range(2)]
    # a hole among the best, and slots all over the stream
    cold = np.unique(np.concatenate([rng.choice(n, 400, replace=False), np.argsort(-scores[0])[:300:2], np.argsort(-scores[1])[:300:2], np.arange(n - 40, n, 3)]))
    for s in cold:
        assert pool.evict(int(s))
    ti, tv, tc = pool.score_topk(qc, qs, 2, k)
    assert S.debug_last_score_set() == 32 and S.last_score_stats()["rows_handed_to_generic_kernel"] == 0
    for j in range(2):
        live = scores[j].copy()
        live[cold] = -np.inf
        assert tc[j] == k and len(set(ti[j])) == k and not set(ti[j]) & set(cold)
        assert np.all(np.abs(tv[j] - live[ti[j]]) <= 1e-3) and np.all(np.abs(tv[j] - np.sort(live)[::-1][:k]) <= 2e-3)


@pytest.mark.parametrize("order", ["random", "rising", "falling", "equal", "negative lambda"])
@pytest.mark.parametrize("codec,nq,k", [(0, 4, 16), (2, 1, 100), (3, 2, 300), (4, 4, 7)])
def test_seeds_of_a_long_row(order, codec, nq, k):
    # one row over all CTAs: few warps append their first sets unfiltered and the others wait for the thresholds these prove, whatever the
    # scores' order.  (The residual term of a negative lambda has the same size: its tiles must not be passed over.)
    n = 150_001
    tiles = np.tile(H.random_tiles(5000, codec, seed=980 + codec), n // 5000 + 1)[:n].copy()
    qc, qs = H.random_queries(nq, 981)
    if order in ("rising", "falling"):
        s = ora.score_tiles(tiles, qc[0], qs[0])
        tiles = tiles[np.argsort(s if order == "rising" else -s, kind="stable")]
    elif order == "equal":
        tiles[:] = tiles[0]
    elif order == "negative lambda":
        tiles["dynamic_lambda"] = np.where(np.arange(n) % 3 == 0, -0.05, 0.0).astype(F)
    idx, sc, cnt = S.score_topk(S.to_device(tiles), S.make_segments([(0, n, 0, nq, 0)]), qc, qs, nq, k)
    for j in range(nq):
        want = ora.score_tiles(tiles, qc[j], qs[j])
        assert cnt[j] == k and len(set(idx[j])) == k
        assert np.all(np.abs(sc[j] - want[idx[j]]) <= 1e-3 * (1 + np.abs(want[idx[j]])))
        rest = np.delete(want, idx[j])
        assert rest.max() <= want[idx[j]].min() + 2e-3 * (1 + np.abs(want).max())
        if order == "equal":
            assert np.array_equal(idx[j], np.arange(k))  # ties go to the lower index
