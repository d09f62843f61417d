"""Dense scores (score_tiles, score_segments, score_all) on the kernels that give a tile to a thread."""
import numpy as np
import pytest

from oracle import pyoracle as ora
from tests import helpers as H

pytestmark = pytest.mark.gpu
S = pytest.importorskip("slhav2_b200")
F = np.float32


@pytest.mark.parametrize("codec", [1, 2, 3, 4, 5])
def test_dense_scores_of_an_arena_with_scattered_cold_slots(codec):
    # every CTA takes several rounds of its staging ring, and in every warp some lanes hold COLD slots: a slot of the ring must
    # not be refilled before the warp's last lane has read its residual bits.  Repeated calls give the same bits.
    n = 40000 + codec
    tiles = np.tile(H.random_tiles(2500, codec, seed=500 + codec, warm_every=9, nocorr_every=6), n // 2500 + 1)[:n]
    pool = S.TilePool(n, 2**40, S.PAGE_OLDEST_FIRST, S.EVICT_IMPORTANCE)
    pool.insert(tiles)
    pool.observe_scores(np.arange(n, dtype=np.uint32), np.random.default_rng(codec).standard_normal(n).astype(F), 1.0)
    pool.set_budget(96 * n * 3 // 5)
    assert pool.enforce_budget()
    now, state = pool.read()[:2]
    cold = state == ora.COLD
    assert 0.2 < cold.mean() < 0.5 and cold[:n // 32 * 32].reshape(-1, 32).any(1).mean() > 0.9
    qc, qs = H.random_queries(1, 510 + codec)
    want = ora.score_tiles(now, qc[0], qs[0])[~cold]
    first = None
    for _ in range(8):
        slots, scores = pool.score_all(qc[0], qs[0])
        assert np.array_equal(slots, np.flatnonzero(~cold))
        assert np.all(np.abs(scores - want) <= 1e-4 * (1 + np.abs(want)))
        first = scores if first is None else first
        assert np.array_equal(scores, first)


@pytest.mark.parametrize("codec", range(7))
@pytest.mark.parametrize("nq", [1, 4, 17])
def test_query_rows_may_start_at_any_float(codec, nq):
    # query rows in device memory that start 4, 8 and 12 bytes behind a 16-byte boundary: the same results as from the boundary
    n, k = 3000, 16
    tiles = H.random_tiles(n, codec, seed=520 + codec)
    qc, qs = H.random_queries(nq, 530)
    dt, ds = S.to_device(tiles), S.to_device(qs)
    long_tiles = S.to_device(np.tile(tiles, 11))  # (score_tiles takes another kernel from 32 768 tiles on)
    seg, off = S.make_segments([(0, n, 0, nq, 0)]), np.arange(nq, dtype=np.uint64) * n

    def scores(q):
        i, s, c = S.score_topk(dt, seg, q, ds, nq, k)
        return [i, s, c, S.score_segments(dt, seg, q, ds, nq, np.zeros((nq, n), F), off, n), S.score_tiles(long_tiles, 11 * n, q, ds, nq, np.zeros((nq, 11 * n), F))]

    want = scores(S.to_device(qc))
    for shift in (1, 2, 3):
        flat = S.to_device(np.concatenate([np.zeros(shift, F), qc.reshape(-1)]))
        for a, b in zip(scores(flat.view(4 * shift, qc.nbytes)), want):
            assert np.array_equal(a, b)
