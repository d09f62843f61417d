"""The streaming kernels where short rows would be scored as a whole: the same shapes at the edges of their blocks and items, with whole rows switched off.  Calls
above what whole rows are taken for (rows above 32 768 tiles, many rows) run on these kernels."""
import numpy as np
import pytest

from tests import helpers as H
from tests import test_gpu_stream_kernel as T
from tests import test_gpu_topk as K

pytestmark = pytest.mark.gpu
S = pytest.importorskip("slhav2_b200")


@pytest.fixture(autouse=True)
def streamed():
    S.debug_stream_all_rows(True)
    yield
    S.debug_stream_all_rows(False)


@pytest.mark.parametrize("codec,nq,kernel", [(5, 1, S.KERNEL_TILE), (5, 6, S.KERNEL_TILE), (5, 64, S.KERNEL_WIDE), (4, 17, S.KERNEL_WIDE), (3, 64, S.KERNEL_WIDE), (0, 4, S.KERNEL_STREAM)])
def test_segments_around_the_block_sizes(codec, nq, kernel):
    T.test_top_k_of_segments_around_the_block_sizes(codec, nq)
    assert S.debug_last_score_kernel() == kernel


@pytest.mark.parametrize("codec,n_seg,longest,nq,k", [(5, 100, 3000, 3, 40), (5, 3000, 20, 2, 7), (5, 160, 9000, 4, 16), (5, 8, 20011, 4, 512), (3, 90, 2500, 6, 300)])
def test_many_ragged_segments(codec, n_seg, longest, nq, k):
    T.test_top_k_of_many_ragged_segments(codec, n_seg, longest, nq, k)
    assert S.debug_last_score_kernel() == (S.KERNEL_TILE if codec == 5 else S.KERNEL_STREAM)


@pytest.mark.parametrize("seed", [0, 2, 3, 5])
def test_mix3_random_shapes(seed):
    T.test_mix3_top_k_of_random_shapes(seed)
    assert S.debug_last_score_kernel() == S.KERNEL_TILE


@pytest.mark.parametrize("nq,n_seg,n", [(2, 1, 5000), (4, 100, 900), (20, 3, 2000)])
def test_mix3_rows_that_are_handed_back(nq, n_seg, n):
    T.test_mix3_rows_that_are_handed_back(nq, n_seg, n)
    assert S.debug_last_score_kernel() == (S.KERNEL_WIDE if nq == 20 else S.KERNEL_TILE)


@pytest.mark.parametrize("n,nq,k,codec,warm,nocorr,foreign", [(12800, 16, 128, 4, 7, 5, None), (9000, 100, 32, 4, 0, 0, None), (20000, 24, 100, 0, 0, 0, 2), (127, 20, 200, 1, 0, 0, None),
                                                              (7000, 64, 512, 3, 0, 0, 1), (9000, 40, 100, 5, 8, 4, None), (7000, 20, 64, 5, 0, 0, 4)])
def test_the_wide_kernel(n, nq, k, codec, warm, nocorr, foreign):
    K.test_wide_scoring_on_the_tcgen05_kernel(n, nq, k, codec, warm, nocorr, foreign)
    assert S.debug_last_score_kernel() == S.KERNEL_WIDE


@pytest.mark.parametrize("n_seg,n,nq", [(3, 5000, 4), (100, 700, 2), (4, 3000, 20)])
def test_a_plan_of_mix3_tiles_takes_int4_tiles_of_its_shape(n_seg, n, nq):
    # a plan keeps the kernel of the tiles that came first: interleaved shares, plain ones, the 64-row kernel
    k, total = 33, n_seg * nq
    rows = [(i * n, n, i * nq, nq, i) for i in range(n_seg)]
    seg = S.make_segments(rows)
    for codec in (5, 1, 5):
        tiles = np.resize(H.random_tiles(3000, codec, seed=840 + codec, warm_every=9), n_seg * n)
        qc, qs = H.random_queries(total, 841)
        idx, sc, cnt = S.score_topk(S.to_device(tiles), seg, qc, qs, total, k)
        assert S.debug_last_score_kernel() == (S.KERNEL_WIDE if nq == 20 else S.KERNEL_TILE) and S.last_score_stats()["rows_handed_to_generic_kernel"] == 0
        T._check_rows(tiles, rows, qc, qs, idx, sc, cnt, k, every=7 if n_seg > 9 else 1)
