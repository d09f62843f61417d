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


class _CapturedStream:
    """A stream of the CUDA runtime in capture mode (relaxed), set as the library's."""

    def __enter__(self):
        import ctypes as C

        S.load_library()
        self.rt, self.stream = C.CDLL("libcudart.so.12"), C.c_void_p()
        assert self.rt.cudaStreamCreateWithFlags(C.byref(self.stream), 1) == 0
        S.set_stream(self.stream.value)
        assert self.rt.cudaStreamBeginCapture(self.stream, 2) == 0
        return self

    def __exit__(self, *exc):
        import ctypes as C

        graph = C.c_void_p()
        self.rt.cudaStreamEndCapture(self.stream, C.byref(graph))
        self.captured = bool(graph.value)
        self.rt.cudaGetLastError()
        S.set_stream(None)
        self.rt.cudaStreamDestroy(self.stream)


def test_dense_calls_with_tables_refuse_a_stream_that_is_captured():
    # a graph would keep the address of the call's host tables: the call fails and so does the capture; afterwards it works as before
    n, nq = 33000, 3
    tiles = np.tile(H.random_tiles(1100, 1, seed=540), 30)
    qc, qs = H.random_queries(nq, 541)
    dt, dq, ds, out = S.to_device(tiles), S.to_device(qc), S.to_device(qs), S.DeviceBuffer(nq * n * 4)
    seg, off = S.make_segments([(0, n, 0, nq, 0)]), np.arange(nq, dtype=np.uint64) * n
    want = S.score_tiles(dt, n, dq, ds, nq, np.zeros((nq, n), F))
    for call in (lambda: S.score_tiles(dt, n, dq, ds, nq, out), lambda: S.score_segments(dt, seg, dq, ds, nq, out, off, n)):
        with _CapturedStream() as cap:
            with pytest.raises(S.SlhaError) as e:
                call()
            assert e.value.code == S.ERR_DEVICE
        assert not cap.captured
        call()
        S.synchronize()
        assert np.array_equal(out.download(F, nq * n).reshape(nq, n), want)


def test_dense_calls_of_different_shapes_queued_behind_one_another():
    # more calls in flight on one stream than the library keeps table slots for, each with tables of its own, some of them large
    import ctypes as C

    tiles = np.tile(H.random_tiles(3000, 4, seed=550), 12)
    qc, qs = H.random_queries(40, 551)
    dt, dq, ds = S.to_device(tiles), S.to_device(qc), S.to_device(qs)
    rng = np.random.default_rng(552)
    shapes = [(int(rng.integers(1, 30000)), int(rng.integers(1, 41))) for _ in range(9)] + [(32000, 9)]
    jobs = []
    for n, nq in shapes:
        parts = 30000 if n > 30000 else min(n, 3)  # (30 000 segments: tables of more than a megabyte)
        cut = np.linspace(0, n, parts + 1).astype(int)
        rows = [(cut[i], cut[i + 1] - cut[i], 0, nq, cut[i]) for i in range(parts)]
        jobs.append((n, nq, S.make_segments(rows), np.arange(nq, dtype=np.uint64) * n, S.DeviceBuffer(nq * n * 4)))
    rt, stream = C.CDLL("libcudart.so.12"), C.c_void_p()
    assert rt.cudaStreamCreateWithFlags(C.byref(stream), 1) == 0
    S.set_stream(stream.value)
    try:
        for n, nq, seg, off, out in jobs:
            S.score_segments(dt, seg, dq, ds, nq, out, off, n)
        S.synchronize()
    finally:
        S.set_stream(None)
        rt.cudaStreamDestroy(stream)
    for n, nq, _, _, out in jobs:
        got = out.download(F, nq * n).reshape(nq, n)
        for j in range(nq):
            want = ora.score_tiles(tiles[:n], qc[j], qs[j])
            assert np.all(np.abs(got[j] - want) <= 1e-4 * (1 + np.abs(want)))
