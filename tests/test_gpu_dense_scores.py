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
        parts = 30000 if n > 30000 else (900 if n > 20000 else min(n, 3))  # (30 000 segments: tables of more than a megabyte; 900: of some 200 KB)
        cut = np.linspace(0, n, parts + 1).astype(int)
        rows = [(cut[i], cut[i + 1] - cut[i], 0, nq, cut[i]) for i in range(parts)]
        jobs.append((n, nq, S.make_segments(rows), np.arange(nq, dtype=np.uint64) * n, S.DeviceBuffer(nq * n * 4)))
    rt, stream = C.CDLL("libcudart.so.12"), C.c_void_p()
    assert rt.cudaStreamCreateWithFlags(C.byref(stream), 1) == 0
    S.set_stream(stream.value)
    try:
        for _ in range(4):
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


SPREADS = [1e-30, 1e-6, 1e-4, 1e-3, 0.088, 1.0, 1e3, 1e5, 1e20]


def _exact_terms(tiles, qc):
    """float64 scores of tiles without a residual term, [query][tile], and the sums of their terms' sizes."""
    lat = np.stack([ora.dequant(tiles[i:i + 1]) for i in range(len(tiles))]).astype(np.float64)
    q = qc.astype(np.float64)
    return q @ lat.T, np.abs(q) @ np.abs(lat).T


def _spread_inputs(codec, nq, seed):
    tiles = H.random_tiles(400, codec, seed=seed + codec, nocorr_every=5)
    tiles["dynamic_lambda"] = 0
    tiles["scale"][100:200] *= F(1e3)
    tiles["scale"][200:300] *= F(1e6)
    tiles["scale"][300:] *= F(1e-6)
    qc, qs = H.random_queries(nq, seed + 1)
    qc *= np.array([SPREADS[j % len(SPREADS)] for j in range(nq)], F)[:, None]
    qc[-1, 5] *= F(300.0)  # (one element far above the others)
    return tiles, qc, qs


# Bound: a query is held to 2^-22 of every element that matters, the levels are exact, and at most 20 sums of float32 are each
# off by 2^-23 of the terms so far (the reference's own latents by 3 x 2^-24): 2.7e-6 of the terms' sizes, whatever the query's size.
SCORE_BOUND = 3e-6


@pytest.mark.parametrize("codec", range(7))
@pytest.mark.parametrize("nq", [9, 18, 64])
def test_dense_scores_are_as_exact_for_small_and_large_queries(codec, nq):
    tiles, qc, qs = _spread_inputs(codec, nq, 560)
    n = len(tiles)
    dt = S.to_device(tiles)
    want, size = _exact_terms(tiles, qc)
    got = [S.score_segments(dt, S.make_segments([(0, n, 0, nq, 0)]), qc, qs, nq, np.zeros((nq, n), F), np.arange(nq, dtype=np.uint64) * n, n)]
    got += [np.concatenate([S.score_segments(dt, S.make_segments([(0, n, 0, 1, 0)]), qc[j:j + 1], qs[j:j + 1], 1, np.zeros((1, n), F), np.zeros(1, np.uint64), n)
                            for j in range(9)])]
    got += [S.score_tiles(S.to_device(np.tile(tiles, 82)), 82 * n, qc[:9], qs[:9], 9)[:, -n:]]
    for g in got:
        assert np.all(np.abs(g - want[:len(g)]) <= SCORE_BOUND * size[:len(g)] + 1e-44)


@pytest.mark.parametrize("codec,nq", [(5, 1), (5, 4), (5, 6)] + [(c, nq) for c in (0, 1, 3, 4, 5, 6) for nq in (18, 64)])
def test_top_k_scores_are_as_exact_for_small_and_large_queries(codec, nq):
    # the tile kernel's codec and the 64-row kernel's
    tiles, qc, qs = _spread_inputs(codec, 9 if nq < 9 else nq, 570)
    n = k = 100 - codec  # (plans are kept by shape, each for one codec)
    for part in range(4):  # (tiles of one scale at a time: the winners are all of them)
        own = tiles[100 * part:100 * part + n]
        dt = S.to_device(own)
        want, size = _exact_terms(own, qc)
        for q0 in range(0, len(qc), nq):
            m = min(nq, len(qc) - q0)
            idx, sc, cnt = S.score_topk(dt, S.make_segments([(0, n, 0, m, 0)]), qc[q0:q0 + m], qs[q0:q0 + m], m, k)
            assert np.all(cnt == k) and S.last_score_stats()["rows_handed_to_generic_kernel"] == 0
            rows = np.arange(q0, q0 + m)[:, None]
            assert np.all(np.sort(idx, 1) == np.arange(n))
            assert np.all(np.abs(sc - want[rows, idx]) <= SCORE_BOUND * size[rows, idx] + 1e-44)


@pytest.mark.parametrize("nq", [4, 17])
@pytest.mark.parametrize("value", [np.inf, -np.inf, np.nan, 1e30])
def test_query_rows_beyond_the_split_take_the_generic_kernel(nq, value):
    n, k = 700, 20
    tiles = H.random_tiles(n, 5, seed=580)
    qc, qs = H.random_queries(nq, 581)
    qc[2, 77] = value
    dt, seg = S.to_device(tiles), S.make_segments([(0, n, 0, nq, 0)])
    idx, sc, _ = S.score_topk(dt, seg, qc, qs, nq, k)
    assert S.last_score_stats()["rows_handed_to_generic_kernel"] == nq
    out = S.score_segments(dt, seg, qc, qs, nq, np.zeros((nq, n), F), np.arange(nq, dtype=np.uint64) * n, n)
    S.debug_force_generic_score(True)
    try:
        gi, gs, _ = S.score_topk(dt, seg, qc, qs, nq, k)
        gout = S.score_segments(dt, seg, qc, qs, nq, np.zeros((nq, n), F), np.arange(nq, dtype=np.uint64) * n, n)
    finally:
        S.debug_force_generic_score(False)
    assert np.array_equal(idx, gi) and np.array_equal(sc, gs, equal_nan=True)
    assert np.array_equal(out[:4], gout[:4], equal_nan=True)  # (dense: the group of four rows that holds it)
    assert np.all(np.abs(out[4:] - gout[4:]) <= 1e-4 * (1 + np.abs(gout[4:])))


@pytest.mark.parametrize("residual", [False, True])
@pytest.mark.parametrize("codec,nq", [(c, nq) for c in range(7) for nq in (1, 4)] + [(2, 20), (2, 64), (5, 20), (5, 64)])
def test_scores_are_no_further_from_64_bits_than_the_generic_kernels(codec, nq, residual):
    # the calls that tensor-core kernels took over from it (float32 products in short chains): 2-norm of the error over six sets of
    # tiles and queries, 5 % for chance (a single set's two errors differ by up to 12 % either way)
    n = 1500 + codec
    k = n // 3
    seg, off = S.make_segments([(0, n, 0, nq, 0)]), np.arange(nq, dtype=np.uint64) * n
    square = np.zeros((2, 2, 2))  # [dense, top-k][tensor cores, generic][error, size]
    for seed in range(590, 650, 10):
        tiles = H.random_tiles(n, codec, seed=seed + codec, nocorr_every=5)
        qc, qs = H.random_queries(nq, seed + 1)
        want = _exact_terms(tiles, qc)[0]
        # a residual a third of the key's size, or none
        tiles["dynamic_lambda"] = 0.0235 * want.std() / 128**0.5 if residual else 0
        lam = tiles["dynamic_lambda"].astype(np.float64)
        bits = np.unpackbits(np.ascontiguousarray(tiles["residual_bitmap"]).view(np.uint8).reshape(n, 32), axis=1)
        want += lam * np.stack([256.0 - 2.0 * (bits != np.unpackbits(q.view(np.uint8))).sum(1) for q in qs])
        dt = S.to_device(tiles)
        for generic in (0, 1):
            S.debug_force_generic_score(bool(generic))
            try:
                out = S.score_segments(dt, seg, qc, qs, nq, np.zeros((nq, n), F), off, n)
                idx, sc, _ = S.score_topk(dt, seg, qc, qs, nq, k)
            finally:
                S.debug_force_generic_score(False)
            w = want[np.arange(nq)[:, None], idx]
            square[0, generic] += ((out - want) ** 2).sum(), (want ** 2).sum()
            square[1, generic] += ((sc - w) ** 2).sum(), (w ** 2).sum()
    error = np.sqrt(square[:, :, 0] / square[:, :, 1])
    assert error[0, 0] <= 1.05 * error[0, 1], error
    assert codec != 5 or error[1, 0] <= 1.05 * error[1, 1], error  # (the other codecs' top-k always had kernels of their own)


def _generic(call):
    S.debug_force_generic_score(True)
    try:
        return call()
    finally:
        S.debug_force_generic_score(False)


@pytest.mark.parametrize("nq", [2, 16])
def test_segments_of_different_codecs_in_one_cta_are_decoded_each_as_its_own(nq):
    # 148 CTAs share about two thousand short segments of six codecs in turn: no row takes the generic kernel, whose sums differ in
    # their last bits.  (NF4 with 16 rows or more passes through the four-row kernel.)
    n_seg, lens = 1998, [17, 40, 129, 64, 5, 200]
    parts = [H.random_tiles(200, c, seed=600 + c, warm_every=5, nocorr_every=3) for c in (1, 3, 4, 5, 2, 6)]
    rows, chunks, tb = [], [], 0
    for i in range(n_seg):
        m = lens[(i // 6) % 6]
        chunks.append(parts[i % 6][:m])
        rows.append((tb, m, i * nq, nq, 0))
        tb += m
    tiles = np.concatenate(chunks)
    row_len = 200
    qc, qs = H.random_queries(n_seg * nq, 601)
    dt, seg, off = S.to_device(tiles), S.make_segments(rows), np.arange(n_seg * nq, dtype=np.uint64) * row_len
    call = lambda: S.score_segments(dt, seg, qc, qs, n_seg * nq, np.zeros((n_seg * nq, row_len), F), off, row_len)  # noqa: E731
    got, gen = call(), _generic(call)
    handed = 0
    for i, (t, m, q0, _, _) in enumerate(rows):
        a, b = got[q0:q0 + nq, :m], gen[q0:q0 + nq, :m]
        assert np.all(np.abs(a - b) <= 1e-4 * (1 + np.abs(b)))
        handed += m >= 40 and np.array_equal(a, b)
        assert np.all(got[q0:q0 + nq, m:] == 0)
        if i % 97 == 0:
            want = ora.score_tiles(tiles[t:t + m], qc[q0], qs[q0])
            assert np.all(np.abs(a[0] - want) <= 1e-4 * (1 + np.abs(want)))
    assert handed == 0


@pytest.mark.parametrize("codecs", [(1, 3), (5, 4), (2, 5), (0, 5)])
@pytest.mark.parametrize("nq", [3, 18])
def test_arenas_whose_tiles_change_codec_all_the_time(codecs, nq):
    # every block holds tiles of two codecs: the tensor-core kernels give such items up, the generic kernel scores them
    n = 33000
    a, b = (np.tile(H.random_tiles(500, c, seed=610 + c, warm_every=4), 66) for c in codecs)
    tiles = np.where((np.arange(n) % 3 == 1), b, a)
    qc, qs = H.random_queries(nq, 611)
    dt = S.to_device(tiles)
    idx, sc, _ = S.score_topk(dt, S.make_segments([(0, n, 0, nq, 0)]), qc, qs, nq, 50)
    out = S.score_segments(dt, S.make_segments([(0, n, 0, nq, 0)]), qc, qs, nq, np.zeros((nq, n), F), np.arange(nq, dtype=np.uint64) * n, n)
    full = S.score_tiles(dt, n, qc, qs, nq)
    for j in range(nq):
        want = ora.score_tiles(tiles, qc[j], qs[j])
        for o in (out[j], full[j]):
            assert np.all(np.abs(o - want) <= 1e-4 * (1 + np.abs(want)))
        assert np.all(np.abs(sc[j] - np.sort(want)[::-1][:50]) <= 1e-3) and np.all(np.abs(sc[j] - want[idx[j]]) <= 1e-3)


def test_a_pool_of_nf4_and_int4_tiles_is_scored_in_one_pass():
    # tiles of both in every CTA's share: the kind that decodes both takes all of them (the generic kernel's sums differ in their last bits)
    n = 36000
    model = S.Model.from_projection(H.make_model_pair(128)[1], 128, 7)
    keys = H.gaussian_keys(620, 1500, 128, outlier_channels=(7, 93))
    qc, qs = H.random_queries(1, 621)
    for first, second in ((S.CODEC_INT4_GROUPED, S.CODEC_NF4), (S.CODEC_NF4, S.CODEC_INT4_SINGLE)):
        pool = S.TilePool(n, 2**40)
        for i in range(n // 1500):
            pool.append_keys(model, keys, (first, second)[i % 2], want_slots=False)
        slots, got = pool.score_all(qc[0], qs[0])
        gen = _generic(lambda: pool.score_all(qc[0], qs[0]))[1]
        tiles = pool.read()[0]
        want = ora.score_tiles(tiles, qc[0], qs[0])
        assert np.array_equal(slots, np.arange(n)) and np.all(np.abs(got - want) <= 1e-4 * (1 + np.abs(want)))
        nf4 = (tiles["flags"] & S.FLAG_NF4) != 0
        assert nf4.mean() == 0.5
        for part in (nf4, ~nf4):
            for b in range(0, n, 3000):
                own = part[b:b + 3000]
                assert not np.array_equal(got[b:b + 3000][own], gen[b:b + 3000][own])
        # the same tiles in an arena of the caller's whose first tile is an NF4 tile
        arena = tiles[np.argsort(~nf4[:1500 * 2], kind="stable")]
        arena = np.tile(arena, 12)
        call = lambda: S.score_tiles(S.to_device(arena), len(arena), qc, qs, 1)  # noqa: E731
        assert not np.array_equal(call()[0][-3000:], _generic(call)[0][-3000:])


@pytest.mark.parametrize("nq,n", [(1, 5000), (4, 9000), (20, 3000)])
def test_int4_tiles_of_the_shape_of_an_earlier_mix3_call_stay_on_the_tensor_cores(nq, n):
    # plans are kept by shape: the one made for MIX3 tiles decodes INT4 / MX-INT4 tiles too, and MIX3 again after them
    k = 33
    qc, qs = H.random_queries(nq, 630)
    seg = S.make_segments([(0, n, 0, nq, 0)])
    for codec in (5, 1, 6, 0, 5):
        tiles = np.tile(H.random_tiles(1000, codec, seed=631 + codec, warm_every=6), n // 1000)
        idx, sc, cnt = S.score_topk(S.to_device(tiles), seg, qc, qs, nq, k)
        assert S.last_score_stats()["rows_handed_to_generic_kernel"] == 0
        for j in range(nq):
            want = ora.score_tiles(tiles, qc[j], qs[j])
            assert cnt[j] == k and np.all(np.abs(sc[j] - np.sort(want)[::-1][:k]) <= 1e-3) and np.all(np.abs(sc[j] - want[idx[j]]) <= 1e-3)


@pytest.mark.parametrize("nq,codec", [(1, 0), (4, 5), (20, 3), (20, 2), (300, 0)])
@pytest.mark.parametrize("tail", [0, 7])
def test_row_offsets_in_device_memory_are_checked_there(nq, codec, tail):
    # the same scores as with offsets in host memory; a row that reaches beyond the destination refuses the call, and no row is written
    n = 700
    tiles = S.to_device(H.random_tiles(n, codec, seed=540 + codec))
    qc, qs = H.random_queries(nq, 541)
    dq, ds = S.to_device(qc), S.to_device(qs)
    seg, row = S.make_segments([(0, n, 0, nq, 0)]), n + tail
    off = np.random.default_rng(nq).permutation(nq).astype(np.uint64) * row
    want = S.score_segments(tiles, seg, dq, ds, nq, np.zeros(nq * row, F), off, row, fill=-3.0)
    out = S.to_device(np.full(nq * row, 9.0, F))
    S.score_segments(tiles, seg, dq, ds, nq, out, S.to_device(off), row, fill=-3.0)
    assert np.array_equal(out.download(F, nq * row), want)
    for bad in (1, 2**63, 2**64 - row):  # (one element too far, and sums that wrap around)
        wrong = off.copy()
        wrong[nq // 2] = (int(wrong.max()) + bad) % 2**64 if bad == 1 else bad
        out = S.to_device(np.full(nq * row, 9.0, F))
        host = np.full(nq * row, 9.0, F)
        for dst in (out, host):
            with pytest.raises(S.SlhaError) as e:
                S.score_segments(tiles, seg, dq, ds, nq, dst, S.to_device(wrong), row, fill=-3.0)
            assert e.value.code == S.ERR_DIMENSION
        assert np.all(out.download(F, nq * row) == 9.0) and np.all(host == 9.0)
    S.score_segments(tiles, seg, dq, ds, nq, out, S.to_device(off), row, fill=-3.0)  # a refused call leaves nothing behind
    assert np.array_equal(out.download(F, nq * row), want)


@pytest.mark.parametrize("nq,per_cta", [(1, 80), (16, 20)])
def test_segments_that_are_left_to_the_generic_arithmetic_leave_the_others_as_they_are(nq, per_cta):
    # more such segments in a CTA (148 SMs) than a short list holds, every second one: the rows of the others keep their bits, in dense calls and in top-k
    m, n_seg = 5, 148 * per_cta
    base = H.random_tiles(1000, 3, seed=540)
    tiles = base[np.random.default_rng(nq).integers(0, 1000, m * n_seg)]
    mixed = tiles.copy()
    odd = np.repeat(np.arange(n_seg) % 2 == 1, nq)
    mixed[m + 2::2 * m] = np.resize(H.random_tiles(100, 4, seed=541), n_seg // 2)
    total = nq * n_seg
    qc, qs = (np.resize(x, (total,) + x.shape[1:]) for x in H.random_queries(97, 542))
    seg = S.make_segments([(m * i, m, nq * i, nq, 0) for i in range(n_seg)])
    off = np.arange(total, dtype=np.uint64) * m

    def run(t):
        dt = S.to_device(t)
        dense = S.score_segments(dt, seg, qc, qs, total, np.zeros((total, m), F), off, m)
        idx, sc, _ = S.score_topk(dt, seg, qc, qs, total, m)
        return dense, idx, sc, S.last_score_stats()["rows_handed_to_generic_kernel"]

    clean, now = run(tiles), run(mixed)
    assert clean[3] == 0 and now[3] == odd.sum()
    for a, b in zip(clean[:3], now[:3]):
        assert a[~odd].tobytes() == b[~odd].tobytes()
    for i in range(1, n_seg, 97):
        if i % 2:
            for j in (nq * i, nq * i + nq - 1):
                want = ora.score_tiles(mixed[m * i:m * i + m], qc[j], qs[j])
                assert np.all(np.abs(now[0][j] - want) <= 1e-3 * (1 + np.abs(want))) and np.all(np.abs(now[2][j] - want[now[1][j]]) <= 1e-3)


def test_nf4_rows_of_many_queries_cost_what_the_same_rows_cost_four_at_a_time():
    # 40 rows a segment, handed on by the 64-row kernel and cut into equal shares again: shares end inside groups of four rows and at ragged ends
    import time

    n, nq, base = 20_013, 40, 9
    tiles = H.random_tiles(2 * n, 2, seed=550, warm_every=11)
    qc, qs = H.random_queries(2 * nq, 551)
    dt, dq, ds = S.to_device(tiles), S.to_device(qc), S.to_device(qs)
    row_len = n + base
    off = S.to_device(np.arange(2 * nq, dtype=np.uint64) * row_len)
    whole = S.make_segments([(0, n, 0, nq, base), (n, n, nq, nq, base)])
    fours = S.make_segments([(i // 10 * n, n, 4 * i, 4, base) for i in range(20)])
    outs, took = [], []
    for seg in (whole, fours):
        out = S.DeviceBuffer(2 * nq * row_len * 4)
        out.upload(np.zeros(2 * nq * row_len, F))
        for rep in range(2):
            S.synchronize()
            t = []
            for _ in range(30):
                t0 = time.perf_counter()
                S.score_segments(dt, seg, dq, ds, 2 * nq, out, off, row_len)
                S.synchronize()
                t.append(time.perf_counter() - t0)
        took.append(float(np.median(t)))
        outs.append(out.download(F, 2 * nq * row_len).reshape(2 * nq, row_len))
    assert outs[0].tobytes() == outs[1].tobytes()
    for j in (0, 3, 39, 40, 77):
        want = ora.score_tiles(tiles[j // nq * n:j // nq * n + n], qc[j], qs[j])
        assert np.all(np.abs(outs[0][j, base:] - want) <= 1e-3 * (1 + np.abs(want)))
    assert took[0] < 1.6 * took[1], took


def test_segments_that_continue_one_another_in_the_tiles_but_not_in_the_row():
    # NF4 rows of two segments each: the second takes the tiles behind the first's and writes them elsewhere in the row, beside ones that do go on
    n, nq, row_len = 700, 16, 4000
    tiles = H.random_tiles(4 * n, 2, seed=560)
    qc, qs = H.random_queries(2 * nq, 561)
    rows = [(0, n, 0, nq, 0), (n, n, 0, nq, 2000), (2 * n, n, nq, nq, 100), (3 * n, n, nq, nq, 100 + n)]
    out = S.score_segments(S.to_device(tiles), S.make_segments(rows), qc, qs, 2 * nq, np.zeros((2 * nq, row_len), F), np.arange(2 * nq, dtype=np.uint64) * row_len, row_len)
    for tb, m, q0, q, base in rows:
        for j in range(q0, q0 + q, 5):
            want = ora.score_tiles(tiles[tb:tb + m], qc[j], qs[j])
            assert np.all(np.abs(out[j, base:base + m] - want) <= 1e-3 * (1 + np.abs(want)))


@pytest.mark.parametrize("n_seg,longest,share,huge", [(40, 3000, 0.5, 0), (700, 200, 0.3, 0), (9, 20000, 0.12, 0), (600, 40, 1.0, 0), (12, 9000, 0.3, 0.5), (800, 150, 0.1, 0.2), (1, 700, 0, 1), (3, 16384, 0, 1)])
def test_what_was_handed_on_is_shared_out_whatever_lies_between(n_seg, longest, share, huge):
    # segments of 16 to 70 rows, some of them NF4, some with a query row beyond the fp16 split (handed on by the 64-row kernel, in groups of unequal cost): those give what the same rows give in
    # fours, bit for bit, the others the oracle's scores
    rng = np.random.default_rng(n_seg)
    nf4 = rng.random(n_seg) < share
    base = {c: H.random_tiles(1000, c, seed=570 + c, warm_every=9) for c in (0, 2, 3, 5)}
    rows, fours, parts, tb, qb = [], [], [], 0, 0
    for i in range(n_seg):
        n, nq = int(rng.integers(1, longest + 1)), int(rng.choice([16, 17, 40, 64, 70]))
        parts.append(base[2 if nf4[i] else int(rng.choice([0, 3, 5]))][rng.integers(0, 1000, n)])
        rows.append((tb, n, qb, nq, 0))
        fours += [(tb, n, qb + q, min(4, nq - q), 0) for q in range(0, nq, 4)]
        tb, qb = tb + n, qb + nq
    tiles = np.concatenate(parts)
    qc, qs = (np.resize(x, (qb,) + x.shape[1:]) for x in H.random_queries(211, 571))
    far, of_far = [], np.zeros(qb, bool)
    for i in np.flatnonzero(rng.random(n_seg) < huge):
        j = int(rng.integers(0, rows[i][3]))
        far.append(rows[i][2] + j)
        qc[far[-1], int(rng.integers(0, 100))] = rng.choice([1e30, -np.inf, np.nan])
        of_far[rows[i][2] + j // 64 * 64:min(rows[i][2] + j // 64 * 64 + 64, rows[i][2] + rows[i][3])] = True
    row_len = max(r[1] for r in rows)
    off = np.arange(qb, dtype=np.uint64) * row_len
    dt = S.to_device(tiles)
    out = S.score_segments(dt, S.make_segments(rows), qc, qs, qb, np.zeros((qb, row_len), F), off, row_len)
    want = S.score_segments(dt, S.make_segments(fours), qc, qs, qb, np.zeros((qb, row_len), F), off, row_len)
    of_nf4 = np.repeat(nf4, [r[3] for r in rows])
    handed = of_nf4 | of_far
    assert out[handed].tobytes() == want[handed].tobytes()
    usual = np.setdiff1d(np.arange(qb), far)
    assert np.all(np.abs(out[usual] - want[usual]) <= 1e-4 * (1 + np.abs(want[usual])))
    for i in range(0, n_seg, max(1, n_seg // 12)):
        t, n, q0, nq, _ = rows[i]
        for j in set((q0, q0 + nq - 1)) - set(far):
            s = ora.score_tiles(tiles[t:t + n], qc[j], qs[j])
            assert np.all(np.abs(out[j, :n] - s) <= 1e-3 * (1 + np.abs(s))) and np.all(out[j, n:] == 0)
