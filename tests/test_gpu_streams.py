"""One thread, several streams: the library's working memory (scratch arena, plans, table slots) is kept per thread, so a call on
another stream has to wait for the work that still uses it.  All arguments lie in device memory: nothing else waits."""
import ctypes as C

import numpy as np
import pytest

from tests import helpers as H

pytestmark = pytest.mark.gpu
S = pytest.importorskip("slhav2_b200")
F = np.float32


class Streams:
    """Streams of the CUDA runtime, made and destroyed here."""

    def __init__(self, n):
        S.load_library()
        self.rt = C.CDLL("libcudart.so.12")
        self.all = [self.make() for _ in range(n)]

    def make(self):
        s = C.c_void_p()
        assert self.rt.cudaStreamCreateWithFlags(C.byref(s), 1) == 0
        return s

    def __enter__(self):
        return self

    def __exit__(self, *exc):
        S.set_stream(None)
        for s in self.all:
            self.rt.cudaStreamSynchronize(s)
            self.rt.cudaStreamDestroy(s)
        self.rt.cudaGetLastError()  # (of a test that failed)


class Job:
    """A score_topk call with its own queries and outputs on the device."""

    def __init__(self, tiles, n, nq, k, seed):
        self.args = tiles, S.make_segments([(0, n, 0, nq, 0)])
        qc, qs = H.random_queries(nq, seed)
        self.q = S.to_device(qc), S.to_device(qs)
        self.nq, self.k = nq, k
        self.out = S.DeviceBuffer(nq * k * 4), S.DeviceBuffer(nq * k * 4), S.DeviceBuffer(nq * 4)

    def run(self):
        S.score_topk(*self.args, *self.q, self.nq, self.k, *self.out)

    def result(self):
        m = self.nq * self.k
        return self.out[0].download(np.uint32, m), self.out[1].download(F, m), self.out[2].download(np.uint32, self.nq)

    def clear(self):
        for b in self.out:
            b.upload(np.zeros(b.nbytes // 4, np.uint32))


@pytest.mark.parametrize("codec", [1, 5])
@pytest.mark.parametrize("shapes", [1, 6])
def test_calls_of_one_thread_that_alternate_between_streams(codec, shapes):
    # the same plan from two streams in turn, and (six shapes, four plans) plans rebuilt while another stream may still use them
    n = 240000
    tiles = S.to_device(np.tile(H.random_tiles(4000, codec, seed=700 + codec, warm_every=7), n // 4000))
    jobs = [Job(tiles, n - 5000 * (i % shapes), 4, 100, 710 + i) for i in range(12)]
    want = []
    for j in jobs:
        j.run()
        S.synchronize()
        want.append(j.result())
        j.clear()
    with Streams(2) as st:
        for _ in range(3):
            for i, j in enumerate(jobs):
                S.set_stream(st.all[i % 2].value)
                j.run()
            for s in st.all:
                assert st.rt.cudaStreamSynchronize(s) == 0
            S.set_stream(None)
            for j, w in zip(jobs, want):
                for a, b in zip(j.result(), w):
                    assert np.array_equal(a, b)
                j.clear()


def test_a_stream_that_was_destroyed_and_one_made_after_it():
    # the new stream may get the old one's handle; the destroyed one's work still runs
    n = 240000
    tiles = S.to_device(np.tile(H.random_tiles(4000, 2, seed=720), n // 4000))
    jobs = [Job(tiles, n, 4, 64, 730 + i) for i in range(8)]
    want = []
    for j in jobs:
        j.run()
        S.synchronize()
        want.append(j.result())
        j.clear()
    with Streams(0) as st:
        for j in jobs:
            s = st.make()
            S.set_stream(s.value)
            j.run()
            assert st.rt.cudaStreamDestroy(s) == 0
        S.set_stream(None)
        assert st.rt.cudaDeviceSynchronize() == 0
    for j, w in zip(jobs, want):
        for a, b in zip(j.result(), w):
            assert np.array_equal(a, b)


def test_score_topk_is_captured_after_calls_on_another_stream():
    # warm-up on one stream, capture on another: the call may neither wait for work outside the graph nor be refused
    n = 50000
    tiles = S.to_device(np.tile(H.random_tiles(5000, 3, seed=740), n // 5000))
    job = Job(tiles, n, 4, 32, 741)
    with Streams(2) as st:
        S.set_stream(st.all[0].value)
        job.run()
        S.synchronize()
        want = job.result()
        job.clear()
        rt, graph, exe = st.rt, C.c_void_p(), C.c_void_p()
        S.set_stream(st.all[1].value)
        assert rt.cudaStreamBeginCapture(st.all[1], 2) == 0
        job.run()
        assert rt.cudaStreamEndCapture(st.all[1], C.byref(graph)) == 0
        assert rt.cudaGraphInstantiate(C.byref(exe), graph, C.c_ulonglong(0)) == 0
        for _ in range(3):
            assert rt.cudaGraphLaunch(exe, st.all[1]) == 0 and rt.cudaStreamSynchronize(st.all[1]) == 0
            S.set_stream(None)
            for a, b in zip(job.result(), want):
                assert np.array_equal(a, b)
            job.clear()
        S.set_stream(st.all[0].value)
        job.run()
        S.synchronize()
        S.set_stream(None)
        for a, b in zip(job.result(), want):
            assert np.array_equal(a, b)
        rt.cudaGraphExecDestroy(exe)
        rt.cudaGraphDestroy(graph)


def test_a_sharded_step_outlives_the_plans_of_other_shapes():
    # the repeated step is a graph over a plan's buffers; five other shapes rebuild all four plans, then the step comes again
    n, nq, k = 60000, 4, 40
    tiles = S.to_device(np.tile(H.random_tiles(5000, 1, seed=750), n // 5000))
    job = Job(tiles, n, nq, k, 751)
    others = [Job(tiles, n - 7000 * (i + 1), 4, 500, 760 + i) for i in range(5)]
    shard = S.Shard(None, 0, 1)
    job.run()
    S.synchronize()
    want = job.result()
    with Streams(1) as st:
        for _ in range(2):
            S.set_stream(st.all[0].value)
            for _ in range(4):  # plain, captured, replayed twice
                job.clear()
                shard.score_topk(*job.args, *job.q, nq, k, *job.out[:2])
                S.synchronize()
                for a, b in zip(job.result()[:2], want):
                    assert np.array_equal(a, b)
            for o in others:
                o.run()
            S.synchronize()
    shard.destroy()


def test_a_new_plan_is_not_made_under_capture():
    # its tables come from host memory that goes away with the call; a pool knows its codec, so no look at a tile stops the call earlier
    n = 3000
    pool = S.TilePool(n + 64, 2**40)
    model = S.Model.from_projection(H.make_model_pair(128)[1], 128, 7)
    pool.append_keys(model, H.gaussian_keys(770, n, 128), S.CODEC_MIXED, want_slots=False)
    qc, qs = H.random_queries(2, 771)
    dq, ds = S.to_device(qc), S.to_device(qs)
    out = S.DeviceBuffer(2 * 29 * 4), S.DeviceBuffer(2 * 29 * 4), S.DeviceBuffer(8)
    with Streams(1) as st:
        graph = C.c_void_p()
        S.set_stream(st.all[0].value)
        assert st.rt.cudaStreamBeginCapture(st.all[0], 2) == 0
        with pytest.raises(S.SlhaError) as e:
            pool.score_topk(dq, ds, 2, 29, *out)
        assert e.value.code == S.ERR_DEVICE
        st.rt.cudaStreamEndCapture(st.all[0], C.byref(graph))
        st.rt.cudaGetLastError()
        assert not graph.value
        pool.score_topk(dq, ds, 2, 29, *out)
        S.synchronize()
        idx = out[0].download(np.uint32, 58).reshape(2, 29)
    want = pool.score_topk(qc, qs, 2, 29)
    assert np.array_equal(idx, want[0])


def test_a_merge_on_a_second_stream_runs_beside_the_scoring_on_the_first():
    # a pipelined step: the merge uses no plan and no scratch, so it may not wait for score calls queued before it
    n, nq, k = 1 << 22, 4, 64
    tiles = S.to_device(np.tile(H.random_tiles(4096, 1, seed=780), n // 4096))
    jobs = [Job(tiles, n, nq, k, 781 + i) for i in range(2)]
    for j in jobs:
        j.run()
    S.synchronize()
    lists = 2
    cand_i = S.to_device(np.concatenate([j.result()[0] for j in jobs]))
    cand_s = S.to_device(np.concatenate([j.result()[1] for j in jobs]))
    out = S.DeviceBuffer(nq * k * 4), S.DeviceBuffer(nq * k * 4)
    S.topk_merge(cand_i, cand_s, lists, nq, k, k, *out)
    S.synchronize()
    want = out[0].download(np.uint32, nq * k), out[1].download(F, nq * k)
    with Streams(2) as st:
        for _ in range(3):
            S.set_stream(st.all[0].value)
            for _ in range(200):  # some 25 ms
                jobs[0].run()
            S.set_stream(st.all[1].value)
            S.topk_merge(cand_i, cand_s, lists, nq, k, k, *out)
            assert st.rt.cudaStreamSynchronize(st.all[1]) == 0
            assert st.rt.cudaStreamQuery(st.all[0]) == 600  # cudaErrorNotReady: the scoring still runs
            st.rt.cudaGetLastError()
            assert st.rt.cudaStreamSynchronize(st.all[0]) == 0
            assert np.array_equal(out[0].download(np.uint32, nq * k), want[0]) and np.array_equal(out[1].download(F, nq * k), want[1])
