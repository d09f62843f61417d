"""The budget question of a decode step, settled by one kernel (pool.cu, enforce_step_kernel): the same slots, states, bytes and order of freed
slots as the phases run one by one from the host give, on both sides of every condition under which the kernel leaves the work to the others."""
import ctypes as C

import numpy as np
import pytest

from tests import helpers as H
from tests.test_gpu_streams import Streams

pytestmark = pytest.mark.gpu
S = pytest.importorskip("slhav2_b200")
F = np.float32


@pytest.mark.parametrize("page,evict,recent,n", [(0, 0, 0, 1), (1, 1, 0, 511), (0, 1, 300, 513), (1, 0, 0, 9000), (1, 1, 100, 9001), (1, 1, 2000, 80000), (0, 1, 75000, 80000)])
def test_a_step_gives_what_the_host_driven_phases_give(page, evict, recent, n):
    rng = np.random.default_rng(n + 10 * page + evict)
    gm = S.Model.from_projection(H.make_model_pair(128, seed=61)[1], 128, 61)
    room = 30000
    keys = H.gaussian_keys(62, 4096, 128)
    pools = [S.TilePool(n + room, 2**40, page, evict, 4, recent) for _ in range(2)]
    at = 0

    def append(m):
        nonlocal at
        pos = ((at + np.arange(m)) // 2).astype(np.uint32)
        which = rng.integers(0, len(keys), m)
        got = [p.append_keys(gm, keys[which], S.CODEC_MIXED if at % 2 else S.CODEC_NF4, positions=pos) for p in pools]
        assert np.array_equal(*got)  # (slots that were freed are taken again in the same order)
        at += m

    def step(budget):
        within = []
        for i, p in enumerate(pools):
            p.set_budget(max(0, int(budget)))
            S.debug_force_generic_score(bool(i))
            try:
                within.append(p.enforce_budget())
            finally:
                S.debug_force_generic_score(False)
        assert within[0] == within[1]
        assert pools[0].stats() == pools[1].stats()

    def live():
        return pools[0].stats()["live_bytes"]

    for b in range(0, n, 50000):
        append(min(50000, n - b))
    sc = (rng.standard_normal(n) * 3).astype(F)
    for p in pools:
        if n != 9001:  # (all of one importance: their keys lie in the slots' order)
            p.observe_scores(np.arange(n, dtype=np.uint32), sc, 0.9)
    step(live())                              # within the budget: nothing
    if n <= 4096:
        step(live() - 32 * (n // 2) - 1)      # page-outs from a list that fits, not all of them
    step(live() - 32 * 7)                     # (more HOT tiles than the list holds, or what is left of them)
    step(96 * n)                              # the rest of the page-outs
    step(96 * n - 1)                          # one eviction
    for m in (1, 8, 40):
        append(m)
        step(live() - 32 * m)                 # exactly the page-outs
        append(m)
        step(live() - 32 * m - 96 * m)        # and evictions
        append(m)
        step(live() - 16 * m)                 # half of the page-outs
    append(5)
    step(live() - 32 * 45 - 80 * 120)         # more evictions than the blocks' smallest keys are kept for (148 blocks)
    append(4097)
    step(live() - 32 * 3)                     # one HOT tile more than the list holds
    step(live() - 32 * 4097)
    append(600)
    step(live() - 32 * 600 - 96 * 3)
    for _ in range(3):                        # down to the slots that only the last phase takes, and to nothing
        step(live() // 2)
    step(96 * 5)
    step(96)
    step(0)
    append(3)
    step(96 * 2)
    for a, b in zip(pools[0].read(), pools[1].read()):
        assert a.tobytes() == b.tobytes()


@pytest.mark.parametrize("n", [1, 15, 256, 257, 65537, 16 * 65536, 16 * 65536 + 1])
def test_observing_a_query_is_observing_its_scores(n):
    # up to 16 x 65 536 slots by one kernel, from there on by three, like a list of slots, in the same order; the counts of both forms of the statistics
    gm = S.Model.from_projection(H.make_model_pair(128, seed=61)[1], 128, 61)
    base = H.gaussian_keys(64, 2048, 128)
    pools = [S.TilePool(n, 2**40) for _ in range(2)]
    for b in range(0, n, 262144):
        keys = np.resize(base, (min(262144, n - b), 128))
        for p in pools:
            p.append_keys(gm, keys, S.CODEC_MIXED)
    qc, qs = H.random_queries(1, 7)
    gone = np.unique(np.array([0, n // 3, n // 2]) % n) if n > 1 else []
    for p in pools:
        for s in gone:
            p.evict(int(s))
    slots, scores = pools[0].score_all(qc, qs)
    pools[0].observe_query(qc, qs, 20.0)
    pools[1].observe_scores(slots, scores, 20.0)
    a, b = pools[0].read()[2], pools[1].read()[2]
    live = np.ones(n, bool)
    live[list(gone)] = False
    assert np.allclose(a[live], b[live], rtol=3e-5, atol=1e-44)  # (a list leaves out COLD slots, so its shares are others: 16 terms a thread, a tree, 256 sums, each way 2^-24 x 280; subnormal weights: their spacing)
    assert abs(float(a[live].astype(np.float64).sum()) - 1.0) < 1e-4
    st = pools[0].stats()
    assert (st["hot"], st["warm"], st["cold"], st["len"]) == (n - len(gone), 0, len(gone), n)
    extra = S.TilePool(40, 2**40)
    extra.insert(H.random_tiles(33, 4, seed=3, nocorr_every=5))
    st = extra.stats()
    assert st["hot"] == 33 and st["nocorr"] == 7


@pytest.mark.parametrize("nq,k", [(1, 1), (256, 1), (257, 1), (4, 64), (5, 64)])
def test_short_host_outputs(nq, k):
    # 1024 bytes are the most that kernels write to the host's page
    tiles = H.random_tiles(300, 0, seed=9)
    pool = S.TilePool(300, 2**40)
    pool.insert(tiles)
    qc, qs = H.random_queries(nq, 11)
    gi, gs, gc = pool.score_topk(qc, qs, nq, k)
    di, ds, dc = S.DeviceBuffer(nq * k * 4), S.DeviceBuffer(nq * k * 4), S.DeviceBuffer(nq * 4)
    pool.score_topk(S.to_device(qc), S.to_device(qs), nq, k, di, ds, dc)
    S.synchronize()
    assert np.array_equal(np.asarray(gi).reshape(-1), di.download(np.uint32, nq * k)) and np.array_equal(np.asarray(gs).reshape(-1), ds.download(F, nq * k))
    assert np.array_equal(gc, dc.download(np.uint32, nq)) and np.all(gc == k)


def test_observing_a_query_is_captured_before_any_other_call():
    # a graph made by the pool's first such call, launched behind and before calls that are not
    gm = S.Model.from_projection(H.make_model_pair(128, seed=61)[1], 128, 61)
    pools = [S.TilePool(3000, 2**40) for _ in range(2)]
    for p in pools:
        p.append_keys(gm, H.gaussian_keys(65, 3000, 128), S.CODEC_MIXED)
    qc, qs = H.random_queries(1, 12)
    dq, ds = S.to_device(qc), S.to_device(qs)
    with Streams(1) as st:
        rt, graph, exe = st.rt, C.c_void_p(), C.c_void_p()
        S.set_stream(st.all[0].value)
        pools[1].observe_query(dq, ds, 3.0)  # (the thread's scratch)
        assert rt.cudaStreamBeginCapture(st.all[0], 2) == 0
        pools[0].observe_query(dq, ds, 3.0)
        assert rt.cudaStreamEndCapture(st.all[0], C.byref(graph)) == 0
        assert rt.cudaGraphInstantiate(C.byref(exe), graph, C.c_ulonglong(0)) == 0
        for direct in (True, False, True, False):
            if direct:
                pools[0].observe_query(dq, ds, 3.0)
            else:
                assert rt.cudaGraphLaunch(exe, st.all[0]) == 0
        for _ in range(3):
            pools[1].observe_query(dq, ds, 3.0)
        S.synchronize()
        rt.cudaGraphExecDestroy(exe)
        rt.cudaGraphDestroy(graph)
        S.set_stream(None)
    assert pools[0].read()[2].tobytes() == pools[1].read()[2].tobytes()


def test_a_pool_is_driven_from_two_streams_in_turn():
    # every call of a step on the other stream than the one before it, as soon as that has given its answer; budgets that are met and that are not
    gm = S.Model.from_projection(H.make_model_pair(128, seed=61)[1], 128, 61)
    keys = H.gaussian_keys(66, 4096, 128)
    pools = [S.TilePool(150_000, 2**40, 1, 1, 4, 50) for _ in range(2)]
    with Streams(2) as st:
        for p in pools:
            turn = 0

            def other():
                nonlocal turn
                turn ^= p is pools[0]
                S.set_stream(st.all[turn].value)

            for i in range(30):
                p.append_keys(gm, keys, S.CODEC_MIXED, position_base=4096 * i)
            S.synchronize()
            for i in range(60):
                live = p.stats()["live_bytes"]
                p.set_budget(live + 1000 if i % 3 else live - 32 * 8 - 96 * 3)
                assert p.enforce_budget()
                other()
                p.append_keys(gm, keys[:8], S.CODEC_MIXED, position_base=130_000 + i)
                S.synchronize()
                p.set_budget(2**40)
                assert p.enforce_budget()
                other()
                p.append_keys(gm, keys[8:9], S.CODEC_MIXED, position_base=140_000 + i)
                S.synchronize()
    assert pools[0].stats() == pools[1].stats()
    for a, b in zip(pools[0].read(), pools[1].read()):
        assert a.tobytes() == b.tobytes()


def test_refused_calls_leave_the_page_for_short_outputs_free():
    # a thread's calls take no longer after hundreds of refused ones (through the device and a copy an output, as without the page, twice as long)
    import time

    tiles = H.random_tiles(4096, 0, seed=9)
    qc, qs = H.random_queries(1, 11)
    dt, dq, ds = S.to_device(tiles), S.to_device(qc), S.to_device(qs)
    good, bad = S.make_segments([(0, 4096, 0, 1, 0)]), S.make_segments([(0, 4096, 0, 1, 0), (0, 100, 0, 1, 0)])
    out = np.zeros((1, 64), np.uint32), np.zeros((1, 64), F), np.zeros(1, np.uint32)

    def took():
        t = []
        for _ in range(300):
            t0 = time.perf_counter()
            S.score_topk(dt, good, dq, ds, 1, 64, *out)
            t.append(time.perf_counter() - t0)
        return float(np.median(t))

    took()
    before = took()
    for _ in range(300):
        with pytest.raises(S.SlhaError):
            S.score_topk(dt, bad, dq, ds, 1, 64, *out)
        with pytest.raises(S.SlhaError):
            S.score_topk(dt, good, dq, ds, 1, 5000, np.zeros((1, 5000), np.uint32), np.zeros((1, 5000), F), out[2])
    after = took()
    assert after < 1.5 * before, (before, after)


_SLEEPER = """
import ctypes, sys, time
rt = ctypes.CDLL("libcudart.so.12")
assert rt.cudaSetDevice(0) == 0 and rt.cudaSetDeviceFlags(4) == 0  # cudaDeviceScheduleBlockingSync
import numpy as np
import slhav2_b200 as S
from tests import helpers as H
from tests.test_gpu_streams import Streams
gm = S.Model.from_projection(H.make_model_pair(128, seed=61)[1], 128, 61)
keys = S.to_device(np.resize(H.gaussian_keys(67, 4096, 128), (262144, 128)))
out = S.DeviceBuffer(262144 * 128)
pool = S.TilePool(1000, 2**40)
pool.append_keys(gm, H.gaussian_keys(68, 900, 128), S.CODEC_MIXED)
with Streams(1) as st:
    S.set_stream(st.all[0].value)
    for call in (pool.stats, pool.enforce_budget):
        call()
        worst = 0.0
        for _ in range(3):
            for _ in range(60):
                gm.encode_keys(keys, S.CODEC_NF4, n=262144, out=out)
            wall, cpu = time.perf_counter(), time.thread_time()
            call()
            wall, cpu = time.perf_counter() - wall, time.thread_time() - cpu
            assert wall > 0.01, wall
            worst = max(worst, cpu / wall)
        print(call.__name__, worst)
        assert worst < 0.3, (call.__name__, worst)
"""


def test_a_thread_that_is_to_sleep_while_it_waits_does():
    # calls behind 60 encodes of 0.7 ms, in a process whose device has cudaDeviceScheduleBlockingSync
    import os
    import subprocess
    import sys

    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", _SLEEPER], cwd=root, capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr


@pytest.mark.parametrize("n,evict,skewed", [(500_003, 1, False), (500_003, 1, True), (16 * 148 * 512 - 1, 1, False), (16 * 148 * 512, 0, False), (16 * 148 * 512 + 1, 1, False)])
def test_a_step_in_a_large_pool(n, evict, skewed):
    # all sixteen slots of a thread's registers (148 SMs) and one more; skewed: one block holds no small key, so that the blocks' least keys bound nothing, more
    # candidates than the list holds lie within the other bound, and the kernel leaves the work to the other one after its scans
    rng = np.random.default_rng(n + evict)
    gm = S.Model.from_projection(H.make_model_pair(128, seed=61)[1], 128, 61)
    keys = S.to_device(np.resize(H.gaussian_keys(62, 4096, 128), (131072, 128)))
    pools = [S.TilePool(n + 4000, 2**40, 1, evict, 4, 500) for _ in range(2)]
    at = 0

    def append(m):
        nonlocal at
        got = [p.append_keys(gm, keys, S.CODEC_MIXED, n=m, position_base=at) for p in pools]
        assert np.array_equal(*got)
        at += m

    def step(budget):
        within, launched = [], []
        for i, p in enumerate(pools):
            p.set_budget(int(budget))
            S.debug_force_generic_score(bool(i))
            before = S.launch_count()
            try:
                within.append(p.enforce_budget())
            finally:
                S.debug_force_generic_score(False)
            launched.append(S.launch_count() - before)
        assert within[0] == within[1] and pools[0].stats() == pools[1].stats()
        return launched[0]

    def live():
        return pools[0].stats()["live_bytes"]

    for b in range(0, n, 131072):
        append(min(131072, n - b))
    slots = np.arange(n, dtype=np.uint32)
    sc = rng.standard_normal(n).astype(F)
    if skewed:
        sc[slots // 512 % 148 == 147] += 30
    for p in pools:
        p.observe_scores(slots, sc, 0.9)
    step(96 * n)                           # everything is paged
    for m, gone in ((8, 1), (8, 8), (1, 60), (20, 90)):
        append(m)
        kernels = step(live() - 32 * m - 96 * gone)
        assert kernels == (2 if skewed and gone >= 60 else 1), (m, gone, kernels)
    append(3)
    assert step(live() - 32 * 2) == 1 and step(live()) == 1
    for a, b in zip(pools[0].read(), pools[1].read()):
        assert a.tobytes() == b.tobytes()
