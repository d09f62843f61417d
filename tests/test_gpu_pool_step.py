"""The budget question of a decode step, settled by one kernel (pool.cu, enforce_step_kernel): the same slots, states, bytes and order of freed
slots as the phases run one by one from the host give, on both sides of every condition under which the kernel leaves the work to the others."""
import numpy as np
import pytest

from tests import helpers as H

pytestmark = pytest.mark.gpu
S = pytest.importorskip("slhav2_b200")
F = np.float32


@pytest.mark.parametrize("page,evict,recent,n", [(0, 0, 0, 1), (1, 1, 0, 511), (0, 1, 300, 513), (1, 0, 0, 9000), (1, 1, 2000, 80000), (0, 1, 75000, 80000)])
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
