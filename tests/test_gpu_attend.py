"""Decode tail on the selected tiles (slha_b200_attend_topk) against the oracle's restatement of the
reference's softmax_into + aggregate_v (scirust/src/metrics.rs:338-420,
scirust/examples/benchmark_decode.rs:28-38, :82-95).  Floating point: weights and outputs within
2e-6 absolute + 2e-5 relative (the device sums in another, fixed order and uses float32 exp)."""
import numpy as np
import pytest

from oracle import pyoracle as ora
from tests import helpers as H

pytestmark = pytest.mark.gpu
S = pytest.importorskip("slhav2_b200")
F = np.float32


def close(a, b):
    return np.all(np.abs(a - b) <= 2e-6 + 2e-5 * np.abs(b))


@pytest.mark.parametrize("n,nq,k,d_v,bf16", [(5000, 4, 256, 128, False), (3000, 3, 100, 96, True), (700, 2, 1024, 128, False),
                                             (4096, 5, 64, 300, False)])
def test_attend_after_topk_matches_the_reference_tail(n, nq, k, d_v, bf16):
    tiles = H.random_tiles(n, 1, seed=n)
    qc, qs = H.random_queries(nq, n + 1)
    dt = S.to_device(tiles)
    # two KV heads' worth of value rows; the query rows alternate between them; reported indices start at 50
    heads = 2
    values = ora.Rng(n + 2).gaussian(heads * n * d_v).reshape(heads * n, d_v)
    if bf16:
        values = H.to_bf16_f32(values).reshape(heads * n, d_v)
        dv = S.to_device((values.view(np.uint32) >> 16).astype(np.uint16))
    else:
        dv = S.to_device(values)
    segs = [(0, n, 0, nq, 50)]
    gi, gs, gc = S.score_topk(dt, S.make_segments(segs), qc, qs, nq, k)
    base = np.array([(j % heads) * n - 50 for j in range(nq)], np.int64).astype(np.uint64)
    scale = float(1.0 / np.sqrt(128.0))
    w_out = np.zeros((nq, k), F)
    out = S.attend_topk(gi, gs, k, scale, dv, d_v, value_dtype=S.BF16 if bf16 else S.F32, top_count=gc, value_row_base=base,
                        weights_out=w_out)
    want, want_w = ora.attend_topk(gi, gs, scale, values, top_count=gc, row_base=base)
    assert close(w_out, want_w) and close(out, want)
    assert np.all(np.abs(w_out.sum(1) - 1.0) <= 1e-5)
    assert np.all(w_out[:, min(k, n):] == 0)  # padding entries weigh nothing


def test_attend_rows_without_winners_and_bad_arguments():
    d_v, k = 64, 16
    values = ora.Rng(3).gaussian(100 * d_v).reshape(100, d_v)
    dv = S.to_device(values)
    idx = np.full((2, k), 0xFFFFFFFF, np.uint32)
    sc = np.full((2, k), -np.inf, F)
    idx[1, :3] = [5, 7, 99]
    sc[1, :3] = [1.0, 0.5, -2.0]
    out = S.attend_topk(idx, sc, k, 0.25, dv, d_v)
    want, _ = ora.attend_topk(idx, sc, 0.25, values)
    assert np.all(out[0] == 0) and close(out, want)
    with pytest.raises(S.SlhaError) as e:
        S.attend_topk(idx, sc, k, float("nan"), dv, d_v)
    assert e.value.code == S.ERR_NONFINITE
    with pytest.raises(S.SlhaError) as e:
        S.attend_topk(idx, sc, k, 0.25, values, d_v)  # host values
    assert e.value.code == S.ERR_DEVICE


@pytest.mark.parametrize("d_v,stride,shift,bf16,k", [(128, 128, 0, True, 2048), (128, 136, 1, True, 100), (130, 130, 0, True, 9), (2104, 2104, 0, True, 33),
                                                     (7, 9, 0, False, 1), (128, 132, 0, False, 700), (128, 128, 1, False, 65), (1100, 1100, 0, False, 17)])
def test_attend_takes_any_row_length_stride_and_alignment(d_v, stride, shift, bf16, k):
    # 16-byte loads where rows allow them, single elements elsewhere; more than 256 vectors per row take a second sweep
    n, nq = 3000, 3
    rng = np.random.default_rng(d_v + k)
    values = rng.standard_normal((n, d_v)).astype(F)
    if bf16:
        values = H.to_bf16_f32(values).reshape(n, d_v)
    esz = 2 if bf16 else 4
    flat = np.zeros(n * stride + shift, np.uint16 if bf16 else F)
    rows = flat[shift:].reshape(n, stride)
    rows[:, :d_v] = (values.view(np.uint32) >> 16).astype(np.uint16) if bf16 else values
    buf = S.to_device(flat)
    idx = np.stack([rng.permutation(n)[:k] for _ in range(nq)]).astype(np.uint32)
    idx[1, ::3] = 0xFFFFFFFF
    sc = (10.0 * rng.standard_normal((nq, k))).astype(F)
    cnt = np.array([k, k, k // 2], np.uint32)
    w_out = np.zeros((nq, k), F)
    out = S.attend_topk(idx, sc, k, 0.1, buf.view(shift * esz, flat.nbytes - shift * esz), d_v, value_dtype=S.BF16 if bf16 else S.F32, top_count=cnt,
                        value_row_stride=stride, weights_out=w_out)
    want, want_w = ora.attend_topk(idx, sc, 0.1, values, top_count=cnt)
    assert close(w_out, want_w) and close(out, want)


@pytest.mark.parametrize("k,bf16", [(64, False), (1000, True), (2048, True)])
def test_attend_rows_that_have_fewer_winners_than_k(k, bf16):
    # the winners a row has are shared by the eight CTAs of its cluster: counts around their multiples, up to k and beyond
    n, d_v = 4000, 128
    counts = np.array([0, 1, 7, 8, 9, k // 8 - 1, k // 8, k // 8 + 1, k // 2 + 3, k - 1, k, k + 5], np.uint32)
    nq = len(counts)
    rng = np.random.default_rng(k)
    values = rng.standard_normal((n, d_v)).astype(F)
    if bf16:
        values = H.to_bf16_f32(values).reshape(n, d_v)
    buf = S.to_device((values.view(np.uint32) >> 16).astype(np.uint16) if bf16 else values)
    idx = np.stack([rng.permutation(n)[:k] for _ in range(nq)]).astype(np.uint32)
    idx[8, ::5] = 0xFFFFFFFF
    sc = (10.0 * rng.standard_normal((nq, k))).astype(F)
    w_out = np.full((nq, k), 7.0, F)
    out = S.attend_topk(idx, sc, k, 0.1, buf, d_v, value_dtype=S.BF16 if bf16 else S.F32, top_count=counts, weights_out=w_out)
    want, want_w = ora.attend_topk(idx, sc, 0.1, values, top_count=np.minimum(counts, k))
    assert close(w_out, want_w) and close(out, want)
    for j in range(nq):
        assert np.all(w_out[j, min(counts[j], k):] == 0)


@pytest.mark.parametrize("nq,k", [(1, 8192), (36, 33), (38, 100), (75, 64), (150, 16), (300, 300), (700, 1), (320, 4096)])
def test_attend_of_many_rows_takes_smaller_clusters(nq, k):
    # eight, four, two and one CTA per row; a CTA alone holds all of a row's weights
    n, d_v = 9000, 96
    rng = np.random.default_rng(nq)
    values = rng.standard_normal((n, d_v)).astype(F)
    idx = np.stack([rng.permutation(n)[:k] for _ in range(nq)]).astype(np.uint32)
    sc = (10.0 * rng.standard_normal((nq, k))).astype(F)
    counts = rng.integers(0, k + 1, nq).astype(np.uint32)
    w_out = np.full((nq, k), 7.0, F)
    out = S.attend_topk(idx, sc, k, 0.1, S.to_device(values), d_v, top_count=counts, weights_out=w_out)
    some = rng.choice(nq, min(nq, 40), replace=False)
    want, want_w = ora.attend_topk(idx[some], sc[some], 0.1, values, top_count=counts[some])
    assert close(w_out[some], want_w) and close(out[some], want)


def test_attention_feeds_attention_queries_and_keys_without_a_wait_between():
    # attend's grids let the next kernel on the stream start early: what they write is the next call's values, queries or keys, in the same
    # buffers call after call (1500 rows: the wide loads of the encoder, full 16-byte value loads)
    n, k, d = 1500, 8, 128
    rng = np.random.default_rng(5)
    gm = S.Model.from_projection(H.orthogonal_projection(11, d), d, 7)
    idx = S.to_device(rng.integers(0, n, (n, k)).astype(np.uint32))
    sc = S.to_device(rng.standard_normal((n, k)).astype(F))
    idx.numel = lambda: n * k  # (attend_topk takes the number of rows from it)
    values = [S.to_device(rng.standard_normal((n, d)).astype(F)) for _ in range(3)]
    mid, out, qc, qs, tiles = [S.DeviceBuffer(n * m) for m in (4 * d, 4 * d, 512, 32, 128)]

    def step(v, wait):
        S.attend_topk(idx, sc, k, 0.7, v, d, out=mid)
        wait()
        S.attend_topk(idx, sc, k, 0.7, mid, d, out=out)
        wait()
        gm.prepare_queries(out, nq=n, q_coarse_out=qc, q_sign_out=qs)
        wait()
        S.attend_topk(idx, sc, k, 0.3, mid, d, out=out)
        wait()
        gm.encode_keys(out, 2, n=n, out=tiles)

    def results():
        S.synchronize()
        return [b.download(np.uint8, b.nbytes) for b in (qc, qs, tiles)]

    want = []
    for v in values:
        step(v, S.synchronize)
        want.append(results())
    for r in range(30):
        for i in range(r % 3 + 1):
            step(values[i], lambda: None)
        assert all(np.array_equal(g, w) for g, w in zip(results(), want[r % 3])), r
