"""Timed cases of the tile hot path, as a program that serves from it calls them: fused score + top-k over resident
tiles, dense scores of a layer, batched encode, the decode tail over the winners, and a decode step on the elastic pool.

All calls go through `slhav2_b200` on device buffers and one stream of the caller's.  The scoring cases' tiles are made
here with torch (seeded keys with per-channel scales and rotary positions, quantised into the 128-byte record), so that
`exact` can score the very same bytes in 64 bits without the library.
"""
import math

import numpy as np
import torch

import slhav2_b200 as S

DEV = "cuda"
ROPE_THETA = 500000.0
LAMBDA_PER_SIGMA = 0.0783  # lambda = 0.0783 sigma_E in an encoded tile
CODECS = ("int4", "mx16", "nf4", "mixed", "tq3", "mix3", "mx32")  # codec ids 0..6
FLAGS = {"nf4": 2, "mixed": 4, "tq3": 8, "mix3": 32}
NF4 = (-1.0, -0.7075, -0.5421, -0.4165, -0.3108, -0.2158, -0.1272, -0.0421, 0.0421, 0.1272, 0.2158, 0.3108, 0.4165, 0.5421, 0.7075, 1.0)
CHUNK = 131072  # keys made at a time
_stream = None


def _use_stream():
    """One non-default stream for torch and the library, made once per process."""
    global _stream
    if _stream is None:
        _stream = torch.cuda.Stream()
    S.set_stream(_stream.cuda_stream)


def listed():
    return [
        # A million tokens of one layer's 8 KV heads (MX-32 tiles, 32 query heads in groups of 4): the long-context step.
        dict(name="topk_1m_mx32", op="topk", codec="mx32", segments=8, tokens=1048576, queries=4, k=2048, ragged=False, residual=False),
        # A whole Llama-3-8B-shaped decode step in one call: 32 layers x 8 KV heads x 32768 tokens, NF4.
        dict(name="topk_llama_nf4", op="topk", codec="nf4", segments=256, tokens=32768, queries=4, k=1024, ragged=False, residual=False),
        # 16 sequences x 32 heads share 8 KV heads of 16384 tokens: 64 queries per tile, TQ3.
        dict(name="topk_batch_tq3", op="topk", codec="tq3", segments=8, tokens=16384, queries=64, k=256, ragged=False, residual=True),
        # A batch of four sequences of different lengths, 8 KV heads each, MIX3 tiles.
        dict(name="topk_ragged_mix3", op="topk", codec="mix3", segments=32, tokens=20011, queries=4, k=512, ragged=True, residual=True),
        # One layer of an ordinary context, mixed 8/4 tiles, as a per-layer decode loop calls it.
        dict(name="topk_layer_mixed", op="topk", codec="mixed", segments=8, tokens=8192, queries=4, k=256, ragged=False, residual=True),
        # The smallest: one head, one query, 4096 tokens.
        dict(name="topk_single_int4", op="topk", codec="int4", segments=1, tokens=4096, queries=1, k=64, ragged=False, residual=False),
        # The llama.cpp shim's dense scores of a layer: a 64-row prompt chunk on a long context ...
        dict(name="dense_mixed_64", op="dense", codec="mixed", segments=8, tokens=32768, queries=64, residual=True),
        # ... and one decoded token on an ordinary one.
        dict(name="dense_mix3_decode", op="dense", codec="mix3", segments=8, tokens=4096, queries=4, residual=True),
        # Prefill: a layer's keys (8 heads x 32768 tokens, bf16) into NF4 tiles.
        dict(name="encode_nf4", op="encode", codec="nf4", keys=262144, d=128, dtype="bf16", rht=False),
        # A prompt chunk of float32 keys wider than the latent, TQ3 with the Hadamard rotation.
        dict(name="encode_tq3_d160_rht", op="encode", codec="tq3", keys=20011, d=160, dtype="f32", rht=True),
        # Decode tail: softmax over 2048 winners of 32 query rows and the weighted sum of their bf16 value rows.
        dict(name="attend_32x2048", op="attend", rows=32, k=2048, heads=8, tokens=131072, d_v=128, dtype="bf16"),
        # Elastic pool of a million slots under a 60 % budget: append one token's 8 keys, prepare and score 4 queries,
        # observe one, enforce the budget, read the counters.
        dict(name="pool_step_1m", op="pool", codec="mixed", slots=1048576, queries=4, k=256, recent=2048),
    ]


def _spread(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["topk"] * 6 + ["dense"] * 2 + ["encode"] * 2 + ["attend", "pool"])
    if op == "topk":
        codec, queries = rng.choice(CODECS), rng.choice([1, 2, 3, 4, 4, 4, 5, 6, 8, 16, 32, 64])
        segments = _spread(rng, 1, 256)
        # tiles x passes over them stay below the listed ones' cost
        most = (262144 if codec == "mix3" else 4194304) if queries <= 4 else (262144 if codec == "mix3" else 2097152) * 4 // queries
        tokens = min(max(192, most // segments), _spread(rng, 192, 1048576))
        ragged = rng.random() < 0.4
        k = min(_spread(rng, 8, 2048), min(_lengths(segments, tokens, ragged)))
        return dict(op=op, codec=codec, segments=segments, tokens=tokens, queries=queries, k=k, ragged=ragged, residual=rng.random() < 0.5)
    if op == "dense":
        queries = rng.choice([1, 4, 4, 6, 8, 16, 33, 64])
        tokens = _spread(rng, 128, 32768)
        segments = rng.choice([1, 2, 4, 8])
        codec = rng.choice(CODECS)
        if codec in ("nf4", "mix3"):
            tokens = min(tokens, 262144 // (segments * queries) * 4)
        return dict(op=op, codec=codec, segments=segments, tokens=tokens, queries=queries, residual=rng.random() < 0.5)
    if op == "encode":
        return dict(op=op, codec=rng.choice(CODECS), keys=_spread(rng, 1, 131072), d=rng.choice([128, 128, 128, 160]), dtype=rng.choice(["bf16", "f32"]),
                    rht=rng.random() < 0.4)
    if op == "attend":
        return dict(op=op, rows=_spread(rng, 1, 256), k=_spread(rng, 16, 2048), heads=8, tokens=_spread(rng, 2048, 131072), d_v=rng.choice([64, 96, 128, 256]),
                    dtype=rng.choice(["bf16", "f32"]))
    return dict(op=op, codec=rng.choice(["mixed", "tq3", "mx16"]), slots=_spread(rng, 32768, 1048576), queries=rng.choice([1, 4, 4, 8]), k=_spread(rng, 64, 512),
                recent=_spread(rng, 64, 2048))


# --------------------------------------------------------------------------- inputs
def _lengths(segments, tokens, ragged):
    return [tokens - ((i * 40503 + 17) % 65536) * (tokens // 2) // 65536 if ragged else tokens for i in range(segments)]


def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    return g


def _projection(seed, d):
    """128 orthonormal rows of d."""
    q, _ = np.linalg.qr(np.random.default_rng(seed).standard_normal((d, d)))
    return np.ascontiguousarray(q.T[:128], np.float32)


def _rope(k, pos):
    d = k.shape[-1]
    inv = ROPE_THETA ** (-torch.arange(0, d, 2, device=DEV, dtype=torch.float64) / d)
    ang = pos.double()[:, None] * inv
    c, s = torch.cos(ang).float(), torch.sin(ang).float()
    a, b = k[:, 0::2].clone(), k[:, 1::2].clone()
    k[:, 0::2] = a * c - b * s
    k[:, 1::2] = a * s + b * c
    return k


def _keys(gen, chan, n, pos):
    """Keys with per-channel scales and rotary positions, float32."""
    return _rope(torch.randn(n, chan.numel(), generator=gen, device=DEV) * chan, pos)


def _bytes_of(x):
    return x.contiguous().view(torch.uint8).reshape(x.shape[0], -1)


def _groups(v, codec):
    """Per tile: 8 group steps, the 128 (or 120) values over their step."""
    n = v.shape[0]
    top = {"int4": 7.0, "mx16": 7.0, "mx32": 7.0, "nf4": 1.0, "tq3": 3.5, "mixed": 7.0, "mix3": 3.5}[codec]
    if codec in ("mixed", "mix3"):
        step = torch.cat([v[:, :8].abs().amax(1, keepdim=True) / 127.0, v[:, 8:120].reshape(n, 7, 16).abs().amax(2) / top], 1)
        dims = torch.cat([torch.zeros(8, dtype=torch.long), torch.arange(112) // 16 + 1]).to(DEV)
        v = v[:, :120]
    else:
        width = {"int4": 128, "mx32": 32}.get(codec, 16)
        step = (v.reshape(n, 128 // width, width).abs().amax(2) / top).repeat_interleave(width // 16, 1)
        dims = torch.arange(128, device=DEV) // 16
    scale = step.amax(1)
    gs = torch.round(step / scale[:, None] * 255.0).clamp(1, 255)
    eff = scale[:, None] * (gs / 255.0)
    return scale, gs.to(torch.uint8), v / eff[:, dims]


def _nibbles(code):
    return code[:, 0::2] | (code[:, 1::2] << 4)


def _codes3(t):
    """3-bit codes as a little-endian bit stream, then one correction bit per value."""
    n, m = t.shape
    code = torch.round(t + 3.5).clamp(0, 7)
    corr = (t > code - 3.5).to(torch.int32).reshape(n, m // 8, 8)
    at = torch.arange(8, device=DEV, dtype=torch.int32)
    word = (code.to(torch.int32).reshape(n, m // 8, 8) << (3 * at)).sum(2)
    return torch.cat([torch.stack([(word >> s) & 255 for s in (0, 8, 16)], 2).reshape(n, -1).to(torch.uint8), (corr << at).sum(2).to(torch.uint8)], 1)


def _tiles(v, codec, gen, pos, head, residual):
    """The 128-byte records of latents v."""
    n = v.shape[0]
    scale, gs, t = _groups(v, codec)
    if codec == "nf4":
        book = torch.tensor(NF4, device=DEV)
        lat = _nibbles(torch.bucketize(t.clamp(-1, 1), (book[1:] + book[:-1]) / 2).to(torch.uint8))
    elif codec == "tq3":
        lat = _codes3(t)
    elif codec == "mixed" or codec == "mix3":
        body = _nibbles((torch.round(t[:, 8:]).clamp(-8, 7) + 8).to(torch.uint8)) if codec == "mixed" else _codes3(t[:, 8:])
        lat = torch.cat([(torch.round(t[:, :8]).clamp(-128, 127) + 128).to(torch.uint8), body], 1)
    else:
        lat = _nibbles((torch.round(t).clamp(-8, 7) + 8).to(torch.uint8))
    bits = torch.randint(0, 256, (n, 32), generator=gen, device=DEV, dtype=torch.uint8)
    # keys of the latent's own width leave rounding noise as their residual, wider ones a part of the key
    sigma = (0.3 if residual else 6e-8) * v.square().mean(1).sqrt()
    meta = torch.stack([scale, sigma * LAMBDA_PER_SIGMA, sigma], 1)
    pos32 = pos.to(torch.int32)
    ids = torch.tensor([head, FLAGS.get(codec, 0)], device=DEV, dtype=torch.int16).expand(n, 2)
    return torch.cat([lat, bits, _bytes_of(meta), _bytes_of(torch.stack([pos32, pos32], 1)), _bytes_of(ids), gs], 1)


def _score_inputs(case, seed):
    lens = _lengths(case["segments"], case["tokens"], case.get("ragged", False))
    tiles = torch.empty(sum(lens), 128, dtype=torch.uint8, device=DEV)
    gen = _gen(seed)
    p = torch.from_numpy(_projection(seed % 65536, 128)).to(DEV)
    chan = torch.exp(0.5 * torch.randn(128, generator=gen, device=DEV))
    rows, at = [], 0
    for i, n in enumerate(lens):
        for t0 in range(0, n, CHUNK):
            m = min(CHUNK, n - t0)
            pos = torch.arange(t0, t0 + m, device=DEV)
            tiles[at + t0:at + t0 + m] = _tiles(_keys(gen, chan, m, pos) @ p.T, case["codec"], gen, pos, i % 8, case["residual"])
        rows.append((at, n, i * case["queries"], case["queries"], 0))
        at += n
    nq = len(lens) * case["queries"]
    qc = torch.randn(nq, 128, generator=gen, device=DEV)
    qs = torch.randint(-2**63, 2**63 - 1, (nq, 4), generator=gen, device=DEV)
    return tiles, rows, qc, qs


def _winners(case, seed):
    gen = _gen(seed)
    values = torch.randn(case["heads"] * case["tokens"], case["d_v"], generator=gen, device=DEV).to(torch.bfloat16 if case["dtype"] == "bf16" else torch.float32)
    k = min(case["k"], case["tokens"])
    index = torch.stack([torch.randperm(case["tokens"], generator=gen, device=DEV)[:k] for _ in range(case["rows"])]).to(torch.int32)
    score = 13.0 * (2.0 + torch.rand(case["rows"], k, generator=gen, device=DEV).square() * 2.5).sort(1, descending=True).values
    base = (torch.arange(case["rows"], device=DEV) * case["heads"] // case["rows"]) * case["tokens"]
    return values, index, score, base


def _raw_keys(case, seed, n, d):
    gen = _gen(seed)
    chan = torch.exp(0.5 * torch.randn(d, generator=gen, device=DEV))
    pos = torch.arange(n, device=DEV)
    return _keys(gen, chan, n, pos).to(torch.bfloat16 if case.get("dtype", "bf16") == "bf16" else torch.float32), pos.to(torch.int32), gen


def prepare(case, seed):
    _use_stream()
    st = dict(case)
    if case["op"] in ("topk", "dense"):
        tiles, rows, qc, qs = _score_inputs(case, seed)
        nq = qc.shape[0]
        st.update(tiles=tiles, segs=S.make_segments(rows), qc=qc, qs=qs, nq=nq)
        if case["op"] == "topk":
            st.update(index=torch.empty(nq, case["k"], dtype=torch.int32, device=DEV), score=torch.empty(nq, case["k"], device=DEV),
                      count=torch.empty(nq, dtype=torch.int32, device=DEV))
        else:
            st.update(out=torch.empty(nq, case["tokens"], device=DEV), offsets=torch.arange(nq, device=DEV) * case["tokens"])
    elif case["op"] == "encode":
        keys, pos, _ = _raw_keys(case, seed, case["keys"], case["d"])
        st.update(model=S.Model.from_projection(_projection(seed % 65536, case["d"]), case["d"], 7, rht=case["rht"]), buf=keys, pos=pos,
                  heads=(pos % 8).to(torch.int16), out=torch.empty(case["keys"], 128, dtype=torch.uint8, device=DEV), codec=CODECS.index(case["codec"]))
    elif case["op"] == "attend":
        values, index, score, base = _winners(case, seed)
        rows, k = index.shape
        st.update(values=values, index=index, score=score, base=base, k=k, out=torch.empty(rows, case["d_v"], device=DEV),
                  weights=torch.empty(rows, k, device=DEV))
    else:
        slots, codec = case["slots"], CODECS.index(case["codec"])
        model = S.Model.from_projection(_projection(seed % 65536, 128), 128, 7)
        pool = S.TilePool(slots, int(0.6 * 128 * slots), S.PAGE_LOWEST_IMPACT_FIRST, S.EVICT_IMPORTANCE, sink_window=4, recent_window=case["recent"])
        fill = (slots - 64) // 8 * 8
        keys, pos, gen = _raw_keys(case, seed, fill, 128)
        new = torch.randn(64, 8, 128, generator=gen, device=DEV).to(torch.bfloat16)
        queries = torch.randn(64, case["queries"], 128, generator=gen, device=DEV)
        torch.cuda.synchronize()
        pool.append_keys(model, keys, codec, n=fill, key_dtype=S.BF16, positions=pos // 8, want_slots=False)
        pool.enforce_budget()
        nq, k = case["queries"], case["k"]
        st.update(model=model, pool=pool, new=new, raw=queries, codec=codec, step=0, token=fill // 8,
                  qc=torch.empty(nq, 128, device=DEV), qs=torch.empty(nq, 4, dtype=torch.int64, device=DEV),
                  index=torch.empty(nq, k, dtype=torch.int32, device=DEV), score=torch.empty(nq, k, device=DEV))
    return st


# --------------------------------------------------------------------------- one pass
def run(st):
    op = st["op"]
    if op == "topk":
        S.score_topk(st["tiles"], st["segs"], st["qc"], st["qs"], st["nq"], st["k"], st["index"], st["score"], st["count"])
        return st["index"], st["score"], st["count"]
    if op == "dense":
        return S.score_segments(st["tiles"], st["segs"], st["qc"], st["qs"], st["nq"], st["out"], st["offsets"], st["tokens"])
    if op == "encode":
        dtype = S.BF16 if st["dtype"] == "bf16" else S.F32
        return st["model"].encode_keys(st["buf"], st["codec"], n=st["keys"], key_dtype=dtype, positions=st["pos"], head_ids=st["heads"], out=st["out"])
    if op == "attend":
        dtype = S.BF16 if st["dtype"] == "bf16" else S.F32
        S.attend_topk(st["index"], st["score"], st["k"], 128.0 ** -0.5, st["values"], st["d_v"], value_dtype=dtype, value_row_base=st["base"], out=st["out"],
                      weights_out=st["weights"])
        return st["out"], st["weights"]
    i, pool, model, nq = st["step"] % 64, st["pool"], st["model"], st["queries"]
    pool.append_keys(model, st["new"][i], st["codec"], n=8, key_dtype=S.BF16, positions=np.full(8, st["token"] + st["step"], np.uint32), want_slots=False)
    model.prepare_queries(st["raw"][i], nq=nq, q_coarse_out=st["qc"], q_sign_out=st["qs"])
    pool.score_topk(st["qc"], st["qs"], nq, st["k"], st["index"], st["score"])
    pool.observe_query(st["qc"], st["qs"], 1.0)
    within = pool.enforce_budget()
    st["step"] += 1
    return st["index"], st["score"], within, pool.stats()


# --------------------------------------------------------------------------- what a pass cannot do without
def work(case):
    op = case["op"]
    if op in ("topk", "dense"):
        tiles, q = sum(_lengths(case["segments"], case["tokens"], case.get("ragged", False))), case["queries"]
        out = 8 * case["segments"] * q * case["k"] if op == "topk" else 4 * tiles * q
        return {"bytes": 128 * tiles + 544 * case["segments"] * q + out, "flops": 2 * 128 * tiles * q}
    if op == "encode":
        d_pad = 1 << (case["d"] - 1).bit_length() if case["rht"] else case["d"]
        return {"bytes": case["keys"] * (case["d"] * (2 if case["dtype"] == "bf16" else 4) + 128), "flops": 2 * case["keys"] * (2 * 128 * case["d"] + 256 * d_pad)}
    if op == "attend":
        n = case["rows"] * min(case["k"], case["tokens"])
        return {"bytes": n * (case["d_v"] * (2 if case["dtype"] == "bf16" else 4) + 12) + case["rows"] * case["d_v"] * 4, "flops": 2 * n * case["d_v"]}
    # the live tiles are read once for the queries' scores and the observed one's, the importances once and back
    live = 0.6 * case["slots"] * 4 / 3
    live = min(live, case["slots"])
    return {"bytes": live * (64 + 32) + case["slots"] + 8 * live, "flops": 2 * 128 * live * case["queries"]}


def tolerance(case):
    """Measured against other orders of the sums (the generic kernel, 64 bits): float32 sums of 128 products, whose
    queries the tensor-core kernels split in two halves of 16 bits; ranks may swap where scores tie that closely."""
    op = case["op"]
    if op == "encode":
        return "exact"  # a tile's bytes are those of the reference's order of operations
    if op == "attend":
        return {"rel": 4e-6, "max": 4e-5}
    if op == "dense":
        return {"rel": 4e-6, "max": 4e-5}
    return {"rel": 4e-6, "max": 4e-5, "differ": 0.01}


# --------------------------------------------------------------------------- the same in 64 bits
def _latents64(tiles, codec):
    b = tiles.to(torch.int64)
    scale = tiles[:, 96:100].contiguous().view(torch.float32).double()
    gs = b[:, 120:128].double() / 255.0

    def level3(lat, m):
        words = lat[:, :3 * m // 8].reshape(-1, m // 8, 3)
        word = words[:, :, 0] | (words[:, :, 1] << 8) | (words[:, :, 2] << 16)
        at = torch.arange(8, device=DEV)
        code = ((word[:, :, None] >> (3 * at)) & 7).reshape(-1, m)
        corr = ((lat[:, 3 * m // 8:m // 2, None] >> at) & 1).reshape(-1, m)
        return code.double() - 3.5 + (corr.double() - 0.5) * 0.5

    def nibbles(lat):
        return torch.stack([lat & 15, lat >> 4], 2).reshape(lat.shape[0], -1)

    lat = b[:, :64]
    if codec in ("mixed", "mix3"):
        body = nibbles(lat[:, 8:]).double() - 8.0 if codec == "mixed" else level3(lat[:, 8:], 112)
        eff = scale * gs
        v = torch.cat([(lat[:, :8].double() - 128.0) * eff[:, :1], body * eff[:, 1:].repeat_interleave(16, 1)], 1)
        return torch.cat([v, torch.zeros(v.shape[0], 8, device=DEV, dtype=torch.float64)], 1)
    if codec == "tq3":
        v = level3(lat, 128)
    elif codec == "nf4":
        v = torch.tensor(NF4, device=DEV).double()[nibbles(lat)]
    else:
        v = nibbles(lat).double() - 8.0
    return v * (scale * gs).repeat_interleave(16, 1)


def _scores64(tiles, codec, qc, qs):
    """[query][tile]"""
    parts = []
    bits = 2 ** torch.arange(8, device=DEV)
    signs = lambda x: 2.0 * ((x[:, :, None].to(torch.int64) & bits) != 0).reshape(x.shape[0], -1).double() - 1.0  # noqa: E731
    q, s = qc.double(), signs(_bytes_of(qs))
    for t0 in range(0, tiles.shape[0], CHUNK):
        t = tiles[t0:t0 + CHUNK]
        lam = t[:, 100:104].contiguous().view(torch.float32).double()[:, 0]
        parts.append(q @ _latents64(t, codec).T + lam * (s @ signs(t[:, 64:96]).T))
    return torch.cat(parts, 1)


def exact(case, seed):
    op = case["op"]
    if op in ("topk", "dense"):
        tiles, rows, qc, qs = _score_inputs(case, seed)
        got = []
        for at, n, q0, q, _ in rows:
            s = _scores64(tiles[at:at + n], case["codec"], qc[q0:q0 + q], qs[q0:q0 + q])
            got.append(s.topk(case["k"], 1).values if op == "topk" else s)
        return (None, torch.cat(got), None) if op == "topk" else torch.cat(got)
    if op == "attend":
        values, index, score, base = _winners(case, seed)
        w = torch.softmax(score.double() * 128.0 ** -0.5, 1)
        rows = values[(index.long() + base[:, None]).reshape(-1)].double().reshape(*index.shape, -1)
        return torch.einsum("rk,rkd->rd", w, rows), w
    return None
