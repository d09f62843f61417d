// Tensor-core kernel of the fused score + top-k path for up to four queries per tile (score_stream_kernel), the pieces the
// other scoring kernels share with it, and the selection routine of the merge kernel.  Included by score.cu.
//
// With a GQA group of four queries the CUDA-core kernel is bound by instruction issue (128 FMAs
// per tile and query plus the nibble decode), not by HBM.  Here the coarse dot product of eq. 2.3
// runs as m16n8k16 MMAs over sets of 16 tiles:
//   A (16 tiles x 16 k slots) = exact fp16 levels made from the tiles' nibbles in registers,
//   B (16 k slots x 8 columns) = the four queries, each as an fp16 hi and lo column
//                                (q = hi + lo keeps ~22 bits), so a thread's two accumulator
//                                columns add up to one query; fragments live in shared memory,
//   D fp32.
// Two arrangements of A exist.  Per scale group (NF4, mixed 8/4, TQ3 and INT4 tiles met in such
// launches): one MMA per 16-dim group, levels n - 8 by an fp16 magic-number trick or NF4 codebook
// entries as hi + lo pairs from a bank-replicated shared-memory table, D started from zero per
// group and folded into the score with the tile's effective group scale on the CUDA cores; the
// MMA's k index is permuted so that the four k slots a thread owns are the four nibbles of one
// 16-bit word, odd slots carry 16x the level and B's even slots 16x the query (all exact).
// Contiguous (launches of INT4 / MX-INT4 tiles only): a thread owns 16 latent bytes of a row, the
// group scale is folded into A exactly, and the eight MMAs of a set chain on two accumulators.
// The Hamming term is 8 XOR + POPC per tile and query.  Tiles are staged by cp.async into a per-warp
// ring whose rows are padded to 144 bytes: every shared-memory address of the inner loop is "row
// base + immediate".  Candidates go to per-row buffers in global memory (see score_stream_kernel).
// A tile of another codec than the launch decodes hands its query rows to score_kernel.
#pragma once

namespace slha {
namespace {

constexpr int MMA_SET_TILES = 16;
constexpr int MMA_ROW = TILE_BYTES + 16;                   // padded row of the staging ring
constexpr int MMA_HALF = 8 * MMA_ROW;                      // row g -> row g + 8
#ifndef SLHA_MMA_DEPTH
#define SLHA_MMA_DEPTH 2
#endif
constexpr uint32_t MMA_CHUNK = 16;  // slots a warp reserves at a time in a row's candidate buffer (larger chunks measured no faster)
// score_stream_kernel: a warp takes sets of U x 16 tiles.  Shared layout: query fragments, sign words, thresholds (the tail) | stage ring, and
// for launches with NF4 tiles (KIND 0) tail | ring of the first warps | NF4 table at 64 KB | ring of the others.
// U = 2 on long shares: 8 x 1M MX-32 tiles 274 -> 247 us a call (16 tiles at a time cost 483 instructions, 32 tiles 2 x 308), 8 x 524 288 mixed and TQ3
// tiles the same as with 1.  Not for NF4, whose 128 registers leave 16 warps an SM (457 us for 256 x 32 768 tiles; 439 with sets of 16 and
// 24 warps), nor for interleaved shares, whose first sets are appended unfiltered (a million MX-16 tiles on one row, k = 100: 81 us, with U = 2 102).
// Plain shares come in two forms.  LONG: U = 2 (not NF4), a first round with few seeds, Hamming distances only where a tile can reach the threshold.  Short ones
// have none of the three (INT4 has the latter two in both forms): each costs set-up or instructions and saves where items are long or few tiles are appended.  Taken
//   INT4, MX-INT4: from 6400 tiles a work item on (the plan's average: segments are cut at the CTAs' shares too), mixed 8/4 and TQ3 from 18 000, or
//     from 10 000 where rows have 1000 k tiles or more (99 segments of 30 303 TQ3 tiles, k = 16 161 / 157, k = 64 166 / 168).  us a call short / long
//     at items of 4878 (200 segments of 8000 tiles, k = 64), 6521 (150 of 12 000), 9756 (200 of 16 000, k = 256), 14 545 (80 of 40 000, k = 1024), 21 399 (256 of 32 768,
//     k = 1024), 27 594 (8 of 524 288): INT4 92 / 94, 88 / 86, 161 / 156, 158 / 152; mixed 91 / 100, 91 / 97, 160 / 164, 158 / 159, 368 / 365, 155 / 139;
//     TQ3 117 / 125, 121 / 126, 211 / 211, 205 / 206, 493 / 485, 219 / 201;
//   NF4: where rows have 200 k tiles or more on the average, so that few are appended: 256 rows of 32 768 tiles, k = 1024 428 / 443, 200 of 20 000, k = 256 218 / 223, 100 of
//     40 000 190 / 190, 200 of 16 000, k = 32 160 / 155, 8 of a million, k = 2048 347 / 324.
constexpr bool stream_long(int kind, bool il, uint64_t item_tiles, uint64_t row_tiles, uint32_t k) {
    return !il && (kind == 0 ? row_tiles >= 200ull * k : item_tiles >= (kind == 3 ? 6400 : row_tiles >= 1000ull * k ? 10000 : 18000));
}
constexpr int stream_sets(int kind, bool long_items) { return long_items && kind != 0 ? 2 : 1; }
constexpr int STREAM_THREADS = 768;  // 24 warps at 80 registers: latencies are hidden with warps (U = 2 with 20 or 16 warps: 251, 254 us)
constexpr int MMA_DEPTH = SLHA_MMA_DEPTH;                  // cp.async ring slots per warp
constexpr int MMA_BQ_BYTES = 9 * 32 * 8;                   // B fragments of a work item: [9][32 lanes] x 8 bytes
constexpr int MMA_TAIL_BYTES = 2560;                       // fragments | sign words 128 | thresholds 16 | bucket mappings 32 + 32 | flag 16
constexpr int STREAM_LUT_BYTES = 256 * 32 * 8;             // NF4 table: [byte][32 lanes] x (hi pair, lo pair)
constexpr uint32_t STREAM_LUT_AT = 0x10000;                // its shared-memory address
constexpr int stream_slot(int u) { return MMA_DEPTH * u * MMA_SET_TILES * MMA_ROW; }  // a warp's ring
constexpr int stream_low_warps(int u) { return ((int)STREAM_LUT_AT - 2048 - MMA_TAIL_BYTES) / stream_slot(u); }  // (dynamic shared memory starts below 2 KB)
constexpr size_t stream_smem_bytes(int kind, int u) {
    const int warps = STREAM_THREADS / 32;
    if (kind != 0) return MMA_TAIL_BYTES + (size_t)warps * stream_slot(u);
    return STREAM_LUT_AT + STREAM_LUT_BYTES + (size_t)(warps > stream_low_warps(u) ? warps - stream_low_warps(u) : 0) * stream_slot(u);
}
constexpr int NF4_LUT_BYTES = 256 * 16 * 8;                // score_dense_kernel: [byte][16 lanes] x (hi pair, lo pair)
constexpr int SEL_HIST_INTS = 4 * 256 + 48;                // block_select_multi: 4 histograms + state

#ifdef SLHA_STREAM_PROBE
// development build only: %globaltimer in nanoseconds
__device__ __forceinline__ unsigned long long probe_now() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;\n" : "=l"(t));
    return t;
}
#endif
__device__ __forceinline__ void mma_f16(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                        uint32_t b0, uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void mma_f16_zero(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                             uint32_t b0, uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};\n"
        : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(0.0f));
}
__device__ __forceinline__ uint32_t prmt(uint32_t a, uint32_t b, uint32_t sel) {
    uint32_t d;
    asm("prmt.b32 %0, %1, %2, %3;\n" : "=r"(d) : "r"(a), "r"(b), "r"(sel));
    return d;
}
__device__ __forceinline__ uint32_t hfma2_u32(uint32_t a, uint32_t b, uint32_t c) {
    uint32_t d;
    asm("fma.rn.f16x2 %0, %1, %2, %3;\n" : "=r"(d) : "r"(a), "r"(b), "r"(c));
    return d;
}
// The four nibbles n0..n3 of a 16-bit word h (n0 lowest) -> half2 (n0 - 8, 16 (n1 - 8))
// and half2 (n2 - 8, 16 (n3 - 8)), exact.  h duplicated into both halves of a word
// has n0 at bit 0 and n1 at bit 20 (after >> 8: n2 and n3); OR-ing those into
// 1024.0h gives (1024 + n0, 1024 + 16 n1), and one fp16 add of (-1032, -1152)
// finishes.  The odd slots carry 16x the level: the B operand carries 16x the query
// in the even slots instead, and the final score is divided by 16 (all exact).
// `magic` is 0x64006400 held in a register the compiler cannot rebuild from an immediate.
__device__ __forceinline__ void int4_quad(uint32_t h, uint32_t magic, uint32_t& lo, uint32_t& hi) {
    const uint32_t t = h * 0x10001u;
    uint32_t v0, v1;
    asm("lop3.b32 %0, %1, 0x00F0000F, %2, 0xEA;\n" : "=r"(v0) : "r"(t), "r"(magic));
    asm("lop3.b32 %0, %1, 0x00F0000F, %2, 0xEA;\n" : "=r"(v1) : "r"(t >> 8), "r"(magic));
    asm("add.rn.f16x2 %0, %1, %2;\n" : "=r"(lo) : "r"(v0), "r"(0xE480E408u));
    asm("add.rn.f16x2 %0, %1, %2;\n" : "=r"(hi) : "r"(v1), "r"(0xE480E408u));
}
__device__ __forceinline__ uint32_t pack_half2(float lo, float hi) {
    __half2 h = __floats2half2_rn(lo, hi);
    return *reinterpret_cast<uint32_t*>(&h);
}
__device__ __forceinline__ float half_residual(float x) {  // x - fp16(x)
    return x - __half2float(__float2half_rn(x));
}
// shared-memory loads on 32-bit shared-window addresses plus an immediate
template <int IMM>
__device__ __forceinline__ uint32_t lds_u16(uint32_t addr) {
    uint16_t v;
    asm volatile("ld.shared.u16 %0, [%1+%2];\n" : "=h"(v) : "r"(addr), "n"(IMM));
    return (uint32_t)v;
}
template <int IMM>
__device__ __forceinline__ uint2 lds_v2(uint32_t addr) {
    uint2 v;
    asm volatile("ld.shared.v2.u32 {%0,%1}, [%2+%3];\n" : "=r"(v.x), "=r"(v.y) : "r"(addr), "n"(IMM));
    return v;
}
template <int IMM>
__device__ __forceinline__ uint4 lds_v4(uint32_t addr) {
    uint4 v;
    asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4+%5];\n"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
                 : "r"(addr), "n"(IMM));
    return v;
}
template <int SRC_IMM, int DST_IMM>
__device__ __forceinline__ void cp_async16_s(uint32_t dst, const unsigned char* src, int src_bytes) {
    asm volatile("cp.async.cg.shared.global [%0+%1], [%2+%3], 16, %4;\n" ::"r"(dst), "n"(DST_IMM), "l"(src), "n"(SRC_IMM),
                 "r"(src_bytes));
}
// the same with an L2 eviction policy: tiles are read once, so their lines are the first to go and the rows'
// candidate buffers and histograms, which the merge reads next, stay in the L2
template <int SRC_IMM, int DST_IMM>
__device__ __forceinline__ void cp_async16_sp(uint32_t dst, const unsigned char* src, int src_bytes, uint64_t policy) {
    asm volatile("cp.async.cg.shared.global.L2::cache_hint [%0+%1], [%2+%3], 16, %4, %5;\n" ::"r"(dst), "n"(DST_IMM), "l"(src),
                 "n"(SRC_IMM), "r"(src_bytes), "l"(policy));
}
__device__ __forceinline__ void sts_v4(uint32_t addr, uint32_t x, uint32_t y, uint32_t z, uint32_t w) {
    asm volatile("st.shared.v4.u32 [%0], {%1,%2,%3,%4};\n" ::"r"(addr), "r"(x), "r"(y), "r"(z), "r"(w) : "memory");
}
// TQ3 rows of a staged 16-tile set, rewritten in place as nibble rows: nibble d of the 64 latent
// bytes becomes 2 code_d + correction_d (codes: 3 bits at bit 3d of bytes 0..47; correction bits:
// bit d of bytes 48..63, taken as zero for a tile flagged as without its correction plane).  A lane rewrites half a
// row (64 dims: 24 code bytes and 8 correction bytes in, 32 bytes out); every lane reads before
// any lane writes.
__device__ __forceinline__ void tq3_to_nibbles(uint32_t set_s, int lane) {
    const uint32_t h = (uint32_t)lane & 1u, row = set_s + (uint32_t)(lane >> 1) * MMA_ROW;
    const uint2 c0 = lds_v2<0>(row + 24u * h), c1 = lds_v2<8>(row + 24u * h), c2 = lds_v2<16>(row + 24u * h);
    uint2 cr = lds_v2<48>(row + 8u * h);
    // a tile flagged as without its correction plane is decoded from the codes alone, whatever the plane's bytes hold
    if (lds_u16<118>(row) & F_NOCORR) cr.x = cr.y = 0u;
    __syncwarp();
    const uint32_t w[7] = {c0.x, c0.y, c1.x, c1.y, c2.x, c2.y, 0u};
    uint32_t o[8];
#pragma unroll
    for (int m = 0; m < 8; ++m) {
        const int wi = (24 * m) >> 5, sh = (24 * m) & 31;
        uint32_t x = __funnelshift_r(w[wi], w[wi + 1], sh) & 0xFFFFFFu;
        x = (x & 0xFFFu) | ((x & 0xFFF000u) << 4);
        x = (x & 0x003F003Fu) | ((x & 0x0FC00FC0u) << 2);
        x = (x & 0x07070707u) | ((x & 0x38383838u) << 1);
        uint32_t c = ((m < 4 ? cr.x : cr.y) >> (8 * (m & 3))) & 0xFFu;
        c = (c | (c << 12)) & 0x000F000Fu;
        c = (c | (c << 6)) & 0x03030303u;
        c = (c | (c << 3)) & 0x11111111u;
        o[m] = (x << 1) | c;
    }
    sts_v4(row + 32u * h, o[0], o[1], o[2], o[3]);
    sts_v4(row + 32u * h + 16u, o[4], o[5], o[6], o[7]);
    __syncwarp();
}
__device__ __forceinline__ int popc8(const uint4& a, const uint4& b, const uint32_t (&q)[8]) {
    return __popc(a.x ^ q[0]) + __popc(a.y ^ q[1]) + __popc(a.z ^ q[2]) + __popc(a.w ^ q[3]) +
           __popc(b.x ^ q[4]) + __popc(b.y ^ q[5]) + __popc(b.z ^ q[6]) + __popc(b.w ^ q[7]);
}

// Pairs of float32 (sm_100's f32x2): each half rounds like the scalar operation
__device__ __forceinline__ uint64_t f2_pack(float lo, float hi) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};\n" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ uint64_t f2_add(uint64_t a, uint64_t b) {
    uint64_t r;
    asm("add.rn.f32x2 %0, %1, %2;\n" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ uint64_t f2_fma(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;\n" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}

// Coarse sums of U sub-sets of 16 tiles for rows g + 16 u (low half of acc[u]) and g + 8 + 16 u (high half), query t.
// hb = shared address of row g of the set + 2t: halfword t of every 8-byte scale
// group holds the four nibbles this thread feeds to the MMA of that group.
// MODE 0: every row uniform INT4, 1: every row NF4, 2: per-row choice, 3: every row mixed 8/4
// (group 0 holds the eight 8-bit head levels, halfword t = dims 2t and 2t+1, which fill k slots
// 2t and 2t+1 as byte - 128 while slots 2t+8 and 2t+9 stay empty; groups 1..7 are INT4 groups of
// dims 16 J - 8 ..; the B operand is arranged to match when the launch scores mixed tiles).
// lut: shared address of this lane's column of the NF4 table, whose entry of byte b lies 256 b further (the table starts at a multiple of
// 64 KB, so that one byte permutation makes an entry's address).
template <int MODE, int J, int U>
__device__ __forceinline__ void coarse_group(uint32_t hb, uint32_t lut, uint32_t magic, uint32_t bqa, const uint32_t (&f)[2 * U],
                                             const uint2 (&gs)[2 * U], uint64_t (&acc)[U]) {
    const uint2 bq = lds_v2<256 * J>(bqa);  // this lane's B fragment of group J
#pragma unroll
    for (int u = 0; u < U; ++u) {
        const uint32_t rb = hb + (uint32_t)(2 * u * MMA_HALF);
        const uint32_t h0 = lds_u16<8 * J>(rb), h1 = lds_u16<8 * J + MMA_HALF>(rb);
        uint32_t a0, a1, a2, a3, l0 = 0, l1 = 0, l2 = 0, l3 = 0;
        if (MODE == 3 && J == 0) {
            // bytes (b0, b1) -> half2 (1024 + b0, 1024 + b1) - 1152
            asm("add.rn.f16x2 %0, %1, %2;\n" : "=r"(a0) : "r"(prmt(h0, magic, 0x7150u)), "r"(0xE480E480u));
            asm("add.rn.f16x2 %0, %1, %2;\n" : "=r"(a1) : "r"(prmt(h1, magic, 0x7150u)), "r"(0xE480E480u));
            a2 = 0u;
            a3 = 0u;
        } else {
            if (MODE == 1 || (MODE == 2 && (f[2 * u] & F_NF4))) {
                const uint2 e0 = lds_v2<0>(prmt(h0, lut, 0x7604u)), e1 = lds_v2<0>(prmt(h0, lut, 0x7614u));
                a0 = e0.x; a2 = e1.x; l0 = e0.y; l2 = e1.y;
            } else {
                int4_quad(h0, magic, a0, a2);
            }
            if (MODE == 1 || (MODE == 2 && (f[2 * u + 1] & F_NF4))) {
                const uint2 e0 = lds_v2<0>(prmt(h1, lut, 0x7604u)), e1 = lds_v2<0>(prmt(h1, lut, 0x7614u));
                a1 = e0.x; a3 = e1.x; l1 = e0.y; l3 = e1.y;
            } else {
                int4_quad(h1, magic, a1, a3);
            }
        }
        float d[4];
        mma_f16_zero(d, a0, a1, a2, a3, bq.x, bq.y);
        if (MODE == 1 || MODE == 2) mma_f16(d, l0, l1, l2, l3, bq.x, bq.y);
        // gs[J] as float (on the ALU / FMA pipes: 2^23 + b as a bit pattern, minus 2^23)
        const uint32_t gw0 = J < 4 ? gs[2 * u].x : gs[2 * u].y, gw1 = J < 4 ? gs[2 * u + 1].x : gs[2 * u + 1].y;
        const uint64_t g2 = f2_add(f2_pack(__uint_as_float(__byte_perm(gw0, 0x4B000000u, 0x7440 + (J & 3))),
                                           __uint_as_float(__byte_perm(gw1, 0x4B000000u, 0x7440 + (J & 3)))),
                                   0xCB000000CB000000ull);
        acc[u] = f2_fma(f2_pack(d[0] + d[1], d[2] + d[3]), g2, acc[u]);
    }
}

template <int MODE, int U>
__device__ __forceinline__ void coarse_set(uint32_t hb, uint32_t lut, uint32_t magic, uint32_t bq, const uint32_t (&f)[2 * U],
                                           const uint2 (&gs)[2 * U], float (&out)[2 * U]) {
    uint64_t acc[U];
#pragma unroll
    for (int u = 0; u < U; ++u) acc[u] = 0ull;
    coarse_group<MODE, 0, U>(hb, lut, magic, bq, f, gs, acc);
    coarse_group<MODE, 1, U>(hb, lut, magic, bq, f, gs, acc);
    coarse_group<MODE, 2, U>(hb, lut, magic, bq, f, gs, acc);
    coarse_group<MODE, 3, U>(hb, lut, magic, bq, f, gs, acc);
    coarse_group<MODE, 4, U>(hb, lut, magic, bq, f, gs, acc);
    coarse_group<MODE, 5, U>(hb, lut, magic, bq, f, gs, acc);
    coarse_group<MODE, 6, U>(hb, lut, magic, bq, f, gs, acc);
    coarse_group<MODE, 7, U>(hb, lut, magic, bq, f, gs, acc);
#pragma unroll
    for (int u = 0; u < U; ++u) asm("mov.b64 {%0, %1}, %2;\n" : "=f"(out[2 * u]), "=f"(out[2 * u + 1]) : "l"(acc[u]));
}

// ---- launches that hold only INT4 / MX-INT4 tiles (KIND 3) --------------------------------
// Thread (g, t) of the warp owns the 16 latent bytes 16t..16t+15 of its rows: dims
// 32t..32t+31, i.e. the two scale groups 2t and 2t+1, fetched with one 16-byte load per row.
// The group scale is folded into the A operand, so the eight MMAs of a set chain on two
// accumulators and nothing is scaled per group afterwards:
//   a nibble n masked in place at bits 0..3 of a 16-bit half is the fp16 value n * 2^-24, at bits 4..7 n * 2^-20;
//   fma(n * 2^-24, gs * 2^8, -8 gs * 2^-16) = fma(n * 2^-20, gs * 2^4, ..) = (n - 8) gs * 2^-16, exact: |(n - 8) gs| <= 2040
//   has 11 significant bits and is a multiple of 2^-24 (one shift per word of eight nibbles; with the nibbles all brought to bits 4..7 it took three).
// k slot pairs (2t, 2t+1) / (2t+8, 2t+9) of MMA 2i take nibbles (0, 4) / (1, 5) of the
// thread's word i, those of MMA 2i+1 nibbles (2, 6) / (3, 7); the B fragments carry the
// queries' dims in the same order.  Sum = 2^-16 sum_d level_d gs_g q_d.
struct Int4Scale {
    uint32_t lo, hi, c;  // half2 (gs * 2^8), (gs * 2^4), (-gs * 2^-13), twice each
};
__device__ __forceinline__ Int4Scale int4c_scale(uint32_t h, uint32_t magic, uint32_t sel) {  // sel: which byte of h
    const uint32_t p = prmt(h, magic, sel);  // 1024 + gs
    Int4Scale s;
    s.hi = hfma2_u32(p, 0x4C004C00u, 0xF400F400u);  // 16 p - 16384
    s.c = hfma2_u32(p, 0x88008800u, 0x30003000u);   // -2^-13 p + 2^-3
    asm("mul.rn.f16x2 %0, %1, %2;\n" : "=r"(s.lo) : "r"(s.hi), "r"(0x4C004C00u));
    return s;
}
__device__ __forceinline__ void int4c_word(uint32_t w, const Int4Scale& s, uint32_t (&o)[4]) {
    const uint32_t v = w >> 8;
    o[0] = hfma2_u32(w & 0x000F000Fu, s.lo, s.c);  // nibbles 0, 4
    o[1] = hfma2_u32(w & 0x00F000F0u, s.hi, s.c);  // nibbles 1, 5
    o[2] = hfma2_u32(v & 0x000F000Fu, s.lo, s.c);  // nibbles 2, 6
    o[3] = hfma2_u32(v & 0x00F000F0u, s.hi, s.c);  // nibbles 3, 7
}
// rb = shared address of row g of the staged set; t = lane & 3
template <int U>
__device__ __forceinline__ void coarse_set_int4c(uint32_t rb, uint32_t t, uint32_t magic, uint32_t bqa, float (&out)[2 * U]) {
    const uint32_t cb = rb + 16u * t, hb = rb + 2u * t;
    const uint2 b0 = lds_v2<0>(bqa), b1 = lds_v2<256>(bqa), b2 = lds_v2<512>(bqa), b3 = lds_v2<768>(bqa);
    const uint2 b4 = lds_v2<1024>(bqa), b5 = lds_v2<1280>(bqa), b6 = lds_v2<1536>(bqa), b7 = lds_v2<1792>(bqa);
    const uint2 bq[8] = {b0, b1, b2, b3, b4, b5, b6, b7};
#pragma unroll
    for (int u = 0; u < U; ++u) {
        const uint32_t cu = cb + (uint32_t)(2 * u * MMA_HALF), hu = hb + (uint32_t)(2 * u * MMA_HALF);
        const uint4 L0 = lds_v4<0>(cu), L1 = lds_v4<MMA_HALF>(cu);
        const uint32_t h0 = lds_u16<120>(hu), h1 = lds_u16<120 + MMA_HALF>(hu);
        const Int4Scale s0[2] = {int4c_scale(h0, magic, 0x5050u), int4c_scale(h0, magic, 0x5151u)};
        const Int4Scale s1[2] = {int4c_scale(h1, magic, 0x5050u), int4c_scale(h1, magic, 0x5151u)};
        const uint32_t w0[4] = {L0.x, L0.y, L0.z, L0.w}, w1[4] = {L1.x, L1.y, L1.z, L1.w};
        // two accumulator chains (even / odd MMAs) halve the dependent MMA latency of a set
        float d[4], e[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            uint32_t o0[4], o1[4];
            int4c_word(w0[i], s0[i >> 1], o0);
            int4c_word(w1[i], s1[i >> 1], o1);
            if (i == 0) {
                mma_f16_zero(d, o0[0], o1[0], o0[1], o1[1], bq[0].x, bq[0].y);
                mma_f16_zero(e, o0[2], o1[2], o0[3], o1[3], bq[1].x, bq[1].y);
            } else {
                mma_f16(d, o0[0], o1[0], o0[1], o1[1], bq[2 * i].x, bq[2 * i].y);
                mma_f16(e, o0[2], o1[2], o0[3], o1[3], bq[2 * i + 1].x, bq[2 * i + 1].y);
            }
        }
        out[2 * u] = (d[0] + e[0]) + (d[1] + e[1]);
        out[2 * u + 1] = (d[2] + e[2]) + (d[3] + e[3]);
    }
}

// four consecutive elements of a query row (a caller's query rows start at any float)
__device__ __forceinline__ float4 load_q4(const float* p) {
    if (reinterpret_cast<uintptr_t>(p) & 15u) return make_float4(p[0], p[1], p[2], p[3]);
    return *reinterpret_cast<const float4*>(p);
}

// A query row is multiplied by a power of two before it is split into fp16 hi + lo, and the finished sums by its inverse: with the
// largest element in [2^target, 2^(target + 1)) the parts hold at least 22 bits of every element down to 2^-(target + 2) of the largest
// (lo ends at 2^-24; unscaled, a row of elements around 1e-3 kept 15 bits and one of 1e-8 none).  `largest`: the bits
// of the row's largest absolute value.  (up, its inverse)
__device__ __forceinline__ float2 split_scale(uint32_t largest, int target) {
    const int e = max(min(target + 127 - (int)(largest >> 23), 126), -126);  // (126: rows of denormals, exact all the same)
    return make_float2(__uint_as_float((uint32_t)(127 + e) << 23), __uint_as_float((uint32_t)(127 - e) << 23));
}
constexpr uint32_t SPLIT_MOST = (127u + 96u) << 23;  // rows with an element of 2^96 or more, infinities and NaN go to the generic kernel
__device__ __forceinline__ uint32_t abs_bits(float x) { return __float_as_uint(x) & 0x7FFFFFFFu; }

// ---- tcgen05 / mbarrier plumbing ------------------------------------------------------------------
constexpr uint32_t TC_SPIN = 1u << 22;            // polls of one mbarrier wait before it gives up (~0.2 s)

// a threshold's score word as a float; words at or below the key of -inf mean "no threshold yet"
__device__ __forceinline__ float thr_float(uint32_t key) { return key > 0x00800000u ? key_score(key) : -INFINITY; }
__device__ __forceinline__ void mbar_init(uint32_t addr, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(addr), "r"(count) : "memory");
}
// false when the phase did not complete within TC_SPIN polls
__device__ __forceinline__ bool mbar_wait(uint32_t addr, uint32_t parity) {
    for (uint32_t i = 0; i < TC_SPIN; ++i) {
        uint32_t ok;
        asm volatile("{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\nselp.u32 %0, 1, 0, p;\n}\n"
                     : "=r"(ok) : "r"(addr), "r"(parity) : "memory");
        if (ok) return true;
        if (i > 64) __nanosleep(64);
    }
    return false;
}
// Named barrier `id` over `nthreads` threads that also tells every one of them whether any brought `fail`: the
// warps of a role leave their loop together, so that none is left waiting at a later barrier of the role.
__device__ __forceinline__ bool role_any(uint32_t id, uint32_t nthreads, bool fail) {
    uint32_t any;
    asm volatile("{\n.reg .pred p, q;\nsetp.ne.u32 q, %1, 0;\nbar.red.or.pred p, %2, %3, q;\nselp.u32 %0, 1, 0, p;\n}\n"
                 : "=r"(any) : "r"((uint32_t)fail), "r"(id), "r"(nthreads) : "memory");
    return any != 0;
}
// K-major, 128-byte swizzle, 8-row groups 1024 bytes apart (tcgen05 shared-memory matrix descriptor)
__device__ __forceinline__ uint64_t tc_desc(uint32_t saddr) {
    return (uint64_t)((saddr & 0x3FFFFu) >> 4) | ((uint64_t)1 << 16) | ((uint64_t)(1024 >> 4) << 32) | ((uint64_t)1 << 46) |
           ((uint64_t)2 << 61);
}
// One lane of a warp, to be called where the warp is known to be converged (a kernel's start; the result stays in a predicate).
// tcgen05 instructions take uniform registers: behind elect.sync and a warp index taken by shuffle the compiler knows a branch to be one
// thread's, behind `threadIdx.x == 0` it issues each of them through a loop over the active lanes (a lone tcgen05.mma: 217 against
// 109 cycles).
__device__ __forceinline__ bool elect_one() {
    uint32_t p;
    asm volatile("{\n.reg .pred p;\nelect.sync _|p, 0xFFFFFFFF;\nselp.u32 %0, 1, 0, p;\n}\n" : "=r"(p));
    return p != 0;
}
__device__ __forceinline__ int uniform_warp() { return __shfl_sync(0xFFFFFFFFu, (int)(threadIdx.x >> 5), 0); }
__device__ __forceinline__ void tc_commit(uint32_t mbar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(mbar) : "memory");
}

// Bucket of a score inside [smin, smin + 256 / inv): monotone in the score.
__device__ __forceinline__ int sel_bucket_f(float sc, float smin, float inv) {
    const int b = (int)((sc - smin) * inv);
    return b < 0 ? 0 : (b > 255 ? 255 : b);
}
__device__ __forceinline__ int sel_bucket(uint32_t h, float smin, float inv) {
    return sel_bucket_f(key_score(h), smin, inv);
}
// Range [lo, hi] (order keys of scores) -> (smin, inv); false when the range cannot
// be bucketed (one single score, or a non-finite bound).
__device__ __forceinline__ bool sel_range(uint32_t lo, uint32_t hi, float& smin, float& inv) {
    smin = key_score(lo);
    const float smax = key_score(hi);
    inv = 256.0f / (smax - smin);
    return hi > lo && isfinite(smin) && isfinite(smax) && isfinite(inv);
}

// Shrinks up to four candidate buffers (keys[q][cap], counts cnt[q]) to between k
// and k + slack entries each and raises pivot[q] accordingly; only buffers with
// more than `trigger` entries are touched.  The four queries share every barrier.
//
// Selection works on the score (high word of the composite key): 256 equal-width
// buckets over [min, max] of the scores at or above the pivot; the bucket in which
// the count from the top reaches k is kept whole if that leaves at most k + slack
// keys, otherwise it becomes the next range.  Scores spread smoothly over such a
// range, so the histogram atomics do not pile up on one address the way the bytes
// of the key do.  Keys below the current pivot are dropped (the pivot is a proven
// lower bound of the query's k-th best key).  The new pivot is the smallest kept
// score.  Queries whose range collapses to one score with too many keys (equal
// scores), or holds a non-finite score, are reported in the returned bit mask
// (uniform over the block) and left for block_select_topk, which also orders by
// index.  hist: SEL_HIST_INTS ints.  All threads of the block must call.
// pivot_only: no selection, the buffers are only purged of keys below the pivot.
__device__ uint32_t block_select_multi(uint64_t* keys, uint32_t cap, int* cnt, int nq, uint32_t k, uint32_t slack,
                                       int trigger, uint64_t* pivot, int* hist, bool pivot_only = false) {
    const int tid = threadIdx.x, nt = blockDim.x, lane = tid & 31, warp = tid >> 5;
    // [q][8]: 0 range lo, 1 range hi, 2 need, 3 active, 4 exact selection wanted, 5 kept, 6 selected, 7 pivotal bucket
    uint32_t* st = reinterpret_cast<uint32_t*>(hist + 1024);
    if (tid < 4) {
        const bool act = tid < nq && cnt[tid] > trigger;
        uint32_t* s = st + 8 * tid;
        s[0] = pivot_only ? (tid < nq ? (uint32_t)(pivot[tid] >> 32) : 0u) : 0xFFFFFFFFu;
        s[1] = 0u;
        s[2] = k;
        s[3] = act && !pivot_only;
        s[4] = 0u;
        s[5] = 0u;
        s[6] = act;
        s[7] = 0u;
        if (act && cnt[tid] > (int)cap) cnt[tid] = (int)cap;
    }
    __syncthreads();
    if (!(st[6] | st[14] | st[22] | st[30])) return 0u;
    // smallest and largest score at or above the pivot
    for (int q = 0; q < nq; ++q) {
        if (!st[8 * q + 3]) continue;
        const uint64_t* kq = keys + (size_t)q * cap;
        const uint32_t floor_h = (uint32_t)(pivot[q] >> 32);
        uint32_t mx = 0u, mn = 0xFFFFFFFFu;
        const int c = cnt[q];
#pragma unroll 4
        for (int i = tid; i < c; i += nt) {
            const uint32_t h = (uint32_t)(kq[i] >> 32);
            if (h >= floor_h) { mx = max(mx, h); mn = min(mn, h); }
        }
        mx = __reduce_max_sync(0xFFFFFFFFu, mx);
        mn = __reduce_min_sync(0xFFFFFFFFu, mn);
        if (lane == 0) { atomicMax(&st[8 * q + 1], mx); atomicMin(&st[8 * q], mn); }
    }
    __syncthreads();
    for (int pass = 0; pass < 12; ++pass) {
        if (!(st[3] | st[11] | st[19] | st[27])) break;
        for (int b = tid; b < 1024; b += nt) hist[b] = 0;
        __syncthreads();
        for (int q = 0; q < nq; ++q) {
            if (!st[8 * q + 3]) continue;
            const uint32_t lo = st[8 * q], hi = st[8 * q + 1];
            float smin, inv;
            if (!sel_range(lo, hi, smin, inv)) continue;  // settled by the scan below
            const uint64_t* kq = keys + (size_t)q * cap;
            // four keys per round: the loads go out together, then the atomics
            const int c = cnt[q];
            for (int i0 = tid; i0 < c; i0 += 4 * nt) {
                uint32_t h[4];
#pragma unroll
                for (int u = 0; u < 4; ++u) h[u] = i0 + u * nt < c ? (uint32_t)(kq[i0 + u * nt] >> 32) : 0u;
#pragma unroll
                for (int u = 0; u < 4; ++u)
                    if (i0 + u * nt < c && h[u] >= lo && h[u] <= hi) atomicAdd(&hist[256 * q + sel_bucket(h[u], smin, inv)], 1);
            }
        }
        __syncthreads();
        bool refine = false;
        if (warp < nq && st[8 * warp + 3]) {
            uint32_t* s = st + 8 * warp;
            const int* hq = hist + 256 * warp;
            const uint32_t lo = s[0], hi = s[1], need = s[2];
            float smin, inv;
            if (!sel_range(lo, hi, smin, inv)) {
                // everything left in the range stays; more than allowed means equal
                // (or non-finite) scores: the exact selection sorts it out
                __syncwarp();
                if (lane == 0) { s[3] = 0u; s[4] = 1u; s[7] = 0u; }
            } else {
                // lane l owns buckets 255-8l .. 248-8l (descending)
                int c[8], tot = 0;
#pragma unroll
                for (int j = 0; j < 8; ++j) { c[j] = hq[255 - 8 * lane - j]; tot += c[j]; }
                int incl = tot;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const int y = __shfl_up_sync(0xFFFFFFFFu, incl, o);
                    if (lane >= o) incl += y;
                }
                const unsigned ok = __ballot_sync(0xFFFFFFFFu, incl >= (int)need);
                if (ok == 0u) {
                    // fewer than `need` keys at or above the pivot: all of them stay
                    if (lane == 0) { s[3] = 0u; s[7] = 0u; }
                } else {
                    int bsel = 0, run = 0, binc = 0;
                    if (lane == __ffs(ok) - 1) {
                        run = incl - tot;
#pragma unroll
                        for (int j = 0; j < 8; ++j) {
                            if (run + c[j] >= (int)need) { bsel = 255 - 8 * lane - j; binc = c[j]; break; }
                            run += c[j];
                        }
                    }
                    const int src = __ffs(ok) - 1;
                    bsel = __shfl_sync(0xFFFFFFFFu, bsel, src);
                    run = __shfl_sync(0xFFFFFFFFu, run, src);
                    binc = __shfl_sync(0xFFFFFFFFu, binc, src);
                    const uint32_t kept = (k - need) + (uint32_t)(run + binc);
                    if (kept <= k + slack) {
                        if (lane == 0) { s[3] = 0u; s[7] = (uint32_t)bsel; }
                    } else {
                        // next range: the scores of the pivotal bucket
                        refine = true;
                        __syncwarp();
                        if (lane == 0) { s[2] = need - (uint32_t)run; s[7] = (uint32_t)bsel; }
                    }
                }
            }
        }
        if (!__syncthreads_or(refine)) continue;
        // smallest and largest score inside the pivotal bucket of the queries still active
        uint32_t nlo[4], nhi[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) { nlo[q] = 0xFFFFFFFFu; nhi[q] = 0u; }
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            if (q >= nq || !st[8 * q + 3]) continue;
            const uint32_t lo = st[8 * q], hi = st[8 * q + 1];
            const int bsel = (int)st[8 * q + 7];
            float smin, inv;
            sel_range(lo, hi, smin, inv);
            const uint64_t* kq = keys + (size_t)q * cap;
            for (int i = tid; i < cnt[q]; i += nt) {
                const uint32_t h = (uint32_t)(kq[i] >> 32);
                if (h >= lo && h <= hi && sel_bucket(h, smin, inv) == bsel) { nlo[q] = min(nlo[q], h); nhi[q] = max(nhi[q], h); }
            }
            nlo[q] = __reduce_min_sync(0xFFFFFFFFu, nlo[q]);
            nhi[q] = __reduce_max_sync(0xFFFFFFFFu, nhi[q]);
        }
        __syncthreads();  // every thread has read the old range
        if (tid < 4 && tid < nq && st[8 * tid + 3]) { st[8 * tid] = 0xFFFFFFFFu; st[8 * tid + 1] = 0u; }
        __syncthreads();
#pragma unroll
        for (int q = 0; q < 4; ++q)
            if (q < nq && st[8 * q + 3] && lane == 0) { atomicMin(&st[8 * q], nlo[q]); atomicMax(&st[8 * q + 1], nhi[q]); }
        __syncthreads();
    }
    // (a range that is still open after the last pass stays whole and goes to the exact selection)
    if (tid < 4) {
        if (st[8 * tid + 3]) { st[8 * tid + 3] = 0u; st[8 * tid + 4] = 1u; st[8 * tid + 7] = 0u; }
        st[8 * tid + 2] = 0xFFFFFFFFu;  // from here on: the smallest score kept
    }
    __syncthreads();
    // compact the selected buffers in place: keys above the last range, and those of
    // the range whose bucket is the pivotal one or higher, stay
    int maxc = 0;
    for (int q = 0; q < nq; ++q)
        if (st[8 * q + 6]) maxc = max(maxc, cnt[q]);
    const int R = (maxc + nt - 1) / nt;
    if (R <= 10) {
        // every warp owns R*32 consecutive slots: it reads them all, the warps' counts are
        // summed once, then it writes its survivors (order preserved, no read-after-write)
        int* wcnt = hist;  // [4][32]
#pragma unroll 1
        for (int q = 0; q < nq; ++q) {
            if (!st[8 * q + 6]) continue;
            const uint32_t rlo = st[8 * q], rhi = st[8 * q + 1];
            int bsel = (int)st[8 * q + 7];
            float smin, inv;
            if (!sel_range(rlo, rhi, smin, inv)) bsel = -1;  // whole range stays
            uint64_t* kq = keys + (size_t)q * cap;
            const int c = cnt[q];
            uint64_t key[10];
            unsigned bal[10];
            int wtot = 0;
            uint32_t km = 0xFFFFFFFFu;
#pragma unroll
            for (int j = 0; j < 10; ++j) {
                bal[j] = 0u;
                key[j] = 0ull;
                if (j < R) {
                    const int i = (warp * R + j) * 32 + lane;
                    const bool in = i < c;
                    key[j] = in ? kq[i] : 0ull;
                    const uint32_t h = (uint32_t)(key[j] >> 32);
                    const bool keep = in && h >= rlo && (h > rhi || bsel < 0 || sel_bucket(h, smin, inv) >= bsel);
                    if (keep) km = min(km, h);
                    bal[j] = __ballot_sync(0xFFFFFFFFu, keep);
                    wtot += __popc(bal[j]);
                }
            }
            km = __reduce_min_sync(0xFFFFFFFFu, km);
            if (lane == 0) {
                wcnt[q * 32 + warp] = wtot;
                if (km != 0xFFFFFFFFu) atomicMin(&st[8 * q + 2], km);
            }
            __syncthreads();
            const int v = lane < (nt >> 5) ? wcnt[q * 32 + lane] : 0;
            int run = __reduce_add_sync(0xFFFFFFFFu, lane < warp ? v : 0);
            const int total = __reduce_add_sync(0xFFFFFFFFu, v);
#pragma unroll
            for (int j = 0; j < 10; ++j) {
                if (j < R) {
                    if (bal[j] >> lane & 1u) kq[run + __popc(bal[j] & ((1u << lane) - 1u))] = key[j];
                    run += __popc(bal[j]);
                }
            }
            if (tid == 0) st[8 * q + 5] = (uint32_t)total;
        }
        __syncthreads();
    } else {
        float smin[4], inv[4];
        uint32_t rlo[4], rhi[4];
        int bsel[4];
        uint32_t kmin[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            kmin[q] = 0xFFFFFFFFu;
            rlo[q] = rhi[q] = 0u;
            bsel[q] = 0;
            smin[q] = inv[q] = 0.0f;
            if (q < nq && st[8 * q + 6]) {
                rlo[q] = st[8 * q];
                rhi[q] = st[8 * q + 1];
                bsel[q] = (int)st[8 * q + 7];
                if (!sel_range(rlo[q], rhi[q], smin[q], inv[q])) bsel[q] = -1;  // whole range stays
            }
        }
        for (int i0 = 0; i0 < maxc; i0 += nt) {
            const int i = i0 + tid;
            uint64_t key[4];
            bool keep[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const bool in = q < nq && st[8 * q + 6] && i < cnt[q];
                key[q] = in ? keys[(size_t)q * cap + i] : 0ull;
                const uint32_t h = (uint32_t)(key[q] >> 32);
                keep[q] = in && h >= rlo[q] && (h > rhi[q] || bsel[q] < 0 || sel_bucket(h, smin[q], inv[q]) >= bsel[q]);
                if (keep[q]) kmin[q] = min(kmin[q], h);
            }
            __syncthreads();  // every read of this round precedes its writes (they land below i0 + nt)
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const unsigned bal = __ballot_sync(0xFFFFFFFFu, keep[q]);
                if (bal) {
                    int base = 0;
                    if (lane == 0) base = (int)atomicAdd(&st[8 * q + 5], (uint32_t)__popc(bal));
                    base = __shfl_sync(0xFFFFFFFFu, base, 0);
                    if (keep[q]) keys[(size_t)q * cap + base + __popc(bal & ((1u << lane) - 1u))] = key[q];
                }
            }
        }
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            if (q >= nq || !st[8 * q + 6]) continue;
            const uint32_t m = __reduce_min_sync(0xFFFFFFFFu, kmin[q]);
            if (lane == 0 && m != 0xFFFFFFFFu) atomicMin(&st[8 * q + 2], m);
        }
        __syncthreads();
    }
    // the new pivot: the smallest score kept, provided k keys were kept (fewer prove nothing)
    if (tid < 4 && st[8 * tid + 6]) {
        cnt[tid] = (int)st[8 * tid + 5];
        const uint64_t np = st[8 * tid + 2] == 0xFFFFFFFFu ? 0ull : (uint64_t)st[8 * tid + 2] << 32;
        if (st[8 * tid + 5] >= k && np > pivot[tid]) pivot[tid] = np;
    }
    uint32_t ties = 0u;
#pragma unroll
    for (int q = 0; q < 4; ++q)
        if (st[8 * q + 6] && st[8 * q + 4] && st[8 * q + 5] > k + slack) ties |= 1u << q;
    __syncthreads();
    return ties;
}


// ---- streaming top-k state shared by all CTAs -----------------------------------------------
// Per query row, in global memory (L2-resident), zeroed by one memset per call:
//   gpivot  best proven lower bound of the row's k-th best composite key (score word in the high half)
//   grange  bucket mapping (smin, inv) of the row's score histogram, 0 = none yet
//   gcount  candidates appended to the row's buffer so far
//   gflag   1 = the generic kernel scores the row's work items instead (a tile of another codec,
//           a query outside the fp16 split, or a full candidate buffer)
//   ghist   256 bucket counts of the appended candidates
// and one candidate buffer of gcap composite keys per row.  A CTA keeps no candidates of its own:
// a tile whose score reaches the row's threshold is appended to the row's buffer (one atomic per
// warp, query and set), counted in the row's histogram, and the threshold is re-derived from that
// histogram from time to time - the counts are of real tiles, so the lower edge of the highest
// bucket whose count from the top reaches k is a proven lower bound of the k-th best score, for
// all CTAs at once.

// A whole warp: the bound that a row's histogram proves (0 = none): the lower edge of the highest bucket whose count from the
// top reaches k, minus half a bucket and a few ulps: every counted key of the buckets from there on is above it whatever
// the rounding of the bucket arithmetic.  r: the row's bucket mapping.
__device__ __forceinline__ uint32_t hist_bound(const uint32_t* hist, float2 r, uint32_t k, int lane) {
    const uint32_t* hq = hist + 248 - 8 * lane;
    uint32_t c[8];  // buckets 255-8l .. 248-8l (descending)
    asm volatile("ld.volatile.global.v4.u32 {%0,%1,%2,%3}, [%4];\n" : "=r"(c[7]), "=r"(c[6]), "=r"(c[5]), "=r"(c[4]) : "l"(hq));
    asm volatile("ld.volatile.global.v4.u32 {%0,%1,%2,%3}, [%4];\n" : "=r"(c[3]), "=r"(c[2]), "=r"(c[1]), "=r"(c[0]) : "l"(hq + 4));
    uint32_t tot = 0;
#pragma unroll
    for (int jj = 0; jj < 8; ++jj) tot += c[jj];
    uint32_t incl = tot;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, incl, o);
        if (lane >= o) incl += y;
    }
    const unsigned ok = __ballot_sync(0xFFFFFFFFu, incl >= k);
    uint32_t ek = 0;
    if (ok != 0u && lane == __ffs(ok) - 1) {
        uint32_t run = incl - tot;
        int b = 0;
#pragma unroll
        for (int jj = 0; jj < 8; ++jj) {
            if (run + c[jj] >= k) { b = 255 - 8 * lane - jj; break; }
            run += c[jj];
        }
        if (b >= 1) {
            const uint32_t e = score_key(r.x + ((float)b - 0.5f) / r.y);
            ek = e > 8u ? e - 8u : 0u;
        }
    }
    return __reduce_max_sync(0xFFFFFFFFu, ek);
}

// A whole warp: raise the threshold of query row Q (shared word *pvh) from the row's histogram
// and from what other CTAs have proven.
__device__ __forceinline__ void stream_refresh_threshold(const ScoreArgs& a, uint32_t Q, float2 r, uint32_t* pvh, int lane) {
    const unsigned long long seen = *reinterpret_cast<volatile unsigned long long*>(a.gpivot + Q);
    uint32_t best = (uint32_t)(seen >> 32);
    if (r.y != 0.0f) {
        const uint32_t ek = hist_bound(a.ghist + (size_t)Q * 256, r, a.k, lane);
        if (ek > best) {
            best = ek;
            if (lane == 0) atomicMax(a.gpivot + Q, (unsigned long long)ek << 32);
        }
    }
    if (lane == 0 && best > *reinterpret_cast<volatile uint32_t*>(pvh)) atomicMax(pvh, best);
}

// A whole warp, once a row's candidates are all in its buffer: the row's threshold from its complete histogram.  Calls whose
// rows are scored in a round or two have raised none, or a stale one, while scoring.
__device__ __forceinline__ unsigned long long final_threshold(const uint32_t* hist, unsigned long long pivot, unsigned long long mapping, uint32_t k, int lane) {
    const float2 r = make_float2(__uint_as_float((uint32_t)mapping), __uint_as_float((uint32_t)(mapping >> 32)));
    const unsigned long long e = r.y != 0.0f ? (unsigned long long)hist_bound(hist, r, k, lane) << 32 : 0ull;
    return e > pivot ? e : pivot;
}

// KIND 0: nibble codecs (INT4, MX-INT4, NF4 through the shared-memory table); 1: the launch scores
// mixed 8/4 tiles; 2: TQ3 tiles, rewritten in shared memory as nibble rows (2 code + correction
// bit) before the INT4 path scores them; 3: INT4 / MX-INT4 tiles only (scale folded into A).
// Separate instantiations.  A tile of another codec than the launch was arranged for flags the
// work item's query rows, which the generic kernel then scores.
// IL: the work items are interleaved shares of whole streams (see the planner); the plain instantiation keeps the
// set arithmetic of contiguous ranges out of its loop.
// LONG: see stream_long.  FULL: what its rows pay for is there (seeds, and the question whether a tile can reach the threshold).
// U: a warp takes U x 16 tiles at a time.  The kernel is bound by instruction issue, and what a set costs beside its sums (fetch, flags, votes, thresholds,
// query fragments) is paid once for both halves of a set of 32.
template <int KIND, bool IL, bool LONG>
__global__ void __launch_bounds__(STREAM_THREADS, 1) score_stream_kernel(ScoreArgs a) {
    extern __shared__ __align__(16) unsigned char smem[];
    dep_launch();
    dep_wait();
    constexpr int U = stream_sets(KIND, LONG), nwarps = STREAM_THREADS / 32, R = 2 * U, SET_TILES = MMA_SET_TILES * U, SET_STRIDE = SET_TILES * MMA_ROW;
    constexpr bool FULL = IL || LONG || KIND == 3;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int g = lane >> 2, t = lane & 3;
    uint2* bq_w = reinterpret_cast<uint2*>(smem);                        // [9][32]
    uint32_t* qs_w = reinterpret_cast<uint32_t*>(smem + MMA_BQ_BYTES);   // [4][8]
    uint32_t* pvh = qs_w + 32;                                           // [4] score word of the row's threshold
    float2* rng = reinterpret_cast<float2*>(pvh + 4);                    // [4] (smin, inv), inv 0 = none yet
    float2* rmap = rng + 4;                                              // [4] (-smin * inv, inv): the same mapping as the hot path uses it
    int* bail = reinterpret_cast<int*>(rmap + 4);                        // [1]
    const uint32_t smem_s = (uint32_t)__cvta_generic_to_shared(smem);
    const uint32_t bqa = smem_s + (uint32_t)lane * 8u;
    const uint32_t qsa = smem_s + MMA_BQ_BYTES + (uint32_t)t * 32u;
    constexpr int LOW = KIND == 0 ? stream_low_warps(U) : nwarps;
    const uint32_t stage_s = warp < LOW ? smem_s + MMA_TAIL_BYTES + (uint32_t)warp * stream_slot(U) : STREAM_LUT_AT + STREAM_LUT_BYTES + (uint32_t)(warp - LOW) * stream_slot(U);

    if (KIND == 0 && smem_s > 2048u) {  // (never: the layout above needs dynamic shared memory to start below 2 KB)
        for (uint32_t i = a.cta_begin[blockIdx.x]; i < a.cta_begin[blockIdx.x + 1]; ++i)
            if (tid < (int)a.stream_items[i].n_queries) a.gflag[a.stream_items[i].query_begin + tid] = 1u;
        return;
    }
    if (KIND == 0) {
        // NF4 codebook as fp16 hi + lo pairs per byte (two nibbles), a column for every lane
        uint2* lut = reinterpret_cast<uint2*>(smem + (STREAM_LUT_AT - smem_s));
        for (int e = tid; e < 256 * 32; e += 32 * nwarps) {
            const int b = e >> 5;
            const float c0 = c_nf4[b & 15], c1 = 16.0f * c_nf4[b >> 4];  // odd slots carry 16x (see int4_quad)
            lut[e] = make_uint2(pack_half2(c0, c1), pack_half2(half_residual(c0), half_residual(c1)));
        }
    }
    const uint32_t lut_lane = STREAM_LUT_AT + (uint32_t)lane * 8u;
    uint32_t magic;  // 1024.0h twice, opaque so that it stays in one register
    asm volatile("mov.u32 %0, 0x64006400;\n" : "=r"(magic));
    // cp.async of a set: lane copies the 16-byte chunks lane, lane+32, .., i.e. chunk (lane & 7) of rows (lane >> 3) + {0, 4, 8, ..}
    const uint32_t dst_lane = (uint32_t)((lane >> 3) * MMA_ROW + (lane & 7) * 16);
    const uint32_t row_lane = (uint32_t)g * MMA_ROW;
    const uint32_t lt_mask = (1u << lane) - 1u, t_mask = 0x11111111u << t;
    uint64_t stream_policy;
    asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;\n" : "=l"(stream_policy));

    const uint32_t item_end = a.cta_begin[blockIdx.x + 1];
    for (uint32_t item_id = a.cta_begin[blockIdx.x]; item_id < item_end; ++item_id) {
        const WorkItem it = a.stream_items[item_id];
        const int nq = (int)it.n_queries;
        // interleaved: this CTA is number il_c of the il_n CTAs that share the stream [tile_begin, + n_tiles); round r of
        // the stream's static deal belongs to CTA r mod il_n.  Otherwise the item is this CTA's own range.
        constexpr bool il = IL;
        const uint32_t il_n = il ? ((it.pad >> 8) & 0x7FFFFFu) : 1u, il_c = il ? it.list_begin : 0u;
        __syncthreads();  // previous item fully retired (and the table is visible)
        // The first sets are fetched before anything else of the item is prepared: the copy runs while the query
        // fragments are built.
        const uint8_t* sbase = a.state ? a.state + it.tile_begin : nullptr;
        const uint32_t n = it.n_tiles;
        uint32_t n_sets = (n + SET_TILES - 1) / SET_TILES;
        const uint32_t n_full = n / SET_TILES;
        const bool mine = t < nq;
        const uint32_t Qt = it.query_begin + (mine ? (uint32_t)t : 0u);  // the row whose scores this thread finishes
        uint64_t* const dst = a.gbuf + (size_t)Qt * a.gcap;                // the row's candidate buffer
        uint32_t* const hrow = a.ghist + (size_t)Qt * 256;                 // and its histogram
        // sets are dealt to the warps round by round: warp w takes set j * nwarps + w of round j
        const unsigned char* tbase = a.tiles + it.tile_begin * TILE_BYTES + lane * 16;
        // This CTA's rounds of the deal, r = il_c, il_c + il_n, ..; an interleaved CTA walks them starting from a place of its
        // own and wraps around (CTA c of C starts c / C of the way through), so that at any moment the CTAs of a stream are
        // spread over the whole stream -- the first thresholds then come from a sample of all positions even when one
        // end of the stream holds nothing to score (the oldest slots of a pool are mostly COLD).
        const uint32_t all_rounds = (n_sets + (uint32_t)nwarps - 1) / (uint32_t)nwarps;
        const uint32_t my_rounds = all_rounds > il_c ? (all_rounds - il_c + il_n - 1) / il_n : 0u;  // (the same for all warps of the CTA)
        const uint32_t first_round = il ? (uint32_t)(((uint64_t)il_c * my_rounds) / il_n) : 0u;
        auto set_of = [&](uint32_t i) {  // the set this warp takes in its i-th iteration
            if (!il) return i * (uint32_t)nwarps + (uint32_t)warp;
            uint32_t j = i + first_round;
            if (j >= my_rounds) j -= my_rounds;
            return (j * il_n + il_c) * (uint32_t)nwarps + (uint32_t)warp;
        };
        uint32_t iss_no = 0, slot_next = 0;
        auto issue = [&]() {
            const uint32_t s_next = iss_no < my_rounds ? set_of(iss_no) : 0xFFFFFFFFu;
            ++iss_no;
            if (s_next < n_sets) {
                const uint32_t dst = stage_s + slot_next + dst_lane;
                const unsigned char* src = tbase + (size_t)s_next * (SET_TILES * TILE_BYTES);
                if (s_next < n_full) {
                    cp_async16_sp<0, 0>(dst, src, 16, stream_policy);
                    cp_async16_sp<512, 4 * MMA_ROW>(dst, src, 16, stream_policy);
                    cp_async16_sp<1024, 8 * MMA_ROW>(dst, src, 16, stream_policy);
                    cp_async16_sp<1536, 12 * MMA_ROW>(dst, src, 16, stream_policy);
                    if (U == 2) {
                        cp_async16_sp<2048, 16 * MMA_ROW>(dst, src, 16, stream_policy);
                        cp_async16_sp<2560, 20 * MMA_ROW>(dst, src, 16, stream_policy);
                        cp_async16_sp<3072, 24 * MMA_ROW>(dst, src, 16, stream_policy);
                        cp_async16_sp<3584, 28 * MMA_ROW>(dst, src, 16, stream_policy);
                    }
                } else {
                    // ragged last set: rows past the end are zero-filled (source not read)
                    const uint32_t r = s_next * SET_TILES + (uint32_t)(lane >> 3);
#pragma unroll 1
                    for (uint32_t q = 0; q < 4u * U; ++q) {
                        const bool in = r + 4u * q < n;
                        cp_async16_s<0, 0>(dst + q * (4u * MMA_ROW), in ? src + 512u * q : a.tiles, in ? 16 : 0);
                    }
                }
            }
            cp_async_commit();
            slot_next = slot_next == (MMA_DEPTH - 1) * SET_STRIDE ? 0u : slot_next + SET_STRIDE;
        };
#pragma unroll
        for (int i = 0; i < MMA_DEPTH - 1; ++i) issue();
        bool row_warm = true;
        if (tid < 4) {
            // start from the threshold other CTAs have already proven for the row, and from the
            // row's bucket mapping if one has been published
            const bool have = tid < nq;
            const unsigned long long pv = have ? *reinterpret_cast<volatile unsigned long long*>(a.gpivot + it.query_begin + tid) : 0ull;
            pvh[tid] = (uint32_t)(pv >> 32);
            row_warm = !have || (uint32_t)(pv >> 32) != 0u;
            const unsigned long long pr = have ? *reinterpret_cast<volatile unsigned long long*>(a.grange + it.query_begin + tid) : 0ull;
            rng[tid] = make_float2(__uint_as_float((uint32_t)pr), __uint_as_float((uint32_t)(pr >> 32)));
            rmap[tid] = make_float2(-rng[tid].x * rng[tid].y, rng[tid].y);
        }
        if (tid == 0) bail[0] = 0;
        if (warp == 1 % nwarps) {
            // sign words of the item's (up to four) queries
            const int qi = lane >> 3;
            qs_w[lane] = qi < nq ? a.q_sign[(size_t)(it.query_begin + qi) * 8 + (lane & 7)] : 0u;
        }
        bool big = false;
        if (warp == 0) {
            // B fragments: column n = g is query g>>1, part g&1 (fp16 hi / lo of the query)
            const int qi = g >> 1;
            const bool have = qi < nq;
            const float* q = a.q_coarse + (size_t)(it.query_begin + (have ? qi : 0)) * D_C;
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                float v[4];
                if (KIND == 3) {
                    // MMA j takes nibbles (o, o + 4 | o + 1, o + 5), o = 2 (j & 1), of the thread's word j >> 1
                    const float* qd = q + 32 * t + 8 * (j >> 1) + 2 * (j & 1);
                    v[0] = qd[0]; v[1] = qd[4]; v[2] = qd[1]; v[3] = qd[5];
                } else {
                    // k slots {2t, 2t+1, 2t+8, 2t+9} of group j carry dims 16j + 4t + {0,1,2,3}; mixed 8/4 tiles:
                    // group 0 = dims 2t, 2t+1 (8-bit levels, plain in both slots, so both carry 16x the
                    // query), groups 1..7 = INT4 groups of dims 16 j - 8 ..
                    const int dim0 = !(KIND == 1) ? 16 * j + 4 * t : (j == 0 ? 0 : 16 * j - 8 + 4 * t);
                    float4 x = load_q4(q + dim0);
                    if (KIND == 1 && j == 0) x = make_float4(q[2 * t], 16.0f * q[2 * t + 1], 0.0f, 0.0f);
                    v[0] = x.x; v[1] = x.y; v[2] = x.z; v[3] = x.w;
                }
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    if (!have) v[i] = 0.0f;
                    if (KIND == 3) {
                        big |= fabsf(v[i]) > 60000.0f;
                    } else {
                        big |= fabsf(v[i]) > (KIND == 1 && j == 0 && i == 1 ? 64000.0f : 4000.0f);  // 16 v must stay inside fp16
                        if (!(i & 1)) v[i] *= 16.0f;  // even slots carry 16x the query (see int4_quad)
                    }
                    if (g & 1) v[i] = half_residual(v[i]);
                }
                bq_w[j * 32 + lane] = make_uint2(pack_half2(v[0], v[1]), pack_half2(v[2], v[3]));
            }
            uint32_t bE = 0;
            if (KIND == 2) {
                // B fragment of the group sums: k slots 2t and 2t+1 = groups 2t and 2t+1 of query g>>1
                float s0 = 0.0f, s1 = 0.0f;
#pragma unroll
                for (int i = 0; i < 16; ++i) {
                    s0 += q[32 * t + i];
                    s1 += q[32 * t + 16 + i];
                }
                if (!have) s0 = s1 = 0.0f;
                big |= fabsf(s0) > 60000.0f || fabsf(s1) > 60000.0f;
                if (g & 1) { s0 = half_residual(s0); s1 = half_residual(s1); }
                bE = pack_half2(s0, s1);
            }
            bq_w[8 * 32 + lane] = make_uint2(bE, 0u);
            if (__any_sync(0xFFFFFFFFu, big) && lane == 0) bail[0] = 1;  // a query too large for the fp16 split
        }
        // (from a barrier's vote, not from the flag word: a fast warp may raise the flag for an undecodable tile meanwhile)
        const bool too_big = __syncthreads_or(big) != 0;
        // The barrier after the first round (below) pays when the round can supply k candidates to a row -- a set per warp
        // of every CTA that works on the row -- and the rows do not already have thresholds (a CTA that starts its
        // second item on rows other CTAs have been scoring for a while).
        const bool all_warm = __syncthreads_and(row_warm) != 0;
        const bool first_round_barrier = !all_warm && !too_big && (uint64_t)a.k <= (uint64_t)SET_TILES * (uint64_t)nwarps * (uint64_t)max((it.pad >> 8) & 0x7FFFFFu, 1u);
        // Of the first round only some warps append unfiltered; the others wait at that barrier with their first set, and filter it by the
        // thresholds of these seeds.  With N tiles in the first round of all CTAs on the row, S seeds and (N - S) k / S of the rest are appended,
        // least at S = sqrt(N k).  (With all 24 warps of 148 CTAs on one row 57 k tiles a row were appended at once: a million MX tiles, k = 100,
        // 81 us, with 7 seeds a CTA 60.)
        const uint32_t parts = max((it.pad >> 8) & 0x7FFFFFu, 1u);
        int seeds = nwarps;
        // (from N = 9 k on, where the seeds number 3 k: with k = 2048 of N = 6912 the seeds hardly prove a threshold before the rest is due,
        // 8 x 131 072 INT4 tiles 85 -> 100 us; and calls of two rounds have little to append: 8 x 8192 mixed tiles 29.1 -> 29.6 us)
        const uint64_t first_tiles = (uint64_t)SET_TILES * (uint64_t)nwarps * parts;
        if (FULL && first_round_barrier && my_rounds > 1u && first_tiles >= 9ull * a.k && (my_rounds > 2u || first_tiles >= 8192u))
            seeds = min(nwarps, max(1, (int)ceilf(sqrtf((float)nwarps * (float)a.k / ((float)SET_TILES * (float)parts)))));
        if (too_big) n_sets = 0;  // (the sets already on their way are waited for at the item's end and never read)

        uint32_t slot = 0, polls = 0;
        uint32_t cur = 0, end = 0;  // this warp's chunk of the buffer of row Qt (the same in the eight lanes of a query)
        bool dead = false;          // this warp met a tile it cannot decode
        const uint32_t rounds = too_big ? 0u : my_rounds;
        for (uint32_t round = 0; round < rounds; ++round) {
            const uint32_t s = set_of(round);
            if (round == (!FULL || warp < seeds ? 1u : 0u) && first_round_barrier) {
                // The seeds of the CTA (and, started together, of the grid) have appended their first sets
                // unfiltered, so the rows' histograms hold a set's candidates per seed: first thresholds now,
                // before the other sets are filtered.  (All warps pass here: `rounds` is the same for all, and at least two where there are
                // fewer seeds than warps.)  Other CTAs may be a little behind: a few tries.
                __syncthreads();
                if (warp < nq) {
                    for (int tries = FULL && seeds < nwarps ? 4 : 1; tries; --tries) {
                        stream_refresh_threshold(a, it.query_begin + (uint32_t)warp, rng[warp], pvh + warp, lane);
                        __syncwarp();
                        if (reinterpret_cast<volatile uint32_t*>(pvh)[warp] != 0u || tries == 1) break;
                        __nanosleep(400);
                    }
                }
                __syncthreads();
            }
            // (the ring advances in every iteration, also when this warp has no set in this round -- the short last round of
            // the stream can come anywhere in a rotated walk -- so that fetches and reads stay in step)
            issue();
            cp_async_wait<MMA_DEPTH - 1>();
            __syncwarp();
            const uint32_t rb = stage_s + slot + row_lane;
            slot = slot == (MMA_DEPTH - 1) * SET_STRIDE ? 0u : slot + SET_STRIDE;
            if (dead || s >= n_sets) continue;
            const bool ragged = s >= n_full;
            const uint32_t t0 = s * SET_TILES + (uint32_t)g;  // row r of this thread is tile t0 + 8 r
            uint32_t f[R], fo = 0, fa = 0xFFFFFFFFu;
            uint2 gs[R];
#pragma unroll
            for (int r = 0; r < R; ++r) {
                if (KIND == 3) {
                    f[r] = lds_u16<118>(rb + (uint32_t)(r * MMA_HALF));
                } else {
                    const uint4 x = lds_v4<112>(rb + (uint32_t)(r * MMA_HALF));  // position, head|flags, gs[8]
                    f[r] = x.y >> 16;
                    gs[r] = make_uint2(x.z, x.w);
                }
                fo |= f[r];
                // (rows past the end of a ragged last set are zero-filled and their scores dropped: they count as tiles of the launch's codec)
                if (KIND == 1 || KIND == 2) fa &= !ragged || t0 + 8u * r < n ? f[r] : 0xFFFFFFFFu;
                if (KIND == 0) fa &= f[r];
            }
            fo = __reduce_or_sync(0xFFFFFFFFu, fo);
            if (KIND != 3) fa = __reduce_and_sync(0xFFFFFFFFu, fa);
            // a launch arranged for mixed 8/4 (TQ3) tiles takes nothing else
            const bool odd = KIND == 3 ? (fo & (F_MIX3 | F_TQ3 | F_MIXED | F_NF4)) != 0
                           : KIND == 2 ? (fo & (F_MIX3 | F_MIXED)) || !(fa & F_TQ3)
                           : KIND == 1 ? (fo & (F_MIX3 | F_TQ3)) || !(fa & F_MIXED)
                                       : (fo & (F_MIX3 | F_TQ3 | F_MIXED)) != 0;
            if (odd) {
                if (lane == 0) bail[0] = 1;  // a codec this launch does not decode: the generic kernel takes the rows
                dead = true;
                continue;
            }
            float c[R];
            const uint32_t hb = rb + 2u * (uint32_t)t;
            if (KIND == 3) {
                coarse_set_int4c<U>(rb, (uint32_t)t, magic, bqa, c);
            } else if (KIND == 2) {
#pragma unroll
                for (int u = 0; u < U; ++u) tq3_to_nibbles(rb - row_lane + (uint32_t)(2 * u * MMA_HALF), lane);
                coarse_set<0, U>(hb, lut_lane, magic, bqa, f, gs, c);
                // level = (2 nibble - 15) / 4, or (2 nibble - 14) / 4 without the correction plane:
                // beside the nibble sums X the score needs 8 c sum_g gs_g Q_g (c = 1 or 2, Q_g = the
                // query's sum over group g), one more MMA with the scale bytes as the A operand
                const uint32_t sel = (t & 1) ? 0x7352u : 0x7150u;
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    uint32_t ga0, ga1;
                    asm("add.rn.f16x2 %0, %1, %2;\n" : "=r"(ga0) : "r"(prmt(t < 2 ? gs[2 * u].x : gs[2 * u].y, magic, sel)), "r"(0xE400E400u));
                    asm("add.rn.f16x2 %0, %1, %2;\n" : "=r"(ga1) : "r"(prmt(t < 2 ? gs[2 * u + 1].x : gs[2 * u + 1].y, magic, sel)), "r"(0xE400E400u));
                    float e[4];
                    mma_f16_zero(e, ga0, ga1, 0u, 0u, lds_v2<256 * 8>(bqa).x, 0u);
                    c[2 * u] = fmaf((f[2 * u] & F_NOCORR) ? 16.0f : 8.0f, e[0] + e[1], c[2 * u]);
                    c[2 * u + 1] = fmaf((f[2 * u + 1] & F_NOCORR) ? 16.0f : 8.0f, e[2] + e[3], c[2 * u + 1]);
                }
            } else if (KIND == 1) {
                coarse_set<3, U>(hb, lut_lane, magic, bqa, f, gs, c);
            } else if (fa & F_NF4) {
                coarse_set<1, U>(hb, lut_lane, magic, bqa, f, gs, c);
            } else if (!(fo & F_NF4)) {
                coarse_set<0, U>(hb, lut_lane, magic, bqa, f, gs, c);
            } else {
                coarse_set<2, U>(hb, lut_lane, magic, bqa, f, gs, c);
            }
            // 1 / (255 x 16 [x 2]); KIND 3: the sums carry 2^-16
            constexpr float unit = KIND == 3 ? 65536.0f / 255.0f : (KIND == 2 ? 1.0f / 8160.0f : 1.0f / 4080.0f);
            const float thr = thr_float(reinterpret_cast<const volatile uint32_t*>(pvh)[t]);
            // The residual term lies in [-256 |lambda|, 256 |lambda|]: rows none of whose tiles can reach the threshold even with the largest
            // term need no Hamming distances (and append nothing).  (257 and the relative slack cover the rounding of the bound
            // itself; a NaN passes.)  Long INT4 launches ask for eight tiles at a time, the others for the set; not asked where most rows are short
            // beside k (a decode step's caches: one tile in seven is appended, and some tile of a set nearly always), see stream_long.
            constexpr int GATE = KIND == 3 && U == 2 ? 1 : R;  // rows asked for at a time
            float sc[R], lam[R];
            uint32_t b[R], some = 0;
            bool p[R];
#pragma unroll
            for (int r = 0; r < R; ++r) {
                const uint2 m = lds_v2<96>(rb + (uint32_t)(r * MMA_HALF));  // scale, lambda
                lam[r] = (f[r] & F_WARM) ? 0.0f : __uint_as_float(m.y);
                sc[r] = c[r] * (__uint_as_float(m.x) * unit);
                p[r] = mine && (!FULL || !(fmaf(fabsf(lam[r]), 257.0f, fmaf(fabsf(sc[r]), 1e-6f, sc[r])) < thr));
                b[r] = 0u;
            }
#pragma unroll
            for (int r0 = 0; r0 < R; r0 += GATE) {
                bool any = false;
#pragma unroll
                for (int r = r0; r < r0 + GATE; ++r) any = any || p[r];
                if (!FULL || __any_sync(0xFFFFFFFFu, any)) {
                    const uint4 qa = lds_v4<0>(qsa), qb = lds_v4<16>(qsa);
                    const uint32_t qs[8] = {qa.x, qa.y, qa.z, qa.w, qb.x, qb.y, qb.z, qb.w};
#pragma unroll
                    for (int r = r0; r < r0 + GATE; ++r) {
                        // Hamming term of query t for the row
                        const uint32_t row = rb + (uint32_t)(r * MMA_HALF);
                        const int h = popc8(lds_v4<64>(row), lds_v4<80>(row), qs);
                        // 256 - 2 h without an integer conversion: (2^23 + h) as a bit pattern, times -2, plus 2^24 + 256 (exact)
                        sc[r] = fmaf(lam[r], fmaf(__uint_as_float(0x4B000000u | (uint32_t)h), -2.0f, 16777472.0f), sc[r]);
                        // (a superset of the composite comparison: the merge drops keys below the final threshold)
                        p[r] = p[r] && !(sc[r] < thr) && (!ragged || t0 + 8u * r < n);
                        if (sbase) p[r] = p[r] && sbase[t0 + 8u * r] != ST_COLD;
                        b[r] = __ballot_sync(0xFFFFFFFFu, p[r]);
                        some |= b[r];
                    }
                }
            }
            if (round == 0) {
                // First set of the warp: a row without a bucket mapping gets one from the scores
                // this warp has just computed for it - their range widened by 1.5 spans on both sides.
                // Any monotone mapping is valid; this one only has to put the final threshold somewhere
                // inside its 256 buckets.  The first CTA to publish wins.
                float mn = INFINITY, mx = -INFINITY;
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    mn = fminf(mn, p[r] ? sc[r] : INFINITY);
                    mx = fmaxf(mx, p[r] ? sc[r] : -INFINITY);
                }
#pragma unroll
                for (int o = 4; o < 32; o <<= 1) {
                    mn = fminf(mn, __shfl_xor_sync(0xFFFFFFFFu, mn, o));
                    mx = fmaxf(mx, __shfl_xor_sync(0xFFFFFFFFu, mx, o));
                }
                if (g == 0 && mine && rng[t].y == 0.0f) {
                    unsigned long long pr = *reinterpret_cast<volatile unsigned long long*>(a.grange + Qt);
                    if (!pr && mx > mn) {
                        const float span = mx - mn, lo = mn - 1.5f * span, inv = 256.0f / (4.0f * span);
                        if (isfinite(lo) && isfinite(inv) && inv > 0.0f) {
                            const unsigned long long mine_r = (unsigned long long)__float_as_uint(lo) | ((unsigned long long)__float_as_uint(inv) << 32);
                            const unsigned long long old = atomicCAS(a.grange + Qt, 0ull, mine_r);
                            pr = old ? old : mine_r;
                        }
                    }
                    if (pr) {
                        rng[t] = make_float2(__uint_as_float((uint32_t)pr), __uint_as_float((uint32_t)(pr >> 32)));
                        rmap[t] = make_float2(-rng[t].x * rng[t].y, rng[t].y);
                    }
                }
                __syncwarp();
            }
            if (some) {
                // The eight lanes of query t append to the row's buffer, slots by ballot.  The warp owns a
                // chunk of slots per row, [cur, end); a set that does not fit takes what is left of it and the start of a new chunk,
                // reserved with one atomic.  What is unused at the end of the work item is zeroed (absent keys).
                uint32_t nn = 0, first[R];
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    first[r] = nn + (uint32_t)__popc(b[r] & t_mask & lt_mask);
                    nn += (uint32_t)__popc(b[r] & t_mask);
                }
                const uint32_t left = end - cur;
                uint32_t fresh = cur;  // where the candidates beyond `left` go, minus `left`
                if (nn > left) {  // (the same in the eight lanes of a query, which are the lanes of t_mask)
                    const uint32_t size = nn - left > MMA_CHUNK ? 2 * MMA_CHUNK : MMA_CHUNK;
                    uint32_t base = 0;
                    if (g == 0) {
                        base = atomicAdd(a.gcount + Qt, size);
                        if (base + size > a.gcap) {
                            // the row's buffer is full: the generic kernel scores the row; this warp's further
                            // candidates of the row land in the buffer's last slots, which nobody reads then
                            a.gflag[Qt] = 1u;
                            base = a.gcap - size;
                        }
                    }
                    base = __shfl_sync(t_mask, base, t);  // lane t is (g = 0, t)
                    fresh = base - left;
                    end = base + size;
                }
                // bucket of the row's histogram: (int)(score * inv - smin * inv), clamped; scores below the
                // mapping (and all scores while the row has no mapping) count in bucket 0, which never decides
                const float2 map = rmap[t];
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    if (p[r]) {
                        dst[(first[r] < left ? cur : fresh) + first[r]] = ((uint64_t)score_key(sc[r]) << 32) | (uint64_t)(~(it.index_base + t0 + 8u * r));
                        atomicAdd(hrow + min(max(__float2int_rz(fmaf(sc[r], map.y, map.x)), 0), 255), 1u);
                    }
                }
                cur = nn > left ? fresh + nn : cur + nn;
            }
            __syncwarp();
            // In turn, a warp raises the threshold of query (warp & 3): early on (the first
            // thresholds come from the barrier after the first round), then every 256 tiles, the warps of a
            // query staggered.  A stale threshold costs appends (each one a store, a
            // histogram count and, downstream, merge work), a refresh costs one 1 KB read of the row's
            // histogram by one warp.
            ++polls;
            constexpr uint32_t every = 16 / U;
            if ((polls & (every - 1u)) == (uint32_t)((warp >> 2) & 3) * (every / 4u) + (every / 4u - 1u) || polls == 4u / U - (U == 1) || polls == 8u / U - (U == 1)) {
                const int q = warp & 3;
                if (q < nq) stream_refresh_threshold(a, it.query_begin + (uint32_t)q, rng[q], pvh + q, lane);
                __syncwarp();
            }
        }
        cp_async_wait<0>();
        if (mine) {  // the unused rest of the warp's last chunk holds absent keys
            for (uint32_t z = cur + (uint32_t)g; z < end; z += 8u) dst[z] = 0ull;
        }
        __syncthreads();
        // rows this CTA could not score on the tensor cores go to the generic kernel as a whole
        if (bail[0] && tid < nq) a.gflag[it.query_begin + tid] = 1u;
    }
}

}  // namespace
}  // namespace slha
