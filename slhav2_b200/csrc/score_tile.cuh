// One thread per tile, tcgen05 with the tiles in TMEM: the top-k of MIX3 tiles (score_mix3_kernel) and dense scores of every codec
// (score_dense_kernel) for up to four queries per tile.  Included by score.cu after score_mma.cuh; score_wide.cuh shares the decode.
//
// A thread reads its tile's 64 latent bytes from shared memory, turns them into exact fp16 products (level x scale byte) in
// registers and writes them as its row of the A operand into TMEM; tcgen05.mma multiplies the 128 rows of a warpgroup with
// the queries (scaled to one size, fp16 hi + lo columns, 22 bits or more) and the thread reads its finished coarse scores back.  Scale, lambda, flags
// and scale bytes are each read by one thread, where the fragments of warp-level MMAs need them in four lanes each.
//
// Bound: the chain of a block (decode, TMEM store, eight or nine MMAs, read-back, filter or finish) with four warpgroups in flight; a scheduler issues in 47 % of the cycles.  Dense scores
// of 8 x 131 072 tiles, us a call for 4 rows / one: mixed 56 / 50 -> 42 / 36, NF4 78 / 72 -> 63 / 54, MIX3 65 / 60 -> 48 / 43 by the sums in pairs (f32x2), full adders in front of
// POPC, row addresses and slot states read ahead, the queries asked for before the tiles.
// MIX3 top-k of 32 ragged segments (485 k tiles x 4 queries): 367 -> 72 us a call streamed (dense scores and a selection: 40); dense MIX3 scores of 8 x 4096
// tiles x 4 rows: 278 -> 17 us a call (6 of kernel).  Top-k of the codecs that score_stream_kernel
// decodes, over long rows, stays there: on 8.4 M MX-INT4 tiles a call takes 308 us with this kernel and 237 with that one, on as many NF4 tiles earlier forms of both took 573 and 462.
#pragma once

namespace slha {
namespace {

constexpr int ST_M = 128;                              // tiles of a warpgroup's block = rows of an MMA
constexpr int ST_WT = 32;                              // tiles of a warp
constexpr int ST_ROW = TILE_BYTES + 16;                // padded row of the staging ring: a warp's 16-byte loads of 32 rows touch every bank once
constexpr int ST_SLOT = ST_WT * ST_ROW;
constexpr int ST_DEPTH = 2;                            // ring slots per warp
constexpr uint32_t ST_CHUNK = 32;                      // slots a warp reserves at a time in a row's candidate buffer
constexpr int ST_B_BYTES = 8192;                       // B operand: up to 3 slabs of 2 KB (64 K slots of 16 rows)
constexpr int ST_TAIL_BYTES = 128 + 16 + 16 + 32 + 32 + 64 + 32 + 256;
// KIND 0: NF4 (and INT4) tiles, 1: mixed 8/4, 2: TQ3, 3: INT4 / MX-INT4, 4: MIX3
constexpr int ST_WG = 4, ST_THREADS = 128 * ST_WG;     // warpgroups per CTA
constexpr uint32_t ST_TMEM = 128;                      // TMEM columns of a warpgroup: A in the first 64 (72 for the 3-bit kinds), accumulators behind it
// Accumulators of 16 columns that a block's MMAs rotate through, added on the CUDA cores: a chain of eight sums in one
// accumulator left 1.1e-7 relative error against 64 bits on MX-INT4 scores, chains of two or three 6.2e-8 (mma.sync: 6.6e-8).  NF4:
// one per scale group of a half.
constexpr int st_accs(int kind) { return kind == 2 || kind == 4 ? 3 : 4; }
constexpr uint32_t st_d_col(int kind) { return kind == 2 || kind == 4 ? 72u : 64u; }
constexpr size_t st_smem_bytes(bool dense) {  // (only dense calls meet NF4 tiles here)
    return 1024 + (dense ? NF4_LUT_BYTES + 4 * UNDONE_WORDS : 0) + ST_B_BYTES + (size_t)(ST_THREADS / 32) * ST_DEPTH * ST_SLOT + ST_TAIL_BYTES;
}

// instruction descriptor: D fp32, A and B fp16, both K-major, N columns, M = 128
__host__ __device__ constexpr uint32_t tc_idesc(uint32_t n) { return (1u << 4) | ((n >> 3) << 17) | ((128u >> 4) << 24); }
// A from TMEM (one row per lane, two fp16 per 32-bit column), B from shared memory
__device__ __forceinline__ void st_mma(uint32_t d_tmem, uint32_t a_tmem, uint64_t db, uint32_t accumulate, uint32_t idesc = tc_idesc(16)) {
    asm volatile(
        "{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\n"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n}\n" ::"r"(d_tmem), "r"(a_tmem), "l"(db), "r"(idesc), "r"(accumulate)
        : "memory");
}
__device__ __forceinline__ void st_tmem_st16(uint32_t taddr, const uint32_t (&v)[16]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};\n" ::"r"(taddr),
                 "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]), "r"(v[10]), "r"(v[11]),
                 "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15])
                 : "memory");
}
__device__ __forceinline__ void st_tmem_st8(uint32_t taddr, const uint32_t (&v)[8]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};\n" ::"r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]),
                 "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7])
                 : "memory");
}
// sixteen columns from each of two places (one statement with the wait, so that nothing reads the registers before it)
__device__ __forceinline__ void st_tmem_ld16x2(uint32_t t0, uint32_t t1, uint32_t (&v)[16], uint32_t (&w)[16]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%32];\n"
                 "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%33];\n"
                 "tcgen05.wait::ld.sync.aligned;\n"
                 : "=&r"(v[0]), "=&r"(v[1]), "=&r"(v[2]), "=&r"(v[3]), "=&r"(v[4]), "=&r"(v[5]), "=&r"(v[6]), "=&r"(v[7]), "=&r"(v[8]), "=&r"(v[9]),
                   "=&r"(v[10]), "=&r"(v[11]), "=&r"(v[12]), "=&r"(v[13]), "=&r"(v[14]), "=&r"(v[15]), "=&r"(w[0]), "=&r"(w[1]), "=&r"(w[2]), "=&r"(w[3]),
                   "=&r"(w[4]), "=&r"(w[5]), "=&r"(w[6]), "=&r"(w[7]), "=&r"(w[8]), "=&r"(w[9]), "=&r"(w[10]), "=&r"(w[11]), "=&r"(w[12]), "=&r"(w[13]),
                   "=&r"(w[14]), "=&r"(w[15])
                 : "r"(t0), "r"(t1)
                 : "memory");
}
// eight columns of three or four accumulators, `step` columns apart
__device__ __forceinline__ void st_ld_accs(uint32_t t, uint32_t (&v)[3][8], uint32_t step = 16u) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%24];\n"
                 "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%8,%9,%10,%11,%12,%13,%14,%15}, [%25];\n"
                 "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%16,%17,%18,%19,%20,%21,%22,%23}, [%26];\n"
                 "tcgen05.wait::ld.sync.aligned;\n"
                 : "=&r"(v[0][0]), "=&r"(v[0][1]), "=&r"(v[0][2]), "=&r"(v[0][3]), "=&r"(v[0][4]), "=&r"(v[0][5]), "=&r"(v[0][6]), "=&r"(v[0][7]),
                   "=&r"(v[1][0]), "=&r"(v[1][1]), "=&r"(v[1][2]), "=&r"(v[1][3]), "=&r"(v[1][4]), "=&r"(v[1][5]), "=&r"(v[1][6]), "=&r"(v[1][7]),
                   "=&r"(v[2][0]), "=&r"(v[2][1]), "=&r"(v[2][2]), "=&r"(v[2][3]), "=&r"(v[2][4]), "=&r"(v[2][5]), "=&r"(v[2][6]), "=&r"(v[2][7])
                 : "r"(t), "r"(t + step), "r"(t + 2u * step)
                 : "memory");
}
__device__ __forceinline__ void st_ld_accs(uint32_t t, uint32_t (&v)[4][8], uint32_t step = 16u) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%32];\n"
                 "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%8,%9,%10,%11,%12,%13,%14,%15}, [%33];\n"
                 "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%16,%17,%18,%19,%20,%21,%22,%23}, [%34];\n"
                 "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%24,%25,%26,%27,%28,%29,%30,%31}, [%35];\n"
                 "tcgen05.wait::ld.sync.aligned;\n"
                 : "=&r"(v[0][0]), "=&r"(v[0][1]), "=&r"(v[0][2]), "=&r"(v[0][3]), "=&r"(v[0][4]), "=&r"(v[0][5]), "=&r"(v[0][6]), "=&r"(v[0][7]),
                   "=&r"(v[1][0]), "=&r"(v[1][1]), "=&r"(v[1][2]), "=&r"(v[1][3]), "=&r"(v[1][4]), "=&r"(v[1][5]), "=&r"(v[1][6]), "=&r"(v[1][7]),
                   "=&r"(v[2][0]), "=&r"(v[2][1]), "=&r"(v[2][2]), "=&r"(v[2][3]), "=&r"(v[2][4]), "=&r"(v[2][5]), "=&r"(v[2][6]), "=&r"(v[2][7]),
                   "=&r"(v[3][0]), "=&r"(v[3][1]), "=&r"(v[3][2]), "=&r"(v[3][3]), "=&r"(v[3][4]), "=&r"(v[3][5]), "=&r"(v[3][6]), "=&r"(v[3][7])
                 : "r"(t), "r"(t + step), "r"(t + 2u * step), "r"(t + 3u * step)
                 : "memory");
}

// One scale byte -> half2 (gs 2^8) for nibbles at bits 0..3 of a half (n 2^-24), (gs 2^4) for bits 4..7 (n 2^-20), and the
// offset -8 gs 2^-16: fma(n 2^-24, gs 2^8, -8 gs 2^-16) = (n - 8) gs 2^-16 has at most 11 significant bits and is a multiple
// of 2^-16, so it is exact in fp16 (subnormal below 2^-14).
struct NibScale { uint32_t g8, g4, c; };
__device__ __forceinline__ NibScale nib_scale(uint32_t gs_dup) {  // gs_dup: half2 of the scale byte as an integer
    NibScale s;
    asm("mul.rn.f16x2 %0, %1, %2;\n" : "=r"(s.g8) : "r"(gs_dup), "r"(0x5C005C00u));  // x 2^8
    asm("mul.rn.f16x2 %0, %1, %2;\n" : "=r"(s.g4) : "r"(gs_dup), "r"(0x4C004C00u));  // x 2^4
    asm("mul.rn.f16x2 %0, %1, %2;\n" : "=r"(s.c) : "r"(gs_dup), "r"(0x88008800u));   // x -2^-13
    return s;
}
// byte J of a word as half2 (b, b), an exact integer
template <int J>
__device__ __forceinline__ uint32_t byte_half2(uint32_t w, uint32_t magic) {
    uint32_t r;
    asm("add.rn.f16x2 %0, %1, %2;\n" : "=r"(r) : "r"(prmt(w, magic, 0x5050u + 0x0101u * J)), "r"(0xE400E400u));
    return r;
}
// eight nibbles -> four columns of A: dims 0,4 | 1,5 | 2,6 | 3,7 of the word
__device__ __forceinline__ void nib_word(uint32_t w, const NibScale& s, uint32_t* o) {
    const uint32_t x = w >> 8;
    o[0] = hfma2_u32(w & 0x000F000Fu, s.g8, s.c);
    o[1] = hfma2_u32(w & 0x00F000F0u, s.g4, s.c);
    o[2] = hfma2_u32(x & 0x000F000Fu, s.g8, s.c);
    o[3] = hfma2_u32(x & 0x00F000F0u, s.g4, s.c);
}
// eight 3-bit codes (the low 24 bits) and their correction bits (the low 8) -> a word of nibbles 2 code + bit.  Every step moves the upper half of each field and takes
// the rest as it is, one LOP3 a step (x where the mask is set, else y); what that leaves between the fields never reaches a place that the last step keeps.
__device__ __forceinline__ uint32_t bit_select(uint32_t x, uint32_t y, uint32_t mask) {
    uint32_t d;
    asm("lop3.b32 %0, %1, %2, %3, 0xE2;\n" : "=r"(d) : "r"(x), "r"(mask), "r"(y));
    return d;
}
__device__ __forceinline__ uint32_t code3_nibbles(uint32_t x, uint32_t c) {
    x = bit_select(x, x << 4, 0x00000FFFu);
    x = bit_select(x, x << 2, 0x003F003Fu);
    x = bit_select(x, x << 1, 0x07070707u);
    c = bit_select(c, c << 12, 0x0000000Fu);
    c = bit_select(c, c << 6, 0x00030003u);
    c = bit_select(c, c << 3, 0x01010101u);
    return bit_select(x << 1, c, 0xEEEEEEEEu);
}
// four head bytes b -> (b - 128) gh 2^(U + 4) (two columns) and (b - 128) gl 2^U (two columns), gh / gl the nibbles of the
// head's scale byte, U = -16 (mixed) or -15 (MIX3, whose other levels are kept halved): products below 2048, exact in fp16
template <bool HALVED>
__device__ __forceinline__ void head_word(uint32_t w, uint32_t gs0, uint32_t magic, uint32_t* o) {
    uint32_t gh, gl, b01, b23;
    asm("add.rn.f16x2 %0, %1, %2;\n" : "=r"(gh) : "r"(0x64006400u | (gs0 >> 4) * 0x10001u), "r"(0xE400E400u));
    asm("add.rn.f16x2 %0, %1, %2;\n" : "=r"(gl) : "r"(0x64006400u | (gs0 & 15u) * 0x10001u), "r"(0xE400E400u));
    asm("mul.rn.f16x2 %0, %1, %2;\n" : "=r"(gh) : "r"(gh), "r"(HALVED ? 0x10001000u : 0x0C000C00u));  // x 2^-11 / 2^-12
    asm("mul.rn.f16x2 %0, %1, %2;\n" : "=r"(gl) : "r"(gl), "r"(HALVED ? 0x02000200u : 0x01000100u));  // x 2^-15 / 2^-16 (subnormal constants)
    asm("add.rn.f16x2 %0, %1, %2;\n" : "=r"(b01) : "r"(prmt(w, magic, 0x7150u)), "r"(0xE480E480u));  // bytes 0, 1 minus 128
    asm("add.rn.f16x2 %0, %1, %2;\n" : "=r"(b23) : "r"(prmt(w, magic, 0x7352u)), "r"(0xE480E480u));
    asm("mul.rn.f16x2 %0, %1, %2;\n" : "=r"(o[0]) : "r"(b01), "r"(gh));
    asm("mul.rn.f16x2 %0, %1, %2;\n" : "=r"(o[1]) : "r"(b23), "r"(gh));
    asm("mul.rn.f16x2 %0, %1, %2;\n" : "=r"(o[2]) : "r"(b01), "r"(gl));
    asm("mul.rn.f16x2 %0, %1, %2;\n" : "=r"(o[3]) : "r"(b23), "r"(gl));
}
// scale bytes (b0, b1) of a word -> half2 times f (a power of two)
__device__ __forceinline__ uint32_t scale_pair(uint32_t w, uint32_t magic, uint32_t sel, uint32_t f) {
    uint32_t t;
    asm("add.rn.f16x2 %0, %1, %2;\n" : "=r"(t) : "r"(prmt(w, magic, sel)), "r"(0xE400E400u));
    asm("mul.rn.f16x2 %0, %1, %2;\n" : "=r"(t) : "r"(t), "r"(f));
    return t;
}

// Quarters Q0 .. Q1 - 1 of a tile's row of the A operand (16 columns each) for the kinds whose scale bytes are folded into it;
// the last quarter brings the extra columns of the 3-bit kinds.
template <int KIND, int Q0, int Q1>
__device__ __forceinline__ void st_fold_row(uint32_t row, uint32_t ta, uint32_t flags, uint32_t gsl, uint32_t gsh, uint32_t magic) {
    const bool nocorr = (flags & F_NOCORR) != 0;  // (the correction plane's bytes are ignored once flagged as dropped)
    const uint32_t gs0 = gsl & 0xFFu;
    uint32_t words[16];  // the latent's sixteen words (only those the quarters need are loaded)
#pragma unroll
    for (int i = 0; i < 16; ++i) words[i] = 0u;
    if (KIND == 2 || KIND == 4) {
        // TQ3: codes in bytes 0..47, correction plane in 48..63.  MIX3: head 0..7, codes 8..49, correction plane 50..63.
        const uint4 a = lds_v4<0>(row), b = lds_v4<16>(row), c = lds_v4<32>(row), d = lds_v4<48>(row);
        words[0] = a.x; words[1] = a.y; words[2] = a.z; words[3] = a.w; words[4] = b.x; words[5] = b.y; words[6] = b.z; words[7] = b.w;
        words[8] = c.x; words[9] = c.y; words[10] = c.z; words[11] = c.w; words[12] = d.x; words[13] = d.y; words[14] = d.z; words[15] = d.w;
    }
#pragma unroll
    for (int Q = Q0; Q < Q1; ++Q) {
        uint32_t w[4];
        if (KIND == 2) {
            const uint32_t cr = nocorr ? 0u : words[12 + Q];
#pragma unroll
            for (int m = 0; m < 4; ++m) {
                const int bit = 96 * Q + 24 * m, wi = bit >> 5, sh = bit & 31;
                w[m] = code3_nibbles(__funnelshift_r(words[wi], words[wi + 1], sh), cr >> (8 * m));
            }
        } else if (KIND == 4) {
            if (Q == 0) {
                w[0] = words[0];
                w[1] = words[1];
            }
#pragma unroll
            for (int m = Q == 0 ? 2 : 0; m < 4; ++m) {
                const int j = 4 * Q + m - 2;  // code word j: dims 8 + 8 j .., codes at bit 64 + 24 j, correction bits at bit 400 + 8 j
                const int bit = 64 + 24 * j, wi = bit >> 5, sh = bit & 31, cb = 400 + 8 * j;
                const uint32_t cr = nocorr ? 0u : words[cb >> 5] >> (cb & 31);
                w[m] = code3_nibbles(__funnelshift_r(words[wi], words[wi + 1 < 16 ? wi + 1 : 15], sh), cr);
            }
        } else {
            const uint4 L = Q == 0 ? lds_v4<0>(row) : (Q == 1 ? lds_v4<16>(row) : (Q == 2 ? lds_v4<32>(row) : lds_v4<48>(row)));
            w[0] = L.x; w[1] = L.y; w[2] = L.z; w[3] = L.w;
        }
        // words 4 Q, 4 Q + 1 share scale byte 2 Q, words 4 Q + 2, 4 Q + 3 scale byte 2 Q + 1 (the mixed layouts' two head words take the
        // place of group 0, whose byte is the head's)
        const uint32_t gw = Q < 2 ? gsl : gsh;
        const NibScale s0 = nib_scale((Q & 1) ? byte_half2<2>(gw, magic) : byte_half2<0>(gw, magic));
        const NibScale s1 = nib_scale((Q & 1) ? byte_half2<3>(gw, magic) : byte_half2<1>(gw, magic));
        uint32_t o[16];
        if ((KIND == 1 || KIND == 4) && Q == 0) {
            head_word<KIND == 4>(w[0], gs0, magic, o);
            head_word<KIND == 4>(w[1], gs0, magic, o + 4);
        } else {
            nib_word(w[0], s0, o);
            nib_word(w[1], s0, o + 4);
        }
        nib_word(w[2], s1, o + 8);
        nib_word(w[3], s1, o + 12);
        st_tmem_st16(ta + 16u * Q, o);
    }
    if (Q1 == 4 && (KIND == 2 || KIND == 4)) {
        // level = (n - 8) / 2 + c / 4 with the nibble n (c = 1, or 2 without the correction plane): eight more K slots carry the
        // scale bytes times c 2^-13, against a sixteenth of the queries' sums over the groups (MIX3: the head's slot meets a zero)
        const uint32_t f = nocorr ? 0x0C000C00u : 0x08000800u;
        uint32_t o[8] = {scale_pair(gsl, magic, 0x7150u, f), scale_pair(gsl, magic, 0x7352u, f), scale_pair(gsh, magic, 0x7150u, f),
                         scale_pair(gsh, magic, 0x7352u, f), 0u, 0u, 0u, 0u};
        st_tmem_st8(ta + 64u, o);
    }
}

// NF4: half H of the latent (four scale groups) as fp16 hi (columns 0..31) and lo (32..63) parts of 1024 times the codebook entries
// (unscaled, the lo parts of the small entries would be subnormal), from the shared-memory table; the scale bytes are applied to the groups' sums instead, because a codebook value times a scale
// byte does not fit fp16.
__device__ __forceinline__ void st_nf4_half(uint32_t row, int h, uint32_t ta, uint32_t flags, uint32_t lut_s, uint32_t lane8, uint32_t magic) {
#pragma unroll
    for (int Q = 0; Q < 2; ++Q) {
        const uint4 L = lds_v4<0>(row + 32u * h + 16u * Q);
        const uint32_t w[4] = {L.x, L.y, L.z, L.w};
        uint32_t hi[16], lo[16];
        if (flags & F_NF4) {
#pragma unroll
            for (int m = 0; m < 4; ++m) {
                const uint2 e0 = lds_v2<0>(lut_s + (((w[m] << 7) & 0x7F80u) | lane8)), e1 = lds_v2<0>(lut_s + (((w[m] >> 1) & 0x7F80u) | lane8));
                const uint2 e2 = lds_v2<0>(lut_s + (((w[m] >> 9) & 0x7F80u) | lane8)), e3 = lds_v2<0>(lut_s + (((w[m] >> 17) & 0x7F80u) | lane8));
                hi[4 * m] = e0.x; hi[4 * m + 1] = e1.x; hi[4 * m + 2] = e2.x; hi[4 * m + 3] = e3.x;
                lo[4 * m] = e0.y; lo[4 * m + 1] = e1.y; lo[4 * m + 2] = e2.y; lo[4 * m + 3] = e3.y;
            }
        } else {  // an INT4 tile in an NF4 launch: levels n - 8
#pragma unroll
            for (int e = 0; e < 16; ++e) {
                const uint32_t b = (w[e >> 2] >> (8 * (e & 3))) & 0xFFu;
                asm("add.rn.f16x2 %0, %1, %2;\n" : "=r"(hi[e]) : "r"(((b | (b << 12)) & 0x000F000Fu) | magic), "r"(0xE408E408u));
                asm("mul.rn.f16x2 %0, %1, %2;\n" : "=r"(hi[e]) : "r"(hi[e]), "r"(0x64006400u));
                lo[e] = 0u;
            }
        }
        __syncwarp();
        st_tmem_st16(ta + 16u * Q, hi);
        st_tmem_st16(ta + 32u + 16u * Q, lo);
    }
}

// s + x into s, what the rounding lost added to e
__device__ __forceinline__ void two_sum(float& s, float x, float& e) {
    const float t = __fadd_rn(s, x), b = __fsub_rn(t, s);
    e = __fadd_rn(e, __fadd_rn(__fsub_rn(s, __fsub_rn(t, b)), __fsub_rn(x, b)));
    s = t;
}
// the same for pairs (a subtraction is a fused step with -1: exact but for the one rounding)
__device__ __forceinline__ void two_sum2(uint64_t& s, uint64_t x, uint64_t& e) {
    constexpr uint64_t M1 = 0xBF800000BF800000ull;
    const uint64_t t = f2_add(s, x), b = f2_fma(s, M1, t);
    e = f2_add(e, f2_add(f2_fma(f2_fma(b, M1, t), M1, s), f2_fma(b, M1, x)));
    s = t;
}
__device__ __forceinline__ uint64_t f2_mul(uint64_t a, uint64_t b) {
    uint64_t r;
    asm("mul.rn.f32x2 %0, %1, %2;\n" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ uint64_t u2_pack(uint32_t lo, uint32_t hi) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};\n" : "=l"(r) : "r"(lo), "r"(hi));
    return r;
}
// Set bits of eight words: four full adders leave four words for POPC, which runs at a quarter of the logic's rate.
__device__ __forceinline__ uint32_t popc8_words(const uint32_t (&x)[8]) {
    const uint32_t s1 = x[0] ^ x[1] ^ x[2], c1 = (x[0] & x[1]) | (x[2] & (x[0] | x[1]));
    const uint32_t s2 = x[3] ^ x[4] ^ x[5], c2 = (x[3] & x[4]) | (x[5] & (x[3] | x[4]));
    const uint32_t s3 = x[6] ^ x[7] ^ s1, c3 = (x[6] & x[7]) | (s1 & (x[6] | x[7]));
    const uint32_t t = c1 ^ c2 ^ c3, u = (c1 & c2) | (c3 & (c1 | c2));
    return (uint32_t)__popc(s2) + (uint32_t)__popc(s3) + 2u * (uint32_t)__popc(t) + 4u * (uint32_t)__popc(u);
}

// a codec a launch of this kind does not decode
__device__ __forceinline__ bool st_alien(int kind, uint32_t flags) {
    if (kind == 0) return (flags & (F_MIXED | F_TQ3 | F_MIX3)) != 0;
    if (kind == 1) return !(flags & F_MIXED) || (flags & (F_TQ3 | F_MIX3 | F_NF4));
    if (kind == 2) return !(flags & F_TQ3) || (flags & (F_MIXED | F_MIX3 | F_NF4));
    if (kind == 3) return (flags & (F_MIXED | F_TQ3 | F_MIX3 | F_NF4)) != 0;
    return !(flags & F_MIX3) || (flags & (F_MIXED | F_TQ3 | F_NF4));
}

// What a thread keeps from one work item to the next.
struct TileCta {
    uint32_t base_s;   // shared memory, 1024-byte aligned: B | [NF4 table] | ring | sign words | thresholds (keys, floats) | mappings | barriers, flags | query scales | [bits of undone items]
    unsigned char* base;
    uint32_t tmem;
    int uw;            // warp index, known to be uniform
    bool leader;       // the thread that issues its warpgroup's MMAs
    bool table;        // the NF4 table is there
    uint32_t phase;    // of the warpgroup's mbarrier
    bool failed;       // a wait of this warp ran out
    bool undone;       // dense: an item was left, see undone_add
    PassWalk walk;     // PASS: where the item lies, of range
    const PassRange* range;
};
template <bool DENSE>
struct TileLayout {
    static constexpr uint32_t LUT = ST_B_BYTES, RING = LUT + (DENSE ? NF4_LUT_BYTES : 0), TAIL = RING + (ST_THREADS / 32) * ST_DEPTH * ST_SLOT, UNDONE = TAIL + ST_TAIL_BYTES;
};
__device__ __forceinline__ unsigned char* tile_base(unsigned char* smem_raw) {
    const uint32_t at = (uint32_t)__cvta_generic_to_shared(smem_raw);
    return smem_raw + (((at + 1023u) & ~1023u) - at);
}
template <bool DENSE>
__device__ __forceinline__ TileCta tile_open(unsigned char* smem_raw) {
    TileCta t;
    t.uw = uniform_warp();
    // (the four warpgroups' leaders sit on different schedulers)
    const bool elected = elect_one();
    t.leader = elected && (t.uw & 3) == (t.uw >> 2);
    t.base = tile_base(smem_raw);
    t.base_s = (uint32_t)__cvta_generic_to_shared(t.base);
    const uint32_t tail_s = t.base_s + TileLayout<DENSE>::TAIL;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(t.base + TileLayout<DENSE>::TAIL + 256u);
    if (threadIdx.x == 0) {
        for (int i = 0; i < ST_WG; ++i) mbar_init(tail_s + 224u + 8 * i, 1);
        tmem_slot[1] = 0u;  // bail
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    if (threadIdx.x < 32) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(tail_s + 256u), "r"(512u) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    t.tmem = *reinterpret_cast<volatile uint32_t*>(tmem_slot);
    t.table = false;
    t.phase = 0u;
    t.failed = t.undone = false;
    t.walk = PassWalk{};
    t.range = nullptr;
    return t;
}
__device__ __forceinline__ void tile_close(const TileCta& t) {
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    if (threadIdx.x < 32) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(t.tmem), "r"(512u) : "memory");
}
// The kind of a work item: what its first tile says.  nf4_too: plain nibble tiles count as NF4 (that kind decodes both).
__device__ __forceinline__ int item_kind(uint32_t tile_flags, bool nf4_too) {
    if (tile_flags & F_MIXED) return 1;
    if (tile_flags & F_TQ3) return 2;
    if (tile_flags & F_MIX3) return 4;
    return (tile_flags & F_NF4) || nf4_too ? 0 : 3;
}
__device__ __forceinline__ uint32_t first_tile_flags(const ScoreArgs& a, const WorkItem& it) {
    return *reinterpret_cast<const uint16_t*>(a.tiles + it.tile_begin * TILE_BYTES + 118);
}

// The work items from item_id on (KINDS: up to the first whose first tile is of another kind); the next item.  it, flags0: item_id's item and its first
// tile's flags, which the caller has read; the next item's when this returns.
// DENSE: every score is written to a.scores (row q at a.row_offset[q] or q * a.score_stride, tile i of the item at
// index_base + i; -inf for COLD slots) and nothing is filtered or appended.  IL: the work items are interleaved shares of
// whole streams (see the planner).  A tile of another codec than KIND's, or a query outside the fp16 split, hands the
// item's query rows to the generic kernel.
template <int KIND, bool IL, bool DENSE, bool KINDS, bool PASS = false>
__device__ __forceinline__ uint32_t tile_run(const ScoreArgs& a, TileCta& cta, uint32_t item_id, uint32_t item_end, WorkItem& it, uint32_t& flags0, bool nf4_too = false) {
    constexpr int NWG = ST_WG, NWARPS = 4 * NWG, NACC = st_accs(KIND);
    constexpr uint32_t STRIDE = ST_TMEM, DCOL = st_d_col(KIND);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, wg = warp >> 2, wq = warp & 3;
    const int uw = cta.uw;
    const bool leader = cta.leader;
    const uint32_t base_s = cta.base_s, tmem = cta.tmem;
    unsigned char* base = cta.base;
    constexpr uint32_t LUT_OFF = TileLayout<DENSE>::LUT, RING_OFF = TileLayout<DENSE>::RING, TAIL_OFF = TileLayout<DENSE>::TAIL;
    const uint32_t B_s = base_s, lut_s = base_s + LUT_OFF, ring_s = base_s + RING_OFF + (uint32_t)warp * (ST_DEPTH * ST_SLOT), tail_s = base_s + TAIL_OFF;
    unsigned char* tail = base + TAIL_OFF;
    uint32_t* qs_w = reinterpret_cast<uint32_t*>(tail);         // [4][8] sign words
    uint32_t* pvh = qs_w + 32;                                   // [4] score word of the row's threshold
    float* thr = reinterpret_cast<float*>(pvh + 4);              // [4] the same as a float (-inf: none)
    float2* rng = reinterpret_cast<float2*>(thr + 4);            // [4] (smin, inv), inv 0 = none yet
    float2* rmap = rng + 4;                                      // [4] (-smin inv, inv)
    uint32_t* flagw = reinterpret_cast<uint32_t*>(rmap + 4);     // mbarriers of the warpgroups (32 bytes), TMEM base, bail
    const uint32_t bar_s = tail_s + 224u, qsw_s = tail_s;
    uint32_t* bail = flagw + 9;
    uint32_t* qmax = flagw + 16;                                 // [4] bits of the row's largest element
    float* qinv = reinterpret_cast<float*>(qmax + 4);            // [4] inverse of the row's scale times the unit of A
    float* qsum = qinv + 4;                                      // [4][16] sums of eight elements (3-bit kinds)

    if (KIND == 0 && !cta.table) {  // NF4 codebook pairs per byte, 16 bank-aligned replicas (read by nobody yet)
        cta.table = true;
        uint2* lut = reinterpret_cast<uint2*>(base + LUT_OFF);
        for (int e = tid; e < 256 * 16; e += blockDim.x) {
            const int b = e >> 4;
            const float c0 = 1024.0f * c_nf4[b & 15], c1 = 1024.0f * c_nf4[b >> 4];
            lut[e] = make_uint2(pack_half2(c0, c1), pack_half2(half_residual(c0), half_residual(c1)));
        }
    }
    const uint32_t ta = tmem + (uint32_t)wg * STRIDE + ((uint32_t)(32 * wq) << 16);  // this warp's lanes of its warpgroup's columns
    uint32_t magic;  // 1024.0h twice, opaque so that it stays in one register
    asm volatile("mov.u32 %0, 0x64006400;\n" : "=r"(magic));
    const uint32_t lane8 = (uint32_t)(lane & 15) * 8u;
    const uint32_t dst_lane = ring_s + (uint32_t)((lane >> 3) * ST_ROW + (lane & 7) * 16), row_lane = ring_s + (uint32_t)lane * ST_ROW;
    const uint32_t lt_mask = (1u << lane) - 1u;
    uint64_t stream_policy;
    asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;\n" : "=l"(stream_policy));
    uint32_t phase = cta.phase;
    bool failed = cta.failed;

    auto next_item = [&]() {  // false at the end, or at an item of another kind (the same in the whole CTA)
        if (PASS) {
            if (!pass_next(a, *cta.range, cta.walk)) {
                item_id = item_end;
                return false;
            }
            ++item_id;
            it = pass_item(a, *cta.range, cta.walk);
        } else {
            if (++item_id >= item_end) return false;
            it = a.stream_items[item_id];
        }
        if (KINDS) flags0 = first_tile_flags(a, it);
        return !KINDS || item_kind(flags0, nf4_too) == KIND;
    };
    do {
        bool gave_up = false;  // this warpgroup met a tile it cannot decode, or a wait of it ran out (the same in the whole warpgroup)
        const int nq = (int)it.n_queries;
        // interleaved: this CTA is number il_c of the il_n CTAs that share the stream [tile_begin, + n_tiles); round r of
        // the stream's static deal belongs to CTA r mod il_n.  Otherwise the item is this CTA's own range.
        const uint32_t il_n = IL ? ((it.pad >> 8) & 0x7FFFFFu) : 1u, il_c = IL ? it.list_begin : 0u;
        const uint8_t* sbase = a.state ? a.state + it.tile_begin : nullptr;
        const uint32_t n = it.n_tiles;
        const uint32_t n_blocks = (n + ST_M - 1) / ST_M;
        // Blocks are dealt to the warpgroups round by round.  An interleaved CTA walks its rounds starting from a place of its
        // own and wraps around (CTA c of C starts c / C of the way through), so that at any moment the CTAs of a stream are
        // spread over the whole stream -- the first thresholds then come from a sample of all positions even when one
        // end of the stream holds nothing to score (the oldest slots of a pool are mostly COLD).
        const uint32_t all_rounds = (n_blocks + NWG - 1) / NWG;
        const uint32_t my_rounds = all_rounds > il_c ? (all_rounds - il_c + il_n - 1) / il_n : 0u;  // (the same for all warps of the CTA)
        const uint32_t first_round = IL ? (uint32_t)(((uint64_t)il_c * my_rounds) / il_n) : 0u;
        auto block_of = [&](uint32_t i) {  // the block this warpgroup takes in its i-th iteration
            if (!IL) return i * (uint32_t)NWG + (uint32_t)wg;
            uint32_t j = i + first_round;
            if (j >= my_rounds) j -= my_rounds;
            return (j * il_n + il_c) * (uint32_t)NWG + (uint32_t)wg;
        };
        auto leave = [&]() {
            const uint32_t bit = undone_bit(PASS ? item_id : item_id - dense_first(a));
            reinterpret_cast<uint32_t*>(base + TileLayout<true>::UNDONE)[bit >> 5] |= 1u << (bit & 31u);
        };
        if (PASS) {  // (a group one of whose rows the 64-row kernel handed on)
            uint32_t f = 0;
            for (int q = 0; q < nq; ++q) f |= a.only_flagged[it.query_begin + q];
            if (f & 2u) {  // (the same in the whole CTA)
                if (a.gflag && tid < nq) a.gflag[it.query_begin + tid] = 1u;
                if (tid == 0) leave();
                cta.undone = true;
                continue;
            }
        }
        const unsigned char* tbase = a.tiles + it.tile_begin * TILE_BYTES + (size_t)wq * (ST_WT * TILE_BYTES) + lane * 16;
        uint32_t iss_no = 0, slot_next = 0;
        auto issue = [&]() {  // lane copies chunk (lane & 7) of rows (lane >> 3) + 0, 4, .. 28 of the warp's 32 tiles
            const uint32_t b = iss_no < my_rounds ? block_of(iss_no) : 0xFFFFFFFFu;
            ++iss_no;
            if (b < n_blocks) {
                const uint32_t dst = dst_lane + slot_next, t0 = b * ST_M + (uint32_t)wq * ST_WT;
                const unsigned char* src = tbase + (size_t)b * (ST_M * TILE_BYTES);
                if (t0 + ST_WT <= n) {
                    cp_async16_sp<0, 0>(dst, src, 16, stream_policy);
                    cp_async16_sp<512, 4 * ST_ROW>(dst, src, 16, stream_policy);
                    cp_async16_sp<1024, 8 * ST_ROW>(dst, src, 16, stream_policy);
                    cp_async16_sp<1536, 12 * ST_ROW>(dst, src, 16, stream_policy);
                    cp_async16_sp<2048, 16 * ST_ROW>(dst, src, 16, stream_policy);
                    cp_async16_sp<2560, 20 * ST_ROW>(dst, src, 16, stream_policy);
                    cp_async16_sp<3072, 24 * ST_ROW>(dst, src, 16, stream_policy);
                    cp_async16_sp<3584, 28 * ST_ROW>(dst, src, 16, stream_policy);
                } else {  // rows past the end are zero-filled (source not read)
                    const uint32_t r = t0 + (uint32_t)(lane >> 3);
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        const bool in = r + 4u * i < n;
                        cp_async16_s<0, 0>(dst + 4u * i * ST_ROW, in ? src + 512 * i : a.tiles, in ? 16 : 0);
                    }
                }
            }
            cp_async_commit();
            slot_next = slot_next == (ST_DEPTH - 1) * ST_SLOT ? 0u : slot_next + ST_SLOT;
        };
        // B: 16-byte chunks of eight k slots, K-major, 128-byte swizzle (chunk i of row r at chunk i ^ (r & 7) of its line), one a thread.
        // Row n = 4 part + q (hi / lo of query q), rows 8..15 zero; k slot 8 i + j holds dim 8 i + {0,4,1,5,2,6,3,7}[j] (see
        // nib_word), NF4: dim 8 i + j.  A row's scale comes from the elements its chunks hold (the mixed layouts drop the last eight).  What the item
        // brings from memory is asked for before the first barrier, and before the tiles: behind 64 KB of them it took 1100 to 2500 cycles.
        static_assert(ST_THREADS >= 16 * 18, "a thread per chunk");
        constexpr bool HEAD = KIND == 1 || KIND == 4, EXTRA = KIND == 2 || KIND == 4;
        const int br = tid / 18, bi = tid % 18, bq = br & 3;
        // (one load for all kinds of chunk and no arithmetic on what comes: a branch would wait for its own loads)
        const bool chunk_of_row = tid < 8 * 18 && bq < nq && bi < 16, head = HEAD && bi < 2;
        float4 qx = make_float4(0.0f, 0.0f, 0.0f, 0.0f), qy = qx;
        {
            const float* q = a.q_coarse + (size_t)(it.query_begin + bq) * D_C + (head ? 4 * bi : 8 * (HEAD ? bi - 1 : bi));
            const int up = head ? 0 : 4;
            if (reinterpret_cast<uintptr_t>(a.q_coarse) & 15u) {  // (the same for all rows)
                if (chunk_of_row) {
                    qx = make_float4(q[0], q[1], q[2], q[3]);
                    qy = make_float4(q[up], q[up + 1], q[up + 2], q[up + 3]);
                }
            } else if (chunk_of_row) {
                qx = *reinterpret_cast<const float4*>(q);
                qy = *reinterpret_cast<const float4*>(q + up);
            }
        }
        uint32_t sign_word = 0u;
        if (warp == 8 && (lane >> 3) < nq) sign_word = a.q_sign[(size_t)(it.query_begin + (lane >> 3)) * 8 + (lane & 7)];
        bool row_warm = true;
        unsigned long long pv = 0ull, pr = 0ull;
        if (!DENSE && tid < nq) {
            pv = *reinterpret_cast<volatile unsigned long long*>(a.gpivot + it.query_begin + tid);
            pr = *reinterpret_cast<volatile unsigned long long*>(a.grange + it.query_begin + tid);
        }
        float* rowp[4];  // dense: where the item's rows start
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const uint32_t Q = it.query_begin + (uint32_t)min(q, nq - 1);
            rowp[q] = !DENSE ? nullptr : a.blocked ? a.scores + it.list_begin + 128u * (uint32_t)q + (size_t)(it.index_base >> 7) * it.pad
                                                   : a.scores + (a.row_offset ? (size_t)a.row_offset[Q] : (size_t)Q * a.score_stride) + it.index_base;
        }
        const uint32_t row_step = DENSE && a.blocked ? it.pad : (uint32_t)ST_M;  // from a block's scores of a row to the next block's
#pragma unroll
        for (int i = 0; i < ST_DEPTH - 1; ++i) issue();
        if (warp == 9 && lane < 4) qmax[lane] = 0u;  // (read last in the set-up of the item before)
        __syncthreads();  // previous item fully retired (and the table is visible)
        if (!DENSE && tid < 4) {
            // start from the threshold other CTAs have already proven for the row, and from the
            // row's bucket mapping if one has been published
            pvh[tid] = (uint32_t)(pv >> 32);
            thr[tid] = thr_float((uint32_t)(pv >> 32));
            row_warm = tid >= nq || (uint32_t)(pv >> 32) != 0u;
            rng[tid] = make_float2(__uint_as_float((uint32_t)pr), __uint_as_float((uint32_t)(pr >> 32)));
            rmap[tid] = make_float2(-rng[tid].x * rng[tid].y, rng[tid].y);
        }
        if (warp == 8) qs_w[lane] = sign_word;  // sign words of the item's (up to four) queries
        float v[8];
        if (KIND == 0 || head) {  // (head: slots 0..3 the scale byte's high nibble's products of dims 4 bi .., 4..7 the low nibble's)
            v[0] = qx.x; v[1] = qx.y; v[2] = qx.z; v[3] = qx.w; v[4] = qy.x; v[5] = qy.y; v[6] = qy.z; v[7] = qy.w;
        } else {
            v[0] = qx.x; v[1] = qy.x; v[2] = qx.y; v[3] = qy.y; v[4] = qx.z; v[5] = qy.z; v[6] = qx.w; v[7] = qy.w;
        }
        if (tid < 4 * 18 && bi < 16) {
            uint32_t largest = 0u;
#pragma unroll
            for (int j = 0; j < 8; ++j) largest = max(largest, abs_bits(v[j]));
            atomicMax(&qmax[bq], largest);
        }
        if (EXTRA && tid < 4 * 18 && bi < 16) qsum[16 * bq + bi] = ((v[0] + v[1]) + (v[2] + v[3])) + ((v[4] + v[5]) + (v[6] + v[7]));  // of a group's half
        __syncthreads();
        if (EXTRA && tid < 8 * 18 && bi == 16) {
#pragma unroll
            for (int g = KIND == 4 ? 1 : 0; g < 8; ++g) v[g] = 0.0625f * (qsum[16 * bq + 2 * g] + qsum[16 * bq + 2 * g + 1]);
        }
        if (tid < 16 * 18) {
            const float up = split_scale(qmax[bq], 14).x;  // (rows 8 .. 15 are zero)
            uint32_t w[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                float x0 = v[2 * j] * up, x1 = v[2 * j + 1] * up;
                if (br >= 4) { x0 = half_residual(x0); x1 = half_residual(x1); }
                w[j] = pack_half2(x0, x1);
            }
            const uint32_t slab = (uint32_t)bi >> 3, chunk = (uint32_t)bi & 7u;
            sts_v4(B_s + slab * 2048u + (uint32_t)br * 128u + ((chunk ^ ((uint32_t)br & 7u)) << 4), w[0], w[1], w[2], w[3]);
        }
        bool big = false;  // a query beyond the fp16 split
        if (tid < 4) {
            big = qmax[tid] >= SPLIT_MOST;
            qinv[tid] = split_scale(qmax[tid], 14).y * (KIND == 0 ? 1.0f / 1024.0f : (KIND == 2 || KIND == 4 ? 32768.0f : 65536.0f));
        }
        if (big) *bail = 1u;
        asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");  // B was written with ordinary stores, the MMA reads it through the async proxy
        // The barrier after the first round (below) pays when the round can supply k candidates to a row -- 32 per warp
        // of every CTA that works on the row -- and the rows do not already have thresholds (a CTA that starts its
        // second item on rows other CTAs have been scoring for a while).
        // (from a barrier's vote, not from the flag word: a fast warp may raise the flag for an undecodable tile meanwhile)
        const bool too_big = __syncthreads_or(big) != 0;
        const bool all_warm = !DENSE && __syncthreads_and(row_warm) != 0;
        const bool first_round_barrier = !DENSE && !all_warm && (uint64_t)a.k <= (uint64_t)(ST_WT * NWARPS) * (uint64_t)max((it.pad >> 8) & 0x7FFFFFu, 1u);
        const uint32_t rounds = too_big ? 0u : my_rounds;  // (copies already on their way are waited for at the item's end and never read)

        auto state_of = [&](uint32_t i) {
            const uint32_t t = i < my_rounds ? block_of(i) * (uint32_t)ST_M + (uint32_t)(wq * ST_WT + lane) : 0xFFFFFFFFu;
            return t < n ? sbase[t] : ST_HOT;
        };
        uint8_t st_next = sbase ? state_of(0) : ST_HOT;
        uint32_t slot = 0, polls = 0;
        uint32_t cur[4] = {0, 0, 0, 0}, end[4] = {0, 0, 0, 0};  // this warp's chunk of every row's buffer
        bool dead = false;                                      // this warp met a tile it cannot decode, or a wait of it ran out
        for (uint32_t round = 0; round < rounds; ++round) {
            if (round == 1 && first_round_barrier) {
                // Every warp of the CTA (and, started together, of the grid) has appended its first tiles
                // unfiltered, so the rows' histograms hold 32 candidates per warp: first thresholds now,
                // before the second blocks are filtered.  (All warps pass here: `rounds` is the same for all.)
                __syncthreads();
                if (warp < nq) {
                    stream_refresh_threshold(a, it.query_begin + (uint32_t)warp, rng[warp], pvh + warp, lane);
                    __syncwarp();
                    if (lane == 0) thr[warp] = thr_float(pvh[warp]);
                }
                __syncthreads();
            }
            if (gave_up) continue;
            const uint32_t b = block_of(round);
            // (the ring advances in every iteration, also when this warpgroup has no block in this round -- the short last round
            // of the stream can come anywhere in a rotated walk -- so that fetches and reads stay in step)
            // issue() refills the slot that was read last, every lane its chunks of other lanes' rows: all lanes have read theirs
            // (they part company over COLD slots, rows past the end and residual words that only some need)
            __syncwarp();
            issue();
            cp_async_wait<ST_DEPTH - 1>();
            __syncwarp();
            const uint32_t row = row_lane + slot;
            slot = slot == (ST_DEPTH - 1) * ST_SLOT ? 0u : slot + ST_SLOT;
            if (b >= n_blocks) {  // (the same in the whole warpgroup)
                if (sbase) st_next = state_of(round + 1);
                continue;
            }
            const uint32_t t0 = b * ST_M + (uint32_t)(wq * ST_WT + lane);
            bool live = t0 < n;
            if (sbase) {  // (the slot's state came with the block before)
                live = live && st_next != ST_COLD;
                st_next = state_of(round + 1);
            }
            const uint2 meta = lds_v2<96>(row);   // scale, lambda
            const uint4 x = lds_v4<112>(row);     // position, head | flags, scale bytes
            const uint32_t flags = x.y >> 16;
            const bool alien = st_alien(KIND, flags);  // (rows past the end are zero-filled and not live)
            if (__any_sync(0xFFFFFFFFu, alien && t0 < n)) {
                if (lane == 0) *bail = 1u;
                dead = true;
            }
            uint64_t cs[2] = {0ull, 0ull}, low[2] = {0ull, 0ull};  // rows 0, 1 and 2, 3
            bool skip = false;
#pragma unroll
            for (int h = 0; h < (KIND == 0 ? 2 : 1); ++h) {  // (NF4: the latent in two halves, whose hi and lo parts fill the same columns)
                if (KIND == 0) st_nf4_half(row, h, ta, flags, lut_s, lane8, magic);
                else st_fold_row<KIND, 0, 4>(row, ta, flags, x.z, x.w, magic);
                asm volatile("tcgen05.wait::st.sync.aligned;\n" ::: "memory");
                asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
                if (role_any(1 + wg, 128, failed || dead)) { skip = true; break; }
                if (leader) {
                        asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
                        const uint32_t at = tmem + (uint32_t)(uw >> 2) * STRIDE, dt = at + DCOL;
                        if (KIND == 0) {
#pragma unroll
                            for (int u = 0; u < 8; ++u) {  // hi parts of the half's four groups, then the lo parts onto them
                                const int g = 4 * h + (u & 3);
                                st_mma(dt + 16u * (u & 3), at + 32u * (u >> 2) + 8u * (u & 3), tc_desc(B_s + 2048u * (g >> 2) + 32u * (g & 3)), u >> 2);
                            }
                        } else {
#pragma unroll
                            for (int ks = 0; ks < (KIND == 2 || KIND == 4 ? 9 : 8); ++ks)
                                st_mma(dt + 16u * (ks % NACC), at + 8u * ks, tc_desc(B_s + 2048u * (ks >> 2) + 32u * (ks & 3)), ks >= NACC ? 1u : 0u);
                        }
                        tc_commit(bar_s + 8 * (uw >> 2));
                }
                __syncwarp();
                failed = !mbar_wait(bar_s + 8 * wg, phase);
                phase ^= 1u;
                if (__any_sync(0xFFFFFFFFu, failed)) {
                    // the wait ran out: the warpgroup stops together at its next barrier, in this item and in all that follow
                    failed = true;
                    if (lane == 0) *bail = 1u;
                    dead = true;
                }
                asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
                uint32_t v[NACC][8];
                st_ld_accs(ta + DCOL, v);
                asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
                // The accumulators' sums with their rounding errors kept (two_sum), so that a score is rounded once here: the
                // generic kernel adds fp32 products in sixteen short chains, and this kernel's error is not to be larger.
#pragma unroll
                for (int p = 0; p < 2; ++p) {
                    if (p && nq <= 2) break;  // (uniform)
                    if (KIND == 0) {
#pragma unroll
                        for (int i = 0; i < NACC; ++i) {
                            // the group's scale byte (byte -> float: 2^23 + b as a bit pattern, minus 2^23), and its products' rounding errors
                            const float gs = __uint_as_float(__byte_perm(h ? x.w : x.z, 0x4B000000u, 0x7440 + i)) - 8388608.0f;
                            const uint64_t hi = u2_pack(v[i][2 * p], v[i][2 * p + 1]), lo = u2_pack(v[i][4 + 2 * p], v[i][4 + 2 * p + 1]);
                            const uint64_t g2 = f2_pack(gs, gs), n2 = f2_pack(-gs, -gs), prod = f2_mul(hi, g2);
                            low[p] = f2_fma(f2_fma(lo, n2, f2_fma(hi, n2, prod)), 0xBF800000BF800000ull, low[p]);
                            if (h == 0 && i == 0) cs[p] = prod;
                            else two_sum2(cs[p], prod, low[p]);
                        }
                    } else {
                        cs[p] = u2_pack(v[0][2 * p], v[0][2 * p + 1]);
                        low[p] = u2_pack(v[0][4 + 2 * p], v[0][4 + 2 * p + 1]);
#pragma unroll
                        for (int i = 1; i < NACC; ++i) {
                            low[p] = f2_add(low[p], u2_pack(v[i][4 + 2 * p], v[i][4 + 2 * p + 1]));
                            two_sum2(cs[p], u2_pack(v[i][2 * p], v[i][2 * p + 1]), low[p]);
                        }
                    }
                }
            }
            if (skip) {  // the item's rows go to the generic kernel: this warpgroup has no more to do for it
                if (lane == 0) *bail = 1u;
                gave_up = true;
                continue;
            }
            // (the row's power of two is exact; the tile's scale comes in the last step, so that the coarse term is rounded once there)
            const float su = __uint_as_float(meta.x) * (1.0f / 255.0f);
            float c[4];
            {
                const ulonglong2 inv = *reinterpret_cast<const ulonglong2*>(qinv);
                cs[0] = f2_mul(f2_add(cs[0], low[0]), inv.x);
                cs[1] = f2_mul(f2_add(cs[1], low[1]), inv.y);
                asm("mov.b64 {%0, %1}, %2;\n" : "=f"(c[0]), "=f"(c[1]) : "l"(cs[0]));
                asm("mov.b64 {%0, %1}, %2;\n" : "=f"(c[2]), "=f"(c[3]) : "l"(cs[1]));
            }
            if (dead) continue;
            const float lam = (flags & F_WARM) ? 0.0f : __uint_as_float(meta.y);
            if (DENSE) {
                const uint4 ra = lds_v4<64>(row), rb = lds_v4<80>(row);
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    if (q >= nq) break;  // (uniform)
                    const uint4 qa = lds_v4<0>(qsw_s + 32u * q), qb = lds_v4<16>(qsw_s + 32u * q);
                    const uint32_t d[8] = {ra.x ^ qa.x, ra.y ^ qa.y, ra.z ^ qa.z, ra.w ^ qa.w, rb.x ^ qb.x, rb.y ^ qb.y, rb.z ^ qb.z, rb.w ^ qb.w};
                    // 256 - 2 h without an integer conversion: (2^23 + h) as a bit pattern, times -2, plus 2^24 + 256 (exact)
                    const float sc = fmaf(c[q], su, lam * fmaf(__uint_as_float(0x4B000000u | popc8_words(d)), -2.0f, 16777472.0f));
                    // (the 32 lanes of a warp hold 32 consecutive tiles: one 128-byte run per row)
                    if (t0 < n) rowp[q][(size_t)b * row_step + (uint32_t)(wq * ST_WT + lane)] = live ? sc : __uint_as_float(a.cold_bits);
                }
                continue;
            }
            // The residual term lies in [-256 lambda, 256 lambda]: a tile that cannot reach a row's threshold even with the
            // largest term needs no Hamming distance (257 and the relative slack cover the rounding of the bound itself).
            uint32_t m = 0;
            if (round == 0) {
                m = live ? (1u << nq) - 1u : 0u;
            } else {
                float4 th;
                asm volatile("ld.volatile.shared.v4.f32 {%0,%1,%2,%3}, [%4];\n" : "=f"(th.x), "=f"(th.y), "=f"(th.z), "=f"(th.w) : "r"(tail_s + 144u));
                const float tq[4] = {th.x, th.y, th.z, th.w};
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const float x = c[q] * su;
                    if (q < nq && live && !(fmaf(fabsf(lam), 257.0f, fmaf(fabsf(x), 1e-6f, x)) < tq[q])) m |= 1u << q;  // (a NaN goes on to the exact test)
                }
            }
            if (__any_sync(0xFFFFFFFFu, m != 0u)) {
                const uint4 ra = lds_v4<64>(row), rb = lds_v4<80>(row);
#pragma unroll
                for (int q = 0; q < 4; ++q)
                    if (m >> q & 1u) {
                        const uint32_t* qw = qs_w + 8 * q;
                        const uint32_t d[8] = {ra.x ^ qw[0], ra.y ^ qw[1], ra.z ^ qw[2], ra.w ^ qw[3], rb.x ^ qw[4], rb.y ^ qw[5], rb.z ^ qw[6], rb.w ^ qw[7]};
                        c[q] = fmaf(c[q], su, lam * fmaf(__uint_as_float(0x4B000000u | popc8_words(d)), -2.0f, 16777472.0f));
                    }
                {
                    if (round == 0) {
                        // First tiles of the warp: a row without a bucket mapping gets one from the scores this warp has just
                        // computed for it - their range widened by 1.5 spans on both sides.  Any monotone mapping is
                        // valid; this one only has to put the final threshold somewhere inside its 256 buckets.  The first
                        // CTA to publish wins.
                        float mn[4], mx[4];
#pragma unroll
                        for (int q = 0; q < 4; ++q) {
                            mn[q] = live ? c[q] : INFINITY;
                            mx[q] = live ? c[q] : -INFINITY;
#pragma unroll
                            for (int o = 1; o < 32; o <<= 1) {
                                mn[q] = fminf(mn[q], __shfl_xor_sync(0xFFFFFFFFu, mn[q], o));
                                mx[q] = fmaxf(mx[q], __shfl_xor_sync(0xFFFFFFFFu, mx[q], o));
                            }
                        }
                        if (lane < nq && rng[lane].y == 0.0f) {
                            const float lo_s = lane == 0 ? mn[0] : (lane == 1 ? mn[1] : (lane == 2 ? mn[2] : mn[3]));
                            const float hi_s = lane == 0 ? mx[0] : (lane == 1 ? mx[1] : (lane == 2 ? mx[2] : mx[3]));
                            const uint32_t Q = it.query_begin + (uint32_t)lane;
                            unsigned long long pr = *reinterpret_cast<volatile unsigned long long*>(a.grange + Q);
                            if (!pr && hi_s > lo_s) {
                                const float span = hi_s - lo_s, lo = lo_s - 1.5f * span, inv = 256.0f / (4.0f * span);
                                if (isfinite(lo) && isfinite(inv) && inv > 0.0f) {
                                    const unsigned long long mine_r = (unsigned long long)__float_as_uint(lo) | ((unsigned long long)__float_as_uint(inv) << 32);
                                    const unsigned long long old = atomicCAS(a.grange + Q, 0ull, mine_r);
                                    pr = old ? old : mine_r;
                                }
                            }
                            if (pr) {
                                rng[lane] = make_float2(__uint_as_float((uint32_t)pr), __uint_as_float((uint32_t)(pr >> 32)));
                                rmap[lane] = make_float2(-rng[lane].x * rng[lane].y, rng[lane].y);
                            }
                        }
                        __syncwarp();
                    }
                    // Filter on the score word alone (a superset of the composite comparison: the merge drops keys below the
                    // final threshold) and append: the warp owns a chunk of 32 slots per row, [cur, end), reserved with one
                    // atomic, and a block brings at most 32 candidates per row, so a fresh chunk always fits them.  The
                    // unused rest of a chunk is zeroed (an absent key) before the next one is taken and at the item's end.
                    const uint32_t nidx = ~(it.index_base + t0);
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        if (q >= nq) break;  // (uniform)
                        const uint32_t key = score_key(c[q]);
                        const bool p = (m >> q & 1u) && key >= reinterpret_cast<const volatile uint32_t*>(pvh)[q];
                        const uint32_t bal = __ballot_sync(0xFFFFFFFFu, p);
                        if (!bal) continue;
                        const uint32_t nn = (uint32_t)__popc(bal), Q = it.query_begin + (uint32_t)q;
                        uint64_t* const dst = a.gbuf + (size_t)Q * a.gcap;
                        if (cur[q] + nn > end[q]) {
                            if (cur[q] + (uint32_t)lane < end[q]) dst[cur[q] + (uint32_t)lane] = 0ull;
                            uint32_t at = 0;
                            if (lane == 0) {
                                at = atomicAdd(a.gcount + Q, ST_CHUNK);
                                if (at + ST_CHUNK > a.gcap) {
                                    // the row's buffer is full: the generic kernel scores the row; this warp's further
                                    // candidates of the row land in the buffer's last chunk, which nobody reads then
                                    a.gflag[Q] = 1u;
                                    at = a.gcap - ST_CHUNK;
                                }
                            }
                            cur[q] = __shfl_sync(0xFFFFFFFFu, at, 0);
                            end[q] = cur[q] + ST_CHUNK;
                        }
                        if (p) {
                            dst[cur[q] + (uint32_t)__popc(bal & lt_mask)] = ((uint64_t)key << 32) | (uint64_t)nidx;
                            // bucket of the row's histogram: (int)(score * inv - smin * inv), clamped; scores below the
                            // mapping (and all scores while the row has no mapping) count in bucket 0, which never decides
                            const float2 r = rmap[q];
                            atomicAdd(a.ghist + (size_t)Q * 256 + min(max(__float2int_rz(fmaf(c[q], r.y, r.x)), 0), 255), 1u);
                        }
                        cur[q] += nn;
                    }
                }
            }
            // In turn, a warp raises the threshold of query (warp & 3): after its 2nd and 4th block (the first
            // thresholds come from the barrier after the first round), then every 8 blocks, the warps of a
            // query staggered.  A stale threshold costs appends (each one a store, a histogram count and,
            // downstream, merge work), a refresh costs one 1 KB read of the row's histogram by one warp.
            ++polls;
            if ((polls & 7u) == (uint32_t)wg * 2u + 1u || polls == 2u || polls == 4u) {
                if (wq < nq) {
                    stream_refresh_threshold(a, it.query_begin + (uint32_t)wq, rng[wq], pvh + wq, lane);
                    __syncwarp();
                    if (lane == 0) thr[wq] = thr_float(*reinterpret_cast<volatile uint32_t*>(pvh + wq));
                }
                __syncwarp();
            }
        }
        cp_async_wait<0>();
        if (!DENSE) {  // the unused rest of the warp's last chunks holds absent keys
#pragma unroll
            for (int q = 0; q < 4; ++q)
                if (cur[q] + (uint32_t)lane < end[q]) a.gbuf[(size_t)(it.query_begin + (uint32_t)q) * a.gcap + cur[q] + (uint32_t)lane] = 0ull;
        }
        __syncthreads();
        if (*reinterpret_cast<volatile uint32_t*>(bail)) {  // (the same in the whole CTA)
            // rows this CTA could not score on the tensor cores go to the generic kernel as a whole; of dense calls the item, at the CTA's end
            if (a.gflag && tid < nq) a.gflag[it.query_begin + tid] = 1u;
            if (DENSE) {
                if (tid == 0) leave();
                cta.undone = true;
            }
        }
        __syncthreads();
        if (tid == 0) *bail = 0u;  // (ordered before the next item's writers by the barrier at its start)
    } while (next_item());
    cta.phase = phase;
    cta.failed = failed;
    return item_id;
}

// Top-k of plans made for MIX3 tiles.  Plans are kept by shape: where a later call of that shape brings INT4 / MX-INT4 tiles, they
// are decoded as those (as the plans of MIX3 tiles did when the generic kernel scored MIX3).
template <bool IL>
__global__ void __launch_bounds__(ST_THREADS, 1) score_mix3_kernel(ScoreArgs a) {
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    dep_launch();
    dep_wait();
    uint32_t i = a.cta_begin[blockIdx.x];
    const uint32_t item_end = a.cta_begin[blockIdx.x + 1];
    WorkItem it = a.stream_items[i];
    uint32_t flags = first_tile_flags(a, it);
    TileCta cta = tile_open<false>(smem_raw);
    if (item_kind(flags, false) == 3) i = tile_run<3, IL, false, true>(a, cta, i, item_end, it, flags);
    if (i < item_end) tile_run<4, IL, false, false>(a, cta, i, item_end, it, flags);
    tile_close(cta);
}

// Dense scores.  Every work item is decoded as what its first tile says (read here: a host that looked would wait for the
// stream); a tile of another kind inside the item hands its rows over as everywhere.  An arena known to hold NF4 beside INT4
// tiles is decoded as NF4 throughout.
// PASS: behind the 64-row kernel, of the rows that it handed on.
template <bool PASS>
__global__ void __launch_bounds__(ST_THREADS, 1) score_dense_kernel(const __grid_constant__ ScoreArgs a) {
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    dep_launch();
    dep_wait();
    if (a.refused && *a.refused) return;
    __shared__ PassRange range;
    if (PASS && (!*a.handoff_any || !pass_range(a, range))) return;
    uint32_t i = PASS ? 0u : dense_first(a);  // PASS: counted
    const uint32_t first = i, item_end = PASS ? 0xFFFFFFFFu : dense_end(a);
    PassWalk walk{};
    if (PASS) walk = pass_first(a, range);
    WorkItem it = PASS ? pass_item(a, range, walk) : a.stream_items[i];
    uint32_t flags = first_tile_flags(a, it);  // (on its way while the CTA is set up, and the first item's queries with it)
    if (threadIdx.x < 4u * it.n_queries) asm volatile("prefetch.global.L1 [%0];\n" ::"l"(a.q_coarse + (size_t)it.query_begin * D_C + 32u * threadIdx.x));
    if (threadIdx.x == 32) asm volatile("prefetch.global.L1 [%0];\n" ::"l"(a.q_sign + (size_t)it.query_begin * 8));
    if (threadIdx.x == 64 && a.row_offset) asm volatile("prefetch.global.L1 [%0];\n" ::"l"(a.row_offset + it.query_begin));
    const bool nf4_too = a.nf4_table == 1u || (a.nf4_table == 2u && (first_tile_flags(a, a.stream_items[0]) & F_NF4));
    uint32_t* const bits = reinterpret_cast<uint32_t*>(tile_base(smem_raw) + TileLayout<true>::UNDONE);
    for (uint32_t w = threadIdx.x; w < min(((PASS ? range.end - range.mine : item_end - first) + 31u) / 32u, (uint32_t)UNDONE_WORDS); w += ST_THREADS) bits[w] = 0u;  // (ordered by tile_open's barrier)
    TileCta cta = tile_open<true>(smem_raw);
    cta.walk = walk;
    cta.range = &range;
    for (;;) {
        switch (item_kind(flags, nf4_too)) {
            case 0: i = tile_run<0, false, true, true, PASS>(a, cta, i, item_end, it, flags, nf4_too); break;
            case 1: i = tile_run<1, false, true, true, PASS>(a, cta, i, item_end, it, flags, nf4_too); break;
            case 2: i = tile_run<2, false, true, true, PASS>(a, cta, i, item_end, it, flags, nf4_too); break;
            case 3: i = tile_run<3, false, true, true, PASS>(a, cta, i, item_end, it, flags, nf4_too); break;
            default: i = tile_run<4, false, true, true, PASS>(a, cta, i, item_end, it, flags, nf4_too); break;
        }
        if (i >= item_end) break;
    }
    tile_close(cta);
    static_assert(4096 + (ST_THREADS / 32) * BLK_BYTES <= TileLayout<true>::UNDONE, "below the bits");
    if (cta.undone) finish_undone<PASS>(a, bits, &range, smem_raw);
}

}  // namespace
}  // namespace slha
