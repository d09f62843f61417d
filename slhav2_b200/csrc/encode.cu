// Key -> tile encode, query preparation and tile decode for sm_100a.
//
// Restates LearnedModel::{latent, reconstruct, sign_bits, encode_with,
// query_coarse} (scirust/src/learned.rs:247-408), the six quantisers
// (scirust/src/attention/slha_v2/codec/*.rs) and the randomised Hadamard
// transform (scirust/src/incoherence.rs:45-125).
//
// Bit-exactness contract: every decision the reference takes on a float
// (round-half-away, `acc < 0.0`, `t - level > 0.0`, first-minimum NF4 search)
// sits on a float32 sum that the reference accumulates strictly left to right
// with a separate multiply and add.  This kernel keeps that order: each thread
// owns whole output rows and walks the contraction index sequentially with
// __fmul_rn / __fadd_rn (never contracted into FMA), divisions are __fdiv_rn and
// square roots __fsqrt_rn.  Parallelism comes from rows x keys, not from
// splitting a sum, so the tile bytes equal the scalar reference's bit for bit.  Where
// only a decision is stored (sign bits, codes), it is taken on a cheaper value with a
// bound on its error, and on the exact one where the bound does not settle it.
#include <cuda_fp16.h>

#include "common.cuh"

namespace slha {
namespace {

constexpr int enc_threads(int kb) { return kb == 32 ? 128 : 256; }  // threads of a CTA that takes kb keys at a time

struct EncodeArgs {
    const void* keys;        // [n][d] f32 or bf16
    int key_dtype;
    uint64_t n;
    uint32_t d, d_pad;
    const float* p;          // [128][d]
    const float* pt;         // [d][128]
    const float* scale;      // [128]
    const float* zt;         // [d_pad][256]
    const float* z;          // [256][d_pad]
    const uint4* zf;         // fp16 B fragments of z, rows at one norm (model_build), or null: every sign from its exact sum
    float z_guard, z_norm;   // a sum further from zero than z_guard |e| + z_norm |e - e'| has the exact sum's sign (see signs_mma)
    const float* diag;       // [d_pad] or null
    float fwht_inv;          // 1/sqrt(d_pad), rounded as the reference rounds it
    float lambda_c;          // sqrt(pi/512) in f32
    const uint32_t* positions;
    uint32_t position_base;
    const uint16_t* heads;
    int codec;
    unsigned char* tiles;    // output tiles (encode)
    const uint32_t* slots;   // optional scatter: tile i goes to tiles[slots[i]]
    float* q_coarse;         // [n][128]  (query mode)
    uint64_t* q_sign;        // [n][4]    (query mode)
    uint64_t one;            // (1.0f, 1.0f): the compiler must not know it (see add2)
    int kb;                  // keys per CTA pass (power of two, <= 16)
};

__device__ __forceinline__ float rnd_half_away(float x) { return roundf(x); }
__device__ __forceinline__ int sat_i32(float x) { return __float2int_rz(x); }  // Rust `x as i32`: NaN -> 0, saturating, like cvt.rzi.s32.f32
__device__ __forceinline__ int clampi(int v, int lo, int hi) { return min(max(v, lo), hi); }
__device__ __forceinline__ uint32_t scale_byte(float step, float global) {
    // `(step / global * 255.0).round().clamp(1.0, 255.0) as u8`  (int4.rs:48-49)
    float r = rnd_half_away(__fmul_rn(__fdiv_rn(step, global), 255.0f));
    if (r != r) return 0;
    return (uint32_t)fminf(fmaxf(r, 1.0f), 255.0f);
}
// `gap`: lowered to the distance of t from the nearest float between two entries.
__device__ __forceinline__ uint32_t nf4_nearest(float t, float& gap) {
    // nf4.rs:7-18: linear scan over the codebook by rounded distance, first minimum wins.  Entry i + 1 beats entry i from a certain float on
    // (rounded differences are monotone in t), so four comparisons with those floats find the entry; each is the smallest t in
    // [-1, 1] with |fl(t - c[i+1])| < |fl(t - c[i])|.  (A difference of two floats is negative exactly where the first is smaller.)
    constexpr uint32_t from[15] = {0xBF5A8F5Bu, 0xBF1FF2E4u, 0xBEF566CFu, 0xBEBA3054u, 0xBE86CF41u, 0xBE2F9DB2u, 0xBDAD5CFBu, 0x31000000u,
                                   0x3DAD5CFCu, 0x3E2F9DB3u, 0x3E86CF42u, 0x3EBA3056u, 0x3EF566D0u, 0x3F1FF2E5u, 0x3F5A8F5Du};
    const auto f = [&](int i) { return __uint_as_float(from[i]); };
    const float d3 = __fsub_rn(t, f(7));
    const bool b3 = d3 >= 0.0f;
    const float d2 = __fsub_rn(t, b3 ? f(11) : f(3));
    const bool b2 = d2 >= 0.0f;
    const float d1 = __fsub_rn(t, b3 ? (b2 ? f(13) : f(9)) : (b2 ? f(5) : f(1)));
    const bool b1 = d1 >= 0.0f;
    const float lo = b2 ? (b1 ? f(6) : f(4)) : (b1 ? f(2) : f(0)), hi = b2 ? (b1 ? f(14) : f(12)) : (b1 ? f(10) : f(8));
    const float d0 = __fsub_rn(t, b3 ? hi : lo);
    const bool b0 = d0 >= 0.0f;
    gap = fminf(fminf(gap, fminf(fabsf(d3), fabsf(d2))), fminf(fabsf(d1), fabsf(d0)));
    return (b3 ? 8u : 0u) | (b2 ? 4u : 0u) | (b1 ? 2u : 0u) | (b0 ? 1u : 0u);
}
// Rows of h in shared memory hold their 16-byte chunks in an order in which eight lanes that each read the same chunk of their own 16 dimensions
// meet all banks.
__device__ __forceinline__ int h_chunk(int c) { return (c & ~3) | ((c & 3) ^ (c >> 3)); }
__device__ __forceinline__ float octet_max(float v) {  // max over the 8 lanes sharing lane >> 3
    v = fmaxf(v, __shfl_xor_sync(0xFFFFFFFFu, v, 1));
    v = fmaxf(v, __shfl_xor_sync(0xFFFFFFFFu, v, 2));
    return fmaxf(v, __shfl_xor_sync(0xFFFFFFFFu, v, 4));
}

// Code of a value from its quotient q by the unit's step: a nibble, an 8-bit head level, or a 3-bit code (corr: its correction bit).  False where q
// may lie on the other side of the next place at which the code changes than a quotient up to 2^-22 (relative) away: halves of
// integers, for 3-bit codes all multiples of a half (a sum with 3.5 is rounded on the way: 2^-21 more), NF4: the floats between two entries.
enum { Q_INT4, Q_NF4, Q_HEAD, Q_CODE3 };
template <int MODE>
__device__ __forceinline__ bool code_of(float q, uint32_t& code, uint32_t& corr) {
    corr = 0u;
    if (MODE == Q_NF4) {
        float gap = 1.0f;
        code = nf4_nearest(fminf(fmaxf(q, -1.0f), 1.0f), gap);
        return gap > 5e-7f && fabsf(q) < 1e30f;
    }
    if (MODE == Q_CODE3) {
        code = (uint32_t)clampi(sat_i32(rnd_half_away(__fadd_rn(q, 3.5f))), 0, 7);
        corr = __fsub_rn(q, __fsub_rn((float)code, 3.5f)) > 0.0f ? 1u : 0u;
        const float h = __fadd_rn(q, q);
        return fabsf(__fsub_rn(h, rintf(h))) > 8e-6f && fabsf(q) < 8.0f;
    }
    constexpr int lo = MODE == Q_HEAD ? -128 : -8, hi = MODE == Q_HEAD ? 127 : 7;
    code = (uint32_t)(clampi(sat_i32(rnd_half_away(q)), lo, hi) - lo);
    return fabsf(__fsub_rn(q, rintf(q))) < 0.5f - (MODE == Q_HEAD ? 6e-5f : 4e-6f) && fabsf(q) < 1.5f * hi;
}
// The codes of a unit's values v (nibbles, head levels, or 3-bit codes two times eight with their correction bits).  Every decision is taken on the
// rounded quotient v / eff; v * (1 / eff) is within 2^-22 of it (half an ulp each for the reciprocal, the product and the quotient), so only
// the values for which that is not enough are divided -- one in 10^5, and the largest of a key's 3-bit codes.  A division is a branch of its
// own to the compiler: sixteen of them in a row, one after the other, took a fifth of the kernel.
template <int MODE>
__device__ __forceinline__ void quantize_values(const float (&v)[16], const float* h, int first, float eff, uint32_t (&w)[2], uint32_t& corr) {
    constexpr int N = MODE == Q_HEAD ? 8 : 16, BITS = MODE == Q_HEAD ? 8 : (MODE == Q_CODE3 ? 3 : 4), PER = N / 2;
    const bool usual = eff >= 8.6736174e-19f && eff <= 1.1529215e18f;  // 2^-60 .. 2^60
    const float inv = __fdiv_rn(1.0f, eff);
    uint32_t again = 0, code, c;
    w[0] = w[1] = corr = 0u;
#pragma unroll
    for (int i = 0; i < N; ++i) {
        const bool sure = code_of<MODE>(__fmul_rn(v[i], inv), code, c);
        w[i / PER] |= code << (BITS * (i % PER));
        corr |= c << i;
        again |= sure ? 0u : 1u << i;
    }
    if (!usual) again = (1u << N) - 1u;
    while (again) {
        const int i = __ffs(again) - 1, dim = first + i;
        again &= again - 1u;
        const float x = h[4 * h_chunk(dim >> 2) + (dim & 3)];
        code_of<MODE>(MODE != Q_NF4 || eff > 0.0f ? __fdiv_rn(x, eff) : 0.0f, code, c);
        const uint32_t at = BITS * (i % PER), keep = ~(((1u << BITS) - 1u) << at);
        if (i < PER) w[0] = (w[0] & keep) | code << at;
        else w[1] = (w[1] & keep) | code << at;
        corr = (corr & ~(1u << i)) | c << i;
    }
}

// Quantise one latent into the 64 latent bytes + scale + 8 scale bytes of a tile in shared memory: eight lanes per key, lane u has scale
// unit u -- 16 dimensions from 16 u on, or for the head + body codecs (mixed.rs:15-33, mix3.rs:13-31) dimensions 0..7 (u = 0) and 16
// from 16 u - 8 on, the last eight dropped.  A lane finds its step and its scale byte for itself, the key's scale takes three shuffles,
// and the lane's bytes lie together in the tile.  All lanes of the warp call; on: the lane has a key.
__device__ __forceinline__ void quantize_unit(const float* h, int codec, unsigned char* tile, int u, bool on) {
    const bool headbody = codec == SLHA_CODEC_MIXED || codec == SLHA_CODEC_MIX3, head = headbody && u == 0;
    float v[16];
#pragma unroll
    for (int c = 0; c < 4; ++c) {
        const int at = h_chunk(headbody ? (u ? 4 * u - 2 + c : (c & 1)) : 4 * u + c);
        const float4 x = reinterpret_cast<const float4*>(h)[at];
        const bool in = !head || c < 2;
        v[4 * c] = in ? x.x : 0.0f;
        v[4 * c + 1] = in ? x.y : 0.0f;
        v[4 * c + 2] = in ? x.z : 0.0f;
        v[4 * c + 3] = in ? x.w : 0.0f;
    }
    float mx = 0.0f;
#pragma unroll
    for (int i = 0; i < 16; ++i) mx = fmaxf(mx, fabsf(v[i]));
    float global;
    uint32_t gsb = 255;
    if (codec == SLHA_CODEC_INT4_SINGLE) {  // int4.rs:9-24
        mx = octet_max(mx);
        global = mx > 0.0f ? __fdiv_rn(mx, 7.0f) : 1.0f;
    } else {
        // step = absmax / {7, 1, 3.5} (int4.rs:34-63, nf4.rs:23-57, tq3.rs:10-49), of the 8-bit head absmax / 127
        if (codec == SLHA_B200_CODEC_INT4_GROUPED32) mx = fmaxf(mx, __shfl_xor_sync(0xFFFFFFFFu, mx, 1));
        const float div = head ? 127.0f : (codec == SLHA_CODEC_TQ3 || codec == SLHA_CODEC_MIX3 ? 3.5f : 7.0f);
        const float step = codec == SLHA_CODEC_NF4 ? mx : __fdiv_rn(mx, div);
        const float g = octet_max(step);
        global = g > 0.0f ? g : 1.0f;
        gsb = scale_byte(step, global);
    }
    const float eff = codec == SLHA_CODEC_INT4_SINGLE ? global : __fmul_rn(global, __fdiv_rn((float)gsb, 255.0f));
    if (!on) return;
    tile[120 + u] = (unsigned char)gsb;
    if (u == 0) *reinterpret_cast<float*>(tile + 96) = global;
    const int first = headbody && !head ? 16 * u - 8 : 16 * u;
    uint32_t w[2], corr;
    if (head) {
        quantize_values<Q_HEAD>(v, h, first, eff, w, corr);
        *reinterpret_cast<uint2*>(tile) = make_uint2(w[0], w[1]);
    } else if (codec == SLHA_CODEC_TQ3 || codec == SLHA_CODEC_MIX3) {
        quantize_values<Q_CODE3>(v, h, first, eff, w, corr);
        // code plane: 6 bytes per unit from byte 0 (TQ3) or 8 (MIX3, whose unit 0 is the head); correction plane behind it
        const int cu = headbody ? u - 1 : u;
        uint16_t* cp = reinterpret_cast<uint16_t*>(tile + (headbody ? 8 : 0) + 6 * cu);
        cp[0] = (uint16_t)w[0];
        cp[1] = (uint16_t)(w[0] >> 16 | w[1] << 8);
        cp[2] = (uint16_t)(w[1] >> 8);
        *reinterpret_cast<uint16_t*>(tile + (headbody ? 50 : 48) + 2 * cu) = (uint16_t)corr;
    } else {
        if (codec == SLHA_CODEC_NF4) quantize_values<Q_NF4>(v, h, first, eff, w, corr);
        else quantize_values<Q_INT4>(v, h, first, eff, w, corr);
        *reinterpret_cast<uint2*>(tile + 8 * u) = make_uint2(w[0], w[1]);
    }
}

// acc[j] += x * v[j] for NK keys whose values lie consecutively (16-byte aligned when NK % 4 == 0),
// each as a separate multiply and add (the reference never fuses them).
template <int NK>
__device__ __forceinline__ void axpy_keys(float (&acc)[NK], float x, const float* v) {
    if (NK % 4 == 0) {
#pragma unroll
        for (int j4 = 0; j4 < NK / 4; ++j4) {
            const float4 b4 = reinterpret_cast<const float4*>(v)[j4];
            acc[4 * j4 + 0] = __fadd_rn(acc[4 * j4 + 0], __fmul_rn(x, b4.x));
            acc[4 * j4 + 1] = __fadd_rn(acc[4 * j4 + 1], __fmul_rn(x, b4.y));
            acc[4 * j4 + 2] = __fadd_rn(acc[4 * j4 + 2], __fmul_rn(x, b4.z));
            acc[4 * j4 + 3] = __fadd_rn(acc[4 * j4 + 3], __fmul_rn(x, b4.w));
        }
    } else {
#pragma unroll
        for (int j = 0; j < NK; ++j) acc[j] = __fadd_rn(acc[j], __fmul_rn(x, v[j]));
    }
}

// NK consecutive floats (16-byte aligned when NK % 4 == 0) to / from registers
template <int NK>
__device__ __forceinline__ void store_keys(float* dst, const float (&v)[NK]) {
    if (NK % 4 == 0) {
#pragma unroll
        for (int j4 = 0; j4 < NK / 4; ++j4)
            reinterpret_cast<float4*>(dst)[j4] = make_float4(v[4 * j4], v[4 * j4 + 1], v[4 * j4 + 2], v[4 * j4 + 3]);
    } else {
#pragma unroll
        for (int j = 0; j < NK; ++j) dst[j] = v[j];
    }
}
template <int NK>
__device__ __forceinline__ void load_keys(float (&v)[NK], const float* src) {
    if (NK % 4 == 0) {
#pragma unroll
        for (int j4 = 0; j4 < NK / 4; ++j4) {
            const float4 x = reinterpret_cast<const float4*>(src)[j4];
            v[4 * j4] = x.x; v[4 * j4 + 1] = x.y; v[4 * j4 + 2] = x.z; v[4 * j4 + 3] = x.w;
        }
    } else {
#pragma unroll
        for (int j = 0; j < NK; ++j) v[j] = src[j];
    }
}

// Packed pairs of float32 (Blackwell f32x2): one instruction works on two independent float32 values, each rounded to
// nearest exactly like the scalar operation.  A multiply-add of a key pair is a packed multiply and a packed sum, two issue
// slots for two multiplies and two additions.  The sum is written as fma(product, one, acc) with `one` = (1, 1) from the
// kernel's arguments: product * 1 is exact, so it rounds once, like an addition.  A plain packed addition would be contracted
// with the multiply before it into one fused multiply-add even when both carry an explicit rounding mode and contraction is
// switched off (seen on sm_100a, CUDA 12.9), and a fused multiply-add rounds once where the reference rounds twice.
// Bound: 65 536 multiplies and additions per key (latent and residual) at d = 128 on 128 fp32 lanes per SM: 568 M keys/s, 461 us for
// 262 144 bf16 keys, which take 747 us.  (With the signs in the same form 1251 us, with scalar sums, three issue slots instead of two, 1327.)
__device__ __forceinline__ uint64_t pack2(float lo, float hi) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};\n" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ void unpack2(uint64_t v, float& lo, float& hi) { asm("mov.b64 {%0, %1}, %2;\n" : "=f"(lo), "=f"(hi) : "l"(v)); }
__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b) {
    uint64_t m;
    asm("mul.rn.f32x2 %0, %1, %2;\n" : "=l"(m) : "l"(a), "l"(b));
    return m;
}
__device__ __forceinline__ uint64_t add2(uint64_t p, uint64_t one, uint64_t acc) {
    uint64_t r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;\n" : "=l"(r) : "l"(p), "l"(one), "l"(acc));
    return r;
}

// acc[r][j] += m[r] * v[j] for an R x K register tile: R output rows (or columns) times K keys, keys in pairs.
// Each output still sums its products in contraction order, one multiply and one add at a time.
template <int R, int K>
__device__ __forceinline__ void outer_keys(uint64_t (&acc)[R][K / 2], const float4& m4, const float* v, uint64_t one) {
    static_assert(R == 4 && K % 4 == 0, "the matrix operand is one 16-byte load");
    uint64_t kv[K / 2];
#pragma unroll
    for (int j4 = 0; j4 < K / 4; ++j4) {
        const float4 x = reinterpret_cast<const float4*>(v)[j4];
        kv[2 * j4] = pack2(x.x, x.y);
        kv[2 * j4 + 1] = pack2(x.z, x.w);
    }
    const uint64_t m[4] = {pack2(m4.x, m4.x), pack2(m4.y, m4.y), pack2(m4.z, m4.z), pack2(m4.w, m4.w)};
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
        for (int j = 0; j < K / 2; ++j) acc[r][j] = add2(mul2(m[r], kv[j]), one, acc[r][j]);
}
template <int R, int K>
__device__ __forceinline__ void zero_tile(uint64_t (&acc)[R][K / 2]) {
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
        for (int j = 0; j < K / 2; ++j) acc[r][j] = 0ull;
}
template <int R, int K>
__device__ __forceinline__ void unpack_tile(const uint64_t (&acc)[R][K / 2], float (&out)[R][K]) {
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
        for (int j = 0; j < K / 2; ++j) unpack2(acc[r][j], out[r][2 * j], out[r][2 * j + 1]);
}

// floats between the rows of the transposed [..][KB] arrays in shared memory
__host__ __device__ constexpr int enc_row_stride(int kb) { return kb >= 8 ? kb + 4 : kb; }

// ---- sign bits on the tensor cores ---------------------------------------------------------------------------------------
// A tile stores only the signs of the 256 projections Z e, and e is exact (in the reference's order) before they are taken.  So the
// sums run as m16n8k16 MMAs over fp16 roundings of Z (its rows scaled to one norm) and of e (scaled by a power of two), and only a sum
// closer to zero than its error bound is taken again in the reference's order.  With z' and e' the roundings, n = d_pad terms:
//   rounding of both factors               |z - z'| |e| + |z'| |e - e'|   (norms, measured: about 2^-12.3 |z| |e| each)
//   fp32 accumulation in the MMAs          2^-13.9 |z| |e|                (17 addends an MMA, each cut at 2^-22 of the largest, 16 MMAs; no document
//                                                                          says how they are summed: measured, addends are kept to 2^-25 of the
//                                                                          largest, and 256 products beside one large end within 2^-17.7)
//   the reference's own sequential sum     2^-16 |z| |e|                  (n + 1 roundings of 2^-24, n <= 256)
// (model_build gives no fragments for n > 256 or a Z of unusual size).  Gaussian rows of Z leave about 1.1 of 256 signs of a key inside
// the bound at d = 128, 1.6 at d_pad = 256.
constexpr int SIGN_LIST = 32;                    // sums of a key that may be taken again before the whole pass is summed exactly
__host__ __device__ constexpr int sign_stride(int kb) { return kb == 32 ? 40 : (kb == 16 ? 24 : kb); }  // words between pairs of rows: conflict-free fragment loads
__host__ __device__ constexpr uint32_t sign_rows(uint32_t dp) { return (dp + 31) / 32 * 32; }
// words of the phase's own shared memory: count | bound [KB] | list | fp16 pairs [rows / 2][stride], later rows of z
__host__ __device__ constexpr uint32_t sign_fixed(int kb) { return 4u + (uint32_t)kb + (uint32_t)(kb * SIGN_LIST / 2); }
__host__ __device__ constexpr uint32_t sign_words(uint32_t dp, int kb) {
    return sign_fixed(kb) + (sign_rows(dp) / 2 * (uint32_t)sign_stride(kb) + 8u > dp + 7u ? sign_rows(dp) / 2 * (uint32_t)sign_stride(kb) + 8u : dp + 7u);
}
__device__ __forceinline__ void mma_16816(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
template <int N>
__device__ __forceinline__ void load_words(float (&v)[N], const float* src) {  // N = 8, 4, 2, 1, aligned to min(N, 4) words
    if (N >= 4) {
#pragma unroll
        for (int q = 0; q < N / 4; ++q) {
            const float4 x = reinterpret_cast<const float4*>(src)[q];
            v[4 * q] = x.x; v[(4 * q + 1) % N] = x.y; v[(4 * q + 2) % N] = x.z; v[(4 * q + 3) % N] = x.w;
        }
    } else if (N == 2) {
        const float2 x = *reinterpret_cast<const float2*>(src);
        v[0] = x.x; v[1 % N] = x.y;
    } else {
        v[0] = *src;
    }
}

// Signs of Z e for the KB columns of buf [dp][KS], into the sign words of the tiles at tl.  All threads of the CTA; buf is complete
// (a barrier lies between its writers and this call) and the `words` words at `w` are free.  meanwhile: work that only reads buf.  False (for
// all threads alike): too many sums lie too close to zero, nothing usable was written.
template <int KB, typename F>
__device__ __forceinline__ bool signs_mma(const EncodeArgs& a, const float* buf, unsigned char* tl, uint32_t* w, uint32_t words, F&& meanwhile) {
    constexpr int KS = enc_row_stride(KB), STR = sign_stride(KB), MT = KB == 32 ? 2 : 1, NT = enc_threads(KB), WARPS = NT / 32;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
    const uint32_t dp = a.d_pad, rows = sign_rows(dp);
    uint32_t* cnt = w;
    float* bound = reinterpret_cast<float*>(cnt + 4);
    uint16_t* list = reinterpret_cast<uint16_t*>(bound + KB);
    uint32_t* eh = w + sign_fixed(KB);
    if (tid == 0) *cnt = 0u;
    // the first fragments are on their way while the keys are scaled; those of every further two steps follow one turn ahead
    const uint4* zf = a.zf + (size_t)(4 * warp) * 32 + lane;
    uint4 ahead[4];
#pragma unroll
    for (int n = 0; n < 4; ++n) ahead[n] = __ldg(zf + n * 32);
    // a warp's keys (KW consecutive columns): largest element, then the scaled fp16 pairs with the norms of what they hold and of what they lost
    constexpr int KW = KB >= WARPS ? KB / WARPS : 1;
    if (KW * warp < KB) {
        const float* col = buf + KW * warp;
        uint32_t mx[KW];
        float ss[KW], lost[KW], sc[KW];
#pragma unroll
        for (int j = 0; j < KW; ++j) { mx[j] = 0u; ss[j] = lost[j] = 0.0f; }
#pragma unroll 4
        for (uint32_t i = lane; i < dp; i += 32) {
            float x[KW];
            load_words<KW>(x, col + (size_t)i * KS);
#pragma unroll
            for (int j = 0; j < KW; ++j) mx[j] = max(mx[j], __float_as_uint(x[j]) & 0x7FFFFFFFu);
        }
#pragma unroll
        for (int j = 0; j < KW; ++j) {
            mx[j] = __reduce_max_sync(0xFFFFFFFFu, mx[j]);
            // 2^p with the largest element in [2^12, 2^13); elements of ordinary size only, so that nothing leaves the normal range
            // (other keys, infinities and NaN among them, become zeros within an infinite bound: summed exactly)
            const bool usual = mx[j] >= (67u << 23) && mx[j] < (187u << 23);  // [2^-60, 2^60)
            sc[j] = usual ? __uint_as_float((266u - (mx[j] >> 23)) << 23) : 0.0f;
        }
#pragma unroll 2
        for (uint32_t r = lane; r < rows / 2; r += 32) {
            float x[KW] = {}, y[KW] = {};
            if (2 * r < dp) load_words<KW>(x, col + (size_t)(2 * r) * KS);
            if (2 * r + 1 < dp) load_words<KW>(y, col + (size_t)(2 * r + 1) * KS);
            float h[KW];
#pragma unroll
            for (int j = 0; j < KW; ++j) {
                const float u = sc[j] != 0.0f ? x[j] * sc[j] : 0.0f, v = sc[j] != 0.0f ? y[j] * sc[j] : 0.0f;
                const __half2 p = __floats2half2_rn(u, v);
                const float2 q = __half22float2(p);
                ss[j] = fmaf(u, u, fmaf(v, v, ss[j]));
                lost[j] = fmaf(u - q.x, u - q.x, fmaf(v - q.y, v - q.y, lost[j]));
                h[j] = *reinterpret_cast<const float*>(&p);
            }
            store_keys<KW>(reinterpret_cast<float*>(eh) + r * STR + KW * warp, h);
        }
#pragma unroll
        for (int j = 0; j < KW; ++j) {
            // sums over the warp in fixed point, rounded up: a lane's eight squares are below 2^29, its lost parts (half an ulp, at most 2) below 2^6
            const float e2 = 8.0f * (float)__reduce_add_sync(0xFFFFFFFFu, (uint32_t)(ss[j] * 0.125f) + 1u);
            const float l2 = 9.5367431640625e-7f * (float)__reduce_add_sync(0xFFFFFFFFu, (uint32_t)(lost[j] * 1048576.0f) + 1u);
            const float lim = a.z_guard * (e2 * rsqrtf(e2)) + a.z_norm * (l2 * rsqrtf(l2));  // (rounding: slack of the two factors)
            if (lane == j) bound[KW * warp + j] = sc[j] != 0.0f ? lim : (mx[j] == 0u ? -1.0f : INFINITY);  // (an all-zero key has no negative sum)
        }
    }
    __syncthreads();
    meanwhile();
    // M = keys (rows of no key give sums nobody reads), N = hyperplanes 32 word .. + 31: one word of every key at a time
    constexpr int HALVES = KB > 8 ? 2 : 1, WORDS = 8 / WARPS;
    uint32_t near[WORDS][MT * HALVES], nears = 0;
    const bool mine = KB >= 8 || g < KB;
#pragma unroll
    for (int wd = 0; wd < WORDS; ++wd) {
        const int word = warp + wd * WARPS;
        float acc[MT][4][4];
#pragma unroll
        for (int m = 0; m < MT; ++m)
#pragma unroll
            for (int n = 0; n < 4; ++n)
#pragma unroll
                for (int c = 0; c < 4; ++c) acc[m][n][c] = 0.0f;
#pragma unroll 2
        for (uint32_t k2 = 0; k2 < rows / 32; ++k2) {
            uint4 b[4];
            const bool last = k2 + 1 == rows / 32;
            const uint4* next = last ? zf + (size_t)(wd + 1) * (4 * WARPS * 32) : zf + (size_t)wd * (4 * WARPS * 32) + (size_t)(k2 + 1) * 1024;
#pragma unroll
            for (int n = 0; n < 4; ++n) {
                b[n] = ahead[n];
                if (!last || wd + 1 < WORDS) ahead[n] = __ldg(next + n * 32);
            }
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const uint32_t* er = eh + (16 * k2 + 8 * h + t) * STR + g;
#pragma unroll
                for (int m = 0; m < MT; ++m) {
                    uint32_t x[4];
                    x[0] = er[16 * m];
                    x[1] = KB > 8 ? er[16 * m + 8] : 0u;
                    x[2] = er[4 * STR + 16 * m];
                    x[3] = KB > 8 ? er[4 * STR + 16 * m + 8] : 0u;
#pragma unroll
                    for (int n = 0; n < 4; ++n) mma_16816(acc[m][n], x, h ? b[n].z : b[n].x, h ? b[n].w : b[n].y);
                }
            }
        }
        // bit 8 n + 2 t + c of the word of key 16 m + 8 half + g
#pragma unroll
        for (int m = 0; m < MT; ++m)
#pragma unroll
            for (int half = 0; half < HALVES; ++half) {
                const int key = 16 * m + 8 * half + g;
                const float lim = mine ? bound[key] : -1.0f;
                uint32_t v = 0, close = 0;  // sign bits shifted in: a sum is close where |sum| - bound is negative
#pragma unroll
                for (int n = 3; n >= 0; --n) {
                    v <<= 6;
                    close <<= 6;
#pragma unroll
                    for (int c = 1; c >= 0; --c) {
                        const float x = acc[m][n][2 * half + c];
                        v = __funnelshift_l(__float_as_uint(x), v, 1);
                        close = __funnelshift_l(__float_as_uint(__fsub_rn(fabsf(x), lim)), close, 1);
                    }
                }
                v &= ~close;
                if (!mine) close = 0u;
                v <<= 2 * t;
                near[wd][m * HALVES + half] = close << (2 * t);
                nears += __popc(close);
                v |= __shfl_xor_sync(0xFFFFFFFFu, v, 1);
                v |= __shfl_xor_sync(0xFFFFFFFFu, v, 2);
                if (t == 0 && mine) reinterpret_cast<uint32_t*>(tl + (size_t)key * TILE_BYTES + 64)[word] = v;
            }
    }
    // the sums to take again go to the list, one reservation per warp
    if (__any_sync(0xFFFFFFFFu, nears != 0u)) {
        uint32_t at = nears;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, at, o);
            if (lane >= o) at += y;
        }
        uint32_t base = 0;
        if (lane == 31) base = atomicAdd(cnt, at);
        at += __shfl_sync(0xFFFFFFFFu, base, 31) - nears;
#pragma unroll
        for (int wd = 0; wd < WORDS; ++wd)
#pragma unroll
            for (int i = 0; i < MT * HALVES; ++i)
                for (uint32_t b = near[wd][i]; b; b &= b - 1u, ++at)
                    if (at < KB * SIGN_LIST) list[at] = (uint16_t)((8 * i + g) << 8 | (32 * (warp + wd * WARPS) + __ffs(b) - 1));
    }
    __syncthreads();
    const uint32_t again = *cnt;
    if (again > KB * SIGN_LIST) return false;
    // The rows of Z are copied together, a warp per row, to the place of the fp16 pairs; then a thread per sum.  (With every thread loading its
    // own row each load met 32 lines, and the phase was bound by the L1's tags.)
    float* zs = reinterpret_cast<float*>(eh);
    const uint32_t stride = (dp + 7) / 4 * 4, room = min((words - sign_fixed(KB)) / stride, (uint32_t)NT);  // (4 words over a multiple of 32: no bank conflicts)
    for (uint32_t e0 = 0; e0 < again; e0 += room) {
        const uint32_t n = min(room, again - e0);
        // (eight rows a warp at a time: their numbers are read before the first copy is issued)
        for (uint32_t e = warp; dp % 4 == 0 && e < n; e += 8 * WARPS) {
            uint32_t row[8];
#pragma unroll
            for (int q = 0; q < 8; ++q) row[q] = e + q * WARPS < n ? (list[e0 + e + q * WARPS] & 255u) * dp : ~0u;
            const uint32_t to = (uint32_t)__cvta_generic_to_shared(zs + e * stride);
            for (uint32_t i = 4 * lane; i < dp; i += 128)
#pragma unroll
                for (int q = 0; q < 8; ++q)
                    if (row[q] != ~0u) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(to + 4 * (q * WARPS * stride + i)), "l"(a.z + row[q] + i));
        }
        // (rows that start at any word: by words, and copied all the same; through registers 300 queries of 202 dimensions took 24.5 us a call, now 15.8)
#pragma unroll 1
        for (uint32_t e = warp; dp % 4 != 0 && e < n; e += WARPS) {
            const float* z = a.z + (list[e0 + e] & 255u) * dp;
            const uint32_t to = (uint32_t)__cvta_generic_to_shared(zs + e * stride);
#pragma unroll 1
            for (uint32_t i = lane; i < dp; i += 32) asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(to + 4 * i), "l"(z + i));
        }
        asm volatile("cp.async.wait_all;\n" ::: "memory");
        __syncthreads();
        if (tid < n) {
            const uint32_t key = list[e0 + tid] >> 8, s = list[e0 + tid] & 255u;
            const float* z = zs + tid * stride;
            const float* x = buf + key;
            float sum = 0.0f;
            uint32_t i = 0;
            for (; i + 32 <= dp; i += 32) {  // all products of a turn before its sums
                float p[32];
#pragma unroll
                for (int j = 0; j < 32; j += 4) {
                    const float4 z4 = *reinterpret_cast<const float4*>(z + i + j);
                    p[j] = __fmul_rn(z4.x, x[(size_t)(i + j) * KS]);
                    p[j + 1] = __fmul_rn(z4.y, x[(size_t)(i + j + 1) * KS]);
                    p[j + 2] = __fmul_rn(z4.z, x[(size_t)(i + j + 2) * KS]);
                    p[j + 3] = __fmul_rn(z4.w, x[(size_t)(i + j + 3) * KS]);
                }
#pragma unroll
                for (int j = 0; j < 32; ++j) sum = __fadd_rn(sum, p[j]);
            }
            for (; i < dp; ++i) sum = __fadd_rn(sum, __fmul_rn(z[i], x[(size_t)i * KS]));
            if (sum < 0.0f) atomicOr(reinterpret_cast<uint32_t*>(tl + (size_t)key * TILE_BYTES + 64) + (s >> 5), 1u << (s & 31u));
        }
        if (e0 + room < again) __syncthreads();
    }
    return true;
}

// Residuals of 32 keys for up to 32 C columns, C columns (32 apart) times 8 keys a thread: e = key - sum_k w_k P[k][column], in place of the key.
template <int C>
__device__ __forceinline__ void residual_columns(const EncodeArgs& a, float* buf, const float* wsT) {
    constexpr int KS = enc_row_stride(32);
    const uint32_t d = a.d, c0 = 8 * (threadIdx.x >> 5) + (threadIdx.x & 7), kg = (threadIdx.x & 31) >> 3;
    const float* mp = a.p + c0;
    const float* wr = wsT + 8 * kg;
    uint64_t acc[C][4] = {};
#pragma unroll 4
    for (int k = 0; k < D_C; ++k) {
        uint64_t kv[4];
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            const float4 x = reinterpret_cast<const float4*>(wr + (size_t)k * KS)[j];
            kv[2 * j] = pack2(x.x, x.y);
            kv[2 * j + 1] = pack2(x.z, x.w);
        }
#pragma unroll
        for (int c = 0; c < C; ++c) {
            const float m = c0 + 32 * c < d ? __ldg(mp + (size_t)k * d + 32 * c) : 0.0f;
            const uint64_t mm = pack2(m, m);
#pragma unroll
            for (int j = 0; j < 4; ++j) acc[c][j] = add2(mul2(mm, kv[j]), a.one, acc[c][j]);
        }
    }
#pragma unroll
    for (int c = 0; c < C; ++c) {
        if (c0 + 32 * c >= d) continue;
        float* row = buf + (size_t)(c0 + 32 * c) * KS + 8 * kg;
        float e[8], kv[8];
        load_keys<8>(kv, row);
#pragma unroll
        for (int j = 0; j < 4; ++j) unpack2(acc[c][j], e[2 * j], e[2 * j + 1]);
#pragma unroll
        for (int j = 0; j < 8; ++j) e[j] = __fsub_rn(kv[j], e[j]);
        store_keys<8>(row, e);
    }
}

// 2^R-point stretches of the Hadamard butterflies of buf [dp][KS] in registers: the stages h, 2 h, .. 2^(R-1) h, each sum and difference the
// reference's.  first: the inputs times the diagonal; last: the outputs times 1/sqrt(dp).
template <int KB, int R>
__device__ __forceinline__ void fwht_stages(float* buf, uint32_t dp, uint32_t log2_h, const float* diag, float inv) {
    constexpr int KS = enc_row_stride(KB), P = 1 << R, NT = enc_threads(KB);
    const bool last = (1u << (log2_h + R)) == dp;
    const uint32_t h = 1u << log2_h;
    for (uint32_t e = threadIdx.x; e < (dp >> R) * KB; e += NT) {
        const uint32_t q = e / KB, at = ((q >> log2_h) << (log2_h + R)) + (q & (h - 1u));
        float* col = buf + (size_t)at * KS + e % KB;
        float x[P];
#pragma unroll
        for (int r = 0; r < P; ++r) {
            x[r] = col[(size_t)(r * h) * KS];
            if (log2_h == 0) x[r] = __fmul_rn(x[r], __ldg(diag + at + r));
        }
#pragma unroll
        for (int o = 1; o < P; o <<= 1)
#pragma unroll
            for (int r = 0; r < P; ++r)
                if (!(r & o)) {
                    const float u = x[r], v = x[r + o];
                    x[r] = __fadd_rn(u, v);
                    x[r + o] = __fsub_rn(u, v);
                }
#pragma unroll
        for (int r = 0; r < P; ++r) col[(size_t)(r * h) * KS] = last ? __fmul_rn(x[r], inv) : x[r];
    }
}

// KB keys per CTA pass (compile time: 32 unless the model dimension leaves no room).  Every
// contraction is walked sequentially by the thread that owns the output element, for all the keys
// the thread holds at once.

// CTAs of KB keys whose registers fit on an SM together: four of 32 keys at head dimension 128 (57 KB of shared memory each), two of 16 or 8.  (16
// keys with 180 registers, one CTA an SM: 20 011 keys of 512 dimensions 772 us, with 127 registers 564.)
constexpr int enc_ctas(int kb) { return kb == 32 ? 4 : (kb >= 8 ? 2 : 1); }

template <bool QUERY, int KB>
__global__ void __launch_bounds__(enc_threads(KB), enc_ctas(KB)) encode_kernel(EncodeArgs a) {
    extern __shared__ __align__(16) unsigned char smem[];
    dep_wait();  // (no dep_launch: CTAs of the next call that came to wait here were spread unevenly over the SMs, 7000 keys of 128 dimensions 42 us -> 55)
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    constexpr int PER = KB >= 2 ? KB / 2 : 1;  // keys per thread where two threads share an output row
    constexpr int NT = enc_threads(KB);
    const uint32_t d = a.d, dp = a.d_pad;
    // shared: tiles [KB][128 B] | buf [d_pad][KS] | h [KB][128] | wsT [128][KS]
    // (buf holds the keys, then in their place the residuals, the sign-LSH input, transposed so that one thread
    // reads the KB values of a contraction index with 16-byte loads).  Rows are KS = KB + 4
    // floats apart: a warp whose lanes walk the rows then spreads its 16-byte accesses over
    // all banks, while lanes that walk the keys of one row stay on consecutive banks.  The sign phase works in the
    // space of h and wsT.
    constexpr int KS = enc_row_stride(KB);
    unsigned char* tl = smem;
    float* buf = reinterpret_cast<float*>(tl + (size_t)KB * TILE_BYTES);
    float* hs = buf + (((size_t)dp * KS + 3) & ~size_t(3));
    float* wsT = hs + (size_t)KB * D_C;  // h_k * s_k of every key, transposed like buf

    for (uint64_t base = (uint64_t)blockIdx.x * KB; base < a.n; base += (uint64_t)gridDim.x * KB) {
        const int nk = (int)min((uint64_t)KB, a.n - base);
        __syncthreads();
        // ---- load keys (transposed: buf[i][j]); absent keys and padding rows are zero ------
        const bool f32 = a.key_dtype == SLHA_B200_F32;
        const uint32_t epc = f32 ? 4u : 8u;  // elements per 16-byte chunk
        if (KB >= 8 && d % epc == 0 && (reinterpret_cast<uintptr_t>(a.keys) & 15) == 0) {
            // 16-byte chunks; the lanes of a warp take the same chunk of consecutive keys, so
            // that their transposed stores fall on consecutive banks.  All loads of a thread
            // are in flight before the first store.  (Ordinary loads: this grid may be resident while the keys are written, see dep_wait.)
            constexpr int U = 512 / NT;
            const uint32_t cpk = d / epc, total = cpk * (uint32_t)KB;
            const uint4* src = reinterpret_cast<const uint4*>(a.keys) + base * cpk;
            for (uint32_t c0 = tid; c0 < total; c0 += U * NT) {
                uint4 v[U];
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const uint32_t c = c0 + u * NT, j = c % KB, ic = c / KB;
                    v[u] = make_uint4(0u, 0u, 0u, 0u);
                    if (c < total && (int)j < nk) v[u] = src[(size_t)j * cpk + ic];
                }
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const uint32_t c = c0 + u * NT, j = c % KB, ic = c / KB;
                    if (c >= total) continue;
                    float* dst = buf + (size_t)(ic * epc) * KS + j;
                    const uint32_t w[4] = {v[u].x, v[u].y, v[u].z, v[u].w};
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        if (f32) {
                            dst[(size_t)q * KS] = __uint_as_float(w[q]);
                        } else {  // bf16 -> f32 widening is exact
                            dst[(size_t)(2 * q) * KS] = __uint_as_float(w[q] << 16);
                            dst[(size_t)(2 * q + 1) * KS] = __uint_as_float(w[q] & 0xFFFF0000u);
                        }
                    }
                }
            }
        } else {
            for (uint32_t e = tid; e < d * (uint32_t)KB; e += NT) {
                const int j = e / d;
                const uint32_t i = e % d;
                float x = 0.0f;
                if (j < nk) {
                    const uint64_t o = (base + j) * d + i;
                    x = f32 ? reinterpret_cast<const float*>(a.keys)[o]
                            : __uint_as_float((uint32_t)reinterpret_cast<const uint16_t*>(a.keys)[o] << 16);
                }
                buf[(size_t)i * KS + j] = x;
            }
        }
        for (uint32_t e = d * KS + tid; e < dp * KS; e += NT) buf[e] = 0.0f;
        __syncthreads();

        // With 32 keys per pass every thread holds a 4 x 8 tile of outputs: four matrix elements (one 16-byte load) and eight key
        // values (two 16-byte loads) feed 32 multiply-adds.  An SM's load path fills 128 bytes of registers a cycle, whether
        // lanes load the same address or not, and its fp32 lanes take 64 cycles for the four warps' steps: 48 cycles of fills here, as many
        // as the arithmetic with 4 x 4 tiles (encode of 262 144 bf16 keys, NF4: 888 us with those and 256 threads).  A warp's tiles
        // form 32 outputs x 32 keys, so that a CTA reads each matrix once.
        const bool tiled = KB == 32 && d % 4 == 0 &&
                           ((reinterpret_cast<uintptr_t>(a.pt) | reinterpret_cast<uintptr_t>(a.p) |
                             reinterpret_cast<uintptr_t>(a.zt) | reinterpret_cast<uintptr_t>(a.scale)) & 15) == 0;
        // ---- latent / q_coarse: rows 4 rl .. +3, keys 8 kl .. +7 ------------
        if (KB == 32 && tiled) {
            const int rl = 8 * warp + (lane & 7), kl = lane >> 3;
            uint64_t acc2[4][4];
            zero_tile<4, 8>(acc2);
            const float4* mp = reinterpret_cast<const float4*>(a.pt) + rl;
#pragma unroll 8
            for (uint32_t i = 0; i < d; ++i)
                outer_keys<4, 8>(acc2, __ldg(mp + (size_t)i * (D_C / 4)), buf + (size_t)i * KS + 8 * kl, a.one);
            float acc[4][8];
            unpack_tile<4, 8>(acc2, acc);
            const float4 s4 = __ldg(reinterpret_cast<const float4*>(a.scale) + rl);
            const float sk[4] = {s4.x, s4.y, s4.z, s4.w};
            const bool whiten = s4.x != 1.0f || s4.y != 1.0f || s4.z != 1.0f || s4.w != 1.0f;  // (a division by one changes nothing, but takes a branch each)
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                float hv[4] = {acc[0][j], acc[1][j], acc[2][j], acc[3][j]};
                if (whiten) {
#pragma unroll
                    for (int r = 0; r < 4; ++r) {
                        hv[r] = QUERY ? __fmul_rn(acc[r][j], sk[r]) : __fdiv_rn(acc[r][j], sk[r]);
                        acc[r][j] = __fmul_rn(hv[r], sk[r]);  // w[k][j] = h_j[k] * s_k, the factor of P[k][:] in the reconstruction
                    }
                }
                store_keys<4>(hs + (size_t)(8 * kl + j) * D_C + 4 * h_chunk(rl), hv);
            }
            if (!QUERY) {
#pragma unroll
                for (int r = 0; r < 4; ++r) store_keys<8>(wsT + (size_t)(4 * rl + r) * KS + 8 * kl, acc[r]);
            }
        } else {
            // row k = u & 127, keys of half (u >> 7)
            for (int u = tid; u < (KB >= 2 ? 2 : 1) * D_C; u += NT) {
                const int k = u & 127, j0 = (u >> 7) * PER;
                float acc[PER];
#pragma unroll
                for (int j = 0; j < PER; ++j) acc[j] = 0.0f;
#pragma unroll KB <= 8 ? 32 : (KB == 16 ? 16 : 8)
                for (uint32_t i = 0; i < d; ++i)
                    axpy_keys<PER>(acc, a.pt[(size_t)i * D_C + k], buf + (size_t)i * KS + j0);
                const float sk = a.scale[k];
#pragma unroll
                for (int j = 0; j < PER; ++j) {
                    const float hv = QUERY ? __fmul_rn(acc[j], sk) : __fdiv_rn(acc[j], sk);
                    hs[(size_t)(j0 + j) * D_C + 4 * h_chunk(k >> 2) + (k & 3)] = hv;
                    // w[k][j] = h_j[k] * s_k, the factor the reconstruction multiplies P[k][:] by
                    acc[j] = __fmul_rn(hv, sk);
                }
                if (!QUERY) store_keys<PER>(wsT + (size_t)k * KS + j0, acc);
            }
        }
        __syncthreads();

        if (QUERY) {
            for (int e = tid; e < nk * D_C; e += NT)
                a.q_coarse[(base + e / D_C) * D_C + (e % D_C)] = hs[(e & ~(D_C - 1)) + 4 * h_chunk((e % D_C) >> 2) + (e & 3)];
            // (the sign-LSH input is the raw query)
        } else {
            // ---- quantise ---------------------------------
            for (int e = tid; e < (KB > 4 ? KB * 8 : 32); e += NT) {
                const int j = min(e >> 3, KB - 1);
                quantize_unit(hs + (size_t)j * D_C, a.codec, tl + (size_t)j * TILE_BYTES, e & 7, (e >> 3) < KB);
            }
            // (no barrier: the residual phase reads the keys and the reconstruction factors, which
            //  the barrier after the latent phase already covers, and does not touch the tiles)
            // ---- residual e = key - sum_k (h_k*s_k) * P[k][:]  (k outer, sequential): a thread owns
            //      column i for half of the keys ---------------------------------------------------
            constexpr int HALVES = KB >= 2 ? 2 : 1;
            // tiled: columns 4 ig .. +3 for keys 8 kg .. +7 (or five or six columns a thread, where fours would take the warps two rounds)
            if (KB == 32 && tiled && d > 128 && d <= 192) {
                if (d <= 160) residual_columns<5>(a, buf, wsT);
                else residual_columns<6>(a, buf, wsT);
            }
            for (uint32_t wt = warp; KB == 32 && tiled && !(d > 128 && d <= 192) && wt < (d + 31) / 32; wt += NT / 32) {
                const uint32_t ig = 8 * wt + (lane & 7), kg = lane >> 3;
                if (ig >= d / 4) continue;
                uint64_t acc2[4][4];
                zero_tile<4, 8>(acc2);
                const float4* mp = reinterpret_cast<const float4*>(a.p) + ig;
                const float* wr = wsT + 8 * kg;
#pragma unroll 8
                for (int k = 0; k < D_C; ++k)
                    outer_keys<4, 8>(acc2, __ldg(mp + (size_t)k * (d / 4)), wr + (size_t)k * KS, a.one);
                float acc[4][8];
                unpack_tile<4, 8>(acc2, acc);
#pragma unroll
                for (int r = 0; r < 4; ++r) {
                    float kv[8];
                    load_keys<8>(kv, buf + (size_t)(4 * ig + r) * KS + 8 * kg);
#pragma unroll
                    for (int j = 0; j < 8; ++j) acc[r][j] = __fsub_rn(kv[j], acc[r][j]);
                    store_keys<8>(buf + (size_t)(4 * ig + r) * KS + 8 * kg, acc[r]);
                }
            }
            for (uint32_t wi = tid; !(KB == 32 && tiled) && wi < HALVES * d; wi += NT) {
                const uint32_t i = wi % d, half = wi / d;
                float acc[PER];
#pragma unroll
                for (int j = 0; j < PER; ++j) acc[j] = 0.0f;
                const float* wr = wsT + half * PER;
#pragma unroll KB <= 8 ? 32 : (KB == 16 ? 16 : 8)
                for (int k = 0; k < D_C; ++k) axpy_keys<PER>(acc, a.p[(size_t)k * d + i], wr + (size_t)k * KS);
                float kv[PER];
                load_keys<PER>(kv, buf + (size_t)i * KS + half * PER);
#pragma unroll
                for (int j = 0; j < PER; ++j) acc[j] = __fsub_rn(kv[j], acc[j]);
                store_keys<PER>(buf + (size_t)i * KS + half * PER, acc);
            }
        }
        __syncthreads();

        // ---- sigma_E (f32, sequential over i) and tile metadata: the last warp (the others go on with the signs where no rotation
        //      changes the residual first) ---------------
        auto metadata = [&]() {
            const int j = tid - (NT - 32);
            if (QUERY || j < 0 || j >= nk) return;
            float ss = 0.0f;
#pragma unroll 8
            for (uint32_t i = 0; i < d; ++i) {
                const float x = buf[(size_t)i * KS + j];
                ss = __fadd_rn(ss, __fmul_rn(x, x));
            }
            const float sigma = __fsqrt_rn(__fdiv_rn(ss, (float)d));
            unsigned char* tile = tl + (size_t)j * TILE_BYTES;
            const uint32_t pos = a.positions ? a.positions[base + j] : a.position_base + (uint32_t)(base + j);
            *reinterpret_cast<float*>(tile + 100) = __fmul_rn(sigma, a.lambda_c);
            *reinterpret_cast<float*>(tile + 104) = sigma;
            *reinterpret_cast<uint32_t*>(tile + 108) = pos;
            *reinterpret_cast<uint32_t*>(tile + 112) = pos;
            const uint32_t head = a.heads ? a.heads[base + j] : 0u;
            uint32_t cflag = 0;
            if (a.codec == SLHA_CODEC_NF4) cflag = F_NF4;
            else if (a.codec == SLHA_CODEC_MIXED) cflag = F_MIXED;
            else if (a.codec == SLHA_CODEC_TQ3) cflag = F_TQ3;
            else if (a.codec == SLHA_CODEC_MIX3) cflag = F_MIX3;
            *reinterpret_cast<uint32_t*>(tile + 116) = head | (cflag << 16);
        };

        // ---- optional randomised Hadamard transform of buf ------------------
        if (a.diag) {
            metadata();
            if (!QUERY) __syncthreads();
            uint32_t at = 0, left = 31 - __clz(dp);
            for (; left >= 4; left -= 4, at += 4) {
                fwht_stages<KB, 4>(buf, dp, at, a.diag, a.fwht_inv);
                __syncthreads();
            }
            if (dp == 1) fwht_stages<KB, 0>(buf, dp, 0, a.diag, a.fwht_inv);
            if (left == 3) fwht_stages<KB, 3>(buf, dp, at, a.diag, a.fwht_inv);
            if (left == 2) fwht_stages<KB, 2>(buf, dp, at, a.diag, a.fwht_inv);
            if (left == 1) fwht_stages<KB, 1>(buf, dp, at, a.diag, a.fwht_inv);
            if (left || at == 0) __syncthreads();
        }

        // ---- sign-LSH ----------------------------------------------------------
        bool signs_done = false;
        if constexpr (KB >= 4) {
            if (a.zf) signs_done = signs_mma<KB>(a, buf, tl, reinterpret_cast<uint32_t*>(hs), (uint32_t)(D_C * (KB + KS)), [&]() { if (!a.diag) metadata(); });
            else if (!a.diag) metadata();
        } else if (!a.diag) {
            metadata();
        }
        if (!signs_done) __syncthreads();
        // every sum in the reference's order, tiled: hyperplanes 4 rg .. +3 for keys 8 kg .. +7
        if (signs_done) {
        } else if (KB == 32 && tiled) {
            for (int u = tid; u < 256; u += NT) {
                const int rg = u & 63, kg = u >> 6;
                uint64_t acc2[4][4];
                zero_tile<4, 8>(acc2);
                const float4* mp = reinterpret_cast<const float4*>(a.zt) + rg;
#pragma unroll 16
                for (uint32_t i = 0; i < dp; ++i)
                    outer_keys<4, 8>(acc2, __ldg(mp + (size_t)i * (D_S / 4)), buf + (size_t)i * KS + 8 * kg, a.one);
                float acc[4][8];
                unpack_tile<4, 8>(acc2, acc);
                // bit s of a key = (acc < 0); this thread holds bits 4 rg .. +3, eight lanes fill a 32-bit word
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    uint32_t v = (acc[0][j] < 0.0f ? 1u : 0u) | (acc[1][j] < 0.0f ? 2u : 0u) |
                                 (acc[2][j] < 0.0f ? 4u : 0u) | (acc[3][j] < 0.0f ? 8u : 0u);
                    v <<= 4 * (lane & 7);
                    v |= __shfl_xor_sync(0xFFFFFFFFu, v, 1);
                    v |= __shfl_xor_sync(0xFFFFFFFFu, v, 2);
                    v |= __shfl_xor_sync(0xFFFFFFFFu, v, 4);
                    const int key = 8 * kg + j, word = (rg >> 3);
                    if ((lane & 7) == 0) reinterpret_cast<uint32_t*>(tl + (size_t)key * TILE_BYTES + 64)[word] = v;
                }
            }
        } else {
            // a thread owns hyperplane s for all KB keys
            for (int s = tid; s < D_S; s += NT) {
                float acc[KB];
#pragma unroll
                for (int j = 0; j < KB; ++j) acc[j] = 0.0f;
                // (16 keys: loads of 16 steps in flight together, as in the two phases above: 7000 keys of 448 dimensions 182 us, with 8 steps 231)
#pragma unroll KB == 16 ? 16 : 8
                for (uint32_t i = 0; i < dp; ++i) axpy_keys<KB>(acc, a.zt[(size_t)i * D_S + s], buf + (size_t)i * KS);
#pragma unroll
                for (int j = 0; j < KB; ++j) {
                    const unsigned b = __ballot_sync(0xFFFFFFFFu, acc[j] < 0.0f);
                    if (lane == 0) reinterpret_cast<uint32_t*>(tl + (size_t)j * TILE_BYTES + 64)[s >> 5] = b;
                }
            }
        }
        __syncthreads();

        // ---- write tiles: 8 x 16 B per tile (query mode: their 32 sign bytes) -----
        if (QUERY) {
            for (int e = tid; e < nk * 8; e += NT)
                reinterpret_cast<uint32_t*>(a.q_sign)[base * 8 + e] = reinterpret_cast<const uint32_t*>(tl + (size_t)(e >> 3) * TILE_BYTES + 64)[e & 7];
        } else {
            for (int e = tid; e < nk * 8; e += NT) {
                const int j = e >> 3, c = e & 7;
                const uint64_t dst = a.slots ? a.slots[base + j] : base + j;
                reinterpret_cast<uint4*>(a.tiles + dst * TILE_BYTES)[c] =
                    reinterpret_cast<const uint4*>(tl + (size_t)j * TILE_BYTES)[c];
            }
        }
    }
}

// reconstruct (learned.rs:276-286) from the dequantised latent of one tile, and
// optionally the sign-sketch estimate of reconstruct_from_tile (learned.rs:290-322)
__global__ void decode_kernel(const unsigned char* tile, const float* p, const float* scale,
                              const float* z, uint32_t d, uint32_t d_pad, int with_residual,
                              float* out) {
    __shared__ float k[D_C];
    __shared__ float sgn[D_S];
    const uint32_t flags = *reinterpret_cast<const uint16_t*>(tile + 118);
    const float sc = *reinterpret_cast<const float*>(tile + 96);
    for (int dd = threadIdx.x; dd < D_C; dd += blockDim.x) {
        // tile.rs:133-255
        float v;
        auto alt = [&](int g) { return __fdiv_rn(__fmul_rn(sc, (float)tile[120 + g]), 255.0f); };
        auto grp = [&](int dim) { return __fmul_rn(sc, __fdiv_rn((float)tile[120 + dim / 16], 255.0f)); };
        auto code3 = [&](int off, int end, int ld) {
            const int bit = 3 * ld, byte = off + (bit >> 3), sh = bit & 7;
            const uint32_t lo = tile[byte], hi = (byte + 1 < end) ? ((uint32_t)tile[byte + 1] << 8) : 0u;
            return (int)(((lo | hi) >> sh) & 7u);
        };
        if (flags & F_MIXED) {
            if (dd < 8) v = __fmul_rn((float)((int)tile[dd] - 128), alt(0));
            else if (dd < 120) {
                const int ld = dd - 8;
                const uint32_t b = tile[8 + (ld >> 1)];
                v = __fmul_rn((float)((int)((ld & 1) ? (b >> 4) : (b & 15)) - 8), alt(1 + ld / 16));
            } else v = 0.0f;
        } else if (flags & F_TQ3) {
            float level = (float)code3(0, 48, dd) - 3.5f;
            if (!(flags & F_NOCORR)) level += ((tile[48 + (dd >> 3)] >> (dd & 7)) & 1) ? 0.25f : -0.25f;
            v = __fmul_rn(level, grp(dd));
        } else if (flags & F_MIX3) {
            if (dd < 8) v = __fmul_rn((float)((int)tile[dd] - 128), alt(0));
            else if (dd >= 120) v = 0.0f;
            else {
                const int ld = dd - 8;
                float level = (float)code3(8, 50, ld) - 3.5f;
                if (!(flags & F_NOCORR)) level += ((tile[50 + (ld >> 3)] >> (ld & 7)) & 1) ? 0.25f : -0.25f;
                v = __fmul_rn(level, alt(1 + ld / 16));
            }
        } else {
            const uint32_t b = tile[dd >> 1];
            const uint32_t nib = (dd & 1) ? (b >> 4) : (b & 15);
            const float cb[16] = {-1.0f,   -0.7075f, -0.5421f, -0.4165f, -0.3108f, -0.2158f,
                                  -0.1272f, -0.0421f, 0.0421f,  0.1272f,  0.2158f,  0.3108f,
                                  0.4165f,  0.5421f,  0.7075f,  1.0f};
            const float level = (flags & F_NF4) ? cb[nib] : (float)((int)nib - 8);
            v = __fmul_rn(level, grp(dd));
        }
        k[dd] = v;
    }
    const float sigma = *reinterpret_cast<const float*>(tile + 104);
    const float rs = __fdiv_rn(__fmul_rn(sigma, __fsqrt_rn(__fdiv_rn(3.14159265358979323846f, 2.0f))), (float)D_S);
    for (int s = threadIdx.x; s < D_S; s += blockDim.x) {
        const uint64_t w = reinterpret_cast<const uint64_t*>(tile + 64)[s >> 6];
        sgn[s] = ((w >> (s & 63)) & 1ull) ? -1.0f : 1.0f;
    }
    __syncthreads();
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < d; i += gridDim.x * blockDim.x) {
        float acc = 0.0f;
        for (int kk = 0; kk < D_C; ++kk)
            acc = __fadd_rn(acc, __fmul_rn(__fmul_rn(k[kk], scale[kk]), p[(size_t)kk * d + i]));
        if (with_residual)
            for (int s = 0; s < D_S; ++s)
                acc = __fadd_rn(acc, __fmul_rn(__fmul_rn(sgn[s], rs), z[(size_t)s * d_pad + i]));
        out[i] = acc;
    }
}

// Z in fp16 as the B operand of m16n8k16 MMAs (columns = hyperplanes), every row scaled to the norm SIGN_NORM: lane (g, t) of a group of 8
// hyperplanes holds k = 2 t, 2 t + 1 and 2 t + 8, 2 t + 9 of hyperplane g for two steps of 16 in one 16-byte word.  A CTA per
// row; stats[row] = (norm of what the rounding lost, norm of what it kept), negative where the row is not of ordinary size.
constexpr double SIGN_NORM = 16.0;
__global__ void __launch_bounds__(128) sign_fragments_kernel(const float* z, uint32_t dp, uint32_t* out, float2* stats) {
    __shared__ double part[4];
    const uint32_t s = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const auto total = [&](double v) {
        for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xFFFFFFFFu, v, o);
        __syncthreads();
        if (lane == 0) part[warp] = v;
        __syncthreads();
        return part[0] + part[1] + part[2] + part[3];
    };
    double n2 = 0.0, lost = 0.0, kept = 0.0;
    for (uint32_t i = threadIdx.x; i < dp; i += 128) n2 += (double)z[(size_t)s * dp + i] * z[(size_t)s * dp + i];
    n2 = total(n2);
    const bool usual = n2 >= 1e-12 && n2 <= 1e12;  // (false for NaN)
    const double scale = usual ? SIGN_NORM / sqrt(n2) : 0.0;
    for (uint32_t i = 2 * threadIdx.x; i < sign_rows(dp); i += 256) {
        uint32_t word = 0;
        for (uint32_t h = 0; h < 2; ++h) {
            const double x = i + h < dp && usual ? z[(size_t)s * dp + i + h] * scale : 0.0;
            const __half r = __float2half_rn((float)x);
            const double k = (double)__half2float(r), l = k - x;
            kept += k * k;
            lost += l * l;
            word |= (uint32_t)__half_as_ushort(r) << (16 * h);
        }
        out[((i / 32 * 32 + s / 8) * 32 + 4 * (s % 8) + i / 2 % 4) * 4 + i / 8 % 4] = word;
    }
    lost = total(lost);
    kept = total(kept);
    if (threadIdx.x == 0) stats[s] = usual ? make_float2((float)sqrt(lost), (float)sqrt(kept)) : make_float2(-1.0f, -1.0f);
}

__global__ void __launch_bounds__(256) transpose_kernel(const float* in, float* out, uint64_t rows, uint64_t cols) {
    for (uint64_t i = (uint64_t)blockIdx.x * 256 + threadIdx.x; i < rows * cols; i += (uint64_t)gridDim.x * 256) out[i] = in[i % rows * cols + i / rows];
}

size_t encode_smem(uint32_t d_pad, int kb) {
    const size_t ks = (size_t)enc_row_stride(kb);
    return (((d_pad * ks + 3) & ~size_t(3)) + (size_t)kb * D_C + ks * D_C) * 4 + (size_t)kb * TILE_BYTES;
}

Status fill_args(const Model* m, size_t n, EncodeArgs& a, int* kb_out) {
    a.d = (uint32_t)m->d;
    a.d_pad = (uint32_t)m->d_pad;
    a.p = m->d_p;
    a.pt = m->d_pt;
    a.scale = m->d_scale;
    a.zt = m->d_zt;
    a.z = m->d_z;
    a.z_guard = m->z_guard;
    a.z_norm = m->z_norm;
    a.diag = m->d_diag;
    a.fwht_inv = 1.0f / sqrtf((float)m->d_pad);
    a.one = 0x3F8000003F800000ull;
    a.lambda_c = sqrtf(3.14159265358979323846f / (2.0f * (float)D_S));
    // 32 keys per CTA pass up to 100 KB of shared memory (d_pad <= 440: 20 011 keys of 440 dimensions 411 us, with 16 keys 530), else fewer
    int kb = 32;
    while (kb > 1 && encode_smem(a.d_pad, kb) > (kb == 32 ? 100 : 200) * 1024) kb >>= 1;
    if (encode_smem(a.d_pad, kb) > 200 * 1024)
        return Status(SLHA_ERR_DIMENSION, "model dimension too large for the encode kernel");
    // The 4 x 8 register tiles, which make 32 keys pay, need d % 4 == 0.  Without them 16 keys are faster where the signs are summed in order too
    // (2400 keys of 258 dimensions 73 us, with 32 keys 117; 60 000: 930, 910) and up to two waves of their CTAs (9000 keys of 202 dimensions 92, 115;
    // 12 000: 131, 117).
    const uint64_t sms = (uint64_t)sm_count(m->device);
    if (kb == 32 && m->d % 4 != 0 && (!m->d_zf || n <= 16 * 2 * 2 * sms)) kb = 16;
    // Few keys: the narrowest CTA of at least 4 keys whose CTAs are all on the GPU at once, one (4 keys) or two (8, 16) an SM.  Measured (us per call,
    // float32, at 592 / 1184 / 2368 / 4736 keys): d = 128: 4 keys 14 / 25 / 45 / 84, 8: 14 / 15 / 19 / 36, 16: 19 / 19 / 20 / 27, 32: 33 / 30 / 30 / 31;
    // d = 320: 4: 30 / 58 / 113 / 224, 8: 36 / 36 / 52 / 102, 16: 59 / 59 / 59 / 84, 32: 89 / 88 / 89 / 89.  With the next width from one CTA an SM on, 2400 keys
    // of 288 dimensions took 89 us instead of 78, 1800 queries of 512 dimensions 85 instead of 54.
    while (kb > 4 && n <= (uint64_t)(kb / 2 * enc_ctas(kb / 2)) * sms) kb >>= 1;
    *kb_out = kb;
    a.kb = kb;
    // (the sign phase works in the space of h and the reconstruction factors)
    a.zf = kb >= 4 && sign_words(a.d_pad, kb) <= (uint32_t)(D_C * (kb + enc_row_stride(kb))) ? m->d_zf : nullptr;
    return Status();
}

template <bool QUERY, int KB>
Status run_encode_kb(Ctx* c, EncodeArgs& a) {
    const size_t smem = encode_smem(a.d_pad, KB);
    const uint64_t groups = (a.n + KB - 1) / KB;
    static thread_local bool configured[16] = {false};  // the attribute is per device
    if (!configured[c->device & 15]) {
        SLHA_CUDA(cudaFuncSetAttribute(encode_kernel<QUERY, KB>, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024));
        configured[c->device & 15] = true;
    }
    // far more CTAs than fit at once (592 are resident at head dimension 128): the hardware hands
    // out a CTA whenever one finishes, which balances the tail and keeps the CTAs sharing an SM in
    // different phases, so that the arithmetic of one covers the loads, quantisation and barriers
    // of the others.  (One resident wave measured 182 M keys/s, 8 CTAs per SM 191, one CTA per pass 199, when the signs were summed in order.)
    const uint32_t grid = (uint32_t)std::min<uint64_t>(groups, 148ull * 64);
    SLHA_CUDA(launch_behind(encode_kernel<QUERY, KB>, dim3(grid), dim3(enc_threads(KB)), smem, c->stream, a));
    count_launch();
    return Status();
}

template <bool QUERY>
Status run_encode(Ctx* c, EncodeArgs& a) {
    switch (a.kb) {
        case 32: return run_encode_kb<QUERY, 32>(c, a);
        case 16: return run_encode_kb<QUERY, 16>(c, a);
        case 8: return run_encode_kb<QUERY, 8>(c, a);
        case 4: return run_encode_kb<QUERY, 4>(c, a);
        case 2: return run_encode_kb<QUERY, 2>(c, a);
        default: return run_encode_kb<QUERY, 1>(c, a);
    }
}

}  // namespace

// No fragments (every sign from its exact sum) where the error bound of signs_mma does not hold: more than 256 dimensions, or rows far
// from ordinary size.
Status build_model_arrays(Ctx* c, Model* m, uint4* d_zf, void* d_stats) {
    const auto grid = [](size_t n) { return (uint32_t)std::min<size_t>((n + 255) / 256, 1184); };
    transpose_kernel<<<grid(D_C * m->d), 256, 0, c->stream>>>(m->d_p, m->d_pt, D_C, m->d);
    transpose_kernel<<<grid(D_S * m->d_pad), 256, 0, c->stream>>>(m->d_z, m->d_zt, D_S, m->d_pad);
    count_launch(2);
    SLHA_CUDA(cudaGetLastError());
    if (m->d_pad > 256) return Status();
    float2 stats[D_S];
    sign_fragments_kernel<<<D_S, 128, 0, c->stream>>>(m->d_z, (uint32_t)m->d_pad, reinterpret_cast<uint32_t*>(d_zf), static_cast<float2*>(d_stats));
    count_launch();
    SLHA_CUDA(cudaGetLastError());
    SLHA_CUDA(cudaMemcpyAsync(stats, d_stats, sizeof stats, cudaMemcpyDeviceToHost, c->stream));
    SLHA_CUDA(cudaStreamSynchronize(c->stream));
    float lost = 0.0f, kept = 0.0f;
    for (const float2& r : stats) {
        if (!(r.y > 0.0f)) return Status();
        lost = std::max(lost, r.x);
        kept = std::max(kept, r.y);
    }
    // MMA accumulation and the reference's own sum: 2^-13.9 + 2^-16 of the norms' product; 2e-4 for the rounding of the bound itself
    m->z_guard = (float)(1.0002 * (lost + (1.0 / 15286.0 + 1.0 / 65536.0) * SIGN_NORM));
    m->z_norm = (float)(1.0002 * kept);
    m->d_zf = d_zf;
    return Status();
}

Status launch_encode(Ctx* c, const Model* m, const void* d_keys, int key_dtype, size_t n,
                     const uint32_t* d_positions, uint32_t position_base, const uint16_t* d_heads,
                     int codec, SciRustSlhaTile* d_tiles, const uint32_t* d_slots) {
    if (n == 0) return Status();
    EncodeArgs a{};
    int kb;
    SLHA_TRY(fill_args(m, n, a, &kb));
    a.keys = d_keys;
    a.key_dtype = key_dtype;
    a.n = n;
    a.positions = d_positions;
    a.position_base = position_base;
    a.heads = d_heads;
    a.codec = codec;
    a.tiles = reinterpret_cast<unsigned char*>(d_tiles);
    a.slots = d_slots;
    return run_encode<false>(c, a);
}

Status launch_prepare_queries(Ctx* c, const Model* m, const float* d_q, size_t nq,
                              float* d_q_coarse, uint64_t* d_q_sign) {
    if (nq == 0) return Status();
    EncodeArgs a{};
    int kb;
    SLHA_TRY(fill_args(m, nq, a, &kb));
    a.keys = d_q;
    a.key_dtype = SLHA_B200_F32;
    a.n = nq;
    a.q_coarse = d_q_coarse;
    a.q_sign = d_q_sign;
    return run_encode<true>(c, a);
}

Status launch_decode(Ctx* c, const Model* m, const SciRustSlhaTile* d_tile, float* d_out,
                     bool with_residual) {
    const uint32_t d = (uint32_t)m->d;
    decode_kernel<<<(d + 127) / 128, 128, 0, c->stream>>>(
        reinterpret_cast<const unsigned char*>(d_tile), m->d_p, m->d_scale, m->d_z, d,
        (uint32_t)m->d_pad, with_residual && !m->rht, d_out);
    count_launch();
    SLHA_CUDA(cudaGetLastError());
    return Status();
}

}  // namespace slha
