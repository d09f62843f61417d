// Wide scoring: many queries per KV head (16 or more: batched decode, prompt chunks).  Included by score.cu after
// score_tile.cuh, whose tile decode it shares.
//
// A CTA takes a block of 128 tiles through tcgen05.mma against up to 64 query rows.  Both terms of eq. 2.3 are contractions here:
//   coarse  A (128 tiles x 128 dims, exact fp16 levels times scale bytes, + 16 K slots for the 3-bit kinds) x the queries, scaled
//           to one size, as fp16 hi, then lo (22 bits or more), accumulated into the same 64 columns,
//   sign    A (128 tiles x 256 residual bits, a bit in place as an fp16 subnormal 2^-24 .. 2^-17) x the queries' signs as
//           +-2^10 .. 2^3: exact integers times 2^-14, from which 256 - 2 hamming = U - 2^15 D, U the sum of the query's signs.
// The 64 Hamming distances of a tile cost 8 XOR + 8 POPC each on the CUDA cores (POPC at a quarter of the issue rate), about 1100
// instructions per tile; spreading the 256 bits costs 136.  The A operand lives in TMEM: thread (tile row, quarter) writes a
// quarter of its tile's row -- quarters 0 and 1 the latent, 2 and 3 the bits -- and after the MMAs finishes 16 of the
// tile's 64 scores.  The MMAs of block b + 1 run while the scores of block b are finished (two accumulators).
//
// MIX3 has three coarse accumulators and reads them back before the next block's MMAs are issued, into the same columns: a
// chain of nine steps in one accumulator leaves 1.5e-7 relative error against 64 bits, where the generic kernel that scored
// these tiles before has 0.9e-7.  (The other kinds' chain of eight is the one they have always had here.)
#pragma once

namespace slha {
namespace {

#ifdef SLHA_STREAM_PROBE
#define WPROBE_DECL unsigned long long wp_t = probe_now(), wp_acc[12] = {0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0}
#define WPROBE_LAP(i) do { const unsigned long long n_ = probe_now(); wp_acc[i] += n_ - wp_t; wp_t = n_; } while (0)
#define WPROBE_OUT(base, cnt) do { if ((threadIdx.x & 31) == 0) for (int i_ = 0; i_ < cnt; ++i_) g_wide_probe[blockIdx.x][base + i_] = wp_acc[i_]; } while (0)
__device__ unsigned long long g_wide_probe[160][24];
#else
#define WPROBE_DECL
#define WPROBE_LAP(i)
#define WPROBE_OUT(base, cnt)
#endif
constexpr int WIDE_M = 128;                         // tiles per block
constexpr int WIDE_NQ = 64;                         // query rows per work item
constexpr int WIDE_THREADS = 512;
constexpr int WIDE_SLAB = WIDE_NQ * 128;            // 64 K slots of B: 64 rows x 128 bytes
constexpr int WIDE_B_BYTES = 3 * WIDE_SLAB;         // one part (hi or lo): K = 64 + 64 + 16
constexpr int WIDE_S_BYTES = 4 * WIDE_SLAB;         // signs: K = 256
constexpr int WIDE_RAW = 128 * ST_ROW;              // one staged block
constexpr int WIDE_RING = 3;
constexpr int WIDE_Q_BYTES = WIDE_NQ * D_C * 4;     // the item's queries in fp32 (item set-up only)
constexpr int WIDE_OUT_BYTES = WIDE_NQ * 128 * 4;   // dense: a block's scores on their way out, a row of them per query; two of these, over the queries
constexpr int WIDE_TAIL = 2048 + 256 + 512 + 512 + 512 + 64 + 2048;  // sign words, threshold keys, sign sums and scales, mappings (2), barrier + flags, minima and maxima / row offsets
constexpr uint32_t WIDE_A_SIGN = 128, WIDE_D = 256;                   // TMEM columns: A latent 0..71, A signs 128..255, accumulators 256.. and 384..
constexpr size_t wide_smem_bytes(bool dense) {
    return 1024 + 2 * WIDE_B_BYTES + WIDE_S_BYTES + (dense ? 2 * WIDE_OUT_BYTES : WIDE_Q_BYTES) + WIDE_RING * WIDE_RAW + WIDE_TAIL;
}

// Threshold refresh of NR consecutive query rows by one warp (all loads of the NR histograms in flight
// together): the lower edge of the highest bucket whose count from the top reaches k, minus half a
// bucket, is a proven bound (see stream_refresh_threshold).
template <int NR>
__device__ __forceinline__ void wide_refresh_rows(const ScoreArgs& a, uint32_t Q0, int nrows, const float2* rng, uint32_t* pvh, int lane) {
    uint32_t c[NR][8];
    unsigned long long seen = 0ull;
    if (lane < nrows) seen = *reinterpret_cast<volatile unsigned long long*>(a.gpivot + Q0 + lane);
#pragma unroll
    for (int r = 0; r < NR; ++r) {
#pragma unroll
        for (int j = 0; j < 8; ++j) c[r][j] = 0u;
        if (r < nrows && rng[r].y != 0.0f) {  // (uniform)
            const uint32_t* hq = a.ghist + (size_t)(Q0 + r) * 256 + 248 - 8 * lane;  // buckets 255-8l .. 248-8l (descending)
            asm volatile("ld.volatile.global.v4.u32 {%0,%1,%2,%3}, [%4];\n" : "=r"(c[r][7]), "=r"(c[r][6]), "=r"(c[r][5]), "=r"(c[r][4]) : "l"(hq));
            asm volatile("ld.volatile.global.v4.u32 {%0,%1,%2,%3}, [%4];\n" : "=r"(c[r][3]), "=r"(c[r][2]), "=r"(c[r][1]), "=r"(c[r][0]) : "l"(hq + 4));
        }
    }
#pragma unroll
    for (int r = 0; r < NR; ++r) {
        if (r >= nrows) break;  // (uniform)
        uint32_t best = (uint32_t)(__shfl_sync(0xFFFFFFFFu, seen, r) >> 32);
        const float2 rr = rng[r];
        if (rr.y != 0.0f) {
            uint32_t tot = 0;
#pragma unroll
            for (int j = 0; j < 8; ++j) tot += c[r][j];
            uint32_t incl = tot;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, incl, o);
                if (lane >= o) incl += y;
            }
            const unsigned ok = __ballot_sync(0xFFFFFFFFu, incl >= a.k);
            uint32_t ek = 0;
            if (ok != 0u && lane == __ffs(ok) - 1) {
                uint32_t run = incl - tot;
                int b = 0;
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    if (run + c[r][j] >= a.k) { b = 255 - 8 * lane - j; break; }
                    run += c[r][j];
                }
                if (b >= 1) {
                    const uint32_t e = score_key(rr.x + ((float)b - 0.5f) / rr.y);
                    ek = e > 8u ? e - 8u : 0u;
                }
            }
            ek = __reduce_max_sync(0xFFFFFFFFu, ek);
            if (ek > best) {
                best = ek;
                if (lane == 0) atomicMax(a.gpivot + Q0 + r, (unsigned long long)ek << 32);
            }
        }
        if (lane == 0 && best > pvh[r]) pvh[r] = best;
    }
}


// Four words of residual bits -> 64 columns: column 16 w + j holds bits j and j + 16 of word w as 2^-24 2^(j & 7).
__device__ __forceinline__ void wide_sign_words(const uint4& x, uint32_t ta) {
    const uint32_t w[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        uint32_t o[16];
#pragma unroll
        for (int j = 0; j < 16; ++j) o[j] = (j < 8 ? w[i] : w[i] >> 8) & (0x00010001u << (j & 7));
        st_tmem_st16(ta + 16u * i, o);
    }
}

// Dense calls: an item's rows go to the four-row kernel's pass.  (CTAs that share the rows may hand them on for different reasons: the pass sees them all, whichever came last.)
__device__ __forceinline__ void wide_hand_on(const ScoreArgs& a, const WorkItem& it, uint32_t as) {
    if (threadIdx.x < it.n_queries) atomicOr(a.handoff + it.query_begin + threadIdx.x, as);
    if (threadIdx.x == 0) *a.handoff_any = 1u;
}
// what an item that wide_body did not score is handed on as: it is NF4 where its first tile is
__device__ __forceinline__ uint32_t wide_hand_as(const ScoreArgs& a, const WorkItem& it) {
    return item_kind(first_tile_flags(a, it), false) == 0 ? 1u : a.handoff_as;
}

// KIND as in score_stream_kernel (1 mixed 8/4, 2 TQ3, 3 INT4 / MX-INT4, 4 MIX3).  DENSE: every score is written to its row of
// a.scores (row q starts at a.row_offset[q]) instead of going through the top-k filter: the dense scores of a layer for
// callers that replace attention logits (the llama.cpp shim).
// The CTA's work items from first_item on.
template <int KIND, bool DENSE>
__device__ __forceinline__ void wide_body(const ScoreArgs& a, unsigned char* smem_raw, uint32_t first_item) {
    constexpr int ACCS = KIND == 4 ? 3 : 1;                            // coarse accumulators
    constexpr uint32_t SIGN_AT = 64u * ACCS, FLIP = ACCS == 1 ? 128u : 0u;  // the signs' columns behind them; the second set of both
    // shared layout (1024-byte aligned base): B hi | B lo | signs | raw ring | queries, later (dense) scores on their way out | tail
    const uint32_t base_s = ((uint32_t)__cvta_generic_to_shared(smem_raw) + 1023u) & ~1023u;
    unsigned char* base = smem_raw + (base_s - (uint32_t)__cvta_generic_to_shared(smem_raw));
    constexpr uint32_t S_OFF = 2 * WIDE_B_BYTES, RAW_OFF = S_OFF + WIDE_S_BYTES, Q_OFF = RAW_OFF + WIDE_RING * WIDE_RAW, TAIL_OFF = Q_OFF + (DENSE ? 2 * WIDE_OUT_BYTES : WIDE_Q_BYTES);
    const uint32_t B_s = base_s, S_s = base_s + S_OFF, raw_s = base_s + RAW_OFF, out_s = base_s + Q_OFF;
    float* qf = reinterpret_cast<float*>(base + Q_OFF);             // [64][128]
    unsigned char* tail = base + TAIL_OFF;
    uint32_t* qs_w = reinterpret_cast<uint32_t*>(tail);            // [64][8]
    uint32_t* pvh = qs_w + 512;                                     // [64] score word of the row's threshold
    float* uq = reinterpret_cast<float*>(pvh + 64);                 // [64] sums of the rows' signs, [64] inverses of the rows' scales times the unit of A
    float2* rng = reinterpret_cast<float2*>(uq + 128);                                          // [64] (smin, inv)
    float2* rmap = rng + 64;                                        // [64] (-smin inv, inv)
    uint32_t* ctl = reinterpret_cast<uint32_t*>(rmap + 64);         // mbarrier (8 bytes), [4] TMEM base, [5] error flag, [6] bail
    float2* colmm = reinterpret_cast<float2*>(ctl + 16);            // [4][64] per tile quarter: (min, max) score of a column
    unsigned long long* roff = reinterpret_cast<unsigned long long*>(colmm);  // DENSE: [64] where the item's rows start in a.scores
    const uint32_t bar_s = base_s + TAIL_OFF + 2048 + 256 + 512 + 512 + 512;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, qt = warp & 3, ch = warp >> 2;
    const int uw = uniform_warp();
    const bool elected = elect_one(), leader = elected && uw == 0;  // the thread that issues the MMAs

    if (tid == 0) {
        mbar_init(bar_s, 1);
        ctl[5] = 0u;
        ctl[6] = 0u;
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(bar_s + 16), "r"(512u) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    const uint32_t tmem = *reinterpret_cast<volatile uint32_t*>(ctl + 4);
    const uint32_t tlane = tmem + ((uint32_t)(32 * qt) << 16);  // this warp's lanes: tile rows 32 qt .. + 31
    uint32_t magic;
    asm volatile("mov.u32 %0, 0x64006400;\n" : "=r"(magic));
    const uint32_t row_off = (uint32_t)(32 * qt + lane) * ST_ROW;
    WPROBE_DECL;
    uint32_t phase = 0;
    bool stop = false;

    const uint32_t item_end = a.cta_begin[blockIdx.x + 1];
    for (uint32_t item_id = first_item; item_id < item_end && !stop; ++item_id) {
        const WorkItem it = a.items[item_id];
        const int nq = (int)it.n_queries;
        const uint32_t n = it.n_tiles, idesc = tc_idesc(((uint32_t)nq + 15u) & ~15u);
        __syncthreads();  // the previous item's MMAs and scores are finished: B, thresholds and sign words may change
        auto fetch = [&](uint32_t b) {  // two 16-byte chunks per thread
            const uint32_t t0 = b * WIDE_M, dst = raw_s + (b % WIDE_RING) * WIDE_RAW;
            const unsigned char* src = a.tiles + (it.tile_begin + t0) * TILE_BYTES;
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const uint32_t chunk = (uint32_t)i * WIDE_THREADS + (uint32_t)tid, row = chunk >> 3;
                const bool in = t0 + row < n;
                cp_async16_s<0, 0>(dst + row * ST_ROW + (chunk & 7u) * 16u, in ? src + (size_t)chunk * 16 : a.tiles, in ? 16 : 0);
            }
            cp_async_commit();
        };
        const uint32_t all_blocks = (n + WIDE_M - 1) / WIDE_M;
        if (all_blocks) fetch(0);
        constexpr bool HEAD = KIND == 1 || KIND == 4, EXTRA = KIND == 2 || KIND == 4;
        bool big = false;  // a query beyond the fp16 split
        {   // four rows a warp, scaled on their way into shared memory (the mixed layouts have no levels behind dim 119)
            constexpr int ROWS = WIDE_NQ / (WIDE_THREADS / 32);
            float4 x[ROWS];
#pragma unroll
            for (int i = 0; i < ROWS; ++i) {
                const int r = ROWS * warp + i;
                x[i] = r < nq && !(HEAD && lane >= 30) ? load_q4(a.q_coarse + (size_t)(it.query_begin + r) * D_C + 4 * lane) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            }
#pragma unroll
            for (int i = 0; i < ROWS; ++i) {
                const int r = ROWS * warp + i;
                const uint32_t largest = __reduce_max_sync(0xFFFFFFFFu, max(max(abs_bits(x[i].x), abs_bits(x[i].y)), max(abs_bits(x[i].z), abs_bits(x[i].w))));
                big |= largest >= SPLIT_MOST;
                const float2 f = split_scale(largest, 14);
                reinterpret_cast<float4*>(qf)[32 * r + lane] = make_float4(x[i].x * f.x, x[i].y * f.x, x[i].z * f.x, x[i].w * f.x);
                if (lane == 0) uq[64 + r] = f.y * (EXTRA ? 32768.0f : 65536.0f);
            }
        }
        qs_w[tid] = (tid >> 3) < nq ? a.q_sign[(size_t)(it.query_begin + (tid >> 3)) * 8 + (tid & 7)] : 0u;
        if (DENSE && tid < WIDE_NQ) roff[tid] = tid >= nq || a.blocked ? 0ull : a.row_offset[it.query_begin + tid];
        if (!DENSE && tid < WIDE_NQ) {
            const bool have = tid < nq;
            const unsigned long long pv = have ? *reinterpret_cast<volatile unsigned long long*>(a.gpivot + it.query_begin + tid) : ~0ull;
            pvh[tid] = (uint32_t)(pv >> 32);
            const unsigned long long pr = have ? *reinterpret_cast<volatile unsigned long long*>(a.grange + it.query_begin + tid) : 0ull;
            rng[tid] = make_float2(__uint_as_float((uint32_t)pr), __uint_as_float((uint32_t)(pr >> 32)));
            rmap[tid] = make_float2(-rng[tid].x * rng[tid].y, rng[tid].y);
        }
        __syncthreads();
        constexpr uint32_t SUMS = WIDE_NQ * D_C;  // behind the queries: [64][8] a sixteenth of their sums over the groups (a group a thread; MIX3: group g is dims 16 g - 8 ..)
        if (EXTRA && DENSE) {
            const int r = tid >> 3, g = tid & 7;
            const float* qg = qf + r * D_C + (KIND == 4 ? 16 * g - 8 : 16 * g);
            float s = 0.0f;
            if (KIND == 2 || g)
#pragma unroll
                for (int d = 0; d < 16; d += 4) {
                    const float4 x = *reinterpret_cast<const float4*>(qg + d);
                    s = s + x.x + x.y + x.z + x.w;
                }
            qf[SUMS + tid] = 0.0625f * s;
            __syncthreads();
        }
        // B rows = queries, K-major, 128-byte swizzle (16-byte chunk i of row r at chunk i ^ (r & 7) of its line); the order of the
        // k slots is that of nib_word / head_word / scale_pair
        for (int u = tid; u < WIDE_NQ * 18; u += WIDE_THREADS) {
            const int r = u / 18, i = u % 18;
            const float* q = qf + r * D_C;
            float v[8];
            if (HEAD && i < 2) {
                const float4 x = *reinterpret_cast<const float4*>(q + 4 * i);
                v[0] = x.x; v[1] = x.y; v[2] = x.z; v[3] = x.w; v[4] = x.x; v[5] = x.y; v[6] = x.z; v[7] = x.w;
            } else if (i < 16) {
                const int d0 = HEAD ? 8 * (i - 1) : 8 * i;
                const float4 x = *reinterpret_cast<const float4*>(q + d0), y = *reinterpret_cast<const float4*>(q + d0 + 4);
                v[0] = x.x; v[1] = y.x; v[2] = x.y; v[3] = y.y; v[4] = x.z; v[5] = y.z; v[6] = x.w; v[7] = y.w;
            } else {
#pragma unroll
                for (int g = 0; g < 8; ++g) {
                    v[g] = i == 16 && EXTRA && DENSE ? qf[SUMS + 8 * r + g] : 0.0f;
                    if (i == 16 && EXTRA && !DENSE && (KIND == 2 || g)) {
                        const float* qg = q + (KIND == 4 ? 16 * g - 8 : 16 * g);
                        float s = 0.0f;
                        for (int d = 0; d < 16; d += 4) {
                            const float4 x = *reinterpret_cast<const float4*>(qg + d);
                            s = s + x.x + x.y + x.z + x.w;
                        }
                        v[g] = 0.0625f * s;
                    }
                }
            }
            uint32_t hi[4], lo[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                hi[j] = pack_half2(v[2 * j], v[2 * j + 1]);
                lo[j] = pack_half2(half_residual(v[2 * j]), half_residual(v[2 * j + 1]));
            }
            const uint32_t at = B_s + (uint32_t)(i >> 3) * WIDE_SLAB + (uint32_t)r * 128u + ((((uint32_t)i & 7u) ^ ((uint32_t)r & 7u)) << 4);
            sts_v4(at, hi[0], hi[1], hi[2], hi[3]);
            sts_v4(at + WIDE_B_BYTES, lo[0], lo[1], lo[2], lo[3]);
        }
        for (int u = tid; u < WIDE_NQ * 32; u += WIDE_THREADS) {
            const int r = u >> 5, i = u & 31, j0 = 4 * (i & 3);  // chunk i: columns j0 .. j0 + 3 of word i / 4
            const uint32_t w = qs_w[8 * r + (i >> 2)];
            uint32_t o[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const uint32_t mag = 0x6400u - (uint32_t)((j0 + j) & 7) * 0x400u;  // 2^(10 - (j & 7)), negative for a set bit
                o[j] = (mag | ((w >> (j0 + j) & 1u) << 15)) | ((mag | ((w >> (j0 + j + 16) & 1u) << 15)) << 16);
            }
            sts_v4(S_s + (uint32_t)(i >> 3) * WIDE_SLAB + (uint32_t)r * 128u + ((((uint32_t)i & 7u) ^ ((uint32_t)r & 7u)) << 4), o[0], o[1], o[2], o[3]);
        }
        if (tid < WIDE_NQ) {
            int c = 0;
            for (int w = 0; w < 8; ++w) c += __popc(qs_w[8 * tid + w]);
            uq[tid] = (float)(256 - 2 * c);
        }
        if (big) ctl[6] = 1u;
        asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");  // B was written with ordinary stores, the MMA reads it through the async proxy
        const bool too_big = __syncthreads_or(big) != 0;  // (from the vote: the flag word may already be raised for a tile)
        const bool need_map = __syncthreads_or(!DENSE && tid < nq && rng[tid].y == 0.0f) != 0;  // a row of the item has no bucket mapping yet
        const uint32_t blocks = too_big ? 0u : all_blocks;
        WPROBE_LAP(0);  // item set-up

        // this thread's quarter of its tile's row of A
        auto stage = [&](uint32_t b) {
            const uint32_t row = raw_s + (b % WIDE_RING) * WIDE_RAW + row_off;
            if (ch < 2) {
                const uint4 x = lds_v4<112>(row);
                const uint32_t flags = x.y >> 16;
                if (ch == 0) {
                    st_fold_row<KIND, 0, 2>(row, tlane, flags, x.z, x.w, magic);
                    if (b * WIDE_M + (uint32_t)(32 * qt + lane) < n && st_alien(KIND, flags)) ctl[6] = 1u;  // the item's rows go to the generic kernel
                } else {
                    st_fold_row<KIND, 2, 4>(row, tlane, flags, x.z, x.w, magic);
                }
            } else if (ch == 2) {
                wide_sign_words(lds_v4<64>(row), tlane + WIDE_A_SIGN);
            } else {
                wide_sign_words(lds_v4<80>(row), tlane + WIDE_A_SIGN + 64u);
            }
            asm volatile("tcgen05.wait::st.sync.aligned;\n" ::: "memory");
            asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
            // (only the issuing warp waits for the others: a barrier of its own, since the others may be at the next one by then)
            if (uw == 0) asm volatile("bar.sync 3, 512;\n" ::: "memory");
            else asm volatile("bar.arrive 3, 512;\n" ::: "memory");
            if (leader) {
                asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
                const uint32_t dt = tmem + WIDE_D + FLIP * (b & 1u);
                // Coarse and sign steps alternate (MMAs that add into the same columns wait for one another).  Coarse: the queries' lo
                // parts first, so that only the hi steps round at the size of the score.
                constexpr int KS = EXTRA ? 9 : 8;
#pragma unroll
                for (int i = 0; i < 2 * KS; ++i) {
                    const int ks = i % KS;
                    st_mma(dt + 64u * (ks % ACCS), tmem + 8u * ks, tc_desc(B_s + (i < KS ? WIDE_B_BYTES : 0) + (uint32_t)(ks >> 2) * WIDE_SLAB + 32u * (ks & 3)),
                           i >= ACCS ? 1u : 0u, idesc);
                    if (i < 16) st_mma(dt + SIGN_AT, tmem + WIDE_A_SIGN + 8u * i, tc_desc(S_s + (uint32_t)(i >> 2) * WIDE_SLAB + 32u * (i & 3)), i ? 1u : 0u, idesc);
                }
                tc_commit(bar_s);
            }
            __syncwarp();
        };
        // A block's scores of a plan of whole rows, where they lie together, leave shared memory by one bulk copy (512 rows of 16 384 TQ3 tiles, k = 256:
        // 50.9 us a call with a store a score, 48.1 with these; a copy for each of 64 rows was no faster).
        auto send = [&](uint32_t b) {
            if (tid != WIDE_THREADS - 32) return;
            float* const to = a.scores + it.list_begin + (size_t)((it.index_base >> 7) + b) * it.pad;
            asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;\ncp.async.bulk.commit_group;\n" ::"l"(to), "r"(out_s + (b & 1u) * WIDE_OUT_BYTES),
                         "r"((uint32_t)nq * 512u) : "memory");
        };
        const int r = 32 * qt + lane;
        const bool cols = 16 * ch < nq;  // this warp has query columns in this item
        const uint32_t Q0 = it.query_begin + 16u * (uint32_t)ch;
        if (blocks) {
            cp_async_wait<0>();
            asm volatile("bar.sync 2, 512;\n" ::: "memory");
            if (blocks > 1) fetch(1);
            stage(0);
            WPROBE_LAP(3);
        }
        for (uint32_t b = 0; b < blocks; ++b) {
            // the accumulators of block b are finished (and its A operand may be overwritten); a wait that ran out anywhere
            // ends the item for all warps together, because barriers follow
            const bool ok = mbar_wait(bar_s, phase);
            phase ^= 1u;
            cp_async_wait<0>();  // this thread's copies of block b + 1
            const bool turned = DENSE && a.blocked;
            if (turned && tid == WIDE_THREADS - 32) asm volatile("cp.async.bulk.wait_group.read 0;\n" ::: "memory");  // (the copy out of the buffer that this block fills)
            if (role_any(1, WIDE_THREADS, !ok)) { stop = true; break; }
            if (turned && b) send(b - 1);
            asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
            WPROBE_LAP(1);  // wait for the accumulators
            if (b + 2 < blocks) fetch(b + 2);
            if (ACCS == 1 && b + 1 < blocks) stage(b + 1);
            WPROBE_LAP(3);  // stage
            const uint32_t t0 = b * WIDE_M + (uint32_t)r;
            const uint32_t row = raw_s + (b % WIDE_RING) * WIDE_RAW + row_off;
            const uint2 meta = lds_v2<96>(row);
            const uint32_t flags = lds_u16<118>(row);
            const bool live = t0 < n;
            const float lam = (flags & F_WARM) ? 0.0f : __uint_as_float(meta.y);
            const float su = __uint_as_float(meta.x) * (1.0f / 255.0f);
            float sc[16];
            if (cols) {
                const uint32_t dt = tlane + WIDE_D + FLIP * (b & 1u) + 16u * (uint32_t)ch;
                uint32_t s[16];
                if constexpr (ACCS == 1) {
                    uint32_t v[16];
                    st_tmem_ld16x2(dt, dt + SIGN_AT, v, s);
#pragma unroll
                    for (int j = 0; j < 16; ++j) sc[j] = __uint_as_float(v[j]);
                } else {
#pragma unroll
                    for (int half = 0; half < 16; half += 8) {
                        uint32_t v[4][8];
                        st_ld_accs(dt + half, v, 64u);  // three accumulators and the signs
#pragma unroll
                        for (int j = 0; j < 8; ++j) {
                            float sum = __uint_as_float(v[0][j]), low = 0.0f;
                            two_sum(sum, __uint_as_float(v[1][j]), low);
                            two_sum(sum, __uint_as_float(v[2][j]), low);
                            sc[half + j] = sum + low;
                            s[half + j] = v[3][j];
                        }
                    }
                }
                const uint64_t su2 = f2_pack(su, su), lam2 = f2_pack(lam, lam);
#pragma unroll
                for (int j = 0; j < 16; j += 4) {
                    const ulonglong2 ux = *reinterpret_cast<const ulonglong2*>(uq + 16 * ch + j), uy = *reinterpret_cast<const ulonglong2*>(uq + 64 + 16 * ch + j);
#pragma unroll
                    for (int p = 0; p < 2; ++p) {
                        const uint64_t h = f2_fma(u2_pack(s[j + 2 * p], s[j + 2 * p + 1]), 0xC7000000C7000000ull, p ? ux.y : ux.x);  // 256 - 2 hamming, exact (-32768 s + u)
                        // (uy is a power of two: the coarse term is rounded once)
                        const uint64_t r2 = f2_fma(f2_mul(f2_pack(sc[j + 2 * p], sc[j + 2 * p + 1]), p ? uy.y : uy.x), su2, f2_mul(lam2, h));
                        asm("mov.b64 {%0, %1}, %2;\n" : "=f"(sc[j + 2 * p]), "=f"(sc[j + 2 * p + 1]) : "l"(r2));
                    }
                }
            }
            if (ACCS > 1 && b + 1 < blocks) stage(b + 1);  // (its barrier: every warp has read this block's accumulators)
            asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
            if (DENSE) {
                if (turned) {
                    const uint32_t to = out_s + (b & 1u) * WIDE_OUT_BYTES + (uint32_t)(16 * ch * 128 + r) * 4u;
                    if (cols) {
#pragma unroll
                        for (int j = 0; j < 16; ++j) asm volatile("st.shared.f32 [%0], %1;\n" ::"r"(to + (uint32_t)(j * 512)), "f"(sc[j]) : "memory");
                        asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
                    }
                } else if (cols) {
#pragma unroll
                    for (int j = 0; j < 16; ++j) {
                        const int q = 16 * ch + j;
                        if (q < nq && live) a.scores[roff[q] + it.index_base + t0] = sc[j];  // (32 consecutive tiles: one 128-byte store per row)
                    }
                }
                continue;
            }
            if (b == 0) {
                // The first block of an item is walked before it is filtered.  (1) Rows without a bucket mapping get one
                // from the block's scores (any monotone mapping is valid): column minima and maxima per tile
                // quarter by a butterfly, combined by one thread per row, one load and one compare-and-swap for all rows
                // at once.  (2) A counting pass puts every score of the block into the rows' histograms without
                // appending anything, and the thresholds are derived -- all CTAs of the grid count their first blocks at
                // about the same time, 128 tiles each; otherwise each CTA would append its whole first block.
                if (need_map) {
                    if (cols) {
                        float mn[16], mx[16];
#pragma unroll
                        for (int j = 0; j < 16; ++j) {
                            mn[j] = live ? sc[j] : INFINITY;
                            mx[j] = live ? sc[j] : -INFINITY;
                        }
#pragma unroll
                        for (int step = 0; step < 4; ++step) {
                            const int half = 8 >> step, off = 16 >> step;
                            const bool up = (lane & off) != 0;
#pragma unroll
                            for (int i = 0; i < half; ++i) {
                                const float rmn = __shfl_xor_sync(0xFFFFFFFFu, up ? mn[i] : mn[i + half], off);
                                const float rmx = __shfl_xor_sync(0xFFFFFFFFu, up ? mx[i] : mx[i + half], off);
                                mn[i] = fminf(up ? mn[i + half] : mn[i], rmn);
                                mx[i] = fmaxf(up ? mx[i + half] : mx[i], rmx);
                            }
                        }
                        mn[0] = fminf(mn[0], __shfl_xor_sync(0xFFFFFFFFu, mn[0], 1));
                        mx[0] = fmaxf(mx[0], __shfl_xor_sync(0xFFFFFFFFu, mx[0], 1));
                        if (!(lane & 1)) colmm[qt * WIDE_NQ + 16 * ch + (lane >> 1)] = make_float2(mn[0], mx[0]);  // column 16 ch + lane / 2
                    }
                    asm volatile("bar.sync 2, 512;\n" ::: "memory");
                    if (tid < nq && rng[tid].y == 0.0f) {
                        float lo_s = INFINITY, hi_s = -INFINITY;
                        for (int w2 = 0; w2 < 4; ++w2) {
                            lo_s = fminf(lo_s, colmm[w2 * WIDE_NQ + tid].x);
                            hi_s = fmaxf(hi_s, colmm[w2 * WIDE_NQ + tid].y);
                        }
                        const uint32_t Q = it.query_begin + (uint32_t)tid;
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
                            const float2 rr = make_float2(__uint_as_float((uint32_t)pr), __uint_as_float((uint32_t)(pr >> 32)));
                            rng[tid] = rr;
                            rmap[tid] = make_float2(-rr.x * rr.y, rr.y);
                        }
                    }
                    asm volatile("bar.sync 2, 512;\n" ::: "memory");
                }
                WPROBE_LAP(4);  // bucket mappings
                if (cols) {
#pragma unroll
                    for (int j = 0; j < 16; ++j) {
                        const int q = 16 * ch + j;
                        if (q >= nq || !live) continue;
                        const float2 rm = rmap[q];
                        atomicAdd(a.ghist + (size_t)(Q0 + (uint32_t)j) * 256 + min(max(__float2int_rz(fmaf(sc[j], rm.y, rm.x)), 0), 255), 1u);
                    }
                }
                asm volatile("bar.sync 2, 512;\n" ::: "memory");
                WPROBE_LAP(5);  // counting pass
                const int rows = min(4, nq - 4 * warp);
                if (rows > 0) wide_refresh_rows<4>(a, it.query_begin + 4u * (uint32_t)warp, rows, rng + 4 * warp, pvh + 4 * warp, lane);
                asm volatile("bar.sync 2, 512;\n" ::: "memory");
                WPROBE_LAP(6);  // thresholds
            }
            if (cols) {
                const uint32_t nidx = ~(it.index_base + t0);
                uint32_t bal[16], pm = 0, mine_cnt = 0;
#pragma unroll
                for (int j = 0; j < 16; ++j) {
                    const int q = 16 * ch + j;
                    bal[j] = 0;
                    if (q >= nq) continue;  // (uniform)
                    const bool p = live && score_key(sc[j]) >= reinterpret_cast<const volatile uint32_t*>(pvh)[q];
                    bal[j] = __ballot_sync(0xFFFFFFFFu, p);
                    if (p) pm |= 1u << j;
                    if (lane == j) mine_cnt = (uint32_t)__popc(bal[j]);
                }
                // slots of the sixteen rows' candidates: lane j reserves for row 16 ch + j, one round trip for all
                uint32_t slot0 = 0;
                if (mine_cnt) slot0 = atomicAdd(a.gcount + Q0 + (uint32_t)lane, mine_cnt);
#pragma unroll
                for (int j = 0; j < 16; ++j) {
                    if (!bal[j]) continue;  // (uniform)
                    const uint32_t base_j = __shfl_sync(0xFFFFFFFFu, slot0, j);
                    if (pm >> j & 1u) {
                        const uint32_t Q = Q0 + (uint32_t)j;
                        const uint32_t at = base_j + (uint32_t)__popc(bal[j] & ((1u << lane) - 1u));
                        if (at < a.gcap) a.gbuf[(size_t)Q * a.gcap + at] = ((uint64_t)score_key(sc[j]) << 32) | (uint64_t)nidx;
                        else a.gflag[Q] = 1u;  // the row's buffer is full: the generic kernel scores the row
                        if (b != 0) {  // (the first block was counted by its counting pass)
                            const float2 rm = rmap[16 * ch + j];
                            atomicAdd(a.ghist + (size_t)Q * 256 + min(max(__float2int_rz(fmaf(sc[j], rm.y, rm.x)), 0), 255), 1u);
                        }
                    }
                }
            }
            WPROBE_LAP(9);  // filter and append
            // thresholds again after every second block; warp w looks after rows 4 w .. 4 w + 3
            if ((b & 1u) == 1u && b + 1 < blocks) {
                const int rows = min(4, nq - 4 * warp);
                if (rows > 0) wide_refresh_rows<4>(a, it.query_begin + 4u * (uint32_t)warp, rows, rng + 4 * warp, pvh + 4 * warp, lane);
                WPROBE_LAP(6);
            }
        }
        cp_async_wait<0>();
        if (warp == 0) WPROBE_OUT(0, 12);
        if (stop && tid == 0) ctl[5] = 1u;
        __syncthreads();
        if (DENSE && a.blocked && blocks && !stop) {
            send(blocks - 1);
            if (tid == WIDE_THREADS - 32) asm volatile("cp.async.bulk.wait_group 0;\n" ::: "memory");  // (the next item's first block fills a buffer behind its barriers)
        }
        // rows this CTA could not score (another codec, a query outside the fp16 split, a wait that ran out) go to the generic kernel, of a dense call to
        // the four-row kernel
        if (*reinterpret_cast<volatile uint32_t*>(ctl + 6) || stop) {
            if (DENSE) wide_hand_on(a, it, wide_hand_as(a, it));
            else if (tid < nq) a.gflag[it.query_begin + tid] = 1u;
        }
        __syncthreads();
        if (tid == 0) ctl[6] = 0u;  // (ordered before the next item's writers by the barrier at its start)
    }
    if (stop) {
        // a wait ran out (the same in all threads): the barrier's phases are no longer known, the remaining items go to the generic kernel too (of a
        // dense call to the four-row kernel)
        for (uint32_t item_id = a.cta_begin[blockIdx.x]; item_id < item_end; ++item_id) {
            const WorkItem it = a.items[item_id];
            if (DENSE) wide_hand_on(a, it, wide_hand_as(a, it));
            else if (tid < (int)it.n_queries) a.gflag[it.query_begin + tid] = 1u;
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(512u) : "memory");
}

template <int KIND>
__global__ void __launch_bounds__(WIDE_THREADS, 1) score_wide_kernel(ScoreArgs a) {
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    dep_launch();
    dep_wait();
    const uint32_t first = a.cta_begin[blockIdx.x];
    // (a plan made for MIX3 tiles also takes INT4 / MX-INT4 tiles of its shape, see score_mix3_kernel)
    if (KIND == 4 && item_kind(first_tile_flags(a, a.items[first]), false) == 3) wide_body<3, false>(a, smem_raw, first);
    else wide_body<KIND, false>(a, smem_raw, first);
}

// Dense scores; a CTA decodes the kind of its first item that is not NF4.  Items of other kinds, and NF4 tiles, whose scale bytes cannot
// be folded into A, go to score_dense_kernel's pass over the flagged rows.
__global__ void __launch_bounds__(WIDE_THREADS, 1) score_wide_dense_kernel(ScoreArgs a) {
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    dep_launch();
    dep_wait();
    if (a.refused && *a.refused) return;
    uint32_t i = a.cta_begin[blockIdx.x];
    const uint32_t item_end = a.cta_begin[blockIdx.x + 1];
    int kind = item_kind(first_tile_flags(a, a.items[i]), false);
    while (kind == 0) {
        wide_hand_on(a, a.items[i], 1u);
        if (++i == item_end) return;
        kind = item_kind(first_tile_flags(a, a.items[i]), false);
    }
    if (kind == 1) wide_body<1, true>(a, smem_raw, i);
    else if (kind == 2) wide_body<2, true>(a, smem_raw, i);
    else if (kind == 4) wide_body<4, true>(a, smem_raw, i);
    else wide_body<3, true>(a, smem_raw, i);
}

}  // namespace
}  // namespace slha
