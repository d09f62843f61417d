// Top-k of rows whose scores have all been written: one CTA per query row.  Included by score.cu after score_merge.cuh.
//
// Where a row is short (a decode step over an ordinary context, a batch of queries on one cache) the streaming top-k has little to stream: its thresholds come
// from the first tiles of every warp, which are appended unfiltered, and the passes behind it (hand-over check, compaction, merge) each cost
// a launch and a chain of latencies.  Scores written as a whole cost four bytes a tile and row, which the L2 keeps, and need no threshold while they
// are made.  Here a row's scores go to registers, a sample of them gives a bound that little more than k reach, every thread keeps the few of its own that do,
// and those are compacted: up to ROW_RANKED are ordered by comparing each with all, more by buckets between the bound and the largest score of the
// sample and by comparing inside a bucket, or, where that is crowded (equal scores, one far from the rest), by a radix sort.
// Bound: the latencies between the block barriers, and for many rows the instructions a score costs.  us a call, streamed and merged / whole rows: 4096
// INT4 tiles, k = 64 19.6 / 10.6, 8 x 8192 mixed tiles x 4 rows, k = 256 26.6 / 13.0, 8 x 16 384 TQ3 x 64 rows 85 / 47 (with events between the two 34 of scores, 22 of selection).  With the
// candidates ordered by buckets alone 13.6 and 48.1; with a histogram of the whole row in place of the sample 20 us for 512 rows of 16 384.
#pragma once

namespace slha {
namespace {

constexpr int ROW_BUCKETS = 1024;
constexpr uint32_t ROW_ABSENT = 0xFFFFFFFFu;      // bits of a score that is not there (no arithmetic gives this NaN)
constexpr int row_own(int r) { return 4 * r < 16 ? 4 * r : 16; }  // candidates a thread keeps
struct RowInfo {
    uint32_t n, index_base;  // scores of the row, reported index of the first
    uint32_t begin, step;    // where they lie: 128 from begin on, the next 128 `step` further, ..
};
struct RowsArgs {
    const float* scores;
    const RowInfo* rows;
    uint32_t* flag;          // [nq] a work item of the row took the generic arithmetic, [nq] it was handed on by the 64-row kernel, [4 nq] whether any was (cleared here)
    uint32_t* stats;         // [nq][2] candidates, the flag
    uint32_t k, cap;         // cap: slots for candidates, row_cap
    uint32_t* out_index;
    float* out_score;
    uint32_t* out_count;
};
// slots: what a sample's bound lets through, see below, and k rounded up to a power of two at least
inline uint32_t row_cap(uint32_t k, uint32_t kp2) { return std::max(kp2, std::min(4u * k + 1024u, 2u * k + 2560u)); }
constexpr int ROW_HIST_INTS = ROW_BUCKETS + 64;
// (the threads' own lists make room for the candidates by buckets)
__host__ __device__ constexpr size_t row_own_slots(uint32_t cap, int nt, int r) { return (size_t)nt * row_own(r) > cap ? (size_t)nt * row_own(r) : cap; }
inline size_t row_smem(uint32_t cap, int nt, int r) { return ((size_t)cap + row_own_slots(cap, nt, r)) * 8 + (size_t)(ROW_HIST_INTS + 64) * 4 + (size_t)(cap + 1) / 2 * 4; }
constexpr uint32_t ROW_RANKED = 192;              // candidates that are ordered by comparing each with all
// Candidates of a bucket up to which the bucket is ordered by comparing each with all.  Above, all candidates are sorted: comparing goes by the bucket's square (us a call by comparing / sorting:
// 4 rows of 6000 equal scores 1004 / 38, of 4096 scores with one 10 000 times the others, k = 4096 466 / 54), sorting by the candidates (4 rows of 30 000, each score thirty times, k = 4096, buckets of
// some hundred 42 / 67).
constexpr uint32_t ROW_CROWD = 512;

// The CTA's hist[ROW_BUCKETS] into c, ROW_BUCKETS / NT a thread; the sum of the counts before the thread's.  (st[16 ..]: a word a warp.)
template <int NT>
__device__ __forceinline__ int row_scan(const int* hist, uint32_t* st, int (&c)[ROW_BUCKETS / NT]) {
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    int sum = 0;
#pragma unroll
    for (int j = 0; j < ROW_BUCKETS / NT; ++j) {
        c[j] = hist[tid * (ROW_BUCKETS / NT) + j];
        sum += c[j];
    }
    int incl = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xFFFFFFFFu, incl, o);
        if ((int)lane >= o) incl += y;
    }
    if (lane == 31) st[16 + warp] = (uint32_t)incl;
    __syncthreads();
    const int before = lane < warp ? (int)st[16 + lane] : 0;
    return incl - sum + __reduce_add_sync(0xFFFFFFFFu, before);
}
// buf[0 .. count) in descending order, there or behind cap: a stable radix sort, six bits at a time where the keys differ.  A warp takes a run of the keys; hist[16 x digit + warp] holds its
// counts, then its places.
template <int NT>
__device__ __forceinline__ const uint64_t* row_sort(uint64_t* buf, uint32_t cap, uint32_t count, int* hist, uint32_t* st) {
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    constexpr int PER = ROW_BUCKETS / NT;
    uint64_t *from = buf, *to = buf + cap;
    if (tid == 0) st[8] = st[9] = 0u;
    __syncthreads();
    uint64_t differ = 0;
    for (uint32_t i = tid; i < count; i += NT) differ |= from[i] ^ from[0];
    const uint32_t lo = __reduce_or_sync(0xFFFFFFFFu, (uint32_t)differ), hi = __reduce_or_sync(0xFFFFFFFFu, (uint32_t)(differ >> 32));
    if (lane == 0) {
        atomicOr(&st[8], lo);
        atomicOr(&st[9], hi);
    }
    __syncthreads();
    differ = (uint64_t)st[9] << 32 | st[8];
    const uint32_t run = (count + NT - 1) / NT * 32, first = min(count, warp * run), end = min(count, first + run);
    for (int shift = 0; shift < 64; shift += 6) {
        if (!(differ >> shift & 63u)) continue;
        for (uint32_t b = tid; b < (uint32_t)ROW_BUCKETS; b += NT) hist[b] = 0;
        __syncthreads();
        for (uint32_t i0 = first; i0 < end; i0 += 32) {
            const bool in = i0 + lane < end;
            const uint32_t digit = in ? 63u - (uint32_t)(from[i0 + lane] >> shift & 63u) : 64u, same = __match_any_sync(0xFFFFFFFFu, digit);
            if (in && (uint32_t)__ffs(same) - 1u == lane) hist[16 * digit + warp] += __popc(same);
            __syncwarp();
        }
        __syncthreads();
        int c[PER], at = row_scan<NT>(hist, st, c);
#pragma unroll
        for (int j = 0; j < PER; ++j) {
            hist[tid * PER + j] = at;
            at += c[j];
        }
        __syncthreads();
        for (uint32_t i0 = first; i0 < end; i0 += 32) {
            const bool in = i0 + lane < end;
            const uint64_t key = in ? from[i0 + lane] : 0ull;
            const uint32_t digit = in ? 63u - (uint32_t)(key >> shift & 63u) : 64u, same = __match_any_sync(0xFFFFFFFFu, digit);
            const int place = in ? hist[16 * digit + warp] : 0;
            __syncwarp();
            if (in) to[place + __popc(same & ((1u << lane) - 1u))] = key;
            if (in && (uint32_t)__ffs(same) - 1u == lane) hist[16 * digit + warp] = place + __popc(same);
            __syncwarp();
        }
        __syncthreads();
        uint64_t* const was = from;
        from = to;
        to = was;
    }
    return from;
}

// R: 4 R scores a thread, n <= 4 R x threads
template <int NT, int R>
__global__ void __launch_bounds__(NT, R <= 2 ? 1536 / NT : R <= 8 ? 2 : 1) topk_rows_kernel(RowsArgs a) {
    extern __shared__ __align__(16) unsigned char smem[];
    const RowInfo info = a.rows[blockIdx.x];  // (the plan's: no kernel writes it)
    dep_launch();
    dep_wait();
    constexpr int OWN = row_own(R), PER = ROW_BUCKETS / NT;
    const uint32_t k = a.k, cap = a.cap, Q = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    uint64_t* buf = reinterpret_cast<uint64_t*>(smem);                     // [cap]
    uint64_t* own = buf + cap + tid;                                       // [OWN], NT apart; then the candidates' places in their buckets
    int* hist = reinterpret_cast<int*>(buf + cap + row_own_slots(cap, NT, R));  // [ROW_BUCKETS + 1]
    uint32_t* st = reinterpret_cast<uint32_t*>(hist + ROW_HIST_INTS);     // 0 candidates, 1 smallest and 2 largest score word, 3 bound's bucket and 10, 11, 13 what a closer look at it needs, 14 the bucket of a lower bound, 5, 8, 9 of a selection step, 12 a bucket is crowded, 16.. warp totals
    const uint32_t n = info.n;
    const float* row = a.scores + info.begin;
    // thread t holds the scores 4 (t + NT j) .. + 3
    auto load4 = [&](int j) {
        const uint32_t e = 4u * (tid + (uint32_t)NT * j);
        uint4 x = e < n ? __ldcg(reinterpret_cast<const uint4*>(row + (size_t)(e >> 7) * info.step + (e & 127u))) : make_uint4(ROW_ABSENT, ROW_ABSENT, ROW_ABSENT, ROW_ABSENT);
        if (e + 3u >= n) {
            if (e + 1u >= n) x.y = ROW_ABSENT;
            if (e + 2u >= n) x.z = ROW_ABSENT;
            x.w = ROW_ABSENT;
        }
        return x;
    };
    uint4 v[R];
#pragma unroll
    for (int j = 0; j < R; ++j) v[j] = load4(j);
    if (tid < 16) st[tid] = tid == 1 || tid == 10 ? 0xFFFFFFFFu : 0u;
    for (int b = (int)tid; b <= ROW_BUCKETS; b += NT) hist[b] = 0;
    __syncthreads();
    // (What one pass over the row computed from the scores is not kept for the next: it would take as many registers as they do.)
    auto fresh = [&]() {
#pragma unroll
        for (int j = 0; j < R; ++j) asm volatile("" : "+r"(v[j].x), "+r"(v[j].y), "+r"(v[j].z), "+r"(v[j].w));
    };
    fresh();
    // Long rows: a bound from a sample, every fourth to sixteenth score all along the row (neighbours resemble one another).  Where `part` of the sample should lie above the k-th score, it is the lower edge of the bucket
    // in which the sample's count from the top reaches 1.25 part + 3 sqrt(part) + 2.
    constexpr int STEP = R >= 16 ? 4 : (R >= 8 ? 2 : 1);
    const bool sampled = R > 2 || n > cap / 2u;
    {
        uint32_t mn = 0xFFFFFFFFu, mx = 0u;
#pragma unroll
        for (int j = 0; j < R; ++j) {
            const uint32_t x[4] = {v[j].x, v[j].y, v[j].z, v[j].w};
#pragma unroll
            for (int c = 0; c < 4; ++c)
                if (sampled ? c == 0 && ((tid + j) & (STEP - 1)) == 0 : R <= 2) {
                    const float s = __uint_as_float(x[c]);
                    if (fabsf(s) < INFINITY) {
                        mn = min(mn, score_key(s));
                        mx = max(mx, score_key(s));
                    }
                }
        }
        mn = __reduce_min_sync(0xFFFFFFFFu, mn);
        mx = __reduce_max_sync(0xFFFFFFFFu, mx);
        if (lane == 0 && mx) {
            atomicMin(&st[1], mn);
            atomicMax(&st[2], mx);
        }
    }
    __syncthreads();
    const bool ranged = st[2] > st[1];
    float low = key_score(ranged ? st[1] : score_key(0.0f)), bound = -INFINITY;
    const float top = key_score(ranged ? st[2] : score_key(1.0f));
    if (sampled && ranged) {
        const float part = (float)k * (0.25f / (float)STEP);
        const int want = (int)(1.25f * part + 3.0f * sqrtf(part)) + 2, most = (int)(cap * 3u / (16u * STEP)), safe = min(most, 3 * want);
        float inv = (float)ROW_BUCKETS / (top - low);  // (a range that overflows puts all in one bucket)
#pragma unroll
        for (int j = 0; j < R; ++j) {
            const float s = __uint_as_float(v[j].x);
            if (((tid + j) & (STEP - 1)) == 0 && fabsf(s) < INFINITY) atomicAdd(&hist[min(max(__float2int_rz((top - s) * inv), 0), ROW_BUCKETS - 1)], 1);
        }
        __syncthreads();
        int c[PER], at = row_scan<NT>(hist, st, c);
#pragma unroll
        for (int j = 0; j < PER; ++j) {
            if (at < want && at + c[j] >= want) {
                st[3] = tid * PER + j + 1;
                if (at + c[j] > most) st[13] = at + 1;
            }
            if (R > 2 && at <= safe && at + c[j] > safe) st[14] = tid * PER + j;  // (shorter rows take 20 us without a bound)
            at += c[j];
            hist[tid * PER + j] = 0;
        }
        __syncthreads();
        if (st[3] && st[3] < (uint32_t)ROW_BUCKETS) bound = top - (float)st[3] / inv;  // (zero: the sample holds too few, all are candidates)
        // Scores far from the rest (an attention sink) leave that bucket with more than the candidates' slots hold: its own scores in buckets, up to three times.  (128 rows of 30 000, one score
        // 10 000 times the others, k = 1024: 449 us a call without, 81 with it.)
        if (__builtin_expect(st[13] != 0u, 0)) {
            float upper = top, lower = low;
#pragma unroll 1
            for (int zoom = 0; zoom < 3 && st[13]; ++zoom) {
                const int b = (int)st[3] - 1, above = (int)st[13] - 1;
                uint32_t mn = 0xFFFFFFFFu, mx = 0u;
#pragma unroll
                for (int j = 0; j < R; ++j) {
                    const float s = __uint_as_float(v[j].x);
                    if (((tid + j) & (STEP - 1)) == 0 && s >= lower && s <= upper && min(max(__float2int_rz((upper - s) * inv), 0), ROW_BUCKETS - 1) == b) {
                        mn = min(mn, score_key(s));
                        mx = max(mx, score_key(s));
                    }
                }
                mn = __reduce_min_sync(0xFFFFFFFFu, mn);
                mx = __reduce_max_sync(0xFFFFFFFFu, mx);
                if (lane == 0 && mx) {
                    atomicMin(&st[10], mn);
                    atomicMax(&st[11], mx);
                }
                __syncthreads();
                lower = key_score(st[10]);
                upper = key_score(st[11]);
                __syncthreads();
                if (!(lower < upper)) break;  // (all equal, the same in every thread)
                if (tid == 0) {
                    st[3] = st[11] = st[13] = 0u;
                    st[10] = 0xFFFFFFFFu;
                }
                inv = (float)ROW_BUCKETS / (upper - lower);
#pragma unroll
                for (int j = 0; j < R; ++j) {
                    const float s = __uint_as_float(v[j].x);
                    if (((tid + j) & (STEP - 1)) == 0 && s >= lower && s <= upper) atomicAdd(&hist[min(max(__float2int_rz((upper - s) * inv), 0), ROW_BUCKETS - 1)], 1);
                }
                __syncthreads();
                int c[PER], at = row_scan<NT>(hist, st, c) + above;
#pragma unroll
                for (int j = 0; j < PER; ++j) {
                    if (at < want && at + c[j] >= want) {
                        st[3] = tid * PER + j + 1;
                        if (at + c[j] > most) st[13] = at + 1;
                    }
                    at += c[j];
                    hist[tid * PER + j] = 0;
                }
                __syncthreads();
                if (st[3]) bound = st[3] < (uint32_t)ROW_BUCKETS ? upper - (float)st[3] / inv : lower;
            }
        }
    }
    // what reaches the bound: the thread's own candidates
    uint32_t mine;
    for (;;) {
        fresh();
        mine = 0;
#pragma unroll
        for (int j = 0; j < R; ++j) {
            const uint32_t x[4] = {v[j].x, v[j].y, v[j].z, v[j].w};
#pragma unroll
            for (int c = 0; c < 4; ++c)
                if (__uint_as_float(x[c]) >= bound) {
                    if (OWN == 4 * R || mine < (uint32_t)OWN) own[mine * NT] = (uint64_t)x[c] << 32 | (uint32_t)(4 * NT * j + c);
                    ++mine;
                }
            asm volatile("" : "+r"(mine) : : "memory");  // (four at a time: all comparisons first would take a register each)
        }
        if (bound <= 0.0f) {  // a NaN counts as -0, as score_kernel's keys have it
#pragma unroll
            for (int j = 0; j < R; ++j) {
                const uint32_t x[4] = {v[j].x, v[j].y, v[j].z, v[j].w};
#pragma unroll
                for (int c = 0; c < 4; ++c)
                    if ((x[c] & 0x7FFFFFFFu) > 0x7F800000u && x[c] != ROW_ABSENT) {
                        if (OWN == 4 * R || mine < (uint32_t)OWN) own[mine * NT] = (uint64_t)0x80000000u << 32 | (uint32_t)(4 * NT * j + c);
                        ++mine;
                    }
                asm volatile("" : "+r"(mine) : : "memory");
            }
        }
        if (__any_sync(0xFFFFFFFFu, mine != 0u)) {
            uint32_t incl = mine;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, incl, o);
                if (lane >= (uint32_t)o) incl += y;
            }
            uint32_t at = 0;
            if (lane == 31) at = atomicAdd(&st[0], incl);
            at = __shfl_sync(0xFFFFFFFFu, at, 31) + incl - mine;
            if (OWN < 4 * R && mine > (uint32_t)OWN) {  // all of the thread's candidates again, for want of room in its own list (read again: the unrolled form cost all launches 1.4 %)
#pragma unroll 1
                for (int j = 0; j < R; ++j) {
                    const uint4 w = load4(j);
                    const uint32_t x[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
                    for (int c = 0; c < 4; ++c) {
                        const float s = __uint_as_float(x[c]);
                        const bool nan = bound <= 0.0f && s != s && x[c] != ROW_ABSENT;
                        if (!(s >= bound || nan)) continue;
                        if (at < cap) buf[at] = make_comp(nan ? -0.0f : s, info.index_base + 4u * (tid + (uint32_t)NT * j) + c);
                        ++at;
                    }
                }
                mine = 0u;
            }
            for (uint32_t h = 0; h < min(mine, (uint32_t)OWN); ++h, ++at) {
                const uint64_t e = own[h * NT];
                if (at < cap) buf[at] = make_comp(__uint_as_float((uint32_t)(e >> 32)), info.index_base + 4u * tid + (uint32_t)e);
            }
        }
        __syncthreads();
        if (st[0] >= k || bound == -INFINITY) break;
        // The sample misled: a bound that three times as many of it reach, in the end none.  (One of some thousand rows for small k; in a call of 32 rows of 32 768 the selection of all
        // scores that follows without a bound took 102 us instead of 33.)
        const float second = top - (float)st[14] * (top - low) / (float)ROW_BUCKETS;
        bound = R > 2 && st[14] && second < bound ? second : -INFINITY;
        __syncthreads();
        if (tid == 0) st[0] = st[14] = 0u;
        __syncthreads();
    }
    const uint32_t got = st[0], m = min(got, k);
    uint32_t* const out_index = a.out_index + (size_t)Q * k;
    float* const out_score = a.out_score + (size_t)Q * k;
    const bool listed = got <= cap;
    bool crowded = false;
    if (listed && got <= ROW_RANKED) {
        // Few candidates: a candidate's place is the number of larger ones, counted by SPLIT threads in turn (a slice of the list each).
        constexpr uint32_t SPLIT = 2;
        const uint32_t i = tid / SPLIT, part = tid % SPLIT;
        for (uint32_t c = i; c < got; c += NT / SPLIT) {
            const uint64_t key = buf[c];
            uint32_t r = 0;
#pragma unroll 8
            for (uint32_t x = part; x < got; x += SPLIT) r += buf[x] > key;
            r += __shfl_xor_sync(3u << (lane & 30u), r, 1);
            if (part == 0 && r < m) {
                out_index[r] = 0xFFFFFFFFu - (uint32_t)key;
                out_score[r] = key_score((uint32_t)(key >> 32));
            }
        }
        for (uint32_t r = m + tid; r < k; r += NT) {
            out_index[r] = 0xFFFFFFFFu;
            out_score[r] = -INFINITY;
        }
    } else if (listed) {
        if (bound > low) low = bound;
        const float inv = (float)ROW_BUCKETS / (top - low);
        const bool apart = inv > 0.0f && inv < INFINITY;
        auto bucket = [&](uint64_t key) { return apart ? min(max(__float2int_rz((top - key_score((uint32_t)(key >> 32))) * inv), 0), ROW_BUCKETS - 1) : 0; };
        // placed[]: the candidates by buckets; a candidate's number in its bucket comes from the counting (any order)
        uint64_t* const placed = buf + cap;
        uint16_t* const number = reinterpret_cast<uint16_t*>(st + 64);
        for (uint32_t i = tid; i < got; i += NT) number[i] = (uint16_t)atomicAdd(&hist[bucket(buf[i])], 1);
        __syncthreads();
        int c[PER], at = row_scan<NT>(hist, st, c);
#pragma unroll
        for (int j = 0; j < PER; ++j) {
            hist[tid * PER + j] = at;
            at += c[j];
            if (c[j] > (int)ROW_CROWD) st[12] = 1u;
        }
        if (tid == NT - 1) hist[ROW_BUCKETS] = at;
        __syncthreads();
        for (uint32_t i = tid; i < got; i += NT) {
            const uint64_t key = buf[i];
            placed[hist[bucket(key)] + (int)number[i]] = key;
        }
        __syncthreads();
        crowded = st[12] != 0u;
        for (uint32_t i = tid; i < got && !crowded; i += NT) {
            const uint64_t key = placed[i];
            const int b = bucket(key);
            const int s0 = hist[b], e0 = hist[b + 1];
            uint32_t r = (uint32_t)s0;
            for (int x = s0; x < e0; ++x) r += placed[x] > key;
            if (r < m) {
                out_index[r] = 0xFFFFFFFFu - (uint32_t)key;
                out_score[r] = key_score((uint32_t)(key >> 32));
            }
        }
        for (uint32_t r = m + tid; r < k; r += NT) {
            out_index[r] = 0xFFFFFFFFu;
            out_score[r] = -INFINITY;
        }
    } else {
        // Too many candidates (many equal scores, or outliers far from the rest): a radix selection of the k-th largest score word, what
        // lies above it, and of the scores equal to it those with the lowest indices.  (More than k are there.  The row is read again: held on to for
        // this, it would cost every launch registers.)
        auto word = [](uint32_t bits) { return (bits & 0x7FFFFFFFu) > 0x7F800000u ? 0x7FFFFFFFu : score_key(__uint_as_float(bits)); };
        uint32_t prefix = 0, need = k;
        for (int shift = 24;; shift -= 8) {
            __syncthreads();
            for (int b = (int)tid; b < 256; b += NT) hist[b] = 0;
            __syncthreads();
#pragma unroll 1
            for (int j = 0; j < R; ++j) {
                const uint4 w = load4(j);
                const uint32_t x[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    const uint32_t h = word(x[c]);
                    const bool in = x[c] != ROW_ABSENT && (shift == 24 || (h >> (shift + 8)) == prefix);
                    const uint32_t b = in ? (h >> shift) & 255u : 256u;
                    // (equal scores meet in one bucket: one atomic per warp and bucket)
                    const uint32_t same = __match_any_sync(0xFFFFFFFFu, b);
                    if (in && (uint32_t)__ffs(same) - 1u == lane) atomicAdd(&hist[b], __popc(same));
                }
            }
            __syncthreads();
            if (tid < 32) {  // lane l owns bins 255-8l .. 248-8l (descending)
                int c[8], tot = 0;
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    c[j] = hist[255 - 8 * (int)tid - j];
                    tot += c[j];
                }
                int incl = tot;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const int y = __shfl_up_sync(0xFFFFFFFFu, incl, o);
                    if ((int)lane >= o) incl += y;
                }
                const unsigned ok = __ballot_sync(0xFFFFFFFFu, incl >= (int)need);
                if ((int)tid == __ffs(ok) - 1) {
                    int run = incl - tot;
#pragma unroll
                    for (int j = 0; j < 8; ++j) {
                        if (run + c[j] >= (int)need) {
                            st[8] = 255u - 8u * tid - (uint32_t)j;
                            st[9] = (uint32_t)run;
                            break;
                        }
                        run += c[j];
                    }
                }
            }
            __syncthreads();
            prefix = (prefix << 8) | st[8];
            need -= st[9];
            if (shift == 0) break;
        }
        __syncthreads();
        if (tid == 0) st[5] = 0u;
        __syncthreads();
#pragma unroll 1
        for (int j = 0; j < R; ++j) {  // (4 NT scores at a time in index order, so that the lowest indices among the equal ones come first)
            const uint4 w = load4(j);
            const uint32_t x[4] = {w.x, w.y, w.z, w.w}, e = info.index_base + 4u * (tid + (uint32_t)NT * j);
            uint32_t eq = 0;
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                if (x[c] == ROW_ABSENT) continue;
                const uint32_t h = word(x[c]);
                if (h > prefix) buf[atomicAdd(&st[5], 1u)] = ((uint64_t)word(x[c]) << 32 | (0xFFFFFFFFu - (e + c)));
                else if (h == prefix) ++eq;
            }
            uint32_t incl = eq;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, incl, o);
                if (lane >= (uint32_t)o) incl += y;
            }
            if (lane == 31) st[16 + warp] = incl;
            __syncthreads();
            uint32_t rank = incl - eq, all = 0;
            for (uint32_t w2 = 0; w2 < NT / 32; ++w2) {
                if (w2 < warp) rank += st[16 + w2];
                all += st[16 + w2];
            }
#pragma unroll
            for (int c = 0; c < 4; ++c)
                if (x[c] != ROW_ABSENT && word(x[c]) == prefix) {
                    if (rank < need) buf[atomicAdd(&st[5], 1u)] = ((uint64_t)word(x[c]) << 32 | (0xFFFFFFFFu - (e + c)));
                    ++rank;
                }
            need -= min(need, all);
            __syncthreads();
        }
    }
    if (__builtin_expect(crowded || !listed, 0)) emit_sorted(row_sort<NT>(buf, cap, listed ? got : k, hist, st), m, k, Q, a.out_index, a.out_score, nullptr);
    if (tid == 0) {
        if (a.out_count) a.out_count[Q] = m;
        a.stats[2 * Q] = got;
        a.stats[2 * Q + 1] = a.flag[Q];
        a.flag[Q] = a.flag[gridDim.x + Q] = 0u;
        if (Q == 0) a.flag[4 * (size_t)gridDim.x] = 0u;
    }
}

}  // namespace
}  // namespace slha
