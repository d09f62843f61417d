// Host side of the scoring path: work decomposition ("plan"), kernel launches.
// Included by score.cu.
#pragma once

#include <memory>

namespace slha {

namespace {

constexpr size_t MAX_SMEM = 227 * 1024;

// slha_b200_debug_force_generic_score: the calling thread's score_topk calls skip the
// tensor-core kernel (a checking aid: both kernels must give the same answers).
thread_local bool g_force_generic = false;
thread_local bool g_stream_all_rows = false;  // slha_b200_debug_stream_all_rows
struct Plan;
thread_local const Plan* g_last_stream_plan = nullptr;  // the calling thread's latest tensor-core call (for its counters)

// Tiles a CTA is given at least: two rounds of score_stream_kernel's 24 warps.  us per call with 512 / 768 / 2048: 4096 INT4 tiles,
// one query 27.4 / 26.7 / 32.9; 8 segments x 2048 tiles 27.4 / 26.9 / 36.2; 4 x 32 768 TQ3 tiles 45.6 / 45.1 / 62.8.
constexpr uint32_t STREAM_LEAST = 768;
// kind of a launch by the flags of a tile (dequant_at's precedence)
int stream_kind(uint32_t flags) { return (flags & F_MIXED) ? 1 : ((flags & F_TQ3) ? 2 : ((flags & F_MIX3) ? 4 : ((flags & F_NF4) ? 0 : 3))); }
// the same for a codec hint: bit 0 NF4 tiles expected, bit 1 mixed 8/4 only, bit 2 TQ3 only, bit 3 MIX3 only
int hint_kind(int hint) { return (hint & 2) ? 1 : ((hint & 4) ? 2 : ((hint & 8) ? 4 : ((hint & 1) ? 0 : 3))); }

template <typename F>
Status launch_tc(Ctx* c, F* kernel, bool* configured, const ScoreArgs& a, uint32_t grid, int threads, size_t smem, bool behind = false) {
    if (!configured[c->device & 15]) {  // (the attribute is per device)
        SLHA_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        configured[c->device & 15] = true;
    }
    if (behind) SLHA_CUDA(launch_behind(kernel, dim3(grid), dim3(threads), smem, c->stream, a));
    else kernel<<<grid, threads, smem, c->stream>>>(a);
    count_launch();
    SLHA_CUDA(cudaGetLastError());
    return Status();
}
template <int KIND, bool IL, bool LONG>
Status launch_stream_t(Ctx* c, const ScoreArgs& a, uint32_t grid) {
    static thread_local bool configured[16] = {false};
    return launch_tc(c, score_stream_kernel<KIND, IL, LONG>, configured, a, grid, STREAM_THREADS, stream_smem_bytes(KIND, stream_sets(KIND, LONG)), true);
}
template <bool IL>
Status launch_mix3(Ctx* c, const ScoreArgs& a, uint32_t grid) {
    static thread_local bool configured[16] = {false};
    return launch_tc(c, score_mix3_kernel<IL>, configured, a, grid, ST_THREADS, st_smem_bytes(false), true);
}
template <bool IL, bool LONG>
Status launch_stream_i(Ctx* c, int kind, const ScoreArgs& a, uint32_t grid) {
    switch (kind) {
        case 0: return launch_stream_t<0, IL, LONG>(c, a, grid);
        case 1: return launch_stream_t<1, IL, LONG>(c, a, grid);
        case 2: return launch_stream_t<2, IL, LONG>(c, a, grid);
        case 3: return launch_stream_t<3, IL, LONG>(c, a, grid);
        default: return launch_mix3<IL>(c, a, grid);
    }
}
Status launch_stream(Ctx* c, int kind, bool il, bool long_items, const ScoreArgs& a, uint32_t grid) {
    if (il) return launch_stream_i<true, false>(c, kind, a, grid);
    return long_items ? launch_stream_i<false, true>(c, kind, a, grid) : launch_stream_i<false, false>(c, kind, a, grid);
}
// tiles a warp takes at a time, and warps of a CTA
uint32_t stream_warp_tiles(int kind, int sets) { return kind == 4 ? ST_WT : (uint32_t)(MMA_SET_TILES * sets); }
uint32_t stream_warps(int kind) { return (uint32_t)(kind == 4 ? ST_THREADS : STREAM_THREADS) / 32; }
static_assert(ST_CHUNK == ST_WT, "a fresh chunk holds what a warp can append at once");
template <bool PASS>
Status launch_dense_t(Ctx* c, const ScoreArgs& a, uint32_t grid, bool behind) {
    static thread_local bool configured[16] = {false};
    return launch_tc(c, score_dense_kernel<PASS>, configured, a, grid, ST_THREADS, st_smem_bytes(true), behind);
}
Status launch_dense(Ctx* c, const ScoreArgs& a, uint32_t grid, bool behind) {
    return a.streams ? launch_dense_t<true>(c, a, grid, behind) : launch_dense_t<false>(c, a, grid, behind);
}
template <int KIND>
Status launch_wide_t(Ctx* c, const ScoreArgs& a, uint32_t grid) {
    static thread_local bool configured[16] = {false};
    return launch_tc(c, score_wide_kernel<KIND>, configured, a, grid, WIDE_THREADS, wide_smem_bytes(false), true);
}
Status launch_wide(Ctx* c, int kind, const ScoreArgs& a, uint32_t grid) {
    switch (kind) {
        case 1: return launch_wide_t<1>(c, a, grid);
        case 2: return launch_wide_t<2>(c, a, grid);
        case 3: return launch_wide_t<3>(c, a, grid);
        default: return launch_wide_t<4>(c, a, grid);
    }
}
Status launch_wide_dense(Ctx* c, const ScoreArgs& a, uint32_t grid, bool behind) {
    static thread_local bool configured[16] = {false};
    return launch_tc(c, score_wide_dense_kernel, configured, a, grid, WIDE_THREADS, wide_smem_bytes(true), behind);
}
template <int NT, int R>
Status launch_rows_t(Ctx* c, const RowsArgs& a, uint32_t nq) {
    static thread_local bool configured[16] = {false};
    if (!configured[c->device & 15]) {
        SLHA_CUDA(cudaFuncSetAttribute(topk_rows_kernel<NT, R>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)row_smem(row_cap(4096, 4096), NT, R)));
        SLHA_CUDA(cudaFuncSetAttribute(topk_rows_kernel<NT, R>, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared));
        configured[c->device & 15] = true;
    }
    SLHA_CUDA(launch_behind(topk_rows_kernel<NT, R>, dim3(nq), dim3(NT), row_smem(a.cap, NT, R), c->stream, a));
    count_launch();
    return Status();
}
constexpr uint32_t ROWS_MOST = 32768;  // scores of a row that topk_rows_kernel takes
Status launch_rows(Ctx* c, const RowsArgs& a, uint32_t nq, uint32_t longest) {
    // (many short rows of which little is selected: more CTAs an SM.  us a call, 256 / 128 threads: 22 528 rows of 174 INT4 tiles k = 16 222 / 198, k = 100 223 / 212; 8000 of 500
    // k = 16 118 / 116, k = 100 119 / 123, k = 500 143 / 167)
    if (nq >= 1024 && (longest <= 256 || (longest <= 1024 && a.k <= 64))) return launch_rows_t<128, 2>(c, a, nq);
    if (longest <= 2048) return launch_rows_t<256, 2>(c, a, nq);
    if (longest <= 4096) return launch_rows_t<512, 2>(c, a, nq);
    if (longest <= 8192) return launch_rows_t<512, 4>(c, a, nq);
    if (longest <= 16384) return launch_rows_t<512, 8>(c, a, nq);
    return launch_rows_t<512, 16>(c, a, nq);
}

size_t score_smem_bytes(int G, int nwarps, bool topk, uint32_t cap) {
    size_t b = (size_t)G * D_C * 4 + 16 * 32 * 4 + (size_t)nwarps * DEPTH * BLK_BYTES;
    if (topk) b += (size_t)G * cap * 8;
    b += (size_t)G * 8 + (size_t)G * 4 + 260 * 4 + 16;
    return b;
}

template <int G, bool TOPK>
Status launch_score_t(Ctx* c, const ScoreArgs& a, uint32_t grid, int threads, size_t smem, bool behind) {
    static thread_local size_t configured[16] = {0};
    int dev = c->device & 15;
    if (configured[dev] < smem) {
        SLHA_CUDA(cudaFuncSetAttribute(score_kernel<G, TOPK>,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize, (int)MAX_SMEM));
        // every kernel of a scoring call asks for the same shared-memory / L1 split, so that an SM does not have to
        // be drained and reconfigured between the kernels of one call
        SLHA_CUDA(cudaFuncSetAttribute(score_kernel<G, TOPK>, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared));
        configured[dev] = MAX_SMEM;
    }
    if (behind) SLHA_CUDA(launch_behind(score_kernel<G, TOPK>, dim3(grid), dim3(threads), smem, c->stream, a));
    else score_kernel<G, TOPK><<<grid, threads, smem, c->stream>>>(a);
    count_launch();
    SLHA_CUDA(cudaGetLastError());
    return Status();
}

// behind: right after a kernel of the same call (see launch_behind)
template <bool TOPK>
Status launch_score(Ctx* c, int G, const ScoreArgs& a, uint32_t grid, int threads, size_t smem, bool behind) {
    switch (G) {
        case 1: return launch_score_t<1, TOPK>(c, a, grid, threads, smem, behind);
        case 2: return launch_score_t<2, TOPK>(c, a, grid, threads, smem, behind);
        default: return launch_score_t<4, TOPK>(c, a, grid, threads, smem, behind);
    }
}

int group_width(uint32_t nq) { return nq >= 3 ? 4 : (int)nq; }

// shared-memory candidate slots of the merge kernel for at most `total` candidates per query
// (k results wanted, kp2 = k rounded up to a power of two).  kp2 + k slots let the merge kernel order
// its winners by bucket placement next to them; more buys nothing: longer inputs go through the
// kernel's bucket pre-filter, which gathers only k plus one bucket of candidates, and a small buffer
// lets more CTAs share an SM.
uint32_t merge_cap(uint64_t total, uint32_t kp2, uint32_t k) {
    // (and room to order up to 1.5 k gathered keys next to themselves: the merge's sort-all path)
    const uint64_t enough = (std::max<uint64_t>((uint64_t)kp2 + k + 256, 2 * ((uint64_t)k + k / 2) + 512) + 255) / 256 * 256;
    return (uint32_t)std::min<uint64_t>(enough, 24576);
}
int merge_threads(uint32_t cap_s) { return cap_s > 4096 ? 512 : 256; }
size_t merge_smem(uint32_t cap_s, uint32_t kp2) {
    return (size_t)cap_s * 8 + 8 + (size_t)(std::max(SEL_HIST_INTS, merge_buckets(kp2, (uint32_t)merge_threads(cap_s)) + 48) + 4) * 4;
}

// Optional per-call CUDA-event timing of the two kernels of score_topk
// (slha_b200_timing_begin / _end).  Events are recorded on the launching stream.
struct Timing {
    std::vector<cudaEvent_t> ev;  // 3 per call: before score, after score, after merge
    uint32_t max_calls = 0, calls = 0;
};
thread_local Timing g_timing;

// Grow-only device buffer owned by a plan (kept when the plan object is recycled).
struct DevBuf {
    void* p = nullptr;
    size_t cap = 0;
    Status ensure(size_t need) {
        need = std::max<size_t>(need, 256);
        if (need <= cap) return Status();
        if (p) cudaFree(p);
        p = nullptr;
        cap = 0;
        const size_t want = need + need / 2;
        void* q = nullptr;
        SLHA_CUDA(cudaMalloc(&q, want));  // (on failure the buffer stays empty: p == nullptr, cap == 0)
        p = q;
        cap = want;
        return Status();
    }
    ~DevBuf() { cudaFree(p); }
};

// Several small host arrays in one upload.
struct Blob {
    std::vector<unsigned char> bytes;
    template <typename T>
    size_t add(const std::vector<T>& v) {
        const size_t at = (bytes.size() + 15) / 16 * 16;
        bytes.resize(at + v.size() * sizeof(T));
        if (!v.empty()) std::memcpy(bytes.data() + at, v.data(), v.size() * sizeof(T));
        return at;
    }
    size_t zeros = 0;  // words of zeros behind them (the last to be added)
    size_t add_zeros(size_t words) {
        zeros = words;
        return (bytes.size() + 15) / 16 * 16;
    }
};

// The cached decomposition of one score_topk call shape.
struct Plan {
    std::vector<unsigned char> key;
    int device = -1;
    uint32_t k = 0, cap = 0, kp2 = 0, nq = 0, n_lists = 0;
    int threads = 128;
    struct Class { int G; uint32_t first, count; };
    std::vector<Class> classes;
    WorkItem* d_items = nullptr;
    uint32_t* d_q_list_begin = nullptr;
    uint32_t* d_q_list_count = nullptr;
    uint64_t* d_cand_keys = nullptr;
    uint32_t* d_cand_cnt = nullptr;
    uint32_t* d_cta_begin = nullptr;  // tensor-core kernel: items [cta_begin[b], cta_begin[b+1]) belong to CTA b
    unsigned long long* d_gpivot = nullptr;  // per query: streaming top-k state (threshold, mapping, count, flag, histogram)
    uint64_t* d_gbuf = nullptr;              // per query: gcap candidate keys of the tensor-core kernel
    uint32_t gcap = 0;
    size_t gstate_bytes = 0;
    // Short shares (below 4096 tiles per CTA, ten rounds): the thresholds raised while scoring are stale or absent, and the compaction or
    // the merge takes the row's threshold from its complete histogram first.  Longer shares have just refreshed theirs: there the
    // extra read of the histogram cost 2 to 6 us of 55 to 100.
    bool late_threshold = false;
    bool state_clean = false;  // the previous call's merge left the streaming state cleared (see StreamLists::finish)
    uint32_t compact_splits = 0, selcap = 0;  // optional compaction pass before the merge (few rows, long buffers)
    // wide scoring (16 or more queries per segment, INT4 / TQ3 launches): work items of up to 64 query rows for score_wide_kernel
    bool wide = false, allow_wide_in = false;
    WorkItem* d_wide_items = nullptr;
    WorkItem* d_stream_items = nullptr;  // interleaved description of every CTA's work for score_stream_kernel (null: the work items themselves)
    uint32_t* d_wide_cta = nullptr;
    uint32_t wide_grid = 0, n_wide_items = 0;
    uint32_t n_items = 0;
    uint32_t max_parts = 1;  // most candidate lists any query has
    uint32_t list_cap = 0;   // slots per candidate list: k plus the slack the tensor-core kernel's last selection may leave
    bool use_mma = false;
    int kind = 3;            // 0 NF4, 1 mixed 8/4, 2 TQ3, 3 INT4, 4 MIX3
    int codec_hint_in = -1;
    bool force_generic_in = false;
    uint32_t mma_grid = 0;
    bool long_items = false; // score_stream_kernel's form for them
    int sets = 1;            // sub-sets of 16 tiles that a warp takes at a time
    DevBuf b_tables, b_keys, b_cnt, b_gpivot, b_gbuf, b_gsel, b_tmp;
    // Two-level merge for calls with few queries and many candidate lists per query (a pool scored
    // by one GQA group: 148 lists each): groups of `group_parts` lists are merged by a CTA each into
    // `n_groups` intermediate (index, score) lists per query, which a second launch merges.
    uint32_t n_groups = 0, group_parts = 0;
    uint32_t* d_vq_begin = nullptr;
    uint32_t* d_vq_count = nullptr;
    uint32_t* d_tmp_index = nullptr;
    float* d_tmp_score = nullptr;
    // Rows whose scores are written as a whole and selected from (score_select.cuh)
    bool rows = false, allow_rows_in = false;
    uint32_t longest = 0;
    uint64_t row_stride = 0;
    RowInfo* d_rows = nullptr;
    uint32_t* d_row_flags = nullptr;  // [nq] generic arithmetic, [nq] handed on by the 64-row kernel, [nq][2] statistics, whether any row was handed on
    WorkItem* d_streams = nullptr;    // of the pass over those, see Streams
    uint32_t n_streams = 0, streams_grid = 0;
    uint64_t last_use = 0;
    bool captured = false;  // a graph of the library's own names this plan's buffers (see plan_epoch)
};
thread_local Plan* g_last_plan = nullptr;    // of the thread's latest score_topk
thread_local uint32_t g_plans_recycled = 0;  // of this thread's captured plans
std::atomic<uint32_t> g_plan_threads{0};

// Cuts of (segment, group of up to `width` query rows) streams into one share per CTA.  `total`: in whole units of each stream, as the shares are filled (counted in
// tiles, 200 segments of 8128 made 149 CTAs, one of them behind all others: 136 us instead of 90).
struct Cuts {
    static uint64_t whole(uint64_t n, uint64_t unit) { return (n + unit - 1) / unit * unit; }
    std::vector<WorkItem> items;
    std::vector<uint32_t> cta{0u};
    uint64_t share = 0, filled = 0, unit;
    Cuts(uint64_t total, int sms, uint64_t unit_tiles, uint64_t least) : unit(unit_tiles) {
        share = (total + sms - 1) / sms;
        share = std::max<uint64_t>(least, whole(share, unit));
    }
    void add(const SlhaB200Segment& s, uint32_t width) {
        for (uint32_t q0 = 0; q0 < s.n_queries; q0 += width)
            for (uint64_t pos = 0; pos < s.n_tiles;) {
                const uint32_t take = (uint32_t)std::min<uint64_t>(s.n_tiles - pos, share - filled);
                WorkItem w{};
                w.tile_begin = s.tile_begin + pos;
                w.n_tiles = take;
                w.index_base = s.index_base + (uint32_t)pos;
                w.query_begin = s.query_begin + q0;
                w.n_queries = std::min<uint32_t>(width, s.n_queries - q0);
                items.push_back(w);
                pos += take;
                filled += whole(take, unit);  // (cuts lie at whole units of a segment)
                if (filled >= share) {
                    filled = 0;
                    cta.push_back((uint32_t)items.size());
                }
            }
    }
    void finish() {
        if (cta.back() != (uint32_t)items.size()) cta.push_back((uint32_t)items.size());
    }
};

// What the four-row kernel's pass behind the 64-row kernel is given (ScoreArgs::streams): that kernel's items put together to whole streams, or, where most are whole streams, the items
// themselves (`all` stays empty).
struct Streams {
    std::vector<WorkItem> all;
    uint32_t n = 0, grid = 0;
    // items: in the order of the streams, and of their tiles
    void make(const std::vector<WorkItem>& items, int sms) {
        auto goes_on = [&](size_t i) {
            if (i == 0) return false;
            const WorkItem &w = items[i], &v = items[i - 1];
            return w.query_begin == v.query_begin && w.n_queries == v.n_queries && w.tile_begin == v.tile_begin + v.n_tiles && w.index_base == v.index_base + v.n_tiles;
        };
        uint64_t blocks = 0;
        for (size_t i = 0; i < items.size(); ++i) {
            n += !goes_on(i);
            blocks += (uint64_t)((items[i].n_queries + 3) / 4) * ((items[i].n_tiles + 127u) / 128u);
        }
        grid = (uint32_t)std::min<uint64_t>(blocks, (uint64_t)sms);
        if (2 * (size_t)n > items.size()) {
            n = (uint32_t)items.size();
            return;
        }
        all.reserve(n);
        for (size_t i = 0; i < items.size(); ++i) {
            if (goes_on(i)) all.back().n_tiles += items[i].n_tiles;
            else all.push_back(items[i]);
        }
    }
};

// Whether a call's rows are scored as a whole (score_select.cuh) rather than streamed: rows of up to ROWS_MOST tiles, scores of 64 MB at most as they are laid out.  `passes`: tiles times
// groups of four query rows, `wide`: 16 rows or more a segment, which the 64-row kernel takes (512 rows of 16 384 TQ3 tiles, k = 256 85 -> 47 us; 1232 of
// 3553 MX tiles 111 -> 53).  Streaming reads a million tiles in 25 us where score_dense_kernel takes 40 (NF4 34, 59), but its set-up, first sets and compaction
// cost about 20 us a call, and appending and merging a row 0.04 (k = 64) to 0.08 us (k = 1024), which selecting from whole rows costs hardly: in pico-
// seconds, 16 a pass (NF4 30, both a little above what was measured) against 18 million a call and per_row a row.  us a call, whole / streamed, k = 64, 256, 1024:
//   64 segments of 16 384 INT4 tiles 51 / 63, 52 / 72, 60 / 90, TQ3 59 / 82, 60 / 95, 68 / 111, NF4 71 / 73, 71 / 86, 80 / 105; 128 of 16 384 INT4 88 / 94, 89 / 108, 106 / 124,
//   NF4 126 / 114, 127 / 122, 143 / 140; 48 of 32 768 INT4 76 / 72, 79 / 85, 86 / 103, NF4 105 / 87, 109 / 99, 116 / 117; 96 of 32 768 INT4 131 / 114, 135 / 133, 147 / 157,
//   mixed 129 / 124, 133 / 136, 144 / 157; 400 of 8192 INT4 141 / 165, 142 / 191, 181 / 234, NF4 201 / 186, 201 / 214, 241 / 256; 1000 of 4096 INT4 198 / 253,
//   200 / 308, 245 / 396, NF4 272 / 294, 273 / 369, 318 / 475.
// Up to 640 000 passes (1 280 000 from k = 512) whole rows are the faster ones however few they are: 19 x 32 768 tiles, one row each, k = 64, 1024 INT4 34 / 45, 37 / 78, NF4 45 / 47, 49 / 79;
// 38 x 32 768, k = 512, 1024 INT4 50 / 94, 52 / 107, NF4 71 / 111, 73 / 131.  (Above, at k = 64, INT4 67 streamed, NF4 74.)
enum RowsRule { ROWS_NO, ROWS_YES, ROWS_UNLESS_NF4 };
RowsRule rows_rule(uint64_t passes, bool wide, size_t nq, uint32_t longest, uint32_t k) {
    const uint64_t unit = wide ? WIDE_M : 32;  // (the 64-row kernel writes blocks of 128 scores)
    if (longest == 0 || longest > ROWS_MOST || nq * Cuts::whole(longest, unit) > (16ull << 20)) return ROWS_NO;
    if (wide || passes <= (k >= 512 ? 1280000 : 640000)) return ROWS_YES;
    const uint64_t saved = 18000000 + nq * (k >= 1024 ? 85000 : k >= 200 ? 75000 : k >= 32 ? 37000 : 25000);
    return 30 * passes <= saved ? ROWS_YES : 16 * passes <= saved ? ROWS_UNLESS_NF4 : ROWS_NO;
}

Status build_rows_plan(Ctx* c, Plan* p, const SlhaB200Segment* segs, size_t n_segs, size_t nq, uint32_t longest, bool allow_wide) {
    const int sms = sm_count(c->device);
    bool wide = true;
    uint64_t total = 0, wtotal = 0;
    std::vector<RowInfo> rows(nq, RowInfo{0u, 0u, 0u, 128u});
    std::vector<uint8_t> taken(nq, 0);
    for (size_t i = 0; i < n_segs; ++i) {
        const SlhaB200Segment& s = segs[i];
        if ((uint64_t)s.query_begin + s.n_queries > nq) return Status(SLHA_ERR_DIMENSION, "segment query range exceeds n_queries");
        for (uint32_t q = 0; q < s.n_queries; ++q) {
            if (taken[s.query_begin + q]) return Status(SLHA_ERR_DIMENSION, "a query row belongs to two segments");
            taken[s.query_begin + q] = s.n_tiles != 0;
            rows[s.query_begin + q] = RowInfo{s.n_tiles, s.index_base, 0u, 128u};
        }
        wide = wide && (s.n_queries >= 16 || s.n_tiles == 0);
        total += Cuts::whole(s.n_tiles, ST_M) * ((s.n_queries + 3) / 4);
        wtotal += Cuts::whole(s.n_tiles, WIDE_M) * ((s.n_queries + WIDE_NQ - 1) / WIDE_NQ);
    }
    wide = wide && allow_wide && wtotal;
    Cuts cuts(wide ? wtotal : total, sms, wide ? WIDE_M : ST_M, wide ? WIDE_M : ST_M);
    for (size_t i = 0; i < n_segs; ++i) {
        SlhaB200Segment s = segs[i];
        s.index_base = 0;  // (where the scores go: a place in the row)
        cuts.add(s, wide ? WIDE_NQ : 4);
    }
    cuts.finish();
    // Where the scores go: rows one behind the other, or where the 64-row kernel writes them, a block of 128 tiles' scores of all the item's rows together.
    p->row_stride = ((uint64_t)longest + 31) / 32 * 32;
    uint64_t floats = nq * p->row_stride;
    Streams streams;
    if (wide) {
        floats = 0;
        size_t at = 0;
        for (size_t i = 0; i < n_segs; ++i)
            for (uint32_t q0 = 0; q0 < segs[i].n_queries && segs[i].n_tiles; q0 += WIDE_NQ) {
                const uint32_t m = std::min<uint32_t>(WIDE_NQ, segs[i].n_queries - q0);
                for (uint32_t q = 0; q < m; ++q) {
                    rows[segs[i].query_begin + q0 + q].begin = (uint32_t)(floats + 128 * q);
                    rows[segs[i].query_begin + q0 + q].step = 128 * m;
                }
                for (uint64_t done = 0; done < segs[i].n_tiles; ++at) {  // (the cuts of this stream, in order)
                    cuts.items[at].list_begin = (uint32_t)floats;
                    cuts.items[at].pad = 128 * m;
                    done += cuts.items[at].n_tiles;
                }
                floats += (uint64_t)(segs[i].n_tiles + 127) / 128 * 128 * m;
            }
    } else {
        for (size_t q = 0; q < nq; ++q) rows[q].begin = (uint32_t)(q * p->row_stride);
    }
    if (wide) streams.make(cuts.items, sms);
    Blob tables;
    const size_t o_n = tables.add(cuts.items), o_nc = tables.add(cuts.cta), o_r = tables.add(rows), o_s = tables.add(streams.all);
    SLHA_TRY(p->b_tables.ensure(tables.bytes.size()));
    SLHA_TRY(p->b_gpivot.ensure((4 * nq + 1) * 4));
    SLHA_TRY(p->b_gbuf.ensure(floats * 4));
    unsigned char* dev = static_cast<unsigned char*>(p->b_tables.p);
    SLHA_TRY(ctx_copy_table(c, dev, tables.bytes.data(), tables.bytes.size()));
    p->d_row_flags = (uint32_t*)p->b_gpivot.p;
    SLHA_CUDA(cudaMemsetAsync(p->d_row_flags, 0, (4 * nq + 1) * 4, c->stream));
    p->d_items = reinterpret_cast<WorkItem*>(dev + o_n);
    p->wide = wide;
    p->n_items = (uint32_t)cuts.items.size();
    p->mma_grid = (uint32_t)cuts.cta.size() - 1;
    p->d_cta_begin = !wide && p->n_items == p->mma_grid ? nullptr : reinterpret_cast<uint32_t*>(dev + o_nc);  // (null: an item a CTA)
    p->d_rows = reinterpret_cast<RowInfo*>(dev + o_r);
    p->d_streams = streams.all.empty() ? p->d_items : reinterpret_cast<WorkItem*>(dev + o_s);
    p->n_streams = streams.n;
    p->streams_grid = streams.grid;
    p->longest = longest;
    p->rows = true;
    return Status();
}

Status build_plan(Ctx* c, const SciRustSlhaTile* tiles, const SlhaB200Segment* segs, size_t n_segs, size_t nq,
                  uint32_t k, int codec_hint, bool allow_wide, bool allow_rows, Plan** out) {
    std::vector<unsigned char> key(sizeof(SlhaB200Segment) * n_segs + 16);
    std::memcpy(key.data(), segs, sizeof(SlhaB200Segment) * n_segs);
    uint64_t nq64 = nq;
    std::memcpy(key.data() + sizeof(SlhaB200Segment) * n_segs, &nq64, 8);
    std::memcpy(key.data() + sizeof(SlhaB200Segment) * n_segs + 8, &k, 4);
    // small per-thread cache of plans (call shapes alternate in practice: appends
    // change a pool's length, layers differ); a recycled plan keeps its device buffers
    static thread_local std::vector<std::unique_ptr<Plan>> cache;
    static thread_local uint64_t tick = 0;
    ++tick;
    for (auto& e : cache)
        if (e->device == c->device && e->codec_hint_in == codec_hint && e->force_generic_in == g_force_generic && e->allow_wide_in == allow_wide && e->allow_rows_in == allow_rows && e->key == key) {
            e->last_use = tick;
            *out = e.get();
            return Status();
        }
    SLHA_TRY(ctx_no_capture(c));  // (a new plan has tables to copy)
    Plan* p;
    if (cache.size() < 4) {
        cache.push_back(std::make_unique<Plan>());
        p = cache.back().get();
    } else {
        p = cache[0].get();
        for (auto& e : cache)
            if (e->last_use < p->last_use) p = e.get();
        if (p->captured) ++g_plans_recycled;
        p->captured = false;
        p->classes.clear();
        p->max_parts = 1;
    }
    // The plan is published (key + device set) only once it is complete: any early return
    // below leaves a slot that no later call can match.
    p->key.clear();
    p->device = -1;
    p->last_use = tick;
    p->codec_hint_in = codec_hint;
    p->force_generic_in = g_force_generic;
    p->allow_wide_in = allow_wide;
    p->allow_rows_in = allow_rows;
    p->wide = p->rows = false;
    p->k = k;
    p->n_lists = 0;
    p->nq = (uint32_t)nq;
    p->kp2 = 2;
    while (p->kp2 < k) p->kp2 <<= 1;
    // Codec hint: -1 = the flags of the first tile of the first non-empty segment decide which kind of tile a streaming launch
    // decodes.  A wrong hint costs speed only (tiles of another kind are handed to the generic kernel).
    auto look = [&]() -> Status {
        p->kind = codec_hint < 0 ? 3 : hint_kind(codec_hint);
        for (size_t i = 0; i < n_segs && codec_hint < 0; ++i)
            if (segs[i].n_tiles) {
                uint16_t flags = 0;
                const unsigned char* t0 = reinterpret_cast<const unsigned char*>(tiles) + segs[i].tile_begin * TILE_BYTES;
                SLHA_CUDA(cudaMemcpyAsync(&flags, t0 + 118, 2, cudaMemcpyDeviceToHost, c->stream));
                SLHA_CUDA(cudaStreamSynchronize(c->stream));
                p->kind = stream_kind(flags);
                break;
            }
        return Status();
    };
    bool looked = false;
    if (allow_rows && !g_force_generic) {
        uint32_t longest = 0;
        uint64_t passes = 0;
        bool wide = true;
        for (size_t i = 0; i < n_segs; ++i) {
            if (segs[i].n_queries) longest = std::max(longest, segs[i].n_tiles);
            wide = wide && (segs[i].n_queries >= 16 || segs[i].n_tiles == 0);
            passes += (uint64_t)segs[i].n_tiles * ((segs[i].n_queries + 3) / 4);
        }
        // The 64-row kernel hands NF4 tiles on to score_dense_kernel, so whether they had better be streamed has to be known first, where the rule for four rows says so (250 NF4 rows on 32 768
        // tiles, k = 16 100 us a call, 130 whole).  Elsewhere nobody looks: a new shape of other tiles would wait 18 us for what saves 5 of 34 on NF4 (64 rows on each of 4 x 3000).
        wide = wide && allow_wide;
        RowsRule rule = rows_rule(passes, wide, nq, longest, k);
        if (rule == ROWS_UNLESS_NF4 || (rule == ROWS_YES && wide && rows_rule(passes, false, nq, longest, k) != ROWS_YES)) {
            SLHA_TRY(look());
            looked = true;
            rule = p->kind == 0 ? ROWS_NO : ROWS_YES;
        }
        if (rule == ROWS_YES) {
            SLHA_TRY(build_rows_plan(c, p, segs, n_segs, nq, longest, wide));
            p->use_mma = true;
            p->key = std::move(key);
            p->device = c->device;
            *out = p;
            return Status();
        }
    }
    p->threads = k > 1024 ? 256 : 128;
    const int nwarps = p->threads / 32;
    const uint32_t round = (uint32_t)nwarps * BLK_TILES;
    uint32_t cap = std::max<uint32_t>(2 * k, k + 2 * round);
    while (cap > k + round && score_smem_bytes(4, nwarps, true, cap) > MAX_SMEM) cap -= round;
    if (score_smem_bytes(4, nwarps, true, cap) > MAX_SMEM || (size_t)p->kp2 * 8 + 2048 > MAX_SMEM)
        return Status(SLHA_ERR_CAPACITY, "top-k: k is too large for the shared-memory selection state");
    p->cap = cap;

    // tensor-core kernel: one persistent CTA per SM
    const int sms = sm_count(c->device);
    {
        if (!looked) SLHA_TRY(look());
        p->use_mma = !g_force_generic;
        p->mma_grid = (uint32_t)sms;
    }
    const uint32_t st_unit = p->kind == 4 ? (uint32_t)ST_M : (uint32_t)MMA_SET_TILES;

    // Work items.  Generic kernel: fixed-size runs, large enough that candidate
    // traffic stays a few percent of the tile stream and small enough to balance
    // the SMs through the hardware CTA scheduler.  Tensor-core kernel: the
    // concatenated tile stream is cut into one equal share per persistent CTA
    // (and at segment ends), so per-item costs are paid once per ~total/grid tiles.
    uint64_t total = 0;
    size_t streams = 0;  // (segment, group of up to four query rows)
    for (size_t i = 0; i < n_segs; ++i) {
        const size_t groups = (segs[i].n_queries + 3) / 4;
        total += (uint64_t)segs[i].n_tiles * groups;
        streams += segs[i].n_tiles ? groups : 0;
    }
    uint32_t item_tiles = std::max<uint32_t>(8192, 8 * k);
    while (item_tiles > 2048 && total / item_tiles < 592) item_tiles /= 2;
    item_tiles = std::max(round, (item_tiles + round - 1) / round * round);
    uint64_t share = (total + p->mma_grid - 1) / std::max<uint32_t>(p->mma_grid, 1);
    share = std::max<uint64_t>(STREAM_LEAST, (share + st_unit - 1) / st_unit * st_unit);
    const uint64_t snap = std::min<uint64_t>(share / 16, 2048);
    uint64_t spare = share * std::max<uint32_t>(p->mma_grid, 1) > total ? share * std::max<uint32_t>(p->mma_grid, 1) - total : 0;  // room the equal shares leave
    uint64_t filled = 0;  // tiles already given to the current CTA (tensor-core mode)
    std::vector<uint32_t> cta_begin(1, 0);
    // Few long streams (a stream = one segment's tiles for one group of up to four query rows; at most half as many as
    // there are CTAs): every stream gets whole CTAs in proportion to its tiles, and the CTAs of a stream take its tiles
    // interleaved -- CTA c of C takes the 24-set chunks c, c + C, c + 2 C .. -- instead of one contiguous range each.
    // Equal ranges are not equal work: where the scores are high (recent tokens) a CTA appends far more candidates, and
    // the CTA with the densest range ended 13 us after the median one; interleaved, every CTA sees the same mix.  The
    // work items below stay contiguous ranges (one per CTA): they are what the generic kernel scores when a row is
    // handed back; the tensor-core kernel reads the interleaved description of the same CTA from `stream_items`.
    std::vector<uint32_t> stream_ctas;
    std::vector<WorkItem> stream_items;
    if (p->use_mma && total > 0) {
        std::vector<uint64_t> st_tiles;
        for (size_t i = 0; i < n_segs; ++i)
            for (uint32_t q0 = 0; q0 < segs[i].n_queries; q0 += 4)
                if (segs[i].n_tiles) st_tiles.push_back(segs[i].n_tiles);
        // Only for short shares (less than 20 000 tiles per CTA: shards of a long context, measured at 7 k and 14 k tiles
        // per CTA): with whole CTAs per stream the streams' CTA counts differ by one (18 or 19 of 148 for eight streams),
        // which costs the slower streams 5 % -- less than the second set-up of a CTA that works on two streams when a
        // share lasts 40 us, more when it lasts 200 us.
        if (!st_tiles.empty() && st_tiles.size() * 2 <= p->mma_grid && total / p->mma_grid < 20000) {
            stream_ctas.resize(st_tiles.size());
            uint32_t used = 0;
            for (size_t j = 0; j < st_tiles.size(); ++j) {
                const uint64_t most = (st_tiles[j] + STREAM_LEAST - 1) / STREAM_LEAST;
                stream_ctas[j] = (uint32_t)std::max<uint64_t>(1, std::min<uint64_t>(most, st_tiles[j] * p->mma_grid / total));
                used += stream_ctas[j];
            }
            while (used < p->mma_grid) {  // the CTAs left over go where a CTA has the most tiles
                size_t best = st_tiles.size();
                uint64_t worst = 0;
                for (size_t j = 0; j < st_tiles.size(); ++j) {
                    const uint64_t per = st_tiles[j] / stream_ctas[j];
                    if (per > worst && (uint64_t)stream_ctas[j] < (st_tiles[j] + STREAM_LEAST - 1) / STREAM_LEAST) { worst = per; best = j; }
                }
                if (best == st_tiles.size()) break;
                ++stream_ctas[best];
                ++used;
            }
        }
    }
    size_t stream_no = 0;

    std::vector<WorkItem> items[3];  // by class G = 1, 2, 4 (generic mode); all in [2] in tensor-core mode
    std::vector<uint32_t> q_begin(nq, 0), q_count(nq, 0);
    uint32_t n_lists = 0;
    for (size_t i = 0; i < n_segs; ++i) {
        const SlhaB200Segment& s = segs[i];
        if ((uint64_t)s.query_begin + s.n_queries > nq)
            return Status(SLHA_ERR_DIMENSION, "segment query range exceeds n_queries");
        for (uint32_t q0 = 0; q0 < s.n_queries; q0 += 4) {
            const uint32_t gq = std::min<uint32_t>(4, s.n_queries - q0);
            const int G = group_width(gq);
            // cut points of this (segment, query group) stream
            std::vector<std::pair<uint32_t, uint32_t>> cuts;  // (offset, length)
            if (!stream_ctas.empty() && s.n_tiles) {
                uint32_t ctas = stream_ctas[stream_no++];
                const uint32_t per = (uint32_t)(((uint64_t)s.n_tiles + ctas - 1) / ctas + st_unit - 1) / st_unit * st_unit;
                ctas = (s.n_tiles + per - 1) / per;  // (rounding to whole sets can leave the last CTA nothing)
                for (uint32_t part = 0; part < ctas; ++part) {
                    cuts.push_back({part * per, std::min<uint32_t>(per, s.n_tiles - part * per)});
                    cta_begin.push_back((uint32_t)items[2].size() + (uint32_t)cuts.size());
                    WorkItem w{};
                    w.tile_begin = s.tile_begin;
                    w.n_tiles = s.n_tiles;
                    w.index_base = s.index_base;
                    w.query_begin = s.query_begin + q0;
                    w.n_queries = gq;
                    w.list_begin = part;                              // this CTA's place among the stream's CTAs
                    w.pad = gq | (ctas << 8) | 0x80000000u;           // their number; bit 31: interleaved
                    stream_items.push_back(w);
                }
            }
            for (uint32_t pos = 0; stream_ctas.empty() && pos < s.n_tiles;) {
                uint32_t take;
                if (p->use_mma) {
                    // A work item costs its set-up and first set (several microseconds) whatever its length, so cuts that
                    // would leave a sliver are moved to the segment's end: a CTA with little room left does not start the
                    // next segment, and a cut that would leave a short rest of a segment takes the rest along.
                    if (pos == 0 && filled > 0 && share - filled < snap && spare >= share - filled) {
                        spare -= share - filled;  // (the grid must not grow beyond one CTA per SM)
                        filled = 0;
                        cta_begin.push_back((uint32_t)items[2].size() + (uint32_t)cuts.size());
                    }
                    take = (uint32_t)std::min<uint64_t>(s.n_tiles - pos, share - filled);
                    const uint32_t rest = s.n_tiles - pos - take;
                    if (rest > 0 && rest < snap) {
                        take += rest;
                        spare += rest;
                    }
                    filled += take;
                } else {
                    take = std::min<uint32_t>(item_tiles, s.n_tiles - pos);
                }
                cuts.push_back({pos, take});
                pos += take;
                if (p->use_mma && filled >= share) {
                    filled = 0;
                    cta_begin.push_back((uint32_t)items[2].size() + (uint32_t)cuts.size());
                }
            }
            const uint32_t parts = (uint32_t)cuts.size();
            p->max_parts = std::max(p->max_parts, parts);
            for (uint32_t g = 0; g < gq; ++g) {
                const uint32_t Q = s.query_begin + q0 + g;
                if (q_count[Q]) return Status(SLHA_ERR_DIMENSION, "a query row belongs to two segments");
                q_begin[Q] = n_lists + g;  // lists of one item are consecutive: stride gq per part
                q_count[Q] = parts;
            }
            for (uint32_t part = 0; part < parts; ++part) {
                WorkItem w;
                w.tile_begin = s.tile_begin + cuts[part].first;
                w.n_tiles = cuts[part].second;
                w.index_base = s.index_base + cuts[part].first;
                w.query_begin = s.query_begin + q0;
                w.n_queries = gq;
                w.list_begin = n_lists + part * gq;
                w.pad = gq | (std::min<uint32_t>(parts, 0xFFFFFFu) << 8);  // low byte: list stride between parts (merge accessor); above: parts of the row group
                items[p->use_mma ? 2 : (G == 1 ? 0 : (G == 2 ? 1 : 2))].push_back(w);
            }
            n_lists += parts * gq;
        }
    }
    p->n_lists = n_lists;
    std::vector<WorkItem> all;
    for (int cls = 0; cls < 3; ++cls) {
        if (items[cls].empty()) continue;
        p->classes.push_back({cls == 0 ? 1 : (cls == 1 ? 2 : 4), (uint32_t)all.size(), (uint32_t)items[cls].size()});
        all.insert(all.end(), items[cls].begin(), items[cls].end());
    }
    if (cta_begin.back() != (uint32_t)all.size()) cta_begin.push_back((uint32_t)all.size());
    if (all.empty()) p->use_mma = false;
    p->mma_grid = (uint32_t)cta_begin.size() - 1;
    // per query: list id of part p is q_begin + p * stride; store stride in the count's high bits
    std::vector<uint32_t> q_stride(nq, 1);
    for (const WorkItem& w : all)
        for (uint32_t g = 0; g < w.n_queries; ++g) q_stride[w.query_begin + g] = w.pad & 0xFFu;
    if (!stream_items.empty() && stream_items.size() != all.size()) return Status(SLHA_ERR_PANIC, "score plan: stream items out of step");
    p->list_cap = (k + std::max<uint32_t>(64, k / 2) + 31) / 32 * 32;
    SLHA_TRY(p->b_keys.ensure((size_t)n_lists * p->list_cap * 8));
    SLHA_TRY(p->b_cnt.ensure((size_t)n_lists * 4));
    // Wide scoring: every segment brings 16 or more queries and the launch holds INT4 / MX-INT4 or TQ3 tiles.  Work items
    // of up to 64 query rows; the (segment, row group) streams are cut into one share per CTA, in whole 128-tile blocks.
    uint32_t wide_parts = 1;
    std::vector<WorkItem> wi;
    std::vector<uint32_t> wcta;
    {
        bool all_wide = p->use_mma && allow_wide && n_segs > 0 && p->kind != 0;
        uint64_t wtotal = 0;
        for (size_t i = 0; i < n_segs && all_wide; ++i) {
            all_wide = segs[i].n_queries >= 16 || segs[i].n_tiles == 0;
            wtotal += (uint64_t)segs[i].n_tiles * ((segs[i].n_queries + WIDE_NQ - 1) / WIDE_NQ);
        }
        if (all_wide && wtotal > 0) {
            uint64_t wshare = (wtotal + sms - 1) / sms;
            wshare = std::max<uint64_t>(WIDE_M, (wshare + WIDE_M - 1) / WIDE_M * WIDE_M);
            wcta.push_back(0);
            uint64_t wfilled = 0;
            for (size_t i = 0; i < n_segs; ++i) {
                const SlhaB200Segment& s = segs[i];
                for (uint32_t q0 = 0; q0 < s.n_queries; q0 += WIDE_NQ) {
                    uint32_t parts = 0;
                    for (uint32_t pos = 0; pos < s.n_tiles;) {
                        const uint32_t take = (uint32_t)std::min<uint64_t>(s.n_tiles - pos, wshare - wfilled);
                        WorkItem w{};
                        w.tile_begin = s.tile_begin + pos;
                        w.n_tiles = take;
                        w.index_base = s.index_base + pos;
                        w.query_begin = s.query_begin + q0;
                        w.n_queries = std::min<uint32_t>(WIDE_NQ, s.n_queries - q0);
                        wi.push_back(w);
                        ++parts;
                        pos += take;
                        wfilled += take;
                        if (wfilled >= wshare) {
                            wfilled = 0;
                            wcta.push_back((uint32_t)wi.size());
                        }
                    }
                    wide_parts = std::max(wide_parts, parts);
                }
            }
            if (wcta.back() != (uint32_t)wi.size()) wcta.push_back((uint32_t)wi.size());
            p->n_wide_items = (uint32_t)wi.size();
            p->wide_grid = (uint32_t)wcta.size() - 1;
            p->wide = true;
        }
    }
    // Streaming top-k state per query row: threshold, bucket mapping, count, flag, 256 bucket counts; and
    // the row's candidate buffer.  In random order about k (1 + ln(n / k)) tiles pass the rising threshold
    // plus the unfiltered first sets of every warp; 16 k slots (at most the longest segment) leave a wide
    // margin, and a row that fills its buffer all the same is scored by the generic kernel.
    // (a warp reserves slots in chunks of up to the tiles it takes at a time, so up to that many per warp and item stay unused)
    uint32_t longest = 0;
    for (size_t i = 0; i < n_segs; ++i) longest = std::max(longest, segs[i].n_tiles);
    p->long_items = stream_long(p->kind, !stream_items.empty(), total / std::max<size_t>(all.size(), 1), total / std::max<size_t>(streams, 1), k);
    p->sets = stream_sets(p->kind, p->long_items);
    const uint32_t st_warps = stream_warps(p->kind), st_tiles = stream_warp_tiles(p->kind, p->sets);
    const uint64_t all_of_a_row = (uint64_t)longest + (uint64_t)st_tiles * st_warps * p->max_parts + 64;
    // (the first set of every warp that scans a row is appended unfiltered: its tiles per warp and item, twice over)
    const uint64_t first_sets = (uint64_t)(2 * st_tiles) * st_warps * p->max_parts;
    uint32_t expect = (uint32_t)std::min<uint64_t>(std::max<uint64_t>(std::max<uint64_t>(16ull * k, 4096), first_sets + 4ull * k), all_of_a_row / 64 * 64);
    // Scores that rise along a long segment bring more (18 to 23 k slots for k = 1024 of 524 288 mixed tiles, 16 k + 10 % of which sent four of
    // 32 rows to the generic kernel: 1860 us instead of 184), so rows have up to 64 k slots where all rows' together stay within 64 MB.
    p->gcap = (uint32_t)std::min<uint64_t>(std::max<uint64_t>(expect, std::min<uint64_t>(65536, (8ull << 20) / nq)), all_of_a_row / 64 * 64);
    // (wide scoring: the first 128-tile block of every item is appended unfiltered, and a CTA sees few blocks)
    if (p->wide) p->gcap = expect = (uint32_t)std::min<uint64_t>(std::max<uint64_t>(expect, 4ull * WIDE_M * wide_parts + 16ull * k), ((uint64_t)longest + 63) / 64 * 64);
    p->gstate_bytes = nq * (1024 + 8 + 8 + 4 + 4 + 4 + 8);  // histogram, threshold, mapping, count, flag, compacted count, statistics
    p->state_clean = false;
    p->late_threshold = p->use_mma && total / (uint64_t)sms < 4096;
    // few rows with long buffers: several CTAs per row compact the survivors before the merge
    // (a slice of at most 1024 slots per CTA: one round of four keys per thread)
    // (up to 256 rows: 128 rows of 15 k MIX3 tiles 69.4 -> 65.0 us, 160 rows of 30 000 INT4 tiles 86.9 -> 82.2; with 1024 rows of 32 768 NF4 tiles the
    // merge's own CTAs fill the GPU and the extra pass costs 28 us of 441; rows of the 64-row kernel are short: 512 of them 10 of 85, 192 7 of 133)
    p->compact_splits = (p->use_mma && (nq < 128 || (nq <= 256 && !p->wide)) && expect >= 8192) ? (uint32_t)std::min<size_t>(64, std::max<size_t>((296 + nq - 1) / nq, (expect + 1023) / 1024)) : 0;
    p->selcap = merge_cap((uint64_t)p->gcap, p->kp2, k);
    if (p->compact_splits) SLHA_TRY(p->b_gsel.ensure(nq * (size_t)p->selcap * 8));
    SLHA_TRY(p->b_gpivot.ensure(p->gstate_bytes));
    if (p->use_mma) SLHA_TRY(p->b_gbuf.ensure(nq * (size_t)p->gcap * 8));
    p->d_gbuf = (uint64_t*)p->b_gbuf.p;
    p->d_cand_keys = (uint64_t*)p->b_keys.p;
    p->d_cand_cnt = (uint32_t*)p->b_cnt.p;
    p->d_gpivot = (unsigned long long*)p->b_gpivot.p;
    p->n_items = (uint32_t)all.size();
    p->n_groups = 0;
    std::vector<uint32_t> vq;
    if (nq <= 64 && p->max_parts >= 24 && !p->use_mma) {
        uint32_t G = 1;
        while (G * G < p->max_parts) ++G;
        const uint32_t ng = (p->max_parts + G - 1) / G;
        vq.resize(2 * (size_t)ng * nq);
        for (uint32_t g = 0; g < ng; ++g)
            for (size_t Q = 0; Q < nq; ++Q) {
                const uint32_t parts = q_count[Q], lo = g * G;
                vq[g * nq + Q] = q_begin[Q] + lo * q_stride[Q];
                vq[(size_t)ng * nq + g * nq + Q] = (parts > lo ? std::min(G, parts - lo) : 0u) | (q_stride[Q] << 24);
            }
        SLHA_TRY(p->b_tmp.ensure((size_t)ng * nq * k * 8));
        p->d_tmp_index = (uint32_t*)p->b_tmp.p;
        p->d_tmp_score = reinterpret_cast<float*>(p->d_tmp_index + (size_t)ng * nq * k);
        p->n_groups = ng;
        p->group_parts = G;
    }
    for (size_t Q = 0; Q < nq; ++Q) q_count[Q] |= q_stride[Q] << 24;
    Blob tables;
    const size_t o_items = tables.add(all), o_stream = tables.add(stream_items), o_cta = tables.add(cta_begin), o_qb = tables.add(q_begin), o_qc = tables.add(q_count);
    const size_t o_vq = tables.add(vq), o_wi = tables.add(wi), o_wcta = tables.add(wcta);
    SLHA_TRY(p->b_tables.ensure(tables.bytes.size()));
    unsigned char* dev = static_cast<unsigned char*>(p->b_tables.p);
    SLHA_TRY(ctx_copy_table(c, dev, tables.bytes.data(), tables.bytes.size()));
    p->d_items = reinterpret_cast<WorkItem*>(dev + o_items);
    p->d_stream_items = stream_items.empty() ? nullptr : reinterpret_cast<WorkItem*>(dev + o_stream);
    p->d_cta_begin = reinterpret_cast<uint32_t*>(dev + o_cta);
    p->d_q_list_begin = reinterpret_cast<uint32_t*>(dev + o_qb);
    p->d_q_list_count = reinterpret_cast<uint32_t*>(dev + o_qc);
    p->d_vq_begin = reinterpret_cast<uint32_t*>(dev + o_vq);
    p->d_vq_count = p->d_vq_begin + vq.size() / 2;
    p->d_wide_items = reinterpret_cast<WorkItem*>(dev + o_wi);
    p->d_wide_cta = reinterpret_cast<uint32_t*>(dev + o_wcta);
    p->key = std::move(key);
    p->device = c->device;
    *out = p;
    return Status();
}

}  // namespace

namespace {
// slha-c/src/lib.rs:244-286 per tile; status = min over bad tiles of (index << 8 | -code)
__global__ void validate_tiles_kernel(const unsigned char* tiles, uint64_t n, unsigned long long* status) {
    const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const unsigned char* t = tiles + i * TILE_BYTES;
    const uint32_t flags = *reinterpret_cast<const uint16_t*>(t + 118);
    const float sc = *reinterpret_cast<const float*>(t + 96), lam = *reinterpret_cast<const float*>(t + 100),
                sg = *reinterpret_cast<const float*>(t + 104);
    int code = 0;
    if (flags & ~0x3Fu) code = 6;
    else if (__popc(flags & (F_NF4 | F_MIXED | F_TQ3 | F_MIX3)) > 1) code = 6;
    else if ((flags & F_NOCORR) && !(flags & (F_TQ3 | F_MIX3))) code = 6;
    else if (!isfinite(sc) || !isfinite(lam) || !isfinite(sg)) code = 5;
    else if (sc < 0.0f || lam < 0.0f || sg < 0.0f) code = 6;
    if (code) atomicMin(status, (unsigned long long)((i << 8) | (uint64_t)code));
}
}  // namespace

Status launch_validate_tiles(Ctx* c, const SciRustSlhaTile* tiles, size_t n, unsigned long long* d_status) {
    if (n == 0) return Status();
    validate_tiles_kernel<<<(uint32_t)((n + 255) / 256), 256, 0, c->stream>>>(
        reinterpret_cast<const unsigned char*>(tiles), n, d_status);
    count_launch();
    SLHA_CUDA(cudaGetLastError());
    return Status();
}

// What a dense call brings from the host, in a kernel's parameters: its tables, copied to `dst`, and with them the check of row offsets in device
// memory (block 0).  An upload between two kernels cost 8 us (8 x 32 768 tiles x 64 rows 57 us a call, now 50).
template <int BYTES>
struct TableParam {
    uint4 w[BYTES / 16];
};
constexpr uint32_t TABLE_SLICE = 2048;  // bytes a block copies (parameters are read one address at a time)
template <int BYTES>
__global__ void __launch_bounds__(256) table_kernel(const __grid_constant__ TableParam<BYTES> table, uint32_t n16, uint32_t with_zeros, uint4* dst, const uint64_t* offsets, uint32_t nq, uint64_t scores_len,
                                                    uint32_t row_len, uint64_t* copy, uint32_t* refused, uint32_t* answer, uint32_t check_no) {
    dep_launch();
    dep_wait();
    const uint32_t i = blockIdx.x * (TABLE_SLICE / 16) + threadIdx.x;
    if (threadIdx.x < TABLE_SLICE / 16 && i < with_zeros) dst[i] = i < n16 ? table.w[i] : make_uint4(0u, 0u, 0u, 0u);
    if (blockIdx.x || !offsets) return;
    bool bad = false;
    for (uint32_t q = threadIdx.x; q < nq; q += blockDim.x) {
        const uint64_t o = offsets[q];
        copy[q] = o;
        bad |= o > scores_len || row_len > scores_len - o;
    }
    bad = __syncthreads_or(bad) != 0;
    if (threadIdx.x == 0) {
        *refused = bad;
        *reinterpret_cast<volatile uint32_t*>(answer) = 2u * check_no + bad;  // (page-locked host memory)
    }
}
constexpr uint32_t ANSWERS = 16;  // words that checks answer in, in turn: one of a call that ended early may still write
thread_local uint32_t g_check_no = 0;
template <int BYTES>
Status launch_table_t(Ctx* c, const Blob& blob, uint4* dst, const uint64_t* offsets, uint32_t nq, uint64_t scores_len, uint32_t row_len, uint64_t* copy, uint32_t* refused, uint32_t* answer,
                      uint32_t check_no) {
    static thread_local TableParam<BYTES> table;
    std::memcpy(&table, blob.bytes.data(), blob.bytes.size());
    const uint32_t n16 = (uint32_t)((blob.bytes.size() + 15) / 16), with_zeros = n16 + (uint32_t)((blob.zeros + 3) / 4);
    const uint32_t blocks = std::max<uint32_t>(1, (uint32_t)(((uint64_t)with_zeros * 16 + TABLE_SLICE - 1) / TABLE_SLICE));
    SLHA_CUDA(launch_behind(table_kernel<BYTES>, dim3(blocks), dim3(256), 0, c->stream, table, n16, with_zeros, dst, offsets, nq, scores_len, row_len, copy, refused, answer, check_no));
    count_launch();
    return Status();
}
// The call's tables to the device (*dev), and the check of `check`'s offsets, if any, with them.
Status send_tables(Ctx* c, Blob& blob, unsigned char** dev, RowCheck* check) {
    SLHA_TRY(ctx_no_capture(c));
    const bool in_params = blob.bytes.size() <= 16384;
    uint64_t* copy = nullptr;
    uint32_t *refused = nullptr, *answer = nullptr, no = 0;
    if (check) {
        if (check->nq > 0xFFFFFFFFull) return Status(SLHA_ERR_DIMENSION, "too many query rows");
        void* mem;
        SLHA_TRY(ctx_device_scratch(c, check->nq * 8 + 8, &mem));
        SLHA_TRY(ctx_answer(c, &check->host, &answer, &check->open));
        g_check_no = g_check_no % 0x7FFFFFFFu + 1u;
        check->no = no = g_check_no;
        check->host += no % ANSWERS;
        answer += no % ANSWERS;
        copy = static_cast<uint64_t*>(mem);
        refused = reinterpret_cast<uint32_t*>(copy + check->nq);
    }
    const uint64_t* offsets = check ? check->offsets : nullptr;
    const uint32_t nq = check ? (uint32_t)check->nq : 0u, row_len = check ? check->row_len : 0u;
    const uint64_t len = check ? check->scores_len : 0ull;
    if (!in_params) blob.bytes.resize((blob.bytes.size() + 15) / 16 * 16 + 4 * blob.zeros);  // (uploaded with the rest)
    if (in_params && !blob.bytes.empty()) SLHA_TRY(ctx_device_scratch(c, (blob.bytes.size() + 15) / 16 * 16 + (blob.zeros + 3) / 4 * 16, (void**)dev));
    else if (!blob.bytes.empty()) SLHA_TRY(ctx_upload(c, blob.bytes.data(), blob.bytes.size(), (void**)dev));
    uint4* dst = in_params ? reinterpret_cast<uint4*>(*dev) : nullptr;
    static const Blob none;
    const Blob& sent = in_params ? blob : none;
    if (in_params || check) {
        if (sent.bytes.size() <= 2048) SLHA_TRY(launch_table_t<2048>(c, sent, dst, offsets, nq, len, row_len, copy, refused, answer, no));
        else if (sent.bytes.size() <= 6144) SLHA_TRY(launch_table_t<6144>(c, sent, dst, offsets, nq, len, row_len, copy, refused, answer, no));
        else SLHA_TRY(launch_table_t<16384>(c, sent, dst, offsets, nq, len, row_len, copy, refused, answer, no));
    }
    if (check) {
        *check->open = check->launched = true;
        check->copy = copy;
        check->refused = refused;
    }
    return Status();
}
Status launch_row_check(Ctx* c, RowCheck* check) {
    unsigned char* dev = nullptr;
    Blob none;
    return send_tables(c, none, &dev, check);
}
// (The host polls the word: recording an event and waiting for it cost 3 us of a call of 17.)
Status checked_offsets(Ctx* c, RowCheck& check, bool* refused) {
    for (uint32_t i = 0; (*check.host >> 1) != check.no; ++i) {
        if (i % 4096 != 4095) continue;
        const cudaError_t e = cudaStreamQuery(c->stream);
        if (e == cudaErrorNotReady) continue;
        SLHA_CUDA(e);
        uint32_t word = 0;  // the stream is idle: the kernel's own word
        SLHA_CUDA(cudaMemcpyAsync(&word, check.refused, 4, cudaMemcpyDeviceToHost, c->stream));
        SLHA_CUDA(cudaStreamSynchronize(c->stream));
        *refused = word != 0;
        *check.open = false;
        return Status();
    }
    *refused = (*check.host & 1u) != 0;
    *check.open = false;
    return Status();
}

Status launch_score_full(Ctx* c, const SciRustSlhaTile* tiles, const uint8_t* state, size_t n,
                         const float* q_coarse, const uint64_t* q_sign, size_t nq, float* scores, int codec_hint) {
    if (n == 0 || nq == 0) return Status();
    // Long arenas: the streaming tensor-core kernel in its dense mode (all query groups of four in one launch, every CTA an
    // equal share of the tiles).  codec_hint -2: codecs the tensor-core kernel does not decode together;
    // bit 0: NF4 tiles beside INT4 ones; -1: not known.
    if (n >= 32768 && n < 0xFFFFFFFFull && codec_hint != -2 && !g_force_generic) {
        const int sms = sm_count(c->device);
        Cuts cuts(Cuts::whole(n, ST_M) * ((nq + 3) / 4), sms, ST_M, 2048);
        cuts.add(SlhaB200Segment{0, (uint32_t)n, 0, (uint32_t)nq, 0}, 4);
        cuts.finish();
        Blob blob;
        const size_t o_items = blob.add(cuts.items), o_cta = blob.add(cuts.cta);
        unsigned char* dev;
        SLHA_TRY(send_tables(c, blob, &dev, nullptr));
        ScoreArgs a{};
        a.cold_bits = 0xFF800000u;
        a.tiles = reinterpret_cast<const unsigned char*>(tiles);
        a.state = state;
        a.items = a.stream_items = reinterpret_cast<const WorkItem*>(dev + o_items);
        a.n_items = (uint32_t)cuts.items.size();
        a.cta_begin = cuts.items.size() + 1 == cuts.cta.size() ? nullptr : reinterpret_cast<const uint32_t*>(dev + o_cta);
        a.q_coarse = q_coarse;
        a.q_sign = reinterpret_cast<const uint32_t*>(q_sign);
        a.scores = scores;
        a.score_stride = n;
        a.nf4_table = codec_hint < 0 ? 2u : (uint32_t)(codec_hint & 1);
        return launch_dense(c, a, (uint32_t)cuts.cta.size() - 1, true);
    }
    const int threads = 128, nwarps = threads / 32;
    const uint32_t item_tiles = 4096;
    const uint32_t chunks = (uint32_t)((n + item_tiles - 1) / item_tiles);
    size_t q0 = 0;
    while (q0 < nq) {
        const size_t gq = std::min<size_t>(4, nq - q0);
        const int G = group_width((uint32_t)gq);
        ScoreArgs a{};
        a.tiles = reinterpret_cast<const unsigned char*>(tiles);
        a.state = state;
        a.items = nullptr;
        a.q_coarse = q_coarse + q0 * D_C;
        a.q_sign = reinterpret_cast<const uint32_t*>(q_sign + q0 * 4);
        a.scores = scores + q0 * n;
        a.cold_bits = 0xFF800000u;
        a.score_stride = n;
        a.total_tiles = n;
        a.item_tiles = item_tiles;
        a.nq_launch = (uint32_t)gq;
        SLHA_TRY(launch_score<false>(c, G, a, chunks, threads, score_smem_bytes(G, nwarps, false, 0), false));
        q0 += gq;
    }
    return Status();
}

// fill of the rows' tails [tail_begin[q], row_len) (one CTA per row)
__global__ void fill_rows_kernel(float* scores, const unsigned long long* row_offset, const uint32_t* tail_begin, uint32_t row_len, float fill, const uint32_t* refused) {
    if (refused && *refused) return;
    float* row = scores + row_offset[blockIdx.x];
    for (uint32_t e = tail_begin[blockIdx.x] + threadIdx.x; e < row_len; e += blockDim.x) row[e] = fill;
}

// Dense scores of whole segments: every query row of a segment against every tile of the segment, row q written at
// scores + row_offsets[q] + index_base + tile, the rest of the row up to row_len set to `fill`.  Where every segment brings 16 query rows or
// more the 64-row kernel comes first and the four-row kernel takes the rows it hands over (it ends at once when there are none).  The host looks at no tile and
// waits for nothing.
Status launch_score_segments(Ctx* c, const SciRustSlhaTile* tiles, const SlhaB200Segment* segs, size_t n_segs, const float* d_q_coarse,
                             const uint64_t* d_q_sign, size_t nq, float* d_scores, const uint64_t* row_offsets,
                             uint32_t row_len, float fill, RowCheck* check) {
    const int sms = sm_count(c->device);
    bool wide = !g_force_generic, fills = false;
    uint64_t total = 0, wtotal = 0;
    std::vector<uint32_t> tail(nq, row_len);
    for (size_t i = 0; i < n_segs; ++i) {
        const SlhaB200Segment& s = segs[i];
        if ((uint64_t)s.query_begin + s.n_queries > nq) return Status(SLHA_ERR_DIMENSION, "segment query range exceeds n_queries");
        if ((uint64_t)s.index_base + s.n_tiles > row_len) return Status(SLHA_ERR_DIMENSION, "segment does not fit a row of row_len scores");
        for (uint32_t q = 0; q < s.n_queries; ++q) tail[s.query_begin + q] = s.index_base + s.n_tiles;
        fills |= s.index_base + s.n_tiles < row_len;
        wide = wide && (s.n_queries >= 16 || s.n_tiles == 0);
        total += Cuts::whole(s.n_tiles, ST_M) * ((s.n_queries + 3) / 4);
        wtotal += Cuts::whole(s.n_tiles, WIDE_M) * ((s.n_queries + WIDE_NQ - 1) / WIDE_NQ);
    }
    Cuts cuts(wide ? wtotal : total, sms, wide ? WIDE_M : ST_M, wide ? WIDE_M : ST_M * 4);
    for (size_t i = 0; i < n_segs; ++i) cuts.add(segs[i], wide ? WIDE_NQ : 4);
    cuts.finish();
    Streams streams;
    if (wide) streams.make(cuts.items, sms);
    std::vector<WorkItem> generic;  // runs of 4096 tiles where score_kernel takes the call
    if (g_force_generic)
        for (const WorkItem& s : cuts.items)
            for (uint32_t pos = 0; pos < s.n_tiles; pos += 4096) {
                WorkItem w = s;
                w.tile_begin += pos;
                w.index_base += pos;
                w.n_tiles = std::min<uint32_t>(4096, s.n_tiles - pos);
                generic.push_back(w);
            }
    Blob blob;
    const size_t o_items = blob.add(cuts.items), o_cta = blob.add(cuts.cta), o_gen = blob.add(generic);
    const size_t o_tail = fills ? blob.add(tail) : 0;
    const size_t o_s = streams.all.empty() ? o_items : blob.add(streams.all);
    const size_t o_rows = check ? 0 : blob.add(std::vector<uint64_t>(row_offsets, row_offsets + nq));
    const size_t o_flag = wide ? blob.add_zeros(nq + 1) : 0;
    unsigned char* dev;
    SLHA_TRY(send_tables(c, blob, &dev, check));
    const unsigned long long* d_row_offsets = reinterpret_cast<const unsigned long long*>(check ? check->copy : reinterpret_cast<const uint64_t*>(dev + o_rows));
    const uint32_t* refused = check ? check->refused : nullptr;
    if (fills) {
        fill_rows_kernel<<<(uint32_t)nq, 256, 0, c->stream>>>(d_scores, d_row_offsets, reinterpret_cast<const uint32_t*>(dev + o_tail), row_len, fill, refused);
        count_launch();
        SLHA_CUDA(cudaGetLastError());
    }
    if (cuts.items.empty()) return Status();
    ScoreArgs a{};
    a.tiles = reinterpret_cast<const unsigned char*>(tiles);
    a.q_coarse = d_q_coarse;
    a.q_sign = reinterpret_cast<const uint32_t*>(d_q_sign);
    a.scores = d_scores;
    a.row_offset = d_row_offsets;
    a.cold_bits = 0xFF800000u;
    a.refused = refused;
    a.items = a.stream_items = reinterpret_cast<const WorkItem*>(dev + o_items);
    a.n_items = (uint32_t)cuts.items.size();
    a.cta_begin = reinterpret_cast<const uint32_t*>(dev + o_cta);
    const uint32_t grid = (uint32_t)cuts.cta.size() - 1;
    if (wide) {
        a.handoff = reinterpret_cast<uint32_t*>(dev + o_flag);
        a.handoff_any = a.handoff + nq;
        a.handoff_as = 1u;
        SLHA_TRY(launch_wide_dense(c, a, grid, true));
        a.only_flagged = a.handoff;
        a.streams = reinterpret_cast<const WorkItem*>(dev + o_s);
        a.n_streams = streams.n;
        a.least_share = 4u;
    } else if (a.n_items == grid) {
        a.cta_begin = nullptr;
    }
    if (!g_force_generic) return launch_dense(c, a, wide ? streams.grid : grid, true);
    a.items = reinterpret_cast<const WorkItem*>(dev + o_gen);
    const int threads = 128, nwarps = threads / 32;
    return launch_score<false>(c, 4, a, (uint32_t)generic.size(), threads, score_smem_bytes(4, nwarps, false, 0), false);
}

// Every score of every row, then the rows' best.
static Status score_topk_rows(Ctx* c, Plan* p, const SciRustSlhaTile* tiles, const uint8_t* state, const float* d_q_coarse, const uint64_t* d_q_sign, size_t nq, uint32_t k,
                              uint32_t* d_out_index, float* d_out_score, uint32_t* d_out_count, int codec_hint) {
    const bool timed = g_timing.calls < g_timing.max_calls;
    cudaEvent_t* tev = timed ? &g_timing.ev[3 * g_timing.calls] : nullptr;
    if (timed) SLHA_CUDA(cudaEventRecord(tev[0], c->stream));
    g_last_stream_plan = p;
    ScoreArgs a{};
    a.tiles = reinterpret_cast<const unsigned char*>(tiles);
    a.state = state;
    a.q_coarse = d_q_coarse;
    a.q_sign = reinterpret_cast<const uint32_t*>(d_q_sign);
    a.scores = reinterpret_cast<float*>(p->b_gbuf.p);
    a.score_stride = p->row_stride;
    a.cold_bits = ROW_ABSENT;
    a.nf4_table = codec_hint < 0 ? 2u : (uint32_t)(codec_hint & 1);
    a.gflag = p->d_row_flags;
    a.items = a.stream_items = p->d_items;
    a.n_items = p->n_items;
    a.cta_begin = p->d_cta_begin;
    if (p->wide) {
        a.blocked = 1u;
        a.handoff = p->d_row_flags + nq;
        a.handoff_any = p->d_row_flags + 4 * nq;
        a.handoff_as = 2u;
        SLHA_TRY(launch_wide_dense(c, a, p->mma_grid, true));
        a.only_flagged = a.handoff;
        a.streams = p->d_streams;
        a.n_streams = p->n_streams;
        a.least_share = 1u;
    }
    SLHA_TRY(launch_dense(c, a, p->wide ? p->streams_grid : p->mma_grid, true));
    if (timed) SLHA_CUDA(cudaEventRecord(tev[1], c->stream));
    RowsArgs r{a.scores, p->d_rows, p->d_row_flags, p->d_row_flags + 2 * nq, k, row_cap(k, p->kp2), d_out_index, d_out_score, d_out_count};
    SLHA_TRY(launch_rows(c, r, (uint32_t)nq, p->longest));
    if (timed) {
        SLHA_CUDA(cudaEventRecord(tev[2], c->stream));
        ++g_timing.calls;
    }
    return Status();
}

Status score_topk_device(Ctx* c, const SciRustSlhaTile* tiles, const uint8_t* state,
                         const SlhaB200Segment* segs, size_t n_segs, const float* d_q_coarse,
                         const uint64_t* d_q_sign, size_t nq, uint32_t k, uint32_t* d_out_index,
                         float* d_out_score, uint32_t* d_out_count, bool prefer_generic, int codec_hint) {
    if (nq == 0) return Status();
    // (4096 winners per row is what the generic kernel's block-wide selection state holds in shared memory beside its
    // tile ring; the plan builder checks the exact figure)
    if (k == 0 || k > 4096) return Status(SLHA_ERR_DIMENSION, "top-k: k must be in 1..4096");
    ctx_uses_plans(c);
    Plan* p = nullptr;
    SLHA_TRY(build_plan(c, tiles, segs, n_segs, nq, k, codec_hint, /*allow_wide=*/state == nullptr, /*allow_rows=*/!prefer_generic && !g_stream_all_rows, &p));
    g_last_plan = p;
    if (p->rows) return score_topk_rows(c, p, tiles, state, d_q_coarse, d_q_sign, nq, k, d_out_index, d_out_score, d_out_count, codec_hint);
    const int nwarps = p->threads / 32;
    const bool timed = g_timing.calls < g_timing.max_calls;
    cudaEvent_t* tev = timed ? &g_timing.ev[3 * g_timing.calls] : nullptr;
    if (timed) SLHA_CUDA(cudaEventRecord(tev[0], c->stream));
    const bool mma = p->use_mma && !prefer_generic;
    ScoreArgs am{};
    if (mma) g_last_stream_plan = p;
    if (mma) {
        if (!p->state_clean) SLHA_CUDA(cudaMemsetAsync(p->d_gpivot, 0, p->gstate_bytes, c->stream));
        p->state_clean = false;
        ScoreArgs& a = am;
        a.tiles = reinterpret_cast<const unsigned char*>(tiles);
        a.state = state;
        a.items = p->d_items;
        a.stream_items = p->d_stream_items ? p->d_stream_items : p->d_items;
        a.n_items = p->n_items;
        a.cta_begin = p->d_cta_begin;
        // (histograms first: they are read with 16-byte loads)
        a.ghist = reinterpret_cast<uint32_t*>(p->d_gpivot);
        a.gpivot = p->d_gpivot + 128 * nq;
        a.grange = a.gpivot + nq;
        a.gcount = reinterpret_cast<uint32_t*>(a.grange + nq);
        a.gflag = a.gcount + nq;
        a.gbuf = p->d_gbuf;
        a.gcap = p->gcap;
        a.q_coarse = d_q_coarse;
        a.q_sign = reinterpret_cast<const uint32_t*>(d_q_sign);
        a.k = k;
        if (p->wide) {
            a.items = p->d_wide_items;
            a.n_items = p->n_wide_items;
            a.cta_begin = p->d_wide_cta;
            SLHA_TRY(launch_wide(c, p->kind, a, p->wide_grid));
        } else if (p->d_stream_items) {
            SLHA_TRY(launch_stream(c, p->kind, true, false, a, p->mma_grid));
        } else {
            SLHA_TRY(launch_stream(c, p->kind, false, p->long_items, a, p->mma_grid));
        }
        // (timing: the first bracket is the tensor-core kernel alone; the generic kernel's pass over handed-back rows, an
        // early exit when there are none, counts with the compaction and the merge)
        if (timed) SLHA_CUDA(cudaEventRecord(tev[1], c->stream));
    }
    for (const Plan::Class& cl : p->classes) {
        ScoreArgs a{};
        a.gflag = mma ? am.gflag : nullptr;  // after the tensor-core kernel: only the work items of rows it handed back
        a.tiles = reinterpret_cast<const unsigned char*>(tiles);
        a.state = state;
        a.items = p->d_items + cl.first;
        a.q_coarse = d_q_coarse;
        a.q_sign = reinterpret_cast<const uint32_t*>(d_q_sign);
        a.k = k;
        a.list_cap = p->list_cap;
        a.cap = p->cap;
        a.cand_keys = p->d_cand_keys;
        a.cand_cnt = p->d_cand_cnt;
        SLHA_TRY(launch_score<true>(c, cl.G, a, cl.count, p->threads, score_smem_bytes(cl.G, nwarps, true, p->cap), mma));
    }
    if (timed && !mma) SLHA_CUDA(cudaEventRecord(tev[1], c->stream));
    static thread_local bool configured[16] = {false};  // the attribute is per device
    if (!configured[c->device & 15]) {
        SLHA_CUDA(cudaFuncSetAttribute(topk_merge_kernel<CompLists>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)MAX_SMEM));
        SLHA_CUDA(cudaFuncSetAttribute(topk_merge_kernel<PairLists>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)MAX_SMEM));
        SLHA_CUDA(cudaFuncSetAttribute(topk_merge_kernel<StreamLists>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)MAX_SMEM));
        SLHA_CUDA(cudaFuncSetAttribute(topk_merge_kernel<CompLists>, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared));
        SLHA_CUDA(cudaFuncSetAttribute(topk_merge_kernel<PairLists>, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared));
        SLHA_CUDA(cudaFuncSetAttribute(topk_merge_kernel<StreamLists>, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared));
        SLHA_CUDA(cudaFuncSetAttribute(stream_compact_kernel<true>, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared));
        SLHA_CUDA(cudaFuncSetAttribute(stream_compact_kernel<false>, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared));
        configured[c->device & 15] = true;
    }
    if (mma) {
        uint32_t* gselcnt = am.gflag + nq;
        const uint32_t cap_s = p->selcap;
        if (p->compact_splits) {
            const dim3 cgrid(p->compact_splits, (uint32_t)nq);
            if (p->late_threshold)
                SLHA_CUDA(launch_behind(stream_compact_kernel<true>, cgrid, dim3(256), 0, c->stream, p->d_gbuf, am.gcount, am.gflag, am.gpivot, p->gcap,
                                        (uint64_t*)p->b_gsel.p, gselcnt, cap_s, p->compact_splits, am.ghist, k));
            else
                SLHA_CUDA(launch_behind(stream_compact_kernel<false>, cgrid, dim3(256), 0, c->stream, p->d_gbuf, am.gcount, am.gflag, am.gpivot, p->gcap,
                                        (uint64_t*)p->b_gsel.p, gselcnt, cap_s, p->compact_splits, am.ghist, k));
            count_launch();
            SLHA_CUDA(cudaGetLastError());
        }
        StreamLists L{p->d_gbuf, am.gcount, am.gflag, am.gpivot, p->gcap,
                      p->compact_splits ? (const uint64_t*)p->b_gsel.p : nullptr, gselcnt, cap_s,
                      CompLists{p->d_cand_keys, p->d_cand_cnt, p->d_q_list_begin, p->d_q_list_count, p->list_cap},
                      am.ghist, p->late_threshold ? k : 0u, gselcnt + nq};
        SLHA_CUDA(launch_behind(topk_merge_kernel<StreamLists>, dim3((uint32_t)nq), dim3(merge_threads(cap_s)), merge_smem(cap_s, p->kp2), c->stream, L, k, p->kp2, cap_s,
                                d_out_index, d_out_score, d_out_count));
        p->state_clean = true;
    } else if (p->n_groups) {
        // few queries, many lists each: groups of lists first, then the groups' results
        CompLists L1{p->d_cand_keys, p->d_cand_cnt, p->d_vq_begin, p->d_vq_count, p->list_cap};
        const uint32_t cap1 = merge_cap((uint64_t)p->group_parts * p->list_cap, p->kp2, k);
        topk_merge_kernel<CompLists><<<p->n_groups * (uint32_t)nq, merge_threads(cap1), merge_smem(cap1, p->kp2), c->stream>>>(
            L1, k, p->kp2, cap1, p->d_tmp_index, p->d_tmp_score, nullptr);
        count_launch();
        SLHA_CUDA(cudaGetLastError());
        PairLists L2{p->d_tmp_index, p->d_tmp_score, p->n_groups, (uint32_t)nq, k, (uint64_t)nq * k, 1u, nullptr, nullptr, nullptr, nullptr, nullptr};
        const uint32_t cap2 = merge_cap((uint64_t)p->n_groups * k, p->kp2, k);
        topk_merge_kernel<PairLists><<<(uint32_t)nq, merge_threads(cap2), merge_smem(cap2, p->kp2), c->stream>>>(
            L2, k, p->kp2, cap2, d_out_index, d_out_score, d_out_count);
    } else {
        CompLists L{p->d_cand_keys, p->d_cand_cnt, p->d_q_list_begin, p->d_q_list_count, p->list_cap};
        const uint32_t cap_s = merge_cap((uint64_t)p->max_parts * p->list_cap, p->kp2, k);
        topk_merge_kernel<CompLists><<<(uint32_t)nq, merge_threads(cap_s), merge_smem(cap_s, p->kp2), c->stream>>>(
            L, k, p->kp2, cap_s, d_out_index, d_out_score, d_out_count);
    }
    count_launch();
    SLHA_CUDA(cudaGetLastError());
    if (timed) {
        SLHA_CUDA(cudaEventRecord(tev[2], c->stream));
        ++g_timing.calls;
    }
    return Status();
}

// A captured score_topk names the buffers of one of the calling thread's plans: its graph may run as long as plan_epoch()
// returns what it returned at the capture (this thread, none of its captured plans rebuilt for another shape).
uint64_t plan_epoch() {
    static thread_local const uint32_t thread_no = ++g_plan_threads;
    return ((uint64_t)thread_no << 32) | g_plans_recycled;
}
void plan_was_captured() {
    if (g_last_plan) g_last_plan->captured = true;
}

void debug_force_generic_score(bool on) { g_force_generic = on; }
void debug_stream_all_rows(bool on) { g_stream_all_rows = on; }
bool debug_general_paths() { return g_force_generic; }

// Counters of the calling thread's latest score_topk call that used the tensor-core kernel.
Status last_score_stats(Ctx* c, uint64_t* out4) {
    out4[0] = out4[1] = out4[2] = out4[3] = 0;
    const Plan* p = g_last_stream_plan;
    if (!p || p->device != c->device || !p->use_mma) return Status();
    const size_t nq = p->nq;
    std::vector<uint32_t> h(2 * nq);
    const uint32_t* stats = p->rows ? p->d_row_flags + 2 * nq : reinterpret_cast<const uint32_t*>(p->d_gpivot + 128 * nq + 2 * nq) + 3 * nq;  // kept by the merge
    SLHA_CUDA(cudaMemcpyAsync(h.data(), stats, 8 * nq, cudaMemcpyDeviceToHost, c->stream));
    SLHA_CUDA(cudaStreamSynchronize(c->stream));
    out4[0] = nq;
    for (size_t q = 0; q < nq; ++q) {
        out4[1] += h[2 * q + 1] != 0;
        out4[2] += h[2 * q];
    }
    out4[3] = p->rows ? p->row_stride : p->gcap;
    return Status();
}

uint32_t last_score_kernel(Ctx* c) {
    const Plan* p = g_last_stream_plan;
    if (!p || p->device != c->device || !p->use_mma) return 0u;
    if (p->rows) return p->wide ? SLHA_B200_KERNEL_ROWS_WIDE : SLHA_B200_KERNEL_ROWS;
    return p->wide ? SLHA_B200_KERNEL_WIDE : p->kind == 4 ? SLHA_B200_KERNEL_TILE : SLHA_B200_KERNEL_STREAM;
}

// Tiles a warp of that call took at a time.
uint32_t last_score_set(Ctx* c) {
    return last_score_kernel(c) == SLHA_B200_KERNEL_STREAM ? (uint32_t)(MMA_SET_TILES * g_last_stream_plan->sets) : 0u;
}

bool timing_active() { return g_timing.calls < g_timing.max_calls; }

Status timing_begin(uint32_t max_calls) {
    for (cudaEvent_t e : g_timing.ev) cudaEventDestroy(e);
    g_timing.ev.assign((size_t)3 * max_calls, nullptr);
    for (cudaEvent_t& e : g_timing.ev) SLHA_CUDA(cudaEventCreate(&e));
    g_timing.max_calls = max_calls;
    g_timing.calls = 0;
    return Status();
}

Status timing_end(Ctx* c, float* score_ms, float* merge_ms, uint32_t capacity, uint32_t* n_out) {
    SLHA_CUDA(cudaStreamSynchronize(c->stream));
    const uint32_t n = std::min(g_timing.calls, capacity);
    for (uint32_t i = 0; i < n; ++i) {
        float a = 0, b = 0;
        SLHA_CUDA(cudaEventElapsedTime(&a, g_timing.ev[3 * i], g_timing.ev[3 * i + 1]));
        SLHA_CUDA(cudaEventElapsedTime(&b, g_timing.ev[3 * i + 1], g_timing.ev[3 * i + 2]));
        if (score_ms) score_ms[i] = a;
        if (merge_ms) merge_ms[i] = b;
    }
    if (n_out) *n_out = g_timing.calls;
    for (cudaEvent_t e : g_timing.ev) cudaEventDestroy(e);
    g_timing.ev.clear();
    g_timing.max_calls = g_timing.calls = 0;
    return Status();
}

Status launch_topk_merge_pairs(Ctx* c, const uint32_t* cand_index, const float* cand_score,
                               uint32_t n_lists, uint64_t list_stride, uint32_t n_queries, uint32_t k_in,
                               uint32_t k_out, uint32_t* out_index, float* out_score, bool lists_sorted) {
    if (n_queries == 0) return Status();
    if (k_out == 0 || k_out > 8192) return Status(SLHA_ERR_DIMENSION, "merge: k_out must be in 1..8192");
    uint32_t kp2 = 2;
    while (kp2 < k_out) kp2 <<= 1;
    PairLists L{cand_index, cand_score, n_lists, n_queries, k_in, list_stride, lists_sorted ? 1u : 0u, nullptr, nullptr, nullptr, nullptr, nullptr};
    static thread_local bool configured[16] = {false};  // the attribute is per device
    if (!configured[c->device & 15]) {
        SLHA_CUDA(cudaFuncSetAttribute(topk_merge_kernel<PairLists>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)MAX_SMEM));
        configured[c->device & 15] = true;
    }
    const uint32_t cap_s = merge_cap((uint64_t)n_lists * k_in, kp2, k_out);
    topk_merge_kernel<PairLists><<<n_queries, merge_threads(cap_s), merge_smem(cap_s, kp2), c->stream>>>(L, k_out, kp2, cap_s, out_index, out_score, nullptr);
    count_launch();
    SLHA_CUDA(cudaGetLastError());
    return Status();
}

// The merge of a sharded step whose lists lie in their owners' memory (see PairLists::bases): lists ordered best first.
Status launch_topk_merge_peers(Ctx* c, const uint32_t* const* d_bases, uint32_t n_lists, uint32_t n_queries, uint32_t k, const uint32_t* d_ready,
                               uint32_t* d_step, uint32_t* d_done, uint32_t* d_status, uint32_t* out_index, float* out_score) {
    if (n_queries == 0) return Status();
    if (k == 0 || k > 8192) return Status(SLHA_ERR_DIMENSION, "merge: k must be in 1..8192");
    uint32_t kp2 = 2;
    while (kp2 < k) kp2 <<= 1;
    PairLists L{nullptr, nullptr, n_lists, n_queries, k, 0, 1u, d_bases, d_ready, d_step, d_done, d_status};
    static thread_local bool configured[16] = {false};  // the attribute is per device
    if (!configured[c->device & 15]) {
        SLHA_CUDA(cudaFuncSetAttribute(topk_merge_kernel<PairLists>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)MAX_SMEM));
        configured[c->device & 15] = true;
    }
    const uint32_t cap_s = merge_cap((uint64_t)n_lists * k, kp2, k);
    topk_merge_kernel<PairLists><<<n_queries, merge_threads(cap_s), merge_smem(cap_s, kp2), c->stream>>>(L, k, kp2, cap_s, out_index, out_score, nullptr);
    count_launch();
    SLHA_CUDA(cudaGetLastError());
    return Status();
}

}  // namespace slha
