// Device-resident CCOS elastic tile pool: the ElasticKvCache of
// scirust/src/ccos.rs with its arena, per-slot state/seq/importance arrays,
// LIFO free list and logical byte counter all kept in HBM.  Every transition
// (insert, page_out, drop_correction, evict, enforce_budget, observe_scores)
// runs as kernels; the host only reads back a 64-byte counter block.
//
// enforce_budget reproduces the reference's four ordered phases
// (ccos.rs:555-614).  A phase sorts its candidates by the reference's key
// (cub::DeviceRadixSort on a unique 64-bit key), prefix-sums the bytes each
// candidate would free, and applies the operation to exactly the prefix the
// reference's sequential loop would have reached.
#include <cooperative_groups.h>
#include <cub/block/block_radix_sort.cuh>
#include <cub/block/block_scan.cuh>
#include <cub/device/device_radix_sort.cuh>
#include <cub/device/device_scan.cuh>
#include <chrono>
#include <vector>

#include "common.cuh"
#include "pool.cuh"

namespace slha {
namespace {

__device__ __forceinline__ uint32_t f32_total_key(float f) {
    uint32_t u = __float_as_uint(f);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ uint32_t corr_bytes(uint32_t flags) {  // tile.rs:118-126
    return (flags & F_TQ3) ? 16u : ((flags & F_MIX3) ? 14u : 0u);
}
__device__ __forceinline__ uint32_t live_bytes_of(uint8_t st, uint32_t flags) {  // ccos.rs:468-482
    if (st == ST_COLD) return 0;
    const uint32_t base = st == ST_HOT ? 128u : 96u;
    return base - ((flags & F_NOCORR) ? corr_bytes(flags) : 0u);
}
__device__ __forceinline__ uint32_t tile_flags(const unsigned char* tiles, uint64_t slot) {
    return *reinterpret_cast<const uint16_t*>(tiles + slot * TILE_BYTES + 118);
}

// ---- insert (ccos.rs:217-259) ------------------------------------------------
// Tile j of the batch takes free_list[free_len-1-j] while the free list lasts
// (LIFO pops), then fresh slots len, len+1, ...
__global__ void insert_kernel(PoolDev p, const unsigned char* src, uint64_t n, uint64_t pops,
                              uint64_t len0, uint64_t free0, uint64_t seq0, const uint32_t* positions, uint32_t position_base, uint32_t* slots_out) {
    dep_launch();
    dep_wait();
    const uint64_t j = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    uint32_t bytes = 0;
    if (j < n) {
        const uint32_t slot = j < pops ? p.free_list[free0 - 1 - j] : (uint32_t)(len0 + (j - pops));
        uint32_t flags = 0;
        if (src) flags = *reinterpret_cast<const uint16_t*>(src + j * TILE_BYTES + 118);
        const uint8_t st = (flags & F_WARM) ? ST_WARM : ST_HOT;
        p.state[slot] = st;
        p.seq[slot] = seq0 + j;
        p.importance[slot] = 0.0f;
        p.pos[slot] = src ? *reinterpret_cast<const uint32_t*>(src + j * TILE_BYTES + 112) : positions ? positions[j] : position_base + (uint32_t)j;
        slots_out[j] = slot;
        bytes = live_bytes_of(st, flags);
    }
    for (int o = 16; o; o >>= 1) bytes += __shfl_xor_sync(0xFFFFFFFFu, bytes, o);
    if ((threadIdx.x & 31) == 0 && bytes) atomicAdd((unsigned long long*)&p.cnt->live, (unsigned long long)bytes);
    if (j == 0) {
        p.cnt->free_len = free0 - pops;
        p.cnt->len = len0 + (n - pops);
        p.cnt->next_seq = seq0 + n;
    }
}
__global__ void scatter_tiles_kernel(unsigned char* tiles, const unsigned char* src,
                                     const uint32_t* slots, uint64_t n) {
    const uint64_t e = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (e < n * 8) {
        const uint64_t j = e >> 3, c = e & 7;
        reinterpret_cast<uint4*>(tiles + (uint64_t)slots[j] * TILE_BYTES)[c] =
            reinterpret_cast<const uint4*>(src + j * TILE_BYTES)[c];
    }
}

// ---- single-slot transitions ---------------------------------------------------
__device__ bool do_page_out(const PoolDev& p, uint32_t slot, int64_t* delta) {  // ccos.rs:365-380
    if (p.state[slot] != ST_HOT) return false;
    unsigned char* t = p.tiles + (uint64_t)slot * TILE_BYTES;
    uint4 z = make_uint4(0, 0, 0, 0);
    reinterpret_cast<uint4*>(t + 64)[0] = z;
    reinterpret_cast<uint4*>(t + 64)[1] = z;
    *reinterpret_cast<float*>(t + 100) = 0.0f;
    *reinterpret_cast<uint16_t*>(t + 118) |= F_WARM;
    p.state[slot] = ST_WARM;
    *delta -= 32;
    return true;
}
__device__ bool do_drop_correction(const PoolDev& p, uint32_t slot, int64_t* delta) {  // ccos.rs:386-397
    unsigned char* t = p.tiles + (uint64_t)slot * TILE_BYTES;
    const uint32_t flags = *reinterpret_cast<uint16_t*>(t + 118);
    const uint32_t nb = corr_bytes(flags);
    if (p.state[slot] == ST_COLD || nb == 0 || (flags & F_NOCORR)) return false;
    for (uint32_t b = 64 - nb; b < 64; ++b) t[b] = 0;
    *reinterpret_cast<uint16_t*>(t + 118) = (uint16_t)(flags | F_NOCORR);
    *delta -= (int64_t)nb;
    return true;
}
__global__ void single_op_kernel(PoolDev p, int op, uint32_t slot, int32_t* result) {
    int64_t delta = 0;
    bool done = false;
    if (slot < p.cnt->len) {
        if (op == 0) done = do_page_out(p, slot, &delta);
        else if (op == 1) done = do_drop_correction(p, slot, &delta);
        else if (p.state[slot] != ST_COLD) {  // evict, ccos.rs:404-438 (no event log)
            delta = -(int64_t)live_bytes_of(p.state[slot], tile_flags(p.tiles, slot));
            p.state[slot] = ST_COLD;
            p.free_list[p.cnt->free_len++] = slot;
            done = true;
        }
    }
    p.cnt->live = (uint64_t)((int64_t)p.cnt->live + delta);
    *result = done ? 1 : 0;
}

// ---- enforce_budget phases -------------------------------------------------------
enum Phase { PH_CORR_HOT = 0, PH_PAGE = 1, PH_CORR_WARM = 2, PH_EVICT = 3, PH_EVICT_PINNED = 4 };
constexpr uint64_t SENTINEL = ~0ull;

// max live position (for the recent-window extension)
__global__ void max_pos_kernel(PoolDev p) {
    const uint64_t len = p.cnt->len;
    uint32_t m = 0;
    for (uint64_t s = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; s < len; s += (uint64_t)gridDim.x * blockDim.x)
        if (p.state[s] != ST_COLD) m = max(m, p.pos[s]);
    for (int o = 16; o; o >>= 1) m = max(m, __shfl_xor_sync(0xFFFFFFFFu, m, o));
    if ((threadIdx.x & 31) == 0) atomicMax(&p.cnt->max_pos, m);
}

__device__ __forceinline__ bool is_pinned(const PoolDev& p, uint32_t pos, uint32_t max_pos) {
    if (pos < p.sink_window) return true;  // ccos.rs:592-594
    return p.recent_window && (max_pos - pos) < p.recent_window;
}

// What phase_key needs of a slot: loaded first, so that a scan can have several slots' loads in flight.
struct SlotMeta {
    uint8_t st;
    uint32_t pos, flags, seq;
    float weight;  // sigma (paging phases) or importance (eviction)
};
// state only: may `phase` act on a slot in state st at all
__device__ __forceinline__ bool phase_looks(int phase, uint8_t st) {
    return phase >= PH_EVICT ? st != ST_COLD : st == (phase == PH_CORR_WARM ? ST_WARM : ST_HOT);
}
// (st is set; the rest is loaded where the phase looks at such slots)
__device__ __forceinline__ void load_meta(const PoolDev& p, int phase, uint64_t s, SlotMeta& m) {
    m.pos = m.flags = m.seq = 0u;
    m.weight = 0.0f;
    if (!phase_looks(phase, m.st)) return;
    const unsigned char* t = p.tiles + s * TILE_BYTES;
    if (phase >= PH_EVICT) m.pos = p.pos[s];
    if (phase == PH_CORR_HOT || phase == PH_CORR_WARM) m.flags = tile_flags(p.tiles, s);
    m.seq = (uint32_t)p.seq[s];
    m.weight = phase >= PH_EVICT ? p.importance[s] : *reinterpret_cast<const float*>(t + 104);
}
// the sort key of slot s in `phase`, or SENTINEL when the phase cannot act on it
__device__ __forceinline__ uint64_t phase_key(const PoolDev& p, int phase, uint64_t s, const SlotMeta& m, uint32_t max_pos) {
    if (!phase_looks(phase, m.st)) return SENTINEL;
    if (phase >= PH_EVICT) {
        const bool pin = p.evict_policy == SLHA_B200_EVICT_IMPORTANCE && is_pinned(p, m.pos, max_pos);
        if ((phase == PH_EVICT_PINNED) != pin) return SENTINEL;
        // ccos.rs:586-603: causal = by seq; importance = (importance, seq)
        return p.evict_policy == SLHA_B200_EVICT_CAUSAL ? (uint64_t)m.seq : ((uint64_t)f32_total_key(m.weight) << 32) | m.seq;
    }
    if (phase != PH_PAGE && (!corr_bytes(m.flags) || (m.flags & F_NOCORR))) return SENTINEL;
    // slots_in_paging_order, ccos.rs:526-539: stable sort of the
    // slot-ascending list by sigma (total order) or by seq
    return p.page_policy == SLHA_B200_PAGE_LOWEST_IMPACT_FIRST ? ((uint64_t)f32_total_key(m.weight) << 32) | (uint32_t)s : (uint64_t)m.seq;
}

// candidate (key, slot) pairs of one phase, compacted in arbitrary order (keys are unique, so the
// sort that follows gives one order): only the slots a phase can act on are sorted, e.g. the few
// HOT tiles just appended for the page-out phase.  n_cand is zero when the kernel starts.
__global__ void phase_build_kernel(PoolDev p, int phase, uint64_t* keys, uint32_t* vals) {
    const uint64_t len = p.cnt->len;
    const bool over = p.cnt->live > p.cnt->budget;
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        p.cnt->phase_deficit = over ? p.cnt->live - p.cnt->budget : 0;
        p.cnt->phase_applied = 0;
    }
    const uint32_t max_pos = p.cnt->max_pos;
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    const uint64_t rounds = over ? (len + stride - 1) / stride : 0;  // whole warps stay together for the ballot
    for (uint64_t r = 0; r < rounds; ++r) {
        const uint64_t s = r * stride + (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
        uint64_t key = SENTINEL;
        if (s < len) {
            SlotMeta m;
            m.st = p.state[s];
            load_meta(p, phase, s, m);
            key = phase_key(p, phase, s, m, max_pos);
        }
        const unsigned hit = __ballot_sync(0xFFFFFFFFu, key != SENTINEL);
        if (hit) {
            const int lane = threadIdx.x & 31;
            uint32_t base = 0;
            if (lane == 0) base = atomicAdd(&p.cnt->n_cand, (uint32_t)__popc(hit));
            base = __shfl_sync(0xFFFFFFFFu, base, 0);
            if (key != SENTINEL) {
                const uint32_t i = base + (uint32_t)__popc(hit & ((1u << lane) - 1u));
                keys[i] = key;
                vals[i] = (uint32_t)s;
            }
        }
    }
}

// Pre-filter of a long candidate list: a phase stops once the bytes it has freed reach the deficit,
// and every operation of a phase frees at least `min_freed` bytes (14 for a dropped correction
// plane, 32 for a page-out, 80 for an eviction), so only the M = deficit / min_freed + 1 smallest
// keys can be reached.  A histogram over the keys' 12 high bits gives the smallest bin prefix that
// holds M candidates; only those candidates are sorted.
constexpr uint32_t PREFILTER_BINS = 4096, PREFILTER_MIN = 65536;
__global__ void phase_hist_kernel(PoolDev p, const uint64_t* keys, uint32_t* hist) {
    __shared__ uint32_t h[PREFILTER_BINS];
    for (uint32_t b = threadIdx.x; b < PREFILTER_BINS; b += blockDim.x) h[b] = 0;
    __syncthreads();
    const uint64_t n = p.cnt->n_cand;
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x)
        atomicAdd(&h[(uint32_t)(keys[i] >> 52)], 1u);
    __syncthreads();
    for (uint32_t b = threadIdx.x; b < PREFILTER_BINS; b += blockDim.x)
        if (h[b]) atomicAdd(&hist[b], h[b]);
}
// keeps the candidates whose bin is at most `last_bin`; n_cand becomes their number (out_n, then copied)
__global__ void phase_filter_kernel(PoolDev p, const uint64_t* keys, const uint32_t* vals, uint32_t last_bin,
                                    uint64_t* keys_out, uint32_t* vals_out, uint32_t* out_n) {
    const uint64_t n = p.cnt->n_cand;
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    const uint64_t rounds = (n + stride - 1) / stride;
    for (uint64_t r = 0; r < rounds; ++r) {
        const uint64_t i = r * stride + (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
        const bool keep = i < n && (uint32_t)(keys[i] >> 52) <= last_bin;
        const unsigned hit = __ballot_sync(0xFFFFFFFFu, keep);
        if (hit) {
            const int lane = threadIdx.x & 31;
            uint32_t base = 0;
            if (lane == 0) base = atomicAdd(out_n, (uint32_t)__popc(hit));
            base = __shfl_sync(0xFFFFFFFFu, base, 0);
            if (keep) {
                const uint32_t o = base + (uint32_t)__popc(hit & ((1u << lane) - 1u));
                keys_out[o] = keys[i];
                vals_out[o] = vals[i];
            }
        }
    }
}
__global__ void phase_set_ncand_kernel(PoolDev p, const uint32_t* n) { p.cnt->n_cand = *n; }

__global__ void phase_weights_kernel(PoolDev p, int phase, const uint64_t* keys_sorted,
                                     const uint32_t* slots_sorted, uint32_t* w) {
    const uint64_t len = p.cnt->n_cand;
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < len; i += (uint64_t)gridDim.x * blockDim.x) {
        uint32_t bytes = 0;
        if (keys_sorted[i] != SENTINEL) {
            const uint32_t s = slots_sorted[i];
            const uint32_t flags = tile_flags(p.tiles, s);
            if (phase == PH_PAGE) bytes = 32;
            else if (phase <= PH_CORR_WARM) bytes = corr_bytes(flags);
            else bytes = live_bytes_of(p.state[s], flags);
        }
        w[i] = bytes;
    }
}

// Apply the phase operation to the sorted prefix whose exclusive byte prefix is
// below the deficit: exactly the items the reference's `for s in order { if
// live <= budget {return}; op(s) }` loop reaches.
__global__ void phase_apply_kernel(PoolDev p, int phase, const uint64_t* keys_sorted,
                                   const uint32_t* slots_sorted, const uint32_t* w,
                                   const uint64_t* excl, uint64_t limit) {
    const uint64_t len = p.cnt->n_cand;
    const uint64_t deficit = p.cnt->phase_deficit;
    const uint64_t free0 = p.cnt->free_len;
    int64_t delta = 0;
    uint32_t applied = 0;
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < len; i += (uint64_t)gridDim.x * blockDim.x) {
        if (keys_sorted[i] == SENTINEL || deficit == 0 || excl[i] >= deficit || i >= limit) continue;
        const uint32_t s = slots_sorted[i];
        if (phase == PH_PAGE) do_page_out(p, s, &delta);
        else if (phase <= PH_CORR_WARM) do_drop_correction(p, s, &delta);
        else {
            delta -= (int64_t)w[i];
            p.state[s] = ST_COLD;
            p.free_list[free0 + i] = s;  // pushes happen in sorted order (applied items are a prefix)
            ++applied;
        }
    }
    for (int o = 16; o; o >>= 1) {
        delta += __shfl_xor_sync(0xFFFFFFFFu, delta, o);
        applied += __shfl_xor_sync(0xFFFFFFFFu, applied, o);
    }
    if ((threadIdx.x & 31) == 0) {
        if (delta) atomicAdd((unsigned long long*)&p.cnt->live_delta, (unsigned long long)delta);
        if (applied) atomicAdd((unsigned long long*)&p.cnt->phase_applied, (unsigned long long)applied);
    }
}
// With an event log attached: (seq, slot, tile) of the slots an eviction phase is about to turn COLD,
// in eviction order (the applied items are a prefix of the sorted candidates), for the host to append.
__global__ void phase_journal_kernel(PoolDev p, const uint64_t* keys_sorted, const uint32_t* slots_sorted, const uint64_t* excl,
                                     unsigned long long* count, uint64_t* seq_out, uint32_t* slot_out, uint4* tiles_out) {
    const uint64_t len = p.cnt->n_cand, deficit = p.cnt->phase_deficit;
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < len; i += (uint64_t)gridDim.x * blockDim.x) {
        if (keys_sorted[i] == SENTINEL || deficit == 0 || excl[i] >= deficit) continue;
        const uint32_t s = slots_sorted[i];
        seq_out[i] = p.seq[s];
        slot_out[i] = s;
        const uint4* src = reinterpret_cast<const uint4*>(p.tiles + (size_t)s * TILE_BYTES);
        for (int j = 0; j < 8; ++j) tiles_out[i * 8 + j] = src[j];
        atomicMax(count, (unsigned long long)(i + 1));
    }
}
__global__ void phase_commit_kernel(PoolDev p) {
    p.cnt->live = (uint64_t)((int64_t)p.cnt->live + (int64_t)p.cnt->live_delta);
    p.cnt->live_delta = 0;
    p.cnt->free_len += p.cnt->phase_applied;
    p.cnt->phase_applied = 0;
}

// ---- enforce_budget in one cooperative launch --------------------------------------
// The host-driven phases above need the candidate count (for the sort) and the prefilter cut on the
// host, one stream round trip each.  When no event log is attached nothing of a phase needs the
// host: this kernel runs every phase with grid-wide barriers in between.  Per phase
//   build    candidates (key, slot) compacted as above, with the smallest and largest key;
//   select   when there are more than EB_CAP candidates, a radix select (12 key bits per level,
//            starting at the highest bit in which the keys differ) finds a key bound below which at
//            least `reach` = deficit / min_freed + 1 and at most EB_CAP candidates lie -- no more
//            than `reach` can be reached before the deficit is covered;
//   finish   one block sorts those (cub::BlockRadixSort), prefix-sums the bytes each would free and
//            applies the operation to exactly the prefix the reference's loop reaches.
// A phase the select cannot bound (a deficit worth more than EB_CAP operations) raises `overflow`
// and ends the kernel; the phases already finished are complete, and the host-driven path then
// continues from the state they left (a finished phase has no candidates left or met the budget).
constexpr int EB_BATCH = 4;  // slots a thread of the scans looks at together
// phase_key of the slots s0, s0 + stride, .. (EB_BATCH of them), the loads of all of them in flight together
__device__ __forceinline__ void phase_keys(const PoolDev& p, int phase, uint64_t s0, uint64_t stride, uint64_t len, uint32_t max_pos, uint64_t (&key)[EB_BATCH]) {
    SlotMeta m[EB_BATCH];
#pragma unroll
    for (int u = 0; u < EB_BATCH; ++u) m[u].st = s0 + u * stride < len ? p.state[s0 + u * stride] : ST_COLD;
#pragma unroll
    for (int u = 0; u < EB_BATCH; ++u) load_meta(p, phase, s0 + u * stride, m[u]);
#pragma unroll
    for (int u = 0; u < EB_BATCH; ++u) key[u] = phase_key(p, phase, s0 + u * stride, m[u], max_pos);
}
constexpr int EB_KEYS = 16;  // slots of a thread whose keys stay in its registers (1.2 million on 148 SMs)
constexpr int EB_FEW = 6;    // and from how many slots a thread on they do (455 000)
constexpr int EB_THREADS = 512, EB_ITEMS = 8, EB_CAP = EB_THREADS * EB_ITEMS, EB_LEVELS = 6, EB_BINS = 4096;
struct EnforceState {
    unsigned long long inv_min_key, max_key;  // ~min and max over the phase's candidates (zero = none yet)
    uint32_t n_keep, overflow, pad[2];
    ulonglong2 bounds[5];                     // ~bound of the phase's candidates and the largest of the blocks' smallest keys, see below
    uint32_t few[5], pad2;                    // how many lie within it
    uint32_t hist[5][EB_LEVELS][EB_BINS];
};

using EbScan32 = cub::BlockScan<uint32_t, EB_THREADS>;
struct CutShared {
    union {
        uint32_t hist[EB_BINS];
        typename EbScan32::TempStorage scan;
    };
    unsigned long long lo_inv, hi;
    uint32_t count, bin, in_bin, cum;
};
// A key bound that at least `reach` of the block's keys (N a thread, SENTINEL where there is none) do not exceed, or all of
// them where there are fewer: a radix select in shared memory, 12 key bits a level from the highest in which the keys differ, until at most `slack`
// more than reach are kept.  All threads of the block call; kept: how many keys are within the bound.
template <int N>
__device__ __forceinline__ uint64_t block_cut(const uint64_t (&k)[N], uint64_t reach, uint32_t slack, CutShared& sm, uint32_t& kept) {
    uint64_t lo = SENTINEL, hi = 0;
    uint32_t n = 0;
#pragma unroll
    for (int j = 0; j < N; ++j)
        if (k[j] != SENTINEL) {
            lo = min(lo, k[j]);
            hi = max(hi, k[j]);
            ++n;
        }
    for (int o = 16; o; o >>= 1) {
        lo = min(lo, __shfl_xor_sync(0xFFFFFFFFu, lo, o));
        hi = max(hi, __shfl_xor_sync(0xFFFFFFFFu, hi, o));
    }
    n = __reduce_add_sync(0xFFFFFFFFu, n);
    __syncthreads();
    if (threadIdx.x == 0) {
        sm.lo_inv = sm.hi = 0ull;
        sm.count = 0u;
    }
    __syncthreads();
    if ((threadIdx.x & 31) == 0 && n) {
        atomicMax(&sm.lo_inv, (unsigned long long)~lo);
        atomicMax(&sm.hi, (unsigned long long)hi);
        atomicAdd(&sm.count, n);
    }
    __syncthreads();
    lo = ~sm.lo_inv;
    hi = sm.hi;
    kept = sm.count;
    if (kept <= reach + slack) return hi;
    uint64_t base = lo, below = 0;
    int shift = max(0, 64 - __clzll((long long)(hi - lo)) - 12);
    for (;;) {
        __syncthreads();
        for (uint32_t b = threadIdx.x; b < EB_BINS; b += EB_THREADS) sm.hist[b] = 0u;
        __syncthreads();
#pragma unroll
        for (int j = 0; j < N; ++j)
            if (k[j] != SENTINEL && k[j] >= base && ((k[j] - base) >> shift) < (uint64_t)EB_BINS) atomicAdd(&sm.hist[(uint32_t)((k[j] - base) >> shift)], 1u);
        __syncthreads();
        uint32_t h[EB_ITEMS], mine = 0, before;
#pragma unroll
        for (int j = 0; j < EB_ITEMS; ++j) {
            h[j] = sm.hist[threadIdx.x * EB_ITEMS + j];
            mine += h[j];
        }
        __syncthreads();
        EbScan32(sm.scan).ExclusiveSum(mine, before);
        uint64_t cum = below + before;
        if (cum < reach && cum + mine >= reach) {  // (one thread: there are more than reach keys)
            for (int j = 0; j < EB_ITEMS; ++j) {
                cum += h[j];
                if (cum >= reach) {
                    sm.bin = threadIdx.x * EB_ITEMS + j;
                    sm.in_bin = h[j];
                    sm.cum = (uint32_t)cum;
                    break;
                }
            }
        }
        __syncthreads();
        const uint32_t b = sm.bin;
        kept = sm.cum;
        if (kept <= reach + slack || shift == 0) {
            const uint64_t bound = base + ((((uint64_t)b + 1) << shift) - 1);
            return bound < base ? SENTINEL - 1 : bound;
        }
        below = kept - sm.in_bin;
        base += (uint64_t)b << shift;
        shift = max(0, shift - 12);
    }
}

// Shared memory of a phase's end (block 0) and of what the blocks do before it.
struct FinishShared {
    using Sort = cub::BlockRadixSort<uint64_t, EB_THREADS, EB_ITEMS, uint32_t>;
    using Scan64 = cub::BlockScan<uint64_t, EB_THREADS>;
    union {
        typename Sort::TempStorage sort;
        typename Scan64::TempStorage scan64;
        typename EbScan32::TempStorage scan32;
        uint32_t hist[EB_BINS];
        struct { uint64_t in[EB_THREADS], key[EB_THREADS]; uint32_t val[EB_THREADS]; } few;
        CutShared cut;
    };
    unsigned long long applied;  // of the phase that ended
    long long delta;
    uint32_t n;
};
// The end of a phase, by one block: the candidates ks / vs [0 .. n), n <= EB_CAP, in order, the operation on exactly the prefix that the reference's loop reaches.  sm.applied and
// sm.delta: what was evicted, and the change of the live bytes.  CUT: for lists of the blocks' smallest keys, of which few are reached (skeys, svals: room for them).
template <bool CUT>
__device__ __forceinline__ void finish_phase(const PoolDev& p, int phase, uint64_t reach, uint64_t deficit, uint64_t free0, const uint64_t* ks, const uint32_t* vs, uint32_t n, uint64_t* skeys,
                                             uint32_t* svals, FinishShared& sm) {
    const int lane = threadIdx.x & 31;
    uint64_t k[EB_ITEMS];
    uint32_t v[EB_ITEMS];
#pragma unroll
    for (int j = 0; j < EB_ITEMS; ++j) {
        const uint32_t i = threadIdx.x * EB_ITEMS + j;
        k[j] = i < n ? ks[i] : SENTINEL;
        v[j] = i < n ? vs[i] : 0u;
    }
    if (CUT && n > EB_THREADS && reach <= EB_THREADS / 2) {  // the blocks' smallest keys together: down to what the count below orders
        uint32_t kept;
        const uint64_t bound = block_cut(k, reach, EB_THREADS / 2, sm.cut, kept);
        if (kept <= EB_THREADS) {
            if (threadIdx.x == 0) sm.n = 0u;
            __syncthreads();
#pragma unroll
            for (int j = 0; j < EB_ITEMS; ++j)
                if (k[j] != SENTINEL && k[j] <= bound) {
                    const uint32_t o = atomicAdd(&sm.n, 1u);
                    skeys[o] = k[j];  // (every key has been read: block_cut's barriers)
                    svals[o] = v[j];
                }
            __syncthreads();
            ks = skeys;
            vs = svals;
            n = kept;
        }
    }
    if (threadIdx.x == 0) {
        sm.applied = 0;
        sm.delta = 0;
    }
    __syncthreads();
    int64_t delta = 0;
    uint32_t applied = 0;
    auto weight = [&](uint64_t key, uint32_t slot) -> uint64_t {
        if (key == SENTINEL) return 0;
        const uint32_t flags = tile_flags(p.tiles, slot);
        return phase == PH_PAGE ? 32 : phase <= PH_CORR_WARM ? corr_bytes(flags) : live_bytes_of(p.state[slot], flags);
    };
    auto apply = [&](uint64_t key, uint32_t slot, uint64_t bytes, uint64_t before, uint32_t place) {
        if (key == SENTINEL || before >= deficit) return;
        if (phase == PH_PAGE) {
            do_page_out(p, slot, &delta);
        } else if (phase <= PH_CORR_WARM) {
            do_drop_correction(p, slot, &delta);
        } else {
            delta -= (int64_t)bytes;
            p.state[slot] = ST_COLD;
            p.free_list[free0 + place] = slot;  // applied items are a prefix of the sorted order
            ++applied;
        }
    };
    if (n <= EB_THREADS) {
        // few candidates (a decode step's page-outs and evictions): every thread counts the keys below its own
        // (keys are unique), n reads of shared memory instead of the radix sort's sixteen passes, and goes on with one of them in order
        const uint32_t i = threadIdx.x;
        const uint64_t own = i < n ? ks[i] : SENTINEL;
        sm.few.in[i] = own;
        __syncthreads();
        uint32_t rank = 0;
#pragma unroll 8
        for (uint32_t e = 0; e < n; ++e) rank += sm.few.in[e] < own;
        if (i < n) {
            sm.few.key[rank] = own;
            sm.few.val[rank] = vs[i];
        }
        __syncthreads();
        const uint64_t key = i < n ? sm.few.key[i] : SENTINEL;
        const uint32_t slot = i < n ? sm.few.val[i] : 0u;
        const uint64_t bytes = weight(key, slot);
        uint64_t before;
        __syncthreads();
        FinishShared::Scan64(sm.scan64).ExclusiveSum(bytes, before);
        apply(key, slot, bytes, before, i);
    } else {
        FinishShared::Sort(sm.sort).Sort(k, v);
        __syncthreads();
        uint64_t w[EB_ITEMS], excl[EB_ITEMS];
#pragma unroll
        for (int j = 0; j < EB_ITEMS; ++j) w[j] = weight(k[j], v[j]);
        FinishShared::Scan64(sm.scan64).ExclusiveSum(w, excl);
#pragma unroll
        for (int j = 0; j < EB_ITEMS; ++j) apply(k[j], v[j], w[j], excl[j], threadIdx.x * EB_ITEMS + j);
    }
    for (int o = 16; o; o >>= 1) {
        delta += __shfl_xor_sync(0xFFFFFFFFu, delta, o);
        applied += __shfl_xor_sync(0xFFFFFFFFu, applied, o);
    }
    if (lane == 0) {
        if (delta) atomicAdd((unsigned long long*)&sm.delta, (unsigned long long)delta);
        if (applied) atomicAdd(&sm.applied, (unsigned long long)applied);
    }
    __syncthreads();
}

// A decode step's budget question in one pass over the slots: no correction planes in the pool, few HOT tiles to page out, few evictions.  Paging every HOT tile
// frees 32 bytes each, so all blocks know the evictions' deficit as soon as they know how many there are, and the states, positions and the largest position come
// from the same loads: three grid barriers and one end instead of seven and two, and the host reads the answer from its own memory instead of waiting for the end and for
// two copies.  Latency bounds it: barriers, a scan whose loads are all in flight at once, and one block's ordering of a few hundred keys.  us of the whole
// call, 8 tiles appended and 8 evicted, with enforce_kernel and with this one: by importance 20 000 slots 94 / 32, 100 000 81 / 42, 1 000 000 132 / 41 (62
// while the positions were read from the tiles, a sector of every line); in causal order 69 / 32, 81 / 35, 121 / 37.  Whatever does not fit is left to enforce_kernel, with nothing changed: that costs the first scan, so the host
// also asks what it knows before (see there).
constexpr uint32_t STEP_BAIL = 1u;                  // a flag of the answer: nothing was done
struct StepState {                                  // zero when the kernel starts, and again when it ends
    struct {
        unsigned long long bound_inv, bound_low;    // ~bound of the candidates and the largest of the blocks' smallest keys, see enforce_kernel
        uint32_t few_n, all_n;                      // how many lie within it, and how many there are
    } set[2];                                       // tiles that are not pinned, then those that are
    uint32_t hot_n, max_pos;
};
struct StepAnswer {                                 // page-locked host memory
    uint64_t live, free_len;
    uint64_t hot;                                   // HOT tiles left
    uint32_t flags, no;                             // no: the call's number, written last
};
__global__ void __launch_bounds__(EB_THREADS) enforce_step_kernel(PoolDev p, uint64_t* hkeys, uint32_t* hvals, uint64_t* skeys, uint32_t* svals, StepState* ss,
                                                                  volatile StepAnswer* answer, uint32_t no) {
    namespace cg = cooperative_groups;
    cg::grid_group grid = cg::this_grid();
    __shared__ FinishShared sm;
    __shared__ uint32_t warp_n[EB_THREADS / 32];
    volatile PoolCounters* cnt = p.cnt;
    const uint64_t len = cnt->len, live = cnt->live, budget = cnt->budget, free0 = cnt->free_len;
    const uint64_t gtid = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x, stride = (uint64_t)gridDim.x * blockDim.x;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    auto say = [&](uint64_t live_now, uint64_t free_now, uint64_t hot, uint32_t flags) {  // block 0's first thread, when nobody reads *ss any more
        *ss = StepState{};
        answer->live = live_now;
        answer->free_len = free_now;
        answer->hot = hot;
        answer->flags = flags;
        __threadfence_system();
        answer->no = no;
    };
    if (live <= budget) {
        grid.sync();  // every block has read the counters: on the answer the caller may change them, on another stream
        if (gtid == 0) say(live, free0, ~0ull, 0u);
        return;
    }
    const bool by_importance = p.evict_policy == SLHA_B200_EVICT_IMPORTANCE, low_impact = p.page_policy == SLHA_B200_PAGE_LOWEST_IMPACT_FIRST;
    uint8_t st[EB_KEYS];
    uint32_t pos[EB_KEYS];
#pragma unroll
    for (int u = 0; u < EB_KEYS; ++u) st[u] = gtid + u * stride < len ? p.state[gtid + u * stride] : ST_COLD;
#pragma unroll
    for (int u = 0; u < EB_KEYS; ++u) pos[u] = by_importance && gtid + u * stride < len ? p.pos[gtid + u * stride] : 0u;
    uint32_t m = 0;
#pragma unroll
    for (int u = 0; u < EB_KEYS; ++u) m = max(m, st[u] != ST_COLD ? pos[u] : 0u);
#pragma unroll 1
    for (int u = 0; u < EB_KEYS; ++u) {
        uint8_t own = st[0];
#pragma unroll
        for (int j = 1; j < EB_KEYS; ++j) own = u == j ? st[j] : own;
        const bool hot = own == ST_HOT;
        const unsigned hit = __ballot_sync(0xFFFFFFFFu, hot);
        if (!hit) continue;
        uint32_t at = 0;
        if (lane == 0) at = atomicAdd(&ss->hot_n, (uint32_t)__popc(hit));
        at = __shfl_sync(0xFFFFFFFFu, at, 0) + (uint32_t)__popc(hit & ((1u << lane) - 1u));
        if (hot && at < (uint32_t)EB_CAP) {
            const uint64_t s = gtid + u * stride;
            hkeys[at] = low_impact ? ((uint64_t)f32_total_key(*reinterpret_cast<const float*>(p.tiles + s * TILE_BYTES + 104)) << 32) | (uint32_t)s : (uint64_t)(uint32_t)p.seq[s];
            hvals[at] = (uint32_t)s;
        }
    }
    if (p.recent_window) {
        m = __reduce_max_sync(0xFFFFFFFFu, m);
        if (lane == 0) warp_n[warp] = m;
        __syncthreads();
        if (threadIdx.x == 0) {
            for (int w = 1; w < EB_THREADS / 32; ++w) m = max(m, warp_n[w]);
            if (m) atomicMax(&ss->max_pos, m);
        }
    }
    grid.sync();
    const uint32_t hot_n = *(volatile uint32_t*)&ss->hot_n, max_pos = *(volatile uint32_t*)&ss->max_pos;
    const uint64_t deficit = live - budget, paged = 32ull * hot_n;
    const bool evicts = paged < deficit;
    const uint64_t rest = evicts ? deficit - paged : 0, reach = rest / 80 + 1;
    const bool fits = hot_n <= (uint32_t)EB_CAP && !(evicts && reach * gridDim.x > 4ull * EB_CAP);
    if (!fits || !evicts) {  // (the same for every block)
        grid.sync();         // the counts have been read
        if (blockIdx.x) return;
        if (fits) finish_phase<false>(p, PH_PAGE, deficit / 32 + 1, deficit, free0, hkeys, hvals, hot_n, skeys, svals, sm);
        if (threadIdx.x == 0) {
            const uint64_t live_now = fits ? (uint64_t)((int64_t)live + sm.delta) : live;
            if (fits) cnt->live = live_now;
            say(live_now, free0, hot_n - (live - live_now) / 32, fits ? 0u : STEP_BAIL);
        }
        return;
    }
    // Pinned tiles go last (by importance only), and only where the others free too little: 96 bytes each, once they are paged.
    uint32_t got[2] = {0u, 0u};
#pragma unroll 1
    for (int pinned = 0; pinned < 2; ++pinned) {
        uint64_t key[EB_KEYS];
        float imp[EB_KEYS];
        uint32_t seq[EB_KEYS];
        auto looks = [&](int u) { return st[u] != ST_COLD && (by_importance && is_pinned(p, pos[u], max_pos)) == (pinned != 0); };
#pragma unroll
        for (int u = 0; u < EB_KEYS; ++u) {
            imp[u] = by_importance && looks(u) ? p.importance[gtid + u * stride] : 0.0f;
            seq[u] = looks(u) ? (uint32_t)p.seq[gtid + u * stride] : 0u;
        }
#pragma unroll
        for (int u = 0; u < EB_KEYS; ++u) key[u] = !looks(u) ? SENTINEL : by_importance ? ((uint64_t)f32_total_key(imp[u]) << 32) | seq[u] : (uint64_t)seq[u];
        auto& set = ss->set[pinned];
        uint64_t* lk = skeys + pinned * EB_CAP;
        uint32_t* lv = svals + pinned * EB_CAP;
        uint32_t kept;
        const uint64_t own = block_cut(key, reach, 4u, sm.cut, kept);
        if (threadIdx.x == 0 && kept >= reach) atomicMax(&set.bound_inv, (unsigned long long)~own);
        if (threadIdx.x == 32) atomicMax(&set.bound_low, ~sm.cut.lo_inv);
        if (threadIdx.x == 64 && sm.cut.count) atomicAdd(&set.all_n, sm.cut.count);
        grid.sync();
        const unsigned long long by_blocks = ~*(volatile unsigned long long*)&set.bound_inv, by_least = *(volatile unsigned long long*)&set.bound_low;
        const uint32_t all_n = *(volatile uint32_t*)&set.all_n;
        const uint64_t bound = reach <= gridDim.x ? min(by_blocks, by_least) : by_blocks;
        uint32_t mine = 0;
#pragma unroll
        for (int j = 0; j < EB_KEYS; ++j) mine += key[j] != SENTINEL && key[j] <= bound;
        if (__any_sync(0xFFFFFFFFu, mine != 0u)) {
            uint32_t incl = mine;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, incl, o);
                if (lane >= o) incl += y;
            }
            uint32_t at = 0;
            if (lane == 31) at = atomicAdd(&set.few_n, incl);
            at = __shfl_sync(0xFFFFFFFFu, at, 31) + incl - mine;
#pragma unroll
            for (int j = 0; j < EB_KEYS; ++j)
                if (key[j] != SENTINEL && key[j] <= bound) {
                    if (at < (uint32_t)EB_CAP) {
                        lk[at] = key[j];
                        lv[at] = (uint32_t)(gtid + j * stride);
                    }
                    ++at;
                }
        }
        grid.sync();
        got[pinned] = *(volatile uint32_t*)&set.few_n;
        if (!by_importance || 96ull * all_n >= rest) break;  // (the same for every block)
    }
    if (blockIdx.x) return;
    __syncthreads();
    if (got[0] > (uint32_t)EB_CAP || got[1] > (uint32_t)EB_CAP) {
        if (threadIdx.x == 0) say(live, free0, hot_n, STEP_BAIL);
        return;
    }
    int64_t delta = 0;
    uint64_t freed = free0;
    if (hot_n) {
        finish_phase<false>(p, PH_PAGE, hot_n, deficit, free0, hkeys, hvals, hot_n, skeys, svals, sm);  // (all of them: the lists of the evictions stay as they are)
        delta += sm.delta;
        __threadfence_block();
        __syncthreads();
    }
#pragma unroll 1
    for (int pinned = 0; pinned < 2; ++pinned) {
        const uint64_t now = (uint64_t)((int64_t)live + delta);
        if (!got[pinned] || now <= budget) continue;
        const uint64_t left = now - budget;
        uint64_t* lk = skeys + pinned * EB_CAP;
        uint32_t* lv = svals + pinned * EB_CAP;
        finish_phase<true>(p, PH_EVICT, left / 80 + 1, left, freed, lk, lv, got[pinned], lk, lv, sm);
        delta += sm.delta;
        freed += sm.applied;
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        const uint64_t live_now = (uint64_t)((int64_t)live + delta);
        cnt->live = live_now;
        cnt->free_len = freed;
        say(live_now, freed, 0, 0u);
    }
}

// FEW: for pools in which a phase's smallest keys are found from registers where that can be done (see below); the other form is the faster one without that code
// (100 000 slots, 1 to 80 evictions: 62 to 71 us of the kernel, 69 to 76 with it).
template <bool FEW>
__global__ void __launch_bounds__(EB_THREADS) enforce_kernel(PoolDev p, uint32_t phase_mask, uint64_t* keys, uint32_t* vals,
                                                             uint64_t* skeys, uint32_t* svals, EnforceState* es) {
    namespace cg = cooperative_groups;
    cg::grid_group grid = cg::this_grid();
    using Scan32 = cub::BlockScan<uint32_t, EB_THREADS>;
    __shared__ FinishShared sm;
    __shared__ uint32_t cut_bin, cut_hist;
    __shared__ unsigned long long cut_cum;
    volatile PoolCounters* cnt = p.cnt;
    const uint64_t len = cnt->len;
    const uint64_t gtid = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x, stride = (uint64_t)gridDim.x * blockDim.x;
    const int lane = threadIdx.x & 31;
    if (cnt->live <= cnt->budget) return;  // (nothing has been written yet: every block sees the same)
    __shared__ uint32_t warp_n[EB_THREADS / 32], block_base;
    __shared__ unsigned long long block_min_inv, block_max;
    const int warp = threadIdx.x >> 5;
    if (p.recent_window) {
        uint32_t m = 0;
        for (uint64_t s0 = gtid; s0 < len; s0 += EB_BATCH * stride) {  // (the loads of a batch are in flight together)
            uint8_t st[EB_BATCH];
            uint32_t pos[EB_BATCH];
#pragma unroll
            for (int u = 0; u < EB_BATCH; ++u) st[u] = s0 + u * stride < len ? p.state[s0 + u * stride] : ST_COLD;
#pragma unroll
            for (int u = 0; u < EB_BATCH; ++u)
                pos[u] = st[u] != ST_COLD ? p.pos[s0 + u * stride] : 0u;
#pragma unroll
            for (int u = 0; u < EB_BATCH; ++u) m = max(m, pos[u]);
        }
        m = __reduce_max_sync(0xFFFFFFFFu, m);
        if (lane == 0) warp_n[warp] = m;
        __syncthreads();
        if (threadIdx.x == 0) {
            for (int w = 1; w < EB_THREADS / 32; ++w) m = max(m, warp_n[w]);
            if (m) atomicMax(&p.cnt->max_pos, m);
        }
        grid.sync();
    }
    const uint32_t max_pos = cnt->max_pos;
    for (int phase = 0; phase < 5; ++phase) {
        if (!((phase_mask >> phase) & 1u)) continue;
        const uint64_t live = cnt->live, budget = cnt->budget;
        if (live <= budget) break;
        const uint64_t deficit = live - budget;
        const uint64_t min_freed = phase == PH_PAGE ? 32 : (phase >= PH_EVICT ? 80 : 14);
        const uint64_t reach = deficit / min_freed + 1;
        // ---- a decode step's deficit (a few operations) in a large pool: every block finds a bound that `reach` of its own keys do not
        //      exceed, and the smallest of the blocks' bounds is one for all candidates; so is the largest of the blocks' smallest keys, where
        //      there are `reach` blocks or more (the better one where keys lie in random order: 1 000 000 slots, 80 evictions 179 -> 132 us).  The few keys
        //      within both go to the last block's sort from registers: one scan and two grid barriers, where the list of all
        //      candidates below takes a write and three reads, global histograms and three barriers.  The block's own selection costs more than the list while
        //      that is read in a round or two (us of the kernel, 16 evictions by importance, without and with: 100 000 slots 65 / 84, 300 000 73 / 88,
        //      500 000 93 / 96, 650 000 101 / 102, 1 000 000 136 / 120; in causal order 59 / 71, 69 / 76, 84 / 81, 93 / 87, 126 / 108;
        //      all with the positions read from the tiles).
        bool few = FEW && reach * gridDim.x <= 4ull * EB_CAP;
        if (FEW && few) {
            uint64_t key[EB_KEYS];
#pragma unroll
            for (int b = 0; b < EB_KEYS; b += EB_BATCH) {
                uint64_t part[EB_BATCH];
                phase_keys(p, phase, gtid + b * stride, stride, len, max_pos, part);
#pragma unroll
                for (int u = 0; u < EB_BATCH; ++u) key[b + u] = part[u];
            }
            uint32_t kept;
            const uint64_t own = block_cut(key, reach, 4u, sm.cut, kept);
            if (threadIdx.x == 0 && kept >= reach) atomicMax(&es->bounds[phase].x, (unsigned long long)~own);  // (a block with fewer keys bounds nothing)
            if (threadIdx.x == 32) atomicMax(&es->bounds[phase].y, ~sm.cut.lo_inv);                            // (SENTINEL from a block without keys)
            grid.sync();
            const ulonglong2 bounds = __ldcg(&es->bounds[phase]);
            const uint64_t bound = reach <= gridDim.x ? min(~bounds.x, bounds.y) : ~bounds.x;
            uint32_t mine = 0;
#pragma unroll
            for (int j = 0; j < EB_KEYS; ++j) mine += key[j] != SENTINEL && key[j] <= bound;
            if (__any_sync(0xFFFFFFFFu, mine != 0u)) {
                uint32_t incl = mine;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, incl, o);
                    if (lane >= o) incl += y;
                }
                uint32_t at = 0;
                if (lane == 31) at = atomicAdd(&es->few[phase], incl);
                at = __shfl_sync(0xFFFFFFFFu, at, 31) + incl - mine;
#pragma unroll
                for (int j = 0; j < EB_KEYS; ++j)
                    if (key[j] != SENTINEL && key[j] <= bound) {
                        if (at < (uint32_t)EB_CAP) {
                            skeys[at] = key[j];
                            svals[at] = (uint32_t)(gtid + j * stride);
                        }
                        ++at;
                    }
            }
            grid.sync();
            const uint32_t got = *(volatile uint32_t*)&es->few[phase];
            if (got == 0) continue;                 // no candidates (every block sees the same)
            few = got <= (uint32_t)EB_CAP;          // (else the general path below)
        }
        // ---- build
        if (!few) {
            // One reservation per block and batch, one minimum and maximum per block: an atomic per warp on the same word
            // costs more than the scan itself (32 k of them for a million slots).
            uint64_t kmin = SENTINEL, kmax = 0;
            const uint64_t batches = (len + EB_BATCH * stride - 1) / (EB_BATCH * stride);
            for (uint64_t r = 0; r < batches; ++r) {
                const uint64_t s0 = r * EB_BATCH * stride + gtid;
                uint64_t key[EB_BATCH];
                phase_keys(p, phase, s0, stride, len, max_pos, key);
                uint32_t mine = 0;
#pragma unroll
                for (int u = 0; u < EB_BATCH; ++u) mine += key[u] != SENTINEL;
                uint32_t incl = mine;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, incl, o);
                    if (lane >= o) incl += y;
                }
                if (lane == 31) warp_n[warp] = incl;
                __syncthreads();
                if (threadIdx.x == 0) {
                    uint32_t tot = 0;
                    for (int w = 0; w < EB_THREADS / 32; ++w) {
                        const uint32_t x = warp_n[w];
                        warp_n[w] = tot;
                        tot += x;
                    }
                    block_base = tot ? atomicAdd(&p.cnt->n_cand, tot) : 0u;
                }
                __syncthreads();
                uint32_t at = block_base + warp_n[warp] + incl - mine;
#pragma unroll
                for (int u = 0; u < EB_BATCH; ++u)
                    if (key[u] != SENTINEL) {
                        keys[at] = key[u];
                        vals[at] = (uint32_t)(s0 + u * stride);
                        ++at;
                        kmin = min(kmin, key[u]);
                        kmax = max(kmax, key[u]);
                    }
                __syncthreads();  // (the counts are reused by the next batch)
            }
            for (int o = 16; o; o >>= 1) {
                kmin = min(kmin, __shfl_xor_sync(0xFFFFFFFFu, kmin, o));
                kmax = max(kmax, __shfl_xor_sync(0xFFFFFFFFu, kmax, o));
            }
            if (threadIdx.x == 0) block_min_inv = block_max = 0ull;
            __syncthreads();
            if (lane == 0 && kmin != SENTINEL) {
                atomicMax(&block_min_inv, (unsigned long long)~kmin);
                atomicMax(&block_max, (unsigned long long)kmax);
            }
            __syncthreads();
            if (threadIdx.x == 0 && block_min_inv) {
                atomicMax(&es->inv_min_key, block_min_inv);
                atomicMax(&es->max_key, block_max);
            }
        }
        if (!few) grid.sync();
        const uint64_t nc = cnt->n_cand;
        if (nc || few) {
            const bool take_all = !few && nc <= (uint64_t)EB_CAP;
            uint64_t base = ~*(volatile unsigned long long*)&es->inv_min_key, thr_rel = ~0ull, below = 0;
            bool bounded = take_all || few;
            if (!bounded && reach <= (uint64_t)EB_CAP) {
                const uint64_t span = *(volatile unsigned long long*)&es->max_key - base;
                int shift = max(0, 64 - __clzll((long long)span) - 12);
                for (int level = 0; level < EB_LEVELS && !bounded; ++level) {
                    uint32_t* ghist = es->hist[phase][level];
                    for (uint32_t b = threadIdx.x; b < EB_BINS; b += EB_THREADS) sm.hist[b] = 0;
                    __syncthreads();
                    for (uint64_t i = gtid; i < nc; i += stride) {
                        const uint64_t k = keys[i];
                        if (k >= base && ((k - base) >> shift) < (uint64_t)EB_BINS) atomicAdd(&sm.hist[(uint32_t)((k - base) >> shift)], 1u);
                    }
                    __syncthreads();
                    for (uint32_t b = threadIdx.x; b < EB_BINS; b += EB_THREADS)
                        if (sm.hist[b]) atomicAdd(&ghist[b], sm.hist[b]);
                    grid.sync();
                    // every block finds the cut itself: the first bin at which `below` + the running count reaches `reach`
                    uint32_t h[EB_ITEMS], mine = 0;
                    for (int j = 0; j < EB_ITEMS; ++j) {
                        h[j] = *(volatile uint32_t*)&ghist[threadIdx.x * EB_ITEMS + j];
                        mine += h[j];
                    }
                    if (threadIdx.x == 0) cut_bin = 0xFFFFFFFFu;
                    __syncthreads();
                    uint32_t before;
                    Scan32(sm.scan32).ExclusiveSum(mine, before);
                    uint64_t cum = below + before;
                    if (cum < reach && cum + mine >= reach) {
                        for (int j = 0; j < EB_ITEMS; ++j) {
                            cum += h[j];
                            if (cum >= reach) {
                                cut_bin = threadIdx.x * EB_ITEMS + j;
                                cut_hist = h[j];
                                cut_cum = cum;
                                break;
                            }
                        }
                    }
                    __syncthreads();
                    const uint32_t b = cut_bin;
                    const uint64_t kept = cut_cum;
                    const uint32_t hb = cut_hist;
                    __syncthreads();
                    if (b == 0xFFFFFFFFu) break;  // fewer candidates than `reach`: all of them are needed, and they do not fit
                    if (kept <= (uint64_t)EB_CAP) {
                        thr_rel = (((uint64_t)b + 1) << shift) - 1;
                        bounded = true;
                    } else if (shift == 0) {
                        break;  // equal keys beyond the block sort's capacity
                    } else {
                        below = kept - hb;
                        base += (uint64_t)b << shift;
                        shift = max(0, shift - 12);
                    }
                }
            }
            if (!bounded) {
                if (gtid == 0) es->overflow = 1;
                return;  // every block takes this branch
            }
            if (!take_all && !few) {
                const uint64_t rounds = (nc + stride - 1) / stride;
                for (uint64_t r = 0; r < rounds; ++r) {
                    const uint64_t i = r * stride + gtid;
                    uint64_t k = 0;
                    bool keep = false;
                    if (i < nc) {
                        k = keys[i];
                        keep = k < base || (k - base) <= thr_rel;
                    }
                    const unsigned hit = __ballot_sync(0xFFFFFFFFu, keep);
                    if (hit) {
                        uint32_t o = 0;
                        if (lane == 0) o = atomicAdd(&es->n_keep, (uint32_t)__popc(hit));
                        o = __shfl_sync(0xFFFFFFFFu, o, 0) + (uint32_t)__popc(hit & ((1u << lane) - 1u));
                        if (keep && o < (uint32_t)EB_CAP) {
                            skeys[o] = k;
                            svals[o] = vals[i];
                        }
                    }
                }
                grid.sync();
            }
            // ---- finish (block 0)
            if (blockIdx.x == 0) {
                const uint64_t* ks = take_all ? keys : skeys;
                const uint32_t* vs = take_all ? vals : svals;
                uint32_t n = take_all ? (uint32_t)nc : (few ? *(volatile uint32_t*)&es->few[phase] : min(*(volatile uint32_t*)&es->n_keep, (uint32_t)EB_CAP));
                finish_phase<FEW>(p, phase, reach, deficit, cnt->free_len, ks, vs, n, skeys, svals, sm);
                if (threadIdx.x == 0) {
                    cnt->live = (uint64_t)((int64_t)live + sm.delta);
                    cnt->free_len += sm.applied;
                    cnt->n_cand = 0;
                    es->inv_min_key = 0;
                    es->max_key = 0;
                    es->n_keep = 0;
                    __threadfence();
                }
            }
        }
        grid.sync();
    }
}

// ---- observe_scores (ccos.rs:275-314) -----------------------------------------
struct ObserveTmp {
    uint32_t max_key;   // order-preserving key of the max live score
    uint32_t bad;       // a live score is non-finite
    uint32_t live;      // number of live entries
    uint32_t pad;
    float sum;
};
// (one set of atomics per CTA, and a grid of a few CTAs per SM: an atomic per warp on the same words costs more than the scan)
__global__ void __launch_bounds__(256) observe_pass1(PoolDev p, const uint32_t* slots, const float* scores, uint64_t n, ObserveTmp* tmp) {
    dep_launch();
    dep_wait();
    __shared__ uint32_t red[3];
    if (threadIdx.x < 3) red[threadIdx.x] = 0u;
    __syncthreads();
    const uint64_t len = p.cnt->len, stride = (uint64_t)gridDim.x * blockDim.x;
    uint32_t mk = 0, bad = 0, live = 0;
    for (uint64_t i0 = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i0 < n; i0 += 4 * stride) {
        uint64_t s[4];
        float v[4];
        uint8_t st[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const uint64_t i = i0 + u * stride;
            s[u] = i < n ? (slots ? slots[i] : i) : len;
            v[u] = i < n ? scores[i] : 0.0f;
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) st[u] = s[u] < len ? p.state[s[u]] : ST_COLD;
#pragma unroll
        for (int u = 0; u < 4; ++u)
            if (st[u] != ST_COLD) {
                ++live;
                if (!isfinite(v[u])) bad = 1;
                mk = max(mk, f32_total_key(v[u]));
            }
    }
    mk = __reduce_max_sync(0xFFFFFFFFu, mk);
    bad = __reduce_or_sync(0xFFFFFFFFu, bad);
    live = __reduce_add_sync(0xFFFFFFFFu, live);
    if ((threadIdx.x & 31) == 0) {
        atomicMax(&red[0], mk);
        if (bad) atomicOr(&red[1], 1u);
        atomicAdd(&red[2], live);
    }
    __syncthreads();
    if (threadIdx.x == 0 && red[2]) {
        atomicMax(&tmp->max_key, red[0]);
        if (red[1]) atomicOr(&tmp->bad, 1u);
        atomicAdd(&tmp->live, red[2]);
    }
}
__device__ __forceinline__ float key_to_f32(uint32_t k) {
    return __uint_as_float((k & 0x80000000u) ? (k & 0x7FFFFFFFu) : ~k);
}
// per-CTA partial sums of exp((s-m)/T) in a fixed order (deterministic)
__global__ void observe_pass2(PoolDev p, const uint32_t* slots, const float* scores, uint64_t n,
                              float temperature, const ObserveTmp* tmp, float* partial) {
    dep_launch();
    dep_wait();
    __shared__ float red[32];
    const uint64_t len = p.cnt->len;
    const float m = key_to_f32(tmp->max_key);
    float acc = 0.0f;
    if (!tmp->bad && tmp->live) {
        const uint64_t per = (n + gridDim.x - 1) / gridDim.x;
        const uint64_t lo = (uint64_t)blockIdx.x * per, hi = min(n, lo + per);
        for (uint64_t i0 = lo + threadIdx.x; i0 < hi; i0 += 4 * blockDim.x) {  // (four entries' loads in flight, added in order)
            uint64_t s[4];
            float v[4];
            uint8_t st[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const uint64_t i = i0 + u * blockDim.x;
                s[u] = i < hi ? (slots ? slots[i] : (uint32_t)i) : len;
                v[u] = i < hi ? scores[i] : 0.0f;
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) st[u] = s[u] < len ? p.state[s[u]] : ST_COLD;
#pragma unroll
            for (int u = 0; u < 4; ++u)
                if (st[u] != ST_COLD) acc += expf((v[u] - m) / temperature);
        }
    }
    for (int o = 16; o; o >>= 1) acc += __shfl_xor_sync(0xFFFFFFFFu, acc, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
    __syncthreads();
    if (threadIdx.x == 0) {
        float t = 0.0f;
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t += red[w];
        partial[blockIdx.x] = t;
    }
}
__global__ void observe_pass3(PoolDev p, const uint32_t* slots, const float* scores, uint64_t n,
                              float temperature, ObserveTmp* tmp, const float* partial, int n_partial) {
    dep_launch();
    dep_wait();
    __shared__ float s_inv, part[256];
    for (int i = threadIdx.x; i < n_partial; i += blockDim.x) part[i] = partial[i];  // (n_partial <= 256)
    __syncthreads();
    if (threadIdx.x == 0) {
        float sum = 0.0f;
#pragma unroll 16
        for (int i = 0; i < n_partial; ++i) sum += part[i];
        s_inv = (tmp->bad || !tmp->live || !isfinite(sum) || sum <= 0.0f) ? 0.0f : 1.0f / sum;
    }
    __syncthreads();
    const float inv = s_inv;
    if (inv == 0.0f) return;
    const uint64_t len = p.cnt->len, stride = (uint64_t)gridDim.x * blockDim.x;
    const float m = key_to_f32(tmp->max_key);
    for (uint64_t i0 = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i0 < n; i0 += 4 * stride) {
        uint64_t s[4];
        float v[4], old[4];
        uint8_t st[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const uint64_t i = i0 + u * stride;
            s[u] = i < n ? (slots ? slots[i] : (uint32_t)i) : len;
            v[u] = i < n ? scores[i] : 0.0f;
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            st[u] = s[u] < len ? p.state[s[u]] : ST_COLD;
            old[u] = !slots && s[u] < len ? p.importance[s[u]] : 0.0f;
        }
#pragma unroll
        for (int u = 0; u < 4; ++u)
            if (st[u] != ST_COLD) {
                const float w = expf((v[u] - m) / temperature) * inv;
                if (slots) atomicAdd(&p.importance[s[u]], w);  // (a caller's list may name a slot twice)
                else p.importance[s[u]] = __fadd_rn(old[u], w);
            }
    }
}

// The three passes over all slots (observe_query) in one: a thread keeps its entries' terms and importances in registers between two grid barriers.  The shares, and so
// the order of the sum, are pass 2's: half a CTA is one of its 256.  Latency bounds it, three loads' and two barriers': a million slots 22 us with the clear
// and the three kernels, 13 with this one.
constexpr int OBSERVE_PARTS = 256, OBSERVE_KEEP = 16;  // entries a thread: up to 1 048 576 slots, since the parts of the sum, and with them its order, stay pass 2's 256
__global__ void __launch_bounds__(512) observe_all_kernel(PoolDev p, const float* scores, uint64_t n, float temperature, ObserveTmp* tmp, float* partial) {
    cooperative_groups::grid_group grid = cooperative_groups::this_grid();
    __shared__ uint32_t red[3];
    __shared__ float warp_sum[16], part[OBSERVE_PARTS], s_inv;
    const int tid = threadIdx.x;
    if (tid < 3) red[tid] = 0u;
    __syncthreads();
    const uint64_t len = p.cnt->len, per = (n + OBSERVE_PARTS - 1) / OBSERVE_PARTS;
    const uint64_t lo = (2ull * blockIdx.x + (tid >> 8)) * per, hi = min(n, lo + per), i0 = lo + (tid & 255);
    float v[OBSERVE_KEEP], old[OBSERVE_KEEP];
    uint32_t on = 0u;
#pragma unroll
    for (int u = 0; u < OBSERVE_KEEP; ++u) {
        const uint64_t i = i0 + 256 * u;
        const bool in = i < hi;
        v[u] = in ? scores[i] : 0.0f;
        if (in && i < len && p.state[i] != ST_COLD) on |= 1u << u;
    }
    uint32_t mk = 0, bad = 0;
#pragma unroll
    for (int u = 0; u < OBSERVE_KEEP; ++u)
        if (on >> u & 1u) {
            if (!isfinite(v[u])) bad = 1;
            mk = max(mk, f32_total_key(v[u]));
        }
#pragma unroll
    for (int u = 0; u < OBSERVE_KEEP; ++u) old[u] = on >> u & 1u ? p.importance[i0 + 256 * u] : 0.0f;
    mk = __reduce_max_sync(0xFFFFFFFFu, mk);
    bad = __reduce_or_sync(0xFFFFFFFFu, bad);
    const uint32_t live = __reduce_add_sync(0xFFFFFFFFu, (uint32_t)__popc(on));
    if ((tid & 31) == 0) {
        atomicMax(&red[0], mk);
        if (bad) atomicOr(&red[1], 1u);
        atomicAdd(&red[2], live);
    }
    __syncthreads();
    if (tid == 0 && red[2]) {
        atomicMax(&tmp->max_key, red[0]);
        if (red[1]) atomicOr(&tmp->bad, 1u);
        atomicAdd(&tmp->live, red[2]);
    }
    grid.sync();
    volatile ObserveTmp* all = tmp;
    const float m = key_to_f32(all->max_key);
    const bool usable = !all->bad && all->live;
    float acc = 0.0f;
    if (usable)
#pragma unroll
        for (int u = 0; u < OBSERVE_KEEP; ++u)
            if (on >> u & 1u) {
                v[u] = expf((v[u] - m) / temperature);
                acc += v[u];
            }
    for (int o = 16; o; o >>= 1) acc += __shfl_xor_sync(0xFFFFFFFFu, acc, o);
    if ((tid & 31) == 0) warp_sum[tid >> 5] = acc;
    __syncthreads();
    if ((tid & 255) == 0) {
        float t = 0.0f;
        for (int w = 0; w < 8; ++w) t += warp_sum[(tid >> 5) + w];
        partial[2 * blockIdx.x + (tid >> 8)] = t;
    }
    grid.sync();
    if (blockIdx.x == 0 && tid == 0) *tmp = ObserveTmp{};  // (everyone has read it)
    if (tid < OBSERVE_PARTS) part[tid] = __ldcg(partial + tid);
    __syncthreads();
    if (tid == 0) {
        float sum = 0.0f;
#pragma unroll 16
        for (int i = 0; i < OBSERVE_PARTS; ++i) sum += part[i];
        s_inv = (!usable || !isfinite(sum) || sum <= 0.0f) ? 0.0f : 1.0f / sum;
    }
    __syncthreads();
    const float inv = s_inv;
    if (inv == 0.0f) return;
#pragma unroll
    for (int u = 0; u < OBSERVE_KEEP; ++u)
        if (on >> u & 1u) p.importance[i0 + 256 * u] = __fadd_rn(old[u], __fmul_rn(v[u], inv));
}

// ---- stats / compaction ---------------------------------------------------------
// The CTAs' sums meet behind a grid barrier and the first CTA answers in the host's memory (a clear and a copy less: 4096 slots
// 23 us a call, now 16; a million with correction planes 46, now 40).
__global__ void __launch_bounds__(512) stats_kernel(PoolDev p, uint32_t* sums, volatile unsigned long long* answer, unsigned long long no, bool planes) {
    __shared__ uint32_t red[5];
    __shared__ unsigned long long total[5];
    if (threadIdx.x < 5) red[threadIdx.x] = 0u, total[threadIdx.x] = 0ull;
    __syncthreads();
    const uint64_t len = p.cnt->len, stride = (uint64_t)gridDim.x * blockDim.x;
    uint32_t v[5] = {0, 0, 0, 0, 0};  // hot, warm, cold, without correction plane, bytes it gave back (per thread: below 2^32 slots)
    if (planes) {
        for (uint64_t s0 = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; s0 < len; s0 += 4 * stride) {
            uint8_t st[4];
            uint32_t flags[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) st[u] = s0 + u * stride < len ? p.state[s0 + u * stride] : 0xFFu;
#pragma unroll
            for (int u = 0; u < 4; ++u) flags[u] = st[u] == ST_HOT || st[u] == ST_WARM ? tile_flags(p.tiles, s0 + u * stride) : 0u;
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                if (st[u] == 0xFFu) continue;
                v[0] += st[u] == ST_HOT;
                v[1] += st[u] == ST_WARM;
                v[2] += st[u] != ST_HOT && st[u] != ST_WARM;
                if (flags[u] & F_NOCORR) { ++v[3]; v[4] += corr_bytes(flags[u]); }
            }
        }
    } else {  // states only, sixteen a load
        for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < len / 16; i += stride) {
            const uint4 x = reinterpret_cast<const uint4*>(p.state)[i];
            const uint32_t w[4] = {x.x, x.y, x.z, x.w};
            uint32_t hot = 0, warm = 0;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                hot += __popc(__vcmpeq4(w[j], 0x01010101u * ST_HOT)) >> 3;
                warm += __popc(__vcmpeq4(w[j], 0x01010101u * ST_WARM)) >> 3;
            }
            v[0] += hot;
            v[1] += warm;
            v[2] += 16u - hot - warm;
        }
        if (blockIdx.x == 0 && threadIdx.x < len % 16) {
            const uint8_t st = p.state[len / 16 * 16 + threadIdx.x];
            v[0] += st == ST_HOT;
            v[1] += st == ST_WARM;
            v[2] += st != ST_HOT && st != ST_WARM;
        }
    }
#pragma unroll
    for (int i = 0; i < 5; ++i) {
        const uint32_t t = __reduce_add_sync(0xFFFFFFFFu, v[i]);
        if ((threadIdx.x & 31) == 0 && t) atomicAdd(&red[i], t);
    }
    __syncthreads();
    if (threadIdx.x < 5) sums[8 * blockIdx.x + threadIdx.x] = red[threadIdx.x];
    cooperative_groups::this_grid().sync();
    if (blockIdx.x) return;
    for (uint32_t i = threadIdx.x; i < 8 * gridDim.x; i += blockDim.x)
        if ((i & 7u) < 5u) atomicAdd(&total[i & 7u], (unsigned long long)__ldcg(sums + i));
    __syncthreads();
    if (threadIdx.x) return;
    for (int i = 0; i < 5; ++i) answer[2 + i] = total[i];
    answer[0] = len;
    answer[1] = p.cnt->live;
    answer[7] = p.cnt->free_len;
    __threadfence_system();
    answer[8] = no;
}
// ordered compaction of the non-COLD (slot, score) pairs; one CTA
__global__ void compact_live_kernel(PoolDev p, const float* scores, uint32_t* slots_out,
                                    float* scores_out, unsigned long long* n_out) {
    __shared__ uint32_t warp_tot[32];
    __shared__ uint32_t base_s;
    const uint64_t len = p.cnt->len;
    if (threadIdx.x == 0) base_s = 0;
    __syncthreads();
    for (uint64_t b = 0; b < len; b += blockDim.x) {
        const uint64_t s = b + threadIdx.x;
        const bool live = s < len && p.state[s] != ST_COLD;
        const unsigned bal = __ballot_sync(0xFFFFFFFFu, live);
        const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
        if (lane == 0) warp_tot[wp] = __popc(bal);
        __syncthreads();
        uint32_t off = base_s;
        for (int w = 0; w < wp; ++w) off += warp_tot[w];
        if (live) {
            const uint32_t o = off + __popc(bal & ((1u << lane) - 1));
            slots_out[o] = (uint32_t)s;
            scores_out[o] = scores[s];
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            uint32_t t = 0;
            for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t += warp_tot[w];
            base_s += t;
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) *n_out = base_s;
}

inline uint32_t grid_for(uint64_t n, int threads = 256) {
    return (uint32_t)std::min<uint64_t>(std::max<uint64_t>(1, (n + threads - 1) / threads), 148 * 8);
}

}  // namespace

Status pool_sync_counters(Ctx* c, Pool* pl) {
    SLHA_CUDA(cudaMemcpyAsync(&pl->h_cnt, pl->dev.cnt, sizeof(PoolCounters), cudaMemcpyDeviceToHost, c->stream));
    SLHA_CUDA(cudaStreamSynchronize(c->stream));
    pl->unread = 0;
    return Status();
}

Status pool_create(Ctx* c, const SlhaB200PoolConfig& cfg, Pool** out) {
    auto* pl = new Pool();
    pl->cfg = cfg;
    pl->device = c->device;
    const uint64_t cap = cfg.capacity_tiles;
    PoolDev& d = pl->dev;
    cudaError_t e = cudaSuccess;
    auto alloc = [&](void** p, size_t bytes) { if (e == cudaSuccess) e = cudaMalloc(p, std::max<size_t>(bytes, 256)); };
    alloc((void**)&d.tiles, cap * TILE_BYTES);
    alloc((void**)&d.state, cap);
    alloc((void**)&d.seq, cap * 8);
    alloc((void**)&d.importance, cap * 4);
    alloc((void**)&d.pos, cap * 4);
    alloc((void**)&d.free_list, cap * 4);
    alloc((void**)&d.cnt, sizeof(PoolCounters));
    if (e != cudaSuccess) {
        pool_destroy(pl);
        return cuda_status(e, "cudaMalloc(pool)");
    }
    d.page_policy = cfg.page_policy;
    d.evict_policy = cfg.evict_policy;
    d.sink_window = cfg.sink_window;
    d.recent_window = cfg.recent_window;
    PoolCounters z{};
    z.budget = cfg.budget_bytes;
    pl->h_cnt = z;
    SLHA_CUDA(cudaMemcpyAsync(d.cnt, &pl->h_cnt, sizeof(z), cudaMemcpyHostToDevice, c->stream));
    SLHA_CUDA(cudaStreamSynchronize(c->stream));
    *out = pl;
    return Status();
}

void pool_destroy(Pool* pl) {
    if (!pl) return;
    cudaFree(pl->dev.tiles);
    cudaFree(pl->dev.state);
    cudaFree(pl->dev.seq);
    cudaFree(pl->dev.importance);
    cudaFree(pl->dev.pos);
    cudaFree(pl->dev.free_list);
    cudaFree(pl->dev.cnt);
    cudaFree(pl->d_observe);
    cudaFree(pl->d_step);
    if (pl->log) eventlog_close(pl->log);
    delete pl;
}

// Reserve slots for n tiles (bookkeeping only); d_slots receives the slot ids.
Status pool_reserve(Ctx* c, Pool* pl, const unsigned char* d_src_tiles, uint64_t n, uint32_t* d_slots, const uint32_t* d_positions, uint32_t position_base) {
    PoolCounters& h = pl->h_cnt;
    if (h.next_seq + n > 0xFFFFFFFFull)
        return Status(SLHA_ERR_CAPACITY, "pool: insertion counter exhausted (2^32 inserts)");
    const uint64_t pops = std::min<uint64_t>(n, h.free_len);
    if (h.len + (n - pops) > pl->cfg.capacity_tiles)
        return Status(SLHA_ERR_CAPACITY, "pool: capacity_tiles exceeded");
    SLHA_CUDA(launch_behind(insert_kernel, dim3((uint32_t)((n + 255) / 256)), dim3(256), 0, c->stream, pl->dev, d_src_tiles, n, pops, h.len, h.free_len,
                            h.next_seq, d_positions, position_base, d_slots));
    count_launch();
    h.free_len -= pops;
    h.len += n - pops;
    h.next_seq += n;
    pl->hot_most += n;
    pl->unread += n;
    return Status();
}

Status pool_scatter(Ctx* c, Pool* pl, const unsigned char* d_src_tiles, const uint32_t* d_slots, uint64_t n) {
    scatter_tiles_kernel<<<(uint32_t)((n * 8 + 255) / 256), 256, 0, c->stream>>>(pl->dev.tiles, d_src_tiles, d_slots, n);
    count_launch();
    SLHA_CUDA(cudaGetLastError());
    return Status();
}

Status pool_single_op(Ctx* c, Pool* pl, int op, uint32_t slot, int32_t* result) {
    if (op == 2 && (pl->log || pl->require_durable)) {
        // evict with an event log attached (ccos.rs:404-438): persist the record, then (and only then) go COLD
        SLHA_TRY(pool_sync_counters(c, pl));
        uint8_t st = ST_COLD;
        if (slot < pl->h_cnt.len) SLHA_CUDA(cudaMemcpyAsync(&st, pl->dev.state + slot, 1, cudaMemcpyDeviceToHost, c->stream));
        SLHA_CUDA(cudaStreamSynchronize(c->stream));
        if (st == ST_COLD) {
            *result = 0;
            return Status();
        }
        uint64_t seq = 0;
        unsigned char tile[TILE_BYTES];
        SLHA_CUDA(cudaMemcpyAsync(&seq, pl->dev.seq + slot, 8, cudaMemcpyDeviceToHost, c->stream));
        SLHA_CUDA(cudaMemcpyAsync(tile, pl->dev.tiles + (size_t)slot * TILE_BYTES, TILE_BYTES, cudaMemcpyDeviceToHost, c->stream));
        SLHA_CUDA(cudaStreamSynchronize(c->stream));
        const bool ok = pl->log && eventlog_append(pl->log, seq, slot, tile, pl->require_durable).ok();
        if (!ok) {
            if (pl->log) ++pl->log_errors;
            if (pl->require_durable) {
                ++pl->blocked_evictions;
                *result = 0;
                return Status();
            }
        }
    }
    int32_t* d_res;
    SLHA_TRY(ctx_device_scratch(c, 256, (void**)&d_res));
    single_op_kernel<<<1, 1, 0, c->stream>>>(pl->dev, op, slot, d_res);
    count_launch();
    SLHA_CUDA(cudaGetLastError());
    SLHA_CUDA(cudaMemcpyAsync(result, d_res, 4, cudaMemcpyDeviceToHost, c->stream));
    return pool_sync_counters(c, pl);
}

// Device memory of enforce_step_kernel: state, lists.
static Status pool_step_memory(Pool* pl) {
    if (!pl->d_step) {
        SLHA_CUDA(cudaMalloc(&pl->d_step, 256 + 3 * (size_t)EB_CAP * 12));
        pl->step_clean = false;
    }
    return Status();
}
// Until the stream's last kernel has answered.  The host polls for as long as a decode step's kernels may take (the answer is there some us before the runtime knows of the kernel's end), but
// not where its threads are to sleep while they wait (cudaDeviceScheduleBlockingSync); behind more work than that it waits for the stream as everywhere.  The library's own stream is drained.
constexpr long POLL_US = 200;
template <typename There>
static Status wait_answer(Ctx* c, There there) {
    unsigned flags = 0;
    SLHA_CUDA(cudaGetDeviceFlags(&flags));
    if ((flags & cudaDeviceScheduleMask) != cudaDeviceScheduleBlockingSync) {
        const auto since = std::chrono::steady_clock::now();
        for (uint32_t i = 1; !there(); ++i)
            if (i % 64 == 0 && std::chrono::steady_clock::now() - since > std::chrono::microseconds(POLL_US)) break;
    }
    if (!there() || c->own_stream) SLHA_CUDA(cudaStreamSynchronize(c->stream));
    return there() ? Status() : Status(SLHA_ERR_DEVICE, "the kernel ended without an answer");
}

// One cooperative launch for all phases, one read-back of the counters.  Sets *done when the
// budget question is settled; leaves it clear when a phase needs the host-driven path.
static Status pool_enforce_budget_fused(Ctx* c, Pool* pl, int32_t* within, bool* done) {
    *done = false;
    static int blocks_per_sm[64] = {0}, sms[64] = {0};
    const int dev = pl->device & 63;
    if (!blocks_per_sm[dev]) {
        int coop = 0, n = 0, b = 0, f = 0;
        SLHA_CUDA(cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, pl->device));
        SLHA_CUDA(cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, pl->device));
        SLHA_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, enforce_kernel<false>, EB_THREADS, 0));
        SLHA_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&f, enforce_kernel<true>, EB_THREADS, 0));
        b = std::min(b, f);
        sms[dev] = n;
        blocks_per_sm[dev] = coop && b > 0 ? std::min(b, 2) : -1;
    }
    if (blocks_per_sm[dev] < 0) return Status();
    const uint64_t len = pl->h_cnt.len, free_before = pl->h_cnt.free_len;  // (the host mirror of both is exact: inserts and calls that read them back move them)
    if (len == 0) return Status();
    Scratch sc{c};
    SLHA_TRY(sc.reserve(pad256(len * 8) + pad256(len * 4) + pad256(EB_CAP * 8) + pad256(EB_CAP * 4) + pad256(sizeof(EnforceState)) + 4096));
    uint64_t* keys = sc.take<uint64_t>(len);
    uint32_t* vals = sc.take<uint32_t>(len);
    uint64_t* skeys = sc.take<uint64_t>(EB_CAP);
    uint32_t* svals = sc.take<uint32_t>(EB_CAP);
    EnforceState* es = sc.take<EnforceState>(1);
    uint32_t mask = 0x1Fu;
    if (pl->cfg.evict_policy != SLHA_B200_EVICT_IMPORTANCE) mask &= ~(1u << PH_EVICT_PINNED);
    const uint32_t cm = pl->codec_mask;
    if (cm && !(cm & 0x80000000u) && !(cm & ((1u << SLHA_CODEC_TQ3) | (1u << SLHA_CODEC_MIX3))))
        mask &= ~((1u << PH_CORR_HOT) | (1u << PH_CORR_WARM));  // no tile with a correction plane can be in the pool
    SLHA_CUDA(cudaMemsetAsync(es, 0, sizeof(EnforceState), c->stream));
    SLHA_CUDA(cudaMemsetAsync(&pl->dev.cnt->max_pos, 0, 8, c->stream));  // max_pos and n_cand
    PoolDev d = pl->dev;
    void* args[] = {&d, &mask, &keys, &vals, &skeys, &svals, &es};
    const uint64_t want = (len + EB_THREADS - 1) / EB_THREADS;
    const unsigned grid = (unsigned)std::max<uint64_t>(1, std::min<uint64_t>(want, (uint64_t)sms[dev] * blocks_per_sm[dev]));
    const uint64_t stride = (uint64_t)grid * EB_THREADS;
    const bool few = len > EB_FEW * stride && len <= EB_KEYS * stride;
    SLHA_CUDA(cudaLaunchCooperativeKernel(few ? (const void*)enforce_kernel<true> : (const void*)enforce_kernel<false>, dim3(grid), dim3(EB_THREADS), args, 0, c->stream));
    count_launch();
    uint32_t overflow = 0;
    SLHA_CUDA(cudaMemcpyAsync(&overflow, &es->overflow, 4, cudaMemcpyDeviceToHost, c->stream));
    SLHA_TRY(pool_sync_counters(c, pl));
    if (overflow) return Status();
    if (pl->h_cnt.free_len > free_before) pl->hot_most = 0;  // evictions follow when every HOT tile is paged
    *within = pl->h_cnt.live <= pl->h_cnt.budget ? 1 : 0;
    *done = true;
    return Status();
}

// The step kernel (see there), where no tile can have a correction plane and a thread's slots fit its registers (1.2 million on 148 SMs).  Not where the
// list of HOT tiles may overflow, nor where the appended tiles alone ask for more evictions than the blocks' smallest keys are kept for (110 on 148 blocks):
// the kernel would find that out after its first scan, 20 to 30 us, and leave the rest to the other.  Sets *done when the budget question is settled.
static Status pool_enforce_budget_step(Ctx* c, Pool* pl, int32_t* within, bool* done) {
    *done = false;
    const uint32_t cm = pl->codec_mask;
    const bool planes = !cm || (cm & (0x80000000u | (1u << SLHA_CODEC_TQ3) | (1u << SLHA_CODEC_MIX3)));
    const uint64_t len = pl->h_cnt.len;
    if (planes || len == 0) return Status();
    static int ctas[64] = {0};
    const int dev = pl->device & 63;
    if (!ctas[dev]) {
        int coop = 0, n = 0, b = 0;
        SLHA_CUDA(cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, pl->device));
        SLHA_CUDA(cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, pl->device));
        SLHA_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, enforce_step_kernel, EB_THREADS, 0));
        ctas[dev] = coop && b > 0 ? n : -1;
    }
    if (ctas[dev] < 0) return Status();
    const uint64_t want = (len + EB_THREADS - 1) / EB_THREADS;
    const unsigned grid = (unsigned)std::min<uint64_t>(want, (uint64_t)ctas[dev]);
    if (len > (uint64_t)EB_KEYS * grid * EB_THREADS) return Status();
    if (pl->hot_most > (uint64_t)EB_CAP) return Status();
    const uint64_t about = pl->h_cnt.live + 96 * pl->unread;  // once they are paged
    if (about > pl->h_cnt.budget && ((about - pl->h_cnt.budget) / 80 + 1) * grid > 4ull * EB_CAP) return Status();
    SLHA_TRY(ctx_no_capture(c));  // (the host waits for the answer)
    SLHA_TRY(pool_step_memory(pl));
    volatile uint32_t* host;
    uint32_t* dev_host;
    bool* open;
    SLHA_TRY(ctx_answer(c, &host, &dev_host, &open));
    volatile StepAnswer* h = reinterpret_cast<volatile StepAnswer*>(host + 64);
    StepState* ss = static_cast<StepState*>(pl->d_step);
    uint64_t* hkeys = reinterpret_cast<uint64_t*>(static_cast<char*>(pl->d_step) + 256);
    uint64_t* skeys = hkeys + EB_CAP;
    uint32_t* hvals = reinterpret_cast<uint32_t*>(skeys + 2 * EB_CAP);
    uint32_t* svals = hvals + EB_CAP;
    if (!pl->step_clean) SLHA_CUDA(cudaMemsetAsync(ss, 0, sizeof(StepState), c->stream));
    pl->step_clean = false;
    PoolDev d = pl->dev;
    static thread_local uint32_t count = 0;
    uint32_t no = count = count % 0x7FFFFFFFu + 1u;
    h->no = 0u;
    StepAnswer* answer = reinterpret_cast<StepAnswer*>(dev_host + 64);
    void* args[] = {&d, &hkeys, &hvals, &skeys, &svals, &ss, &answer, &no};
    SLHA_CUDA(cudaLaunchCooperativeKernel((const void*)enforce_step_kernel, dim3(grid), dim3(EB_THREADS), args, 0, c->stream));
    count_launch();
    SLHA_TRY(wait_answer(c, [&] { return h->no == no; }));
    pl->h_cnt.live = h->live;
    pl->h_cnt.free_len = h->free_len;
    pl->unread = 0;
    pl->step_clean = true;
    if (h->hot != ~0ull) pl->hot_most = h->hot;
    if (h->flags) return Status();
    *within = pl->h_cnt.live <= pl->h_cnt.budget ? 1 : 0;
    *done = true;
    return Status();
}

Status pool_enforce_budget(Ctx* c, Pool* pl, int32_t* within) {
    if (!pl->log && !pl->require_durable && !debug_general_paths()) {
        bool done = false;
        SLHA_TRY(pool_enforce_budget_step(c, pl, within, &done));
        if (done) return Status();
        SLHA_TRY(pool_enforce_budget_fused(c, pl, within, &done));
        if (done) return Status();
    }
    SLHA_TRY(pool_sync_counters(c, pl));
    PoolCounters& h = pl->h_cnt;
    if (h.live <= h.budget) {
        *within = 1;
        return Status();
    }
    const uint64_t len = h.len;
    size_t tmp_sort = 0, tmp_scan = 0;
    cub::DeviceRadixSort::SortPairs(nullptr, tmp_sort, (uint64_t*)nullptr, (uint64_t*)nullptr,
                                    (uint32_t*)nullptr, (uint32_t*)nullptr, (int)len);
    cub::DeviceScan::ExclusiveSum(nullptr, tmp_scan, (uint32_t*)nullptr, (uint64_t*)nullptr, (int)len);
    const size_t tmp_bytes = std::max(tmp_sort, tmp_scan);
    Scratch sc{c};
    SLHA_TRY(sc.reserve(pad256(len * 8) * 3 + pad256(len * 4) * 3 + pad256(tmp_bytes) + 4096));
    uint64_t* keys = sc.take<uint64_t>(len);
    uint64_t* keys_s = sc.take<uint64_t>(len);
    uint64_t* excl = sc.take<uint64_t>(len);
    uint32_t* vals = sc.take<uint32_t>(len);
    uint32_t* vals_s = sc.take<uint32_t>(len);
    uint32_t* w = sc.take<uint32_t>(len);
    void* tmp = sc.take<unsigned char>(tmp_bytes);
    const uint32_t grid = grid_for(len);

    SLHA_CUDA(cudaMemsetAsync(&pl->dev.cnt->max_pos, 0, 4, c->stream));
    if (pl->cfg.recent_window) {
        max_pos_kernel<<<grid, 256, 0, c->stream>>>(pl->dev);
        count_launch();
    }
    const int phases[5] = {PH_CORR_HOT, PH_PAGE, PH_CORR_WARM, PH_EVICT, PH_EVICT_PINNED};
    for (int ph : phases) {
        if (ph == PH_EVICT_PINNED && pl->cfg.evict_policy != SLHA_B200_EVICT_IMPORTANCE) continue;
        // a pool that has only ever been appended to with codecs without a correction plane (every
        // codec but TQ3 and MIX3) has no candidate for the two correction phases: no scan for them
        const uint32_t cm = pl->codec_mask;
        const bool no_corr_planes = cm && !(cm & 0x80000000u) && !(cm & ((1u << SLHA_CODEC_TQ3) | (1u << SLHA_CODEC_MIX3)));
        if (no_corr_planes && (ph == PH_CORR_HOT || ph == PH_CORR_WARM)) continue;
        SLHA_CUDA(cudaMemsetAsync(&pl->dev.cnt->n_cand, 0, 4, c->stream));
        phase_build_kernel<<<grid, 256, 0, c->stream>>>(pl->dev, ph, keys, vals);
        count_launch();
        SLHA_CUDA(cudaGetLastError());
        // the host needs the candidate count for the sort (and learns whether the budget is met)
        SLHA_TRY(pool_sync_counters(c, pl));
        if (pl->h_cnt.live <= pl->h_cnt.budget) break;
        int nc = (int)pl->h_cnt.n_cand;
        if (nc == 0) continue;
        uint64_t* keys_in = keys;
        uint32_t* vals_in = vals;
        if ((uint32_t)nc >= PREFILTER_MIN) {
            // only the smallest keys can be reached before the deficit is covered (see phase_hist_kernel)
            const uint64_t min_freed = ph == PH_PAGE ? 32 : (ph >= PH_EVICT ? 80 : 14);
            const uint64_t reach = (pl->h_cnt.live - pl->h_cnt.budget) / min_freed + 1;
            uint32_t* d_hist = reinterpret_cast<uint32_t*>(excl);  // (free until the scan; 8 bytes x len >= 16 KB + 4 here)
            SLHA_CUDA(cudaMemsetAsync(d_hist, 0, (PREFILTER_BINS + 1) * 4, c->stream));
            phase_hist_kernel<<<grid_for((uint64_t)nc), 256, 0, c->stream>>>(pl->dev, keys, d_hist);
            std::vector<uint32_t> hh(PREFILTER_BINS);
            SLHA_CUDA(cudaMemcpyAsync(hh.data(), d_hist, PREFILTER_BINS * 4, cudaMemcpyDeviceToHost, c->stream));
            SLHA_CUDA(cudaStreamSynchronize(c->stream));
            uint64_t cum = 0;
            uint32_t last = PREFILTER_BINS - 1;
            for (uint32_t b = 0; b < PREFILTER_BINS; ++b) {
                cum += hh[b];
                if (cum >= reach) { last = b; break; }
            }
            if (cum < (uint64_t)nc) {  // the filter drops something: compact into the sorted-side buffers, sort back
                phase_filter_kernel<<<grid_for((uint64_t)nc), 256, 0, c->stream>>>(pl->dev, keys, vals, last, keys_s, vals_s, d_hist + PREFILTER_BINS);
                phase_set_ncand_kernel<<<1, 1, 0, c->stream>>>(pl->dev, d_hist + PREFILTER_BINS);
                count_launch(3);
                SLHA_CUDA(cudaGetLastError());
                nc = (int)cum;
                std::swap(keys, keys_s);
                std::swap(vals, vals_s);
                keys_in = keys;
                vals_in = vals;
            }
        }
        const uint32_t cgrid = grid_for((uint64_t)nc);
        size_t tb = tmp_bytes;
        SLHA_CUDA(cub::DeviceRadixSort::SortPairs(tmp, tb, keys_in, keys_s, vals_in, vals_s, nc, 0, 64, c->stream));
        phase_weights_kernel<<<cgrid, 256, 0, c->stream>>>(pl->dev, ph, keys_s, vals_s, w);
        tb = tmp_bytes;
        SLHA_CUDA(cub::DeviceScan::ExclusiveSum(tmp, tb, w, excl, nc, c->stream));
        uint64_t limit = ~0ull;
        if (ph >= PH_EVICT && (pl->log || pl->require_durable)) {
            // persist first (ccos.rs:411-432): the records of the slots this phase will evict, in order
            unsigned long long* d_cnt;
            uint64_t* d_seq;
            uint32_t* d_slot;
            uint4* d_tiles;
            SLHA_TRY(ctx_device_scratch(c, 256, (void**)&d_cnt));
            SLHA_TRY(ctx_device_scratch(c, (size_t)nc * 8, (void**)&d_seq));
            SLHA_TRY(ctx_device_scratch(c, (size_t)nc * 4, (void**)&d_slot));
            SLHA_TRY(ctx_device_scratch(c, (size_t)nc * TILE_BYTES, (void**)&d_tiles));
            SLHA_CUDA(cudaMemsetAsync(d_cnt, 0, 8, c->stream));
            phase_journal_kernel<<<cgrid, 256, 0, c->stream>>>(pl->dev, keys_s, vals_s, excl, d_cnt, d_seq, d_slot, d_tiles);
            count_launch();
            unsigned long long m = 0;
            SLHA_CUDA(cudaMemcpyAsync(&m, d_cnt, 8, cudaMemcpyDeviceToHost, c->stream));
            SLHA_CUDA(cudaStreamSynchronize(c->stream));
            std::vector<uint64_t> hseq(m);
            std::vector<uint32_t> hslot(m);
            std::vector<unsigned char> htiles((size_t)m * TILE_BYTES);
            if (m) {
                SLHA_CUDA(cudaMemcpyAsync(hseq.data(), d_seq, m * 8, cudaMemcpyDeviceToHost, c->stream));
                SLHA_CUDA(cudaMemcpyAsync(hslot.data(), d_slot, m * 4, cudaMemcpyDeviceToHost, c->stream));
                SLHA_CUDA(cudaMemcpyAsync(htiles.data(), d_tiles, (size_t)m * TILE_BYTES, cudaMemcpyDeviceToHost, c->stream));
                SLHA_CUDA(cudaStreamSynchronize(c->stream));
            }
            // all records of the phase in one write (the same bytes in the same order as one append per eviction)
            uint64_t written = 0;
            const bool ok = m == 0 || (pl->log && eventlog_append_batch(pl->log, m, hseq.data(), hslot.data(), htiles.data(), pl->require_durable, &written).ok());
            if (!ok) {
                if (pl->log) ++pl->log_errors;
                if (pl->require_durable) {
                    // record `written` could not be persisted: its slot stays live; the reference goes on to try (and be
                    // refused) every remaining live slot
                    limit = written;
                    pl->blocked_evictions += (uint64_t)nc - written;
                    if (pl->log) pl->log_errors += (uint64_t)nc - written - 1;
                }
            }
        }
        phase_apply_kernel<<<cgrid, 256, 0, c->stream>>>(pl->dev, ph, keys_s, vals_s, w, excl, limit);
        phase_commit_kernel<<<1, 1, 0, c->stream>>>(pl->dev);
        count_launch(3);
        SLHA_CUDA(cudaGetLastError());
    }
    SLHA_TRY(pool_sync_counters(c, pl));
    *within = pl->h_cnt.live <= pl->h_cnt.budget ? 1 : 0;
    return Status();
}

Status pool_observe(Ctx* c, Pool* pl, const uint32_t* d_slots, const float* d_scores, uint64_t n, float temperature) {
    if (n == 0 || !std::isfinite(temperature) || temperature <= 0.0f) return Status();
    const int nparts = OBSERVE_PARTS;
    if (!pl->d_observe) {
        SLHA_CUDA(cudaMalloc(&pl->d_observe, 2 * sizeof(ObserveTmp) + nparts * 4));
        pl->observe_clean = false;
    }
    ObserveTmp* tmp = reinterpret_cast<ObserveTmp*>(pl->d_observe);
    ObserveTmp* all = tmp + 1;  // observe_all_kernel's, zero between its calls
    float* partial = reinterpret_cast<float*>(tmp + 2);
    // (not into a graph: whether the state needs its clear is known when a call is made, not when a graph is launched)
    if (!d_slots && n <= (uint64_t)OBSERVE_PARTS * 256 * OBSERVE_KEEP && !ctx_capturing(c)) {
        static int fits[64] = {0};
        const int dev = pl->device & 63;
        if (!fits[dev]) {
            int coop = 0, b = 0;
            SLHA_CUDA(cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, pl->device));
            SLHA_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, observe_all_kernel, 512, 0));
            fits[dev] = coop && b * sm_count(c->device) >= OBSERVE_PARTS / 2 ? 1 : -1;
        }
        if (fits[dev] > 0) {
            if (!pl->observe_clean) SLHA_CUDA(cudaMemsetAsync(all, 0, sizeof(ObserveTmp), c->stream));
            pl->observe_clean = false;
            void* args[] = {&pl->dev, &d_scores, &n, &temperature, &all, &partial};
            SLHA_CUDA(cudaLaunchCooperativeKernel((const void*)observe_all_kernel, dim3(OBSERVE_PARTS / 2), dim3(512), args, 0, c->stream));
            count_launch();
            pl->observe_clean = true;
            return Status();
        }
    }
    SLHA_CUDA(cudaMemsetAsync(tmp, 0, sizeof(ObserveTmp), c->stream));
    const uint32_t grid = std::min<uint32_t>(grid_for(n), (uint32_t)sm_count(c->device) * 4);
    observe_pass1<<<grid, 256, 0, c->stream>>>(pl->dev, d_slots, d_scores, n, tmp);
    SLHA_CUDA(launch_behind(observe_pass2, dim3(nparts), dim3(256), 0, c->stream, pl->dev, d_slots, d_scores, n, temperature, tmp, partial));
    SLHA_CUDA(launch_behind(observe_pass3, dim3(grid), dim3(256), 0, c->stream, pl->dev, d_slots, d_scores, n, temperature, tmp, partial, nparts));
    count_launch(3);
    SLHA_CUDA(cudaGetLastError());
    return Status();
}

Status pool_stats(Ctx* c, Pool* pl, uint64_t out[8]) {
    SLHA_TRY(ctx_no_capture(c));  // (the host waits for the answer)
    volatile uint32_t* host;
    uint32_t *dev, *sums;
    bool* open;
    SLHA_TRY(ctx_answer(c, &host, &dev, &open));
    volatile uint64_t* h = reinterpret_cast<volatile uint64_t*>(host + 32);  // (behind the answers to checks)
    unsigned long long* answer = reinterpret_cast<unsigned long long*>(dev + 32);
    // (a pool that has only ever been appended to with codecs without a correction plane holds no tile that dropped one)
    const uint32_t cm = pl->codec_mask;
    bool planes = !cm || (cm & (0x80000000u | (1u << SLHA_CODEC_TQ3) | (1u << SLHA_CODEC_MIX3)));
    const uint32_t grid = (uint32_t)std::min<uint64_t>((pl->h_cnt.len + (planes ? 512u : 8192u)) / (planes ? 512u : 8192u), (uint64_t)sm_count(c->device));
    SLHA_TRY(ctx_device_scratch(c, (size_t)grid * 32, (void**)&sums));
    static thread_local unsigned long long count = 0;
    unsigned long long no = ++count;
    h[8] = 0;
    void* args[] = {&pl->dev, &sums, &answer, &no, &planes};
    SLHA_CUDA(cudaLaunchCooperativeKernel((const void*)stats_kernel, dim3(grid), dim3(512), args, 0, c->stream));
    count_launch();
    SLHA_TRY(wait_answer(c, [&] { return h[8] == no; }));
    for (int i = 0; i < 8; ++i) out[i] = h[i];
    return Status();
}

Status pool_compact_live(Ctx* c, Pool* pl, const float* d_scores, uint32_t* d_slots_out, float* d_scores_out,
                         unsigned long long* d_n_out) {
    compact_live_kernel<<<1, 1024, 0, c->stream>>>(pl->dev, d_scores, d_slots_out, d_scores_out, d_n_out);
    count_launch();
    SLHA_CUDA(cudaGetLastError());
    return Status();
}

}  // namespace slha

namespace slha {
// ElasticKvCache::rehydrate (ccos.rs:451-466): the most recent record with that eviction seq comes back as a
// fresh admission (new seq, importance 0), WARM when its tile carries the WARM flag, else HOT.
Status pool_rehydrate(Ctx* c, Pool* pl, uint64_t seq, int64_t* slot_out) {
    *slot_out = -1;
    if (!pl->log) return Status();
    bool found = false;
    uint32_t old_slot = 0;
    unsigned char tile[TILE_BYTES];
    SLHA_TRY(eventlog_fetch_by_seq(pl->log, seq, &found, &old_slot, tile));
    if (!found) return Status();
    unsigned char* d_tile;
    uint32_t* d_slot;
    SLHA_TRY(ctx_device_scratch(c, TILE_BYTES, (void**)&d_tile));
    SLHA_TRY(ctx_device_scratch(c, 256, (void**)&d_slot));
    SLHA_CUDA(cudaMemcpyAsync(d_tile, tile, TILE_BYTES, cudaMemcpyHostToDevice, c->stream));
    SLHA_TRY(pool_reserve(c, pl, d_tile, 1, d_slot));
    SLHA_TRY(pool_scatter(c, pl, d_tile, d_slot, 1));
    uint32_t slot = 0;
    SLHA_CUDA(cudaMemcpyAsync(&slot, d_slot, 4, cudaMemcpyDeviceToHost, c->stream));
    SLHA_CUDA(cudaStreamSynchronize(c->stream));
    pl->codec_mask |= 0x80000000u;
    *slot_out = (int64_t)slot;
    return Status();
}
}  // namespace slha
