// Decode tail on the selected tiles: softmax over the k winners of every query row, then the
// weighted sum of their value rows -- the two steps that follow scoring in the reference's decode
// proxy (scirust/examples/benchmark_decode.rs:82-95: metrics::softmax_into, scirust/src/metrics.rs:338-420,
// then aggregate_v, benchmark_decode.rs:28-38), applied to the top-k instead of the whole context.
// The k (index, score) pairs stay in HBM; what crosses PCIe afterwards is one d_v-vector per query
// row instead of k pairs.
//
// One query row is shared by the SPLIT CTAs of a cluster (eight or fewer, see launch_attend_topk), each taking an equal run of the winners the row has.  Every CTA
// finds the row's maximum itself (k scores, a few KB from the L2) and weighs its own run; the normalisers and the
// partial sums of the value rows meet in distributed shared memory, added in a fixed order, so a call is one launch and
// writes nothing but its results.  Bound: the gather of k value rows per query row (HBM); a thread keeps twelve 16-byte
// loads in flight.  32 rows x 2048 winners of 128 bf16 values (17 MB): 8.7 us a call (2.0 TB/s); with
// one-element loads, four in flight, partial sums through memory and a second launch to add them it was 31.9 us.
#include <cooperative_groups.h>
#include <cuda_bf16.h>

#include <cfloat>

#include "runtime.cuh"

namespace slha {
namespace {

constexpr int ATT_THREADS = 256;
constexpr int ATT_FLIGHT = 12; // value loads a thread issues before it uses the first

// VEC columns of a value row (4 or 16 bytes; one element of a float32 or bfloat16 row), loaded when `p` holds, else zero.
// (Predicated loads in volatile statements, so that a thread's loads stay together in front of their uses.  Coherent ones: this grid may be
// resident while the values are written, see dep_wait.)
template <typename T, int VEC>
struct Values {
    uint32_t x[VEC == 1 ? 1 : 4];
    __device__ __forceinline__ void load(const T* src, bool p) {
        if constexpr (VEC > 1) {
            asm volatile("{\n.reg .pred p;\nsetp.ne.u32 p, %5, 0;\nmov.u32 %0, 0;\nmov.u32 %1, 0;\nmov.u32 %2, 0;\nmov.u32 %3, 0;\n"
                         "@p ld.global.v4.u32 {%0,%1,%2,%3}, [%4];\n}\n"
                         : "=&r"(x[0]), "=&r"(x[1]), "=&r"(x[2]), "=&r"(x[3]) : "l"(src), "r"((uint32_t)p));
        } else if constexpr (sizeof(T) == 4) {
            asm volatile("{\n.reg .pred p;\nsetp.ne.u32 p, %2, 0;\nmov.u32 %0, 0;\n@p ld.global.u32 %0, [%1];\n}\n" : "=&r"(x[0]) : "l"(src), "r"((uint32_t)p));
        } else {
            uint16_t h;
            asm volatile("{\n.reg .pred p;\nsetp.ne.u32 p, %2, 0;\nmov.u16 %0, 0;\n@p ld.global.u16 %0, [%1];\n}\n" : "=&h"(h) : "l"(src), "r"((uint32_t)p));
            x[0] = h;
        }
    }
    __device__ __forceinline__ void hold() {  // nothing that uses the values is moved above this point
        if constexpr (VEC > 1) asm volatile("" : "+r"(x[0]), "+r"(x[1]), "+r"(x[2]), "+r"(x[3]));
        else asm volatile("" : "+r"(x[0]));
    }
    __device__ __forceinline__ float get(int i) const {
        if constexpr (sizeof(T) == 4) return __uint_as_float(x[i]);
        else return __uint_as_float((i & 1) ? (x[i >> 1] & 0xFFFF0000u) : (x[i >> 1] << 16));
    }
};

__device__ __forceinline__ float block_reduce(float v, float* sh, bool is_max) {
    for (int o = 16; o; o >>= 1) {
        const float y = __shfl_xor_sync(0xFFFFFFFFu, v, o);
        v = is_max ? fmaxf(v, y) : v + y;
    }
    __syncthreads();
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = v;
    __syncthreads();
    float r = sh[0];
    for (int w = 1; w < (int)(blockDim.x >> 5); ++w) r = is_max ? fmaxf(r, sh[w]) : r + sh[w];
    return r;
}

// weights_out (optional): [nq][k] softmax weights (0 for absent entries).  VEC 1 takes any alignment, stride and d_v.
template <typename T, int VEC, int SPLIT>
__global__ void __cluster_dims__(SPLIT, 1, 1) __launch_bounds__(ATT_THREADS)
    attend_kernel(const uint32_t* top_index, const float* top_score, const uint32_t* top_count, uint32_t k, float scale, const T* values,
                  size_t d_v, size_t row_stride, const uint64_t* row_base, float* out, float* weights_out) {
    dep_wait();  // (no dep_launch: CTAs of the next call that came to wait here were spread unevenly, 256 rows x 2048 winners 37 us -> 49, now 35)
    namespace cg = cooperative_groups;
    cg::cluster_group cluster = cg::this_cluster();
    extern __shared__ float sm[];  // weights | indices of the CTA's run
    __shared__ float red[8], own_sum, slot[ATT_THREADS * VEC], part_out[ATT_THREADS * VEC];
    const uint32_t Q = blockIdx.y, part = cluster.block_rank(), tid = threadIdx.x;
    const uint32_t n = top_count ? min(top_count[Q], k) : k;
    const float* sc = top_score + (size_t)Q * k;
    const uint32_t* ix = top_index + (size_t)Q * k;
    // softmax_into: logits = score * scale, maximum subtracted, normalised (absent entries weigh nothing)
    float mx = -INFINITY;
    for (uint32_t i = tid; i < n; i += ATT_THREADS)
        if (ix[i] != 0xFFFFFFFFu) mx = fmaxf(mx, sc[i] * scale);
    mx = block_reduce(mx, red, true);
    const uint32_t run = (n + SPLIT - 1) / SPLIT, lo = min(n, part * run), len = min(n, lo + run) - lo;  // this CTA's winners
    float* w = sm;
    uint32_t* wi = reinterpret_cast<uint32_t*>(sm + (k + SPLIT - 1) / SPLIT);
    float sum = 0.0f;
    for (uint32_t j = tid; j < len; j += ATT_THREADS) {
        const uint32_t i = lo + j, id = ix[i];
        const bool have = id != 0xFFFFFFFFu;
        const float e = have && mx > -INFINITY ? expf(sc[i] * scale - mx) : 0.0f;
        w[j] = e;
        wi[j] = have ? id : 0xFFFFFFFFu;
        sum += e;
    }
    sum = block_reduce(sum, red, false);
    if (tid == 0) own_sum = sum;
    cluster.sync();  // (also: this CTA's weights and indices are visible to all its threads)
    float total = 0.0f;
    for (int r = 0; r < SPLIT; ++r) total += *cluster.map_shared_rank(&own_sum, r);
    const float inv = (total > 0.0f && isfinite(total)) ? 1.0f / total : 0.0f;
    if (weights_out)
        for (uint32_t j = tid; j < len; j += ATT_THREADS) weights_out[(size_t)Q * k + lo + j] = w[j] * inv;
    const uint64_t base = row_base ? row_base[Q] : 0ull;
    const uint32_t all = (uint32_t)(d_v / VEC);  // column vectors of a value row
    for (uint32_t v0 = 0; v0 < all; v0 += ATT_THREADS) {
        // threads cover the row's column vectors, row groups take alternate winners
        const uint32_t cols = min(all - v0, (uint32_t)ATT_THREADS), groups = ATT_THREADS / cols, grp = tid / cols, col = tid % cols;
        float acc[VEC];
#pragma unroll
        for (int e = 0; e < VEC; ++e) acc[e] = 0.0f;
        if (grp < groups) {
            const T* src = values + (size_t)(v0 + col) * VEC;
            for (uint32_t j0 = grp; j0 < len; j0 += ATT_FLIGHT * groups) {
                Values<T, VEC> x[ATT_FLIGHT];
                float wt[ATT_FLIGHT];
#pragma unroll
                for (int f = 0; f < ATT_FLIGHT; ++f) {
                    const uint32_t j = j0 + f * groups;
                    const uint32_t id = j < len ? wi[j] : 0xFFFFFFFFu;
                    const bool have = id != 0xFFFFFFFFu;
                    x[f].load(src + (base + id) * row_stride, have);
                    wt[f] = have ? w[j] : 0.0f;
                }
#pragma unroll
                for (int f = 0; f < ATT_FLIGHT; ++f) x[f].hold();
#pragma unroll
                for (int f = 0; f < ATT_FLIGHT; ++f)
#pragma unroll
                    for (int e = 0; e < VEC; ++e) acc[e] = fmaf(wt[f], x[f].get(e), acc[e]);
            }
        }
        // the row groups' sums, then the CTAs' sums, in a fixed order
#pragma unroll
        for (int e = 0; e < VEC; ++e) slot[e * ATT_THREADS + tid] = acc[e];
        __syncthreads();
        for (uint32_t c = tid; c < cols * VEC; c += ATT_THREADS) {
            float t = 0.0f;
            for (uint32_t g = 0; g < groups; ++g) t += slot[(c % VEC) * ATT_THREADS + g * cols + c / VEC];
            part_out[c] = t;
        }
        cluster.sync();
        const uint32_t share = (cols * VEC + SPLIT - 1) / SPLIT, c0 = part * share;
        for (uint32_t c = c0 + tid; c < min(c0 + share, cols * VEC); c += ATT_THREADS) {
            float t = 0.0f;
#pragma unroll
            for (int r = 0; r < SPLIT; ++r) t += cluster.map_shared_rank(part_out, r)[c];
            out[(size_t)Q * d_v + (size_t)v0 * VEC + c] = t * inv;
        }
        cluster.sync();  // the peers have read this CTA's sums
    }
    if (weights_out && n < k)
        for (uint32_t i = n + part * ATT_THREADS + tid; i < k; i += SPLIT * ATT_THREADS) weights_out[(size_t)Q * k + i] = 0.0f;
}

template <typename T, int VEC, int SPLIT>
Status launch_attend_t(Ctx* c, const uint32_t* d_index, const float* d_score, const uint32_t* d_count, size_t nq, uint32_t k, float scale,
                       const void* d_values, size_t d_v, size_t row_stride, const uint64_t* d_row_base, float* d_out, float* d_weights) {
    const size_t smem = (size_t)((k + SPLIT - 1) / SPLIT) * 8;
    if (smem > 16 * 1024) SLHA_CUDA(cudaFuncSetAttribute(attend_kernel<T, VEC, SPLIT>, cudaFuncAttributeMaxDynamicSharedMemorySize, 8192 * 8));
    SLHA_CUDA(launch_behind(attend_kernel<T, VEC, SPLIT>, dim3(SPLIT, (uint32_t)nq), dim3(ATT_THREADS), smem, c->stream, d_index, d_score, d_count, k, scale,
                            (const T*)d_values, d_v, row_stride, d_row_base, d_out, d_weights));
    count_launch();
    return Status();
}

}  // namespace

Status launch_attend_topk(Ctx* c, const uint32_t* d_index, const float* d_score, const uint32_t* d_count, size_t nq, uint32_t k,
                          float scale, const void* d_values, int value_dtype, size_t d_v, size_t row_stride,
                          const uint64_t* d_row_base, float* d_out, float* d_weights) {
    if (nq == 0 || d_v == 0) return Status();
    if (k == 0 || k > 8192) return Status(SLHA_ERR_DIMENSION, "attend_topk: k must be in 1..8192");
    if (!isfinite(scale)) return Status(SLHA_ERR_NONFINITE, "attend_topk: scale is not finite");
    // 16-byte loads where every value row starts and ends on a 16-byte boundary, else one element at a time
    const size_t esz = value_dtype == SLHA_B200_BF16 ? 2 : 4;
    const bool vec = reinterpret_cast<uintptr_t>(d_values) % 16 == 0 && d_v * esz % 16 == 0 && row_stride * esz % 16 == 0;
    // CTAs per row: the most that keep the grid within two CTAs an SM.  With eight for every row, calls of many rows ran in waves of CTAs
    // with little to gather each: 128 bf16 values, 100 rows of 64 winners 22.4 us (now 8.6), of 2048 31.1 (16.7), 256 rows of 64
    // 43.4 (8.8), of 2048 63.9 (35.1).
    // Three an SM where a row's values are long: from 320 KB rather two CTAs a row than one (150 rows of 2048 winners of 256 bf16 values
    // 57.8 -> 35.0 us), from 768 KB of float32 also four and eight (75 rows of 2048 x 256 29.0 -> 24.9; bf16 there 22.8 -> 24.9).
    const size_t long_row = (size_t)k * d_v * esz, sms = (size_t)sm_count(c->device);
    auto per_sm = [&](int ctas) { return (ctas == 2 ? long_row >= (320u << 10) : esz == 4 && long_row >= (768u << 10)) ? 3u : 2u; };
    int split = 8;
    while (split > 1 && nq * (size_t)split > per_sm(split) * sms) split >>= 1;
#define SLHA_ATTEND_S(T, V, S) launch_attend_t<T, V, S>(c, d_index, d_score, d_count, nq, k, scale, d_values, d_v, row_stride, d_row_base, d_out, d_weights)
#define SLHA_ATTEND(T, V) (split == 8 ? SLHA_ATTEND_S(T, V, 8) : split == 4 ? SLHA_ATTEND_S(T, V, 4) : split == 2 ? SLHA_ATTEND_S(T, V, 2) : SLHA_ATTEND_S(T, V, 1))
    if (value_dtype == SLHA_B200_BF16) return vec ? SLHA_ATTEND(__nv_bfloat16, 8) : SLHA_ATTEND(__nv_bfloat16, 1);
    return vec ? SLHA_ATTEND(float, 4) : SLHA_ATTEND(float, 1);
#undef SLHA_ATTEND_S
#undef SLHA_ATTEND
}

}  // namespace slha
