// Host runtime of libslha_b200: execution context, scratch arena, staging,
// model construction (.slhw parsing, sign-LSH matrix generation) and registry.
#include "runtime.cuh"

#include <sys/stat.h>

#include <atomic>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <memory>
#include <mutex>
#include <shared_mutex>
#include <unordered_map>

namespace slha {

Status cuda_status(cudaError_t e, const char* what) {
    cudaGetLastError();  // (reported here, not once more by the next call's launch check)
    return Status(SLHA_ERR_DEVICE, std::string("CUDA error: ") + cudaGetErrorString(e) + " in " + what);
}

static std::atomic<uint64_t> g_launches{0};
static thread_local uint64_t g_thread_launches = 0;
void count_launch(int n) {
    g_launches.fetch_add((uint64_t)n, std::memory_order_relaxed);
    g_thread_launches += (uint64_t)n;
}
int sm_count(int device) {
    static std::atomic<int> known[16];
    std::atomic<int>& n = known[device & 15];
    int v = n.load(std::memory_order_relaxed);
    if (v == 0) {
        if (cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, device) != cudaSuccess || v < 1) {
            cudaGetLastError();
            return 148;
        }
        n.store(v, std::memory_order_relaxed);
    }
    return v;
}
uint64_t launch_count() { return g_launches.load(std::memory_order_relaxed); }

// ---- per-thread context ------------------------------------------------------
namespace {
struct Block {
    char* p = nullptr;
    size_t cap = 0, off = 0;
};
// The small tables that calls upload (ctx_upload): a copy may read its slot until the slot's event, so a slot is written again
// only after that.  One wait per stream, for its newest event in half the ring, covers the half; a wait for an event that is long
// over still costs 1.4 us.  Short tables lie
// in ordinary memory, whose copies the driver sends along with its commands (8 KB: 2.0 us against 3.6 us for the copy
// engine), longer ones in page-locked memory (60 KB: 5.1 us against 2.3 us of the host's time).  Given back when the thread ends.
constexpr int UPLOAD_SLOTS = 16, UPLOAD_HALF = UPLOAD_SLOTS / 2;
constexpr size_t UPLOAD_SHORT = (size_t)16 << 10;
constexpr size_t UPLOAD_MOST = (size_t)256 << 10;  // larger tables are copied from where they lie, and waited for
struct UploadSlot {
    std::vector<unsigned char> table;
    void* p = nullptr;
    size_t cap = 0;
    cudaEvent_t done = nullptr;  // recorded where the call that used the slot ends
    unsigned long long stream = 0;
    bool pending = false;
    ~UploadSlot() {
        if (pending) cudaEventSynchronize(done);
        if (done) cudaEventDestroy(done);
        if (p) cudaFreeHost(p);
    }
};
// Working memory (the scratch arena, the plans' buffers) across streams: a call on a caller-supplied stream may return while its
// kernels still use it; the event marks the end of that work, and a later call that uses the same memory on ANOTHER stream (by its
// id: the handle of a destroyed stream may come again) waits for it first.  On the same stream, stream order suffices.  The two are
// told apart so that a call without a plan (a merge on a second stream) runs beside the scoring of the next step.
struct LastUse {
    cudaEvent_t done = nullptr;
    unsigned long long stream = 0;
    bool queued = false;
};
// (at the thread's end, when any device may be current)
void drain(int device) {
    if (cudaSetDevice(device) == cudaSuccess) cudaDeviceSynchronize();
}
struct Answer {
    int device = 0;
    uint32_t* host = nullptr;
    uint32_t* dev = nullptr;
    bool open = false;  // a kernel may still write there: nobody has seen its answer (a call that ended by an exception)
    ~Answer() {
        if (open) drain(device);
        if (host) cudaFreeHost(host);
    }
};
// Where kernels write a call's short host outputs.  Empty between calls: what a failed call has left is given back at its end (see ~CallScope).
constexpr size_t OUT_PAGE = 4096, OUT_BYTES = 1024;
struct OutPage {
    int device = 0;
    unsigned char* host = nullptr;
    unsigned char* dev = nullptr;
    size_t used = 0;
    uint64_t launched = 0;  // the thread's launches when the call under way took its first part
    ~OutPage() {
        if (used) drain(device);
        if (host) cudaFreeHost(host);
    }
};
struct ThreadState {
    int device = 0;
    bool device_chosen = false;
    cudaStream_t user_stream = nullptr;
    bool has_user_stream = false;
    Ctx ctx[16];
    bool ctx_init[16] = {false};
    std::vector<Block> blocks[16];
    std::vector<std::pair<void*, size_t>> hblocks[16];
    UploadSlot upload[16][UPLOAD_SLOTS];
    uint32_t upload_next[16] = {0};
    UploadSlot* upload_used[16] = {nullptr};  // by the call under way
    LastUse arena[16], plans[16];
    Answer answer[16];
    OutPage outs[16];
    bool plans_used[16] = {false};            // by the call under way
};
thread_local ThreadState tls;
}  // namespace

void tls_set_device(int dev) {
    tls.device = dev;
    tls.device_chosen = true;
}
void tls_set_stream(void* s) {
    tls.user_stream = (cudaStream_t)s;
    tls.has_user_stream = s != nullptr;
}

Status get_ctx(Ctx** out) {
    int n = 0;
    cudaError_t e = cudaGetDeviceCount(&n);
    if (e != cudaSuccess || n == 0) {
        cudaGetLastError();
        return Status(SLHA_ERR_DEVICE, "no CUDA device is available (this library has no CPU fallback)");
    }
    int dev = tls.device;
    if (dev < 0 || dev >= n || dev >= 16) return Status(SLHA_ERR_DEVICE, "invalid device index");
    SLHA_CUDA(cudaSetDevice(dev));
    Ctx& c = tls.ctx[dev];
    if (!tls.ctx_init[dev]) {
        c.device = dev;
        SLHA_CUDA(cudaStreamCreateWithFlags(&c.lib_stream, cudaStreamNonBlocking));
        tls.ctx_init[dev] = true;
    }
    c.stream = tls.has_user_stream ? tls.user_stream : c.lib_stream;
    c.own_stream = !tls.has_user_stream;
    *out = &c;
    return Status();
}
bool sync_by_default(const Ctx* c) { return c->own_stream; }

Status ctx_device_scratch(Ctx* c, size_t bytes, void** out) {
    bytes = pad256(std::max<size_t>(bytes, 256));
    auto& blocks = tls.blocks[c->device];
    for (Block& b : blocks) {
        if (b.cap - b.off >= bytes) {
            *out = b.p + b.off;
            b.off += bytes;
            return Status();
        }
    }
    Block nb;
    nb.cap = std::max<size_t>(bytes, blocks.empty() ? (size_t)8 << 20 : blocks.back().cap * 2);
    SLHA_CUDA(cudaMalloc((void**)&nb.p, nb.cap));
    nb.off = bytes;
    *out = nb.p;
    blocks.push_back(nb);
    return Status();
}
Status ctx_host_scratch(Ctx* c, size_t bytes, void** out) {
    void* p = nullptr;
    SLHA_CUDA(cudaMallocHost(&p, std::max<size_t>(bytes, 256)));
    tls.hblocks[c->device].push_back({p, bytes});
    *out = p;
    return Status();
}

namespace {
// (an error means that another stream's capture forbids to ask)
bool capturing(cudaStream_t s) {
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(s, &cap) == cudaSuccess) return cap != cudaStreamCaptureStatusNone;
    cudaGetLastError();
    return true;
}
unsigned long long stream_id(cudaStream_t s) {
    unsigned long long id = 0;
    if (cudaStreamGetId(s, &id) != cudaSuccess) cudaGetLastError();
    return id;
}
// (a stream under capture runs nothing now, a graph may not wait for work outside it, and asking for the stream's id would end the capture)
void wait_for(const LastUse& u, cudaStream_t s) {
    if (u.queued && !capturing(s) && stream_id(s) != u.stream) cudaStreamWaitEvent(s, u.done, 0);
}
bool mark(LastUse& u, cudaStream_t s, unsigned long long id) {
    if (!u.done && cudaEventCreateWithFlags(&u.done, cudaEventDisableTiming) != cudaSuccess) return false;
    if (cudaEventRecord(u.done, s) != cudaSuccess) return false;
    u.stream = id;
    u.queued = true;
    return true;
}
}  // namespace

bool ctx_capturing(Ctx* c) { return capturing(c->stream); }
Status ctx_no_capture(Ctx* c) {
    if (!capturing(c->stream)) return Status();
    // a graph would keep the address of host memory that this call's successors write again: refused, and the capture ends
    // as invalid, like everywhere the library has to wait for a stream
    SLHA_CUDA(cudaStreamSynchronize(c->stream));
    return Status(SLHA_ERR_DEVICE, "this call cannot be captured into a graph");
}
Status ctx_upload(Ctx* c, const void* src, size_t bytes, void** dev) {
    SLHA_TRY(ctx_no_capture(c));
    SLHA_TRY(ctx_device_scratch(c, bytes, dev));
    return ctx_copy_table(c, *dev, src, bytes);
}
Status ctx_copy_table(Ctx* c, void* dev, const void* src, size_t bytes) {
    if (bytes > UPLOAD_MOST) {
        SLHA_CUDA(cudaMemcpyAsync(dev, src, bytes, cudaMemcpyHostToDevice, c->stream));
        SLHA_CUDA(cudaStreamSynchronize(c->stream));
        return Status();
    }
    if (UploadSlot* before = tls.upload_used[c->device]) {  // a second table of the same call
        SLHA_CUDA(cudaEventRecord(before->done, c->stream));
        before->stream = stream_id(c->stream);
        before->pending = true;
    }
    const uint32_t at = tls.upload_next[c->device]++ % UPLOAD_SLOTS;
    UploadSlot* const ring = tls.upload[c->device];
    if (at % UPLOAD_HALF == 0) {
        for (int i = UPLOAD_HALF - 1; i >= 0; --i) {
            if (!ring[at + i].pending) continue;
            SLHA_CUDA(cudaEventSynchronize(ring[at + i].done));
            for (int j = i; j >= 0; --j)
                if (ring[at + j].stream == ring[at + i].stream) ring[at + j].pending = false;
        }
    }
    UploadSlot& s = ring[at];
    const bool brief = bytes <= UPLOAD_SHORT;
    if (!brief && s.cap < bytes) {
        if (s.p) SLHA_CUDA(cudaFreeHost(s.p));
        s.p = nullptr;
        s.cap = 0;
        size_t want = (size_t)64 << 10;
        while (want < bytes) want <<= 1;
        SLHA_CUDA(cudaMallocHost(&s.p, want));
        s.cap = want;
    }
    if (!s.done) SLHA_CUDA(cudaEventCreateWithFlags(&s.done, cudaEventDisableTiming));
    if (brief) s.table.assign(static_cast<const unsigned char*>(src), static_cast<const unsigned char*>(src) + bytes);
    else std::memcpy(s.p, src, bytes);
    SLHA_CUDA(cudaMemcpyAsync(dev, brief ? s.table.data() : s.p, bytes, cudaMemcpyHostToDevice, c->stream));
    tls.upload_used[c->device] = &s;  // (its event is recorded at the call's end)
    return Status();
}
Status ctx_answer(Ctx* c, volatile uint32_t** host, uint32_t** dev, bool** open) {
    Answer& a = tls.answer[c->device];
    if (!a.host) {
        a.device = c->device;
        SLHA_CUDA(cudaHostAlloc((void**)&a.host, 512, cudaHostAllocMapped | cudaHostAllocPortable));
        std::memset(a.host, 0, 512);
    }
    if (!a.dev) SLHA_CUDA(cudaHostGetDevicePointer((void**)&a.dev, a.host, 0));
    *host = a.host;
    *dev = a.dev;
    *open = &a.open;
    return Status();
}
void ctx_uses_plans(Ctx* c) {
    wait_for(tls.plans[c->device], c->stream);
    tls.plans_used[c->device] = true;
}

CallScope::CallScope() {
    st = get_ctx(&c);
    if (!st.ok()) return;
    auto& blocks = tls.blocks[c->device];
    tls.upload_used[c->device] = nullptr;
    tls.plans_used[c->device] = false;
    wait_for(tls.arena[c->device], c->stream);
    // the previous call has returned, so its staging memory may be reused; when
    // the arena had to chain blocks, replace them by one block of the total size
    if (blocks.size() > 1) {
        size_t total = 0;
        cudaStreamSynchronize(c->stream);
        for (Block& b : blocks) { total += b.cap; cudaFree(b.p); }
        blocks.clear();
        Block nb;
        nb.cap = total;
        if (cudaMalloc((void**)&nb.p, nb.cap) == cudaSuccess) blocks.push_back(nb);
        else cudaGetLastError();
    }
    for (Block& b : blocks) b.off = 0;
    for (auto& hb : tls.hblocks[c->device]) cudaFreeHost(hb.first);
    tls.hblocks[c->device].clear();
}

CallScope::~CallScope() {
    if (!c) return;
    // A call that failed behind stage_out: nothing writes its part of the page where nothing was launched, and nothing once the stream is drained.
    OutPage& page = tls.outs[c->device];
    if (page.used) {
        if (page.launched == g_thread_launches || cudaStreamSynchronize(c->stream) == cudaSuccess) page.used = 0;
        else cudaGetLastError();
    }
    UploadSlot* up = tls.upload_used[c->device];
    if (c->own_stream && !up) return;  // library stream: the call drained it before returning
    bool arena = false;
    for (const Block& b : tls.blocks[c->device]) arena |= b.off != 0;
    const bool plans = tls.plans_used[c->device];
    if ((!up && !arena && !plans) || capturing(c->stream)) return;
    const unsigned long long id = stream_id(c->stream);
    bool ok = true;
    if (up) {
        ok = cudaEventRecord(up->done, c->stream) == cudaSuccess;
        up->stream = id;
        up->pending = ok;
    }
    if (arena) ok &= mark(tls.arena[c->device], c->stream, id);
    if (plans) ok &= mark(tls.plans[c->device], c->stream, id);
    if (!ok) {
        cudaGetLastError();
        cudaStreamSynchronize(c->stream);  // no event to be had: drain instead
    }
}

bool is_device_ptr(const void* p) {
    cudaPointerAttributes a;
    if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    return a.type == cudaMemoryTypeDevice || a.type == cudaMemoryTypeManaged;
}

Status stage_in(Ctx* c, const void* p, size_t bytes, const void** dev) {
    if (p == nullptr || bytes == 0 || is_device_ptr(p)) {
        *dev = p;
        return Status();
    }
    void* d;
    SLHA_TRY(ctx_device_scratch(c, bytes, &d));
    SLHA_CUDA(cudaMemcpyAsync(d, p, bytes, cudaMemcpyHostToDevice, c->stream));
    *dev = d;
    return Status();
}

Status stage_out(Ctx* c, void* user, size_t bytes, StagedOut* out, bool in_place_if_pinned) {
    out->user = user;
    out->bytes = bytes;
    if (user == nullptr || bytes == 0 || is_device_ptr(user)) {
        out->dev = user;
        out->is_host = false;
        return Status();
    }
    // Page-locked host memory the GPU can address (cudaHostAlloc, cudaHostRegister with mapping) is written in place by the
    // kernels: the results cross the bus while the kernel that produces them runs, instead of in a copy queued behind it.
    // Only for outputs that the call's kernels write once and never read (the caller says so).
    cudaPointerAttributes a;
    if (in_place_if_pinned && cudaPointerGetAttributes(&a, user) == cudaSuccess && a.type == cudaMemoryTypeHost && a.devicePointer != nullptr) {
        out->dev = a.devicePointer;
        out->is_host = false;
        return Status();
    }
    cudaGetLastError();
    out->is_host = true;
    // Few bytes (a call's counts): the kernels write page-locked memory of the thread, from where finish_outputs copies them.  A copy behind the
    // kernels took 7 us.
    if (in_place_if_pinned && bytes <= OUT_BYTES && !capturing(c->stream)) {
        OutPage& o = tls.outs[c->device];
        if (!o.host) {
            o.device = c->device;
            SLHA_CUDA(cudaHostAlloc((void**)&o.host, OUT_PAGE, cudaHostAllocMapped | cudaHostAllocPortable));
            SLHA_CUDA(cudaHostGetDevicePointer((void**)&o.dev, o.host, 0));
        }
        const size_t take = (bytes + 15) / 16 * 16;
        if (o.used + take <= OUT_PAGE) {
            if (!o.used) o.launched = g_thread_launches;
            out->dev = o.dev + o.used;
            out->page = o.host + o.used;
            o.used += take;
            return Status();
        }
    }
    return ctx_device_scratch(c, bytes, &out->dev);
}

Status finish_outputs(Ctx* c, std::vector<StagedOut>& outs, bool force_sync) {
    bool any = false;
    for (StagedOut& o : outs)
        if (o.is_host && o.bytes) {
            if (!o.page) SLHA_CUDA(cudaMemcpyAsync(o.user, o.dev, o.bytes, cudaMemcpyDeviceToHost, c->stream));
            any = true;
        }
    if (any || force_sync) SLHA_CUDA(cudaStreamSynchronize(c->stream));
    for (StagedOut& o : outs)
        if (o.page) {
            std::memcpy(o.user, o.page, o.bytes);
            tls.outs[c->device].used -= (o.bytes + 15) / 16 * 16;
        }
    return Status();
}

// ---- model registry ------------------------------------------------------------
// Handles are addresses of small heap tokens.  A released token is kept forever
// in a retired list so that its address can never become a live handle again
// (same guarantee as slha-c/src/lib.rs:124-205).
namespace {
struct Token { uint64_t opaque; };
struct Registry {
    std::shared_mutex mu;
    std::unordered_map<const void*, std::pair<std::unique_ptr<Token>, std::shared_ptr<Model>>> live;
    std::vector<std::unique_ptr<Token>> retired;
};
Registry& registry() {
    static Registry* r = new Registry();
    return *r;
}
}  // namespace

std::shared_ptr<Model> model_lookup(const SlhaModel* handle, Status* st) {
    if (handle == nullptr) {
        *st = Status(SLHA_ERR_NULL, "model handle is NULL");
        return nullptr;
    }
    if (reinterpret_cast<uintptr_t>(handle) % alignof(uint64_t) != 0) {
        *st = Status(SLHA_ERR_INVALID_HANDLE, "model handle is misaligned");
        return nullptr;
    }
    Registry& r = registry();
    std::shared_lock<std::shared_mutex> lk(r.mu);
    auto it = r.live.find(handle);
    if (it == r.live.end()) {
        *st = Status(SLHA_ERR_INVALID_HANDLE, "model handle is not a live SLHA handle");
        return nullptr;
    }
    return it->second.second;
}
SlhaModel* model_register(std::shared_ptr<Model> m) {
    Registry& r = registry();
    auto tok = std::make_unique<Token>();
    const void* key = tok.get();
    std::unique_lock<std::shared_mutex> lk(r.mu);
    r.live.emplace(key, std::make_pair(std::move(tok), std::move(m)));
    return reinterpret_cast<SlhaModel*>(const_cast<void*>(key));
}
bool model_unregister(SlhaModel* handle) {
    Registry& r = registry();
    std::unique_lock<std::shared_mutex> lk(r.mu);
    auto it = r.live.find(handle);
    if (it == r.live.end()) return false;
    r.retired.push_back(std::move(it->second.first));
    r.live.erase(it);
    return true;
}

// ---- model construction -----------------------------------------------------------
namespace {
// SplitMix64 + Box-Muller, scirust/src/rng.rs:13-51.  The matrix is generated on
// the host with libm logf/cosf (what Rust's f32::ln / f32::cos call) and uploaded.
struct Rng {
    uint64_t state;
    explicit Rng(uint64_t seed) : state(seed ^ 0x9E3779B97F4A7C15ull) {}
    uint64_t next_u64() {
        state += 0x9E3779B97F4A7C15ull;
        uint64_t z = state;
        z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
        z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
        return z ^ (z >> 31);
    }
    float next_unit() { return (float)(next_u64() >> 40) * (1.0f / (float)(1ull << 24)); }
    float next_gaussian() {
        float u1 = next_unit();
        if (!(u1 > 1.0e-7f)) u1 = 1.0e-7f;
        const float u2 = next_unit();
        const float r = sqrtf(-2.0f * logf(u1));
        return r * cosf(2.0f * 3.14159265358979323846f * u2);
    }
};
void free_model(Model* m) {
    cudaFree(m->block);
    delete m;
}
}  // namespace

Status model_build(Ctx* c, const float* p, size_t d, uint64_t seed, bool rht, const float* scale,
                   const float* z, std::shared_ptr<Model>* out) {
    if (d == 0 || d > (1u << 20)) return Status(SLHA_ERR_DIMENSION, "projection must be D_C x d with 0 < d <= 2^20");
    for (size_t i = 0; i < (size_t)D_C * d; ++i)
        if (!std::isfinite(p[i])) return Status(SLHA_ERR_NONFINITE, "projection contains a non-finite value");
    std::shared_ptr<Model> m(new Model(), free_model);
    m->d = d;
    m->rht = rht;
    m->device = c->device;
    size_t dp = d;
    if (rht) {  // incoherence.rs:29-35 next_pow2
        dp = 1;
        while (dp < d) dp <<= 1;
    }
    m->d_pad = dp;
    // one allocation; P, scale, Z and the diagonal go up in one copy, the transposed copies and the fragments of Z are made there
    const size_t zfb = (dp + 31) / 32 * 32 * 32 * 16;
    size_t at[8] = {0};
    at[1] = pad256(D_C * d * 4);              // 0 P, 1 scale
    at[2] = at[1] + pad256(D_C * 4);          // 2 Z
    at[3] = at[2] + pad256(D_S * dp * 4);     // 3 diagonal
    at[4] = at[3] + pad256(rht ? dp * 4 : 0); // 4 P transposed, from here on made on the device
    at[5] = at[4] + pad256(D_C * d * 4);      // 5 Z transposed
    at[6] = at[5] + pad256(D_S * dp * 4);     // 6 fragments
    at[7] = at[6] + (dp <= 256 ? zfb : 0);    // 7 figures of the fragments' rounding
    std::unique_ptr<float[]> host(new float[at[4] / 4]);
    const auto part = [&](int i) { return host.get() + at[i] / 4; };
    std::memcpy(part(0), p, D_C * d * 4);
    for (int k = 0; k < D_C; ++k) {
        if (scale && (!std::isfinite(scale[k]) || scale[k] <= 0.0f))
            return Status(SLHA_ERR_NONFINITE, "whitening scale must be finite and positive");
        part(1)[k] = scale ? scale[k] : 1.0f;
    }
    if (rht) {  // learned.rs:158-165 + incoherence.rs:89-97
        Rng r(seed ^ 0xA2A2A2A2A2A2A2A2ull);
        for (size_t i = 0; i < dp; ++i) part(3)[i] = r.next_unit() < 0.5f ? -1.0f : 1.0f;
    }
    if (z) {
        std::memcpy(part(2), z, D_S * dp * 4);
    } else {  // learned.rs:168-170
        Rng r(seed);
        float* zp = part(2);
        for (size_t i = 0; i < D_S * dp; ++i) zp[i] = r.next_gaussian();
    }
    SLHA_CUDA(cudaMalloc(&m->block, at[7] + D_S * 8 + 256));
    SLHA_CUDA(cudaMemcpyAsync(m->block, host.get(), at[4], cudaMemcpyHostToDevice, c->stream));
    const auto array = [&](int i) { return reinterpret_cast<float*>((char*)m->block + at[i]); };
    m->d_p = array(0);
    m->d_scale = array(1);
    m->d_z = array(2);
    m->d_diag = rht ? array(3) : nullptr;
    m->d_pt = array(4);
    m->d_zt = array(5);
    SLHA_TRY(build_model_arrays(c, m.get(), reinterpret_cast<uint4*>(array(6)), array(7)));
    SLHA_CUDA(cudaStreamSynchronize(c->stream));
    *out = std::move(m);
    return Status();
}

Status model_load_slhw(Ctx* c, const char* path, std::shared_ptr<Model>* out) {
    // weights.rs:284-311: regular file, <= 256 MiB
    struct stat sb;
    if (stat(path, &sb) != 0) return Status(SLHA_ERR_IO, std::string("weights: cannot stat ") + path);
    if (!S_ISREG(sb.st_mode)) return Status(SLHA_ERR_IO, std::string("weights: ") + path + " is not a regular file");
    if ((uint64_t)sb.st_size > 256ull * 1024 * 1024) return Status(SLHA_ERR_IO, "weights: file above the 256 MiB safety cap");
    FILE* f = std::fopen(path, "rb");
    if (!f) return Status(SLHA_ERR_IO, std::string("weights: cannot read ") + path);
    std::vector<unsigned char> b((size_t)sb.st_size);
    const size_t got = b.empty() ? 0 : std::fread(b.data(), 1, b.size(), f);
    std::fclose(f);
    if (got != b.size()) return Status(SLHA_ERR_IO, std::string("weights: short read on ") + path);
    // weights.rs:159-270
    auto u32_at = [&](size_t o) {
        return (uint32_t)b[o] | ((uint32_t)b[o + 1] << 8) | ((uint32_t)b[o + 2] << 16) | ((uint32_t)b[o + 3] << 24);
    };
    if (b.size() < 24) return Status(SLHA_ERR_IO, "weights: truncated header");
    if (u32_at(0) != 0x534C4857u) return Status(SLHA_ERR_IO, "weights: bad magic (not an SLHW file)");
    const uint32_t version = u32_at(4);
    size_t header;
    if (version == 1) header = 24;
    else if (version == 2) header = 28;
    else return Status(SLHA_ERR_IO, "weights: unsupported version " + std::to_string(version) + " (supported: 1 and 2)");
    if (b.size() < header) return Status(SLHA_ERR_IO, "weights: truncated header");
    const size_t d = u32_at(8);
    if (d <= (size_t)D_C)
        return Status(SLHA_ERR_IO, "weights: invalid dimension " + std::to_string(d) + " (must be greater than D_C=128)");
    uint64_t seed = 0;
    for (int i = 0; i < 8; ++i) seed |= (uint64_t)b[12 + i] << (8 * i);
    if (b[20] > 1) return Status(SLHA_ERR_IO, "weights: invalid RHT flag " + std::to_string(b[20]) + " (expected 0 or 1)");
    if (b[21] || b[22] || b[23]) return Status(SLHA_ERR_IO, "weights: non-zero reserved header bytes");
    const size_t expected = header + (size_t)D_C * d * 4;
    if (b.size() != expected)
        return Status(SLHA_ERR_IO, "weights: size mismatch (got " + std::to_string(b.size()) + ", expected " + std::to_string(expected) + ")");
    if (version == 2) {  // FNV-1a over the 24-byte header and the payload, weights.rs:68-80
        uint32_t h = 0x811C9DC5u;
        for (size_t i = 0; i < 24; ++i) { h ^= b[i]; h *= 0x01000193u; }
        for (size_t i = 28; i < b.size(); ++i) { h ^= b[i]; h *= 0x01000193u; }
        if (h != u32_at(24)) return Status(SLHA_ERR_IO, "weights: checksum mismatch");
    }
    std::vector<float> p((size_t)D_C * d);
    std::memcpy(p.data(), b.data() + header, p.size() * 4);
    for (size_t i = 0; i < p.size(); ++i)
        if (!std::isfinite(p[i]))
            return Status(SLHA_ERR_IO, "weights: non-finite projection value at index " + std::to_string(i));
    return model_build(c, p.data(), d, seed, b[20] == 1, nullptr, nullptr, out);
}

Status validate_tile_host(const SciRustSlhaTile& t) {
    const uint16_t known = F_WARM | F_NF4 | F_MIXED | F_TQ3 | F_NOCORR | F_MIX3;
    if (t.flags & ~known) {
        char buf[64];
        std::snprintf(buf, sizeof buf, "tile contains unknown flag bits: 0x%04x", t.flags);
        return Status(SLHA_ERR_INVALID_TILE, buf);
    }
    if (__builtin_popcount(t.flags & (F_NF4 | F_MIXED | F_TQ3 | F_MIX3)) > 1)
        return Status(SLHA_ERR_INVALID_TILE, "tile selects more than one latent codec");
    if ((t.flags & F_NOCORR) && !(t.flags & (F_TQ3 | F_MIX3)))
        return Status(SLHA_ERR_INVALID_TILE, "correction-drop flag requires the TQ3 or MIX3 codec");
    if (!std::isfinite(t.scale) || !std::isfinite(t.dynamic_lambda) || !std::isfinite(t.residual_sigma))
        return Status(SLHA_ERR_NONFINITE, "tile metadata contains a non-finite float");
    if (t.scale < 0.0f || t.dynamic_lambda < 0.0f || t.residual_sigma < 0.0f)
        return Status(SLHA_ERR_INVALID_TILE, "tile scale, dynamic lambda, and residual sigma must be non-negative");
    return Status();
}

}  // namespace slha
