// Context lifetime, error reporting and host/device staging.
#include <algorithm>
#include <atomic>
#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <optional>
#include <thread>

#include "dt_core.cuh"

namespace dt {

static thread_local std::string g_last_error;

std::string fmt(const char *f, ...) {
    char buf[1024];
    va_list ap;
    va_start(ap, f);
    vsnprintf(buf, sizeof(buf), f, ap);
    va_end(ap);
    return std::string(buf);
}

void set_last_error(const std::string &msg) { g_last_error = msg; }
void clear_last_error() { g_last_error.clear(); }

void check_shape(int ndim, const int64_t *shape, const char *who) {
    DT_CHECK_ARG(ndim >= 1 && ndim <= 16 && shape, "%s: bad ndim %d", who, ndim);
    int64_t total = 1;
    for (int i = 0; i < ndim; i++) {
        DT_CHECK_ARG(shape[i] >= 1, "%s: shape[%d] = %lld must be >= 1", who, i,
                     (long long)shape[i]);
        DT_CHECK_ARG(shape[i] <= (int64_t(1) << 62) / total,
                     "%s: the element count overflows at shape[%d] = %lld", who, i,
                     (long long)shape[i]);
        total *= shape[i];
    }
}

bool is_device_ptr(const void *p) {
    if (!p) return false;
    cudaPointerAttributes attr;
    cudaError_t e = cudaPointerGetAttributes(&attr, p);
    if (e != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    return attr.type == cudaMemoryTypeDevice || attr.type == cudaMemoryTypeManaged;
}

bool pdl_enabled() {
    static const bool on = [] {
        const char *e = std::getenv("DT_DISABLE_PDL");
        return !(e && e[0] == '1');
    }();
    return on;
}

bool graphs_enabled() {
    static const bool on = [] {
        const char *e = std::getenv("DT_DISABLE_GRAPHS");
        return !(e && e[0] == '1');
    }();
    return on;
}

void release_plan(dt_ctx *ctx, std::shared_ptr<void> &plan) {
    if (!plan) return;
    DT_CUDA(cudaStreamSynchronize(ctx->stream));
    plan.reset();
}

void SweepGraph::reset() {
    if (exec_) cudaGraphExecDestroy(exec_);
    exec_ = nullptr;
    launches_ = 0;
}

void SweepGraph::run(dt_ctx *ctx, const std::function<void()> &fn) {
    if (!exec_) {
        if (failed_ || !graphs_enabled()) {
            fn();
            return;
        }
        std::optional<CaptureStream> on(ctx);
        const int64_t l0 = ctx->launches;
        auto give_up = [&](cudaGraph_t g) {
            if (g) cudaGraphDestroy(g);
            cudaGetLastError();
            ctx->launches = l0;
            failed_ = true;
        };
        DT_CUDA(cudaStreamBeginCapture(ctx->stream, cudaStreamCaptureModeRelaxed));
        cudaGraph_t g = nullptr;
        try {
            fn();
        } catch (const Error &e) {
            cudaStreamEndCapture(ctx->stream, &g);
            if (e.code == DT_ERR_NOMEM) {
                // Out of memory (or over the context's cap): the call fails and
                // the next one captures again.
                if (g) cudaGraphDestroy(g);
                cudaGetLastError();
                ctx->launches = l0;
                throw;
            }
            give_up(g);
            on.reset();
            fn();
            return;
        } catch (...) {
            cudaStreamEndCapture(ctx->stream, &g);
            give_up(g);
            on.reset();
            fn();
            return;
        }
        if (cudaStreamEndCapture(ctx->stream, &g) != cudaSuccess || !g) {
            give_up(g);
            on.reset();
            fn();
            return;
        }
        if (cudaGraphInstantiateWithFlags(&exec_, g, 0) != cudaSuccess) {
            exec_ = nullptr;
            give_up(g);
            on.reset();
            fn();
            return;
        }
        cudaGraphDestroy(g);
        launches_ = ctx->launches - l0;
        ctx->launches = l0;
    }
    DT_CUDA(cudaGraphLaunch(exec_, ctx->stream));
    ctx->launches += launches_;
}

void raise_smem_limit(dt_ctx *ctx, const void *kernel, size_t bytes) {
    static std::mutex mu;
    static std::map<std::pair<const void *, int>, size_t> limits;
    std::lock_guard<std::mutex> lock(mu);
    size_t &cur = limits[{kernel, ctx->device}];
    if (bytes <= cur) return;
    DT_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes));
    cur = bytes;
}

void *DevArena::take(size_t bytes) {
    bytes = (bytes + 255) & ~size_t(255);
    size_t off = 0;
    auto at = used_.begin();
    for (; at != used_.end() && at->first - off < bytes; ++at) off = at->first + at->second;
    used_.insert(at, {off, bytes});
    need = std::max(need, off + bytes);
    if (cap && off + bytes > cap)
        fail(DT_ERR_CUDA, fmt("internal: sweep arena of %zu bytes exceeded", cap));
    return base + off;
}

void DevArena::give(void *p) {
    const size_t off = (size_t)(static_cast<char *>(p) - base);
    for (auto it = used_.begin(); it != used_.end(); ++it)
        if (it->first == off) {
            used_.erase(it);
            return;
        }
}

bool release_idle(dt_ctx *ctx) {
    cudaStreamCaptureStatus st;
    if (cudaStreamIsCapturing(ctx->stream, &st) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    if (st != cudaStreamCaptureStatusNone) return false;
    // A running call holds a reference of its own to the plan it uses.
    auto &kept = ctx->hooi_plans_fp64;
    for (size_t k = kept.size(); k-- > 0;)
        if (kept[k].use_count() == 1) {
            release_plan(ctx, kept[k]);
            kept.erase(kept.begin() + k);
            return true;
        }
    if (ctx->hooi_plan_mixed.use_count() == 1) {
        release_plan(ctx, ctx->hooi_plan_mixed);
        return true;
    }
    return release_batched_scratch(ctx);
}

bool DevMem::try_alloc(dt_ctx *ctx, size_t bytes) {
    release();
    if (bytes == 0) return true;
    if (ctx->arena) {
        p_ = ctx->arena->take(bytes);
        arena_ = ctx->arena;
        bytes_ = bytes;
        return true;
    }
    for (;;) {
        if (!ctx->mem_limit || ctx->mem_in_use + bytes <= ctx->mem_limit) {
            const cudaError_t e = cudaMallocAsync(&p_, bytes, ctx->stream);
            if (e == cudaSuccess) break;
            p_ = nullptr;
            if (e != cudaErrorMemoryAllocation) DT_CUDA(e);
            cudaGetLastError();
        }
        if (!release_idle(ctx)) return false;
    }
    ctx_ = ctx;
    bytes_ = bytes;
    ctx->mem_in_use += bytes;
    ctx->mem_peak = std::max(ctx->mem_peak, ctx->mem_in_use);
    return true;
}

void DevMem::alloc(dt_ctx *ctx, size_t bytes) {
    if (try_alloc(ctx, bytes)) return;
    if (ctx->mem_limit && ctx->mem_in_use + bytes > ctx->mem_limit)
        fail(DT_ERR_NOMEM, fmt("device allocation of %zu bytes would exceed the context's "
                               "limit (%llu of %llu bytes in use)",
                               bytes, (unsigned long long)ctx->mem_in_use,
                               (unsigned long long)ctx->mem_limit));
    fail(DT_ERR_NOMEM, fmt("device allocation of %zu bytes failed", bytes));
}

void DevMem::release() {
    if (arena_) arena_->give(p_);
    arena_ = nullptr;
    if (p_ && ctx_) {
        cudaFreeAsync(p_, ctx_->stream);
        ctx_->mem_in_use -= bytes_;
    }
    p_ = nullptr;
    bytes_ = 0;
}

void ChunkedUpload::start(dt_ctx *c, const void *host, int64_t count, size_t esz) {
    constexpr int kc = dt_ctx::kCopyChunks;
    if (!c->copy_stream) {
        DT_CUDA(cudaStreamCreateWithFlags(&c->copy_stream, cudaStreamNonBlocking));
        for (cudaEvent_t &e : c->copy_ev)
            DT_CUDA(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
    }
    n = count;
    step = std::max<int64_t>(1024, ((n + kc - 1) / kc + 1023) / 1024 * 1024);
    chunks = (int)((n + step - 1) / step);
    dst.alloc(c, (size_t)n * esz);
    // The copies follow the context stream's earlier work (dst's allocation).
    DT_CUDA(cudaEventRecord(c->copy_ev[kc], c->stream));
    DT_CUDA(cudaStreamWaitEvent(c->copy_stream, c->copy_ev[kc], 0));
    for (int q = 0; q < chunks; q++) {
        DT_CUDA(cudaMemcpyAsync(static_cast<char *>(dst.get()) + offset(q) * esz,
                                static_cast<const char *>(host) + offset(q) * esz,
                                (size_t)length(q) * esz, cudaMemcpyHostToDevice, c->copy_stream));
        DT_CUDA(cudaEventRecord(c->copy_ev[q], c->copy_stream));
    }
}

void ChunkedUpload::wait(dt_ctx *c, int q) const {
    DT_CUDA(cudaStreamWaitEvent(c->stream, c->copy_ev[q], 0));
}

DevView::DevView(dt_ctx *ctx, const void *p, size_t bytes, bool is_input, bool is_output)
    : ctx_(ctx), user_(const_cast<void *>(p)), dptr_(nullptr), bytes_(bytes),
      output_(is_output), staged_(false) {
    if (bytes == 0) return;
    if (!p) fail(DT_ERR_ARG, "null buffer");
    if (is_device_ptr(p)) {
        dptr_ = user_;
        return;
    }
    staged_ = true;
    mem_.alloc(ctx, bytes);
    dptr_ = mem_.get();
    if (is_input)
        DT_CUDA(cudaMemcpyAsync(dptr_, p, bytes, cudaMemcpyHostToDevice, ctx->stream));
}

void copy_out(dt_ctx *ctx, void *user, const void *src, size_t bytes) {
    if (bytes == 0) return;
    if (!user) fail(DT_ERR_ARG, "null output buffer");
    DT_CUDA(cudaMemcpyAsync(user, src, bytes, cudaMemcpyDefault, ctx->stream));
}

namespace {

struct BlockList {
    const unsigned long long *src[kMaxCopyBlocks];
    unsigned long long *dst[kMaxCopyBlocks];
    long long words[kMaxCopyBlocks];
    int count;
};

// Every block in one grid-stride pass: 8-byte words, consecutive threads on
// consecutive words.
__global__ void copy_blocks_kernel(BlockList b) {
    const long long stride = (long long)gridDim.x * blockDim.x;
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    for (int k = 0; k < b.count; k++)
        for (long long i = t; i < b.words[k]; i += stride) b.dst[k][i] = b.src[k][i];
}

// How a kernel on the context's GPU may store to p: directly (device or managed
// memory of that GPU), by way of the host (host memory), or not at all.
enum class Reach { Direct, Host, No };

Reach reach(const dt_ctx *ctx, const void *p) {
    cudaPointerAttributes attr;
    if (cudaPointerGetAttributes(&attr, p) != cudaSuccess) {
        cudaGetLastError();
        return Reach::No;
    }
    if (attr.type == cudaMemoryTypeUnregistered || attr.type == cudaMemoryTypeHost)
        return Reach::Host;
    return attr.device == ctx->device ? Reach::Direct : Reach::No;
}

}  // namespace

void OutBlocks::add(void *dst, const void *src, size_t bytes) {
    if (!dst || bytes == 0) return;
    DT_CHECK_ARG(n_ < kMaxCopyBlocks, "OutBlocks: more than %d blocks", kMaxCopyBlocks);
    dst_[n_] = dst;
    src_[n_] = src;
    bytes_[n_++] = bytes;
}

// A copy into pageable memory holds the calling thread for ~12 us each, and one
// into pinned memory costs its own slot on the stream; the kernel stores to
// pinned memory across PCIe, in order with the rest of its blocks.
void OutBlocks::queue() {
    BlockList b{};
    size_t staged = 0;
    long long most = 0;
    bool one_launch = true;
    for (int k = 0; k < n_ && one_launch; k++) {
        void *to = dst_[k];
        one_launch = (reinterpret_cast<uintptr_t>(src_[k]) | bytes_[k]) % 8 == 0;
        const size_t at = static_cast<char *>(to) - static_cast<char *>(ctx_->host_stage);
        if (!ctx_->host_stage || at >= dt_ctx::kHostStageBytes) {
            const Reach r = reach(ctx_, to);
            if (r == Reach::Host) {
                if (staged + bytes_[k] > dt_ctx::kOutStageBytes) one_launch = false;
                if (!one_launch) break;
                if (!ctx_->out_stage)
                    DT_CUDA(cudaHostAlloc(&ctx_->out_stage, dt_ctx::kOutStageBytes,
                                          cudaHostAllocDefault));
                stage_[k] = to = static_cast<char *>(ctx_->out_stage) + staged;
                staged += bytes_[k];
            } else if (r == Reach::No || reinterpret_cast<uintptr_t>(to) % 8 != 0) {
                one_launch = false;
            }
        }
        b.src[k] = static_cast<const unsigned long long *>(src_[k]);
        b.dst[k] = static_cast<unsigned long long *>(to);
        b.words[k] = (long long)(bytes_[k] / 8);
        most = std::max(most, b.words[k]);
    }
    if (!one_launch) {
        for (int k = 0; k < n_; k++) {
            stage_[k] = nullptr;
            copy_out(ctx_, dst_[k], src_[k], bytes_[k]);
        }
        return;
    }
    if (n_ == 0) return;
    b.count = n_;
    const int threads = 256;
    const long long want = (most + threads - 1) / threads;
    const unsigned blocks = (unsigned)std::max(1LL, std::min<long long>(want, 2LL * ctx_->num_sms));
    DT_LAUNCH(ctx_, copy_blocks_kernel, blocks, threads, 0, b);
}

void OutBlocks::finish() {
    for (int k = 0; k < n_; k++)
        if (stage_[k]) std::memcpy(dst_[k], stage_[k], bytes_[k]);
}

namespace {

constexpr size_t kChunk = size_t(1) << 20, kStageFrom = size_t(1) << 20;
constexpr size_t kCopyThreads = 4;
static_assert(2 * kCopyThreads * kChunk <= dt_ctx::kBigStageBytes, "two slots per thread");

struct Chunk {
    char *dev, *host;
    size_t bytes;
};

// fn(0) .. fn(n - 1) over a few threads; the first CUDA error is thrown here.
void over_threads(dt_ctx *ctx, size_t n, const std::function<cudaError_t(size_t)> &fn) {
    const size_t most =
        std::max<size_t>(1, std::min<size_t>(kCopyThreads, std::thread::hardware_concurrency() / 2));
    std::atomic<size_t> next{0};
    std::atomic<int> err{(int)cudaSuccess};
    auto work = [&] {
        cudaSetDevice(ctx->device);
        for (size_t i; (i = next.fetch_add(1)) < n;) {
            const cudaError_t e = fn(i);
            if (e != cudaSuccess) err.store((int)e);
        }
    };
    std::vector<std::thread> pool;
    pool.reserve(kCopyThreads);
    try {
        for (size_t k = 1; k < std::min(most, n); k++) pool.emplace_back(work);
    } catch (...) {  // no more threads or memory for one: the ones there do it
    }
    work();
    for (auto &t : pool) t.join();
    DT_CUDA((cudaError_t)err.load());
}

// What `later` is given from now on runs after what `earlier` has been given.
void stream_after(cudaStream_t later, cudaStream_t earlier) {
    cudaEvent_t ev;
    DT_CUDA(cudaEventCreateWithFlags(&ev, cudaEventDisableTiming));
    cudaError_t e = cudaEventRecord(ev, earlier);
    if (e == cudaSuccess) e = cudaStreamWaitEvent(later, ev, 0);
    cudaEventDestroy(ev);  // (its place in the streams stays)
    DT_CUDA(e);
}

// The pieces in chunks, dealt to kCopyThreads lanes; lane l has two slots of the
// pinned staging, so one chunk's DMA runs while the other is copied by the host.
// run(stream, chunks of the lane, its slots, its events) on a thread of its own
// where there is one.  The DMA goes to ctx->stream; cudaStreamPerThread, which names
// another stream in each thread, is stood in for by the context's own stream, which
// starts after what the caller's has been given and which that waits for in turn.
// 281 k rows of 16, 10 sweeps, both ways: 15.0 ms a call and 41 ms for
// a context's first one with 8 MB of staging; 15.2 and 54 ms with 32 MB filled and
// drained whole (pinning them is the difference), 18 ms with 8 MB in such rounds.
void over_lanes(dt_ctx *ctx, const std::vector<HostPiece> &pieces,
                const std::function<cudaError_t(cudaStream_t, const std::vector<Chunk> &,
                                                char *const *, const cudaEvent_t *)> &run) {
    const bool stand_in = ctx->stream == cudaStreamPerThread;
    const cudaStream_t dma = stand_in ? ctx->own_stream : ctx->stream;
    if (stand_in) stream_after(dma, ctx->stream);
    std::vector<Chunk> lane[kCopyThreads];
    size_t n = 0;
    for (const HostPiece &p : pieces)
        for (size_t o = 0; o < p.bytes; o += kChunk)
            lane[n++ % kCopyThreads].push_back({static_cast<char *>(p.dev) + o,
                                                static_cast<char *>(p.host) + o,
                                                std::min(kChunk, p.bytes - o)});
    auto one_lane = [&](size_t l) {
        char *slot[2];
        cudaEvent_t ev[2] = {};
        cudaError_t e = cudaSuccess;
        for (int s = 0; s < 2; s++) {
            slot[s] = static_cast<char *>(ctx->big_stage) + (2 * l + s) * kChunk;
            if (e == cudaSuccess) e = cudaEventCreateWithFlags(&ev[s], cudaEventDisableTiming);
        }
        if (e == cudaSuccess) e = run(dma, lane[l], slot, ev);
        for (cudaEvent_t x : ev)
            if (x) cudaEventDestroy(x);
        return e;
    };
    // (After an error too: the caller's stream then frees what the DMA may still use.)
    try {
        over_threads(ctx, kCopyThreads, one_lane);
    } catch (...) {
        if (stand_in) stream_after(ctx->stream, dma);
        throw;
    }
    if (stand_in) stream_after(ctx->stream, dma);
}

// Whether the pieces go through the staging: enough bytes, and memory to pin.
bool staged(dt_ctx *ctx, const std::vector<HostPiece> &pieces) {
    size_t total = 0;
    for (const HostPiece &p : pieces) total += p.bytes;
    if (total < kStageFrom) return false;
    if (!ctx->big_stage &&
        cudaHostAlloc(&ctx->big_stage, dt_ctx::kBigStageBytes, cudaHostAllocDefault) != cudaSuccess) {
        cudaGetLastError();
        ctx->big_stage = nullptr;
    }
    return ctx->big_stage != nullptr;
}

}  // namespace

void upload_pieces(dt_ctx *ctx, const std::vector<HostPiece> &pieces) {
    if (!staged(ctx, pieces)) {
        for (const HostPiece &p : pieces)
            DT_CUDA(cudaMemcpyAsync(p.dev, p.host, p.bytes, cudaMemcpyHostToDevice, ctx->stream));
        return;
    }
    // An earlier call's DMA out of the staging is done: every call that uses it
    // ends with a synchronisation.
    over_lanes(ctx, pieces, [&](cudaStream_t dma, const std::vector<Chunk> &cs,
                                char *const *slot, const cudaEvent_t *ev) {
        cudaError_t e = cudaSuccess;
        for (size_t i = 0; i < cs.size() && e == cudaSuccess; i++) {
            const int s = i & 1;
            if (i >= 2) e = cudaEventSynchronize(ev[s]);  // the slot's last DMA
            if (e != cudaSuccess) break;
            std::memcpy(slot[s], cs[i].host, cs[i].bytes);
            e = cudaMemcpyAsync(cs[i].dev, slot[s], cs[i].bytes, cudaMemcpyHostToDevice, dma);
            if (e == cudaSuccess) e = cudaEventRecord(ev[s], dma);
        }
        return e;
    });
}

void download_pieces(dt_ctx *ctx, const std::vector<HostPiece> &pieces) {
    if (!staged(ctx, pieces)) {
        for (const HostPiece &p : pieces)
            DT_CUDA(cudaMemcpyAsync(p.host, p.dev, p.bytes, cudaMemcpyDeviceToHost, ctx->stream));
        DT_CUDA(cudaStreamSynchronize(ctx->stream));
        return;
    }
    over_lanes(ctx, pieces, [&](cudaStream_t dma, const std::vector<Chunk> &cs,
                                char *const *slot, const cudaEvent_t *ev) {
        auto fetch = [&](size_t i) {
            const int s = i & 1;
            const cudaError_t e = cudaMemcpyAsync(slot[s], cs[i].dev, cs[i].bytes,
                                                  cudaMemcpyDeviceToHost, dma);
            return e == cudaSuccess ? cudaEventRecord(ev[s], dma) : e;
        };
        cudaError_t e = cs.empty() ? cudaSuccess : fetch(0);
        for (size_t i = 0; i < cs.size() && e == cudaSuccess; i++) {
            if (i + 1 < cs.size()) e = fetch(i + 1);
            if (e == cudaSuccess) e = cudaEventSynchronize(ev[i & 1]);
            if (e == cudaSuccess) std::memcpy(cs[i].host, slot[i & 1], cs[i].bytes);
        }
        return e;
    });
}

void *host_stage(dt_ctx *ctx) {
    if (!ctx->host_stage)
        DT_CUDA(cudaHostAlloc(&ctx->host_stage, dt_ctx::kHostStageBytes, cudaHostAllocDefault));
    return ctx->host_stage;
}

void DevView::finish() {
    if (output_ && staged_ && bytes_) {
        DT_CUDA(cudaMemcpyAsync(user_, dptr_, bytes_, cudaMemcpyDeviceToHost, ctx_->stream));
        DT_CUDA(cudaStreamSynchronize(ctx_->stream));
    }
}

}  // namespace dt

using namespace dt;

extern "C" {

const char *dt_last_error(void) { return g_last_error.c_str(); }

int dt_ctx_create(int device, dt_ctx **out) {
    return guard([&] {
        DT_CHECK_ARG(out, "dt_ctx_create: null output pointer");
        int n = 0;
        DT_CUDA(cudaGetDeviceCount(&n));
        DT_CHECK_ARG(device >= 0 && device < n, "dt_ctx_create: device %d out of range (%d)",
                     device, n);
        DT_CUDA(cudaSetDevice(device));
        cudaDeviceProp prop;
        DT_CUDA(cudaGetDeviceProperties(&prop, device));
        if (prop.major < 10)
            fail(DT_ERR_UNSUPPORTED,
                 fmt("device %d is sm_%d%d; this library is built for sm_100a", device,
                     prop.major, prop.minor));
        auto *ctx = new dt_ctx();
        ctx->device = device;
        ctx->num_sms = prop.multiProcessorCount;
        // Keep freed stream-ordered allocations cached in the device's pool:
        // with the default threshold of 0 every synchronisation returns them
        // to the driver and the next cudaMallocAsync has to map pages again.
        cudaMemPool_t pool;
        DT_CUDA(cudaDeviceGetDefaultMemPool(&pool, device));
        uint64_t keep = ~0ULL;
        DT_CUDA(cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep));
        DT_CUDA(cudaStreamCreateWithFlags(&ctx->own_stream, cudaStreamNonBlocking));
        ctx->stream = ctx->own_stream;
        DT_CUDA(cudaEventCreate(&ctx->ev_start));
        DT_CUDA(cudaEventCreate(&ctx->ev_stop));
        *out = ctx;
    });
}

int dt_ctx_destroy(dt_ctx *ctx) {
    return guard([&] {
        if (!ctx) return;
        cudaSetDevice(ctx->device);
        detach_sptensors(ctx);
        if (ctx->stream) cudaStreamSynchronize(ctx->stream);
        ctx->hooi_plans_fp64.clear();
        ctx->hooi_plan_mixed.reset();
        ctx->batched.reset();
        ctx->summary.reset();
        if (ctx->stream) cudaStreamSynchronize(ctx->stream);
        if (ctx->ev_start) cudaEventDestroy(ctx->ev_start);
        if (ctx->ev_stop) cudaEventDestroy(ctx->ev_stop);
        if (ctx->copy_stream) {
            cudaStreamSynchronize(ctx->copy_stream);
            for (cudaEvent_t e : ctx->copy_ev)
                if (e) cudaEventDestroy(e);
            cudaStreamDestroy(ctx->copy_stream);
        }
        if (ctx->own_stream) cudaStreamDestroy(ctx->own_stream);
        if (ctx->host_stage) cudaFreeHost(ctx->host_stage);
        if (ctx->out_stage) cudaFreeHost(ctx->out_stage);
        if (ctx->big_stage) cudaFreeHost(ctx->big_stage);
        delete ctx;
    });
}

int dt_ctx_set_stream(dt_ctx *ctx, void *stream) {
    return guard([&] {
        check_ctx(ctx);
        ctx->stream = stream ? static_cast<cudaStream_t>(stream) : ctx->own_stream;
    });
}

int dt_ctx_set_mem_limit(dt_ctx *ctx, uint64_t bytes) {
    return guard([&] {
        check_ctx(ctx);
        ctx->mem_limit = bytes;
    });
}

int dt_ctx_mem_usage(dt_ctx *ctx, uint64_t *in_use, uint64_t *peak) {
    return guard([&] {
        check_ctx(ctx);
        if (in_use) *in_use = ctx->mem_in_use;
        if (peak) *peak = ctx->mem_peak;
    });
}

int dt_ctx_synchronize(dt_ctx *ctx) {
    return guard([&] {
        check_ctx(ctx);
        DT_CUDA(cudaSetDevice(ctx->device));
        DT_CUDA(cudaStreamSynchronize(ctx->stream));
    });
}

int64_t dt_ctx_kernel_launches(dt_ctx *ctx) { return ctx ? ctx->launches : -1; }

}  // extern "C"
