// Plan compiler and executor behind the C ABI of include/msnh_b200.h.
//
// A plan is built once per (net, batch, dtype): shape inference -> fusion of conv + BatchNorm +
// activation + residual add into one tensor-core launch -> zero-copy placement of route/concat
// inputs as channel slices of the concat buffer -> liveness-based static arena -> weight folding
// and packing -> one list of kernel launches with resolved pointers and TMA tensor maps, captured
// as a CUDA graph. Running a plan is one H2D copy, one graph launch and (optionally) one sync.
// It stands in for NetBuilder's GPU loop and memory pools (src/net/MsnhNetBuilder.cpp:565-620,
// :820-1007 in the reference) and for the per-layer forwardGPU bodies.
#include "plan_internal.h"
#include <atomic>
#ifdef __SSE2__
#include <emmintrin.h>
#endif

using namespace msnh;

namespace msnh {

const char *const kLaunchNames[] = {"input_nchw_to_nhwc", "conv_umma", "conv_direct", "dwconv", "scale_bias_act",
                                    "add_n", "binary", "maxpool", "avgpool", "upsample", "slice", "pad", "softmax",
                                    "yolo_decode", "collect_zero", "yolo_collect", "input_nchw_to_patches",
                                    "yolo_decode_collect", "focus_slices", "bilinear", "deconv_col2im", "clip", "remap", "reduce", "prelu", "maxpool_depth", "conv_split", "input_nchw_to_row_patches"};

int fail(MsnhB200Ctx *ctx, int code, const char *fmt, ...) {
    char buf[1024];
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(buf, sizeof(buf), fmt, ap);
    va_end(ap);
    if (ctx) ctx->last_error = buf;
    return code;
}

int caught(MsnhB200Ctx *ctx) noexcept {
    int code = MSNH_B200_ERR_STATE;
    try {
        try { throw; }
        catch (const std::bad_alloc &) { code = MSNH_B200_ERR_NOMEM; return fail(ctx, code, "out of host memory"); }
        catch (const std::length_error &) { code = MSNH_B200_ERR_NOMEM; return fail(ctx, code, "out of host memory"); }
        catch (const std::exception &e) { return fail(ctx, code, "%s", e.what()); }
        catch (...) { return fail(ctx, code, "unknown exception"); }
    } catch (...) { return code; }                            // (no room for the text)
}

PlanDebugOptions PlanDebugOptions::from_env() {
    auto flag = [](const char *name) { const char *e = std::getenv(name); return e != nullptr; };
    auto num = [](const char *name, int unset) { const char *e = std::getenv(name); return e ? atoi(e) : unset; };
    PlanDebugOptions o;
    { const char *e = std::getenv("MSNH_B200_NO_PDL"); o.no_pdl = e && e[0] == '1'; }
    o.no_merge = flag("MSNH_B200_NO_MERGE");
    o.build_trace = flag("MSNH_B200_BUILD_TRACE");
    o.trace_tune = flag("MSNH_B200_TRACE_TUNE");
    o.dw_simple = flag("MSNH_B200_DW_SIMPLE");
    o.conv_simple = flag("MSNH_B200_CONV_SIMPLE");
    o.dw_th = num("MSNH_B200_DW_TH", 0);
    o.dw_stages = num("MSNH_B200_DW_STAGES", 0);
    o.autotune = num("MSNH_B200_AUTOTUNE", -1);
    o.trace_tile = num("MSNH_B200_TRACE_TILE", 0);
    o.forced_mm = num("MSNH_B200_M_MULT", 0);
    o.forced_bn = num("MSNH_B200_BN", 0);
    o.fp32_split = num("MSNH_B200_FP32_SPLIT", 0);
    o.conv_split = num("MSNH_B200_CONV_SPLIT", 0);
    o.k_split = num("MSNH_B200_K_SPLIT", 0);
    o.stream_k = num("MSNH_B200_STREAM_K", 0);
    o.pair = num("MSNH_B200_PAIR", 0);
    return o;
}
int check_device_flag(MsnhB200Ctx *ctx, volatile int *flag) {
    const int code = *flag;
    if (code != 0) {
        *flag = 0;
        return fail(ctx, MSNH_B200_ERR_DEVICE_TIMEOUT, "a bounded wait inside the conv kernel ran out (code %d)", code);
    }
    return MSNH_B200_OK;
}
int alloc_device_flag(MsnhB200Ctx *ctx, volatile int **flag, int **dev_flag) {
    void *host = nullptr, *dev = nullptr;
    CUDA_TRY(ctx, cudaHostAlloc(&host, sizeof(int), cudaHostAllocMapped));
    *flag = static_cast<volatile int *>(host);
    **flag = 0;
    CUDA_TRY(ctx, cudaHostGetDevicePointer(&dev, host, 0));
    *dev_flag = static_cast<int *>(dev);
    return MSNH_B200_OK;
}

bool is_pageable(const void *p) {
    cudaPointerAttributes a;
    if (cudaPointerGetAttributes(&a, p) != cudaSuccess) { cudaGetLastError(); return true; }
    return a.type == cudaMemoryTypeUnregistered;
}
// Copies of pageable memory from here on are the pool's. A synchronous call with an image of so many KB, its copy through the
// driver's own single-threaded staging / through the pool, in us:
//     KB                                        300      432      588      768      972     2028     3072     17328
//     image in the caller's cache            53 / 60  57 / 67  67 / 79  82 / 90  99 / 98  149 / 155  217 / 169  1275 / 485
//     image elsewhere in memory              67 / 57  78 / 64  95 / 72  120 / 78 142 / 87 243 / 129  340 / 165  1630 / 493
// The line lies between the two: what the pool loses to waking up in the one it more than wins in the other.
constexpr size_t kPoolBytes = 512 * 1024;
// What a thread copies and PCIe carries at a time: 5 us of PCIe, less where that would leave threads of the pool without a chunk
// (an image of 602 KB: a call of ResNet-18 343 -> 336 us, of MobileNetV2 296 -> 290)
constexpr size_t kCopyChunk = 256 * 1024, kMinChunk = 64 * 1024;
constexpr int kMinWorkers = 3;              // with fewer threads beside the caller the driver's staging is as fast
// Hands a cache line this core is done with down to the cache all cores share (a hint; processors without it ignore it).
static inline void demote_line(const void *p) {
#ifdef __SSE2__
    asm volatile("cldemote %0" ::"m"(*static_cast<const char *>(p)));
#else
    (void)p;
#endif
}
// memcpy for a pool thread that fills staging (dst 16-byte aligned). It writes past the caches: staging filled through the caches
// of eight cores leaves the device to fetch every line from one of them (19 MB took 1.7 ms to arrive that way, 1.0 ms through
// the driver's staging, 0.49 ms like this). And it hands the caller's lines back: left in eight cores' caches they made the
// caller's next write of those 19 MB take 2.8 ms instead of 1.1.
static void copy_past_caches(uint8_t *dst, const uint8_t *src, size_t n) {
#ifdef __SSE2__
    size_t i = 0;
    for (; i + 64 <= n; i += 64) {
        const __m128i a = _mm_loadu_si128(reinterpret_cast<const __m128i *>(src + i)), b = _mm_loadu_si128(reinterpret_cast<const __m128i *>(src + i + 16));
        const __m128i c = _mm_loadu_si128(reinterpret_cast<const __m128i *>(src + i + 32)), d = _mm_loadu_si128(reinterpret_cast<const __m128i *>(src + i + 48));
        demote_line(src + i);
        _mm_stream_si128(reinterpret_cast<__m128i *>(dst + i), a); _mm_stream_si128(reinterpret_cast<__m128i *>(dst + i + 16), b);
        _mm_stream_si128(reinterpret_cast<__m128i *>(dst + i + 32), c); _mm_stream_si128(reinterpret_cast<__m128i *>(dst + i + 48), d);
    }
    std::memcpy(dst + i, src + i, n - i);
    _mm_sfence();
#else
    std::memcpy(dst, src, n);
#endif
}
static HostPool &pool_of(MsnhB200Ctx *ctx) {
    if (!ctx->pool) ctx->pool.reset(new HostPool(HostPool::default_workers()));
    return *ctx->pool;
}
static int pinned_staging(MsnhB200Plan *pl, size_t bytes) {
    if (pl->staging_busy) CUDA_TRY(pl->ctx, cudaEventSynchronize(pl->ev_copy));       // the copy before has left it
    pl->staging_busy = false;
    if (pl->h_pinned_bytes >= bytes) return MSNH_B200_OK;
    if (pl->h_pinned) cudaFreeHost(pl->h_pinned);
    pl->h_pinned = nullptr; pl->h_pinned_bytes = 0;
    CUDA_TRY(pl->ctx, cudaMallocHost(reinterpret_cast<void **>(&pl->h_pinned), bytes));
    pl->h_pinned_bytes = bytes;
    return MSNH_B200_OK;
}
void parallel_memcpy(MsnhB200Ctx *ctx, void *dst, const void *src, size_t bytes) {
    if (bytes < kPoolBytes) { std::memcpy(dst, src, bytes); return; }
    pool_of(ctx).run(static_cast<int>((bytes + kCopyChunk - 1) / kCopyChunk), [=](int i) {
        const size_t at = i * kCopyChunk, n = std::min(kCopyChunk, bytes - at);
        uint8_t *to = static_cast<uint8_t *>(dst) + at;
        std::memcpy(to, static_cast<const uint8_t *>(src) + at, n);
        for (size_t k = 0; k < n; k += 64) demote_line(to + k);        // the caller reads it next
    });
}
int copy_in(MsnhB200Plan *pl, void *dev, const void *host, size_t bytes) {
    MsnhB200Ctx *ctx = pl->ctx;
    if (bytes < kPoolBytes || !is_pageable(host) || HostPool::default_workers() < kMinWorkers || pool_of(ctx).workers() < kMinWorkers) {
        CUDA_TRY(ctx, cudaMemcpyAsync(dev, host, bytes, cudaMemcpyHostToDevice, ctx->stream));
        return MSNH_B200_OK;
    }
    const size_t chunk = std::min(kCopyChunk, std::max(kMinChunk, (bytes / 8 + 4095) / 4096 * 4096));
    const int n = static_cast<int>((bytes + chunk - 1) / chunk), part = static_cast<int>(kStagingBytes / kStagingParts / chunk), ring = kStagingParts * part;
    { const int rc = pinned_staging(pl, std::min(n, ring) * chunk); if (rc) return rc; }
    HostPool &pool = pool_of(ctx);
    uint8_t *pinned = pl->h_pinned;
    std::atomic<int> open{ring};                 // chunks before this one may be written: what lay in their place has been sent
    pool.begin(n, [=, &open](int i) {
        for (int spins = 0; open.load(std::memory_order_acquire) <= i; ++spins) {
            if (spins < 200) std::this_thread::yield();
            else std::this_thread::sleep_for(std::chrono::microseconds(20));           // (the stream is busy with something long)
        }
        const size_t at = i * chunk;
        copy_past_caches(pinned + static_cast<size_t>(i % ring) * chunk, static_cast<const uint8_t *>(host) + at, std::min(chunk, bytes - at));
    });
    // send what is ready, in order and up to the ring's end; copy along while the next chunk is not
    cudaError_t e = cudaSuccess;
    int parts_sent = 0, parts_left = 0;          // parts of the ring behind which an event is queued, and those whose event has come
    for (int sent = 0; sent < n && e == cudaSuccess;) {
        const int writable = open.load(std::memory_order_relaxed);
        if (parts_left < parts_sent && pool.all_started(writable)) {
            const cudaEvent_t ev = pl->ev_part[parts_left % kStagingParts];
            e = sent < writable ? cudaEventQuery(ev) : cudaEventSynchronize(ev);
            if (e == cudaSuccess) open.store(ring + ++parts_left * part, std::memory_order_release);
            else if (e == cudaErrorNotReady) e = cudaSuccess;
        }
        int ready = sent;
        while (ready < n && pool.done(ready) && (ready == sent || ready % ring)) ++ready;
        if (ready == sent) { if (!pool.help(writable)) std::this_thread::yield(); continue; }
        const size_t at = sent * chunk, end = std::min(ready * chunk, bytes);
        e = cudaMemcpyAsync(static_cast<uint8_t *>(dev) + at, pinned + static_cast<size_t>(sent % ring) * chunk, end - at, cudaMemcpyHostToDevice, ctx->stream);
        sent = ready;
        for (; n > ring && e == cudaSuccess && (parts_sent + 1) * part <= sent; ++parts_sent) e = cudaEventRecord(pl->ev_part[parts_sent % kStagingParts], ctx->stream);
    }
    open.store(n, std::memory_order_release);
    pool.finish();
    CUDA_TRY(ctx, e);
    CUDA_TRY(ctx, cudaEventRecord(pl->ev_copy, ctx->stream));
    pl->staging_busy = true;
    return MSNH_B200_OK;
}
int copy_out(MsnhB200Plan *pl, void *host, const void *dev, size_t bytes) {
    MsnhB200Ctx *ctx = pl->ctx;
    if (bytes < kPoolBytes || !is_pageable(host) || HostPool::default_workers() < kMinWorkers || pool_of(ctx).workers() < kMinWorkers) {
        CUDA_TRY(ctx, cudaMemcpyAsync(host, dev, bytes, cudaMemcpyDeviceToHost, ctx->stream));
        CUDA_TRY(ctx, cudaStreamSynchronize(ctx->stream));
        return MSNH_B200_OK;
    }
    // in pieces of half the staging at most, so that one crosses PCIe while the one before it is copied on
    const size_t piece = std::min(kStagingBytes / 2, (bytes / 2 + kCopyChunk - 1) / kCopyChunk * kCopyChunk);
    const int n = static_cast<int>((bytes + piece - 1) / piece);
    { const int rc = pinned_staging(pl, std::min(bytes, 2 * piece)); if (rc) return rc; }
    auto fetch = [&](int k) -> cudaError_t {
        const size_t at = k * piece;
        const cudaError_t e = cudaMemcpyAsync(pl->h_pinned + (k & 1) * piece, static_cast<const uint8_t *>(dev) + at, std::min(piece, bytes - at), cudaMemcpyDeviceToHost, ctx->stream);
        return e == cudaSuccess ? cudaEventRecord(pl->ev_part[k & 1], ctx->stream) : e;
    };
    for (int k = 0; k < n && k < 2; ++k) CUDA_TRY(ctx, fetch(k));
    for (int k = 0; k < n; ++k) {
        const size_t at = k * piece;
        CUDA_TRY(ctx, cudaEventSynchronize(pl->ev_part[k & 1]));
        parallel_memcpy(ctx, static_cast<uint8_t *>(host) + at, pl->h_pinned + (k & 1) * piece, std::min(piece, bytes - at));
        if (k + 2 < n) CUDA_TRY(ctx, fetch(k + 2));
    }
    return MSNH_B200_OK;
}

}  // namespace msnh

// ------------------------------------------------------------------------------------------------
// C ABI
// ------------------------------------------------------------------------------------------------
extern "C" {

int msnh_b200_device_count(int *count) {
    if (!count) return MSNH_B200_ERR_ARG;
    int n = 0;
    if (cudaGetDeviceCount(&n) != cudaSuccess) { *count = 0; cudaGetLastError(); return MSNH_B200_ERR_CUDA; }
    *count = n;
    return MSNH_B200_OK;
}

int msnh_b200_ctx_create(int device, MsnhB200Ctx **out) try {
    if (!out) return MSNH_B200_ERR_ARG;
    *out = nullptr;
    int n = 0;
    if (cudaGetDeviceCount(&n) != cudaSuccess || device < 0 || device >= n) { cudaGetLastError(); return MSNH_B200_ERR_CUDA; }
    MsnhB200Ctx *ctx = new MsnhB200Ctx();
    ctx->device = device;
    cudaDeviceProp prop;
    if (cudaSetDevice(device) != cudaSuccess || cudaGetDeviceProperties(&prop, device) != cudaSuccess) { delete ctx; return MSNH_B200_ERR_CUDA; }
    if (prop.major != 10) { delete ctx; return MSNH_B200_ERR_UNSUPPORTED; }   // sm_100a code only
    ctx->sm_count = prop.multiProcessorCount;
    ctx->pdl = !PlanDebugOptions::from_env().no_pdl;
    cudaDriverGetVersion(&ctx->driver_version);
    if (cudaStreamCreateWithFlags(&ctx->stream, cudaStreamNonBlocking) != cudaSuccess) { delete ctx; return MSNH_B200_ERR_CUDA; }
    cudaDriverEntryPointQueryResult q;
    void *fn = nullptr;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &q) != cudaSuccess || !fn) { delete ctx; return MSNH_B200_ERR_CUDA; }
    ctx->encode_tiled = reinterpret_cast<EncodeTiledFn>(fn);
    fn = nullptr;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeIm2col", &fn, cudaEnableDefault, &q) != cudaSuccess || !fn) { delete ctx; return MSNH_B200_ERR_CUDA; }
    ctx->encode_im2col = reinterpret_cast<EncodeIm2colFn>(fn);
    if (alloc_device_flag(ctx, &ctx->err_flag, &ctx->dev_err_flag) != MSNH_B200_OK) {
        const bool got = ctx->err_flag != nullptr;
        if (got) cudaFreeHost(const_cast<int *>(ctx->err_flag));
        delete ctx;
        return got ? MSNH_B200_ERR_CUDA : MSNH_B200_ERR_NOMEM;
    }
    *out = ctx;
    return MSNH_B200_OK;
} catch (...) { return caught(nullptr); }

int msnh_b200_ctx_destroy(MsnhB200Ctx *ctx) {
    if (!ctx) return MSNH_B200_ERR_ARG;
    cudaSetDevice(ctx->device);
    if (ctx->flush_buf) cudaFree(ctx->flush_buf);
    if (ctx->err_flag) cudaFreeHost(const_cast<int *>(ctx->err_flag));
    if (ctx->stream) cudaStreamDestroy(ctx->stream);
    delete ctx;
    return MSNH_B200_OK;
}

const char *msnh_b200_last_error(MsnhB200Ctx *ctx) { return ctx ? ctx->last_error.c_str() : "null context"; }

int msnh_b200_host_alloc(MsnhB200Ctx *ctx, size_t bytes, void **ptr) try {
    if (!ctx || !ptr) return MSNH_B200_ERR_ARG;
    CUDA_TRY(ctx, cudaSetDevice(ctx->device));
    CUDA_TRY(ctx, cudaMallocHost(ptr, bytes));
    return MSNH_B200_OK;
} catch (...) { return caught(ctx); }
int msnh_b200_host_free(MsnhB200Ctx *ctx, void *ptr) try {
    if (!ctx) return MSNH_B200_ERR_ARG;
    CUDA_TRY(ctx, cudaFreeHost(ptr));
    return MSNH_B200_OK;
} catch (...) { return caught(ctx); }

int msnh_b200_plan_create(MsnhB200Ctx *ctx, const MsnhB200Op *ops, int n_ops, int in_c, int in_h, int in_w, int batch,
                          int dtype, uint32_t flags, MsnhB200Plan **out) try {
    if (!ctx || !ops || !out || n_ops <= 0) return fail(ctx, MSNH_B200_ERR_ARG, "plan_create: null or empty argument");
    *out = nullptr;
    if (in_c <= 0 || in_h <= 0 || in_w <= 0 || batch <= 0) return fail(ctx, MSNH_B200_ERR_ARG, "plan_create: bad input shape %dx%dx%d batch %d", in_c, in_h, in_w, batch);
    if (dtype != MSNH_B200_F32 && dtype != MSNH_B200_F16) return fail(ctx, MSNH_B200_ERR_ARG, "plan_create: dtype %d", dtype);
    std::unique_ptr<MsnhB200Plan> pl(new MsnhB200Plan());
    pl->ctx = ctx; pl->in_c = in_c; pl->in_h = in_h; pl->in_w = in_w; pl->batch = batch; pl->dtype = dtype; pl->flags = flags;
    pl->ops.resize(n_ops);
    for (int i = 0; i < n_ops; ++i) {
        pl->ops[i].d = ops[i];
        std::string err;
        int rc = infer_shape(pl.get(), i, err);
        if (rc) return fail(ctx, rc, "op %d (kind %d): %s", i, ops[i].kind, err.c_str());
        if (ops[i].act < 0 || ops[i].act >= MSNH_ACT_COUNT) return fail(ctx, MSNH_B200_ERR_UNSUPPORTED, "op %d: activation %d not supported", i, ops[i].act);
    }
    // fp32 detection nets: fp32 arithmetic throughout unless tf32 is asked for (see MSNH_PLAN_TF32_DETECT), convs on split operands
    if (dtype == MSNH_B200_F32 && !(flags & MSNH_PLAN_TF32_DETECT))
        for (int i = 0; i < n_ops; ++i) if (ops[i].kind == MSNH_OP_YOLO) { pl->split_fp32 = !(flags & MSNH_PLAN_NO_TENSOR_CORE); pl->flags |= MSNH_PLAN_NO_TENSOR_CORE; break; }
    *out = pl.release();
    return MSNH_B200_OK;
} catch (...) { return caught(ctx); }

int msnh_b200_plan_op_shape(MsnhB200Plan *pl, int op, int *c, int *h, int *w) {
    if (!pl || op < 0 || op >= static_cast<int>(pl->ops.size())) return MSNH_B200_ERR_ARG;
    if (c) *c = pl->ops[op].out.C; if (h) *h = pl->ops[op].out.H; if (w) *w = pl->ops[op].out.W;
    return MSNH_B200_OK;
}

int msnh_b200_plan_weight_count(MsnhB200Plan *pl, int op, int slot, size_t *count) {
    if (!pl || !count || op < 0 || op >= static_cast<int>(pl->ops.size()) || slot < 0 || slot >= MSNH_W_SLOTS) return MSNH_B200_ERR_ARG;
    *count = pl->ops[op].wcount[slot];
    return MSNH_B200_OK;
}

int msnh_b200_plan_set_weights(MsnhB200Plan *pl, int op, int slot, const float *data, size_t count) try {
    if (!pl) return MSNH_B200_ERR_ARG;
    if (pl->finalized) return fail(pl->ctx, MSNH_B200_ERR_STATE, "set_weights after finalize");
    if (!data || op < 0 || op >= static_cast<int>(pl->ops.size()) || slot < 0 || slot >= MSNH_W_SLOTS) return fail(pl->ctx, MSNH_B200_ERR_ARG, "set_weights: bad argument");
    if (count != pl->ops[op].wcount[slot]) return fail(pl->ctx, MSNH_B200_ERR_ARG, "set_weights: op %d slot %d expects %zu floats, got %zu", op, slot, pl->ops[op].wcount[slot], count);
    pl->ops[op].w[slot].assign(data, data + count);
    return MSNH_B200_OK;
} catch (...) { return caught(pl ? pl->ctx : nullptr); }

// The debug switches as they stand now. MSNH_B200_CONV_SPLIT takes any fp32 plan that may use the tensor cores to the split-operand convs.
static void read_debug_options(MsnhB200Plan *pl) {
    pl->dbg = PlanDebugOptions::from_env();
    if (pl->dbg.conv_split && pl->dtype == MSNH_B200_F32 && !(pl->flags & MSNH_PLAN_NO_TENSOR_CORE)) { pl->split_fp32 = true; pl->flags |= MSNH_PLAN_NO_TENSOR_CORE; }
}

int msnh_b200_plan_use_pack(MsnhB200Plan *pl, const char *path, uint64_t weights_tag, int *usable) try {
    if (!pl || !path || !*path) return MSNH_B200_ERR_ARG;
    if (pl->finalized) return fail(pl->ctx, MSNH_B200_ERR_STATE, "use_pack after finalize");
    pl->pack_path = path; pl->pack_tag = weights_tag;
    read_debug_options(pl);
    if (usable) *usable = pack_probe(pl) ? 1 : 0;
    return MSNH_B200_OK;
} catch (...) { return caught(pl ? pl->ctx : nullptr); }

// The result a synchronous run brings back with it: that of the plan's only output op, when it is a candidate list or small.
static int early_result_setup(MsnhB200Plan *pl) {
    int op = -1, outputs = 0;
    for (size_t i = 0; i < pl->ops.size(); ++i)
        if (pl->ops[i].d.is_output) { op = static_cast<int>(i); ++outputs; }
    if (outputs != 1 || (pl->flags & MSNH_PLAN_KEEP_ALL)) return MSNH_B200_OK;
    const OpState &o = pl->ops[op];
    size_t floats;
    if (o.d.kind == MSNH_OP_YOLO_COLLECT) {
        bool found = false;
        for (const Launch &L : pl->launches) found = found || (L.kind == L_COLLECT_ZERO && L.op == op);
        if (!found) return MSNH_B200_OK;
        floats = static_cast<size_t>(pl->batch) * kEarlyRows * 8;
        CUDA_TRY(pl->ctx, cudaMallocHost(reinterpret_cast<void **>(&pl->h_early_counts), sizeof(int) * pl->batch));
    } else {
        floats = static_cast<size_t>(pl->batch) * o.out.C * o.out.H * o.out.W;
        if (floats * sizeof(float) > kEarlyOutputBytes) return MSNH_B200_OK;
    }
    CUDA_TRY(pl->ctx, cudaMallocHost(reinterpret_cast<void **>(&pl->h_early), floats * sizeof(float)));
    pl->early_op = op;
    return MSNH_B200_OK;
}

int msnh_b200_plan_finalize(MsnhB200Plan *pl) try {
    if (!pl) return MSNH_B200_ERR_ARG;
    MsnhB200Ctx *ctx = pl->ctx;
    if (pl->finalized) return fail(ctx, MSNH_B200_ERR_STATE, "finalize called twice");
    if (pl->finalize_failed) return fail(ctx, MSNH_B200_ERR_STATE, "an earlier finalize of this plan failed: destroy it and build a new one");
    CUDA_TRY(ctx, cudaSetDevice(ctx->device));
    read_debug_options(pl);
    int rc = build_launches(pl);
    if (rc) {
        // weights that were merely missing can still be set; anything later leaves half-built state behind
        bool missing_weights = rc == MSNH_B200_ERR_STATE && pl->launches.empty() && pl->tensors.empty();
        if (!missing_weights) pl->finalize_failed = true;
        for (OpState &o : pl->ops) o.consumers.clear();
        return rc;
    }
    CUDA_TRY(ctx, cudaEventCreate(&pl->ev0));
    CUDA_TRY(ctx, cudaEventCreate(&pl->ev1));
    CUDA_TRY(ctx, cudaEventCreateWithFlags(&pl->ev_copy, cudaEventDisableTiming));
    for (cudaEvent_t &e : pl->ev_part) CUDA_TRY(ctx, cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
    { const int rc2 = early_result_setup(pl); if (rc2) return rc2; }
    for (OpState &o : pl->ops) for (int s = 0; s < MSNH_W_SLOTS; ++s) { std::vector<float>().swap(o.w[s]); }
    if (!(pl->flags & MSNH_PLAN_NO_GRAPH)) {
        CUDA_TRY(ctx, cudaStreamBeginCapture(ctx->stream, cudaStreamCaptureModeThreadLocal));
        for (const Launch &L : pl->launches) launch_one(ctx, L, ctx->stream);
        cudaError_t e = cudaStreamEndCapture(ctx->stream, &pl->graph);
        if (e != cudaSuccess) return fail(ctx, MSNH_B200_ERR_CUDA, "graph capture failed: %s", cudaGetErrorString(e));
        CUDA_TRY(ctx, cudaGraphInstantiate(&pl->graph_exec, pl->graph, 0));
    }
    CUDA_TRY(ctx, cudaGetLastError());
    pl->finalized = true;
    return MSNH_B200_OK;
} catch (...) {
    if (pl && !pl->finalized) pl->finalize_failed = true;
    return caught(pl ? pl->ctx : nullptr);
}

int msnh_b200_plan_input_buffer(MsnhB200Plan *pl, float **dev_ptr) try {
    if (!pl || !dev_ptr) return MSNH_B200_ERR_ARG;
    if (!pl->finalized) return fail(pl->ctx, MSNH_B200_ERR_STATE, "plan not finalized");
    *dev_ptr = pl->d_input;
    return MSNH_B200_OK;
} catch (...) { return caught(pl ? pl->ctx : nullptr); }

static const Launch *collect_launch(const MsnhB200Plan *pl, int op) {
    for (const Launch &L : pl->launches) if (L.kind == L_COLLECT_ZERO && L.op == op) return &L;
    return nullptr;
}

static int run_common(MsnhB200Plan *pl, int n_images, int sync) {
    MsnhB200Ctx *ctx = pl->ctx;
    pl->early_valid = false;
    CUDA_TRY(ctx, cudaEventRecord(pl->ev0, ctx->stream));
    if (pl->graph_exec) CUDA_TRY(ctx, cudaGraphLaunch(pl->graph_exec, ctx->stream));
    else for (const Launch &L : pl->launches) launch_one(ctx, L, ctx->stream);
    CUDA_TRY(ctx, cudaEventRecord(pl->ev1, ctx->stream));
    pl->timed_steps = 1;
    if (sync) {
        if (pl->early_op >= 0) {
            const OpState &o = pl->ops[pl->early_op];
            if (o.d.kind == MSNH_OP_YOLO_COLLECT) {
                const Launch *zl = collect_launch(pl, pl->early_op);
                launch_candidates_to_host(zl->rows, zl->max_rows, zl->counts, pl->h_early, kEarlyRows, pl->h_early_counts, n_images, ctx->stream);
            } else {
                TView v = view_of(pl, o.tensor);
                v.N = n_images;
                launch_readback(ctx, pl->tensors[o.tensor].dtype, v, pl->h_early, static_cast<size_t>(n_images) * o.out.C * o.out.H * o.out.W, ctx->stream);
            }
            CUDA_TRY(ctx, cudaGetLastError());
        }
        CUDA_TRY(ctx, cudaStreamSynchronize(ctx->stream));
        const int rc = check_device_flag(pl);
        if (rc) return rc;
        pl->early_valid = pl->early_op >= 0; pl->early_images = n_images;
    }
    return MSNH_B200_OK;
}

int msnh_b200_plan_run(MsnhB200Plan *pl, const float *host_nchw, int n_images) try {
    if (!pl || !host_nchw) return MSNH_B200_ERR_ARG;
    MsnhB200Ctx *ctx = pl->ctx;
    if (!pl->finalized) return fail(ctx, MSNH_B200_ERR_STATE, "plan not finalized");
    if (n_images < 1 || n_images > pl->batch) return fail(ctx, MSNH_B200_ERR_ARG, "n_images %d outside 1..%d", n_images, pl->batch);
    CUDA_TRY(ctx, cudaSetDevice(ctx->device));
    const size_t bytes = static_cast<size_t>(n_images) * pl->in_c * pl->in_h * pl->in_w * sizeof(float);
    { const int rc = copy_in(pl, pl->d_input, host_nchw, bytes); if (rc) return rc; }
    return run_common(pl, n_images, 1);
} catch (...) { return caught(pl ? pl->ctx : nullptr); }

int msnh_b200_plan_run_device(MsnhB200Plan *pl, const float *dev_nchw, int n_images, int sync) try {
    if (!pl) return MSNH_B200_ERR_ARG;
    MsnhB200Ctx *ctx = pl->ctx;
    if (!pl->finalized) return fail(ctx, MSNH_B200_ERR_STATE, "plan not finalized");
    if (n_images < 1 || n_images > pl->batch) return fail(ctx, MSNH_B200_ERR_ARG, "n_images %d outside 1..%d", n_images, pl->batch);
    CUDA_TRY(ctx, cudaSetDevice(ctx->device));
    if (dev_nchw && dev_nchw != pl->d_input) {
        const size_t bytes = static_cast<size_t>(n_images) * pl->in_c * pl->in_h * pl->in_w * sizeof(float);
        CUDA_TRY(ctx, cudaMemcpyAsync(pl->d_input, dev_nchw, bytes, cudaMemcpyDeviceToDevice, ctx->stream));
    }
    return run_common(pl, n_images, sync);
} catch (...) { return caught(pl ? pl->ctx : nullptr); }

int msnh_b200_plan_run_timed(MsnhB200Plan *pl, int n_images, int steps, float *total_ms) try {
    if (!pl || !total_ms || steps < 1) return MSNH_B200_ERR_ARG;
    MsnhB200Ctx *ctx = pl->ctx;
    if (!pl->finalized) return fail(ctx, MSNH_B200_ERR_STATE, "plan not finalized");
    if (n_images < 1 || n_images > pl->batch) return fail(ctx, MSNH_B200_ERR_ARG, "n_images %d outside 1..%d", n_images, pl->batch);
    CUDA_TRY(ctx, cudaSetDevice(ctx->device));
    CUDA_TRY(ctx, cudaStreamSynchronize(ctx->stream));
    pl->early_valid = false;
    CUDA_TRY(ctx, cudaEventRecord(pl->ev0, ctx->stream));
    for (int s = 0; s < steps; ++s) {
        if (pl->graph_exec) CUDA_TRY(ctx, cudaGraphLaunch(pl->graph_exec, ctx->stream));
        else for (const Launch &L : pl->launches) launch_one(ctx, L, ctx->stream);
    }
    CUDA_TRY(ctx, cudaEventRecord(pl->ev1, ctx->stream));
    CUDA_TRY(ctx, cudaStreamSynchronize(ctx->stream));
    CUDA_TRY(ctx, cudaEventElapsedTime(total_ms, pl->ev0, pl->ev1));
    pl->timed_steps = steps;
    return check_device_flag(pl);
} catch (...) { return caught(pl ? pl->ctx : nullptr); }

int msnh_b200_plan_run_instrumented(MsnhB200Plan *pl, int n_images, int steps, float *ms, int capacity) try {
    if (!pl || !ms || steps < 1) return MSNH_B200_ERR_ARG;
    MsnhB200Ctx *ctx = pl->ctx;
    if (!pl->finalized) return fail(ctx, MSNH_B200_ERR_STATE, "plan not finalized");
    const int n = static_cast<int>(pl->launches.size());
    if (capacity < n) return fail(ctx, MSNH_B200_ERR_ARG, "run_instrumented: capacity %d < %d launches", capacity, n);
    CUDA_TRY(ctx, cudaSetDevice(ctx->device));
    pl->early_valid = false;
    std::vector<cudaEvent_t> ev(static_cast<size_t>(n) + 1);
    for (auto &e : ev) CUDA_TRY(ctx, cudaEventCreate(&e));
    for (int k = 0; k < n; ++k) ms[k] = 0.f;
    for (int s = 0; s < steps; ++s) {
        CUDA_TRY(ctx, cudaEventRecord(ev[0], ctx->stream));
        for (int k = 0; k < n; ++k) {
            launch_one(ctx, pl->launches[k], ctx->stream);
            CUDA_TRY(ctx, cudaEventRecord(ev[k + 1], ctx->stream));
        }
        CUDA_TRY(ctx, cudaStreamSynchronize(ctx->stream));
        for (int k = 0; k < n; ++k) {
            float t = 0.f;
            CUDA_TRY(ctx, cudaEventElapsedTime(&t, ev[k], ev[k + 1]));
            ms[k] += t;
        }
    }
    for (int k = 0; k < n; ++k) ms[k] /= steps;
    for (auto &e : ev) cudaEventDestroy(e);
    (void)n_images;
    return check_device_flag(pl);
} catch (...) { return caught(pl ? pl->ctx : nullptr); }

int msnh_b200_plan_read_output(MsnhB200Plan *pl, int op, float *host, size_t count) try {
    if (!pl || !host) return MSNH_B200_ERR_ARG;
    MsnhB200Ctx *ctx = pl->ctx;
    if (!pl->finalized) return fail(ctx, MSNH_B200_ERR_STATE, "plan not finalized");
    if (op < 0 || op >= static_cast<int>(pl->ops.size())) return fail(ctx, MSNH_B200_ERR_ARG, "read_output: op %d", op);
    const OpState &o = pl->ops[op];
    if (!(o.d.is_output || (pl->flags & MSNH_PLAN_KEEP_ALL))) return fail(ctx, MSNH_B200_ERR_STATE, "op %d is not an output of this plan", op);
    if (o.d.kind == MSNH_OP_YOLO_COLLECT) return fail(ctx, MSNH_B200_ERR_ARG, "use plan_read_candidates for op %d", op);
    const size_t per = static_cast<size_t>(o.out.C) * o.out.H * o.out.W;
    if (count == 0 || count % per || count / per > static_cast<size_t>(pl->batch)) return fail(ctx, MSNH_B200_ERR_ARG, "read_output: count %zu is not 1..%d images of %zu", count, pl->batch, per);
    if (op == pl->early_op && pl->early_valid && count / per <= static_cast<size_t>(pl->early_images)) {     // came back with the run
        std::memcpy(host, pl->h_early, count * sizeof(float));
        return MSNH_B200_OK;
    }
    CUDA_TRY(ctx, cudaSetDevice(ctx->device));
    if (pl->readback_elems < count) {
        if (pl->d_readback) cudaFree(pl->d_readback);
        pl->d_readback = nullptr; pl->readback_elems = 0;
        CUDA_TRY(ctx, cudaMalloc(reinterpret_cast<void **>(&pl->d_readback), count * sizeof(float)));
        pl->readback_elems = count;
    }
    TView v = view_of(pl, o.tensor);
    v.N = static_cast<int>(count / per);
    const int dt = pl->tensors[o.tensor].dtype;
    launch_readback(ctx, dt, v, pl->d_readback, count, ctx->stream);
    return copy_out(pl, host, pl->d_readback, count * sizeof(float));
} catch (...) { return caught(pl ? pl->ctx : nullptr); }

int msnh_b200_plan_read_candidates(MsnhB200Plan *pl, int op, int n_images, float *rows, int max_rows, int *counts) try {
    if (!pl || !rows || !counts) return MSNH_B200_ERR_ARG;
    MsnhB200Ctx *ctx = pl->ctx;
    if (!pl->finalized) return fail(ctx, MSNH_B200_ERR_STATE, "plan not finalized");
    if (op < 0 || op >= static_cast<int>(pl->ops.size()) || pl->ops[op].d.kind != MSNH_OP_YOLO_COLLECT) return fail(ctx, MSNH_B200_ERR_ARG, "op %d is not a yolo collect op", op);
    if (n_images < 1 || n_images > pl->batch || max_rows < 1) return fail(ctx, MSNH_B200_ERR_ARG, "read_candidates: bad n_images / max_rows");
    const Launch *zl = collect_launch(pl, op);
    if (!zl) return fail(ctx, MSNH_B200_ERR_STATE, "collect launch missing");
    bool early = op == pl->early_op && pl->early_valid && n_images <= pl->early_images;        // they came back with the run, all of them
    for (int i = 0; early && i < n_images; ++i) early = std::min(pl->h_early_counts[i], zl->max_rows) <= kEarlyRows;
    if (early) {
        for (int i = 0; i < n_images; ++i) {
            counts[i] = std::min(pl->h_early_counts[i], std::min(zl->max_rows, max_rows));
            // rows in excess of the caller's buffer: the first ones in scan order would be as arbitrary as the first that were appended
            std::memcpy(rows + static_cast<size_t>(i) * max_rows * 8, pl->h_early + static_cast<size_t>(i) * kEarlyRows * 8, sizeof(float) * 8 * counts[i]);
        }
    } else {
        CUDA_TRY(ctx, cudaSetDevice(ctx->device));
        CUDA_TRY(ctx, cudaMemcpyAsync(pl->h_counts, zl->counts, sizeof(int) * n_images, cudaMemcpyDeviceToHost, ctx->stream));
        CUDA_TRY(ctx, cudaStreamSynchronize(ctx->stream));
        for (int i = 0; i < n_images; ++i) {
            int c = std::min(pl->h_counts[i], std::min(zl->max_rows, max_rows));
            counts[i] = c;
            if (c > 0)
                CUDA_TRY(ctx, cudaMemcpyAsync(rows + static_cast<size_t>(i) * max_rows * 8, zl->rows + static_cast<size_t>(i) * zl->max_rows * 8,
                                              sizeof(float) * 8 * c, cudaMemcpyDeviceToHost, ctx->stream));
        }
        CUDA_TRY(ctx, cudaStreamSynchronize(ctx->stream));
    }
    // restore the reference's scan order (the device appends in arbitrary order)
    struct Row { float v[8]; };
    for (int i = 0; i < n_images; ++i) {
        Row *r = reinterpret_cast<Row *>(rows + static_cast<size_t>(i) * max_rows * 8);
        std::sort(r, r + counts[i], [](const Row &a, const Row &b) { return a.v[7] < b.v[7]; });
    }
    return MSNH_B200_OK;
} catch (...) { return caught(pl ? pl->ctx : nullptr); }


int msnh_b200_plan_last_ms(MsnhB200Plan *pl, float *ms) {
    if (!pl || !ms) return MSNH_B200_ERR_ARG;
    // the events of the last run are looked at when somebody asks (a run that nobody has waited for yet keeps the figure before it)
    float t = 0.f;
    if (pl->timed_steps > 0 && cudaEventElapsedTime(&t, pl->ev0, pl->ev1) == cudaSuccess) { pl->last_ms = t / pl->timed_steps; pl->timed_steps = 0; }
    else cudaGetLastError();
    *ms = pl->last_ms;
    return MSNH_B200_OK;
}

int msnh_b200_plan_stats(MsnhB200Plan *pl, int *launches, size_t *arena_bytes) {
    if (!pl) return MSNH_B200_ERR_ARG;
    if (launches) *launches = static_cast<int>(pl->launches.size());
    if (arena_bytes) *arena_bytes = pl->arena_bytes;
    return MSNH_B200_OK;
}

const char *msnh_b200_plan_describe(MsnhB200Plan *pl) { return pl ? pl->description.c_str() : ""; }

int msnh_b200_plan_profile(MsnhB200Plan *pl, int iters, float *ms, int capacity) try {
    if (!pl || !ms || iters < 1) return MSNH_B200_ERR_ARG;
    MsnhB200Ctx *ctx = pl->ctx;
    if (!pl->finalized) return fail(ctx, MSNH_B200_ERR_STATE, "plan not finalized");
    const int n = static_cast<int>(pl->launches.size());
    if (capacity < n) return fail(ctx, MSNH_B200_ERR_ARG, "profile: capacity %d < %d launches", capacity, n);
    CUDA_TRY(ctx, cudaSetDevice(ctx->device));
    { float settled; msnh_b200_plan_last_ms(pl, &settled); pl->timed_steps = 0; }     // (the events below are those of the last run)
    pl->early_valid = false;
    if (!ctx->flush_buf) {
        ctx->flush_elems = static_cast<size_t>(256) * 1024 * 1024 / sizeof(float);   // 256 MiB > 126 MB L2
        CUDA_TRY(ctx, cudaMalloc(reinterpret_cast<void **>(&ctx->flush_buf), ctx->flush_elems * sizeof(float)));
    }
    // one full forward first so every launch sees real inputs
    for (const Launch &L : pl->launches) launch_one(ctx, L, ctx->stream);
    CUDA_TRY(ctx, cudaStreamSynchronize(ctx->stream));
    for (int k = 0; k < n; ++k) {
        float total = 0.f;
        for (int it = 0; it < iters; ++it) {
            launch_fill(ctx, ctx->flush_buf, ctx->flush_elems, 0.f, ctx->stream);
            CUDA_TRY(ctx, cudaEventRecord(pl->ev0, ctx->stream));
            launch_one(ctx, pl->launches[k], ctx->stream);
            CUDA_TRY(ctx, cudaEventRecord(pl->ev1, ctx->stream));
            CUDA_TRY(ctx, cudaStreamSynchronize(ctx->stream));
            float t = 0.f;
            CUDA_TRY(ctx, cudaEventElapsedTime(&t, pl->ev0, pl->ev1));
            total += t;
        }
        ms[k] = total / iters;
    }
    return check_device_flag(pl);
} catch (...) { return caught(pl ? pl->ctx : nullptr); }

int msnh_b200_plan_read_trace(MsnhB200Plan *pl, int launch, long long *stamps, int capacity, int *ctas) try {
    if (!pl || !stamps || !ctas) return MSNH_B200_ERR_ARG;
    MsnhB200Ctx *ctx = pl->ctx;
    if (launch < 0 || launch >= static_cast<int>(pl->launches.size())) return fail(ctx, MSNH_B200_ERR_ARG, "read_trace: launch %d", launch);
    const Launch &L = pl->launches[launch];
    if (L.kind != L_CONV_UMMA || !L.up.trace) return fail(ctx, MSNH_B200_ERR_STATE, "launch %d has no trace (plan needs MSNH_PLAN_TRACE)", launch);
    const int n = L.grid * kTraceSlots;
    if (capacity < n) return fail(ctx, MSNH_B200_ERR_ARG, "read_trace: capacity %d < %d", capacity, n);
    CUDA_TRY(ctx, cudaSetDevice(ctx->device));
    CUDA_TRY(ctx, cudaStreamSynchronize(ctx->stream));
    CUDA_TRY(ctx, cudaMemcpy(stamps, L.up.trace, sizeof(long long) * n, cudaMemcpyDeviceToHost));
    CUDA_TRY(ctx, cudaMemset(L.up.trace, 0, sizeof(long long) * n));
    *ctas = L.grid;
    return MSNH_B200_OK;
} catch (...) { return caught(pl ? pl->ctx : nullptr); }

int msnh_b200_plan_destroy(MsnhB200Plan *pl) {
    if (!pl) return MSNH_B200_ERR_ARG;
    cudaSetDevice(pl->ctx->device);
    if (pl->graph_exec) cudaGraphExecDestroy(pl->graph_exec);
    if (pl->graph) cudaGraphDestroy(pl->graph);
    if (pl->ev0) cudaEventDestroy(pl->ev0);
    if (pl->ev1) cudaEventDestroy(pl->ev1);
    if (pl->ev_copy) cudaEventDestroy(pl->ev_copy);
    for (cudaEvent_t e : pl->ev_part) if (e) cudaEventDestroy(e);
    if (pl->h_pinned) cudaFreeHost(pl->h_pinned);
    if (pl->h_early) cudaFreeHost(pl->h_early);
    if (pl->h_early_counts) cudaFreeHost(pl->h_early_counts);
    for (void *d : pl->dev_allocs) cudaFree(d);
    if (pl->arena) cudaFree(pl->arena);
    if (pl->d_input) cudaFree(pl->d_input);
    if (pl->d_readback) cudaFree(pl->d_readback);
    if (pl->d_u8) cudaFree(pl->d_u8);
    if (pl->h_counts) cudaFreeHost(pl->h_counts);
    for (auto &sl : pl->slots) {
        for (cudaGraphExec_t g : sl.graph_exec) if (g) cudaGraphExecDestroy(g);
        if (sl.err_flag) cudaFreeHost(const_cast<int *>(sl.err_flag));
        if (sl.d_stage) cudaFree(sl.d_stage);
        if (sl.d_result) cudaFree(sl.d_result);
        if (sl.h_result) cudaFreeHost(sl.h_result);
        if (sl.h_counts) cudaFreeHost(sl.h_counts);
        if (sl.h2d_done) cudaEventDestroy(sl.h2d_done);
        if (sl.consumed) cudaEventDestroy(sl.consumed);
        if (sl.done) cudaEventDestroy(sl.done);
        for (cudaEvent_t e : sl.piece) if (e) cudaEventDestroy(e);
        if (sl.fwd_done) cudaEventDestroy(sl.fwd_done);
    }
    if (pl->copy_stream) cudaStreamDestroy(pl->copy_stream);
    if (pl->d2h_stream) cudaStreamDestroy(pl->d2h_stream);
    delete pl;
    return MSNH_B200_OK;
}

}  // extern "C"
