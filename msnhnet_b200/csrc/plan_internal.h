// Shared declarations of the plan compiler and executor behind include/msnh_b200.h: the context, the plan's data model
// (ops, tensors, buffers, launches), the debug switches, and the functions its translation units call across files:
//   plan.cu          context, plan lifetime, run / read-back entry points
//   plan_shapes.cu   shape inference and validation of the op list
//   plan_build.cu    lowering: fusion, tensors, zero-copy concat, launches, liveness arena, description
//   plan_tiles.cu    tensor maps; tile-shape model and measured choice of the tensor-core conv; depthwise tiles
//   plan_pack.cu     weight arena staging and the pack cache file
//   plan_launch.cu   the only file that compiles the kernels: one launch per Launch record, small launch wrappers
//   plan_stream.cu   preprocessing, device NMS and the pipelined streaming calls
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>
#include <algorithm>
#include <cmath>
#include <cstdarg>
#include <cstdio>
#include <chrono>
#include <cstdlib>
#include <cstring>
#include <functional>
#include <thread>
#include <array>
#include <map>
#include <memory>
#include <mutex>
#include <new>
#include <stdexcept>
#include <string>
#include <vector>

#include "../../include/msnh_b200.h"
#include "host_pool.h"
#include "kernel_params.h"

// ------------------------------------------------------------------------------------------------
// context
// ------------------------------------------------------------------------------------------------
typedef CUresult (*EncodeTiledFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                  const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
typedef CUresult (*EncodeIm2colFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                   const cuuint64_t *, const int *, const int *, cuuint32_t, cuuint32_t,
                                   const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle,
                                   CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

struct MsnhB200Ctx {
    int device = 0;
    int sm_count = 148;
    int driver_version = 0;
    cudaStream_t stream = nullptr;
    EncodeTiledFn encode_tiled = nullptr;
    EncodeIm2colFn encode_im2col = nullptr;
    int *dev_err_flag = nullptr;    // device address of *err_flag
    volatile int *err_flag = nullptr;   // pinned host memory the kernels write an error code to: looking at it costs no copy
    std::unique_ptr<msnh::HostPool> pool;   // copies of pageable memory (started by the first large one)
    bool pdl = true;                // programmatic dependent launch between consecutive kernels (MSNH_B200_NO_PDL=1 turns it off)
    float *flush_buf = nullptr;     // > L2 size, for per-launch profiling
    size_t flush_elems = 0;
    std::string last_error;
};

namespace msnh {

// records the message on the context (when there is one) and returns `code`
int fail(MsnhB200Ctx *ctx, int code, const char *fmt, ...);
// the status of the exception being handled: what a C entry point that allocates or starts threads returns for it
int caught(MsnhB200Ctx *ctx) noexcept;
#define CUDA_TRY(ctx, expr)                                                                          \
    do {                                                                                             \
        cudaError_t e_ = (expr);                                                                     \
        if (e_ != cudaSuccess)                                                                       \
            return fail(ctx, MSNH_B200_ERR_CUDA, "%s failed: %s (%s:%d)", #expr, cudaGetErrorString(e_), \
                        __FILE__, __LINE__);                                                         \
    } while (0)

// Debug switches, read from the environment once per plan_finalize (and context creation). They change how a plan is
// built, never what it computes (the two that force the shares of a k: in the order of its sums, that is in the last bits).
struct PlanDebugOptions {
    bool no_pdl = false;        // MSNH_B200_NO_PDL=1: plain stream order between kernels
    bool no_merge = false;      // MSNH_B200_NO_MERGE: no sibling 1x1 / SPP pool merging
    bool build_trace = false;   // MSNH_B200_BUILD_TRACE: wall-clock of each build stage on stderr
    bool trace_tune = false;    // MSNH_B200_TRACE_TUNE: traced plans take the measured tile shapes too
    bool dw_simple = false;     // MSNH_B200_DW_SIMPLE: depthwise 3x3 without the shared-memory tile kernel
    int dw_th = 0, dw_stages = 0;   // MSNH_B200_DW_TH, MSNH_B200_DW_STAGES: force the depthwise tile height / ring depth
    bool conv_simple = false;   // MSNH_B200_CONV_SIMPLE: CUDA-core convs without the shared-memory tiled kernel
    int autotune = -1;          // MSNH_B200_AUTOTUNE: -1 unset (time six runners-up), 0 off, n runners-up
    int trace_tile = 0;         // MSNH_B200_TRACE_TILE: which tile of a CTA the producer / MMA stamps describe
    int forced_mm = 0, forced_bn = 0;   // MSNH_B200_M_MULT, MSNH_B200_BN: force the conv tile shape
    int fp32_split = 0;         // MSNH_B200_FP32_SPLIT: shares of the fp32 conv's k (1..8), a CTA each; negative: all of them in one CTA
    int conv_split = 0;         // MSNH_B200_CONV_SPLIT: shares of the split-operand fp32 conv's k (1..8, a CTA each where the clusters fit; negative:
                                // all of them in one CTA)
    int k_split = 0;            // MSNH_B200_K_SPLIT: shares of the tensor-core conv's k in fp32 plans (1: one; 2, 4, 8: a CTA each where
                                // the clusters fit; negative: all of them in one CTA)
    int stream_k = 0;           // MSNH_B200_STREAM_K: -1 by cost, 0 never, 1 wherever possible
    int pair = 0;               // MSNH_B200_PAIR: 1 = CTA pairs wherever possible
    static PlanDebugOptions from_env();
    // any switch that forces tile shapes: such plans neither take shapes from a pack file nor write one
    bool forces_tiles() const { return forced_mm || forced_bn || pair == 1 || stream_k != 0 || k_split != 0; }
};

// ------------------------------------------------------------------------------------------------
// plan data model
// ------------------------------------------------------------------------------------------------
struct Shape { int C = 0, H = 0, W = 0; };

// Where a tensor lives: a root buffer of the arena plus a channel offset (concat slices).
struct Tensor {
    Shape s;
    int   dtype = MSNH_B200_F16;
    int   buffer = -1;     // root buffer id
    int   c_off = 0;
    int   ldc = 0;
    bool  placed = false;  // already a slice of some concat buffer
};

struct Buffer {
    int    ldc = 0, dtype = 0;
    size_t pixels = 0;     // batch*H*W
    size_t bytes = 0, offset = 0;
    int    first = 1 << 30, last = -1;
    bool   persistent = false;
    int    alias_of = -1;  // buffer merged into another one (nested concat): root id
    int    alias_c_off = 0;
};

enum LaunchKind { L_INPUT = 0, L_CONV_UMMA, L_CONV_DIRECT, L_DWCONV, L_SBA, L_ADD, L_BINARY, L_MAXPOOL, L_AVGPOOL,
                  L_UPSAMPLE, L_SLICE, L_PAD, L_SOFTMAX, L_YOLO, L_COLLECT_ZERO, L_COLLECT, L_INPUT_PATCH, L_COLLECT_RAW, L_FOCUS,
                  L_BILINEAR, L_COL2IM, L_CLIP, L_REMAP, L_REDUCE, L_PRELU, L_MAXPOOL_DEPTH, L_CONV_SPLIT, L_INPUT_ROWS };
extern const char *const kLaunchNames[];

struct Launch {
    int kind = 0;
    int op = -1;               // primary op (for describe / parity)
    int dtype = 0;
    TView in{}, out{};
    bool vec = false;
    // generic params
    int kh = 1, kw = 1, sh = 1, sw = 1, ph = 0, pw = 0, dh = 1, dw = 1, groups = 1;
    int act1 = 0, act2 = 0; float act1_p = 0.f, act2_p = 0.f;
    const float *scale = nullptr, *bias = nullptr;
    const float *bias2 = nullptr; int act_mid = 0; float act_mid_p = 0.f;   // deconv gather: BatchNorm behind the layer (scale, bias2)
    const void *weights = nullptr; int cin_pad = 0;
    const void *res = nullptr; int ldc_res = 0;
    AddInputs add{};
    float fval = 0.f; int ival = 0, ival2 = 0;
    int slice_o[3] = {0, 0, 0}, slice_s[3] = {1, 1, 1};
    float anchors[6] = {0, 0, 0, 0, 0, 0};
    int yolo_type = 0; float yolo_ratio = 1.f;   // decode parameters of a fused decode + collect launch
    FocusParams focus{};                         // merged stride-2 slices
    bool focus_planar = false;                   // ... read straight from the planar fp32 image (in.ptr = the input staging)
    PoolSet pools{};                             // L_MAXPOOL: the pools this launch computes (n == 0: the one in kh.. / out)
    YoloHeadSet heads{};                         // L_COLLECT_RAW: the heads this launch decodes and scans
    // yolo collect
    float *rows = nullptr; int *counts = nullptr; int max_rows = 0;
    // umma
    CUtensorMap map_a, map_b, map_c, map_c2, map_res;
    TView out2{};              // second output of two 1x1 convs over the same input merged into this launch (ptr == nullptr: none)
    int split_n = 0;           // its first channel in the merged channel range (split operands: act_mid is its activation)
    ConvUmmaParams up{};
    ConvSplitParams sp{}; int sp_bn = 0, sp_split = 1;   // L_CONV_SPLIT: channels of a tile; CTAs of a cluster its shares are spread over
    int grid = 0; size_t smem = 0;
    // depthwise 3x3 on shared-memory tiles (map_a = the input's 4-D tensor map; grid / smem above)
    bool dw_tile = false; DwTileParams dwp{};
    bool tiled = false;        // L_CONV_DIRECT: dense conv on aligned views -> the shared-memory-tiled CUDA-core kernels
    int fp_shares = 1;         // ... fp32: shares the k of a tile is summed in (1..8)
    int fp_split = 1;          // ... and the CTAs of a cluster they are spread over: 1, or fp_shares
    // accounting
    double flops = 0, bytes = 0;
    std::string note;
};

// Pinned staging of a plan: a ring that larger images and results go round, in parts the copy engine and the threads hand each
// other. PCIe moves it in 0.3 ms: room for threads that are late.
constexpr size_t kStagingBytes = 16 << 20;
constexpr int kStagingParts = 4;
// Pieces a long streaming result crosses PCIe in: pop copies one on to the caller's buffer while the next crosses. After the last
// batch nothing else hides that copy (four batches of FCN-S-320, 16 images and 13 MB of results each: 6.34 -> 6.20 ms).
constexpr int kResultPieces = 4;

struct OpState {
    MsnhB200Op d{};
    Shape out;
    int out_dtype = 0;
    std::vector<float> w[MSNH_W_SLOTS];
    size_t wcount[MSNH_W_SLOTS] = {0, 0, 0, 0, 0, 0};
    // fusion results
    int absorbed_into = -1;     // op index of the launch that computes this op's value
    int tensor = -1;            // tensor id holding this op's value
    bool decode_in_collect = false;   // YOLO head whose decode runs inside the collect launch (its tensor is never written)
    std::vector<int> consumers;
};

// A launch while it is being planned: tensors by id, arena pointers patched in after allocation.
struct Pending { Launch L; int in_t = -1, out_t = -1, res_t = -1; std::vector<int> add_t; int c_off_out = 0; int c_sub = -1; int c_in_off = 0; int c_in_sub = -1;
                 int out2_t = -1;      // second output tensor of a merged pair of 1x1 convs
                 std::vector<int> more_in_t, more_out_t; };   // further heads of a collect launch / further pools over one input

}  // namespace msnh

struct MsnhB200Plan {
    MsnhB200Ctx *ctx = nullptr;
    int in_c = 0, in_h = 0, in_w = 0, batch = 0, dtype = 0;
    uint32_t flags = 0;
    bool split_fp32 = false;                        // convs in fp32 arithmetic on the tensor cores (conv_split.cuh) where they can: the default of
                                                    // fp32 detection nets. Never where the caller asked for MSNH_PLAN_NO_TENSOR_CORE
    msnh::PlanDebugOptions dbg;                     // the debug switches as they stood when plan_finalize began
    std::vector<msnh::OpState> ops;
    std::vector<msnh::Tensor> tensors;
    std::vector<msnh::Buffer> buffers;
    std::vector<msnh::Launch> launches;
    int input_tensor = -1;
    bool finalized = false;
    bool finalize_failed = false;                   // build_launches failed part-way: the plan can only be destroyed
    // device memory
    uint8_t *arena = nullptr; size_t arena_bytes = 0;
    float *sk_ws = nullptr; int *sk_flags = nullptr;   // stream-K hand-over slots and flags (freed with dev_allocs)
    unsigned char *d_u8 = nullptr; size_t d_u8_bytes = 0;        // raw image staging of plan_preprocess_u8
    float *d_nms_boxes = nullptr; int *d_nms_counts = nullptr;   // device NMS output: [batch][kNmsMaxCandidates][8], [batch]
    bool stream_nms = false; float nms_thresh = 0.f, nms_sigma = 0.3f; int nms_soft = 0;   // streaming: NMS on the device
    float *d_input = nullptr;                       // fp32 NCHW staging
    float *d_readback = nullptr; size_t readback_elems = 0;
    std::vector<void *> dev_allocs;                 // weight arena, workspaces
    // Weight arena: every packed tensor of the plan (conv weights, scale / bias tables, slopes) sits in ONE device
    // allocation filled by one copy. While the launches are being planned the tensors are laid out in `pack_host`
    // and launches hold offsets (tagged pointers); the offsets become device pointers once the size is known.
    // With a pack file (plan_use_pack) the laid-out bytes come from the file and the repacking is skipped.
    std::vector<uint8_t> pack_host;
    size_t pack_cursor = 0;
    bool   pack_loaded = false;                     // arena bytes come from the pack file
    std::string pack_path; uint64_t pack_tag = 0;   // set by plan_use_pack
    std::vector<std::array<int32_t, 3>> pack_picks; // conv tile shapes (sub-tiles, channels, form) in launch order: stored in / taken from the pack
    uint8_t *d_pack = nullptr;
    std::vector<uint8_t> pack_blob; uint64_t pack_blob_bytes = 0, pack_blob_key = 0, pack_blob_tag = 0;   // a probed pack file: its arena bytes until they are copied
    uint8_t *h_pinned = nullptr; size_t h_pinned_bytes = 0; bool staging_busy = false;   // pinned staging (kStagingBytes at most) for callers whose memory is pageable; a copy out of it may be under way (ev_copy)
    int *h_counts = nullptr;                        // pinned
    // Results of the last synchronous run, written to pinned memory behind its kernels so that the read call finds them there:
    // candidate counts and the first kEarlyRows rows per image, or the one small output of a classifier.
    int early_op = -1;                              // the op they belong to (-1: the plan has none that qualifies)
    bool early_valid = false; int early_images = 0;
    float *h_early = nullptr; int *h_early_counts = nullptr;
    cudaGraph_t graph = nullptr; cudaGraphExec_t graph_exec = nullptr;
    cudaEvent_t ev0 = nullptr, ev1 = nullptr, ev_copy = nullptr;
    cudaEvent_t ev_part[msnh::kStagingParts] = {};  // the copies of a part of the staging have left or arrived
    float last_ms = 0.f; int timed_steps = 0;       // last_ms is brought up to date from the events when it is asked for (0 steps: it is)
    std::string description;
    // pipelined streaming (plan_stream_push / pop): two slots, a copy stream next to the compute stream
    struct StreamSlot {
        float *d_stage = nullptr;        // this slot's fp32 NCHW input staging on the device
        float *h_result = nullptr;       // pinned: candidate rows or output floats of the batch
        int   *h_counts = nullptr;       // pinned: candidate counts per image
        float *d_result = nullptr;       // device: this slot's copy of an output (candidates go straight to h_result)
        cudaEvent_t h2d_done = nullptr, consumed = nullptr, fwd_done = nullptr, done = nullptr;
        int n_images = 0; bool busy = false;
        bool in_pieces = false; cudaEvent_t piece[msnh::kResultPieces - 1] = {};   // a long result comes in pieces; the last one is `done`
        // A batch's kernels report a wait that ran out here and not on the context, so that the pop of this batch says so: the next
        // batch already runs when this one is popped. (pinned and mapped, like the context's)
        volatile int *err_flag = nullptr; int *dev_err_flag = nullptr;
        // The plan's launches as this slot runs them, put together by the first push of their kind: [0] with the plan's input buffer
        // as the image, [1] with the slot's staging buffer (float pushes: no device copy).
        std::vector<msnh::Launch> launches[2]; cudaGraphExec_t graph_exec[2] = {nullptr, nullptr};
    } slots[2];
    cudaStream_t copy_stream = nullptr, d2h_stream = nullptr;   // host->device of the next batch / device->host of the last
    int stream_op = -1, stream_cap = 0; size_t stream_result_floats = 0;
    int push_count = 0, pop_count = 0;
};

namespace msnh {

inline int esize(int dtype) { return dtype == MSNH_B200_F16 ? 2 : 4; }
inline int vec_of(int dtype) { return dtype == MSNH_B200_F16 ? 8 : 4; }
inline int round_up(int x, int m) { return (x + m - 1) / m * m; }

inline int grid_for(const MsnhB200Ctx *ctx, size_t work_items, int block) {
    size_t blocks = (work_items + block - 1) / block;
    size_t cap = static_cast<size_t>(ctx->sm_count) * 8;   // multiple of the SM count, grid-stride beyond
    if (blocks > cap) blocks = cap;
    if (blocks < 1) blocks = 1;
    return static_cast<int>(blocks);
}

// ---- plan_shapes.cu ----
int infer_shape(MsnhB200Plan *pl, int i, std::string &err);

// ---- plan_build.cu ----
int new_tensor(MsnhB200Plan *pl, Shape s, int dtype);
int new_buffer(MsnhB200Plan *pl, int tensor);
int root_of(MsnhB200Plan *pl, int buf, int *c_off);
TView view_of(MsnhB200Plan *pl, int tensor);
void touch(MsnhB200Plan *pl, int tensor, int step);
int build_launches(MsnhB200Plan *pl);

// ---- plan_tiles.cu ----
CUtensorMapDataType tm_type(int dtype);
// state of the measured tile-shape choice that lives across the launches of one build
struct TileTuning { bool autotune = false; cudaEvent_t ev0 = nullptr, ev1 = nullptr; size_t umma_seen = 0; };
int tile_tuning_begin(MsnhB200Plan *pl, TileTuning &tt);
int tile_tuning_end(MsnhB200Plan *pl, TileTuning &tt);
// tile shape, ring sizes, grid, shared memory and tensor maps of a tensor-core conv launch whose views are resolved
int configure_conv_umma(MsnhB200Plan *pl, TileTuning &tt, Launch &L);
// shares of the k of a CUDA-core fp32 conv launch, and the CTAs they are spread over
void configure_conv_fp32(MsnhB200Plan *pl, Launch &L);
// shares, tiles, grid and tensor maps of a split-operand fp32 conv launch whose views are resolved
int configure_conv_split(MsnhB200Plan *pl, Launch &L);
// the shared-memory tile form of a 3x3 depthwise launch, where it applies (sets L.dw_tile)
void configure_dw_tile(MsnhB200Plan *pl, Launch &L);

// ---- plan_pack.cu ----
// A slot of n elements in the weight arena: `dev` is the slot's offset as a tagged pointer (resolved by
// resolve_pack), `host` its zero-filled staging bytes to fill right away -- valid until the next reserve -- or nullptr
// when the arena is loaded from a pack file.
constexpr uintptr_t kPackTag = static_cast<uintptr_t>(1) << 44;
template <typename T> struct PackSlot { T *host; void *dev; };
uint8_t *reserve_pack_bytes(MsnhB200Plan *pl, size_t bytes, void **dev);
template <typename T> PackSlot<T> reserve_pack(MsnhB200Plan *pl, size_t n) {
    void *dev = nullptr;
    uint8_t *host = reserve_pack_bytes(pl, n * sizeof(T), &dev);
    return {reinterpret_cast<T *>(host), dev};
}
template <typename T> void *upload(MsnhB200Plan *pl, const std::vector<T> &host) {
    PackSlot<T> s = reserve_pack<T>(pl, host.size());
    if (s.host && !host.empty()) std::memcpy(s.host, host.data(), host.size() * sizeof(T));
    return s.dev;
}
template <typename P> void resolve_pack(const MsnhB200Plan *pl, P *&p) {
    const uintptr_t v = reinterpret_cast<uintptr_t>(p);
    if (v & kPackTag) p = reinterpret_cast<P *>(pl->d_pack + (v & (kPackTag - 1)));
}
// A pack file that matches this plan (op list, shapes, flags, blob tag) and whose checksum holds: its arena bytes and
// stored tile shapes are kept in the plan for pack_load_arena. False: there is none, or it does not fit.
bool pack_probe(MsnhB200Plan *pl);
int pack_load_arena(MsnhB200Plan *pl);        // cudaMalloc + copy of the probed bytes (pl->d_pack)
void pack_write(MsnhB200Plan *pl);            // best effort: temporary file unique to this process, then rename

// ---- plan_launch.cu ----
void launch_one(MsnhB200Ctx *ctx, const Launch &L, cudaStream_t st);
void prepare_conv_umma_launch(const Launch &L);   // dynamic shared memory opt-in of the kernel instantiation L runs
int conv_umma_max_clusters(int split);   // k-split convs: clusters of `split` CTAs that run at once
int conv_split_max_clusters(int split);  // the same of the split-operand fp32 conv
void prepare_conv_split_launch();        // shared memory opt-in of its kernels
void launch_readback(MsnhB200Ctx *ctx, int dtype, const TView &v, float *dst_nchw, size_t count, cudaStream_t st);
void launch_preprocess_u8(const unsigned char *src, float *dst, const PrepParams &p, int n_images, cudaStream_t st);
int prepare_yolo_nms(MsnhB200Ctx *ctx);           // shared memory opt-in of the NMS kernel
void launch_yolo_nms(const float *rows, const int *counts, int max_rows, float nms_thresh, int use_soft_nms, float sigma,
                     float *boxes, int box_pitch, int *box_counts, int n_images, cudaStream_t st);
void prepare_dw_tile_launch(int dtype);
void prepare_conv_fp32_launch();                  // shared memory opt-in of the fp32 conv kernels
void launch_fill(MsnhB200Ctx *ctx, float *dst, size_t n, float value, cudaStream_t st);

void launch_candidates_to_host(const float *rows, int max_rows, const int *counts, float *host_rows, int cap, int *host_counts, int n_images, cudaStream_t st);

// ---- plan.cu ----
int check_device_flag(MsnhB200Ctx *ctx, volatile int *flag);      // reads and clears an error word
inline int check_device_flag(MsnhB200Plan *pl) { return check_device_flag(pl->ctx, pl->ctx->err_flag); }
int alloc_device_flag(MsnhB200Ctx *ctx, volatile int **flag, int **dev_flag);   // a pinned, mapped word that kernels write error codes to
constexpr int kEarlyRows = 512;                     // candidate rows per image that come back with a synchronous run
constexpr size_t kEarlyOutputBytes = 1 << 20;       // largest output that does
// Copy to / from the caller's memory that ends or begins on ctx->stream: pageable memory of half a megabyte or more goes through
// pinned staging, chunk by chunk, copied by the pool's threads.
bool is_pageable(const void *p);
int copy_in(MsnhB200Plan *pl, void *dev, const void *host, size_t bytes);
int copy_out(MsnhB200Plan *pl, void *host, const void *dev, size_t bytes);   // the data is there when it returns
void parallel_memcpy(MsnhB200Ctx *ctx, void *dst, const void *src, size_t bytes);

}  // namespace msnh
