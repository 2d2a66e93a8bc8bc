// fp32 convolution on the tensor cores: every fp32 operand is the sum of four bf16 numbers, and a product that of ten
// tensor-core products. What the fp32 plans of detection nets run (boxes decoded through exp() do not hold
// through tf32's 10 mantissa bits); the CUDA-core form of the same arithmetic is conv_fp32_kernel (conv_tiled.cuh). Replaces the
// reference's im2col + cublasSgemm (src/layers/MsnhConvolutionalLayer.cpp:1026-1160).
#pragma once
#include "conv_umma.cuh"

namespace msnh {

// ---------------------------------------------------------------------------------------------------------------------------
// x = x0 + x1 + x2 + x3 exactly: x0 the nearest number of 4 significant bits, x1 and x2 the nearest bf16 (8 bits) of what is left, x3 the rest;
// w the same. Weights are split on the host, activations here. Of the sixteen products ten are taken; the largest of the others, x2 w2, x1 w3
// and x3 w1, are below 2^-26 of x w and some 2^-29: a product keeps more than an fp32 one would.
//
// The sums. The tensor core adds into its fp32 accumulator without rounding to nearest: what does not fit 24 bits is cut off, always
// towards zero, and layers upon layers would multiply such a loss. Products of two 4-bit numbers have 8 bits, so a sum of 32 hardly ever
// needs more than 24: x0 w0 is accumulated over one k-block at a time (32 values of k, two tensor-core steps), and so is x0 w1 + x1 w0, some 2^-5
// of it; both are added up over the k-blocks in registers with ordinary rounded additions. The other seven products, some 2^-10, stay in an accumulator of
// their own over the whole share of k. What a sum of 32 products loses on average, relative (a simulation that fits the tensor core's results):
//     bits of x0, w0                       4         5         6         8        11 (tf32)
//     normal                            3e-10     1e-9      3.4e-9    2.5e-8    1.0e-7
//     normal, behind a LeakyReLU        1.2e-9    3.4e-9    1.0e-8
//     positive activations and weights  5e-10     1.6e-9    5e-9      3.3e-8
// YOLOv5m, whose 94 convs multiply it most, needs 2e-9: with 6 bits its heads (352, 640 pixels) were 1.6 and 2.3 times as far from the net in 64 bits as
// with fp32 FMAs, with tf32 parts, four products and a factor that made up for the mean loss on normal data 1.9 and 3.3 times.
// (inf and NaN stay whole in x0, with the other parts zero; where the large sum is not finite it is the result and the small ones, which hold inf * 0, are dropped.)
//
// Roles of the 28 warps, connected by rings of mbarriers. A wait costs a single thread some 170 cycles even where it passes, so the
// MMA threads have one a k-block: ready(k-block) counts the four splitting warps, the weights' bytes and the sixteen adding warps
// that have emptied the accumulator; the two commits, done(k-block), free the slot and the weights and say that the sums are there.
//   0      loads activations, fp32 as they are: 128 pixels x 32 values of k (one filter tap), im2col or 2-D TMA, 128-byte swizzle
//   1      loads the weights' four parts: 4 x kBn channels x 32 values of k, one 3-D TMA, 64-byte swizzle
//   4-11   split: shared memory -> registers -> TMEM, a pixel (TMEM lane) per thread, 16 columns (two values each) of every part; two groups
//          of four warps take k-blocks in turn. With the parts in TMEM the tensor core reads only the weights from shared memory and an
//          MMA of N channels takes N / 2 cycles.
//   2, 3   issue the MMAs, 2 those of x0 w0, x0 w1 and x1 w0, 3 those of the other seven products: an accumulator has one issuer, so that the order of
//          its sums is fixed. 20 of N = kBn for a k-block (two steps x ten products), half as many where a tap's last channels end
//   12-27  add up: the k-block's sums, TMEM -> registers, kBn / 4 channels of a pixel per thread; at the end of a share of k to shared memory, and
//          where a tile's k is one share after every kSpFlush k-blocks (a chain of rounded additions over all of them would lose more than the shares
//          of conv_fp32_kernel); then scale / bias, activation, residual and the store, in rows of 16-byte vectors
// TMEM: columns 0-319 a ring of accumulators of x0 w0 | x0 w1 + x1 w0 and those of the other products, then three slots of x0 | x1 | x2 | x3
// (320 + 64 s).
//
// The k of a tile is summed in p.shares shares that are added in their order. How many comes from the layer and one image
// (configure_conv_split), so an image has the same bits in a plan of any batch size. kSplit: a cluster of that many CTAs sums one
// each, one tile per cluster, and every CTA finishes every shares-th row through distributed shared memory. Else a CTA walks tiles
// and sums a tile's shares one after the other.
//
// Measured against fp32 FMAs on the CUDA cores (conv_fp32_kernel), a forward in us: YOLOv3-tiny-416, one image 441 -> 243 and sixteen
// 3984 -> 1726; YOLOv5m-352, three images 2973 -> 1520; YOLOv5m-640, two 4717 -> 2381; YOLOv4-416, one 3520 -> 1835. (Two tf32 parts and four products:
// 219, 1532, 1308, 1942 and 1548.) Norm error against 64 bits, FMAs / here in one share: 27 values of k 9.4e-8 / 2.6e-8, 64 1.44e-7 / 2.6e-8,
// 576 1.6e-7 / 3.6e-8, 2304 3.1e-7 / 5.3e-8, 4608 4.3e-7 / 7.4e-8 (normal data; tests/test_conv_split_precision_gpu.py has other kinds). Heads of whole nets against the
// net in 64 bits: YOLOv3-tiny-416 7e-7 / 1.5e-7, YOLOv5m-640 2.1-2.9e-6 / 0.8-1.1e-6, YOLOv4-416 1.0-1.2e-6 / 2.2-2.7e-7.
// ---------------------------------------------------------------------------------------------------------------------------
__device__ __forceinline__ void tma_load_3d(uint32_t dst, const CUtensorMap *map, uint32_t bar, int c0, int c1, int c2) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
        ::"r"(dst), "l"(map), "r"(bar), "r"(c0), "r"(c1), "r"(c2) : "memory");
}
// D (TMEM) += A (TMEM) x B (shared memory), bf16
__device__ __forceinline__ void tcgen05_mma_ts_bf16(uint32_t tmem_d, uint32_t tmem_a, uint64_t desc_b, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
        ::"r"(tmem_d), "r"(tmem_a), "l"(desc_b), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void tmem_st_32x32b_x8(uint32_t taddr, const uint32_t (&r)[8]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%8], {%0, %1, %2, %3, %4, %5, %6, %7};"
                 ::"r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(taddr) : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_ld_32x32b_x8(uint32_t taddr, uint32_t *r) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]) : "r"(taddr) : "memory");
}
__device__ __forceinline__ void tmem_ld_32x32b_x4(uint32_t taddr, uint32_t *r) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(taddr) : "memory");
}
template <int N>                       // N columns (a multiple of four) without waiting for them
__device__ __forceinline__ void tmem_ld_columns(uint32_t taddr, uint32_t (&r)[N]) {
#pragma unroll
    for (int c = 0; c + 8 <= N; c += 8) tmem_ld_32x32b_x8(taddr + static_cast<uint32_t>(c), r + c);
    if constexpr (N % 8 != 0) tmem_ld_32x32b_x4(taddr + static_cast<uint32_t>(N - 4), r + N - 4);
}

// Sixteen values (as bits) to their leading parts, two to a register, and what those leave. kCareful: for values that round to infinity,
// which are cut off in place of it, and for inf and NaN, which leave nothing. Returns a NaN where the careful form is needed, else zero.
template <bool kCareful>
__device__ __forceinline__ float split_lead(uint32_t (&x)[16], uint32_t (&part)[8]) {
    float bad = 0.f;
#pragma unroll
    for (int q = 0; q < 16; q += 2) {
        uint32_t h[2];
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const uint32_t u = x[q + e];
            h[e] = (u + (1u << (kSplitLeadCut - 1))) & ~((1u << kSplitLeadCut) - 1u);
            if (kCareful) {
                const uint32_t mag = u & 0x7fffffffu;
                if (mag >= kSplitLeadMax) h[e] = mag > 0x7f800000u ? 0x7fc00000u : u & 0xffff0000u;
                x[q + e] = mag >= 0x7f800000u ? 0u : __float_as_uint(__fsub_rn(__uint_as_float(u), __uint_as_float(h[e])));
            } else {
                x[q + e] = __float_as_uint(__fsub_rn(__uint_as_float(u), __uint_as_float(h[e])));
                bad = __fmaf_rn(__uint_as_float(x[q + e]), 0.f, bad);
            }
        }
        part[q / 2] = __byte_perm(h[0], h[1], 0x7632);
    }
    return bad;
}
// their next parts, the nearest bf16, and what those leave
__device__ __forceinline__ void split_next(uint32_t (&x)[16], uint32_t (&part)[8]) {
#pragma unroll
    for (int q = 0; q < 8; ++q) {
        asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(part[q]) : "f"(__uint_as_float(x[2 * q + 1])), "f"(__uint_as_float(x[2 * q])));
        x[2 * q] = __float_as_uint(__fsub_rn(__uint_as_float(x[2 * q]), __uint_as_float(part[q] << 16)));
        x[2 * q + 1] = __float_as_uint(__fsub_rn(__uint_as_float(x[2 * q + 1]), __uint_as_float(part[q] & 0xffff0000u)));
    }
}

// The end of a tile: scale / bias, activation, residual (+ second activation), store. Of kThreads threads each has four channels of
// every kRows-th row; rows row0, row0 + step, ... are these threads'. A thread's scale and bias are loaded long before its
// sums are there, its rows kBatch at a time: row by row, with the tables read for each, the end of a tile of 128 x 64 took 9000
// cycles, most of them latency. `sum` gives the sums at a byte offset into the tile.
template <int kBn, int kThreads, int kBatch>
struct SplitFinish {
    static constexpr int kQuads = kBn / 4, kRows = kThreads / kQuads;
    int row, col, c, cout;
    const TView &out;
    float4 sc, bi;
    bool live;
    __device__ __forceinline__ SplitFinish(const ConvSplitParams &p, const TView &out1, const TView &out2, int n0, int t)
        : row(t / kQuads), col(4 * (t % kQuads)), c(n0 + col), cout(n0 < p.split_n ? p.split_n : p.cout), out(n0 < p.split_n ? out1 : out2), live(t < kRows * kQuads && c < cout) {
        if (live) { sc = __ldg(reinterpret_cast<const float4 *>(p.scale + c)); bi = __ldg(reinterpret_cast<const float4 *>(p.bias + c)); }   // (padded past the last channel tile)
    }
    template <typename Sum>
    __device__ __forceinline__ void operator()(const ConvSplitParams &p, int m0, int row0, int step, Sum &&sum) const {
        if (!live) return;
        const int rows = min(kUmmaM, p.m_total - m0);
        const bool whole = c + 4 <= cout;
        float *const dst0 = static_cast<float *>(out.ptr) + (c < p.split_n ? c : c - p.split_n);
        for (int j = row0 + row * step; j < rows; j += kBatch * kRows * step) {
            float y[4 * kBatch], rr[4 * kBatch];
#pragma unroll
            for (int q = 0; q < kBatch; ++q) {
                const int r = min(j + q * kRows * step, rows - 1);                    // (rows past the last are computed and not stored)
                sum(4u * static_cast<uint32_t>(r * (kBn + 4) + col), y + 4 * q);
                if (p.res) {
                    const float *rp = static_cast<const float *>(p.res) + static_cast<size_t>(m0 + r) * p.ldc_res + c;
                    if (whole) {
                        const float4 t = *reinterpret_cast<const float4 *>(rp);
                        rr[4 * q] = t.x; rr[4 * q + 1] = t.y; rr[4 * q + 2] = t.z; rr[4 * q + 3] = t.w;
                    } else {
#pragma unroll
                        for (int e = 0; e < 4; ++e) rr[4 * q + e] = c + e < cout ? rp[e] : 0.f;
                    }
                }
            }
#pragma unroll
            for (int q = 0; q < 4 * kBatch; q += 4) { y[q] = fmaf(y[q], sc.x, bi.x); y[q + 1] = fmaf(y[q + 1], sc.y, bi.y); y[q + 2] = fmaf(y[q + 2], sc.z, bi.z); y[q + 3] = fmaf(y[q + 3], sc.w, bi.w); }
            activate_all(y, c < p.split_n ? p.act1 : p.act1_b, c < p.split_n ? p.act1_param : p.act1_b_param);
            if (p.res) {
#pragma unroll
                for (int q = 0; q < 4 * kBatch; ++q) y[q] = __fadd_rn(y[q], rr[q]);
                activate_all(y, p.act2, p.act2_param);
            }
#pragma unroll
            for (int q = 0; q < kBatch; ++q) {
                const int r = j + q * kRows * step;
                if (r >= rows) break;
                float *dst = dst0 + static_cast<size_t>(m0 + r) * out.ldc;
                if (whole) *reinterpret_cast<float4 *>(dst) = make_float4(y[4 * q], y[4 * q + 1], y[4 * q + 2], y[4 * q + 3]);
                else {
#pragma unroll
                    for (int e = 0; e < 4; ++e) if (c + e < cout) dst[e] = y[4 * q + e];
                }
            }
        }
    }
    static __device__ __forceinline__ void activate_all(float (&v)[4 * kBatch], int act, float param) {      // (one branch for all of them)
        if (act == MSNH_ACT_NONE) return;
        if (act == MSNH_ACT_LEAKY) {
#pragma unroll
            for (int e = 0; e < 4 * kBatch; ++e) v[e] = activate(v[e], MSNH_ACT_LEAKY, param);
        } else if (act == MSNH_ACT_HARD_SWISH) {
#pragma unroll
            for (int e = 0; e < 4 * kBatch; ++e) v[e] = activate(v[e], MSNH_ACT_HARD_SWISH, param);
        } else {
#pragma unroll
            for (int e = 0; e < 4 * kBatch; ++e) v[e] = activate_slow(v[e], act, param);
        }
    }
};

template <int kBn, bool kSplit>
__global__ void __launch_bounds__(kSpThreads, 1)
conv_split_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b, const __grid_constant__ TView out, const __grid_constant__ TView out2, const __grid_constant__ ConvSplitParams p) {
    constexpr int kCols = kBn / 4;                                   // channels of a pixel an adding thread holds
    constexpr int kPitch = kBn + 4;                                  // floats of a row of the tile of sums
    constexpr uint32_t kABytes = kUmmaM * 128, kPartBytes = kBn * 64, kBBytes = 4 * kPartBytes;
    // TMEM columns 0-319: accumulators of x0 w0 and of x0 w1 + x1 w0 side by side (a ring) and of the other products (twice where there is room)
    constexpr uint32_t kMain = kBn >= 48 ? 2 : 4, kSmall = kBn == 64 ? 1 : 2, kSmallCol = 2 * kMain * kBn, kSlotCol = 320;
    static_assert((2 * kMain + kSmall) * kBn <= kSlotCol && kSlotCol + 64 * kSpSlots <= 512, "TMEM columns");
    extern __shared__ uint8_t smem_raw[];
    const uint32_t a_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    const uint32_t b_base = a_base + kSpAStages * kABytes;
    const uint32_t sum_base = b_base + kSpBStages * kBBytes;         // [128][kPitch] floats
    const uint32_t bar_base = sum_base + kUmmaM * kPitch * 4;
    auto full_a  = [&](uint32_t s) { return bar_base + 8u * s; };
    auto empty_a = [&](uint32_t s) { return bar_base + 8u * (8 + s); };
    auto ready   = [&](uint32_t s) { return bar_base + 8u * (16 + s); };
    auto done    = [&](uint32_t s) { return bar_base + 8u * (24 + s); };
    auto s_full  = [&](uint32_t s) { return bar_base + 8u * (32 + s); };
    auto s_empty = [&](uint32_t s) { return bar_base + 8u * (34 + s); };
    __shared__ uint32_t tmem_base_slot;
    __shared__ int cta_abort_slot;
    volatile int *cta_abort = &cta_abort_slot;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int num_tiles = p.tiles_m * p.tiles_n, num_k = p.taps * p.chunks_per_tap;
    int rank = 0;
    if constexpr (kSplit) asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
    const int first_tile = kSplit ? static_cast<int>(blockIdx.x) / p.shares : static_cast<int>(blockIdx.x);
    const int tile_stride = kSplit ? num_tiles : static_cast<int>(gridDim.x);
    const int share_first = kSplit ? rank : 0, share_end = kSplit ? rank + 1 : p.shares;

    pdl_launch_dependents();
    if (threadIdx.x < 36) {             // a barrier per thread
        const uint32_t t = threadIdx.x;
        mbar_init(bar_base + 8u * t, t < 8 ? 1u : t < 16 ? 4u : t < 24 ? 4 + 1 + 16u : t < 32 ? 2u : t < 34 ? 1u : 16u);      // full_a, empty_a, ready, done, s_full, s_empty
        if (t == 0) cta_abort_slot = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (threadIdx.x == 96) {
        asm volatile("prefetch.tensormap [%0];" ::"l"(&map_b) : "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(&map_a) : "memory");
    }
    if (warp == 2) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base_slot)), "r"(512u) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tcgen05_fence_before();
    __syncthreads();
    tcgen05_fence_after();
    const uint32_t tmem = tmem_base_slot;

    if (warp == 0) {
        // ------------------------------ activations ------------------------------
        if (elect_one()) {
            uint32_t stage = 0, phase = 1;
            bool ok = true;
            const bool im2col = p.a_mode == A_MODE_IM2COL;
            pdl_wait();                     // the activations are the previous kernel's output
            for (int tile = first_tile; tile < num_tiles && ok; tile += tile_stride) {
                const int m0 = tile / p.tiles_n * kUmmaM;
                const int img = m0 / (p.oh * p.ow), rem = m0 - img * p.oh * p.ow, y0 = rem / p.ow, x0 = rem - y0 * p.ow;
                const int cx = x0 * p.stride_w - p.pad_w, cy = y0 * p.stride_h - p.pad_h;
                const int k0 = kSplit ? num_k * rank / p.shares : 0, k1 = kSplit ? num_k * (rank + 1) / p.shares : num_k;
                const int tap = k0 / p.chunks_per_tap, r = tap / p.kw;
                int chunk = k0 - tap * p.chunks_per_tap, s = tap - r * p.kw, off_h = r * p.dil_h, off_w = s * p.dil_w;
                for (int kt = k0; kt < k1; ++kt) {
                    ok = mbar_wait(empty_a(stage), phase, cta_abort, p.err_flag, DEV_ERR_WAIT_EMPTY);
                    if (!ok) break;
                    mbar_expect_tx(full_a(stage), kABytes);
                    if (im2col) tma_load_im2col_4d(a_base + stage * kABytes, &map_a, full_a(stage), 32 * chunk, cx, cy, img, static_cast<uint16_t>(off_w), static_cast<uint16_t>(off_h));
                    else        tma_load_2d(a_base + stage * kABytes, &map_a, full_a(stage), 32 * chunk, m0);
                    if (++stage == kSpAStages) { stage = 0; phase ^= 1u; }
                    if (++chunk == p.chunks_per_tap) {
                        chunk = 0; off_w += p.dil_w;
                        if (++s == p.kw) { s = 0; off_w = 0; off_h += p.dil_h; }
                    }
                }
            }
        }
    } else if (warp == 1) {
        // ------------------------------ weights (constants: asked for while the previous kernel still runs) ------------------------------
        if (elect_one()) {
            uint32_t stage = 0, at = 0, freed = 0, phase = 0, ahead = kSpBStages;     // (the first stages are free)
            bool ok = true;
            for (int tile = first_tile; tile < num_tiles && ok; tile += tile_stride) {
                const int n0 = tile % p.tiles_n * kBn;
                const int k0 = kSplit ? num_k * rank / p.shares : 0, k1 = kSplit ? num_k * (rank + 1) / p.shares : num_k;
                const int tap = k0 / p.chunks_per_tap;
                int chunk = k0 - tap * p.chunks_per_tap, c_tap = tap * p.cin_pad;
                for (int kt = k0; kt < k1; ++kt) {
                    if (ahead) --ahead;
                    else {
                        ok = mbar_wait(done(freed), phase, cta_abort, p.err_flag, DEV_ERR_WAIT_EMPTY);
                        if (!ok) break;
                        if (++freed == kSpRing) { freed = 0; phase ^= 1u; }
                    }
                    mbar_expect_tx(ready(at), kBBytes);
                    tma_load_3d(b_base + stage * kBBytes, &map_b, ready(at), c_tap + 32 * chunk, n0, 0);
                    if (++stage == kSpBStages) stage = 0;
                    if (++at == kSpRing) at = 0;
                    if (++chunk == p.chunks_per_tap) { chunk = 0; c_tap += p.cin_pad; }
                }
            }
        }
    } else if (warp < 4) {
        // ------------------------------ MMA issuers: the products of every k-block shared between them ------------------------------
        if (elect_one()) {
            constexpr uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | (static_cast<uint32_t>(kBn >> 3) << 17) | (static_cast<uint32_t>(kUmmaM >> 4) << 24);
            const uint32_t issuer = static_cast<uint32_t>(warp - 2);
            const uint64_t desc_b0 = make_smem_desc(b_base, 64);
            uint32_t at = 0, phase = 0, stage = 0, slot = 0, acc = 0;
            uint32_t small = 0, small_phase = 1;
            bool ok = true;
            for (int tile = first_tile; tile < num_tiles && ok; tile += tile_stride)
                for (int share = share_first; share < share_end && ok; ++share) {
                    const int k0 = num_k * share / p.shares, k1 = num_k * (share + 1) / p.shares;
                    int chunk = k0 % p.chunks_per_tap;
                    if (issuer == 1) {
                        ok = mbar_wait(s_empty(small), small_phase, cta_abort, p.err_flag, DEV_ERR_WAIT_ACC_EMPTY);
                        if (!ok) break;
                    }
                    const uint32_t d_small = tmem + kSmallCol + kBn * small;
                    uint32_t more = 0;                                          // the share's first MMA begins its small sums
                    for (int kt = k0; kt < k1; ++kt) {
                        const bool last = ++chunk == p.chunks_per_tap;
                        if (last) chunk = 0;
                        ok = mbar_wait(ready(at), phase, cta_abort, p.err_flag, DEV_ERR_WAIT_FULL);
                        if (!ok) break;
                        tcgen05_fence_after();
                        const uint64_t w0 = desc_b0 + static_cast<uint64_t>(stage) * (kBBytes >> 4), w1 = w0 + (kPartBytes >> 4), w2 = w1 + (kPartBytes >> 4), w3 = w2 + (kPartBytes >> 4);
                        const uint32_t x0 = tmem + kSlotCol + 64u * slot, x1 = x0 + 16u, x2 = x1 + 16u, x3 = x2 + 16u, d_main = tmem + 2 * kBn * acc, d_mid = d_main + kBn;
                        auto step = [&](uint32_t k, uint32_t more_main, uint32_t more_small) {
                            if (issuer == 0) {
                                tcgen05_mma_ts_bf16(d_mid, x0 + 8 * k, w1 + 2 * k, idesc, more_main);
                                tcgen05_mma_ts_bf16(d_main, x0 + 8 * k, w0 + 2 * k, idesc, more_main);
                                tcgen05_mma_ts_bf16(d_mid, x1 + 8 * k, w0 + 2 * k, idesc, 1u);
                            } else {
                                tcgen05_mma_ts_bf16(d_small, x1 + 8 * k, w1 + 2 * k, idesc, more_small);
                                tcgen05_mma_ts_bf16(d_small, x0 + 8 * k, w2 + 2 * k, idesc, 1u);
                                tcgen05_mma_ts_bf16(d_small, x2 + 8 * k, w0 + 2 * k, idesc, 1u);
                                tcgen05_mma_ts_bf16(d_small, x1 + 8 * k, w2 + 2 * k, idesc, 1u);
                                tcgen05_mma_ts_bf16(d_small, x2 + 8 * k, w1 + 2 * k, idesc, 1u);
                                tcgen05_mma_ts_bf16(d_small, x0 + 8 * k, w3 + 2 * k, idesc, 1u);
                                tcgen05_mma_ts_bf16(d_small, x3 + 8 * k, w0 + 2 * k, idesc, 1u);
                            }
                        };
                        step(0u, 0u, more);
                        if (!last || p.tail_steps == 2) step(1u, 1u, 1u);
                        more = 1;
                        tcgen05_commit(done(at));
                        if (++at == kSpRing) { at = 0; phase ^= 1u; }
                        if (++stage == kSpBStages) stage = 0;
                        if (++slot == kSpSlots) slot = 0;
                        if (++acc == kMain) acc = 0;
                    }
                    if (!ok) break;
                    if (issuer == 1) tcgen05_commit(s_full(small));
                    if (++small == kSmall) { small = 0; small_phase ^= 1u; }
                }
        }
    } else if (warp >= 4 && warp < 12) {
        // ------------------------------ split: fp32 in shared memory -> four bf16 parts in TMEM ------------------------------
        const int group = (warp - 4) >> 2;
        const uint32_t row = static_cast<uint32_t>((warp & 3) * 32 + lane), swz = row & 7u;
        const uint32_t lanes = static_cast<uint32_t>((warp & 3) * 32) << 16;
        const int k_tile = kSplit ? num_k * (rank + 1) / p.shares - num_k * rank / p.shares : num_k;
        const int tiles_here = first_tile < num_tiles ? (num_tiles - first_tile + tile_stride - 1) / tile_stride : 0;
        const long long total = static_cast<long long>(tiles_here) * k_tile;
        uint32_t stage = static_cast<uint32_t>(group), a_phase = 0, slot = static_cast<uint32_t>(group), at = slot, freed = at + kSpRing - kSpSlots, s_phase = 1;
        for (long long q = group; q < total; q += 2) {
            bool ok = mbar_wait(full_a(stage), a_phase, cta_abort, p.err_flag, DEV_ERR_WAIT_FULL);
            if (!__all_sync(0xffffffffu, ok)) break;
            const uint32_t src = a_base + stage * kABytes + row * 128u, dst = tmem + lanes + kSlotCol + 64u * slot;
            uint32_t x[16];
            auto fetch = [&](uint32_t h) {          // half a row
#pragma unroll
                for (uint32_t j = 0; j < 4; ++j)
                    asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(x[4 * j]), "=r"(x[4 * j + 1]), "=r"(x[4 * j + 2]), "=r"(x[4 * j + 3]) : "r"(src + (((j + 4u * h) ^ swz) << 4)) : "memory");
            };
            fetch(0);
            if (q >= kSpSlots) {                    // the slot's k-block before this one
                ok = mbar_wait(done(freed), s_phase, cta_abort, p.err_flag, DEV_ERR_WAIT_EMPTY);
                if (!__all_sync(0xffffffffu, ok)) break;
            }
            tcgen05_fence_after();
#pragma unroll
            for (uint32_t h = 0; h < 2; ++h) {
                uint32_t part[8];
                if (h == 1) fetch(1);
                const float bad = split_lead<false>(x, part);
                if (__any_sync(0xffffffffu, bad != 0.f)) { fetch(h); split_lead<true>(x, part); }
                tmem_st_32x32b_x8(dst + 8u * h, part);
                split_next(x, part);
                tmem_st_32x32b_x8(dst + 16u + 8u * h, part);
                split_next(x, part);
                tmem_st_32x32b_x8(dst + 32u + 8u * h, part);
#pragma unroll
                for (int q = 0; q < 8; ++q) part[q] = __byte_perm(x[2 * q], x[2 * q + 1], 0x7632);      // (what is left has two bits)
                tmem_st_32x32b_x8(dst + 48u + 8u * h, part);
            }
            tmem_st_wait();
            tcgen05_fence_before();
            __syncwarp();
            // (the stage is given back behind the last use of its values: an arrive overtakes loads that nothing has waited for)
            if (lane == 0) { mbar_arrive(empty_a(stage)); mbar_arrive(ready(at)); }
            stage += 2; if (stage >= kSpAStages) { stage -= kSpAStages; a_phase ^= 1u; }
            slot += 2; if (slot >= kSpSlots) slot -= kSpSlots;
            at += 2; if (at >= kSpRing) at -= kSpRing;
            freed += 2; if (freed >= kSpRing) { freed -= kSpRing; s_phase ^= 1u; }
        }
    } else if (warp >= 12) {
        // ------------------------------ sums in registers, epilogue ------------------------------
        const int t = static_cast<int>(threadIdx.x) - 12 * 32;
        const int part = (warp - 12) >> 2;
        const uint32_t row = static_cast<uint32_t>((warp & 3) * 32 + lane);
        const uint32_t from = tmem + (static_cast<uint32_t>((warp & 3) * 32) << 16) + static_cast<uint32_t>(part * kCols);
        const uint32_t mine = sum_base + 4u * (row * kPitch + static_cast<uint32_t>(part * kCols));
        uint32_t at = 0, phase = 0, from_acc = 0, small = 0, small_phase = 0;
        bool ok = true;
        if (lane == 0)
            for (uint32_t a = 0; a < kMain; ++a) mbar_arrive(ready(a));                 // all accumulators are free
        auto load = [&](uint32_t at, uint32_t (&v)[kCols]) {
            tmem_ld_columns(at, v);
            tmem_ld_wait();
#pragma unroll
            for (int c = 0; c < kCols; ++c) asm volatile("" : "+r"(v[c]));      // (no use of them moves up past the wait)
        };
        for (int tile = first_tile; tile < num_tiles && ok; tile += tile_stride) {
            const SplitFinish<kBn, 512, 4> finish(p, out, out2, tile % p.tiles_n * kBn, t);
            bool begun = false;                       // sums of this tile are in shared memory
            for (int share = share_first; share < share_end && ok; ++share) {
                const int k0 = num_k * share / p.shares, k1 = num_k * (share + 1) / p.shares;
                float acc[kCols], mid[kCols];
#pragma unroll
                for (int c = 0; c < kCols; ++c) acc[c] = mid[c] = 0.f;
                // the sums so far to shared memory, behind those that are there: earlier k-blocks and shares, in their order
                auto flush = [&]() {
#pragma unroll
                    for (int c = 0; c < kCols; c += 4) {
                        const uint32_t to = mine + 4u * static_cast<uint32_t>(c);
                        if (begun) {
                            float4 s;
                            asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(s.x), "=f"(s.y), "=f"(s.z), "=f"(s.w) : "r"(to) : "memory");
                            acc[c] = __fadd_rn(s.x, acc[c]); acc[c + 1] = __fadd_rn(s.y, acc[c + 1]); acc[c + 2] = __fadd_rn(s.z, acc[c + 2]); acc[c + 3] = __fadd_rn(s.w, acc[c + 3]);
                        }
                        asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(to), "f"(acc[c]), "f"(acc[c + 1]), "f"(acc[c + 2]), "f"(acc[c + 3]) : "memory");
                        acc[c] = acc[c + 1] = acc[c + 2] = acc[c + 3] = 0.f;
                    }
                    begun = true;
                };
                for (int kt = k0; kt < k1; ++kt) {
                    ok = mbar_wait(done(at), phase, cta_abort, p.err_flag, DEV_ERR_WAIT_ACC_FULL);
                    ok = __all_sync(0xffffffffu, ok);
                    if (!ok) break;
                    tcgen05_fence_after();
                    uint32_t v[kCols];
                    load(from + 2 * kBn * from_acc, v);
#pragma unroll
                    for (int c = 0; c < kCols; ++c) acc[c] = __fadd_rn(acc[c], __uint_as_float(v[c]));
                    load(from + 2 * kBn * from_acc + kBn, v);
                    tcgen05_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(ready((at + kMain) % kSpRing));      // the accumulators are the k-block's that comes kMain later
                    if (++at == kSpRing) { at = 0; phase ^= 1u; }
                    if (++from_acc == kMain) from_acc = 0;
#pragma unroll
                    for (int c = 0; c < kCols; ++c) mid[c] = __fadd_rn(mid[c], __uint_as_float(v[c]));
                    if (!kSplit && p.shares == 1 && kt % kSpFlush == kSpFlush - 1 && kt + 1 < k1) flush();
                }
                if (!ok) break;
                ok = mbar_wait(s_full(small), small_phase, cta_abort, p.err_flag, DEV_ERR_WAIT_ACC_FULL);
                ok = __all_sync(0xffffffffu, ok);
                if (!ok) break;
                tcgen05_fence_after();
                {
                    uint32_t v[kCols];
                    load(from + kSmallCol + kBn * small, v);
#pragma unroll
                    for (int c = 0; c < kCols; ++c) mid[c] = __fadd_rn(mid[c], __uint_as_float(v[c]));
                }
                tcgen05_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(s_empty(small));
                if (++small == kSmall) { small = 0; small_phase ^= 1u; }
                // (a large sum that is not finite may have gone to shared memory: the small sums are asked, which are then not finite either)
#pragma unroll
                for (int c = 0; c < kCols; ++c) if ((__float_as_uint(mid[c]) & 0x7f800000u) != 0x7f800000u) acc[c] = __fadd_rn(acc[c], mid[c]);
                flush();
            }
            if constexpr (!kSplit) {
                // the sixteen warps decide together: they meet at the tile of sums
                uint32_t all_ok;
                asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.u32 q, %1, 0;\n\tbar.red.and.pred p, 1, 512, q;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                             : "=r"(all_ok) : "r"(static_cast<uint32_t>(ok)) : "memory");
                ok = all_ok != 0;
                if (!ok) break;
                if (p.res) pdl_wait();                               // the residual is an earlier kernel's output
                finish(p, tile / p.tiles_n * kUmmaM, 0, 1, [&](uint32_t at, float *y) {
                    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(y[0]), "=f"(y[1]), "=f"(y[2]), "=f"(y[3]) : "r"(sum_base + at) : "memory");
                });
                asm volatile("bar.sync 1, 512;" ::: "memory");        // the tile of sums is free for the next tile
            }
        }
    }

    tcgen05_fence_before();
    __syncthreads();
    if constexpr (kSplit) {
        const SplitFinish<kBn, kSpThreads, 1> finish(p, out, out2, first_tile % p.tiles_n * kBn, static_cast<int>(threadIdx.x));
        cluster_sync_all();          // every share of the tile is in some CTA's shared memory
        if (*cta_abort == 0) {
            if (p.res) pdl_wait();
            finish(p, first_tile / p.tiles_n * kUmmaM, rank, p.shares, [&](uint32_t at, float *y) {
#pragma unroll
                for (int q = 0; q < kUmmaMaxKSplit; ++q)
                    if (q < p.shares) {
                        float4 s;
                        asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(s.x), "=f"(s.y), "=f"(s.z), "=f"(s.w) : "r"(map_to_cta(sum_base + at, q)) : "memory");
                        if (q == 0) { y[0] = s.x; y[1] = s.y; y[2] = s.z; y[3] = s.w; }
                        else { y[0] = __fadd_rn(y[0], s.x); y[1] = __fadd_rn(y[1], s.y); y[2] = __fadd_rn(y[2], s.z); y[3] = __fadd_rn(y[3], s.w); }
                    }
            });
        }
        __syncwarp();
        cluster_sync_all();          // nobody leaves while a peer still reads its shared memory
    }
    if (warp == 2) {
        __syncwarp();
        tcgen05_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
    }
}

}  // namespace msnh
