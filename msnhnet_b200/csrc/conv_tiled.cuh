// Dense convolutions on the CUDA cores in fp32 arithmetic.
//
// conv_fp32_kernel (below) serves the plans that must reproduce the reference's fp32 results (its GPU path is fp32 Sgemm
// throughout, src/layers/MsnhConvolutionalLayer.cpp:1026-1160): fp32 detection nets without tensor cores, whose exp()-decoded boxes do not survive
// tf32's 10-bit mantissa, and fp32 plans built without tensor cores.
// conv_tiled_kernel: an implicit GEMM with shared-memory tiles for 16-bit plans built without tensor cores (the cross-check of
// the tensor-core kernel).
// D[m][n] = sum_k A[m][k] * B[n][k]: m = output pixel (linear over image, row, column), n = output channel, k = (filter
// tap, input channel) tap-major like the packed weights [Cout][tap][cin_pad]. A CTA of 256 threads computes 128 pixels x
// 64 channels; a k-step stages 128 x BK input values (gathered with the conv's stride / padding / dilation, zero outside the
// plane) and 64 x BK weights in shared memory as fp32, k-major, so that the inner loop reads them without bank conflicts;
// the next k-step's global loads are in flight while this one's products are summed. A thread owns 8 pixels x 4 channels.
#pragma once
#include "common.cuh"
#include "layer_kernels.cuh"
#include "conv_umma.cuh"   // packed fp32 pairs, cluster barrier

namespace msnh {

template <typename T>
__global__ void __launch_bounds__(kCtThreads)
conv_tiled_kernel(TView in, TView out, const T *__restrict__ w, const ConvTiledParams p) {
    constexpr int V = Elem<T>::kVec;           // elements per 16-byte vector
    constexpr int BK = 4 * V;                  // k elements per step: four vectors per pixel / per output channel
    __shared__ float As[BK][kCtBM + 4];
    __shared__ float Bs[BK][kCtBN + 4];
    pdl_prologue();
    const int tid = threadIdx.x;
    const int m_total = out.N * out.H * out.W;
    const int m0 = blockIdx.x * kCtBM, n0 = blockIdx.y * kCtBN;
    const int cin = in.C, cout = out.C;
    // this thread's global loads: two pixels (64 apart) x one vector of A, one output channel x one vector of B
    const int kq = tid & 3;                    // which of the four vectors of the k-step
    const int lrow = tid >> 2;                 // 0..63
    int pn[2], py[2], px[2]; bool pvalid[2];
#pragma unroll
    for (int j = 0; j < 2; ++j) {
        const int m = m0 + lrow + 64 * j;
        pvalid[j] = m < m_total;
        const int mm = pvalid[j] ? m : 0;
        pn[j] = mm / (out.H * out.W);
        const int rem = mm - pn[j] * out.H * out.W;
        py[j] = rem / out.W; px[j] = rem - py[j] * out.W;
    }
    const int co_ld = n0 + lrow;               // (lrow < 64: every thread loads one vector of B)
    const T *wrow = w + static_cast<size_t>(co_ld < cout ? co_ld : 0) * p.kh * p.kw * p.cin_pad;
    // compute mapping: pixels tm + 16 i (i < 8), channels 4 tn .. 4 tn + 3
    const int tm = tid & 15, tn = tid >> 4;
    float acc[8][4];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[i][e] = 0.f;

    const int chunks = (cin + BK - 1) / BK;
    const int steps = p.kh * p.kw * chunks;
    float ra[2][V], rb[V];
    auto load_step = [&](int step) {
        const int tap = step / chunks, c = (step - tap * chunks) * BK + kq * V;
        const int r = tap / p.kw, s = tap - r * p.kw;
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            const int iy = py[j] * p.sh - p.ph + r * p.dh, ix = px[j] * p.sw - p.pw + s * p.dw;
            const bool inside = pvalid[j] && iy >= 0 && iy < in.H && ix >= 0 && ix < in.W && c < cin;
            if (inside) {
                const T *src = static_cast<const T *>(in.ptr) + pix_off(in, pn[j], iy, ix) + c;
                if (c + V <= in.ldc) VecIO<T, V>::ld(src, ra[j]);
                else {
#pragma unroll
                    for (int e = 0; e < V; ++e) ra[j][e] = c + e < cin ? Elem<T>::ld(src + e) : 0.f;
                }
#pragma unroll
                for (int e = 0; e < V; ++e) if (c + e >= cin) ra[j][e] = 0.f;     // pad channels of the pitch hold no data
            } else {
#pragma unroll
                for (int e = 0; e < V; ++e) ra[j][e] = 0.f;
            }
        }
        if (co_ld < cout && c < p.cin_pad) VecIO<T, V>::ld(wrow + static_cast<size_t>(tap) * p.cin_pad + c, rb);
        else {
#pragma unroll
            for (int e = 0; e < V; ++e) rb[e] = 0.f;
        }
    };
    load_step(0);
    for (int step = 0; step < steps; ++step) {
#pragma unroll
        for (int e = 0; e < V; ++e) {
            As[kq * V + e][lrow] = ra[0][e];
            As[kq * V + e][lrow + 64] = ra[1][e];
            Bs[kq * V + e][lrow] = rb[e];
        }
        __syncthreads();
        if (step + 1 < steps) load_step(step + 1);          // in flight under the arithmetic below
#pragma unroll
        for (int k = 0; k < BK; ++k) {
            float a[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) a[i] = As[k][tm + 16 * i];
            const float4 b = *reinterpret_cast<const float4 *>(&Bs[k][4 * tn]);
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                acc[i][0] = fmaf(a[i], b.x, acc[i][0]); acc[i][1] = fmaf(a[i], b.y, acc[i][1]);
                acc[i][2] = fmaf(a[i], b.z, acc[i][2]); acc[i][3] = fmaf(a[i], b.w, acc[i][3]);
            }
        }
        __syncthreads();
    }
    // epilogue: scale / bias, activation, residual (+ second activation), store
    const int c0 = n0 + 4 * tn;
    if (c0 >= cout) return;
    float sc[4], bi[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
        sc[e] = (p.scale && c0 + e < cout) ? p.scale[c0 + e] : 1.f;
        bi[e] = (p.bias && c0 + e < cout) ? p.bias[c0 + e] : 0.f;
    }
    const T *res = static_cast<const T *>(p.res);
    const bool vec_ok = c0 + 4 <= cout && (out.ldc & 3) == 0 && (reinterpret_cast<uintptr_t>(out.ptr) & 15) == 0;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int m = m0 + tm + 16 * i;
        if (m >= m_total) continue;
        float y[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            y[e] = activate(fmaf(acc[i][e], sc[e], bi[e]), p.act1, p.act1_param);
            if (res && c0 + e < cout) y[e] = activate(y[e] + Elem<T>::ld(res + static_cast<size_t>(m) * p.ldc_res + c0 + e), p.act2, p.act2_param);
            if (sizeof(T) == 4 && out.tf32) y[e] = round_tf32(y[e]);
        }
        T *dst = static_cast<T *>(out.ptr) + static_cast<size_t>(m) * out.ldc + c0;
        if (vec_ok) {
            if constexpr (sizeof(T) == 4) *reinterpret_cast<float4 *>(dst) = make_float4(y[0], y[1], y[2], y[3]);
            else {
                const __half2 lo = __floats2half2_rn(y[0], y[1]), hi = __floats2half2_rn(y[2], y[3]);
                *reinterpret_cast<uint2 *>(dst) = make_uint2(*reinterpret_cast<const uint32_t *>(&lo), *reinterpret_cast<const uint32_t *>(&hi));
            }
        } else {
#pragma unroll
            for (int e = 0; e < 4; ++e) if (c0 + e < cout) Elem<T>::st(dst + e, y[e]);
        }
    }
}

// ---------------------------------------------------------------------------------------------------------------------------
// conv_fp32_kernel: the fp32 form, for plans that ask for no tensor cores and for views TMA cannot read (fp32 detection nets run
// conv_split.cuh). Same GEMM view; A and B are streams of 16-byte vectors (k = four input channels of one filter
// tap, taps in order), so a k-step of four vectors may straddle taps and a 3-channel stem wastes nothing but its pad channel.
// What bounds it is the FMA pipe (128 lanes per SM and cycle) and, close behind, the register fill from shared memory; the rest
// of its design serves the layers that do not fill the chip - a plane of 11 x 11 pixels under 768 channels is six tiles of
// pixels and one chain of 3456 products:
//  * a CTA of four warps computes tiles of 64 pixels x 64 channels, a thread 8 x 4 of them. Neighbouring lanes share the pixel
//    rows they read: a 16-byte load whose lane pairs agree takes 2.3 SM cycles, one whose lane pairs differ 4.1 (measured), so
//    per k the eight pixel values cost as much as the four channel values. Scalar FMAs: the packed form reads six registers at
//    a time and reaches 54 TFLOP/s from registers alone, the scalar one 72.
//  * the k of a tile is summed in 1..8 shares that are added in their order; how many is fixed by the layer and one image, never
//    by the batch (configure_conv_fp32). Where tiles are few a cluster takes them, a CTA each: every CTA leaves its sum in its
//    own shared memory and reduces every size-th row of the tile from all of them through distributed shared memory, in rank order:
//    deterministic, no workspace, no second launch. Where the tiles fill the chip one CTA sums them one after the other (kShares).
//  * operands stay k-contiguous in shared memory as cp.async wrote them (row pitch 20 floats: the eight rows of a load
//    fall in different banks); a ring of four k-steps, cp.async also zero-fills the padding, pad channels and ragged edges. A
//    loader thread keeps its source addresses and moves them along while its vectors stay inside one filter tap.
// Measured against the 128 x 64 tile form above: 3x3 384->384 at 11x11, three images 514 -> 46 us; YOLOv5m-352, three images
// 14.9 -> 2.9 ms a forward; YOLOv3-tiny-416, one image 3.0 -> 0.43 ms. Layers that fill the chip run at 41 TFLOP/s (3x3
// 512->512 at 38x38, eight images), where loads from shared memory and FMAs take the SM equally long; the k-step by CTAs an SM is in
// the table at configure_conv_fp32.
// ---------------------------------------------------------------------------------------------------------------------------
__device__ __forceinline__ void cp_async16(uint32_t dst, const void *src, uint32_t bytes) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}

template <bool kShares>        // one CTA sums all shares of a tile's k, one after the other (no cluster)
__global__ void __launch_bounds__(kFpThreads, 4)
conv_fp32_kernel(TView in, TView out, const float *__restrict__ w, const ConvTiledParams p) {
    constexpr int BM = kFpBM, BN = kFpBN, T = kFpThreads, PITCH = kFpPitch, LROWS = T / 4, LA = BM / LROWS, LB = BN / LROWS;
    constexpr int kStageFloats = (BM + BN) * PITCH, kCPitch = BN + 4;
    extern __shared__ __align__(16) float fp_smem[];
    const uint32_t smem = smem_u32(fp_smem);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int m_total = out.N * out.H * out.W, cout = out.C;
    const int m0 = blockIdx.x * BM, n0 = blockIdx.y * BN;
    const int splits = gridDim.z, rank = blockIdx.z;
    const int cvecs = p.cin_pad >> 2, kvecs = p.kh * p.kw * cvecs, steps = (kvecs + 3) >> 2;
    const int step0 = static_cast<int>(static_cast<long long>(steps) * rank / splits), step1 = static_cast<int>(static_cast<long long>(steps) * (rank + 1) / splits);

    // loader: vector kq of a k-step for pixels and channels lrow, lrow + LROWS, ...
    const int kq = tid & 3, lrow = tid >> 2;
    int a_pix[LA], ay[LA], ax[LA];                                // pixel index of the filter's first tap, its row and column
#pragma unroll
    for (int j = 0; j < LA; ++j) {
        const int m = m0 + lrow + LROWS * j;
        const int mm = m < m_total ? m : 0;
        const int n = mm / (out.H * out.W), rem = mm - n * out.H * out.W;
        const int oy = rem / out.W, ox = rem - oy * out.W;
        ay[j] = oy * p.sh - p.ph; ax[j] = ox * p.sw - p.pw;
        a_pix[j] = (n * in.H + ay[j]) * in.W + ax[j];
        if (m >= m_total) ay[j] = -(1 << 28);                     // a row past the last pixel is never inside the plane
    }
    int v = step0 * 4 + kq, r, s, c4;                             // next vector of this thread's column: tap (r, s), vector c4
    { const int tap = v / cvecs; c4 = v - tap * cvecs; r = tap / p.kw; s = tap - r * p.kw; }
    const float *a_src[LA], *b_src[LB]; uint32_t a_take[LA], b_take[LB];   // sources of the next step; 16 or 0 bytes of them
    auto aim = [&]() {                                            // a new filter tap: where this thread's pixels are under it
        const int dy = r * p.dh, dx = s * p.dw, dpix = dy * in.W + dx;
#pragma unroll
        for (int j = 0; j < LA; ++j) {
            const bool inside = v < kvecs && static_cast<unsigned>(ay[j] + dy) < static_cast<unsigned>(in.H) && static_cast<unsigned>(ax[j] + dx) < static_cast<unsigned>(in.W);
            a_take[j] = inside ? 16u : 0u;
            a_src[j] = static_cast<const float *>(in.ptr) + (inside ? static_cast<size_t>(a_pix[j] + dpix) * in.ldc + 4 * c4 : 0);
        }
    };
    aim();
#pragma unroll
    for (int j = 0; j < LB; ++j) {
        b_take[j] = n0 + lrow + LROWS * j < cout ? 16u : 0u;
        b_src[j] = w + (b_take[j] ? (static_cast<size_t>(n0 + lrow + LROWS * j) * kvecs + v) * 4 : 0);
    }
    const uint32_t a_dst = smem + static_cast<uint32_t>(lrow * PITCH + kq * 4) * 4u;
    const uint32_t b_dst = a_dst + static_cast<uint32_t>(BM * PITCH) * 4u;
    auto load_step = [&](int slot) {
        const uint32_t off = static_cast<uint32_t>(slot * kStageFloats) * 4u;
        const uint32_t bytes = static_cast<uint32_t>(min(16, (in.C - 4 * c4) * 4));       // pad channels of the pitch hold no data
        const bool live = v < kvecs;
#pragma unroll
        for (int j = 0; j < LA; ++j) { cp_async16(a_dst + off + static_cast<uint32_t>(LROWS * j * PITCH) * 4u, a_src[j], min(a_take[j], bytes)); a_src[j] += a_take[j]; }
#pragma unroll
        for (int j = 0; j < LB; ++j) {
            cp_async16(b_dst + off + static_cast<uint32_t>(LROWS * j * PITCH) * 4u, live ? b_src[j] : w, live ? b_take[j] : 0u);
            b_src[j] += b_take[j];
        }
        v += 4; c4 += 4;
        if (c4 >= cvecs) {
            do { c4 -= cvecs; if (++s == p.kw) { s = 0; ++r; } } while (c4 >= cvecs);
            aim();
        }
    };

    // arithmetic: a warp covers 64 pixels x 16 channels, a thread pixels tm + 8 i and channels tn + 4 j
    const int tm = (lane >> 1) & 7, tn = (lane & 1) + 2 * (lane >> 4) + 16 * warp;
    float acc[8][4];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;

    // kShares: the sum of the shares behind this one. Touched once a share, so it stays on the stack (its address is shown to an empty
    // asm): in registers it would push the addresses of the main loop out of theirs.
    float sum[kShares ? 8 : 1][4];
    int share = 0, share_end = step1;
    bool first = true;
    if constexpr (kShares) {
        asm volatile("" ::"l"(&sum[0][0]) : "memory");
        share_end = steps / p.shares;
        while (share_end == 0) share_end = static_cast<int>(static_cast<long long>(steps) * (++share + 1) / p.shares);   // (more shares than k-steps)
    }
    auto fold = [&](bool first) {                                 // this share to the sum of those before it, in their order
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) acc[i][j] = (first ? 0.f : sum[i][j]) + acc[i][j];
    };
    pdl_wait();
#pragma unroll
    for (int q = 0; q < kFpStages - 1; ++q) {
        if (step0 + q < step1) load_step(q);
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    int slot = 0;
    for (int step = step0; step < step1; ++step) {
        asm volatile("cp.async.wait_group %0;" ::"n"(kFpStages - 2) : "memory");
        __syncthreads();                            // this k-step has landed, and everybody is done with the slot loaded next
        if (step + kFpStages - 1 < step1) load_step((slot + kFpStages - 1) & (kFpStages - 1));
        asm volatile("cp.async.commit_group;" ::: "memory");
        const float *As = fp_smem + slot * kStageFloats + tm * PITCH, *Bs = fp_smem + slot * kStageFloats + (BM + tn) * PITCH;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            float4 a[8], b[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) b[j] = *reinterpret_cast<const float4 *>(Bs + 4 * j * PITCH + 4 * q);
#pragma unroll
            for (int i = 0; i < 8; ++i) a[i] = *reinterpret_cast<const float4 *>(As + 8 * i * PITCH + 4 * q);
#pragma unroll
            for (int i = 0; i < 8; ++i) {
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(a[i].x, b[j].x, acc[i][j]);
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(a[i].y, b[j].y, acc[i][j]);
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(a[i].z, b[j].z, acc[i][j]);
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(a[i].w, b[j].w, acc[i][j]);
            }
        }
        slot = (slot + 1) & (kFpStages - 1);
        if constexpr (kShares) {
            if (step + 1 == share_end) {
                fold(first);
                first = false;
                if (step + 1 < steps) {
#pragma unroll
                    for (int i = 0; i < 8; ++i)
#pragma unroll
                        for (int j = 0; j < 4; ++j) { sum[i][j] = acc[i][j]; acc[i][j] = 0.f; }
                    do share_end = static_cast<int>(static_cast<long long>(steps) * (++share + 1) / p.shares); while (share_end == step + 1);
                }
            }
        }
    }
    // Only now may the next kernel's CTAs come in: launched at the start of this one they would pile up on the SMs that have
    // room, that is on those that this layer leaves idle, and stay there.
    pdl_launch_dependents();
    // this CTA's sums -> shared memory (over the ring: everybody has to be done reading it)
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) fp_smem[(tm + 8 * i) * kCPitch + tn + 4 * j] = acc[i][j];
    if (splits > 1) cluster_sync_all(); else __syncthreads();

    // this CTA's rows of the tile: sum over the cluster, scale / bias, activation, residual (+ second activation), store
    const float *res = static_cast<const float *>(p.res);
    const bool out_vec = (out.ldc & 3) == 0 && (reinterpret_cast<uintptr_t>(out.ptr) & 15) == 0;
    const bool res_vec = res && (p.ldc_res & 3) == 0 && (reinterpret_cast<uintptr_t>(res) & 15) == 0;
    const int col = 4 * (tid & 15), c0 = n0 + col;
    if (c0 < cout) {
        float sc[4], bi[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            sc[e] = (p.scale && c0 + e < cout) ? p.scale[c0 + e] : 1.f;
            bi[e] = (p.bias && c0 + e < cout) ? p.bias[c0 + e] : 0.f;
        }
        for (int row = rank + splits * (tid >> 4); row < BM && m0 + row < m_total; row += splits * (T / 16)) {
            const int m = m0 + row;
            float y[4] = {0.f, 0.f, 0.f, 0.f};
            if (splits == 1) ld_vec(fp_smem + row * kCPitch + col, y);
            else {
                const uint32_t at = smem + static_cast<uint32_t>(row * kCPitch + col) * 4u;
                for (int q = 0; q < splits; ++q) {
                    float4 t;
                    asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(t.x), "=f"(t.y), "=f"(t.z), "=f"(t.w) : "r"(map_to_cta(at, q)) : "memory");
                    y[0] += t.x; y[1] += t.y; y[2] += t.z; y[3] += t.w;
                }
            }
            float rr[4] = {0.f, 0.f, 0.f, 0.f};
            if (res) {
                const float *rp = res + static_cast<size_t>(m) * p.ldc_res + c0;
                if (res_vec && c0 + 4 <= cout) ld_vec(rp, rr);
                else {
#pragma unroll
                    for (int e = 0; e < 4; ++e) if (c0 + e < cout) rr[e] = rp[e];
                }
            }
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                y[e] = activate(fmaf(y[e], sc[e], bi[e]), p.act1, p.act1_param);
                if (res) y[e] = activate(y[e] + rr[e], p.act2, p.act2_param);
                if (out.tf32) y[e] = round_tf32(y[e]);
            }
            float *dst = static_cast<float *>(out.ptr) + static_cast<size_t>(m) * out.ldc + c0;
            if (out_vec && c0 + 4 <= cout) st_vec(dst, y);
            else {
#pragma unroll
                for (int e = 0; e < 4; ++e) if (c0 + e < cout) dst[e] = y[e];
            }
        }
    }
    if (splits > 1) cluster_sync_all();              // nobody leaves while a peer still reads its shared memory
}

}  // namespace msnh
