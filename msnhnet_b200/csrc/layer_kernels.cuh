// Memory-bound layer kernels on channels-last tensors. One thread moves one 16-byte channel
// vector (8 fp16 / 4 fp32) whenever the channel count and pitches allow (V = Elem<T>::kVec),
// otherwise one element (V = 1). Consecutive threads walk consecutive channel vectors of the same
// pixel, so every warp access is a run of full 128-byte lines. Grids are sized by the caller as a
// multiple of the SM count and kernels use grid-stride loops.
//
// These replace src/layers/cuda/*.cu and the elementwise kernels of
// src/core/cuda/MsnhBlasGPU.cu; each kernel cites the function it stands in for.
#pragma once
#include <float.h>
#include "common.cuh"

namespace msnh {

template <typename T, int V> struct VecIO {
    __device__ __forceinline__ static void ld(const T *p, float (&v)[V]) {
        if constexpr (V == 1) v[0] = Elem<T>::ld(p); else ld_vec(p, v);
    }
    __device__ __forceinline__ static void st(T *p, const float (&v)[V]) {
        if constexpr (V == 1) Elem<T>::st(p, v[0]); else st_vec(p, v);
    }
    // store of computed values into `out`: rounds to tf32 first when the view asks for it
    __device__ __forceinline__ static void st_out(const TView &out, T *p, float (&v)[V]) {
        if constexpr (sizeof(T) == 4) {
            if (out.tf32) {
#pragma unroll
                for (int e = 0; e < V; ++e) v[e] = round_tf32(v[e]);
            }
        }
        st(p, v);
    }
};
template <typename T> __device__ __forceinline__ void st_out(const TView &out, T *p, float v) {
    Elem<T>::st(p, sizeof(T) == 4 && out.tf32 ? round_tf32(v) : v);
}

__device__ __forceinline__ size_t pix_off(const TView &t, int n, int h, int w) {
    return (static_cast<size_t>(n) * t.H + h) * t.W * static_cast<size_t>(t.ldc) + static_cast<size_t>(w) * t.ldc;
}

// ---- network input: planar fp32 CHW images -> channels-last T, pad channels written as zero ----
// (the reference uploads the planar image as is, src/net/MsnhNetBuilder.cpp:843,938)
template <typename T>
__global__ void nchw_f32_to_nhwc_kernel(const float *__restrict__ src, TView dst) {
    pdl_prologue();
    const size_t plane = static_cast<size_t>(dst.H) * dst.W;
    const size_t total = plane * dst.N;
    for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < total;
         i += static_cast<size_t>(gridDim.x) * blockDim.x) {
        const size_t n = i / plane, hw = i - n * plane;
        T *d = static_cast<T *>(dst.ptr) + i * dst.ldc;
        const float *s = src + n * dst.C * plane + hw;
        constexpr int V = Elem<T>::kVec;
        for (int c0 = 0; c0 < dst.ldc; c0 += V) {            // ldc is a multiple of one 16-byte vector
            float v[V];
#pragma unroll
            for (int e = 0; e < V; ++e) {
                v[e] = c0 + e < dst.C ? __ldg(s + static_cast<size_t>(c0 + e) * plane) : 0.f;
                if (sizeof(T) == 4 && dst.tf32) v[e] = round_tf32(v[e]);
            }
            st_vec(d + c0, v);
        }
    }
}

// ---- network input -> patch matrix of the first conv: dst[pixel][tap*cin + c] = image value under
//      tap (r,s) of output pixel `pixel`, zero outside the image and in the pad columns. One thread
//      per output pixel; reads are coalesced along the image row, the write is one contiguous row.
template <typename T>
__global__ void nchw_f32_to_patches_kernel(const float *__restrict__ src, TView dst, int cin, int H, int W, int kh, int kw,
                                           int sh, int sw, int ph, int pw, int dh, int dw) {
    pdl_prologue();
    const size_t oplane = static_cast<size_t>(dst.H) * dst.W;
    const size_t total = oplane * dst.N;
    const size_t iplane = static_cast<size_t>(H) * W;
    for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < total;
         i += static_cast<size_t>(gridDim.x) * blockDim.x) {
        const size_t n = i / oplane, rem = i - n * oplane;
        const int oy = static_cast<int>(rem / dst.W), ox = static_cast<int>(rem - static_cast<size_t>(oy) * dst.W);
        T *d = static_cast<T *>(dst.ptr) + i * dst.ldc;
        const float *s = src + n * cin * iplane;
        int k = 0;
        for (int r = 0; r < kh; ++r) {
            const int iy = oy * sh - ph + r * dh;
            for (int q = 0; q < kw; ++q) {
                const int ix = ox * sw - pw + q * dw;
                const bool in = iy >= 0 && iy < H && ix >= 0 && ix < W;
                for (int c = 0; c < cin; ++c, ++k) {
                    float v = in ? s[static_cast<size_t>(c) * iplane + static_cast<size_t>(iy) * W + ix] : 0.f;
                    if (sizeof(T) == 4 && dst.tf32) v = round_tf32(v);
                    Elem<T>::st(d + k, v);
                }
            }
        }
        for (; k < dst.ldc; ++k) Elem<T>::st(d + k, 0.f);
    }
}

// Same, for a compile-time receptive field (the 3-channel 3x3 stem of every detector here): the
// whole patch row lives in registers and leaves as 16-byte vectors.
template <typename T, int CIN, int KH, int KW>
__global__ void nchw_f32_to_patches_fixed_kernel(const float *__restrict__ src, TView dst, int H, int W,
                                                 int sh, int sw, int ph, int pw, int dh, int dw) {
    pdl_prologue();
    constexpr int K = CIN * KH * KW;
    constexpr int V = Elem<T>::kVec;
    constexpr int KP = (K + 15) / 16 * 16;
    const size_t oplane = static_cast<size_t>(dst.H) * dst.W;
    const size_t total = oplane * dst.N;
    const size_t iplane = static_cast<size_t>(H) * W;
    for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < total;
         i += static_cast<size_t>(gridDim.x) * blockDim.x) {
        const size_t n = i / oplane, rem = i - n * oplane;
        const int oy = static_cast<int>(rem / dst.W), ox = static_cast<int>(rem - static_cast<size_t>(oy) * dst.W);
        const float *s = src + n * CIN * iplane;
        float v[KP];
#pragma unroll
        for (int k = K; k < KP; ++k) v[k] = 0.f;
#pragma unroll
        for (int r = 0; r < KH; ++r) {
            const int iy = oy * sh - ph + r * dh;
#pragma unroll
            for (int q = 0; q < KW; ++q) {
                const int ix = ox * sw - pw + q * dw;
                const bool in = iy >= 0 && iy < H && ix >= 0 && ix < W;
                const size_t off = static_cast<size_t>(in ? iy : 0) * W + (in ? ix : 0);
#pragma unroll
                for (int c = 0; c < CIN; ++c) {
                    float x = in ? __ldg(s + static_cast<size_t>(c) * iplane + off) : 0.f;
                    if (sizeof(T) == 4 && dst.tf32) x = round_tf32(x);
                    v[(r * KW + q) * CIN + c] = x;
                }
            }
        }
        T *d = static_cast<T *>(dst.ptr) + i * dst.ldc;
#pragma unroll
        for (int k = 0; k < KP; k += V) {
            float t[V];
#pragma unroll
            for (int e = 0; e < V; ++e) t[e] = v[k + e];
            st_vec(d + k, t);
        }
    }
}

// Row patches: for every image row and output column the kw pixels under a filter row, [row][output column][pixel * C + c], padded with
// zeros; a conv reads them as kh x 1. A CTA stages `rows` image rows in shared memory, their padding included, and writes the patches of a row as
// one stream of 16-byte vectors; a vector's place inside a patch decides what it gathers, and the number of threads is a multiple of the
// vectors of a patch, so that a thread's gather is the same throughout. Bound by the writes: 32 images of 224 x 224 under a 7-wide
// filter at stride 2 are 77 MB.
template <typename T>
__global__ void __launch_bounds__(256)
nchw_f32_to_row_patches_kernel(const float *__restrict__ src, TView dst, int C, int H, int W, int kw, int sw, int pw, int rows) {
    constexpr int V = Elem<T>::kVec;
    extern __shared__ float row_smem[];
    const int pieces = dst.ldc / V, threads = blockDim.x / pieces * pieces, t = threadIdx.x;
    const int width = pw + max(W, (dst.W - 1) * sw + kw - pw);
    int at[V];                                     // offset of a vector's values in the staged row (output column 0); negative: pad channel
    const int piece = t % pieces;
#pragma unroll
    for (int e = 0; e < V; ++e) {
        const int v = piece * V + e, s = v / C;
        at[e] = s < kw ? (v - s * C) * width + s : -1;
    }
    const int warp = t >> 5, lane = t & 31, warps = blockDim.x >> 5;
    pdl_prologue();
    for (int row0 = blockIdx.x * rows; row0 < dst.N * H; row0 += gridDim.x * rows) {
        const int here = min(rows, dst.N * H - row0);
        for (int q = warp; q < here * C; q += warps) {                 // a warp per row and channel
            const int r = q / C, c = q - r * C, n = (row0 + r) / H, y = row0 + r - n * H;
            const float *s = src + (static_cast<size_t>(n * C + c) * H + y) * W;
            float *to = row_smem + q * width;
#pragma unroll 4
            for (int i = lane; i < width; i += 32) {
                const int x = i - pw;
                const float v = x >= 0 && x < W ? __ldg(s + x) : 0.f;
                to[i] = dst.tf32 ? round_tf32(v) : v;
            }
        }
        __syncthreads();
        if (t < threads)
            for (int r = 0; r < here; ++r) {
                T *d = static_cast<T *>(dst.ptr) + static_cast<size_t>(row0 + r) * dst.W * dst.ldc;
                const float *from = row_smem + r * C * width;
#pragma unroll 2
                for (int i = t; i < dst.W * pieces; i += threads) {
                    const int x = i / pieces * sw;
                    float v[V];
#pragma unroll
                    for (int e = 0; e < V; ++e) v[e] = at[e] >= 0 ? from[at[e] + x] : 0.f;
                    st_vec(d + static_cast<size_t>(i) * V, v);
                }
            }
        __syncthreads();
    }
}

// The same for fp16 and the 3x3x3 stem without dilation. The kernel above converts every image value nine times and reads it as
// often through L1 (27 loads and conversions per pixel: 85 us for eight images of 608 x 608, 225 MB). Here a CTA of 128 threads
// stages the input rows of 128 x 4 output pixels in shared memory as interleaved fp16 pixels, so that the nine values of a filter
// row are contiguous, and a thread puts a pixel's 32 columns together from 15 words with funnel shifts: 51 us. kSw: horizontal stride.
constexpr int kPatchTx = 128, kPatchTy = 4;
template <int kSw>
__global__ void __launch_bounds__(kPatchTx)
nchw_f32_to_patches3_kernel(const float *__restrict__ src, TView dst, int H, int W, int sh, int ph, int pw) {
    constexpr int kCols = ((kPatchTx - 1) * kSw + 3 + 1) / 2 * 2, kPitch = kCols * 3 / 2 + 1;       // pixels, words per staged row
    __shared__ uint32_t rows[(kPatchTy - 1) * 2 + 3][kPitch];
    __shared__ uint4 staged[kPatchTx / 32][128];           // a warp's 32 patches, 16-byte pieces XOR-swizzled against bank conflicts
    pdl_prologue();
    const int ox0 = blockIdx.x * kPatchTx, oy0 = blockIdx.y * kPatchTy, n = blockIdx.z;
    const int ix0 = ox0 * kSw - pw, iy0 = oy0 * sh - ph, n_rows = (kPatchTy - 1) * sh + 3;
    const size_t plane = static_cast<size_t>(H) * W;
    const float *s = src + static_cast<size_t>(n) * 3 * plane;
    for (int i = threadIdx.x; i < n_rows * (kCols / 2); i += kPatchTx) {
        const int r = i / (kCols / 2), pair = i - r * (kCols / 2);
        const int iy = iy0 + r, ix = ix0 + 2 * pair;
        const bool row_ok = static_cast<unsigned>(iy) < static_cast<unsigned>(H);
        const bool ok0 = row_ok && static_cast<unsigned>(ix) < static_cast<unsigned>(W), ok1 = row_ok && static_cast<unsigned>(ix + 1) < static_cast<unsigned>(W);
        float v[6];
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const float *p = s + c * plane + static_cast<size_t>(row_ok ? iy : 0) * W;
            v[c] = ok0 ? __ldg(p + ix) : 0.f;
            v[3 + c] = ok1 ? __ldg(p + ix + 1) : 0.f;
        }
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            const __half2 h = __floats2half2_rn(v[2 * k], v[2 * k + 1]);
            rows[r][3 * pair + k] = *reinterpret_cast<const uint32_t *>(&h);
        }
    }
    __syncthreads();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, swz = (lane >> 1) & 3;
    uint4 *mine = staged[warp];
    const int first = 3 * kSw * static_cast<int>(threadIdx.x), word = first >> 1, shift = (first & 1) * 16;      // first half of a filter row
    for (int y = 0; y < kPatchTy && oy0 + y < dst.H; ++y) {
        uint32_t o[16];
#pragma unroll
        for (int r = 0; r < 3; ++r) {
            uint32_t a[5];
#pragma unroll
            for (int k = 0; k < 5; ++k) a[k] = rows[y * sh + r][word + k];
            if (r != 1) {                          // halves 0..8 (18..26) of the patch: whole words, then a low half
                const int at = r == 0 ? 0 : 9;
#pragma unroll
                for (int k = 0; k < 4; ++k) o[at + k] = __funnelshift_rc(a[k], a[k + 1], shift);
                o[at + 4] = (a[4] >> shift) & 0xffffu;
            } else {                               // halves 9..17: a high half, then whole words
                o[4] |= (a[0] >> shift) << 16;
#pragma unroll
                for (int k = 0; k < 4; ++k) o[5 + k] = __funnelshift_rc(a[k], a[k + 1], 16 + shift);
            }
        }
        o[14] = o[15] = 0u;
        // out through shared memory, so that a warp writes 512 contiguous bytes at a time (16 bytes every 64 make L2 merge half sectors)
        __syncwarp();
#pragma unroll
        for (int k = 0; k < 4; ++k) mine[lane * 4 + (k ^ swz)] = make_uint4(o[4 * k], o[4 * k + 1], o[4 * k + 2], o[4 * k + 3]);
        __syncwarp();
        uint4 *d = reinterpret_cast<uint4 *>(static_cast<__half *>(dst.ptr) + ((static_cast<size_t>(n) * dst.H + oy0 + y) * dst.W + ox0 + 32 * warp) * 32);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const int pix = 8 * k + (lane >> 2);
            if (ox0 + 32 * warp + pix < dst.W) d[32 * k + lane] = mine[pix * 4 + ((lane & 3) ^ ((pix >> 1) & 3))];
        }
    }
}

// ---- read-back for outputs and parity dumps: channels-last T -> planar fp32 ----
template <typename T>
__global__ void nhwc_to_nchw_f32_kernel(TView src, float *__restrict__ dst) {
    pdl_prologue();
    const size_t plane = static_cast<size_t>(src.H) * src.W;
    const size_t total = plane * src.N * src.C;
    for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < total;
         i += static_cast<size_t>(gridDim.x) * blockDim.x) {
        const size_t hw = i % plane;
        const size_t nc = i / plane;
        const size_t c = nc % src.C, n = nc / src.C;
        dst[i] = Elem<T>::ld(static_cast<const T *>(src.ptr) + (n * plane + hw) * src.ldc + c);
    }
}

// ---- y = act(x * scale[c] + bias[c]) : standalone BatchNorm (folded), activation, copy ----
// (BatchNormLayer::forwardGPU's copy+norm+scale+bias+activation, src/layers/MsnhBatchNormLayer.cpp:355-358;
//  ActivationsGPU::gpuActivateArray, src/layers/cuda/MsnhActivationsGPU.cu:5-199;
//  BlasGPU copy kernels used by route, src/core/cuda/MsnhBlasGPU.cu:5-66)
template <typename T, int V>
__global__ void scale_bias_act_kernel(TView in, TView out, const float *__restrict__ scale,
                                      const float *__restrict__ bias, int act, float act_param) {
    pdl_prologue();
    constexpr int U = 4;                         // independent vectors in flight per thread
    const int cv = in.C / V;
    const size_t total = static_cast<size_t>(in.N) * in.H * in.W * cv;
    const size_t stride = static_cast<size_t>(gridDim.x) * blockDim.x;
    for (size_t i0 = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i0 < total; i0 += U * stride) {
        float v[U][V];
        size_t pix[U]; int c[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const size_t i = i0 + u * stride;
            pix[u] = i / cv; c[u] = static_cast<int>(i - pix[u] * cv) * V;
            if (i < total) VecIO<T, V>::ld(static_cast<const T *>(in.ptr) + pix[u] * in.ldc + c[u], v[u]);
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            if (i0 + u * stride >= total) break;
            if (scale) {
#pragma unroll
                for (int e = 0; e < V; ++e) v[u][e] = fmaf(v[u][e], __ldg(scale + c[u] + e), __ldg(bias + c[u] + e));
            }
            switch (act) {
                case MSNH_ACT_NONE: break;
                case MSNH_ACT_LEAKY:
#pragma unroll
                    for (int e = 0; e < V; ++e) v[u][e] = v[u][e] > 0.f ? v[u][e] : act_param * v[u][e];
                    break;
                case MSNH_ACT_RELU:
#pragma unroll
                    for (int e = 0; e < V; ++e) v[u][e] = v[u][e] > 0.f ? v[u][e] : 0.f;
                    break;
                default:
#pragma unroll
                    for (int e = 0; e < V; ++e) v[u][e] = activate(v[u][e], act, act_param);
                    break;
            }
            VecIO<T, V>::st_out(out, static_cast<T *>(out.ptr) + pix[u] * out.ldc + c[u], v[u]);
        }
    }
}

// ---- y = act(a (op) b [...]) : shortcut / block sums / varop ----
// (BlasGPU::gpuAxpy chains in Route addModel 1 and the block layers, src/core/cuda/MsnhBlasGPU.cu:40-66;
//  BlasGPU::gpuArithmetic, src/core/cuda/MsnhBlasGPU.cu:68-140)
template <typename T, int V>
__global__ void add_n_kernel(AddInputs ins, TView out, int act, float act_param) {
    pdl_prologue();
    const int cv = out.C / V;
    const size_t total = static_cast<size_t>(out.N) * out.H * out.W * cv;
    // (32-bit index arithmetic: the plan refuses tensors of 2^31 or more vectors)
    for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < static_cast<unsigned>(total); i += gridDim.x * blockDim.x) {
        const unsigned pix = i / cv;
        const int c = static_cast<int>(i - pix * cv) * V;
        float acc[V];
#pragma unroll
        for (int e = 0; e < V; ++e) acc[e] = 0.f;
        for (int k = 0; k < ins.n; ++k) {
            float v[V];
            VecIO<T, V>::ld(static_cast<const T *>(ins.ptr[k]) + static_cast<size_t>(pix) * ins.ldc[k] + c, v);
#pragma unroll
            for (int e = 0; e < V; ++e) acc[e] += v[e];
        }
#pragma unroll
        for (int e = 0; e < V; ++e) acc[e] = activate(acc[e], act, act_param);
        VecIO<T, V>::st_out(out, static_cast<T *>(out.ptr) + static_cast<size_t>(pix) * out.ldc + c, acc);
    }
}

template <typename T, int V>
__global__ void binary_kernel(TView a, const void *bptr, int ldb, float cval, int kind, TView out) {
    pdl_prologue();
    const int cv = out.C / V;
    const size_t total = static_cast<size_t>(out.N) * out.H * out.W * cv;
    // (32-bit index arithmetic: the plan refuses tensors of 2^31 or more vectors)
    for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < static_cast<unsigned>(total); i += gridDim.x * blockDim.x) {
        const unsigned pix = i / cv;
        const int c = static_cast<int>(i - pix * cv) * V;
        float x[V], y[V];
        VecIO<T, V>::ld(static_cast<const T *>(a.ptr) + static_cast<size_t>(pix) * a.ldc + c, x);
        if (bptr) VecIO<T, V>::ld(static_cast<const T *>(bptr) + static_cast<size_t>(pix) * ldb + c, y);
        else {
#pragma unroll
            for (int e = 0; e < V; ++e) y[e] = cval;
        }
#pragma unroll
        for (int e = 0; e < V; ++e) {
            switch (kind) {
                case MSNH_BIN_ADD:     x[e] = x[e] + y[e]; break;
                case MSNH_BIN_SUB:     x[e] = x[e] - y[e]; break;
                case MSNH_BIN_SUB_INV: x[e] = y[e] - x[e]; break;
                case MSNH_BIN_MUL:     x[e] = x[e] * y[e]; break;
                case MSNH_BIN_DIV:     x[e] = x[e] / y[e]; break;
                case MSNH_BIN_DIV_INV: x[e] = y[e] / x[e]; break;
                // one-operand forms (y = the layer's constant): the library functions the reference calls
                case MSNH_UN_ABS:      x[e] = fabsf(x[e]); break;
                case MSNH_UN_ACOS:     x[e] = acosf(x[e]); break;
                case MSNH_UN_ASIN:     x[e] = asinf(x[e]); break;
                case MSNH_UN_ATAN:     x[e] = atanf(x[e]); break;
                case MSNH_UN_COS:      x[e] = cosf(x[e]); break;
                case MSNH_UN_COSH:     x[e] = coshf(x[e]); break;
                case MSNH_UN_SIN:      x[e] = sinf(x[e]); break;
                case MSNH_UN_SINH:     x[e] = sinhf(x[e]); break;
                case MSNH_UN_TAN:      x[e] = tanf(x[e]); break;
                case MSNH_UN_TANH:     x[e] = tanhf(x[e]); break;
                case MSNH_UN_EXP:      x[e] = expf(x[e]); break;
                case MSNH_UN_POW:      x[e] = powf(x[e], y[e]); break;
                case MSNH_UN_LOG:      x[e] = logf(x[e]); break;
                case MSNH_UN_LOG10:    x[e] = log10f(x[e]); break;
                case MSNH_UN_SQRT:     x[e] = sqrtf(x[e]); break;
                default: break;
            }
        }
        VecIO<T, V>::st_out(out, static_cast<T *>(out.ptr) + static_cast<size_t>(pix) * out.ldc + c, x);
    }
}

// ---- max pool: window max over the taps that fall inside the plane ----
// (maxpoolNormalKernel, src/layers/cuda/MsnhMaxPoolLayerGPU.cu:35-91: padding never wins the max)
template <typename T, int V>
__global__ void maxpool_kernel(TView in, TView out, int kh, int kw, int sh, int sw, int ph, int pw) {
    pdl_prologue();
    const int cv = out.C / V;
    const size_t total = static_cast<size_t>(out.N) * out.H * out.W * cv;
    // (32-bit index arithmetic: the plan refuses tensors of 2^31 or more vectors)
    for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < static_cast<unsigned>(total); i += gridDim.x * blockDim.x) {
        unsigned pix = i / cv;
        const int c = static_cast<int>(i - pix * cv) * V;
        const int ow = static_cast<int>(pix % out.W); pix /= out.W;
        const int oh = static_cast<int>(pix % out.H);
        const int n  = static_cast<int>(pix / out.H);
        float m[V];
#pragma unroll
        for (int e = 0; e < V; ++e) m[e] = -FLT_MAX;
        const int h0 = oh * sh - ph, w0 = ow * sw - pw;
        const int hb = max(h0, 0), he = min(h0 + kh, in.H);
        const int wb = max(w0, 0), we = min(w0 + kw, in.W);
        for (int h = hb; h < he; ++h)
            for (int w = wb; w < we; ++w) {
                float v[V];
                VecIO<T, V>::ld(static_cast<const T *>(in.ptr) + pix_off(in, n, h, w) + c, v);
#pragma unroll
                for (int e = 0; e < V; ++e) m[e] = fmaxf(m[e], v[e]);
            }
        VecIO<T, V>::st_out(out, static_cast<T *>(out.ptr) + pix_off(out, n, oh, ow) + c, m);
    }
}

// 16 bytes of elements rounded to tf32 when the view asks for it
template <typename T> __device__ __forceinline__ uint4 round_out16(const TView &out, uint4 v) {
    if constexpr (sizeof(T) == 4) {
        if (out.tf32) {
            v.x = __float_as_uint(round_tf32(__uint_as_float(v.x))); v.y = __float_as_uint(round_tf32(__uint_as_float(v.y)));
            v.z = __float_as_uint(round_tf32(__uint_as_float(v.z))); v.w = __float_as_uint(round_tf32(__uint_as_float(v.w)));
        }
    }
    return v;
}
// maximum of two 16-byte vectors of elements
template <typename T>
__device__ __forceinline__ uint4 vec_max16(uint4 a, uint4 b) {
    uint4 r;
    if constexpr (sizeof(T) == 2) {
        const __half2 *x = reinterpret_cast<const __half2 *>(&a), *y = reinterpret_cast<const __half2 *>(&b);
        __half2 *z = reinterpret_cast<__half2 *>(&r);
#pragma unroll
        for (int e = 0; e < 4; ++e) z[e] = __hmax2(x[e], y[e]);
    } else {
        const float *x = reinterpret_cast<const float *>(&a), *y = reinterpret_cast<const float *>(&b);
        float *z = reinterpret_cast<float *>(&r);
#pragma unroll
        for (int e = 0; e < 4; ++e) z[e] = fmaxf(x[e], y[e]);
    }
    return r;
}
// 2 x 2 pools, vector channels: CTAs walk output rows with a power-of-two grid of (channel
// vector, pixel) threads, so that no division is left per value, the window's loads are independent of one another, and the
// maximum is taken on the stored type. 64 channels at 320 x 320, 16 images, fp16: 78 -> 54 us for 262 MB (3 x 3 windows gain
// nothing from it and stay with the kernel above).
template <typename T>
__global__ void maxpool2_rows_kernel(TView in, TView out, int sh, int sw, int ph, int pw, int lanes_c_log2) {
    constexpr int V = Elem<T>::kVec, K = 2;
    pdl_prologue();
    const int cv = out.C / V, rows = out.N * out.H;
    const int tc = threadIdx.x & ((1 << lanes_c_log2) - 1), tp = threadIdx.x >> lanes_c_log2;
    const int step_c = 1 << lanes_c_log2, step_p = blockDim.x >> lanes_c_log2;
    uint4 lowest;
    if constexpr (sizeof(T) == 2) lowest = make_uint4(0xfc00fc00u, 0xfc00fc00u, 0xfc00fc00u, 0xfc00fc00u);       // -FLT_MAX as fp16: -inf
    else lowest = make_uint4(0xff7fffffu, 0xff7fffffu, 0xff7fffffu, 0xff7fffffu);
    for (int row = blockIdx.x; row < rows; row += gridDim.x) {
        const int n = row / out.H, oh = row - n * out.H, h0 = oh * sh - ph;
        const T *img = static_cast<const T *>(in.ptr) + static_cast<size_t>(n) * in.H * in.W * in.ldc;
        T *dst = static_cast<T *>(out.ptr) + pix_off(out, n, oh, 0);
        for (int ow = tp; ow < out.W; ow += step_p) {
            const int w0 = ow * sw - pw;
            for (int c = tc; c < cv; c += step_c) {
                uint4 v[K * K];
#pragma unroll
                for (int r = 0; r < K; ++r)
#pragma unroll
                    for (int q = 0; q < K; ++q) {
                        const bool inside = static_cast<unsigned>(h0 + r) < static_cast<unsigned>(in.H) && static_cast<unsigned>(w0 + q) < static_cast<unsigned>(in.W);
                        v[r * K + q] = inside ? *reinterpret_cast<const uint4 *>(img + (static_cast<size_t>(h0 + r) * in.W + w0 + q) * in.ldc + c * V) : lowest;
                    }
                uint4 m = lowest;
#pragma unroll
                for (int k = 0; k < K * K; ++k) m = vec_max16<T>(m, v[k]);
                *reinterpret_cast<uint4 *>(dst + static_cast<size_t>(ow) * out.ldc + c * V) = round_out16<T>(out, m);
            }
        }
    }
}

// Stride-1 max pool that keeps the plane size (the SPP pools: 5x5 / 9x9 / 13x13 over a 19x19 plane):
// a block stages the whole plane of G 16-byte channel groups of one image in shared memory and takes
// the window max as a row pass followed by a column pass (kh + kw reads per output instead of kh * kw).
// Shared memory: 2 * H * W * G * 16 bytes.
// Up to three such pools over the same input (the SPP block: one tensor through a 5, a 9 and a 13 window) run as one
// launch: the plane is staged once and every pool takes its own row pass and column pass over it.
template <typename T>
__global__ void maxpool_plane_kernel(TView in, const __grid_constant__ PoolSet ps, int G) {
    pdl_prologue();
    extern __shared__ uint4 plane_smem[];
    constexpr int V = 16 / static_cast<int>(sizeof(T));
    const int hw = in.H * in.W;
    uint4 *src = plane_smem, *rowmax = plane_smem + hw * G;
    const int cv = in.C / V;
    const int groups = (cv + G - 1) / G;
    for (int blk = blockIdx.x; blk < in.N * groups; blk += gridDim.x) {
        const int n = blk / groups, g0 = (blk - n * groups) * G;
        const int ng = min(G, cv - g0);
        const T *ibase = static_cast<const T *>(in.ptr) + pix_off(in, n, 0, 0) + g0 * V;
        for (int i = threadIdx.x; i < hw * ng; i += blockDim.x) {
            const int pix = i / ng, g = i - pix * ng;
            src[pix * G + g] = *reinterpret_cast<const uint4 *>(ibase + static_cast<size_t>(pix) * in.ldc + g * V);
        }
        __syncthreads();
#pragma unroll 1
        for (int q = 0; q < ps.n; ++q) {
            const TView &out = ps.out[q];
            const int kh = ps.kh[q], kw = ps.kw[q], ph = ps.ph[q], pw = ps.pw[q];
            T *obase = static_cast<T *>(out.ptr) + pix_off(out, n, 0, 0) + g0 * V;
            for (int i = threadIdx.x; i < hw * ng; i += blockDim.x) {
                const int pix = i / ng, g = i - pix * ng;
                const int h = pix / in.W, w = pix - h * in.W;
                const int wb = max(w - pw, 0), we = min(w - pw + kw, in.W);
                uint4 m = src[(h * in.W + wb) * G + g];
                for (int x = wb + 1; x < we; ++x) m = vec_max16<T>(m, src[(h * in.W + x) * G + g]);
                rowmax[pix * G + g] = m;
            }
            __syncthreads();
            for (int i = threadIdx.x; i < hw * ng; i += blockDim.x) {
                const int pix = i / ng, g = i - pix * ng;
                const int h = pix / in.W, w = pix - h * in.W;
                const int hb = max(h - ph, 0), he = min(h - ph + kh, in.H);
                uint4 m = rowmax[(hb * in.W + w) * G + g];
                for (int y = hb + 1; y < he; ++y) m = vec_max16<T>(m, rowmax[(y * in.W + w) * G + g]);
                *reinterpret_cast<uint4 *>(obase + static_cast<size_t>(pix) * out.ldc + g * V) = round_out16<T>(out, m);
            }
            __syncthreads();
        }
    }
}

// ---- local / global average pool: mean over the valid taps ----
// (localAvgPoolNormalKernel, src/layers/cuda/MsnhLocalAvgPoolLayerGPU.cu:5-79)
// Latency bounds it: a classifier's global pool is some hundred vectors of outputs with a chain of 49 loads each. Eight loads are
// in flight at a time and small pools run as one-warp blocks, so that the vectors spread over the SMs: a call of
// MobileNetV2 with one image (1280 channels of 7x7) 290 -> 285 us, of ResNet-18 fp32 243 -> 239.
template <typename T, int V>
__global__ void avgpool_kernel(TView in, TView out, int kh, int kw, int sh, int sw, int ph, int pw) {
    pdl_prologue();
    const int cv = out.C / V;
    const size_t total = static_cast<size_t>(out.N) * out.H * out.W * cv;
    // (32-bit index arithmetic: the plan refuses tensors of 2^31 or more vectors)
    for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < static_cast<unsigned>(total); i += gridDim.x * blockDim.x) {
        unsigned pix = i / cv;
        const int c = static_cast<int>(i - pix * cv) * V;
        const int ow = static_cast<int>(pix % out.W); pix /= out.W;
        const int oh = static_cast<int>(pix % out.H);
        const int n  = static_cast<int>(pix / out.H);
        float s[V];
#pragma unroll
        for (int e = 0; e < V; ++e) s[e] = 0.f;
        const int h0 = oh * sh - ph, w0 = ow * sw - pw;
        const int hb = max(h0, 0), he = min(h0 + kh, in.H);
        const int wb = max(w0, 0), we = min(w0 + kw, in.W);
        // taps in row order, eight loads in flight
        const int taps = max(he - hb, 0) * max(we - wb, 0), cols = we - wb;
        const T *at = static_cast<const T *>(in.ptr) + pix_off(in, n, hb, wb) + c;
        for (int t = 0, x = 0; t < taps; t += 8) {
            float v[8][V];
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                if (t + k < taps) VecIO<T, V>::ld(at, v[k]);
                at += in.ldc;
                if (++x == cols) { x = 0; at += static_cast<size_t>(in.W - cols) * in.ldc; }
            }
#pragma unroll
            for (int k = 0; k < 8; ++k)
                if (t + k < taps) {
#pragma unroll
                    for (int e = 0; e < V; ++e) s[e] += v[k][e];
                }
        }
        const float cnt = static_cast<float>(max(he - hb, 0) * max(we - wb, 0));
#pragma unroll
        for (int e = 0; e < V; ++e) s[e] = s[e] / cnt;
        VecIO<T, V>::st_out(out, static_cast<T *>(out.ptr) + pix_off(out, n, oh, ow) + c, s);
    }
}

// ---- nearest upsample: out[h][w] = scale * in[h/sh][w/sw] ----
// (upSampleKernel after a zero fill, src/core/cuda/MsnhBlasGPU.cu:541-578)
template <typename T, int V>
__global__ void upsample_kernel(TView in, TView out, int sh, int sw, float scale) {
    pdl_prologue();
    const int cv = out.C / V;
    const size_t total = static_cast<size_t>(out.N) * out.H * out.W * cv;
    // (32-bit index arithmetic: the plan refuses tensors of 2^31 or more vectors)
    for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < static_cast<unsigned>(total); i += gridDim.x * blockDim.x) {
        unsigned pix = i / cv;
        const int c = static_cast<int>(i - pix * cv) * V;
        const int ow = static_cast<int>(pix % out.W); pix /= out.W;
        const int oh = static_cast<int>(pix % out.H);
        const int n  = static_cast<int>(pix / out.H);
        float v[V];
        VecIO<T, V>::ld(static_cast<const T *>(in.ptr) + pix_off(in, n, oh / sh, ow / sw) + c, v);
        if (scale != 1.f) {
#pragma unroll
            for (int e = 0; e < V; ++e) v[e] *= scale;
        }
        VecIO<T, V>::st_out(out, static_cast<T *>(out.ptr) + pix_off(out, n, oh, ow) + c, v);
    }
}

// ---- strided slice: out[c][h][w] = in[c*s0+o0][h*s1+o1][w*s2+o2] ----
// (sliceKernel, src/layers/cuda/MsnhSliceLayerGPU.cu:5-41)
template <typename T>
__global__ void slice_kernel(TView in, TView out, int o0, int s0, int o1, int s1, int o2, int s2) {
    pdl_prologue();
    const int total = out.N * out.H * out.W;                 // one thread per output pixel
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < total; i += gridDim.x * blockDim.x) {
        int pix = i;
        const int ow = pix % out.W; pix /= out.W;
        const int oh = pix % out.H;
        const int n  = pix / out.H;
        const T *src = static_cast<const T *>(in.ptr) + pix_off(in, n, oh * s1 + o1, ow * s2 + o2) + o0;
        T *dst = static_cast<T *>(out.ptr) + pix_off(out, n, oh, ow);
        for (int c = 0; c < out.C; ++c) {
            if constexpr (sizeof(T) == 4) dst[c] = out.tf32 ? round_tf32(src[c * s0]) : src[c * s0]; else dst[c] = src[c * s0];
        }
    }
}

// Up to four stride-2 spatial slices of one image-like tensor whose results sit side by side in one concat
// buffer (the "Focus" stem of YOLOv5: src/layers/MsnhSliceLayer.cpp + RouteLayer, models/yolov5m/yolov5m.msnhnet:6-58)
// as one pass: a thread loads the 16-byte pixels the slices pick from its 2x2 input block and writes the output
// pixel's channel groups. C = channels per slice (compile time, so the output pixel stays in registers).
template <typename T, int C>
__global__ void focus_kernel(TView in, TView out, FocusParams fp) {
    pdl_prologue();
    constexpr int V = Elem<T>::kVec;
    constexpr int OUTV = (4 * C + V - 1) / V;             // 16-byte vectors of the output pixel that the slices touch
    const int total = out.N * out.H * out.W;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < total; i += gridDim.x * blockDim.x) {
        int pix = i;
        const int ow = pix % out.W; pix /= out.W;
        const int oh = pix % out.H;
        const int n  = pix / out.H;
        float x[4][V];
#pragma unroll
        for (int k = 0; k < 4; ++k)
            if (k < fp.n) ld_vec(static_cast<const T *>(in.ptr) + pix_off(in, n, oh * 2 + fp.o1[k], ow * 2 + fp.o2[k]), x[k]);
        float y[OUTV * V];
#pragma unroll
        for (int e = 0; e < OUTV * V; ++e) y[e] = 0.f;
#pragma unroll
        for (int k = 0; k < 4; ++k)
            if (k < fp.n) {
#pragma unroll
                for (int c = 0; c < C; ++c) y[k * C + c] = x[k][c];
            }
        T *dst = static_cast<T *>(out.ptr) + pix_off(out, n, oh, ow);
#pragma unroll
        for (int q = 0; q < OUTV; ++q) {
            float v[V];
#pragma unroll
            for (int e = 0; e < V; ++e) v[e] = y[q * V + e];
            VecIO<T, V>::st_out(out, dst + q * V, v);
        }
    }
}
// The same straight from the network input as the caller hands it over (planar fp32, [N][C][H][W]): where the image
// feeds nothing but those slices, the channels-last copy of the image is never written.
template <typename T, int C>
__global__ void focus_planar_kernel(const float *__restrict__ src, int H, int W, TView out, FocusParams fp) {
    pdl_prologue();
    constexpr int V = Elem<T>::kVec;
    constexpr int OUTV = (4 * C + V - 1) / V;
    const int total = out.N * out.H * out.W;
    const size_t plane = static_cast<size_t>(H) * W;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < total; i += gridDim.x * blockDim.x) {
        int pix = i;
        const int ow = pix % out.W; pix /= out.W;
        const int oh = pix % out.H;
        const int n  = pix / out.H;
        float y[OUTV * V];
#pragma unroll
        for (int e = 0; e < OUTV * V; ++e) y[e] = 0.f;
        const float *img = src + static_cast<size_t>(n) * C * plane;
#pragma unroll
        for (int k = 0; k < 4; ++k)
            if (k < fp.n) {
                const size_t off = static_cast<size_t>(oh * 2 + fp.o1[k]) * W + (ow * 2 + fp.o2[k]);
#pragma unroll
                for (int c = 0; c < C; ++c) y[k * C + c] = __ldg(img + c * plane + off);
            }
        T *dst = static_cast<T *>(out.ptr) + pix_off(out, n, oh, ow);
#pragma unroll
        for (int q = 0; q < OUTV; ++q) {
            float v[V];
#pragma unroll
            for (int e = 0; e < V; ++e) v[e] = y[q * V + e];
            VecIO<T, V>::st_out(out, dst + q * V, v);
        }
    }
}

// ---- constant padding ----
// (paddingKernel, src/layers/cuda/MsnhPaddingLayerGPU.cu:5-53)
template <typename T, int V>
__global__ void pad_kernel(TView in, TView out, int top, int left, float val) {
    pdl_prologue();
    const int cv = out.C / V;
    const size_t total = static_cast<size_t>(out.N) * out.H * out.W * cv;
    // (32-bit index arithmetic: the plan refuses tensors of 2^31 or more vectors)
    for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < static_cast<unsigned>(total); i += gridDim.x * blockDim.x) {
        unsigned pix = i / cv;
        const int c = static_cast<int>(i - pix * cv) * V;
        const int ow = static_cast<int>(pix % out.W); pix /= out.W;
        const int oh = static_cast<int>(pix % out.H);
        const int n  = static_cast<int>(pix / out.H);
        const int ih = oh - top, iw = ow - left;
        float v[V];
        if (ih >= 0 && ih < in.H && iw >= 0 && iw < in.W)
            VecIO<T, V>::ld(static_cast<const T *>(in.ptr) + pix_off(in, n, ih, iw) + c, v);
        else {
#pragma unroll
            for (int e = 0; e < V; ++e) v[e] = val;
        }
        VecIO<T, V>::st_out(out, static_cast<T *>(out.ptr) + pix_off(out, n, oh, ow) + c, v);
    }
}

// ---- softmax over `len` consecutive channel-major values per (image, group): one warp per row,
//      warp-shuffle max and sum ----
// (softmaxKernel, src/core/cuda/MsnhBlasGPU.cu:456-499, without its int truncation of the max)
// The row is addressed in the reference's planar order: element j of group g of image n is
// channel (g*len + j) / (H*W), pixel (g*len + j) % (H*W).
template <typename T>
__global__ void softmax_kernel(TView in, TView out, int groups, float temperature) {
    pdl_prologue();
    const int warps_per_block = blockDim.x >> 5;
    const int lane = threadIdx.x & 31;
    const size_t plane = static_cast<size_t>(in.H) * in.W;
    const size_t per_img = plane * in.C;
    const size_t len = per_img / groups;
    const size_t rows = static_cast<size_t>(in.N) * groups;
    for (size_t row = blockIdx.x * static_cast<size_t>(warps_per_block) + (threadIdx.x >> 5); row < rows;
         row += static_cast<size_t>(gridDim.x) * warps_per_block) {
        const size_t n = row / groups, g = row - n * groups;
        auto addr = [&](const TView &t, size_t j) {
            const size_t flat = g * len + j;
            const size_t c = flat / plane, hw = flat - c * plane;
            return (n * plane + hw) * t.ldc + c;
        };
        float mx = -FLT_MAX;
        for (size_t j = lane; j < len; j += 32) mx = fmaxf(mx, Elem<T>::ld(static_cast<const T *>(in.ptr) + addr(in, j)));
        for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
        float sum = 0.f;
        for (size_t j = lane; j < len; j += 32)
            sum += expf(Elem<T>::ld(static_cast<const T *>(in.ptr) + addr(in, j)) / temperature - mx / temperature);
        for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
        for (size_t j = lane; j < len; j += 32) {
            const float e = expf(Elem<T>::ld(static_cast<const T *>(in.ptr) + addr(in, j)) / temperature - mx / temperature);
            st_out(out, static_cast<T *>(out.ptr) + addr(out, j), e / sum);
        }
    }
}

// ---- depthwise conv (groups == Cin == Cout), BatchNorm/bias + activation fused ----
// (the reference runs one im2col + Sgemm per channel, src/layers/MsnhConvolutionalLayer.cpp:1028-1066)
// Weights are repacked to [tap][C] so a thread's V channels of one tap are one 16-byte load.
template <typename T, int V>
__global__ void dwconv_kernel(TView in, TView out, const T *__restrict__ w, const float *__restrict__ scale,
                              const float *__restrict__ bias, int kh, int kw, int sh, int sw, int ph, int pw,
                              int dh, int dw, int act, float act_param) {
    pdl_prologue();
    const int cv = out.C / V;
    const size_t total = static_cast<size_t>(out.N) * out.H * out.W * cv;
    // (32-bit index arithmetic: the plan refuses tensors of 2^31 or more vectors)
    for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < static_cast<unsigned>(total); i += gridDim.x * blockDim.x) {
        unsigned pix = i / cv;
        const int c = static_cast<int>(i - pix * cv) * V;
        const int ow = static_cast<int>(pix % out.W); pix /= out.W;
        const int oh = static_cast<int>(pix % out.H);
        const int n  = static_cast<int>(pix / out.H);
        float acc[V];
#pragma unroll
        for (int e = 0; e < V; ++e) acc[e] = 0.f;
        for (int r = 0; r < kh; ++r) {
            const int ih = oh * sh - ph + r * dh;
            if (ih < 0 || ih >= in.H) continue;
            for (int s = 0; s < kw; ++s) {
                const int iw = ow * sw - pw + s * dw;
                if (iw < 0 || iw >= in.W) continue;
                float x[V], f[V];
                VecIO<T, V>::ld(static_cast<const T *>(in.ptr) + pix_off(in, n, ih, iw) + c, x);
                VecIO<T, V>::ld(w + static_cast<size_t>(r * kw + s) * out.C + c, f);
#pragma unroll
                for (int e = 0; e < V; ++e) acc[e] = fmaf(x[e], f[e], acc[e]);
            }
        }
#pragma unroll
        for (int e = 0; e < V; ++e) {
            const float sc = scale ? scale[c + e] : 1.f, bi = bias ? bias[c + e] : 0.f;
            acc[e] = activate(fmaf(acc[e], sc, bi), act, act_param);
        }
        VecIO<T, V>::st_out(out, static_cast<T *>(out.ptr) + pix_off(out, n, oh, ow) + c, acc);
    }
}

// 3x3 depthwise conv, dilation 1, stride S = 1 or 2, on 16-byte channel vectors: a thread computes a strip of
// four output pixels of one row for V channels, so every input vector it loads feeds up to three taps of up to
// two outputs (18 or 27 loads per four outputs instead of 36) and the nine weight vectors, scale and bias are
// read once per strip. The activation switch sits outside the arithmetic.
template <typename T, int V, int S>
__global__ void dwconv3x3_kernel(TView in, TView out, const T *__restrict__ w, const float *__restrict__ scale,
                                 const float *__restrict__ bias, int ph, int pw, int act, float act_param) {
    pdl_prologue();
    constexpr int TW = 4;                        // output pixels per thread
    constexpr int IW = (TW - 1) * S + 3;         // input columns they read
    const int cv = out.C / V;
    const int strips = (out.W + TW - 1) / TW;
    const int total = out.N * out.H * strips * cv;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < total; i += gridDim.x * blockDim.x) {
        int rest = i / cv;
        const int c = (i - rest * cv) * V;
        const int strip = rest % strips; rest /= strips;
        const int oh = rest % out.H;
        const int n = rest / out.H;
        const int ow0 = strip * TW;
        const int iw0 = ow0 * S - pw;
        float acc[TW][V];
#pragma unroll
        for (int t = 0; t < TW; ++t)
#pragma unroll
            for (int e = 0; e < V; ++e) acc[t][e] = 0.f;
#pragma unroll
        for (int r = 0; r < 3; ++r) {
            const int ih = oh * S - ph + r;
            if (ih < 0 || ih >= in.H) continue;
            const T *row = static_cast<const T *>(in.ptr) + pix_off(in, n, ih, 0) + c;
            float x[IW][V];
#pragma unroll
            for (int q = 0; q < IW; ++q) {
                const int iw = iw0 + q;
                if (iw >= 0 && iw < in.W) VecIO<T, V>::ld(row + static_cast<size_t>(iw) * in.ldc, x[q]);
                else {
#pragma unroll
                    for (int e = 0; e < V; ++e) x[q][e] = 0.f;
                }
            }
#pragma unroll
            for (int s = 0; s < 3; ++s) {
                float f[V];
                VecIO<T, V>::ld(w + static_cast<size_t>(r * 3 + s) * out.C + c, f);
#pragma unroll
                for (int t = 0; t < TW; ++t)
#pragma unroll
                    for (int e = 0; e < V; ++e) acc[t][e] = fmaf(x[t * S + s][e], f[e], acc[t][e]);
            }
        }
        float sc[V], bi[V];
#pragma unroll
        for (int e = 0; e < V; ++e) { sc[e] = scale ? scale[c + e] : 1.f; bi[e] = bias ? bias[c + e] : 0.f; }
        T *orow = static_cast<T *>(out.ptr) + pix_off(out, n, oh, 0) + c;
#pragma unroll
        for (int t = 0; t < TW; ++t) {
            if (ow0 + t >= out.W) break;
#pragma unroll
            for (int e = 0; e < V; ++e) acc[t][e] = fmaf(acc[t][e], sc[e], bi[e]);
            switch (act) {
                case MSNH_ACT_NONE: break;
                case MSNH_ACT_RELU6:
#pragma unroll
                    for (int e = 0; e < V; ++e) acc[t][e] = fminf(fmaxf(acc[t][e], 0.f), 6.f);
                    break;
                case MSNH_ACT_RELU:
#pragma unroll
                    for (int e = 0; e < V; ++e) acc[t][e] = acc[t][e] > 0.f ? acc[t][e] : 0.f;
                    break;
                case MSNH_ACT_LEAKY:
#pragma unroll
                    for (int e = 0; e < V; ++e) acc[t][e] = acc[t][e] > 0.f ? acc[t][e] : act_param * acc[t][e];
                    break;
                default:
#pragma unroll
                    for (int e = 0; e < V; ++e) acc[t][e] = activate(acc[t][e], act, act_param);
                    break;
            }
            VecIO<T, V>::st_out(out, orow + static_cast<size_t>(ow0 + t) * out.ldc, acc[t]);
        }
    }
}

// ---- CUDA-core direct convolution: any kernel / stride / padding / dilation / groups ----
// Slow and simple: the device-side cross-check of the tensor-core kernel and the fallback for
// shapes it does not take (grouped non-depthwise convs). Weights in the tensor-core packing
// [Cout][tap][cin_pad] (cin_pad = per-group input channels rounded up to a 16-byte multiple).
template <typename T>
__global__ void conv_direct_kernel(TView in, TView out, const T *__restrict__ w, int cin_pad,
                                   const float *__restrict__ scale, const float *__restrict__ bias,
                                   int kh, int kw, int sh, int sw, int ph, int pw, int dh, int dw, int groups,
                                   const T *__restrict__ res, int ldc_res, int act1, float act1_param,
                                   int act2, float act2_param) {
    pdl_prologue();
    const size_t total = static_cast<size_t>(out.N) * out.H * out.W * out.C;
    const int cin_g = in.C / groups, cout_g = out.C / groups;
    for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < total;
         i += static_cast<size_t>(gridDim.x) * blockDim.x) {
        size_t pix = i / out.C;
        const int co = static_cast<int>(i - pix * out.C);
        const size_t opix = pix;
        const int ow = static_cast<int>(pix % out.W); pix /= out.W;
        const int oh = static_cast<int>(pix % out.H);
        const int n  = static_cast<int>(pix / out.H);
        const int g = co / cout_g;
        float acc = 0.f;
        for (int r = 0; r < kh; ++r) {
            const int ih = oh * sh - ph + r * dh;
            if (ih < 0 || ih >= in.H) continue;
            for (int s = 0; s < kw; ++s) {
                const int iw = ow * sw - pw + s * dw;
                if (iw < 0 || iw >= in.W) continue;
                const T *x = static_cast<const T *>(in.ptr) + pix_off(in, n, ih, iw) + g * cin_g;
                const T *f = w + (static_cast<size_t>(co) * kh * kw + r * kw + s) * cin_pad;
                for (int ci = 0; ci < cin_g; ++ci) acc = fmaf(Elem<T>::ld(x + ci), Elem<T>::ld(f + ci), acc);
            }
        }
        float y = activate(fmaf(acc, scale ? scale[co] : 1.f, bias ? bias[co] : 0.f), act1, act1_param);
        if (res) y = activate(y + Elem<T>::ld(res + opix * ldc_res + co), act2, act2_param);
        if (sizeof(T) == 4 && out.tf32) y = round_tf32(y);
        Elem<T>::st(static_cast<T *>(out.ptr) + opix * out.ldc + co, y);
    }
}

// ---- YOLO head decode ----
// (YoloLayer::forwardGPU and its five kernels, src/layers/MsnhYoloLayer.cpp:145-214,
//  src/layers/cuda/MsnhYoloLayerGPU.cu:4-93; math as the CPU path, src/layers/MsnhYoloLayer.cpp:217-284)
// in : [N][H][W][3*(5+cls)] raw head logits (T), out: same shape, always fp32.
// channel a*(5+cls)+k of anchor a: k=0 x, 1 y, 2 w, 3 h, 4 objectness, 5.. class scores.
// value k (0 x, 1 y, 2 w, 3 h, >= 4 objectness / class score) of anchor a at grid cell (col, row) from its raw logit t
__device__ __forceinline__ float yolo_decode_value(float t, int k, int a, int col, int row, int yolo_type, float ratio,
                                                   const YoloAnchors &an) {
    const float sg = 1.f / (1.f + expf(-t));
    if (k >= 4) return sg;
    if (k < 2) {
        const float grid = k == 0 ? static_cast<float>(col) : static_cast<float>(row);
        return (yolo_type == MSNH_YOLO_V5) ? (2.f * sg - 0.5f + grid) * ratio : (sg + grid) * ratio;
    }
    const float side = k == 2 ? an.w[a] : an.h[a];
    return (yolo_type == MSNH_YOLO_V5) ? side * powf(2.f * sg, 2.f) : side * expf(t);
}

template <typename T>
__global__ void yolo_decode_kernel(TView in, TView out, int classes, int yolo_type, float ratio, YoloAnchors an) {
    pdl_prologue();
    const int per = 5 + classes;
    const size_t total = static_cast<size_t>(in.N) * in.H * in.W * in.C;
    for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < total;
         i += static_cast<size_t>(gridDim.x) * blockDim.x) {
        size_t pix = i / in.C;
        const int c = static_cast<int>(i - pix * in.C);
        const size_t opix = pix;
        const int col = static_cast<int>(pix % in.W); pix /= in.W;
        const int row = static_cast<int>(pix % in.H);
        const int a = c / per, k = c - a * per;
        const float t = Elem<T>::ld(static_cast<const T *>(in.ptr) + opix * in.ldc + c);
        const float y = yolo_decode_value(t, k, a, col, row, yolo_type, ratio, an);
        static_cast<float *>(out.ptr)[opix * out.ldc + c] = y;
    }
}

// ---- candidate collection: what YoloOutLayer does on the host after its shuffle + D2H ----
// (src/layers/MsnhYoloOutLayer.cpp:119-165; shuffleDataKernel, src/layers/cuda/MsnhYoloOutLayerGPU.cu:5-28)
// One thread per (image, cell, anchor) of a decoded head. Cells whose objectness exceeds the
// threshold append {x,y,w,h,conf,bestClsConf,bestClsIdx,order} to the image's row list through
// an atomic counter. `order` = order_base + anchor*H*W + cell is the candidate's index in the
// reference's scan, so the host can restore the reference's candidate order exactly.
__global__ void yolo_collect_kernel(TView dec, int classes, float conf_thresh, int order_base,
                                    float *__restrict__ rows, int max_rows, int *__restrict__ counts) {
    pdl_prologue();
    const int per = 5 + classes;
    const int plane = dec.H * dec.W;
    const size_t total = static_cast<size_t>(dec.N) * plane * 3;
    for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < total;
         i += static_cast<size_t>(gridDim.x) * blockDim.x) {
        const int a = static_cast<int>(i % 3);
        const size_t pix = i / 3;
        const int n = static_cast<int>(pix / plane), cell = static_cast<int>(pix - static_cast<size_t>(n) * plane);
        const float *p = static_cast<const float *>(dec.ptr) + pix * dec.ldc + a * per;
        const float conf = p[4];
        if (!(conf > conf_thresh)) continue;
        float best = p[5]; int best_i = 0;
        for (int k = 1; k < classes; ++k) { const float v = p[5 + k]; if (v > best) { best = v; best_i = k; } }
        const int slot = atomicAdd(counts + n, 1);
        if (slot < max_rows) {
            float *r = rows + (static_cast<size_t>(n) * max_rows + slot) * 8;
            r[0] = p[0]; r[1] = p[1]; r[2] = p[2]; r[3] = p[3]; r[4] = conf; r[5] = best;
            r[6] = static_cast<float>(best_i); r[7] = static_cast<float>(order_base + a * plane + cell);
        }
    }
}

// Decode and collect in one pass over the RAW head logits: only the objectness of every (cell, anchor) is
// decoded; the box and the class scores are decoded for the cells that pass. Same values, row for row,
// as yolo_decode_kernel followed by yolo_collect_kernel, without writing the decoded tensor.
// All heads of the net go through ONE launch (items = (image, cell, anchor) of head 0, then of head 1, ...), and the
// class scores of a cell that passes are scanned by its whole warp (three scores per lane, then a shuffle arg-max that
// keeps the lowest index among equal maxima, as the reference's first-greater scan does): one passing cell no longer
// holds its warp for eighty dependent loads.
template <typename T>
__global__ void yolo_decode_collect_kernel(const __grid_constant__ YoloHeadSet hs, float conf_thresh, float *__restrict__ rows, int max_rows,
                                           int *__restrict__ counts) {
    pdl_prologue();
    const int total = hs.h[hs.n - 1].end;
    const int lane = threadIdx.x & 31;
    for (int i0 = blockIdx.x * blockDim.x + threadIdx.x - lane; i0 < total; i0 += gridDim.x * blockDim.x) {
        const int i = i0 + lane;
        bool pass = false;
        const T *p = nullptr;
        float conf = 0.f, ratio = 1.f;
        int a = 0, n = 0, cell = 0, row = 0, col = 0, plane = 1, classes = 0, yolo_type = 0, order_base = 0;
        YoloAnchors an{};
        if (i < total) {
            int start = 0;
#pragma unroll
            for (int h = 0; h < 4; ++h) {
                if (h < hs.n && i >= start && i < hs.h[h].end) {
                    const YoloHead &hd = hs.h[h];
                    const int j = i - start;
                    a = j % 3;
                    const int pix = j / 3;
                    plane = hd.in.H * hd.in.W;
                    n = pix / plane; cell = pix - n * plane;
                    row = cell / hd.in.W; col = cell - row * hd.in.W;
                    classes = hd.classes; yolo_type = hd.yolo_type; order_base = hd.order_base; ratio = hd.ratio; an = hd.an;
                    p = static_cast<const T *>(hd.in.ptr) + static_cast<size_t>(pix) * hd.in.ldc + a * (5 + classes);
                }
                if (h < hs.n) start = hs.h[h].end;
            }
            conf = yolo_decode_value(Elem<T>::ld(p + 4), 4, a, col, row, yolo_type, ratio, an);
            pass = conf > conf_thresh;
        }
        unsigned todo = __ballot_sync(0xffffffffu, pass);
        float best = 0.f; int best_i = 0;
        while (todo) {
            const int src = __ffs(todo) - 1;
            todo &= todo - 1;
            const T *ps = reinterpret_cast<const T *>(__shfl_sync(0xffffffffu, reinterpret_cast<unsigned long long>(p), src));
            const int cls = __shfl_sync(0xffffffffu, classes, src);
            float b = -INFINITY; int bi = 0x7fffffff;
            for (int k = lane; k < cls; k += 32) {
                const float v = yolo_decode_value(Elem<T>::ld(ps + 5 + k), 5, 0, 0, 0, 0, 1.f, an);
                if (v > b) { b = v; bi = k; }
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                const float ov = __shfl_xor_sync(0xffffffffu, b, o);
                const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
                if (ov > b || (ov == b && oi < bi)) { b = ov; bi = oi; }
            }
            if (lane == src) { best = b; best_i = bi; }
        }
        if (pass) {
            const int slot = atomicAdd(counts + n, 1);
            if (slot < max_rows) {
                float *r = rows + (static_cast<size_t>(n) * max_rows + slot) * 8;
#pragma unroll
                for (int k = 0; k < 4; ++k) r[k] = yolo_decode_value(Elem<T>::ld(p + k), k, a, col, row, yolo_type, ratio, an);
                r[4] = conf; r[5] = best;
                r[6] = static_cast<float>(best_i); r[7] = static_cast<float>(order_base + a * plane + cell);
            }
        }
    }
}

// The candidates of a batch to pinned host memory, a CTA per image: the count and the first `cap` rows of those there are. A few
// KB of posted writes in one launch, in place of a copy of every row a slot could hold.
__global__ void candidates_to_host_kernel(const float4 *__restrict__ rows, int max_rows, const int *__restrict__ counts, float4 *host_rows, int cap, int *host_counts) {
    const int n = blockIdx.x, count = counts[n], take = 2 * min(min(count, max_rows), cap);
    if (threadIdx.x == 0) host_counts[n] = count;
    for (int i = threadIdx.x; i < take; i += blockDim.x) host_rows[static_cast<size_t>(n) * cap * 2 + i] = rows[static_cast<size_t>(n) * max_rows * 2 + i];
}

// ---- raw 8-bit image -> the net's fp32 planar input ----
// What the reference's C API does on the host before the forward (src/c_api/MsnhnetLib.cpp:540-600, :754-778 with
// src/utils/MsnhCVUtil.cpp:91-373 and the bilinear MatOp::resize, src/cv/MsnhCVMatOp.cpp:142-160, :399-434):
// optional RGB<->BGR swap, optional pad-to-square with 127-gray bars, bilinear resize in float32 with the
// source's operation order (result through a float -> uint16 conversion, clamped to 255), optional second
// channel swap, then one affine formula per mode. One thread per output pixel; every float operation is a
// round-to-nearest intrinsic so the result equals the host code bit for bit (built without FMA contraction).
__device__ __forceinline__ int prep_src(const unsigned char *src, const PrepParams &p, int yy, int xx, int k, int top, int left) {
    yy -= top; xx -= left;
    if (yy < 0 || yy >= p.h || xx < 0 || xx >= p.w) return 127;
    return src[(static_cast<size_t>(yy) * p.w + xx) * 3 + k];
}
__global__ void preprocess_u8_kernel(const unsigned char *__restrict__ src, float *__restrict__ out, PrepParams p,
                                     size_t src_image_bytes, size_t out_image_floats) {
    const int x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y;
    if (x >= p.out_w || y >= p.out_h) return;
    src += blockIdx.z * src_image_bytes;            // blockIdx.z: image of a batch of same-sized images
    out += blockIdx.z * out_image_floats;
    int sw = p.w, sh = p.h, top = 0, left = 0;
    if (p.letterbox) {
        const int diff = abs(p.w - p.h);
        if (p.w > p.h) { top = diff / 2; sh = p.w; } else if (p.w < p.h) { left = diff / 2; sw = p.h; }
    }
    const bool same = sw == p.out_w && sh == p.out_h;
    int h0 = y, h1 = y, w0 = x, w1 = x;
    float wh1 = 0.f, wh0 = 0.f, ww1 = 0.f, ww0 = 0.f;
    if (!same) {
        const float fx = __fdiv_rn(__fmul_rn(1.f, static_cast<float>(sw)), static_cast<float>(p.out_w));
        const float fy = __fdiv_rn(__fmul_rn(1.f, static_cast<float>(sh)), static_cast<float>(p.out_h));
        float ih = __fsub_rn(__fmul_rn(__fadd_rn(static_cast<float>(y), 0.5f), fy), 0.5f); ih = ih < 0.f ? 0.f : ih;
        float iw = __fsub_rn(__fmul_rn(__fadd_rn(static_cast<float>(x), 0.5f), fx), 0.5f); iw = iw < 0.f ? 0.f : iw;
        h0 = __float2int_rz(ih); h1 = min(h0 + 1, sh - 1);
        w0 = __float2int_rz(iw); w1 = min(w0 + 1, sw - 1);
        wh1 = __fsub_rn(static_cast<float>(h1), ih); wh0 = __fsub_rn(ih, static_cast<float>(h0));
        ww1 = __fsub_rn(static_cast<float>(w1), iw); ww0 = __fsub_rn(iw, static_cast<float>(w0));
    }
    const size_t plane = static_cast<size_t>(p.out_w) * p.out_h;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const int k1 = p.rev_out ? 2 - k : k;             // channel of the resized image that lands in plane k
        const int ks = p.rev_in ? 2 - k1 : k1;            // channel of the caller's image behind it
        int u;
        if (same) u = prep_src(src, p, y, x, ks, top, left);
        else {
            const float p00 = static_cast<float>(prep_src(src, p, h0, w0, ks, top, left)), p01 = static_cast<float>(prep_src(src, p, h0, w1, ks, top, left));
            const float p10 = static_cast<float>(prep_src(src, p, h1, w0, ks, top, left)), p11 = static_cast<float>(prep_src(src, p, h1, w1, ks, top, left));
            const float t = __fmul_rn(wh1, __fadd_rn(__fmul_rn(ww1, p00), __fmul_rn(ww0, p01)));
            const float b = __fmul_rn(wh0, __fadd_rn(__fmul_rn(ww1, p10), __fmul_rn(ww0, p11)));
            const int r16 = __float2int_rz(__fadd_rn(t, b)) & 0xFFFF;    // float -> uint16 as the host conversion does
            u = r16 > 255 ? 255 : r16;
        }
        const float uf = static_cast<float>(u);
        float v;
        switch (p.mode) {
            case MSNH_PREP_GOOGLENET: {
                const float a = k == 0 ? (0.229f / 0.5f) : (k == 1 ? (0.224f / 0.5f) : (0.225f / 0.5f));
                const float c = k == 0 ? ((0.485f - 0.5f) / 0.5f) : (k == 1 ? ((0.456f - 0.5f) / 0.5f) : ((0.406f - 0.5f) / 0.5f));
                v = __fadd_rn(__fmul_rn(__fdiv_rn(uf, 255.0f), a), c);
                break;
            }
            case MSNH_PREP_TRANSFORMED: v = __fdiv_rn(__fsub_rn(__fdiv_rn(uf, 255.0f), p.mean[k]), p.std[k]); break;
            case MSNH_PREP_CAFFE: v = __fsub_rn(uf, k == 0 ? 123.68f : (k == 1 ? 116.779f : 103.939f)); break;
            default: v = __fdiv_rn(uf, 255.0f); break;    // MSNH_PREP_UNIT and MSNH_PREP_PAD_SQUARE
        }
        out[k * plane + static_cast<size_t>(y) * p.out_w + x] = v;
    }
}

// ---- bilinear resize (upsample type bilinear) ----
// (bilinearResizeKernel, src/core/cuda/MsnhBlasGPU.cu:580-654; Blas::cpuBilinearResize, src/core/MsnhBlas.cpp:2400-2464)
// rh / rw are the reference's source steps, computed on the host in float as it does:
// align_corners 0: in/out; 1: (in-1)/(out-1).
template <typename T, int V>
__global__ void bilinear_kernel(TView in, TView out, float rh, float rw, int align) {
    pdl_prologue();
    const int cv = out.C / V;
    const size_t total = static_cast<size_t>(out.N) * out.H * out.W * cv;
    // (32-bit index arithmetic: the plan refuses tensors of 2^31 or more vectors)
    for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < static_cast<unsigned>(total); i += gridDim.x * blockDim.x) {
        unsigned pix = i / cv;
        const int c = static_cast<int>(i - pix * cv) * V;
        const int ow = static_cast<int>(pix % out.W); pix /= out.W;
        const int oh = static_cast<int>(pix % out.H);
        const int n  = static_cast<int>(pix / out.H);
        float h1r, w1r;
        if (align == 0) {
            h1r = fmaxf(__fsub_rn(__fmul_rn(rh, oh + 0.5f), 0.5f), 0.f);
            w1r = fmaxf(__fsub_rn(__fmul_rn(rw, ow + 0.5f), 0.5f), 0.f);
        } else {
            h1r = __fmul_rn(rh, static_cast<float>(oh));
            w1r = __fmul_rn(rw, static_cast<float>(ow));
        }
        const int h1 = static_cast<int>(h1r), w1 = static_cast<int>(w1r);
        const int h1p = h1 < in.H - 1 ? 1 : 0, w1p = w1 < in.W - 1 ? 1 : 0;
        const float lh1 = h1r - h1, lh0 = 1.f - lh1, lw1 = w1r - w1, lw0 = 1.f - lw1;
        const T *base = static_cast<const T *>(in.ptr) + c;
        float a[V], b[V], d[V], e[V], y[V];
        VecIO<T, V>::ld(base + pix_off(in, n, h1, w1), a);
        VecIO<T, V>::ld(base + pix_off(in, n, h1, w1 + w1p), b);
        VecIO<T, V>::ld(base + pix_off(in, n, h1 + h1p, w1), d);
        VecIO<T, V>::ld(base + pix_off(in, n, h1 + h1p, w1 + w1p), e);
#pragma unroll
        for (int k = 0; k < V; ++k) y[k] = lh0 * (lw0 * a[k] + lw1 * b[k]) + lh1 * (lw0 * d[k] + lw1 * e[k]);
        VecIO<T, V>::st_out(out, static_cast<T *>(out.ptr) + pix_off(out, n, oh, ow) + c, y);
    }
}

// ---- transposed convolution, second half: gather of the per-tap products (+bias, +activation) ----
// The first half is a 1x1 tensor-core convolution that leaves, for every INPUT pixel, the kh*kw*Cout products
// W[ci][co][ky][kx] * x[ci] summed over ci, stored tap-major ([ky][kx][co]). An output pixel (oy, ox) sums the
// taps whose input pixel exists: iy = (oy + pad - ky) / stride when that division is exact and in range, so only
// ky = (oy + pad) mod stride, + stride, ... are visited. Same sums as Gemm::cpuCol2Im over the GEMM result
// (src/core/MsnhGemm.cpp:115-154, src/layers/MsnhDeConvolutionalLayer.cpp:113-127), taps in its order (ky, then kx).
// What follows the layer in the net rides along: y = act(sum + bias); then, when given, the BatchNorm behind it
// (y * scale2 + bias2, its activation) and the tensor a route adds (+ res, its activation).
template <typename T, int V>
__global__ void col2im_kernel(TView col, TView out, int kh, int kw, int sh, int sw, int ph, int pw,
                              const float *__restrict__ bias, int act, float act_p, Col2ImTail tail, int lanes_c_log2) {
    pdl_prologue();
    // One output row (n, oh) per CTA turn. The CTA's threads form a (channel vector, pixel) grid whose first extent is
    // a power of two (lanes_c = 1 << lanes_c_log2 <= channel vectors), so a thread finds its pixel and channel with
    // shifts; the row index costs one 32-bit division per row.
    const int cv = out.C / V;
    const int rows = out.N * out.H;
    const int tc = threadIdx.x & ((1 << lanes_c_log2) - 1), tp = threadIdx.x >> lanes_c_log2;
    const int step_c = 1 << lanes_c_log2, step_p = blockDim.x >> lanes_c_log2;
    for (int row = blockIdx.x; row < rows; row += gridDim.x) {
        const int n = row / out.H, oh = row - n * out.H;
        const int ty0 = oh + ph;
        const int ky0 = ty0 % sh, iy0 = ty0 / sh;
        const T *col_img = static_cast<const T *>(col.ptr) + static_cast<size_t>(n) * col.H * col.W * col.ldc;
        T *out_row = static_cast<T *>(out.ptr) + pix_off(out, n, oh, 0);
        const T *res_row = tail.res ? static_cast<const T *>(tail.res) + (static_cast<size_t>(n) * out.H + oh) * out.W * static_cast<size_t>(tail.ldc_res) : nullptr;
        for (int ow = tp; ow < out.W; ow += step_p)
        for (int cvec = tc; cvec < cv; cvec += step_c) {
            const int c = cvec * V;
            float s[V];
#pragma unroll
            for (int e = 0; e < V; ++e) s[e] = 0.f;
            const int tx0 = ow + pw;
            int kx0, ix0;
            if (sw == 2) { kx0 = tx0 & 1; ix0 = tx0 >> 1; } else if (sw == 1) { kx0 = 0; ix0 = tx0; } else { kx0 = tx0 % sw; ix0 = tx0 / sw; }
            for (int ky = ky0, iy = iy0; ky < kh && iy >= 0; ky += sh, --iy) {
                if (iy >= col.H) continue;
                for (int kx = kx0, ix = ix0; kx < kw && ix >= 0; kx += sw, --ix) {
                    if (ix >= col.W) continue;
                    float v[V];
                    VecIO<T, V>::ld(col_img + (static_cast<size_t>(iy) * col.W + ix) * col.ldc + (ky * kw + kx) * out.C + c, v);
#pragma unroll
                    for (int e = 0; e < V; ++e) s[e] += v[e];
                }
            }
            // per-channel tables are padded to a multiple of 8 floats and 16-byte aligned: vector loads when V allows
            auto add_table = [&](const float *tab, bool mul) {
                float t[V];
                if constexpr (V % 4 == 0) {
#pragma unroll
                    for (int e = 0; e < V; e += 4) {
                        const float4 q = __ldg(reinterpret_cast<const float4 *>(tab + c + e));
                        t[e] = q.x; t[e + 1] = q.y; t[e + 2] = q.z; t[e + 3] = q.w;
                    }
                } else {
#pragma unroll
                    for (int e = 0; e < V; ++e) t[e] = tab[c + e];
                }
#pragma unroll
                for (int e = 0; e < V; ++e) s[e] = mul ? s[e] * t[e] : s[e] + t[e];
            };
            auto act_all = [&](int a, float ap) {
                if (a == MSNH_ACT_NONE) return;
                if (a == MSNH_ACT_RELU) {
#pragma unroll
                    for (int e = 0; e < V; ++e) s[e] = fmaxf(s[e], 0.f);
                    return;
                }
#pragma unroll
                for (int e = 0; e < V; ++e) s[e] = activate(s[e], a, ap);
            };
            if (bias) add_table(bias, false);
            act_all(act, act_p);
            if (tail.scale2) { add_table(tail.scale2, true); add_table(tail.bias2, false); act_all(tail.act_mid, tail.act_mid_p); }
            if (res_row) {
                float r[V];
                VecIO<T, V>::ld(res_row + static_cast<size_t>(ow) * tail.ldc_res + c, r);
#pragma unroll
                for (int e = 0; e < V; ++e) s[e] += r[e];
                act_all(tail.act2, tail.act2_p);
            }
            VecIO<T, V>::st_out(out, out_row + static_cast<size_t>(ow) * out.ldc + c, s);
        }
    }
}

// ---- PReLU: x > 0 ? x : slope[c] * x (Activations::activatePRelu, src/layers/MsnhActivations.cpp:411-470) ----
template <typename T, int V>
__global__ void prelu_kernel(TView in, TView out, const float *__restrict__ slope) {
    pdl_prologue();
    const int cv = out.C / V;
    const size_t total = static_cast<size_t>(out.N) * out.H * out.W * cv;
    // (32-bit index arithmetic: the plan refuses tensors of 2^31 or more vectors)
    for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < static_cast<unsigned>(total); i += gridDim.x * blockDim.x) {
        const unsigned pix = i / cv;
        const int c = static_cast<int>(i - pix * cv) * V;
        float v[V];
        VecIO<T, V>::ld(static_cast<const T *>(in.ptr) + static_cast<size_t>(pix) * in.ldc + c, v);
#pragma unroll
        for (int e = 0; e < V; ++e) v[e] = v[e] > 0.f ? v[e] : v[e] * slope[c + e];
        VecIO<T, V>::st_out(out, static_cast<T *>(out.ptr) + static_cast<size_t>(pix) * out.ldc + c, v);
    }
}

// ---- depth max pooling: out channel g = max over input channels g, g + out.C, g + 2 out.C, ... of the same pixel ----
// (MaxPoolLayer::forward with maxPoolDepth, src/layers/MsnhMaxPoolLayer.cpp:244-270; forwardDepthGPU,
// src/layers/cuda/MsnhMaxPoolLayerGPU.cu)
template <typename T>
__global__ void maxpool_depth_kernel(TView in, TView out) {
    pdl_prologue();
    const size_t total = static_cast<size_t>(out.N) * out.H * out.W * out.C;
    for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < total;
         i += static_cast<size_t>(gridDim.x) * blockDim.x) {
        const size_t pix = i / out.C;
        const int g = static_cast<int>(i - pix * out.C);
        const T *src = static_cast<const T *>(in.ptr) + pix * in.ldc;
        float m = -FLT_MAX;
        for (int k = g; k < in.C; k += out.C) m = fmaxf(m, Elem<T>::ld(src + k));
        st_out(out, static_cast<T *>(out.ptr) + pix * out.ldc + g, m);
    }
}

// ---- clip: min(max(x, lo), hi) (clipKernel, src/layers/cuda/MsnhClipLayerGPU.cu) ----
template <typename T, int V>
__global__ void clip_kernel(TView in, TView out, float lo, float hi) {
    pdl_prologue();
    const int cv = out.C / V;
    const size_t total = static_cast<size_t>(out.N) * out.H * out.W * cv;
    // (32-bit index arithmetic: the plan refuses tensors of 2^31 or more vectors)
    for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < static_cast<unsigned>(total); i += gridDim.x * blockDim.x) {
        const unsigned pix = i / cv;
        const int c = static_cast<int>(i - pix * cv) * V;
        float v[V];
        VecIO<T, V>::ld(static_cast<const T *>(in.ptr) + static_cast<size_t>(pix) * in.ldc + c, v);
#pragma unroll
        for (int e = 0; e < V; ++e) v[e] = fminf(fmaxf(v[e], lo), hi);
        VecIO<T, V>::st_out(out, static_cast<T *>(out.ptr) + static_cast<size_t>(pix) * out.ldc + c, v);
    }
}

// ---- view / permute / pixel shuffle: element i of the output's planar (C,H,W) order comes from element g(i) of
//      the input's planar order; both tensors live channels-last here, so the kernel converts on either side ----
// kind 0 view: g(i) = i (src/layers/MsnhViewLayer.cpp); kind 1 permute: input axis d[k] becomes output axis k
// (src/layers/MsnhPermuteLayer.cpp:127-183, permuteKernel in src/layers/cuda/MsnhPermuteLayerGPU.cu);
// kind 2 pixel shuffle with factor d[0], the reference's own index formula
// (src/layers/MsnhPixelShuffleLayer.cpp:98-104, src/layers/cuda/MsnhPixelShuffleLayerGPU.cu).
template <typename T>
__global__ void remap_kernel(TView in, TView out, int kind, int d0, int d1, int d2) {
    pdl_prologue();
    const size_t total = static_cast<size_t>(out.N) * out.H * out.W * out.C;
    const int in_plane = in.H * in.W;
    for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < total;
         i += static_cast<size_t>(gridDim.x) * blockDim.x) {
        size_t pix = i / out.C;
        const int oc = static_cast<int>(i - pix * out.C);
        const int ow = static_cast<int>(pix % out.W); pix /= out.W;
        const int oh = static_cast<int>(pix % out.H);
        const int n  = static_cast<int>(pix / out.H);
        int ic, ih, iw;
        if (kind == 1) {
            int idx[3];
            idx[d0] = oc; idx[d1] = oh; idx[d2] = ow;
            ic = idx[0]; ih = idx[1]; iw = idx[2];
        } else {
            long long j;
            if (kind == 0) j = (static_cast<long long>(oc) * out.H + oh) * out.W + ow;
            else j = static_cast<long long>(oc * d0 + ow % d0) * in_plane + static_cast<long long>(oh) * in.W + ow / d0;
            ic = static_cast<int>(j / in_plane);
            const int r = static_cast<int>(j - static_cast<long long>(ic) * in_plane);
            ih = r / in.W; iw = r - ih * in.W;
        }
        T v = static_cast<const T *>(in.ptr)[pix_off(in, n, ih, iw) + ic];
        if constexpr (sizeof(T) == 4) { if (out.tf32) v = round_tf32(v); }
        static_cast<T *>(out.ptr)[pix_off(out, n, oh, ow) + oc] = v;
    }
}

// ---- reduction: sum or mean over one axis (0 C, 1 H, 2 W) or over the whole image (-1), one image at a time ----
// (src/layers/MsnhReductionLayer.cpp:76-160). One warp per output value; lanes stride over the reduced axis.
template <typename T>
__global__ void reduce_kernel(TView in, TView out, int axis, int mean) {
    pdl_prologue();
    const int lane = threadIdx.x & 31;
    const size_t warp = (blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x) >> 5;
    const size_t warps = (static_cast<size_t>(gridDim.x) * blockDim.x) >> 5;
    const size_t total = static_cast<size_t>(out.N) * out.H * out.W * out.C;
    for (size_t o = warp; o < total; o += warps) {
        size_t pix = o / out.C;
        const int oc = static_cast<int>(o - pix * out.C);
        const int ow = static_cast<int>(pix % out.W); pix /= out.W;
        const int oh = static_cast<int>(pix % out.H);
        const int n  = static_cast<int>(pix / out.H);
        const T *src = static_cast<const T *>(in.ptr);
        float s = 0.f;
        int len;
        if (axis == 0)      { len = in.C; for (int k = lane; k < len; k += 32) s += Elem<T>::ld(src + pix_off(in, n, oh, ow) + k); }
        else if (axis == 1) { len = in.H; for (int k = lane; k < len; k += 32) s += Elem<T>::ld(src + pix_off(in, n, k, ow) + oc); }
        else if (axis == 2) { len = in.W; for (int k = lane; k < len; k += 32) s += Elem<T>::ld(src + pix_off(in, n, oh, k) + oc); }
        else {
            len = in.H * in.W * in.C;
            const int hw = in.H * in.W;
            for (int p = lane; p < hw; p += 32) {
                const T *px = src + (static_cast<size_t>(n) * hw + p) * in.ldc;
                for (int k = 0; k < in.C; ++k) s += Elem<T>::ld(px + k);
            }
        }
#pragma unroll
        for (int d = 16; d > 0; d >>= 1) s += __shfl_xor_sync(0xffffffffu, s, d);
        if (mean) s = s / static_cast<float>(len);
        if (lane == 0) st_out(out, static_cast<T *>(out.ptr) + pix_off(out, n, oh, ow) + oc, s);
    }
}

// ---- L2 flush helper for per-launch profiling ----
__global__ void fill_kernel(float *p, size_t n, float v) {
    pdl_prologue();
    for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < n;
         i += static_cast<size_t>(gridDim.x) * blockDim.x) p[i] = v;
}

}  // namespace msnh
