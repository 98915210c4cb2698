// cnn.cu -- the learned subgrid closure's convolutional network on the tensor cores.
//
// Network: L periodic 3x3 convolutions (stride 1, "same" with periodic wrap, as the doubly
// periodic QG domain), GELU after every layer but the last.  Activations are NHWC BF16 with
// the channel count padded to a multiple of 16; weights are FP32 masters with BF16 copies in
// two layouts (forward: [tap][cout][cin], backward-data: [tap'][cin][cout] with the taps
// mirrored); products run on the BF16 tensor cores with FP32 accumulation: tcgen05.mma with
// the accumulator tile in TMEM (default; forward, backward-data and weight gradients), or the
// warp-level mma.m16n8k16 path (selectable with qgn_cnn_set_engine or QGN_CNN_MMA=sync).  An inference
// whose tiles fit one CTA each runs all layers in one cooperative launch (k_cnn_fused);
// QGN_CNN_MMA=layers keeps one tcgen05 launch per layer.
//
// Kernels (one CTA = 8 warps = 128 consecutive pixels of one image row, persistent over rows):
//   k_conv<CIN,COUT,EPI>  implicit GEMM  out[p, n] = sum_{tap, k} in[p + tap, k] w[tap, n, k]
//                         EPI_GELU:      A = bf16(GELU(Z)), D = GELU'(Z) (FP32), Z = acc + bias
//                         EPI_LINEAR:    Y = acc + bias (FP32)
//                         EPI_GELU_GRAD: G = bf16(acc * D)   (backward through a layer)
//   k_wgrad<CIN,COUT>     dW[tap, n, k] partials = sum_p G[p, n] in[p + tap, k] per row chunk
//   k_reduce_*            deterministic chunk sums of dW and the bias gradient
//   k_mse                 loss and dL/dY = 2 (Y - T)/count, as BF16 G of the last layer
//   k_adam                Adam on the FP32 masters, refreshing both BF16 layouts
//   k_conv_tc<CIN,COUT,EPI>  the implicit GEMM on tcgen05 (TMEM accumulators)
//   k_wgrad_tc<CX,SWAP>   the weight- and bias-gradient partials on tcgen05 (MN-major operands)
//   k_cnn_fused           every layer of a small-batch inference, rows exchanged through L2
#include "qgn_internal.cuh"
#include "cnn.cuh"
#include "tmap.cuh"

#include <cuda_bf16.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstdlib>
#include <cstring>
#include <new>
#include <random>
#include <string>
#include <vector>

namespace qgn {
namespace cnn {

constexpr int kTileP = 128;          // pixels per CTA tile (one row segment)
constexpr int kWarps = 8;
constexpr int kThreads = kWarps * 32;
// Warps of the fused small-batch inference (one CTA per SM: shared memory).  It has one tile per
// CTA and per layer, with nothing to overlap its epilogue (TMEM loads, bias, GELU, BF16 packing,
// staged stores), so 16 warps each drain 16 accumulator columns: the 128^2 batch-1 inference ran
// 58.2 -> 53.7 us on B200.
constexpr int kFusedWarps = 16;
constexpr int kFusedThreads = kFusedWarps * 32;
// Warps of the layer kernels k_conv_tc and k_wgrad_tc by role: these drain accumulators, one more
// loads rows, one issues the MMAs
constexpr int kEpiWarps = 16;        // k_conv_tc
constexpr int kDrainWarps = 8;       // k_wgrad_tc
constexpr int kConvThreads = (kEpiWarps + 2) * 32;
constexpr int kWgThreads = (kDrainWarps + 2) * 32;
constexpr int kMseThreads = 1024;
constexpr int kWChunkRows = 16;      // image rows per weight-gradient partial of the mma.sync engine

// EPI_PLANAR: as EPI_LINEAR but the FP32 output is planar, out[n][pixel] (the closure's input
// to its forward transform)
// EPI_GELU_ACT: as EPI_GELU without the FP32 pre-activation (inference: only the BF16
// activation feeds the next layer)
enum { EPI_GELU = 0, EPI_LINEAR = 1, EPI_GELU_GRAD = 2, EPI_PLANAR = 3, EPI_GELU_ACT = 4 };

__device__ __forceinline__ float gelu(float z) { return 0.5f * z * (1.0f + erff(z * 0.70710678118654752f)); }
__device__ __forceinline__ float gelu_grad(float z) {
    return 0.5f * (1.0f + erff(z * 0.70710678118654752f)) + z * 0.39894228040143268f * expf(-0.5f * z * z);
}

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ void ldsm_x4(uint32_t addr, uint32_t& r0, uint32_t& r1, uint32_t& r2, uint32_t& r3) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n"
                 : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3)
                 : "r"(addr));
}
__device__ __forceinline__ void ldsm_x4_t(uint32_t addr, uint32_t& r0, uint32_t& r1, uint32_t& r2, uint32_t& r3) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n"
                 : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3)
                 : "r"(addr));
}

// D += A(16x16, row) * B(16x8, col), BF16 in, FP32 accumulate
__device__ __forceinline__ void mma_bf16(float* d, uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                         uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
        "{%0,%1,%2,%3};\n"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

template <int C>
struct RowPad {
    static constexpr int LD = C + 8;   // bf16 elements per pixel in shared memory (16-byte skew)
};

// copy pixels [w0-1, w0+128] (periodic) of image row (b, h) into smem rows of LD elements
template <int C>
__device__ __forceinline__ void load_row(const __nv_bfloat16* __restrict__ src, int b, int h, int H, int W, int w0,
                                         int halo, __nv_bfloat16* dst) {
    constexpr int V = C / 8;   // 16-byte vectors per pixel
    const int npix = kTileP + 2 * halo;
    const size_t rowbase = ((size_t)b * H + h) * W;
    for (int i = threadIdx.x; i < npix * V; i += kThreads) {
        const int px = i / V, v = i % V;
        int w = w0 - halo + px;
        w = (w % W + W) % W;
        const uint4 val = *reinterpret_cast<const uint4*>(src + (rowbase + w) * C + v * 8);
        *reinterpret_cast<uint4*>(dst + px * RowPad<C>::LD + v * 8) = val;
    }
}

// ---- implicit-GEMM periodic 3x3 convolution -------------------------------------------------
template <int CIN, int COUT, int EPI>
__global__ void __launch_bounds__(kThreads, 1)
    k_conv(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ wt, const float* __restrict__ bias,
           int B, int H, int W, float* __restrict__ outf, __nv_bfloat16* __restrict__ outb,
           const float* __restrict__ dact) {
    QGN_PDL_ENTRY();
    static_assert(CIN % 16 == 0 && COUT % 16 == 0, "channel counts are padded to 16");
    constexpr int LDI = RowPad<CIN>::LD;
    constexpr int NT = COUT / 8;       // n-tiles of 8 output channels per warp
    extern __shared__ __align__(16) unsigned char smraw[];
    __nv_bfloat16* ws = reinterpret_cast<__nv_bfloat16*>(smraw);           // [9][COUT][LDI]
    __nv_bfloat16* xs = ws + 9 * COUT * LDI;                                 // [3][130][LDI]
    const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
    // weights once per CTA
    for (int i = threadIdx.x; i < 9 * COUT * (CIN / 8); i += kThreads) {
        const int row = i / (CIN / 8), v = i % (CIN / 8);
        *reinterpret_cast<uint4*>(ws + row * LDI + v * 8) = *reinterpret_cast<const uint4*>(wt + (size_t)row * CIN + v * 8);
    }
    const int segs = W / kTileP;
    const int ntiles = B * H * segs;
    for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
        const int seg = tile % segs;
        const int h = (tile / segs) % H;
        const int b = tile / (segs * H);
        const int w0 = seg * kTileP;
        __syncthreads();   // previous tile's readers of xs are done (and the weights are in)
        for (int r = 0; r < 3; ++r)
            load_row<CIN>(x, b, (h + r - 1 + H) % H, H, W, w0, 1, xs + r * (kTileP + 2) * LDI);
        __syncthreads();
        float acc[NT][4];
#pragma unroll
        for (int j = 0; j < NT; ++j) acc[j][0] = acc[j][1] = acc[j][2] = acc[j][3] = 0.f;
        const int pbase = warp * 16;
#pragma unroll 1
        for (int tap = 0; tap < 9; ++tap) {
            const int dh = tap / 3, dw = tap % 3;      // offsets +1 (halo included)
            const __nv_bfloat16* xr = xs + dh * (kTileP + 2) * LDI;
            const __nv_bfloat16* wr = ws + tap * COUT * LDI;
#pragma unroll
            for (int kc = 0; kc < CIN / 16; ++kc) {
                uint32_t a0, a1, a2, a3;
                {
                    const int prow = pbase + (lane % 8) + 8 * ((lane / 8) % 2);
                    const int kcol = kc * 16 + 8 * (lane / 16);
                    ldsm_x4(smem_u32(xr + (prow + dw) * LDI + kcol), a0, a1, a2, a3);
                }
#pragma unroll
                for (int j = 0; j < NT; j += 2) {
                    uint32_t b0, b1, b2, b3;
                    const int n = j * 8 + (lane % 8) + 8 * (lane / 16);
                    const int kcol = kc * 16 + 8 * ((lane / 8) % 2);
                    ldsm_x4(smem_u32(wr + n * LDI + kcol), b0, b1, b2, b3);
                    mma_bf16(acc[j], a0, a1, a2, a3, b0, b1);
                    mma_bf16(acc[j + 1], a0, a1, a2, a3, b2, b3);
                }
            }
        }
        // epilogue: thread holds pixels g, g+8 of the warp's 16 and channels 2t, 2t+1 of each n-tile
        const int g = lane / 4, t = lane % 4;
        const size_t prow0 = ((size_t)b * H + h) * W + w0 + pbase;
#pragma unroll
        for (int j = 0; j < NT; ++j) {
            const int n = j * 8 + 2 * t;
#pragma unroll
            for (int half = 0; half < 2; ++half) {
                const size_t p = prow0 + g + 8 * half;
                float v0 = acc[j][2 * half], v1 = acc[j][2 * half + 1];
                if (EPI == EPI_PLANAR) {
                    const size_t np = (size_t)B * H * W;
                    outf[(size_t)n * np + p] = v0 + bias[n];
                    outf[(size_t)(n + 1) * np + p] = v1 + bias[n + 1];
                } else if (EPI == EPI_GELU || EPI == EPI_LINEAR || EPI == EPI_GELU_ACT) {
                    v0 += bias[n];
                    v1 += bias[n + 1];
                    if (EPI == EPI_GELU || EPI == EPI_GELU_ACT) {
                        if (EPI == EPI_GELU)
                            *reinterpret_cast<float2*>(outf + p * COUT + n) =
                                make_float2(gelu_grad(v0), gelu_grad(v1));
                        *reinterpret_cast<__nv_bfloat162*>(outb + p * COUT + n) =
                            __floats2bfloat162_rn(gelu(v0), gelu(v1));
                    } else {
                        *reinterpret_cast<float2*>(outf + p * COUT + n) = make_float2(v0, v1);
                    }
                } else {
                    const float2 d = *reinterpret_cast<const float2*>(dact + p * COUT + n);
                    *reinterpret_cast<__nv_bfloat162*>(outb + p * COUT + n) = __floats2bfloat162_rn(v0 * d.x, v1 * d.y);
                }
            }
        }
    }
}

// ---- weight gradient: partial[chunk][tap][n][k] = sum over the chunk's pixels of G[p,n] in[p+tap,k]
template <int CIN, int COUT>
__global__ void __launch_bounds__(kThreads, 1)
    k_wgrad(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ gr, int B, int H, int W,
            float* __restrict__ part) {
    QGN_PDL_ENTRY();
    constexpr int LDI = RowPad<CIN>::LD, LDG = RowPad<COUT>::LD;
    constexpr int MT = CIN / 16, NT = COUT / 8;
    constexpr int TILES = MT * NT;                  // 16x8 output tiles of dW[tap]
    constexpr int PERW = (TILES + kWarps - 1) / kWarps;
    static_assert(TILES % kWarps == 0 || TILES < kWarps, "tiles split evenly over warps");
    extern __shared__ __align__(16) unsigned char smraw[];
    __nv_bfloat16* xs = reinterpret_cast<__nv_bfloat16*>(smraw);    // [130][LDI]
    __nv_bfloat16* gs = xs + (kTileP + 2) * LDI;                      // [128][LDG]
    const int tap = blockIdx.y;
    const int dh = tap / 3 - 1, dw = tap % 3 - 1;
    const int chunk = blockIdx.x;
    const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
    const int segs = W / kTileP;
    const int rows_total = B * H;
    const int r0 = chunk * kWChunkRows, r1 = min(rows_total, r0 + kWChunkRows);
    float acc[PERW][4];
#pragma unroll
    for (int i = 0; i < PERW; ++i) acc[i][0] = acc[i][1] = acc[i][2] = acc[i][3] = 0.f;
    for (int row = r0; row < r1; ++row) {
        const int b = row / H, h = row % H;
        for (int seg = 0; seg < segs; ++seg) {
            const int w0 = seg * kTileP;
            __syncthreads();
            load_row<CIN>(x, b, (h + dh + H) % H, H, W, w0, 1, xs);
            load_row<COUT>(gr, b, h, H, W, w0, 0, gs);
            __syncthreads();
#pragma unroll 1
            for (int kp = 0; kp < kTileP / 16; ++kp) {
#pragma unroll
                for (int i = 0; i < PERW; ++i) {
                    const int tt = warp * PERW + i;
                    if (tt >= TILES) break;
                    const int mt = tt / NT, nt = tt % NT;
                    uint32_t a0, a1, a2, a3, b0, b1, b2, b3;
                    {
                        // A = in^T (rows k = input channel, cols = pixel): transposed 8x8 loads
                        const int mj = lane / 8, r = lane % 8;
                        const int p = kp * 16 + r + 8 * (mj / 2) + 1 + dw;     // +1: halo offset
                        const int k = mt * 16 + 8 * (mj % 2);
                        ldsm_x4_t(smem_u32(xs + p * LDI + k), a0, a1, a2, a3);
                    }
                    {
                        // B = G (rows = pixel, cols n): b0 = pixels 0-7, b1 = pixels 8-15 (transposed)
                        const int mj = lane / 8, r = lane % 8;
                        const int p = kp * 16 + r + 8 * (mj % 2);
                        const int n = (nt & ~1) * 8 + 8 * (mj / 2);
                        ldsm_x4_t(smem_u32(gs + p * LDG + n), b0, b1, b2, b3);
                    }
                    if (nt % 2 == 0) mma_bf16(acc[i], a0, a1, a2, a3, b0, b1);
                    else mma_bf16(acc[i], a0, a1, a2, a3, b2, b3);
                }
            }
        }
    }
    // acc[i]: rows k = mt*16 + g (+8), cols n = nt*8 + 2t (+1)
    const int g = lane / 4, t = lane % 4;
    float* out = part + ((size_t)chunk * 9 + tap) * COUT * CIN;
#pragma unroll
    for (int i = 0; i < PERW; ++i) {
        const int tt = warp * PERW + i;
        if (tt >= TILES) break;
        const int mt = tt / NT, nt = tt % NT;
#pragma unroll
        for (int half = 0; half < 2; ++half) {
            const int k = mt * 16 + g + 8 * half;
            const int n = nt * 8 + 2 * t;
            out[(size_t)n * CIN + k] = acc[i][2 * half];
            out[(size_t)(n + 1) * CIN + k] = acc[i][2 * half + 1];
        }
    }
}

// dw[i] = sum of nchunks partials of n weights, db likewise of nb biases: a block sums 64 outputs, its
// four groups of threads a quarter of the partials each, then the quarters in order.  (One thread per
// output ran 147 dependent loads deep, 15.8 us for 64 x 64 x 9, and the biases' one block 12.5 us more.)
constexpr int kRedOut = 64;
__global__ void __launch_bounds__(4 * kRedOut)
    k_reduce_wgrad(const float* __restrict__ part, int nchunks, int n, float* __restrict__ dw,
                   const float* __restrict__ bpart, int nbchunks, int nb, float* __restrict__ db) {
    QGN_PDL_ENTRY();
    __shared__ float sm[4][kRedOut];
    const int o = threadIdx.x % kRedOut, q = threadIdx.x / kRedOut;
    int i = blockIdx.x * kRedOut + o;
    const int wblocks = (n + kRedOut - 1) / kRedOut;   // (the blocks of the weights; one more for the biases)
    if ((int)blockIdx.x >= wblocks) {
        part = bpart;
        nchunks = nbchunks;
        dw = db;
        n = nb;
        i = o;
    }
    const int c0 = nchunks * q / 4, c1 = nchunks * (q + 1) / 4;
    float s = 0.f;
    if (i < n) {
#pragma unroll 8
        for (int c = c0; c < c1; ++c) s += part[(size_t)c * n + i];
    }
    sm[q][o] = s;
    __syncthreads();
    if (q == 0 && i < n) dw[i] = ((s + sm[1][o]) + sm[2][o]) + sm[3][o];
}

// bias gradient: per-block column sums of G, then a chunk reduction
__global__ void k_bias_part(const __nv_bfloat16* __restrict__ gr, long long npix, int C, int pix_per_block,
                            float* __restrict__ part) {
    QGN_PDL_ENTRY();
    const long long p0 = (long long)blockIdx.x * pix_per_block;
    const long long p1 = min(npix, p0 + pix_per_block);
    for (int c = threadIdx.x; c < C; c += blockDim.x) {
        float s = 0.f;
        for (long long p = p0; p < p1; ++p) s += __bfloat162float(gr[p * C + c]);
        part[(size_t)blockIdx.x * C + c] = s;
    }
}

// MSE over the real output channels; G = bf16(2 (Y - T) / count), zero in padded channels.  One
// thread per four channels of a pixel: 16-byte loads, none of them for padded groups.
__global__ void __launch_bounds__(kMseThreads) k_mse(const float* __restrict__ y, const float* __restrict__ tgt, long long npix, int C, int creal,
                      double inv_count, __nv_bfloat16* __restrict__ g, double* __restrict__ loss_part) {
    QGN_PDL_ENTRY();
    __shared__ double red[kMseThreads / 32];
    double s = 0.0;
    const float gs = (float)(2.0 * inv_count);
    const long long n4 = npix * (C / 4);
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n4; i += (long long)gridDim.x * blockDim.x) {
        const int c0 = 4 * (int)((unsigned long long)i % (unsigned)(C / 4));
        float gv[4] = {0.f, 0.f, 0.f, 0.f};
        if (c0 < creal) {
            const float4 a = reinterpret_cast<const float4*>(y)[i], b = reinterpret_cast<const float4*>(tgt)[i];
            const float d[4] = {a.x - b.x, a.y - b.y, a.z - b.z, a.w - b.w};
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                if (c0 + k < creal) {
                    s += (double)d[k] * (double)d[k];
                    gv[k] = gs * d[k];
                }
            }
        }
        __nv_bfloat162 o[2] = {__floats2bfloat162_rn(gv[0], gv[1]), __floats2bfloat162_rn(gv[2], gv[3])};
        reinterpret_cast<uint2*>(g)[i] = *reinterpret_cast<const uint2*>(o);
    }
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (threadIdx.x % 32 == 0) red[threadIdx.x / 32] = s;
    __syncthreads();
    if (threadIdx.x == 0) {
        double tot = 0.0;
        for (int i = 0; i < (int)(blockDim.x / 32); ++i) tot += red[i];
        loss_part[blockIdx.x] = tot * inv_count;
    }
}

// Adam (bias-corrected) on FP32 masters [9][cout][cin]; refreshes the forward ([tap][cout][cin])
// and backward-data ([8-tap][cin][cout]) BF16 copies
__global__ void k_adam(float* __restrict__ w, float* __restrict__ m, float* __restrict__ v,
                       const float* __restrict__ g, int n, int cout, int cin, float lr, float b1, float b2, float eps,
                       float c1, float c2, __nv_bfloat16* __restrict__ wf, __nv_bfloat16* __restrict__ wb) {
    QGN_PDL_ENTRY();
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const float gi = g[i];
        const float mi = b1 * m[i] + (1.f - b1) * gi;
        const float vi = b2 * v[i] + (1.f - b2) * gi * gi;
        m[i] = mi;
        v[i] = vi;
        const float wi = w[i] - lr * (mi / c1) / (sqrtf(vi / c2) + eps);
        w[i] = wi;
        if (wf) {
            const int tap = i / (cout * cin), r = i % (cout * cin);
            const int co = r / cin, ci = r % cin;
            const __nv_bfloat16 bv = __float2bfloat16_rn(wi);
            wf[i] = bv;
            wb[((size_t)(8 - tap) * cin + ci) * cout + co] = bv;
        }
    }
}

__global__ void k_adam_bias(float* __restrict__ w, float* __restrict__ m, float* __restrict__ v,
                            const float* __restrict__ g, int n, float lr, float b1, float b2, float eps, float c1,
                            float c2) {
    QGN_PDL_ENTRY();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float gi = g[i];
    const float mi = b1 * m[i] + (1.f - b1) * gi;
    const float vi = b2 * v[i] + (1.f - b2) * gi * gi;
    m[i] = mi;
    v[i] = vi;
    w[i] = w[i] - lr * (mi / c1) / (sqrtf(vi / c2) + eps);
}

__global__ void k_weights_bf16(const float* __restrict__ w, int n, int cout, int cin, __nv_bfloat16* __restrict__ wf,
                               __nv_bfloat16* __restrict__ wb) {
    QGN_PDL_ENTRY();
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const int tap = i / (cout * cin), r = i % (cout * cin);
        const int co = r / cin, ci = r % cin;
        const __nv_bfloat16 bv = __float2bfloat16_rn(w[i]);
        wf[i] = bv;
        wb[((size_t)(8 - tap) * cin + ci) * cout + co] = bv;
    }
}

// gather batch samples: dst[b] = src[idx[b]] (rows of `bytes` bytes, 16-byte multiples)
__global__ void k_gather(const unsigned char* __restrict__ src, const int* __restrict__ idx, int nb, size_t bytes,
                         unsigned char* __restrict__ dst) {
    QGN_PDL_ENTRY();
    const size_t vec = bytes / 16;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < vec * nb; i += (size_t)gridDim.x * blockDim.x) {
        const size_t b = i / vec, o = i % vec;
        reinterpret_cast<uint4*>(dst)[i] = reinterpret_cast<const uint4*>(src + (size_t)idx[b] * bytes)[o];
    }
}

// ---- the same convolution on the 5th-generation tensor cores (tcgen05, accumulator in TMEM) ----
// One tile = 128 consecutive pixels of an image row (GEMM M = 128) x all COUT output channels
// with K = 9 taps x CIN (kind::f16, BF16 in, FP32 accumulate); the FP32 tile lives in TMEM (COUT columns, one lane per pixel) and
// the epilogue reads it back with tcgen05.ld.  Operands sit in shared memory:
//   input rows of 64 channels   [pixel][128 B] in the 128-byte swizzle (16-byte piece c of a pixel at
//               c ^ (address / 128 % 8)), as one tensor-map copy of 128 pixels writes them, with the
//               two pixels of the periodic halo on either side.  The A tile of tap (dh, dw) starts
//               at pixel dw - 1: the swizzle goes by address, so a shift by whole pixels (128 B) is a
//               shift of the start address.  Eight-pixel groups 1024 B apart (SBO);
//   input rows of 16 channels   canonical K-major no-swizzle layout (core matrices of 8 rows x 16
//               bytes): [2 channel groups][130 pixels][8 channels], pixels 16 B apart, 8-pixel
//               groups 128 B apart (SBO), the two halves of a K step 130*16 B apart (LBO);
//   weights     no-swizzle, chunks of eight input channels: SBO 128 B, LBO one chunk.
// Each CTA takes a contiguous range of tiles ordered row-fastest, so consecutive tiles of a column
// of rows share two of their three input rows: one new row per tile.  Completion is signalled by
// tcgen05.commit on mbarriers; every wait is bounded, and a wait that runs out records an error,
// waits once more for the MMAs in flight, frees the TMEM and returns.
namespace tc {

constexpr int kPixS = kTileP + 2;        // staged pixels per input row (periodic halo)
constexpr int kSlots = 6;                // input-row ring of the layer kernel
constexpr int kAccSlots = 8;             // accumulator ring of the layer kernel
constexpr long long kWaitLimit = 1LL << 22;

constexpr int imax(int a, int b) { return a > b ? a : b; }

// a staged row of C channels: 64 channels swizzled, halo pixels in the eight-pixel blocks before and
// after the 128 pixels at MAIN; 16 channels in two planes
template <int C>
struct Row {
    static constexpr bool SWZ = C == 64;
    static constexpr int MAIN = SWZ ? 1024 : 0;
    static constexpr int BYTES = SWZ ? 1024 + kTileP * 128 + 1024 : ((C / 8) * kPixS * 16 + 1023) / 1024 * 1024;
};

// Shared-memory plan of the layer kernel
template <int CIN, int COUT>
struct Lay {
    static constexpr int SLOT_BYTES = Row<CIN>::BYTES;
    static constexpr int W_OFF = kSlots * SLOT_BYTES;
    static constexpr int W_BYTES = 9 * (CIN / 8) * COUT * 16;
    static constexpr int BAR_OFF = (W_OFF + W_BYTES + 1023) / 1024 * 1024;
    static constexpr int NB = 3 * COUT;                      // operand rows: the three tap rows
    static constexpr int OPS_END = BAR_OFF + 1024;
    static constexpr int STG_OFF = OPS_END;                 // output staging, 2 KB per epilogue warp
    static constexpr int SMEM = STG_OFF + kEpiWarps * 2048;
    static constexpr int TMEM_COLS = kAccSlots * COUT;       // the accumulators of eight output rows
};

// Shared-memory operand descriptors, version 1: the low word holds the start address and the leading
// byte offset, the high word the stride byte offset and the swizzle.  Addresses and offsets are in
// 16-byte units below 2^14, so a later start address is a sum on the low word.
struct Desc {
    uint32_t lo, hi;
    __device__ __forceinline__ Desc at(uint32_t bytes) const { return Desc{lo + (bytes >> 4), hi}; }
};
__device__ __forceinline__ Desc sdesc(uint32_t saddr, uint32_t lbo, uint32_t sbo) {   // no swizzle
    return Desc{(saddr >> 4) | ((lbo >> 4) << 16), (sbo >> 4) | (1u << 14)};
}
// an operand in the 128-byte swizzle, groups of eight 128-byte rows 1024 B apart
__device__ __forceinline__ Desc sdesc128(uint32_t saddr) {
    return Desc{(saddr >> 4) | (64u << 16), 64u | (1u << 14) | (2u << 29)};
}

// M = 128, N = COUT, BF16 x BF16 -> F32, both operands K-major
template <int N>
__host__ __device__ constexpr uint32_t idesc() {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
}

// the same with N at run time (a multiple of 16, at most 256)
__device__ __forceinline__ uint32_t idesc_n(int n) { return idesc<0>() | ((uint32_t)(n >> 3) << 17); }

__device__ __forceinline__ void mma(uint32_t tmem, Desc a, Desc b, uint32_t id, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t.reg .b64 da, db;\n\tsetp.ne.b32 p, %6, 0;\n\t"
        "mov.b64 da, {%1, %2};\n\tmov.b64 db, {%3, %4};\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %5, p;\n\t}\n" ::"r"(tmem),
        "r"(a.lo), "r"(a.hi), "r"(b.lo), "r"(b.hi), "r"(id), "r"(accumulate));
}

// One lane of a converged warp, always the same one.  The MMAs are issued under it and not under
// `lane == 0`: their operands live in uniform registers, and only this form tells the compiler that
// what one thread computes is the warp's -- under a lane test every MMA moved its descriptors there
// by itself and took about 110 cycles to issue, whatever its size.
__device__ __forceinline__ bool elect_one() {
    uint32_t p;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}\n" : "=r"(p));
    return p != 0;
}

__device__ __forceinline__ bool bar_wait(uint32_t bar, uint32_t parity) {
    for (long long i = 0; i < kWaitLimit; ++i) {
        uint32_t ok;
        asm volatile(
            "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}\n"
            : "=r"(ok)
            : "r"(bar), "r"(parity)
            : "memory");
        if (ok) return true;
    }
    return false;
}

// bounded wait of one role of a layer kernel; gives up at once when another role has.  False: the
// role leaves its loop (and so, through the flag, do the others).
__device__ __forceinline__ bool role_wait(uint32_t bar, uint32_t parity, volatile int* gave_up) {
    for (long long i = 0; i < kWaitLimit; ++i) {
        uint32_t ok;
        asm volatile(
            "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}\n"
            : "=r"(ok)
            : "r"(bar), "r"(parity)
            : "memory");
        if (ok) return true;
        if (*gave_up) return false;
    }
    *gave_up = 1;
    return false;
}
__device__ __forceinline__ void arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(bar)
                 : "memory");
}
__device__ __forceinline__ void bar_init(uint32_t bar, int count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(bar), "r"(count) : "memory");
}

__device__ __forceinline__ void cp16(uint32_t saddr, const void* g) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(saddr), "l"(g) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
__device__ __forceinline__ void cp_wait_all() { asm volatile("cp.async.wait_all;\n" ::: "memory"); }

__device__ __forceinline__ void tmem_ld8(uint32_t taddr, float* v) {
    uint32_t r[8];
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = __uint_as_float(r[i]);
}
template <int NC>
__device__ __forceinline__ void tmem_ld(uint32_t taddr, float* v);
template <>
__device__ __forceinline__ void tmem_ld<16>(uint32_t taddr, float* v) {
    uint32_t r[16];
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                   "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
                 : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}
template <>
__device__ __forceinline__ void tmem_ld<32>(uint32_t taddr, float* v) {
    tmem_ld<16>(taddr, v);
    tmem_ld<16>(taddr + 16, v + 16);
}

// The 9*CIN/16 MMAs of one tile into the accumulator at TMEM address dacc, then a commit that
// arrives on the mbarrier at bar when they have completed.  ra: shared addresses of the ring
// slots holding input rows h-1, h, h+1; w: the layer's weights.  One thread issues.
template <int CIN, int COUT>
__device__ __forceinline__ void issue_tile(uint32_t dacc, const uint32_t* ra, uint32_t w, uint32_t bar) {
    const Desc b0 = sdesc(w, COUT * 16, 128);
    const Desc a0[3] = {sdesc(ra[0], kPixS * 16, 128), sdesc(ra[1], kPixS * 16, 128), sdesc(ra[2], kPixS * 16, 128)};
#pragma unroll
    for (int tap = 0; tap < 9; ++tap) {
#pragma unroll
        for (int kc = 0; kc < CIN / 16; ++kc)
            mma(dacc, a0[tap / 3].at((2 * kc * kPixS + tap % 3) * 16), b0.at((tap * (CIN / 8) + 2 * kc) * COUT * 16),
                idesc<COUT>(), (tap | kc) ? 1u : 0u);
    }
    commit(bar);
}

// a layer's weights [9][COUT][CIN] (BF16) into the K-major operand layout [9][CIN/8][COUT][8];
// cin and cout are powers of two (16 or 64), so the index split is shifts and masks
template <int NT>
__device__ __forceinline__ void fetch_weights(const __nv_bfloat16* __restrict__ wt, int cin, int cout, uint32_t w) {
    const int c8n = cin >> 3;
    const int lc8 = __ffs(c8n) - 1, lco = __ffs(cout) - 1;
    for (int i = threadIdx.x; i < 9 * cout * c8n; i += NT) {
        const int c8 = i & (c8n - 1), n = (i >> lc8) & (cout - 1), tap = i >> (lc8 + lco);
        cp16(w + (uint32_t)(((tap * c8n + c8) * cout + n) * 16), wt + ((size_t)tap * cout + n) * cin + c8 * 8);
    }
}

// the same into the layer kernel's operand layout [3 dw][CIN/8][3 COUT][8]: for one horizontal tap the
// three tap rows stacked, dh = +1 first
template <int CIN, int COUT, int NT>
__device__ __forceinline__ void fetch_weights_stacked(const __nv_bfloat16* __restrict__ wt, uint32_t w) {
    constexpr int C8 = CIN / 8;
    for (int i = threadIdx.x; i < 9 * COUT * C8; i += NT) {
        const int c8 = i % C8, n = (i / C8) % COUT, tap = i / (C8 * COUT);
        const int dh = tap / 3, dw = tap % 3;
        cp16(w + (uint32_t)(((dw * C8 + c8) * 3 * COUT + (2 - dh) * COUT + n) * 16), wt + ((size_t)tap * COUT + n) * CIN + c8 * 8);
    }
}

// one input row (image b, row hh, pixels w0-1 .. w0+128 periodic) into a ring slot, asynchronously
template <int CIN, int NT>
__device__ __forceinline__ void fetch_row(const __nv_bfloat16* __restrict__ x, int b, int hh, int H, int W, int w0,
                                         uint32_t slot_addr, int tid) {
    const size_t row = ((size_t)b * H + hh) * W;
    for (int i = tid; i < kPixS * (CIN / 8); i += NT) {
        const int c8 = i % (CIN / 8), px = i / (CIN / 8);
        int ww = w0 - 1 + px;   // in [-1, W]: one periodic wrap at either end
        ww = ww < 0 ? ww + W : (ww >= W ? ww - W : ww);
        cp16(slot_addr + (uint32_t)((c8 * kPixS + px) * 16), x + (row + ww) * CIN + c8 * 8);
    }
}

// 128 pixels of 64 channels (row `row` of the map, pixels w0 ..) into swizzled shared memory; the
// copy's bytes complete on bar
__device__ __forceinline__ void tma_row(uint32_t dst, const CUtensorMap* map, int w0, int row, uint32_t bar) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], "
        "[%5];\n" ::"r"(dst),
        "l"(map), "r"(0), "r"(w0), "r"(row), "r"(bar)
        : "memory");
}
__device__ __forceinline__ void arrive_tx(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(bar), "r"(bytes) : "memory");
}

// One warp loads a row with its periodic halo (image row `row`, pixels w0-1 .. w0+128) into the slot
// at `slot` and commits its cp.async group.  64 channels: the 128 pixels by tensor-map copy (its 16 KB
// are an arrival on `full` of their own, made here) and the two halo pixels by cp.async; 16 channels:
// all by cp.async.  The caller arrives once more when the group has completed.
template <int C>
__device__ __forceinline__ void load_row_warp(const CUtensorMap* map, const __nv_bfloat16* __restrict__ x, int row, int W,
                                              int w0, uint32_t slot, uint32_t full, int lane) {
    if constexpr (Row<C>::SWZ) {
        const uint32_t main = slot + Row<C>::MAIN;
        if (lane == 0) {
            arrive_tx(full, kTileP * 128);
            tma_row(main, map, w0, row, full);
        }
        if (lane < 16) {   // pixel w0-1 in the last row of the block before, w0+128 in the first one after
            const int side = lane / 8, c = lane % 8;
            const int ww = side ? (w0 + kTileP == W ? 0 : w0 + kTileP) : (w0 == 0 ? W - 1 : w0 - 1);
            cp16(main + (side ? kTileP * 128 + c * 16 : -128 + ((c ^ 7) * 16)), x + ((size_t)row * W + ww) * C + c * 8);
        }
    } else {
        fetch_row<C, 32>(x, 0, row, 0, W, w0, slot, lane);   // (b = 0: `row` counts all images' rows)
    }
    cp_commit();
}
// arrivals per use of a row's full barrier
template <int C>
__host__ __device__ constexpr int row_arrivals() { return Row<C>::SWZ ? 2 : 1; }

}  // namespace tc

// Epilogue of one tile of the fused inference: warp w reads TMEM lanes 32 (w % 4).. (one pixel per thread) and a block
// of columns, applies bias and, but for the last layer, GELU, and writes the tile through
// XOR-swizzled shared-memory staging so that the global stores are contiguous 16-byte pieces.
// The tile's outputs are contiguous in global memory: pixels p0 .. p0+127, COUT channels each.
// Columns of the accumulator each epilogue thread drains (NW warps: four TMEM sub-partitions,
// NW/4 column blocks each when COUT = 64; four warps when COUT = 16) and the first of them.
template <int COUT, int NW>
__host__ __device__ constexpr int epi_ncol() { return COUT == 64 ? 64 / (NW / 4) : 16; }
template <int COUT, int NW>
__device__ __forceinline__ int epi_n0(int warp) { return COUT == 64 ? epi_ncol<COUT, NW>() * (warp / 4) : 0; }

template <int CIN, int COUT, int EPI, int NW>
__device__ __forceinline__ void conv_tc_epilogue(uint32_t tacc, size_t p0, const float* breg,
                                                 float* __restrict__ outf, __nv_bfloat16* __restrict__ outb,
                                                 unsigned char* stf, unsigned char* stb, size_t npix) {
    const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
    constexpr int NCOL = epi_ncol<COUT, NW>();
    constexpr int NT = NW * 32;
    constexpr int CF = COUT / 4;        // 16-byte pieces per staged FP32 row
    constexpr int CB = COUT / 8;        // 16-byte pieces per staged BF16 row
    const bool reads = COUT == 64 || warp < 4;
    const int px = 32 * (warp % 4) + lane;
    const int n0 = epi_n0<COUT, NW>(warp);
    if (reads) {
        float v[NCOL];
        tc::tmem_ld<NCOL>(tacc + ((uint32_t)(32 * (warp % 4)) << 16) + (uint32_t)n0, v);
#pragma unroll
        for (int j = 0; j < NCOL; j += 4) {
            const int c = (n0 + j) / 4;
            float4* fz = reinterpret_cast<float4*>(stf + (px * CF + (c ^ (px % CF))) * 16);
            uint2* fb = reinterpret_cast<uint2*>(stb + (px * CB + (((n0 + j) / 8) ^ (px % CB))) * 16 + ((n0 + j) % 8) * 2);
            const float4 z = make_float4(v[j] + breg[j], v[j + 1] + breg[j + 1], v[j + 2] + breg[j + 2],
                                         v[j + 3] + breg[j + 3]);
            if (EPI == EPI_GELU_ACT) {
                __nv_bfloat162 g2[2] = {__floats2bfloat162_rn(gelu(z.x), gelu(z.y)),
                                        __floats2bfloat162_rn(gelu(z.z), gelu(z.w))};
                *fb = *reinterpret_cast<const uint2*>(g2);
            } else {
                *fz = z;
            }
        }
    }
    __syncthreads();
    if (EPI == EPI_LINEAR) {
        for (int i = threadIdx.x; i < kTileP * CF; i += NT) {
            const int r = i / CF, c = i % CF;
            *reinterpret_cast<float4*>(outf + (p0 + r) * COUT + c * 4) =
                *reinterpret_cast<const float4*>(stf + (r * CF + (c ^ (r % CF))) * 16);
        }
    }
    if (EPI == EPI_PLANAR) {   // out[n][p0 + r]: each channel's 128 pixels are contiguous
        for (int i = threadIdx.x; i < COUT * kTileP; i += NT) {
            const int n = i / kTileP, r = i % kTileP;
            const int c = n / 4;
            outf[(size_t)n * npix + p0 + r] =
                reinterpret_cast<const float*>(stf + (r * CF + (c ^ (r % CF))) * 16)[n % 4];
        }
    }
    if (EPI == EPI_GELU_ACT) {
        for (int i = threadIdx.x; i < kTileP * CB; i += NT) {
            const int r = i / CB, c = i % CB;
            *reinterpret_cast<uint4*>(outb + (p0 + r) * COUT + c * 8) =
                *reinterpret_cast<const uint4*>(stb + (r * CB + (c ^ (r % CB))) * 16);
        }
    }
}

// One layer for a batch, persistent over the CTA's tiles, with the warps split by role so that the
// row loads, the MMAs and the epilogue of different tiles overlap:
//   loader    one warp: streams the input rows of the CTA's tiles into the ring (two rows in flight
//             behind the one being issued), one 'full' barrier per slot;
//   issuer    one thread: multiplies each input row by the weights of all three tap rows at once, N =
//             3 COUT, into the accumulators of the three output rows that it belongs to, which are
//             neighbours in a ring of eight in TMEM; commits the row's slot to its 'empty' barrier
//             and the output row that it completes to its 'full' one;
//   epilogue  sixteen warps, each 32 pixels x 16 channels: accumulator to registers, bias, GELU, BF16
//             packing, and stores through a 2 KB staging block of the warp's own (XOR-swizzled, so
//             that the global stores are whole 32- and 64-byte sectors): no block-wide barrier.
// An MMA here costs the shared-memory bytes of its operands (128 B per clock): 4 KB of pixels and 2 KB
// of weights per 16 channels when each tap row was an MMA of its own with N = 64 (63 cycles measured,
// 36 of them per tile), 4 + 6 KB for the three together.  The sum of an output is formed in the same
// order either way (dh, dw, channels).
// 64 -> 64 at batch 32 on 128^2 (B200, ncu): loads, MMAs and epilogue one after another in the same warps
// 152 us with an FP32 second output; the split in roles 118 us, 92 us without it (inference); this form 86
// and 69 us.  Of the 69, the GELUs (8192 per tile, 32 instructions each) are 29 us of issue and the MMAs
// 15, on different warps, and neither is the bound: all sixteen epilogue warps take the same tile, wait for
// its tcgen05.ld together and then issue together (at batch 8: tensor pipe 19 %, issue slots 34 %, long
// scoreboard 3.5 of the stalls per issued instruction).
// EPI_GELU stores GELU'(z) in FP32 beside the activation, where the backward pass only multiplies by
// it: the error function is evaluated once per training step instead of twice.
template <int CIN, int COUT, int EPI>
__global__ void __launch_bounds__(kConvThreads, 1)
    k_conv_tc(const __grid_constant__ CUtensorMap xmap, const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ wt, const float* __restrict__ bias,
              int B, int H, int W, float* __restrict__ outf, __nv_bfloat16* __restrict__ outb,
              const float* __restrict__ dact, int* __restrict__ err) {
    QGN_PDL_ENTRY();
    using L = tc::Lay<CIN, COUT>;
    static_assert(COUT == 16 || COUT == 64, "N of the MMA");
    static_assert(COUT == 64 || EPI == EPI_LINEAR || EPI == EPI_PLANAR, "narrow outputs are the last layer's");
    constexpr int NCOL = 16;                              // channels per epilogue thread
    constexpr int EW = COUT == 64 ? kEpiWarps : 4;        // epilogue warps with work
    constexpr int NS = tc::kSlots, NA = tc::kAccSlots;
    extern __shared__ __align__(1024) unsigned char smtc[];
    uint32_t* tslot = reinterpret_cast<uint32_t*>(smtc + L::BAR_OFF + 240);
    volatile int* gave_up = reinterpret_cast<volatile int*>(smtc + L::BAR_OFF + 248);
    const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
    const uint32_t in_a = smem_u32(smtc), w_a = smem_u32(smtc + L::W_OFF);
    const uint32_t full = smem_u32(smtc + L::BAR_OFF), empty = full + 8 * NS, accf = empty + 8 * NS, acce = accf + 8 * NA,
                   drained = acce + 8 * NA;

    // this CTA's tiles: a contiguous range of t = ((b * segs + seg) * H + h), rows fastest.  Its
    // maximal runs of consecutive rows of one (b, seg) read cnt + 2 rows each; loaders and issuer
    // count the rows of all runs in the same order, row n in slot n % NS.
    const int segs = W / kTileP;
    const int ntiles = B * H * segs;
    const int per = (ntiles + gridDim.x - 1) / gridDim.x;
    const int t0 = blockIdx.x * per, t1 = min(ntiles, t0 + per);

    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(tslot)),
                     "r"((uint32_t)L::TMEM_COLS));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n");
    }
    if (threadIdx.x == 0) {
        *gave_up = 0;
        for (int i = 0; i < NS; ++i) {
            tc::bar_init(full + 8 * i, tc::row_arrivals<CIN>());
            tc::bar_init(empty + 8 * i, 1);
        }
        for (int i = 0; i < NA; ++i) {
            tc::bar_init(accf + 8 * i, 1);
            tc::bar_init(acce + 8 * i, EW);
        }
        tc::bar_init(drained, 1);
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    tc::fetch_weights_stacked<CIN, COUT, kConvThreads>(wt, w_a);
    tc::cp_commit();
    tc::cp_wait_all();
    asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    const uint32_t tmem = *tslot;

    if (warp < EW) {   // ---- epilogue
        const int pw = 32 * (warp % 4);                   // first pixel of the warp
        const int n0 = NCOL * (warp / 4);                 // first channel
        float breg[NCOL];
        if constexpr (EPI != EPI_GELU_GRAD) {
#pragma unroll
            for (int j = 0; j < NCOL; ++j) breg[j] = bias[n0 + j];
        }
        unsigned char* stg = smtc + L::STG_OFF + warp * 2048;
        for (int t = t0, i = 0; t < t1; ++t, ++i) {
            const int h = t % H, bs = t / H;
            const size_t p0 = ((size_t)(bs / segs) * H + h) * W + (bs % segs) * kTileP + pw;
            const int buf = i % NA;
            float4 dv[4];   // EPI_GELU_GRAD: the tile's GELU', 64 bytes of eight pixels per load
            if constexpr (EPI == EPI_GELU_GRAD) {
#pragma unroll
                for (int k = 0; k < 4; ++k)
                    dv[k] = *reinterpret_cast<const float4*>(dact + (p0 + 8 * k + lane / 4) * COUT + n0 + 4 * (lane % 4));
            }
            const bool ok = tc::role_wait(accf + 8 * buf, (i / NA) & 1, gave_up);
            if (!__all_sync(0xffffffffu, ok)) break;
            asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
            float v[NCOL];
            tc::tmem_ld<NCOL>(tmem + ((uint32_t)pw << 16) + (uint32_t)(buf * COUT + n0), v);
            asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
            __syncwarp();
            if (lane == 0) tc::arrive(acce + 8 * buf);
            if constexpr (EPI != EPI_GELU_GRAD) {
#pragma unroll
                for (int j = 0; j < NCOL; ++j) v[j] += breg[j];
            }
            if constexpr (EPI == EPI_PLANAR) {   // out[n][pixel]: 128 bytes per channel and warp
                const size_t npix = (size_t)B * H * W;
#pragma unroll
                for (int j = 0; j < NCOL; ++j) outf[(size_t)(n0 + j) * npix + p0 + lane] = v[j];
            } else {
                // FP32 staging: 64 bytes per pixel; lane = pixel, or four lanes per pixel
                auto fpiece = [&](int px, int c) {
                    return reinterpret_cast<float4*>(stg + px * 64 + ((c ^ ((px >> 1) & 3)) * 16));
                };
                auto put_f32 = [&]() {   // v -> outf
#pragma unroll
                    for (int c = 0; c < 4; ++c)
                        *fpiece(lane, c) = make_float4(v[4 * c], v[4 * c + 1], v[4 * c + 2], v[4 * c + 3]);
                    __syncwarp();
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        const int px = 8 * k + lane / 4, c = lane % 4;
                        *reinterpret_cast<float4*>(outf + (p0 + px) * COUT + n0 + 4 * c) = *fpiece(px, c);
                    }
                    __syncwarp();
                };
                if constexpr (EPI == EPI_LINEAR) {
                    put_f32();
                } else {
                    __nv_bfloat162 o[NCOL / 2];
                    if constexpr (EPI == EPI_GELU_GRAD) {
#pragma unroll
                        for (int k = 0; k < 4; ++k) *fpiece(8 * k + lane / 4, lane % 4) = dv[k];
                        __syncwarp();
#pragma unroll
                        for (int c = 0; c < 4; ++c) {
                            const float4 d = *fpiece(lane, c);
                            o[2 * c] = __floats2bfloat162_rn(v[4 * c] * d.x, v[4 * c + 1] * d.y);
                            o[2 * c + 1] = __floats2bfloat162_rn(v[4 * c + 2] * d.z, v[4 * c + 3] * d.w);
                        }
                        __syncwarp();
                    } else {
#pragma unroll
                        for (int k = 0; k < NCOL / 2; ++k) {
                            const float a = v[2 * k], b = v[2 * k + 1];
                            o[k] = __floats2bfloat162_rn(gelu(a), gelu(b));
                            if constexpr (EPI == EPI_GELU) {
                                v[2 * k] = gelu_grad(a);
                                v[2 * k + 1] = gelu_grad(b);
                            }
                        }
                    }
                    if constexpr (EPI == EPI_GELU) put_f32();
                    // BF16 output, 32 bytes per pixel
                    auto bpiece = [&](int px, int c) {
                        return reinterpret_cast<uint4*>(stg + px * 32 + ((c ^ ((px >> 2) & 1)) * 16));
                    };
#pragma unroll
                    for (int c = 0; c < 2; ++c) *bpiece(lane, c) = *reinterpret_cast<const uint4*>(&o[4 * c]);
                    __syncwarp();
#pragma unroll
                    for (int k = 0; k < 2; ++k) {
                        const int px = 16 * k + lane / 2, c = lane % 2;
                        *reinterpret_cast<uint4*>(outb + (p0 + px) * COUT + n0 + 8 * c) = *bpiece(px, c);
                    }
                    __syncwarp();
                }
            }
        }
    } else if (warp == kEpiWarps) {   // ---- loader
        int n = 0;             // rows issued
        bool ok = true;
        for (int t = t0; t < t1 && ok;) {
            const int h0 = t % H, bs = t / H;
            const int cnt = min(t1 - t, H - h0);
            const int b = bs / segs, w0 = (bs % segs) * kTileP;
            for (int i = 0; i < cnt + 2; ++i, ++n) {
                ok = __all_sync(0xffffffffu, tc::role_wait(empty + 8 * (n % NS), ((n / NS) & 1) ^ 1, gave_up));
                if (!ok) break;
                tc::load_row_warp<CIN>(&xmap, x, b * H + (h0 - 1 + i + H) % H, W, w0,
                                       in_a + (uint32_t)((n % NS) * L::SLOT_BYTES), full + 8 * (n % NS), lane);
                if (n >= 2) {   // the cp.async part of row n - 2 has landed
                    asm volatile("cp.async.wait_group 2;\n" ::: "memory");
                    asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
                    __syncwarp();
                    if (lane == 0) tc::arrive(full + 8 * ((n - 2) % NS));
                }
            }
            t += cnt;
        }
        tc::cp_wait_all();
        asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
        __syncwarp();
        if (lane == 0) {
            for (int k = n >= 2 ? n - 2 : 0; k < n; ++k) tc::arrive(full + 8 * (k % NS));
            // after a wait that ran out, the tensor-map copies in flight still write this CTA's memory
            if (!ok)
                for (int k = n > NS ? n - NS : 0; k < n; ++k) tc::bar_wait(full + 8 * (k % NS), (k / NS) & 1);
        }
    } else if (warp == kEpiWarps + 1) {   // ---- MMA issuer (one lane; the warp waits with it)
        int n = 0, o = 0;      // input rows, and output rows of the earlier runs
        bool ok = true;
        for (int t = t0; t < t1 && ok;) {
            const int cnt = min(t1 - t, H - t % H);
            // input row i of the run belongs to its output rows i - 2 (dh = +1), i - 1 and i (dh = -1)
            for (int i = 0; i < cnt + 2; ++i, ++n) {
                ok = tc::role_wait(full + 8 * (n % NS), (n / NS) & 1, gave_up);
                if (i < cnt)   // output row i starts here: its accumulator has been read
                    ok = ok && tc::role_wait(acce + 8 * ((o + i) % NA), (((o + i) / NA) & 1) ^ 1, gave_up);
                ok = __all_sync(0xffffffffu, ok);
                if (!ok) break;
                asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
                if (tc::elect_one()) {
                    constexpr bool SWZ = tc::Row<CIN>::SWZ;
                    const uint32_t ra = in_a + (uint32_t)((n % NS) * L::SLOT_BYTES + tc::Row<CIN>::MAIN);
                    const tc::Desc a0 = SWZ ? tc::sdesc128(ra - 128) : tc::sdesc(ra, tc::kPixS * 16, 128);
                    const tc::Desc b0 = tc::sdesc(w_a, L::NB * 16, 128);
                    // output rows jlo .. jhi; the ring's end may split them.  Everything that an MMA needs
                    // beyond a sum per descriptor is formed here, once per row: this thread shares its
                    // scheduler with the epilogue's warps (with the split worked out per MMA, a row's
                    // MMAs took 190 cycles each to issue)
                    const int jlo = max(i - 2, 0), jhi = min(i, cnt - 1);
                    const int s1 = (o + jlo) % NA, c1 = min(jhi - jlo + 1, NA - s1), c2 = jhi - jlo + 1 - c1;
                    const tc::Desc b1 = b0.at((jlo - (i - 2)) * COUT * 16), b2 = b1.at(c1 * COUT * 16);
                    const uint32_t d1 = tmem + (uint32_t)(s1 * COUT);   // the second part starts at slot 0
                    const uint32_t id1 = tc::idesc_n(c1 * COUT), id2 = tc::idesc_n(c2 * COUT);
                    // the first product starts output row i (an accumulator of its own, the last one)
                    if (i < cnt) {
                        const int sn = (o + i) % NA;
                        tc::mma(tmem + (uint32_t)(sn * COUT), a0, b0.at(2 * COUT * 16), tc::idesc<COUT>(), 0u);
                        const int m1 = c2 > 0 ? c1 : c1 - 1;            // earlier rows in each part
                        if (m1 > 0) tc::mma(d1, a0, b1, tc::idesc_n(m1 * COUT), 1u);
                        if (c2 > 1) tc::mma(tmem, a0, b2, tc::idesc<COUT>(), 1u);
                    } else {
                        tc::mma(d1, a0, b1, id1, 1u);
                        if (c2 > 0) tc::mma(tmem, a0, b2, id2, 1u);
                    }
#pragma unroll
                    for (int dw = 0; dw < 3; ++dw) {
#pragma unroll
                        for (int kc = 0; kc < CIN / 16; ++kc) {
                            if (dw == 0 && kc == 0) continue;
                            const tc::Desc a = a0.at(SWZ ? dw * 128 + kc * 32 : (2 * kc * tc::kPixS + dw) * 16);
                            const int bo = (dw * (CIN / 8) + 2 * kc) * L::NB * 16;
                            tc::mma(d1, a, b1.at(bo), id1, 1u);
                            if (c2 > 0) tc::mma(tmem, a, b2.at(bo), id2, 1u);
                        }
                    }
                    tc::commit(empty + 8 * (n % NS));
                    if (i >= 2) tc::commit(accf + 8 * ((o + i - 2) % NA));
                }
                __syncwarp();
            }
            o += cnt;
            t += cnt;
        }
        if (tc::elect_one()) {
            tc::commit(drained);   // every MMA issued, also after a wait that ran out
            tc::bar_wait(drained, 0);
        }
    }
    __syncwarp();
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    if (threadIdx.x == 0 && *gave_up) atomicOr(err, 1);
    if (warp == 0) {
        asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"((uint32_t)L::TMEM_COLS));
    }
}

// ---- all layers of an inference in one launch (small batches) --------------------------------
// When every tile (one image row segment) of a batch has a CTA of its own, the network runs as a
// single cooperative launch: CTA t computes tile t of every layer in turn.  Layer l of tile
// (b, h) needs layer l-1 of rows h-1, h, h+1: its own row is its own previous output, the other
// two come from the CTAs of the neighbouring rows, which publish each finished layer by
// incrementing their flag (release after a device-scope fence; the reader polls with an acquire
// load, bounded).  Flags count up across launches: a CTA reads its own flag at entry (every flag
// holds the same value between launches, since each launch adds L-1 to each) and waits for its
// neighbours' flags to reach that base + l.  Each layer writes its own activation buffer, so no
// row is overwritten while a neighbour may still read it.  The next layer's weights are fetched
// while the epilogue drains the accumulator.  A wait that runs out sets bit 2 of the error word
// and the CTA skips its remaining layers; its neighbours then run out too, so the launch ends.
constexpr int kMaxFusedLayers = 8;
constexpr long long kFlagLimit = 1LL << 21;

struct FusedArgs {
    const __nv_bfloat16* x;                       // input [B][H][W][ci[0]]
    __nv_bfloat16* act[kMaxFusedLayers];          // act[l]: input of layer l (l >= 1), [B][H][W][ci[l]]
    const __nv_bfloat16* wt[kMaxFusedLayers];     // [9][co][ci] BF16
    const float* bias[kMaxFusedLayers];
    int ci[kMaxFusedLayers], co[kMaxFusedLayers];
    int L, B, H, W, planar;
    float* y;                                     // last layer: planar [co][B*H*W] or [B][H][W][co]
    unsigned int* flags;                          // one per tile
    int* err;
};

namespace tc {
// shared-memory plan of the fused kernel: three row slots (rows h-1, h, h+1) of up to 64
// channels, one weight block, the accumulator barrier, FP32 and BF16 output staging; the
// operand region also covers reads under the swapped reading of the descriptor strides
struct FusedLay {
    static constexpr int SLOT_BYTES = 8 * kPixS * 16;
    static constexpr int IN_BYTES = 3 * SLOT_BYTES;
    static constexpr int W_OFF = (IN_BYTES + 1023) / 1024 * 1024;
    static constexpr int W_BYTES = 9 * 8 * 64 * 16;
    static constexpr int BAR_OFF = (W_OFF + W_BYTES + 1023) / 1024 * 1024;
    static constexpr int A_LAST = 2 * SLOT_BYTES + (6 * kPixS + 2) * 16;
    static constexpr int B_LAST = W_OFF + (8 * 8 + 8 - 2) * 64 * 16;
    static constexpr int A_END = A_LAST + imax(kPixS * 16 + 15 * 128, 15 * kPixS * 16 + 128) + 128;
    static constexpr int B_END = B_LAST + imax(64 * 16 + 7 * 128, 7 * 64 * 16 + 128) + 128;
    static constexpr int OPS_END = (imax(BAR_OFF + 64, imax(A_END, B_END)) + 1023) / 1024 * 1024;
    static constexpr int STF_OFF = OPS_END;
    static constexpr int STB_OFF = STF_OFF + kTileP * 64 * 4;
    static constexpr int SMEM = STB_OFF + kTileP * 64 * 2;
    static constexpr int TMEM_COLS = 64;
};

__device__ __forceinline__ bool wait_flag(const unsigned int* f, unsigned int target) {
    for (long long i = 0; i < kFlagLimit; ++i) {
        unsigned int v;
        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];\n" : "=r"(v) : "l"(f) : "memory");
        if ((int)(v - target) >= 0) return true;
        __nanosleep(64);
    }
    return false;
}
}  // namespace tc

// One layer of the fused inference for this CTA's tile.  Returns false if a wait ran out.
template <int CIN, int COUT, int EPI>
__device__ __forceinline__ bool fused_layer(const FusedArgs& a, int l, int t, int tup, int tdn, int b, int h, int w0,
                                            unsigned int base, uint32_t in_a, uint32_t w_a, uint32_t bar_a,
                                            uint32_t& phase, uint32_t tmem, unsigned char* stf, unsigned char* stb) {
    using FL = tc::FusedLay;
    const int H = a.H, W = a.W;
    const __nv_bfloat16* src = l == 0 ? a.x : a.act[l];
    // the own row needs no wait: it is this CTA's previous output (or the input)
    tc::fetch_row<CIN, kFusedThreads>(src, b, h, H, W, w0, in_a + (uint32_t)FL::SLOT_BYTES, threadIdx.x);
    tc::cp_commit();
    // the epilogue's bias columns, loaded while the rows and the MMAs are in flight
    const int warp = threadIdx.x / 32;
    constexpr int NCOL = epi_ncol<COUT, kFusedWarps>();
    float breg[NCOL];
    {
        const int n0 = epi_n0<COUT, kFusedWarps>(warp);
#pragma unroll
        for (int j = 0; j < NCOL; ++j) breg[j] = a.bias[l][n0 + j];
    }
    bool ok = true;
    if (l > 0 && threadIdx.x == 0)
        ok = tc::wait_flag(a.flags + tup, base + (unsigned)l) && tc::wait_flag(a.flags + tdn, base + (unsigned)l);
    if (__syncthreads_or(!ok)) {
        if (threadIdx.x == 0) atomicOr(a.err, 2);
        tc::cp_wait_all();
        return false;
    }
    tc::fetch_row<CIN, kFusedThreads>(src, b, (h - 1 + H) % H, H, W, w0, in_a, threadIdx.x);
    tc::fetch_row<CIN, kFusedThreads>(src, b, (h + 1) % H, H, W, w0, in_a + 2u * (uint32_t)FL::SLOT_BYTES, threadIdx.x);
    tc::cp_commit();
    tc::cp_wait_all();   // the rows and this layer's weights
    asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
    __syncthreads();
    if (warp == 0 && tc::elect_one()) {
        asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
        const uint32_t ra[3] = {in_a, in_a + (uint32_t)FL::SLOT_BYTES, in_a + 2u * (uint32_t)FL::SLOT_BYTES};
        tc::issue_tile<CIN, COUT>(tmem, ra, w_a, bar_a);
    }
    __syncwarp();
    ok = tc::bar_wait(bar_a, phase);
    phase ^= 1u;
    if (__syncthreads_or(!ok)) {
        if (threadIdx.x == 0) atomicOr(a.err, 1);
        tc::bar_wait(bar_a, phase ^ 1u);   // once more, bounded, before the caller frees the TMEM
        return false;
    }
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    // the MMAs have read the weights: fetch the next layer's while the accumulator drains
    if (l + 1 < a.L) {
        tc::fetch_weights<kFusedThreads>(a.wt[l + 1], a.ci[l + 1], a.co[l + 1], w_a);
        tc::cp_commit();
    }
    const size_t p0 = ((size_t)b * H + h) * W + w0;
    conv_tc_epilogue<CIN, COUT, EPI, kFusedWarps>(tmem, p0, breg, a.y, EPI == EPI_GELU_ACT ? a.act[l + 1] : nullptr,
                                                  stf, stb, (size_t)a.B * H * W);
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    if (l + 1 < a.L) {   // publish the row
        __threadfence();
        __syncthreads();
        if (threadIdx.x == 0) atomicAdd(a.flags + t, 1u);
    } else {
        __syncthreads();
    }
    return true;
}

template <int EPI>
__device__ __forceinline__ bool fused_dispatch(const FusedArgs& a, int l, int t, int tup, int tdn, int b, int h,
                                               int w0, unsigned int base, uint32_t in_a, uint32_t w_a, uint32_t bar_a,
                                               uint32_t& phase, uint32_t tmem, unsigned char* stf, unsigned char* stb) {
    const int ci = a.ci[l], co = a.co[l];
    if (ci == 16 && co == 64)
        return fused_layer<16, 64, EPI>(a, l, t, tup, tdn, b, h, w0, base, in_a, w_a, bar_a, phase, tmem, stf, stb);
    if (ci == 64 && co == 64)
        return fused_layer<64, 64, EPI>(a, l, t, tup, tdn, b, h, w0, base, in_a, w_a, bar_a, phase, tmem, stf, stb);
    if (ci == 64 && co == 16)
        return fused_layer<64, 16, EPI>(a, l, t, tup, tdn, b, h, w0, base, in_a, w_a, bar_a, phase, tmem, stf, stb);
    return fused_layer<16, 16, EPI>(a, l, t, tup, tdn, b, h, w0, base, in_a, w_a, bar_a, phase, tmem, stf, stb);
}

__global__ void __launch_bounds__(kFusedThreads, 1) k_cnn_fused(FusedArgs a) {
    QGN_PDL_ENTRY();
    using FL = tc::FusedLay;
    extern __shared__ __align__(1024) unsigned char smtc[];
    uint64_t* bar = reinterpret_cast<uint64_t*>(smtc + FL::BAR_OFF);
    uint32_t* tslot = reinterpret_cast<uint32_t*>(smtc + FL::BAR_OFF + 32);
    unsigned int* sbase = reinterpret_cast<unsigned int*>(smtc + FL::BAR_OFF + 40);
    const int warp = threadIdx.x / 32;
    const uint32_t bar_a = smem_u32(bar), in_a = smem_u32(smtc), w_a = smem_u32(smtc + FL::W_OFF);
    const int H = a.H, segs = a.W / kTileP;
    const int t = blockIdx.x;
    const int h = t % H, bs = t / H;
    const int w0 = (bs % segs) * kTileP, b = bs / segs;
    const int tup = t - h + (h - 1 + H) % H, tdn = t - h + (h + 1) % H;

    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(tslot)),
                     "r"((uint32_t)FL::TMEM_COLS));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n");
    }
    if (threadIdx.x == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(bar_a));
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
        unsigned int v;
        asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];\n" : "=r"(v) : "l"(a.flags + t) : "memory");
        *sbase = v;
    }
    tc::fetch_weights<kFusedThreads>(a.wt[0], a.ci[0], a.co[0], w_a);
    tc::cp_commit();
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    const uint32_t tmem = *tslot;
    const unsigned int base = *sbase;
    unsigned char* stf = smtc + FL::STF_OFF;
    unsigned char* stb = smtc + FL::STB_OFF;
    uint32_t phase = 0u;
    for (int l = 0; l < a.L; ++l) {
        bool ok;
        if (l + 1 < a.L)
            ok = fused_dispatch<EPI_GELU_ACT>(a, l, t, tup, tdn, b, h, w0, base, in_a, w_a, bar_a, phase, tmem, stf, stb);
        else if (a.planar)
            ok = fused_dispatch<EPI_PLANAR>(a, l, t, tup, tdn, b, h, w0, base, in_a, w_a, bar_a, phase, tmem, stf, stb);
        else
            ok = fused_dispatch<EPI_LINEAR>(a, l, t, tup, tdn, b, h, w0, base, in_a, w_a, bar_a, phase, tmem, stf, stb);
        if (!ok) break;
    }
    tc::cp_wait_all();
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    if (warp == 0) {
        asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"((uint32_t)FL::TMEM_COLS));
    }
}

// ---- weight gradient on tcgen05 -------------------------------------------------------------
// dW[dh, dw][n][k] = sum_p G[p][n] X[p + (dh, dw)][k] as MMAs over K = 16 pixels, both operands read
// MN-major (channels contiguous) straight from the NHWC rows staged as for the forward pass.  The M
// side G has 64 channels, X 16 or 64.  For the last layer (64 -> 16) the two change places: with q = p
// + tap the sum is over X[q] G[q - tap], the same with all taps mirrored (SWAP).
// An input row r of X belongs to the taps dh = +1, 0, -1 of the G rows r - 1, r, r + 1, so one CTA makes
// all nine taps from one pass over its rows: for every 16 pixels
//   [G row r-1; G row r] x X row r    M = 128: two rows of G as the two 64-channel blocks of the A
//                                     operand, their distance in the ring being the block stride (LBO);
//                                     zero blocks before and after the ring stand in for a row that is
//                                     not the CTA's, and for the second row where the ring wraps
//   G row r+1 x X row r               M = 64
// and, when X has 64 channels, its three horizontal taps are the three 64-column blocks of one B
// operand with N = 192, one pixel (128 bytes of the swizzled row) apart.  Operand bytes in shared memory
// are what an MMA costs: 18 KB per 16 pixels for the nine taps, 36 KB as nine products with M = N = 64.
// On B200 an M = 64 accumulator holds row m in TMEM lane 32 (m / 16) + m % 16; an MN-major no-swizzle
// descriptor takes the stride between 8-pixel (K) groups as its leading byte offset and the stride
// between 8-channel groups as its stride byte offset, a swizzled one the stride between 64-channel
// blocks and the stride between 8-pixel groups (measured with known operands).
// Roles as in k_conv_tc: a loader (one ring of X rows, one of G rows), an MMA issuer, and eight warps
// that sum G over the staged pixels (the bias gradient) while the MMAs run, then write the accumulators
// as one partial per chunk of at most kWgRows rows, which bounds the length of the FP32 sums in TMEM.
// 64 -> 64 at batch 32 on 128^2 (B200, ncu): one CTA per tap row 195 us with one stage in flight, 146 us
// with the roles split, 89 us with swizzled tensor-map rows and MMAs issued from uniform registers;
// this form 51 us with partials of 28 rows, its traffic alone 20.  16 rows, the mma.sync engine's length,
// keep the FP32 sums as short as there: six layers' gradients at batch 32 1.27 -> 1.32 ms.
constexpr int kWgRows = 16;          // most row segments per partial
namespace tc {
template <int CX>
struct WgLay {
    static constexpr int NX = 4, NG = 6;                   // ring slots
    static constexpr int XB = Row<CX>::BYTES, GB = kTileP * 128;
    static constexpr int Z1_OFF = 0;                       // zeros, below every G slot
    static constexpr int G_OFF = GB;
    static constexpr int Z2_OFF = G_OFF + NG * GB;         // zeros, above every G slot
    static constexpr int X_OFF = Z2_OFF + GB;
    static constexpr int SUM_OFF = X_OFF + NX * XB;        // bias sums [256][8]
    static constexpr int BAR_OFF = SUM_OFF + kDrainWarps * 32 * 8 * 4;
    static constexpr int SMEM = BAR_OFF + 256;
    static constexpr int N = 3 * CX;                       // accumulator columns of the three dw
    static constexpr int TMEM_COLS = 2 * N <= 128 ? 128 : 512;
    static_assert(Z2_OFF / 16 < (1 << 14), "block strides fit the descriptor");
    // reads of a no-swizzle X slot, under either reading of LBO/SBO
    static_assert(Row<CX>::SWZ || (16 * 7 + 2) * 16 + (CX / 8 - 1) * kPixS * 16 + 2 * 128 <= XB, "X reads");
};

// BF16 x BF16 -> F32, both operands MN-major
__host__ __device__ constexpr uint32_t idesc_mn(int m, int n) {
    return (1u << 4) | (1u << 7) | (1u << 10) | (1u << 15) | (1u << 16) | ((uint32_t)(n >> 3) << 17) |
           ((uint32_t)(m >> 4) << 24);
}
// an MN-major operand in the 128-byte swizzle: 64-channel blocks `block` bytes apart
__device__ __forceinline__ Desc sdesc128_mn(uint32_t saddr, uint32_t block) {
    return Desc{(saddr >> 4) | ((block >> 4) << 16), 64u | (1u << 14) | (2u << 29)};
}
}  // namespace tc

// part[chunk][tap][n][k] and bpart[chunk][n] over the chunk's row segments (ordered as the tiles of
// k_conv_tc), chunk = blockIdx.x, + gridDim.x, ...  SWAP: x is the 16-channel gradient, gr the
// 64-channel input, and part is [8 - tap][k][n] of what the kernel forms.
template <int CX, bool SWAP>
__global__ void __launch_bounds__(kWgThreads, 1)
    k_wgrad_tc(const __grid_constant__ CUtensorMap xmap, const __grid_constant__ CUtensorMap gmap,
               const __nv_bfloat16* __restrict__ x, int B, int H, int W, int rows_per_chunk, int chunks,
               float* __restrict__ part, float* __restrict__ bpart, int* __restrict__ err) {
    QGN_PDL_ENTRY();
    using L = tc::WgLay<CX>;
    constexpr int N = L::N, NX = L::NX, NG = L::NG;
    extern __shared__ __align__(1024) unsigned char smw[];
    uint32_t* tslot = reinterpret_cast<uint32_t*>(smw + L::BAR_OFF + 240);
    volatile int* gave_up = reinterpret_cast<volatile int*>(smw + L::BAR_OFF + 248);
    const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
    const uint32_t base_a = smem_u32(smw);
    const uint32_t fullx = smem_u32(smw + L::BAR_OFF), emptyx = fullx + 8 * NX, fullg = emptyx + 8 * NX,
                   emptyg = fullg + 8 * NG, accf = emptyg + 8 * NG, acce = accf + 8, drained = acce + 8;
    const int segs = W / kTileP;
    const int ntiles = B * H * segs;

    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(tslot)),
                     "r"((uint32_t)L::TMEM_COLS));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n");
    }
    if (threadIdx.x == 0) {
        *gave_up = 0;
        for (int i = 0; i < NX; ++i) {
            tc::bar_init(fullx + 8 * i, tc::row_arrivals<CX>());
            tc::bar_init(emptyx + 8 * i, SWAP ? 1 + kDrainWarps : 1);
        }
        for (int i = 0; i < NG; ++i) {
            tc::bar_init(fullg + 8 * i, 1);
            tc::bar_init(emptyg + 8 * i, SWAP ? 1 : 1 + kDrainWarps);
        }
        tc::bar_init(accf, 1);
        tc::bar_init(acce, kDrainWarps);
        tc::bar_init(drained, 1);
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    for (int i = threadIdx.x; i < L::GB / 16; i += kWgThreads) {
        *reinterpret_cast<uint4*>(smw + L::Z1_OFF + i * 16) = make_uint4(0, 0, 0, 0);
        *reinterpret_cast<uint4*>(smw + L::Z2_OFF + i * 16) = make_uint4(0, 0, 0, 0);
    }
    asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    const uint32_t tmem = *tslot;

    // Every role walks the same rows: the chunk's runs of consecutive rows of one (b, seg), cnt G rows
    // and cnt + 2 X rows each; X row i of a run goes with the G rows i - 2, i - 1 and i.
    bool ok = true;
    if (warp < kDrainWarps) {   // ---- bias sums, then the accumulators
        // sums: channel group tid % GROUPS, every PX-th pixel of the staged gradient rows
        constexpr int GROUPS = SWAP ? CX / 8 : 8, PX = kDrainWarps * 32 / GROUPS;
        const int c8 = threadIdx.x % GROUPS, pq = threadIdx.x / GROUPS;
        int n = 0, e = 0;      // rows summed, chunks done
        for (int c = blockIdx.x; c < chunks && ok; c += gridDim.x, ++e) {
            float bs[8] = {};
            const int t1 = min(ntiles, (c + 1) * rows_per_chunk);
            for (int t = c * rows_per_chunk; t < t1 && ok;) {
                const int cnt = min(t1 - t, H - t % H);
                for (int i = 0; i < (SWAP ? cnt + 2 : cnt); ++i, ++n) {
                    const uint32_t f = SWAP ? fullx + 8 * (n % NX) : fullg + 8 * (n % NG);
                    ok = __all_sync(0xffffffffu, tc::role_wait(f, (n / (SWAP ? NX : NG)) & 1, gave_up));
                    if (!ok) break;
                    if (!SWAP || (i >= 1 && i <= cnt)) {   // (the halo rows are other rows' gradients)
                        const unsigned char* s = SWAP ? smw + L::X_OFF + (n % NX) * L::XB : smw + L::G_OFF + (n % NG) * L::GB;
#pragma unroll
                        for (int p0 = 0; p0 < kTileP; p0 += PX) {
                            const int px = p0 + pq;
                            const uint4 v = *reinterpret_cast<const uint4*>(
                                s + (SWAP ? (c8 * tc::kPixS + px + 1) * 16 : px * 128 + ((c8 ^ (px & 7)) * 16)));
                            const __nv_bfloat162* p = reinterpret_cast<const __nv_bfloat162*>(&v);
#pragma unroll
                            for (int k = 0; k < 4; ++k) {
                                const float2 q = __bfloat1622float2(p[k]);
                                bs[2 * k] += q.x;
                                bs[2 * k + 1] += q.y;
                            }
                        }
                    }
                    __syncwarp();
                    if (lane == 0) tc::arrive(SWAP ? emptyx + 8 * (n % NX) : emptyg + 8 * (n % NG));
                }
                t += cnt;
            }
            ok = ok && __all_sync(0xffffffffu, tc::role_wait(accf, e & 1, gave_up));
            if (ok) {
                asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
                // warp w reads TMEM lanes 32 (w % 4) .. and half of the columns.  First accumulator: rows
                // 0..63 dh = +1, 64..127 dh = 0; second (M = 64, lanes 0..15 of each quarter): dh = -1
                constexpr int HALF = N / 2, STEP = HALF % 16 == 0 ? 16 : 8;
                const int q4 = warp % 4, c0 = (warp / 4) * HALF;
                float* out = part + (size_t)c * 9 * 64 * CX;
#pragma unroll
                for (int d = 0; d < 2; ++d) {
                    const int m = d == 0 ? (32 * q4 + lane) % 64 : 16 * q4 + lane;
                    const int dh = d == 0 ? (q4 < 2 ? 1 : 0) : -1;
                    for (int cc = 0; cc < HALF; cc += STEP) {
                        float v[STEP];
                        const uint32_t ta = tmem + ((uint32_t)(32 * q4) << 16) + (uint32_t)(d * N + c0 + cc);
                        if constexpr (STEP == 16) tc::tmem_ld<16>(ta, v);
                        else tc::tmem_ld8(ta, v);
                        if (d == 0 || lane < 16) {
                            const int dw = (c0 + cc) / CX, k = (c0 + cc) % CX;   // (a step stays in one tap)
                            const int tap = 3 * (dh + 1) + dw;
                            if constexpr (SWAP) {
#pragma unroll
                                for (int j = 0; j < STEP; ++j) out[((size_t)(8 - tap) * CX + k + j) * 64 + m] = v[j];
                            } else {
                                float4* o = reinterpret_cast<float4*>(out + ((size_t)tap * 64 + m) * CX + k);
#pragma unroll
                                for (int j = 0; j < STEP / 4; ++j)
                                    o[j] = make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
                            }
                        }
                    }
                }
                asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
                __syncwarp();
                if (lane == 0) tc::arrive(acce);
            }
            // the channels' sums over the warps' threads, in a fixed order (every warp comes here, also
            // after a wait that ran out: `ok` then ends the loop)
            float* sb = reinterpret_cast<float*>(smw + L::SUM_OFF);
#pragma unroll
            for (int k = 0; k < 8; ++k) sb[threadIdx.x * 8 + k] = bs[k];
            asm volatile("bar.sync 1, %0;\n" ::"r"(kDrainWarps * 32) : "memory");
            if (threadIdx.x < GROUPS * 8) {
                float s = 0.f;
                for (int q = 0; q < PX; ++q) s += sb[(q * GROUPS + threadIdx.x / 8) * 8 + threadIdx.x % 8];
                bpart[(size_t)c * GROUPS * 8 + threadIdx.x] = s;
            }
            uint32_t any;           // the warps leave the loop together
            asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.u32 q, %1, 0;\n\tbar.red.or.pred p, 1, %2, q;\n\t"
                         "selp.u32 %0, 1, 0, p;\n\t}\n"
                         : "=r"(any)
                         : "r"(ok ? 0u : 1u), "r"(kDrainWarps * 32)
                         : "memory");
            ok = any == 0;
        }
    } else if (warp == kDrainWarps) {   // ---- loader
        int n = 0, ng = 0;     // X rows and G rows issued
        for (int c = blockIdx.x; c < chunks && ok; c += gridDim.x) {
            const int t1 = min(ntiles, (c + 1) * rows_per_chunk);
            for (int t = c * rows_per_chunk; t < t1 && ok;) {
                const int h0 = t % H, bs = t / H;
                const int cnt = min(t1 - t, H - h0);
                const int b = bs / segs, w0 = (bs % segs) * kTileP;
                for (int i = 0; i < cnt + 2; ++i, ++n) {
                    ok = tc::role_wait(emptyx + 8 * (n % NX), ((n / NX) & 1) ^ 1, gave_up);
                    if (i < cnt) ok = ok && tc::role_wait(emptyg + 8 * (ng % NG), ((ng / NG) & 1) ^ 1, gave_up);
                    ok = __all_sync(0xffffffffu, ok);
                    if (!ok) break;
                    if (i < cnt) {
                        if (lane == 0) {
                            tc::arrive_tx(fullg + 8 * (ng % NG), L::GB);
                            tc::tma_row(base_a + (uint32_t)(L::G_OFF + (ng % NG) * L::GB), &gmap, w0, b * H + h0 + i,
                                        fullg + 8 * (ng % NG));
                        }
                        ++ng;
                    }
                    tc::load_row_warp<CX>(&xmap, x, b * H + (h0 - 1 + i + H) % H, W, w0,
                                          base_a + (uint32_t)(L::X_OFF + (n % NX) * L::XB), fullx + 8 * (n % NX), lane);
                    if (n >= 2) {   // the cp.async part of row n - 2 has landed
                        asm volatile("cp.async.wait_group 2;\n" ::: "memory");
                        asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
                        __syncwarp();
                        if (lane == 0) tc::arrive(fullx + 8 * ((n - 2) % NX));
                    }
                }
                t += cnt;
            }
        }
        tc::cp_wait_all();
        asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
        __syncwarp();
        if (lane == 0) {
            for (int k = n >= 2 ? n - 2 : 0; k < n; ++k) tc::arrive(fullx + 8 * (k % NX));
            // after a wait that ran out, the tensor-map copies in flight still write this CTA's memory
            if (!ok) {
                for (int k = n > NX ? n - NX : 0; k < n; ++k) tc::bar_wait(fullx + 8 * (k % NX), (k / NX) & 1);
                for (int k = ng > NG ? ng - NG : 0; k < ng; ++k) tc::bar_wait(fullg + 8 * (k % NG), (k / NG) & 1);
            }
        }
    } else {   // ---- MMA issuer (one lane; the warp waits with it)
        int n = 0, g0 = 0, e = 0;   // X rows, G rows of the earlier runs, chunks
        for (int c = blockIdx.x; c < chunks && ok; c += gridDim.x, ++e) {
            const int t1 = min(ntiles, (c + 1) * rows_per_chunk);
            ok = __all_sync(0xffffffffu, tc::role_wait(acce, (e & 1) ^ 1, gave_up));
            uint32_t more1 = 0u, more2 = 0u;   // the accumulators hold earlier sums of this chunk
            for (int t = c * rows_per_chunk; t < t1 && ok;) {
                const int cnt = min(t1 - t, H - t % H);
                for (int i = 0; i < cnt + 2; ++i, ++n) {
                    ok = tc::role_wait(fullx + 8 * (n % NX), (n / NX) & 1, gave_up);
                    if (i < cnt) ok = ok && tc::role_wait(fullg + 8 * ((g0 + i) % NG), ((g0 + i) / NG) & 1, gave_up);
                    ok = __all_sync(0xffffffffu, ok);
                    if (!ok) break;
                    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
                    const bool pair = i >= 1;   // G row i - 1 or i - 2 exists
                    if (tc::elect_one()) {
                        constexpr bool XS = tc::Row<CX>::SWZ;
                        const uint32_t xs = base_a + (uint32_t)(L::X_OFF + (n % NX) * L::XB);
                        const tc::Desc x0 = XS ? tc::sdesc128_mn(xs + tc::Row<CX>::MAIN - 128, 128)
                                               : tc::sdesc(xs, 128, tc::kPixS * 16);
                        const uint32_t gs = base_a + (uint32_t)L::G_OFF, z1 = base_a + (uint32_t)L::Z1_OFF,
                                       z2 = base_a + (uint32_t)L::Z2_OFF;
                        // the 16-pixel products of one A operand with the X row (slot pixel 0 is w0 - 1)
                        auto products = [&](uint32_t d, tc::Desc a, int m, uint32_t accumulate) {
#pragma unroll
                            for (int kc = 0; kc < kTileP / 16; ++kc) {
                                if constexpr (XS) {
                                    tc::mma(d, a.at(kc * 2048), x0.at(kc * 2048), tc::idesc_mn(m, N),
                                            kc > 0 ? 1u : accumulate);
                                } else {
#pragma unroll
                                    for (int dw = 0; dw < 3; ++dw)
                                        tc::mma(d + (uint32_t)(dw * CX), a.at(kc * 2048), x0.at((16 * kc + dw) * 16),
                                                tc::idesc_mn(m, CX), kc > 0 ? 1u : accumulate);
                                }
                            }
                        };
                        if (i < cnt) products(tmem + (uint32_t)N, tc::sdesc128_mn(gs + (uint32_t)(((g0 + i) % NG) * L::GB), 128), 64, more2);
                        if (pair) {
                            const uint32_t ga = gs + (uint32_t)(((g0 + i + 2 * NG - 2) % NG) * L::GB);   // row i - 2
                            const uint32_t gb = gs + (uint32_t)(((g0 + i + NG - 1) % NG) * L::GB);       // row i - 1
                            const bool ha = i >= 2, hb = i - 1 < cnt;
                            if (ha && hb && gb > ga) {
                                products(tmem, tc::sdesc128_mn(ga, gb - ga), 128, more1);
                            } else {
                                if (ha) products(tmem, tc::sdesc128_mn(ga, z2 - ga), 128, more1);
                                if (hb) products(tmem, tc::sdesc128_mn(z1, gb - z1), 128, ha ? 1u : more1);
                            }
                        }
                        tc::commit(emptyx + 8 * (n % NX));
                        if (i >= 2) tc::commit(emptyg + 8 * ((g0 + i - 2) % NG));
                    }
                    __syncwarp();
                    more2 = 1u;
                    if (pair) more1 = 1u;
                }
                g0 += cnt;
                t += cnt;
            }
            if (ok && tc::elect_one()) tc::commit(accf);
            __syncwarp();
        }
        if (tc::elect_one()) {
            tc::commit(drained);   // every MMA issued, also after a wait that ran out
            tc::bar_wait(drained, 0);
        }
    }
    __syncwarp();
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    if (threadIdx.x == 0 && *gave_up) atomicOr(err, 4);
    if (warp == 0) {
        asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"((uint32_t)L::TMEM_COLS));
    }
}

template <int CIN, int COUT>
constexpr int conv_smem() {
    return (9 * COUT + 3 * (kTileP + 2)) * RowPad<CIN>::LD * 2;
}
template <int CIN, int COUT>
constexpr int wgrad_smem() {
    return ((kTileP + 2) * RowPad<CIN>::LD + kTileP * RowPad<COUT>::LD) * 2;
}

}  // namespace cnn
}  // namespace qgn

using namespace qgn;
using namespace qgn::cnn;

struct qgn_cnn {
    int cin = 0, width = 0, cout = 0, layers = 0;   // real channel counts
    int H = 0, W = 0, max_batch = 0;
    int device = 0;
    cudaStream_t stream = nullptr;
    std::vector<int> ci, co;                         // padded channel counts per layer
    std::vector<float*> w, bias, mw, vw, mb, vb, gw, gb;
    std::vector<__nv_bfloat16*> wf, wb;
    std::vector<float*> z;                           // per layer (FP32): GELU'(pre-activation); last: the output
    std::vector<__nv_bfloat16*> act;                 // act[0] = input batch, act[l+1] = GELU(z[l])
    __nv_bfloat16* gA = nullptr;                     // backward: G of the current layer
    __nv_bfloat16* gB = nullptr;
    float* grads = nullptr;                          // gw and gb of every layer, as in qgn_cnn_get_weights
    float* part = nullptr;                           // weight-gradient partials
    float* bpart = nullptr;                          // bias-gradient partials
    size_t part_elems = 0;
    double* loss_part = nullptr;
    double* loss_host = nullptr;
    float* ytgt = nullptr;                           // gathered targets
    long long adam_t = 0;
    int engine = 0;                                  // 0: tcgen05, all layers in one launch when the
                                                     // tiles fit one CTA each; 1: mma.sync; 2: tcgen05
                                                     // one launch per layer
    int* d_err = nullptr;                            // device error word of the tcgen05 kernels
    unsigned int* flags = nullptr;                   // per-tile layer counters of the fused inference
    int fused_tiles = -1;                            // tile count the flags were last used with
    int fused_max_tiles = 0;                         // co-resident CTAs of the fused kernel
    std::vector<void*> owned;
    std::string last_error;
};

namespace {

int cnn_err(qgn_cnn* n, int code, const std::string& m) {
    if (n) n->last_error = m;
    return code;
}

#define NCK(call)                                                                                      \
    do {                                                                                               \
        cudaError_t _e = (call);                                                                       \
        if (_e != cudaSuccess) return cnn_err(net, QGN_ERR_CUDA, std::string(#call) + ": " + cudaGetErrorString(_e)); \
    } while (0)

int pad16(int c) { return (c + 15) / 16 * 16; }

template <class T>
cudaError_t nalloc(qgn_cnn* net, T** p, size_t count) {
    cudaError_t e = cudaMalloc((void**)p, sizeof(T) * (count ? count : 1));
    if (e == cudaSuccess) {
        net->owned.push_back(*p);
        cudaMemsetAsync(*p, 0, sizeof(T) * (count ? count : 1), net->stream);
    }
    return e;
}

size_t npix(const qgn_cnn* n, int batch) { return (size_t)batch * n->H * n->W; }

int conv_grid(const qgn_cnn* n, int batch) {
    const int tiles = batch * n->H * (n->W / kTileP);
    return std::max(1, std::min(tiles, 148));
}

// The tensor map of `rows` image rows of W pixels x 64 channels (BF16, NHWC), copied 128 pixels at a
// time into the 128-byte swizzle
cudaError_t row_map(const __nv_bfloat16* p, int W, int rows, CUtensorMap* map) {
    const cuuint64_t dims[3] = {64, (cuuint64_t)W, (cuuint64_t)rows}, strides[2] = {128, (cuuint64_t)W * 128};
    const cuuint32_t box[3] = {64, kTileP, 1};
    return tensor_map(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, p, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_128B);
}

template <int CIN, int COUT, int EPI>
cudaError_t launch_conv_t(qgn_cnn* n, const __nv_bfloat16* x, const __nv_bfloat16* wt, const float* bias, int batch,
                          float* outf, __nv_bfloat16* outb, const float* dact) {
    if (n->engine != 1) {
        constexpr int SM = tc::Lay<CIN, COUT>::SMEM;
        if (cudaError_t e = smem_opt_in(k_conv_tc<CIN, COUT, EPI>, SM); e != cudaSuccess) return e;
        CUtensorMap map = {};
        if (CIN == 64)
            if (cudaError_t e = row_map(x, n->W, batch * n->H, &map); e != cudaSuccess) return e;
        ::qgn::launch(k_conv_tc<CIN, COUT, EPI>, conv_grid(n, batch), kConvThreads, SM, n->stream, map, x, wt, bias, batch,
                      n->H, n->W, outf, outb, dact, n->d_err);
        return cudaGetLastError();
    }
    constexpr int SM = conv_smem<CIN, COUT>();
    if (cudaError_t e = smem_opt_in(k_conv<CIN, COUT, EPI>, SM); e != cudaSuccess) return e;
    ::qgn::launch(k_conv<CIN, COUT, EPI>, conv_grid(n, batch), kThreads, SM, n->stream, x, wt, bias, batch, n->H, n->W, outf,
                                                                             outb, dact);
    return cudaGetLastError();
}

// the layers of a network of width 64: 16 or 64 channels in and 64 out, or (the last) 64 in, 16 out
template <int EPI>
cudaError_t launch_conv(qgn_cnn* n, int cin, int cout, const __nv_bfloat16* x, const __nv_bfloat16* wt,
                        const float* bias, int batch, float* outf, __nv_bfloat16* outb, const float* dact) {
    if constexpr (EPI == EPI_LINEAR || EPI == EPI_PLANAR) {
        if (cin == 64 && cout == 16) return launch_conv_t<64, 16, EPI>(n, x, wt, bias, batch, outf, outb, dact);
    } else {
        if (cin == 16 && cout == 64) return launch_conv_t<16, 64, EPI>(n, x, wt, bias, batch, outf, outb, dact);
        if (cin == 64 && cout == 64) return launch_conv_t<64, 64, EPI>(n, x, wt, bias, batch, outf, outb, dact);
    }
    return cudaErrorInvalidValue;
}

// partials of the tcgen05 weight gradient: row segments per partial and their number
int wg_rows(const qgn_cnn* n, int batch) {
    const int tiles = batch * n->H * (n->W / kTileP);
    const int waves = (tiles + 148 * kWgRows - 1) / (148 * kWgRows);   // the fewest with partials that short
    return (tiles + 148 * waves - 1) / (148 * waves);
}
int wg_chunks(const qgn_cnn* n, int batch) {
    const int tiles = batch * n->H * (n->W / kTileP), r = wg_rows(n, batch);
    return (tiles + r - 1) / r;
}

// weight-gradient partials of one layer into part (*nchunks of them); the tcgen05 kernel also leaves
// as many bias-gradient partials in bpart
template <int CX, bool SWAP>
cudaError_t launch_wgrad_tc(qgn_cnn* n, const __nv_bfloat16* x, const __nv_bfloat16* g, int batch, int* nchunks) {
    constexpr int SM = tc::WgLay<CX>::SMEM;
    if (cudaError_t e = smem_opt_in(k_wgrad_tc<CX, SWAP>, SM); e != cudaSuccess) return e;
    CUtensorMap xm = {}, gm = {};
    if (CX == 64)
        if (cudaError_t e = row_map(x, n->W, batch * n->H, &xm); e != cudaSuccess) return e;
    if (cudaError_t e = row_map(g, n->W, batch * n->H, &gm); e != cudaSuccess) return e;
    const int chunks = *nchunks = wg_chunks(n, batch);
    ::qgn::launch(k_wgrad_tc<CX, SWAP>, std::min(chunks, 148), kWgThreads, SM, n->stream, xm, gm, x, batch, n->H, n->W,
                  wg_rows(n, batch), chunks, n->part, n->bpart, n->d_err);
    return cudaGetLastError();
}

template <int CIN, int COUT>
cudaError_t launch_wgrad_t(qgn_cnn* n, const __nv_bfloat16* x, const __nv_bfloat16* g, int batch, int* nchunks) {
    if (n->engine != 1) {
        if constexpr (COUT == 64) return launch_wgrad_tc<CIN, false>(n, x, g, batch, nchunks);
        else return launch_wgrad_tc<COUT, true>(n, g, x, batch, nchunks);
    }
    const int chunks = (batch * n->H + kWChunkRows - 1) / kWChunkRows;
    *nchunks = chunks;
    constexpr int SM = wgrad_smem<CIN, COUT>();
    if (cudaError_t e = smem_opt_in(k_wgrad<CIN, COUT>, SM); e != cudaSuccess) return e;
    ::qgn::launch(k_wgrad<CIN, COUT>, dim3(chunks, 9), kThreads, SM, n->stream, x, g, batch, n->H, n->W, n->part);
    return cudaGetLastError();
}

cudaError_t launch_wgrad(qgn_cnn* n, int cin, int cout, const __nv_bfloat16* x, const __nv_bfloat16* g, int batch,
                         int* nchunks) {
    if (cin == 16 && cout == 64) return launch_wgrad_t<16, 64>(n, x, g, batch, nchunks);
    if (cin == 64 && cout == 64) return launch_wgrad_t<64, 64>(n, x, g, batch, nchunks);
    if (cin == 64 && cout == 16) return launch_wgrad_t<64, 16>(n, x, g, batch, nchunks);
    return cudaErrorInvalidValue;
}

// forward of a batch: layer 0 reads x0 (default act[0]); the last layer's FP32 output goes
// to ylast (default z[L-1]).  grads: the hidden layers' GELU' go to z[l] for the backward pass.
int forward(qgn_cnn* net, int batch, bool grads, const __nv_bfloat16* x0 = nullptr, float* ylast = nullptr,
            bool planar = false) {
    const int L = net->layers;
    for (int l = 0; l < L; ++l) {
        const bool last = l == L - 1;
        const __nv_bfloat16* in = (l == 0 && x0) ? x0 : net->act[l];
        float* y = ylast ? ylast : net->z[l];
        const int ci = net->ci[l], co = net->co[l];
        cudaError_t e =
            last && planar ? launch_conv<EPI_PLANAR>(net, ci, co, in, net->wf[l], net->bias[l], batch, y, nullptr, nullptr)
            : last    ? launch_conv<EPI_LINEAR>(net, ci, co, in, net->wf[l], net->bias[l], batch, y, nullptr, nullptr)
            : grads   ? launch_conv<EPI_GELU>(net, ci, co, in, net->wf[l], net->bias[l], batch, net->z[l],
                                              net->act[l + 1], nullptr)
                      : launch_conv<EPI_GELU_ACT>(net, ci, co, in, net->wf[l], net->bias[l], batch, nullptr,
                                                  net->act[l + 1], nullptr);
        NCK(e);
    }
    return QGN_OK;
}

// backward from the BF16 output gradient in gA; fills gw/gb of every layer
int backward(qgn_cnn* net, int batch) {
    const int L = net->layers;
    __nv_bfloat16* gcur = net->gA;
    __nv_bfloat16* gnext = net->gB;
    const long long np = (long long)npix(net, batch);
    for (int l = L - 1; l >= 0; --l) {
        int chunks = 0;
        NCK(launch_wgrad(net, net->ci[l], net->co[l], net->act[l], gcur, batch, &chunks));
        const int nw = 9 * net->co[l] * net->ci[l];
        const float* bpart = net->bpart;
        int nbias = chunks;
        if (net->engine == 1) {
            const int ppb = 1024;
            nbias = (int)((np + ppb - 1) / ppb);
            ::qgn::launch(k_bias_part, nbias, 64, 0, net->stream, gcur, np, net->co[l], ppb, net->part + (size_t)chunks * nw);
            NCK(cudaGetLastError());
            bpart = net->part + (size_t)chunks * nw;
        }
        ::qgn::launch(k_reduce_wgrad, (nw + kRedOut - 1) / kRedOut + 1, 4 * kRedOut, 0, net->stream, net->part, chunks, nw,
                      net->gw[l], bpart, nbias, net->co[l], net->gb[l]);
        NCK(cudaGetLastError());
        if (l > 0) {
            NCK(launch_conv<EPI_GELU_GRAD>(net, net->co[l], net->ci[l], gcur, net->wb[l], nullptr, batch, nullptr,
                                           gnext, net->z[l - 1]));
            std::swap(gcur, gnext);
        }
    }
    return QGN_OK;
}

int mse(qgn_cnn* net, int batch, const float* tgt) {
    const int L = net->layers;
    const long long np = (long long)npix(net, batch);
    const int C = net->co[L - 1];
    const double inv = 1.0 / ((double)np * net->cout);
    ::qgn::launch(k_mse, 148, kMseThreads, 0, net->stream, net->z[L - 1], tgt, np, C, net->cout, inv, net->gA, net->loss_part);
    NCK(cudaGetLastError());
    return QGN_OK;
}

int check_err(qgn_cnn* net) {
    int h = 0;
    NCK(cudaMemcpyAsync(&h, net->d_err, sizeof(int), cudaMemcpyDeviceToHost, net->stream));
    NCK(cudaStreamSynchronize(net->stream));
    if (h) {
        net->fused_tiles = -1;   // the layer counters may be uneven: the next fused launch clears them
        NCK(cudaMemsetAsync(net->d_err, 0, sizeof(int), net->stream));   // reported once
        return cnn_err(net, QGN_ERR_CUDA,
                       (h & 2)   ? "the fused inference timed out waiting for a neighbouring row"
                       : (h & 4) ? "a tensor-core weight gradient timed out waiting for its MMAs"
                                 : "a tensor-core convolution timed out waiting for its MMAs");
    }
    return QGN_OK;
}

// the fused single-launch inference applies: tcgen05 engine, at most kMaxFusedLayers layers,
// 128-pixel row segments, at least 3 rows, and one co-resident CTA per tile
bool fused_ok(qgn_cnn* net, int batch) {
    if (net->engine != 0 || net->layers > kMaxFusedLayers || net->H < 3 || net->W % kTileP != 0) return false;
    if (net->fused_max_tiles == 0) {
        int dev = 0, sms = 0, per = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        if (smem_opt_in(k_cnn_fused, tc::FusedLay::SMEM) != cudaSuccess ||
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_cnn_fused, kFusedThreads, tc::FusedLay::SMEM) !=
                cudaSuccess)
            per = 0;
        net->fused_max_tiles = per > 0 ? sms * per : -1;
    }
    return (long long)batch * net->H * (net->W / kTileP) <= net->fused_max_tiles;
}

int forward_fused(qgn_cnn* net, int batch, const __nv_bfloat16* x, float* y, bool planar) {
    const int L = net->layers;
    const int tiles = batch * net->H * (net->W / kTileP);
    if (tiles != net->fused_tiles) {
        NCK(cudaMemsetAsync(net->flags, 0, sizeof(unsigned int) * tiles, net->stream));
        net->fused_tiles = tiles;
    }
    FusedArgs a = {};
    a.x = x;
    for (int l = 0; l < L; ++l) {
        a.act[l] = net->act[l];
        a.wt[l] = net->wf[l];
        a.bias[l] = net->bias[l];
        a.ci[l] = net->ci[l];
        a.co[l] = net->co[l];
    }
    a.L = L;
    a.B = batch;
    a.H = net->H;
    a.W = net->W;
    a.planar = planar ? 1 : 0;
    a.y = y;
    a.flags = net->flags;
    a.err = net->d_err;
    // cooperative: every CTA is resident at once, which the waits on neighbouring rows need
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(tiles);
    cfg.blockDim = dim3(kFusedThreads);
    cfg.dynamicSmemBytes = tc::FusedLay::SMEM;
    cfg.stream = net->stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    NCK(smem_opt_in(k_cnn_fused, tc::FusedLay::SMEM));   // per device: a no-op after the first
    NCK(cudaLaunchKernelEx(&cfg, k_cnn_fused, a));
    return QGN_OK;
}

int read_loss(qgn_cnn* net, double* loss) {
    NCK(cudaMemcpyAsync(net->loss_host, net->loss_part, sizeof(double) * 148, cudaMemcpyDeviceToHost, net->stream));
    NCK(cudaStreamSynchronize(net->stream));
    if (int rc = check_err(net)) return rc;
    double s = 0.0;
    for (int i = 0; i < 148; ++i) s += net->loss_host[i];
    if (loss) *loss = s;
    return QGN_OK;
}

}  // namespace

namespace qgn {
namespace cnn {
int padded_in(const qgn_cnn* net) { return net->ci[0]; }
int padded_out(const qgn_cnn* net) { return net->co[net->layers - 1]; }
int height(const qgn_cnn* net) { return net->H; }
int width(const qgn_cnn* net) { return net->W; }
int real_out(const qgn_cnn* net) { return net->cout; }
int infer(qgn_cnn* net, const void* x, float* y, int batch, cudaStream_t stream, bool planar) {
    if (batch < 1 || batch > net->max_batch) return QGN_ERR_ARG;
    cudaStream_t own = net->stream;
    net->stream = stream;
    const __nv_bfloat16* xb = static_cast<const __nv_bfloat16*>(x);
    const int rc = fused_ok(net, batch) ? forward_fused(net, batch, xb, y, planar) : forward(net, batch, false, xb, y, planar);
    net->stream = own;
    return rc;
}
}  // namespace cnn
}  // namespace qgn

extern "C" {

int qgn_cnn_create(int cin, int width, int cout, int layers, int H, int W, int max_batch, unsigned long long seed,
                   qgn_cnn** out) {
    if (!out) return QGN_ERR_ARG;
    *out = nullptr;
    if (cin < 1 || cin > 16 || cout < 1 || cout > 16 || width != 64 || layers < 2 || layers > 16) return QGN_ERR_CONFIG;
    if (H < 1 || W < kTileP || W % kTileP != 0 || max_batch < 1) return QGN_ERR_CONFIG;
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev < 1) return QGN_ERR_NO_DEVICE;
    qgn_cnn* net = new (std::nothrow) qgn_cnn();
    if (!net) return QGN_ERR_CUDA;
    net->cin = cin;
    net->width = width;
    net->cout = cout;
    net->layers = layers;
    net->H = H;
    net->W = W;
    net->max_batch = max_batch;
    cudaGetDevice(&net->device);
    auto fail = [&](int code) {
        qgn_cnn_destroy(net);
        return code;
    };
    if (cudaStreamCreateWithFlags(&net->stream, cudaStreamNonBlocking) != cudaSuccess) return fail(QGN_ERR_CUDA);
    for (int l = 0; l < layers; ++l) {
        net->ci.push_back(l == 0 ? pad16(cin) : width);
        net->co.push_back(l == layers - 1 ? pad16(cout) : width);
    }
    const size_t NP = npix(net, max_batch);
    net->w.resize(layers); net->bias.resize(layers); net->mw.resize(layers); net->vw.resize(layers);
    net->mb.resize(layers); net->vb.resize(layers); net->gw.resize(layers); net->gb.resize(layers);
    net->wf.resize(layers); net->wb.resize(layers); net->z.resize(layers); net->act.resize(layers + 1);
    size_t part = 0;
    // gradients in one allocation, in the order of qgn_cnn_get_weights: one copy reads them back
    size_t np = 0;
    for (int l = 0; l < layers; ++l) np += 9ull * net->co[l] * net->ci[l] + net->co[l];
    if (nalloc(net, &net->grads, np)) return fail(QGN_ERR_CUDA);
    np = 0;
    for (int l = 0; l < layers; ++l) {
        net->gw[l] = net->grads + np;
        np += 9ull * net->co[l] * net->ci[l];
        net->gb[l] = net->grads + np;
        np += net->co[l];
    }
    // most partials of any batch up to max_batch: 148 in every wave of CTAs
    const size_t max_chunks = 148 * (((size_t)max_batch * H * (W / kTileP) + 148 * kWgRows - 1) / (148 * kWgRows));
    std::mt19937_64 rng(seed);
    for (int l = 0; l < layers; ++l) {
        const int nw = 9 * net->co[l] * net->ci[l];
        if (nalloc(net, &net->w[l], nw) || nalloc(net, &net->mw[l], nw) || nalloc(net, &net->vw[l], nw) ||
            nalloc(net, &net->wf[l], nw) || nalloc(net, &net->wb[l], nw) ||
            nalloc(net, &net->bias[l], net->co[l]) || nalloc(net, &net->mb[l], net->co[l]) ||
            nalloc(net, &net->vb[l], net->co[l]) || nalloc(net, &net->z[l], NP * net->co[l]) || nalloc(net, &net->act[l], NP * net->ci[l]))
            return fail(QGN_ERR_CUDA);
        // He initialisation over the real fan-in, zeros in padded channels
        const int real_in = l == 0 ? cin : width, real_out = l == layers - 1 ? cout : width;
        std::normal_distribution<float> nd(0.f, std::sqrt(2.0f / (9.0f * real_in)) * (l == layers - 1 ? 0.1f : 1.0f));
        std::vector<float> hw(nw, 0.f);
        for (int tap = 0; tap < 9; ++tap)
            for (int o = 0; o < real_out; ++o)
                for (int i = 0; i < real_in; ++i) hw[((size_t)tap * net->co[l] + o) * net->ci[l] + i] = nd(rng);
        if (cudaMemcpyAsync(net->w[l], hw.data(), sizeof(float) * nw, cudaMemcpyHostToDevice, net->stream) !=
            cudaSuccess)
            return fail(QGN_ERR_CUDA);
        cudaStreamSynchronize(net->stream);
        ::qgn::launch(k_weights_bf16, (nw + 255) / 256, 256, 0, net->stream, net->w[l], nw, net->co[l], net->ci[l], net->wf[l],
                                                                  net->wb[l]);
        const size_t chunks = (size_t)((max_batch * H + kWChunkRows - 1) / kWChunkRows);
        // (the mma.sync engine's bias partials follow its weight partials)
        part = std::max(part, std::max(chunks * nw + ((NP + 1023) / 1024) * (size_t)net->co[l], max_chunks * nw));
    }
    if (nalloc(net, &net->bpart, max_chunks * net->width) || nalloc(net, &net->act[layers], 16) || nalloc(net, &net->gA, NP * net->width) ||
        nalloc(net, &net->gB, NP * net->width) || nalloc(net, &net->part, part) ||
        nalloc(net, &net->loss_part, 148) || nalloc(net, &net->ytgt, NP * pad16(cout)) ||
        nalloc(net, &net->d_err, 1) || nalloc(net, &net->flags, 1024))
        return fail(QGN_ERR_CUDA);
    net->part_elems = part;
    if (const char* e = std::getenv("QGN_CNN_MMA"))
        net->engine = (std::string(e) == "sync") ? 1 : (std::string(e) == "layers") ? 2 : 0;
    if (cudaMallocHost((void**)&net->loss_host, sizeof(double) * 148) != cudaSuccess) return fail(QGN_ERR_CUDA);
    if (cudaStreamSynchronize(net->stream) != cudaSuccess) return fail(QGN_ERR_CUDA);
    *out = net;
    return QGN_OK;
}

int qgn_cnn_padded_channels(const qgn_cnn* net, int* cin_padded, int* cout_padded) {
    if (!net) return QGN_ERR_ARG;
    if (cin_padded) *cin_padded = net->ci[0];
    if (cout_padded) *cout_padded = net->co[net->layers - 1];
    return QGN_OK;
}

// weights: per layer [9][cout_p][cin_p] FP32 then bias [cout_p], layers in order
long long qgn_cnn_num_params(const qgn_cnn* net) {
    if (!net) return -1;
    long long n = 0;
    for (int l = 0; l < net->layers; ++l) n += 9LL * net->co[l] * net->ci[l] + net->co[l];
    return n;
}

int qgn_cnn_get_weights(qgn_cnn* net, float* host) {
    if (!net || !host) return QGN_ERR_ARG;
    size_t off = 0;
    for (int l = 0; l < net->layers; ++l) {
        const size_t nw = 9ull * net->co[l] * net->ci[l];
        NCK(cudaMemcpyAsync(host + off, net->w[l], sizeof(float) * nw, cudaMemcpyDeviceToHost, net->stream));
        off += nw;
        NCK(cudaMemcpyAsync(host + off, net->bias[l], sizeof(float) * net->co[l], cudaMemcpyDeviceToHost, net->stream));
        off += net->co[l];
    }
    NCK(cudaStreamSynchronize(net->stream));
    return QGN_OK;
}

int qgn_cnn_set_weights(qgn_cnn* net, const float* host) {
    if (!net || !host) return QGN_ERR_ARG;
    size_t off = 0;
    for (int l = 0; l < net->layers; ++l) {
        const int nw = 9 * net->co[l] * net->ci[l];
        NCK(cudaMemcpyAsync(net->w[l], host + off, sizeof(float) * nw, cudaMemcpyHostToDevice, net->stream));
        off += nw;
        NCK(cudaMemcpyAsync(net->bias[l], host + off, sizeof(float) * net->co[l], cudaMemcpyHostToDevice, net->stream));
        off += net->co[l];
        ::qgn::launch(k_weights_bf16, (nw + 255) / 256, 256, 0, net->stream, net->w[l], nw, net->co[l], net->ci[l], net->wf[l],
                                                                  net->wb[l]);
        NCK(cudaGetLastError());
    }
    NCK(cudaStreamSynchronize(net->stream));
    net->adam_t = 0;
    for (int l = 0; l < net->layers; ++l) {
        const int nw = 9 * net->co[l] * net->ci[l];
        NCK(cudaMemsetAsync(net->mw[l], 0, sizeof(float) * nw, net->stream));
        NCK(cudaMemsetAsync(net->vw[l], 0, sizeof(float) * nw, net->stream));
        NCK(cudaMemsetAsync(net->mb[l], 0, sizeof(float) * net->co[l], net->stream));
        NCK(cudaMemsetAsync(net->vb[l], 0, sizeof(float) * net->co[l], net->stream));
    }
    NCK(cudaStreamSynchronize(net->stream));
    return QGN_OK;
}

// inference: x = BF16 [batch][H][W][cin_p] (device), y = FP32 [batch][H][W][cout_p] (device).
// Runs on `stream` (NULL: the network's own stream), ordered after the caller's work there.
int qgn_cnn_forward(qgn_cnn* net, const void* x, float* y, int batch, void* stream) {
    QGN_NVTX("qgn_cnn_forward");
    if (!net || !x || !y || batch < 1 || batch > net->max_batch) return QGN_ERR_ARG;
    return qgn::cnn::infer(net, x, y, batch, stream ? static_cast<cudaStream_t>(stream) : net->stream, false);
}

// gradients of the MSE loss at the current weights for x (BF16 [batch][H][W][cin_p]) and
// targets y (FP32 [batch][H][W][cout_p]); host output in the get_weights layout
int qgn_cnn_gradients(qgn_cnn* net, const void* x, const float* y, int batch, float* grads_host, double* loss) {
    if (!net || !x || !y || batch < 1 || batch > net->max_batch) return QGN_ERR_ARG;
    const size_t xb = npix(net, batch) * net->ci[0] * sizeof(__nv_bfloat16);
    NCK(cudaMemcpyAsync(net->act[0], x, xb, cudaMemcpyDeviceToDevice, net->stream));
    if (reinterpret_cast<uintptr_t>(y) % 16 != 0) {   // k_mse loads 16 bytes at a time
        const size_t yb = npix(net, batch) * net->co[net->layers - 1] * sizeof(float);
        NCK(cudaMemcpyAsync(net->ytgt, y, yb, cudaMemcpyDeviceToDevice, net->stream));
        y = net->ytgt;
    }
    int rc = forward(net, batch, true);
    if (rc == QGN_OK) rc = mse(net, batch, y);
    if (rc == QGN_OK) rc = backward(net, batch);
    if (rc == QGN_OK) rc = read_loss(net, loss);
    if (rc != QGN_OK) return rc;
    if (grads_host) {
        NCK(cudaMemcpyAsync(grads_host, net->grads, sizeof(float) * (size_t)qgn_cnn_num_params(net),
                            cudaMemcpyDeviceToHost, net->stream));
        NCK(cudaStreamSynchronize(net->stream));
    }
    return QGN_OK;
}

// one Adam step on the batch idx[0..batch) (device int32) of a dataset: x_all BF16
// [n][H][W][cin_p], y_all FP32 [n][H][W][cout_p]; loss (before the update) optional
int qgn_cnn_train_step(qgn_cnn* net, const void* x_all, const float* y_all, const int* idx, int batch, float lr,
                       double* loss) {
    QGN_NVTX("qgn_cnn_train_step");
    if (!net || !x_all || !y_all || !idx || batch < 1 || batch > net->max_batch || !(lr > 0)) return QGN_ERR_ARG;
    const int L = net->layers;
    const size_t xs = (size_t)net->H * net->W * net->ci[0] * sizeof(__nv_bfloat16);
    const size_t ys = (size_t)net->H * net->W * net->co[L - 1] * sizeof(float);
    ::qgn::launch(k_gather, 148 * 4, 256, 0, net->stream, static_cast<const unsigned char*>(x_all), idx, batch, xs,
                                              reinterpret_cast<unsigned char*>(net->act[0]));
    NCK(cudaGetLastError());
    ::qgn::launch(k_gather, 148 * 4, 256, 0, net->stream, reinterpret_cast<const unsigned char*>(y_all), idx, batch, ys,
                                              reinterpret_cast<unsigned char*>(net->ytgt));
    NCK(cudaGetLastError());
    int rc = forward(net, batch, true);
    if (rc == QGN_OK) rc = mse(net, batch, net->ytgt);
    if (rc == QGN_OK) rc = backward(net, batch);
    if (rc != QGN_OK) return rc;
    net->adam_t += 1;
    const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
    const float c1 = 1.f - std::pow(b1, (float)net->adam_t), c2 = 1.f - std::pow(b2, (float)net->adam_t);
    for (int l = 0; l < L; ++l) {
        const int nw = 9 * net->co[l] * net->ci[l];
        ::qgn::launch(k_adam, (nw + 255) / 256, 256, 0, net->stream, net->w[l], net->mw[l], net->vw[l], net->gw[l], nw, net->co[l],
                                                          net->ci[l], lr, b1, b2, eps, c1, c2, net->wf[l], net->wb[l]);
        NCK(cudaGetLastError());
        ::qgn::launch(k_adam_bias, 1, 64, 0, net->stream, net->bias[l], net->mb[l], net->vb[l], net->gb[l], net->co[l], lr, b1, b2,
                                               eps, c1, c2);
        NCK(cudaGetLastError());
    }
    if (loss) return read_loss(net, loss);
    return QGN_OK;
}

int qgn_cnn_set_engine(qgn_cnn* net, int engine) {
    if (!net || engine < 0 || engine > 2) return QGN_ERR_ARG;
    if (cudaStreamSynchronize(net->stream) != cudaSuccess) return QGN_ERR_CUDA;
    net->engine = engine;
    return QGN_OK;
}

// failure injection for tests: set the fused inference's layer counter of one tile.  A large
// value makes that tile's CTA wait, in the next fused launch, for neighbour counters that
// never reach it; the bounded wait runs out and qgn_cnn_check reports it.
int qgn_cnn_debug_set_counter(qgn_cnn* net, int tile, unsigned int value) {
    if (!net || tile < 0 || tile >= 1024) return QGN_ERR_ARG;
    NCK(cudaMemcpyAsync(net->flags + tile, &value, sizeof(value), cudaMemcpyHostToDevice, net->stream));
    NCK(cudaStreamSynchronize(net->stream));
    return QGN_OK;
}

int qgn_cnn_check(qgn_cnn* net) {
    if (!net) return QGN_ERR_ARG;
    return check_err(net);
}

int qgn_cnn_stream(qgn_cnn* net, void** stream) {
    if (!net || !stream) return QGN_ERR_ARG;
    *stream = net->stream;
    return QGN_OK;
}

const char* qgn_cnn_last_error(const qgn_cnn* net) { return net ? net->last_error.c_str() : "NULL network"; }

int qgn_cnn_destroy(qgn_cnn* net) {
    if (!net) return QGN_OK;
    if (net->stream) cudaStreamSynchronize(net->stream);
    for (void* p : net->owned) cudaFree(p);
    if (net->loss_host) cudaFreeHost(net->loss_host);
    if (net->stream) cudaStreamDestroy(net->stream);
    delete net;
    return QGN_OK;
}

}  // extern "C"
