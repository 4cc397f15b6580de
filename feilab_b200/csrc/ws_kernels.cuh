// ws_kernels.cuh -- the kernels of the warm-start U-Net besides the 3x3
// tensor-core convolutions (ws_conv.cuh): weight gradients by mma.sync, the rest
// SIMT.  Activations are NHWC BF16
// images [n][H][W][C]; arithmetic is FP32; every reduction is two-level with
// a fixed order (partial sums per block, then one pass over the partials), so
// results do not depend on scheduling.
#pragma once
#include <cuda_bf16.h>
#include <cstdint>

#include "pdl.cuh"

namespace ws {

__device__ __forceinline__ float bf(const __nv_bfloat16 v) { return __bfloat162float(v); }
__device__ __forceinline__ __nv_bfloat16 tobf(float v) { return __float2bfloat16_rn(v); }

// ------------------------------------------------------------ slice layout
// Slices in the layout of the C ABI: [S][N0][N1], Y (N1) fastest, as the
// reference's images (X*N1 + Y).  The network image of slice s is
// [Hp][Wp] with h = Y, w = X (Hp, Wp: N1, N0 rounded up to multiples of 8).

// Per-slice sums of squares of Re(Ahwb), in two steps of fixed order: block
// (c, s) of kSumSqChunks per slice writes part[s][c], then k_slice_sumsq_fin
// (one warp per slice) ss[s].  One block per slice took 559 us for 8 slices of
// 1024 x 300 (one SM each); this takes 10 us.
constexpr int kSumSqChunks = 64;

__global__ void __launch_bounds__(256) k_slice_sumsq(const float2 *__restrict__ Ahwb, int N0, int N1, double *__restrict__ part)
{
    icon::pdl_wait();
    __shared__ double red[256];
    const int c = blockIdx.x, s = blockIdx.y, n = N0 * N1;
    const float2 *base = Ahwb + (size_t)s * n;
    const int i0 = (int)((long long)n * c / kSumSqChunks), i1 = (int)((long long)n * (c + 1) / kSumSqChunks);
    double acc = 0.0;
#pragma unroll 4
    for (int i = i0 + threadIdx.x; i < i1; i += 256) {
        double v = base[i].x;
        acc += v * v;
    }
    red[threadIdx.x] = acc;
    __syncthreads();
    for (int o = 128; o > 0; o >>= 1) {
        if ((int)threadIdx.x < o) red[threadIdx.x] += red[threadIdx.x + o];
        __syncthreads();
    }
    if (threadIdx.x == 0) part[s * kSumSqChunks + c] = red[0];
}

__global__ void k_slice_sumsq_fin(const double *__restrict__ part, double *__restrict__ ss)
{
    icon::pdl_wait();
    double v = 0.0;
    for (int c = threadIdx.x; c < kSumSqChunks; c += 32) v += part[blockIdx.x * kSumSqChunks + c];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if (threadIdx.x == 0) ss[blockIdx.x] = v;
}

// Network input x[s][h][w] = Re(Ahwb[s][w][h]) / scale_s for h < N1, w < N0,
// zero in the padding; scale_s = sqrt(ss/(N0 N1)), or 1 when zero.
__global__ void k_net_input(const float2 *__restrict__ Ahwb, const double *__restrict__ ss, int N0, int N1, int Hp,
                            int Wp, int S, float *__restrict__ x, float *__restrict__ scale)
{
    icon::pdl_wait();
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    const size_t total = (size_t)S * Hp * Wp;
    if (i >= total) return;
    const int w = (int)(i % Wp), h = (int)((i / Wp) % Hp), s = (int)(i / ((size_t)Wp * Hp));
    const double q = ss[s] / ((double)N0 * N1);
    const float sc = q > 0 ? (float)sqrt(q) : 1.f;
    if (h == 0 && w == 0) scale[s] = sc;
    x[i] = (h < N1 && w < N0) ? Ahwb[((size_t)s * N0 + w) * N1 + h].x / sc : 0.f;
}

// Training target t[s][h][w] = m[s][w][h] / (scale_s * gain), zero in the padding.
__global__ void k_net_target(const float *__restrict__ m, const float *__restrict__ scale, float gain, int N0, int N1,
                             int Hp, int Wp, int S, float *__restrict__ t)
{
    icon::pdl_wait();
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    const size_t total = (size_t)S * Hp * Wp;
    if (i >= total) return;
    const int w = (int)(i % Wp), h = (int)((i / Wp) % Hp), s = (int)(i / ((size_t)Wp * Hp));
    t[i] = (h < N1 && w < N0) ? m[((size_t)s * N0 + w) * N1 + h] / (scale[s] * gain) : 0.f;
}

// m0[s][X][Y] = scale_s * gain * y[s][Y][X].
__global__ void k_net_output(const float *__restrict__ y, const float *__restrict__ scale, float gain, int N0, int N1,
                             int Hp, int Wp, int S, float *__restrict__ m)
{
    icon::pdl_wait();
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    const size_t total = (size_t)S * N0 * N1;
    if (i >= total) return;
    const int Y = (int)(i % N1), X = (int)((i / N1) % N0), s = (int)(i / ((size_t)N1 * N0));
    m[i] = (scale[s] * gain) * y[((size_t)s * Hp + Y) * Wp + X];
}

// ------------------------------------------------------------ first layer
// 3x3 convolution of the one-channel input to 16 channels, bias, ReLU; two
// neighbouring pixels (W is even) a thread, so that a shared-memory load of four
// weights feeds eight multiply-adds.  w: [9][16] FP32, tap = 3*dy + dx.
// 8 x 304 x 1024 pixels: 38 us; one pixel a thread and a load per weight took 50.
__global__ void __launch_bounds__(128) k_conv_in(const float *__restrict__ x, const float *__restrict__ w,
                                                 const float *__restrict__ bias, int n, int H, int W,
                                                 __nv_bfloat16 *__restrict__ y)
{
    icon::pdl_wait();
    __shared__ __align__(16) float sw[9 * 16 + 16];
    for (int i = threadIdx.x; i < 9 * 16; i += blockDim.x) sw[i] = w[i];
    for (int i = threadIdx.x; i < 16; i += blockDim.x) sw[144 + i] = bias[i];
    __syncthreads();
    const size_t p2 = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (2 * p2 >= (size_t)n * H * W) return;
    const int xw = 2 * (int)(p2 % (W / 2)), xh = (int)((p2 / (W / 2)) % H), im = (int)(p2 / ((size_t)(W / 2) * H));
    float in[3][4];
#pragma unroll
    for (int r = 0; r < 3; ++r) {
        const int hh = xh + r - 1;
        const float *row = x + ((size_t)im * H + hh) * W + xw;
        const bool on = hh >= 0 && hh < H;
        const float2 mid = on ? *reinterpret_cast<const float2 *>(row) : make_float2(0.f, 0.f);
        in[r][0] = on && xw > 0 ? row[-1] : 0.f;
        in[r][1] = mid.x;
        in[r][2] = mid.y;
        in[r][3] = on && xw + 2 < W ? row[2] : 0.f;
    }
    __align__(16) __nv_bfloat16 o[2][16];
#pragma unroll
    for (int c = 0; c < 16; c += 4) {
        const float4 b4 = *reinterpret_cast<const float4 *>(sw + 144 + c);
        float a[2][4] = {{b4.x, b4.y, b4.z, b4.w}, {b4.x, b4.y, b4.z, b4.w}};
#pragma unroll
        for (int t = 0; t < 9; ++t) {
            const float4 w4 = *reinterpret_cast<const float4 *>(sw + t * 16 + c);
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                const float v = in[t / 3][t % 3 + q];
                a[q][0] = fmaf(w4.x, v, a[q][0]);
                a[q][1] = fmaf(w4.y, v, a[q][1]);
                a[q][2] = fmaf(w4.z, v, a[q][2]);
                a[q][3] = fmaf(w4.w, v, a[q][3]);
            }
        }
#pragma unroll
        for (int q = 0; q < 2; ++q)
#pragma unroll
            for (int k = 0; k < 4; ++k) o[q][c + k] = tobf(fmaxf(a[q][k], 0.f));
    }
    uint4 *d = reinterpret_cast<uint4 *>(y + 2 * p2 * 16);
#pragma unroll
    for (int q = 0; q < 2; ++q) {
        d[2 * q] = reinterpret_cast<uint4 *>(o[q])[0];
        d[2 * q + 1] = reinterpret_cast<uint4 *>(o[q])[1];
    }
}

// Weight and bias gradients of the first layer.  A block takes kInRows image
// rows, kInCols pixels wide, at a time (tile = blockIdx.x + k*gridDim.x), its
// input with the border and its output gradients in shared memory.  Thread =
// (row group, dy, channel): it walks its rows' pixels with the three dx inputs
// in registers, two shared loads and three multiply-adds a pixel; the dy = 1
// threads also sum the bias.  part[blk][160] = dw[9][16], db[16], the row
// groups' sums added in order.  16 x 512 x 256 pixels: 61 us; one thread
// per weight walking 2048 pixels of global memory took 1669.
constexpr int kInRows = 8, kInCols = 64, kInGroups = 4;

__global__ void __launch_bounds__(48 * kInGroups) k_conv_in_wgrad(const float *__restrict__ x,
                                                                  const __nv_bfloat16 *__restrict__ gz, int n, int H,
                                                                  int W, float *__restrict__ part)
{
    icon::pdl_wait();
    constexpr int T = 48 * kInGroups;
    __shared__ float sx[kInRows + 2][kInCols + 2];
    __shared__ float sg[kInRows][kInCols][17];
    __shared__ float red[kInGroups][160];
    const int t = threadIdx.x, c = t & 15, dy = (t >> 4) % 3, grp = t / 48;
    const int tw = (W + kInCols - 1) / kInCols, th = (H + kInRows - 1) / kInRows;
    const long long tiles = (long long)n * tw * th;
    float acc[3] = {0.f, 0.f, 0.f}, bacc = 0.f;
    for (long long tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
        const int w0 = (int)(tile % tw) * kInCols, h0 = (int)((tile / tw) % th) * kInRows, im = (int)(tile / ((long long)tw * th));
        __syncthreads();
        for (int i = t; i < (kInRows + 2) * (kInCols + 2); i += T) {
            const int px = i % (kInCols + 2), r = i / (kInCols + 2), hh = h0 + r - 1, ww = w0 + px - 1;
            sx[r][px] = (hh >= 0 && hh < H && ww >= 0 && ww < W) ? x[((size_t)im * H + hh) * W + ww] : 0.f;
        }
        for (int i = t; i < kInRows * kInCols * 2; i += T) {     // 8 channels a piece
            const int q = i & 1, px = (i >> 1) % kInCols, r = (i >> 1) / kInCols, hh = h0 + r, ww = w0 + px;
            uint4 v = make_uint4(0, 0, 0, 0);
            if (hh < H && ww < W) v = *reinterpret_cast<const uint4 *>(gz + (((size_t)im * H + hh) * W + ww) * 16 + 8 * q);
            const __nv_bfloat16 *e = reinterpret_cast<const __nv_bfloat16 *>(&v);
#pragma unroll
            for (int k = 0; k < 8; ++k) sg[r][px][8 * q + k] = bf(e[k]);
        }
        __syncthreads();
        for (int r = grp; r < kInRows; r += kInGroups) {
            float x0 = sx[r + dy][0], x1 = sx[r + dy][1];
#pragma unroll 8
            for (int px = 0; px < kInCols; ++px) {
                const float g = sg[r][px][c], x2 = sx[r + dy][px + 2];
                acc[0] = fmaf(g, x0, acc[0]);
                acc[1] = fmaf(g, x1, acc[1]);
                acc[2] = fmaf(g, x2, acc[2]);
                bacc += g;
                x0 = x1;
                x1 = x2;
            }
        }
    }
#pragma unroll
    for (int dx = 0; dx < 3; ++dx) red[grp][(3 * dy + dx) * 16 + c] = acc[dx];
    if (dy == 1) red[grp][144 + c] = bacc;
    __syncthreads();
    if (t < 160) {
        float a = red[0][t];
        for (int k = 1; k < kInGroups; ++k) a += red[k][t];
        part[(size_t)blockIdx.x * 160 + t] = a;
    }
}

// ------------------------------------------------------------ pool / upsample
// 2x2 average pooling; C a multiple of 8 (8 channels per thread).
__global__ void k_pool2(const __nv_bfloat16 *__restrict__ in, int n, int H, int W, int C, __nv_bfloat16 *__restrict__ out)
{
    icon::pdl_wait();
    const int Ho = H / 2, Wo = W / 2, C8 = C / 8;
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (size_t)n * Ho * Wo * C8) return;
    const int c8 = (int)(i % C8);
    const size_t q = i / C8;
    const int wo = (int)(q % Wo), ho = (int)((q / Wo) % Ho), im = (int)(q / ((size_t)Wo * Ho));
    float acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    for (int dy = 0; dy < 2; ++dy)
        for (int dx = 0; dx < 2; ++dx) {
            const uint4 v =
                *reinterpret_cast<const uint4 *>(in + (((size_t)im * H + 2 * ho + dy) * W + 2 * wo + dx) * C + 8 * c8);
            const __nv_bfloat16 *e = reinterpret_cast<const __nv_bfloat16 *>(&v);
#pragma unroll
            for (int k = 0; k < 8; ++k) acc[k] += bf(e[k]);
        }
    __align__(16) __nv_bfloat16 o[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) o[k] = tobf(0.25f * acc[k]);
    *reinterpret_cast<uint4 *>(out + (((size_t)im * Ho + ho) * Wo + wo) * C + 8 * c8) = *reinterpret_cast<uint4 *>(o);
}

// Gradient of the pooling, added to what the skip connection left there, through
// the ReLU of y, the pooled image: gin[2h+dy][2w+dx] = y > 0 ? gin + gout[h][w] / 4
// : 0 (H, W = input size).
__global__ void k_pool2_bwd(const __nv_bfloat16 *__restrict__ gout, int n, int H, int W, int C,
                            const __nv_bfloat16 *__restrict__ y, __nv_bfloat16 *__restrict__ gin)
{
    icon::pdl_wait();
    const int Ho = H / 2, Wo = W / 2, C8 = C / 8;
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (size_t)n * H * W * C8) return;
    const int c8 = (int)(i % C8);
    const size_t q = i / C8;
    const int w = (int)(q % W), h = (int)((q / W) % H), im = (int)(q / ((size_t)W * H));
    const uint4 g = *reinterpret_cast<const uint4 *>(gout + (((size_t)im * Ho + h / 2) * Wo + w / 2) * C + 8 * c8);
    const __nv_bfloat16 *ge = reinterpret_cast<const __nv_bfloat16 *>(&g);
    const uint4 yv = *reinterpret_cast<const uint4 *>(y + q * C + 8 * c8);
    const __nv_bfloat16 *ye = reinterpret_cast<const __nv_bfloat16 *>(&yv);
    uint4 *dst = reinterpret_cast<uint4 *>(gin + q * C + 8 * c8);
    __align__(16) __nv_bfloat16 o[8];
    const uint4 old = *dst;
    const __nv_bfloat16 *oe = reinterpret_cast<const __nv_bfloat16 *>(&old);
#pragma unroll
    for (int k = 0; k < 8; ++k) o[k] = bf(ye[k]) > 0.f ? tobf(bf(oe[k]) + 0.25f * bf(ge[k])) : tobf(0.f);
    *dst = *reinterpret_cast<uint4 *>(o);
}

// Nearest 2x upsampling: out[h][w] = in[h/2][w/2] (H, W = output size).
__global__ void k_up2(const __nv_bfloat16 *__restrict__ in, int n, int H, int W, int C, __nv_bfloat16 *__restrict__ out)
{
    icon::pdl_wait();
    const int C8 = C / 8;
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (size_t)n * H * W * C8) return;
    const int c8 = (int)(i % C8);
    const size_t q = i / C8;
    const int w = (int)(q % W), h = (int)((q / W) % H), im = (int)(q / ((size_t)W * H));
    *reinterpret_cast<uint4 *>(out + q * C + 8 * c8) =
        *reinterpret_cast<const uint4 *>(in + (((size_t)im * (H / 2) + h / 2) * (W / 2) + w / 2) * C + 8 * c8);
}

// Gradient of the upsampling, through the ReLU of y, the upsampled image: gin[h][w]
// = y > 0 ? sum of gout over its 2x2 block : 0 (H, W = input size).
__global__ void k_up2_bwd(const __nv_bfloat16 *__restrict__ gout, int n, int H, int W, int C,
                          const __nv_bfloat16 *__restrict__ y, __nv_bfloat16 *__restrict__ gin)
{
    icon::pdl_wait();
    const int C8 = C / 8;
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (size_t)n * H * W * C8) return;
    const int c8 = (int)(i % C8);
    const size_t q = i / C8;
    const int w = (int)(q % W), h = (int)((q / W) % H), im = (int)(q / ((size_t)W * H));
    const uint4 yv = *reinterpret_cast<const uint4 *>(y + q * C + 8 * c8);
    const __nv_bfloat16 *ye = reinterpret_cast<const __nv_bfloat16 *>(&yv);
    float acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    for (int dy = 0; dy < 2; ++dy)
        for (int dx = 0; dx < 2; ++dx) {
            const uint4 v = *reinterpret_cast<const uint4 *>(
                gout + (((size_t)im * 2 * H + 2 * h + dy) * (2 * W) + 2 * w + dx) * C + 8 * c8);
            const __nv_bfloat16 *e = reinterpret_cast<const __nv_bfloat16 *>(&v);
#pragma unroll
            for (int k = 0; k < 8; ++k) acc[k] += bf(e[k]);
        }
    __align__(16) __nv_bfloat16 o[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) o[k] = bf(ye[k]) > 0.f ? tobf(acc[k]) : tobf(0.f);
    *reinterpret_cast<uint4 *>(gin + q * C + 8 * c8) = *reinterpret_cast<uint4 *>(o);
}

// ------------------------------------------------------------ weight gradients
// dW[tap][co][ci] = sum over pixels of gz[p][co] * X[p shifted by tap][ci] for
// a 3x3 convolution whose input is X0 (c0 channels) concatenated with X1 (c1
// channels), and db[co] = sum gz[p][co]: nine matrix products with the pixels
// as the inner dimension, 16 to 128 rows and 16 to 192 columns, on the tensor
// cores by warp-level mma (m16n8k16, BF16 products, FP32 sums).  (The tiles are
// too small for tcgen05: of its 64 rows at least 48 would be padding at 16
// channels, and its operands could not share one staged row between the three
// dx, which here are the same shared-memory rows read one pixel on.)
//
// A CTA of four warps takes an output tile of 16 WCO MC x 16 MI channels and a
// contiguous share of the image rows, cut into 64 pixels wide strips.  It
// walks down a strip with a ring of rows in shared memory (cp.async, two rows
// ahead; five of X, so that each row of X is loaded once for its three dy, and
// three of gz) whose 16-byte pieces are XOR-swizzled by the pixel, so that
// every ldmatrix is free of bank conflicts at any dx.  A warp's tile is
// 16 WCO x 16; the KW warps of one tile take the strip's 16-pixel steps in
// turn.  Per step and warp: WCO + 9 ldmatrix and 18 WCO mma.  Every warp writes
// its own partial sums, part[split KW + k] = dW[tap][co][ci], db[co], added in
// order by k_sum_parts.  16 x 512 x 256 pixels, all 13 layers: 0.89 ms; one multiply-add a thread from
// shared memory took 11.8 ms.
constexpr int kWgStrip = 64, kWgXRows = 5, kWgGRows = 3;

__device__ __forceinline__ void ldsm_t(uint32_t (&r)[4], uint32_t addr)
{
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(addr));
}
__device__ __forceinline__ void mma_16816(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1)
{
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// 16-byte copy, or 16 zero bytes where !on.
__device__ __forceinline__ void cp16_or_zero(uint32_t dst, const void *src, bool on)
{
    const int n = on ? 16 : 0;
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(n) : "memory");
}

// Byte offset of 16-byte piece `ch` of pixel px in a row of PC pieces per pixel.
template <int PC>
__device__ __forceinline__ uint32_t wg_off(int px, int ch)
{
    const int sw = PC == 2 ? (px >> 2) & 1 : PC == 4 ? (px >> 1) & 3 : px & 7;
    return (uint32_t)((px * PC + (ch ^ sw)) * 16);
}

template <int WCO, int MC, int MI, int KW>
struct WgShape {
    static_assert(MC * MI * KW == 4, "four warps");
    static constexpr int CO = 16 * WCO * MC, CI = 16 * MI, GC = CO / 8, XC = CI / 8;
    static constexpr int XB = (kWgStrip + 2) * XC * 16, GB = kWgStrip * GC * 16;   // bytes of a staged row
    static constexpr int SMEM = kWgXRows * XB + kWgGRows * GB;
};

template <int WCO, int MC, int MI, int KW>
__global__ void __launch_bounds__(128) k_wgrad3x3(const __nv_bfloat16 *__restrict__ X0, int c0, int up0,
                                                   const __nv_bfloat16 *__restrict__ X1, int c1,
                                                   const __nv_bfloat16 *__restrict__ gz, int N, int n, int H, int W,
                                                   float *__restrict__ part)
{
    icon::pdl_wait();
    using S = WgShape<WCO, MC, MI, KW>;
    extern __shared__ __align__(128) unsigned char wg_smem[];
    const uint32_t sx = (uint32_t)__cvta_generic_to_shared(wg_smem), sg = sx + kWgXRows * S::XB;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int kw = warp % KW, mi = (warp / KW) % MI, mc = warp / (KW * MI);
    const int co0 = blockIdx.y * S::CO, ci0 = blockIdx.z * S::CI, Cin = c0 + c1;
    const bool second = ci0 >= c0;                       // tiles do not straddle the inputs
    const __nv_bfloat16 *X = second ? X1 + (ci0 - c0) : X0 + ci0;
    const int CX = second ? c1 : c0, up = second ? 0 : up0;   // up0: X0 is read as its 2x nearest upsampling
    const bool bias = blockIdx.z == 0 && mi == 0;
    // ldmatrix addresses within a row: gz pieces (pixel, co), X pieces (pixel + dx, ci).
    const int lr = lane & 7, lm = lane >> 3;
    uint32_t aoff[WCO], xoff[3];
#pragma unroll
    for (int v = 0; v < WCO; ++v) aoff[v] = wg_off<S::GC>(lr + 8 * (lm >> 1), 2 * (mc * WCO + v) + (lm & 1));
#pragma unroll
    for (int dx = 0; dx < 3; ++dx) xoff[dx] = wg_off<S::XC>(lr + 8 * (lm & 1) + dx, 2 * mi + (lm >> 1));
    float acc[WCO][9][2][4], bacc[WCO][4];
#pragma unroll
    for (int v = 0; v < WCO; ++v) {
#pragma unroll
        for (int t = 0; t < 9; ++t)
#pragma unroll
            for (int j = 0; j < 2; ++j)
#pragma unroll
                for (int q = 0; q < 4; ++q) acc[v][t][j][q] = 0.f;
#pragma unroll
        for (int q = 0; q < 4; ++q) bacc[v][q] = 0.f;
    }
    const int strips = (W + kWgStrip - 1) / kWgStrip;
    const long long rows = (long long)n * strips * H;    // (image, strip, row), row fastest
    long long r = rows * blockIdx.x / gridDim.x;
    const long long r_end = rows * (blockIdx.x + 1) / gridDim.x;
    while (r < r_end) {
        const int h0 = (int)(r % H), w0 = (int)((r / H) % strips) * kWgStrip, im = (int)(r / ((long long)H * strips));
        const int cnt = (int)min((long long)(H - h0), r_end - r);
        auto load_x = [&](int j) {                       // row h0 + j (j >= -1) into slot (j + 1) % kWgXRows
            const int hh = h0 + j;
            const uint32_t dst = sx + ((j + 1) % kWgXRows) * S::XB;
            const bool in = hh >= 0 && hh < H;
            const __nv_bfloat16 *src = X + ((size_t)im * (H >> up) + (in ? hh >> up : 0)) * (W >> up) * CX;
            for (int i = tid; i < (kWgStrip + 2) * S::XC; i += 128) {
                const int px = i / S::XC, ch = i % S::XC, ww = w0 + px - 1;
                const bool on = in && ww >= 0 && ww < W;
                cp16_or_zero(dst + wg_off<S::XC>(px, ch), src + (on ? (ww >> up) * CX + 8 * ch : 0), on);
            }
        };
        auto load_g = [&](int j) {
            const uint32_t dst = sg + (j % kWgGRows) * S::GB;
            const __nv_bfloat16 *src = gz + ((size_t)im * H + h0 + j) * W * N + co0;
            for (int i = tid; i < kWgStrip * S::GC; i += 128) {
                const int px = i / S::GC, ch = i % S::GC, ww = w0 + px;
                const bool on = ww < W;
                cp16_or_zero(dst + wg_off<S::GC>(px, ch), src + (on ? (size_t)ww * N + 8 * ch : 0), on);
            }
        };
        auto issue = [&](int j) {                        // what step j needs beyond step j - 1
            if (j < cnt) {
                load_x(j + 1);
                load_g(j);
            }
            asm volatile("cp.async.commit_group;" ::: "memory");
        };
        __syncthreads();                                 // the last strip's rows are consumed
        load_x(-1);
        load_x(0);
        issue(0);
        issue(1);
        for (int j = 0; j < cnt; ++j) {
            asm volatile("cp.async.wait_group 1;" ::: "memory");
            __syncthreads();                             // step j has landed, step j - 1 is consumed
            issue(j + 2);
            const uint32_t grow = sg + (j % kWgGRows) * S::GB;
#pragma unroll
            for (int k = 0; k < kWgStrip / 16 / KW; ++k) {
                const int ks = k * KW + kw;
                uint32_t a[WCO][4];
#pragma unroll
                for (int v = 0; v < WCO; ++v) ldsm_t(a[v], grow + aoff[v] + ks * 16 * S::GC * 16);
                if (bias) {
#pragma unroll
                    for (int v = 0; v < WCO; ++v) mma_16816(bacc[v], a[v], 0x3f803f80u, 0x3f803f80u);   // times one
                }
#pragma unroll
                for (int dy = 0; dy < 3; ++dy) {
                    const uint32_t xrow = sx + ((j + dy) % kWgXRows) * S::XB + ks * 16 * S::XC * 16;
#pragma unroll
                    for (int dx = 0; dx < 3; ++dx) {
                        uint32_t b[4];
                        ldsm_t(b, xrow + xoff[dx]);
#pragma unroll
                        for (int v = 0; v < WCO; ++v) {
                            mma_16816(acc[v][3 * dy + dx][0], a[v], b[0], b[1]);
                            mma_16816(acc[v][3 * dy + dx][1], a[v], b[2], b[3]);
                        }
                    }
                }
            }
        }
        r += cnt;
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    // Accumulator (g, t): rows co = g, g + 8, columns ci = 2t, 2t + 1 of each half.
    const size_t ps = (size_t)blockIdx.x * KW + kw;
    const int g = lane >> 2, t2 = 2 * (lane & 3);
    part += ps * (size_t)(9 * Cin + 1) * N;
#pragma unroll
    for (int v = 0; v < WCO; ++v) {
        const int co = co0 + (mc * WCO + v) * 16 + g, ci = ci0 + mi * 16 + t2;
#pragma unroll
        for (int t = 0; t < 9; ++t)
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                float *o = part + ((size_t)t * N + co) * Cin + ci + 8 * j;
                *reinterpret_cast<float2 *>(o) = make_float2(acc[v][t][j][0], acc[v][t][j][1]);
                *reinterpret_cast<float2 *>(o + (size_t)8 * Cin) = make_float2(acc[v][t][j][2], acc[v][t][j][3]);
            }
        if (bias && t2 == 0) {
            part[(size_t)9 * N * Cin + co] = bacc[v][0];
            part[(size_t)9 * N * Cin + co + 8] = bacc[v][2];
        }
    }
}

// out[i] = sum over s < nsplit of part[s][i]: 32 V outputs a block, V adjacent
// ones a thread; of the block's W warps, warp w takes the parts s = w, w + W, ...
// in order, and the W sums are added in order.  One load a thread in flight per
// eight parts or so: with 32 warps and V = 1 throughout, a layer of 56 parts of
// 590 KB took 32 us, its 4608 blocks of 1024 threads mostly starting and ending;
// 9 us so.  (One thread per output walking every part: 876 us over the sums of a
// backward pass, 223 us with 32 warps and V = 1, 140 us so.)
constexpr int kSumWarps = 32;

template <int V>
__global__ void __launch_bounds__(32 * kSumWarps) k_sum_parts(const float *__restrict__ part, int nsplit, size_t len, float *__restrict__ out)
{
    icon::pdl_wait();
    __shared__ float red[kSumWarps][32 * V + 1];
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31, W = blockDim.x >> 5;
    const size_t i = ((size_t)blockIdx.x * 32 + lane) * V;
    float a[V];
#pragma unroll
    for (int v = 0; v < V; ++v) a[v] = 0.f;
    if (i < len) {
#pragma unroll 8
        for (int s = w; s < nsplit; s += W) {
            if constexpr (V == 4) {
                const float4 q = *reinterpret_cast<const float4 *>(part + (size_t)s * len + i);
                a[0] += q.x;
                a[1] += q.y;
                a[2] += q.z;
                a[3] += q.w;
            } else {
                a[0] += part[(size_t)s * len + i];
            }
        }
    }
#pragma unroll
    for (int v = 0; v < V; ++v) red[w][lane * V + v] = a[v];
    __syncthreads();
    const size_t o = (size_t)blockIdx.x * 32 * V + threadIdx.x;
    if (threadIdx.x < 32 * V && o < len) {
        float b = 0.f;
        for (int k = 0; k < W; ++k) b += red[k][threadIdx.x];
        out[o] = b;
    }
}

// ------------------------------------------------------------ output layer
// y[p] = b + sum_c w[c] * d[p][c] (1x1 convolution of 16 channels to one).
__global__ void k_conv_out(const __nv_bfloat16 *__restrict__ d, const float *__restrict__ w, const float *__restrict__ b,
                           size_t npix, float *__restrict__ y)
{
    icon::pdl_wait();
    const size_t p = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= npix) return;
    const uint4 *v = reinterpret_cast<const uint4 *>(d + p * 16);
    float a = b[0];
#pragma unroll
    for (int q = 0; q < 2; ++q) {
        const uint4 u = v[q];
        const __nv_bfloat16 *e = reinterpret_cast<const __nv_bfloat16 *>(&u);
#pragma unroll
        for (int k = 0; k < 8; ++k) a = fmaf(w[8 * q + k], bf(e[k]), a);
    }
    y[p] = a;
}

// Mean squared error over the valid pixels (h < Hv, w < Wv) of S images
// [S][Hp][Wp]: dy = 2 (y - t) / count (zero in the padding); per-block partial
// sums of (y - t)^2 in double to lpart[blockIdx.x].  blockDim = 256.
__global__ void k_mse(const float *__restrict__ y, const float *__restrict__ t, int S, int Hp, int Wp, int Hv, int Wv,
                      float *__restrict__ dy, double *__restrict__ lpart)
{
    icon::pdl_wait();
    __shared__ double red[256];
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    const size_t total = (size_t)S * Hp * Wp;
    double l = 0.0;
    if (i < total) {
        const int w = (int)(i % Wp), h = (int)((i / Wp) % Hp);
        float g = 0.f;
        if (h < Hv && w < Wv) {
            const float e = y[i] - t[i];
            l = (double)e * e;
            g = 2.f * e / ((float)S * Hv * Wv);
        }
        dy[i] = g;
    }
    red[threadIdx.x] = l;
    __syncthreads();
    for (int o = blockDim.x / 2; o > 0; o >>= 1) {
        if ((int)threadIdx.x < o) red[threadIdx.x] += red[threadIdx.x + o];
        __syncthreads();
    }
    if (threadIdx.x == 0) lpart[blockIdx.x] = red[0];
}

// Backward of the output layer and of the ReLU before it: gd[p][c] = d[p][c] > 0 ?
// dy[p] * w[c] : 0 (BF16), and per-block
// partial sums of dw[c] = sum dy[p] d[p][c] and db = sum dy[p] (part[blk][17])
// over the pixels p = thread + k * threads, summed in a thread, then over its
// warp and the block in fixed order.  (One pixel per thread, a 17-wide tree in
// every block and 8192 partial sums: 50 + 462 us for 16 x 512 x 256 pixels;
// 592 blocks: 25 + 5 us.)
constexpr int kOutBlocks = 4 * icon::kSMs;

__global__ void __launch_bounds__(256) k_conv_out_bwd(const __nv_bfloat16 *__restrict__ d, const float *__restrict__ dy,
                                                      const float *__restrict__ w, size_t npix,
                                                      __nv_bfloat16 *__restrict__ gd, float *__restrict__ part)
{
    icon::pdl_wait();
    __shared__ float red[8][17];
    float loc[17], wv[16];
#pragma unroll
    for (int k = 0; k < 17; ++k) loc[k] = 0.f;
#pragma unroll
    for (int k = 0; k < 16; ++k) wv[k] = w[k];
    for (size_t p = (size_t)blockIdx.x * 256 + threadIdx.x; p < npix; p += (size_t)gridDim.x * 256) {
        const float g = dy[p];
        const uint4 *v = reinterpret_cast<const uint4 *>(d + p * 16);
        __align__(16) __nv_bfloat16 o[16];
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            const uint4 u = v[q];
            const __nv_bfloat16 *e = reinterpret_cast<const __nv_bfloat16 *>(&u);
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                loc[8 * q + k] = fmaf(g, bf(e[k]), loc[8 * q + k]);
                o[8 * q + k] = bf(e[k]) > 0.f ? tobf(g * wv[8 * q + k]) : tobf(0.f);
            }
        }
        loc[16] += g;
        uint4 *dst = reinterpret_cast<uint4 *>(gd + p * 16);
        dst[0] = reinterpret_cast<uint4 *>(o)[0];
        dst[1] = reinterpret_cast<uint4 *>(o)[1];
    }
#pragma unroll
    for (int k = 0; k < 17; ++k) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) loc[k] += __shfl_xor_sync(0xffffffffu, loc[k], o);
        if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5][k] = loc[k];
    }
    __syncthreads();
    if (threadIdx.x < 17) {
        float a = red[0][threadIdx.x];
        for (int k = 1; k < 8; ++k) a += red[k][threadIdx.x];
        part[(size_t)blockIdx.x * 17 + threadIdx.x] = a;
    }
}

// ------------------------------------------------------------ optimiser
// Adam on the FP32 master parameters (bias-corrected, no weight decay).
__global__ void k_adam(float *__restrict__ p, const float *__restrict__ g, float *__restrict__ m, float *__restrict__ v,
                       size_t n, float lr, float b1, float b2, float eps, float c1, float c2)
{
    icon::pdl_wait();
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float gi = g[i];
    const float mi = b1 * m[i] + (1.f - b1) * gi;
    const float vi = b2 * v[i] + (1.f - b2) * gi * gi;
    m[i] = mi;
    v[i] = vi;
    p[i] -= lr * (mi / c1) / (sqrtf(vi / c2) + eps);
}

// BF16 copies of a 3x3 layer's weights: wb[tap][N][Cin] = w, and the weights
// of its input gradient wt[tap][Cin][N] = w[8 - tap][N][Cin] (flipped taps,
// swapped channels).
__global__ void k_weights_bf16(const float *__restrict__ w, int N, int Cin, __nv_bfloat16 *__restrict__ wb,
                               __nv_bfloat16 *__restrict__ wt)
{
    icon::pdl_wait();
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (size_t)9 * N * Cin) return;
    const int ci = (int)(i % Cin), co = (int)((i / Cin) % N), tap = (int)(i / ((size_t)Cin * N));
    const __nv_bfloat16 v = tobf(w[i]);
    wb[i] = v;
    wt[((size_t)(8 - tap) * Cin + ci) * N + co] = v;
}

}  // namespace ws
