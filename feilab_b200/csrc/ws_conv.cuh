// ws_conv.cuh -- 3x3 convolution (stride 1, zero padding 1) of NHWC BF16
// activations as an implicit GEMM on the sm_100a tensor cores.
//
// One CTA computes a tile of 128 output pixels (one image row, w0..w0+127)
// by N output channels: D[128][N] = sum over K of A[128][K] * B[N][K]^T with
// K = taps x input channels.  For every (input tensor, chunk of cc channels,
// tap) step, TMA loads the 128 x cc input box shifted by the tap (zero fill
// outside the image gives the padding) and the N x cc weight box, both into
// swizzled K-major shared-memory tiles; one thread issues cc/16
// tcgen05.mma (M = 128, K = 16) per step into an FP32 accumulator in tensor
// memory.  A ring of kStages stages keeps the loads ahead of the MMAs.  The
// epilogue (four warps, one pixel per thread) reads the accumulator with
// tcgen05.ld, adds the bias, applies ReLU, rounds to BF16 and stores the
// pixel's channels; the channels can be split over two outputs (the gradient
// of a concatenated input) and added to what an output holds.
//
// Two input tensors are read as one concatenated input (the decoder's skip
// connections), so the concatenation is never stored.  Weights are
// [tap][N][Cin] BF16 with tap = 3*dy + dx.
#pragma once
#include "pdl.cuh"
#include "ws_tc.cuh"

namespace ws {

constexpr int kConvStages = 4;
constexpr int kConvThreads = 128;
constexpr int kTileM = 128;

struct ConvArgs {
    int nin;                 // input tensors (1 or 2), concatenated along channels
    int cin0, cin1;          // their channels
    int H, W;                // image size (output = input size)
    int cc;                  // channels per K step (16, 32 or 64; divides cin0 and cin1)
    int N;                   // output channels (multiple of 16, <= 256)
    int nsplit;              // out0 takes channels [0, nsplit), out1 [nsplit, N)
    __nv_bfloat16 *out0, *out1;
    int acc0, acc1;          // 1: add to the output's values
    const __nv_bfloat16 *mask0;   // out0 is zeroed where this image of its shape is not positive (ReLU gradient), or null
    const float *bias;       // [N] or null
    int relu;
    int *err;                // device error flag
    // Limit of the pipeline's load and MMA waits (normally kWaitNs).  The
    // waits that drain copies and MMAs before the CTA exits always use
    // kWaitNs, so nothing is left in flight.
    unsigned long long wait_ns;
    // Test of the bounded waits: the first stage's barrier expects 16 bytes
    // more than its loads deliver, so the wait for it can only run out.
    int hold;
};

// v = 0 where y is not positive.
__device__ __forceinline__ void relu_mask(float (&v)[16], const __nv_bfloat16 *y)
{
#pragma unroll
    for (int q = 0; q < 2; ++q) {
        const uint4 u = reinterpret_cast<const uint4 *>(y)[q];
        const __nv_bfloat16 *e = reinterpret_cast<const __nv_bfloat16 *>(&u);
#pragma unroll
        for (int i = 0; i < 8; ++i)
            if (!(__bfloat162float(e[i]) > 0.f)) v[8 * q + i] = 0.f;
    }
}

__host__ __device__ inline size_t conv_stage_a_bytes(int cc) { return (size_t)kTileM * cc * 2; }
__host__ __device__ inline size_t conv_stage_b_bytes(int N, int cc) { return (((size_t)N * cc * 2) + 1023) & ~(size_t)1023; }
__host__ __device__ inline size_t conv_smem_bytes(int N, int cc)
{
    return 1024 /* alignment slack */ + kConvStages * (conv_stage_a_bytes(cc) + conv_stage_b_bytes(N, cc)) +
           (2 * kConvStages + 1) * 8 + 16 + (size_t)N * 4;
}
__host__ __device__ inline uint32_t conv_tmem_cols(int N)
{
    uint32_t c = 32;
    while ((int)c < N) c <<= 1;
    return c;
}

__global__ void __launch_bounds__(kConvThreads, 1)
k_conv3x3_tc(const __grid_constant__ CUtensorMap in0, const __grid_constant__ CUtensorMap in1,
             const __grid_constant__ CUtensorMap wmap, ConvArgs a)
{
    icon::pdl_wait();
    extern __shared__ unsigned char smem_raw[];
    unsigned char *base = reinterpret_cast<unsigned char *>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    const size_t abytes = conv_stage_a_bytes(a.cc), bbytes = conv_stage_b_bytes(a.N, a.cc);
    unsigned char *sa = base;
    unsigned char *sb = base + kConvStages * abytes;
    uint64_t *full = reinterpret_cast<uint64_t *>(sb + kConvStages * bbytes);
    uint64_t *empty = full + kConvStages;
    uint64_t *done = empty + kConvStages;
    uint32_t *tslot = reinterpret_cast<uint32_t *>(done + 1);
    float *sbias = reinterpret_cast<float *>(tslot + 4);

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int w0 = blockIdx.x * kTileM, h = blockIdx.y, img = blockIdx.z;
    const uint32_t ncols = conv_tmem_cols(a.N);
    const int sw = a.cc * 2;                       // swizzle span = row bytes of a tile
    const int chunks0 = a.cin0 / a.cc, chunks = chunks0 + (a.nin > 1 ? a.cin1 / a.cc : 0);
    const int steps = 9 * chunks;
    const uint32_t tx = (uint32_t)(kTileM * a.cc * 2 + a.N * a.cc * 2);
    const uint32_t idesc = idesc_bf16(kTileM, a.N);

    if (tid == 0) {
        for (int s = 0; s < kConvStages; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], 1);
        }
        mbar_init(done, 1);
        mbar_fence_init();
        tma_prefetch_desc(&in0);
        if (a.nin > 1) tma_prefetch_desc(&in1);
        tma_prefetch_desc(&wmap);
    }
    for (int i = tid; i < a.N; i += kConvThreads) sbias[i] = a.bias ? a.bias[i] : 0.f;
    if (warp == 0) tmem_alloc(tslot, ncols);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tslot;

    bool ok = true;
    if (warp == 0) {
        if (lane == 0) {
            // Step k: global chunk g = k / 9 (tensor 0's chunks, then tensor
            // 1's), tap = k % 9.
            auto issue = [&](int k) {
                const int s = k % kConvStages, g = k / 9, tap = k - 9 * g, dy = tap / 3, dx = tap - 3 * dy;
                const bool second = g >= chunks0;
                const int c0 = (second ? g - chunks0 : g) * a.cc;
                const int wc0 = (second ? a.cin0 : 0) + c0;
                mbar_expect_tx(&full[s], tx + ((a.hold && k == 0) ? 16u : 0u));
                tma_load_4d(sa + s * abytes, second ? &in1 : &in0, c0, w0 + dx - 1, h + dy - 1, img, &full[s]);
                tma_load_3d(sb + s * bbytes, &wmap, wc0, 0, tap, &full[s]);
            };
            const int pre = steps < kConvStages ? steps : kConvStages;
            for (int k = 0; k < pre; ++k) issue(k);
            int issued = pre;
            for (int k = 0; k < steps && ok; ++k) {
                const int s = k % kConvStages;
                if (!mbar_wait(&full[s], (uint32_t)((k / kConvStages) & 1), a.err, kErrLoadWait, a.wait_ns)) {
                    ok = false;
                    break;
                }
                tc_fence_after();
                const uint32_t a0 = smem_u32(sa + s * abytes), b0 = smem_u32(sb + s * bbytes);
                for (int kk = 0; kk < a.cc / 16; ++kk) {
                    const uint64_t ad = smem_desc_kmajor(a0 + kk * 32, sw);
                    const uint64_t bd = smem_desc_kmajor(b0 + kk * 32, sw);
                    mma_bf16(tmem, ad, bd, idesc, (k > 0) || (kk > 0));
                }
                mma_commit(&empty[s]);
                // Refill the stage of step k-1 once its MMAs are done (step
                // k's MMAs stay queued meanwhile).
                if (k >= 1 && issued < steps) {
                    const int kp = k - 1, sp = kp % kConvStages;
                    if (!mbar_wait(&empty[sp], (uint32_t)((kp / kConvStages) & 1), a.err, kErrMmaWait, a.wait_ns)) {
                        ok = false;
                        break;
                    }
                    issue(issued++);
                }
            }
            mma_commit(done);
            if (!ok) {
                // Let the copies already issued land before the CTA exits.
                for (int k = 0; k < issued; ++k) {
                    const int s = k % kConvStages;
                    mbar_wait(&full[s], (uint32_t)((k / kConvStages) & 1), a.err, kErrLoadWait);
                }
            }
        }
        __syncwarp();
    }
    const bool fin = mbar_wait(done, 0, a.err, kErrDoneWait);
    tc_fence_after();
    if (fin && *a.err == kErrNone) {
        const int px = w0 + tid;
        const bool valid = px < a.W;
        const size_t pix = ((size_t)img * a.H + h) * a.W + px;
        for (int c = 0; c < a.N; c += 16) {
            float v[16];
            __syncwarp();
            tmem_ld16(tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)c, v);
            if (!valid) continue;
#pragma unroll
            for (int i = 0; i < 16; ++i) {
                v[i] += sbias[c + i];
                if (a.relu) v[i] = fmaxf(v[i], 0.f);
            }
            const bool first = c < a.nsplit;
            const int C = first ? a.nsplit : a.N - a.nsplit;
            __nv_bfloat16 *dst = (first ? a.out0 : a.out1) + pix * C + (first ? c : c - a.nsplit);
            if (first ? a.acc0 : a.acc1) {
                const __nv_bfloat162 *old = reinterpret_cast<const __nv_bfloat162 *>(dst);
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    float2 o = __bfloat1622float2(old[i]);
                    v[2 * i] += o.x;
                    v[2 * i + 1] += o.y;
                }
            }
            if (first && a.mask0) relu_mask(v, a.mask0 + pix * C + c);
            uint4 pk[2];
            uint32_t *pw = reinterpret_cast<uint32_t *>(pk);
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                __nv_bfloat162 t = __floats2bfloat162_rn(v[2 * i], v[2 * i + 1]);
                pw[i] = *reinterpret_cast<uint32_t *>(&t);
            }
            uint4 *d4 = reinterpret_cast<uint4 *>(dst);
            d4[0] = pk[0];
            d4[1] = pk[1];
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) tmem_dealloc(tmem, ncols);
}

// ---------------------------------------------------- small layers ----
// The same convolution for layers whose weights and input tile fit beside each
// other's CTAs in shared memory (conv_halo_rows): the layers of the two finest
// levels, which hold most of the pixels and are bound by moving them.  The
// kernel above loads every pixel nine times, shifted by each tap, in boxes of
// 32 or 64 byte rows, and the weights once per 128 pixels.  Here a CTA keeps
// the weights and walks over tiles of 128 pixels x TH rows; a tile's input
// with its border is loaded once (cp.async, zeros outside the image) into
// planes of 8 channels, 16 bytes a pixel.  In this unswizzled K-major layout
// consecutive pixels are consecutive 16-byte rows, so the tap (dy, dx) of
// image row r is the same planes read from pixel (r + dy) * 130 + dx on: nine
// descriptors of one tile.  The MMAs of a tile run in the order of the kernel
// above (chunks, taps, 16-channel steps), so the sums are the same bit for
// bit.  Several CTAs per SM overlap one's loads with another's MMAs and
// stores; a tile's loads start as soon as the previous tile's MMAs have read
// the planes, ahead of its epilogue.  8 x 304 x 1024 pixels:
// 16 -> 16 channels 171 -> 66 us, 48 -> 16 383 -> 205, 32 -> 32 at half size 54
// -> 43.  An input that is the 2x upsampling of a stored image is read from
// that image (up0), which saves the pass that stored it (64 us).
constexpr int kHaloW = kTileM + 2;

__host__ __device__ inline size_t conv_halo_smem(int N, int cin, int th)
{
    return 128 + (size_t)9 * N * cin * 2 + (size_t)(th + 2) * kHaloW * cin * 2 + (size_t)N * 4 + 32;
}
// Rows per tile of k_conv3x3_halo, or 0: accumulators in at most 128 TMEM
// columns and two CTAs per SM (for 48 -> 16 channels four rows with two CTAs
// take 203 us, two rows with three 238).
__host__ __device__ inline int conv_halo_rows(int N, int cin)
{
    for (int th = 4; th >= 2; th -= 2)
        if (th * N <= 128 && conv_halo_smem(N, cin, th) <= 110 * 1024) return th;
    return 0;
}

// 32 bytes of a thread in one store.
__device__ __forceinline__ void store32(void *p, const uint32_t (&v)[8])
{
    asm volatile("st.global.v8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(p), "r"(v[0]), "r"(v[1]), "r"(v[2]),
                 "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7])
                 : "memory");
}
__device__ __forceinline__ void halo_cp16(uint32_t dst, const void *src, bool on)
{
    const int n = on ? 16 : 0;
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(n) : "memory");
}

struct HaloArgs {
    ConvArgs c;
    const __nv_bfloat16 *in0, *in1, *w;
    int lg0, lg1;            // log2 of the 16-byte pieces per pixel of the two inputs
    int up0;                 // in0 is [nimg][H/2][W/2][cin0], read as its 2x nearest upsampling
    int nimg;
};

template <int TH>
__global__ void __launch_bounds__(kConvThreads) k_conv3x3_halo(const HaloArgs h)
{
    icon::pdl_wait();
    extern __shared__ unsigned char smem_raw[];
    const ConvArgs &a = h.c;
    unsigned char *base = reinterpret_cast<unsigned char *>(((uintptr_t)smem_raw + 127) & ~(uintptr_t)127);
    const int cin = a.cin0 + a.cin1, N = a.N, W = a.W, H = a.H;
    constexpr uint32_t plane = (TH + 2) * kHaloW * 16;    // bytes of 8 channels of a tile
    const uint32_t sw = smem_u32(base), sx = sw + 9 * N * cin * 2;
    float *sbias = reinterpret_cast<float *>(base + 9 * N * cin * 2 + (cin / 8) * plane);
    uint64_t *done = reinterpret_cast<uint64_t *>(((uintptr_t)(sbias + N) + 7) & ~(uintptr_t)7);
    uint32_t *tslot = reinterpret_cast<uint32_t *>(done + 1);
    const int tid = threadIdx.x, warp = tid >> 5;
    uint32_t ncols = 32;
    while ((int)ncols < TH * N) ncols <<= 1;
    if (tid == 0) {
        mbar_init(done, 1);
        mbar_fence_init();
    }
    for (int i = tid; i < N; i += kConvThreads) sbias[i] = a.bias ? a.bias[i] : 0.f;
    // Weights [tap][N][cin] into [tap][piece of 8 channels][N] of 16 bytes.
    for (int i = tid; i < 9 * N * (cin / 8); i += kConvThreads) {
        const int ch = i % (cin / 8), tn = i / (cin / 8), n = tn % N, tap = tn / N;
        halo_cp16(sw + ((tap * (cin / 8) + ch) * N + n) * 16, h.w + (size_t)tn * cin + 8 * ch, true);
    }
    const int tw = (W + kTileM - 1) / kTileM, th = (H + TH - 1) / TH;
    const long long tiles = (long long)h.nimg * th * tw;
    auto load = [&](long long t) {                        // a tile's input with its border
        const int w0 = (int)(t % tw) * kTileM - 1, h0 = (int)((t / tw) % th) * TH - 1, img = (int)(t / ((long long)tw * th));
#pragma unroll
        for (int s = 0; s < 2; ++s) {
            if (s == 1 && a.nin < 2) break;
            const __nv_bfloat16 *in = s ? h.in1 : h.in0;
            const int lg = s ? h.lg1 : h.lg0, C = s ? a.cin1 : a.cin0;
            const uint32_t dst = sx + (s ? (a.cin0 / 8) * plane : 0);
            for (int r = 0; r < TH + 2; ++r) {
                const int hh = h0 + r;
                const bool row = hh >= 0 && hh < H;
                const int up = s == 0 ? h.up0 : 0;
                const __nv_bfloat16 *src = in + ((size_t)img * (H >> up) + (row ? hh >> up : 0)) * (W >> up) * C;
                for (int i = tid; i < kHaloW << lg; i += kConvThreads) {
                    const int px = i >> lg, ch = i & ((1 << lg) - 1), ww = w0 + px;
                    const bool on = row && ww >= 0 && ww < W;
                    halo_cp16(dst + ch * plane + (r * kHaloW + px) * 16, src + (on ? (ww >> up) * C + 8 * ch : 0), on);
                }
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    long long t = blockIdx.x;
    if (t < tiles) load(t);
    if (warp == 0) tmem_alloc(tslot, ncols);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tslot;
    const uint32_t idesc = idesc_bf16(kTileM, N);
    const int chunks = cin / a.cc;
    const bool clean = *a.err == kErrNone;                // an earlier unread error: no output, as above
    bool ok = true;
    for (uint32_t phase = 0; t < tiles && ok; t += gridDim.x, phase ^= 1) {
        // The tile's planes (and at first the weights) in place for the MMAs;
        // the accumulators read by the previous tile's epilogue.
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        tc_fence_before();
        __syncthreads();
        tc_fence_after();
        if (tid == 0) {
            bool first = true;
            for (int g = 0; g < chunks; ++g)
                for (int tap = 0; tap < 9; ++tap)
                    for (int kk = 0; kk < a.cc / 16; ++kk) {
                        const int p = (g * a.cc + 16 * kk) / 8;      // first of the step's two planes
                        const uint64_t bd = smem_desc_planar(sw + ((tap * (cin / 8) + p) * N) * 16, N * 16);
                        const uint32_t a0 = sx + p * plane + ((tap / 3) * kHaloW + tap % 3) * 16;
#pragma unroll
                        for (int r = 0; r < TH; ++r)
                            mma_bf16(tmem + r * N, smem_desc_planar(a0 + r * kHaloW * 16, plane), bd, idesc, !first);
                        first = false;
                    }
            mma_commit(done);
        }
        ok = mbar_wait(done, phase, a.err, kErrDoneWait, a.wait_ns);
        ok = __syncthreads_and(ok) != 0;
        if (!ok) {                                        // a second bounded wait before shared memory and TMEM go
            mbar_wait(done, phase, a.err, kErrDoneWait);
            break;
        }
        tc_fence_after();
        if (t + gridDim.x < tiles) load(t + gridDim.x);
        const int px = (int)(t % tw) * kTileM + tid, h0 = (int)((t / tw) % th) * TH, img = (int)(t / ((long long)tw * th));
#pragma unroll
        for (int r = 0; r < TH; ++r) {
            const bool valid = clean && px < W && h0 + r < H;
            const size_t pix = ((size_t)img * H + h0 + r) * W + px;
            for (int c = 0; c < N; c += 16) {
                float v[16];
                __syncwarp();
                tmem_ld16(tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)(r * N + c), v);
                if (!valid) continue;
#pragma unroll
                for (int i = 0; i < 16; ++i) {
                    v[i] += sbias[c + i];
                    if (a.relu) v[i] = fmaxf(v[i], 0.f);
                }
                const bool f = c < a.nsplit;
                const int C = f ? a.nsplit : N - a.nsplit;
                __nv_bfloat16 *dst = (f ? a.out0 : a.out1) + pix * C + (f ? c : c - a.nsplit);
                if (f ? a.acc0 : a.acc1) {
                    const __nv_bfloat162 *old = reinterpret_cast<const __nv_bfloat162 *>(dst);
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        const float2 o = __bfloat1622float2(old[i]);
                        v[2 * i] += o.x;
                        v[2 * i + 1] += o.y;
                    }
                }
                if (f && a.mask0) relu_mask(v, a.mask0 + pix * C + c);
                uint32_t pk[8];
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const __nv_bfloat162 q = __floats2bfloat162_rn(v[2 * i], v[2 * i + 1]);
                    pk[i] = *reinterpret_cast<const uint32_t *>(&q);
                }
                if (((uintptr_t)dst & 31) == 0) {
                    store32(dst, pk);
                } else {
                    reinterpret_cast<uint4 *>(dst)[0] = make_uint4(pk[0], pk[1], pk[2], pk[3]);
                    reinterpret_cast<uint4 *>(dst)[1] = make_uint4(pk[4], pk[5], pk[6], pk[7]);
                }
            }
        }
        __syncwarp();
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    tc_fence_before();
    __syncthreads();
    if (warp == 0) tmem_dealloc(tmem, ncols);
}

}  // namespace ws
