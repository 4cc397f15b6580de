// tools.cu -- the steps either side of the ICON solve that the reference does
// in its companion tools, on the GPU: stack pre-processing (ICONPreProcess)
// and, in mask.cu, volume assembly with the cross-validation mask
// (ICONMask3).  C ABI in include/icon_tools.h.
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <string>
#include <vector>

#include "icon_b200.h"
#include "icon_tools.h"
#include "pdl.cuh"

extern "C" void icon_internal_set_error(const char *msg);

namespace {

icon_status tools_fail(icon_status st, const std::string &msg)
{
    icon_internal_set_error(msg.c_str());
    return st;
}

constexpr int kPreThreads = 1024;
constexpr int kPreMaxProjections = 1024;

// Variance factors of the projections, passed by value (8 KB of kernel
// parameters) so the call needs no device memory.
struct PreFactors {
    double f[kPreMaxProjections];
};

// One cluster of RANKS CTAs per projection k of in[nz][ny][nx]
// (ICONPreProcess.c:29-85):
//   mode  = bin of the most pixels (first on ties) of a 256-bin histogram of
//           the central region (10 % margins), bin index
//           floor((v - min) / step), step = (max - min) / 256 in double; the
//           largest pixel falls in bin 256, which is not counted
//   v    -= mode                                (float result)
//   with factor[k] > 0: mean = sum v / size, var = sum (v - mean)^2 / size
//           (double), v = v / sqrt(var) * sqrt(factor[k])
// out may equal in.
//
// The four passes over a projection (extrema, histogram, moments, result) are
// bound by memory: 78 us for 61 projections of 1024 x 1024 read and written
// once.  A CTA takes a band of whole rows and keeps the first of them in
// shared memory (its first pass fills them); the rest of the passes read L2 as far
// as it holds the bands in flight (one CTA runs per SM), and DRAM again beyond.  Extrema, bin counts and moments are
// combined over the cluster through distributed shared memory in rank order.
// The size of the clusters: one CTA runs per SM, so a call takes as many rounds as its
// CTAs fill the SMs, and a round about 12 us plus 0.6 ns a pixel of a CTA's band
// (one CTA: 61 x 1024 x 1024 in one round 634 us, 81 x 100 x 100 20). pre_ranks takes
// the size of the least rounds x (20,000 + pixels of a band).  With clusters of 8
// throughout many small projections were slower than with one CTA each: 200 of 2000 x
// 30 129 -> 338 us, now 90; 41 of 128 x 128 28 -> 38, now 16; large ones gain from
// fewer rounds: 61 x 1024 x 1024 398 -> 329 us (one CTA per projection, six passes and
// divisions in double for every pixel 2374), 61 x 2048 x 2048 1590 -> 1228.
constexpr int kPreMaxRanks = 8;
inline int pre_ranks(long long size, int nz)
{
    long long best = 0;
    int ranks = 1;
    for (int r = 1; r <= kPreMaxRanks; r *= 2) {
        const int places = icon::kSMs / r * r;            // clusters of 8: 18
        const long long cost = ((long long)nz * r + places - 1) / places * (20000 + size / r);
        if (r == 1 || cost < best) {
            best = cost;
            ranks = r;
        }
    }
    return ranks;
}
constexpr int kPreCache = 184 * 1024;   // shared memory for rows

// Sum over the block of one double per thread (fixed order), to every thread.
__device__ double block_sum(double v, double *red)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    __syncthreads();                       // red free
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
    __syncthreads();
    double r = 0.0;
    for (int i = 0; i < (int)blockDim.x / 32; ++i) r += red[i];
    return r;
}

// VEC: rows are read and written as float4 (nx a multiple of 4, both stacks
// on 16-byte boundaries).
template <bool VEC, int RANKS>
__global__ void __launch_bounds__(kPreThreads, 1) __cluster_dims__(RANKS, 1, 1)
    k_preprocess(const float *in, float *out, int nx, int ny, int normalize, int cache_rows,
                 const __grid_constant__ PreFactors factor)
{
    namespace cg = cooperative_groups;
    cg::cluster_group cl = cg::this_cluster();
    extern __shared__ __align__(16) float cache[];   // [cache_rows][nx]
    __shared__ double red[kPreThreads / 32];
    __shared__ float ext[2];                         // this CTA's extrema, read by the cluster
    __shared__ int hist[8][256];                     // warps w share copy w % 8
    __shared__ int bins[256];                        // this CTA's counts, read by the cluster
    __shared__ double mom[2], mode_s;                // this CTA's moments
    const int k = blockIdx.x / RANKS, rank = (int)cl.block_rank();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, W = blockDim.x >> 5;
    const size_t size = (size_t)nx * ny;
    const float *p = in + (size_t)k * size;
    float *q = out + (size_t)k * size;
    const int y0 = (int)((long long)ny * rank / RANKS), y1 = (int)((long long)ny * (rank + 1) / RANKS);
    const int xe = (int)(nx * 0.1), ye = (int)(ny * 0.1);
    const int xr = nx - xe, yr = ny - ye;            // core: xe <= x < xr, ye <= y < yr
    // Calls f(x, v) for the pixels x of row y that this lane takes.
    auto row = [&](const float *r, auto f) {
        if constexpr (VEC) {
            for (int x = 4 * lane; x < nx; x += 128) {
                const float4 v = *reinterpret_cast<const float4 *>(r + x);
                f(x, v.x);
                f(x + 1, v.y);
                f(x + 2, v.z);
                f(x + 3, v.w);
            }
        } else {
            for (int x = lane; x < nx; x += 32) f(x, r[x]);
        }
    };
    // Row y from the cache when it is there.
    auto source = [&](int y) { return y - y0 < cache_rows ? cache + (size_t)(y - y0) * nx : p + (size_t)y * nx; };

    // Extrema of the core; fills the cache.
    float lo = p[(size_t)ye * nx + xe], hi = lo;
    for (int y = y0 + warp; y < y1; y += W) {
        const bool core = y >= ye && y < yr, keep = y - y0 < cache_rows;
        float *c = cache + (size_t)(y - y0) * nx;
        row(p + (size_t)y * nx, [&](int x, float v) {
            if (keep) c[x] = v;
            if (core && x >= xe && x < xr) {
                lo = fminf(lo, v);
                hi = fmaxf(hi, v);
            }
        });
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        lo = fminf(lo, __shfl_xor_sync(0xffffffffu, lo, o));
        hi = fmaxf(hi, __shfl_xor_sync(0xffffffffu, hi, o));
    }
    float *red_f = reinterpret_cast<float *>(&hist[0][0]);   // [2][32], before the counts
    if (lane == 0) {
        red_f[warp] = lo;
        red_f[32 + warp] = hi;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int i = 1; i < W; ++i) {
            lo = fminf(lo, red_f[i]);
            hi = fmaxf(hi, red_f[32 + i]);
        }
        ext[0] = lo;
        ext[1] = hi;
    }
    cl.sync();
    lo = cl.map_shared_rank(ext, 0)[0];
    hi = cl.map_shared_rank(ext, 0)[1];
    for (int r = 1; r < RANKS; ++r) {
        lo = fminf(lo, cl.map_shared_rank(ext, r)[0]);
        hi = fmaxf(hi, cl.map_shared_rank(ext, r)[1]);
    }
    const double mn = lo, mx = hi;
    const double step = (mx - mn) / 256.0;
    double mode = mn;   // a constant core has no spread (the reference divides by zero there)
    if (step > 0.0) {
        for (int i = threadIdx.x; i < 8 * 256; i += blockDim.x) (&hist[0][0])[i] = 0;
        __syncthreads();
        const double inv = 1.0 / step;
        int *h = hist[warp & 7];
        for (int y = max(y0, ye) + warp; y < min(y1, yr); y += W)
            row(source(y), [&](int x, float v) {
                if (x < xe || x >= xr) return;
                // The quotient's floor by a product (its nearest whole number
                // read from the low bits of t + 1.5 2^52, all in the FP64 pipe),
                // and by the division itself where the product is near a
                // whole number (or not finite).
                const double t = ((double)v - mn) * inv, big = t + 6755399441055744.0, d = t - (big - 6755399441055744.0);
                int b = __double2loint(big) - (d < 0.0);
                if (!(fabs(d) > 1e-6)) b = (int)floor(((double)v - mn) / step);
                if (b >= 0 && b < 256) atomicAdd(&h[b], 1);
            });
        __syncthreads();
        if (threadIdx.x < 256) {
            int c = 0;
            for (int i = 0; i < 8; ++i) c += hist[i][threadIdx.x];
            bins[threadIdx.x] = c;
        }
        cl.sync();
        // First bin with the largest count, over the cluster.
        if (threadIdx.x < 256) {
            int c = 0;
            for (int r = 0; r < RANKS; ++r) c += cl.map_shared_rank(bins, r)[threadIdx.x];
            hist[0][threadIdx.x] = c;
        }
        __syncthreads();
        if (threadIdx.x < 32) {
            int best = -1, bi = 0;
            for (int i = lane; i < 256; i += 32)
                if (best < hist[0][i]) {
                    best = hist[0][i];
                    bi = i;
                }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                const int ob = __shfl_xor_sync(0xffffffffu, best, o), oi = __shfl_xor_sync(0xffffffffu, bi, o);
                if (ob > best || (ob == best && oi < bi)) {
                    best = ob;
                    bi = oi;
                }
            }
            if (lane == 0) mode_s = bi * step + mn;
        }
        __syncthreads();
        mode = mode_s;
    }
    const double f = normalize ? factor.f[k] : 0.0;
    double scale = 1.0;
    if (f > 0.0) {
        // var = (sum v^2 - (sum v)^2 / size) / size in double.  At least one pixel
        // of the mode's bin lies within a bin of 0, so var is no less than about
        // mean^2 / size and the difference keeps all but size 2^-53 of its digits
        // (2e-9 for 4096 x 4096).  (The mean of float quotients v / size that the
        // reference subtracts is within 2^-24 of the mean, and moves the variance by
        // the square of that.)
        double s1 = 0.0, s2 = 0.0;
        for (int y = y0 + warp; y < y1; y += W)
            row(source(y), [&](int, float v0) {
                const double v = (double)(float)((double)v0 - mode);
                s1 += v;
                s2 += v * v;
            });
        s1 = block_sum(s1, red);
        s2 = block_sum(s2, red);
        if (threadIdx.x == 0) {
            mom[0] = s1;
            mom[1] = s2;
        }
        cl.sync();
        s1 = s2 = 0.0;
        for (int r = 0; r < RANKS; ++r) {
            const double *m = cl.map_shared_rank(mom, r);
            s1 += m[0];
            s2 += m[1];
        }
        const double var = (s2 - s1 * s1 / (double)size) / (double)size;
        scale = sqrt(f) / sqrt(var < 0.0 ? 0.0 : var);   // rounding of the sums for a constant stack
    }
    for (int y = y0 + warp; y < y1; y += W) {
        const float *r = source(y);
        float *o = q + (size_t)y * nx;
        auto result = [&](float v0) {
            const float v = (float)((double)v0 - mode);
            return f > 0.0 ? (float)((double)v * scale) : v;
        };
        if constexpr (VEC) {
            for (int x = 4 * lane; x < nx; x += 128) {
                const float4 v = *reinterpret_cast<const float4 *>(r + x);
                *reinterpret_cast<float4 *>(o + x) = make_float4(result(v.x), result(v.y), result(v.z), result(v.w));
            }
        } else {
            for (int x = lane; x < nx; x += 32) o[x] = result(r[x]);
        }
    }
    cl.sync();   // no CTA leaves while another reads its shared memory
}

template <int RANKS>
cudaError_t pre_launch(bool vec, const float *in, float *out, int nx, int ny, int nz, bool norm, const PreFactors &f,
                       cudaStream_t st)
{
    const size_t row = sizeof(float) * (size_t)nx;
    const int cache_rows = (int)std::min<size_t>(kPreCache / row, (size_t)(ny + RANKS - 1) / RANKS);
    const auto kern = vec ? k_preprocess<true, RANKS> : k_preprocess<false, RANKS>;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kPreCache);
    if (e != cudaSuccess) return e;
    kern<<<nz * RANKS, kPreThreads, cache_rows * row, st>>>(in, out, nx, ny, norm ? 1 : 0, cache_rows, f);
    return cudaGetLastError();
}

}  // namespace

extern "C" {

icon_status icon_preprocess(const float *d_in, float *d_out, int nx, int ny, int nz, const float *h_tilt_deg,
                            int thickness, void *stream)
{
    if (!d_in || !d_out || nx < 1 || ny < 1 || nz < 1) return tools_fail(ICON_ERR_INVALID, "icon_preprocess: bad argument");
    if ((nx - 2 * (int)(nx * 0.1)) < 1 || (ny - 2 * (int)(ny * 0.1)) < 1)
        return tools_fail(ICON_ERR_INVALID, "icon_preprocess: image too small");
    if (nz > kPreMaxProjections) return tools_fail(ICON_ERR_INVALID, "icon_preprocess: more than 1024 projections");
    cudaStream_t st = (cudaStream_t)stream;
    const bool norm = h_tilt_deg && thickness > 0;
    PreFactors f{};
    if (norm) {
        // ICONPreProcess.c:73-85 with angle = -tilt (:283): 0.33 t / cos(angle in radians, pi = 3.1415926)
        for (int k = 0; k < nz; ++k) {
            const float angle = -h_tilt_deg[k];
            f.f[k] = 0.33 * thickness / std::cos(angle / 180.0 * 3.1415926);
            if (!(f.f[k] > 0.0)) return tools_fail(ICON_ERR_INVALID, "icon_preprocess: tilt angle gives a non-positive variance");
        }
    }
    const bool vec = nx % 4 == 0 && ((uintptr_t)d_in & 15) == 0 && ((uintptr_t)d_out & 15) == 0;
    cudaError_t e = cudaSuccess;
    switch (pre_ranks((long long)nx * ny, nz)) {
    case 1: e = pre_launch<1>(vec, d_in, d_out, nx, ny, nz, norm, f, st); break;
    case 2: e = pre_launch<2>(vec, d_in, d_out, nx, ny, nz, norm, f, st); break;
    case 4: e = pre_launch<4>(vec, d_in, d_out, nx, ny, nz, norm, f, st); break;
    default: e = pre_launch<8>(vec, d_in, d_out, nx, ny, nz, norm, f, st); break;
    }
    if (e != cudaSuccess) return tools_fail(ICON_ERR_CUDA, std::string("icon_preprocess: ") + cudaGetErrorString(e));
    return ICON_OK;
}

icon_status icon_preprocess_host(const float *h_in, float *h_out, int nx, int ny, int nz, const float *h_tilt_deg,
                                 int thickness)
{
    if (!h_in || !h_out || nx < 1 || ny < 1 || nz < 1) return tools_fail(ICON_ERR_INVALID, "icon_preprocess_host: bad argument");
    const size_t bytes = sizeof(float) * (size_t)nx * ny * nz;
    float *d = nullptr;
    if (cudaMalloc(&d, bytes) != cudaSuccess) {
        cudaGetLastError();
        return tools_fail(ICON_ERR_NOMEM, "icon_preprocess_host: device memory for the stack");
    }
    icon_status rc = ICON_OK;
    cudaError_t e = cudaMemcpy(d, h_in, bytes, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) rc = icon_preprocess(d, d, nx, ny, nz, h_tilt_deg, thickness, nullptr);
    if (e == cudaSuccess && rc == ICON_OK) e = cudaMemcpy(h_out, d, bytes, cudaMemcpyDeviceToHost);
    cudaFree(d);
    if (e != cudaSuccess) return tools_fail(ICON_ERR_CUDA, std::string("icon_preprocess_host: ") + cudaGetErrorString(e));
    return rc;
}

}  // extern "C"
