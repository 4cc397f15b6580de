// icon_kern_b.cu -- the batched FFT kernels for one slice-group size,
// ICON_KB (1, 2, 4 or 8, set by the build), and their host launchers.
#define ICON_KERNELS_TEMPLATES_ONLY
#include "icon_kernels.cuh"
#include "icon_launch.h"

#ifndef ICON_KB
#error "compile with -DICON_KB=<1|2|4|8>"
#endif

namespace icon {

template <int B>
void Launch<B>::xpass_fwd(bool real_in, int E, dim3 grid, int threads, size_t smem, cudaStream_t st, const Geo &g,
                          const void *in, float2 *G1)
{
    // n0 >= 128 is k_xtoep's and k_xtoep_real's (icon_api.cu: xt_ok); only the complex
    // image of the measured Toeplitz iterations comes here with E = 32.
    if (E == 32) pdl(k_xpass_fwd<false, B, 32>, grid, threads, smem, st, g, in, G1);
    else if (real_in && g.n0 / 2 >= 16)   // half-length FFT per slice: half the threads and buffer
        pdl(k_xpass_fwd_r2c<B, 16>, grid, threads / 2, smem / 2, st, g, (const float *)in, G1);
    else if (real_in) pdl(k_xpass_fwd<true, B, 16>, grid, threads, smem, st, g, in, G1);
    else pdl(k_xpass_fwd<false, B, 16>, grid, threads, smem, st, g, in, G1);
}

template <int B>
void Launch<B>::xpass_fwd_full(int E, dim3 grid, int threads, size_t smem, cudaStream_t st, const Geo &g,
                               const float *in, float2 *G1)
{
    if (g.n0 / 2 >= E) {   // half-length FFT per slice, as xpass_fwd
        if (E == 32) pdl(k_xpass_fwd_r2c<B, 32, true>, grid, threads / 2, smem / 2, st, g, in, G1);
        else pdl(k_xpass_fwd_r2c<B, 16, true>, grid, threads / 2, smem / 2, st, g, in, G1);
        return;
    }
    pdl(k_xpass_fwd<true, B, 16, true>, grid, threads, smem, st, g, in, G1);   // n0 = 16
}

// The four-step register FFT (k_ytoep4) for n1 = 32 R, R in
// {4, 6, 8, 10, 12, 16, 20, 24, 32}; blockDim = n1*B/32, shared memory
// n1*B float2.
template <int B, int MODE>
static void launch_ytoep4(dim3 grid, cudaStream_t st, const Geo &g, float2 *G1, const float2 *Gh, double *part)
{
    const int threads = g.n1 * B / 32;
    const size_t smem = ytoep4_smem(g.n1, B);
    switch (g.n1 / 32) {
    case 4: pdl(k_ytoep4<B, 4, MODE>, grid, threads, smem, st, g, G1, Gh, part); break;
    case 6: pdl(k_ytoep4<B, 6, MODE>, grid, threads, smem, st, g, G1, Gh, part); break;
    case 8: pdl(k_ytoep4<B, 8, MODE>, grid, threads, smem, st, g, G1, Gh, part); break;
    case 10: pdl(k_ytoep4<B, 10, MODE>, grid, threads, smem, st, g, G1, Gh, part); break;
    case 12: pdl(k_ytoep4<B, 12, MODE>, grid, threads, smem, st, g, G1, Gh, part); break;
    case 16: pdl(k_ytoep4<B, 16, MODE>, grid, threads, smem, st, g, G1, Gh, part); break;
    case 20: pdl(k_ytoep4<B, 20, MODE>, grid, threads, smem, st, g, G1, Gh, part); break;
    case 24: pdl(k_ytoep4<B, 24, MODE>, grid, threads, smem, st, g, G1, Gh, part); break;
    default: pdl(k_ytoep4<B, 32, MODE>, grid, threads, smem, st, g, G1, Gh, part); break;
    }
}

template <int B>
void Launch<B>::ypass_toep(int E, dim3 grid, int threads, size_t smem, cudaStream_t st, const Geo &g, float2 *G1,
                           const float2 *Gh)
{
    if (ytoep4_fits(g.n1)) launch_ytoep4<B, 0>(grid, st, g, G1, Gh, nullptr);
    else if (E == 32) pdl(k_ypass_toep<B, 32>, grid, threads, smem, st, g, G1, Gh);
    else pdl(k_ypass_toep<B, 16>, grid, threads, smem, st, g, G1, Gh);
}

template <int B>
void Launch<B>::ypass_toep_quad(int E, dim3 grid, int threads, size_t smem, cudaStream_t st, const Geo &g,
                                const float2 *G1, double *part)
{
    if (ytoep4_fits(g.n1)) launch_ytoep4<B, 1>(grid, st, g, const_cast<float2 *>(G1), nullptr, part);
    else if (E == 32) pdl(k_ypass_toep_quad<B, 32>, grid, threads, smem, st, g, G1, part);
    else pdl(k_ypass_toep_quad<B, 16>, grid, threads, smem, st, g, G1, part);
}

// k_xtoep for one (BH, NA, NB) shape: grid (N1 * B/BH, G), half-groups fastest.
template <int B, int BH, int LA, int LNB>
static void xt_go(int mode, cudaStream_t st, int G, const XtArgs &a)
{
    using S = XtShape<BH, LA, LNB>;
    const dim3 grid((unsigned)(a.N1 * (B / BH)), (unsigned)G);
    const size_t smem = xtoep_smem(S::N, BH);
    if (mode == 0) pdl(k_xtoep<B, BH, LA, LNB, 0>, grid, S::T, smem, st, a);
    else if (mode == 1) {
        // After a y-pass of many small blocks the early launch of fewer blocks than
        // the SMs hold at once costs more than the gap that it saves (they seem to settle
        // on the SMs that empty first): one slice, an iteration of 1024 x 300 57 us (80
        // when early), 2048 x 100 54 (86), 4096 x 100 84 (103); four of 2048 x 40 51 (59). Above three fifths of what fits, and after
        // y-passes of fewer blocks, the early launch is ahead by 1 to 3 us (8 slices of
        // 1024 x 100 51 us, 53 without).
        const int fit = kSMs * (int)(227 * 1024 / (smem + 1024)), blocks = (int)(grid.x * grid.y);
        const bool early = S::N * G < 2048 || 5 * blocks > 3 * fit;
        pdl_if(early, k_xtoep<B, BH, LA, LNB, 1>, grid, S::T, smem, st, a);
    }
    else pdl(k_xtoep<B, BH, LA, LNB, 2>, grid, S::T, smem, st, a);
}
template <int B, int BH, int LA, int LNB>
static cudaError_t xt_attr()
{
    const int bytes = (int)xtoep_smem(XtShape<BH, LA, LNB>::N, BH);
    cudaError_t e = cudaFuncSetAttribute((const void *)k_xtoep<B, BH, LA, LNB, 0>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (e != cudaSuccess) return e;
    e = cudaFuncSetAttribute((const void *)k_xtoep<B, BH, LA, LNB, 2>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             bytes);
    if (e != cudaSuccess) return e;
    return cudaFuncSetAttribute((const void *)k_xtoep<B, BH, LA, LNB, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                bytes);
}

// Slices per CTA: all B below n0 = 1024, there 4 (four CTAs of 128 threads per SM
// overlap one's loads with another's transforms: 40.3 us a launch against 41.4 of
// two CTAs with all 8, 24 slices of 512 x 256), then at most 8192 / n0 (a CTA's
// transposed values stay at 64 KB, two CTAs per SM).
#define ICON_XT_SHAPES(X)                            \
    X(128, B, 2, 0)                                   \
    X(256, B, 3, 0)                                   \
    X(512, B, 4, 0)                                   \
    X(1024, (B < 4 ? B : 4), 5, 0)                    \
    X(2048, (B < 4 ? B : 4), 3, 3)                    \
    X(4096, (B < 2 ? B : 2), 4, 3)                    \
    X(8192, 1, 4, 4)

// k_xtoep_real for n0, by its half length: all B slices up to 1024, then at
// most 8192 / N.
#define ICON_XTR_SHAPES(X)                           \
    X(128, B, 1, 0)                                   \
    X(256, B, 2, 0)                                   \
    X(512, B, 3, 0)                                   \
    X(1024, B, 4, 0)                                  \
    X(2048, B, 5, 0)                                  \
    X(4096, (B < 4 ? B : 4), 3, 3)                    \
    X(8192, (B < 2 ? B : 2), 4, 3)

template <int B, int BH, int LA, int LNB>
static void xtr_go(cudaStream_t st, int G, const XtArgs &a)
{
    using S = XtShape<BH, LA, LNB>;
    pdl(k_xtoep_real<B, BH, LA, LNB>, dim3((unsigned)(a.N1 * (B / BH)), (unsigned)G), xtr_threads(S::T),
                                     sizeof(float2) * S::N * BH, st, a);
}
template <int B, int BH, int LA, int LNB>
static cudaError_t xtr_attr()
{
    return cudaFuncSetAttribute((const void *)k_xtoep_real<B, BH, LA, LNB>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)sizeof(float2) * XtShape<BH, LA, LNB>::N * BH);
}

template <int B>
void Launch<B>::xtoep_real(cudaStream_t st, int G, const XtArgs &a)
{
    switch (a.n0) {
#define X(N, BH, LA, LNB) \
    case N: xtr_go<B, BH, LA, LNB>(st, G, a); break;
        ICON_XTR_SHAPES(X)
#undef X
    default: break;
    }
}

template <int B>
bool Launch<B>::xtoep(int mode, cudaStream_t st, int G, const XtArgs &a)
{
    switch (a.n0) {
#define X(N, BH, LA, LNB) \
    case N: xt_go<B, BH, LA, LNB>(mode, st, G, a); return true;
        ICON_XT_SHAPES(X)
#undef X
    default: return false;
    }
}

template <int B>
cudaError_t Launch<B>::xtoep_prepare(int n0)
{
    cudaError_t e = cudaSuccess;
    switch (n0) {
#define X(N, BH, LA, LNB) \
    case N: e = xt_attr<B, BH, LA, LNB>(); break;
        ICON_XT_SHAPES(X)
#undef X
    default: break;
    }
    if (e != cudaSuccess) return e;
    switch (n0) {
#define X(N, BH, LA, LNB) \
    case N: return xtr_attr<B, BH, LA, LNB>();
        ICON_XTR_SHAPES(X)
#undef X
    default: return cudaSuccess;
    }
}

// Threads of k_yfwd4, at least the FFT's R B.  What is left after the FFT are the
// entries of a CTA, 850 or so where a real image's 61 tilts put two rows' on it,
// and the FFT of few threads is a chain that only other CTAs on the SM cover.  So: few
// CTAs take their entries by 256 threads (24 slices of 64 x 100 34 us the call, 51
// with 128, 66 with 64), many by 128 (24 of 2048 x 40 422 us, 516 with 256, 488 with
// 64); one row's entries (complex images) or a reprojection line's by 64 (lines of 8
// slices of 4096 x 40 158 us the call, 170 and 261; 8 complex slices of 4096 x 100
// 554, 607 and 844).
static int yfwd_threads(int fft_threads, bool herm, dim3 grid, const Geo &g)
{
    const long long entries = (long long)g.M * (g.thi - g.tlo + 1) * 2;
    const int want = !herm || entries < 64LL * g.n0 ? 64 : grid.x * grid.y <= 800 ? 256 : 128;
    return fft_threads > want ? fft_threads : want;
}

template <int B, int R>
static void yfwd4_go(bool herm, dim3 grid, cudaStream_t st, const Geo &g, const float2 *G1, float2 *P)
{
    const int threads = yfwd_threads(R * B, herm, grid, g);
    const size_t smem = yfwd4_smem(32 * R, B);
    if (herm) pdl(k_yfwd4<B, R, true>, grid, threads, smem, st, g, G1, P);
    else pdl(k_yfwd4<B, R, false>, grid, threads, smem, st, g, G1, P);
}

template <int B>
void Launch<B>::ypass_fwd(int E, bool herm, dim3 grid, int threads, size_t smem, cudaStream_t st, const Geo &g,
                          const float2 *G1, float2 *P)
{
    switch (yadj4_fits(g.n1) ? g.n1 / 32 : 0) {
    case 4: yfwd4_go<B, 4>(herm, grid, st, g, G1, P); return;
    case 8: yfwd4_go<B, 8>(herm, grid, st, g, G1, P); return;
    case 16: yfwd4_go<B, 16>(herm, grid, st, g, G1, P); return;
    case 32: yfwd4_go<B, 32>(herm, grid, st, g, G1, P); return;
    default: break;
    }
    if (E == 32) {
        if (herm) pdl(k_ypass_fwd<B, 32, true>, grid, threads, smem, st, g, G1, P);
        else pdl(k_ypass_fwd<B, 32, false>, grid, threads, smem, st, g, G1, P);
    } else {
        if (herm) pdl(k_ypass_fwd<B, 16, true>, grid, threads, smem, st, g, G1, P);
        else pdl(k_ypass_fwd<B, 16, false>, grid, threads, smem, st, g, G1, P);
    }
}

template <int B>
void Launch<B>::interp_fin(int mode, bool herm, dim3 grid, cudaStream_t st, const Geo &g, const float2 *P, float2 *f,
                           double *part)
{
    // After the y-pass of a complex image, whose last rows are among its heaviest, the
    // early launch costs more than the gap that it saves: 24 slices of 2048 x 40 462 us
    // the call (526 when early), one of 1024 x 100 41 (56). Small calls keep it (64 x 40
    // 21.4 us, 23.2 without).
    const bool early = herm || g.n0 * (int)grid.y < 2048;
    if (mode == 0) pdl_if(early, k_interp_fin<0, B>, grid, 256, 0, st, g, P, f, part);
    else if (mode == 1) pdl_if(early, k_interp_fin<1, B>, grid, 256, 0, st, g, P, f, part);
    else pdl_if(early, k_interp_fin<2, B>, grid, 256, 0, st, g, P, f, part);
}

template <int B>
void Launch<B>::ypass_adj(int E, dim3 grid, int threads, size_t smem, cudaStream_t st, const Geo &g, const float2 *f,
                          float2 *G1)
{
    switch (yadj4_fits(g.n1) ? g.n1 / 32 : 0) {
    case 4: pdl(k_yadj4<B, 4>, grid, threads, smem, st, g, f, G1); break;
    case 8: pdl(k_yadj4<B, 8>, grid, threads, smem, st, g, f, G1); break;
    case 16: pdl(k_yadj4<B, 16>, grid, threads, smem, st, g, f, G1); break;
    case 32: pdl(k_yadj4<B, 32>, grid, threads, smem, st, g, f, G1); break;
    default:
        if (E == 32) pdl(k_ypass_adj<B, 32, false>, grid, threads, smem, st, g, f, G1);
        else if (threads == g.n1 * B / 16) pdl(k_ypass_adj<B, 16, false>, grid, threads, smem, st, g, f, G1);
        else pdl(k_ypass_adj<B, 16, true>, grid, threads, smem, st, g, f, G1);
    }
}

template <int B>
void Launch<B>::xpass_adj(int mode, int E, dim3 grid, int threads, size_t smem, cudaStream_t st, const Geo &g,
                          const float2 *G1, float2 *out, const float2 *Ahwb, double *part)
{
    if (E == 32) {
        pdl(k_xpass_adj<1, B, 32>, grid, threads, smem, st, g, G1, out, Ahwb, part);   // mode 0: k_xtoep
    } else {
        if (mode == 0) pdl(k_xpass_adj<0, B, 16>, grid, threads, smem, st, g, G1, out, Ahwb, part);
        else pdl(k_xpass_adj<1, B, 16>, grid, threads, smem, st, g, G1, out, Ahwb, part);
    }
}

template <int B>
void Launch<B>::rows_fwd(int E, dim3 grid, int threads, size_t smem, cudaStream_t st, const Geo &g, const Geo1 &g1,
                         const float *rows, size_t sstride, size_t istride, int skip, int S, float2 *f,
                         float2 *bout)
{
    if (E == 32) pdl(k_rows_fwd<B, 32>, grid, threads, smem, st, g, g1, rows, sstride, istride, skip, S, f, bout);
    else pdl(k_rows_fwd<B, 16>, grid, threads, smem, st, g, g1, rows, sstride, istride, skip, S, f, bout);
}

template <int B>
void Launch<B>::alpha(cudaStream_t st, int G, const double *rtr, int nr, const double *rtar, int na, double *alpha,
                      double *hist_alpha, double *hist_rtr)
{
    pdl(k_alpha<B>, G, kAlphaThreads, 0, st, rtr, nr, rtar, na, alpha, hist_alpha, hist_rtr);
}

template <int B, typename T, bool IN>
static void img_move(cudaStream_t st, int G, const T *src, T *dst, int S, int N0, int N1)
{
    using I = ImgTile<T, B>;
    const dim3 grid((N1 + I::TY - 1) / I::TY, (N0 + I::TX - 1) / I::TX, G);
    pdl(k_img_move<T, B, IN>, grid, 256, 0, st, src, dst, S, N0, N1);
}
template <int B>
void Launch<B>::img_in(cudaStream_t st, int G, const float *src, float *dst, int S, int N0, int N1)
{
    img_move<B, float, true>(st, G, src, dst, S, N0, N1);
}
template <int B>
void Launch<B>::img_in(cudaStream_t st, int G, const float2 *src, float2 *dst, int S, int N0, int N1)
{
    img_move<B, float2, true>(st, G, src, dst, S, N0, N1);
}
template <int B>
void Launch<B>::img_out(cudaStream_t st, int G, const float *src, float *dst, int S, int N0, int N1)
{
    img_move<B, float, false>(st, G, src, dst, S, N0, N1);
}
template <int B>
void Launch<B>::img_out(cudaStream_t st, int G, const float2 *src, float2 *dst, int S, int N0, int N1)
{
    img_move<B, float2, false>(st, G, src, dst, S, N0, N1);
}
template <int B>
void Launch<B>::nodes_in(cudaStream_t st, int G, const float2 *src, float2 *dst, int S, int M)
{
    pdl(k_nodes_in<B>, dim3((M + 127) / 128, G), 128, 0, st, src, dst, S, M);
}
template <int B>
void Launch<B>::nodes_out(cudaStream_t st, int G, const float2 *src, float2 *dst, int S, int M)
{
    pdl(k_nodes_out<B>, dim3((M + 127) / 128, G), 128, 0, st, src, dst, S, M);
}

template <int B>
void Launch<B>::img_out_file(dim3 grid, cudaStream_t st, const float *m, float *out, int S, int N0, int N1)
{
    pdl(k_img_out_file<B>, grid, 256, 0, st, m, out, S, N0, N1);
}

template <int B>
void Launch<B>::row_adj(int E, dim3 grid, int threads, size_t smem, cudaStream_t st, const Geo &g, const Geo1 &g1,
                        const float2 *f, float *out, int S)
{
    if (E == 32) pdl(k_row_adj<B, 32>, grid, threads, smem, st, g, g1, f, out, S);
    else pdl(k_row_adj<B, 16>, grid, threads, smem, st, g, g1, f, out, S);
}

template <int B>
void Launch<B>::update(dim3 grid, cudaStream_t st, float *m, const float2 *rhat, const double *alpha, int per_group,
                       int clamp, int data_type, float thr, double *step_part)
{
    if (step_part) pdl(k_update<B, true>, grid, 256, 0, st, m, rhat, alpha, per_group, clamp, data_type, thr, step_part);
    else pdl(k_update<B, false>, grid, 256, 0, st, m, rhat, alpha, per_group, clamp, data_type, thr, (double *)nullptr);
}

template <int B>
void Launch<B>::update_re(dim3 grid, cudaStream_t st, float *m, const float *rre, const double *alpha, int per_group,
                          int clamp, int data_type, float thr)
{
    pdl(k_update<B, false, float>, grid, 256, 0, st, m, rre, alpha, per_group, clamp, data_type, thr, (double *)nullptr);
}

// The dynamic shared-memory limit is a property of the kernel function, not
// of a plan: plans of different sizes share the variants of one B, so every
// variant gets the device's opt-in maximum (what a launch actually asks for
// still sets the occupancy).  Lowering it to one plan's size would make a
// larger plan's next launch fail.  Only the variants that a plan of these
// sizes launches are set: all of a B's take 0.3 ms of the small plans' 1.4.
template <int B>
cudaError_t Launch<B>::set_smem(int ex, int ey, int n1, int n1t)
{
    int dev = 0, optin = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    if (e != cudaSuccess) return e;
    auto set = [&](const void *fn) {
        cudaError_t r = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, optin);
        if (r != cudaSuccess && e == cudaSuccess) e = r;
    };
    if (ex == 32) {
        set((const void *)k_xpass_fwd<false, B, 32>);
        set((const void *)k_xpass_fwd_r2c<B, 32, true>);
        set((const void *)k_xpass_adj<1, B, 32>);
        set((const void *)k_rows_fwd<B, 32>);
        set((const void *)k_row_adj<B, 32>);
    } else {
        set((const void *)k_xpass_fwd<true, B, 16>);
        set((const void *)k_xpass_fwd<false, B, 16>);
        set((const void *)k_xpass_fwd_r2c<B, 16>);
        set((const void *)k_xpass_fwd_r2c<B, 16, true>);
        set((const void *)k_xpass_fwd<true, B, 16, true>);
        set((const void *)k_xpass_adj<0, B, 16>);
        set((const void *)k_xpass_adj<1, B, 16>);
        set((const void *)k_rows_fwd<B, 16>);
        set((const void *)k_row_adj<B, 16>);
    }
    switch (yadj4_fits(n1) ? n1 / 32 : 0) {
#define X(R) \
    case R: \
        set((const void *)k_yfwd4<B, R, false>); \
        set((const void *)k_yfwd4<B, R, true>); \
        set((const void *)k_yadj4<B, R>); \
        break;
        X(4) X(8) X(16) X(32)
#undef X
    default:
        if (ey == 32) {
            set((const void *)k_ypass_fwd<B, 32, false>);
            set((const void *)k_ypass_fwd<B, 32, true>);
            set((const void *)k_ypass_adj<B, 32, false>);
        } else {
            set((const void *)k_ypass_fwd<B, 16, false>);
            set((const void *)k_ypass_fwd<B, 16, true>);
            set((const void *)k_ypass_adj<B, 16, false>);
            set((const void *)k_ypass_adj<B, 16, true>);
        }
    }
    switch (ytoep4_fits(n1t) ? n1t / 32 : 0) {
#define X(R) \
    case R: \
        set((const void *)k_ytoep4<B, R, 0>); \
        set((const void *)k_ytoep4<B, R, 1>); \
        break;
        X(4) X(6) X(8) X(10) X(12) X(16) X(20) X(24) X(32)
#undef X
    default:
        if (ey == 32) {
            set((const void *)k_ypass_toep<B, 32>);
            set((const void *)k_ypass_toep_quad<B, 32>);
        } else {
            set((const void *)k_ypass_toep<B, 16>);
            set((const void *)k_ypass_toep_quad<B, 16>);
        }
    }
    return e;
}

template struct Launch<ICON_KB>;

}  // namespace icon
