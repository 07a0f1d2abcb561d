// Device-side bodies of the 2D projectors, shared by the single-problem
// kernels (proj2d.cu) and the batched persistent kernels (batch2d.cu): one
// ray of a forward projection, one pixel of a backprojection.
//
// Model: cuda/2d/par_fp.cu (FPhorizontal_simple / FPvertical_simple, 53-200),
// cuda/2d/fan_fp.cu (FanFPhorizontal / FanFPvertical, 55-193),
// cuda/2d/par_bp.cu (devBP / devBP_SS, 52-137) and cuda/2d/fan_bp.cu
// (devFanBP / devFanBP_SS, 57-161), with explicit FP32 linear interpolation
// and a zero border in place of texture fetches.
#pragma once

#include <cuda_runtime.h>

#include "proj2d.h"

namespace b2t {

// linear interpolation of a 1D line at continuous index q (texel i at q = i),
// zero outside [0, n)
__device__ __forceinline__ float lerp_line(const float *__restrict__ p, long long stride, int n, float q)
{
    const float fl = floorf(q);
    const int k = (int)fl;
    const float f = q - fl;
    const float a = (k >= 0 && k < n) ? __ldg(p + (long long)k * stride) : 0.0f;
    const float b = (k + 1 >= 0 && k + 1 < n) ? __ldg(p + (long long)(k + 1) * stride) : 0.0f;
    return fmaf(f, b - a, a);
}

// Reciprocal: the hardware's approximation (one ulp) and one Newton-Raphson
// step r + r (1 - x r), whose residual is exact to FP32 in a fused
// multiply-add; within one ulp of 1 / x.
__device__ __forceinline__ float rcp_approx(float x)
{
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
__device__ __forceinline__ float rcp_newton(float x)
{
    const float r = rcp_approx(x);
    return fmaf(r, fmaf(-x, r, 1.0f), r);
}

// Partial sums of a line integral and of a pixel's backprojection: the slices
// (views) are cut into this many ranges of equal length, each summed on its
// own and the partial sums then added in order.  The fixed cut lets the line
// kernels (lines2d.cu) give the ranges of a short problem to different warps
// and still return the bits of the kernels that run them one after another.
constexpr int FP2D_PARTS = 4;
constexpr int BP2D_PARTS = 8;

__host__ __device__ __forceinline__ int part_begin(int p, int n, int parts)
{
    return (int)((long long)n * p / parts);
}

// Parts of a ray's slices begin at multiples of four (the direct bodies sum
// four slices at a time and test once for the end of a part).
__host__ __device__ __forceinline__ int slice_begin(int p, int n)
{
    return p < FP2D_PARTS ? part_begin(p, n, FP2D_PARTS) & ~3 : n;
}

// A ray: sample position q(slice) = A slice + B in texels (texel i at q = i)
// of the line along the other axis; horizontal: slices are columns.
struct Ray2D {
    float A, B, corr;
    bool horizontal;
};

// Sub-ray r of R of detector det of a parallel view (corr: see V.corr).
__device__ __forceinline__ Ray2D par_ray2d(const ParFPView &V, int det, int r, int R)
{
    Ray2D q;
    q.A = V.slicestep;
    q.B = fmaf((float)det + (0.5f + (float)r) / (float)R - 0.5f, V.detstep, V.p0) - 0.5f;
    q.corr = V.corr;
    q.horizontal = !V.vertical;
    return q;
}

// Whether a fan view's rays to detector det march over columns: the choice of
// every ray, in float as the reference evaluates it.
__device__ __forceinline__ bool fan_horizontal(const b2t_view2d &V, int det)
{
    const float fdx = fabsf(fmaf((float)det, V.det_u[0], V.det_s[0]) + 0.5f - V.src[0]);
    const float fdy = fabsf(fmaf((float)det, V.det_u[1], V.det_s[1]) + 0.5f - V.src[1]);
    return !(fdy > fdx);
}

// Sub-ray r of R of detector det of a fan view, scaled for the mean over R.
__device__ __forceinline__ Ray2D fan_ray2d(const b2t_view2d &V, bool horizontal, int W, int H, int det, int r, int R,
                                           float out_scale)
{
    Ray2D q;
    q.horizontal = horizontal;
    // ray set-up in FP64: the source sits far from the origin
    const double fdet = det + (0.5 + r) / (double)R;
    const double DX = V.det_s[0] + fdet * V.det_u[0];
    const double DY = V.det_s[1] + fdet * V.det_u[1];
    if (horizontal) {
        const double alpha = (V.src[1] - DY) / (V.src[0] - DX);
        const double beta = V.src[1] - alpha * V.src[0];
        q.corr = (float)(sqrt(alpha * alpha + 1.0) * out_scale / R);
        q.B = (float)(-alpha * (0.5 - 0.5 * W) - beta + 0.5 * H - 0.5);
        q.A = (float)-alpha;
    } else {
        const double alpha = (V.src[0] - DX) / (V.src[1] - DY);
        const double beta = V.src[0] - alpha * V.src[1];
        q.corr = (float)(sqrt(alpha * alpha + 1.0) * out_scale / R);
        q.B = (float)(-alpha * (0.5 - 0.5 * H) + beta + 0.5 * W - 0.5);
        q.A = (float)-alpha;
    }
    return q;
}

// Sum of the samples of a ray over slices s0, s0 + ds, ...; with ds = 1 from
// slice 0 all of them, in FP2D_PARTS partial sums.  COLS: the slices are
// columns.
//
// Bound by the latency of the loads; the compiler unrolls one plain loop with
// four samples' loads in flight, and a loop within a loop costs it (one view of
// a 4096^2 image over rows: 283 us; a loop for every part 373 us; the choice of
// direction inside the loop over sub-rays, or that loop around a single
// ray, 300 to 470 us; run-time strides took the batched projections 1.15 to 1.18
// times as long).  Hence the three tests in place of four loops, and the
// branches on direction and on one sub-ray around everything else.
template <bool COLS>
__device__ __forceinline__ float sum_slices2d(const float *vol, long long pitch, int W, int H, const Ray2D &q, int s0,
                                              int ds)
{
    const int n0 = COLS ? W : H;
    auto sample = [&](int sl) {
        const float x = fmaf((float)sl, q.A, q.B);
        return COLS ? lerp_line(vol + sl, pitch, H, x) : lerp_line(vol + (long long)sl * pitch, 1, W, x);
    };
    float tot = 0.0f, sum = 0.0f;
    if (ds != 1) {
        for (int sl = s0; sl < n0; sl += ds) sum += sample(sl);
        return sum;
    }
    static_assert(FP2D_PARTS == 4, "three ends between parts");
    const int e1 = slice_begin(1, n0), e2 = slice_begin(2, n0), e3 = slice_begin(3, n0);
    auto fold = [&](int sl) {
        if (sl == e1 || sl == e2 || sl == e3) {
            tot += sum;
            sum = 0.0f;
        }
    };
    int sl = 0;
#pragma unroll 1
    for (; sl + 3 < n0; sl += 4) {
        float v[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) v[i] = sample(sl + i);
        fold(sl);
#pragma unroll
        for (int i = 0; i < 4; ++i) sum += v[i];
    }
    fold(sl);
    for (; sl < n0; ++sl) sum += sample(sl);
    return tot + sum;
}

// Sum over the R sub-rays of detector det: of a parallel view unscaled (all
// share V.corr), of a fan view scaled.
template <bool COLS>
__device__ __forceinline__ float par_rays2d(const float *vol, long long pitch, int W, int H, const ParFPView &V, int det,
                                            int R, int s0, int ds)
{
    if (R == 1) return sum_slices2d<COLS>(vol, pitch, W, H, par_ray2d(V, det, 0, 1), s0, ds);
    float acc = 0.0f;
    for (int r = 0; r < R; ++r) acc += sum_slices2d<COLS>(vol, pitch, W, H, par_ray2d(V, det, r, R), s0, ds);
    return acc;
}
template <bool COLS>
__device__ __forceinline__ float fan_rays2d(const float *vol, long long pitch, int W, int H, const b2t_view2d &V, int det,
                                            int R, float out_scale, int s0, int ds)
{
    auto ray = [&](int r, int n, float acc) {
        const Ray2D q = fan_ray2d(V, COLS, W, H, det, r, n, out_scale);
        return fmaf(sum_slices2d<COLS>(vol, pitch, W, H, q, s0, ds), q.corr, acc);
    };
    if (R == 1) return ray(0, 1, 0.0f);
    float acc = 0.0f;
    for (int r = 0; r < R; ++r) acc = ray(r, R, acc);
    return acc;
}

// Parallel-beam line integral of detector `det` (R sub-rays), scaled; over
// slices s0, s0 + ds, ... (all slices by default; a partial sum otherwise).
__device__ __forceinline__ float fp2d_par_ray(const float *vol, long long pitch, int W, int H, const ParFPView &V,
                                              int det, int R, int s0 = 0, int ds = 1)
{
    const float acc = V.vertical ? par_rays2d<false>(vol, pitch, W, H, V, det, R, s0, ds)
                                 : par_rays2d<true>(vol, pitch, W, H, V, det, R, s0, ds);
    return __fmul_rn(acc, V.corr / (float)R);  // (not fused into an accumulating caller)
}

// Fan-beam line integral of detector `det` (R sub-rays), scaled; over slices
// s0, s0 + ds, ... as fp2d_par_ray.
__device__ __forceinline__ float fp2d_fan_ray(const float *vol, long long pitch, int W, int H, const b2t_view2d &V,
                                              int det, int R, float out_scale, int s0 = 0, int ds = 1)
{
    return fan_horizontal(V, det) ? fan_rays2d<true>(vol, pitch, W, H, V, det, R, out_scale, s0, ds)
                                  : fan_rays2d<false>(vol, pitch, W, H, V, det, R, out_scale, s0, ds);
}

// Backprojection sum of pixel (X, Y) over views [0, nviews) of `views`
// (sinogram rows row0 .. row0 + nviews - 1), R x R sub-pixels, unscaled, in
// BP2D_PARTS partial sums.  ONE: R is 1 (the short ranges of a batch's small
// problems show the loops over sub-pixels).
template <bool ONE>
__device__ __forceinline__ float bp2d_pixel_sum(const float *sino, long long sino_pitch, int row0, int nviews,
                                                const BPView2D *views, int W, int H, int ndet, int R, int kind, int fbp,
                                                int X, int Y)
{
    const float sub = 1.0f / (float)R;
    auto add_view = [&](int i, float &acc) {
        const BPView2D &C = views[i];
        const float *row = sino + (long long)(row0 + i) * sino_pitch;
        for (int ix = 0; ix < (ONE ? 1 : R); ++ix) {
            for (int iy = 0; iy < (ONE ? 1 : R); ++iy) {
                float x = (float)X - 0.5f * (float)W + 0.5f;
                float y = (float)Y - 0.5f * (float)H + 0.5f;
                if (!ONE && R > 1) {
                    x += -0.5f + 0.5f * sub + (float)ix * sub;
                    y += -0.5f + 0.5f * sub + (float)iy * sub;
                }
                if (kind == B2T_GEOM_PAR2D) {
                    // T - 1/2, T = x c - y s + offset (par_bp.cu:78-81)
                    const float q = fmaf(x, C.c[0], fmaf(-y, C.c[1], C.c[2] - 0.5f));
                    acc = fmaf(lerp_line(row, 1, ndet, q), C.c[3], acc);
                } else {
                    // world y is flipped (fan_bp.cu:73)
                    const float yw = -y;
                    const float num = fmaf(x, C.c[1], fmaf(yw, C.c[2], C.c[0]));
                    const float den = fmaf(x, C.c[4], fmaf(yw, C.c[5], C.c[3]));
                    const float fr = rcp_newton(den);
                    const float w = fbp ? fr * fr : fr;
                    acc = fmaf(lerp_line(row, 1, ndet, fmaf(num, fr, -0.5f)), w, acc);
                }
            }
        }
    };
    float tot = 0.0f;
    if (nviews <= BP2D_PARTS) {
        // a view or none in every part (4096^2, one view: 180 us with the loop below)
        for (int i = 0; i < nviews; ++i) {
            float acc = 0.0f;
            add_view(i, acc);
            tot += acc;
        }
        return tot;
    }
    for (int p = 0; p < BP2D_PARTS; ++p) {
        const int end = part_begin(p + 1, nviews, BP2D_PARTS);
        float acc = 0.0f;
        for (int i = part_begin(p, nviews, BP2D_PARTS); i < end; ++i) add_view(i, acc);
        tot += acc;
    }
    return tot;
}

__device__ __forceinline__ float bp2d_pixel(const float *sino, long long sino_pitch, int row0, int nviews,
                                            const BPView2D *views, int W, int H, int ndet, int R, int kind, int fbp,
                                            int X, int Y)
{
    return R == 1 ? bp2d_pixel_sum<true>(sino, sino_pitch, row0, nviews, views, W, H, ndet, 1, kind, fbp, X, Y)
                  : bp2d_pixel_sum<false>(sino, sino_pitch, row0, nviews, views, W, H, ndet, R, kind, fbp, X, Y);
}

}  // namespace b2t
