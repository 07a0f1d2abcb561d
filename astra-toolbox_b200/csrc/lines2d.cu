// 2D forward and back projection from lines of texel pairs.
//
// Same models, and the same bits, as the direct bodies in proj2d_dev.cuh (the
// reference's cuda/2d/par_fp.cu:53-200, fan_fp.cu:55-193, par_bp.cu:52-137,
// fan_bp.cu:57-161): linear samples of lines, of the image's rows or columns
// in a forward projection and of the sinogram's rows in a backprojection.
//
// The direct bodies load two texels per sample, test both against the ends of
// the line and, where a ray marches over columns, touch one cache line per
// lane (10.2 ms for both directions at 1024^2 x 1440 views, 1536 detectors).
// Here a line is held as pairs (v[k], v[k + 1] - v[k]) of neighbouring texels
// inside zeros: a sample is one 8-byte load with neighbouring lanes on
// neighbouring pairs, and one FMA; positions and texel splits of two samples
// share packed f32x2 instructions (1.4 ms at the same size).
//   - FP: the image's rows and, transposed, its columns are copied once per
//     call (fp2d_lines); rays read the copy through L1.
//   - BP: every CTA stages the pairs its pixels sample in shared memory, some
//     views at a time, straight from the sinogram (bp2d_lines).
//
// Ranges of slices (FP) or views (BP) are summed separately and then in order
// (FP2D_PARTS, BP2D_PARTS), so that a problem with few rays or pixels spreads
// one ray's or pixel's ranges over the warps of a CTA.
#include <cuda_runtime.h>

#include <algorithm>
#include <climits>
#include <cmath>
#include <memory>
#include <type_traits>

#include "b2t_internal.h"
#include "f32x2.cuh"
#include "proj2d.h"
#include "proj2d_dev.cuh"
#include "tma.h"

namespace b2t {

namespace {

constexpr float SPLIT_M = 12582912.0f;        // 1.5 * 2^23: q + M rounded down holds floor(q) in its bits
constexpr uint32_t SPLIT_BITS = 0x4B400000u;  // bits of SPLIT_M
constexpr int LINE_BORDER = 2;                // zero texels on both sides of a line
constexpr int LINES_THREADS = 256;
constexpr int LINES_WARPS = LINES_THREADS / 32;
constexpr int LINES_MAX_WIN = 160;            // pairs of a staged sinogram row (bp2d_lines), even

// Pairs of line l at out[l * pitch + k + 2], k in [-2, n + 2).
struct LineSet {
    float2 *out;
    int lines, n, pitch;
    int transposed;  // line l is column l of the source
};
struct BuildLines {
    const float *src;
    long long src_pitch;
    LineSet set[2];
    int nsets;
};

// One 32 x 32 tile of pairs per block: 32 lines x 32 texels of set
// blockIdx.z, staged in shared memory when the lines are source columns.
__global__ void __launch_bounds__(LINES_THREADS) build_lines_kernel(const BuildLines B)
{
    __shared__ float t[33][33];
    const LineSet S = B.set[blockIdx.z];
    const int l0 = blockIdx.y * 32;
    const int k0 = (int)blockIdx.x * 32 - LINE_BORDER;
    if (l0 >= S.lines || k0 >= S.n + LINE_BORDER) return;
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    if (S.transposed) {
        // t[texel][line], read along the source rows
        for (int j = ty; j < 33; j += LINES_WARPS) {
            const int k = k0 + j, l = l0 + tx;
            t[j][tx] = (k >= 0 && k < S.n && l < S.lines) ? __ldg(B.src + (long long)k * B.src_pitch + l) : 0.0f;
        }
        __syncthreads();
        const int k = k0 + tx;
        if (k >= S.n + LINE_BORDER) return;
        for (int j = ty; j < 32 && l0 + j < S.lines; j += LINES_WARPS) {
            const float a = t[tx][j], b = t[tx + 1][j];
            S.out[(size_t)(l0 + j) * S.pitch + k + LINE_BORDER] = make_float2(a, b - a);
        }
    } else {
        const int k = k0 + tx;
        if (k >= S.n + LINE_BORDER) return;
        for (int j = ty; j < 32 && l0 + j < S.lines; j += LINES_WARPS) {
            const float *row = B.src + (long long)(l0 + j) * B.src_pitch;
            const float a = (k >= 0 && k < S.n) ? __ldg(row + k) : 0.0f;
            const float b = (k + 1 >= 0 && k + 1 < S.n) ? __ldg(row + k + 1) : 0.0f;
            S.out[(size_t)(l0 + j) * S.pitch + k + LINE_BORDER] = make_float2(a, b - a);
        }
    }
}

// The pair of the texel whose split bits are `bits` on the line at byte
// address `line` (of texel 0, less the split's constant bits, which the wide
// multiply-add takes back).
__device__ __forceinline__ float2 ld_pair(unsigned long long line, int bits)
{
    return __ldg(reinterpret_cast<const float2 *>(line + (unsigned long long)(uint32_t)bits * 8u));
}

__device__ __forceinline__ int floor_texel(float q) { return __float_as_int(__fadd_rd(q, SPLIT_M)) - (int)SPLIT_BITS; }

// ---------------------------------------------------------------------------
// forward projection
// ---------------------------------------------------------------------------

constexpr int FP2D_GROUPS = LINES_WARPS / FP2D_PARTS;  // groups of 16 detectors x 4 views per CTA

// CAP views' constants travel in the launch parameters.
template <int CAP> struct FP2DLinesLaunch {
    // texel 0 of line 0 and byte pitch of a line: rows (rays that march over
    // rows, [0]) and columns ([1])
    const char *line0[2];
    uint32_t pitch[2];
    float *sino;
    long long sino_pitch;
    int W, H, ndet, rays, accumulate, a0, nviews;
    float out_scale;
    const float *res_b, *res_w;  // SIRT's residual in place of the projection: (b - A x) w
    union {
        ParFPView par[CAP];
        b2t_view2d fan[CAP];
    };
};

// A lane's ray: position A slice + B, byte address of texel 0 of line 0 (less
// the split's constant bits), byte pitch of a line, and the slices [lo, hi] where its
// base texel lies in [-2, n] (lo > hi: none; the ray then reads the border
// of line 0, so that it needs no test); n0 slices, n texels a line.
struct LineRay {
    float A, B;
    unsigned long long row;
    uint32_t pitch;
    int lo, hi, n0, n;
};

__device__ __forceinline__ void clip_line(LineRay &r)
{
    const int n = r.n;
    // a quarter texel inside the border: every slice with a sample in the line
    // is kept, and rounding cannot leave the border (A = 0: infinities of one
    // sign, or of both when the whole ray lies inside)
    const float s1 = (-1.75f - r.B) / r.A, s2 = ((float)n + 0.75f - r.B) / r.A;
    const float a = fmaxf(0.0f, fminf(s1, s2)), b = fminf((float)(r.n0 - 1), fmaxf(s1, s2));
    int lo = (int)ceilf(a), hi = (int)floorf(b);
    // the base texel is monotone in the slice, so inside at both ends is
    // inside everywhere between (an ill-conditioned ray is cut to where it is)
    auto inside = [&](int s) {
        const int k = floor_texel(fmaf((float)s, r.A, r.B));
        return k >= -LINE_BORDER && k <= n;
    };
    while (lo <= hi && !inside(lo)) ++lo;
    while (lo <= hi && !inside(hi)) --hi;
    r.lo = lo;
    r.hi = hi;
    if (lo > hi) {
        r.A = 0.0f;
        r.B = -(float)LINE_BORDER;
        r.pitch = 0;
    }
}

// Sums of the lane's two rays over range p of their slices.
template <bool SAME_LINE>
__device__ __forceinline__ void sum_part(const LineRay (&ray)[2], bool mixed, int p, float (&sum)[2])
{
    int lo[2], hi[2];
    int ulo = INT_MAX, uhi = INT_MIN, ilo = INT_MIN, ihi = INT_MAX;
#pragma unroll
    for (int j = 0; j < 2; ++j) {
        lo[j] = max(ray[j].lo, slice_begin(p, ray[j].n0));
        hi[j] = min(ray[j].hi, slice_begin(p + 1, ray[j].n0) - 1);
        if (ray[j].lo <= ray[j].hi) {
            const bool some = lo[j] <= hi[j];
            ulo = min(ulo, some ? lo[j] : INT_MAX);
            uhi = max(uhi, some ? hi[j] : INT_MIN);
            ilo = max(ilo, some ? lo[j] : INT_MAX);
            ihi = min(ihi, some ? hi[j] : INT_MIN);
        }
        sum[j] = 0.0f;
    }
    // the warp's slices: those of any ray [ulo, uhi], those of every ray [ilo, ihi]
    ulo = __reduce_min_sync(0xffffffffu, ulo);
    uhi = __reduce_max_sync(0xffffffffu, uhi);
    ilo = __reduce_max_sync(0xffffffffu, ilo);
    ihi = __reduce_min_sync(0xffffffffu, ihi);
    if (ulo > uhi) return;
    const int f0 = ilo <= ihi ? max(ilo, ulo) : uhi + 1, f1 = min(ihi, uhi);

    // Slices [s0, s1] of both rays, UNR at a time with their loads in flight
    // together.  CLAMP: base texels are clamped into the zero border (slices
    // at which some ray of the warp is outside its line).
    const uint64_t A2 = pk2(ray[0].A, ray[1].A), B2 = pk2(ray[0].B, ray[1].B);
    const uint64_t M2 = pk2(SPLIT_M, SPLIT_M), nM2 = pk2(-SPLIT_M, -SPLIT_M), one2 = pk2(1.0f, 1.0f);
    auto slices = [&](int s0, int s1, auto clamp) {
        constexpr bool CLAMP = decltype(clamp)::value;
        constexpr int UNR = 4;
        uint64_t s2 = pk2((float)s0, (float)s0);
        unsigned long long r0 = ray[0].row + (unsigned long long)(uint32_t)s0 * ray[0].pitch;
        unsigned long long r1 = ray[1].row + (unsigned long long)(uint32_t)s0 * ray[1].pitch;
        auto sample = [&](float2 &f, float2 &v0, float2 &v1) {
            const uint64_t q = fma2(s2, A2, B2);
            const uint64_t t = add2_rd(q, M2);
            f = upk2(sub2(q, add2(t, nM2)));
            const float2 tb = upk2(t);
            int b0 = __float_as_int(tb.x), b1 = __float_as_int(tb.y);
            if (CLAMP) {
                b0 = min(max(b0, (int)SPLIT_BITS - LINE_BORDER), (int)SPLIT_BITS + ray[0].n);
                b1 = min(max(b1, (int)SPLIT_BITS - LINE_BORDER), (int)SPLIT_BITS + ray[1].n);
            }
            v0 = ld_pair(r0, b0);
            v1 = ld_pair(SAME_LINE ? r0 : r1, b1);
            s2 = add2(s2, one2);
            r0 += ray[0].pitch;
            if (!SAME_LINE) r1 += ray[1].pitch;
        };
        int s = s0;
        for (; s + UNR - 1 <= s1; s += UNR) {
            float2 f[UNR], v0[UNR], v1[UNR];
#pragma unroll
            for (int i = 0; i < UNR; ++i) sample(f[i], v0[i], v1[i]);
#pragma unroll
            for (int i = 0; i < UNR; ++i) {
                sum[0] += fmaf(f[i].x, v0[i].y, v0[i].x);
                sum[1] += fmaf(f[i].y, v1[i].y, v1[i].x);
            }
        }
        for (; s <= s1; ++s) {
            float2 f, v0, v1;
            sample(f, v0, v1);
            sum[0] += fmaf(f.x, v0.y, v0.x);
            sum[1] += fmaf(f.y, v1.y, v1.x);
        }
    };
    if (mixed) {
        // rays over rows and over columns in one warp: their slice counts
        // differ, so a slice is tested against each ray's own range
        for (int s = ulo; s <= uhi; ++s) {
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                if (s >= lo[j] && s <= hi[j]) {
                    const float q = fmaf((float)s, ray[j].A, ray[j].B);
                    const float t = __fadd_rd(q, SPLIT_M);
                    const float f = q - (t - SPLIT_M);
                    const float2 v = ld_pair(ray[j].row + (unsigned long long)(uint32_t)s * ray[j].pitch, __float_as_int(t));
                    sum[j] += fmaf(f, v.y, v.x);
                }
            }
        }
        return;
    }
    slices(ulo, f0 - 1, std::true_type{});
    slices(f0, f1, std::false_type{});
    slices(max(f0, f1 + 1), uhi, std::true_type{});
}

// A warp traces 16 neighbouring detectors of 4 consecutive views: lane
// (detector & 7, view), two rays 8 detectors apart per lane.  Neighbouring
// views sample nearly the same texels at the same slice, so a load of the
// warp falls within about 16 pairs, one or two cache lines (against three or
// four for 32 detectors of one view).  A CTA traces two such groups, each
// group's FP2D_PARTS ranges of slices one warp each: four times the warps of
// one per group, which a small problem needs (128^2 x 180 parallel: 33 us with
// one warp, 24 with two, 18 with four) and a large one does not lose by
// (1024^2 x 1440: 0.89, 0.97, 0.84 ms).  Bound by the latency of L2: 44 % of the
// issue rate, seven sectors in ten miss L1.
template <int KIND, int CAP>
__global__ void __launch_bounds__(LINES_THREADS) fp2d_lines_kernel(const __grid_constant__ FP2DLinesLaunch<CAP> L)
{
    __shared__ float red[FP2D_GROUPS][FP2D_PARTS][64];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int grp = warp / FP2D_PARTS, part = warp % FP2D_PARTS;
    const int v_raw = (int)blockIdx.x * 4 + (lane >> 3);
    const int vi = min(v_raw, L.nviews - 1);
    const int det0 = ((int)blockIdx.y * FP2D_GROUPS + grp) * 16 + (lane & 7);
    float acc[2] = {0.0f, 0.0f};
    const int R = L.rays;
    for (int r = 0; r < R; ++r) {
        LineRay ray[2];
        float corr[2];
        bool cols[2];
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            const int det = min(det0 + 8 * j, L.ndet - 1);
            Ray2D q;
            if constexpr (KIND == B2T_GEOM_PAR2D) q = par_ray2d(L.par[vi], det, r, R);
            else q = fan_ray2d(L.fan[vi], fan_horizontal(L.fan[vi], det), L.W, L.H, det, r, R, L.out_scale);
            const int o = q.horizontal ? 1 : 0;
            ray[j].A = q.A;
            ray[j].B = q.B;
            ray[j].row = reinterpret_cast<unsigned long long>(o ? L.line0[1] : L.line0[0]) - SPLIT_BITS * 8ull;
            ray[j].pitch = o ? L.pitch[1] : L.pitch[0];
            ray[j].n0 = o ? L.W : L.H;
            ray[j].n = o ? L.H : L.W;
            corr[j] = q.corr;
            clip_line(ray[j]);
            cols[j] = q.horizontal;
        }
        // a warp whose rays choose different lines (views around 45 degrees)
        // of different counts
        const bool mixed = L.W != L.H && !__all_sync(0xffffffffu, cols[0] && cols[1]) &&
                           __any_sync(0xffffffffu, cols[0] || cols[1]);
        // a parallel view's rays are on the same line at every slice (a ray
        // that misses the image then reads the border of that line)
        if constexpr (KIND == B2T_GEOM_PAR2D) ray[0].pitch = ray[1].pitch = L.par[vi].vertical ? L.pitch[0] : L.pitch[1];
        float sum[2], tot[2] = {0.0f, 0.0f};
        sum_part<KIND == B2T_GEOM_PAR2D>(ray, mixed, part, sum);
        red[grp][part][lane] = sum[0];
        red[grp][part][lane + 32] = sum[1];
        __syncthreads();
        if (part == 0) {
#pragma unroll
            for (int p = 0; p < FP2D_PARTS; ++p) {
                tot[0] += red[grp][p][lane];
                tot[1] += red[grp][p][lane + 32];
            }
        }
        if (R > 1) __syncthreads();
#pragma unroll
        for (int j = 0; j < 2; ++j) acc[j] = KIND == B2T_GEOM_PAR2D ? acc[j] + tot[j] : fmaf(tot[j], corr[j], acc[j]);
    }
    if (part != 0 || v_raw >= L.nviews) return;
#pragma unroll
    for (int j = 0; j < 2; ++j) {
        const int det = det0 + 8 * j;
        if (det >= L.ndet) continue;
        if constexpr (KIND == B2T_GEOM_PAR2D) acc[j] = __fmul_rn(acc[j], L.par[vi].corr / (float)R);
        const long long i = (long long)(L.a0 + vi) * L.sino_pitch + det;
        if (L.res_w) L.sino[i] = (L.res_b[i] - acc[j]) * L.res_w[i];
        else L.sino[i] = L.accumulate ? L.sino[i] + acc[j] : acc[j];
    }
}

// ---------------------------------------------------------------------------
// backprojection
// ---------------------------------------------------------------------------

template <int CAP> struct BP2DLinesLaunch {
    const float *sino;  // row of the launch's first view
    long long sino_pitch;
    float *vol;
    long long vol_pitch;
    int W, H, ndet, fbp, nviews, accumulate;
    int win;  // pairs per staged row
    float out_scale;
    SirtUpdate2D upd;  // x set: SIRT's update in place of the backprojection
    BPView2D views[CAP];  // parallel: c[2] less 1/2
};

// A staged view: its constants and the shared-memory byte address of its
// pairs, less the first texel and the split's constant bits (pair k of the
// view at rb + 8 bits(k)); wide: its footprint exceeds the window.
struct alignas(16) BPRecord {
    float c[6];
    uint32_t rb;
    int wide;
};

__device__ __forceinline__ float2 lds_pair(uint32_t a)
{
    float2 v;
    asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(a));
    return v;
}

// Position of one pixel (the packed form below rounds alike).
template <int KIND> __device__ __forceinline__ float bp_position(const float *c, float x, float y)
{
    if constexpr (KIND == B2T_GEOM_PAR2D) {
        return fmaf(x, c[0], fmaf(-y, c[1], c[2]));
    } else {
        const float num = fmaf(x, c[1], fmaf(-y, c[2], c[0])), den = fmaf(x, c[4], fmaf(-y, c[5], c[3]));
        return fmaf(num, rcp_newton(den), -0.5f);
    }
}

// Positions and weights of the lane's pixels x, x + 8, ... (pairs in f32x2)
// of one row.
template <int KIND, int PX>
__device__ __forceinline__ void bp_positions(const float *c, const uint64_t (&x2)[PX / 2], float y, int fbp,
                                             uint64_t (&q)[PX / 2], float (&w)[PX])
{
    if constexpr (KIND == B2T_GEOM_PAR2D) {
        const float in = fmaf(-y, c[1], c[2]);
#pragma unroll
        for (int i = 0; i < PX / 2; ++i) {
            q[i] = fma2(x2[i], pk2(c[0], c[0]), pk2(in, in));
            w[2 * i] = w[2 * i + 1] = c[3];
        }
    } else {
        const float yw = -y;
        const float inn = fmaf(yw, c[2], c[0]), ind = fmaf(yw, c[5], c[3]);
#pragma unroll
        for (int i = 0; i < PX / 2; ++i) {
            const uint64_t num = fma2(x2[i], pk2(c[1], c[1]), pk2(inn, inn));
            // rcp_newton of both denominators
            const float2 den = upk2(fma2(x2[i], pk2(c[4], c[4]), pk2(ind, ind)));
            const uint64_t nden = fma2(x2[i], pk2(-c[4], -c[4]), pk2(-ind, -ind));
            const uint64_t r0 = pk2(rcp_approx(den.x), rcp_approx(den.y));
            const uint64_t fr = fma2(r0, fma2(nden, r0, pk2(1.0f, 1.0f)), r0);
            q[i] = fma2(num, fr, pk2(-0.5f, -0.5f));
            const float2 wu = upk2(fbp ? mul2(fr, fr) : fr);
            w[2 * i] = wu.x;
            w[2 * i + 1] = wu.y;
        }
    }
}

// A warp owns 8 PX x 4 pixels: lane (x & 7, y), PX pixels 8 apart along x,
// so that one load of a warp covers an 8 x 4 patch, whose samples lie within
// about nine pairs.  A CTA has 8 / WS such warps stacked along y, each with
// its BP2D_PARTS / WS ranges of views over WS warps.  The CTA stages, ROWS
// views at a time (ROWS / WS of each of the WS ranges), the window of pairs
// that its pixels sample, zeros outside the detector, into one of two
// buffers.  Parallel views are bound by the shared-memory data pipe (78 %, issue
// 72 %), fan views by instruction issue (69 %, data pipe 56 %): 1024^2 x 1440 takes
// 0.62 ms parallel and 0.94 ms fan; reading bordered pairs of the sinogram
// through L1 instead took 0.84 and 1.56 ms.
template <int KIND, int PX, int WS, int ROWS, int CAP>
__global__ void __launch_bounds__(LINES_THREADS) bp2d_lines_kernel(const __grid_constant__ BP2DLinesLaunch<CAP> L)
{
    constexpr int WY = LINES_WARPS / WS, NP = BP2D_PARTS / WS, NV = ROWS / WS;
    extern __shared__ __align__(16) unsigned char smraw[];
    __shared__ int2 window[ROWS];  // first texel and pairs of a staged view (0: none)
    BPRecord *rec = reinterpret_cast<BPRecord *>(smraw);                           // [2][ROWS]
    float2 *rows = reinterpret_cast<float2 *>(smraw + 2 * ROWS * sizeof(BPRecord));  // [2][ROWS][win]
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int X0 = blockIdx.x * 8 * PX, Y0 = blockIdx.y * 4 * WY;
    const int group = warp % WS;
    const int win = L.win;

    const int X = X0 + (lane & 7), Y = Y0 + 4 * (warp / WS) + (lane >> 3);
    uint64_t x2[PX / 2];
#pragma unroll
    for (int i = 0; i < PX / 2; ++i)
        x2[i] = pk2((float)(X + 16 * i) - 0.5f * (float)L.W + 0.5f, (float)(X + 16 * i + 8) - 0.5f * (float)L.W + 0.5f);
    const float y = (float)Y - 0.5f * (float)L.H + 0.5f;
    const float cx0 = (float)X0 - 0.5f * (float)L.W + 0.5f, cx1 = (float)(X0 + 8 * PX - 1) - 0.5f * (float)L.W + 0.5f;
    const float cy0 = (float)Y0 - 0.5f * (float)L.H + 0.5f, cy1 = (float)(Y0 + 4 * WY - 1) - 0.5f * (float)L.H + 0.5f;

    const uint64_t M2 = pk2(SPLIT_M, SPLIT_M), nM2 = pk2(-SPLIT_M, -SPLIT_M);
    float tot[PX], sum[PX];
#pragma unroll
    for (int i = 0; i < PX; ++i) tot[i] = 0.0f;
    int buf = 0;
#pragma unroll 1
    for (int p = 0; p < NP; ++p) {
#pragma unroll
        for (int i = 0; i < PX; ++i) sum[i] = 0.0f;
        const int len = (L.nviews + BP2D_PARTS - 1) / BP2D_PARTS;  // longest range
#pragma unroll 1
        for (int c0 = 0; c0 < len; c0 += NV, buf ^= 1) {
            // a lane per view: its record and the texels that the corners of
            // the CTA's pixels bound (a view's map is monotone along rows
            // and columns)
            if (threadIdx.x < ROWS) {
                const int j = threadIdx.x;
                const int part = (j / NV) * NP + p;
                const int v = part_begin(part, L.nviews, BP2D_PARTS) + c0 + j % NV;
                int2 w = make_int2(0, 0);
                if (v < part_begin(part + 1, L.nviews, BP2D_PARTS)) {
                    const BPView2D &C = L.views[v];
                    int kmin = INT_MAX, kmax = INT_MIN;
                    bool ok = true;
#pragma unroll
                    for (int c = 0; c < 4; ++c) {
                        const float cx = (c & 1) ? cx1 : cx0, cy = (c & 2) ? cy1 : cy0;
                        const float q = bp_position<KIND>(C.c, cx, cy);
                        if constexpr (KIND != B2T_GEOM_PAR2D) ok = ok && fmaf(cx, C.c[4], fmaf(-cy, C.c[5], C.c[3])) > 1e-6f;
                        ok = ok && fabsf(q) < 1.0e6f;
                        const int k = floor_texel(q);
                        kmin = min(kmin, k - 1);
                        kmax = max(kmax, k + 1);
                    }
                    ok = ok && kmax - kmin < win;
                    BPRecord r;
#pragma unroll
                    for (int i = 0; i < 6; ++i) r.c[i] = C.c[i];
                    r.rb = smem_u32(rows + (size_t)(buf * ROWS + j) * win) - ((uint32_t)kmin + SPLIT_BITS) * 8u;
                    r.wide = !ok;
                    rec[buf * ROWS + j] = r;
                    if (ok) w = make_int2(kmin, kmax - kmin + 1);
                }
                window[j] = w;
            }
            __syncthreads();
            // a warp per view, four views' loads in flight
#pragma unroll 1
            for (int j0 = warp; j0 < ROWS; j0 += 4 * LINES_WARPS) {
                float a[4][2], b[4][2];
                int cnt[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const int j = j0 + i * LINES_WARPS;
                    const int2 w = j < ROWS ? window[j] : make_int2(0, 0);
                    cnt[i] = w.y;
                    const int v = part_begin((j / NV) * NP + p, L.nviews, BP2D_PARTS) + c0 + j % NV;
                    const float *row = L.sino + (long long)v * L.sino_pitch;
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        const int e = lane + 32 * h, t = w.x + e;
                        a[i][h] = (e < w.y && (unsigned)t < (unsigned)L.ndet) ? __ldg(row + t) : 0.0f;
                        b[i][h] = (e < w.y && (unsigned)(t + 1) < (unsigned)L.ndet) ? __ldg(row + t + 1) : 0.0f;
                    }
                }
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const int j = j0 + i * LINES_WARPS;
                    float2 *dst = rows + (size_t)(buf * ROWS + j) * win;
#pragma unroll
                    for (int h = 0; h < 2; ++h)
                        if (lane + 32 * h < cnt[i]) dst[lane + 32 * h] = make_float2(a[i][h], b[i][h] - a[i][h]);
                    if (cnt[i] > 64) {  // (a detector finer than the pixels)
                        const int v = part_begin((j / NV) * NP + p, L.nviews, BP2D_PARTS) + c0 + j % NV;
                        const float *row = L.sino + (long long)v * L.sino_pitch;
                        for (int e = lane + 64; e < cnt[i]; e += 32) {
                            const int t = window[j].x + e;
                            const float fa = (unsigned)t < (unsigned)L.ndet ? __ldg(row + t) : 0.0f;
                            const float fb = (unsigned)(t + 1) < (unsigned)L.ndet ? __ldg(row + t + 1) : 0.0f;
                            dst[e] = make_float2(fa, fb - fa);
                        }
                    }
                }
            }
            __syncthreads();
            const int part = group * NP + p;
            const int v0 = part_begin(part, L.nviews, BP2D_PARTS) + c0;
            const int nv = min(NV, part_begin(part + 1, L.nviews, BP2D_PARTS) - v0);
            const BPRecord *rc = rec + buf * ROWS + group * NV;
#pragma unroll 2
            for (int j = 0; j < nv; ++j) {
                const float4 ra = *reinterpret_cast<const float4 *>(&rc[j]);
                const float4 rd = *reinterpret_cast<const float4 *>(&rc[j].c[4]);
                const float c[6] = {ra.x, ra.y, ra.z, ra.w, rd.x, rd.y};
                const uint32_t rb = __float_as_uint(rd.z);
                uint64_t q[PX / 2];
                float w[PX];
                bp_positions<KIND, PX>(c, x2, y, L.fbp, q, w);
                if (__float_as_int(rd.w) == 0) {
                    float f[PX];
                    float2 val[PX];
#pragma unroll
                    for (int i = 0; i < PX / 2; ++i) {
                        const uint64_t t = add2_rd(q[i], M2);
                        const float2 fu = upk2(sub2(q[i], add2(t, nM2))), tb = upk2(t);
                        f[2 * i] = fu.x;
                        f[2 * i + 1] = fu.y;
                        val[2 * i] = lds_pair((uint32_t)__float_as_int(tb.x) * 8u + rb);
                        val[2 * i + 1] = lds_pair((uint32_t)__float_as_int(tb.y) * 8u + rb);
                    }
#pragma unroll
                    for (int i = 0; i < PX; ++i) sum[i] = fmaf(fmaf(f[i], val[i].y, val[i].x), w[i], sum[i]);
                } else {
                    const float *row = L.sino + (long long)(v0 + j) * L.sino_pitch;
#pragma unroll
                    for (int i = 0; i < PX; ++i) {
                        const float2 qu = upk2(q[i / 2]);
                        sum[i] = fmaf(lerp_line(row, 1, L.ndet, (i & 1) ? qu.y : qu.x), w[i], sum[i]);
                    }
                }
            }
        }
        if constexpr (WS == 1) {
#pragma unroll
            for (int i = 0; i < PX; ++i) tot[i] += sum[i];
        } else {
            // (the partial sums of a warp's ranges wait in shared memory)
            float *red = reinterpret_cast<float *>(rows + (size_t)2 * ROWS * win);
#pragma unroll
            for (int i = 0; i < PX; ++i) red[((warp / WS) * BP2D_PARTS + group * NP + p) * 32 * PX + 32 * i + lane] = sum[i];
        }
    }
    auto store = [&](int px, int py, float t) {
        if (px >= L.W || py >= L.H) return;
        const float r = __fmul_rn(t, L.out_scale);
        const long long i = (long long)py * L.vol_pitch + px;
        if (L.upd.x) {
            const SirtUpdate2D &U = L.upd;
            U.x[i] = sirt_clamp(fmaf(U.w[i], r, U.x[i]), U.use_min, U.min_value, U.use_max, U.max_value,
                                U.min_mask ? U.min_mask + i : nullptr, U.max_mask ? U.max_mask + i : nullptr);
            return;
        }
        float *o = L.vol + i;
        *o = L.accumulate ? *o + r : r;
    };
    if constexpr (WS > 1) {
        float *red = reinterpret_cast<float *>(rows + (size_t)2 * ROWS * win);
        __syncthreads();
        for (int e = threadIdx.x; e < WY * 32 * PX; e += LINES_THREADS) {
            const int wy = e / (32 * PX), k = e % (32 * PX);
            float t = 0.0f;
#pragma unroll
            for (int p = 0; p < BP2D_PARTS; ++p) t += red[(wy * BP2D_PARTS + p) * 32 * PX + k];
            store(X0 + (k & 7) + 8 * (k >> 5), Y0 + 4 * wy + ((k & 31) >> 3), t);
        }
    } else {
#pragma unroll
        for (int i = 0; i < PX; ++i) store(X + 8 * i, Y, tot[i]);
    }
}

b2t_status build_lines(const float *src, long long src_pitch, const LineSet *sets, int nsets, cudaStream_t s)
{
    BuildLines B;
    B.src = src;
    B.src_pitch = src_pitch;
    B.nsets = nsets;
    int kt = 0, lt = 0;
    for (int i = 0; i < nsets; ++i) {
        B.set[i] = sets[i];
        kt = std::max(kt, (sets[i].n + 2 * LINE_BORDER + 31) / 32);
        lt = std::max(lt, (sets[i].lines + 31) / 32);
    }
    if (lt > 65535) return fail(B2T_ERR_NO_MEMORY, "2D line copy: too many lines");
    build_lines_kernel<<<dim3((unsigned)kt, (unsigned)lt, (unsigned)nsets), LINES_THREADS, 0, s>>>(B);
    count_launches(1);
    B2T_CUDA_TRY(cudaGetLastError(), "2D line copy launch");
    return B2T_OK;
}

// Bytes of `lines` lines of n texels, added to total.
size_t lines_bytes(size_t lines, size_t n, size_t &total)
{
    const size_t b = lines * (n + 2 * LINE_BORDER) * sizeof(float2);
    total += b;
    return b;
}

template <int KIND, int CAP>
cudaError_t launch_fp(const FP2DLinesLaunch<CAP> &L, cudaStream_t s)
{
    constexpr int D = 16 * FP2D_GROUPS;
    fp2d_lines_kernel<KIND, CAP><<<dim3((L.nviews + 3) / 4, (L.ndet + D - 1) / D), LINES_THREADS, 0, s>>>(L);
    return cudaGetLastError();
}

// Texels that a diagonal step of one pixel along each axis covers in view C,
// at most: exact for a parallel view; for a fan view at the corner nearest to
// the source.
float bp_step(int kind, const BPView2D &C, const b2t_dims2d &d)
{
    if (kind == B2T_GEOM_PAR2D) return std::fabs(C.c[0]) + std::fabs(C.c[1]);
    float step = 0.0f;
    for (int k = 0; k < 4; ++k) {
        const float x = ((k & 1) ? 0.5f : -0.5f) * (float)d.vol_width, y = ((k & 2) ? 0.5f : -0.5f) * (float)d.vol_height;
        const float den = C.c[3] + x * C.c[4] + y * C.c[5];
        const float q = (C.c[0] + x * C.c[1] + y * C.c[2]) / den;
        step = std::max(step, (std::fabs(C.c[1] - q * C.c[4]) + std::fabs(C.c[2] - q * C.c[5])) / std::fabs(den));
    }
    return step;
}

template <int KIND, int PX, int WS, int ROWS, int CAP>
cudaError_t launch_bp_shape(BP2DLinesLaunch<CAP> &L, float step, cudaStream_t s)
{
    constexpr int TX = 8 * PX, WY = LINES_WARPS / WS, TY = 4 * WY;
    // the widest footprint of a tile, with a texel on both sides and one for
    // rounding, up to LINES_MAX_WIN pairs (wider ones are read from the sinogram)
    const float span = step * (float)(std::max(TX, TY)) + 4.0f;
    L.win = span < (float)LINES_MAX_WIN ? ((int)span + 2) & ~1 : LINES_MAX_WIN;
    auto bytes = [](int win) {
        return 2 * ROWS * (sizeof(BPRecord) + (size_t)win * sizeof(float2)) +
               (WS > 1 ? (size_t)WY * BP2D_PARTS * 32 * PX * sizeof(float) : 0);
    };
    const size_t smem = bytes(L.win);
    auto kern = bp2d_lines_kernel<KIND, PX, WS, ROWS, CAP>;
    // the kernel's own maximum in every call: the limit belongs to the kernel,
    // and a call of another thread may set it between here and the launch
    const cudaError_t e =
        cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes(LINES_MAX_WIN));
    if (e != cudaSuccess) return e;
    kern<<<dim3((L.W + TX - 1) / TX, (L.H + TY - 1) / TY), LINES_THREADS, smem, s>>>(L);
    return cudaGetLastError();
}

// Warps over the ranges of a pixel's views as long as the launch stays within
// about 24 warps per SM: at 256^2 x 180 parallel, 1 / 2 / 4 / 8 warps per
// 32 x 4 pixels (512 tiles) take 25.5 / 19.6 / 16.2 / 20.6 us, at 128^2 x 180
// 25.2 / 19.2 / 13.0 / 9.5 us, at 512^2 x 720 109 / 119 / 158 / 227 us.
constexpr long long LINES_BP_WARPS = 3600;

template <int KIND, int CAP>
cudaError_t launch_bp(BP2DLinesLaunch<CAP> &L, float step, cudaStream_t s)
{
    const long long tiles = (long long)((L.W + 31) / 32) * ((L.H + 3) / 4);
    if (8 * tiles <= LINES_BP_WARPS) return launch_bp_shape<KIND, 4, 8, 64>(L, step, s);
    if (4 * tiles <= LINES_BP_WARPS) return launch_bp_shape<KIND, 4, 4, 64>(L, step, s);
    if (2 * tiles <= LINES_BP_WARPS) return launch_bp_shape<KIND, 4, 2, 32>(L, step, s);
    return launch_bp_shape<KIND, 4, 1, 32>(L, step, s);
}

// Views that a small launch's parameters hold (6 KB instead of 24 KB, which
// the driver copies at every launch).
constexpr int LINES_SMALL_VIEWS = 256;

// Which lines the rays of the scan march over: of the image's rows, of its
// columns.  A parallel view's rays share the choice; a fan view's rays make it
// one by one (fan_ray2d), from |x| and |y| of source to detector, in 32 bits:
// all alike when both ends of the detector choose so, on the same side and by
// more than rounding could change.
struct LineNeed {
    bool rows = false, cols = false;
};
LineNeed lines_needed(const b2t_geom2d *g)
{
    LineNeed need;
    for (uint32_t i = 0; i < g->dims.angles && !(need.rows && need.cols); ++i) {
        const b2t_view2d &V = g->views[i];
        if (g->kind == B2T_GEOM_PAR2D) {
            (std::fabs(V.src[0]) <= std::fabs(V.src[1]) ? need.rows : need.cols) = true;
            continue;
        }
        const double n = (double)g->dims.dets - 1.0;
        double d[2][2], margin = 1.0;  // [end][axis]
        for (int k = 0; k < 2; ++k) {
            for (int e = 0; e < 2; ++e) d[e][k] = e * n * V.det_u[k] + V.det_s[k] + 0.5 - V.src[k];
            margin += std::fabs((double)V.src[k]) + std::fabs((double)V.det_s[k]) + n * std::fabs((double)V.det_u[k]);
        }
        margin *= 1e-5;
        auto all = [&](int k) {  // every ray is longer along axis k
            return d[0][k] * d[1][k] > 0.0 && std::fabs(d[0][k]) - std::fabs(d[0][1 - k]) > margin &&
                   std::fabs(d[1][k]) - std::fabs(d[1][1 - k]) > margin;
        };
        if (!all(0)) need.rows = true;
        if (!all(1)) need.cols = true;
    }
    return need;
}

template <int CAP>
b2t_status fp_run(const b2t_geom2d *g, uint32_t det_supersample, const float *vol, size_t vol_pitch, float *sino,
                  size_t sino_pitch, int32_t mode, const float *res_b, const float *res_w, cudaStream_t s)
{
    const b2t_dims2d &d = g->dims;
    const LineNeed need = lines_needed(g);
    const bool rows = need.rows, cols = need.cols;
    size_t total = 0;
    const size_t row_bytes = rows ? lines_bytes(d.vol_height, d.vol_width, total) : 0;
    if (cols) lines_bytes(d.vol_width, d.vol_height, total);
    Scratch sc;
    B2T_TRY(sc.alloc(total, s, "b2t_fp2d scratch (line copy)"));
    const std::unique_ptr<FP2DLinesLaunch<CAP>> keep(new FP2DLinesLaunch<CAP>);
    FP2DLinesLaunch<CAP> &L = *keep;
    L.res_b = res_b;
    L.res_w = res_w;
    L.pitch[0] = (d.vol_width + 2 * LINE_BORDER) * (uint32_t)sizeof(float2);
    L.pitch[1] = (d.vol_height + 2 * LINE_BORDER) * (uint32_t)sizeof(float2);
    L.line0[0] = sc.as<char>() + LINE_BORDER * sizeof(float2);
    L.line0[1] = L.line0[0] + row_bytes;
    LineSet sets[2];
    int nsets = 0;
    if (rows)
        sets[nsets++] = {sc.as<float2>(), (int)d.vol_height, (int)d.vol_width, (int)d.vol_width + 2 * LINE_BORDER, 0};
    if (cols)
        sets[nsets++] = {reinterpret_cast<float2 *>(sc.as<char>() + row_bytes), (int)d.vol_width, (int)d.vol_height,
                         (int)d.vol_height + 2 * LINE_BORDER, 1};
    B2T_TRY(build_lines(vol, (long long)vol_pitch, sets, nsets, s));
    L.sino = sino;
    L.sino_pitch = (long long)sino_pitch;
    L.W = d.vol_width; L.H = d.vol_height; L.ndet = d.dets;
    L.rays = det_supersample;
    L.accumulate = (mode == B2T_MODE_ADD) ? 1 : 0;
    L.out_scale = g->output_scale;
    for (uint32_t c0 = 0; c0 < d.angles; c0 += CAP) {
        const uint32_t cn = std::min(d.angles - c0, (uint32_t)CAP);
        L.a0 = (int)c0;
        L.nviews = (int)cn;
        for (uint32_t i = 0; i < cn; ++i) {
            if (g->kind == B2T_GEOM_PAR2D) par_fp_view(g->views[c0 + i], d, g->output_scale, L.par[i]);
            else L.fan[i] = g->views[c0 + i];
        }
        const cudaError_t e = g->kind == B2T_GEOM_PAR2D ? launch_fp<B2T_GEOM_PAR2D, CAP>(L, s) : launch_fp<B2T_GEOM_FAN2D, CAP>(L, s);
        count_launches(1);
        B2T_CUDA_TRY(e, "fp2d launch");
    }
    return B2T_OK;
}

template <int CAP>
b2t_status bp_run(const b2t_geom2d *g, int32_t fbp_weight, const float *sino, size_t sino_pitch, float *vol,
                  size_t vol_pitch, int32_t mode, const SirtUpdate2D *update, cudaStream_t s)
{
    const b2t_dims2d &d = g->dims;
    const std::unique_ptr<BP2DLinesLaunch<CAP>> keep(new BP2DLinesLaunch<CAP>);
    BP2DLinesLaunch<CAP> &L = *keep;
    L.upd = update ? *update : SirtUpdate2D{};
    L.sino_pitch = (long long)sino_pitch;
    L.vol = vol;
    L.vol_pitch = (long long)vol_pitch;
    L.W = d.vol_width; L.H = d.vol_height; L.ndet = d.dets;
    L.fbp = fbp_weight ? 1 : 0;
    L.out_scale = g->output_scale;
    for (uint32_t c0 = 0; c0 < d.angles; c0 += CAP) {
        const uint32_t cn = std::min(d.angles - c0, (uint32_t)CAP);
        L.sino = sino + (size_t)c0 * sino_pitch;
        L.nviews = (int)cn;
        float step = 0.0f;
        L.accumulate = (c0 > 0 || mode == B2T_MODE_ADD) ? 1 : 0;
        for (uint32_t i = 0; i < cn; ++i) {
            bp2d_view(g->kind, L.fbp, g->views[c0 + i], L.views[i]);
            if (g->kind == B2T_GEOM_PAR2D) L.views[i].c[2] -= 0.5f;
            step = std::max(step, bp_step(g->kind, L.views[i], d));
        }
        const cudaError_t e =
            g->kind == B2T_GEOM_PAR2D ? launch_bp<B2T_GEOM_PAR2D, CAP>(L, step, s) : launch_bp<B2T_GEOM_FAN2D, CAP>(L, step, s);
        count_launches(1);
        B2T_CUDA_TRY(e, "bp2d launch");
    }
    return B2T_OK;
}

}  // namespace

b2t_status fp2d_lines(const b2t_geom2d *g, uint32_t det_supersample, const float *vol, size_t vol_pitch, float *sino,
                      size_t sino_pitch, int32_t mode, const float *res_b, const float *res_w, cudaStream_t s)
{
    auto run = g->dims.angles <= LINES_SMALL_VIEWS ? fp_run<LINES_SMALL_VIEWS> : fp_run<FP2D_MAX_VIEWS>;
    return run(g, det_supersample, vol, vol_pitch, sino, sino_pitch, mode, res_b, res_w, s);
}

// Calls that the copy into lines, a launch and an allocation, costs more than it
// gives.  Lines and direct kernel, whole calls: 64^2 and up to 64 views 14.3 to 15.7
// and 12.3 to 14.6 us; 96^2 parallel, up to 16 views, 15.4 to 16.9 and 14.2 to 15.6 us.
// One or two fan views whose rays march over rows, where the direct kernel's
// loads are coalesced: 96^2 and 128^2 14.7 to 15.2 and 12.1 to 13.4 us, 4096^2
// (the copy is 200 MB) 391 to 395 and 283 to 300 us; between them the lines win (256^2
// 21 and 23 us, 1024^2 51 and 78 us), as they do where rays march over columns (4096^2
// 398 and 1055 us).
bool fp2d_few_rays(const b2t_geom2d *g)
{
    const b2t_dims2d &d = g->dims;
    const uint32_t n = std::max(d.vol_width, d.vol_height);
    if (n <= 64 && d.angles <= 64) return true;
    if (g->kind == B2T_GEOM_PAR2D) return n <= 96 && d.angles <= 16;
    return d.angles <= 2 && (n <= 128 || n >= 4096) && !lines_needed(g).cols;
}

// A warp that runs all BP2D_PARTS ranges itself goes through the staging of
// each of them, and with a view or less a range that is all it does.  Lines and
// direct kernel (parallel) at 1024^2: 1 view 25.3 and 14.2 us, 8 views 29.4 and 19.5
// us, 10 views (which the direct kernel sums in parts as well) 31.4 and 31.5 us; at
// 4096^2 333 and 54, 393 and 240, 403 and 419 us; fan 435 and 262 us (8 views), 450 and
// 478 us (10).  Images of less than LINES_BP_WARPS tiles leave room on the GPU and
// wait for the staging longer: 512^2 fan, 10 views 15.1 and 12.8 us, 12 15.5 and 14.7
// us, 16 17.0 and 19.0 us.  With the ranges split over warps the calls take the
// same time.
bool bp2d_few_views(const b2t_dims2d &d)
{
    const long long tiles = (long long)((d.vol_width + 31) / 32) * ((d.vol_height + 3) / 4);
    if (2 * tiles <= LINES_BP_WARPS) return false;
    return d.angles <= (uint32_t)(tiles <= LINES_BP_WARPS ? 12 : BP2D_PARTS);
}

b2t_status bp2d_lines(const b2t_geom2d *g, int32_t fbp_weight, const float *sino, size_t sino_pitch, float *vol,
                      size_t vol_pitch, int32_t mode, const SirtUpdate2D *update, cudaStream_t s)
{
    auto run = g->dims.angles <= LINES_SMALL_VIEWS ? bp_run<LINES_SMALL_VIEWS> : bp_run<BP2D_MAX_VIEWS>;
    return run(g, fbp_weight, sino, sino_pitch, vol, vol_pitch, mode, update, s);
}

}  // namespace b2t
