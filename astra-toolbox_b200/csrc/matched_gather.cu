// Exact adjoint of the forward projector, gathered per voxel (projection
// kernel "matched_bp") for the views of the slab forward projector: views that
// march along x or y and whose detector v axis has no component along the
// marching axis or the in-plane axis (every circular orbit, parallel or cone).
//
// The reference scatters each ray with atomic adds (its only matched
// backprojector, cuda/3d/cone_cyl.cu:309-470); matched.cu does the same for
// every view.  For the views here the sum can be turned round.  At slice s the
// samples of detector column u share the in-plane position q1(u, s), and their
// z positions are equally spaced, q2 = P(u, s) + v Q(u, s).  With
// hat(t) = max(0, 1 - |t|),
//
//   vol(s, k1, z) += sum_u hat(q1(u, s) - k1) c_u(z),
//   c_u(z) = sum_v hat(q2(u, v, s) - z) y(u, v) w(u, v),
//
// where the inner sum has at most ceil(2 / Q) terms and c_u serves the two
// texels k1 on either side of q1.
//
//   matched_prep_kernel writes the projections times their ray factors w in
//   FP32 as rows along v (lanes run along z, so their samples lie side by
//   side) and, per view and column, the coefficients of q1, P and Q and whether
//   the column is other than zero (beside an object it mostly is not).
//
//   matched_gather_kernel: a CTA owns T x T x 64 voxels in shared memory (T 8
//   or 16) and runs over all views.  A warp owns one slice (x for x-major views,
//   y for y-major ones), each lane two z.  It walks the columns u that meet its
//   T texels in the order of rising q1 (their data prepared 32 at a time, one
//   column a lane, and read back from shared memory), keeping the sums of texels k1 and k1 + 1
//   in registers until q1 leaves k1: every branch is uniform over the warp, and
//   no two warps share an accumulator, so there are no atomics and the result
//   does not depend on the order of the blocks.
//
// Bound by instruction issue (0.75 a cycle and scheduler; a column of 64 voxels
// takes about 75 instructions, a third of them for its up to four terms).
// Whole calls on dense projections, scattered and gathered: 192^3 x 240 views,
// 288^2 detector 5.36 and 4.59 ms, 256^3 x 360 19.0 and 15.6 ms.  Which calls are
// gathered is decided by the volume and the scan (matched_gather_eligible) and, on
// the device, by how many rays hold a value (matched.cu).
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cfloat>
#include <cmath>
#include <vector>

#include "b2t_internal.h"
#include "f32x2.cuh"
#include "proj3d.h"

namespace b2t {

namespace {

constexpr int MG_Z = 64;            // voxels of a tile along z, two a lane
constexpr int MG_ZP = MG_Z + 1;     // row pitch of a tile (the final reads run along x)
constexpr int MG_PAD = 8;           // zeros after each row of weighted projections: the most terms of c_u(z)
constexpr int MG_MAX_VIEWS = 448;   // views per launch of the preparation (parameter limit)
constexpr float MG_M = 12582912.0f;  // 1.5 * 2^23
constexpr int MG_BITS = 0x4B400000;  // bits of MG_M

// Column u of a view, with t = s - the middle slice: q1 (plus one half) =
// A t + B, P = p0 + p1 t, Q = q0 + q1 t.  From the middle slice on, and worked
// out in FP64 before they are rounded, the coefficients leave positions closer
// to the 64-bit ones than the forward projector's own: the result is 6.1e-6
// from FP64 at 100^3 (cone), 8.8e-6 scattered.
struct MGColumn {
    float A, B, p0, p1, q0, q1, pad0, pad1;
};
// A view's in-plane coefficients (of [1, u']), its denominator made positive.
struct MGRecord {
    float e0, e1, m0, m1, n0, n1, mz, nz;
};

struct MGPrep {
    const void *proj;
    long long proj_pitch;
    float *rows;        // [view][u][pitch]
    MGColumn *cols;     // [view][u]
    MGRecord *recs;     // [view]
    int *live;          // [view][u]: 1 where the column holds a value other than zero (cleared before)
    int *bad;           // [view]: 1 where some weighted value is infinite or NaN (cleared before)
    int nu, nv, na, pitch, half;
    int nviews, first;  // views of this launch, index of its first one in the gather's order
    const int *run;     // 0 there: the call is scattered (null: gathered)
    float f1[2], f2[2], mul[2];
    float mid[2];       // middle slice of either direction
    signed char dir[MG_MAX_VIEWS];
    FPView views[MG_MAX_VIEWS];
};

struct MGLaunch {
    const float *rows;
    const MGColumn *cols;
    const MGRecord *recs;
    const int *live, *bad;
    int nu, nv, pitch, half;
    int nx, ny, nz;
    int nx_views, nviews;  // x-major views come first
    int nzb, splits;
    const int *run;        // as above
    void *out;             // volume [z][y][x], or FP32 partial sums [split][z][y][x]
    long long out_pitch;
    int accumulate;
};

template <typename T> __device__ __forceinline__ float mg_load(T v) { return (float)v; }
template <typename T> __device__ __forceinline__ T mg_store(float v);
template <> __device__ __forceinline__ float mg_store<float>(float v) { return v; }
template <> __device__ __forceinline__ __half mg_store<__half>(float v) { return __float2half_rn(v); }
template <> __device__ __forceinline__ __nv_bfloat16 mg_store<__nv_bfloat16>(float v) { return __float2bfloat16_rn(v); }

// Tiles of 32 columns x 32 rows of one view, transposed through shared memory; a
// block takes several (a block that has nothing to do, in a call that is
// scattered, takes as long to launch as one that has).
constexpr int PREP_TILES = 6;
template <typename T> __global__ void __launch_bounds__(256) matched_prep_kernel(const __grid_constant__ MGPrep L)
{
    __shared__ float tile[32][33];
    if (L.run && *L.run == 0) return;
    const int i = blockIdx.z;
    const FPView &V = L.views[i];
    const int dir = L.dir[i];
    const long long gi = L.first + i;
    const int u0 = blockIdx.x * 32;
    const int u = u0 + threadIdx.x;
    const float uu = (float)u + 0.5f - 0.5f * (float)L.nu;
    const float den = fmaf(uu, V.e[1], V.e[0]);
    const float inv = 1.0f / den;
    const float A1 = fmaf(uu, V.m1[1], V.m1[0]) * inv;
    for (int v0 = blockIdx.y * 32; v0 < L.pitch; v0 += gridDim.y * 32) {
        for (int r = threadIdx.y; r < 32; r += 8) {
            const int v = v0 + r;
            float y = 0.0f;
            if (u < L.nu && v < L.nv) {
                const float vv = (float)v + 0.5f - 0.5f * (float)L.nv;
                const float A2 = fmaf(vv, V.m2[2], fmaf(uu, V.m2[1], V.m2[0])) * inv;
                const float sc = sqrtf(fmaf(A1 * A1, L.f1[dir], fmaf(A2 * A2, L.f2[dir], 1.0f))) * L.mul[dir];
                y = mg_load(static_cast<const T *>(L.proj)[((size_t)v * L.na + V.a) * L.proj_pitch + u]) * sc;
            }
            tile[r][threadIdx.x] = y;
        }
        __syncthreads();
        for (int r = threadIdx.y; r < 32; r += 8) {
            const int v = v0 + threadIdx.x;
            const float y = tile[threadIdx.x][r];
            const bool any = __any_sync(0xffffffffu, y != 0.0f);
            const bool off = __any_sync(0xffffffffu, !(fabsf(y) <= FLT_MAX));
            if (u0 + r >= L.nu) continue;
            if (v < L.pitch) L.rows[(gi * L.nu + u0 + r) * L.pitch + v] = y;
            if (any && threadIdx.x == 0) L.live[gi * L.nu + u0 + r] = 1;
            if (off && threadIdx.x == 0) L.bad[gi] = 1;
        }
        __syncthreads();
    }
    if (blockIdx.y == 0 && threadIdx.y == 0 && u < L.nu) {
        // rows are counted from `half`, near the detector's centre
        const double du = u + 0.5 - 0.5 * L.nu, dvc = L.half + 0.5 - 0.5 * L.nv, mid = L.mid[dir];
        const double di = 1.0 / (V.e[0] + du * V.e[1]);
        auto along = [&](double m, double n) { return (n + m * mid) * di; };
        const double m1 = V.m1[0] + du * V.m1[1], n1 = V.n1[0] + du * V.n1[1];
        const double m2 = V.m2[0] + du * V.m2[1] + dvc * V.m2[2], n2 = V.n2[0] + du * V.n2[1] + dvc * V.n2[2];
        MGColumn c;
        c.A = (float)(m1 * di);
        c.B = (float)(along(m1, n1) + 0.5);
        c.p0 = (float)(along(m2, n2) + 0.5);
        c.p1 = (float)(m2 * di);
        c.q0 = (float)along(V.m2[2], V.n2[2]);
        c.q1 = (float)(V.m2[2] * di);
        c.pad0 = c.pad1 = 0.0f;
        L.cols[gi * L.nu + u] = c;
        if (u == 0) {
            const float sg = den < 0.0f ? -1.0f : 1.0f;
            MGRecord r;
            r.e0 = sg * V.e[0];
            r.e1 = sg * V.e[1];
            r.m0 = sg * V.m1[0];
            r.m1 = sg * V.m1[1];
            r.n0 = sg * V.n1[0];
            r.n1 = sg * V.n1[1];
            r.mz = sg * V.m2[2];
            r.nz = sg * V.n2[2];
            L.recs[gi] = r;
        }
    }
}

__device__ __forceinline__ uint64_t add2_rp(uint64_t a, uint64_t b)
{
    uint64_t d;
    asm("add.rp.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}

// A column's data for a warp's slice: the fraction f1 of q1, P, Q and -1 / Q,
// each twice (both halves of a packed operand).
struct MGStep {
    float4 fP, Qn;
};

// What a warp walks: n columns from `us` on, in steps of du.
struct MGWalk {
    const MGColumn *cols;  // the view's columns
    const float *rows;     // the view's weighted rows
    const int *live;       // the view's columns with any value in them
    int n, us, du, pitch, half;
    float t, vlo, vhi;  // slice from the middle one; the row indices (from `half`) that are clamped to
    uint64_t nz2;       // minus the lane's two z
    int ka;             // the tile's first texel
    float *acc;         // its sums, texel stride `stride`
    int stride;
    MGStep *steps;      // the warp's 32 columns
    int *texels;        // and their base texels k1
};

// NT: terms of c_u(z), at least 2 / Q for every column of the walk.  The NT rows
// read may lie outside the support of hat, where its zero takes them out;
// GUARD: some value of the view is infinite or NaN, and those rows are left
// out by a comparison.
template <int T, int NT, bool GUARD> __device__ __forceinline__ void mg_walk(const MGWalk &W, int lane)
{
    const uint64_t M2 = pk2(MG_M, MG_M), nM2 = pk2(-MG_M, -MG_M), one2 = pk2(1.0f, 1.0f);
    const float tlo = MG_M + W.vlo, thi = MG_M + W.vhi;
    int cur = W.ka - 2;
    uint64_t acc0 = pk2(0.0f, 0.0f), acc1 = acc0;
    auto flush = [&](int k, uint64_t a) {
        if (k < W.ka || k >= W.ka + T) return;
        float *p = W.acc + (k - W.ka) * W.stride;
        const float2 v = upk2(a);
        p[0] += v.x;
        p[32] += v.y;
    };
    for (int b = 0; b < W.n; b += 32) {
        // lane j: column b + j of the walk
        const int u = W.us + W.du * min(b + lane, W.n - 1);
        const float4 c0 = __ldg(reinterpret_cast<const float4 *>(W.cols + u));
        const float2 c1 = __ldg(reinterpret_cast<const float2 *>(W.cols + u) + 2);
        const float q = fmaf(c0.x, W.t, c0.y);
        const float tq = __fadd_rd(q, MG_M);
        const int k1 = __float_as_int(tq) - MG_BITS;
        const float f1 = q - (tq - MG_M);
        const float P = fmaf(c0.w, W.t, c0.z), Q = fmaf(c1.y, W.t, c1.x), ninv = -1.0f / Q;
        const unsigned met = __ballot_sync(0xffffffffu, b + lane < W.n && k1 >= W.ka - 1 && k1 < W.ka + T);
        const unsigned live = met & __ballot_sync(0xffffffffu, __ldg(W.live + u) != 0);
        if (live == 0) continue;
        // from the first to the last live column (q1 is monotone: all of them meet the tile)
        const int j0 = __ffs((int)live) - 1, j1 = 31 - __clz((int)live);
        const int kp = __shfl_up_sync(0xffffffffu, k1, 1);
        const unsigned moved = __ballot_sync(0xffffffffu, k1 != (lane == j0 ? cur : kp));
        __syncwarp();
        W.steps[lane].fP = make_float4(f1, f1, P, P);
        W.steps[lane].Qn = make_float4(Q, Q, ninv, ninv);
        W.texels[lane] = k1;
        __syncwarp();
        // row index of column j: (float as bits) + row, in 32-bit wrap-around
        const uint32_t rstep = (uint32_t)(W.du * W.pitch);
        uint32_t row = (uint32_t)((W.us + W.du * (b + j0)) * W.pitch + W.half - MG_BITS);
        for (int j = j0; j <= j1; ++j, row += rstep) {
            if ((moved >> j) & 1u) {
                const int k = W.texels[j];
                flush(cur, acc0);
                if (k == cur + 1) {
                    acc0 = acc1;
                } else {
                    flush(cur + 1, acc1);
                    acc0 = pk2(0.0f, 0.0f);
                }
                acc1 = pk2(0.0f, 0.0f);
                cur = k;
            }
            if (!((live >> j) & 1u)) continue;
            const float4 s0 = W.steps[j].fP, s1 = W.steps[j].Qn;
            const uint64_t f2 = pk2(s0.x, s0.y), Q2 = pk2(s1.x, s1.y), n2 = pk2(s1.z, s1.w);
            // first row with q2 - z >= -1: v = ceil((z - 1 - P) / Q); a row that
            // rounding puts on the wrong side of that line has a weight of 1e-5
            const uint64_t Pz = add2(pk2(s0.z, s0.w), W.nz2);
            const float2 tv = upk2(add2_rp(fma2(Pz, n2, n2), M2));
            const float ta = fminf(fmaxf(tv.x, tlo), thi), tb = fminf(fmaxf(tv.y, tlo), thi);
            uint64_t d = fma2(add2(pk2(ta, tb), nM2), Q2, Pz);
            const float *pa = W.rows + (uint32_t)(__float_as_int(ta) + row);
            const float *pb = W.rows + (uint32_t)(__float_as_int(tb) + row);
            uint64_t c = 0;
#pragma unroll
            for (int k = 0; k < NT; ++k) {
                const float2 df = upk2(d);
                const float ha = __saturatef(1.0f - fabsf(df.x)), hb = __saturatef(1.0f - fabsf(df.y));
                float ya = __ldg(pa + k), yb = __ldg(pb + k);
                if (GUARD) {
                    ya = ha > 0.0f ? ya : 0.0f;
                    yb = hb > 0.0f ? yb : 0.0f;
                }
                const uint64_t h = pk2(ha, hb), y = pk2(ya, yb);
                c = k == 0 ? mul2(h, y) : fma2(h, y, c);
                if (k + 1 < NT) d = add2(d, Q2);
            }
            acc0 = fma2(sub2(one2, f2), c, acc0);
            acc1 = fma2(f2, c, acc1);
        }
    }
    flush(cur, acc0);
    flush(cur + 1, acc1);
}

// Shared memory of a CTA of T x T x MG_Z voxels: the sums, then the warps' columns.
template <int T> constexpr int mg_smem() { return T * T * MG_ZP * 4 + T * 32 * (int)(sizeof(MGStep) + sizeof(int)); }

template <typename S, int T>
__global__ void __launch_bounds__(32 * T, 1024 / (32 * T)) matched_gather_kernel(const __grid_constant__ MGLaunch L)
{
    extern __shared__ __align__(16) float sums[];  // [y][x][MG_ZP]
    static_assert(T * T * MG_ZP % 4 == 0, "the columns' float4 are aligned");
    if (L.run && *L.run == 0) return;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    MGStep *steps = reinterpret_cast<MGStep *>(sums + T * T * MG_ZP);
    int *texels = reinterpret_cast<int *>(steps + T * 32);
    const int x0 = blockIdx.x * T, y0 = blockIdx.y * T;
    const int split = blockIdx.z / L.nzb;
    const int z0 = (blockIdx.z - split * L.nzb) * MG_Z;
    for (int i = threadIdx.x; i < T * T * MG_ZP; i += 32 * T) sums[i] = 0.0f;
    __syncthreads();
    for (int dir = 0; dir < 2; ++dir) {
        const int first = dir == 0 ? 0 : L.nx_views;
        const int count = dir == 0 ? L.nx_views : L.nviews - L.nx_views;
        const int s = (dir == 0 ? x0 : y0) + warp;
        const int lo = first + (int)((long long)count * split / L.splits);
        const int hi = first + (int)((long long)count * (split + 1) / L.splits);
        if (s < (dir == 0 ? L.nx : L.ny)) {
            MGWalk W;
            W.pitch = L.pitch;
            W.half = L.half;
            const float sf = (float)s;
            W.t = sf - 0.5f * (float)((dir == 0 ? L.nx : L.ny) - 1);
            W.vlo = (float)-L.half;
            W.vhi = (float)(L.nv - L.half);
            W.nz2 = pk2(-(float)(z0 + lane), -(float)(z0 + lane + 32));
            W.ka = dir == 0 ? y0 : x0;
            W.stride = (dir == 0 ? T : 1) * MG_ZP;
            W.acc = sums + (dir == 0 ? warp : warp * T) * MG_ZP + lane;
            W.steps = steps + warp * 32;
            W.texels = texels + warp * 32;
            const float umax = (float)(L.nu - 1), uc = 0.5f * (float)L.nu - 0.5f;
            for (int i = lo; i < hi; ++i) {
                const float4 ra = __ldg(reinterpret_cast<const float4 *>(L.recs + i));
                const float4 rb = __ldg(reinterpret_cast<const float4 *>(L.recs + i) + 1);
                // columns at which q1 (plus one half) is ka - 1 and ka + T:
                // u' = ((y - 1/2) e0 - a) / (b - (y - 1/2) e1) with
                // q1 - 1/2 = (a + b u') / (e0 + e1 u').  The divisor has the
                // sign of dq1/du' wherever some column reaches y; else y lies
                // past the value that q1 tends to where the denominator grows
                const float a = fmaf(ra.z, sf, rb.x), b = fmaf(ra.w, sf, rb.y);
                const float slope = fmaf(b, ra.x, -a * ra.y);
                float ue[2];
#pragma unroll
                for (int k = 0; k < 2; ++k) {
                    const float y = (float)(W.ka - 1 + k * (T + 1)) - 0.5f;
                    const float dv = fmaf(-y, ra.y, b);
                    const float far = ra.y > 0.0f ? umax + 2.0f : -2.0f;
                    const float w = fmaf(y, ra.x, -a) / dv + uc;
                    ue[k] = dv * slope > 0.0f ? fminf(fmaxf(w, -2.0f), umax + 2.0f) : far;
                }
                // a hundredth of a column on either side for rounding
                const int ua = max(0, (int)floorf(fminf(ue[0], ue[1]) - 0.01f));
                const int ub = min(L.nu - 1, (int)ceilf(fmaxf(ue[0], ue[1]) + 0.01f));
                if (ua > ub) continue;
                const bool up = slope > 0.0f;
                W.us = up ? ua : ub;
                W.n = ub - ua + 1;
                W.du = up ? 1 : -1;
                W.cols = L.cols + (long long)i * L.nu;
                W.live = L.live + (long long)i * L.nu;
                W.rows = L.rows + (long long)i * L.nu * L.pitch;
                const float dmax = fmaxf(fmaf((float)ua - uc, ra.y, ra.x), fmaf((float)ub - uc, ra.y, ra.x));
                const float terms = 2.0f * dmax / fmaf(rb.z, sf, rb.w) * 1.00001f;
                if (__ldg(L.bad + i)) mg_walk<T, MG_PAD, true>(W, lane);
                else if (terms <= 2.0f) mg_walk<T, 2, false>(W, lane);
                else if (terms <= 3.0f) mg_walk<T, 3, false>(W, lane);
                else if (terms <= 4.0f) mg_walk<T, 4, false>(W, lane);
                else mg_walk<T, MG_PAD, false>(W, lane);
            }
        }
        __syncthreads();  // the other direction's warps take other rows of the tile
    }
    S *out = static_cast<S *>(L.out) + (size_t)split * L.nz * L.ny * L.out_pitch;
    for (int i = threadIdx.x; i < T * T * MG_Z; i += 32 * T) {
        const int x = i % T, y = (i / T) % T, z = i / (T * T);
        if (x0 + x >= L.nx || y0 + y >= L.ny || z0 + z >= L.nz) continue;
        float r = sums[(y * T + x) * MG_ZP + z];
        S *o = out + ((size_t)(z0 + z) * L.ny + y0 + y) * L.out_pitch + x0 + x;
        if (L.accumulate) r += mg_load(*o);
        *o = mg_store<S>(r);
    }
}

// out (=|+=) the sum of the partial volumes, in order.
template <typename T>
__global__ void matched_fold_splits(const float *__restrict__ part, int splits, int nx, long long rows, T *out,
                                    long long pitch, int accumulate, const int *__restrict__ run)
{
    if (run && *run == 0) return;
    const long long n = rows * nx;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        float r = part[i];
        for (int k = 1; k < splits; ++k) r += part[k * n + i];
        const long long row = i / nx;
        T *o = out + row * pitch + (i - row * nx);
        if (accumulate) r += mg_load(*o);
        *o = mg_store<T>(r);
    }
}

// Which calls are gathered.  A gather takes time by columns x z of the tiles it
// launches, whether they hold voxels, have rows or not; a scatter by the samples
// of the rays there are.  Gathered over scattered time on dense projections
// (cone, magnification 1.5, 1.2 pixels):
//  - MG_MIN_SHARE: of the tiles' voxels in all waves of blocks, weighted by the
//    tile's borders, the share that lies in the volume and before the detector.
//    192^3 0.89: 0.80 to 0.89; 256^3 and 256^2 x 128 0.87: 0.75 to 0.91; 224^2 x
//    168 0.87: 0.77 to 0.86; 128^3 0.79: 0.89 to 1.03; 224^3 0.77: 0.87 to 0.98; 192^2 x
//    144 0.66: 1.04 to 1.15; 160^3 0.51: 1.06 to 1.25; 96^3 0.66: 1.06 to 1.23;
//    256^3 with 300, 250 and 160 of the 320 rows of its shadow: 0.90, 1.09, 1.62.
//  - MG_MAX_SPACING of the rows, in texels at the volume's middle: 0.57 0.68, 0.8
//    0.82, 0.97 0.88, 1.0 0.91, 1.22 1.2.
//  - MG_MAX_COLUMNS, of the columns, on average over the views (on a full orbit
//    1.12 times that of a view along an axis): 0.34 0.69, 1.0 0.84, 1.1 0.87, 1.5 0.95,
//    2.2 1.08 to 1.16.
//  - MG_MIN_WORK, voxels times views: 192^3 x 60 (4.2e8) 0.80, 128^2 x 64 x 120
//    (1.3e8) 1.00, 96^3 x 60 (5e7) 1.06.
constexpr double MG_MIN_SHARE = 0.85;
constexpr double MG_MAX_SPACING = 1.0;
constexpr double MG_MAX_COLUMNS = 1.15;
constexpr double MG_MIN_WORK = 3e8;

// Tiles of 16 x 16 voxels unless the blocks of 8 x 8 ones fill the GPU's
// slots (two blocks of 16 warps an SM, or four of 8) so much better that it
// makes up for their wider borders (9 / 8 texels' columns a
// tile instead of 17 / 16, and the walks' set-up twice as often).
struct MGTiling {
    int tile, nzb, splits;
    double share;  // voxels of the volume to those of all slots' waves
};
b2t_status mg_tiling(const b2t_dims3d &d, MGTiling &t)
{
    int dev = 0, sms = 0;
    B2T_CUDA_TRY(cudaGetDevice(&dev), "matched bp device");
    B2T_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev), "matched bp SM count");
    t.nzb = (int)((d.vol_z + MG_Z - 1) / MG_Z);
    auto blocks = [&](int T) { return (long long)((d.vol_x + T - 1) / T) * ((d.vol_y + T - 1) / T) * t.nzb; };
    auto cost = [&](int T, long long n) {  // of n blocks
        const long long slots = (T == 8 ? 4LL : 2LL) * sms;
        return (double)((n + slots - 1) / slots * slots) * T * T * (T == 8 ? 1.1 : 1.0);
    };
    t.tile = cost(8, blocks(8)) < cost(16, blocks(16)) ? 8 : 16;
    // small volumes: the views split over several blocks a tile, as many as
    // the slots hold
    const long long n = blocks(t.tile);
    t.splits = (int)std::max<long long>(
        1, std::min<long long>({(t.tile == 8 ? 4LL : 2LL) * sms / n, 8, (long long)d.angles / 8}));
    t.share = (double)d.vol_x * d.vol_y * d.vol_z * t.splits / (cost(t.tile, n * t.splits) * MG_Z);
    return B2T_OK;
}

// The view in FP64 terms of its rounded coefficients: one sign of the
// denominator over the detector, rows along +z at least 1/4 texel apart at
// every slice and on average at most MG_MAX_SPACING, and columns that do not
// turn round between the slices.
bool gather_view_ok(const FPView &w, const b2t_dims3d &d, int dir)
{
    if (w.e[2] != 0.0f || w.m1[2] != 0.0f || w.n1[2] != 0.0f) return false;
    const double n0 = dir == 0 ? d.vol_x : d.vol_y;
    const double ulo = 0.5 - 0.5 * d.det_u, uhi = -ulo;
    const double dlo = w.e[0] + w.e[1] * ulo, dhi = w.e[0] + w.e[1] * uhi;
    if (!(dlo * dhi > 0.0)) return false;
    if (std::max(std::abs(dlo), std::abs(dhi)) > 1e3 * std::min(std::abs(dlo), std::abs(dhi))) return false;
    double slope[2];
    if (!((w.m2[2] * 0.5 * (n0 - 1.0) + w.n2[2]) / w.e[0] <= MG_MAX_SPACING)) return false;
    for (int k = 0; k < 2; ++k) {
        const double s = k == 0 ? 0.0 : n0 - 1.0;
        const double q = w.m2[2] * s + w.n2[2];
        for (double den : {dlo, dhi})
            if (!(q / den >= 0.2501)) return false;
        const double a = w.m1[0] * s + w.n1[0], b = w.m1[1] * s + w.n1[1];
        slope[k] = b * w.e[0] - a * w.e[1];
        // columns at least a fiftieth of a texel apart
        if (!(std::abs(slope[k]) >= 0.02 * std::max(dlo * dlo, dhi * dhi))) return false;
    }
    return slope[0] * slope[1] > 0.0;
}

template <typename T>
b2t_status launch_prep(const MGPrep &L, dim3 grid, cudaStream_t s)
{
    matched_prep_kernel<T><<<grid, dim3(32, 8), 0, s>>>(L);
    count_launches(1);
    B2T_CUDA_TRY(cudaGetLastError(), "matched bp (gather) preparation launch");
    return B2T_OK;
}

template <typename S, int T> b2t_status launch_gather_tile(const MGLaunch &L, cudaStream_t s)
{
    auto kern = matched_gather_kernel<S, T>;
    B2T_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, mg_smem<T>()),
                 "matched bp (gather) smem attribute");
    const dim3 grid((L.nx + T - 1) / T, (L.ny + T - 1) / T, L.nzb * L.splits);
    kern<<<grid, 32 * T, mg_smem<T>(), s>>>(L);
    count_launches(1);
    B2T_CUDA_TRY(cudaGetLastError(), "matched bp (gather) launch");
    return B2T_OK;
}

template <typename S> b2t_status launch_gather(const MGLaunch &L, int tile, cudaStream_t s)
{
    return tile == 16 ? launch_gather_tile<S, 16>(L, s) : launch_gather_tile<S, 8>(L, s);
}

template <typename T>
b2t_status launch_split_fold(const float *part, int splits, const b2t_dims3d &d, void *vol, size_t pitch, int accumulate,
                             const int *run, cudaStream_t s)
{
    matched_fold_splits<T><<<1184, 256, 0, s>>>(part, splits, (int)d.vol_x, (long long)d.vol_y * d.vol_z,
                                                static_cast<T *>(vol), (long long)pitch, accumulate, run);
    count_launches(1);
    B2T_CUDA_TRY(cudaGetLastError(), "matched bp (gather) fold launch");
    return B2T_OK;
}

}  // namespace

bool matched_gather_eligible(const b2t_geom3d *g, const b2t_params3d *p, const std::vector<int> &dirs,
                             const std::vector<FPView> &coeffs, bool pays)
{
    const b2t_dims3d &d = g->dims;
    if (p->det_supersample != 1 || d.angles == 0) return false;
    // positions and row indices are split in FP32 around 1.5 * 2^23
    if (d.vol_x > 32768 || d.vol_y > 32768 || d.vol_z > 32768 || d.det_u > 32768 || d.det_v > 32768) return false;
    MGTiling t{};
    if (pays) {
        if ((double)d.vol_x * d.vol_y * d.vol_z * d.angles < MG_MIN_WORK) return false;
        if (mg_tiling(d, t) != B2T_OK || t.share < MG_MIN_SHARE) return false;
    }
    double columns = 0.0;
    for (uint32_t a = 0; a < d.angles; ++a) {
        if (dirs[a] > 1) return false;
        const FPView &w = coeffs[a];
        if (!gather_view_ok(w, d, dirs[a])) return false;
        // the volume's middle: spacing of the rows, of the columns
        const double mid = 0.5 * ((dirs[a] == 0 ? d.vol_x : d.vol_y) - 1.0);
        const double rows = (w.m2[2] * mid + w.n2[2]) / w.e[0];
        const double k1 = w.m1[0] * mid + w.n1[0], k1u = w.m1[1] * mid + w.n1[1];
        columns += std::abs(k1u * w.e[0] - k1 * w.e[1]) / ((double)w.e[0] * w.e[0]);
        if (pays && t.share * std::min(1.0, rows * d.det_v / d.vol_z) < MG_MIN_SHARE) return false;
    }
    return !pays || columns <= MG_MAX_COLUMNS * d.angles;
}

b2t_status matched_gather(const b2t_geom3d *g, const b2t_params3d *p, const void *proj, size_t proj_pitch, void *vol,
                          size_t vol_pitch, int32_t dtype, int accumulate, const std::vector<int> &dirs,
                          const std::vector<FPView> &coeffs, const int *run, cudaStream_t s)
{
    const b2t_dims3d &d = g->dims;
    MGLaunch L{};
    L.nu = (int)d.det_u;
    L.nv = (int)d.det_v;
    L.half = L.nv / 2;
    L.pitch = (L.nv + MG_PAD + 7) & ~7;
    L.nx = (int)d.vol_x;
    L.ny = (int)d.vol_y;
    L.nz = (int)d.vol_z;
    L.nviews = (int)d.angles;
    std::vector<uint32_t> order;
    for (int dir = 0; dir < 2; ++dir) {
        for (uint32_t a = 0; a < d.angles; ++a)
            if (dirs[a] == dir) order.push_back(a);
        if (dir == 0) L.nx_views = (int)order.size();
    }
    MGTiling t;
    B2T_TRY(mg_tiling(d, t));
    const int tile = t.tile;
    L.nzb = t.nzb;
    L.splits = t.splits;
    Scratch rows, cols, recs, live, part;
    const size_t ncol = (size_t)d.angles * d.det_u;
    B2T_TRY(rows.alloc(ncol * L.pitch * sizeof(float), s, "matched bp weighted rows"));
    B2T_TRY(cols.alloc(ncol * sizeof(MGColumn), s, "matched bp columns"));
    B2T_TRY(recs.alloc(d.angles * sizeof(MGRecord), s, "matched bp views"));
    const size_t flags = (ncol + d.angles) * sizeof(int);  // live, then bad
    B2T_TRY(live.alloc(flags, s, "matched bp live columns"));
    B2T_CUDA_TRY(cudaMemsetAsync(live.as<void>(), 0, flags, s), "matched bp live columns");
    const size_t vox = (size_t)d.vol_x * d.vol_y * d.vol_z;
    if (L.splits > 1) B2T_TRY(part.alloc(L.splits * vox * sizeof(float), s, "matched bp partial volumes"));
    L.run = run;
    L.rows = rows.as<float>();
    L.cols = cols.as<MGColumn>();
    L.recs = recs.as<MGRecord>();
    L.live = live.as<int>();
    L.bad = L.live + ncol;
    {
        auto *Pp = new MGPrep;
        MGPrep &P = *Pp;
        P.proj = proj;
        P.proj_pitch = (long long)proj_pitch;
        P.run = run;
        P.rows = rows.as<float>();
        P.cols = cols.as<MGColumn>();
        P.recs = recs.as<MGRecord>();
        P.live = live.as<int>();
        P.bad = P.live + ncol;
        P.nu = L.nu;
        P.nv = L.nv;
        P.na = (int)d.angles;
        P.pitch = L.pitch;
        P.half = L.half;
        P.mid[0] = 0.5f * (float)(L.nx - 1);
        P.mid[1] = 0.5f * (float)(L.ny - 1);
        for (int dir = 0; dir < 2; ++dir)
            fp_scale(g->kind, dir, g->vol_scale, false, p->output_scale, P.f1[dir], P.f2[dir], P.mul[dir]);
        b2t_status st = B2T_OK;
        for (size_t c0 = 0; c0 < order.size() && st == B2T_OK; c0 += MG_MAX_VIEWS) {
            P.first = (int)c0;
            P.nviews = (int)std::min(order.size() - c0, (size_t)MG_MAX_VIEWS);
            for (int i = 0; i < P.nviews; ++i) {
                const uint32_t a = order[c0 + i];
                P.views[i] = coeffs[a];
                P.dir[i] = (signed char)dirs[a];
            }
            const dim3 grid((L.nu + 31) / 32, (L.pitch + 32 * PREP_TILES - 1) / (32 * PREP_TILES), P.nviews);
            if (dtype == B2T_F32) st = launch_prep<float>(P, grid, s);
            else if (dtype == B2T_F16) st = launch_prep<__half>(P, grid, s);
            else st = launch_prep<__nv_bfloat16>(P, grid, s);
        }
        delete Pp;
        B2T_TRY(st);
    }
    if (L.splits > 1) {
        L.out = part.as<void>();
        L.out_pitch = L.nx;
        L.accumulate = 0;
        B2T_TRY(launch_gather<float>(L, tile, s));
        if (dtype == B2T_F32) return launch_split_fold<float>(part.as<float>(), L.splits, d, vol, vol_pitch, accumulate, run, s);
        if (dtype == B2T_F16) return launch_split_fold<__half>(part.as<float>(), L.splits, d, vol, vol_pitch, accumulate, run, s);
        return launch_split_fold<__nv_bfloat16>(part.as<float>(), L.splits, d, vol, vol_pitch, accumulate, run, s);
    }
    L.out = vol;
    L.out_pitch = (long long)vol_pitch;
    L.accumulate = accumulate;
    if (dtype == B2T_F32) return launch_gather<float>(L, tile, s);
    if (dtype == B2T_F16) return launch_gather<__half>(L, tile, s);
    return launch_gather<__nv_bfloat16>(L, tile, s);
}

}  // namespace b2t
