// Ray-driven 3D forward projection from a "bilinear cell" copy of the volume.
//
// Same model as fp3d_kernel (the reference's cone_FP_t / par3D_FP_t,
// cuda/3d/cone_fp.cu:154-231, cuda/3d/par3d_fp.cu:152-230): per ray, the
// slices of the view's dominant axis are sampled bilinearly at unit steps.
//
// The direct-load kernel issues four scalar loads per sample and is bound by
// the L1/TEX pipeline (about seven sectors per warp load).  Here the volume is
// first rewritten, once per call and per marching direction present, into a
// grid of cells: the cell at texel (k1, k2) of slice s holds everything the
// bilinear sample with base texel (k1, k2) needs, so a sample is one aligned
// vector load:
//   FP32 storage:      float4 (c0, c1, c2, c3) with
//                      c0 = v00, c1 = v10 - v00, c2 = v01 - v00,
//                      c3 = v11 - v10 - v01 + v00,
//                      value = c0 + f1 c1 + f2 (c2 + f1 c3)  (three FMAs);
//   FP16/BF16 storage: the four corner values (8 bytes), interpolated in FP32
//                      (no re-rounding of the stored data).
// Cells cover padded texel indices -2..n+1 in both plane axes (the texture
// border is zero), so every ray's clipped slice range stays inside the grid
// exactly as in fp3d_kernel.  Two cell layouts: the columns layout (cells
// contiguous along z, build_cells_cols, fp3d_col_kernel) for x- and y-major
// views, whose warps follow detector columns; the rows layout (contiguous
// along the first plane axis, build_cells, fp3d_cell_kernel) for z-major
// views.  fp3d_cells_build / fp3d_cells_project split the layout pass from
// the projection, so that a streamed call lays a volume out once for all of
// its angle blocks.
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cstdio>
#include <cstdlib>
#include <map>
#include <mutex>
#include <string>
#include <vector>

#include "b2t_internal.h"
#include "proj3d.h"

namespace b2t {

namespace {

template <typename T> __device__ __forceinline__ float vload(const T *p);
template <> __device__ __forceinline__ float vload<float>(const float *p) { return __ldg(p); }
template <> __device__ __forceinline__ float vload<__half>(const __half *p) { return __half2float(__ldg(p)); }
template <> __device__ __forceinline__ float vload<__nv_bfloat16>(const __nv_bfloat16 *p)
{
    return __bfloat162float(__ldg(p));
}
template <typename T> __device__ __forceinline__ T vstore(float v);
template <> __device__ __forceinline__ float vstore<float>(float v) { return v; }
template <> __device__ __forceinline__ __half vstore<__half>(float v) { return __float2half_rn(v); }
template <> __device__ __forceinline__ __nv_bfloat16 vstore<__nv_bfloat16>(float v) { return __float2bfloat16_rn(v); }

template <typename T> struct CellDtype;
template <> struct CellDtype<float> { static constexpr int32_t value = B2T_F32; };
template <> struct CellDtype<__half> { static constexpr int32_t value = B2T_F16; };
template <> struct CellDtype<__nv_bfloat16> { static constexpr int32_t value = B2T_BF16; };

// Cell storage per type: 16 bytes (float coefficients) or 8 bytes (corners).
template <typename T> struct CellT;
template <> struct CellT<float> { using type = float4; };
template <> struct CellT<__half> { using type = uint2; };
template <> struct CellT<__nv_bfloat16> { using type = uint2; };

__device__ __forceinline__ float4 make_cell(float v00, float v10, float v01, float v11, float *)
{
    return make_float4(v00, v10 - v00, v01 - v00, (v11 - v10) - (v01 - v00));
}

template <typename H> __device__ __forceinline__ uint2 pack_corners(float v00, float v10, float v01, float v11);
template <> __device__ __forceinline__ uint2 pack_corners<__half>(float v00, float v10, float v01, float v11)
{
    __half2 a = __floats2half2_rn(v00, v10), b = __floats2half2_rn(v01, v11);
    return make_uint2(*reinterpret_cast<unsigned *>(&a), *reinterpret_cast<unsigned *>(&b));
}
template <> __device__ __forceinline__ uint2 pack_corners<__nv_bfloat16>(float v00, float v10, float v01, float v11)
{
    __nv_bfloat162 a = __floats2bfloat162_rn(v00, v10), b = __floats2bfloat162_rn(v01, v11);
    return make_uint2(*reinterpret_cast<unsigned *>(&a), *reinterpret_cast<unsigned *>(&b));
}

// Interpolate a cell at weights (f1, f2).
__device__ __forceinline__ float interp(const float4 &c, float f1, float f2)
{
    return fmaf(f2, fmaf(f1, c.w, c.z), fmaf(f1, c.y, c.x));
}
template <typename H> __device__ __forceinline__ float interp_corners(uint2 c, float f1, float f2);
template <> __device__ __forceinline__ float interp_corners<__half>(uint2 c, float f1, float f2)
{
    const float2 a = __half22float2(*reinterpret_cast<__half2 *>(&c.x));
    const float2 b = __half22float2(*reinterpret_cast<__half2 *>(&c.y));
    const float r0 = fmaf(f1, a.y - a.x, a.x), r1 = fmaf(f1, b.y - b.x, b.x);
    return fmaf(f2, r1 - r0, r0);
}
template <> __device__ __forceinline__ float interp_corners<__nv_bfloat16>(uint2 c, float f1, float f2)
{
    const float2 a = __bfloat1622float2(*reinterpret_cast<__nv_bfloat162 *>(&c.x));
    const float2 b = __bfloat1622float2(*reinterpret_cast<__nv_bfloat162 *>(&c.y));
    const float r0 = fmaf(f1, a.y - a.x, a.x), r1 = fmaf(f1, b.y - b.x, b.x);
    return fmaf(f2, r1 - r0, r0);
}

// Builds the cells of direction `dir`: cell index (j2 * n0 + s) * m1 + j1 for
// dir 0 / 1, (s * m2 + j2) * m1 + j1 for dir 2, m = n + 4, j = k + 2.
template <typename T>
__global__ void build_cells(const T *__restrict__ vol, size_t pitch, int nx, int ny, int nz, int dir,
                            typename CellT<T>::type *__restrict__ cells)
{
    const int j1 = blockIdx.x * blockDim.x + threadIdx.x;
    const int j2 = blockIdx.y;
    const int s = blockIdx.z;
    int n1, n2;
    if (dir == 0) { n1 = ny; n2 = nz; }
    else if (dir == 1) { n1 = nx; n2 = nz; }
    else { n1 = nx; n2 = ny; }
    const int m1 = n1 + 4, m2 = n2 + 4;
    if (j1 >= m1) return;
    const int k1 = j1 - 2, k2 = j2 - 2;
    float v[4];
#pragma unroll
    for (int c = 0; c < 4; ++c) {
        const int a1 = k1 + (c & 1), a2 = k2 + (c >> 1);
        float val = 0.0f;
        if (a1 >= 0 && a1 < n1 && a2 >= 0 && a2 < n2) {
            int x, y, z;
            if (dir == 0) { x = s; y = a1; z = a2; }
            else if (dir == 1) { x = a1; y = s; z = a2; }
            else { x = a1; y = a2; z = s; }
            val = vload(vol + ((size_t)z * ny + y) * pitch + x);
        }
        v[c] = val;
    }
    size_t idx;
    if (dir == 2) idx = ((size_t)s * m2 + j2) * m1 + j1;
    else {
        const int n0 = (dir == 0) ? nx : ny;
        idx = ((size_t)j2 * n0 + s) * m1 + j1;
    }
    if constexpr (sizeof(typename CellT<T>::type) == 16) {
        cells[idx] = make_cell(v[0], v[1], v[2], v[3], nullptr);
    } else {
        cells[idx] = pack_corners<T>(v[0], v[1], v[2], v[3]);
    }
}

template <typename T>
__device__ __forceinline__ void store_cell(typename CellT<T>::type *dst, float v00, float v10, float v01, float v11)
{
    if constexpr (sizeof(typename CellT<T>::type) == 16) {
        *dst = make_cell(v00, v10, v01, v11, nullptr);
    } else {
        *dst = pack_corners<T>(v00, v10, v01, v11);
    }
}

// Builds the columns layout of direction dir (0: slices along x, k1 = y;
// 1: slices along y, k1 = x; k2 = z for both): cell (j1, s, j2) at
// (j1 n0 + s) m2 + j2, j = k + 2, m = n + 4.  A CTA stages a tile of the
// volume in shared memory, read along x, and writes 32 x 32 cells along j2:
//   dir 0: blockIdx = (j2 tile, s tile, j1), tile[p][zi][xi] = vol(s0 + xi, k1 + p, k2_0 + zi);
//   dir 1: blockIdx = (j2 tile, j1 tile, s), tile[0][zi][xi] = vol(k1_0 + xi, s, k2_0 + zi).
// Rows of 33 floats keep the column reads of the write phase conflict-free.
template <typename T>
__global__ void __launch_bounds__(256) build_cells_cols(const T *__restrict__ vol, size_t pitch, int nx, int ny,
                                                        int nz, int dir, typename CellT<T>::type *__restrict__ cells)
{
    __shared__ float t[2][33][33];
    const int n0 = (dir == 0) ? nx : ny;
    const int m1 = ((dir == 0) ? ny : nx) + 4, m2 = nz + 4;
    const int j2_0 = blockIdx.x * 32, k2_0 = j2_0 - 2;
    const int tid = threadIdx.x;
    const int ji = tid & 31, j2 = j2_0 + ji;
    if (dir == 0) {
        const int s0 = blockIdx.y * 32, j1 = blockIdx.z, k1 = j1 - 2;
        for (int e = tid; e < 2 * 33 * 32; e += 256) {
            const int xi = e & 31, zi = (e >> 5) % 33, pk = e / (33 * 32);
            const int x = s0 + xi, y = k1 + pk, z = k2_0 + zi;
            float val = 0.0f;
            if (x < nx && y >= 0 && y < ny && z >= 0 && z < nz) val = vload(vol + ((size_t)z * ny + y) * pitch + x);
            t[pk][zi][xi] = val;
        }
        __syncthreads();
        if (j2 >= m2) return;
        for (int si = tid >> 5; si < 32 && s0 + si < n0; si += 8)
            store_cell<T>(cells + ((size_t)j1 * n0 + s0 + si) * m2 + j2, t[0][ji][si], t[1][ji][si], t[0][ji + 1][si],
                          t[1][ji + 1][si]);
    } else {
        const int j1_0 = blockIdx.y * 32, k1_0 = j1_0 - 2, sl = blockIdx.z;
        for (int e = tid; e < 33 * 33; e += 256) {
            const int xi = e % 33, zi = e / 33;
            const int x = k1_0 + xi, z = k2_0 + zi;
            float val = 0.0f;
            if (x >= 0 && x < nx && z >= 0 && z < nz) val = vload(vol + ((size_t)z * ny + sl) * pitch + x);
            t[0][zi][xi] = val;
        }
        __syncthreads();
        if (j2 >= m2) return;
        for (int i1 = tid >> 5; i1 < 32 && j1_0 + i1 < m1; i1 += 8)
            store_cell<T>(cells + ((size_t)(j1_0 + i1) * n0 + sl) * m2 + j2, t[0][ji][i1], t[0][ji][i1 + 1],
                          t[0][ji + 1][i1], t[0][ji + 1][i1 + 1]);
    }
}

__device__ __forceinline__ void clip_slices_c(float A, float B, float lo, float hi, float &smin, float &smax)
{
    if (fabsf(A) < 1e-12f) {
        if (!(B >= lo && B <= hi)) {
            smin = 1.0f;
            smax = 0.0f;
        }
        return;
    }
    float s1 = (lo - B) / A, s2 = (hi - B) / A;
    smin = fmaxf(smin, fminf(s1, s2));
    smax = fminf(smax, fmaxf(s1, s2));
}

// Base texel of sample position qh = qm + 1/2 by rounding down: qh + M
// rounded toward -inf holds floor(qh) in its mantissa (|qh| < 2^22); the
// same texel and weight as split_texel_c up to exact ties, where both give
// the same value.
constexpr float SPLIT_M = 12582912.0f;  // 1.5 * 2^23
__device__ __forceinline__ int floor_texel(float qh) { return __float_as_int(__fadd_rd(qh, SPLIT_M)) - 0x4B400000; }

__device__ __forceinline__ bool texel_ok_f(float A, float Bh, int s, int n)
{
    const int k = floor_texel(fmaf(A, (float)s, Bh));
    return k >= -2 && k <= n;
}

template <typename T>
__device__ __forceinline__ float cell_value(const typename CellT<T>::type *p, float f1, float f2)
{
    if constexpr (sizeof(typename CellT<T>::type) == 16) {
        return interp(__ldg(p), f1, f2);
    } else {
        return interp_corners<T>(__ldg(p), f1, f2);
    }
}

// One ray through the rows layout (ray set-up and slice clipping of
// fp3d_kernel): acc + the sum of its samples times the ray length factor.
// L.vol points at the cell of slice 0, texels (k1 = 0, k2 = 0); the cell of
// slice s, texels (k1, k2) is at L.vol + s st0 + k1 + k2 st2 (strides in
// cells).  UNR independent accumulators keep UNR cell loads in flight.
template <typename T, int UNR>
__device__ __forceinline__ float trace_rows(const FPLaunch &L, const FPView &V, float uu, float vv, float acc)
{
    using C = typename CellT<T>::type;
    const float n0 = (float)L.n0;
    const float den = fmaf(vv, V.e[2], fmaf(uu, V.e[1], V.e[0]));
    const float inv = 1.0f / den;
    const float A1 = fmaf(vv, V.m1[2], fmaf(uu, V.m1[1], V.m1[0])) * inv;
    const float A2 = fmaf(vv, V.m2[2], fmaf(uu, V.m2[1], V.m2[0])) * inv;
    const float B1 = fmaf(vv, V.n1[2], fmaf(uu, V.n1[1], V.n1[0])) * inv;
    const float B2 = fmaf(vv, V.n2[2], fmaf(uu, V.n2[1], V.n2[0])) * inv;
    float smin = 0.0f, smax = n0 - 1.0f;
    clip_slices_c(A1, B1, -1.6f, (float)L.n1 - 0.4f, smin, smax);
    clip_slices_c(A2, B2, -1.6f, (float)L.n2 - 0.4f, smin, smax);
    int s_lo = max(0, (int)ceilf(fmaxf(smin, -1.0f)));
    int s_hi = min(L.n0 - 1, (int)floorf(fminf(smax, n0)));
    // sample positions plus one half: texel floor(), weight frac()
    const float B1h = B1 + 0.5f, B2h = B2 + 0.5f;
    for (int it = 0; it < 3 && s_lo <= s_hi; ++it) {
        if (texel_ok_f(A1, B1h, s_lo, L.n1) && texel_ok_f(A2, B2h, s_lo, L.n2)) break;
        ++s_lo;
    }
    for (int it = 0; it < 3 && s_lo <= s_hi; ++it) {
        if (texel_ok_f(A1, B1h, s_hi, L.n1) && texel_ok_f(A2, B2h, s_hi, L.n2)) break;
        --s_hi;
    }
    if (!(texel_ok_f(A1, B1h, s_lo, L.n1) && texel_ok_f(A2, B2h, s_lo, L.n2) &&
          texel_ok_f(A1, B1h, s_hi, L.n1) && texel_ok_f(A2, B2h, s_hi, L.n2)))
        s_hi = s_lo - 1;
    // the base texels are monotone in s, so the checks at both ends keep
    // every access inside the cell grid.  The cell address is formed from
    // the bits of the rounded-down sums (k + 0x4B400000) with 32 x 32 ->
    // 64-bit multiply-adds; the constant offset wraps around in 64 bits
    constexpr uint32_t cb = (uint32_t)sizeof(C);
    const uint32_t st0b = (uint32_t)(L.st0 * cb), st2b = (uint32_t)(L.st2 * cb);
    const unsigned long long base0 =
        reinterpret_cast<unsigned long long>(L.vol) - 0x4B400000ull * ((unsigned long long)st2b + cb);
    auto sample = [&](int sl) -> float {
        const float q1 = fmaf(A1, (float)sl, B1h), q2 = fmaf(A2, (float)sl, B2h);
        const float t1 = __fadd_rd(q1, SPLIT_M), t2 = __fadd_rd(q2, SPLIT_M);
        const float f1 = q1 - (t1 - SPLIT_M), f2 = q2 - (t2 - SPLIT_M);
        const unsigned long long a = base0 + (unsigned long long)(uint32_t)sl * st0b +
                                     (unsigned long long)(uint32_t)__float_as_int(t2) * st2b +
                                     (unsigned long long)(uint32_t)__float_as_int(t1) * cb;
        return cell_value<T>(reinterpret_cast<const C *>(a), f1, f2);
    };
    float sum[UNR];
#pragma unroll
    for (int k = 0; k < UNR; ++k) sum[k] = 0.0f;
    int s = s_lo;
    for (; s + UNR - 1 <= s_hi; s += UNR) {
#pragma unroll
        for (int k = 0; k < UNR; ++k) sum[k] += sample(s + k);
    }
    for (; s <= s_hi; ++s) sum[0] += sample(s);
#pragma unroll
    for (int w = UNR / 2; w >= 1; w /= 2) {
#pragma unroll
        for (int k = 0; k < w; ++k) sum[k] += sum[k + w];
    }
    return fmaf(sum[0], sqrtf(fmaf(A1 * A1, L.f1, fmaf(A2 * A2, L.f2, 1.0f))) * L.mul, acc);
}

template <typename T>
__device__ __forceinline__ void store_ray(const FPLaunch &L, int a, int u, int v, float acc)
{
    T *out = static_cast<T *>(L.proj) + ((size_t)v * L.na + a) * L.proj_pitch + u;
    if (L.accumulate) acc += (float)(*out);
    *out = vstore<T>(acc);
}

// Rows layout (k1 stride 1), used for z-major views: a CTA traces one
// 32 x VROWS tile of detector pixels for VPC consecutive views (threadIdx.z
// selects the view).  Neighbouring views sample nearly the same cells at the
// same slice (the orbit turns by a fraction of a degree per view), and the
// warps of one CTA share an SM, so the views of a CTA reuse each other's
// cells in L1 instead of fetching them again from L2.
template <typename T, int VPC, int VROWS>
__global__ void __launch_bounds__(32 * VROWS * VPC, 2048 / (32 * VROWS * VPC)) fp3d_cell_kernel(const __grid_constant__ FPLaunch L)
{
    const int vi = blockIdx.x * VPC + threadIdx.z;
    if (vi >= L.nviews) return;
    const FPView &V = L.views[vi];
    const int u = blockIdx.y * 32 + threadIdx.x;
    const int v = blockIdx.z * VROWS + threadIdx.y;
    if (u >= L.nu || v >= L.nv) return;
    const int R = L.rays;
    float acc = 0.0f;
    for (int iu = 0; iu < R; ++iu) {
        for (int iv = 0; iv < R; ++iv) {
            float uu = (float)u + 0.5f - 0.5f * (float)L.nu;
            float vv = (float)v + 0.5f - 0.5f * (float)L.nv;
            if (R > 1) {
                uu += -0.5f + (0.5f + (float)iu) / (float)R;
                vv += -0.5f + (0.5f + (float)iv) / (float)R;
            }
            acc = trace_rows<T, 2>(L, V, uu, vv, acc);
        }
    }
    if (R > 1) acc /= (float)(R * R);
    store_ray<T>(L, V.a, u, v, acc);
}

// Columns layout (cell of slice s, texels (k1, k2) at L.vol + s st0 + k1 st1
// + k2), used for x- and y-major views: a warp traces
// 32 consecutive detector rows of one column, a CTA VCOLS columns for VPC
// consecutive views.  For a detector whose v axis is parallel to the
// volume's z axis (circular orbits, parallel or cone) the rays of one column
// lie in one plane containing z, so at every slice they share the in-plane
// texel k1 and their k2 run along the contiguous axis: a warp's 16-byte
// loads fall on three or four 128-byte lines instead of the seven to nine a
// detector row needs when its rays cross several k2 rows.  Four loads in
// flight per thread cover the L2 latency: 32 registers and four CTAs per SM
// with 32-bit cell indices (IDX32, a cell array of fewer than 2^32 cells),
// else 64-bit addresses at 40 registers and three CTAs.
// The ray set-up is the rows tracer's, written out here: the shared form
// spilled at 40 registers.
template <typename T, int VPC, int VCOLS, bool IDX32>
__global__ void __launch_bounds__(32 * VCOLS * VPC, (IDX32 ? 2048 : 1536) / (32 * VCOLS * VPC)) fp3d_col_kernel(const __grid_constant__ FPLaunch L)
{
    using C = typename CellT<T>::type;
    const int vi = blockIdx.x * VPC + threadIdx.z;
    if (vi >= L.nviews) return;
    const FPView &V = L.views[vi];
    const int v = blockIdx.z * 32 + threadIdx.x;
    const int u = blockIdx.y * VCOLS + threadIdx.y;
    if (u >= L.nu || v >= L.nv) return;
    const C *__restrict__ cells = static_cast<const C *>(L.vol);
    const long long st0 = L.st0, st1 = L.st1;  // slice and k1 strides; k2 stride 1
    const int R = L.rays;
    const float n0 = (float)L.n0;
    float acc = 0.0f;
    for (int iu = 0; iu < R; ++iu) {
        for (int iv = 0; iv < R; ++iv) {
            float uu = (float)u + 0.5f - 0.5f * (float)L.nu;
            float vv = (float)v + 0.5f - 0.5f * (float)L.nv;
            if (R > 1) {
                uu += -0.5f + (0.5f + (float)iu) / (float)R;
                vv += -0.5f + (0.5f + (float)iv) / (float)R;
            }
            const float den = fmaf(vv, V.e[2], fmaf(uu, V.e[1], V.e[0]));
            const float inv = 1.0f / den;
            const float A1 = fmaf(vv, V.m1[2], fmaf(uu, V.m1[1], V.m1[0])) * inv;
            const float A2 = fmaf(vv, V.m2[2], fmaf(uu, V.m2[1], V.m2[0])) * inv;
            const float B1 = fmaf(vv, V.n1[2], fmaf(uu, V.n1[1], V.n1[0])) * inv;
            const float B2 = fmaf(vv, V.n2[2], fmaf(uu, V.n2[1], V.n2[0])) * inv;
            float smin = 0.0f, smax = n0 - 1.0f;
            clip_slices_c(A1, B1, -1.6f, (float)L.n1 - 0.4f, smin, smax);
            clip_slices_c(A2, B2, -1.6f, (float)L.n2 - 0.4f, smin, smax);
            int s_lo = max(0, (int)ceilf(fmaxf(smin, -1.0f)));
            int s_hi = min(L.n0 - 1, (int)floorf(fminf(smax, n0)));
            const float B1h = B1 + 0.5f, B2h = B2 + 0.5f;
            for (int it = 0; it < 3 && s_lo <= s_hi; ++it) {
                if (texel_ok_f(A1, B1h, s_lo, L.n1) && texel_ok_f(A2, B2h, s_lo, L.n2)) break;
                ++s_lo;
            }
            for (int it = 0; it < 3 && s_lo <= s_hi; ++it) {
                if (texel_ok_f(A1, B1h, s_hi, L.n1) && texel_ok_f(A2, B2h, s_hi, L.n2)) break;
                --s_hi;
            }
            if (!(texel_ok_f(A1, B1h, s_lo, L.n1) && texel_ok_f(A2, B2h, s_lo, L.n2) &&
                  texel_ok_f(A1, B1h, s_hi, L.n1) && texel_ok_f(A2, B2h, s_hi, L.n2)))
                s_hi = s_lo - 1;
            constexpr uint32_t cb = (uint32_t)sizeof(C);
            const uint32_t st0b = (uint32_t)(st0 * cb), st1b = (uint32_t)(st1 * cb);
            const unsigned long long base0 = reinterpret_cast<unsigned long long>(cells) -
                                             0x4B400000ull * ((unsigned long long)st1b + cb);
            // IDX32 (a cell array of fewer than 2^32 cells): the cell index
            // from the array's first cell, k + 2 >= 0 on both plane axes, in
            // 32-bit arithmetic (the constant offset wraps around), then one
            // wide multiply-add for the address; 32 registers, four CTAs per SM
            const C *arr = cells - 2 * st1 - 2;
            const uint32_t s0 = (uint32_t)st0, s1 = (uint32_t)st1;
            const uint32_t ibase = 2u * s1 + 2u - 0x4B400000u * (s1 + 1u);
            auto sample = [&](int sl) -> float {
                const float q1 = fmaf(A1, (float)sl, B1h), q2 = fmaf(A2, (float)sl, B2h);
                const float t1 = __fadd_rd(q1, SPLIT_M), t2 = __fadd_rd(q2, SPLIT_M);
                const float f1 = q1 - (t1 - SPLIT_M), f2 = q2 - (t2 - SPLIT_M);
                if constexpr (IDX32) {
                    const uint32_t idx = (uint32_t)sl * s0 + (uint32_t)__float_as_int(t1) * s1 +
                                         (uint32_t)__float_as_int(t2) + ibase;
                    return cell_value<T>(arr + idx, f1, f2);
                } else {
                    const unsigned long long a = base0 + (unsigned long long)(uint32_t)sl * st0b +
                                                 (unsigned long long)(uint32_t)__float_as_int(t1) * st1b +
                                                 (unsigned long long)(uint32_t)__float_as_int(t2) * cb;
                    return cell_value<T>(reinterpret_cast<const C *>(a), f1, f2);
                }
            };
            float sum0 = 0.0f, sum1 = 0.0f, sum2 = 0.0f, sum3 = 0.0f;
            int s = s_lo;
            for (; s + 3 <= s_hi; s += 4) {
                sum0 += sample(s);
                sum1 += sample(s + 1);
                sum2 += sample(s + 2);
                sum3 += sample(s + 3);
            }
            for (; s <= s_hi; ++s) sum0 += sample(s);
            sum0 += sum2;
            sum1 += sum3;
            const float sc = sqrtf(fmaf(A1 * A1, L.f1, fmaf(A2 * A2, L.f2, 1.0f))) * L.mul;
            acc = fmaf(sum0 + sum1, sc, acc);
        }
    }
    if (R > 1) acc /= (float)(R * R);
    store_ray<T>(L, V.a, u, v, acc);
}

// Launches of the cell kernels since the last b2t_fp_path_stats.
static std::atomic<unsigned long long> g_cell_launches{0};

// Launch shape of the cell forward projector: views per CTA.
struct CellShape {
    int vpc;
};

// Shapes chosen by b2t_autotune_fp3d, per problem class, for this process.
static std::mutex g_shape_mutex;
static std::map<std::string, CellShape> g_shapes;
// Set by the autotuner while it times one candidate on this thread.
static thread_local const CellShape *t_shape_override = nullptr;

static std::string shape_key(const b2t_geom3d *g, const b2t_params3d *p, int32_t dtype)
{
    const b2t_dims3d &d = g->dims;
    char buf[160];
    std::snprintf(buf, sizeof(buf), "%d/%d/%u/%u/%u/%u/%u/%u/%u", g->kind, dtype, d.vol_x, d.vol_y, d.vol_z, d.angles,
                  d.det_u, d.det_v, p->det_supersample);
    return buf;
}

// The autotuner's candidate while it runs; else B2T_FP_VPC (1, 2, 4 or 8)
// from the environment; else the tuned shape of this problem class; else 4
// views per CTA.
static CellShape choose_shape(const std::string &key)
{
    if (t_shape_override) return *t_shape_override;
    if (const char *e = std::getenv("B2T_FP_VPC")) {
        const int v = std::atoi(e);
        return CellShape{(v == 1 || v == 2 || v == 8) ? v : 4};
    }
    std::lock_guard<std::mutex> lock(g_shape_mutex);
    auto it = g_shapes.find(key);
    return it != g_shapes.end() ? it->second : CellShape{4};
}

template <typename T, int VPC, int VROWS>
static b2t_status launch_cells_shape(const FPLaunch &P, int nviews, const b2t_dims3d &d, cudaStream_t s)
{
    dim3 grid((unsigned)((nviews + VPC - 1) / VPC), (d.det_u + 31) / 32, (d.det_v + VROWS - 1) / VROWS);
    fp3d_cell_kernel<T, VPC, VROWS><<<grid, dim3(32, VROWS, VPC), 0, s>>>(P);
    count_launches(1);
    g_cell_launches.fetch_add(1);
    B2T_CUDA_TRY(cudaGetLastError(), "fp3d_cell_kernel launch");
    return B2T_OK;
}

template <typename T>
static b2t_status launch_cells(const FPLaunch &P, int nviews, const b2t_dims3d &d, const CellShape &shape,
                               cudaStream_t s)
{
    switch (shape.vpc) {
    case 1: return launch_cells_shape<T, 1, 8>(P, nviews, d, s);
    case 2: return launch_cells_shape<T, 2, 4>(P, nviews, d, s);
    case 8: return launch_cells_shape<T, 8, 2>(P, nviews, d, s);
    default: return launch_cells_shape<T, 4, 4>(P, nviews, d, s);
    }
}

template <typename T, int VPC, int VCOLS>
static b2t_status launch_cols_shape(const FPLaunch &P, int nviews, const b2t_dims3d &d, cudaStream_t s)
{
    dim3 grid((unsigned)((nviews + VPC - 1) / VPC), (d.det_u + VCOLS - 1) / VCOLS, (d.det_v + 31) / 32);
    // the cell count of the columns layout, (n1 + 4) n0 (n2 + 4)
    const unsigned long long cells = (unsigned long long)(P.n1 + 4) * (unsigned long long)P.st1;
    if (cells < (1ull << 32))
        fp3d_col_kernel<T, VPC, VCOLS, true><<<grid, dim3(32, VCOLS, VPC), 0, s>>>(P);
    else
        fp3d_col_kernel<T, VPC, VCOLS, false><<<grid, dim3(32, VCOLS, VPC), 0, s>>>(P);
    count_launches(1);
    g_cell_launches.fetch_add(1);
    B2T_CUDA_TRY(cudaGetLastError(), "fp3d_col_kernel launch");
    return B2T_OK;
}

template <typename T>
static b2t_status launch_cols(const FPLaunch &P, int nviews, const b2t_dims3d &d, const CellShape &shape,
                              cudaStream_t s)
{
    switch (shape.vpc) {
    case 1: return launch_cols_shape<T, 1, 16>(P, nviews, d, s);
    case 2: return launch_cols_shape<T, 2, 8>(P, nviews, d, s);
    case 8: return launch_cols_shape<T, 8, 2>(P, nviews, d, s);
    default: return launch_cols_shape<T, 4, 4>(P, nviews, d, s);
    }
}

template <typename T>
b2t_status build_cells_t(const b2t_geom3d *g, const void *vol, size_t vol_pitch, const bool need[3],
                         const bool slab[3], cudaStream_t s, FPCells &c)
{
    using C = typename CellT<T>::type;
    const b2t_dims3d &d = g->dims;
    const int nx = d.vol_x, ny = d.vol_y, nz = d.vol_z;
    c.dtype = CellDtype<T>::value;
    c.vol_x = d.vol_x;
    c.vol_y = d.vol_y;
    c.vol_z = d.vol_z;
    for (int dir = 0; dir < 3; ++dir) {
        c.base[dir] = nullptr;
        c.slab[dir] = false;
        if (!need[dir]) continue;
        if (slab[dir]) {
            // slab copy for the TMA-staged kernel (fp3d_slab.cu)
            if (!c.mem[dir]) c.mem[dir].reset(new Scratch);
            B2T_TRY(c.mem[dir]->alloc(fp_slab_copy_bytes(d, dir), s, "b2t_fp3d scratch (slab copy)"));
            B2T_TRY(fp_slab_build(d, vol, vol_pitch, CellDtype<T>::value, dir, c.mem[dir]->as<void>(), s));
            c.slab[dir] = true;
            c.base[dir] = c.mem[dir]->as<void>();
            continue;
        }
        int n0, n1, n2;
        if (dir == 0) { n0 = nx; n1 = ny; n2 = nz; }
        else if (dir == 1) { n0 = ny; n1 = nx; n2 = nz; }
        else { n0 = nz; n1 = nx; n2 = ny; }
        const long long m1 = n1 + 4, m2 = n2 + 4;
        const size_t count = (size_t)m1 * m2 * n0;
        if (!c.mem[dir]) c.mem[dir].reset(new Scratch);
        B2T_TRY(c.mem[dir]->alloc(count * sizeof(C), s, "b2t_fp3d scratch (cells)"));
        C *cells = c.mem[dir]->as<C>();
        if (dir == 2) {
            // rows layout: cell (s, j2, j1) at (s m2 + j2) m1 + j1
            dim3 grid((unsigned)((m1 + 127) / 128), (unsigned)m2, (unsigned)n0);
            build_cells<T><<<grid, 128, 0, s>>>(static_cast<const T *>(vol), vol_pitch, nx, ny, nz, dir, cells);
            c.st0[dir] = m1 * m2;
            c.st1[dir] = 1;
            c.st2[dir] = m1;
        } else {
            // columns layout: cell (j1, s, j2) at (j1 n0 + s) m2 + j2
            dim3 grid((unsigned)((m2 + 31) / 32), (unsigned)((dir == 0 ? n0 : m1) + 31) / 32,
                      (unsigned)(dir == 0 ? m1 : n0));
            build_cells_cols<T><<<grid, 256, 0, s>>>(static_cast<const T *>(vol), vol_pitch, nx, ny, nz, dir, cells);
            c.st0[dir] = m2;
            c.st1[dir] = (long long)n0 * m2;
            c.st2[dir] = 1;
        }
        count_launches(1);
        B2T_CUDA_TRY(cudaGetLastError(), "cell layout launch");
        c.base[dir] = cells + 2 * c.st1[dir] + 2 * c.st2[dir];
    }
    return B2T_OK;
}

template <typename T>
b2t_status project_cells_t(const b2t_geom3d *g, const b2t_params3d *p, const FPCells &c, void *proj,
                           size_t proj_pitch, int32_t mode, const std::vector<int> &dirs, cudaStream_t s)
{
    const b2t_dims3d &d = g->dims;
    const int nx = d.vol_x, ny = d.vol_y, nz = d.vol_z;
    bool need[3] = {false, false, false};
    for (int dd : dirs) need[dd] = true;
    const CellShape shape = choose_shape(shape_key(g, p, CellDtype<T>::value));
    FPLaunch *Lp = new FPLaunch;
    FPLaunch &P = *Lp;
    const bool force_noncube = p->det_supersample > 1;
    b2t_status st = B2T_OK;
    for (int dir = 0; dir < 3 && st == B2T_OK; ++dir) {
        if (!need[dir]) continue;
        if (c.slab[dir]) {
            if (!fp_slab_eligible(g, p, dir, dirs)) {
                st = fail(B2T_ERR_UNSUPPORTED, "b2t_fp3d: views or parameters differ from those the slab copy was "
                                               "built for");
                break;
            }
            st = fp_slab_project(g, p, c.base[dir], dir, proj, proj_pitch, c.dtype, mode, dirs, s);
            continue;
        }
        P.proj = proj;
        P.proj_pitch = (long long)proj_pitch;
        P.nu = d.det_u;
        P.nv = d.det_v;
        P.na = d.angles;
        P.rays = p->det_supersample;
        P.accumulate = (mode == B2T_MODE_ADD) ? 1 : 0;
        fp_scale(g->kind, dir, g->vol_scale, force_noncube, p->output_scale, P.f1, P.f2, P.mul);
        if (dir == 0) { P.n0 = nx; P.n1 = ny; P.n2 = nz; }
        else if (dir == 1) { P.n0 = ny; P.n1 = nx; P.n2 = nz; }
        else { P.n0 = nz; P.n1 = nx; P.n2 = ny; }
        P.st0 = c.st0[dir];
        P.st1 = c.st1[dir];
        P.st2 = c.st2[dir];
        P.vol = c.base[dir];
        std::vector<int> views;
        for (uint32_t a = 0; a < d.angles; ++a)
            if (dirs[a] == dir) views.push_back((int)a);
        for (size_t c0 = 0; c0 < views.size() && st == B2T_OK; c0 += FP_MAX_VIEWS) {
            const size_t cn = std::min(views.size() - c0, (size_t)FP_MAX_VIEWS);
            P.nviews = (int)cn;
            for (size_t i = 0; i < cn; ++i) {
                const int a = views[c0 + i];
                fp_view_coeffs(g->kind, g->views[a], d, dir, P.views[i]);
                P.views[i].a = a;
            }
            st = (dir == 2) ? launch_cells<T>(P, (int)cn, d, shape, s) : launch_cols<T>(P, (int)cn, d, shape, s);
            if (st != B2T_OK) break;
        }
    }
    delete Lp;
    return st;
}

}  // namespace

b2t_status fp3d_autotune_impl(const b2t_geom3d *g, const b2t_params3d *p, const void *vol, size_t vol_pitch,
                              void *proj, size_t proj_pitch, int32_t dtype, cudaStream_t s, int32_t *vpc_out)
{
    B2T_TRY(validate3d(g, "b2t_autotune_fp3d"));
    if (!p || !vol || !proj) return fail(B2T_ERR_INVALID_ARG, "b2t_autotune_fp3d: null argument");
    if (!dtype_valid(dtype)) return fail(B2T_ERR_INVALID_ARG, "b2t_autotune_fp3d: bad dtype %d", dtype);
    static const CellShape cands[] = {{1}, {2}, {4}, {8}};
    cudaEvent_t e0 = nullptr, e1 = nullptr;
    B2T_CUDA_TRY(cudaEventCreate(&e0), "autotune event");
    cudaError_t ce = cudaEventCreate(&e1);
    if (ce != cudaSuccess) {
        cudaEventDestroy(e0);
        return cuda_fail(ce, "autotune event");
    }
    CellShape best{4};
    float best_ms = 1e30f;
    b2t_status st = B2T_OK;
    for (const CellShape &c : cands) {
        t_shape_override = &c;
        // one untimed run, then the best of two timed runs of the whole call
        st = fp3d_impl(g, p, vol, vol_pitch, proj, proj_pitch, dtype, B2T_MODE_SET, s);
        float ms = 1e30f;
        for (int rep = 0; rep < 2 && st == B2T_OK; ++rep) {
            cudaEventRecord(e0, s);
            st = fp3d_impl(g, p, vol, vol_pitch, proj, proj_pitch, dtype, B2T_MODE_SET, s);
            cudaEventRecord(e1, s);
            ce = cudaEventSynchronize(e1);
            if (ce != cudaSuccess) {
                st = cuda_fail(ce, "autotune timing");
                break;
            }
            float t = 0.0f;
            cudaEventElapsedTime(&t, e0, e1);
            ms = std::min(ms, t);
        }
        t_shape_override = nullptr;
        if (st != B2T_OK) break;
        if (ms < best_ms) {
            best_ms = ms;
            best = c;
        }
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    if (st != B2T_OK) return st;
    {
        std::lock_guard<std::mutex> lock(g_shape_mutex);
        g_shapes[shape_key(g, p, dtype)] = best;
    }
    if (vpc_out) *vpc_out = best.vpc;
    return B2T_OK;
}

unsigned long long fp_cell_launches_take() { return g_cell_launches.exchange(0); }

FPCells::FPCells() = default;
FPCells::~FPCells() = default;

b2t_status fp3d_cells_build(const b2t_geom3d *g, const b2t_params3d *p, const void *vol, size_t vol_pitch,
                            int32_t dtype, const bool need[3], bool choose, cudaStream_t s, FPCells &c)
{
    if (vol_pitch == 0) vol_pitch = g->dims.vol_x;
    std::vector<int> dirs(g->dims.angles);
    for (uint32_t a = 0; a < g->dims.angles; ++a) dirs[a] = dominant_axis(g->kind, g->views[a], g->dims);
    bool slab[3] = {false, false, false}, cells_chosen = false;
    for (int dir = 0; dir < 2; ++dir) {
        if (!need[dir]) continue;
        if (dtype != B2T_F32) {
            slab[dir] = fp_slab_pays(g, dir, dirs, dtype) && fp_slab_eligible(g, p, dir, dirs);
        } else if (fp_slab_eligible(g, p, dir, dirs)) {
            slab[dir] = !choose || fp_slab_pays(g, dir, dirs, dtype);
            cells_chosen = cells_chosen || !slab[dir];
        }
    }
    if (dtype == B2T_F32) {
        const b2t_status st = build_cells_t<float>(g, vol, vol_pitch, need, slab, s, c);
        if (st != B2T_ERR_NO_MEMORY || !cells_chosen) return st;
        clear_error();  // the slab copy is half the size
        return fp3d_cells_build(g, p, vol, vol_pitch, dtype, need, false, s, c);
    }
    if (dtype == B2T_F16) return build_cells_t<__half>(g, vol, vol_pitch, need, slab, s, c);
    return build_cells_t<__nv_bfloat16>(g, vol, vol_pitch, need, slab, s, c);
}

b2t_status fp3d_cells_project(const b2t_geom3d *g, const b2t_params3d *p, const FPCells &c, void *proj,
                              size_t proj_pitch, int32_t mode, cudaStream_t s)
{
    const b2t_dims3d &d = g->dims;
    if (d.vol_x != c.vol_x || d.vol_y != c.vol_y || d.vol_z != c.vol_z)
        return fail(B2T_ERR_INVALID_ARG, "fp3d_cells_project: the cells were built for another volume");
    if (proj_pitch == 0) proj_pitch = d.det_u;
    std::vector<int> dirs(d.angles);
    for (uint32_t a = 0; a < d.angles; ++a) {
        dirs[a] = dominant_axis(g->kind, g->views[a], d);
        if (!c.base[dirs[a]]) return fail(B2T_ERR_INVALID_ARG, "fp3d_cells_project: no cells for view %u", a);
    }
    if (c.dtype == B2T_F32) return project_cells_t<float>(g, p, c, proj, proj_pitch, mode, dirs, s);
    if (c.dtype == B2T_F16) return project_cells_t<__half>(g, p, c, proj, proj_pitch, mode, dirs, s);
    return project_cells_t<__nv_bfloat16>(g, p, c, proj, proj_pitch, mode, dirs, s);
}

b2t_status fp3d_cells(const b2t_geom3d *g, const b2t_params3d *p, const void *vol, size_t vol_pitch, void *proj,
                      size_t proj_pitch, int32_t dtype, int32_t mode, const std::vector<int> &dirs, cudaStream_t s)
{
    bool need[3] = {false, false, false};
    for (int dd : dirs) need[dd] = true;
    FPCells c;
    B2T_TRY(fp3d_cells_build(g, p, vol, vol_pitch, dtype, need, true, s, c));
    if (dtype == B2T_F32) return project_cells_t<float>(g, p, c, proj, proj_pitch, mode, dirs, s);
    if (dtype == B2T_F16) return project_cells_t<__half>(g, p, c, proj, proj_pitch, mode, dirs, s);
    return project_cells_t<__nv_bfloat16>(g, p, c, proj, proj_pitch, mode, dirs, s);
}

}  // namespace b2t
