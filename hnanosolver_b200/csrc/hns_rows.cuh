// 7-point stencils over half z-rows, shared by the FP32 and the reduced-precision steps.
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <cstdint>

#include "hns_internal.cuh"
#include "hns_stencil.cuh"
#include "hns_types.cuh"

namespace hns {
namespace dev {

// ---- stencils over half z-rows ------------------------------------------------------------
//
// The divergence, the gradient subtraction and the refinement residual are 7-point stencils in
// leaf slot order, where a leaf's z-row (x, y) = (a, b) is 8 contiguous slots. A thread covers
// z = 4h .. 4h + 3 of one row (128 threads per leaf, kRowLeaves leaves per 256-thread CTA): it
// loads its half row and the same half of the four x/y neighbour rows (the row of the leaf
// across a face at the leaf's edge; a missing leaf reads 0) as vector loads, and the two z
// neighbours past its ends (the row's other half, or the leaf across the z face). The leaves'
// face neighbours come straight from the 27-neighbour table: no staging, no barrier. Measured
// on a 45,198-leaf grid, one leaf per thread in 256-thread CTAs beat 128- and 512-thread CTAs
// and two or three leaves per thread for all three stencils.
constexpr int kRowThreads = 256;
constexpr int kRowLeaves = kRowThreads / 128;

struct HalfRow {
    int64_t leaf, own;   // own: slot of the half row's first voxel (a multiple of 4)
    int row, h, a, b;    // row = 8 a + b
    int nx, ny, nz;      // leaf across the x face / y face this row touches (itself inside), across
                         // the z face this half touches (-z for h = 0, +z for h = 1); -1 missing
};

// The half row of this thread in leaf group g (the kRowLeaves leaves one CTA covers); false
// past the last leaf.
__device__ __forceinline__ bool half_row(const TopoView& t, HalfRow& r, int64_t g) {
    r.leaf = g * kRowLeaves + (threadIdx.x >> 7);
    if (r.leaf >= t.num_leaves) return false;
    r.row = (threadIdx.x >> 1) & 63, r.h = threadIdx.x & 1, r.a = r.row >> 3, r.b = r.row & 7;
    r.own = (r.leaf << 9) + 8 * r.row + 4 * r.h;
    const int* nb = t.nbr27 + r.leaf * 27;
    // nbr27: (dx+1)*9 + (dy+1)*3 + (dz+1); entry 13 is the leaf itself.
    r.nx = __ldg(nb + (r.a == 7 ? 22 : r.a == 0 ? 4 : 13));
    r.ny = __ldg(nb + (r.b == 7 ? 16 : r.b == 0 ? 10 : 13));
    r.nz = __ldg(nb + (r.h ? 14 : 12));
    return true;
}

// Slots of the same half row in the four x/y neighbour rows (the half row itself where the
// neighbour leaf is missing: its values are then replaced by 0).
struct NbrRows {
    int64_t xp, xm, yp, ym;
    bool zxp, zxm, zyp, zym;  // missing neighbour: read as 0
};

__device__ __forceinline__ NbrRows nbr_rows(const HalfRow& r) {
    auto across = [&](int n, int rw) -> int64_t { return n < 0 ? r.own : ((int64_t)n << 9) + 8 * rw + 4 * r.h; };
    NbrRows q;
    q.xp = r.a < 7 ? r.own + 64 : across(r.nx, r.b);
    q.xm = r.a > 0 ? r.own - 64 : across(r.nx, 56 + r.b);
    q.yp = r.b < 7 ? r.own + 8 : across(r.ny, 8 * r.a);
    q.ym = r.b > 0 ? r.own - 8 : across(r.ny, 8 * r.a + 7);
    q.zxp = r.a == 7 && r.nx < 0, q.zxm = r.a == 0 && r.nx < 0, q.zyp = r.b == 7 && r.ny < 0, q.zym = r.b == 0 && r.ny < 0;
    return q;
}

// Slots of the z neighbours past the half row's ends: the row's other half, and the voxel
// across the z face (-1 when that leaf is missing).
__device__ __forceinline__ void z_ends(const HalfRow& r, int64_t& zin, int64_t& zface) {
    zin = r.h ? r.own - 1 : r.own + 4;
    zface = r.nz < 0 ? -1 : ((int64_t)r.nz << 9) + 8 * r.row + (r.h ? 0 : 7);
}

__device__ __forceinline__ void ld_half4(const double* __restrict__ q, double v[4]) {
    const double2 x0 = __ldg(reinterpret_cast<const double2*>(q));
    const double2 x1 = __ldg(reinterpret_cast<const double2*>(q) + 1);
    v[0] = x0.x, v[1] = x0.y, v[2] = x1.x, v[3] = x1.y;
}

// Velocity of four voxels from slot s (a multiple of 4): 12 interleaved components, 24 bytes in
// BF16 (three 8-byte loads) or 48 in FP32 (three 16-byte loads).
__device__ __forceinline__ float bf16_bits(uint32_t w, int hi) { return __uint_as_float(hi ? (w & 0xFFFF0000u) : (w << 16)); }

__device__ __forceinline__ void vel_half_row(const __nv_bfloat16* __restrict__ v, int64_t s, float3 u[4]) {
    const uint2* q = reinterpret_cast<const uint2*>(v + 3 * s);
    const uint2 w0 = __ldg(q), w1 = __ldg(q + 1), w2 = __ldg(q + 2);
    const uint32_t w[6] = {w0.x, w0.y, w1.x, w1.y, w2.x, w2.y};
#pragma unroll
    for (int z = 0; z < 4; ++z) {
        const int e = 3 * z;
        u[z] = make_float3(bf16_bits(w[e >> 1], e & 1), bf16_bits(w[(e + 1) >> 1], (e + 1) & 1),
                           bf16_bits(w[(e + 2) >> 1], (e + 2) & 1));
    }
}
__device__ __forceinline__ void vel_half_row(const float* __restrict__ v, int64_t s, float3 u[4]) {
    const float4* q = reinterpret_cast<const float4*>(v + 3 * s);
    const float4 a = __ldg(q), b = __ldg(q + 1), c = __ldg(q + 2);
    u[0] = make_float3(a.x, a.y, a.z);
    u[1] = make_float3(a.w, b.x, b.y);
    u[2] = make_float3(b.z, b.w, c.x);
    u[3] = make_float3(c.y, c.z, c.w);
}

__device__ __forceinline__ uint32_t bf16x2_bits(float lo, float hi) {
    const __nv_bfloat162 r = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&r);
}
__device__ __forceinline__ void store_vel_half_row(__nv_bfloat16* v, int64_t s, const float3 u[4]) {
    uint2* q = reinterpret_cast<uint2*>(v + 3 * s);
    q[0] = make_uint2(bf16x2_bits(u[0].x, u[0].y), bf16x2_bits(u[0].z, u[1].x));
    q[1] = make_uint2(bf16x2_bits(u[1].y, u[1].z), bf16x2_bits(u[2].x, u[2].y));
    q[2] = make_uint2(bf16x2_bits(u[2].z, u[3].x), bf16x2_bits(u[3].y, u[3].z));
}
__device__ __forceinline__ void store_vel_half_row(float* v, int64_t s, const float3 u[4]) {
    float4* q = reinterpret_cast<float4*>(v + 3 * s);
    q[0] = make_float4(u[0].x, u[0].y, u[0].z, u[1].x);
    q[1] = make_float4(u[1].y, u[1].z, u[2].x, u[2].y);
    q[2] = make_float4(u[2].z, u[3].x, u[3].y, u[3].z);
}

// Element-wise forms of the same, for velocity arrays that are not 8-byte (BF16) or 16-byte
// (FP32) aligned; kVec selects the vector form.
template <bool kVec, typename V>
__device__ __forceinline__ void vel_row(const V* __restrict__ v, int64_t s, float3 u[4]) {
    if constexpr (kVec) {
        vel_half_row(v, s, u);
    } else {
#pragma unroll
        for (int z = 0; z < 4; ++z) u[z] = vload(v, s + z);
    }
}
// The same of an array that the kernel writes (in place, the thread's own voxels): plain loads.
template <bool kVec>
__device__ __forceinline__ void vel_row_rw(const float* v, int64_t s, float3 u[4]) {
    if constexpr (kVec) {
        const float4* q = reinterpret_cast<const float4*>(v + 3 * s);
        const float4 a = q[0], b = q[1], c = q[2];
        u[0] = make_float3(a.x, a.y, a.z), u[1] = make_float3(a.w, b.x, b.y);
        u[2] = make_float3(b.z, b.w, c.x), u[3] = make_float3(c.y, c.z, c.w);
    } else {
#pragma unroll
        for (int z = 0; z < 4; ++z) u[z] = make_float3(v[3 * (s + z)], v[3 * (s + z) + 1], v[3 * (s + z) + 2]);
    }
}
template <bool kVec>
__device__ __forceinline__ void vel_row_rw(const __nv_bfloat16* v, int64_t s, float3 u[4]) {
    uint32_t w[6];
    if constexpr (kVec) {
        const uint2* q = reinterpret_cast<const uint2*>(v + 3 * s);
        const uint2 a = q[0], b = q[1], c = q[2];
        w[0] = a.x, w[1] = a.y, w[2] = b.x, w[3] = b.y, w[4] = c.x, w[5] = c.y;
    } else {
        const unsigned short* q = reinterpret_cast<const unsigned short*>(v) + 3 * s;
#pragma unroll
        for (int i = 0; i < 6; ++i) w[i] = (uint32_t)q[2 * i] | ((uint32_t)q[2 * i + 1] << 16);
    }
#pragma unroll
    for (int z = 0; z < 4; ++z) {
        const int e = 3 * z;
        u[z] = make_float3(bf16_bits(w[e >> 1], e & 1), bf16_bits(w[(e + 1) >> 1], (e + 1) & 1),
                           bf16_bits(w[(e + 2) >> 1], (e + 2) & 1));
    }
}
template <bool kVec, typename V>
__device__ __forceinline__ void store_vel_row(V* v, int64_t s, const float3 u[4]) {
    if constexpr (kVec) {
        store_vel_half_row(v, s, u);
    } else {
#pragma unroll
        for (int z = 0; z < 4; ++z) vstore(v, s + z, u[z]);
    }
}

__device__ __forceinline__ float vel_z(const __nv_bfloat16* __restrict__ v, int64_t s) {
    return __bfloat162float(__ldg(v + 3 * s + 2));
}
__device__ __forceinline__ float vel_z(const float* __restrict__ v, int64_t s) { return __ldg(v + 3 * s + 2); }

// Four scalars from slot s (a multiple of 4) as FP32, and back; element-wise where the array is not
// aligned to four of them.
template <bool kVec>
__device__ __forceinline__ void scalar_row(const float* __restrict__ p, int64_t s, float v[4]) {
    if constexpr (kVec) {
        const float4 a = __ldg(reinterpret_cast<const float4*>(p + s));
        v[0] = a.x, v[1] = a.y, v[2] = a.z, v[3] = a.w;
    } else {
#pragma unroll
        for (int z = 0; z < 4; ++z) v[z] = __ldg(p + s + z);
    }
}
template <bool kVec>
__device__ __forceinline__ void scalar_row(const __half* __restrict__ p, int64_t s, float v[4]) {
    if constexpr (kVec) {
        const uint2 a = __ldg(reinterpret_cast<const uint2*>(p + s));
        v[0] = __half2float(__ushort_as_half((unsigned short)(a.x & 0xFFFFu)));
        v[1] = __half2float(__ushort_as_half((unsigned short)(a.x >> 16)));
        v[2] = __half2float(__ushort_as_half((unsigned short)(a.y & 0xFFFFu)));
        v[3] = __half2float(__ushort_as_half((unsigned short)(a.y >> 16)));
    } else {
#pragma unroll
        for (int z = 0; z < 4; ++z) v[z] = sload(p, s + z);
    }
}
template <bool kVec>
__device__ __forceinline__ void store_scalar_row(float* p, int64_t s, const float v[4]) {
    if constexpr (kVec) {
        *reinterpret_cast<float4*>(p + s) = make_float4(v[0], v[1], v[2], v[3]);
    } else {
#pragma unroll
        for (int z = 0; z < 4; ++z) p[s + z] = v[z];
    }
}
template <bool kVec>
__device__ __forceinline__ void store_scalar_row(__half* p, int64_t s, const float v[4]) {
    if constexpr (kVec) {
        const __half2 a = __floats2half2_rn(v[0], v[1]), b = __floats2half2_rn(v[2], v[3]);
        *reinterpret_cast<uint2*>(p + s) = make_uint2(*reinterpret_cast<const uint32_t*>(&a), *reinterpret_cast<const uint32_t*>(&b));
    } else {
#pragma unroll
        for (int z = 0; z < 4; ++z) sstore(p, s + z, v[z]);
    }
}
// Whether an array allows the vector forms.
inline bool row_aligned(const void* p, size_t element) { return (reinterpret_cast<uintptr_t>(p) & (4 * element - 1)) == 0; }

// Divergence (divergence, src/Cuda/Kernel.cu:432-453) of a reduced-precision velocity into
// FP32: per voxel the face velocities are the means of the centre and the neighbour (0 for a
// missing neighbour), div = (xp - xm + yp - ym + zp - zm) / dx.
// `c` receives the half row's own velocities.
template <bool kVec, typename V>
__device__ __forceinline__ void half_row_divergence(const HalfRow& r, const V* __restrict__ vel, float inv_dx, float3 c[4],
                                                    float d[4]) {
    const NbrRows q = nbr_rows(r);
    float3 xp[4], xm[4], yp[4], ym[4];
    vel_row<kVec>(vel, r.own, c);
    vel_row<kVec>(vel, q.xp, xp);
    vel_row<kVec>(vel, q.xm, xm);
    vel_row<kVec>(vel, q.yp, yp);
    vel_row<kVec>(vel, q.ym, ym);
    int64_t zin_s, zface_s;
    z_ends(r, zin_s, zface_s);
    const float zin = vel_z(vel, zin_s), zface = zface_s < 0 ? 0.f : vel_z(vel, zface_s);
    const float zlo = r.h ? zin : zface, zhi = r.h ? zface : zin;
#pragma unroll
    for (int z = 0; z < 4; ++z) {
        const float vxp = (c[z].x + (q.zxp ? 0.f : xp[z].x)) * 0.5f;
        const float vxm = (c[z].x + (q.zxm ? 0.f : xm[z].x)) * 0.5f;
        const float vyp = (c[z].y + (q.zyp ? 0.f : yp[z].y)) * 0.5f;
        const float vym = (c[z].y + (q.zym ? 0.f : ym[z].y)) * 0.5f;
        const float vzp = (c[z].z + (z < 3 ? c[z + 1].z : zhi)) * 0.5f;
        const float vzm = (c[z].z + (z > 0 ? c[z - 1].z : zlo)) * 0.5f;
        d[z] = (vxp - vxm + vyp - vym + vzp - vzm) * inv_dx;
    }
}

// kVec: the velocity's vector form; kVecOut: the divergence's.
template <typename V, bool kVec, bool kVecOut>
__global__ void __launch_bounds__(kRowThreads) divergence_rows_kernel(TopoView t, const V* __restrict__ vel,
                                                                      float* __restrict__ div, float inv_dx) {
    HalfRow r;
    if (!half_row(t, r, blockIdx.x)) return;
    float3 c[4];
    float d[4];
    half_row_divergence<kVec>(r, vel, inv_dx, c, d);
    store_scalar_row<kVecOut>(div, r.own, d);
}

// u - grad p with an FP32 pressure (subtractPressureGradient, src/Cuda/Kernel.cu:495-541), FP32
// velocity; vel and out may be the same array. kWalls: zero-gradient walls, a missing neighbour's
// pressure is the voxel's own (else 0).
template <bool kWalls, bool kVec, bool kVecP>
__global__ void __launch_bounds__(kRowThreads) gradient_rows_kernel(TopoView t, const float* vel, const float* __restrict__ p,
                                                                    float* out, float inv_dx) {
    HalfRow r;
    if (!half_row(t, r, blockIdx.x)) return;
    const NbrRows q = nbr_rows(r);
    float c[4], xp[4], xm[4], yp[4], ym[4];
    scalar_row<kVecP>(p, r.own, c);
    scalar_row<kVecP>(p, q.xp, xp);
    scalar_row<kVecP>(p, q.xm, xm);
    scalar_row<kVecP>(p, q.yp, yp);
    scalar_row<kVecP>(p, q.ym, ym);
    int64_t zin_s, zface_s;
    z_ends(r, zin_s, zface_s);
    const float zin = __ldg(p + zin_s), zface = zface_s >= 0 ? __ldg(p + zface_s) : kWalls ? c[r.h ? 3 : 0] : 0.f;
    const float zlo = r.h ? zin : zface, zhi = r.h ? zface : zin;
    float3 u[4];
    vel_row_rw<kVec>(vel, r.own, u);
    const float h = 0.5f * inv_dx;
#pragma unroll
    for (int z = 0; z < 4; ++z) {
        auto n = [&](bool missing, float v) { return missing ? (kWalls ? c[z] : 0.f) : v; };
        const float gx = (n(q.zxp, xp[z]) - n(q.zxm, xm[z])) * h;
        const float gy = (n(q.zyp, yp[z]) - n(q.zym, ym[z])) * h;
        const float gz = ((z < 3 ? c[z < 3 ? z + 1 : 3] : zhi) - (z > 0 ? c[z > 0 ? z - 1 : 0] : zlo)) * h;
        u[z] = make_float3(u[z].x - gx, u[z].y - gy, u[z].z - gz);
    }
    store_vel_row<kVec>(out, r.own, u);
}

// u -= grad p with p in FP64 (0 outside the domain), central differences
// (subtractPressureGradient, src/Cuda/Kernel.cu:495-541), velocity in reduced precision or
// FP32, in place.
template <typename V, bool kVec>
__global__ void __launch_bounds__(kRowThreads) gradient_mixed_kernel(TopoView t, V* __restrict__ vel,
                                                                   const double* __restrict__ p, float inv_dx) {
    HalfRow r;
    if (!half_row(t, r, blockIdx.x)) return;
    const NbrRows q = nbr_rows(r);
    double c[4], xp[4], xm[4], yp[4], ym[4];
    ld_half4(p + r.own, c);
    ld_half4(p + q.xp, xp);
    ld_half4(p + q.xm, xm);
    ld_half4(p + q.yp, yp);
    ld_half4(p + q.ym, ym);
    int64_t zin_s, zface_s;
    z_ends(r, zin_s, zface_s);
    const double zin = __ldg(p + zin_s), zface = zface_s < 0 ? 0.0 : __ldg(p + zface_s);
    const double zlo = r.h ? zin : zface, zhi = r.h ? zface : zin;
    float3 u[4];
    vel_row_rw<kVec>(vel, r.own, u);
    const double hh = 0.5 * (double)inv_dx;
#pragma unroll
    for (int z = 0; z < 4; ++z) {
        const float gx = (float)(((q.zxp ? 0.0 : xp[z]) - (q.zxm ? 0.0 : xm[z])) * hh);
        const float gy = (float)(((q.zyp ? 0.0 : yp[z]) - (q.zym ? 0.0 : ym[z])) * hh);
        const float gz = (float)(((z < 3 ? c[z + 1] : zhi) - (z > 0 ? c[z - 1] : zlo)) * hh);
        u[z] = make_float3(u[z].x - gx, u[z].y - gy, u[z].z - gz);
    }
    store_vel_row<kVec>(vel, r.own, u);
}

inline unsigned row_blocks(const Context& c) { return (unsigned)((c.topo.num_leaves + kRowLeaves - 1) / kRowLeaves); }

}  // namespace dev
}  // namespace hns
