// MacCormack advection of the velocity and at most one scalar from a leaf tile in shared memory
// (advect_vector, src/Cuda/Kernel.cu:349-426, and advect_scalar, Kernel.cu:294-344, along one
// shared trace; samplers read 0 outside the domain), for both storages: FP32 fields, and BF16
// velocity with an FP16 scalar (FP32 arithmetic).
//
// The leaf's voxels and a one-voxel halo, a tile of 10^3 cells (u, v, w, s), are read once into
// shared memory. A trace cell whose eight corners lie in the tile is eight shared-memory loads at
// fixed offsets from one base index (a back trace shorter than a voxel per axis, and a forward
// trace that ends within a voxel of the start); other cells take the leaf-table path, reading the
// arrays. The clamp's six face neighbours always lie in the tile. Cells of missing leaves hold 0.
// One CTA of 256 threads per leaf, two voxels per thread.
//
// What bounds it: instruction issue and the shared-memory pipe, far above DRAM (16 or 32 bytes a
// voxel). Hence
//   - cells of the 16-bit storage stay packed in 8 bytes and are widened after the load (exactly),
//     half the shared-memory traffic of FP32 cells for four more instructions a cell;
//   - the lerps run on pairs of channels, (u, v) and (w, s), with packed FP32 operations (one issue
//     for two roundings, the same bits as scalar operations);
//   - the clamp's minimum and maximum take three operands an instruction.
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <cstdint>

#include "hns_stencil.cuh"
#include "hns_types.cuh"

namespace hns {
namespace dev {

constexpr int kTileHalo = 1;
constexpr int kTileSide = 8 + 2 * kTileHalo;
constexpr int kTileCells = kTileSide * kTileSide * kTileSide;
constexpr int kTileThreads = 256;
constexpr int kTileFill = (kTileCells + kTileThreads - 1) / kTileThreads;  // cells a thread fills

// A pair of FP32 values in one 64-bit register.
using F2 = unsigned long long;
__device__ __forceinline__ F2 f2(float lo, float hi) {
    F2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ void un2(F2 v, float& lo, float& hi) { asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v)); }
__device__ __forceinline__ F2 sub2(F2 a, F2 b) {
    F2 r;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ F2 mul2(F2 a, F2 b) {
    F2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ F2 fma2(F2 a, F2 b, F2 c) {
    F2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
// a + p q on both halves, rounded after each operation. The assembler contracts a packed product
// and the sum that takes it into one rounding, whatever the compiler is told about contraction; a
// sum written as product * one + a with a `one` it cannot know (a kernel argument, 1) it leaves
// alone, and that is the rounded sum exactly.
__device__ __forceinline__ F2 mul_add2(F2 p, F2 q, F2 a, F2 one) { return fma2(mul2(p, q), one, a); }
// lerp1 (a + w (b - a)) on both halves.
__device__ __forceinline__ F2 lerp2(F2 a, F2 b, F2 w, F2 one) { return mul_add2(w, sub2(b, a), a, one); }

__device__ __forceinline__ float min3(float a, float b, float c) {
    float r;
    asm("min.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}
__device__ __forceinline__ float max3(float a, float b, float c) {
    float r;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}

// Four channels of a cell: (u, v) and (w, s).
struct Ch4 {
    F2 uv, ws;
};

// FP32 storage: a cell is its four values. A quarter-warp's 16-byte loads are one z-row of voxels,
// so with strides that are multiples of 8 cells their bank groups are set by z alone.
struct TileF32 {
    using V = float;
    using S = float;
    using Cell = float4;
    static constexpr int kSY = 16, kSX = kTileSide * kSY, kCtasPerSm = 4;
    static __device__ __forceinline__ Cell read(const V* __restrict__ vel, const S* __restrict__ s0, int64_t s) {
        return make_float4(__ldg(vel + 3 * s), __ldg(vel + 3 * s + 1), __ldg(vel + 3 * s + 2), s0 ? __ldg(s0 + s) : 0.f);
    }
    static __device__ __forceinline__ Cell zero() { return make_float4(0.f, 0.f, 0.f, 0.f); }
    static __device__ __forceinline__ Ch4 widen(const Cell& c) { return Ch4{f2(c.x, c.y), f2(c.z, c.w)}; }
};

// BF16 velocity and FP16 scalar: a cell is u | v << 16, w | s << 16. A half-warp's 8-byte loads are
// two z-rows, whose 8-cell halves of the banks differ with a y stride of 8 mod 16 cells.
struct TileHalf {
    using V = __nv_bfloat16;
    using S = __half;
    using Cell = uint2;
    static constexpr int kSY = 24, kSX = kTileSide * kSY, kCtasPerSm = 5;
    static __device__ __forceinline__ Cell read(const V* __restrict__ vel, const S* __restrict__ s0, int64_t s) {
        const unsigned short* v = reinterpret_cast<const unsigned short*>(vel) + 3 * s;
        const uint32_t u = __ldg(v), w = __ldg(v + 2), vv = __ldg(v + 1);
        const uint32_t h = s0 ? (uint32_t)__half_as_ushort(__ldg(s0 + s)) : 0u;
        return make_uint2(u | (vv << 16), w | (h << 16));
    }
    static __device__ __forceinline__ Cell zero() { return make_uint2(0u, 0u); }
    static __device__ __forceinline__ Ch4 widen(const Cell& c) {
        return Ch4{f2(__uint_as_float(c.x << 16), __uint_as_float(c.x & 0xFFFF0000u)),
                   f2(__uint_as_float(c.y << 16), __half2float(__ushort_as_half((unsigned short)(c.y >> 16))))};
    }
};

// Trilinear sample of the four channels at (x, y, z) (global voxel units): lerps along z, then y,
// then x (TrilinearSampler::sample, src/Utils/Stencils.hpp:118-153). I: the slot type of the
// leaf-table path.
template <typename T, typename I>
__device__ __forceinline__ Ch4 tile_sample(const typename T::Cell* __restrict__ tile, const TopoView& t, const LeafNbhd& L,
                                           const typename T::V* __restrict__ vel, const typename T::S* __restrict__ s0,
                                           float x, float y, float z, F2 one) {
    const int i = __float2int_rd(x), j = __float2int_rd(y), k = __float2int_rd(z);
    const float tx = x - (float)i, ty = y - (float)j, tz = z - (float)k;
    const int cx = i - (L.lx << 3) + kTileHalo, cy = j - (L.ly << 3) + kTileHalo, cz = k - (L.lz << 3) + kTileHalo;
    typename T::Cell c[8];
    if ((unsigned)cx <= (unsigned)(kTileSide - 2) && (unsigned)cy <= (unsigned)(kTileSide - 2) &&
        (unsigned)cz <= (unsigned)(kTileSide - 2)) {
        const typename T::Cell* b = tile + cx * T::kSX + cy * T::kSY + cz;
#pragma unroll
        for (int q = 0; q < 8; ++q) c[q] = b[(q >> 2) * T::kSX + ((q >> 1) & 1) * T::kSY + (q & 1)];
    } else {
        TapsT<I> tp;
        taps_at(tp, t, L, x, y, z);
#pragma unroll
        for (int q = 0; q < 8; ++q) c[q] = tp.s[q] < 0 ? T::zero() : T::read(vel, s0, (int64_t)tp.s[q]);
    }
    const F2 wx = f2(tx, tx), wy = f2(ty, ty), wz = f2(tz, tz);
    Ch4 h[2];
#pragma unroll
    for (int a = 0; a < 2; ++a) {
        const Ch4 v0 = T::widen(c[4 * a]), v1 = T::widen(c[4 * a + 1]), v2 = T::widen(c[4 * a + 2]), v3 = T::widen(c[4 * a + 3]);
        h[a].uv = lerp2(lerp2(v0.uv, v1.uv, wz, one), lerp2(v2.uv, v3.uv, wz, one), wy, one);
        h[a].ws = lerp2(lerp2(v0.ws, v1.ws, wz, one), lerp2(v2.ws, v3.ws, wz, one), wy, one);
    }
    return Ch4{lerp2(h[0].uv, h[1].uv, wx, one), lerp2(h[0].ws, h[1].ws, wx, one)};
}

template <typename T, typename I>
__global__ void __launch_bounds__(kTileThreads, T::kCtasPerSm)
    advect_tile_kernel(TopoView t, const typename T::V* __restrict__ vel, const typename T::S* __restrict__ s0,
                       typename T::V* __restrict__ vel_out, typename T::S* __restrict__ s0_out, float sdt, float one_arg) {
    __shared__ typename T::Cell tile[kTileSide * T::kSX];
    __shared__ LeafNbhd L;
    const F2 one = f2(one_arg, one_arg);  // 1 (mul_add2)
    const int64_t leaf = blockIdx.x;
    load_nbhd(L, t, leaf);
    __syncthreads();
    // The fill: every load of the thread's cells is issued before any is stored.
    typename T::Cell raw[kTileFill];
#pragma unroll
    for (int m = 0; m < kTileFill; ++m) {
        const int q = threadIdx.x + m * kTileThreads;
        raw[m] = T::zero();
        if (q < kTileCells) {
            const int lx = q / (kTileSide * kTileSide) - kTileHalo, ly = (q / kTileSide) % kTileSide - kTileHalo,
                      lz = q % kTileSide - kTileHalo;
            const int r = (lx < 0 ? 0 : lx > 7 ? 18 : 9) + (ly < 0 ? 0 : ly > 7 ? 6 : 3) + (lz < 0 ? 0 : lz > 7 ? 2 : 1);
            const int l = L.nb[r];
            if (l >= 0) raw[m] = T::read(vel, s0, ((int64_t)l << 9) | (((lx & 7) << 6) | ((ly & 7) << 3) | (lz & 7)));
        }
    }
#pragma unroll
    for (int m = 0; m < kTileFill; ++m) {
        const int q = threadIdx.x + m * kTileThreads;
        if (q < kTileCells)
            tile[(q / (kTileSide * kTileSide)) * T::kSX + ((q / kTileSide) % kTileSide) * T::kSY + q % kTileSide] = raw[m];
    }
    __syncthreads();
#pragma unroll 1
    for (int half = 0; half < 2; ++half) {
        const int n = (int)threadIdx.x + half * kTileThreads;
        const int a = n >> 6, b = (n >> 3) & 7, cz = n & 7;
        const int i = (L.lx << 3) + a, j = (L.ly << 3) + b, k = (L.lz << 3) + cz;
        const typename T::Cell* centre = tile + (a + kTileHalo) * T::kSX + (b + kTileHalo) * T::kSY + (cz + kTileHalo);
        const Ch4 o = T::widen(*centre);
        float ou, ov, ow, od;
        un2(o.uv, ou, ov), un2(o.ws, ow, od);
        const float bx = (float)i - ou * sdt, by = (float)j - ov * sdt, bz = (float)k - ow * sdt;
        const Ch4 f = tile_sample<T, I>(tile, t, L, vel, s0, bx, by, bz, one);
        float fu, fv, fw, fd;
        un2(f.uv, fu, fv), un2(f.ws, fw, fd);
        const Ch4 g = tile_sample<T, I>(tile, t, L, vel, s0, bx + fu * sdt, by + fv * sdt, bz + fw * sdt, one);
        // f + 0.5 (o - g)
        const F2 half2 = f2(0.5f, 0.5f);
        float cu, cv, cw, cd;
        un2(mul_add2(half2, sub2(o.uv, g.uv), f.uv, one), cu, cv);
        un2(mul_add2(half2, sub2(o.ws, g.ws), f.ws, one), cw, cd);
        // The clamp set: the centre, the six face neighbours and the forward sample.
        float mn[4], mx[4];
        constexpr int kOff[6] = {-T::kSX, T::kSX, -T::kSY, T::kSY, -1, 1};
        float e[6][4];
#pragma unroll
        for (int q = 0; q < 6; ++q) {
            const Ch4 w = T::widen(centre[kOff[q]]);
            un2(w.uv, e[q][0], e[q][1]), un2(w.ws, e[q][2], e[q][3]);
        }
        const float ov4[4] = {ou, ov, ow, od}, fv4[4] = {fu, fv, fw, fd}, cv4[4] = {cu, cv, cw, cd};
        float r[4];
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            mn[c] = min3(min3(ov4[c], e[0][c], e[1][c]), min3(e[2][c], e[3][c], e[4][c]), fminf(e[5][c], fv4[c]));
            mx[c] = max3(max3(ov4[c], e[0][c], e[1][c]), max3(e[2][c], e[3][c], e[4][c]), fmaxf(e[5][c], fv4[c]));
            r[c] = fmaxf(mn[c], fminf(cv4[c], mx[c]));
        }
        const int64_t s = (leaf << 9) + n;
        if (vel_out != nullptr) vstore(vel_out, s, make_float3(r[0], r[1], r[2]));
        if (s0_out != nullptr) sstore(s0_out, s, r[3]);
    }
}

}  // namespace dev
}  // namespace hns
