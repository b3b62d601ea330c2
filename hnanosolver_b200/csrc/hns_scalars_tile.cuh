// HNS_Advance's multi-field advection (advect_scalars, src/Cuda/Kernel.cu:163-289) of up to five FP32
// fields from leaf tiles in shared memory: the back-trace uses the voxel's own velocity, the
// taps' weight-sum trilinear (setupInterpolation, Kernel.cu:204-233) reads slot 0 outside the
// domain, and the MacCormack correction is clamped to the centre, its six face neighbours and the
// forward sample. The operations of advect_scalars_kernel in its order, so the same bits.
//
// The gather form makes 24 loads of the velocity and 23 of each field a voxel, each with its own
// 64-bit address: bound by the load pipe and issue (313 us for four fields on 3.4M voxels, where the
// bytes need 24 us). Here the leaf and a one-voxel halo are read once into two tiles of 16-byte
// cells, (u, v, w, field 4) and fields 0..3, a missing leaf's cells as copies of slot 0, and each
// tap is one or two 16-byte shared-memory loads with the sums on pairs of fields.
#pragma once

#include "hns_advect_tile.cuh"

namespace hns {
namespace dev {

constexpr int kScalarsPerPass = 5;

struct ScalarPass {
    const float* in[kScalarsPerPass];
    float* out[kScalarsPerPass];
};

// kCount fields, the fifth beside the velocity.
template <int kCount>
struct ScalarCell {
    float4 v, f;
    static __device__ __forceinline__ ScalarCell read(const float* __restrict__ vel, const ScalarPass& P, int64_t s) {
        ScalarCell c;
        c.v = make_float4(__ldg(vel + 3 * s), __ldg(vel + 3 * s + 1), __ldg(vel + 3 * s + 2), kCount > 4 ? __ldg(P.in[4] + s) : 0.f);
        c.f = make_float4(__ldg(P.in[0] + s), kCount > 1 ? __ldg(P.in[1] + s) : 0.f, kCount > 2 ? __ldg(P.in[2] + s) : 0.f,
                          kCount > 3 ? __ldg(P.in[3] + s) : 0.f);
        return c;
    }
};

// Cell and trilinear weights of a trace's end (interp_setup's order).
__device__ __forceinline__ void trace_weights(float x, float y, float z, int& i0, int& j0, int& k0, float w[8]) {
    i0 = __float2int_rd(x), j0 = __float2int_rd(y), k0 = __float2int_rd(z);
    const float tx = x - (float)i0, ty = y - (float)j0, tz = z - (float)k0;
    const float itx = 1.0f - tx, ity = 1.0f - ty, itz = 1.0f - tz;
    const float w00 = itx * ity, w10 = tx * ity, w01 = itx * ty, w11 = tx * ty;
    w[0] = w00 * itz, w[1] = w10 * itz, w[2] = w01 * itz, w[3] = w11 * itz;
    w[4] = w00 * tz, w[5] = w10 * tz, w[6] = w01 * tz, w[7] = w11 * tz;
}

// The cell at floor(x), floor(y), floor(z) of a trace: its corners (x fastest, interp_setup's order)
// from the tiles, or through the leaf table when it is not in them, and the weights.
template <int kCount, bool kVelocity, typename I>
__device__ __forceinline__ void scalar_taps(const float4* __restrict__ tv, const float4* __restrict__ tf, const TopoView& t,
                                            const LeafNbhd& L, const float* __restrict__ vel, const ScalarPass& P, float x,
                                            float y, float z, float4 cv[8], float4 cf[8], float w[8]) {
    int i0, j0, k0;
    trace_weights(x, y, z, i0, j0, k0, w);
    const int cx = i0 - (L.lx << 3) + kTileHalo, cy = j0 - (L.ly << 3) + kTileHalo, cz = k0 - (L.lz << 3) + kTileHalo;
    if ((unsigned)cx <= (unsigned)(kTileSide - 2) && (unsigned)cy <= (unsigned)(kTileSide - 2) &&
        (unsigned)cz <= (unsigned)(kTileSide - 2)) {
        const int b = cx * TileF32::kSX + cy * TileF32::kSY + cz;
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            const int e = b + (q & 1) * TileF32::kSX + ((q >> 1) & 1) * TileF32::kSY + (q >> 2);
            cf[q] = tf[e];
            if constexpr (kVelocity || kCount > 4) cv[q] = tv[e];
        }
    } else {
        I idx[8];
        float unused[8];
        interp_setup_fast<I>(t, L, x, y, z, idx, unused);
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            const ScalarCell<kCount> c = ScalarCell<kCount>::read(vel, P, (int64_t)idx[q]);
            cf[q] = c.f, cv[q] = c.v;
        }
    }
}

template <int kCount, typename I>
__global__ void __launch_bounds__(kTileThreads, 3)
    advect_scalars_tile_kernel(TopoView t, const float* __restrict__ vel, ScalarPass P, float sdt) {
    extern __shared__ float4 tiles[];
    __shared__ LeafNbhd L;
    float4* tv = tiles;
    float4* tf = tiles + kTileSide * TileF32::kSX;
    const int64_t leaf = blockIdx.x;
    load_nbhd(L, t, leaf);
    __syncthreads();
    ScalarCell<kCount> raw[kTileFill];
#pragma unroll
    for (int m = 0; m < kTileFill; ++m) {
        const int q = min((int)threadIdx.x + m * kTileThreads, kTileCells - 1);
        const int lx = q / (kTileSide * kTileSide) - kTileHalo, ly = (q / kTileSide) % kTileSide - kTileHalo,
                  lz = q % kTileSide - kTileHalo;
        const int r = (lx < 0 ? 0 : lx > 7 ? 18 : 9) + (ly < 0 ? 0 : ly > 7 ? 6 : 3) + (lz < 0 ? 0 : lz > 7 ? 2 : 1);
        const int l = L.nb[r];
        // Outside the domain: slot 0.
        const int64_t s = l < 0 ? 0 : ((int64_t)l << 9) | (((lx & 7) << 6) | ((ly & 7) << 3) | (lz & 7));
        raw[m] = ScalarCell<kCount>::read(vel, P, s);
    }
#pragma unroll
    for (int m = 0; m < kTileFill; ++m) {
        const int q = (int)threadIdx.x + m * kTileThreads;
        if (q < kTileCells) {
            const int e = (q / (kTileSide * kTileSide)) * TileF32::kSX + ((q / kTileSide) % kTileSide) * TileF32::kSY + q % kTileSide;
            tv[e] = raw[m].v;
            tf[e] = raw[m].f;
        }
    }
    __syncthreads();
#pragma unroll 1
    for (int half = 0; half < 2; ++half) {
        const int n = (int)threadIdx.x + half * kTileThreads;
        const int a = n >> 6, b = (n >> 3) & 7, d = n & 7;
        const int i = (L.lx << 3) + a, j = (L.ly << 3) + b, k = (L.lz << 3) + d;
        const int centre = (a + kTileHalo) * TileF32::kSX + (b + kTileHalo) * TileF32::kSY + (d + kTileHalo);
        const float4 vc = tv[centre];
        const float bx = (float)i - vc.x * sdt, by = (float)j - vc.y * sdt, bz = (float)k - vc.z * sdt;
        float4 cv[8], cf[8];
        float w[8];
        float3 vf = make_float3(0.f, 0.f, 0.f);
        F2 pf[2] = {f2(0.f, 0.f), f2(0.f, 0.f)}, pb[2] = {pf[0], pf[0]};
        float pf4 = 0.f, pb4 = 0.f;
        scalar_taps<kCount, true, I>(tv, tf, t, L, vel, P, bx, by, bz, cv, cf, w);
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            vf.x = vf.x + cv[q].x * w[q];
            vf.y = vf.y + cv[q].y * w[q];
            vf.z = vf.z + cv[q].z * w[q];
            const F2 ww = f2(w[q], w[q]);
            pf[0] = fma2(f2(cf[q].x, cf[q].y), ww, pf[0]);
            if constexpr (kCount > 2) pf[1] = fma2(f2(cf[q].z, cf[q].w), ww, pf[1]);
            if constexpr (kCount > 4) pf4 = __fmaf_rn(cv[q].w, w[q], pf4);
        }
        scalar_taps<kCount, false, I>(tv, tf, t, L, vel, P, bx + vf.x * sdt, by + vf.y * sdt, bz + vf.z * sdt, cv, cf, w);
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            const F2 ww = f2(w[q], w[q]);
            pb[0] = fma2(f2(cf[q].x, cf[q].y), ww, pb[0]);
            if constexpr (kCount > 2) pb[1] = fma2(f2(cf[q].z, cf[q].w), ww, pb[1]);
            if constexpr (kCount > 4) pb4 = __fmaf_rn(cv[q].w, w[q], pb4);
        }
        constexpr int kOff[6] = {-TileF32::kSX, TileF32::kSX, -TileF32::kSY, TileF32::kSY, -1, 1};
        float4 e[6];
        float e4[6];
#pragma unroll
        for (int q = 0; q < 6; ++q) {
            e[q] = tf[centre + kOff[q]];
            e4[q] = kCount > 4 ? tv[centre + kOff[q]].w : 0.f;
        }
        const float4 fc = tf[centre];
        float f[5], g[5];
        un2(pf[0], f[0], f[1]), un2(pf[1], f[2], f[3]), f[4] = pf4;
        un2(pb[0], g[0], g[1]), un2(pb[1], g[2], g[3]), g[4] = pb4;
        const int64_t s = (leaf << 9) + n;
#pragma unroll
        for (int c = 0; c < kCount; ++c) {
            auto ch = [&](const float4& v, float v4) { return c == 0 ? v.x : c == 1 ? v.y : c == 2 ? v.z : c == 3 ? v.w : v4; };
            const float po = ch(fc, vc.w), corr = __fmaf_rn(0.5f, po - g[c], f[c]);
            const float mn = min3(min3(po, ch(e[0], e4[0]), ch(e[1], e4[1])), min3(ch(e[2], e4[2]), ch(e[3], e4[3]), ch(e[4], e4[4])),
                                  fminf(ch(e[5], e4[5]), f[c]));
            const float mx = max3(max3(po, ch(e[0], e4[0]), ch(e[1], e4[1])), max3(ch(e[2], e4[2]), ch(e[3], e4[3]), ch(e[4], e4[4])),
                                  fmaxf(ch(e[5], e4[5]), f[c]));
            P.out[c][s] = fmaxf(mn, fminf(corr, mx));
        }
    }
}

// ---- the same on FP16 fields along a BF16 velocity ---------------------------------------------
//
// A cell is the velocity and up to five fields in 16 bytes (u | v << 16, w | s4 << 16, s0 | s1 << 16,
// s2 | s3 << 16; absent fields 0), so a tap is one shared-memory load for all of them; sums in FP32,
// the clamp's bounds on the FP16 values themselves (exact). Bound by issue. Packed into such records
// in global memory by a pass of its own and gathered from there, four fields on 95.6M voxels took
// 0.58 + 2.45 ms and 16 bytes of scratch a voxel; from the tile they take 2.20 ms and none. Three CTAs
// an SM with more registers took 0.25 ms more than four.
struct HalfScalarPass {
    const __half* in[kScalarsPerPass];
    __half* out[kScalarsPerPass];
    int count;
};

template <int kCount>
__device__ __forceinline__ uint4 half_cell(const __nv_bfloat16* __restrict__ vel, const HalfScalarPass& P, int64_t s) {
    const unsigned short* v = reinterpret_cast<const unsigned short*>(vel) + 3 * s;
    uint32_t h[kScalarsPerPass];
#pragma unroll
    for (int c = 0; c < kScalarsPerPass; ++c) h[c] = c < kCount ? (uint32_t)__half_as_ushort(__ldg(P.in[c < kCount ? c : 0] + s)) : 0u;
    return make_uint4((uint32_t)__ldg(v) | ((uint32_t)__ldg(v + 1) << 16), (uint32_t)__ldg(v + 2) | (h[4] << 16),
                      h[0] | (h[1] << 16), h[2] | (h[3] << 16));
}

__device__ __forceinline__ float cell_u(const uint4& c) { return __uint_as_float(c.x << 16); }
__device__ __forceinline__ float cell_v(const uint4& c) { return __uint_as_float(c.x & 0xFFFF0000u); }
__device__ __forceinline__ float cell_w(const uint4& c) { return __uint_as_float(c.y << 16); }
__device__ __forceinline__ __half2 as_half2(uint32_t w) { return *reinterpret_cast<const __half2*>(&w); }
__device__ __forceinline__ F2 half2_f2(uint32_t w) {
    const float2 f = __half22float2(as_half2(w));
    return f2(f.x, f.y);
}

// The eight cells of a trace, from the tile or through the leaf table, and their weights.
template <int kCount, typename I>
__device__ __forceinline__ void half_taps(const uint4* __restrict__ tile, const TopoView& t, const LeafNbhd& L,
                                          const __nv_bfloat16* __restrict__ vel, const HalfScalarPass& P, float x, float y,
                                          float z, uint4 c[8], float w[8]) {
    int i0, j0, k0;
    trace_weights(x, y, z, i0, j0, k0, w);
    const int cx = i0 - (L.lx << 3) + kTileHalo, cy = j0 - (L.ly << 3) + kTileHalo, cz = k0 - (L.lz << 3) + kTileHalo;
    if ((unsigned)cx <= (unsigned)(kTileSide - 2) && (unsigned)cy <= (unsigned)(kTileSide - 2) &&
        (unsigned)cz <= (unsigned)(kTileSide - 2)) {
        const uint4* b = tile + cx * TileF32::kSX + cy * TileF32::kSY + cz;
#pragma unroll
        for (int q = 0; q < 8; ++q) c[q] = b[(q & 1) * TileF32::kSX + ((q >> 1) & 1) * TileF32::kSY + (q >> 2)];
    } else {
        I idx[8];
        float unused[8];
        interp_setup_fast<I>(t, L, x, y, z, idx, unused);
#pragma unroll
        for (int q = 0; q < 8; ++q) c[q] = half_cell<kCount>(vel, P, (int64_t)idx[q]);
    }
}

// Weighted sums of the eight cells' fields.
template <int kCount>
__device__ __forceinline__ void half_sums(const uint4 c[8], const float w[8], float s[5]) {
    F2 a = f2(0.f, 0.f), b = a;
    float e = 0.f;
#pragma unroll
    for (int q = 0; q < 8; ++q) {
        const F2 ww = f2(w[q], w[q]);
        a = fma2(half2_f2(c[q].z), ww, a);
        if constexpr (kCount > 2) b = fma2(half2_f2(c[q].w), ww, b);
        if constexpr (kCount > 4) e = __fmaf_rn(__half2float(__high2half(as_half2(c[q].y))), w[q], e);
    }
    un2(a, s[0], s[1]), un2(b, s[2], s[3]), s[4] = e;
}

template <int kCount, typename I>
__global__ void __launch_bounds__(kTileThreads, 4)
    advect_scalars_half_tile_kernel(TopoView t, const __nv_bfloat16* __restrict__ vel, HalfScalarPass P, float sdt) {
    __shared__ uint4 tile[kTileSide * TileF32::kSX];
    __shared__ LeafNbhd L;
    const int64_t leaf = blockIdx.x;
    load_nbhd(L, t, leaf);
    __syncthreads();
    uint4 raw[kTileFill];
#pragma unroll
    for (int m = 0; m < kTileFill; ++m) {
        const int q = min((int)threadIdx.x + m * kTileThreads, kTileCells - 1);
        const int lx = q / (kTileSide * kTileSide) - kTileHalo, ly = (q / kTileSide) % kTileSide - kTileHalo,
                  lz = q % kTileSide - kTileHalo;
        const int r = (lx < 0 ? 0 : lx > 7 ? 18 : 9) + (ly < 0 ? 0 : ly > 7 ? 6 : 3) + (lz < 0 ? 0 : lz > 7 ? 2 : 1);
        const int l = L.nb[r];
        // Outside the domain: slot 0.
        raw[m] = half_cell<kCount>(vel, P, l < 0 ? 0 : ((int64_t)l << 9) | (((lx & 7) << 6) | ((ly & 7) << 3) | (lz & 7)));
    }
#pragma unroll
    for (int m = 0; m < kTileFill; ++m) {
        const int q = (int)threadIdx.x + m * kTileThreads;
        if (q < kTileCells)
            tile[(q / (kTileSide * kTileSide)) * TileF32::kSX + ((q / kTileSide) % kTileSide) * TileF32::kSY + q % kTileSide] = raw[m];
    }
    __syncthreads();
#pragma unroll 1
    for (int half = 0; half < 2; ++half) {
        const int n = (int)threadIdx.x + half * kTileThreads;
        const int a = n >> 6, b = (n >> 3) & 7, d = n & 7;
        const int i = (L.lx << 3) + a, j = (L.ly << 3) + b, k = (L.lz << 3) + d;
        const uint4* centre = tile + (a + kTileHalo) * TileF32::kSX + (b + kTileHalo) * TileF32::kSY + (d + kTileHalo);
        const uint4 o = *centre;
        const float bx = (float)i - cell_u(o) * sdt, by = (float)j - cell_v(o) * sdt, bz = (float)k - cell_w(o) * sdt;
        uint4 c[8];
        float w[8], pf[5], pb[5];
        half_taps<kCount, I>(tile, t, L, vel, P, bx, by, bz, c, w);
        float3 vf = make_float3(0.f, 0.f, 0.f);
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            vf.x = vf.x + cell_u(c[q]) * w[q];
            vf.y = vf.y + cell_v(c[q]) * w[q];
            vf.z = vf.z + cell_w(c[q]) * w[q];
        }
        half_sums<kCount>(c, w, pf);
        half_taps<kCount, I>(tile, t, L, vel, P, bx + vf.x * sdt, by + vf.y * sdt, bz + vf.z * sdt, c, w);
        half_sums<kCount>(c, w, pb);
        // The clamp set, on the FP16 values: the centre and the six face neighbours.
        constexpr int kOff[6] = {-TileF32::kSX, TileF32::kSX, -TileF32::kSY, TileF32::kSY, -1, 1};
        __half2 mn[3] = {as_half2(o.z), as_half2(o.w), as_half2(o.y)}, mx[3] = {mn[0], mn[1], mn[2]};
#pragma unroll
        for (int q = 0; q < 6; ++q) {
            const uint4 e = centre[kOff[q]];
            const __half2 h[3] = {as_half2(e.z), as_half2(e.w), as_half2(e.y)};
#pragma unroll
            for (int g = 0; g < 3; ++g)
                if (g == 0 || (g == 1 && kCount > 2) || (g == 2 && kCount > 4)) mn[g] = __hmin2(mn[g], h[g]), mx[g] = __hmax2(mx[g], h[g]);
        }
        const int64_t s = (leaf << 9) + n;
        auto ch = [&](const __half2 v[3], int q) {
            return q == 0 ? __low2float(v[0]) : q == 1 ? __high2float(v[0]) : q == 2 ? __low2float(v[1]) : q == 3 ? __high2float(v[1])
                                                                                                              : __high2float(v[2]);
        };
        const __half2 oc[3] = {as_half2(o.z), as_half2(o.w), as_half2(o.y)};
#pragma unroll
        for (int q = 0; q < kCount; ++q) {
            const float corr = __fmaf_rn(0.5f, ch(oc, q) - pb[q], pf[q]);
            sstore(P.out[q], s, fmaxf(fminf(ch(mn, q), pf[q]), fminf(corr, fmaxf(ch(mx, q), pf[q]))));
        }
    }
}

}  // namespace dev
}  // namespace hns
