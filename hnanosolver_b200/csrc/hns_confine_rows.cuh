// Vorticity confinement (vorticityConfinement, src/Cuda/Kernel.cu:682-727) over half z-rows
// (hns_rows.cuh), for offsets |fs| <= 1, in two passes: |curl| of every voxel into an array, then per
// voxel its curl again, the gradient of |curl| from its neighbours' entries and the force.
//
// Bound by issue (two curls, a square root, three divisions a voxel), not by memory. A leaf tile in
// shared memory (1,728 staged velocities, 1,000 curls for a leaf's 512 voxels, one scalar load and
// shared store at a time) took 1.9 ms for 95.6M BF16 voxels and 97 us for 3.3M FP32 ones; a row's
// vector loads of its neighbour rows, twice, and one FP32 array more take 1.22 ms and 79 us. A face
// neighbour outside the domain has a curl too (of the voxels inside next to it): the rows that
// meet one compute it from single loads.
// The values and the order of every operation are the tile's.
#pragma once

#include "hns_rows.cuh"

namespace hns {
namespace dev {

// nbr27 entry of the leaf that holds local coordinates (a, b, d) in [-8, 15].
__device__ __forceinline__ int near_leaf(const int* __restrict__ nb, int a, int b, int d) {
    return __ldg(nb + ((a >> 3) + 1) * 9 + ((b >> 3) + 1) * 3 + ((d >> 3) + 1));
}

template <typename V>
__device__ __forceinline__ float3 near_vel(const int* __restrict__ nb, const V* __restrict__ vel, int a, int b, int d) {
    const int l = near_leaf(nb, a, b, d);
    return l < 0 ? make_float3(0.f, 0.f, 0.f) : vload(vel, ((int64_t)l << 9) + local_offset(a, b, d));
}

// |curl| times factor at local cell (a, b, d) of the leaf whose table is nb, any cell in [-1, 8].
template <typename V>
__device__ __forceinline__ float near_curl_mag(const int* __restrict__ nb, const V* __restrict__ vel, int a, int b, int d,
                                               float factor) {
    const float3 px = near_vel(nb, vel, a + 1, b, d), mx = near_vel(nb, vel, a - 1, b, d);
    const float3 py = near_vel(nb, vel, a, b + 1, d), my = near_vel(nb, vel, a, b - 1, d);
    const float3 pz = near_vel(nb, vel, a, b, d + 1), mz = near_vel(nb, vel, a, b, d - 1);
    const float ox = ((py.z - my.z) - (pz.y - mz.y)) * factor;
    const float oy = ((pz.x - mz.x) - (px.z - mx.z)) * factor;
    const float oz = ((px.y - mx.y) - (py.x - my.x)) * factor;
    return __fsqrt_rn(ox * ox + oy * oy + oz * oz);
}

// Curl times factor of the half row's voxels; u receives their velocities.
template <typename V>
__device__ __forceinline__ void half_row_curl(const HalfRow& r, const NbrRows& q, const V* __restrict__ vel, float factor,
                                              float3 u[4], float3 w[4]) {
    float3 xp[4], xm[4], yp[4], ym[4];
    vel_row<true>(vel, r.own, u);
    vel_row<true>(vel, q.xp, xp);
    vel_row<true>(vel, q.xm, xm);
    vel_row<true>(vel, q.yp, yp);
    vel_row<true>(vel, q.ym, ym);
    int64_t zin_s, zface_s;
    z_ends(r, zin_s, zface_s);
    const float3 zero = make_float3(0.f, 0.f, 0.f);
    const float3 zin = vload(vel, zin_s), zface = zface_s < 0 ? zero : vload(vel, zface_s);
    const float3 zlo = r.h ? zin : zface, zhi = r.h ? zface : zin;
#pragma unroll
    for (int z = 0; z < 4; ++z) {
        const float3 px = q.zxp ? zero : xp[z], mx = q.zxm ? zero : xm[z], py = q.zyp ? zero : yp[z], my = q.zym ? zero : ym[z];
        const float3 pz = z < 3 ? u[z < 3 ? z + 1 : 3] : zhi, mz = z > 0 ? u[z > 0 ? z - 1 : 0] : zlo;
        w[z] = make_float3(((py.z - my.z) - (pz.y - mz.y)) * factor, ((pz.x - mz.x) - (px.z - mx.z)) * factor,
                           ((px.y - mx.y) - (py.x - my.x)) * factor);
    }
}

__device__ __forceinline__ float curl_mag(const float3& w) { return __fsqrt_rn(w.x * w.x + w.y * w.y + w.z * w.z); }

template <typename V>
__global__ void __launch_bounds__(kRowThreads) curl_rows_kernel(TopoView t, const V* __restrict__ vel, float* __restrict__ mag,
                                                                float factor) {
    HalfRow r;
    if (!half_row(t, r, blockIdx.x)) return;
    const NbrRows q = nbr_rows(r);
    float3 u[4], w[4];
    half_row_curl(r, q, vel, factor, u, w);
    float m[4];
#pragma unroll
    for (int z = 0; z < 4; ++z) m[z] = curl_mag(w[z]);
    store_scalar_row<true>(mag, r.own, m);
}

// u + scale (N x omega) dt per voxel, then the step's velocity source, gravity and scalar sources
// (After, called with the row's first slot and its four velocities), into out.
template <typename V, typename After>
__global__ void __launch_bounds__(kRowThreads) confine_rows_kernel(TopoView t, const V* __restrict__ vel, V* __restrict__ out,
                                                                   const float* __restrict__ mag, float dt, float inv_dx,
                                                                   float scale, int fs, After after) {
    HalfRow r;
    if (!half_row(t, r, blockIdx.x)) return;
    const NbrRows q = nbr_rows(r);
    const float factor = 0.5f * inv_dx;
    float3 u[4], w[4];
    half_row_curl(r, q, vel, factor, u, w);
    float c[4], xp[4], xm[4], yp[4], ym[4], zlo, zhi;
    if (fs != 0) {
        const int* nb = t.nbr27 + r.leaf * 27;
        scalar_row<true>(mag, r.own, c);
        auto side = [&](bool missing, int64_t slot, int a, int b, float m[4]) {
            if (!missing) {
                scalar_row<true>(mag, slot, m);
            } else {
#pragma unroll
                for (int z = 0; z < 4; ++z) m[z] = near_curl_mag(nb, vel, a, b, 4 * r.h + z, factor);
            }
        };
        side(q.zxp, q.xp, r.a + 1, r.b, xp);
        side(q.zxm, q.xm, r.a - 1, r.b, xm);
        side(q.zyp, q.yp, r.a, r.b + 1, yp);
        side(q.zym, q.ym, r.a, r.b - 1, ym);
        int64_t zin_s, zface_s;
        z_ends(r, zin_s, zface_s);
        const float zin = __ldg(mag + zin_s);
        const float zface = zface_s >= 0 ? __ldg(mag + zface_s) : near_curl_mag(nb, vel, r.a, r.b, r.h ? 8 : -1, factor);
        zlo = r.h ? zin : zface, zhi = r.h ? zface : zin;
    }
#pragma unroll
    for (int z = 0; z < 4; ++z) {
        float px, mx, py, my, pz, mz;  // |curl| one voxel up and down each axis
        if (fs == 0) {
            px = mx = py = my = pz = mz = curl_mag(w[z]);
        } else {
            px = xp[z], mx = xm[z], py = yp[z], my = ym[z];
            pz = z < 3 ? c[z < 3 ? z + 1 : 3] : zhi, mz = z > 0 ? c[z > 0 ? z - 1 : 0] : zlo;
        }
        const bool up = fs >= 0;  // fs = -1: the samples trade places
        const float gx = ((up ? px : mx) - (up ? mx : px)) * 0.5f * inv_dx;
        const float gy = ((up ? py : my) - (up ? my : py)) * 0.5f * inv_dx;
        const float gz = ((up ? pz : mz) - (up ? mz : pz)) * 0.5f * inv_dx;
        const float glen = sqrtf(gx * gx + gy * gy + gz * gz) + 1e-5f;
        const float nx = gx / glen, ny = gy / glen, nz = gz / glen;
        const float ox = w[z].x, oy = w[z].y, oz = w[z].z;
        const float fx = scale * (ny * oz - nz * oy), fy = scale * (nz * ox - nx * oz), fz = scale * (nx * oy - ny * ox);
        u[z] = make_float3(u[z].x + fx * dt, u[z].y + fy * dt, u[z].z + fz * dt);
    }
    after(r.own, u);
    store_vel_row<true>(out, r.own, u);
}

// Both passes; `mag`: a float per voxel of scratch. All three arrays are the steps' own scratch, whose
// rows are 16-byte aligned.
template <typename V, typename After>
void launch_confine_rows(const Context& c, const V* vel, V* out, float* mag, float dt, float scale, int fs, const After& after) {
    const float inv_dx = 1.0f / c.dx;
    if (fs != 0) {
        curl_rows_kernel<V><<<row_blocks(c), kRowThreads, 0, c.stream>>>(c.topo.view, vel, mag, 0.5f * inv_dx);
        HNS_LAUNCHED();
    }
    confine_rows_kernel<V, After><<<row_blocks(c), kRowThreads, 0, c.stream>>>(c.topo.view, vel, out, mag, dt, inv_dx, scale, fs,
                                                                              after);
    HNS_LAUNCHED();
}

}  // namespace dev
}  // namespace hns
