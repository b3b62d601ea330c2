// Adjoint (reverse-mode) kernels of the step's operators: MacCormack advection of a scalar
// and of the velocity, divergence, the red-black SOR solve from p = 0, gradient subtraction and
// vorticity confinement. Each computes the transpose of the derivative of its forward operator
// (hns_kernels.cu, hns_advance.cu) at the given inputs and ADDS it into the caller's adjoint
// arrays, so adjoints of several uses of one field accumulate.
//
// The derivatives are those of the forward arithmetic with exact real operations: the
// positions of a trace and the floor() of a trilinear sample are recomputed exactly as the
// forward computes them, and the MacCormack clamp routes the adjoint to the value it selected
// (the corrected value, or the minimum or maximum of the clamp set). Scatters (the transposes
// of trilinear samples and of the curl) use FP32 atomics; everything else is a gather.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>

#include "hns_confine.cuh"
#include "hns_internal.cuh"
#include "hns_stencil.cuh"

namespace hns {
namespace {

constexpr int kThreads = 256;

unsigned blocks_for(int64_t n) { return (unsigned)((n + kThreads - 1) / kThreads); }

__device__ __forceinline__ void coords_of(const TopoView& t, int64_t s, int& i, int& j, int& k) {
    const int4 o = t.origin[s >> 9];
    const int n = (int)(s & 511);
    i = o.x + ((n >> 6) & 7);
    j = o.y + ((n >> 3) & 7);
    k = o.z + (n & 7);
}

// Slot of the voxel at (i, j, k), -1 outside the domain (the dense leaf table).
__device__ __forceinline__ int64_t slot_at(const TopoView& t, int i, int j, int k) {
    const int li = (i >> 3) - t.lo_x, lj = (j >> 3) - t.lo_y, lk = (k >> 3) - t.lo_z;
    if (li < 0 || lj < 0 || lk < 0 || li >= t.dim_x || lj >= t.dim_y || lk >= t.dim_z) return -1;
    const int l = t.lookup[((int64_t)li * t.dim_y + lj) * t.dim_z + lk];
    return l < 0 ? -1 : ((int64_t)l << 9) + (((i & 7) << 6) | ((j & 7) << 3) | (k & 7));
}

__device__ __forceinline__ float val_s(const float* d, int64_t s) { return s < 0 ? 0.f : __ldg(d + s); }

__device__ __forceinline__ float dot3(float3 a, float3 b) { return a.x * b.x + a.y * b.y + a.z * b.z; }

// The clamp of MacCormack (advect_scalar / advect_vector): out = max(mn, min(corr, mx)) with
// mn/mx over {centre, 6 face neighbours, forward sample}. Returns which value the output is:
// -1 corr, 0 centre, 1..6 a neighbour (+x, -x, +y, -y, +z, -z), 7 the forward sample.
__device__ __forceinline__ int clamp_pick(float corr, float ctr, const float nbr[6], float fwd) {
    float mn = ctr, mx = ctr;
    int imn = 0, imx = 0;
#pragma unroll
    for (int q = 0; q < 6; ++q) {
        if (nbr[q] < mn) mn = nbr[q], imn = q + 1;
        if (nbr[q] > mx) mx = nbr[q], imx = q + 1;
    }
    if (fwd < mn) mn = fwd, imn = 7;
    if (fwd > mx) mx = fwd, imx = 7;
    if (corr > mx) return imx;
    if (corr < mn) return imn;
    return -1;
}

__device__ __forceinline__ void face_offset(int q, int& di, int& dj, int& dk) {
    di = q == 0 ? 1 : q == 1 ? -1 : 0;
    dj = q == 2 ? 1 : q == 3 ? -1 : 0;
    dk = q == 4 ? 1 : q == 5 ? -1 : 0;
}

// ---- advection ------------------------------------------------------------------------------

// The scalars of one reverse pass beside the velocity.
struct ScalarBars {
    const float* in[kMaxAdvectFields];
    const float* out_bar[kMaxAdvectFields];
    float* in_bar[kMaxAdvectFields];
    int count;
};

// Interleaves the velocity and the first scalar (0 without one) of a slot: one 16-byte gather per tap.
__global__ void __launch_bounds__(kThreads) pack_step_records_kernel(const float* __restrict__ vel,
                                                                     const float* __restrict__ s0,
                                                                     float4* __restrict__ in4, int64_t n) {
    const int64_t s = (int64_t)blockIdx.x * kThreads + threadIdx.x;
    if (s >= n) return;
    in4[s] = make_float4(__ldg(vel + 3 * s), __ldg(vel + 3 * s + 1), __ldg(vel + 3 * s + 2), s0 ? __ldg(s0 + s) : 0.f);
}

// Adjoint of advect_vector (vel_out_bar, null: none) and advect_scalar (every scalar of F) along
// one trace of vel: vel_bar += (d out / d vel)^T out_bar, through the advected velocity and through
// the trace, and in_bar += (d out / d in)^T out_bar per scalar. The positions of the trace, the
// samples and so the clamp decisions are the forward's (taps_at, tri_lerp). One thread per voxel.
//
// Bound by the scatters' L2 atomics: the taps' adjoints of the velocity and of the first scalar
// are one 16-byte vector reduction per tap into rec4 (fold_step_records_kernel adds it to the
// caller's arrays), the position adjoints of all fields are summed before the velocity's scatter,
// and the taps are gathered as 16-byte records (in4). Further scalars are scattered by themselves.
// On a 128^3 box with one scalar, the packing and the fold included: 776 -> 243 us against a launch
// per field with scalar atomics.
template <typename I>
__global__ void __launch_bounds__(kThreads) adj_advect_step_kernel(TopoView t, const float4* __restrict__ in4,
                                                                   const float* __restrict__ vel_out_bar, ScalarBars F,
                                                                   float4* __restrict__ rec4, float sdt) {
    __shared__ dev::LeafNbhd L;
    const dev::VoxelIdx vx = dev::voxel_of_block();
    dev::load_nbhd(L, t, vx.leaf);
    __syncthreads();
    const int i = (L.lx << 3) + (vx.n >> 6), j = (L.ly << 3) + ((vx.n >> 3) & 7), k = (L.lz << 3) + (vx.n & 7);
    const int64_t s = (vx.leaf << 9) + vx.n;
    const float4 o4 = __ldg(in4 + s);
    const float o[4] = {o4.x, o4.y, o4.z, o4.w};
    const float bx = (float)i - o[0] * sdt, by = (float)j - o[1] * sdt, bz = (float)k - o[2] * sdt;
    dev::TapsT<I> tb, tf;
    auto sample = [&](const dev::TapsT<I>& T, float r[4]) {
        float v[4][8];
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            const float4 a = T.s[q] < 0 ? make_float4(0.f, 0.f, 0.f, 0.f) : __ldg(in4 + T.s[q]);
            v[0][q] = a.x, v[1][q] = a.y, v[2][q] = a.z, v[3][q] = a.w;
        }
#pragma unroll
        for (int c = 0; c < 4; ++c) r[c] = dev::tri_lerp(T, v[c]);
    };
    float pf[4], pb[4];
    dev::taps_at(tb, t, L, bx, by, bz);
    sample(tb, pf);
    dev::taps_at(tf, t, L, bx + pf[0] * sdt, by + pf[1] * sdt, bz + pf[2] * sdt);
    sample(tf, pb);
    // Weight of tap q (index a*4 + b*2 + c) and its position derivatives.
    auto weight = [](const dev::TapsT<I>& T, int q) {
        return ((q & 4) ? T.tx : 1.f - T.tx) * ((q & 2) ? T.ty : 1.f - T.ty) * ((q & 1) ? T.tz : 1.f - T.tz);
    };
    auto grad = [](const dev::TapsT<I>& T, int q) {
        const float wx = (q & 4) ? T.tx : 1.f - T.tx, wy = (q & 2) ? T.ty : 1.f - T.ty, wz = (q & 1) ? T.tz : 1.f - T.tz;
        return make_float3(((q & 4) ? wy : -wy) * wz, ((q & 2) ? wx : -wx) * wz, ((q & 1) ? wx : -wx) * wy);
    };
    I ns[6];
    dev::face_slots(L, (I)s, vx.n, ns);  // -x, +x, -y, +y, -z, +z
    // The adjoints of the centre, the two samples and the clamp's neighbour of each component.
    float4 nbr4[6];
#pragma unroll
    for (int q = 0; q < 6; ++q) nbr4[q] = ns[q] < 0 ? make_float4(0.f, 0.f, 0.f, 0.f) : __ldg(in4 + ns[q]);
    auto route = [&](float ob, float po, float fwd_s, float back_s, const float nv[6], float& g_po, float& g_pf, float& g_pb) {
        const float corr = fwd_s + 0.5f * (po - back_s);
        const int pick = clamp_pick(corr, po, nv, fwd_s);
        g_po = g_pf = g_pb = 0.f;
        if (pick < 0) {
            g_pf = ob, g_po = 0.5f * ob, g_pb = -0.5f * ob;
        } else if (pick == 0) {
            g_po = ob;
        } else if (pick == 7) {
            g_pf = ob;
        } else {
            return pick - 1;
        }
        return -1;
    };
    float gpo[4], gpf[4], gpb[4];
#pragma unroll
    for (int c = 0; c < 4; ++c) {
        const float* ob_p = c < 3 ? vel_out_bar : F.count > 0 ? F.out_bar[0] : nullptr;
        const float ob = ob_p == nullptr ? 0.f : c < 3 ? __ldg(ob_p + 3 * s + c) : __ldg(ob_p + s);
        float nv[6];  // clamp_pick's order: +x, -x, +y, -y, +z, -z
#pragma unroll
        for (int q = 0; q < 6; ++q) {
            const float4 a = nbr4[q ^ 1];
            nv[q] = c == 0 ? a.x : c == 1 ? a.y : c == 2 ? a.z : a.w;
        }
        const int pick = route(ob, o[c], pf[c], pb[c], nv, gpo[c], gpf[c], gpb[c]);
        if (pick >= 0 && ob != 0.f) {
            I at = ns[1];
#pragma unroll
            for (int q = 1; q < 6; ++q) at = pick == q ? ns[q ^ 1] : at;
            if (at >= 0) atomicAdd(reinterpret_cast<float*>(rec4 + at) + c, ob);  // outside is the constant 0
        }
    }
    // The adjoint of a sample's position: the sum over its taps of (the samples' adjoints . the
    // tap's values) times the weight's gradient; fb at fwd, bb at back.
    float3 fb = make_float3(0.f, 0.f, 0.f), bb = make_float3(0.f, 0.f, 0.f);
    auto position = [&](const dev::TapsT<I>& T, const float g[4], float3& r) {
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            if (T.s[q] < 0) continue;
            const float4 a = __ldg(in4 + T.s[q]);
            float d = 0.f;
            if (g[0] != 0.f) d += g[0] * a.x;
            if (g[1] != 0.f) d += g[1] * a.y;
            if (g[2] != 0.f) d += g[2] * a.z;
            if (g[3] != 0.f) d += g[3] * a.w;
            const float3 w = grad(T, q);
            r.x += d * w.x, r.y += d * w.y, r.z += d * w.z;
        }
    };
    // The scalar shares the velocity's records but not its adjoint: where one of them has none, a trace of
    // a velocity that is not finite (weights NaN) adds nothing to it.
    auto part = [](float g, float w) { return g != 0.f ? g * w : 0.f; };
    auto nonzero = [](const float g[4]) { return g[0] != 0.f || g[1] != 0.f || g[2] != 0.f || g[3] != 0.f; };
    if (nonzero(gpb)) {
        position(tf, gpb, fb);
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            const float w = weight(tf, q);
            if (tf.s[q] >= 0) dev::red4(rec4 + tf.s[q], part(gpb[0], w), part(gpb[1], w), part(gpb[2], w), part(gpb[3], w));
        }
    }
    for (int c = 1; c < F.count; ++c) {
        const float ob = __ldg(F.out_bar[c] + s);
        if (ob == 0.f) continue;
        const float* __restrict__ d = F.in[c];
        float vb[8], vf[8], nv[6];
#pragma unroll
        for (int q = 0; q < 8; ++q) vb[q] = val_s(d, tb.s[q]), vf[q] = val_s(d, tf.s[q]);
#pragma unroll
        for (int q = 0; q < 6; ++q) nv[q] = val_s(d, ns[q ^ 1]);
        float g_po, g_pf, g_pb;
        const int pick = route(ob, __ldg(d + s), dev::tri_lerp(tb, vb), dev::tri_lerp(tf, vf), nv, g_po, g_pf, g_pb);
        if (pick >= 0) {
            I at = ns[1];
#pragma unroll
            for (int q = 1; q < 6; ++q) at = pick == q ? ns[q ^ 1] : at;
            if (at >= 0) atomicAdd(F.in_bar[c] + at, ob);
        }
        if (g_po != 0.f) atomicAdd(F.in_bar[c] + s, g_po);
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            const float3 wf = grad(tf, q), wb = grad(tb, q);
            if (g_pb != 0.f) {
                if (tf.s[q] >= 0) atomicAdd(F.in_bar[c] + tf.s[q], g_pb * weight(tf, q));
                fb.x += g_pb * vf[q] * wf.x, fb.y += g_pb * vf[q] * wf.y, fb.z += g_pb * vf[q] * wf.z;
            }
            if (g_pf != 0.f) {
                if (tb.s[q] >= 0) atomicAdd(F.in_bar[c] + tb.s[q], g_pf * weight(tb, q));
                bb.x += g_pf * vb[q] * wb.x, bb.y += g_pf * vb[q] * wb.y, bb.z += g_pf * vb[q] * wb.z;
            }
        }
    }
    // fwd = back + vf sdt: the forward sample of the velocity takes fwd_bar sdt, back takes fwd_bar.
    gpf[0] += fb.x * sdt, gpf[1] += fb.y * sdt, gpf[2] += fb.z * sdt;
    if (nonzero(gpf)) {
        position(tb, gpf, bb);
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            const float w = weight(tb, q);
            if (tb.s[q] >= 0) dev::red4(rec4 + tb.s[q], part(gpf[0], w), part(gpf[1], w), part(gpf[2], w), part(gpf[3], w));
        }
    }
    // back = x - vo sdt.
    bb.x += fb.x, bb.y += fb.y, bb.z += fb.z;
    dev::red4(rec4 + s, gpo[0] - sdt * bb.x, gpo[1] - sdt * bb.y, gpo[2] - sdt * bb.z, gpo[3]);
}

// Adds the records of adj_advect_step_kernel into the velocity's and the first scalar's adjoints.
__global__ void __launch_bounds__(kThreads) fold_step_records_kernel(const float4* __restrict__ rec4,
                                                                     float* __restrict__ vel_bar,
                                                                     float* __restrict__ in_bar, int64_t n) {
    const int64_t s = (int64_t)blockIdx.x * kThreads + threadIdx.x;
    if (s >= n) return;
    const float4 a = __ldg(rec4 + s);
    vel_bar[3 * s] += a.x;
    vel_bar[3 * s + 1] += a.y;
    vel_bar[3 * s + 2] += a.z;
    if (in_bar != nullptr) in_bar[s] += a.w;
}

// ---- projection -----------------------------------------------------------------------------

// Adjoint of divergence (a gather): vel_bar(s) += inv_dx / 2 (div_bar(s - e_d) - div_bar(s + e_d)).
__global__ void __launch_bounds__(kThreads) adj_divergence_kernel(TopoView t, const float* __restrict__ div_bar,
                                                                  float* __restrict__ vel_bar, float h, int64_t n) {
    const int64_t s = (int64_t)blockIdx.x * kThreads + threadIdx.x;
    if (s >= n) return;
    int i, j, k;
    coords_of(t, s, i, j, k);
    vel_bar[3 * s] += h * (val_s(div_bar, slot_at(t, i - 1, j, k)) - val_s(div_bar, slot_at(t, i + 1, j, k)));
    vel_bar[3 * s + 1] += h * (val_s(div_bar, slot_at(t, i, j - 1, k)) - val_s(div_bar, slot_at(t, i, j + 1, k)));
    vel_bar[3 * s + 2] += h * (val_s(div_bar, slot_at(t, i, j, k - 1)) - val_s(div_bar, slot_at(t, i, j, k + 1)));
}

// Adjoint of subtract_gradient (out = vel - grad p) with respect to p (a gather):
// p_bar(s) += inv_dx / 2 sum_d (out_bar_d(s + e_d) - out_bar_d(s - e_d)).
__global__ void __launch_bounds__(kThreads) adj_gradient_kernel(TopoView t, const float* __restrict__ out_bar,
                                                                float* __restrict__ p_bar, float h, int64_t n) {
    const int64_t s = (int64_t)blockIdx.x * kThreads + threadIdx.x;
    if (s >= n) return;
    int i, j, k;
    coords_of(t, s, i, j, k);
    auto ob = [&](int64_t q, int c) { return q < 0 ? 0.f : __ldg(out_bar + 3 * q + c); };
    const float g = (ob(slot_at(t, i + 1, j, k), 0) - ob(slot_at(t, i - 1, j, k), 0)) +
                    (ob(slot_at(t, i, j + 1, k), 1) - ob(slot_at(t, i, j - 1, k), 1)) +
                    (ob(slot_at(t, i, j, k + 1), 2) - ob(slot_at(t, i, j, k - 1), 2));
    p_bar[s] += h * g;
}

// Adjoint of one colour-c half-sweep of redBlackGaussSeidelUpdate, in place on lam. The forward
// half-sweep sets p(c) = (1 - omega) p(c) + omega / 6 (sum of the neighbours - div dx^2) on
// colour c and keeps colour c'; its transpose, from the adjoint lam' after it, gives
//   lam(c') = lam'(c') + omega / 6 sum of the (colour c) neighbours of lam',
//   div_bar(c) -= dx^2 omega / 6 lam'(c),   lam(c) = (1 - omega) lam'(c).
// The last factor is uniform over a colour, so the caller keeps it as a scale per colour: the
// true lam is scale_colour x the stored values. This launch writes colour c' fully scaled
// (keep = the old scale of c', nbr = omega / 6 x the scale of c) and only reads colour c, so it
// runs in place; the caller then sets the scale of c' to 1 and multiplies that of c by
// (1 - omega).
//
// One thread per z-row of a leaf (64 per leaf, 4 leaves per CTA): it loads its row and the four
// x/y neighbour rows as 32-byte vectors (the neighbour leaf's row across a face, zeros for a
// missing leaf) and the two values across the z faces, updates the 4 voxels of colour c' and
// stores them one by one (the row's colour-c values are read by other threads), and updates
// div_bar on the 4 voxels of colour c of its row, which only it touches.
constexpr int kRowLeavesPerBlock = 4;

__device__ __forceinline__ void ld_row(const float* __restrict__ p, float v[8]) {
    const float4 lo = *reinterpret_cast<const float4*>(p), hi = *reinterpret_cast<const float4*>(p + 4);
    v[0] = lo.x, v[1] = lo.y, v[2] = lo.z, v[3] = lo.w, v[4] = hi.x, v[5] = hi.y, v[6] = hi.z, v[7] = hi.w;
}

__global__ void __launch_bounds__(64 * kRowLeavesPerBlock) adj_rbgs_colour_kernel(TopoView t, float* lam,
                                                                                  float* __restrict__ div_bar,
                                                                                  int colour, float keep, float nbr,
                                                                                  float dmul) {
    const int64_t leaf = (int64_t)blockIdx.x * kRowLeavesPerBlock + (threadIdx.x >> 6);
    if (leaf >= t.num_leaves) return;
    const int r = threadIdx.x & 63, a = r >> 3, b = r & 7;
    const int* nb = t.nbr27 + leaf * 27;
    // nbr27: (dx+1)*9 + (dy+1)*3 + (dz+1); entry 13 is the leaf itself.
    const int nx = __ldg(nb + (a == 7 ? 22 : a == 0 ? 4 : 13)), ny = __ldg(nb + (b == 7 ? 16 : b == 0 ? 10 : 13));
    const int nzm = __ldg(nb + 12), nzp = __ldg(nb + 14);
    const int64_t own = (leaf << 9) + 8 * r;
    // Rows (a +- 1, b) and (a, b +- 1): in this leaf, or across the face (missing: this row, zeroed).
    auto across = [&](int n, int row) -> int64_t { return n < 0 ? own : ((int64_t)n << 9) + 8 * row; };
    const int64_t oxp = a < 7 ? own + 64 : across(nx, b), oxm = a > 0 ? own - 64 : across(nx, 56 + b);
    const int64_t oyp = b < 7 ? own + 8 : across(ny, 8 * a), oym = b > 0 ? own - 8 : across(ny, 8 * a + 7);
    const bool zxp = a == 7 && nx < 0, zxm = a == 0 && nx < 0, zyp = b == 7 && ny < 0, zym = b == 0 && ny < 0;
    float c[8], xp[8], xm[8], yp[8], ym[8];
    ld_row(lam + own, c);
    ld_row(lam + oxp, xp);
    ld_row(lam + oxm, xm);
    ld_row(lam + oyp, yp);
    ld_row(lam + oym, ym);
    const float zlo = nzm < 0 ? 0.f : lam[((int64_t)nzm << 9) + 8 * r + 7];
    const float zhi = nzp < 0 ? 0.f : lam[((int64_t)nzp << 9) + 8 * r];
    float d[8];
    ld_row(div_bar + own, d);
    const int pc = (a + b + colour) & 1;  // z parity of colour c in this row
#pragma unroll
    for (int z = 0; z < 8; ++z) {
        if ((z & 1) == pc) {
            d[z] -= dmul * c[z];
        } else {
            const float sx = (zxp ? 0.f : xp[z]) + (zxm ? 0.f : xm[z]);
            const float sy = (zyp ? 0.f : yp[z]) + (zym ? 0.f : ym[z]);
            const float sz = (z < 7 ? c[z + 1] : zhi) + (z > 0 ? c[z - 1] : zlo);
            lam[own + z] = keep * c[z] + nbr * (sx + sy + sz);
        }
    }
    *reinterpret_cast<float4*>(div_bar + own) = make_float4(d[0], d[1], d[2], d[3]);
    *reinterpret_cast<float4*>(div_bar + own + 4) = make_float4(d[4], d[5], d[6], d[7]);
}

// ---- vorticity confinement ------------------------------------------------------------------

__device__ __forceinline__ float3 ldv(const float* vel, int64_t q) {
    return q < 0 ? make_float3(0.f, 0.f, 0.f) : make_float3(__ldg(vel + 3 * q), __ldg(vel + 3 * q + 1), __ldg(vel + 3 * q + 2));
}

// Curl at (i, j, k) from its six face neighbours (computeVorticityMag's differences).
__device__ __forceinline__ float3 curl_at(const TopoView& t, const float* vel, int i, int j, int k, float f) {
    const float3 px = ldv(vel, slot_at(t, i + 1, j, k)), mx = ldv(vel, slot_at(t, i - 1, j, k));
    const float3 py = ldv(vel, slot_at(t, i, j + 1, k)), my = ldv(vel, slot_at(t, i, j - 1, k));
    const float3 pz = ldv(vel, slot_at(t, i, j, k + 1)), mz = ldv(vel, slot_at(t, i, j, k - 1));
    return make_float3(((py.z - my.z) - (pz.y - mz.y)) * f, ((pz.x - mz.x) - (px.z - mx.z)) * f,
                       ((px.y - mx.y) - (py.x - my.x)) * f);
}

__device__ __forceinline__ void add_v(float* bar, int64_t q, int c, float a) {
    if (q >= 0 && a != 0.f) atomicAdd(bar + 3 * q + c, a);
}

// Transpose of the curl at (i, j, k): scatters the adjoint w of the curl into vel_bar.
__device__ __forceinline__ void curl_adjoint(const TopoView& t, float* vel_bar, int i, int j, int k, float3 w, float f) {
    const int64_t px = slot_at(t, i + 1, j, k), mx = slot_at(t, i - 1, j, k);
    const int64_t py = slot_at(t, i, j + 1, k), my = slot_at(t, i, j - 1, k);
    const int64_t pz = slot_at(t, i, j, k + 1), mz = slot_at(t, i, j, k - 1);
    add_v(vel_bar, py, 2, w.x * f), add_v(vel_bar, my, 2, -w.x * f);
    add_v(vel_bar, pz, 1, -w.x * f), add_v(vel_bar, mz, 1, w.x * f);
    add_v(vel_bar, pz, 0, w.y * f), add_v(vel_bar, mz, 0, -w.y * f);
    add_v(vel_bar, px, 2, -w.y * f), add_v(vel_bar, mx, 2, w.y * f);
    add_v(vel_bar, px, 1, w.z * f), add_v(vel_bar, mx, 1, -w.z * f);
    add_v(vel_bar, py, 0, -w.z * f), add_v(vel_bar, my, 0, w.z * f);
}

// Adjoint of vorticityConfinement: out = vel + dt scale (N x omega), N = g / (|g| + 1e-5),
// g = (|omega| at +-fs along each axis) differences * inv_dx / 2, omega = curl * inv_dx / 2.
__global__ void __launch_bounds__(kThreads) adj_confinement_kernel(TopoView t, const float* __restrict__ vel,
                                                                   const float* __restrict__ out_bar,
                                                                   float* __restrict__ vel_bar, float dt, float inv_dx,
                                                                   float scale, int fs, int64_t n) {
    const int64_t s = (int64_t)blockIdx.x * kThreads + threadIdx.x;
    if (s >= n) return;
    const float3 ob = make_float3(__ldg(out_bar + 3 * s), __ldg(out_bar + 3 * s + 1), __ldg(out_bar + 3 * s + 2));
    atomicAdd(vel_bar + 3 * s, ob.x);
    atomicAdd(vel_bar + 3 * s + 1, ob.y);
    atomicAdd(vel_bar + 3 * s + 2, ob.z);
    // Offset 0 (|factor_scale| < 1): both |omega| samples are the same voxel, the gradient is
    // identically 0 and so is the force; the terms below would cancel only up to rounding.
    if (fs == 0 || (ob.x == 0.f && ob.y == 0.f && ob.z == 0.f)) return;
    int i, j, k;
    coords_of(t, s, i, j, k);
    const float f = 0.5f * inv_dx;
    const float3 w = curl_at(t, vel, i, j, k, f);
    // |omega| at the six offset voxels (+x, -x, +y, -y, +z, -z), which may lie outside the domain.
    float3 wv[6];
    float m[6];
#pragma unroll
    for (int q = 0; q < 6; ++q) {
        int di, dj, dk;
        face_offset(q, di, dj, dk);
        wv[q] = curl_at(t, vel, i + fs * di, j + fs * dj, k + fs * dk, f);
        m[q] = sqrtf(dot3(wv[q], wv[q]));
    }
    const float3 g = make_float3((m[0] - m[1]) * f, (m[2] - m[3]) * f, (m[4] - m[5]) * f);
    const float gn = sqrtf(dot3(g, g));
    const float glen = gn + 1e-5f;
    const float3 N = make_float3(g.x / glen, g.y / glen, g.z / glen);
    // f = scale (N x omega); out_bar . (dt f).
    const float3 fb = make_float3(ob.x * dt * scale, ob.y * dt * scale, ob.z * dt * scale);
    // d(N x w) = dN x w + N x dw:  N_bar = w x fb, w_bar = fb x N.
    const float3 Nb = make_float3(w.y * fb.z - w.z * fb.y, w.z * fb.x - w.x * fb.z, w.x * fb.y - w.y * fb.x);
    const float3 wb = make_float3(fb.y * N.z - fb.z * N.y, fb.z * N.x - fb.x * N.z, fb.x * N.y - fb.y * N.x);
    curl_adjoint(t, vel_bar, i, j, k, wb, f);
    // N = g / glen: g_bar = N_bar / glen - g (N_bar . g) / (glen^2 |g|).
    float3 gb = make_float3(Nb.x / glen, Nb.y / glen, Nb.z / glen);
    if (gn > 0.f) {
        const float c = dot3(Nb, g) / (glen * glen * gn);
        gb.x -= c * g.x, gb.y -= c * g.y, gb.z -= c * g.z;
    }
    const float mb[6] = {gb.x * f, -gb.x * f, gb.y * f, -gb.y * f, gb.z * f, -gb.z * f};
#pragma unroll
    for (int q = 0; q < 6; ++q) {
        if (m[q] <= 0.f || mb[q] == 0.f) continue;
        int di, dj, dk;
        face_offset(q, di, dj, dk);
        const float r = mb[q] / m[q];
        curl_adjoint(t, vel_bar, i + fs * di, j + fs * dj, k + fs * dk, make_float3(r * wv[q].x, r * wv[q].y, r * wv[q].z), f);
    }
}

// The same for fs = 1 or -1 as gathers, in three passes without atomics (the scatter form above
// makes 84 of them a voxel). With w_bar(t) the adjoint of the curl at t,
//   1. per voxel s: gb(s), the adjoint of the gradient of |omega|, and wb(s) = fb x N, the part of
//      w_bar(s) that comes from N x omega;
//   2. per voxel t: w_bar(t) = wb(t) + f omega(t) / |omega(t)| sum over the axes of
//      gb_d(t - fs e_d) - gb_d(t + fs e_d), the adjoint of |omega(t)| as its neighbours read it;
//   3. per voxel u: vel_bar(u) += out_bar(u) + the transpose of the curl at u's face neighbours.
// A face neighbour outside the domain has a curl too (its own neighbours inside make it), with
// wb = 0: pass 3 computes its w_bar from gb where it meets one.
// 28,103 leaves: 3.0 -> 1.0 ms.
__global__ void __launch_bounds__(kThreads) adj_confine_force_kernel(TopoView t, const float* __restrict__ vel,
                                                                     const float* __restrict__ out_bar,
                                                                     float* __restrict__ wb_out, float* __restrict__ gb_out,
                                                                     float dt, float inv_dx, float scale, int fs) {
    __shared__ dev::LeafNbhd L;
    __shared__ dev::ConfineTile T;
    const int64_t leaf = blockIdx.x;
    dev::load_nbhd(L, t, leaf);
    __syncthreads();
    const float f = 0.5f * inv_dx;
    dev::confine_tile(L, vel, T, f);
    for (int n = threadIdx.x; n < 512; n += kThreads) {
        const int a = n >> 6, b = (n >> 3) & 7, d = n & 7, c = dev::conf_wi(a, b, d);
        const int64_t s = (leaf << 9) + n;
        const float3 ob = dev::ld3(out_bar, s);
        if (ob.x == 0.f && ob.y == 0.f && ob.z == 0.f) {  // no adjoint, whatever the velocity (0 times infinity is not 0)
            dev::st3(wb_out, s, make_float3(0.f, 0.f, 0.f));
            dev::st3(gb_out, s, make_float3(0.f, 0.f, 0.f));
            continue;
        }
        const float3 w = make_float3(T.w[0][c], T.w[1][c], T.w[2][c]);
        const float3 g = make_float3((T.m[dev::conf_wi(a + fs, b, d)] - T.m[dev::conf_wi(a - fs, b, d)]) * f,
                                     (T.m[dev::conf_wi(a, b + fs, d)] - T.m[dev::conf_wi(a, b - fs, d)]) * f,
                                     (T.m[dev::conf_wi(a, b, d + fs)] - T.m[dev::conf_wi(a, b, d - fs)]) * f);
        const float gn = sqrtf(dot3(g, g)), glen = gn + 1e-5f;
        const float3 N = make_float3(g.x / glen, g.y / glen, g.z / glen);
        const float3 fb = make_float3(ob.x * dt * scale, ob.y * dt * scale, ob.z * dt * scale);
        const float3 Nb = make_float3(w.y * fb.z - w.z * fb.y, w.z * fb.x - w.x * fb.z, w.x * fb.y - w.y * fb.x);
        dev::st3(wb_out, s, make_float3(fb.y * N.z - fb.z * N.y, fb.z * N.x - fb.x * N.z, fb.x * N.y - fb.y * N.x));
        float3 gb = make_float3(Nb.x / glen, Nb.y / glen, Nb.z / glen);
        if (gn > 0.f) {
            const float q = dot3(Nb, g) / (glen * glen * gn);
            gb.x -= q * g.x, gb.y -= q * g.y, gb.z -= q * g.z;
        }
        dev::st3(gb_out, s, gb);
    }
}

// omega / |omega| times the adjoint of |omega|, from the six face neighbours' slots (-x, +x, ...; -1
// outside): pass 2's second term.
__device__ __forceinline__ float3 magnitude_part(const float* __restrict__ vel, const float* __restrict__ gb,
                                                 const int64_t ns[6], float f, int fs) {
    float3 v[6];
#pragma unroll
    for (int q = 0; q < 6; ++q) v[q] = ldv(vel, ns[q]);
    const float3 w = make_float3(((v[3].z - v[2].z) - (v[5].y - v[4].y)) * f, ((v[5].x - v[4].x) - (v[1].z - v[0].z)) * f,
                                 ((v[1].y - v[0].y) - (v[3].x - v[2].x)) * f);
    const float m = sqrtf(dot3(w, w));
    auto at = [&](int64_t q, int c) { return q < 0 ? 0.f : __ldg(gb + 3 * q + c); };
    const float sum = (at(ns[0], 0) - at(ns[1], 0)) + (at(ns[2], 1) - at(ns[3], 1)) + (at(ns[4], 2) - at(ns[5], 2));
    if (m <= 0.f || sum == 0.f) return make_float3(0.f, 0.f, 0.f);  // no neighbour has an adjoint: 0 for any omega
    const float r = (fs > 0 ? sum : -sum) * f / m;
    return make_float3(r * w.x, r * w.y, r * w.z);
}

__global__ void __launch_bounds__(kThreads) adj_confine_curl_kernel(TopoView t, const float* __restrict__ vel,
                                                                    const float* __restrict__ gb, float* __restrict__ wb,
                                                                    float f, int fs) {
    __shared__ dev::LeafNbhd L;
    const dev::VoxelIdx v = dev::voxel_of_block();
    dev::load_nbhd(L, t, v.leaf);
    __syncthreads();
    const int64_t s = (v.leaf << 9) + v.n;
    int64_t ns[6];
    dev::face_slots(L, s, v.n, ns);
    const float3 r = magnitude_part(vel, gb, ns, f, fs);
    wb[3 * s] += r.x;
    wb[3 * s + 1] += r.y;
    wb[3 * s + 2] += r.z;
}

__global__ void __launch_bounds__(kThreads) adj_confine_gather_kernel(TopoView t, const float* __restrict__ vel,
                                                                      const float* __restrict__ out_bar,
                                                                      const float* __restrict__ gb,
                                                                      const float* __restrict__ wb,
                                                                      float* __restrict__ vel_bar, float f, int fs) {
    __shared__ dev::LeafNbhd L;
    const dev::VoxelIdx v = dev::voxel_of_block();
    dev::load_nbhd(L, t, v.leaf);
    __syncthreads();
    const int i = (L.lx << 3) + (v.n >> 6), j = (L.ly << 3) + ((v.n >> 3) & 7), k = (L.lz << 3) + (v.n & 7);
    const int64_t s = (v.leaf << 9) + v.n;
    int64_t ns[6];
    dev::face_slots(L, s, v.n, ns);
    float3 w[6];  // w_bar at -x, +x, -y, +y, -z, +z
#pragma unroll
    for (int q = 0; q < 6; ++q) {
        if (ns[q] >= 0) {
            w[q] = dev::ld3(wb, ns[q]);
            continue;
        }
        int di, dj, dk;
        face_offset(q ^ 1, di, dj, dk);  // face_offset's order is +x, -x, ...
        int64_t around[6];
#pragma unroll
        for (int o = 0; o < 6; ++o) {
            int ei, ej, ek;
            face_offset(o ^ 1, ei, ej, ek);
            around[o] = slot_at(t, i + di + ei, j + dj + ej, k + dk + ek);
        }
        w[q] = magnitude_part(vel, gb, around, f, fs);
    }
    const float3 ob = dev::ld3(out_bar, s);
    vel_bar[3 * s] += ob.x + f * ((w[4].y - w[5].y) - (w[2].z - w[3].z));
    vel_bar[3 * s + 1] += ob.y + f * ((w[0].z - w[1].z) - (w[4].x - w[5].x));
    vel_bar[3 * s + 2] += ob.z + f * ((w[2].x - w[3].x) - (w[0].y - w[1].y));
}

__global__ void __launch_bounds__(kThreads) accumulate_kernel(const float* __restrict__ src, float* __restrict__ dst,
                                                              int64_t n) {
    const int64_t s = (int64_t)blockIdx.x * kThreads + threadIdx.x;
    if (s < n) dst[s] += __ldg(src + s);
}

}  // namespace

// The adjoints' scratch block of 8 n floats: lam, p_bar and div_bar of the projection, then the
// records of the advection that follows it.
float* adj_scratch(Context& c) { return c.scratch_f32("adjoint_work", 8 * (size_t)c.num_voxels()); }

// That block where the context has it, else `floats` n of scratch: a projection or a confinement that is
// differentiated alone needs no records. (The block is not made from the smaller one by growing it, which
// would free what a captured call uses.)
float* adj_scratch(Context& c, const char* own, size_t floats) {
    const auto block = c.scratch.find("adjoint_work");
    return block != c.scratch.end() && block->second.ptr ? adj_scratch(c)
                                                         : c.scratch_f32(own, floats * (size_t)c.num_voxels());
}

void launch_adj_accumulate(const Context& c, const float* src, float* dst, int64_t n) {
    if (n <= 0) return;
    accumulate_kernel<<<blocks_for(n), kThreads, 0, c.stream>>>(src, dst, n);
    HNS_LAUNCHED();
}

void launch_adj_advect(Context& c, const float* vel, const float* vel_out_bar, const float* const* in,
                       const float* const* out_bar, float* const* in_bar, int nscalars, float* vel_bar, float dt,
                       float* work) {
    const int64_t n = c.num_voxels();
    if (n == 0) return;
    if (work == nullptr) work = adj_scratch(c);
    auto* rec4 = reinterpret_cast<float4*>(work);
    auto* in4 = rec4 + n;
    int base = 0;
    do {
        ScalarBars f{};
        f.count = std::min(kMaxAdvectFields, nscalars - base);
        for (int q = 0; q < f.count; ++q)
            f.in[q] = in[base + q], f.out_bar[q] = out_bar[base + q], f.in_bar[q] = in_bar[base + q];
        pack_step_records_kernel<<<blocks_for(n), kThreads, 0, c.stream>>>(vel, f.count > 0 ? f.in[0] : nullptr, in4, n);
        HNS_LAUNCHED();
        HNS_CUDA(cudaMemsetAsync(rec4, 0, sizeof(float4) * (size_t)n, c.stream));
        const unsigned blocks = (unsigned)(2 * c.topo.num_leaves);
        const float sdt = dt * (1.0f / c.dx);
        if (c.topo.num_leaves < (int64_t(1) << 22))
            adj_advect_step_kernel<int32_t><<<blocks, kThreads, 0, c.stream>>>(c.topo.view, in4, vel_out_bar, f, rec4, sdt);
        else
            adj_advect_step_kernel<int64_t><<<blocks, kThreads, 0, c.stream>>>(c.topo.view, in4, vel_out_bar, f, rec4, sdt);
        HNS_LAUNCHED();
        fold_step_records_kernel<<<blocks_for(n), kThreads, 0, c.stream>>>(rec4, vel_bar, f.count > 0 ? f.in_bar[0] : nullptr,
                                                                           n);
        HNS_LAUNCHED();
        vel_out_bar = nullptr;  // further scalars' passes
        base += f.count;
    } while (base < nscalars);
}

void launch_adj_divergence(const Context& c, const float* div_bar, float* vel_bar) {
    const int64_t n = c.num_voxels();
    if (n == 0) return;
    adj_divergence_kernel<<<blocks_for(n), kThreads, 0, c.stream>>>(c.topo.view, div_bar, vel_bar, 0.5f / c.dx, n);
    HNS_LAUNCHED();
}

void launch_adj_gradient(const Context& c, const float* out_bar, float* p_bar) {
    const int64_t n = c.num_voxels();
    if (n == 0) return;
    adj_gradient_kernel<<<blocks_for(n), kThreads, 0, c.stream>>>(c.topo.view, out_bar, p_bar, 0.5f / c.dx, n);
    HNS_LAUNCHED();
}

void launch_adj_rbgs_colour(const Context& c, float* lam, float* div_bar, int colour, float keep, float nbr, float dmul) {
    const int64_t L = c.topo.num_leaves;
    if (L == 0) return;
    adj_rbgs_colour_kernel<<<(unsigned)((L + kRowLeavesPerBlock - 1) / kRowLeavesPerBlock), 64 * kRowLeavesPerBlock, 0,
                             c.stream>>>(c.topo.view, lam, div_bar, colour, keep, nbr, dmul);
    HNS_LAUNCHED();
}

void launch_adj_confinement(Context& c, const float* vel, const float* out_bar, float* vel_bar, float dt, float scale,
                            float factor_scale, float* work) {
    const int64_t n = c.num_voxels();
    if (n == 0) return;
    const int fs = (int)factor_scale;
    if (fs == 1 || fs == -1) {
        if (work == nullptr) work = adj_scratch(c, "adjoint_confinement_work", 6);
        float *wb = work, *gb = work + 3 * n;
        const float f = 0.5f * (1.0f / c.dx);
        adj_confine_force_kernel<<<(unsigned)c.topo.num_leaves, kThreads, 0, c.stream>>>(c.topo.view, vel, out_bar, wb, gb, dt,
                                                                                         1.0f / c.dx, scale, fs);
        HNS_LAUNCHED();
        adj_confine_curl_kernel<<<(unsigned)(2 * c.topo.num_leaves), kThreads, 0, c.stream>>>(c.topo.view, vel, gb, wb, f, fs);
        HNS_LAUNCHED();
        adj_confine_gather_kernel<<<(unsigned)(2 * c.topo.num_leaves), kThreads, 0, c.stream>>>(c.topo.view, vel, out_bar, gb,
                                                                                                wb, vel_bar, f, fs);
        HNS_LAUNCHED();
        return;
    }
    adj_confinement_kernel<<<blocks_for(n), kThreads, 0, c.stream>>>(c.topo.view, vel, out_bar, vel_bar, dt, 1.0f / c.dx,
                                                                     scale, fs, n);
    HNS_LAUNCHED();
}

}  // namespace hns

// ---- C ABI -----------------------------------------------------------------------------------

namespace hns {

// The adjoint of `iterations` red-black iterations from p = 0 (the forward's
// HNS_SOLVE_ZERO_INIT): the half-sweeps' transposes in reverse order, black first, in place on
// a copy of p_bar with one scale per colour (adj_rbgs_colour_kernel). The adjoint with respect
// to the initial p is not needed (p starts at 0), so lam is never rescaled at the end.
void adj_rbgs(Context& c, const float* p_bar, float* div_bar, int iterations, float omega, float* lam) {
    if (iterations <= 0) return;
    if (!aligned16(div_bar)) {  // both forms move its rows as 16-byte vectors
        const size_t bytes = (size_t)c.num_voxels() * sizeof(float);
        float* d = c.scratch_f32("adjoint_div_aligned", (size_t)c.num_voxels());
        HNS_CUDA(cudaMemcpyAsync(d, div_bar, bytes, cudaMemcpyDeviceToDevice, c.stream));
        adj_rbgs(c, p_bar, d, iterations, omega, lam);
        HNS_CUDA(cudaMemcpyAsync(div_bar, d, bytes, cudaMemcpyDeviceToDevice, c.stream));
        return;
    }
    if (use_chip(c, 2 * iterations) && aligned16(p_bar) && chip_takes(c, ChipUse::kTransposed)) {
        launch_chip_transpose(c, c.split_faces(), p_bar, div_bar, iterations, omega);
        return;
    }
    const size_t n = (size_t)c.num_voxels();
    if (lam == nullptr) lam = c.scratch_f32("adjoint_lam", n);
    HNS_CUDA(cudaMemcpyAsync(lam, p_bar, n * sizeof(float), cudaMemcpyDeviceToDevice, c.stream));
    const float a = omega * dev::kInv6;
    const float dx2 = c.dx * c.dx;
    float scale[2] = {1.f, 1.f};  // red, black
    for (int it = 0; it < iterations; ++it)
        for (int colour = 1; colour >= 0; --colour) {
            const int other = colour ^ 1;
            launch_adj_rbgs_colour(c, lam, div_bar, colour, scale[other], a * scale[colour], dx2 * a * scale[colour]);
            scale[other] = 1.f;
            scale[colour] *= 1.f - omega;
        }
}

namespace {

// vel_bar (the adjoint of the projected velocity) -> the adjoint of the velocity before the
// projection: vel_bar - D^T M^T G^T vel_bar, accumulated in place. lam: 3 n floats of scratch.
void adj_project(Context& c, float* vel_bar, int iterations, float omega, float* lam) {
    const size_t n = (size_t)c.num_voxels();
    float* p_bar = lam + n;
    float* div_bar = lam + 2 * n;
    HNS_CUDA(cudaMemsetAsync(p_bar, 0, n * sizeof(float), c.stream));
    HNS_CUDA(cudaMemsetAsync(div_bar, 0, n * sizeof(float), c.stream));
    launch_adj_gradient(c, vel_bar, p_bar);
    adj_rbgs(c, p_bar, div_bar, iterations, omega, lam);
    launch_adj_divergence(c, div_bar, vel_bar);
}

float default_omega(const Context& c, float omega) {
    return omega > 0.f ? omega : (float)(2.0f / (1.0f + std::sin(3.14159 * (double)c.dx)));
}

void need(const void* p, const char* what) {
    if (!p) fail(HNS_ERR_INVALID_ARG, std::string("null ") + what);
}

}  // namespace
}  // namespace hns

using namespace hns;

extern "C" {

HNS_API hns_status hns_adjoint_advect_scalar(hns_ctx* ctx, const float* vel, const float* in, const float* out_bar,
                                             float* in_bar, float* vel_bar, float dt) {
    return guarded([&] {
        Context* c = check_ctx(ctx);
        need(vel, "velocity"), need(in, "field"), need(out_bar, "output adjoint"), need(in_bar, "field adjoint");
        need(vel_bar, "velocity adjoint");
        DeviceGuard g(c->device);
        launch_adj_advect(*c, vel, nullptr, &in, &out_bar, &in_bar, 1, vel_bar, dt);
    });
}

HNS_API hns_status hns_adjoint_advect_vec3(hns_ctx* ctx, const float* vel, const float* out_bar, float* vel_bar, float dt) {
    return guarded([&] {
        Context* c = check_ctx(ctx);
        need(vel, "velocity"), need(out_bar, "output adjoint"), need(vel_bar, "velocity adjoint");
        DeviceGuard g(c->device);
        launch_adj_advect(*c, vel, out_bar, nullptr, nullptr, nullptr, 0, vel_bar, dt);
    });
}

HNS_API hns_status hns_adjoint_divergence(hns_ctx* ctx, const float* div_bar, float* vel_bar) {
    return guarded([&] {
        Context* c = check_ctx(ctx);
        need(div_bar, "divergence adjoint"), need(vel_bar, "velocity adjoint");
        DeviceGuard g(c->device);
        launch_adj_divergence(*c, div_bar, vel_bar);
    });
}

HNS_API hns_status hns_adjoint_subtract_gradient(hns_ctx* ctx, const float* out_bar, float* vel_bar, float* p_bar) {
    return guarded([&] {
        Context* c = check_ctx(ctx);
        need(out_bar, "output adjoint"), need(p_bar, "pressure adjoint");
        DeviceGuard g(c->device);
        if (vel_bar != nullptr) launch_adj_accumulate(*c, out_bar, vel_bar, 3 * c->num_voxels());  // d out / d vel = I
        launch_adj_gradient(*c, out_bar, p_bar);
    });
}

HNS_API hns_status hns_adjoint_rbgs(hns_ctx* ctx, const float* p_bar, float* div_bar, int iterations, float omega) {
    return guarded([&] {
        Context* c = check_ctx(ctx);
        need(p_bar, "pressure adjoint"), need(div_bar, "divergence adjoint");
        if (iterations < 0) fail(HNS_ERR_INVALID_ARG, "negative iteration count");
        DeviceGuard g(c->device);
        adj_rbgs(*c, p_bar, div_bar, iterations, omega);  // hns_rbgs takes omega as given
    });
}

HNS_API hns_status hns_adjoint_project(hns_ctx* ctx, float* vel_bar, int iterations, float omega) {
    return guarded([&] {
        Context* c = check_ctx(ctx);
        need(vel_bar, "velocity adjoint");
        if (iterations < 0) fail(HNS_ERR_INVALID_ARG, "negative iteration count");
        DeviceGuard g(c->device);
        adj_project(*c, vel_bar, iterations, default_omega(*c, omega), adj_scratch(*c, "adjoint_project_work", 3));
    });
}

HNS_API hns_status hns_adjoint_vorticity_confinement(hns_ctx* ctx, const float* vel, const float* out_bar, float* vel_bar,
                                                     float dt, float scale, float factor_scale) {
    return guarded([&] {
        Context* c = check_ctx(ctx);
        need(vel, "velocity"), need(out_bar, "output adjoint"), need(vel_bar, "velocity adjoint");
        if (!std::isfinite(factor_scale) || std::fabs(factor_scale) > 1e6f) fail(HNS_ERR_INVALID_ARG, "factor_scale out of range");
        DeviceGuard g(c->device);
        launch_adj_confinement(*c, vel, out_bar, vel_bar, dt, scale, factor_scale);
    });
}

HNS_API hns_status hns_adjoint_step_plain(hns_ctx* ctx, const float* vel_in, const float* const* scalars_in, int nscalars,
                                          const float* vel_out_bar, const float* const* scalars_out_bar, float* vel_in_bar,
                                          float* const* scalars_in_bar, float dt, int iterations, float omega) {
    return guarded([&] {
        Context* c = check_ctx(ctx);
        need(vel_in, "velocity"), need(vel_out_bar, "output velocity adjoint"), need(vel_in_bar, "velocity adjoint");
        if (nscalars < 0) fail(HNS_ERR_INVALID_ARG, "negative scalar count");
        if (nscalars > 0) need(scalars_in, "scalars"), need(scalars_out_bar, "scalar adjoints"), need(scalars_in_bar, "scalar adjoints");
        for (int q = 0; q < nscalars; ++q)
            need(scalars_in[q], "scalar"), need(scalars_out_bar[q], "scalar adjoint"), need(scalars_in_bar[q], "scalar adjoint");
        if (iterations < 0) fail(HNS_ERR_INVALID_ARG, "negative iteration count");
        DeviceGuard g(c->device);
        const int64_t n3 = 3 * c->num_voxels();
        // Adjoint of the advected velocity: the output adjoint through the projection.
        float* adv_bar = c->scratch_f32("adjoint_adv_bar", (size_t)n3);
        HNS_CUDA(cudaMemcpyAsync(adv_bar, vel_out_bar, (size_t)n3 * sizeof(float), cudaMemcpyDeviceToDevice, c->stream));
        adj_project(*c, adv_bar, iterations, default_omega(*c, omega), adj_scratch(*c));
        // Velocity self-advection and the scalars' advection along the same velocity.
        launch_adj_advect(*c, vel_in, adv_bar, scalars_in, scalars_out_bar, scalars_in_bar, nscalars, vel_in_bar, dt);
    });
}

}  // extern "C"
