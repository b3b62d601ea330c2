// Adjoint of the fire step: HNS_Advance (src/Cuda/HNanoSolver.cu:252-452) with a force model,
// one substep, no disturbance re-solve, no collider. Reverse mode through
//   adv  = advect_vector(vel)                            (Kernel.cu:349-426)
//   adv2 = confinement(adv) + dt src_vel + gravity       (Kernel.cu:682-727, 739-745, 834-838)
//   s1   = s + dt src for temperature, density, fuel     (Kernel.cu:732-737)
//   div  = divergence(adv2) [+ expansion burn]           (Kernel.cu:432-453, 641-677)
//   s2   = burn(s1)                                      (Kernel.cu:568-588 or 641-677)
//   adv3 = adv2 + e_y (b_T(T2) - alpha D1) dt            (Kernel.cu:546-563, plus the density term)
//   vel' = adv3 - grad p, p = M div                      (Kernel.cu:459-541)
//   s'   = advect_scalars(vel', s2)                      (Kernel.cu:163-289)
// with the forward recomputed from the step's inputs. M is the step's solve: `iterations`
// red-black iterations from p = 0 (hns_advance_model), whose transpose is the transposed sweeps
// in reverse; or a solve run to a tolerance (hns_advance_mixed), taken as exact: p = L^-1 (dx^2
// div), and L is symmetric, so div_bar = dx^2 L^-1 p_bar is one more refined solve.
//
// As for the other adjoints, branches (the MacCormack clamp, trace cells, the burn's min and
// thresholds, the buoyancy's T > ambient) are frozen at the forward's values, out-of-domain taps
// of advect_scalars read slot 0 (so their adjoint lands on slot 0, as the forward read it), and
// the trilinear scatters use FP32 atomics.
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <cmath>
#include <string>

#include "hns_internal.cuh"
#include "hns_stencil.cuh"

namespace hns {
namespace {

constexpr int kThreads = 256;
constexpr int kFields = 5;  // density, temperature, fuel, waste, flame
enum { kD = 0, kT = 1, kF = 2, kW = 3, kFL = 4 };

unsigned blocks_for(int64_t n) { return (unsigned)((n + kThreads - 1) / kThreads); }

// The advected fields of the step and their adjoints, up to kFields of them in any order.
struct AdvectedBars {
    const float* d[kFields];        // the fields the advection read
    const float* out_bar[kFields];  // the adjoints of the advected fields
    float* d_bar[kFields];          // += the adjoints of d
    int count;
};

// Interleaves the fields the adjoint gathers: fields 0..3 of a slot, and its velocity with field 4.
__global__ void __launch_bounds__(kThreads) pack_records_kernel(AdvectedBars F, const float* __restrict__ vel,
                                                                float4* __restrict__ in4, float4* __restrict__ vel_in4,
                                                                int64_t n) {
    const int64_t s = (int64_t)blockIdx.x * kThreads + threadIdx.x;
    if (s >= n) return;
    float v[kFields];
#pragma unroll
    for (int c = 0; c < kFields; ++c) v[c] = c < F.count ? __ldg(F.d[c] + s) : 0.f;
    in4[s] = make_float4(v[0], v[1], v[2], v[3]);
    vel_in4[s] = make_float4(__ldg(vel + 3 * s), __ldg(vel + 3 * s + 1), __ldg(vel + 3 * s + 2), v[4]);
}

__device__ __forceinline__ float comp(const float4& a, const float4& b, int c) {
    return c == 0 ? a.x : c == 1 ? a.y : c == 2 ? a.z : c == 3 ? a.w : b.w;
}

// Adjoint of advect_scalars for all fields along vel (the projected velocity), one thread per
// voxel: the trace, the taps and their weights are computed once for all fields, and the position
// adjoints of every field are summed before they are scattered to the velocity.
//   d_bar += (d out / d d)^T out_bar,  vel_bar += (d out / d vel)^T out_bar.
// Bound by the scatters' L2 atomics and the taps' gathers, so both go by records of 16 bytes: in4
// and vel_in4 hold the gathered fields (pack_records_kernel), rec4 one float4 per slot that
// receives the adjoints of fields 0..3 of a tap in one vector reduction, vel4 the three velocity
// components and field 4; fold_records_kernel adds both into the caller's arrays. Weights and
// slots as setupInterpolation (src/Cuda/Kernel.cu:204-233) computes them in the forward
// (interp_setup_fast, x fastest in the tap index), an out-of-domain tap reading slot 0. Slot 0
// takes the adjoints of all of those taps, one after the other on one address, which is most of
// what is left: the records make it one reduction per tap for all fields where each field's
// launch queued by itself. (Summing them per warp first takes 5 ms less but sums them in another
// order, up to 9e-4 away from the sums of one tap at a time.) On a 28,103-leaf grid with four
// fields 45.7 ms in four launches -> 8 ms.
template <typename I>
__global__ void __launch_bounds__(kThreads, 2) adj_advect_scalars_kernel(TopoView t, AdvectedBars F,
                                                                      const float4* __restrict__ in4,
                                                                      const float4* __restrict__ vel_in4,
                                                                      float4* __restrict__ rec4,
                                                                      float4* __restrict__ vel4, float sdt) {
    __shared__ dev::LeafNbhd L;
    const dev::VoxelIdx vx = dev::voxel_of_block();
    dev::load_nbhd(L, t, vx.leaf);
    __syncthreads();
    const int i = (L.lx << 3) + (vx.n >> 6), j = (L.ly << 3) + ((vx.n >> 3) & 7), k = (L.lz << 3) + (vx.n & 7);
    const int64_t s = (vx.leaf << 9) + vx.n;
    const float4 vc = __ldg(vel_in4 + s), dc = __ldg(in4 + s);
    const float bx = (float)i - vc.x * sdt, by = (float)j - vc.y * sdt, bz = (float)k - vc.z * sdt;
    I bs[8], fs[8];
    float bw[8], fw[8];
    dev::interp_setup_fast(t, L, bx, by, bz, bs, bw);
    float pf[kFields] = {}, pb[kFields] = {};
    float3 vf = make_float3(0.f, 0.f, 0.f);
#pragma unroll
    for (int q = 0; q < 8; ++q) {
        const float4 a = __ldg(vel_in4 + bs[q]), d = __ldg(in4 + bs[q]);
        vf.x = vf.x + a.x * bw[q];
        vf.y = vf.y + a.y * bw[q];
        vf.z = vf.z + a.z * bw[q];
#pragma unroll
        for (int c = 0; c < kFields; ++c) pf[c] = __fmaf_rn(comp(d, a, c), bw[q], pf[c]);
    }
    const float fx = bx + vf.x * sdt, fy = by + vf.y * sdt, fz = bz + vf.z * sdt;
    dev::interp_setup_fast(t, L, fx, fy, fz, fs, fw);
#pragma unroll
    for (int q = 0; q < 8; ++q) {
        const float4 d = __ldg(in4 + fs[q]);
        const float w = F.count > 4 ? __ldg(&vel_in4[fs[q]].w) : 0.f;
#pragma unroll
        for (int c = 0; c < kFields; ++c) pb[c] = __fmaf_rn(c < 4 ? comp(d, d, c) : w, fw[q], pb[c]);
    }
    // The clamp: which value of {centre, x-1, x+1, y-1, y+1, z-1, z+1, the forward sample}, in the
    // forward's order, the output is, and so where its adjoint goes.
    I ns[6];
    dev::face_slots(L, (I)s, vx.n, ns);
    float mn[kFields], mx[kFields];
    int imn[kFields], imx[kFields];  // -2 centre, 0..5 a neighbour, 6 the forward sample
#pragma unroll
    for (int c = 0; c < kFields; ++c) mn[c] = mx[c] = comp(dc, vc, c), imn[c] = imx[c] = -2;
#pragma unroll
    for (int q = 0; q < 6; ++q) {
        ns[q] = ns[q] < 0 ? I(0) : ns[q];
        const float4 d = __ldg(in4 + ns[q]);
        const float w = F.count > 4 ? __ldg(&vel_in4[ns[q]].w) : 0.f;
#pragma unroll
        for (int c = 0; c < kFields; ++c) {
            const float a = c < 4 ? comp(d, d, c) : w;
            if (a < mn[c]) mn[c] = a, imn[c] = q;
            if (a > mx[c]) mx[c] = a, imx[c] = q;
        }
    }
    float gpf[kFields] = {}, gpb[kFields] = {}, own[kFields] = {};
#pragma unroll
    for (int c = 0; c < kFields; ++c) {
        const float ob = c < F.count ? __ldg(F.out_bar[c] + s) : 0.f;
        const float corr = __fmaf_rn(0.5f, comp(dc, vc, c) - pb[c], pf[c]);
        if (pf[c] < mn[c]) mn[c] = pf[c], imn[c] = 6;
        if (pf[c] > mx[c]) mx[c] = pf[c], imx[c] = 6;
        const int pick = corr > mx[c] ? imx[c] : corr < mn[c] ? imn[c] : -1;
        if (pick == -1) {
            gpf[c] = ob, own[c] = 0.5f * ob, gpb[c] = -0.5f * ob;
        } else if (pick == -2) {
            own[c] = ob;
        } else if (pick == 6) {
            gpf[c] = ob;
        } else if (ob != 0.f) {
            I at = ns[0];
#pragma unroll
            for (int q = 1; q < 6; ++q) at = pick == q ? ns[q] : at;
            atomicAdd(c < 4 ? reinterpret_cast<float*>(rec4 + at) + c : &vel4[at].w, ob);
        }
    }
    // Positions: pf at back, pb at fwd = back + vf(back) sdt, back = x - vc sdt. A weight's
    // derivative in x is +-wy wz. The adjoint of a sample's position is the sum over its taps of
    // (the fields' adjoints . the tap's values) times the weight's gradient.
    auto grad = [](float x, float y, float z, int q) {
        const float tx = x - (float)__float2int_rd(x), ty = y - (float)__float2int_rd(y), tz = z - (float)__float2int_rd(z);
        const float wx = (q & 1) ? tx : 1.0f - tx, wy = (q & 2) ? ty : 1.0f - ty, wz = (q & 4) ? tz : 1.0f - tz;
        return make_float3(((q & 1) ? wy : -wy) * wz, ((q & 2) ? wx : -wx) * wz, ((q & 4) ? wx : -wx) * wy);
    };
    // The fields share records but not adjoints: one without an adjoint takes nothing, also where the trace
    // of a velocity that is not finite makes the weights NaN.
    auto part = [](float g, float w) { return g != 0.f ? g * w : 0.f; };
    const bool fwd = gpb[0] != 0.f || gpb[1] != 0.f || gpb[2] != 0.f || gpb[3] != 0.f || gpb[4] != 0.f;
    const bool back = gpf[0] != 0.f || gpf[1] != 0.f || gpf[2] != 0.f || gpf[3] != 0.f || gpf[4] != 0.f;
    float3 fb = make_float3(0.f, 0.f, 0.f), bb = make_float3(0.f, 0.f, 0.f);
    if (fwd) {
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            const float4 d = __ldg(in4 + fs[q]);
            float a = 0.f;
#pragma unroll
            for (int c = 0; c < 4; ++c) a += gpb[c] != 0.f ? gpb[c] * comp(d, d, c) : 0.f;
            if (gpb[4] != 0.f) a += gpb[4] * __ldg(&vel_in4[fs[q]].w);
            const float3 w = grad(fx, fy, fz, q);
            fb.x += a * w.x, fb.y += a * w.y, fb.z += a * w.z;
            const float m = fw[q];
            dev::red4(rec4 + fs[q], part(gpb[0], m), part(gpb[1], m), part(gpb[2], m), part(gpb[3], m));
            if (gpb[4] != 0.f) atomicAdd(&vel4[fs[q]].w, gpb[4] * m);
        }
    }
    const float3 vfb = make_float3(fb.x * sdt, fb.y * sdt, fb.z * sdt);
    const bool trace = vfb.x != 0.f || vfb.y != 0.f || vfb.z != 0.f;
    if (back || trace) {
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            const float4 u = __ldg(vel_in4 + bs[q]), d = __ldg(in4 + bs[q]);
            float a = trace ? vfb.x * u.x + vfb.y * u.y + vfb.z * u.z : 0.f;
#pragma unroll
            for (int c = 0; c < kFields; ++c) a += gpf[c] != 0.f ? gpf[c] * comp(d, u, c) : 0.f;
            const float3 w = grad(bx, by, bz, q);
            bb.x += a * w.x, bb.y += a * w.y, bb.z += a * w.z;
            const float m = bw[q];
            if (back) dev::red4(rec4 + bs[q], part(gpf[0], m), part(gpf[1], m), part(gpf[2], m), part(gpf[3], m));
            if (trace || gpf[4] != 0.f)
                dev::red4(vel4 + bs[q], part(vfb.x, m), part(vfb.y, m), part(vfb.z, m), part(gpf[4], m));
        }
    }
    bb.x += fb.x, bb.y += fb.y, bb.z += fb.z;
    dev::red4(rec4 + s, own[0], own[1], own[2], own[3]);
    dev::red4(vel4 + s, -sdt * bb.x, -sdt * bb.y, -sdt * bb.z, own[4]);
}

// Adds the records of adj_advect_scalars_kernel into the fields' and the velocity's adjoints.
__global__ void __launch_bounds__(kThreads) fold_records_kernel(AdvectedBars F, const float4* __restrict__ rec4,
                                                                const float4* __restrict__ vel4,
                                                                float* __restrict__ vel_bar, int64_t n) {
    const int64_t s = (int64_t)blockIdx.x * kThreads + threadIdx.x;
    if (s >= n) return;
    const float4 a = __ldg(rec4 + s), b = __ldg(vel4 + s);
    const float v[kFields] = {a.x, a.y, a.z, a.w, b.w};
#pragma unroll
    for (int c = 0; c < kFields; ++c)
        if (c < F.count) F.d_bar[c][s] += v[c];
    vel_bar[3 * s] += b.x;
    vel_bar[3 * s + 1] += b.y;
    vel_bar[3 * s + 2] += b.z;
}

// s1 = s + dt src (add_scalar_source, out of place; the forward's arithmetic).
__global__ void __launch_bounds__(kThreads) add_source_kernel(const float* __restrict__ in, const float* __restrict__ src,
                                                              float* __restrict__ out, float dt, int64_t n) {
    const int64_t s = (int64_t)blockIdx.x * kThreads + threadIdx.x;
    if (s < n) out[s] = src ? in[s] + dt * __ldg(src + s) : in[s];
}

struct PointwiseIn {
    const float* s1[kFields];  // the fields after the sources, before the burn (null: absent)
    const float* mid_bar[kFields];  // adjoints of the burned fields (what the advection read)
    float* in_bar[kFields];    // the step's input adjoints (+=)
};

// Transposes of the sources (identity), the burn and the buoyancy, per voxel. adv3_bar: the
// adjoint of the forced velocity before the projection; div_bar: of the divergence (the
// oxygen burn's expansion term).
template <int kModel>
__global__ void __launch_bounds__(kThreads) adj_burn_buoy_kernel(PointwiseIn P, const float* __restrict__ adv3_bar,
                                                                 const float* __restrict__ div_bar, float gain,
                                                                 float expansion, float rate, float heat, float ignition,
                                                                 float alpha, float dt, float ambient, float strength,
                                                                 int64_t n) {
    const int64_t s = (int64_t)blockIdx.x * kThreads + threadIdx.x;
    if (s >= n) return;
    auto val = [&](int f) { return P.s1[f] ? P.s1[f][s] : 0.f; };
    auto bar = [&](int f) { return P.mid_bar[f] ? P.mid_bar[f][s] : 0.f; };
    const float T1 = val(kT), F1 = val(kF), W = val(kW), FL = val(kFL);
    // The burn, recomputed, with its branches.
    float T2 = T1, dbF = 0.f, dbW = 0.f, dF = 1.f, dFLb = 0.f;
    bool burning = false, fl_keeps = true;
    if constexpr (kModel == HNS_COMBUSTION_RATE) {
        if (F1 > 0.0f && T1 >= ignition) {
            const float rdt = rate * dt, b = fminf(F1, rdt);
            burning = true;
            dbF = F1 < rdt ? 1.f : 0.f;
            T2 = T1 + b * heat;
        }
    } else if constexpr (kModel == HNS_COMBUSTION_OXYGEN) {
        float F = F1;
        if (F < 0.001f) F = 0.0f, dF = 0.f;
        const float oxy = 1.0f - F - W;
        if (oxy >= 0.0f) {
            burning = true;
            const float burn = fminf(oxy, F);
            if (oxy < F) dbF = -1.f, dbW = -1.f;
            else dbF = 1.f, dbW = 0.f;
            T2 = T1 + burn * gain;
            const float cand = fminf(1.0f, burn * 10.0f);
            fl_keeps = FL >= cand;
            dFLb = (!fl_keeps && burn * 10.0f < 1.0f) ? 10.f : 0.f;
        }
    }
    // Buoyancy: adv3.y = adv2.y + (b_T(T2) - alpha D1) dt.
    const float ay = adv3_bar[3 * s + 1] * dt;
    const float dbt = (T2 > ambient && (T2 - ambient) * strength > 0.0f) ? strength : 0.0f;
    const float T2b = bar(kT) + ay * dbt;
    const float D1b = bar(kD) - ay * alpha;
    float T1b = T2b, F1b = bar(kF), Wb = bar(kW), FLb = bar(kFL);
    if constexpr (kModel == HNS_COMBUSTION_RATE) {
        if (burning) {
            const float bb = -bar(kF) + T2b * heat;
            F1b = bar(kF) + bb * dbF;
        }
    } else if constexpr (kModel == HNS_COMBUSTION_OXYGEN) {
        if (burning) {
            const float bb = -bar(kF) + 2.0f * bar(kW) + gain * T2b + expansion * div_bar[s] + dFLb * bar(kFL);
            F1b = bar(kF) + bb * dbF;
            Wb = bar(kW) + bb * dbW;
            FLb = fl_keeps ? bar(kFL) : 0.f;
        }
        F1b *= dF;
    }
    // The sources are additive: the adjoints pass to the step's inputs unchanged.
    const float outb[kFields] = {D1b, T1b, F1b, Wb, FLb};
#pragma unroll
    for (int f = 0; f < kFields; ++f)
        if (P.in_bar[f]) P.in_bar[f][s] += outb[f];
}

float* sf(Context& c, const std::string& name, size_t count) { return c.scratch_f32("fire_adj_" + name, count); }

}  // namespace

// The projection of the adjoint: refined (exact) when solve is given, else `iterations` red-black
// iterations (omega as the step uses it).
struct FireAdjointSolve {
    int iterations = 0;
    float omega = 0.f;
    const hns_mixed_desc* refined = nullptr;
};

void adjoint_fire(Context& c, const hns_fire_f32& in, const hns_fire_sources_f32& src, const hns_fire_f32& out_bar,
                  const hns_fire_f32& in_bar, float dt, const hns_combustion_params& P, const hns_force_model& M,
                  const FireAdjointSolve& S) {
    const size_t n = (size_t)c.num_voxels();
    const int64_t nn = (int64_t)n;
    const float* sin[kFields] = {in.density, in.temperature, in.fuel, in.waste, in.flame};
    const float* sbar_out[kFields] = {out_bar.density, out_bar.temperature, out_bar.fuel, out_bar.waste, out_bar.flame};
    float* sbar_in[kFields] = {in_bar.density, in_bar.temperature, in_bar.fuel, in_bar.waste, in_bar.flame};
    const float* srcs[kFields] = {src.density, src.temperature, src.fuel, nullptr, nullptr};
    static const char* nm[kFields] = {"density", "temperature", "fuel", "waste", "flame"};

    // One scratch block of 16 n floats whose parts the phases use in turn: the forward's adv2, adv3
    // and div; the scalar advection's records; then p_bar, div_bar, the velocity's adjoints and the
    // self-advection's records. Fewer bytes to allocate on a grid's first pass, which costs more
    // than the pass itself.
    float* arena = sf(c, "arena", 16 * n);

    // ---- the forward, recomputed ----
    float* adv = sf(c, "adv", 3 * n);
    float* adv2 = arena;
    float* adv3 = arena + 3 * n;
    float* div = arena + 6 * n;
    FieldSet none{};
    launch_advect_fused(c, in.velocity, adv, none, dt);
    launch_confine_sources(c, adv, adv2, div, dt, P.vorticityScale, P.factorScale, src.velocity, P.gravity);
    float* s1[kFields] = {};
    float* s2[kFields] = {};
    for (int f = 0; f < kFields; ++f) {
        if (!sin[f]) continue;
        s1[f] = sf(c, std::string("s1_") + nm[f], n);
        s2[f] = sf(c, std::string("s2_") + nm[f], n);
        add_source_kernel<<<blocks_for(nn), kThreads, 0, c.stream>>>(sin[f], srcs[f], s1[f], dt, nn);
        HNS_LAUNCHED();
        HNS_CUDA(cudaMemcpyAsync(s2[f], s1[f], n * sizeof(float), cudaMemcpyDeviceToDevice, c.stream));
    }
    launch_div_combust_buoy(c, adv2, adv3, div, s2[kF], s2[kW], s2[kT], s2[kFL],
                            M.density_buoyancy != 0.0f ? s2[kD] : nullptr, P, M, dt);
    float* velp = sf(c, "velp", 3 * n);
    double* p64 = nullptr;
    if (S.refined) {
        p64 = reinterpret_cast<double*>(sf(c, "p64", 2 * n));
        const float om = S.refined->omega > 0.f ? S.refined->omega : 1.9f;
        refine_solve<__half>(c, div, p64, S.refined->max_outer, S.refined->inner_iterations, om, S.refined->tolerance,
                             S.refined->flags);
        HNS_CUDA(cudaMemcpyAsync(velp, adv3, 3 * n * sizeof(float), cudaMemcpyDeviceToDevice, c.stream));
        launch_gradient_f64(c, velp, p64);
    } else {
        float* p = sf(c, "p", n);
        rbgs_solve(c, div, p, S.iterations, S.omega, HNS_SOLVE_ZERO_INIT);
        launch_subtract_gradient(c, adv3, p, velp);
    }

    // ---- reverse ----
    float* vb = sf(c, "vb", 3 * n);
    HNS_CUDA(cudaMemcpyAsync(vb, out_bar.velocity, 3 * n * sizeof(float), cudaMemcpyDeviceToDevice, c.stream));
    float* mid[kFields] = {};
    AdvectedBars bars{};
    for (int f = 0; f < kFields; ++f) {
        if (!sin[f]) continue;
        mid[f] = sf(c, std::string("mid_") + nm[f], n);
        HNS_CUDA(cudaMemsetAsync(mid[f], 0, n * sizeof(float), c.stream));
        if (!sbar_out[f]) continue;
        bars.d[bars.count] = s2[f];
        bars.out_bar[bars.count] = sbar_out[f];
        bars.d_bar[bars.count] = mid[f];
        ++bars.count;
    }
    if (bars.count > 0) {
        auto* rec4 = reinterpret_cast<float4*>(arena);
        auto* vel4 = reinterpret_cast<float4*>(arena + 4 * n);
        auto* in4 = reinterpret_cast<float4*>(arena + 8 * n);
        auto* vel_in4 = reinterpret_cast<float4*>(arena + 12 * n);
        pack_records_kernel<<<blocks_for(nn), kThreads, 0, c.stream>>>(bars, velp, in4, vel_in4, nn);
        HNS_LAUNCHED();
        HNS_CUDA(cudaMemsetAsync(rec4, 0, 8 * n * sizeof(float), c.stream));  // rec4 and vel4
        const float sdt = dt * (1.0f / c.dx);
        const unsigned blocks = (unsigned)(2 * c.topo.num_leaves);
        if (c.topo.num_leaves < (int64_t(1) << 22))
            adj_advect_scalars_kernel<int32_t><<<blocks, kThreads, 0, c.stream>>>(c.topo.view, bars, in4, vel_in4, rec4,
                                                                                  vel4, sdt);
        else
            adj_advect_scalars_kernel<int64_t><<<blocks, kThreads, 0, c.stream>>>(c.topo.view, bars, in4, vel_in4, rec4,
                                                                                  vel4, sdt);
        HNS_LAUNCHED();
        fold_records_kernel<<<blocks_for(nn), kThreads, 0, c.stream>>>(bars, rec4, vel4, vb, nn);
        HNS_LAUNCHED();
    }
    // The projection: vel' = adv3 - grad p, p = M div.
    float* pbar = arena;
    float* dbar = arena + n;
    HNS_CUDA(cudaMemsetAsync(pbar, 0, n * sizeof(float), c.stream));
    HNS_CUDA(cudaMemsetAsync(dbar, 0, n * sizeof(float), c.stream));
    launch_adj_gradient(c, vb, pbar);
    if (S.refined) {
        // div_bar = dx^2 L^-1 p_bar: the refined solve of p_bar as a divergence.
        const float om = S.refined->omega > 0.f ? S.refined->omega : 1.9f;
        refine_solve<__half>(c, pbar, p64, S.refined->max_outer, S.refined->inner_iterations, om, S.refined->tolerance,
                             S.refined->flags);
        convert_array(c, p64, HNS_DTYPE_F64, dbar, HNS_DTYPE_F32, nn);
    } else {
        adj_rbgs(c, pbar, dbar, S.iterations, S.omega, arena + 8 * n);
    }
    // adv2_bar = adv3_bar (the buoyancy adds to adv2) + D^T div_bar.
    float* adv2b = arena + 2 * n;
    HNS_CUDA(cudaMemcpyAsync(adv2b, vb, 3 * n * sizeof(float), cudaMemcpyDeviceToDevice, c.stream));
    launch_adj_divergence(c, dbar, adv2b);
    // Burn, buoyancy and sources, per voxel.
    PointwiseIn pin{};
    for (int f = 0; f < kFields; ++f) {
        pin.s1[f] = s1[f];
        pin.mid_bar[f] = mid[f];
        pin.in_bar[f] = sin[f] ? sbar_in[f] : nullptr;
    }
    const unsigned g = blocks_for(nn);
    if (M.combustion == HNS_COMBUSTION_OXYGEN)
        adj_burn_buoy_kernel<HNS_COMBUSTION_OXYGEN><<<g, kThreads, 0, c.stream>>>(
            pin, vb, dbar, P.temperatureRelease, P.expansionRate, M.burn_rate, M.heat_release, M.ignition_temp,
            M.density_buoyancy, dt, P.ambientTemp, P.buoyancyStrength, nn);
    else if (M.combustion == HNS_COMBUSTION_RATE)
        adj_burn_buoy_kernel<HNS_COMBUSTION_RATE><<<g, kThreads, 0, c.stream>>>(
            pin, vb, dbar, P.temperatureRelease, P.expansionRate, M.burn_rate, M.heat_release, M.ignition_temp,
            M.density_buoyancy, dt, P.ambientTemp, P.buoyancyStrength, nn);
    else
        adj_burn_buoy_kernel<HNS_COMBUSTION_NONE><<<g, kThreads, 0, c.stream>>>(
            pin, vb, dbar, P.temperatureRelease, P.expansionRate, M.burn_rate, M.heat_release, M.ignition_temp,
            M.density_buoyancy, dt, P.ambientTemp, P.buoyancyStrength, nn);
    HNS_LAUNCHED();
    // Confinement and the velocity's self-advection.
    float* advb = arena + 5 * n;
    HNS_CUDA(cudaMemsetAsync(advb, 0, 3 * n * sizeof(float), c.stream));
    launch_adj_confinement(c, adv, adv2b, advb, dt, P.vorticityScale, P.factorScale, arena + 8 * n);
    launch_adj_advect(c, in.velocity, advb, nullptr, nullptr, nullptr, 0, in_bar.velocity, dt, arena + 8 * n);
}

}  // namespace hns

using namespace hns;

namespace {

void check_fire_adjoint(const hns_fire_f32* out_bar, const hns_fire_f32* in_bar, const hns_combustion_params* params,
                        const hns_force_model& M) {
    if (!out_bar || !in_bar || !params) fail(HNS_ERR_INVALID_ARG, "null argument");
    if (!out_bar->velocity || !in_bar->velocity) fail(HNS_ERR_INVALID_ARG, "the velocity adjoints are required");
    if (params->substeps > 1) fail(HNS_ERR_UNSUPPORTED, "the fire adjoint takes one substep");
    if (params->disturbanceEnable > 0.0f) fail(HNS_ERR_UNSUPPORTED, "the fire adjoint takes no disturbance re-solve");
    check_force_model(M);
}

void check_fields_f32(const hns_fire_f32& in, const hns_fire_f32& out_bar, const hns_fire_f32& in_bar,
                      const hns_force_model& M) {
    const float* a[6] = {in.velocity, in.density, in.temperature, in.fuel, in.waste, in.flame};
    const float* b[6] = {in_bar.velocity, in_bar.density, in_bar.temperature, in_bar.fuel, in_bar.waste, in_bar.flame};
    for (int q = 0; q < 6; ++q)
        if ((a[q] == nullptr) != (b[q] == nullptr)) fail(HNS_ERR_INVALID_ARG, "each field needs its input adjoint");
    (void)out_bar;
    if (!in.temperature) fail(HNS_ERR_INVALID_ARG, "the step needs a temperature field");
    if (M.combustion != HNS_COMBUSTION_NONE && !in.fuel) fail(HNS_ERR_INVALID_ARG, "the burn needs a fuel field");
    if (M.combustion == HNS_COMBUSTION_OXYGEN && (!in.waste || !in.flame))
        fail(HNS_ERR_INVALID_ARG, "the oxygen burn needs waste and flame fields");
    if (M.density_buoyancy != 0.0f && !in.density) fail(HNS_ERR_INVALID_ARG, "the density buoyancy needs a density field");
}

}  // namespace

extern "C" {

HNS_API hns_status hns_adjoint_advance(hns_ctx* ctx, const hns_fire_f32* in, const hns_fire_sources_f32* sources,
                                       const hns_fire_f32* out_bar, const hns_fire_f32* in_bar, float dt, int iterations,
                                       const hns_combustion_params* params, const hns_force_model* model) {
    return guarded([&] {
        Context* c = check_ctx(ctx);
        if (!in || !in->velocity) fail(HNS_ERR_INVALID_ARG, "null fields");
        if (iterations < 0) fail(HNS_ERR_INVALID_ARG, "negative iteration count");
        const hns_force_model M = model ? *model : hns_force_model{};
        check_fire_adjoint(out_bar, in_bar, params, M);
        check_fields_f32(*in, *out_bar, *in_bar, M);
        DeviceGuard dg(c->device);
        FireAdjointSolve S;
        S.iterations = iterations;
        S.omega = 2.0f / (1.0f + sinf(3.14159f * c->dx));  // HNS_Advance's (src/Cuda/HNanoSolver.cu:365)
        adjoint_fire(*c, *in, sources ? *sources : hns_fire_sources_f32{}, *out_bar, *in_bar, dt, *params, M, S);
    });
}

HNS_API hns_status hns_adjoint_advance_mixed(hns_ctx* ctx, const hns_fire_fields* in, const hns_fire_sources* sources,
                                             const hns_fire_f32* out_bar, const hns_fire_f32* in_bar, float dt,
                                             const hns_combustion_params* params, const hns_force_model* model,
                                             const hns_mixed_desc* solve) {
    return guarded([&] {
        Context* c = check_ctx(ctx);
        if (!in || !in->velocity || !solve) fail(HNS_ERR_INVALID_ARG, "null fields or solve description");
        if (solve->max_outer <= 0 || solve->max_outer > 1000 || solve->inner_iterations <= 0 || !(solve->tolerance > 0.0))
            fail(HNS_ERR_INVALID_ARG, "bad solve description");
        const hns_force_model M = model ? *model : hns_force_model{};
        check_fire_adjoint(out_bar, in_bar, params, M);
        DeviceGuard dg(c->device);
        const size_t n = (size_t)c->num_voxels();
        // The BF16/FP16 inputs as FP32: the step's arithmetic is FP32 on these values.
        const void* hin[6] = {in->velocity, in->density, in->temperature, in->fuel, in->waste, in->flame};
        static const char* nm[6] = {"velocity", "density", "temperature", "fuel", "waste", "flame"};
        float* f32[6] = {};
        for (int q = 0; q < 6; ++q) {
            if (!hin[q]) continue;
            if (((uintptr_t)hin[q]) & 1u) fail(HNS_ERR_INVALID_ARG, "BF16/FP16 arrays must be 2-byte aligned");
            const size_t cnt = q == 0 ? 3 * n : n;
            f32[q] = c->scratch_f32(std::string("fire_adjm_in_") + nm[q], cnt);
            convert_array(*c, hin[q], q == 0 ? HNS_DTYPE_BF16 : HNS_DTYPE_F16, f32[q], HNS_DTYPE_F32, (int64_t)cnt);
        }
        const hns_fire_f32 fin{f32[0], f32[1], f32[2], f32[3], f32[4], f32[5]};
        check_fields_f32(fin, *out_bar, *in_bar, M);
        hns_fire_sources_f32 fs{};
        if (sources) {
            const void* hs[4] = {sources->velocity, sources->temperature, sources->density, sources->fuel};
            const float** ps[4] = {&fs.velocity, &fs.temperature, &fs.density, &fs.fuel};
            static const char* sn[4] = {"velocity", "temperature", "density", "fuel"};
            for (int q = 0; q < 4; ++q) {
                if (!hs[q]) continue;
                const size_t cnt = q == 0 ? 3 * n : n;
                float* d = c->scratch_f32(std::string("fire_adjm_src_") + sn[q], cnt);
                convert_array(*c, hs[q], q == 0 ? HNS_DTYPE_BF16 : HNS_DTYPE_F16, d, HNS_DTYPE_F32, (int64_t)cnt);
                *ps[q] = d;
            }
        }
        FireAdjointSolve S;
        S.refined = solve;
        adjoint_fire(*c, fin, fs, *out_bar, *in_bar, dt, *params, M, S);
    });
}

}  // extern "C"
