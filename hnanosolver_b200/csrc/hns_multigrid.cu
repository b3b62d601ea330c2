// Geometric multigrid V-cycle for the inner solve of the FP64 refinement (HNS_SOLVE_MULTIGRID):
// the preconditioner the reference declares for the projection but never implements
// (restrict_to_2x2x2 / prolongate / compute_residual / update_pressure,
// src/Cuda/Kernels.cuh:52-60).
//
// Levels live inside the leaf structure: level l has s = 8 >> l cells per leaf side (8, 4, 2, 1),
// so every level shares the leaf table and the 27-neighbour table, and a cell's face
// neighbour is in its own leaf or in the face-neighbour leaf. Cells of a leaf are stored at
// (x s + y) s + z. With unit fine spacing the level-l operator is
// A_l u = (sum of the 6 face neighbours - 6 u) / 4^l, zero outside the domain (the fine
// system's p = 0 walls). The cycle: red-black Gauss-Seidel smoothing (red by global cell
// parity), the residual, restriction by the mean of the 8 children, on down to one cell per
// leaf, where SOR sweeps solve the leaf-level system; then each coarse correction goes back
// into the fine cells, interpolated trilinearly between cell centres, and post-smoothing.
// FP32 throughout; the FP64 outer refinement around it measures the residual exactly, so the
// cycle only has to reduce the error. Every kernel returns at once when the refinement has
// converged.
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <cmath>
#include <cstdint>
#include <map>
#include <mutex>
#include <string>
#include <utility>

#include "hns_internal.cuh"

namespace hns {
namespace {

constexpr int kThreads = 256;
constexpr int kLevels = 4;
// Cycle parameters: smoothing iterations before and after the coarse correction, and SOR
// iterations (factor kCoarseOmega) at the one-cell-per-leaf level.
constexpr int kPreSmooth = 3, kPostSmooth = 3, kCoarseIters = 60;
constexpr float kCoarseOmega = 1.9f;

__device__ __forceinline__ bool done(const double* check, double tol2) {
    return check != nullptr && check[0] <= tol2 * check[1];
}

// Cell q of level with 2^lg cells per leaf side: its leaf and coordinates within the leaf.
struct Cell {
    int64_t leaf;
    int x, y, z;
};

__device__ __forceinline__ Cell cell_of(int64_t q, int lg) {
    Cell c;
    c.leaf = q >> (3 * lg);
    const int loc = (int)(q & ((1 << (3 * lg)) - 1)), m = (1 << lg) - 1;
    c.x = loc >> (2 * lg);
    c.y = (loc >> lg) & m;
    c.z = loc & m;
    return c;
}

// u at (x, y, z) of leaf `leaf`, each coordinate in [-1, s]: a coordinate outside [0, s) is in
// the neighbour leaf across that face, edge or corner (0 when that leaf does not exist).
__device__ __forceinline__ float at(const TopoView& t, const float* __restrict__ u, int64_t leaf, int lg, int x, int y,
                                    int z) {
    const int s = 1 << lg;
    int dx = 0, dy = 0, dz = 0;
    if (x < 0) dx = -1, x += s;
    if (x >= s) dx = 1, x -= s;
    if (y < 0) dy = -1, y += s;
    if (y >= s) dy = 1, y -= s;
    if (z < 0) dz = -1, z += s;
    if (z >= s) dz = 1, z -= s;
    int64_t l = leaf;
    if (dx | dy | dz) {
        const int n = __ldg(t.nbr27 + leaf * 27 + (dx + 1) * 9 + (dy + 1) * 3 + (dz + 1));
        if (n < 0) return 0.f;
        l = n;
    }
    return u[(l << (3 * lg)) + (((x << lg) + y) << lg) + z];
}

__device__ __forceinline__ float nbr_sum(const TopoView& t, const float* __restrict__ u, const Cell& c, int lg) {
    return at(t, u, c.leaf, lg, c.x + 1, c.y, c.z) + at(t, u, c.leaf, lg, c.x - 1, c.y, c.z) +
           at(t, u, c.leaf, lg, c.x, c.y + 1, c.z) + at(t, u, c.leaf, lg, c.x, c.y - 1, c.z) +
           at(t, u, c.leaf, lg, c.x, c.y, c.z + 1) + at(t, u, c.leaf, lg, c.x, c.y, c.z - 1);
}

// One colour of SOR on level lg: u = (1 - omega) u + omega (sum - h2 b) / 6, h2 = 4^l.
__global__ void __launch_bounds__(kThreads) mg_smooth_kernel(TopoView t, float* u, const float* __restrict__ b, int lg,
                                                             int64_t cells, int colour, float omega, float h2,
                                                             const double* __restrict__ check, double tol2) {
    if (done(check, tol2)) return;
    const int64_t q = (int64_t)blockIdx.x * kThreads + threadIdx.x;
    if (q >= cells) return;
    const Cell c = cell_of(q, lg);
    const int4 o = t.origin[c.leaf];
    // Global cell coordinates: leaf origins are multiples of 8 fine voxels, 2^lg cells per leaf.
    const int gx = ((o.x >> 3) << lg) + c.x, gy = ((o.y >> 3) << lg) + c.y, gz = ((o.z >> 3) << lg) + c.z;
    if (((gx + gy + gz) & 1) != colour) return;
    const float g = (nbr_sum(t, u, c, lg) - h2 * __ldg(b + q)) * (1.0f / 6.0f);
    u[q] = u[q] + omega * (g - u[q]);
}

// r = b - (sum - 6 u) / h2.
__global__ void __launch_bounds__(kThreads) mg_residual_kernel(TopoView t, const float* __restrict__ u,
                                                               const float* __restrict__ b, float* __restrict__ r, int lg,
                                                               int64_t cells, float inv_h2, const double* __restrict__ check,
                                                               double tol2) {
    if (done(check, tol2)) return;
    const int64_t q = (int64_t)blockIdx.x * kThreads + threadIdx.x;
    if (q >= cells) return;
    const Cell c = cell_of(q, lg);
    r[q] = __ldg(b + q) - (nbr_sum(t, u, c, lg) - 6.0f * u[q]) * inv_h2;
}

// Coarse right-hand side: the mean of the 8 children's residuals (coarse level lg).
__global__ void __launch_bounds__(kThreads) mg_restrict_kernel(const float* __restrict__ r_fine, float* __restrict__ b,
                                                               int lg, int64_t cells, const double* __restrict__ check,
                                                               double tol2) {
    if (done(check, tol2)) return;
    const int64_t q = (int64_t)blockIdx.x * kThreads + threadIdx.x;
    if (q >= cells) return;
    const Cell c = cell_of(q, lg);
    const int lf = lg + 1;
    const int64_t base = c.leaf << (3 * lf);
    float sum = 0.f;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        const int x = 2 * c.x + (k >> 2), y = 2 * c.y + ((k >> 1) & 1), z = 2 * c.z + (k & 1);
        sum += __ldg(r_fine + base + (((x << lf) + y) << lf) + z);
    }
    b[q] = 0.125f * sum;
}

// u_fine += the coarse correction interpolated trilinearly between cell centres (fine level
// lg): along each axis a fine cell takes 3/4 of its parent and 1/4 of the parent's neighbour on
// its side (0 outside the domain).
__global__ void __launch_bounds__(kThreads) mg_prolong_kernel(TopoView t, const float* __restrict__ u_coarse,
                                                              float* __restrict__ u_fine, int lg, int64_t cells,
                                                              const double* __restrict__ check, double tol2) {
    if (done(check, tol2)) return;
    const int64_t q = (int64_t)blockIdx.x * kThreads + threadIdx.x;
    if (q >= cells) return;
    const Cell c = cell_of(q, lg);
    const int lc = lg - 1;
    const int X = c.x >> 1, Y = c.y >> 1, Z = c.z >> 1;
    const int dx = (c.x & 1) ? 1 : -1, dy = (c.y & 1) ? 1 : -1, dz = (c.z & 1) ? 1 : -1;
    float sum = 0.f;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        const int a = k >> 2, b = (k >> 1) & 1, e = k & 1;
        const float w = (a ? 0.25f : 0.75f) * (b ? 0.25f : 0.75f) * (e ? 0.25f : 0.75f);
        sum += w * at(t, u_coarse, c.leaf, lc, X + a * dx, Y + b * dy, Z + e * dz);
    }
    u_fine[q] += sum;
}

unsigned blocks(int64_t cells) { return (unsigned)((cells + kThreads - 1) / kThreads); }

// ---- V-cycle of the FP16 inner solve (colour-split fine level) ------------------------------
// Coarse levels as above (2^LG cells per leaf side, cell (x, y, z) of leaf l at
// (l << 3 LG) + ((x << LG) + y << LG) + z, FP32), with the operator corrected at the walls: the
// fine system's p = 0 sits at the ghost cell's centre, half a fine cell past the wall, and a
// coarse ghost value of 0 would put it half a coarse cell past it. The coarse ghost value is
// instead extrapolated linearly through that point, -gamma u with gamma = (2^l - 1) / (2^l + 1)
// at level l, which adds gamma to the diagonal for each missing face neighbour. A numpy model of
// the cycle on a 160^3 shell gives 0.16 per cycle with the correction against 0.54-1.1 without.
// Face neighbours come from the colour-split face table nb8 ({+x, -x, +y, -y, +z, -z, the leaf,
// 0}, a missing leaf = num_leaves).

template <int LG>
struct LevelCell {
    int leaf, x, y, z;
};

template <int LG>
__device__ __forceinline__ LevelCell<LG> level_cell(int64_t q) {
    constexpr int m = (1 << LG) - 1;
    LevelCell<LG> c;
    c.leaf = (int)(q >> (3 * LG));
    c.x = (int)(q >> (2 * LG)) & m;
    c.y = (int)(q >> LG) & m;
    c.z = (int)q & m;
    return c;
}

// Sum of the face neighbours of cell (x, y, z) of `leaf` at level LG present in the domain, and
// the number missing.
template <int LG, bool kRead = true>
__device__ __forceinline__ float level_nsum(const int4* __restrict__ nb8, const float* u, int leaf, int x, int y,
                                            int z, int num_leaves, int& missing) {
    constexpr int s = 1 << LG, m = s - 1;
    const int4 f0 = __ldg(nb8 + 2 * leaf), f1 = __ldg(nb8 + 2 * leaf + 1);
    auto at = [&](int l, int a, int b, int c) -> float {
        if (l >= num_leaves) {
            ++missing;
            return 0.f;
        }
        return kRead ? u[((int64_t)l << (3 * LG)) + (((a << LG) + b) << LG) + c] : 0.f;
    };
    missing = 0;
    float sum = at(x < m ? leaf : f0.x, (x + 1) & m, y, z);
    sum += at(x > 0 ? leaf : f0.y, (x - 1) & m, y, z);
    sum += at(y < m ? leaf : f0.z, x, (y + 1) & m, z);
    sum += at(y > 0 ? leaf : f0.w, x, (y - 1) & m, z);
    sum += at(z < m ? leaf : f1.x, x, y, (z + 1) & m);
    sum += at(z > 0 ? leaf : f1.y, x, y, (z - 1) & m);
    return sum;
}

// The kernels of the FP16 cycle start while the preceding ones still run (programmatic dependent
// launches) and wait before they read what those write. Such arrays are read by plain loads, through
// pointers without __restrict__: a non-coherent load (__ldg, or one that the compiler makes of a const
// __restrict__ pointer) is only allowed on memory that nothing writes while the kernel lives, and may
// be moved above the wait.

// One colour of SOR at the coarsest level (one cell per leaf): u += omega ((sum - h2 b) / (6 + gamma
// missing) - u), the colour being the leaf's parity.
__global__ void __launch_bounds__(kThreads) coarsest_sweep_kernel(TopoView t, const int4* __restrict__ nb8, float* u,
                                                                  const float* b, int colour, int zero,
                                                                  float omega, float h2, float gamma,
                                                                  const double* __restrict__ check, double tol2) {
    if (done(check, tol2)) return;
    // Programmatic dependent launches: the next kernel of the cycle may be scheduled now; u and
    // b are read after griddepcontrol.wait (a no-op for an ordinary launch).
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const int num_leaves = (int)t.num_leaves;
    const int64_t q = (int64_t)blockIdx.x * kThreads + threadIdx.x;
    if (q >= num_leaves) return;
    const int4 o = t.origin[q];
    if ((((o.x + o.y + o.z) >> 3) & 1) != colour) {
        if (zero) {  // from u = 0 the other colour writes 0
            asm volatile("griddepcontrol.wait;" ::: "memory");
            u[q] = 0.f;
        }
        return;
    }
    asm volatile("griddepcontrol.wait;" ::: "memory");
    int missing;
    if (zero) {
        // u = 0 before this sweep: no neighbour is read.
        float unused = level_nsum<0, false>(nb8, u, (int)q, 0, 0, 0, num_leaves, missing);
        (void)unused;
        u[q] = omega * (-h2 * b[q]) / (6.0f + gamma * (float)missing);
        return;
    }
    const float sum = level_nsum<0>(nb8, u, (int)q, 0, 0, 0, num_leaves, missing);
    const float uq = u[q];
    u[q] = uq + omega * ((sum - h2 * b[q]) / (6.0f + gamma * (float)missing) - uq);
}

// All SOR sweeps of the coarsest level (one cell per leaf) in one launch of a thread-block
// cluster, in place of two launches per sweep. CTA r of the cluster holds the cells of leaves
// [r P, r P + P) (P = ceil(L / CTAs)): their values u (and a zero past them, the value of
// a missing neighbour), right-hand sides b and a 32-byte record per cell, made once per context
// by coarse_table_kernel: the six face neighbours as (CTA rank << 16) | index in that CTA's u,
// the diagonal 6 + gamma missing, the cell's index; colour-0 records from the front of the
// table, colour-1 records from the back. Neighbours' values are read through the cluster's
// shared memory window (distributed shared memory), and a cluster barrier separates the
// colours. The arithmetic is coarsest_sweep_kernel's, in its order: the values are its values.
// The cluster has 16 CTAs (a non-portable size) where the device schedules that, else 8.
constexpr int kCoarseThreads = 1024, kCoarseUnroll = 3;
constexpr int kCoarseCellBytes = 32 + 4 + 4;  // the record, u, b (plus 4 bytes: u's zero)

__device__ __forceinline__ void cluster_barrier() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

__device__ __forceinline__ uint32_t cluster_ctarank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}

// The shared::cluster address of shared::cta address `a` in the CTA of rank `rank`.
__device__ __forceinline__ uint32_t cluster_map(uint32_t a, uint32_t rank) {
    uint32_t d;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(rank));
    return d;
}

__device__ __forceinline__ float ld_cluster(uint32_t addr) {
    float v;
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(addr));
    return v;
}

// The records of CTA r's cells (block r of one per CTA of the cluster), and its colour counts.
__global__ void __launch_bounds__(kCoarseThreads) coarse_table_kernel(TopoView t, const int4* __restrict__ nb8,
                                                                      uint4* __restrict__ table, int* __restrict__ counts,
                                                                      int per_cta, float gamma) {
    __shared__ int s_count[2];
    const int P = per_cta, tid = (int)threadIdx.x, r = (int)blockIdx.x;
    const int num_leaves = (int)t.num_leaves;
    const int lo = r * P, n = max(0, min(num_leaves - lo, P));
    if (tid == 0) s_count[0] = s_count[1] = 0;
    __syncthreads();
    uint4* rec = table + (size_t)2 * P * r;
    for (int i = tid; i < n; i += kCoarseThreads) {
        const int leaf = lo + i;
        const int4 f0 = nb8[2 * leaf], f1 = nb8[2 * leaf + 1];
        const int nbl[6] = {f0.x, f0.y, f0.z, f0.w, f1.x, f1.y};
        uint32_t w[6];
        int missing = 0;
#pragma unroll
        for (int k = 0; k < 6; ++k) {
            const int m = nbl[k];
            if (m >= num_leaves) {
                ++missing;
                w[k] = ((uint32_t)r << 16) | (uint32_t)P;
            } else {
                const int q = m / P;
                w[k] = ((uint32_t)q << 16) | (uint32_t)(m - q * P);
            }
        }
        const float d = 6.0f + gamma * (float)missing;
        const int4 o = t.origin[leaf];
        const int slot = (((o.x + o.y + o.z) >> 3) & 1) == 0 ? atomicAdd(&s_count[0], 1)
                                                               : P - 1 - atomicAdd(&s_count[1], 1);
        rec[2 * slot] = make_uint4(w[0], w[1], w[2], w[3]);
        rec[2 * slot + 1] = make_uint4(w[4], w[5], __float_as_uint(d), (uint32_t)i);
    }
    __syncthreads();
    if (tid == 0) {
        counts[2 * r] = s_count[0];
        counts[2 * r + 1] = s_count[1];
    }
}

__global__ void __launch_bounds__(kCoarseThreads, 1)
    coarsest_cluster_kernel(const uint4* __restrict__ table, const int* __restrict__ counts, float* __restrict__ u_out,
                            const float* b, int num_leaves, int per_cta, int sweeps, float omega, float h2,
                            const double* __restrict__ check, double tol2) {
    extern __shared__ __align__(16) unsigned char coarse_smem[];
    __shared__ float s_skip;
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const int P = per_cta, tid = (int)threadIdx.x;
    uint4* srec = reinterpret_cast<uint4*>(coarse_smem);
    float* su = reinterpret_cast<float*>(srec + 2 * P);  // P + 1 values, su[P] = 0
    float* sb = su + P + 1;
    const uint32_t rank = cluster_ctarank();
    const int lo = (int)rank * P, n = max(0, min(num_leaves - lo, P));
    const int c0 = __ldg(counts + 2 * rank), c1 = __ldg(counts + 2 * rank + 1);
    // The records (the topology only) before the wait on the preceding kernel.
    const uint4* g = table + (size_t)2 * P * rank;
    for (int k = tid; k < 2 * P; k += kCoarseThreads) srec[k] = __ldg(g + k);
    if (tid == 0) {
        su[P] = 0.f;
        s_skip = 0.f;
    }
    asm volatile("griddepcontrol.wait;" ::: "memory");
    if (rank == 0 && tid == 0 && done(check, tol2)) s_skip = 1.f;
    for (int i = tid; i < n; i += kCoarseThreads) sb[i] = b[lo + i];
    cluster_barrier();
    // Every CTA takes rank 0's decision, so all or none reach the sweeps' barriers; rank 0's
    // memory stays until each has read it.
    if (ld_cluster(cluster_map((uint32_t)__cvta_generic_to_shared(&s_skip), 0)) != 0.f) {
        cluster_barrier();
        return;
    }
    const uint32_t su_addr = (uint32_t)__cvta_generic_to_shared(su);
    for (int it = 0; it < sweeps; ++it) {
        for (int colour = 0; colour < 2; ++colour) {
            const int begin = colour ? P - c1 : 0, end = colour ? P : c0;
            if (it == 0 && colour == 0) {
                // u = 0 before this sweep: no neighbour is read, the other colour is set to 0.
                for (int j = begin + tid; j < end; j += kCoarseThreads) {
                    const uint4 q = srec[2 * j + 1];
                    su[q.w] = omega * (-h2 * sb[q.w]) / __uint_as_float(q.z);
                }
                for (int j = P - c1 + tid; j < P; j += kCoarseThreads) su[srec[2 * j + 1].w] = 0.f;
            } else {
                // kCoarseUnroll cells per thread at a time: every load issued before the first use.
                for (int j0 = begin + tid; j0 < end; j0 += kCoarseUnroll * kCoarseThreads) {
                    uint4 qa[kCoarseUnroll], qb[kCoarseUnroll];
                    float v[kCoarseUnroll][6];
#pragma unroll
                    for (int k = 0; k < kCoarseUnroll; ++k) {
                        const int j = j0 + k * kCoarseThreads;
                        if (j < end) {
                            qa[k] = srec[2 * j];
                            qb[k] = srec[2 * j + 1];
                        }
                    }
#pragma unroll
                    for (int k = 0; k < kCoarseUnroll; ++k) {
                        if (j0 + k * kCoarseThreads < end) {
                            const uint32_t w[6] = {qa[k].x, qa[k].y, qa[k].z, qa[k].w, qb[k].x, qb[k].y};
#pragma unroll
                            for (int e = 0; e < 6; ++e)
                                v[k][e] = ld_cluster(cluster_map(su_addr + ((w[e] & 0xffffu) << 2), w[e] >> 16));
                        }
                    }
#pragma unroll
                    for (int k = 0; k < kCoarseUnroll; ++k) {
                        if (j0 + k * kCoarseThreads < end) {
                            float sum = v[k][0];
                            sum += v[k][1];
                            sum += v[k][2];
                            sum += v[k][3];
                            sum += v[k][4];
                            sum += v[k][5];
                            const uint32_t i = qb[k].w;
                            const float uq = su[i];
                            su[i] = uq + omega * ((sum - h2 * sb[i]) / __uint_as_float(qb[k].z) - uq);
                        }
                    }
                }
            }
            cluster_barrier();
        }
    }
    // After the last barrier no CTA reads another's memory.
    for (int i = tid; i < n; i += kCoarseThreads) u_out[lo + i] = su[i];
}

// The same sweep at level 1 (4^3 cells per leaf) by rows: one thread per z-row (4 contiguous
// floats), which updates its 2 cells of the colour from 16-byte loads of the row, its right-hand
// side and its 4 x/y neighbour rows (across a face, the neighbour leaf's row; a missing leaf adds
// gamma to the diagonal) and the values past its z ends, and stores the row back whole (no other
// thread writes it in this sweep). Neighbours are summed in the order +x, -x, +y, -y, +z, -z:
// 7 loads for 2 updates. Selects pick the colour's two cells
// before the arithmetic: a loop over the four that skips two ran all four for half the lanes each (95.6M
// voxels 19.5 -> 17.5 us).
__global__ void __launch_bounds__(kThreads) level1_smooth_rows_kernel(const int4* __restrict__ nb8, float* u,
                                                                      const float* b, int num_leaves,
                                                                      int colour, float omega, float h2,
                                                                      float gamma, const double* __restrict__ check,
                                                                      double tol2) {
    if (done(check, tol2)) return;
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const int64_t tid = (int64_t)blockIdx.x * kThreads + threadIdx.x;
    if (tid >= ((int64_t)num_leaves << 4)) return;
    const int leaf = (int)(tid >> 4), x = (int)(tid >> 2) & 3, y = (int)tid & 3;
    const int4 f0 = __ldg(nb8 + 2 * leaf), f1 = __ldg(nb8 + 2 * leaf + 1);
    auto row_of = [&](int l, int a, int c2) { return ((int64_t)l << 6) + (((a << 2) + c2) << 2); };
    const int lxp = x < 3 ? leaf : f0.x, lxm = x > 0 ? leaf : f0.y, lyp = y < 3 ? leaf : f0.z, lym = y > 0 ? leaf : f0.w;
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const float4 z4 = make_float4(0.f, 0.f, 0.f, 0.f);
    auto ld4 = [&](int l, int64_t off) { return l < num_leaves ? *reinterpret_cast<const float4*>(u + off) : z4; };
    const int64_t own = row_of(leaf, x, y);
    // The row's cells of the colour are z = p and p + 2: one of them lies at a z end of the leaf.
    const bool p = ((x + y + colour) & 1) != 0;
    const int lz = p ? f1.x : f1.y;
    const float4 bb = *reinterpret_cast<const float4*>(b + own), c = *reinterpret_cast<const float4*>(u + own);
    const float4 xp = ld4(lxp, row_of(lxp, (x + 1) & 3, y)), xm = ld4(lxm, row_of(lxm, (x - 1) & 3, y));
    const float4 yp = ld4(lyp, row_of(lyp, x, (y + 1) & 3)), ym = ld4(lym, row_of(lym, x, (y - 1) & 3));
    const float end = lz < num_leaves ? u[row_of(lz, x, y) + (p ? 0 : 3)] : 0.f;
    const int lateral = (lxp >= num_leaves) + (lxm >= num_leaves) + (lyp >= num_leaves) + (lym >= num_leaves);
    const int ends = lz >= num_leaves;
    auto relax = [&](float vxp, float vxm, float vyp, float vym, float vzp, float vzm, float vb, float vc, int missing) {
        float sum = vxp;
        sum += vxm;
        sum += vyp;
        sum += vym;
        sum += vzp;
        sum += vzm;
        return vc + omega * ((sum - h2 * vb) / (6.0f + gamma * (float)missing) - vc);
    };
    auto lo = [&](const float4& v) { return p ? v.y : v.x; };
    auto hi = [&](const float4& v) { return p ? v.w : v.z; };
    const float mid = p ? c.z : c.y;  // between the two
    const float r0 = relax(lo(xp), lo(xm), lo(yp), lo(ym), mid, p ? c.x : end, lo(bb), lo(c), lateral + (p ? 0 : ends));
    const float r1 = relax(hi(xp), hi(xm), hi(yp), hi(ym), p ? end : c.w, mid, hi(bb), hi(c), lateral + (p ? ends : 0));
    *reinterpret_cast<float4*>(u + own) = p ? make_float4(c.x, r0, c.z, r1) : make_float4(r0, c.y, r1, c.w);
}

// The same at level 2 (2^3 cells per leaf): one thread per (leaf, x), whose four cells hold two of the
// colour, (y, z) = (0, p) and (1, 1 - p); 8 loads for the two updates, where a thread per cell of the colour
// made 16 (95.6M voxels 5.9 -> 4.9 us).
__global__ void __launch_bounds__(kThreads) level2_smooth_kernel(const int4* __restrict__ nb8, float* u,
                                                                 const float* b, int num_leaves, int colour,
                                                                 float omega, float h2, float gamma,
                                                                 const double* __restrict__ check, double tol2) {
    if (done(check, tol2)) return;
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const int64_t tid = (int64_t)blockIdx.x * kThreads + threadIdx.x;
    if (tid >= ((int64_t)num_leaves << 1)) return;
    const int leaf = (int)(tid >> 1), x = (int)tid & 1;
    const int4 f0 = __ldg(nb8 + 2 * leaf), f1 = __ldg(nb8 + 2 * leaf + 1);
    const bool p = ((x + colour) & 1) != 0;
    const int lx = x ? f0.x : f0.y, lza = p ? f1.x : f1.y, lzb = p ? f1.y : f1.x;
    asm volatile("griddepcontrol.wait;" ::: "memory");
    auto quad = [&](const float* q, int l, int cx) { return *reinterpret_cast<const float4*>(q + ((int64_t)l << 3) + 4 * cx); };
    auto cell = [&](int l, int y, int z) { return l < num_leaves ? u[((int64_t)l << 3) + 4 * x + 2 * y + z] : 0.f; };
    // A quad's cells: .x (0, 0), .y (0, 1), .z (1, 0), .w (1, 1).
    const float4 c = quad(u, leaf, x), in = quad(u, leaf, x ^ 1), bb = quad(b, leaf, x);
    const float4 out = lx < num_leaves ? quad(u, lx, x ^ 1) : make_float4(0.f, 0.f, 0.f, 0.f);
    const float ym = cell(f0.w, 1, p ? 1 : 0), yp = cell(f0.z, 0, p ? 0 : 1);
    const float za = cell(lza, 0, p ? 0 : 1), zb = cell(lzb, 1, p ? 1 : 0);
    auto relax = [&](float vxp, float vxm, float vyp, float vym, float vzp, float vzm, float vb, float vc, int missing) {
        float sum = vxp;
        sum += vxm;
        sum += vyp;
        sum += vym;
        sum += vzp;
        sum += vzm;
        return vc + omega * ((sum - h2 * vb) / (6.0f + gamma * (float)missing) - vc);
    };
    auto lo = [&](const float4& v) { return p ? v.y : v.x; };  // (0, p)
    auto hi = [&](const float4& v) { return p ? v.z : v.w; };  // (1, 1 - p)
    auto plus = [&](float i, float o) { return x ? o : i; };   // across +x: the other half inside, or the next leaf
    const int mx = lx >= num_leaves;
    const float ra = relax(plus(lo(in), lo(out)), plus(lo(out), lo(in)), p ? c.w : c.z, ym, p ? za : c.y, p ? c.x : za, lo(bb), lo(c),
                           mx + (f0.w >= num_leaves) + (lza >= num_leaves));
    const float rb = relax(plus(hi(in), hi(out)), plus(hi(out), hi(in)), yp, p ? c.x : c.y, p ? c.w : zb, p ? zb : c.z, hi(bb), hi(c),
                           mx + (f0.z >= num_leaves) + (lzb >= num_leaves));
    *reinterpret_cast<float4*>(u + ((int64_t)leaf << 3) + 4 * x) = p ? make_float4(c.x, ra, rb, c.w) : make_float4(ra, c.y, c.z, rb);
}

// bc (level LG - 1) = the mean of the residuals b - (sum - (6 + gamma missing) u) / h2 of each
// coarse cell's 8 children at level LG.
template <int LG>
__global__ void __launch_bounds__(kThreads) mgl_restrict_kernel(const int4* __restrict__ nb8, const float* u,
                                                                const float* b, float* bc,
                                                                int num_leaves, float inv_h2, float gamma,
                                                                const double* __restrict__ check, double tol2) {
    if (done(check, tol2)) return;
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const int64_t q = (int64_t)blockIdx.x * kThreads + threadIdx.x;
    if (q >= ((int64_t)num_leaves << (3 * (LG - 1)))) return;
    const LevelCell<LG - 1> cc = level_cell<LG - 1>(q);
    float sum = 0.f;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        const int x = 2 * cc.x + (k >> 2), y = 2 * cc.y + ((k >> 1) & 1), z = 2 * cc.z + (k & 1);
        const int64_t f = ((int64_t)cc.leaf << (3 * LG)) + (((x << LG) + y) << LG) + z;
        int missing;
        const float ns = level_nsum<LG>(nb8, u, cc.leaf, x, y, z, num_leaves, missing);
        sum += b[f] - (ns - (6.0f + gamma * (float)missing) * u[f]) * inv_h2;
    }
    bc[q] = 0.125f * sum;
}

// The same from level 1 to level 2, one thread per level-2 column (X, Y) (two cells): the 2 x 2 rows of
// level 1 under it and the 8 beside them as 16-byte loads. Each cell's children are added in the
// order of mgl_restrict_kernel, each one's neighbours in the sweeps' order. The first
// red sweep of level 2 from u = 0 is made in passing. 95.6M voxels: 34 -> 19 us.
__global__ void __launch_bounds__(kThreads, 3) restrict_level1_kernel(const int4* __restrict__ nb8,
                                                                      const float* u, const float* b, float* b2, float* u2,
                                                                      int num_leaves, float inv_h2,
                                                                      float gamma, float omega2, float h22, float gamma2,
                                                                      const double* __restrict__ check, double tol2) {
    if (done(check, tol2)) return;
    const int64_t tid = (int64_t)blockIdx.x * kThreads + threadIdx.x;
    if (tid >= ((int64_t)num_leaves << 2)) return;
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const int leaf = (int)(tid >> 2), X = (int)(tid >> 1) & 1, Y = (int)tid & 1;
    const int4 f0 = __ldg(nb8 + 2 * leaf), f1 = __ldg(nb8 + 2 * leaf + 1);
    const int lxp = X < 1 ? leaf : f0.x, lxm = X > 0 ? leaf : f0.y, lyp = Y < 1 ? leaf : f0.z, lym = Y > 0 ? leaf : f0.w;
    const bool mxp = lxp >= num_leaves, mxm = lxm >= num_leaves, myp = lyp >= num_leaves, mym = lym >= num_leaves;
    const bool mzp = f1.x >= num_leaves, mzm = f1.y >= num_leaves;
    asm volatile("griddepcontrol.wait;" ::: "memory");
    auto ld4 = [&](const float* p, int l, int x, int y) {
        return *reinterpret_cast<const float4*>(p + ((int64_t)l << 6) + (((x & 3) << 2) + (y & 3)) * 4);
    };
    const float4 z4 = make_float4(0.f, 0.f, 0.f, 0.f);
    const int x0 = 2 * X, y0 = 2 * Y;
    float4 c[2][2], r[2][2], xp[2], xm[2], yp[2], ym[2];
    float zlo[2][2], zhi[2][2];
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            c[i][j] = ld4(u, leaf, x0 + i, y0 + j);
            r[i][j] = ld4(b, leaf, x0 + i, y0 + j);
            const int row = ((x0 + i) * 4 + y0 + j) * 4;
            zlo[i][j] = mzm ? 0.f : u[((int64_t)f1.y << 6) + row + 3];
            zhi[i][j] = mzp ? 0.f : u[((int64_t)f1.x << 6) + row];
        }
#pragma unroll
    for (int k = 0; k < 2; ++k) {  // k: the coordinate along the side
        xp[k] = mxp ? z4 : ld4(u, lxp, x0 + 2, y0 + k);
        xm[k] = mxm ? z4 : ld4(u, lxm, x0 - 1, y0 + k);
        yp[k] = myp ? z4 : ld4(u, lyp, x0 + k, y0 + 2);
        ym[k] = mym ? z4 : ld4(u, lym, x0 + k, y0 - 1);
    }
    auto at = [](const float4& v, int z) { return z == 0 ? v.x : z == 1 ? v.y : z == 2 ? v.z : v.w; };
    float m[2];
#pragma unroll
    for (int Z = 0; Z < 2; ++Z) {
        float sum = 0.f;
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            const int i = k >> 2, j = (k >> 1) & 1, z = 2 * Z + (k & 1);
            const int missing = (i ? mxp : mxm) + (j ? myp : mym) + (z == 3 && mzp) + (z == 0 && mzm);
            float ns = at(i ? xp[j] : c[1][j], z);
            ns += at(i ? c[0][j] : xm[j], z);
            ns += at(j ? yp[i] : c[i][1], z);
            ns += at(j ? c[i][0] : ym[i], z);
            ns += z < 3 ? at(c[i][j], z + 1) : zhi[i][j];
            ns += z > 0 ? at(c[i][j], z - 1) : zlo[i][j];
            sum += at(r[i][j], z) - (ns - (6.0f + gamma * (float)missing) * at(c[i][j], z)) * inv_h2;
        }
        m[Z] = 0.125f * sum;
    }
    const int lateral = mxp + mxm + myp + mym;
    float w[2];
#pragma unroll
    for (int Z = 0; Z < 2; ++Z) {
        const int missing = lateral + (Z ? mzp : mzm);
        w[Z] = ((X + Y + Z) & 1) ? 0.f : omega2 * (-h22 * m[Z]) / (6.0f + gamma2 * (float)missing);
    }
    const int64_t off = ((int64_t)leaf << 3) + (((X << 1) + Y) << 1);
    *reinterpret_cast<float2*>(b2 + off) = make_float2(m[0], m[1]);
    *reinterpret_cast<float2*>(u2 + off) = make_float2(w[0], w[1]);
}

// Prolongation, one thread per coarse cell (level LC, 2^LC cells per leaf side): the coarse
// correction at the cell and its 26 neighbours (across faces, edges and corners of the leaf from
// the 27-neighbour table, 0 outside the domain), then each of the cell's 8 children at level
// LC + 1 takes the trilinear interpolation between cell centres: along each axis 3/4 of the
// parent and 1/4 of the parent's neighbour on the child's side.
template <int LC>
__device__ __forceinline__ void gather27(const TopoView& t, const float* uc, int leaf, int X, int Y, int Z,
                                         float v[27]) {
    constexpr int sc = 1 << LC;
#pragma unroll
    for (int k = 0; k < 27; ++k) {
        int cx = X + k / 9 - 1, cy = Y + (k / 3) % 3 - 1, cz = Z + k % 3 - 1;
        const int ox = cx < 0 ? -1 : (cx >= sc ? 1 : 0), oy = cy < 0 ? -1 : (cy >= sc ? 1 : 0),
                  oz = cz < 0 ? -1 : (cz >= sc ? 1 : 0);
        int l = leaf;
        if (ox | oy | oz) l = __ldg(t.nbr27 + (int64_t)leaf * 27 + (ox + 1) * 9 + (oy + 1) * 3 + (oz + 1));
        cx -= ox * sc, cy -= oy * sc, cz -= oz * sc;
        v[k] = l < 0 ? 0.f : uc[((int64_t)l << (3 * LC)) + (((cx << LC) + cy) << LC) + cz];
    }
}

// The interpolated value of child (i, j, k) (each 0 or 1) from the gathered neighbourhood.
__device__ __forceinline__ float interp8(const float v[27], int i, int j, int k) {
    const int sx = i ? 1 : -1, sy = j ? 1 : -1, sz = k ? 1 : -1;
    float sum = 0.f;
#pragma unroll
    for (int q = 0; q < 8; ++q) {
        const int a = q >> 2, bb = (q >> 1) & 1, e = q & 1;
        const float w = (a ? 0.25f : 0.75f) * (bb ? 0.25f : 0.75f) * (e ? 0.25f : 0.75f);
        sum += w * v[(1 + a * sx) * 9 + (1 + bb * sy) * 3 + (1 + e * sz)];
    }
    return sum;
}

// The colour-split FP16 layout of the inner solve: a leaf's colour-0 values, then its colour-1 values;
// row (x, y) at R = 32 ((x + y) & 1) + 4 x + (y >> 1) within a colour, entry z >> 1 of the row.
__device__ __forceinline__ float h16(const __half* p, uint32_t i) { return __half2float(p[i]); }

// The 8 values of a row, packed: its entries in the two colour blocks, at row position R (colour c
// holds z = 2 j + ((x + y + c) & 1) at entries 4 R + j).
struct Row16 {
    uint2 c0, c1;
};
__device__ __forceinline__ Row16 row16(const __half* p, int l, int R) {
    const uint2* q = reinterpret_cast<const uint2*>(p + ((uint32_t)l << 9) + 4 * R);
    return Row16{q[0], q[64]};
}
// Value z of a row with x + y of parity kPar.
template <int kPar>
__device__ __forceinline__ float row_at(const Row16& r, int z) {
    const uint2 v = ((z + kPar) & 1) ? r.c1 : r.c0;
    const uint32_t w = (z & 4) ? v.y : v.x;
    return __half2float(__ushort_as_half((unsigned short)((z & 2) ? (w >> 16) : (w & 0xFFFFu))));
}

// Fine level of the FP16 cycle: b1 (4^3 cells per leaf) = the mean of the residuals
// r^ - (sum - 6 e) (unit spacing; a missing leaf is the zero leaf past the last one, p = 0 outside
// the domain) of each level-1 cell's 8 voxels, e and r^ in the colour-split layout.
//
// One thread per level-1 column (X, Y): the 2 x 2 fine rows under it, whose parities the code then
// knows (no selects), and the 8 rows beside them, each loaded once for the two or more voxels that
// read it: 32 row loads for 32 voxels where a thread per fine row made 48, and no shuffles (95.6M
// voxels 75 -> 55 us, 23.1M voxels 28 -> 23 us; the bytes need 65 and 16, less what stays in L2). The column's first red sweep of level 1 from u = 0 is made
// in passing.
template <int kPar>
__device__ __forceinline__ void row_residual(const Row16& c, const Row16& xp, const Row16& xm, const Row16& yp,
                                             const Row16& ym, const Row16& rh, float zlo, float zhi, float part[4]) {
#pragma unroll
    for (int Z = 0; Z < 4; ++Z) {
        float sum = 0.f;
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            const int z = 2 * Z + k;
            const float zm = z > 0 ? row_at<kPar>(c, z > 0 ? z - 1 : 0) : zlo, zp = z < 7 ? row_at<kPar>(c, z < 7 ? z + 1 : 7) : zhi;
            sum += row_at<kPar>(rh, z) - (row_at<kPar ^ 1>(xp, z) + row_at<kPar ^ 1>(xm, z) + row_at<kPar ^ 1>(yp, z) +
                                          row_at<kPar ^ 1>(ym, z) + zp + zm - 6.0f * row_at<kPar>(c, z));
        }
        part[Z] = sum;
    }
}

__global__ void __launch_bounds__(kThreads, 3) mg16_restrict_kernel(const int4* __restrict__ nb8, const __half* e,
                                                                    const __half* __restrict__ rhat, float* __restrict__ b1,
                                                                    float* __restrict__ u1, int num_leaves, float omega,
                                                                    float h2, float gamma, const double* __restrict__ check,
                                                                    double tol2) {
    if (done(check, tol2)) return;
    const int64_t tid = (int64_t)blockIdx.x * kThreads + threadIdx.x;
    if (tid >= ((int64_t)num_leaves << 4)) return;
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const int leaf = (int)(tid >> 4), X = (int)(tid >> 2) & 3, Y = (int)tid & 3;
    const int4 f0 = __ldg(nb8 + 2 * leaf), f1 = __ldg(nb8 + 2 * leaf + 1);
    // Row (2 X + i, 2 Y + j) lies at 8 X + Y + 4 i, past 32 where i + j is odd.
    const int R = 8 * X + Y;
    const int lxp = X < 3 ? leaf : f0.x, lxm = X > 0 ? leaf : f0.y, lyp = Y < 3 ? leaf : f0.z, lym = Y > 0 ? leaf : f0.w;
    const int Rxp = 8 * ((X + 1) & 3) + Y, Rxm = 8 * ((X + 3) & 3) + 4 + Y;  // rows (2 X + 2, .), (2 X - 1, .)
    const int Ryp = 8 * X + ((Y + 1) & 3), Rym = 8 * X + ((Y + 3) & 3);      // rows (., 2 Y + 2), (., 2 Y - 1)
    Row16 rh[2][2], c[2][2], xp[2], xm[2], yp[2], ym[2];
    float zlo[2][2], zhi[2][2];
    asm volatile("griddepcontrol.wait;" ::: "memory");  // e is the preceding half-sweep's
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            const int q = R + 4 * i + 32 * ((i + j) & 1);
            c[i][j] = row16(e, leaf, q);
            rh[i][j] = row16(rhat, leaf, q);
            // z = 7 of the leaf below, z = 0 of the leaf above.
            const int par = (i + j) & 1;
            zlo[i][j] = h16(e, ((uint32_t)f1.y << 9) + (par ? 0 : 256) + 4 * q + 3);
            zhi[i][j] = h16(e, ((uint32_t)f1.x << 9) + (par ? 256 : 0) + 4 * q);
        }
#pragma unroll
    for (int k = 0; k < 2; ++k) {  // k: the coordinate along the side
        xp[k] = row16(e, lxp, Rxp + (k ? 32 : 0));
        xm[k] = row16(e, lxm, Rxm + (k ? 0 : 32));
        yp[k] = row16(e, lyp, Ryp + (k ? 4 + 32 : 0));
        ym[k] = row16(e, lym, Rym + (k ? 4 : 32));
    }
    float part[2][2][4];
    row_residual<0>(c[0][0], c[1][0], xm[0], c[0][1], ym[0], rh[0][0], zlo[0][0], zhi[0][0], part[0][0]);
    row_residual<1>(c[0][1], c[1][1], xm[1], yp[0], c[0][0], rh[0][1], zlo[0][1], zhi[0][1], part[0][1]);
    row_residual<1>(c[1][0], xp[0], c[0][0], c[1][1], ym[1], rh[1][0], zlo[1][0], zhi[1][0], part[1][0]);
    row_residual<0>(c[1][1], xp[1], c[0][1], yp[1], c[1][0], rh[1][1], zlo[1][1], zhi[1][1], part[1][1]);
    float m[4];
#pragma unroll
    for (int Z = 0; Z < 4; ++Z)
        m[Z] = 0.125f * ((part[0][0][Z] + part[0][1][Z]) + (part[1][0][Z] + part[1][1][Z]));
    // The first red sweep of level 1 from u = 0 reads no neighbour: made here.
    const int lateral = (lxp >= num_leaves) + (lxm >= num_leaves) + (lyp >= num_leaves) + (lym >= num_leaves);
    float w[4];
#pragma unroll
    for (int Z = 0; Z < 4; ++Z) {
        const int missing = lateral + (Z == 3 && f1.x >= num_leaves) + (Z == 0 && f1.y >= num_leaves);
        w[Z] = ((X + Y + Z) & 1) ? 0.f : omega * (-h2 * m[Z]) / (6.0f + gamma * (float)missing);
    }
    const int64_t off = ((int64_t)leaf << 6) + (((X << 2) + Y) << 2);
    *reinterpret_cast<float4*>(b1 + off) = make_float4(m[0], m[1], m[2], m[3]);
    *reinterpret_cast<float4*>(u1 + off) = make_float4(w[0], w[1], w[2], w[3]);
}

// e (FP16, colour-split) += the level-1 correction interpolated trilinearly, one rounding per
// value. Along z each voxel takes 3/4 of its parent Z = z / 2 and 1/4 of Z - 1 (z even) or Z + 1
// (odd), and the same along x and y; 0 where a leaf is missing.
//
// One thread per level-1 column (X, Y): its 2 x 2 fine rows, from the 3 x 3 level-1 columns around
// it (4 contiguous floats each, and one value past each end), interpolated along z once for the
// rows that share them. A thread per fine row loaded 4 columns and 12 table entries for 8 voxels and
// was bound by issue: 95.6M voxels 102 -> 51 us, 23.1M voxels 37 -> 20 us.
__global__ void __launch_bounds__(kThreads, 3) mg16_prolong_kernel(TopoView t, const float* u1, __half* e,
                                                                   const double* __restrict__ check, double tol2) {
    if (done(check, tol2)) return;
    const int64_t tid = (int64_t)blockIdx.x * kThreads + threadIdx.x;
    if (tid >= (t.num_leaves << 4)) return;
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const int leaf = (int)(tid >> 4), X = (int)(tid >> 2) & 3, Y = (int)tid & 3;
    const int* nb = t.nbr27 + (int64_t)leaf * 27;
    const int lm0 = __ldg(nb + 12), lp0 = __ldg(nb + 14);
    asm volatile("griddepcontrol.wait;" ::: "memory");
    uint2* row = reinterpret_cast<uint2*>(e + ((uint32_t)leaf << 9) + 4 * (8 * X + Y));
    Row16 raw[2][2];
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            const uint2* q = row + 4 * i + 32 * ((i + j) & 1);
            raw[i][j] = Row16{q[0], q[64]};
        }
    float v[3][3][8];  // per column, along z: the fine voxels' interpolants
#pragma unroll
    for (int a = 0; a < 3; ++a)
#pragma unroll
        for (int b = 0; b < 3; ++b) {
            const int cx = X + a - 1, cy = Y + b - 1;
            const int ox = a == 0 ? (cx < 0 ? -1 : 0) : a == 2 ? (cx > 3 ? 1 : 0) : 0;
            const int oy = b == 0 ? (cy < 0 ? -1 : 0) : b == 2 ? (cy > 3 ? 1 : 0) : 0;
            int l = leaf, lm = lm0, lp = lp0;
            if (ox | oy) {
                const int* k = nb + (ox + 1) * 9 + (oy + 1) * 3;
                lm = __ldg(k), l = __ldg(k + 1), lp = __ldg(k + 2);
            }
            const int off = (((cx & 3) << 2) + (cy & 3)) << 2;
            const float4 m = l < 0 ? make_float4(0.f, 0.f, 0.f, 0.f)
                                   : *reinterpret_cast<const float4*>(u1 + ((int64_t)l << 6) + off);
            const float lo = lm < 0 ? 0.f : u1[((int64_t)lm << 6) + off + 3];
            const float hi = lp < 0 ? 0.f : u1[((int64_t)lp << 6) + off];
            const float col[6] = {lo, m.x, m.y, m.z, m.w, hi};
#pragma unroll
            for (int Z = 0; Z < 4; ++Z) {
                const float p = 0.75f * col[Z + 1];
                v[a][b][2 * Z] = fmaf(0.25f, col[Z], p);
                v[a][b][2 * Z + 1] = fmaf(0.25f, col[Z + 2], p);
            }
        }
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            const int par = (i + j) & 1, sx = i ? 2 : 0, sy = j ? 2 : 0;  // the columns the row leans to
            uint32_t h[8];
#pragma unroll
            for (int z = 0; z < 8; ++z) {
                float sum = 0.f;
                sum = fmaf(0.5625f, v[1][1][z], sum);
                sum = fmaf(0.1875f, v[1][sy][z], sum);
                sum = fmaf(0.1875f, v[sx][1][z], sum);
                sum = fmaf(0.0625f, v[sx][sy][z], sum);
                const float old = par ? row_at<1>(raw[i][j], z) : row_at<0>(raw[i][j], z);
                h[z] = __half_as_ushort(__float2half_rn(old + sum));
            }
            uint2* q = row + 4 * i + 32 * par;
            // Colour c holds z = 2 j + ((i + j + c) & 1).
            q[0] = make_uint2(h[par] | (h[2 + par] << 16), h[4 + par] | (h[6 + par] << 16));
            q[64] = make_uint2(h[1 - par] | (h[3 - par] << 16), h[5 - par] | (h[7 - par] << 16));
        }
}

// u (level LG) += the correction uc (level LG - 1), one thread per coarse cell.
template <int LG>
__global__ void __launch_bounds__(kThreads) mgl_prolong_kernel(TopoView t, const float* uc, float* u,
                                                               const double* __restrict__ check, double tol2) {
    if (done(check, tol2)) return;
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const int64_t q = (int64_t)blockIdx.x * kThreads + threadIdx.x;
    if (q >= (t.num_leaves << (3 * (LG - 1)))) return;
    const LevelCell<LG - 1> c = level_cell<LG - 1>(q);
    float v[27];
    gather27<LG - 1>(t, uc, c.leaf, c.x, c.y, c.z, v);
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        const int i = k >> 2, j = (k >> 1) & 1, l = k & 1;
        const int64_t f = ((int64_t)c.leaf << (3 * LG)) + ((((2 * c.x + i) << LG) + 2 * c.y + j) << LG) + 2 * c.z + l;
        u[f] += interp8(v, i, j, l);
    }
}

// The same from level 2 to level 1, one thread per level-2 column (X, Y): its two cells' 16 children
// are the 2 x 2 rows of level 1 above them, read and written as 16 bytes each; the 3 x 3 level-2
// columns around it are read once (8 bytes and one value past each end). The sums are interp8's, in
// its order. 95.6M voxels: 28 -> 14 us.
__global__ void __launch_bounds__(kThreads, 3) prolong_level2_kernel(TopoView t, const float* uc, float* u,
                                                                     const double* __restrict__ check, double tol2) {
    if (done(check, tol2)) return;
    const int64_t tid = (int64_t)blockIdx.x * kThreads + threadIdx.x;
    if (tid >= (t.num_leaves << 2)) return;
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const int leaf = (int)(tid >> 2), X = (int)(tid >> 1) & 1, Y = (int)tid & 1;
    const int* nb = t.nbr27 + (int64_t)leaf * 27;
    // The leaves of the columns: this one's and the one across the x side, the y side, both.
    int l[2][2][3];
#pragma unroll
    for (int a = 0; a < 2; ++a)
#pragma unroll
        for (int c = 0; c < 2; ++c) {
            const int* k = nb + 12 + (a ? (X ? 9 : -9) : 0) + (c ? (Y ? 3 : -3) : 0);
#pragma unroll
            for (int e = 0; e < 3; ++e) l[a][c][e] = __ldg(k + e);
        }
    l[0][0][1] = leaf;
    asm volatile("griddepcontrol.wait;" ::: "memory");
    float4* rows = reinterpret_cast<float4*>(u + ((int64_t)leaf << 6)) + 8 * X + 2 * Y;
    float4 f[2][2];
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 2; ++j) f[i][j] = rows[4 * i + j];
    // v[a][c][.]: the level-2 values Z = -1 .. 2 of column (a, c): 0 the own one, 1 the one on the
    // other side within the leaf, 2 the one across the leaf's side.
    float v[3][3][4];
#pragma unroll
    for (int a = 0; a < 3; ++a)
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const int cx = a == 0 ? X : X ^ 1, cy = c == 0 ? Y : Y ^ 1;
            const int off = ((cx << 1) + cy) << 1;
            const int(&q)[3] = l[a == 2][c == 2];
            const float2 m = q[1] < 0 ? make_float2(0.f, 0.f)
                                      : *reinterpret_cast<const float2*>(uc + ((int64_t)q[1] << 3) + off);
            v[a][c][0] = q[0] < 0 ? 0.f : uc[((int64_t)q[0] << 3) + off + 1];
            v[a][c][1] = m.x, v[a][c][2] = m.y;
            v[a][c][3] = q[2] < 0 ? 0.f : uc[((int64_t)q[2] << 3) + off];
        }
    // The neighbour on child i's side lies across the leaf's side where i == X, else within.
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            float add[4];
#pragma unroll
            for (int z = 0; z < 4; ++z) {
                const int Z = (z >> 1) + 1, zo = (z & 1) ? Z + 1 : Z - 1;
                float sum = 0.f;
#pragma unroll
                for (int q = 0; q < 8; ++q) {
                    const int a = q >> 2, c = (q >> 1) & 1, zz = (q & 1) ? zo : Z;
                    const float w = (a ? 0.25f : 0.75f) * (c ? 0.25f : 0.75f) * ((q & 1) ? 0.25f : 0.75f);
                    const float x0 = a ? (i == X ? v[2][0][zz] : v[1][0][zz]) : v[0][0][zz];
                    const float x1 = a ? (i == X ? v[2][1][zz] : v[1][1][zz]) : v[0][1][zz];
                    const float x2 = a ? (i == X ? v[2][2][zz] : v[1][2][zz]) : v[0][2][zz];
                    sum += w * (c ? (j == Y ? x2 : x1) : x0);
                }
                add[z] = sum;
            }
            float4 r = f[i][j];
            r.x += add[0], r.y += add[1], r.z += add[2], r.w += add[3];
            rows[4 * i + j] = r;
        }
}

}  // namespace

// One V-cycle on rhs b0 (n FP32 values, slot order) into u0 (n FP32, overwritten; starts at 0).
void mg_vcycle(Context& c, const float* b0, float* u0, const double* check, double tol2) {
    const int64_t L = c.topo.num_leaves;
    if (L == 0) return;
    const TopoView t = c.topo.view;
    float* u[kLevels];
    const float* b[kLevels];
    float* bw[kLevels];
    float* r[kLevels];
    int64_t cells[kLevels];
    for (int l = 0; l < kLevels; ++l) {
        const int lg = 3 - l;
        cells[l] = L << (3 * lg);
        r[l] = c.scratch_f32("mg_r" + std::to_string(l), (size_t)cells[l]);
        if (l == 0) {
            u[l] = u0, b[l] = b0, bw[l] = nullptr;
        } else {
            u[l] = c.scratch_f32("mg_u" + std::to_string(l), (size_t)cells[l]);
            bw[l] = c.scratch_f32("mg_b" + std::to_string(l), (size_t)cells[l]);
            b[l] = bw[l];
        }
    }
    auto smooth = [&](int l, int iters, float omega) {
        const float h2 = (float)(1 << (2 * l));
        for (int it = 0; it < iters; ++it)
            for (int colour = 0; colour < 2; ++colour) {
                mg_smooth_kernel<<<blocks(cells[l]), kThreads, 0, c.stream>>>(t, u[l], b[l], 3 - l, cells[l], colour, omega,
                                                                              h2, check, tol2);
                HNS_LAUNCHED();
            }
    };
    HNS_CUDA(cudaMemsetAsync(u0, 0, sizeof(float) * (size_t)cells[0], c.stream));
    for (int l = 0; l + 1 < kLevels; ++l) {
        if (l > 0) HNS_CUDA(cudaMemsetAsync(u[l], 0, sizeof(float) * (size_t)cells[l], c.stream));
        smooth(l, kPreSmooth, 1.0f);
        mg_residual_kernel<<<blocks(cells[l]), kThreads, 0, c.stream>>>(t, u[l], b[l], r[l], 3 - l, cells[l],
                                                                         1.0f / (float)(1 << (2 * l)), check, tol2);
        HNS_LAUNCHED();
        mg_restrict_kernel<<<blocks(cells[l + 1]), kThreads, 0, c.stream>>>(r[l], bw[l + 1], 3 - (l + 1), cells[l + 1],
                                                                             check, tol2);
        HNS_LAUNCHED();
    }
    HNS_CUDA(cudaMemsetAsync(u[kLevels - 1], 0, sizeof(float) * (size_t)cells[kLevels - 1], c.stream));
    smooth(kLevels - 1, kCoarseIters, kCoarseOmega);
    for (int l = kLevels - 2; l >= 0; --l) {
        mg_prolong_kernel<<<blocks(cells[l]), kThreads, 0, c.stream>>>(t, u[l + 1], u[l], 3 - l, cells[l], check, tol2);
        HNS_LAUNCHED();
        smooth(l, kPostSmooth, 1.0f);
    }
}

// One V-cycle of the FP16 inner solve L e = r^ (unit spacing) on the colour-split layout: e is
// refined in place (e_zero: e = 0 before the cycle). Fine level: kMgNu red-black iterations of
// the colour-split half-sweep at omega = 1 before and after the coarse correction; levels with
// 4, 2 and 1 cells per leaf side in FP32 with the wall-corrected operator, kMgNu iterations
// before and after at the first two, SOR sweeps at the last (coarsest_schedule).
namespace {
constexpr int kMgNu = 2;

// SOR sweeps and factor at the coarsest level (one cell per leaf), from how many leaves deep the
// domain is (D, max_leaf_depth): clamp(2 D + 2, 10, 20) sweeps at clamp(2 / (1 + sin(pi / 2 D)),
// 1.5, 1.75), the optimal SOR factor for an extent of 2 D cells. Measured (ms per step, cycles
// per solve 6 on the shell, 8-10 on the fire): shell512 (D = 4) 10 at 1.5: 3.90, 20 at 1.5: 4.17,
// 5 at 1.5: 3.76 (2 doubled the cycles); fire1024 (D = 15) 10 at 1.5: 29.9, 5 at 1.5: 41 with a
// solve above the tolerance at the outer cap, 20 at 1.5: 24.3, 20 at 1.75: 21.3, 40 at 1.8: 22.0.
void coarsest_schedule(Context& c, int& sweeps, float& omega) {
    const int d = std::max(1, max_leaf_depth(c));
    sweeps = std::min(20, std::max(10, 2 * d + 2));
    omega = std::min(1.75f, std::max(1.5f, 2.0f / (1.0f + std::sin(3.14159265f / (2.0f * (float)d)))));
}

// Kernels of the cycle are programmatic dependent launches: each lets the next be scheduled
// at its start and reads the data the preceding ones wrote after griddepcontrol.wait.
template <typename... KArgs, typename... Args>
void launch_pdl(const Context& c, void (*kern)(KArgs...), int64_t threads, Args... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(blocks(threads));
    cfg.blockDim = dim3(kThreads);
    cfg.stream = c.stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = c.add_inner_window(attr, 1);
    HNS_CUDA(cudaLaunchKernelEx(&cfg, kern, args...));
    HNS_LAUNCHED();
}

// Cell size squared, and what a missing neighbour adds to the diagonal, at level l.
float level_h2(int l) { return (float)(1 << (2 * l)); }
float level_gamma(int l) { return (float)((1 << l) - 1) / (float)((1 << l) + 1); }

// kMgNu red-black iterations at level l = 1 or 2. begun: the first red sweep, from u = 0, is made
// already (by the restriction).
void smooth_level(Context& c, const int4* nb8, float* u, const float* b, int l, bool begun, const double* check,
                  double tol2) {
    const int L = (int)c.topo.num_leaves;
    for (int s = begun ? 1 : 0; s < 2 * kMgNu; ++s) {
        if (l == 1)
            launch_pdl(c, level1_smooth_rows_kernel, (int64_t)L << 4, nb8, u, b, L, s & 1, 1.0f, level_h2(l), level_gamma(l),
                       check, tol2);
        else
            launch_pdl(c, level2_smooth_kernel, (int64_t)L << 1, nb8, u, b, L, s & 1, 1.0f, level_h2(l), level_gamma(l), check,
                       tol2);
    }
}

}  // namespace

// Settings shared by the contexts of a process on one device (raise_device_setting).
size_t raise_device_setting(int device, int which, size_t value) {
    static std::mutex mu;
    static std::map<std::pair<int, int>, size_t> in_force;
    std::lock_guard<std::mutex> lock(mu);
    size_t& cur = in_force[{device, which}];
    if (value <= cur) return cur;
    if (which == 0)
        HNS_CUDA(cudaFuncSetAttribute(coarsest_cluster_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)value));
    else
        HNS_CUDA(cudaDeviceSetLimit(cudaLimitPersistingL2CacheSize, value));
    cur = value;
    return cur;
}

namespace {
// The coarsest level's `sweeps` SOR sweeps from u = 0 (level 3, one cell per leaf): one cluster
// launch where the option allows it, the leaves fit the cluster's shared memory and the device
// can schedule the cluster, else two launches per sweep. Both give the same values.
void coarsest_solve(Context& c, const int4* nb8, float* u, const float* b, int sweeps, float omega,
                    const double* check, double tol2) {
    const int64_t L = c.topo.num_leaves;
    const float h2 = 64.0f, gamma = 7.0f / 9.0f;  // level 3: (2^3)^2, (2^3 - 1) / (2^3 + 1)
    auto per_cta = [&](int ctas) { return (L + ctas - 1) / ctas; };
    auto smem_of = [&](int ctas) { return (size_t)per_cta(ctas) * kCoarseCellBytes + 4; };
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[2];
    auto configure = [&](int ctas) {
        cfg.gridDim = dim3(ctas);
        cfg.blockDim = dim3(kCoarseThreads);
        cfg.dynamicSmemBytes = smem_of(ctas);
        cfg.stream = c.stream;
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = ctas;
        attr[0].val.clusterDim.y = 1;
        attr[0].val.clusterDim.z = 1;
        attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[1].val.programmaticStreamSerializationAllowed = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
    };
    bool fresh = false;
    if (c.coarse_solve == HNS_COARSE_CLUSTER && sweeps >= 1 && c.coarse_cluster_ok != 0 &&
        (c.coarse_cluster_ok < 0 || c.coarse_table_leaves != L)) {
        // The cluster size: the larger of 16 and 8 that holds the level and that the device schedules.
        c.coarse_cluster_ok = 0;
        int optin = 0;
        HNS_CUDA(cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, c.device));
        HNS_CUDA(cudaFuncSetAttribute(coarsest_cluster_kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
        for (int ctas : {16, 8}) {
            if (smem_of(ctas) + 16 > (size_t)optin) continue;  // + the kernel's static shared memory
            raise_device_setting(c.device, 0, smem_of(ctas));
            configure(ctas);
            int clusters = 0;
            if (cudaOccupancyMaxActiveClusters(&clusters, coarsest_cluster_kernel, &cfg) != cudaSuccess) {
                (void)cudaGetLastError();  // not schedulable at this size: try the next
                continue;
            }
            if (clusters >= 1) {
                c.coarse_cluster_ok = ctas;
                break;
            }
        }
        if (c.coarse_cluster_ok > 0) {
            const int ctas = c.coarse_cluster_ok;
            auto* table = reinterpret_cast<uint4*>(c.scratch_f32("mg16_coarse_records", (size_t)8 * L + 8 * ctas));
            auto* counts = reinterpret_cast<int*>(c.scratch_f32("mg16_coarse_counts", 2 * 16));
            coarse_table_kernel<<<ctas, kCoarseThreads, 0, c.stream>>>(c.topo.view, nb8, table, counts,
                                                                       (int)per_cta(ctas), gamma);
            HNS_LAUNCHED();
            if (!c.stream_capturing()) c.coarse_table_leaves = L;
            fresh = true;
        }
    }
    if (c.coarse_solve != HNS_COARSE_CLUSTER || sweeps < 1 || c.coarse_cluster_ok <= 0) {
        for (int s = 0; s < 2 * sweeps; ++s)
            launch_pdl(c, coarsest_sweep_kernel, L, c.topo.view, nb8, u, b, s & 1, (int)(s == 0), omega, h2, gamma, check, tol2);
        return;
    }
    const int ctas = c.coarse_cluster_ok;
    configure(ctas);
    // The kernel reads its records before griddepcontrol.wait: after a table made in this call,
    // an ordinary launch.
    cfg.numAttrs = fresh ? 1 : 2;
    const auto* table = reinterpret_cast<const uint4*>(c.scratch_f32("mg16_coarse_records", (size_t)8 * L + 8 * ctas));
    const auto* counts = reinterpret_cast<const int*>(c.scratch_f32("mg16_coarse_counts", 2 * 16));
    HNS_CUDA(cudaLaunchKernelEx(&cfg, coarsest_cluster_kernel, table, counts, u, b, (int)L, (int)per_cta(ctas), sweeps,
                                omega, h2, check, tol2));
    HNS_LAUNCHED();
}
}  // namespace

void mg16_vcycle(Context& c, const int* nb8, const void* rhat, void* e, bool e_zero, const double* check, double tol2) {
    const int64_t L = c.topo.num_leaves;
    if (L == 0) return;
    const TopoView t = c.topo.view;
    const auto* f8 = reinterpret_cast<const int4*>(nb8);
    const auto* r = static_cast<const __half*>(rhat);
    auto* eh = static_cast<__half*>(e);
    float* u[4] = {nullptr, nullptr, nullptr, nullptr};
    float* b[4] = {nullptr, nullptr, nullptr, nullptr};
    for (int l = 1; l < 4; ++l) {
        const size_t cells = (size_t)L << (3 * (3 - l));
        u[l] = c.scratch_f32("mg16_u" + std::to_string(l), cells);
        b[l] = c.scratch_f32("mg16_b" + std::to_string(l), cells);
    }
    auto fine = [&](bool zero_first) {
        for (int it = 0; it < kMgNu; ++it) {
            launch_rbgs_split_half(c, nb8, rhat, e, 0, zero_first && it == 0, 1.0f, check, tol2, false, true);
            launch_rbgs_split_half(c, nb8, rhat, e, 1, false, 1.0f, check, tol2, false, true);
        }
    };
    fine(e_zero);
    launch_pdl(c, mg16_restrict_kernel, L << 4, f8, (const __half*)eh, r, b[1], u[1], (int)L, 1.0f,
               level_h2(1), level_gamma(1), check, tol2);
    smooth_level(c, f8, u[1], b[1], 1, true, check, tol2);
    launch_pdl(c, restrict_level1_kernel, L << 2, f8, (const float*)u[1], (const float*)b[1], b[2], u[2], (int)L, 0.25f,
               level_gamma(1), 1.0f, level_h2(2), level_gamma(2), check, tol2);
    smooth_level(c, f8, u[2], b[2], 2, true, check, tol2);
    launch_pdl(c, mgl_restrict_kernel<1>, L, f8, (const float*)u[2], (const float*)b[2], b[3], (int)L, 1.0f / 16.0f,
               0.6f, check, tol2);
    int coarse_sweeps;
    float coarse_omega;
    coarsest_schedule(c, coarse_sweeps, coarse_omega);
    coarsest_solve(c, f8, u[3], b[3], coarse_sweeps, coarse_omega, check, tol2);
    launch_pdl(c, mgl_prolong_kernel<1>, L, t, (const float*)u[3], u[2], check, tol2);
    smooth_level(c, f8, u[2], b[2], 2, false, check, tol2);
    launch_pdl(c, prolong_level2_kernel, L << 2, t, (const float*)u[2], u[1], check, tol2);
    smooth_level(c, f8, u[1], b[1], 1, false, check, tol2);
    launch_pdl(c, mg16_prolong_kernel, L << 4, t, (const float*)u[1], eh, check, tol2);
    fine(false);
}

}  // namespace hns
