// Topology built on the device from a list of active voxels: the replacement for the
// reference's domain set-up -- the velocity grid's topology dilated by `padding` voxels with
// 26-neighbour (face, edge and vertex) dilation (src/SOP/HNanoSolver/SOP_HNanoSolver.cpp:280-285)
// and the ValueOnIndex grid built from the voxel list with voxelsToGrid
// (src/Cuda/HNanoSolver.cu:498-504). The solver's grids are leaf-dense, so the build produces
// the set of leaves that the dilated voxels touch, in NanoVDB leaf order, and the leaf tables.
//
//   1. The voxels' bounding box (and the check of their range): one read of the list.
//   2. A flag per leaf of the dilated bounding box, in the leaf lookup table that the grid needs
//      anyway: per voxel the leaves its dilation box reaches (per axis: -1 when z & 7 < padding,
//      +1 when (z & 7) + padding >= 8), found once per warp for its voxels of one leaf.
//   3. NanoVDB leaf order is root tile, then upper-node child, then lower-node child, each in
//      x, y, z order (PointsToGrid orders leaves this way). A lower node is 16^3 leaves, so the flags
//      are counted and then numbered node by node, the nodes in that order: one CTA per node of
//      the box, no sort.
//   4. Leaf origins and the table entries as the leaves are numbered, then the 27-neighbour table;
//      only the origins go back to the host (the context keeps a host copy).
// Bound by the two reads of the voxel list and by the call's allocations and three host waits: the
// band of a 512^3 shell (12M voxels, padding 2, 46,000 leaves), context made and destroyed, took
// 8.7 ms with a radix sort of one key per voxel (1.4 ms of kernels, 300 MB of temporary arrays), 2.1 ms
// with the tables in three allocations, and takes 1.7 ms with them in two, in a process that does
// nothing else (0.23 ms of kernels; an allocation and its release cost the host 0.6 ms, and more beside
// other contexts: 2.3 to 3.4 ms with three taking turns).
#include <cuda_runtime.h>

#include <algorithm>
#include <climits>
#include <cstdint>
#include <string>
#include <vector>

#include "hns_internal.cuh"

namespace hns {
namespace {

constexpr int kTopoThreads = 256;
// |coordinate| bound: the key holds a 12-bit biased root tile index per axis (coordinate >> 12).
constexpr int32_t kCoordLimit = (1 << 23) - 64;
constexpr int kMaxPadding = 8;

unsigned grid_for(int64_t n) { return (unsigned)((n + kTopoThreads - 1) / kTopoThreads); }

struct Box {
    int lo[3], dim[3];  // in leaf units
};

// Step 1: bounds[0..2] minima, [3..5] maxima of the coordinates, [6] set when one is out of range.
__global__ void __launch_bounds__(kTopoThreads) bounds_kernel(const int32_t* __restrict__ ijk, int64_t n,
                                                              int* __restrict__ bounds) {
    int lo[3] = {INT_MAX, INT_MAX, INT_MAX}, hi[3] = {INT_MIN, INT_MIN, INT_MIN};
    for (int64_t q = (int64_t)blockIdx.x * kTopoThreads + threadIdx.x; q < n; q += (int64_t)gridDim.x * kTopoThreads)
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            const int v = __ldg(ijk + 3 * q + d);
            lo[d] = min(lo[d], v), hi[d] = max(hi[d], v);
        }
    __shared__ int red[6];
    if (threadIdx.x < 6) red[threadIdx.x] = threadIdx.x < 3 ? INT_MAX : INT_MIN;
    __syncthreads();
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        lo[d] = __reduce_min_sync(0xffffffffu, lo[d]);
        hi[d] = __reduce_max_sync(0xffffffffu, hi[d]);
    }
    if ((threadIdx.x & 31) == 0)
        for (int d = 0; d < 3; ++d) atomicMin(red + d, lo[d]), atomicMax(red + 3 + d, hi[d]);
    __syncthreads();
    if (threadIdx.x < 3) {
        atomicMin(bounds + threadIdx.x, red[threadIdx.x]);
        if (red[threadIdx.x] <= -kCoordLimit) atomicExch(bounds + 6, 1);
    } else if (threadIdx.x < 6) {
        atomicMax(bounds + threadIdx.x, red[threadIdx.x]);
        if (red[threadIdx.x] >= kCoordLimit) atomicExch(bounds + 6, 1);
    }
}

// Step 2: flags (one int per leaf of the box, 0 before) of the leaves the dilated voxels touch.
__global__ void __launch_bounds__(kTopoThreads) flag_kernel(const int32_t* __restrict__ ijk, int64_t n, int padding, Box box,
                                                            int* flags) {
    const int64_t q = (int64_t)blockIdx.x * kTopoThreads + threadIdx.x;
    const bool live = q < n;
    int c[3] = {0, 0, 0};
    uint32_t reach[3] = {0u, 0u, 0u};  // per axis bit 0: -1, bit 1: 0, bit 2: +1
    if (live)
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            const int v = __ldg(ijk + 3 * q + d);
            c[d] = (v >> 3) - box.lo[d];
            reach[d] = 2u | ((v & 7) < padding ? 1u : 0u) | ((v & 7) + padding >= 8 ? 4u : 0u);
        }
    const uint32_t row = ((reach[1] & 1u) ? reach[2] : 0u) | ((reach[1] & 2u) ? reach[2] << 3 : 0u) | ((reach[1] & 4u) ? reach[2] << 6 : 0u);
    const uint32_t m = ((reach[0] & 1u) ? row : 0u) | ((reach[0] & 2u) ? row << 9 : 0u) | ((reach[0] & 4u) ? row << 18 : 0u);
    // The warp's voxels by leaf: the lanes of one leaf share its reached neighbours out. (Bit k of m:
    // neighbour (k / 9, k / 3 % 3, k % 3) - 1; at most 2^28 leaves in the box.)
    const int leaf = live ? (int)(((int64_t)c[0] * box.dim[1] + c[1]) * box.dim[2] + c[2]) : -1;
    const unsigned mates = __match_any_sync(0xffffffffu, leaf);
    uint32_t all = __reduce_or_sync(mates, m);
    if (!live) return;
    unsigned below;
    asm("mov.u32 %0, %%lanemask_lt;" : "=r"(below));
    const int size = __popc(mates);
    int turn = __popc(mates & below);
    for (; all; all &= all - 1, turn = turn == 0 ? size - 1 : turn - 1) {
        if (turn != 0) continue;
        const int k = __ffs(all) - 1;
        int* f = flags + ((int64_t)(c[0] + k / 9 - 1) * box.dim[1] + (c[1] + k / 3 % 3 - 1)) * box.dim[2] + (c[2] + k % 3 - 1);
        // A flag already set is not written again: the list's voxels set few flags many times (a stale 0
        // from this SM's cache costs a write).
        if (*f == 0) *f = 1;
    }
}

// The part of the box that lower node (x, y, z) (coordinates in units of 16 leaves) covers.
struct NodePart {
    int lo[3], dim[3];  // box-relative
    __device__ __forceinline__ int64_t entry(const Box& box, int q) const {
        const int x = q / (dim[1] * dim[2]), r = q - x * dim[1] * dim[2], y = r / dim[2], z = r - y * dim[2];
        return ((int64_t)(lo[0] + x) * box.dim[1] + (lo[1] + y)) * box.dim[2] + (lo[2] + z);
    }
    __device__ __forceinline__ int size() const { return dim[0] * dim[1] * dim[2]; }
};

__device__ __forceinline__ NodePart node_part(const Box& box, const int3& node) {
    NodePart p;
    const int n[3] = {node.x, node.y, node.z};
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        const int a = max(16 * n[d] - box.lo[d], 0), b = min(16 * n[d] + 16 - box.lo[d], box.dim[d]);
        p.lo[d] = a, p.dim[d] = b - a;
    }
    return p;
}

// Step 3a: flagged leaves per lower node.
__global__ void __launch_bounds__(kTopoThreads) node_count_kernel(const int3* __restrict__ nodes, Box box,
                                                                  const int* __restrict__ flags, int* __restrict__ counts) {
    __shared__ int total;
    if (threadIdx.x == 0) total = 0;
    __syncthreads();
    const NodePart p = node_part(box, nodes[blockIdx.x]);
    int c = 0;
    for (int q = threadIdx.x; q < p.size(); q += kTopoThreads) c += flags[p.entry(box, q)];
    c = __reduce_add_sync(0xffffffffu, c);
    if ((threadIdx.x & 31) == 0 && c) atomicAdd(&total, c);
    __syncthreads();
    if (threadIdx.x == 0) counts[blockIdx.x] = total;
}

// Inclusive scan of one value per thread over a CTA of kTopoThreads threads; `sums` has a word per
// warp. Returns the thread's inclusive sum; `total` receives the CTA's.
__device__ __forceinline__ int block_scan(int v, int* sums, int& total) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int u = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v += u;
    }
    if (lane == 31) sums[w] = v;
    __syncthreads();
    int before = 0;
    total = 0;
#pragma unroll
    for (int k = 0; k < kTopoThreads / 32; ++k) {
        if (k < w) before += sums[k];
        total += sums[k];
    }
    __syncthreads();
    return before + v;
}

// Step 3b: first leaf number of each node (exclusive scan, one CTA), the total after the last.
__global__ void __launch_bounds__(kTopoThreads) node_scan_kernel(int* counts, int n) {
    __shared__ int sums[kTopoThreads / 32];
    int base = 0;
    for (int q0 = 0; q0 < n; q0 += kTopoThreads) {
        const int q = q0 + (int)threadIdx.x, v = q < n ? counts[q] : 0;
        int total;
        const int inc = block_scan(v, sums, total);
        if (q < n) counts[q] = base + inc - v;
        base += total;
    }
    if (threadIdx.x == 0) counts[n] = base;
}

// Step 4: numbers each node's leaves in x, y, z order: their origins (int4, and packed for the
// host) and the lookup table's entries (in place of the flags).
__global__ void __launch_bounds__(kTopoThreads) number_kernel(const int3* __restrict__ nodes, Box box,
                                                              const int* __restrict__ first, int* __restrict__ lookup,
                                                              int4* __restrict__ org, int* __restrict__ org3) {
    __shared__ int sums[kTopoThreads / 32];
    const NodePart p = node_part(box, nodes[blockIdx.x]);
    int base = first[blockIdx.x];
    for (int q0 = 0; q0 < p.size(); q0 += kTopoThreads) {
        const int q = q0 + (int)threadIdx.x;
        const int64_t e = q < p.size() ? p.entry(box, q) : 0;
        const int v = q < p.size() ? lookup[e] : 0;
        int total;
        const int l = base + block_scan(v, sums, total) - v;
        if (q < p.size()) {
            lookup[e] = v ? l : -1;
            if (v) {
                const int z = (int)(e % box.dim[2]), y = (int)((e / box.dim[2]) % box.dim[1]),
                          x = (int)(e / ((int64_t)box.dim[1] * box.dim[2]));
                const int o[3] = {8 * (x + box.lo[0]), 8 * (y + box.lo[1]), 8 * (z + box.lo[2])};
                org[l] = make_int4(o[0], o[1], o[2], 0);
                org3[3 * l] = o[0], org3[3 * l + 1] = o[1], org3[3 * l + 2] = o[2];
            }
        }
        base += total;
    }
}

__global__ void nbr27_kernel(const int4* __restrict__ org, int64_t n, TopoView t, int* __restrict__ nbr) {
    const int64_t l = (int64_t)blockIdx.x * kTopoThreads + threadIdx.x;
    if (l >= n) return;
    const int4 o = org[l];
    for (int q = 0; q < 27; ++q) {
        const int a = (o.x >> 3) + q / 9 - 1 - t.lo_x, b = (o.y >> 3) + (q / 3) % 3 - 1 - t.lo_y,
                  c = (o.z >> 3) + q % 3 - 1 - t.lo_z;
        int v = -1;
        if ((unsigned)a < (unsigned)t.dim_x && (unsigned)b < (unsigned)t.dim_y && (unsigned)c < (unsigned)t.dim_z)
            v = t.lookup[((int64_t)a * t.dim_y + b) * t.dim_z + c];
        nbr[l * 27 + q] = v;
    }
}

}  // namespace

// Largest dense leaf table accepted, as in the host build.
constexpr int64_t kMaxLookupEntriesDevice = int64_t(1) << 28;

void Topology::build_from_voxels(const int32_t* ijk, int64_t n, bool ijk_on_device, int padding, cudaStream_t s) {
    if (n <= 0) fail(HNS_ERR_INVALID_ARG, "no active voxels");
    if (padding < 0 || padding > kMaxPadding) fail(HNS_ERR_INVALID_ARG, "padding must be in [0, 8] voxels");
    if (n > (int64_t(1) << 31) - 1) fail(HNS_ERR_UNSUPPORTED, "more than 2^31-1 active voxels");
    DeviceBuffer d_ijk;
    const int32_t* dv = ijk;
    if (!ijk_on_device) {
        d_ijk.alloc(sizeof(int32_t) * 3 * (size_t)n);
        HNS_CUDA(cudaMemcpyAsync(d_ijk.ptr, ijk, sizeof(int32_t) * 3 * (size_t)n, cudaMemcpyHostToDevice, s));
        dv = d_ijk.as<int32_t>();
    }
    DeviceBuffer small(sizeof(int) * 7);
    const int init[7] = {INT_MAX, INT_MAX, INT_MAX, INT_MIN, INT_MIN, INT_MIN, 0};
    HNS_CUDA(cudaMemcpyAsync(small.ptr, init, sizeof(init), cudaMemcpyHostToDevice, s));
    bounds_kernel<<<(unsigned)std::min<int64_t>(grid_for(n), 2048), kTopoThreads, 0, s>>>(dv, n, small.as<int>());
    HNS_LAUNCHED();
    int b[7];
    HNS_CUDA(cudaMemcpyAsync(b, small.ptr, sizeof(b), cudaMemcpyDeviceToHost, s));
    HNS_CUDA(cudaStreamSynchronize(s));
    if (b[6]) fail(HNS_ERR_INVALID_ARG, "a voxel coordinate is outside +-(2^23 - 64)");
    Box box;
    int64_t entries = 1;
    for (int d = 0; d < 3; ++d) {
        // The outermost voxels' dilation boxes reach the outermost leaves: the leaves' bounding box.
        box.lo[d] = (b[d] - padding) >> 3;
        box.dim[d] = ((b[3 + d] + padding) >> 3) - box.lo[d] + 1;
        entries *= box.dim[d];
    }
    if (entries > kMaxLookupEntriesDevice)
        fail(HNS_ERR_UNSUPPORTED, "leaf bounding box exceeds the dense leaf table limit of 2^28 entries");
    // The box's lower nodes (16^3 leaves) in NanoVDB order: by root tile (32^3 nodes), then by node,
    // each in x, y, z order.
    std::vector<int3> nodes;
    int lo[3], hi[3];
    for (int d = 0; d < 3; ++d) lo[d] = box.lo[d] >> 4, hi[d] = (box.lo[d] + box.dim[d] - 1) >> 4;
    auto tile = [](int node) { return node >> 5; };
    auto span = [&](int d, int t, auto&& body) {
        for (int v = std::max(lo[d], 32 * t); v <= std::min(hi[d], 32 * t + 31); ++v) body(v);
    };
    for (int rx = tile(lo[0]); rx <= tile(hi[0]); ++rx)
        for (int ry = tile(lo[1]); ry <= tile(hi[1]); ++ry)
            for (int rz = tile(lo[2]); rz <= tile(hi[2]); ++rz)
                span(0, rx, [&](int x) { span(1, ry, [&](int y) { span(2, rz, [&](int z) { nodes.push_back(make_int3(x, y, z)); }); }); });
    const int num_nodes = (int)nodes.size();
    DeviceBuffer d_nodes(sizeof(int3) * nodes.size()), first(sizeof(int) * (nodes.size() + 1));
    HNS_CUDA(cudaMemcpyAsync(d_nodes.ptr, nodes.data(), d_nodes.bytes, cudaMemcpyHostToDevice, s));
    d_lookup.alloc(sizeof(int32_t) * (size_t)entries);
    HNS_CUDA(cudaMemsetAsync(d_lookup.ptr, 0, d_lookup.bytes, s));
    flag_kernel<<<grid_for(n), kTopoThreads, 0, s>>>(dv, n, padding, box, d_lookup.as<int>());
    HNS_LAUNCHED();
    node_count_kernel<<<(unsigned)num_nodes, kTopoThreads, 0, s>>>(d_nodes.as<int3>(), box, d_lookup.as<int>(), first.as<int>());
    HNS_LAUNCHED();
    node_scan_kernel<<<1, kTopoThreads, 0, s>>>(first.as<int>(), num_nodes);
    HNS_LAUNCHED();
    int L = 0;
    HNS_CUDA(cudaMemcpyAsync(&L, first.as<int>() + num_nodes, sizeof(int), cudaMemcpyDeviceToHost, s));
    HNS_CUDA(cudaStreamSynchronize(s));

    num_leaves = L;
    int4* d_origin;
    int* d_nbr27;
    alloc_leaves(L, d_origin, d_nbr27);
    // The origins for the host pass through the neighbour table's memory, which is written after.
    int* org3 = d_nbr27;
    number_kernel<<<(unsigned)num_nodes, kTopoThreads, 0, s>>>(d_nodes.as<int3>(), box, first.as<int>(), d_lookup.as<int>(),
                                                               d_origin, org3);
    HNS_LAUNCHED();
    origins.resize((size_t)L * 3);
    HNS_CUDA(cudaMemcpyAsync(origins.data(), org3, sizeof(int32_t) * origins.size(), cudaMemcpyDeviceToHost, s));
    nanovdb_order = true;
    view.lookup = d_lookup.as<int>();
    view.lo_x = box.lo[0], view.lo_y = box.lo[1], view.lo_z = box.lo[2];
    view.dim_x = box.dim[0], view.dim_y = box.dim[1], view.dim_z = box.dim[2];
    nbr27_kernel<<<grid_for(L), kTopoThreads, 0, s>>>(d_origin, L, view, d_nbr27);
    HNS_LAUNCHED();
    HNS_CUDA(cudaStreamSynchronize(s));
}

}  // namespace hns
