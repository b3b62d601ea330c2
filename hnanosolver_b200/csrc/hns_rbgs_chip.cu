// The red-black SOR solve held on the chip: every half-sweep of a solve in one cooperative launch
// whose CTAs, all resident, keep their leaves' values in shared memory from the first half-sweep to
// the last and exchange only the faces between CTAs.
//
// Why. A half-sweep of a grid of a few million voxels is bound by its launch, by L2 latency and by
// the drain between the colours, not by bytes. The 148 SMs hold 33 MB of shared memory between
// them, where the values and the right-hand side of up to 3.5 million voxels fit with a halo.
//
// Measured, us per half-sweep, one launch per colour -> here; alone / three contexts taking turns on
// streams of their own (per solve of one of them):
//   leaves                 59                    592                   1,776                  2,368
//   FP32       2.1 -> 1.1 / 2.1 -> 0.4  2.0 -> 1.2 / 2.1 -> 0.7  2.1 -> 2.0 / 1.8 -> 1.3  2.7 -> 2.5 / 1.8 -> 1.6
//   walls      2.1 -> 1.2 / 2.1 -> 0.4  2.1 -> 1.4 / 2.1 -> 0.8  2.3 -> 2.2 / 1.8 -> 1.5  3.0 -> 2.8 / 1.8 -> 1.8
//   transpose                           4.7 -> 1.3 / 2.9 -> 0.8  7.2 -> 2.1 / 3.8 -> 1.4  8.3 -> 2.7 / 4.5 -> 1.8
// and the transpose of 4,096 leaves 12.1 -> 3.4 / 7.3 -> 3.3, of 6,512 16.5 -> 4.8 / 11.4 -> 4.8. What is left
// is the shared-memory pipe and instruction issue, and for small grids the exchange's L2 round trip
// (1.1 us with nothing else to do).
//
// Partition. CTA k owns the P leaves from k P (the caller's leaf order, which is spatially compact
// for NanoVDB-ordered grids; any order is correct). Leaves are stored colour-split, as in
// hns_rbgs_split.cu: a warp relaxes the 32 rows of one parity of a + b of one leaf, its loads from
// shared memory free of bank conflicts. Where a leaf's neighbour is in another CTA, the face of
// the neighbour that it reads (32 values of one colour) passes through `faces` in global memory:
// its owner stores it as it computes it, and at the start of the next half-sweep the reader's CTA
// brings all such faces into shared memory together, so that their latency is paid once.
//
// Order. Every value in `faces` is stored together with a tag, as one 8-byte word: the number of
// the half-sweep that made it, counted on from launch to launch (ChipTags). A reader polls the words
// themselves until they carry the tag it waits for, so a half-sweep costs one store and one load
// through L2 between CTAs, with no fence, flag or grid barrier (with flags behind a fence a
// half-sweep of a 64^3 box took 3.9 us). A word is safe to overwrite: the
// thread that writes a face value of half-sweep h has read, for the same update, the neighbour's
// value of half-sweep h - 1 across that face, and that value was stored after the neighbour had
// read the word of half-sweep h - 2. Waits are bounded (kChipMaxPolls polls): one that gives up
// raises the device error flag and the abort word, and every CTA that waits returns, its leaves not
// stored; one that has no neighbour in another CTA runs to the end and stores its own.
//
// The arithmetic of each update is that of the launch-per-colour kernels in the same order, so
// the values are the same to the bit.
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <type_traits>

#include "hns_internal.cuh"
#include "hns_relax16.cuh"

namespace hns {
namespace {

constexpr uint32_t kChipMaxPolls = 1u << 20;
constexpr size_t kChipSmSmem = 233472;   // an SM's shared memory, 228 KB
constexpr size_t kChipMaxSmem = 232448;  // 227 KB, the most one CTA can have
constexpr size_t kChipReserve = 1536;    // of each CTA: 1 KB of the system's, its static shared memory

// The largest grids, in leaves per SM, whose solves are held here (chip_takes). A solve holds every SM
// from its first half-sweep to its last, so beyond some size launches per colour, between which other
// streams' kernels run, finish more solves. Launches per colour -> here, us, alone / three contexts in turn:
//   FP32, 100 iterations    2,368 leaves 558 -> 505 / 372 -> 327    2,369 (256 threads) 566 -> 498 / 361 -> 504
//                           4,096 673 -> 626 / 398 -> 624           6,512 848 -> 896 / 622 -> 895
//   checked every 10, 100   592 leaves 406 -> 384 / 207 -> 198      750 465 -> 474 / 225 -> 212
//     (loaded and stored    900 479 -> 506 / 234 -> 241             1,776 551 -> 591 / 292 -> 361
//     at every check)
//   FP16, a step of 90      1,184 leaves 504 -> 446 / 375 -> 257    1,776 499 -> 504 / 377 -> 317
//                           1,777 513 -> 587 / 369 -> 317           2,368 592 -> 630 / 380 -> 392
// The transpose, whose form launched per colour is far slower, takes every size that fits.
constexpr int kChipLeavesPerSm = 16, kChipLeavesPerSmChecked = 5, kChipLeavesPerSmHalf = 12;

enum ChipMode { kDirichlet = 0, kWalls = 1, kTranspose = 2 };

// Four values of a row, one colour.
template <typename T>
struct Row;
template <>
struct Row<float> {
    using V = float4;
    static __device__ __forceinline__ V zero() { return make_float4(0.f, 0.f, 0.f, 0.f); }
};
template <>
struct Row<__half> {
    using V = uint2;
    static __device__ __forceinline__ V zero() { return make_uint2(0u, 0u); }
};

__device__ __forceinline__ float at(const float4& v, int j) { return j == 0 ? v.x : j == 1 ? v.y : j == 2 ? v.z : v.w; }
__device__ __forceinline__ uint32_t at(const uint2& v, int j) {
    const uint32_t w = (j & 2) ? v.y : v.x;
    return (j & 1) ? (w >> 16) : (w & 0xFFFFu);
}

// A tagged word: a value (FP32; one or two FP16) and the number of the half-sweep that made it.
__device__ __forceinline__ void put2(uint64_t* p, uint32_t v0, uint32_t v1, uint32_t tag) {
    asm volatile("st.relaxed.gpu.global.v2.b64 [%0], {%1, %2};" ::"l"(p), "l"((uint64_t)tag << 32 | v0),
                 "l"((uint64_t)tag << 32 | v1)
                 : "memory");
}
__device__ __forceinline__ void get2(const uint64_t* p, uint64_t& a, uint64_t& b) {
    asm volatile("ld.relaxed.gpu.global.v2.b64 {%0, %1}, [%2];" : "=l"(a), "=l"(b) : "l"(p) : "memory");
}
constexpr int kFaceWords = 32;  // of one colour on a leaf face (FP16 x and y faces use 16 of them)

// Offset in a leaf of the two (FP32, and z faces) or four (FP16 x and y faces) values of colour k
// that piece i of face f holds. An x or y face holds its rows by parity q of a + b, four rows r of
// four values each; a z face the one value of each of the 32 rows of one parity.
template <int kPerPiece>
__device__ __forceinline__ int face_offset(int f, int k, int i) {
    if (f >= 4) return 256 * k + 128 * (f == 4 ? k ^ 1 : k) + 8 * i + (f == 4 ? 3 : 0);
    const int q = kPerPiece == 2 ? i >> 3 : i >> 2, r = kPerPiece == 2 ? (i >> 1) & 3 : i & 3;
    const int j = kPerPiece == 2 ? 2 * (i & 1) : 0;
    if (f < 2) return 256 * k + 128 * q + (f == 0 ? 112 : 0) + 4 * r + j;
    return 256 * k + 128 * q + 16 * (2 * r + (f == 2 ? q ^ 1 : q)) + (f == 2 ? 12 : 0) + j;
}

// Arguments of one launch.
template <typename T>
struct ChipArgs {
    const int* nb8;   // face neighbours of each leaf, num_leaves where there is none
    const T* rhs;     // the right-hand side (kTranspose: unused)
    T* e;             // the values, read unless zero_init, written at the end
    float* bar;       // kTranspose: the divergence's adjoint, in place
    uint64_t* faces;  // [colour][leaf][face][kFaceWords] tagged words
    unsigned* abort_word;
    uint32_t tag0;    // the launch's tags are tag0 .. tag0 + half_sweeps
    int num_leaves, per_cta, half_sweeps;
    bool zero_init;
    bool rhs_slots, e_slots;  // the arrays are in slot order (else colour-split)
    float omega, dx2;
    const double* check;  // return at once when it has passed
    const double* check_mid;  // tested before half-sweep mid_half; end there when it has passed
    int mid_half;
    double tol2;
    unsigned long long* counters;
    uint32_t max_polls;  // after which a wait gives up
    uint32_t refuse;     // the test hook of the timeout path: ~0, with which no tag is accepted; else 0
};

// Row (a, b) of `leaf`: its values of colour 0 and 1. Slot order holds z = 0 .. 7 in a row; entry j
// of colour c is z = 2 j + ((a + b + c) & 1).
__device__ __forceinline__ void load_row(const float* p, bool slots, int64_t leaf, int a, int b, int pos, float4& c0, float4& c1) {
    if (slots) {
        const float4* q = reinterpret_cast<const float4*>(p + (leaf << 9) + 64 * a + 8 * b);
        const float4 x = q[0], y = q[1];
        const float4 even = make_float4(x.x, x.z, y.x, y.z), odd = make_float4(x.y, x.w, y.y, y.w);
        c0 = ((a + b) & 1) ? odd : even;
        c1 = ((a + b) & 1) ? even : odd;
    } else {
        const float4* q = reinterpret_cast<const float4*>(p + (leaf << 9) + pos);
        c0 = q[0], c1 = q[64];
    }
}
__device__ __forceinline__ void load_row(const __half* p, bool, int64_t leaf, int, int, int pos, uint2& c0, uint2& c1) {
    const uint2* q = reinterpret_cast<const uint2*>(p + (leaf << 9) + pos);
    c0 = q[0], c1 = q[64];
}
__device__ __forceinline__ void store_row(float* p, bool slots, int64_t leaf, int a, int b, int pos, float4 c0, float4 c1) {
    if (slots) {
        const float4 even = ((a + b) & 1) ? c1 : c0, odd = ((a + b) & 1) ? c0 : c1;
        float4* q = reinterpret_cast<float4*>(p + (leaf << 9) + 64 * a + 8 * b);
        q[0] = make_float4(even.x, odd.x, even.y, odd.y);
        q[1] = make_float4(even.z, odd.z, even.w, odd.w);
    } else {
        float4* q = reinterpret_cast<float4*>(p + (leaf << 9) + pos);
        q[0] = c0, q[64] = c1;
    }
}
__device__ __forceinline__ void store_row(__half* p, bool, int64_t leaf, int, int, int pos, uint2 c0, uint2 c1) {
    uint2* q = reinterpret_cast<uint2*>(p + (leaf << 9) + pos);
    q[0] = c0, q[64] = c1;
}

__device__ __forceinline__ float4 scaled(float4 b, float dx2) { return make_float4(b.x * dx2, b.y * dx2, b.z * dx2, b.w * dx2); }
__device__ __forceinline__ uint2 scaled(uint2 b, float) { return b; }

// Face neighbours of the row: values of the other colour at entry j, and across the z face.
// P: z parity of the colour in this row (z = 2 j + P).
template <int P, typename V, typename Z>
__device__ __forceinline__ void z_pair(const V& K, Z ZC, int j, Z& zp, Z& zm) {
    zm = P ? at(K, j) : (j > 0 ? at(K, j - 1) : ZC);
    zp = P ? (j < 3 ? at(K, j + 1) : ZC) : at(K, j);
}

// One row's update; B is the right-hand side times dx^2 (FP32), n4 the count of in-domain
// neighbours of entry j (walls only), keep / nbr the transpose's factors.
template <int P, ChipMode kMode>
__device__ __forceinline__ float4 update(const float4& XP, const float4& XM, const float4& YP, const float4& YM,
                                         const float4& K, float ZC, const float4& B, const float4& C, float omega,
                                         float keep, float nbr, int n_xy, bool z_missing) {
    float v[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        float zp, zm;
        z_pair<P>(K, ZC, j, zp, zm);
        const float c = at(C, j);
        if constexpr (kMode == kTranspose) {
            const float sx = at(XP, j) + at(XM, j), sy = at(YP, j) + at(YM, j), sz = zp + zm;
            v[j] = keep * c + nbr * (sx + sy + sz);
        } else {
            const float sum = at(XP, j) + at(XM, j) + at(YP, j) + at(YM, j) + zp + zm;
            float pgs;
            if constexpr (kMode == kWalls) {
                const int n = n_xy - ((z_missing && j == (P ? 3 : 0)) ? 1 : 0);
                pgs = (sum - at(B, j)) / (float)n;
            } else {
                pgs = (sum - at(B, j)) * dev::kInv6;
            }
            v[j] = c + omega * (pgs - c);
        }
    }
    return make_float4(v[0], v[1], v[2], v[3]);
}
template <int P, ChipMode kMode>
__device__ __forceinline__ uint2 update(const uint2& XP, const uint2& XM, const uint2& YP, const uint2& YM, const uint2& K,
                                        uint32_t ZC, const uint2& B, const uint2& C, float omega, float, float, int, bool) {
    uint32_t r[2];
#pragma unroll
    for (int q = 0; q < 2; ++q) {
        float v[2];
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const int j = 2 * q + i;
            uint32_t zp, zm;
            z_pair<P>(K, ZC, j, zp, zm);
            v[i] = relax16::relax1(at(XP, j), at(XM, j), at(YP, j), at(YM, j), zp, zm, at(B, j), at(C, j), omega);
        }
        const __half2 h = __floats2half2_rn(v[0], v[1]);
        r[q] = *reinterpret_cast<const uint32_t*>(&h);
    }
    return make_uint2(r[0], r[1]);
}

template <typename T, ChipMode kMode, int kChipThreads>
__global__ void __launch_bounds__(kChipThreads, 1024 / kChipThreads) rbgs_chip_kernel(ChipArgs<T> A) {
    using V = typename Row<T>::V;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ int num_foreign;
    if (A.check != nullptr && A.check[0] <= A.tol2 * A.check[1]) return;
    const int P = A.per_cta, leaf0 = (int)blockIdx.x * P, count = min(P, A.num_leaves - leaf0);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    // es: the values, then the zero leaf (local leaf P: what a missing neighbour reads), then the
    // foreign faces of local leaf l at halo(l, f); bs: the right-hand side.
    T* es = reinterpret_cast<T*>(smem_raw);
    const int halo0 = (P + 1) * 512;
    T* bs = es + halo0 + (size_t)P * 6 * 32;
    int* nbs = reinterpret_cast<int*>(bs + (size_t)P * 512);  // face table, 8 per leaf
    int* foreign = nbs + 8 * P;                               // 8 l + f of each foreign face
    if (tid == 0) num_foreign = 0;
    __syncthreads();
    // Face table: a local leaf 0 .. P - 1, P for a missing neighbour, -1 - g for leaf g of another CTA.
    for (int q = tid; q < count * 6; q += kChipThreads) {
        const int l = q / 6, f = q - 6 * l;
        const int g = A.nb8[8 * (leaf0 + l) + f];
        int v = P;
        if (g < A.num_leaves) {
            v = g - leaf0;
            if (v < 0 || v >= count) {
                v = -1 - g;
                foreign[atomicAdd(&num_foreign, 1)] = 8 * l + f;
            }
        }
        nbs[8 * l + f] = v;
    }
    for (int q = tid; q < 128; q += kChipThreads) reinterpret_cast<V*>(es + (size_t)P * 512)[q] = Row<T>::zero();
    for (int q = tid; q < count * 6 * 8; q += kChipThreads) reinterpret_cast<V*>(es + halo0)[q] = Row<T>::zero();
    for (int q = tid; q < count * 64; q += kChipThreads) {
        const int l = q >> 6, r = q & 63, a = (r >> 2) & 7, w = r >> 5, b = 2 * (r & 3) + ((a + w) & 1);
        V c0 = Row<T>::zero(), c1 = c0;
        if (!A.zero_init) load_row(A.e, A.e_slots, leaf0 + l, a, b, 4 * r, c0, c1);
        store_row(es, false, l, a, b, 4 * r, c0, c1);
        if constexpr (kMode == kTranspose)
            load_row(A.bar, A.rhs_slots, leaf0 + l, a, b, 4 * r, c0, c1);
        else
            load_row(A.rhs, A.rhs_slots, leaf0 + l, a, b, 4 * r, c0, c1);
        if constexpr (kMode != kTranspose) c0 = scaled(c0, A.dx2), c1 = scaled(c1, A.dx2);
        store_row(bs, false, l, a, b, 4 * r, c0, c1);
    }
    __syncthreads();
    const int nf = num_foreign;
    const int64_t colour_stride = (int64_t)A.num_leaves * 6 * kFaceWords;
    constexpr bool kHalf = sizeof(T) == 2;
    constexpr int kPieces = kFaceWords / 2;  // 16 bytes each
    // Stores the values of colour k on the faces that touch other CTAs.
    auto put_faces = [&](int k, uint32_t tag) {
        for (int q = tid; q < nf * kPieces; q += kChipThreads) {
            const int i = q & (kPieces - 1), lf = foreign[q / kPieces], l = lf >> 3, f = lf & 7;
            if (kHalf && f < 4 && i >= 8) continue;
            uint64_t* dst = A.faces + k * colour_stride + ((int64_t)(leaf0 + l) * 6 + f) * kFaceWords + 2 * i;
            const T* src = es + 512 * l + face_offset<kHalf ? 4 : 2>(f, k, i);
            if constexpr (kHalf) {
                const auto* u = reinterpret_cast<const unsigned short*>(src);
                if (f < 4) {
                    const uint2 v = *reinterpret_cast<const uint2*>(src);
                    put2(dst, v.x, v.y, tag);
                } else {
                    put2(dst, u[0], u[4], tag);
                }
            } else {
                const auto* u = reinterpret_cast<const uint32_t*>(src);
                put2(dst, u[0], f < 4 ? u[1] : u[4], tag);
            }
        }
    };
    // Brings the other CTAs' faces of colour k, tagged `tag`, into the halo; true if a wait gave up.
    auto get_faces = [&](int k, uint32_t tag) {
        const uint64_t* faces = A.faces + k * colour_stride;
        const uint32_t want = tag | A.refuse;
        bool failed = false;
        for (int q = tid; q < nf * kPieces; q += kChipThreads) {
            const int i = q & (kPieces - 1), lf = foreign[q / kPieces], l = lf >> 3, f = lf & 7;
            if (kHalf && f < 4 && i >= 8) continue;
            const uint64_t* src = faces + ((int64_t)(-1 - nbs[lf]) * 6 + (f ^ 1)) * kFaceWords + 2 * i;
            uint64_t x, y;
            uint32_t polls = 0;
            for (;;) {
                get2(src, x, y);
                if ((uint32_t)(x >> 32) == want && (uint32_t)(y >> 32) == want) break;
                if (++polls >= A.max_polls) {
                    atomicExch(A.abort_word, A.tag0);
                    if (A.counters != nullptr) atomicExch(A.counters + 1, 1ull);
                    failed = true;
                    break;
                }
                if ((polls & 63u) == 0 && *reinterpret_cast<volatile unsigned*>(A.abort_word) == A.tag0) {
                    failed = true;
                    break;
                }
            }
            T* dst = es + halo0 + (l * 6 + f) * 32;
            if constexpr (!kHalf) {
                *reinterpret_cast<uint2*>(dst + 2 * i) = make_uint2((uint32_t)x, (uint32_t)y);
            } else if (f < 4) {
                *reinterpret_cast<uint2*>(dst + 4 * i) = make_uint2((uint32_t)x, (uint32_t)y);
            } else {
                *reinterpret_cast<uint32_t*>(dst + 2 * i) = ((uint32_t)x & 0xFFFFu) | ((uint32_t)y << 16);
            }
        }
        return failed;
    };
    if (!A.zero_init) put_faces(1, A.tag0);  // half-sweep 0 reads the colour it does not update
    // This thread's rows: row (a, b) of parity w of every 16th leaf from warp / 2 (a task is the 32
    // rows of one parity of one leaf, so w, a and b are the thread's for good).
    const int w = warp & 1, a = lane >> 2, b = 2 * (lane & 3) + ((a + w) & 1), b4 = 4 * (b >> 1);
    float scale[2] = {1.f, 1.f};  // kTranspose: the uniform factor of each colour (adj_rbgs)
    const float step = A.omega * dev::kInv6;
    int h = 0;
    for (; h < A.half_sweeps; ++h) {
        if (h == A.mid_half && A.check_mid != nullptr && A.check_mid[0] <= A.tol2 * A.check_mid[1]) break;
        // The colour this half-sweep updates; the transpose of black, then red, updates the other.
        const int colour = h & 1;
        float keep = 0.f, nbr = 0.f, dmul = 0.f;
        if constexpr (kMode == kTranspose) {
            const int from = colour ^ 1;
            keep = scale[colour], nbr = step * scale[from], dmul = A.dx2 * step * scale[from];
            scale[colour] = 1.f;
            scale[from] *= 1.f - A.omega;
        }
        const uint32_t tag = A.tag0 + (uint32_t)h;  // of the other colour's faces; this half-sweep's are tag + 1
        if (h > 0 || !A.zero_init) {
            if (__syncthreads_or(get_faces(colour ^ 1, tag))) return;
        }
        // Offsets in a leaf: the row's own entries, and those of rows (a +- 1, b), (a, b +- 1) of the
        // other colour (`oc`: its block, `op`: the other parity's rows in it).
        const int own0 = 256 * colour + 128 * w + 4 * lane, oc = 256 * (colour ^ 1), op = oc + 128 * (w ^ 1);
        const int ixp = op + 16 * (a + 1) + b4, ixm = op + 16 * (a - 1) + b4;
        const int iyp = op + 16 * a + 4 * ((b + 1) >> 1), iym = op + 16 * a + 4 * ((b - 1) >> 1);
        // Across the faces: a neighbour of this CTA at these offsets of its leaf, or the halo.
        const int jx = op + (a == 7 ? 0 : 112) + b4, jy = op + 16 * a + (b == 7 ? 0 : 12);
        const int kx = halo0 + (a == 7 ? 0 : 32) + 16 * (w ^ 1) + b4;
        const int ky = halo0 + (b == 7 ? 64 : 96) + 16 * (w ^ 1) + 4 * (a >> 1);
        const int fx = a == 7 ? 0 : 1, fy = b == 7 ? 2 : 3;
        auto sweep = [&](auto parity) {
            constexpr int p = decltype(parity)::value;
            const int jz = oc + 128 * w + 4 * lane + (p ? 0 : 3), kz = halo0 + (p ? 128 : 160) + lane;
            for (int l = warp >> 1; l < count; l += kChipThreads / 64) {
                const int* nb = nbs + 8 * l;
                const int nx = nb[fx], ny = nb[fy], nz = nb[p ? 4 : 5];
                const int leaf = 512 * l, halo = 192 * l, own = leaf + own0;
                const int ax = nx < 0 ? halo + kx : 512 * nx + jx;
                const int ay = ny < 0 ? halo + ky : 512 * ny + jy;
                const int az = nz < 0 ? halo + kz : 512 * nz + jz;
                V B;
                if constexpr (kMode == kTranspose)
                    B = Row<T>::zero();
                else
                    B = *reinterpret_cast<const V*>(bs + own);
                const V C = *reinterpret_cast<const V*>(es + own), K = *reinterpret_cast<const V*>(es + (own ^ 256));
                const V XP = *reinterpret_cast<const V*>(es + (a == 7 ? ax : leaf + ixp));
                const V XM = *reinterpret_cast<const V*>(es + (a == 0 ? ax : leaf + ixm));
                const V YP = *reinterpret_cast<const V*>(es + (b == 7 ? ay : leaf + iyp));
                const V YM = *reinterpret_cast<const V*>(es + (b == 0 ? ay : leaf + iym));
                const T Zs = es[az];
                int n_xy = 6;
                if constexpr (kMode == kWalls)
                    n_xy -= ((a == 7 || a == 0) && nx == P ? 1 : 0) + ((b == 7 || b == 0) && ny == P ? 1 : 0);
                if constexpr (kHalf)
                    *reinterpret_cast<V*>(es + own) = update<p, kMode>(XP, XM, YP, YM, K, (uint32_t)__half_as_ushort(Zs), B, C,
                                                                       A.omega, keep, nbr, n_xy, nz == P);
                else
                    *reinterpret_cast<V*>(es + own) =
                        update<p, kMode>(XP, XM, YP, YM, K, Zs, B, C, A.omega, keep, nbr, n_xy, nz == P);
                if constexpr (kMode == kTranspose) {
                    // The divergence's adjoint at the row's voxels of the colour that is read.
                    float4* d = reinterpret_cast<float4*>(reinterpret_cast<float*>(bs) + (own ^ 256));
                    float4 x = *d;
                    x.x -= dmul * K.x, x.y -= dmul * K.y, x.z -= dmul * K.z, x.w -= dmul * K.w;
                    *d = x;
                }
            }
        };
        if ((w + colour) & 1)
            sweep(std::integral_constant<int, 1>{});
        else
            sweep(std::integral_constant<int, 0>{});
        __syncthreads();
        if (h + 1 < A.half_sweeps) put_faces(colour, tag + 1u);
    }
    if (A.counters != nullptr && blockIdx.x == 0 && tid == 0) atomicAdd(A.counters, (unsigned long long)h);
    for (int q = tid; q < count * 64; q += kChipThreads) {
        const int l = q >> 6, r = q & 63, a = (r >> 2) & 7, w = r >> 5, b = 2 * (r & 3) + ((a + w) & 1);
        V c0, c1;
        if constexpr (kMode != kTranspose) {
            load_row(es, false, l, a, b, 4 * r, c0, c1);
            store_row(A.e, A.e_slots, leaf0 + l, a, b, 4 * r, c0, c1);
        } else {
            load_row(bs, false, l, a, b, 4 * r, c0, c1);
            store_row(A.bar, A.rhs_slots, leaf0 + l, a, b, 4 * r, c0, c1);
        }
    }
}

// Shared memory of a CTA of per_cta leaves: values, the zero leaf, six halo faces a leaf, the
// right-hand side, the face table and the list of foreign faces.
template <typename T>
size_t chip_smem(int64_t per_cta) {
    return ((2 * (size_t)per_cta + 1) * 512 + (size_t)per_cta * 6 * 32) * sizeof(T) + (size_t)per_cta * 14 * sizeof(int);
}

// How a launch divides the grid: four CTAs an SM, so that one CTA's exchange overlaps the others'
// updates, of 128 threads up to four leaves a CTA (256 fill the SM's registers, so that other streams
// wait: HNS_Advance on 1,493 leaves, us alone / three contexts in turn: 788 / 626 with 256 threads, 835 /
// 513 with 128). The transpose also of 256 beyond, and one CTA of 1,024 threads an SM for the last 5 %
// of the sizes that fit.
struct ChipShape {
    int64_t per_cta;  // 0: the grid does not fit
    int threads;
};
template <typename T>
ChipShape chip_shape(const Context& c, bool transpose) {
    const int64_t L = c.topo.num_leaves, sms = c.sm_count();
    if (L <= 0) return {0, 0};
    const int64_t quarter = (L + 4 * sms - 1) / (4 * sms), whole = (L + sms - 1) / sms;
    if (4 * quarter <= kChipLeavesPerSm) return {quarter, 128};
    if (transpose && chip_smem<T>(quarter) <= kChipSmSmem / 4 - kChipReserve) return {quarter, 256};
    if (transpose && chip_smem<T>(whole) <= kChipMaxSmem - kChipReserve) return {whole, 1024};
    return {0, 0};
}

template <typename T, ChipMode kMode>
auto chip_kernel(int threads) {
    auto kern = rbgs_chip_kernel<T, kMode, 128>;
    if constexpr (kMode == kTranspose) {
        if (threads == 256) kern = rbgs_chip_kernel<T, kMode, 256>;
        if (threads == 1024) kern = rbgs_chip_kernel<T, kMode, 1024>;
    }
    // The same limit for every context of the process, so none lowers another's.
    HNS_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(kChipMaxSmem - kChipReserve)));
    return kern;
}

// Whether every CTA of a launch is resident at once, as a cooperative launch must be. Asked before each
// solve: a program may prefer L1 over shared memory (cudaDeviceSetCacheConfig), which leaves room for
// one CTA an SM. (A carveout preference of the kernel's own would overrule that, but was slower where
// several contexts solve: with 40 % of shared memory no two grids share the SMs, HNS_Advance on 1,493
// leaves 454 -> 670 us, and with all of it the adjoint step of a 128^3 box 703 -> 744.)
template <typename T, ChipMode kMode>
bool chip_resident(const Context& c) {
    const ChipShape shape = chip_shape<T>(c, kMode == kTranspose);
    if (shape.per_cta <= 0) return false;
    int per_sm = 0;
    HNS_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, chip_kernel<T, kMode>(shape.threads), shape.threads,
                                                           chip_smem<T>(shape.per_cta)));
    return (int64_t)per_sm * c.sm_count() >= (c.topo.num_leaves + shape.per_cta - 1) / shape.per_cta;
}

template <typename T, ChipMode kMode>
void launch_chip(Context& c, ChipArgs<T> A) {
    const int64_t L = c.topo.num_leaves;
    const ChipShape shape = chip_shape<T>(c, kMode == kTranspose);
    A.num_leaves = (int)L;
    A.per_cta = (int)shape.per_cta;
    auto kern = chip_kernel<T, kMode>(shape.threads);
    const unsigned blocks = (unsigned)((L + A.per_cta - 1) / A.per_cta);
    // Face words and the abort word, cleared where the tags need it (ChipTags).
    const size_t words = (size_t)L * 2 * 6 * kFaceWords;
    auto* w = reinterpret_cast<uint64_t*>(c.scratch_f32("chip_faces", 2 * words + 2));
    const ChipTags::Launch tags = c.chip_tags.take((uint32_t)A.half_sweeps, c.stream_capturing());
    if (tags.clear) {
        const cudaError_t cleared = cudaMemsetAsync(w, 0, words * 8 + 8, c.stream);
        if (cleared != cudaSuccess) c.chip_tags = ChipTags();
        HNS_CUDA(cleared);
    }
    A.faces = w;
    A.abort_word = reinterpret_cast<unsigned*>(w + words);
    A.tag0 = tags.first;
    const bool stall = c.first_wait_polls >= 0;
    A.refuse = stall ? ~0u : 0u;
    A.max_polls = stall ? std::min((uint32_t)c.first_wait_polls, kChipMaxPolls) : kChipMaxPolls;
    A.counters = c.counters;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(blocks);
    cfg.blockDim = dim3((unsigned)shape.threads);
    cfg.dynamicSmemBytes = chip_smem<T>(A.per_cta);
    cfg.stream = c.stream;
    // Cooperative: every CTA resident at once, which the waits rely on.
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    HNS_CUDA(cudaLaunchKernelEx(&cfg, kern, A));
    HNS_LAUNCHED();
}

}  // namespace

bool chip_takes(const Context& c, ChipUse use, bool walls) {
    if (use == ChipUse::kTransposed) return chip_resident<float, kTranspose>(c);
    const int per_sm = use == ChipUse::kChecked ? kChipLeavesPerSmChecked
                       : use == ChipUse::kHalf  ? kChipLeavesPerSmHalf
                                                : kChipLeavesPerSm;
    if (c.topo.num_leaves > (int64_t)per_sm * c.sm_count()) return false;
    return use == ChipUse::kHalf ? chip_resident<__half, kDirichlet>(c)
           : walls               ? chip_resident<float, kWalls>(c)
                                 : chip_resident<float, kDirichlet>(c);
}

void launch_chip_solve_f32(Context& c, const int* nb8, const float* rhs, bool rhs_slots, float* e, bool e_slots,
                           int half_sweeps, bool e_zero, float omega, float dx2, bool walls, const double* check,
                           const double* check_mid, int mid_half, double tol2) {
    ChipArgs<float> A = {};
    A.nb8 = nb8, A.rhs = rhs, A.e = e, A.rhs_slots = rhs_slots, A.e_slots = e_slots;
    A.half_sweeps = half_sweeps, A.zero_init = e_zero, A.omega = omega, A.dx2 = dx2;
    A.check = check, A.check_mid = check_mid, A.mid_half = mid_half, A.tol2 = tol2;
    if (walls) launch_chip<float, kWalls>(c, A);
    else launch_chip<float, kDirichlet>(c, A);
}

void launch_chip_solve_f16(Context& c, const int* nb8, const void* rhs, void* e, int half_sweeps, bool e_zero, float omega,
                           const double* check, double tol2) {
    ChipArgs<__half> A = {};
    A.nb8 = nb8, A.rhs = static_cast<const __half*>(rhs), A.e = static_cast<__half*>(e);
    A.half_sweeps = half_sweeps, A.zero_init = e_zero, A.omega = omega, A.dx2 = 1.0f, A.check = check, A.tol2 = tol2;
    launch_chip<__half, kDirichlet>(c, A);
}

void launch_chip_transpose(Context& c, const int* nb8, const float* p_bar, float* div_bar, int iterations, float omega) {
    ChipArgs<float> A = {};
    A.nb8 = nb8, A.e = const_cast<float*>(p_bar), A.bar = div_bar, A.rhs_slots = true, A.e_slots = true;
    A.half_sweeps = 2 * iterations, A.omega = omega, A.dx2 = c.dx * c.dx;
    launch_chip<float, kTranspose>(c, A);
}

}  // namespace hns
