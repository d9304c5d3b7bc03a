// gpu_build.cu — BVH construction on the GPU (see gpu_build.hpp).
//
//  1. prep: per triangle its box, its shading normal, input validation, and
//     the scene box / centroid box (warp-reduced float atomics);
//  2. 63-bit Morton code of each centroid on a grid of 2^21 cubic cells per
//     axis over the centroid box's largest extent (dense scenes keep a
//     spatial order far below the triangle size);
//  3. stable LSD radix sort of (code, triangle) in seven 9-bit passes, tiles
//     of 4,096 put in digit order in shared memory;
//  4. Karras (2012): internal node i of the n-1 finds its key range and
//     split by binary searches on the common-prefix length of the sorted
//     keys (ties between equal codes broken by sorted position); or
//     locally-ordered clustering of the sorted triangles (Meister & Bittner
//     2018), rounds of mutual-nearest-neighbour merges within a window of
//     the cluster array;
//  5. every node is finished from the leaves upwards (Karras: a walk, the
//     second thread to reach a node finishes it; clustering: round by round):
//     box, triangle count and the SAH decision
//     cost(n) = min(N A, C_trav A + cost(l) + cost(r)), a subtree of at most
//     max_leaf triangles becoming one leaf when that is not dearer;
//     With the SAH-optimal collapse that also computes, per node, the costs C(n, i) of representing its subtree by at most i roots (wide
//     nodes or leaf slots of up to 4 triangles) and their decisions, as
//     collapse.cpp does on the host;
//  6. collapse to 8-wide nodes, one wide level per launch: the children by
//     the greedy rule of collapse.cpp (expand the largest-area internal child
//     until 8) or by those decisions, octant slots, margin inflation and
//     outward quantisation in FP32 with directed rounding (conservative by
//     construction; the host collapse uses FP64), children and leaf
//     triangles allocated with atomics.
#include "gpu_build.hpp"

#include <algorithm>
#include <cfloat>
#include <chrono>
#include <cmath>
#include <cstring>
#include <vector>

#include "../../../include/fnd_rt.h"
#include "../core/core.hpp"
#include "../rt/device_scene.hpp"
#include "collapse.hpp"
#include "wide_bvh.hpp"

namespace Foundation {
namespace RT {
namespace {

constexpr uint32_t kFull = 0xFFFFFFFFu;
constexpr uint32_t kLeafRef = 0x80000000u;  // reference to a sorted single-triangle leaf
constexpr uint32_t kLeafNode = 0x80000000u;  // count word: this subtree is one leaf
constexpr uint32_t kNone = 0xFFFFFFFFu;
constexpr uint32_t kDpLeaf = 0x80u;  // decision byte 0: this subtree is one leaf slot
constexpr int kMaxLevels = kMaxStack / 2;  // wide levels the traversal stack allows
constexpr uint32_t kPrepBadIndex = 1u, kPrepNonFinite = 2u;

struct Buffers {
    float4 *blo, *bhi;            // triangle boxes (original order)
    unsigned long long *keys;     // sorted codes
    uint32_t* vals;               // triangle ids
    unsigned long long* keys2;    // radix-sort ping-pong
    uint32_t* vals2;
    uint32_t* cnt;                // digit-major tile counts, then the digits' totals
    uint32_t *left, *right;       // internal node children (kLeafRef | sorted index for leaves)
    uint32_t *parent_i, *parent_l;
    float4 *nlo, *nhi;            // internal node boxes; nlo.w: triangle count | kLeafNode (bits), nhi.w: SAH cost
    uint32_t* flag;               // refit arrival counters
    float* bounds;                // scene lo[3], hi[3], centroid lo[3], hi[3]
    uint32_t* status;
    uint32_t* counters;           // [1] tris, [2] leaves, [4..] per-level queue counts (wide nodes of a level)
    uint2 *qa, *qb;               // collapse queues (binary ref, wide node)
    // SAH-optimal collapse (null: greedy), per internal node k:
    float* dpc;                   // [8 k + i - 1]: C(k, i), least cost of k's subtree as at most i roots
    uint2* dpch;                  // byte i - 1, i >= 2: 0 = C(k, i - 1), else roots given to the left child;
                                  // byte 0: roots given to the left child when k is a wide node, | kDpLeaf when
                                  // C(k, 1) is one leaf slot
    float c_tri;                  // cost of a triangle test relative to a wide-node visit
    uint32_t width;               // children per wide node (2..8)
};

__device__ __forceinline__ void atomic_min_f(float* a, float v) {
    if (v >= 0.0f)
        atomicMin(reinterpret_cast<int*>(a), __float_as_int(v));
    else
        atomicMax(reinterpret_cast<unsigned*>(a), __float_as_uint(v));
}
__device__ __forceinline__ void atomic_max_f(float* a, float v) {
    if (v >= 0.0f)
        atomicMax(reinterpret_cast<int*>(a), __float_as_int(v));
    else
        atomicMin(reinterpret_cast<unsigned*>(a), __float_as_uint(v));
}

__global__ void init_bounds_kernel(float* b) {
    const int i = threadIdx.x;
    if (i < 12) b[i] = (i % 6) < 3 ? __int_as_float(0x7F800000) : __int_as_float(0xFF800000);
}

// Grid-stride over the triangles: each thread folds its triangles' boxes and
// centroids into its own bounds, the block reduces them, and one thread per
// block updates the scene bounds (a few thousand atomics in all, not one set
// per warp).
__global__ void __launch_bounds__(256) prep_kernel(const float* __restrict__ verts, uint32_t nv,
                                                   const uint32_t* __restrict__ idx, uint32_t nt, Buffers B,
                                                   float4* __restrict__ shade) {
    __shared__ float s_red[8][12];
    float lo[3], hi[3], c[3], cmax[3];
    for (int a = 0; a < 3; ++a) {
        lo[a] = c[a] = __int_as_float(0x7F800000);
        hi[a] = cmax[a] = __int_as_float(0xFF800000);
    }
    for (uint32_t t = blockIdx.x * blockDim.x + threadIdx.x; t < nt; t += gridDim.x * blockDim.x) {
        uint32_t vi[3];
        bool ok = true;
        for (int k = 0; k < 3; ++k) {
            vi[k] = idx[3 * (size_t)t + k];
            if (vi[k] >= nv) ok = false;
        }
        if (!ok) {
            atomicOr(B.status, kPrepBadIndex);
            continue;
        }
        float v[9];
        bool finite = true;
        for (int k = 0; k < 3; ++k)
            for (int a = 0; a < 3; ++a) {
                v[3 * k + a] = verts[3 * (size_t)vi[k] + a];
                finite = finite && isfinite(v[3 * k + a]);
            }
        if (!finite) atomicOr(B.status, kPrepNonFinite);
        float tlo[3], thi[3];
        for (int a = 0; a < 3; ++a) {
            tlo[a] = fminf(fminf(v[a], v[3 + a]), v[6 + a]);
            thi[a] = fmaxf(fmaxf(v[a], v[3 + a]), v[6 + a]);
            const float cc = __fmul_rn(0.5f, __fadd_rn(tlo[a], thi[a]));
            lo[a] = fminf(lo[a], tlo[a]);
            hi[a] = fmaxf(hi[a], thi[a]);
            c[a] = fminf(c[a], cc);
            cmax[a] = fmaxf(cmax[a], cc);
        }
        B.blo[t] = make_float4(tlo[0], tlo[1], tlo[2], 0.0f);
        B.bhi[t] = make_float4(thi[0], thi[1], thi[2], 0.0f);
        // geometric normal (winding order), the host's expression tree
        const float e1x = __fsub_rn(v[3], v[0]), e1y = __fsub_rn(v[4], v[1]), e1z = __fsub_rn(v[5], v[2]);
        const float e2x = __fsub_rn(v[6], v[0]), e2y = __fsub_rn(v[7], v[1]), e2z = __fsub_rn(v[8], v[2]);
        float nx = __fsub_rn(__fmul_rn(e1y, e2z), __fmul_rn(e1z, e2y));
        float ny = __fsub_rn(__fmul_rn(e1z, e2x), __fmul_rn(e1x, e2z));
        float nz = __fsub_rn(__fmul_rn(e1x, e2y), __fmul_rn(e1y, e2x));
        const float l = __fsqrt_rn(__fadd_rn(__fadd_rn(__fmul_rn(nx, nx), __fmul_rn(ny, ny)), __fmul_rn(nz, nz)));
        if (l > 0.0f) {
            nx = __fdiv_rn(nx, l);
            ny = __fdiv_rn(ny, l);
            nz = __fdiv_rn(nz, l);
        } else {
            nx = ny = 0.0f;
            nz = 1.0f;
        }
        shade[t] = make_float4(nx, ny, nz, 0.0f);
    }
    for (int o = 16; o > 0; o >>= 1)
        for (int a = 0; a < 3; ++a) {
            lo[a] = fminf(lo[a], __shfl_xor_sync(kFull, lo[a], o));
            hi[a] = fmaxf(hi[a], __shfl_xor_sync(kFull, hi[a], o));
            c[a] = fminf(c[a], __shfl_xor_sync(kFull, c[a], o));
            cmax[a] = fmaxf(cmax[a], __shfl_xor_sync(kFull, cmax[a], o));
        }
    const uint32_t warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    if ((threadIdx.x & 31u) == 0)
        for (int a = 0; a < 3; ++a) {
            s_red[warp][a] = lo[a];
            s_red[warp][3 + a] = hi[a];
            s_red[warp][6 + a] = c[a];
            s_red[warp][9 + a] = cmax[a];
        }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (uint32_t w = 1; w < nw; ++w)
            for (int a = 0; a < 3; ++a) {
                lo[a] = fminf(lo[a], s_red[w][a]);
                hi[a] = fmaxf(hi[a], s_red[w][3 + a]);
                c[a] = fminf(c[a], s_red[w][6 + a]);
                cmax[a] = fmaxf(cmax[a], s_red[w][9 + a]);
            }
        if (lo[0] <= hi[0])
            for (int a = 0; a < 3; ++a) {
                atomic_min_f(B.bounds + a, lo[a]);
                atomic_max_f(B.bounds + 3 + a, hi[a]);
                atomic_min_f(B.bounds + 6 + a, c[a]);
                atomic_max_f(B.bounds + 9 + a, cmax[a]);
            }
    }
}

// bits 0..20 of v to positions 0, 3, 6, ... 60
__device__ __forceinline__ unsigned long long spread3(unsigned long long v) {
    v &= 0x1FFFFFull;
    v = (v | (v << 32)) & 0x1F00000000FFFFull;
    v = (v | (v << 16)) & 0x1F0000FF0000FFull;
    v = (v | (v << 8)) & 0x100F00F00F00F00Full;
    v = (v | (v << 4)) & 0x10C30C30C30C30C3ull;
    v = (v | (v << 2)) & 0x1249249249249249ull;
    return v;
}

// The grid's cells are cubes: every axis is scaled by the centroid box's
// largest extent, so a flat scene's thin axis takes few of the code's bits
// and the first splits of the order are along the long axes.
__global__ void __launch_bounds__(256) morton_kernel(uint32_t nt, Buffers B) {
    const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= nt) return;
    const float4 lo = B.blo[t], hi = B.bhi[t];
    const float c[3] = {__fmul_rn(0.5f, __fadd_rn(lo.x, hi.x)), __fmul_rn(0.5f, __fadd_rn(lo.y, hi.y)),
                        __fmul_rn(0.5f, __fadd_rn(lo.z, hi.z))};
    unsigned long long q[3];
    const float emax = fmaxf(fmaxf(B.bounds[9] - B.bounds[6], B.bounds[10] - B.bounds[7]), B.bounds[11] - B.bounds[8]);
    for (int a = 0; a < 3; ++a) {
        const float u = emax > 0.0f ? (c[a] - B.bounds[6 + a]) * (2097152.0f / emax) : 0.0f;
        q[a] = (unsigned long long)fminf(fmaxf(u, 0.0f), 2097151.0f);
    }
    B.keys[t] = spread3(q[0]) | (spread3(q[1]) << 1) | (spread3(q[2]) << 2);
    B.vals[t] = t;
}

// ---- stable LSD radix sort ---------------------------------------------------
// (code, triangle) pairs by 63-bit codes, seven passes of 9 bits. A block owns
// a tile of 4,096 pairs. Per pass: the tiles' digit counts (digit-major), an
// exclusive scan of each digit's row over the tiles, and the scatter, in which
// a warp ranks its 512 pairs in order by matching digits, the block puts the
// tile in digit order in shared memory, and whole runs of a digit go out
// together. Bound: per pass 12 bytes in and out per pair, and at a million
// pairs the latency of three launches. The earlier form (eight 8-bit passes,
// five launches each, every pair stored on its own by a warp that owned 2,048)
// took 828 us for 1.1M pairs; this one 231 us.
constexpr int kSortBlock = 256;
constexpr int kSortWarps = kSortBlock / 32;
constexpr int kSortItems = 16;                       // pairs per thread
constexpr uint32_t kSortTile = kSortBlock * kSortItems;
constexpr int kDigitBits = 9, kDigits = 1 << kDigitBits, kSortPasses = 7;
static_assert(kDigitBits * kSortPasses >= 63, "the passes cover the codes' bits");
constexpr uint32_t kScanRow = 1024;                  // tiles of one digit scanned at a time

template <typename T>
__device__ __forceinline__ T block_exclusive(T v, T& total, T* s_warp) {
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    T incl = v;
    for (int o = 1; o < 32; o <<= 1) {
        const T x = __shfl_up_sync(kFull, incl, o);
        if ((int)lane >= o) incl += x;
    }
    if (lane == 31) s_warp[warp] = incl;
    __syncthreads();
    const uint32_t nw = blockDim.x >> 5;
    if (warp == 0) {
        T w = lane < nw ? s_warp[lane] : T(0);
        for (int o = 1; o < 32; o <<= 1) {
            const T x = __shfl_up_sync(kFull, w, o);
            if ((int)lane >= o) w += x;
        }
        if (lane < nw) s_warp[lane] = w;
    }
    __syncthreads();
    total = s_warp[nw - 1];
    const T before = warp ? s_warp[warp - 1] : T(0);
    __syncthreads();
    return before + incl - v;
}

__device__ __forceinline__ uint32_t digit_of(unsigned long long k, uint32_t shift) {
    return (uint32_t)(k >> shift) & (uint32_t)(kDigits - 1);
}

__global__ void __launch_bounds__(kSortBlock) hist_kernel(const unsigned long long* __restrict__ keys, uint32_t n,
                                                          uint32_t shift, uint32_t tiles, uint32_t* __restrict__ cnt) {
    __shared__ uint32_t s_cnt[kDigits];
    for (int d = threadIdx.x; d < kDigits; d += kSortBlock) s_cnt[d] = 0;
    __syncthreads();
    const uint32_t base = blockIdx.x * kSortTile + threadIdx.x;
#pragma unroll
    for (int k = 0; k < kSortItems; ++k) {
        const uint32_t i = base + k * kSortBlock;
        if (i < n) atomicAdd(&s_cnt[digit_of(keys[i], shift)], 1u);
    }
    __syncthreads();
    for (int d = threadIdx.x; d < kDigits; d += kSortBlock) cnt[(size_t)d * tiles + blockIdx.x] = s_cnt[d];
}

// One block per digit: its row's exclusive scan in place, its total.
__global__ void __launch_bounds__(kScanRow) scan_rows_kernel(uint32_t* __restrict__ cnt, uint32_t tiles,
                                                             uint32_t* __restrict__ totals) {
    __shared__ uint32_t s_warp[32];
    uint32_t* row = cnt + (size_t)blockIdx.x * tiles;
    uint32_t carry = 0;
    for (uint32_t at = 0; at < tiles; at += kScanRow) {
        const uint32_t k = at + threadIdx.x;
        const uint32_t v = k < tiles ? row[k] : 0u;
        uint32_t total;
        const uint32_t before = block_exclusive(v, total, s_warp);
        if (k < tiles) row[k] = carry + before;
        carry += total;
    }
    if (threadIdx.x == 0) totals[blockIdx.x] = carry;
}

struct SortShared {
    unsigned long long key[kSortTile];
    uint32_t val[kSortTile];
    uint32_t cnt[kSortWarps][kDigits];  // digit counts of a warp, then its first position per digit
    uint32_t out[kDigits];              // global position of a digit's first pair, less its position in the tile
    uint32_t warp[32];
};

__global__ void __launch_bounds__(kSortBlock) scatter_kernel(const unsigned long long* __restrict__ keys,
                                                             const uint32_t* __restrict__ vals, uint32_t n,
                                                             uint32_t shift, uint32_t tiles,
                                                             const uint32_t* __restrict__ cnt,
                                                             const uint32_t* __restrict__ totals,
                                                             unsigned long long* __restrict__ ok_,
                                                             uint32_t* __restrict__ ov) {
    extern __shared__ __align__(16) unsigned char s_raw[];
    SortShared& S = *reinterpret_cast<SortShared*>(s_raw);
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    for (int d = threadIdx.x; d < kSortWarps * kDigits; d += kSortBlock) (&S.cnt[0][0])[d] = 0;
    __syncthreads();
    const uint32_t tile0 = blockIdx.x * kSortTile;
    const uint32_t base = tile0 + warp * (32 * kSortItems) + lane;
    unsigned long long k[kSortItems];
    uint32_t v[kSortItems], rank[kSortItems];
#pragma unroll
    for (int j = 0; j < kSortItems; ++j) {
        const uint32_t i = base + 32 * j;
        k[j] = i < n ? keys[i] : ~0ull;
        v[j] = i < n ? vals[i] : 0u;
    }
    // ranks within the warp's pairs of a digit, in input order
#pragma unroll
    for (int j = 0; j < kSortItems; ++j) {
        const bool ok = base + 32 * j < n;
        const uint32_t d = ok ? digit_of(k[j], shift) : (uint32_t)kDigits;
        const uint32_t peers = __match_any_sync(kFull, d);
        const uint32_t lead = (uint32_t)__ffs(peers) - 1u;
        uint32_t start = 0;
        if (ok && lane == lead) {
            start = S.cnt[warp][d];
            S.cnt[warp][d] = start + (uint32_t)__popc(peers);
        }
        rank[j] = __shfl_sync(kFull, start, lead) + (uint32_t)__popc(peers & ((1u << lane) - 1u));
        __syncwarp();
    }
    __syncthreads();
    // the tile's digit order: digit d of warp w starts at the digits before it
    // plus the pairs of d in the warps before it; thread t has two digits
    {
        const int d0 = 2 * threadIdx.x;
        uint32_t sum[2];
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            uint32_t run = 0;
#pragma unroll
            for (int w = 0; w < kSortWarps; ++w) {
                const uint32_t x = S.cnt[w][d0 + q];
                S.cnt[w][d0 + q] = run;
                run += x;
            }
            sum[q] = run;
        }
        uint32_t total;
        const uint32_t first = block_exclusive(sum[0] + sum[1], total, S.warp);
        // the digits' global starts: the totals of the digits before, this
        // tile's place in the digit's row
        const uint32_t t0 = totals[d0], t1 = totals[d0 + 1];
        const uint32_t g0 = block_exclusive(t0 + t1, total, S.warp);
        S.out[d0] = g0 + cnt[(size_t)d0 * tiles + blockIdx.x] - first;
        S.out[d0 + 1] = g0 + t0 + cnt[(size_t)(d0 + 1) * tiles + blockIdx.x] - (first + sum[0]);
#pragma unroll
        for (int w = 0; w < kSortWarps; ++w) {
            S.cnt[w][d0] += first;
            S.cnt[w][d0 + 1] += first + sum[0];
        }
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < kSortItems; ++j)
        if (base + 32 * j < n) {
            const uint32_t at = S.cnt[warp][digit_of(k[j], shift)] + rank[j];
            S.key[at] = k[j];
            S.val[at] = v[j];
        }
    __syncthreads();
    const uint32_t here = min(kSortTile, n - tile0);
#pragma unroll
    for (int j = 0; j < kSortItems; ++j) {
        const uint32_t i = threadIdx.x + j * kSortBlock;
        if (i < here) {
            const unsigned long long key = S.key[i];
            const uint32_t to = S.out[digit_of(key, shift)] + i;
            ok_[to] = key;
            ov[to] = S.val[i];
        }
    }
}

// ---- hierarchy (Karras 2012) -------------------------------------------------
__device__ __forceinline__ int prefix(const unsigned long long* k, int n, int i, int j) {
    if (j < 0 || j >= n) return -1;
    const unsigned long long a = k[i], b = k[j];
    if (a != b) return __clzll(a ^ b);
    return 64 + __clz((uint32_t)i ^ (uint32_t)j);
}

__global__ void __launch_bounds__(256) hierarchy_kernel(int n, Buffers B) {
    const int i = (int)(blockIdx.x * blockDim.x + threadIdx.x);
    if (i >= n - 1) return;
    const unsigned long long* k = B.keys;
    const int d = prefix(k, n, i, i + 1) - prefix(k, n, i, i - 1) > 0 ? 1 : -1;
    const int dmin = prefix(k, n, i, i - d);
    int lmax = 2;
    while (prefix(k, n, i, i + lmax * d) > dmin) lmax <<= 1;
    int l = 0;
    for (int t = lmax >> 1; t >= 1; t >>= 1)
        if (prefix(k, n, i, i + (l + t) * d) > dmin) l += t;
    const int j = i + l * d;
    const int dnode = prefix(k, n, i, j);
    int s = 0;
    for (int div = 2;; div <<= 1) {
        const int t = (l + div - 1) / div;
        if (prefix(k, n, i, i + (s + t) * d) > dnode) s += t;
        if (t <= 1) break;
    }
    const int gamma = i + s * d + min(d, 0);
    const int lo = min(i, j), hi = max(i, j);
    const uint32_t lc = lo == gamma ? (kLeafRef | (uint32_t)gamma) : (uint32_t)gamma;
    const uint32_t rc = hi == gamma + 1 ? (kLeafRef | (uint32_t)(gamma + 1)) : (uint32_t)(gamma + 1);
    B.left[i] = lc;
    B.right[i] = rc;
    if (lc & kLeafRef)
        B.parent_l[gamma] = (uint32_t)i;
    else
        B.parent_i[gamma] = (uint32_t)i;
    if (rc & kLeafRef)
        B.parent_l[gamma + 1] = (uint32_t)i;
    else
        B.parent_i[gamma + 1] = (uint32_t)i;
}

__host__ __device__ __forceinline__ float half_area(float4 lo, float4 hi) {
    const float dx = hi.x - lo.x, dy = hi.y - lo.y, dz = hi.z - lo.z;
    return dx * dy + dy * dz + dz * dx;
}

// ---- finishing an internal node ------------------------------------------------
struct RefBox {
    float4 lo, hi;
    uint32_t count;  // | kLeafNode when the subtree is one leaf
    float cost;
};

__device__ __forceinline__ RefBox ref_box(const Buffers& B, uint32_t ref) {
    RefBox r;
    if (ref & kLeafRef) {
        const uint32_t t = B.vals[ref & ~kLeafRef];
        r.lo = B.blo[t];
        r.hi = B.bhi[t];
        r.count = 1u | kLeafNode;
        r.cost = half_area(r.lo, r.hi);
    } else {
        r.lo = __ldcg(B.nlo + ref);
        r.hi = __ldcg(B.nhi + ref);
        r.count = __float_as_uint(r.lo.w);
        r.cost = r.hi.w;
    }
    return r;
}

// C(ref, 1..8) of a child: a single-triangle leaf costs c_tri x its half area
// whatever the number of roots.
__device__ __forceinline__ void dp_child(const Buffers& B, uint32_t ref, const RefBox& box, float c[8]) {
    if (ref & kLeafRef) {
        const float v = B.c_tri * box.cost;
#pragma unroll
        for (int i = 0; i < 8; ++i) c[i] = v;
    } else {
        const float4 a = __ldcg(reinterpret_cast<const float4*>(B.dpc + 8 * (size_t)ref));
        const float4 b = __ldcg(reinterpret_cast<const float4*>(B.dpc + 8 * (size_t)ref) + 1);
        c[0] = a.x, c[1] = a.y, c[2] = a.z, c[3] = a.w, c[4] = b.x, c[5] = b.y, c[6] = b.z, c[7] = b.w;
    }
}

// Box, count, cost and, for the SAH-optimal collapse, the dynamic programme of
// internal node p, whose children are finished.
__device__ __forceinline__ void finish_node(const Buffers& B, uint32_t p, uint32_t left, uint32_t right,
                                            uint32_t max_leaf, float trav_cost) {
    const RefBox l = ref_box(B, left), r = ref_box(B, right);
    float4 lo = make_float4(fminf(l.lo.x, r.lo.x), fminf(l.lo.y, r.lo.y), fminf(l.lo.z, r.lo.z), 0.0f);
    float4 hi = make_float4(fmaxf(l.hi.x, r.hi.x), fmaxf(l.hi.y, r.hi.y), fmaxf(l.hi.z, r.hi.z), 0.0f);
    const uint32_t cnt = (l.count & ~kLeafNode) + (r.count & ~kLeafNode);
    const float a = half_area(lo, hi);
    const float split = trav_cost * a + l.cost + r.cost;
    const bool leaf = cnt <= max_leaf && (float)cnt * a <= split;
    lo.w = __uint_as_float(cnt | (leaf ? kLeafNode : 0u));
    hi.w = leaf ? (float)cnt * a : split;
    B.nlo[p] = lo;
    B.nhi[p] = hi;
    if (B.dpc) {
        // SAH-optimal collapse: wide node at cost a, leaf slot at c_tri a cnt
        float cl[8], cr[8], sp[7];  // sp[i - 2]: the subtree as i roots, split between the children
        uint32_t sj[7];             // and the left child's share
        dp_child(B, left, l, cl);
        dp_child(B, right, r, cr);
#pragma unroll
        for (int i = 0; i < 7; ++i) {
            sp[i] = FLT_MAX;
            sj[i] = 1;
        }
        // j roots left, k right, in ascending j for every sum
#pragma unroll
        for (int j = 1; j <= 7; ++j)
#pragma unroll
            for (int k = 1; k <= 7; ++k)
                if (j + k <= 8) {
                    const float v = cl[j - 1] + cr[k - 1];
                    if (v < sp[j + k - 2]) {
                        sp[j + k - 2] = v;
                        sj[j + k - 2] = (uint32_t)j;
                    }
                }
        // (constant indices: the tables stay in registers)
        const uint32_t width = B.width;
        const float at_width = width == 8u   ? sp[6]
                               : width == 7u ? sp[5]
                               : width == 6u ? sp[4]
                               : width == 5u ? sp[3]
                               : width == 4u ? sp[2]
                               : width == 3u ? sp[1]
                                             : sp[0];
        const uint32_t j_width = width == 8u   ? sj[6]
                                 : width == 7u ? sj[5]
                                 : width == 6u ? sj[4]
                                 : width == 5u ? sj[3]
                                 : width == 4u ? sj[2]
                                 : width == 3u ? sj[1]
                                               : sj[0];
        float c[8];
        const float node_cost = a + at_width;
        c[0] = node_cost;
        uint32_t as_leaf = 0;
        if (cnt <= (uint32_t)kMaxLeafTris) {
            const float leaf_cost = B.c_tri * a * (float)cnt;
            if (leaf_cost <= node_cost) {
                c[0] = leaf_cost;
                as_leaf = kDpLeaf;
            }
        }
        uint2 ch = make_uint2(j_width | as_leaf, 0u);
#pragma unroll
        for (int i = 2; i <= 8; ++i) {
            const bool two = sp[i - 2] < c[i - 2];
            c[i - 1] = two ? sp[i - 2] : c[i - 2];
            const uint32_t w = two ? sj[i - 2] : 0u;
            if (i <= 4)
                ch.x |= w << 8 * (i - 1);
            else
                ch.y |= w << 8 * (i - 5);
        }
        float4* dc = reinterpret_cast<float4*>(B.dpc + 8 * (size_t)p);
        dc[0] = make_float4(c[0], c[1], c[2], c[3]);
        dc[1] = make_float4(c[4], c[5], c[6], c[7]);
        B.dpch[p] = ch;
    }
}

// The same as a call, for the clustering kernels, which are there for something
// else. (In the walk of refit_kernel the call costs 10%.)
__device__ __noinline__ void finish_made_node(const Buffers& B, uint32_t p, uint32_t max_leaf, float trav_cost) {
    finish_node(B, p, B.left[p], B.right[p], max_leaf, trav_cost);
}

// ---- hierarchy by locally-ordered clustering (Meister & Bittner 2018) -----------
// Clusters start as the sorted single triangles. Each round, every cluster
// finds the neighbour within r positions of the current cluster array whose
// merged box has the least half area (ties: the nearer-to-the-front
// neighbour, which orders every pair by (area, lower index, higher index)
// alike from both ends); mutual neighbours merge into a new internal node at
// the lower position, and the array is compacted in order. The least pair of
// a round is always mutual, so every round of two or more clusters merges at
// least one pair. Internal nodes are numbered down from n - 2 in creation
// order, so the last merge, the root, is node 0 as in the Karras tree, and
// the same collapse follows.
//
// A round is two launches: one finds the neighbours of a tile and of the r
// clusters around it (so a tile knows its mutual pairs by itself), counts
// merges and survivors, and its last block to finish scans the tiles' counts;
// the other merges and compacts. Once kPlocSmall clusters are left one block
// runs the remaining rounds in shared memory. The nodes that a round makes are
// finished (finish_node) by further blocks of the next round's first launch:
// their children are older, so no bottom-up walk, which took 250 us for 1.05M
// triangles, follows; the first launches take 34 us more for it, the last
// kernel 40. Bound: at a million clusters the
// 32-byte cluster records read twice and written once per round, then launch
// latency. The earlier form (four launches a round down to one cluster,
// sixteen consecutive clusters per thread) took 1,110 us for 1.1M triangles.
constexpr int kPlocBlock = 256;
constexpr int kPlocMaxRadius = 64;
constexpr uint32_t kPlocItems = 2;
constexpr uint32_t kPlocTile = kPlocBlock * kPlocItems;  // clusters per block
constexpr uint32_t kPlocSmall = 1024;                    // clusters the last kernel takes
constexpr uint32_t kPlocGone = 0xFFFFFFFFu;              // merged into a lower position
constexpr uint32_t kTellRoot = 8;                        // page-locked word of the root's RootInfo

struct PlocState {
    uint32_t count;      // clusters
    uint32_t next_node;  // internal nodes 0 .. next_node - 1 are still to be made
    uint32_t made_end;   // next_node .. made_end - 1 were made by the round before
    uint32_t pad;
};

// Cluster records: lo.w holds the cluster's reference (bits).
__global__ void __launch_bounds__(kPlocBlock) ploc_init_kernel(uint32_t n, Buffers B, float4* __restrict__ lo,
                                                               float4* __restrict__ hi, PlocState* st,
                                                               uint32_t* ticket) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i == 0) {
        *st = PlocState{n, n - 1u, n - 1u, 0u};
        *ticket = 0;
    }
    if (i >= n) return;
    const uint32_t t = B.vals[i];
    const float4 l = B.blo[t];
    lo[i] = make_float4(l.x, l.y, l.z, __uint_as_float(kLeafRef | i));
    hi[i] = B.bhi[t];
}

// The nearest of the clusters within r of i (positions 0 .. count - 1; at(j)
// gives a position's index in lo / hi).
template <typename At>
__device__ __forceinline__ int ploc_nearest(const float4* lo, const float4* hi, int i, int count, int r, At at) {
    const float4 alo = lo[at(i)], ahi = hi[at(i)];
    float best = __int_as_float(0x7F800000);
    int bj = i;
    const int jlo = max(0, i - r), jhi = min(count - 1, i + r);
    for (int j = jlo; j <= jhi; ++j) {
        if (j == i) continue;
        const float4 olo = lo[at(j)], ohi = hi[at(j)];
        // the lower position's box first, so both ends compute the same bits
        const float4 plo = j < i ? olo : alo, phi = j < i ? ohi : ahi;
        const float4 qlo = j < i ? alo : olo, qhi = j < i ? ahi : ohi;
        const float dx = fmaxf(phi.x, qhi.x) - fminf(plo.x, qlo.x);
        const float dy = fmaxf(phi.y, qhi.y) - fminf(plo.y, qlo.y);
        const float dz = fmaxf(phi.z, qhi.z) - fminf(plo.z, qlo.z);
        // one rounding order wherever this is inlined, so a pair has one area
        // in both kernels; overflowing extents compare as +inf, so the order
        // stays total
        const float area = __fmaf_rn(dz, dx, __fmaf_rn(dy, dz, __fmul_rn(dx, dy)));
        const float d = fminf(area, __int_as_float(0x7F800000));
        if (d < best || bj == i) {
            best = d;
            bj = j;
        }
    }
    return bj;
}

// (merges << 32) | survivors of a cluster: `partner` is its own position when
// it stays alone, the higher one it merges with, or kPlocGone.
__device__ __forceinline__ unsigned long long ploc_weight(uint32_t i, uint32_t partner) {
    return partner == kPlocGone ? 0ull : partner == i ? 1ull : (1ull << 32) + 1ull;
}

__global__ void __launch_bounds__(kPlocBlock) ploc_pair_kernel(const PlocState* __restrict__ st,
                                                               PlocState* __restrict__ next,
                                                               const float4* __restrict__ lo,
                                                               const float4* __restrict__ hi,
                                                               uint32_t* __restrict__ partner,
                                                               unsigned long long* __restrict__ tsum,
                                                               PlocState* seen, uint32_t* ticket, int r, uint32_t tile_blocks,
                                                               Buffers B, uint32_t max_leaf, float trav_cost) {
    __shared__ float4 s_lo[kPlocTile + 4 * kPlocMaxRadius], s_hi[kPlocTile + 4 * kPlocMaxRadius];
    __shared__ int s_nn[kPlocTile + 2 * kPlocMaxRadius];
    __shared__ unsigned long long s_warp[32];
    __shared__ bool s_last;
    if (blockIdx.x >= tile_blocks) {
        // beside the tiles: the nodes that the round before has made
        const uint32_t end = st->made_end;
        for (uint32_t p = st->next_node + (blockIdx.x - tile_blocks) * kPlocBlock + threadIdx.x; p < end;
             p += (gridDim.x - tile_blocks) * kPlocBlock)
            finish_made_node(B, p, max_leaf, trav_cost);
        return;
    }
    const int count = (int)st->count;
    const int b0 = (int)(blockIdx.x * kPlocTile);
    if (b0 < count) {
        for (int k = threadIdx.x; k < (int)kPlocTile + 4 * r; k += kPlocBlock) {
            const int g = b0 - 2 * r + k;
            if (g >= 0 && g < count) {
                s_lo[k] = lo[g];
                s_hi[k] = hi[g];
            }
        }
        __syncthreads();
        for (int k = threadIdx.x; k < (int)kPlocTile + 2 * r; k += kPlocBlock) {
            const int i = b0 - r + k;
            if (i >= 0 && i < count)
                s_nn[k] = ploc_nearest(s_lo, s_hi, i, count, r, [&](int j) { return j - b0 + 2 * r; });
        }
        __syncthreads();
        unsigned long long v = 0;
#pragma unroll
        for (uint32_t q = 0; q < kPlocItems; ++q) {
            const int i = b0 + (int)(threadIdx.x * kPlocItems + q);
            if (i >= count) continue;
            const int j = s_nn[i - b0 + r];
            const bool mutual = j != i && s_nn[j - b0 + r] == i;
            const uint32_t p = !mutual ? (uint32_t)i : i < j ? (uint32_t)j : kPlocGone;
            partner[i] = p;
            v += ploc_weight((uint32_t)i, p);
        }
        unsigned long long total;
        block_exclusive(v, total, s_warp);
        if (threadIdx.x == 0) tsum[blockIdx.x] = total;
    }
    // the last block scans the tiles' sums and writes the next round's state
    if (threadIdx.x == 0) {
        __threadfence();
        s_last = atomicAdd(ticket, 1u) == tile_blocks - 1u;
    }
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    const uint32_t tiles = ((uint32_t)count + kPlocTile - 1) / kPlocTile;
    unsigned long long carry = 0;
    for (uint32_t c0 = 0; c0 < tiles; c0 += 4 * kPlocBlock) {
        const uint32_t k = c0 + 4u * threadIdx.x;
        unsigned long long c[4], v = 0;
        for (uint32_t j = 0; j < 4; ++j) {
            c[j] = k + j < tiles ? __ldcg(tsum + k + j) : 0ull;
            v += c[j];
        }
        unsigned long long total;
        unsigned long long run = carry + block_exclusive(v, total, s_warp);
        for (uint32_t j = 0; j < 4; ++j) {
            if (k + j < tiles) tsum[k + j] = run;
            run += c[j];
        }
        carry += total;
    }
    if (threadIdx.x == 0) {
        *next = PlocState{(uint32_t)carry, st->next_node - (uint32_t)(carry >> 32), st->next_node, 0u};
        *seen = *next;  // (page-locked host memory)
        *ticket = 0;
    }
}

// Clusters a (lower position) and b become internal node `node`.
__device__ __forceinline__ void ploc_join(const Buffers& B, uint32_t node, float4& alo, float4& ahi, float4 blo,
                                          float4 bhi) {
    const uint32_t a = __float_as_uint(alo.w), b = __float_as_uint(blo.w);
    B.left[node] = a;
    B.right[node] = b;
    alo = make_float4(fminf(alo.x, blo.x), fminf(alo.y, blo.y), fminf(alo.z, blo.z), __uint_as_float(node));
    ahi = make_float4(fmaxf(ahi.x, bhi.x), fmaxf(ahi.y, bhi.y), fmaxf(ahi.z, bhi.z), 0.0f);
}

__global__ void __launch_bounds__(kPlocBlock) ploc_merge_kernel(const PlocState* __restrict__ st,
                                                                const unsigned long long* __restrict__ tsum,
                                                                const uint32_t* __restrict__ partner,
                                                                const float4* __restrict__ lin,
                                                                const float4* __restrict__ hin,
                                                                float4* __restrict__ lout, float4* __restrict__ hout,
                                                                Buffers B) {
    __shared__ unsigned long long s_warp[32];
    const uint32_t count = st->count, next_node = st->next_node;
    if (blockIdx.x * kPlocTile >= count) return;
    const uint32_t base = blockIdx.x * kPlocTile + threadIdx.x * kPlocItems;
    uint32_t p[kPlocItems];
    unsigned long long v = 0;
#pragma unroll
    for (uint32_t q = 0; q < kPlocItems; ++q) {
        p[q] = base + q < count ? partner[base + q] : kPlocGone;
        v += ploc_weight(base + q, p[q]);
    }
    unsigned long long total;
    unsigned long long run = tsum[blockIdx.x] + block_exclusive(v, total, s_warp);
#pragma unroll
    for (uint32_t q = 0; q < kPlocItems; ++q) {
        const uint32_t i = base + q;
        if (p[q] == kPlocGone) continue;
        float4 lo = lin[i], hi = hin[i];
        if (p[q] != i) ploc_join(B, next_node - 1u - (uint32_t)(run >> 32), lo, hi, lin[p[q]], hin[p[q]]);
        lout[(uint32_t)run] = lo;
        hout[(uint32_t)run] = hi;
        run += ploc_weight(i, p[q]);
    }
}

// The rounds of at most kPlocSmall clusters, by one block. Every round merges
// a pair, so there are fewer rounds than clusters; the bound only guards.
__global__ void __launch_bounds__(kPlocSmall) ploc_small_kernel(const PlocState* __restrict__ st, PlocState* seen,
                                                                const float4* __restrict__ lin,
                                                                const float4* __restrict__ hin, int r, Buffers B,
                                                                uint32_t max_leaf, float trav_cost) {
    __shared__ float4 s_lo[kPlocSmall], s_hi[kPlocSmall];
    __shared__ int s_nn[kPlocSmall];
    __shared__ uint32_t s_made[kPlocSmall + 1];  // next_node before each round, and after the last
    __shared__ unsigned long long s_warp[32];
    uint32_t rounds = 0;
    uint32_t count = st->count, next_node = st->next_node;
    const uint32_t i = threadIdx.x;
    if (count > kPlocSmall) {  // the host sees the count and reports it
        if (i == 0) *seen = *st;
        return;
    }
    if (i < count) {
        s_lo[i] = lin[i];
        s_hi[i] = hin[i];
    }
    __syncthreads();
    for (uint32_t round = 0; count > 1u && round < kPlocSmall; ++round) {
        if (i < count) s_nn[i] = ploc_nearest(s_lo, s_hi, (int)i, (int)count, r, [](int j) { return j; });
        __syncthreads();
        uint32_t p = kPlocGone;
        if (i < count) {
            const int j = s_nn[i];
            const bool mutual = j != (int)i && s_nn[j] == (int)i;
            p = !mutual ? i : (int)i < j ? (uint32_t)j : kPlocGone;
        }
        unsigned long long total;
        const unsigned long long run = block_exclusive(ploc_weight(i, p), total, s_warp);
        float4 lo, hi;
        if (p != kPlocGone) {
            lo = s_lo[i];
            hi = s_hi[i];
            if (p != i) ploc_join(B, next_node - 1u - (uint32_t)(run >> 32), lo, hi, s_lo[p], s_hi[p]);
        }
        __syncthreads();
        if (p != kPlocGone) {
            s_lo[(uint32_t)run] = lo;
            s_hi[(uint32_t)run] = hi;
        }
        __syncthreads();
        if ((uint32_t)(total >> 32) == 0u) break;
        if (i == 0) s_made[rounds] = next_node;
        rounds++;
        count = (uint32_t)total;
        next_node -= (uint32_t)(total >> 32);
    }
    // the nodes of the last merge before this kernel, then of each round here
    const uint32_t first = st->next_node, end = st->made_end;
    for (uint32_t p = first + i; p < end; p += kPlocSmall) finish_made_node(B, p, max_leaf, trav_cost);
    if (i == 0) s_made[rounds] = next_node;
    for (uint32_t k = 0; k < rounds; ++k) {
        __threadfence_block();
        __syncthreads();
        const uint32_t p = s_made[k + 1] + i;
        if (p < s_made[k]) finish_made_node(B, p, max_leaf, trav_cost);
    }
    __syncthreads();
    if (i == 0) *seen = PlocState{count, next_node, next_node, 0u};
}

// Bound: the memory traffic of the node records near the leaves, then the
// dependent steps of the walk's upper levels. A node is two vectors (count and
// cost in their w), its decisions one 8-byte word, the programme's tables stay
// in registers (loops unrolled): with byte-wise stores, separate count and cost
// arrays and tables in local memory 1.1M triangles took 343 us.
__global__ void __launch_bounds__(256) refit_kernel(uint32_t n, Buffers B, uint32_t max_leaf, float trav_cost) {
    const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n || n < 2) return;
    uint32_t p = B.parent_l[k];
    // a root path has fewer than n nodes; the bound only guards the walk
    for (uint32_t steps = 0; p != kNone; ++steps) {
        if (steps >= n) {
            atomicOr(B.status, 8u);
            return;
        }
        __threadfence();
        if (atomicAdd(B.flag + p, 1u) == 0u) return;  // the sibling subtree is not finished yet
        __threadfence();
        const uint32_t left = B.left[p], right = B.right[p], up = B.parent_i[p];
        finish_node(B, p, left, right, max_leaf, trav_cost);
        p = up;
    }
}

// ---- collapse to 8-wide nodes -------------------------------------------------
struct CollapseArgs {
    Buffers B;
    const float* verts;
    const uint32_t* idx;
    WideNode* nodes;
    float4* tris;  // three vertices per triangle
    float margin;
    int level;
};

// Eight lanes make one wide node, a lane per child: 16 nodes per block at a
// time. Bound: the dependent loads of the binary tree (children, decisions,
// boxes) and, at the leaves, the scattered vertex reads. One thread per node
// kept its eight children's boxes, slots and stacks in local memory and left
// most of the chip idle: 1.1M triangles, 85,751 nodes, 1098 us over all levels;
// eight lanes: 318 us.
constexpr int kCollapseBlock = 128;

__device__ __forceinline__ float group_min(float v) {
    for (int o = 4; o > 0; o >>= 1) v = fminf(v, __shfl_xor_sync(kFull, v, o, 8));
    return v;
}
__device__ __forceinline__ float group_max(float v) {
    for (int o = 4; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(kFull, v, o, 8));
    return v;
}
template <typename T>
__device__ __forceinline__ T group_get(T v, int src) {
    return __shfl_sync(kFull, v, src, 8);
}

__global__ void __launch_bounds__(kCollapseBlock) collapse_kernel(const CollapseArgs A) {
    __shared__ __align__(16) WideNode s_node[kCollapseBlock / 8];
    __shared__ uint32_t s_leaves;
    const Buffers& B = A.B;
    uint32_t* counters = B.counters;
    const uint32_t count = counters[4 + A.level];
    const uint2* qin = (A.level & 1) ? B.qb : B.qa;
    uint2* qout = (A.level & 1) ? B.qa : B.qb;
    const int lane = threadIdx.x & 31, c = lane & 7;      // c: this lane's child
    const uint32_t gmask = 0xFFu << (lane & 24);          // the lanes of this node
    WideNode& nd = s_node[threadIdx.x >> 3];
    uint32_t first_next = 0;  // wide index of the next level's first node
    for (int l = 0; l <= A.level; ++l) first_next += counters[4 + l];
    uint32_t leaves = 0;
    if (threadIdx.x == 0) s_leaves = 0;
    __syncthreads();
    const uint32_t warps = gridDim.x * (kCollapseBlock / 32);
    const uint32_t warp = blockIdx.x * (kCollapseBlock / 32) + (threadIdx.x >> 5);
    for (uint32_t base = 4u * warp; base < count; base += 4u * warps) {  // the same for the whole warp
        const uint32_t it = base + (uint32_t)(lane >> 3);
        const bool node = it < count;
        const uint2 item = node ? qin[it] : make_uint2(kLeafRef, 0u);
        const bool inner = node && !(item.x & kLeafRef);
        // ---- the children: lane c of the first nk holds child c ----------------
        uint32_t kid = item.x;
        int nk = node ? 1 : 0;
        bool dp_leaf = true;
        if (B.dpc) {
            // the SAH-optimal decisions, all open subtrees split at once, in
            // left-to-right order: (subtree, roots it may become)
            uint32_t roots = 0;
            if (inner) {
                const uint32_t j = B.dpch[item.x].x & (kDpLeaf - 1u);
                kid = c == 0 ? B.left[item.x] : B.right[item.x];
                roots = c == 0 ? j : B.width - j;
                nk = 2;
            }
            for (int round = 0; round < kWidth; ++round) {
                uint32_t split = 0;  // roots of the left part, 0: done
                if (inner && c < nk && roots >= 2u && !(kid & kLeafRef)) {
                    const uint2 w = B.dpch[kid];
                    while (roots >= 2u) {
                        split = (roots > 4u ? w.y >> 8 * (roots - 5u) : w.x >> 8 * (roots - 1u)) & 255u;
                        if (split) break;
                        --roots;
                    }
                }
                const uint32_t splits = __ballot_sync(kFull, split != 0u);
                if (splits == 0u) break;
                // entry e becomes entries at e + (splits before it)
                const int total = nk + __popc(splits & gmask);
                if (total > kWidth && inner) {
                    if (c == 0) atomicOr(B.status, 8u);  // more than 8 roots: malformed decisions
                }
                // lane d of the new list: its old entry e and which part
                int e = 0, second = 0;
                for (int q = 0, at = 0; q < kWidth; ++q) {  // at: first new entry of old entry q
                    const int two = (splits >> ((lane & 24) + q)) & 1;
                    if (q < nk && at <= c) {
                        e = q;
                        second = two ? c - at : 0;
                    }
                    at += 1 + two;
                }
                const uint32_t ok_kid = group_get(kid, e), ok_split = group_get(split, e), ok_roots = group_get(roots, e);
                kid = ok_kid;
                roots = ok_roots;
                if (inner && ok_split) {
                    kid = second ? B.right[ok_kid] : B.left[ok_kid];
                    roots = second ? ok_roots - ok_split : ok_split;
                }
                nk = min(total, kWidth);
            }
            if (inner && c < nk) dp_leaf = (kid & kLeafRef) || (B.dpch[kid].x & kDpLeaf);
        } else {
            // greedy: the largest inner child is opened until there are width
            float area = -1.0f;
            auto look = [&] {  // area of an openable child, -1 for the others
                area = -1.0f;
                if (node && c < nk && !(kid & kLeafRef)) {
                    const float4 lo = __ldcg(B.nlo + kid);
                    if (!(__float_as_uint(lo.w) & kLeafNode))
                        area = fmaxf(half_area(lo, __ldcg(B.nhi + kid)), -1.0f);  // (a NaN: not opened)
                }
            };
            look();
            for (int round = 0; round < kWidth; ++round) {
                float best = area;
                int pick = c;
                for (int o = 1; o < 8; o <<= 1) {
                    const float b2 = __shfl_xor_sync(kFull, best, o, 8);
                    const int p2 = __shfl_xor_sync(kFull, pick, o, 8);
                    if (b2 > best || (b2 == best && p2 < pick)) {
                        best = b2;
                        pick = p2;
                    }
                }
                const bool open = best > -1.0f && nk < (int)B.width;
                if (__ballot_sync(kFull, open) == 0u) break;
                const uint32_t p = group_get(kid, pick);
                if (open) {
                    if (c == pick) kid = B.left[p];
                    if (c == nk) kid = B.right[p];
                    nk++;
                    if (c == pick || c == nk - 1) look();
                }
            }
        }
        const bool have = node && c < nk;
        // ---- child boxes inflated by the margin (one ulp outward when the
        // subtraction rounds back), node box
        float clo[3] = {FLT_MAX, FLT_MAX, FLT_MAX}, chi[3] = {-FLT_MAX, -FLT_MAX, -FLT_MAX};
        uint32_t cnt = 0;
        bool is_leaf = false;
        if (have) {
            float4 lo, hi;
            if (kid & kLeafRef) {
                const uint32_t t = B.vals[kid & ~kLeafRef];
                lo = B.blo[t];
                hi = B.bhi[t];
                cnt = 1;
                is_leaf = true;
            } else {
                lo = __ldcg(B.nlo + kid);
                hi = __ldcg(B.nhi + kid);
                const uint32_t w = __float_as_uint(lo.w);
                is_leaf = (B.dpc && inner) ? dp_leaf : (w & kLeafNode) != 0u;
                cnt = w & ~kLeafNode;
            }
            const float l3[3] = {lo.x, lo.y, lo.z}, h3[3] = {hi.x, hi.y, hi.z};
#pragma unroll
            for (int a = 0; a < 3; ++a) {
                float x = l3[a] - A.margin, y = h3[a] + A.margin;
                if (!(x < l3[a])) x = nextafterf(l3[a], -INFINITY);
                if (!(y > h3[a])) y = nextafterf(h3[a], INFINITY);
                clo[a] = x;
                chi[a] = y;
            }
        }
        float nlo[3], nhi[3];
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            nlo[a] = group_min(clo[a]);
            nhi[a] = group_max(chi[a]);
        }
        // ---- octant slots, greedy on the corner score (as collapse.cpp): of the
        // children without a slot and the free slots, the best pair first (the
        // lower child, then the lower slot, on equal scores)
        const float dx = 0.5f * (clo[0] + chi[0]) - 0.5f * (nlo[0] + nhi[0]);
        const float dy = 0.5f * (clo[1] + chi[1]) - 0.5f * (nlo[1] + nhi[1]);
        const float dz = 0.5f * (clo[2] + chi[2]) - 0.5f * (nlo[2] + nhi[2]);
        int slot = have ? -1 : 8;
        uint32_t used = 0;
        for (int round = 0; round < kWidth; ++round) {
            if (__ballot_sync(kFull, slot < 0) == 0u) break;
            float bv = -INFINITY;
            int bs = 8;
            if (slot < 0) {
#pragma unroll
                for (int q = 0; q < kWidth; ++q) {
                    // (a NaN counts as -inf, so all lanes agree)
                    const float sc = fmaxf(((q & 1) ? dx : -dx) + ((q & 2) ? dy : -dy) + ((q & 4) ? dz : -dz), -INFINITY);
                    if (!(used >> q & 1u) && (sc > bv || bs == 8)) {
                        bv = sc;
                        bs = q;
                    }
                }
            }
            float v = bv;
            int who = bs < 8 ? c : 8;
            for (int o = 1; o < 8; o <<= 1) {
                const float v2 = __shfl_xor_sync(kFull, v, o, 8);
                const int w2 = __shfl_xor_sync(kFull, who, o, 8);
                if (w2 < 8 && (who == 8 || v2 > v || (v2 == v && w2 < who))) {
                    v = v2;
                    who = w2;
                }
            }
            const int won = group_get(bs, who & 7);
            if (who < 8) used |= 1u << won;
            if (c == who) slot = won;
        }
        // ---- grid step 2^e per axis: the least e with 255 2^e >= the node's
        // extent rounded up (all in FP32; 255 2^e and 2^-e are exact)
        int ex[3];
        bool bad = false;
        {
            const float ext = __fsub_ru(c == 0 ? nhi[0] : c == 1 ? nhi[1] : nhi[2], c == 0 ? nlo[0] : c == 1 ? nlo[1] : nlo[2]);
            int e = ext > 0.0f ? ilogbf(ext) - 8 : -100;
            while (e <= 100 && ldexpf(255.0f, e) < ext) e++;
            while (e > -100 && ldexpf(255.0f, e - 1) >= ext) e--;
            bad = node && (e < -100 || e > 100);
#pragma unroll
            for (int a = 0; a < 3; ++a) ex[a] = group_get(e, a);
        }
        // ---- room for the children and triangles: one atomic each per warp ----
        const uint32_t inner_m = __ballot_sync(kFull, have && !is_leaf);
        uint32_t tri_before = 0, node_tris = 0;  // this node's triangles in lower slots; all of them
        uint32_t int_slots = 0;                  // slots of inner children
#pragma unroll
        for (int q = 0; q < kWidth; ++q) {
            const int qs = group_get(slot, q);
            const uint32_t qc = group_get(have && is_leaf ? cnt : 0u, q);
            if (qs < slot) tri_before += qc;
            node_tris += qc;
            if ((inner_m >> ((lane & 24) + q)) & 1u) int_slots |= 1u << qs;
        }
        const uint32_t n_int = (uint32_t)__popc(int_slots);
        uint32_t int_base = 0, tri_base = 0;
        {
            // exclusive sums over the warp's four nodes
            uint32_t ib = 0, tb = 0, it_all = 0, tt_all = 0;
#pragma unroll
            for (int g = 0; g < 4; ++g) {
                const uint32_t gi = __shfl_sync(kFull, n_int, 8 * g), gt = __shfl_sync(kFull, node_tris, 8 * g);
                if (8 * g < (lane & 24)) {
                    ib += gi;
                    tb += gt;
                }
                it_all += gi;
                tt_all += gt;
            }
            if (lane == 0) {
                if (it_all) int_base = atomicAdd(counters + 4 + A.level + 1, it_all);
                if (tt_all) tri_base = atomicAdd(counters + 1, tt_all);
            }
            int_base = __shfl_sync(kFull, int_base, 0) + ib;
            tri_base = __shfl_sync(kFull, tri_base, 0) + tb;
        }
        // ---- the record ---------------------------------------------------------
        uint4* words = reinterpret_cast<uint4*>(&nd);
        if (c < 5) words[c] = make_uint4(0u, 0u, 0u, 0u);
        __syncwarp();
        if (have) {
            // outward: the offsets from p rounded down / up before the
            // exact scaling by 2^-e, so p + ql 2^e <= lo and p + qh 2^e >= hi
            // hold exactly; qh <= 255 since hi - p <= the node's extent
#pragma unroll
            for (int a = 0; a < 3; ++a) {
                const float inv_step = ldexpf(1.0f, -ex[a]);
                const float ql = floorf(__fmul_rd(__fsub_rd(clo[a], nlo[a]), inv_step));
                const float qh = ceilf(__fmul_ru(__fsub_ru(chi[a], nlo[a]), inv_step));
                nd.qlo[a][slot] = (uint8_t)fminf(fmaxf(ql, 0.0f), 255.0f);
                nd.qhi[a][slot] = (uint8_t)fminf(fmaxf(qh, 0.0f), 255.0f);
            }
            nd.meta[slot] = is_leaf ? (uint8_t)(kMetaLeafFlag | ((cnt - 1u) << 5) | tri_before) : kMetaInternal;
        }
        if (node && c == 0) {
#pragma unroll
            for (int a = 0; a < 3; ++a) {
                nd.p[a] = nlo[a];
                nd.e[a] = (uint8_t)(ex[a] + 127);
            }
            nd.imask = (uint8_t)int_slots;
            nd.child_base = n_int ? first_next + int_base : 0u;
            nd.tri_base = node_tris ? tri_base : 0u;
        }
        __syncwarp();
        if (node && c < 5) reinterpret_cast<uint4*>(A.nodes + item.y)[c] = words[c];
        __syncwarp();
        // ---- the children's queue entries, the leaves' triangles -----------------
        bool bad_tree = false;
        if (have && !is_leaf) {
            const uint32_t at = int_base + (uint32_t)__popc(int_slots & ((1u << slot) - 1u));
            qout[at] = make_uint2(kid, first_next + at);
        }
        if (have && is_leaf) {
            // a leaf's triangles: its binary subtree's leaves, left to right
            // (a Morton-order range for the Karras tree, not for clusters)
            leaves++;
            uint32_t st[2 * kMaxLeafTris];
            int sp = 0;
            st[sp++] = kid;
            uint32_t i = 0;
            for (int step = 0; sp > 0 && i < cnt && step < 4 * kMaxLeafTris; ++step) {
                const uint32_t ref = st[--sp];
                if (!(ref & kLeafRef)) {
                    if (sp + 2 > 2 * kMaxLeafTris) break;
                    st[sp++] = B.right[ref];
                    st[sp++] = B.left[ref];
                    continue;
                }
                const uint32_t t = B.vals[ref & ~kLeafRef];
                const size_t d = 3 * ((size_t)tri_base + tri_before + i);
                float v[9];
                for (int k = 0; k < 3; ++k)
                    for (int q = 0; q < 3; ++q) v[3 * k + q] = A.verts[3 * (size_t)A.idx[3 * (size_t)t + k] + q];
                A.tris[d + 0] = make_float4(v[0], v[1], v[2], __uint_as_float(t));
                A.tris[d + 1] = make_float4(v[3], v[4], v[5], 0.0f);
                A.tris[d + 2] = make_float4(v[6], v[7], v[8], 0.0f);
                i++;
            }
            bad_tree = i != cnt;
        }
        if (bad && c < 3) atomicOr(B.status, 4u);
        if (bad_tree) atomicOr(B.status, 8u);
    }
    leaves = __reduce_add_sync(kFull, leaves);
    if (lane == 0 && leaves) atomicAdd(&s_leaves, leaves);
    __syncthreads();
    if (threadIdx.x == 0 && s_leaves) atomicAdd(counters + 2, s_leaves);
}

__global__ void instance_shade_kernel(const float* __restrict__ inv, const uint32_t* __restrict__ prefix,
                                      const uint32_t* __restrict__ off, const float4* const* __restrict__ blas,
                                      uint32_t n_inst, uint32_t total, float4* __restrict__ out) {
    const uint32_t g = blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= total) return;
    uint32_t lo = 0, hi = n_inst;  // prefix[lo] <= g < prefix[hi]
    while (hi - lo > 1) {
        const uint32_t mid = (lo + hi) >> 1;
        if (prefix[mid] <= g)
            lo = mid;
        else
            hi = mid;
    }
    const uint32_t t = g - prefix[lo];
    const float4 n = blas[lo][t];
    const float* m = inv + 12 * (size_t)lo;
    float w[3];
    for (int j = 0; j < 3; ++j) w[j] = m[j] * n.x + m[4 + j] * n.y + m[8 + j] * n.z;
    const float l = sqrtf(w[0] * w[0] + w[1] * w[1] + w[2] * w[2]);
    const float k = l > 0.0f ? 1.0f / l : 0.0f;
    out[(size_t)off[lo] + t] = l > 0.0f ? make_float4(w[0] * k, w[1] * k, w[2] * k, 0.0f) : make_float4(0, 0, 1, 0);
}

// The collapse's first queue entry, level 0 of one node.
// The collapse's first item, and what the host asks of the root (`told`).
struct RootInfo {
    float4 lo, hi;
    float wide_cost;
};
__global__ void root_kernel(Buffers B, uint2 item, bool internal, RootInfo* told) {
    B.qa[0] = item;
    B.counters[4] = 1u;
    if (internal) *told = RootInfo{B.nlo[0], B.nhi[0], B.dpc ? B.dpc[0] : 0.0f};
}

// The status word and `n` words behind `at` into page-locked host memory. The
// device tells the host its few answers by kernels: a copy of some bytes holds
// the stream for 8 us, and with one per clustering round (and seven more) an
// upload of 1.05M triangles, its trace and its end took 1,595 us instead of
// 1,348.
__global__ void __launch_bounds__(128) tell_kernel(const uint32_t* __restrict__ status, const uint32_t* __restrict__ at,
                                                   uint32_t n, uint32_t* told) {
    if (threadIdx.x == 0) told[0] = *status;
    for (uint32_t i = threadIdx.x; i < n; i += blockDim.x) told[4 + i] = at[i];
}

__global__ void interleave_kernel(const float4* __restrict__ planes, uint32_t n, float4* __restrict__ tris) {
    const size_t j = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (j < 3 * (size_t)n) tris[j] = planes[(j % 3) * n + j / 3];
}

__global__ void write_ids_kernel(float4* shade, const uint32_t* ids, uint32_t nt) {
    const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t < nt) reinterpret_cast<uint32_t*>(shade + t)[3] = ids[t];
}

double Ms(std::chrono::steady_clock::time_point t0) {
    return std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t0).count();
}

void Check(cudaError_t e, const char* what) {
    if (e != cudaSuccess)
        RtCore::Fail(e == cudaErrorMemoryAllocation ? FND_ERR_OUT_OF_MEMORY : FND_ERR_CUDA, "%s: %s", what,
                   cudaGetErrorString(e));
}

// Owner of the temporary device allocations of one build (stream order).
struct Scratch {
    cudaMemPool_t pool;
    cudaStream_t s;
    std::vector<void*> ptrs;
    Scratch(cudaMemPool_t pool, cudaStream_t s) : pool(pool), s(s) {}
    Scratch(const Scratch&) = delete;
    Scratch& operator=(const Scratch&) = delete;
    template <typename T>
    T* get(size_t count) {
        void* p = nullptr;
        Check(cudaMallocFromPoolAsync(&p, std::max<size_t>(count, 1) * sizeof(T), pool, s), "GPU build scratch");
        ptrs.push_back(p);
        return static_cast<T*>(p);
    }
    ~Scratch() {
        for (void* p : ptrs) cudaFreeAsync(p, s);
    }
};

void RadixSort(Buffers& B, uint32_t n, cudaStream_t s) {
    const uint32_t tiles = (n + kSortTile - 1) / kSortTile;
    uint32_t* totals = B.cnt + (size_t)kDigits * tiles;
    Check(cudaFuncSetAttribute(scatter_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(SortShared)),
          "radix sort shared memory");
    for (int pass = 0; pass < kSortPasses; ++pass) {
        const uint32_t shift = (uint32_t)(pass * kDigitBits);
        hist_kernel<<<tiles, kSortBlock, 0, s>>>(B.keys, n, shift, tiles, B.cnt);
        scan_rows_kernel<<<kDigits, kScanRow, 0, s>>>(B.cnt, tiles, totals);
        scatter_kernel<<<tiles, kSortBlock, sizeof(SortShared), s>>>(B.keys, B.vals, n, shift, tiles, B.cnt, totals,
                                                                     B.keys2, B.vals2);
        std::swap(B.keys, B.keys2);
        std::swap(B.vals, B.vals2);
    }
    Check(cudaGetLastError(), "radix sort launch");
}

// The clustering rounds of ploc_*_kernel. Each round's grids are sized by
// the cluster count read back one round late (an upper bound: counts only
// fall), so the host never waits for the round it has just queued.
void PlocHierarchy(Buffers& B, uint32_t n, int r, uint32_t max_leaf, float trav_cost, GpuBuildResources& res,
                   cudaStream_t s) {
    Scratch S(res.pool, s);
    float4* lo[2] = {S.get<float4>(n), S.get<float4>(n)};
    float4* hi[2] = {S.get<float4>(n), S.get<float4>(n)};
    uint32_t* partner = S.get<uint32_t>(n);
    unsigned long long* tsum = S.get<unsigned long long>((n + kPlocTile - 1) / kPlocTile);
    PlocState* st = S.get<PlocState>(2);
    uint32_t* ticket = S.get<uint32_t>(1);
    PlocState* h = reinterpret_cast<PlocState*>(res.pinned);  // one slot per round in flight
    cudaEvent_t* ev = res.ev;
    ploc_init_kernel<<<(n + kPlocBlock - 1) / kPlocBlock, kPlocBlock, 0, s>>>(n, B, lo[0], hi[0], st, ticket);
    uint32_t bound = n;  // at least the clusters of the round about to be queued
    int cur = 0;
    // every round of two or more clusters merges a pair: at most n - 1 rounds
    for (uint32_t round = 0; bound > kPlocSmall && round <= n; ++round) {
        const uint32_t tiles = (bound + kPlocTile - 1) / kPlocTile;
        // as many blocks again for the nodes to finish
        ploc_pair_kernel<<<2 * tiles, kPlocBlock, 0, s>>>(st + cur, st + (cur ^ 1), lo[cur], hi[cur], partner, tsum,
                                                          h + (round & 1), ticket, r, tiles, B, max_leaf, trav_cost);
        Check(cudaEventRecord(ev[round & 1], s), "event");
        ploc_merge_kernel<<<tiles, kPlocBlock, 0, s>>>(st + cur, tsum, partner, lo[cur], hi[cur], lo[cur ^ 1],
                                                       hi[cur ^ 1], B);
        cur ^= 1;
        if (round == 0) continue;
        Check(cudaEventSynchronize(ev[(round - 1) & 1]), "clustering round");
        const uint32_t c = h[(round - 1) & 1].count;
        if (round > 1 && c >= bound) break;  // a round without a merge
        bound = c;
    }
    ploc_small_kernel<<<1, kPlocSmall, 0, s>>>(st + cur, h, lo[cur], hi[cur], r, B, max_leaf, trav_cost);
}

// After the stream has passed PlocHierarchy's kernels.
void CheckClustered(const GpuBuildResources& res) {
    const PlocState* h = reinterpret_cast<const PlocState*>(res.pinned);
    CHECK_CODE(h->count == 1 && h->next_node == 0, FND_ERR_INVALID_SCENE, "GPU build: clustering stopped at %u clusters",
               h->count);
}

}  // namespace

void BuildWideGpu(const float* d_verts, uint32_t nv, const uint32_t* d_idx, uint32_t nt, const GpuBuildParams& p,
                  GpuBuildResources& res, GpuBuildOutput& out, cudaStream_t s) {
    CHECK_CODE(nt >= 1 && nt <= kGpuBuildMaxTris, FND_ERR_INVALID_ARG, "GPU build takes 1..%u triangles, not %u",
               kGpuBuildMaxTris, nt);
    CHECK_CODE(p.max_leaf >= 1 && p.max_leaf <= (uint32_t)kMaxLeafTris, FND_ERR_INVALID_ARG, "max_leaf %u",
               p.max_leaf);
    CHECK_CODE(p.width >= 2 && p.width <= (uint32_t)kWidth, FND_ERR_INVALID_ARG, "node width %u not in 2..%d",
               p.width, kWidth);
    CHECK_CODE(p.ploc_radius <= (uint32_t)kPlocMaxRadius, FND_ERR_INVALID_ARG, "clustering radius %u above %d",
               p.ploc_radius, kPlocMaxRadius);
    int dev = 0, sms = 0;
    Check(cudaGetDevice(&dev), "cudaGetDevice");
    Check(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev), "SM count");
    const auto t0 = std::chrono::steady_clock::now();
    Scratch S(res.pool, s);
    Buffers B{};
    const uint32_t n = nt;
    B.blo = S.get<float4>(n);
    B.bhi = S.get<float4>(n);
    B.keys = S.get<unsigned long long>(n);
    B.vals = S.get<uint32_t>(n);
    B.keys2 = S.get<unsigned long long>(n);
    B.vals2 = S.get<uint32_t>(n);
    B.cnt = S.get<uint32_t>((uint64_t)kDigits * ((n + kSortTile - 1) / kSortTile) + kDigits);
    B.left = S.get<uint32_t>(n);
    B.right = S.get<uint32_t>(n);
    const bool walk = p.ploc_radius == 0;  // nodes finished by refit_kernel, not by the clustering
    if (walk) {
        B.parent_i = S.get<uint32_t>(n);
        B.parent_l = S.get<uint32_t>(n);
        B.flag = S.get<uint32_t>(n);
    }
    B.nlo = S.get<float4>(n);
    B.nhi = S.get<float4>(n);
    B.bounds = S.get<float>(12);
    B.status = S.get<uint32_t>(1);
    B.counters = S.get<uint32_t>(4 + kMaxLevels + 2);
    B.width = p.width;
    B.qa = S.get<uint2>(n);
    B.qb = S.get<uint2>(n);
    if (p.sah_collapse && n >= 2) {
        B.dpc = S.get<float>(8ull * n);
        B.dpch = S.get<uint2>(n);
        B.c_tri = p.c_tri;
    }
    auto keep = [&](void** p, size_t bytes, const char* what) {
        Check(cudaMallocFromPoolAsync(p, bytes, res.pool, s), what);
    };
    keep(&out.d_tri_shade, 16ull * n, "shading normals");
    float4* shade = static_cast<float4*>(out.d_tri_shade);
    Check(cudaMemsetAsync(B.status, 0, 4, s), "memset");
    if (walk) {
        Check(cudaMemsetAsync(B.flag, 0, 4ull * n, s), "memset");
        Check(cudaMemsetAsync(B.parent_i, 0xFF, 4ull * n, s), "memset");
        Check(cudaMemsetAsync(B.parent_l, 0xFF, 4ull * n, s), "memset");
    }
    Check(cudaMemsetAsync(B.counters, 0, 4ull * (4 + kMaxLevels + 2), s), "memset");
    init_bounds_kernel<<<1, 32, 0, s>>>(B.bounds);
    const uint32_t g256 = (n + 255) / 256;
    prep_kernel<<<std::max(1u, std::min(g256, 8u * (uint32_t)sms)), 256, 0, s>>>(d_verts, nv, d_idx, n, B, shade);
    uint32_t* pinned = res.pinned;
    float h_bounds[12];
    tell_kernel<<<1, 128, 0, s>>>(B.status, reinterpret_cast<const uint32_t*>(B.bounds), 12, pinned);
    Check(cudaGetLastError(), "prep launch");
    Check(cudaStreamSynchronize(s), "prep");
    uint32_t h_status = pinned[0];
    std::memcpy(h_bounds, pinned + 4, sizeof(h_bounds));
    CHECK_CODE(!(h_status & kPrepBadIndex), FND_ERR_INVALID_ARG, "vertex index out of range (nv = %u)", nv);
    CHECK_CODE(!(h_status & kPrepNonFinite), FND_ERR_INVALID_ARG, "non-finite vertex coordinate");
    for (int a = 0; a < 3; ++a) {
        out.lo[a] = h_bounds[a];
        out.hi[a] = h_bounds[3 + a];
    }
    out.margin = SceneMargin(out.lo, out.hi) * p.margin_scale;
    morton_kernel<<<g256, 256, 0, s>>>(n, B);
    RadixSort(B, n, s);
    if (n >= 2) {
        if (walk) {
            hierarchy_kernel<<<(n - 1 + 255) / 256, 256, 0, s>>>((int)n, B);
            refit_kernel<<<g256, 256, 0, s>>>(n, B, p.max_leaf, p.trav_cost);
        } else {
            PlocHierarchy(B, n, (int)p.ploc_radius, p.max_leaf, p.trav_cost, res, s);
        }
    }
    Check(cudaGetLastError(), "hierarchy launch");
    // root item: internal node 0, or the single leaf
    static_assert(kTellRoot >= 2 * sizeof(PlocState) / 4 && 4 * kTellRoot % alignof(RootInfo) == 0 &&
                      kTellRoot + sizeof(RootInfo) / 4 <= kGpuBuildPinnedWords,
                  "behind the clustering's states");
    RootInfo* told = reinterpret_cast<RootInfo*>(pinned + kTellRoot);
    root_kernel<<<1, 1, 0, s>>>(B, make_uint2(n >= 2 ? 0u : kLeafRef, 0u), n >= 2, told);
    float root_cost = 0.0f, wide_cost = 0.0f;
    float4 rlo{}, rhi{};
    Check(cudaGetLastError(), "root launch");
    Check(cudaStreamSynchronize(s), "LBVH");
    if (n >= 2) {
        if (!walk) CheckClustered(res);
        wide_cost = told->wide_cost;
        rlo = told->lo;
        rhi = told->hi;
    }
    out.build_ms = Ms(t0);
    const auto t1 = std::chrono::steady_clock::now();
    WideNode* nodes = S.get<WideNode>(n);
    keep(&out.d_tris, 48ull * n, "triangles");
    CollapseArgs A{};
    A.B = B;
    A.verts = d_verts;
    A.idx = d_idx;
    A.nodes = nodes;
    A.tris = static_cast<float4*>(out.d_tris);
    A.margin = out.margin;
    const int grid = std::max(1, sms * 8);
    // scenes of ordinary depth end within the first levels; the rest is
    // queued only when the last of them left nodes
    constexpr int kFirstLevels = 12;
    uint32_t h_counters[4 + kMaxLevels + 2];
    static_assert(4 + sizeof(h_counters) / 4 <= kGpuBuildPinnedWords, "the counters fit the page-locked words");
    for (int level = 0; level < kMaxLevels;) {
        const int end = level == 0 ? kFirstLevels : kMaxLevels;
        for (; level < end; ++level) {
            A.level = level;
            collapse_kernel<<<grid, kCollapseBlock, 0, s>>>(A);
        }
        tell_kernel<<<1, 128, 0, s>>>(B.status, B.counters, sizeof(h_counters) / 4, pinned);
        Check(cudaGetLastError(), "collapse launch");
        Check(cudaStreamSynchronize(s), "collapse");
        h_status = pinned[0];
        std::memcpy(h_counters, pinned + 4, sizeof(h_counters));
        if (h_counters[4 + level] == 0) break;
    }
    CHECK_CODE(h_counters[4 + kMaxLevels] == 0, FND_ERR_INVALID_SCENE,
               "wide BVH deeper than the traversal stack bound %d", kMaxLevels);
    CHECK_CODE(!(h_status & 4u), FND_ERR_INVALID_SCENE, "child box quantisation failed (scene extent out of range)");
    CHECK_CODE(!(h_status & 8u), FND_ERR_INVALID_SCENE, "GPU build: malformed hierarchy");
    CHECK_CODE(h_counters[1] == n, FND_ERR_INVALID_SCENE, "collapse placed %u of %u triangles", h_counters[1], n);
    out.num_nodes = 0;
    for (int l = 0; l < kMaxLevels; ++l) out.num_nodes += h_counters[4 + l];
    out.num_refs = n;
    out.leaves = h_counters[2];
    out.depth = 0;
    for (int l = 0; l < kMaxLevels; ++l)
        if (h_counters[4 + l]) out.depth = (uint32_t)l + 1;
    out.num_binary_nodes = 2 * n - 1;
    root_cost = rhi.w;
    const float ra = n >= 2 ? half_area(rlo, rhi) : 0.0f;
    out.sah_cost = n >= 2 && ra > 0.0f ? (double)root_cost / (double)ra : 0.0;
    if (B.dpc)
        LOG_RUNTIME(FndRt, INFO, "SAH-optimal collapse: wide-tree cost %.4f (root half-area normalised)",
                    ra > 0.0f ? (double)wide_cost / (double)ra : 0.0);
    // exact-size node array
    keep(&out.d_nodes, sizeof(WideNode) * (size_t)out.num_nodes, "wide nodes");
    Check(cudaMemcpyAsync(out.d_nodes, nodes, sizeof(WideNode) * (size_t)out.num_nodes, cudaMemcpyDeviceToDevice, s),
          "node copy");
    Check(cudaStreamSynchronize(s), "node copy");
    out.collapse_ms = Ms(t1);
}

cudaError_t CreateGpuBuildResources(int device, GpuBuildResources& r) {
    cudaError_t e = cudaSuccess;
    if (!r.pool) {
        cudaMemPoolProps props{};
        props.allocType = cudaMemAllocationTypePinned;
        props.location.type = cudaMemLocationTypeDevice;
        props.location.id = device;
        e = cudaMemPoolCreate(&r.pool, &props);
        if (e != cudaSuccess) return e;
        uint64_t bytes = kGpuBuildPoolKeep;
        e = cudaMemPoolSetAttribute(r.pool, cudaMemPoolAttrReleaseThreshold, &bytes);
        if (e != cudaSuccess) return e;
    }
    if (!r.pinned) {
        e = cudaHostAlloc(reinterpret_cast<void**>(&r.pinned), 4 * kGpuBuildPinnedWords, cudaHostAllocDefault);
        if (e != cudaSuccess) return e;
    }
    for (cudaEvent_t& ev : r.ev)
        if (!ev && e == cudaSuccess) e = cudaEventCreateWithFlags(&ev, cudaEventDisableTiming);
    return e;
}

void FreeGpuBuildResources(GpuBuildResources& r) {
    for (cudaEvent_t ev : r.ev)
        if (ev) cudaEventDestroy(ev);
    if (r.pinned) cudaFreeHost(r.pinned);
    if (r.pool) cudaMemPoolDestroy(r.pool);
    r = GpuBuildResources{};
}

cudaError_t InstanceShade(const float* d_inv, const uint32_t* d_prefix, const uint32_t* d_prim_offset,
                          const float4* const* d_blas_shade, uint32_t n_inst, uint32_t total, float4* d_out,
                          cudaStream_t s) {
    if (total == 0 || n_inst == 0) return cudaSuccess;
    instance_shade_kernel<<<(total + 255) / 256, 256, 0, s>>>(d_inv, d_prefix, d_prim_offset, d_blas_shade, n_inst,
                                                                total, d_out);
    return cudaGetLastError();
}

cudaError_t InterleaveTriangles(const float4* d_planes, uint32_t n, float4* d_tris, cudaStream_t s) {
    if (n == 0) return cudaSuccess;
    interleave_kernel<<<(uint32_t)((3 * (size_t)n + 255) / 256), 256, 0, s>>>(d_planes, n, d_tris);
    return cudaGetLastError();
}

cudaError_t WriteMaterialIds(float4* d_tri_shade, const uint32_t* d_ids, uint32_t nt, cudaStream_t s) {
    if (nt == 0) return cudaSuccess;
    write_ids_kernel<<<(nt + 255) / 256, 256, 0, s>>>(d_tri_shade, d_ids, nt);
    return cudaGetLastError();
}

}  // namespace RT
}  // namespace Foundation
