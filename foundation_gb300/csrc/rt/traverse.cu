// traverse.cu — persistent closest-hit / any-hit traversal of the compressed
// 8-wide BVH (sm_103a), for one scene (trace_kernel) or for a table of
// (scene, ray batch, query kind) jobs in one launch (batch_kernel).
//
// Structure (after Aila & Laine, "Understanding the Efficiency of Ray
// Traversal on GPUs", HPG 2009, and Ylitie, Karras & Laine, HPG 2017):
//  * persistent warps: the grid is sized to fill every SM once; each warp
//    pulls rays from a global counter with one atomicAdd per refill and hands
//    the new rays to its idle lanes (dynamic fetch: a warp refills once at
//    least `refill_min` lanes are idle, so long rays do not hold 31 idle
//    lanes hostage);
//  * one thread per ray while rays are left to fetch (then, and in small
//    batches, lanes without work share the others' rays: persistent_trace);
//    the traversal state is a "node group" (base index of a node's internal
//    children + the ordered bit mask of children still to
//    visit), the triangles of hit leaves wait in a ring of the warp (warp_trace.cuh);
//  * a node's hit mask goes to the ray's traversal order through a shared
//    8 x 256-byte table in the single-scene and batched kernels (one load in
//    place of three conditional bit swaps); the two-level kernel, whose
//    shared memory already holds the world rays, keeps the swaps;
//  * the stack holds node groups; its first kShort entries live in shared
//    memory (one column per thread, bank-conflict free), deeper entries in a
//    thread-local array; the depth bound kMaxStack is checked on the host at
//    scene upload and again on every push (a failed push latches
//    kStatusStackOverflow and ends the ray instead of writing out of bounds).
// Block size, short-stack depth and the thresholds are launch parameters
// chosen by the autotuner (capi/capi_batch.cpp); every combination below is
// compiled. Two-level scenes (instances) run the same loop with kTwoLevel: a
// lane descending into an instance pushes a return marker and swaps its ray
// and node arrays to the instance's object space.
//
// What bounds it: instruction issue (about 80% of the slots busy, the rest
// short waits; DRAM moves rays and hits only while the tree fits L2). 64
// registers a thread and 32 warps per SM: at 56 registers (36 warps) the loop
// spills about ten words a node step (8.4M incoherent Cornell rays 1.92 ms
// against 1.77), at 72 (28 warps) it lacks warps (1.81 ms).
#include <algorithm>
#include <cfloat>

#include "traverse.cuh"
#include "ray_sort.hpp"
#include "traverse_launch.hpp"
#include "warp_trace.cuh"

namespace Foundation {
namespace RT {

namespace {

// The largest batch for it (117 thousand rays on the full chip): there the two
// loops of persistent_trace cross. 100,000 / 150,000 incoherent rays, second
// loop alone against both: 556 / 671 us and 600 / 628 on the sphere scene, 276
// / 332 and 281 / 292 on the 1M soup, 62 / 72 and 63 / 67 on Cornell.
uint32_t FewRays(uint32_t warps) { return 24u * warps; }

// ---- work sources -----------------------------------------------------------
// One scene, one ray array, one query kind for the whole launch.
struct SingleSource {
    static constexpr bool kCounted = false;
    DeviceScene scene;
    const float4* rays;
    void* hits;
    uint8_t* occluded;
    const uint32_t* order;  // fetch position -> ray index (coherence order), or null
    uint32_t n;
    struct Lane {};
    __device__ __forceinline__ uint32_t map(uint32_t pos) const { return order ? __ldg(order + pos) : pos; }
    __device__ __forceinline__ void load(uint32_t id, float4& r0, float4& r1, Lane&) const {
        r0 = __ldcs(rays + 2 * (size_t)id);
        r1 = __ldcs(rays + 2 * (size_t)id + 1);
    }
    __device__ __forceinline__ const DeviceScene& scene_of(const Lane&) const { return scene; }
    __device__ __forceinline__ bool any_of(const Lane&, bool dflt) const { return dflt; }
    __device__ __forceinline__ void store(uint32_t id, const Lane&, bool any, uint32_t prim, float t) const {
        if (any) {
            __stcs(occluded + id, (uint8_t)(prim != FND_INVALID_ID ? 1 : 0));
        } else {
            const uint2 o = make_uint2(prim, prim == FND_INVALID_ID ? 0x7F800000u : __float_as_uint(t));
            __stcs(reinterpret_cast<uint2*>(hits) + id, o);
        }
    }
};

// A job table; a global ray id is mapped to its job by binary search over
// the prefix of ray counts (kept in shared memory when it fits).
struct BatchSource {
    static constexpr bool kCounted = false;
    const BatchJob* jobs;
    const uint32_t* prefix;  // njobs + 1 entries
    uint32_t njobs;
    uint32_t n;
    struct Lane {
        uint32_t job;
        uint32_t local;
        DeviceScene scene;
        bool any;
    };
    __device__ __forceinline__ uint32_t map(uint32_t pos) const { return pos; }
    __device__ __forceinline__ void load(uint32_t id, float4& r0, float4& r1, Lane& ln) const {
        uint32_t lo = 0, hi = njobs;  // prefix[lo] <= id < prefix[hi]
        while (hi - lo > 1) {
            const uint32_t mid = (lo + hi) >> 1;
            if (prefix[mid] <= id)
                lo = mid;
            else
                hi = mid;
        }
        ln.job = lo;
        ln.local = id - prefix[lo];
        const BatchJob& j = jobs[lo];
        ln.scene = j.scene;
        ln.any = j.any != 0;
        r0 = __ldcs(j.rays + 2 * (size_t)ln.local);
        r1 = __ldcs(j.rays + 2 * (size_t)ln.local + 1);
    }
    __device__ __forceinline__ const DeviceScene& scene_of(const Lane& ln) const { return ln.scene; }
    __device__ __forceinline__ bool any_of(const Lane& ln, bool) const { return ln.any; }
    __device__ __forceinline__ void store(uint32_t, const Lane& ln, bool any, uint32_t prim, float t) const {
        const BatchJob& j = jobs[ln.job];
        if (any) {
            __stcs(static_cast<uint8_t*>(j.out) + ln.local, (uint8_t)(prim != FND_INVALID_ID ? 1 : 0));
        } else {
            const uint2 o = make_uint2(prim, prim == FND_INVALID_ID ? 0x7F800000u : __float_as_uint(t));
            __stcs(reinterpret_cast<uint2*>(j.out) + ln.local, o);
        }
    }
};

// Rays against a two-level scene: the top level's leaves are instances.
struct InstancedSource {
    static constexpr bool kCounted = false;
    DeviceScene scene;  // the top level
    const InstanceRec* inst;
    uint32_t num_inst;
    const float4* rays;
    void* hits;
    uint8_t* occluded;
    uint32_t n;
    struct Lane {};
    __device__ __forceinline__ uint32_t map(uint32_t pos) const { return pos; }
    __device__ __forceinline__ void load(uint32_t id, float4& r0, float4& r1, Lane&) const {
        r0 = __ldg(rays + 2 * (size_t)id);
        r1 = __ldg(rays + 2 * (size_t)id + 1);
    }
    __device__ __forceinline__ const DeviceScene& scene_of(const Lane&) const { return scene; }
    __device__ __forceinline__ bool any_of(const Lane&, bool dflt) const { return dflt; }
    __device__ __forceinline__ void store(uint32_t id, const Lane&, bool any, uint32_t prim, float t) const {
        if (any) {
            __stcs(occluded + id, (uint8_t)(prim != FND_INVALID_ID ? 1 : 0));
        } else {
            const uint2 o = make_uint2(prim, prim == FND_INVALID_ID ? 0x7F800000u : __float_as_uint(t));
            __stcs(reinterpret_cast<uint2*>(hits) + id, o);
        }
    }
};

// A batch of at most few_rays runs the second loop (kFew) only: few lanes of a
// warp take rays (LanesPerWarp), and the others help. A larger one runs the
// first until no rays are left to fetch and lanes have nothing to do, and hands
// what is left to the second. Helping: a lane without work takes the top of
// another's stack, so a ray is followed by several lanes that share its slot;
// every step tests all its triangles, so the ring is empty whenever a lane
// changes rays.
template <class Src, int kKind, bool kStats, int kShort, bool kTwoLevel = false, bool kMulti = false,
          bool kPlanes = false>
__device__ __forceinline__ void persistent_trace(const Src& src, const Common& C, uint32_t w, uint32_t tab,
                                                 float4* s_world = nullptr) {
    uint2 l_stack[kMaxStack - kShort];
    LaneState st{};
    typename Src::Lane ln{};
    if (src.n > C.few_rays)
        trace_loop<Src, kKind, kStats, kShort, kTwoLevel, kMulti, kPlanes, false>(src, C, w, tab, s_world, st, ln, l_stack);
    if (kHelps<kTwoLevel, kPlanes> || src.n <= C.few_rays)
        help_loop<Src, kKind, kStats, kShort, kTwoLevel, kMulti, kPlanes>(src, C, w, tab, s_world, st, ln, l_stack);
}

// 32 resident warps per SM (64 registers a thread).
constexpr int MinBlocks(int block) { return 1024 / block; }

// Few rays: no more blocks than have rays to take, if those take all of them at
// once (grid is then set).
bool SmallGrid(uint32_t n, int block, uint32_t full_warps, int& grid) {
    const uint64_t per_block = (uint64_t)LanesPerWarp(n, full_warps) * ((uint32_t)block / 32u);
    const uint64_t need = ((uint64_t)n + per_block - 1) / per_block;
    if (need > (uint64_t)grid) return false;
    grid = (int)need;
    return true;
}

// Clears the fetch counter, unless it is clear already, or drops it where every
// warp takes its one run of rays: a launch and a trip to L2 less (1,000 / 10,000
// incoherent Cornell rays 25.8 / 36.0 us with it, 23.0 / 33.0 without; on the
// sphere scene 65.7 / 122.4 and 62.5 / 117.2).
cudaError_t ReadyCounter(bool small, bool ready, uint32_t*& counter, cudaStream_t stream) {
    if (small) counter = nullptr;
    return small || ready ? cudaSuccess : cudaMemsetAsync(counter, 0, sizeof(uint32_t), stream);
}

template <bool kAny, bool kStats, int kShort, int kBlock, bool kPlanes = false>
__global__ void __launch_bounds__(kBlock, MinBlocks(kBlock)) trace_kernel(const TraceLaunch L) {
    using W = WarpShared<kShort, false>;
    __shared__ __align__(16) uint8_t s_mem[kTableBytes + W::kBytes * (kBlock / 32)];
    SingleSource src;
    src.scene = L.scene;
    src.rays = L.rays;
    src.hits = L.hits;
    src.occluded = L.occluded;
    src.order = L.order;
    src.n = L.n_dev ? min(*L.n_dev, L.n) : L.n;
    if (src.n == 0) return;  // an empty queue of the path tracer
    if (L.ray_total && blockIdx.x == 0 && threadIdx.x == 0) atomicAdd(L.ray_total, (unsigned long long)src.n);
    fill_tables(s_mem);
    const Common C{L.counter, L.status, L.stats, L.refill_min, L.few_rays, L.full_warps, L.postpone_min ? L.postpone_min : kWaitMin};
    persistent_trace<SingleSource, kAny ? 1 : 0, kStats, kShort, false, false, kPlanes>(
        src, C, shared_addr(s_mem + kTableBytes + W::kBytes * (threadIdx.x >> 5)), shared_addr(s_mem));
}

template <int kShort, int kBlock>
__global__ void __launch_bounds__(kBlock, MinBlocks(kBlock)) batch_kernel(const BatchLaunch B) {
    using W = WarpShared<kShort, true>;
    __shared__ __align__(16) uint8_t s_mem[kTableBytes + W::kBytes * (kBlock / 32)];
    fill_tables(s_mem);
    BatchSource src;
    src.jobs = B.jobs;
    src.prefix = B.prefix;
    src.njobs = B.njobs;
    src.n = B.total;
    const Common C{B.counter, B.status, nullptr, B.refill_min, B.few_rays, B.full_warps, B.postpone_min ? B.postpone_min : kWaitMin};
    persistent_trace<BatchSource, 2, false, kShort, false, true>(
        src, C, shared_addr(s_mem + kTableBytes + W::kBytes * (threadIdx.x >> 5)), shared_addr(s_mem));
}

template <bool kAny>
__global__ void __launch_bounds__(128, 8) instanced_trace_kernel(const InstancedLaunch L) {
    using W = WarpShared<8, true>;
    __shared__ __align__(16) uint8_t s_mem[W::kBytes * 4];
    __shared__ float4 s_world[3 * 128];
    InstancedSource src;
    src.scene = L.tlas;
    src.inst = L.inst;
    src.num_inst = L.num_inst;
    src.rays = L.rays;
    src.hits = L.hits;
    src.occluded = L.occluded;
    src.n = L.n_dev ? min(*L.n_dev, L.n) : L.n;
    if (L.ray_total && blockIdx.x == 0 && threadIdx.x == 0) atomicAdd(L.ray_total, (unsigned long long)src.n);
    const Common C{L.counter, L.status, nullptr, 8u, L.few_rays, L.full_warps, kWaitMin};
    persistent_trace<InstancedSource, kAny ? 1 : 0, false, 8, true, true>(
        src, C, shared_addr(s_mem + W::kBytes * (threadIdx.x >> 5)), 0u, s_world);
}

__global__ void fill_miss_kernel(uint2* hits, uint8_t* occluded, uint32_t cap, const uint32_t* n_dev) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t n = n_dev ? min(*n_dev, cap) : cap;
    if (i >= n) return;
    if (hits) hits[i] = make_uint2(FND_INVALID_ID, 0x7F800000u);
    if (occluded) occluded[i] = 0;
}

// ---- variant tables ---------------------------------------------------------
template <bool kAny, bool kStats, int kShort, int kBlock>
const void* trace_ptr() {
    return reinterpret_cast<const void*>(&trace_kernel<kAny, kStats, kShort, kBlock>);
}

int block_index(int block) { return block == 64 ? 0 : (block == 256 ? 2 : 1); }
int short_index(int s) { return s == 4 ? 0 : (s == 16 ? 2 : 1); }

template <bool kAny>
const void* select_trace(const TraceConfig& c, bool stats) {
    if (stats) return kAny ? trace_ptr<true, true, 8, 128>() : trace_ptr<false, true, 8, 128>();
    static const void* table[3][3] = {
        {trace_ptr<kAny, false, 4, 64>(), trace_ptr<kAny, false, 8, 64>(), trace_ptr<kAny, false, 16, 64>()},
        {trace_ptr<kAny, false, 4, 128>(), trace_ptr<kAny, false, 8, 128>(), trace_ptr<kAny, false, 16, 128>()},
        {trace_ptr<kAny, false, 4, 256>(), trace_ptr<kAny, false, 8, 256>(), trace_ptr<kAny, false, 16, 256>()},
    };
    return table[block_index(c.block)][short_index(c.short_stack)];
}

const void* select_batch(const TraceConfig& c) {
    static const void* table[3][3] = {
        {(const void*)&batch_kernel<4, 64>, (const void*)&batch_kernel<8, 64>, (const void*)&batch_kernel<16, 64>},
        {(const void*)&batch_kernel<4, 128>, (const void*)&batch_kernel<8, 128>, (const void*)&batch_kernel<16, 128>},
        {(const void*)&batch_kernel<4, 256>, (const void*)&batch_kernel<8, 256>, (const void*)&batch_kernel<16, 256>},
    };
    return table[block_index(c.block)][short_index(c.short_stack)];
}

int normalized_block(int b) { return b == 64 || b == 256 ? b : 128; }

}  // namespace

bool ValidTraceConfig(const TraceConfig& c) {
    return (c.block == 64 || c.block == 128 || c.block == 256) &&
           (c.short_stack == 4 || c.short_stack == 8 || c.short_stack == 16) && c.refill_min >= 1 &&
           c.refill_min <= 32 && c.postpone_min <= 32 && c.blocks_per_sm >= 0 && c.blocks_per_sm <= 32 &&
           ValidSortBits(c.sort_bits);
}

cudaError_t TraceOccupancy(int variant, int* blocks_per_sm) {
    TraceConfig c{};
    return TraceOccupancyFor(c, variant, blocks_per_sm);
}

cudaError_t TraceOccupancyFor(const TraceConfig& c, int variant, int* blocks_per_sm) {
    const bool any = variant == 1 || variant == 3, stats = variant >= 2;
    const void* fn = variant == 4 ? select_batch(c) : (any ? select_trace<true>(c, stats) : select_trace<false>(c, stats));
    const int block = stats ? 128 : normalized_block(c.block);
    return cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks_per_sm, fn, block, 0);
}

cudaError_t LaunchTraceConfigured(const TraceLaunch& L, bool any, bool stats, const TraceConfig& c, int grid,
                                  cudaStream_t stream) {
    if (L.n == 0) return cudaSuccess;
    if (L.scene.num_nodes == 0) {
        const uint32_t threads = 256;
        fill_miss_kernel<<<(L.n + threads - 1) / threads, threads, 0, stream>>>(
            any ? nullptr : reinterpret_cast<uint2*>(L.hits), any ? L.occluded : nullptr, L.n, L.n_dev);
        return cudaGetLastError();
    }
    const void* fn = any ? select_trace<true>(c, stats) : select_trace<false>(c, stats);
    int block = stats ? 128 : normalized_block(c.block);
    if (L.scene.tri_stride == 1) {  // triangle planes: the default shape
        fn = any ? reinterpret_cast<const void*>(&trace_kernel<true, false, 8, 128, true>)
                 : reinterpret_cast<const void*>(&trace_kernel<false, false, 8, 128, true>);
        block = 128;
    }
    TraceLaunch arg = L;
    arg.refill_min = c.refill_min ? c.refill_min : L.refill_min;
    arg.postpone_min = c.postpone_min;
    arg.full_warps = (uint32_t)(grid * (block / 32));
    arg.few_rays = L.scene.tri_stride == 1 ? 0u : FewRays(arg.full_warps);
    const bool small = !L.n_dev && L.n <= arg.few_rays && SmallGrid(L.n, block, arg.full_warps, grid);
    if (const cudaError_t e = ReadyCounter(small, L.counter_ready, arg.counter, stream)) return e;
    void* params[] = {&arg};
    return cudaLaunchKernel(fn, dim3(grid), dim3(block), params, 0, stream);
}

cudaError_t LaunchTrace(const TraceLaunch& L, bool any, bool stats, int grid, cudaStream_t stream) {
    TraceConfig c{};
    c.refill_min = L.refill_min;
    return LaunchTraceConfigured(L, any, stats, c, grid, stream);
}

cudaError_t LaunchInstanced(const InstancedLaunch& L, bool any, int sm_count, cudaStream_t stream) {
    if (L.n == 0) return cudaSuccess;
    const void* fn = any ? reinterpret_cast<const void*>(&instanced_trace_kernel<true>)
                         : reinterpret_cast<const void*>(&instanced_trace_kernel<false>);
    int blocks = 0;
    cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks, fn, 128, 0);
    if (e != cudaSuccess) return e;
    InstancedLaunch arg = L;
    int grid = sm_count * (blocks > 0 ? blocks : 1);
    arg.full_warps = (uint32_t)(4 * grid);
    arg.few_rays = FewRays(arg.full_warps);
    const bool small = !L.n_dev && L.n <= arg.few_rays && SmallGrid(L.n, 128, arg.full_warps, grid);
    e = ReadyCounter(small, L.counter_ready, arg.counter, stream);
    if (e != cudaSuccess) return e;
    void* params[] = {&arg};
    return cudaLaunchKernel(fn, dim3(grid), dim3(128), params, 0, stream);
}

cudaError_t LaunchBatch(const BatchLaunch& B, const TraceConfig& c, int grid, cudaStream_t stream) {
    if (B.total == 0) return cudaSuccess;
    BatchLaunch arg = B;
    arg.refill_min = c.refill_min ? c.refill_min : B.refill_min;
    arg.postpone_min = c.postpone_min;
    const int block = normalized_block(c.block);
    arg.full_warps = (uint32_t)(grid * (block / 32));
    arg.few_rays = FewRays(arg.full_warps);
    const bool small = B.total <= arg.few_rays && SmallGrid(B.total, block, arg.full_warps, grid);
    if (const cudaError_t e = ReadyCounter(small, false, arg.counter, stream)) return e;
    void* params[] = {&arg};
    return cudaLaunchKernel(select_batch(c), dim3(grid), dim3(block), params, 0, stream);
}

}  // namespace RT
}  // namespace Foundation
