// path_rays.cuh — the rays of a warp's paths, traced together by the warp: the
// path kernels (tail.cu, train_paths.cu) hold one path per lane, and between
// two vertices each lane has up to three rays from one point: the path's next
// segment and the shadow rays to a light and to the sun.
//
// A warp's rays go through the batch kernels' loop in the form that lets lanes
// without work help (rt/warp_trace.cuh): triangle tests fill whole rounds, a
// lane without a ray takes stacked nodes of another's, and the shadow rays of
// one vertex run beside the segment to the next. What bounds these kernels is
// the latency of their longest paths (a few rays per lane in flight on the
// whole chip). One thread per ray with its own stack, the three rays in turn,
// against this: the 65,536 training paths of a frame with their six optimiser
// steps 640 and 500 us (with 200 instances 1,440 and 930), a whole frame of
// 640x360 990 and 790 us (5,020 and 1,820), of 192x108 724 and 560 (2,250 and
// 1,290), of 1920x1080 x 2 4,130 and 4,025 us. 128 registers and 16 warps per
// SM with one level: with 80 and 64 registers the training took 560 and 620 us
// against those 500, and with 168 (12 warps) 464 against 455 since (kCounted).
#pragma once

#include "../rt/warp_trace.cuh"
#include "pt_math.cuh"

namespace Foundation {
namespace PT {

namespace {

constexpr int kPathStack = 8;  // shared stack entries of a lane
// The warp turns to finished rays once this many lanes are done while rays wait
// (1, 4, 16, 32: 640x360 792, 785, 806, 813 us).
constexpr uint32_t kPathRefill = 4;

// Shared memory of one warp (byte offsets): the loop's own, then per lane the
// rays' origin with the light ray's length, the next segment's direction and
// the light ray's, the hit (id, t bits), whether each shadow ray is blocked;
// the list of the warp's rays (kind * 32 + lane), the loop's fetch counter and,
// with two levels, the world rays of lanes inside an instance.
template <bool kTwoLevel>
struct PathShared {
    using W = RT::WarpShared<kPathStack, kTwoLevel>;
    static constexpr uint32_t kOrigin = W::kBytes, kDir = kOrigin + 512, kLight = kDir + 512, kHit = kLight + 512;
    static constexpr uint32_t kBlocked = kHit + 256, kList = kBlocked + 256, kFetch = kList + 96;
    static constexpr uint32_t kWorld = kFetch + 32, kBytes = kWorld + (kTwoLevel ? 1536 : 0);
};

__device__ __forceinline__ void sts8(uint32_t a, uint32_t v) {
    asm volatile("st.shared.u8 [%0], %1;" ::"r"(a), "r"(v) : "memory");
}

// A lane's rays from o: the next segment (d), to the light (ld, up to lt), to the sun.
struct LaneRays {
    bool next, light, sun;
    float3 o, d, ld;
    float lt;
};
struct LaneHits {
    bool hit, light_blocked, sun_blocked;
    uint32_t prim;
    float t;
};

template <bool kTwoLevel>
struct PathSource {
    using P = PathShared<kTwoLevel>;
    static constexpr bool kCounted = true;
    RT::DeviceScene scene;  // two levels: the top one
    const RT::InstanceRec* inst;
    uint32_t num_inst;
    float3 sun;
    uint32_t w;  // the warp's shared memory
    uint32_t n;
    struct Lane {
        bool any;
    };
    __device__ __forceinline__ uint32_t map(uint32_t pos) const { return RT::lds8(w + P::kList + pos); }
    __device__ __forceinline__ void load(uint32_t id, float4& r0, float4& r1, Lane& ln) const {
        const uint32_t kind = id >> 5, at = w + 16u * (id & 31u);
        const float inf = __int_as_float(0x7F800000);
        r0 = RT::lds128(at + P::kOrigin);
        r1 = kind == 2u ? make_float4(sun.x, sun.y, sun.z, inf)
                        : RT::lds128(at + (kind == 0u ? P::kDir : P::kLight));
        r1.w = kind == 1u ? r0.w : inf;
        r0.w = 0.0f;
        ln.any = kind != 0u;
    }
    __device__ __forceinline__ const RT::DeviceScene& scene_of(const Lane&) const { return scene; }
    __device__ __forceinline__ bool any_of(const Lane& ln, bool) const { return ln.any; }
    __device__ __forceinline__ void store(uint32_t id, const Lane&, bool any, uint32_t prim, float t) const {
        if (any)
            RT::sts32(w + P::kBlocked + 4u * (id - 32u), prim != FND_INVALID_ID ? 1u : 0u);
        else
            RT::sts64(w + P::kHit + 8u * id, prim, __float_as_uint(t));
    }
};

// All lanes of the warp call it together; region: the warp's PathShared, tab:
// the block's tables (one level; fill_tables).
template <bool kTwoLevel>
__device__ __forceinline__ void trace_path_rays(const RT::DeviceScene& scene, const RT::InstanceRec* inst,
                                                uint32_t num_inst, uint32_t* status, float3 sun, uint8_t* region,
                                                const uint8_t* tab, const LaneRays& r, LaneHits& h) {
    using P = PathShared<kTwoLevel>;
    const uint32_t lane = threadIdx.x & 31u, below = (1u << lane) - 1u;
    const uint32_t w = RT::shared_addr(region);
    RT::sts128(w + P::kOrigin + 16u * lane, r.o.x, r.o.y, r.o.z, r.lt);
    RT::sts128(w + P::kDir + 16u * lane, r.d.x, r.d.y, r.d.z, 0.0f);
    RT::sts128(w + P::kLight + 16u * lane, r.ld.x, r.ld.y, r.ld.z, 0.0f);
    // the list, the long rays first
    const uint32_t mn = __ballot_sync(RT::kFull, r.next), ml = __ballot_sync(RT::kFull, r.light);
    const uint32_t ms = __ballot_sync(RT::kFull, r.sun);
    const uint32_t nn = (uint32_t)__popc(mn), nl = nn + (uint32_t)__popc(ml);
    if (r.next) sts8(w + P::kList + (uint32_t)__popc(mn & below), lane);
    if (r.light) sts8(w + P::kList + nn + (uint32_t)__popc(ml & below), 32u | lane);
    if (r.sun) sts8(w + P::kList + nl + (uint32_t)__popc(ms & below), 64u | lane);
    if (lane == 0u) RT::sts32(w + P::kFetch, 0u);
    __syncwarp();
    using Src = PathSource<kTwoLevel>;
    Src src;
    src.scene = scene;
    src.inst = inst;
    src.num_inst = num_inst;
    src.sun = sun;
    src.w = w;
    src.n = nl + (uint32_t)__popc(ms);
    const RT::Common C{reinterpret_cast<uint32_t*>(region + P::kFetch), status, nullptr, kPathRefill, 0u, 0u, 1u};
    uint2 l_stack[RT::kMaxStack - kPathStack];
    RT::LaneState st{};
    typename Src::Lane ln{};
    // (the loop indexes the world rays by thread of the block)
    float4* world = kTwoLevel ? reinterpret_cast<float4*>(region + P::kWorld) - 3u * (threadIdx.x - lane) : nullptr;
    RT::help_loop<Src, 2, false, kPathStack, kTwoLevel, kTwoLevel, false>(src, C, w, RT::shared_addr(tab), world, st, ln,
                                                                          l_stack);
    __syncwarp();
    const uint2 hit = RT::lds64(w + P::kHit + 8u * lane);
    h.prim = hit.x;
    h.t = __uint_as_float(hit.y);
    h.hit = hit.x != FND_INVALID_ID;
    h.light_blocked = RT::lds32(w + P::kBlocked + 4u * lane) != 0u;
    h.sun_blocked = RT::lds32(w + P::kBlocked + 128u + 4u * lane) != 0u;
    __syncwarp();
}

// Shared memory of a block of path kernels.
template <bool kTwoLevel, int kBlock>
struct PathBlock {
    static constexpr uint32_t kTables = kTwoLevel ? 0 : RT::kTableBytes;
    static constexpr uint32_t kBytes = kTables + PathShared<kTwoLevel>::kBytes * (kBlock / 32);
    __device__ static __forceinline__ uint8_t* region(uint8_t* mem) {
        return mem + kTables + PathShared<kTwoLevel>::kBytes * (threadIdx.x >> 5);
    }
};

}  // namespace

}  // namespace PT
}  // namespace Foundation
