// warp_trace.cuh — the traversal loop of a warp: node steps with one ray per
// lane, triangle tests shared by the warp (sm_103a). Included by the ray batch
// kernels (traverse.cu) and by the path kernels (pt/).
#pragma once

#include <cfloat>

#include "../../../include/fnd_rt.h"
#include "traverse.cuh"

namespace Foundation {
namespace RT {

namespace {

constexpr uint32_t kFull = 0xFFFFFFFFu;
constexpr uint32_t kTriGroupFlag = 0x80000000u;
// Lanes that only wait for their triangles before a part-filled round runs. Any
// value from 2 to 16 is within 1% on incoherent and camera rays; 1 costs 1%.
constexpr uint32_t kWaitMin = 4;
// With no rays left to fetch, a warp turns to helping once at most this many of
// its lanes have work (8.4M / 1M rays on Cornell: 0 (never) 1.70 ms / 263 us,
// 16 1.66 / 237, 28 1.65 / 237).
constexpr uint32_t kHelpAt = 28;

struct Common {
    uint32_t* counter;  // null (few rays, a source that is not kCounted): every warp takes its one run of them
    uint32_t* status;
    unsigned long long* stats;
    uint32_t refill_min;
    uint32_t few_rays, full_warps;  // (see persistent_trace)
    uint32_t wait_min;  // flush the ring once this many lanes only wait for their pairs
};

// Lanes of a warp that take rays, for n rays on a grid of `warps` warps. The
// time of a small batch is the latency of its longest rays, and a warp's
// triangle rounds serve all its rays in turn, so a batch finishes sooner on
// few lanes of many warps, where the others help (persistent_trace). Twice the
// lanes that an even spread asks for, so that warps with short rays fetch more.
// us per pass, 32 lanes without helping / this rule: 1,000 incoherent rays on
// the sphere scene 368 / 65, on the 1M soup 167 / 59; 10,000 398 / 111 and 204
// / 82; 30,000 372 / 239 and 200 / 154. Factors 8, 4, 2 and 1 in place of two:
// 10,000 rays 234, 154, 111, 99 on the spheres, 121, 98, 82, 80 on the soup;
// 30,000 on Cornell 46, 41, 39, 46. Not below two lanes: short rays gain from a
// neighbour's warm cache (300 segments on Cornell 37 us, 40 with one lane).
__host__ __device__ __forceinline__ uint32_t LanesPerWarp(uint32_t n, uint32_t warps) {
    const uint64_t l = (2ull * n + warps - 1) / (warps ? warps : 1u);
    return l >= 32 ? 32u : l < 2 ? 2u : (uint32_t)l;
}
constexpr uint32_t kInstanceMarker = 0xFFFFFFFFu;  // stack entry: return to the top level

// ---- shared memory by 32-bit address ------------------------------------------
// One address per warp region, kept in a register: through generic pointers
// the compiler forms the shared window's base anew at nearly every access.
__device__ __forceinline__ uint32_t shared_addr(const void* p) {
    uint32_t a = (uint32_t)__cvta_generic_to_shared(p), r;
    asm volatile("mov.u32 %0, %1;" : "=r"(r) : "r"(a));
    return r;
}
__device__ __forceinline__ uint32_t lds8(uint32_t a) {
    uint32_t v;
    asm volatile("ld.shared.u8 %0, [%1];" : "=r"(v) : "r"(a) : "memory");
    return v;
}
__device__ __forceinline__ uint32_t lds32(uint32_t a) {
    uint32_t v;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(a) : "memory");
    return v;
}
__device__ __forceinline__ uint2 lds64(uint32_t a) {
    uint2 v;
    asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(a) : "memory");
    return v;
}
__device__ __forceinline__ float4 lds128(uint32_t a) {
    float4 v;
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
                 : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
                 : "r"(a)
                 : "memory");
    return v;
}
__device__ __forceinline__ void sts32(uint32_t a, uint32_t v) {
    asm volatile("st.shared.u32 [%0], %1;" ::"r"(a), "r"(v) : "memory");
}
__device__ __forceinline__ void sts64(uint32_t a, uint32_t x, uint32_t y) {
    asm volatile("st.shared.v2.u32 [%0], {%1, %2};" ::"r"(a), "r"(x), "r"(y) : "memory");
}
__device__ __forceinline__ void sts128(uint32_t a, float x, float y, float z, float w) {
    asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(a), "f"(x), "f"(y), "f"(z), "f"(w) : "memory");
}

// Inclusive prefix sum over the warp. The shuffle's own in-range predicate
// takes the place of a lane compare per step.
__device__ __forceinline__ uint32_t warp_inclusive_sum(uint32_t v) {
#pragma unroll
    for (int o = 1; o < 32; o <<= 1)
        asm volatile(
            "{\n\t.reg .u32 t;\n\t.reg .pred p;\n\t"
            "shfl.sync.up.b32 t|p, %0, %1, 0, 0xFFFFFFFF;\n\t"
            "@p add.u32 %0, %0, t;\n\t}"
            : "+r"(v)
            : "r"(o));
    return v;
}

// ---- the warp's queue of triangle tests ---------------------------------------
// After a node step each lane holds the hit leaf slots of its node; lane by
// lane they are uneven (most lanes have none, a few have several). The lanes
// append one range (the node's first triangle, the slot's meta byte, the
// owner lane) per hit leaf to a ring of the warp in shared memory, and the
// warp tests the ranges' triangles 32 at a time, one per lane, whatever lanes
// and node steps they came from: an owner's traversal goes on while its
// ranges wait, against the best t known so far, so every round but a flush is
// nearly full. The ray constants come from the owner's slot, written when the
// ray was fetched, and a hit is merged into the owner's best (smaller t, on
// equal t the lower id). The result does not depend on the order of the
// tests: a triangle tested late can only have been worth a few node visits
// more. A ray is finished once its traversal is and the ring has passed its
// last range.
constexpr uint32_t kRing = 64;  // ranges

// Shared memory of one warp (byte offsets): per lane the ray's constants
// (origin and tmin; -Sx, -Sy, Sz and kz; inverse direction and octx), its
// best hit (t bits, id) and the merge slot, then the ring, with kMulti (lanes
// of one warp in different scenes) the triangle records of each lane's scene
// and its hit-id offset, and the lanes' stacks. The origin and the inverse
// direction are read back for each node: they are dead before the node
// test's widest point, where registers are scarce.
template <int kShort, bool kMulti>
struct WarpShared {
    static constexpr uint32_t kRayA = 0, kRayB = 512, kRayC = 1024, kBest = 1536, kWin = 1792, kRanges = 2048;
    static constexpr uint32_t kTris = kRanges + 8 * kRing, kPrimOff = kTris + (kMulti ? 256 : 0);
    static constexpr uint32_t kStack = kPrimOff + (kMulti ? 128 : 0), kBytes = kStack + 256 * kShort;
};

// Group bit <-> slot (see persistent_trace).
__device__ __forceinline__ uint32_t octx_of(const RayState& r) { return (r.oct ^ 7u) | 24u; }

template <int kShort, bool kMulti>
__device__ __forceinline__ void store_ray(uint32_t w, uint32_t lane, const RayState& r) {
    using W = WarpShared<kShort, kMulti>;
    sts128(w + 16u * lane + W::kRayA, r.ox, r.oy, r.oz, r.tmin);
    sts128(w + 16u * lane + W::kRayB, r.nSx, r.nSy, r.Sz, __int_as_float(r.kz));
    sts128(w + 16u * lane + W::kRayC, r.ix, r.iy, r.iz, __uint_as_float(octx_of(r)));
}
// kMulti: the lane's triangle records and hit-id offset.
template <int kShort>
__device__ __forceinline__ void store_scene(uint32_t w, uint32_t lane, const DeviceScene& sc, uint32_t prim_off) {
    using W = WarpShared<kShort, true>;
    const unsigned long long v = (unsigned long long)sc.v0;
    sts64(w + 8u * lane + W::kTris, (uint32_t)v, (uint32_t)(v >> 32));
    sts32(w + 4u * lane + W::kPrimOff, prim_off);
}
__device__ __forceinline__ const float4* lds_ptr(uint32_t a) {
    const uint2 v = lds64(a);
    return (const float4*)((unsigned long long)v.y << 32 | v.x);
}

// ---- the persistent traversal loop ----------------------------------------
// kKind: 0 closest, 1 any, 2 per-lane (from the source). kTwoLevel: the
// source is an InstancedSource (triangle leaves of the top level are
// instances; per-lane node / triangle arrays). w: this warp's region of
// shared memory, tab: the tables of fill_tables. kPlanes: the scene's
// triangles are three planes (tri_stride 1), not records.
//
// A node group is one word: the internal children still to visit in bits
// 24..31, the highest bit first (bit 24 + j is slot j ^ 7 ^ oct, so the
// highest bit is the nearest along the ray's octant), and the node's imask
// in bits 0..7.
// What the first loop hands to the second: a lane's traversal and its ray, and
// whether rays are left. (The ring is empty there.)
struct LaneState {
    uint32_t ray_id, ng_base, ng_group;
    float best_t;
    int sp;
    bool active, exhausted;
};

// Helping is not for two-level scenes (a lane's slot changes with its
// instance), nor for scenes made by hand, whose depth no upload has checked:
// sharing a stack would hide that it is too deep.
template <bool kTwoLevel, bool kPlanes>
constexpr bool kHelps = !kTwoLevel && !kPlanes;

// One of the two loops of persistent_trace (kFew: the second). l_stack: the
// lane's entries past the shared ones.
template <class Src, int kKind, bool kStats, int kShort, bool kTwoLevel, bool kMulti, bool kPlanes, bool kFew>
__device__ __forceinline__ void trace_loop(const Src& src, const Common& C, uint32_t w, uint32_t tab, float4* s_world,
                                           LaneState& st, typename Src::Lane& lane_src, uint2* l_stack) {
    using W = WarpShared<kShort, kMulti>;
    // two-level: each lane's triangles and hit-id offset come from its own slot
    // (the lanes of a warp sit in different instances)
    static_assert(!kTwoLevel || kMulti, "two-level traversal needs per-lane scenes");
    uint32_t lane, below;
    asm volatile("mov.u32 %0, %%laneid;" : "=r"(lane));
    asm volatile("mov.u32 %0, %%lanemask_lt;" : "=r"(below));
    const uint32_t wl = w + 8u * lane;  // the lane's 8-byte slots
    const uint32_t n = src.n;

    uint32_t slot = lane;  // kSteal: the lane whose ray this one follows
    typename Src::Lane ln = lane_src;
    bool active = st.active, exhausted = st.exhausted, any_hit = kKind == 1 || (kKind == 2 && st.active && src.any_of(ln, false));
    uint32_t ray_id = st.ray_id;
    float best_t = st.best_t, tmin = 0.0f;  // best_t: the culling bound (the hit itself is in shared memory)
    uint32_t ng_base = st.ng_base, ng_group = st.ng_group;
    int sp = st.sp;
    // the warp's ring: ranges head .. tail - 1 (modulo 2^32), with `tris` triangles written
    uint32_t head = 0, tail = 0, tris = 0;
    uint32_t my_end = 0;  // the ring position after this lane's last range
    unsigned long long st_nodes = 0, st_tris = 0;
    uint32_t st_wnode = 0, st_wtri = 0;  // warp steps, counted by the lowest active lane
    // two-level state: the arrays the lane traverses now, its instance, and
    // the instances of a top-level leaf still to enter
    bool in_blas = false, moved = false;  // moved: the lane's ray is an object-space one, the world one is in s_world
    DeviceScene cur{};
    uint32_t tl_base = 0, tl_mask = 0;

    // the first kShort entries in shared memory, deeper ones in local memory
    auto push = [&](uint32_t x, uint32_t y) -> bool {
        if (sp < kShort)
            sts64(wl + W::kStack + 256u * (uint32_t)sp, x, y);
        else if (sp < kMaxStack)
            l_stack[sp - kShort] = make_uint2(x, y);
        else
            return false;
        sp++;
        return true;
    };
    // the root as a pseudo group: one internal child in slot 0
    auto start = [&](uint32_t num_nodes, uint32_t octx) {
        ng_base = 0;
        ng_group = num_nodes ? (1u << octx) | 1u : 0u;  // (an empty scene: a miss)
    };
    // two-level: descend into instance I (from the top level). Its
    // object-space ray replaces the lane's ray, and the world ray's constants
    // wait in s_world for the return; an identity instance keeps them.
    auto enter_instance = [&](const InstanceRec& I) {
        if constexpr (kTwoLevel) {
            cur = I.blas;
            in_blas = true;
            moved = !(__ldg(&I.flags) & kInstanceIdentity);
            if (moved) {
                for (int q = 0; q < 3; ++q) s_world[3 * threadIdx.x + q] = lds128(wl + 8u * lane + W::kRayA + 512u * q);
                float inv[12];
                for (int q = 0; q < 12; ++q) inv[q] = __ldg(I.inv + q);
                float4 r0, r1, o0, o1;
                src.load(ray_id, r0, r1, ln);
                instance_ray(inv, r0, r1, o0, o1);
                store_ray<kShort, kMulti>(w, lane, setup_ray(o0, o1));
            }
            store_scene<kShort>(w, lane, cur, __ldg(&I.prim_offset));
            start(cur.num_nodes, lds32(wl + 8u * lane + W::kRayC + 12u));
        }
    };
    const uint32_t lanes = kFew && n <= C.few_rays ? LanesPerWarp(n, C.full_warps) : 32u;
    constexpr bool kHelp = kHelps<kTwoLevel, kPlanes>;
    constexpr bool kSteal = kFew && kHelp;
    // kSteal in a batch: the followed ray's scene (cur) and kind
    constexpr bool kOwnScene = kSteal && kMulti, kOwnKind = kSteal && kKind == 2;
    bool follows_any = any_hit;
    if constexpr (kOwnScene) cur = src.scene_of(ln);
    for (;;) {
        // ---- finished rays out, new rays in ----------------------------------
        // ready: lanes without a ray, or with one whose traversal and ranges
        // are done. A warp turns to them once there are refill_min (or, when
        // no rays are left, all).
        const bool work = ng_group >= (1u << 24) && (!kTwoLevel || tl_mask == 0u);
        const uint32_t working = __ballot_sync(kFull, work);
        const uint32_t holders = kFew ? kFull >> (32u - lanes) : kFull;
        // kSteal (the ring is empty here): a ray is done when no lane follows it
        const uint32_t followed = kSteal ? __reduce_or_sync(kFull, work ? 1u << slot : 0u) : 0u;
        const bool done = !work && (kSteal ? !(followed >> lane & 1u)
                                           : (!kTwoLevel || tl_mask == 0u) && (int)(my_end - head) <= 0);
        const uint32_t ready = __ballot_sync(kFull, done) & holders;
        if (ready == holders || (!exhausted && (uint32_t)__popc(ready) >= (kFew ? min(C.refill_min, lanes) : C.refill_min))) {
            const bool mine = done && (!kFew || lane < lanes);
            if (mine && active) {
                const uint2 bst = lds64(wl + W::kBest);
                src.store(ray_id, ln, any_hit, bst.y, __uint_as_float(bst.x));
                active = false;
            }
            if (exhausted) break;
            const uint32_t cnt = (uint32_t)__popc(ready);
            uint32_t base = 0;
            if (kFew && !Src::kCounted && !C.counter) {
                base = (blockIdx.x * blockDim.x + threadIdx.x) / 32u * lanes;
                exhausted = true;
            } else {
                if (lane == 0) base = atomicAdd(C.counter, cnt);
                base = __shfl_sync(kFull, base, 0);
                exhausted = base + cnt >= n;
            }
            const uint32_t pos = base + (uint32_t)__popc(ready & below);
            if (mine && pos < n) {
                const uint32_t id = src.map(pos);
                float4 r0, r1;
                src.load(id, r0, r1, ln);
                if (kKind == 2) any_hit = src.any_of(ln, false);
                const RayState r = setup_ray(r0, r1);
                store_ray<kShort, kMulti>(w, lane, r);
                if constexpr (kMulti) store_scene<kShort>(w, lane, src.scene_of(ln), 0u);
                tmin = r.tmin;
                ray_id = id;
                slot = lane;
                if constexpr (kOwnScene) cur = src.scene_of(ln);
                if constexpr (kOwnKind) follows_any = any_hit;
                best_t = r.tmax;
                sts64(wl + W::kBest, __float_as_uint(r.tmax), FND_INVALID_ID);
                start(src.scene_of(ln).num_nodes, octx_of(r));
                active = true;
                if constexpr (kTwoLevel) {
                    in_blas = false;
                    moved = false;
                    cur = src.scene;
                }
            }
            my_end = mine ? head : my_end;
            continue;
        }

        if constexpr (kSteal) {
            // the k-th lane without work takes the top of the k-th stack
            const uint32_t from = __ballot_sync(kFull, sp > 0 && sp <= kShort);
            const uint32_t idle = ~working;
            if (from && idle) {
                const uint32_t rank = (uint32_t)__popc(from & below);
                const bool gives = (from >> lane & 1u) && rank < (uint32_t)__popc(idle);
                if (gives) {
                    sp--;
                    sts32(w + 8u * rank + W::kWin, lane);
                }
                __syncwarp();
                const uint32_t k = (uint32_t)__popc(idle & below);
                const bool takes = !work && k < (uint32_t)__popc(from);
                const uint32_t victim = takes ? lds32(w + 8u * k + W::kWin) : lane;
                const uint32_t top = __shfl_sync(kFull, (uint32_t)sp, victim);
                const uint32_t whose = __shfl_sync(kFull, slot, victim);
                if constexpr (kOwnScene) {  // (lanes that take nothing read their own)
                    cur.nodes = (const uint4*)__shfl_sync(kFull, (unsigned long long)cur.nodes, victim);
                    cur.num_nodes = __shfl_sync(kFull, cur.num_nodes, victim);
                    cur.num_tris = __shfl_sync(kFull, cur.num_tris, victim);
                }
                if constexpr (kOwnKind) follows_any = __shfl_sync(kFull, follows_any ? 1 : 0, victim) != 0;
                if (takes) {
                    const uint2 e = lds64(w + 8u * victim + W::kStack + 256u * top);
                    ng_base = e.x;
                    ng_group = e.y;
                    slot = whose;
                    best_t = bound_of(__uint_as_float(lds32(w + 8u * slot + W::kBest)));
                }
                __syncwarp();
            }
        }
        const uint32_t ws = kSteal ? w + 8u * slot : wl;  // the slots of the followed ray
        // ---- one node --------------------------------------------------------
        uint32_t leaves = 0, tri_base = 0, meta0 = 0, meta1 = 0;
        if (kSteal ? ng_group >= (1u << 24) : work) {
            const DeviceScene& sc = kTwoLevel || kOwnScene ? cur : src.scene_of(ln);
            const uint32_t wr = kSteal ? w + 16u * slot : wl + 8u * lane;
            const float4 ra = lds128(wr + W::kRayA), rc = lds128(wr + W::kRayC);
            const uint32_t octx = __float_as_uint(rc.w);
            const uint32_t b = 31u - (uint32_t)__clz(ng_group);
            ng_group &= ~(1u << b);
            const uint32_t child = ng_base + (uint32_t)__popc(ng_group & ~(kFull << (b ^ octx)));
            uint32_t fail = 0;
            if (ng_group >= (1u << 24) && !push(ng_base, ng_group)) fail = kStatusStackOverflow;
            if (child >= sc.num_nodes) fail |= kStatusBadIndex;
            if (!fail) {
                RayState r;
                r.ox = ra.x;
                r.oy = ra.y;
                r.oz = ra.z;
                r.tmin = kSteal ? ra.w : tmin;
                r.ix = rc.x;
                r.iy = rc.y;
                r.iz = rc.z;
                const SlotHits h = intersect_slots(r, sc.nodes, child, best_t);
                if (kStats) {
                    st_nodes++;
                    if (lane == (uint32_t)__ffs(__activemask()) - 1u) st_wnode++;
                }
                const uint32_t inner = h.hitm & h.imask;
                const uint32_t order = kTwoLevel ? xor_permute8(inner, octx & 7u) : lds8(tab + ((octx & 7u) << 8) + inner);
                ng_base = h.child_base;
                ng_group = order << 24 | h.imask;
                leaves = h.hitm & leaf_slots(h);
                tri_base = h.tri_base;
                meta0 = h.meta[0];
                meta1 = h.meta[1];
                // a node's triangles (at most 4 from offset 31 on) must lie
                // inside the triangle arrays; only near their end each range
                // is looked at
                if (leaves && (sc.num_tris < 35u || tri_base > sc.num_tris - 35u)) {
                    for (uint32_t q = leaves; q; q &= q - 1u) {
                        const uint32_t m = meta_of(h, (uint32_t)__ffs(q) - 1u);
                        if ((uint64_t)tri_base + (m & 31u) + (m >> 5 & 3u) >= sc.num_tris) fail = kStatusBadIndex;
                    }
                }
            }
            if (fail) {  // the ray ends with the hits found so far
                atomicOr(C.status, fail);
                ng_group = 0;
                leaves = 0;
                sp = 0;
            }
        }
        if constexpr (kTwoLevel) {
            // a top-level leaf holds instances: its slots become one mask
            while (!in_blas && leaves) {
                const uint32_t s = (uint32_t)__ffs(leaves) - 1u;
                leaves &= leaves - 1u;
                const uint32_t m = __byte_perm(s < 4u ? meta0 : meta1, 0u, 0x4440u | (s & 3u));
                tl_base = tri_base;
                tl_mask |= ((2u << (m >> 5 & 3u)) - 1u) << (m & 31u);
            }
            // the lane enters the first valid one and publishes its
            // object-space ray (the ring is empty here: see flush below)
            while (!in_blas && tl_mask) {
                const uint32_t k = (uint32_t)__ffs(tl_mask) - 1u;
                tl_mask &= tl_mask - 1u;
                const uint32_t iid = __float_as_uint(__ldg(cur.v0 + 3 * (size_t)(tl_base + k)).w);
                if (iid >= src.num_inst) {
                    atomicOr(C.status, kStatusBadIndex);
                    continue;
                }
                // resume order after the instance: this leaf's other
                // instances, then the node's other children
                const bool ok = (ng_group < (1u << 24) || push(ng_base, ng_group)) &&
                                (!tl_mask || push(tl_base | kTriGroupFlag, tl_mask)) && push(kInstanceMarker, 0u);
                tl_mask = 0;
                if (!ok) {
                    atomicOr(C.status, kStatusStackOverflow);
                    ng_group = 0;
                    sp = 0;
                    break;
                }
                const InstanceRec& I = src.inst[iid];
                enter_instance(I);
            }
        }
        // ---- its leaves into the ring ------------------------------------------
        // positions by the bits of the lanes' range counts (at most 8 each)
        uint32_t at = 0;
        bool fresh = __ballot_sync(kFull, leaves != 0u) != 0u;
        if (fresh) {
            const uint32_t cnt = (uint32_t)__popc(leaves);
            const uint32_t b0 = __ballot_sync(kFull, cnt & 1u), b1 = __ballot_sync(kFull, cnt & 2u);
            at = tail + (uint32_t)__popc(b0 & below) + 2u * (uint32_t)__popc(b1 & below);
            tail += (uint32_t)__popc(b0) + 2u * (uint32_t)__popc(b1);
            if (__ballot_sync(kFull, cnt > 3u)) {
                const uint32_t b2 = __ballot_sync(kFull, cnt & 4u), b3 = __ballot_sync(kFull, cnt & 8u);
                at += 4u * (uint32_t)__popc(b2 & below) + 8u * (uint32_t)__popc(b3 & below);
                tail += 4u * (uint32_t)__popc(b2) + 8u * (uint32_t)__popc(b3);
            }
            if (cnt) my_end = at + cnt;
        }
        // ---- rounds: whenever 32 triangles wait, and all of them when several
        // lanes only wait for theirs or no lane can go on ---------------------
        // (two-level: after every step, as a lane's slot changes with its instance)
        // (few lanes: likewise, for the latency)
        const bool leave = !kFew && kHelp && exhausted && (uint32_t)__popc(working) <= kHelpAt;
        const bool flush = kTwoLevel || kFew || leave || working == 0u || 32u - (uint32_t)__popc(working | ready) >= C.wait_min;
        for (;;) {
            if (fresh) {
                // ranges [head, head + kRing) are written; more as rounds make room
                uint32_t sum = 0;
                while (leaves && at - head < kRing) {
                    const uint32_t s = 31u - (uint32_t)__clz(leaves);
                    leaves &= ~(1u << s);
                    // (meta byte, owner lane, 0, 0)
                    const uint32_t y = __byte_perm(s < 4u ? meta0 : meta1, kSteal ? slot : lane, 0x5540u | (s & 3u));
                    sum += (y >> 5 & 3u) + 1u;
                    sts64(w + W::kRanges + 8u * (at & (kRing - 1u)), tri_base, y);
                    at++;
                }
                tris += __reduce_add_sync(kFull, sum);
                fresh = tail - head > kRing;
                __syncwarp();
            }
            if (tris < 32u && !fresh && !(flush && tris)) break;
            // the ranges that fit 32 lanes, in ring order: one lane per range
            // finds its first position, then one lane per triangle its range
            const bool have = lane < tail - head;
            const uint2 e = lds64(w + W::kRanges + 8u * ((head + lane) & (kRing - 1u)));
            const uint32_t cnt = have ? (e.y >> 5 & 3u) + 1u : 0u;
            const uint32_t inc = warp_inclusive_sum(cnt);
            const uint32_t starts = __reduce_or_sync(kFull, have && inc <= 32u ? 1u << (inc - cnt) : 0u);
            const uint32_t nr = (uint32_t)__popc(starts);
            const uint32_t np = __shfl_sync(kFull, inc, nr - 1u);
            const uint32_t upto = starts & (below * 2u + 1u);
            const uint32_t from = (uint32_t)__popc(upto) - 1u;
            const uint32_t first = __shfl_sync(kFull, e.x + (e.y & 31u), from);
            const uint32_t own = w + 8u * __shfl_sync(kFull, e.y >> 8, from);
            bool hit = false;
            float t = 0.0f;
            uint32_t pid = 0;
            if (lane < np) {
                const uint32_t ti = first + (lane - (31u - (uint32_t)__clz(upto)));
                const float4 a = lds128(2u * own - w + W::kRayA);
                const float4 b = lds128(2u * own - w + W::kRayB);
                RayState rq;
                rq.ox = a.x;
                rq.oy = a.y;
                rq.oz = a.z;
                rq.tmin = a.w;
                rq.nSx = b.x;
                rq.nSy = b.y;
                rq.Sz = b.z;
                rq.kz = __float_as_int(b.w);
                const DeviceScene& sc = src.scene_of(ln);
                const float4* p0 = kMulti ? lds_ptr(own + W::kTris) : sc.v0;
                p0 += (kPlanes ? 1u : 3u) * (size_t)ti;
                const float4* p1 = kPlanes ? sc.v1 + ti : p0 + 1;
                const float4* p2 = kPlanes ? sc.v2 + ti : p0 + 2;
                const float4 v0 = __ldg(p0);
                hit = intersect_tri(rq, v0, __ldg(p1), __ldg(p2), __uint_as_float(lds32(own + W::kBest)), t);
                pid = __float_as_uint(v0.w);
                if constexpr (kTwoLevel) pid += lds32(w + (own - w) / 2u + W::kPrimOff);  // global id of an instance's triangle
                if (kStats) {
                    st_tris++;
                    if (lane == 0u) st_wtri++;
                }
            }
            head += nr;
            tris -= np;
            if (__ballot_sync(kFull, hit)) {
                // one hit per owner at a time
                do {
                    if (hit) sts32(own + W::kWin, lane);
                    __syncwarp();
                    if (hit && lds32(own + W::kWin) == lane) {
                        const uint2 bst = lds64(own + W::kBest);
                        const float bt = __uint_as_float(bst.x);
                        if (t < bt || (t == bt && pid < bst.y)) sts64(own + W::kBest, __float_as_uint(t), pid);
                        hit = false;
                    }
                    __syncwarp();
                } while (__ballot_sync(kFull, hit));
                const uint2 bst = lds64(ws + W::kBest);
                best_t = bound_of(__uint_as_float(bst.x));
                if ((kKind == 1 || (kKind == 2 && (kOwnKind ? follows_any : any_hit))) && (kSteal || active) && bst.y != FND_INVALID_ID) {
                    ng_group = 0;  // found: only the ranges already in the ring remain
                    sp = 0;
                    if (kTwoLevel) tl_mask = 0;
                }
            }
            __syncwarp();
        }
        // ---- next group ----------------------------------------------------
        if (ng_group < (1u << 24) && sp > 0 && (!kTwoLevel || tl_mask == 0u)) {
            auto pop = [&] {
                sp--;
                return sp < kShort ? lds64(wl + W::kStack + 256u * (uint32_t)sp) : l_stack[sp - kShort];
            };
            uint2 e = pop();
            if constexpr (kTwoLevel) {
                if (e.x == kInstanceMarker) {
                    // back to the top level: the world ray again
                    if (moved)
                        for (int q = 0; q < 3; ++q) {
                            const float4 v = s_world[3 * threadIdx.x + q];
                            sts128(wl + 8u * lane + W::kRayA + 512u * q, v.x, v.y, v.z, v.w);
                        }
                    cur = src.scene;
                    in_blas = false;
                    e = sp > 0 ? pop() : make_uint2(0u, 0u);
                }
                if (e.x & kTriGroupFlag) {  // a top-level leaf's other instances
                    tl_base = e.x & ~kTriGroupFlag;
                    tl_mask = e.y;
                    e.y = 0;
                }
            }
            ng_base = e.x;
            ng_group = e.y;
        }
        if (leave) break;
    }
    if constexpr (kHelp && !kFew) {
        st.ray_id = ray_id;
        st.ng_base = ng_base;
        st.ng_group = ng_group;
        st.best_t = best_t;
        st.sp = sp;
        st.active = active;
        st.exhausted = exhausted;
        lane_src = ln;
    }
    if (kStats) {
        for (int o = 16; o > 0; o >>= 1) {
            st_nodes += __shfl_down_sync(kFull, st_nodes, o);
            st_tris += __shfl_down_sync(kFull, st_tris, o);
            st_wnode += __shfl_down_sync(kFull, st_wnode, o);
            st_wtri += __shfl_down_sync(kFull, st_wtri, o);
        }
        if (lane == 0) {
            atomicAdd(C.stats + 0, st_nodes);
            atomicAdd(C.stats + 1, st_tris);
            atomicAdd(C.stats + 2, (unsigned long long)st_wnode);
            atomicAdd(C.stats + 3, (unsigned long long)st_wtri);
        }
    }
}

// The second loop as a call: its registers are its own, and the first loop is
// compiled as if it were alone (inlined, the pair cost the first loop 3%).
template <class Src, int kKind, bool kStats, int kShort, bool kTwoLevel, bool kMulti, bool kPlanes>
__device__ __noinline__ void help_loop(const Src& src, const Common& C, uint32_t w, uint32_t tab, float4* s_world,
                                       LaneState& st, typename Src::Lane& ln, uint2* l_stack) {
    trace_loop<Src, kKind, kStats, kShort, kTwoLevel, kMulti, kPlanes, true>(src, C, w, tab, s_world, st, ln, l_stack);
}

// Fills the 8 x 256 byte table of xor_permute8 (all threads of the block).
constexpr int kTableBytes = 2048;
__device__ __forceinline__ void fill_tables(uint8_t* t) {
    for (uint32_t i = threadIdx.x; i < 2048u; i += blockDim.x) t[i] = (uint8_t)xor_permute8(i & 255u, i >> 8);
    __syncthreads();
}

}  // namespace

}  // namespace RT
}  // namespace Foundation
