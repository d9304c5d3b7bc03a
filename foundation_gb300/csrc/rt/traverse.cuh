// traverse.cuh — device-side scene view, ray set-up, watertight triangle test
// and compressed 8-wide node test shared by every traversal kernel
// (closest hit, any hit, the batched multi-scene launch and the integrator's
// extend / shadow stages).
#pragma once

#include <cstdint>
#include <cstring>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include "../../../include/fnd_rt.h"
#include "../bvh/wide_bvh.hpp"
#include "device_scene.hpp"

namespace Foundation {
namespace RT {

// Per-ray state for the node test (origin, sanitised inverse direction,
// direction-sign octant) and for the watertight triangle test (shear
// constants of Woop, Benthin & Wald 2013, dominant axis kz).
struct RayState {
    float ox, oy, oz;
    float ix, iy, iz;
    float nSx, nSy, Sz;  // -Sx, -Sy, Sz
    float tmin, tmax;
    uint32_t oct;
    int kz;
};

__device__ __forceinline__ float sanitize_dir(float d) {
    // keep the sign (also of -0.0); 2^-64 keeps the inverse finite
    return fabsf(d) < 5.421010862427522e-20f ? copysignf(5.421010862427522e-20f, d) : d;
}

// The culling bound of a best t (or a ray's length) for intersect_slots: the
// same value, with +0 for -0. A hit at the origin often has t = -0, and against
// a node's tn = +0 the sign of -0 - (+0) would say that the box is missed, with
// triangles of equal t and lower id in it. (Once per bound, not per node.)
__device__ __forceinline__ float bound_of(float t) { return __fadd_rn(t, 0.0f); }

__device__ __forceinline__ RayState setup_ray(float4 r0, float4 r1) {
    RayState s;
    s.ox = r0.x;
    s.oy = r0.y;
    s.oz = r0.z;
    s.tmin = r0.w;
    s.tmax = bound_of(r1.w);
    s.ix = __fdiv_rn(1.0f, sanitize_dir(r1.x));
    s.iy = __fdiv_rn(1.0f, sanitize_dir(r1.y));
    s.iz = __fdiv_rn(1.0f, sanitize_dir(r1.z));
    s.oct = (signbit(r1.x) ? 1u : 0u) | (signbit(r1.y) ? 2u : 0u) | (signbit(r1.z) ? 4u : 0u);
    const float ax = fabsf(r1.x), ay = fabsf(r1.y), az = fabsf(r1.z);
    const int kz = (ax >= ay) ? (ax >= az ? 0 : 2) : (ay >= az ? 1 : 2);
    s.kz = kz;
    const float dkz = kz == 0 ? r1.x : (kz == 1 ? r1.y : r1.z);
    const float dkx = kz == 0 ? r1.y : (kz == 1 ? r1.z : r1.x);
    const float dky = kz == 0 ? r1.z : (kz == 1 ? r1.x : r1.y);
    s.nSx = -__fdiv_rn(dkx, dkz);
    s.nSy = -__fdiv_rn(dky, dkz);
    s.Sz = __fdiv_rn(1.0f, dkz);
    return s;
}

// Cyclic permutation (kx, ky, kz) = (kz+1, kz+2, kz) mod 3.
__device__ __forceinline__ void permute(const RayState& r, float a0, float a1, float a2, float& x, float& y, float& z) {
    x = r.kz == 0 ? a1 : (r.kz == 1 ? a2 : a0);
    y = r.kz == 0 ? a2 : (r.kz == 1 ? a0 : a1);
    z = r.kz == 0 ? a0 : (r.kz == 1 ? a1 : a2);
}

__device__ __forceinline__ float edge_fallback(float ax, float by, float ay, float bx) {
    return __double2float_rn(__dsub_rn(__dmul_rn((double)ax, (double)by), __dmul_rn((double)ay, (double)bx)));
}

// Watertight test, non-culling, same FP32 expression tree as the CPU
// restatement: every operation is an explicit round-to-nearest intrinsic so
// the compiler cannot contract or reorder it. Returns t (NaN-free) on a hit
// with t in [tmin, tmax]; out_u/out_v/out_det for barycentrics on request.
template <bool kBary = false>
__device__ __forceinline__ bool intersect_tri(const RayState& r, float4 v0, float4 v1, float4 v2, float tmax,
                                              float& t_out, float* bary = nullptr) {
    float Ax, Ay, Az, Bx, By, Bz, Cx, Cy, Cz;
    permute(r, __fsub_rn(v0.x, r.ox), __fsub_rn(v0.y, r.oy), __fsub_rn(v0.z, r.oz), Ax, Ay, Az);
    permute(r, __fsub_rn(v1.x, r.ox), __fsub_rn(v1.y, r.oy), __fsub_rn(v1.z, r.oz), Bx, By, Bz);
    permute(r, __fsub_rn(v2.x, r.ox), __fsub_rn(v2.y, r.oy), __fsub_rn(v2.z, r.oz), Cx, Cy, Cz);
    const float ax = __fmaf_rn(r.nSx, Az, Ax), ay = __fmaf_rn(r.nSy, Az, Ay);
    const float bx = __fmaf_rn(r.nSx, Bz, Bx), by = __fmaf_rn(r.nSy, Bz, By);
    const float cx = __fmaf_rn(r.nSx, Cz, Cx), cy = __fmaf_rn(r.nSy, Cz, Cy);
    float U = __fsub_rn(__fmul_rn(cx, by), __fmul_rn(cy, bx));
    float V = __fsub_rn(__fmul_rn(ax, cy), __fmul_rn(ay, cx));
    float W = __fsub_rn(__fmul_rn(bx, ay), __fmul_rn(by, ax));
    if (U == 0.0f || V == 0.0f || W == 0.0f) {
        U = edge_fallback(cx, by, cy, bx);
        V = edge_fallback(ax, cy, ay, cx);
        W = edge_fallback(bx, ay, by, ax);
    }
    if ((U < 0.0f || V < 0.0f || W < 0.0f) && (U > 0.0f || V > 0.0f || W > 0.0f)) return false;
    const float det = __fadd_rn(__fadd_rn(U, V), W);
    if (det == 0.0f) return false;
    const float az = __fmul_rn(r.Sz, Az), bz = __fmul_rn(r.Sz, Bz), cz = __fmul_rn(r.Sz, Cz);
    const float T = __fmaf_rn(W, cz, __fmaf_rn(V, bz, __fmul_rn(U, az)));
    const float t = __fdiv_rn(T, det);
    if (!(t >= r.tmin && t <= tmax)) return false;
    t_out = t;
    if (kBary) {
        bary[0] = U;
        bary[1] = V;
        bary[2] = W;
        bary[3] = det;
    }
    return true;
}

// Packed FP32 pairs for the child-box test: a slot's two plane FMAs in one
// fma.rm.f32x2 (sm_100 family). Each lane rounds exactly like the scalar
// __fmaf_rd (tests/test_minmax_gpu.py checks it on the GPU); the host build
// evaluates the scalar form.
struct F2 {
#if defined(__CUDA_ARCH__)
    unsigned long long v;
#else
    float x, y;
#endif
};
__device__ __forceinline__ F2 pack_f2(float a, float b) {
    F2 r;
#if defined(__CUDA_ARCH__)
    asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(a), "f"(b));
#else
    r.x = a;
    r.y = b;
#endif
    return r;
}
// out = a * b + c per lane, rounded down
__device__ __forceinline__ void fma_rd_f2(F2 a, F2 b, F2 c, float out[2]) {
#if defined(__CUDA_ARCH__)
    unsigned long long d;
    asm("fma.rm.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a.v), "l"(b.v), "l"(c.v));
    asm("mov.b64 {%0, %1}, %2;" : "=f"(out[0]), "=f"(out[1]) : "l"(d));
#else
    out[0] = __fmaf_rd(a.x, b.x, c.x);
    out[1] = __fmaf_rd(a.y, b.y, c.y);
#endif
}

// A quantised plane (byte k of word) as the float 1 + q 2^-15, exactly: one
// PRMT puts the byte into bits 8..15 of 1.0f's mantissa.
__device__ __forceinline__ float plane_value(uint32_t word, uint32_t k) {
    return __uint_as_float(__byte_perm(word, 0x3F800000u, 0x7604u | k << 4));
}

// max / min of three (one instruction on the sm_100 family; NaN operands
// are dropped like nested fmaxf / fminf, which tests/test_minmax_gpu.py
// checks on the GPU).
__device__ __forceinline__ float max3f(float a, float b, float c) {
#if defined(__CUDA_ARCH__)
    float r;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
#else
    return fmaxf(fmaxf(a, b), c);
#endif
}
__device__ __forceinline__ float min3f(float a, float b, float c) {
#if defined(__CUDA_ARCH__)
    float r;
    asm("min.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
#else
    return fminf(fminf(a, b), c);
#endif
}

// Bit 7 of each byte of w gathered into bits 0..3: the product places bits
// 7, 15, 23 and 31 at 28..31 and its other partial products at distinct
// lower positions, so no carry reaches the result.
__device__ __forceinline__ uint32_t meta_leaf_bits(uint32_t w) { return ((w & 0x80808080u) * 0x00204081u) >> 28; }

// Bit s of the 8-bit mask m moved to bit s ^ oct.
__device__ __forceinline__ uint32_t xor_permute8(uint32_t m, uint32_t oct) {
    if (oct & 1u) m = ((m & 0x55u) << 1) | ((m >> 1) & 0x55u);
    if (oct & 2u) m = ((m & 0x33u) << 2) | ((m >> 2) & 0x33u);
    if (oct & 4u) m = ((m & 0x0Fu) << 4) | (m >> 4);
    return m;
}

// Tests the 8 child boxes of one compressed node against the ray: which slots
// were hit, and the node's words that say what the slots hold. tfar: a bound_of.
struct SlotHits {
    uint32_t child_base;
    uint32_t tri_base;
    uint32_t imask;    // slots of internal children
    uint32_t hitm;     // bit s: slot s's box was hit (an empty slot's bit means nothing)
    uint32_t meta[2];  // the 8 meta bytes
};

__device__ __forceinline__ SlotHits intersect_slots(const RayState& r, const uint4* __restrict__ nodes, uint32_t idx,
                                                    float tfar) {
    const uint4* n = nodes + 5 * (size_t)idx;
    const uint4 w0 = __ldg(n + 0);
    const uint4 w1 = __ldg(n + 1);
    const uint4 w2 = __ldg(n + 2);
    const uint4 w3 = __ldg(n + 3);
    const uint4 w4 = __ldg(n + 4);
    const float sx = __uint_as_float((w0.w & 0xFFu) << 23) * (32768.0f * r.ix);
    const float sy = __uint_as_float(((w0.w >> 8) & 0xFFu) << 23) * (32768.0f * r.iy);
    const float sz = __uint_as_float(((w0.w >> 16) & 0xFFu) << 23) * (32768.0f * r.iz);
    const float bx = (__uint_as_float(w0.x) - r.ox) * r.ix;
    const float by = (__uint_as_float(w0.y) - r.oy) * r.iy;
    const float bz = (__uint_as_float(w0.z) - r.oz) * r.iz;
    const uint32_t imask = w0.w >> 24;
    // near / far plane words per axis, chosen by the direction signs
    const bool fx = signbit(r.ix), fy = signbit(r.iy), fz = signbit(r.iz);
    const uint32_t nx0 = fx ? w3.z : w2.x, nx1 = fx ? w3.w : w2.y;
    const uint32_t gx0 = fx ? w2.x : w3.z, gx1 = fx ? w2.y : w3.w;
    const uint32_t ny0 = fy ? w4.x : w2.z, ny1 = fy ? w4.y : w2.w;
    const uint32_t gy0 = fy ? w2.z : w4.x, gy1 = fy ? w2.w : w4.y;
    const uint32_t nz0 = fz ? w4.z : w3.x, nz1 = fz ? w4.w : w3.y;
    const uint32_t gz0 = fz ? w3.x : w4.z, gz1 = fz ? w3.y : w4.w;
    // A plane's t is q * s + b with q the quantised byte. The byte is read
    // as the float v = 1 + q 2^-15 (plane_value) and the step taken as
    // S = 2^15 s (exact), near planes rounded down and far planes up:
    //   near: rd(v S + rd(b - S)) <= rd(q s + b) <= rn(q s + b)
    //   far:  ru(v S + ru(b - S)) >= ru(q s + b) >= rn(q s + b)
    // so every child box is at least as wide as under round-to-nearest
    // fma(q, s, b), the culling stays conservative and the hits exact.
    // A slot's near and far plane go through one packed FMA, the far one
    // negated (ru(x) = -rd(-x)), so both round down and one pair of constants
    // per axis serves both: 12 registers across the eight slots, 18 with the
    // constants duplicated for slot pairs.
    const F2 sx2 = pack_f2(sx, -sx), sy2 = pack_f2(sy, -sy), sz2 = pack_f2(sz, -sz);
    const F2 bx2 = pack_f2(__fmaf_rd(-1.0f, sx, bx), __fmaf_rd(1.0f, sx, -bx));
    const F2 by2 = pack_f2(__fmaf_rd(-1.0f, sy, by), __fmaf_rd(1.0f, sy, -by));
    const F2 bz2 = pack_f2(__fmaf_rd(-1.0f, sz, bz), __fmaf_rd(1.0f, sz, -bz));
    // the boxes alone: bit s of miss for slot s (empty slots included)
    const float ntfar = -tfar;
    uint32_t miss = 0;
#pragma unroll
    for (int pr = 3; pr >= 0; --pr) {
        const uint32_t k = 2u * (pr & 1);
        float nx[2], ny[2], nz[2], gx[2], gy[2], gz[2];
#pragma unroll
        for (uint32_t e = 0; e < 2; ++e) {
            nx[e] = plane_value(pr < 2 ? nx0 : nx1, k + e);
            gx[e] = plane_value(pr < 2 ? gx0 : gx1, k + e);
            ny[e] = plane_value(pr < 2 ? ny0 : ny1, k + e);
            gy[e] = plane_value(pr < 2 ? gy0 : gy1, k + e);
            nz[e] = plane_value(pr < 2 ? nz0 : nz1, k + e);
            gz[e] = plane_value(pr < 2 ? gz0 : gz1, k + e);
        }
#pragma unroll
        for (int e = 1; e >= 0; --e) {
            // miss: the sign of tf - tn, shifted in (a difference and a funnel
            // shift: the compare and select of the plain form both go to the
            // integer pipe, the busier one). Equal infinities give a NaN of
            // positive sign and equal values +0, a hit as under tn <= tf; only
            // tf = -0 against tn = +0 would differ, hence bound_of.
            float tx[2], ty[2], tz[2];  // near t, -(far t)
            fma_rd_f2(pack_f2(nx[e], gx[e]), sx2, bx2, tx);
            fma_rd_f2(pack_f2(ny[e], gy[e]), sy2, by2, ty);
            fma_rd_f2(pack_f2(nz[e], gz[e]), sz2, bz2, tz);
            const float tn = max3f(tx[0], ty[0], fmaxf(tz[0], r.tmin));
            const float ntf = max3f(tx[1], ty[1], fmaxf(tz[1], ntfar));
#if defined(__CUDA_ARCH__)
            miss = __funnelshift_l(__float_as_uint(__fsub_rn(-ntf, tn)), miss, 1);
#else
            const float span = -ntf - tn;  // (a host NaN's sign may be set)
            miss = miss << 1 | (span == span && signbit(span) ? 1u : 0u);
#endif
        }
    }
    SlotHits out;
    out.child_base = w1.x;
    out.tri_base = w1.y;
    out.imask = imask;
    out.hitm = ~miss & 0xFFu;
    out.meta[0] = w1.z;
    out.meta[1] = w1.w;
    return out;
}

// The leaf slots of a node, by the 0x80 flag of their meta bytes.
__device__ __forceinline__ uint32_t leaf_slots(const SlotHits& h) {
    return meta_leaf_bits(h.meta[0]) | meta_leaf_bits(h.meta[1]) << 4;
}
// Meta byte of slot s.
__device__ __forceinline__ uint32_t meta_of(const SlotHits& h, uint32_t s) {
    return __byte_perm(s < 4u ? h.meta[0] : h.meta[1], 0u, 0x4440u | (s & 3u));
}

// The same as one group of internal children in traversal order (bit i is
// slot i ^ oct, in bits 0..7, with the node's imask in bits 8..15) and the
// triangle mask (bit k: triangle tri_base + k) of the hit leaf children.
struct NodeHits {
    uint32_t child_base;
    uint32_t tri_base;
    uint32_t group;  // imask << 8 | ordered internal hits
    uint32_t tris;
};

__device__ __forceinline__ NodeHits intersect_node(const RayState& r, const uint4* __restrict__ nodes, uint32_t idx,
                                                   float tfar) {
    const SlotHits h = intersect_slots(r, nodes, idx, bound_of(tfar));
    uint32_t lh = h.hitm & leaf_slots(h), tris = 0;
    while (lh) {  // about one hit leaf per three nodes on incoherent rays
        const uint32_t s = (uint32_t)__ffs(lh) - 1u;
        lh &= lh - 1u;
        const uint32_t meta = meta_of(h, s);
        tris |= ((2u << ((meta >> 5) & 3u)) - 1u) << (meta & 31u);
    }
    NodeHits out;
    out.child_base = h.child_base;
    out.tri_base = h.tri_base;
    out.group = (h.imask << 8) | xor_permute8(h.hitm & h.imask, r.oct);
    out.tris = tris;
    return out;
}

}  // namespace RT
}  // namespace Foundation

namespace Foundation {
namespace RT {

// Reached by tests only, from here on (intersect_node too): the plain form that
// the warp loop (warp_trace.cuh) is tested against, on the host as well. Single-
// ray traversal with a thread-local stack and no warp refill; the node and
// triangle tests and the tie rule are the persistent kernels'. Returns true on a
// hit (best_t / best_p updated; the caller initialises best_t to the ray's tmax).
template <bool kAny>
__device__ __forceinline__ bool trace_single(const DeviceScene& sc, const RayState& r, float& best_t,
                                             uint32_t& best_p, uint32_t* status) {
    best_p = FND_INVALID_ID;
    if (sc.num_nodes == 0) return false;
    uint2 stack[kMaxStack];
    int sp = 0;
    uint32_t ng_base = 0, ng_group = (1u << 8) | (1u << r.oct), tg_base = 0, tg_mask = 0;
    for (;;) {
        if (ng_group & 0xFFu) {
            const uint32_t b = (uint32_t)__ffs(ng_group & 0xFFu) - 1u;
            ng_group &= ~(1u << b);
            const uint32_t slot = b ^ r.oct;
            const uint32_t child = ng_base + (uint32_t)__popc((ng_group >> 8) & ((1u << slot) - 1u));
            if (ng_group & 0xFFu) {
                if (sp >= kMaxStack) {
                    atomicOr(status, kStatusStackOverflow);
                    break;
                }
                stack[sp++] = make_uint2(ng_base, ng_group);
            }
            if (child >= sc.num_nodes) {
                atomicOr(status, kStatusBadIndex);
                break;
            }
            const NodeHits h = intersect_node(r, sc.nodes, child, best_t);
            ng_base = h.child_base;
            ng_group = h.group;
            tg_base = h.tri_base;
            tg_mask = h.tris;
            if (tg_mask && (uint64_t)tg_base + (uint64_t)(32 - __clz(tg_mask)) > sc.num_tris) {
                atomicOr(status, kStatusBadIndex);
                break;
            }
        }
        while (tg_mask) {
            const uint32_t k = (uint32_t)__ffs(tg_mask) - 1u;
            tg_mask &= tg_mask - 1u;
            const uint32_t ti = tg_base + k;
            const size_t at = (size_t)ti * sc.tri_stride;
            const float4 v0 = __ldg(sc.v0 + at);
            float t;
            if (intersect_tri(r, v0, __ldg(sc.v1 + at), __ldg(sc.v2 + at), best_t, t)) {
                const uint32_t pid = __float_as_uint(v0.w);
                if (kAny) {
                    best_t = t;
                    best_p = pid;
                    return true;
                }
                if (best_p == FND_INVALID_ID || t < best_t || (t == best_t && pid < best_p)) {
                    best_t = t;
                    best_p = pid;
                }
            }
        }
        if (ng_group & 0xFFu) continue;
        if (sp == 0) break;
        const uint2 e = stack[--sp];
        ng_base = e.x;
        ng_group = e.y;
    }
    return best_p != FND_INVALID_ID;
}

// World ray -> object space of an instance: o' = inv * (o, 1), d' = inv * (d, 0),
// each component summed left to right with round-to-nearest operations (the
// oracle evaluates the same expression); t is the same parameter in both
// spaces, so tmin / tmax carry over.
__device__ __forceinline__ void instance_ray(const float* inv, float4 r0, float4 r1, float4& o0, float4& o1) {
    float o[3], d[3];
    for (int i = 0; i < 3; ++i) {
        const float* m = inv + 4 * i;
        o[i] = __fadd_rn(__fadd_rn(__fadd_rn(__fmul_rn(m[0], r0.x), __fmul_rn(m[1], r0.y)), __fmul_rn(m[2], r0.z)), m[3]);
        d[i] = __fadd_rn(__fadd_rn(__fmul_rn(m[0], r1.x), __fmul_rn(m[1], r1.y)), __fmul_rn(m[2], r1.z));
    }
    o0 = make_float4(o[0], o[1], o[2], r0.w);
    o1 = make_float4(d[0], d[1], d[2], r1.w);
}

// Two-level traversal: the top-level tree's leaves are instances (the plane
// record's index word holds the instance id); each instance's bottom level
// is traversed in object space with trace_single. Ties across instances
// break by the global id (prim_offset + bottom-level id), as within a scene.
template <bool kAny>
__device__ __forceinline__ bool trace_two_level(const DeviceScene& tlas, const InstanceRec* __restrict__ inst,
                                                uint32_t num_inst, float4 r0, float4 r1, float& best_t,
                                                uint32_t& best_p, uint32_t* status) {
    best_p = FND_INVALID_ID;
    if (tlas.num_nodes == 0) return false;
    const RayState r = setup_ray(r0, r1);
    uint2 stack[kMaxStack];
    int sp = 0;
    uint32_t ng_base = 0, ng_group = (1u << 8) | (1u << r.oct), tg_base = 0, tg_mask = 0;
    for (;;) {
        if (ng_group & 0xFFu) {
            const uint32_t b = (uint32_t)__ffs(ng_group & 0xFFu) - 1u;
            ng_group &= ~(1u << b);
            const uint32_t slot = b ^ r.oct;
            const uint32_t child = ng_base + (uint32_t)__popc((ng_group >> 8) & ((1u << slot) - 1u));
            if (ng_group & 0xFFu) {
                if (sp >= kMaxStack) {
                    atomicOr(status, kStatusStackOverflow);
                    break;
                }
                stack[sp++] = make_uint2(ng_base, ng_group);
            }
            if (child >= tlas.num_nodes) {
                atomicOr(status, kStatusBadIndex);
                break;
            }
            const NodeHits h = intersect_node(r, tlas.nodes, child, best_t);
            ng_base = h.child_base;
            ng_group = h.group;
            tg_base = h.tri_base;
            tg_mask = h.tris;
            if (tg_mask && (uint64_t)tg_base + (uint64_t)(32 - __clz(tg_mask)) > tlas.num_tris) {
                atomicOr(status, kStatusBadIndex);
                break;
            }
        }
        while (tg_mask) {
            const uint32_t k = (uint32_t)__ffs(tg_mask) - 1u;
            tg_mask &= tg_mask - 1u;
            const uint32_t id = __float_as_uint(__ldg(tlas.v0 + (size_t)(tg_base + k) * tlas.tri_stride).w);
            if (id >= num_inst) {
                atomicOr(status, kStatusBadIndex);
                continue;
            }
            const InstanceRec& I = inst[id];
            RayState ro = r;  // an identity instance keeps the world ray
            if (!(__ldg(&I.flags) & kInstanceIdentity)) {
                float inv[12];
                for (int q = 0; q < 12; ++q) inv[q] = __ldg(I.inv + q);
                float4 o0, o1;
                instance_ray(inv, r0, r1, o0, o1);
                ro = setup_ray(o0, o1);
            }
            const DeviceScene blas = I.blas;
            float t = best_t;
            uint32_t p;
            if (trace_single<kAny>(blas, ro, t, p, status)) {
                const uint32_t gid = __ldg(&I.prim_offset) + p;
                if (kAny) {
                    best_t = t;
                    best_p = gid;
                    return true;
                }
                if (best_p == FND_INVALID_ID || t < best_t || (t == best_t && gid < best_p)) {
                    best_t = t;
                    best_p = gid;
                }
            }
        }
        if (ng_group & 0xFFu) continue;
        if (sp == 0) break;
        const uint2 e = stack[--sp];
        ng_base = e.x;
        ng_group = e.y;
    }
    return best_p != FND_INVALID_ID;
}

}  // namespace RT
}  // namespace Foundation
