// integrator.cu — wavefront path-tracing stages (sm_103a): generate, shade,
// shadow resolve, finalize. The extend and shadow traversals are the
// persistent trace kernels of rt/traverse.cu reading their ray counts from
// the device queues.
//
// Light transport (same definitions as the FP64 oracle, oracle/pt_oracle.cpp):
//  * pinhole camera (glm lookAt convention), one jittered sample per path;
//  * surfaces two-sided (geometric normal flipped towards the incoming ray),
//    emitters one-sided (they emit on the side their winding normal faces)
//    and black;
//  * next-event estimation at every non-emissive hit: one point on one quad
//    light (uniform light choice, uniform point on the quad) weighted by the
//    power heuristic against the BSDF pdf, plus one shadow ray towards the
//    directional sun when there is one; BSDF-sampled hits on emitters are
//    weighted by the power heuristic against the light pdf; escaping rays
//    collect the constant sky radiance;
//  * Russian roulette from bounce `rr_start` with survival probability
//    clamp(max(throughput), 0.05, 1); at most `max_depth` surface interactions.
#include "integrator.hpp"

#include "../../../include/fnd_rt.h"
#include "pt_math.cuh"
#include "shade.cuh"

namespace Foundation {
namespace PT {
namespace {

constexpr uint32_t kFull = 0xFFFFFFFFu;
constexpr int kBlock = 256;
constexpr int kShadeBlock = 128, kShadeBlocksPerSm = 6;

__device__ __forceinline__ float3 ld3(const float* p) { return f3(p[0], p[1], p[2]); }
__device__ __forceinline__ float3 xyz(float4 v) { return f3(v.x, v.y, v.z); }

__device__ __forceinline__ void add_radiance(float4* fb, uint32_t pixel, float3 L) {
    atomicAdd(fb + pixel, make_float4(L.x, L.y, L.z, 0.0f));
}

// Pixel and sample of path i of the wave, and its generator after the two
// numbers that generate_kernel places the ray in the pixel with (a, b).
__device__ __forceinline__ Pcg32 camera_path(const PathBuffers& B, const RenderParams& R, uint32_t i, uint32_t& pixel,
                                             uint32_t& sample, float& a, float& b) {
    const uint32_t npix = R.width * R.height, at = B.wave_pixel + i;  // (below 2^26 + 2^28)
    pixel = at % npix;
    sample = B.wave_sample + at / npix + R.sample_offset;
    Pcg32 rng = camera_path_rng(R.seed, pixel, sample);
    a = rng.uniform();
    b = rng.uniform();
    return rng;
}

// Writes the camera rays only: the rest of a new path (generator, throughput
// one) is made again by the first shade stage, which costs less than to
// write and read it (4.1M paths: 36 bytes each way, 45 us).
__global__ void __launch_bounds__(kBlock) generate_kernel(const PathBuffers B, const RenderParams R, uint32_t wave_n) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (blockIdx.x == 0)
        for (uint32_t k = threadIdx.x; k < (uint32_t)kCounts; k += blockDim.x) B.counts[k] = k == kCountExt ? wave_n : 0u;
    if (i >= wave_n) return;
    uint32_t pixel, sample;
    float a, b;
    camera_path(B, R, i, pixel, sample, a, b);
    const uint32_t px = pixel % R.width, py = pixel / R.width;
    const float sx = (2.0f * ((float)px + a) / (float)R.width - 1.0f) * R.tan_half * R.aspect;
    const float sy = (1.0f - 2.0f * ((float)py + b) / (float)R.height) * R.tan_half;
    const float3 d = normalize(ld3(R.fwd) + ld3(R.right) * sx + ld3(R.up) * sy);
    B.ext_rays[0][2 * (size_t)i] = make_float4(R.eye[0], R.eye[1], R.eye[2], 0.0f);
    B.ext_rays[0][2 * (size_t)i + 1] = make_float4(d.x, d.y, d.z, __int_as_float(0x7F800000));
}

// One interaction of each queued path. What bounds it: the latency of its
// dependent gathers (queue entry, path state, hit, shading record, material)
// and of the queue appends, not bytes (DRAM at 11%) nor issue (25%). Hence as
// many warps as registers allow without spills that show: 80 registers, six
// blocks of 128 (24 warps per SM). Plain 1080p frame of 2 spp with four, five,
// six and eight such blocks 4,102, 4,090, 4,038 and 4,036 us, with three of 256
// 4,046; the cache frame 1,366, 1,365, 1,362, 1,367 and 1,365.
// kFirst: the camera rays' hits (see generate_kernel).
template <uint32_t kMode, bool kFirst>
__global__ void __launch_bounds__(kShadeBlock, kShadeBlocksPerSm)
    shade_kernel(const PathBuffers B, const RenderParams R, const ShadeScene S, const CacheIO C, uint32_t bounce) {
    const uint32_t n = B.counts[kCountExt + bounce];
    const uint32_t cur = bounce & 1u, nxt = cur ^ 1u;
    const uint32_t stride = gridDim.x * blockDim.x;
    const uint32_t lane = threadIdx.x & 31u, below = (1u << lane) - 1u;
    for (uint32_t base = blockIdx.x * blockDim.x + (threadIdx.x & ~31u); base < n; base += stride) {
        const uint32_t j = base + lane;
        uint32_t flags = 0, pixel = 0, sample = 0;
        Pcg32 rng{};
        VertexOut v;
        v.shadow = v.sun = v.query = v.next = false;
        if (j < n) {
            const uint2 hit = B.hits[j];
            const float4 r0 = B.ext_rays[cur][2 * (size_t)j];
            const float4 r1 = B.ext_rays[cur][2 * (size_t)j + 1];
            VertexIn in;
            if constexpr (kFirst) {
                float a, b;
                rng = camera_path(B, R, j, pixel, sample, a, b);
                in.beta = f3(1.0f, 1.0f, 1.0f);
                in.last_pdf = 0.0f;
            } else {
                const float4 beta4 = B.beta[cur][j];
                const uint4 rs = B.rng[cur][j];
                rng = unpack_rng(rs);
                sample = rs.z;
                pixel = rs.w & ~kQueryNextFlag;
                flags = rs.w & kQueryNextFlag;
                in.beta = xyz(beta4);
                in.last_pdf = beta4.w;
            }
            in.o = xyz(r0);
            in.d = xyz(r1);
            in.hit = hit.x != FND_INVALID_ID;
            in.prim = hit.x;
            in.t = __uint_as_float(hit.y);
            in.query_here = flags != 0u;
            shade_vertex<kMode>(R, S, C.specular_alpha, bounce, R.max_depth, in, rng, v);
            if (max3(v.add) > 0.0f) add_radiance(B.fb, pixel, v.add);
        }
        // the warp's entries of all queues by one atomic instruction (lane q
        // adds for queue q): each answer is a trip to L2
        const uint32_t ml = __ballot_sync(kFull, v.shadow), ms = __ballot_sync(kFull, v.sun);
        const uint32_t mn = __ballot_sync(kFull, v.next), mq = kMode == 1u ? __ballot_sync(kFull, v.query) : 0u;
        uint32_t* counter = lane == 0u   ? B.counts + kCountShadow + bounce
                            : lane == 1u ? B.counts + kCountExt + bounce + 1u
                                         : C.query_count;
        const uint32_t count = lane == 0u   ? (uint32_t)__popc(ml) + (uint32_t)__popc(ms)
                               : lane == 1u ? (uint32_t)__popc(mn)
                               : lane == 2u ? (uint32_t)__popc(mq)
                                            : 0u;
        const uint32_t at = count ? atomicAdd(counter, count) : 0u;
        const uint32_t at_sh = __shfl_sync(kFull, at, 0), at_next = __shfl_sync(kFull, at, 1);
        if (v.shadow) {
            const uint32_t k = at_sh + (uint32_t)__popc(ml & below);
            B.sh_rays[2 * (size_t)k] = make_float4(v.surf_o.x, v.surf_o.y, v.surf_o.z, 0.0f);
            B.sh_rays[2 * (size_t)k + 1] = make_float4(v.sh_d.x, v.sh_d.y, v.sh_d.z, v.sh_tmax);
            B.sh_contrib[k] = make_float4(v.sh_c.x, v.sh_c.y, v.sh_c.z, __uint_as_float(pixel));
        }
        if (v.sun) {
            const uint32_t k = at_sh + (uint32_t)__popc(ml) + (uint32_t)__popc(ms & below);
            B.sh_rays[2 * (size_t)k] = make_float4(v.surf_o.x, v.surf_o.y, v.surf_o.z, 0.0f);
            B.sh_rays[2 * (size_t)k + 1] = make_float4(R.sun_dir[0], R.sun_dir[1], R.sun_dir[2],
                                                       __int_as_float(0x7F800000));
            B.sh_contrib[k] = make_float4(v.sun_c.x, v.sun_c.y, v.sun_c.z, __uint_as_float(pixel));
        }
        if (kMode == 1u) {
            const uint32_t k = __shfl_sync(kFull, at, 2) + (uint32_t)__popc(mq & below);
            if (v.query && k < C.query_cap) {
                v.cp.wo_aux.w = __uint_as_float(pixel);
                C.queries[k] = v.cp;
            }
        }
        if (v.next) {
            const uint32_t k = at_next + (uint32_t)__popc(mn & below);
            if (kMode == 1u && v.query_next) flags = kQueryNextFlag;
            B.ext_rays[nxt][2 * (size_t)k] = make_float4(v.surf_o.x, v.surf_o.y, v.surf_o.z, 0.0f);
            B.ext_rays[nxt][2 * (size_t)k + 1] =
                make_float4(v.next_d.x, v.next_d.y, v.next_d.z, __int_as_float(0x7F800000));
            B.beta[nxt][k] = make_float4(v.beta.x, v.beta.y, v.beta.z, v.pdf);
            B.rng[nxt][k] = pack_rng(rng, sample, pixel | flags);
        }
    }
}

__global__ void __launch_bounds__(kBlock) resolve_kernel(const PathBuffers B, uint32_t bounce) {
    const uint32_t n = B.counts[kCountShadow + bounce];
    const uint32_t stride = gridDim.x * blockDim.x;
    for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += stride) {
        if (B.sh_occluded[k]) continue;
        const float4 c = B.sh_contrib[k];
        add_radiance(B.fb, __float_as_uint(c.w), f3(c.x, c.y, c.z));
    }
}

__global__ void __launch_bounds__(kBlock) finalize_kernel(const float4* fb, float* rgb, uint32_t npix, float scale) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= npix) return;
    const float4 v = fb[i];
    rgb[3 * (size_t)i + 0] = v.x * scale;
    rgb[3 * (size_t)i + 1] = v.y * scale;
    rgb[3 * (size_t)i + 2] = v.z * scale;
}

}  // namespace

cudaError_t LaunchGenerate(const PathBuffers& B, const RenderParams& R, uint32_t wave_n, cudaStream_t s) {
    const uint32_t blocks = (wave_n + kBlock - 1) / kBlock;
    generate_kernel<<<blocks ? blocks : 1, kBlock, 0, s>>>(B, R, wave_n);
    return cudaGetLastError();
}

cudaError_t LaunchShade(const PathBuffers& B, const RenderParams& R, const ShadeScene& S, const CacheIO& C,
                        uint32_t bounce, int grid, cudaStream_t s) {
    grid *= kBlock / kShadeBlock;
    if (C.mode == 1u && bounce == 0)
        shade_kernel<1u, true><<<grid, kShadeBlock, 0, s>>>(B, R, S, C, bounce);
    else if (C.mode == 1u)
        shade_kernel<1u, false><<<grid, kShadeBlock, 0, s>>>(B, R, S, C, bounce);
    else if (bounce == 0)
        shade_kernel<0u, true><<<grid, kShadeBlock, 0, s>>>(B, R, S, C, bounce);
    else
        shade_kernel<0u, false><<<grid, kShadeBlock, 0, s>>>(B, R, S, C, bounce);
    return cudaGetLastError();
}

cudaError_t LaunchResolve(const PathBuffers& B, uint32_t bounce, int grid, cudaStream_t s) {
    resolve_kernel<<<grid, kBlock, 0, s>>>(B, bounce);
    return cudaGetLastError();
}

cudaError_t LaunchFinalize(const PathBuffers& B, float* rgb, uint32_t npix, float scale, cudaStream_t s) {
    finalize_kernel<<<(npix + kBlock - 1) / kBlock, kBlock, 0, s>>>(B.fb, rgb, npix, scale);
    return cudaGetLastError();
}

}  // namespace PT
}  // namespace Foundation
