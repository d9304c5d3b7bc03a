// product_check.cu — TEST HARNESS: reaches into a live context of the library,
// for states that no call of the API produces by itself. Links libfnd_rt.so.
#include <cuda_runtime.h>

#include <cstdint>

#include "../../foundation_gb300/csrc/capi/context.hpp"
#include "../../foundation_gb300/csrc/rt/traverse_launch.hpp"

// Sets the context's status word, as a kernel that has given up on a wait (or
// met a bad index) does. Returns 0 on success, 1 on a CUDA error.
extern "C" int product_latch_status(fnd_rt_ctx* ctx, uint32_t bits) {
    return cudaStreamSynchronize(ctx->stream) == cudaSuccess &&
                   cudaMemcpy(ctx->d_status, &bits, sizeof(bits), cudaMemcpyDefault) == cudaSuccess
               ? 0
               : 1;
}

// Resident blocks of 128 threads per SM of the path kernels.
extern "C" int product_tail_blocks(int two_level) { return Foundation::PT::TailBlocksPerSm(two_level != 0); }
extern "C" int product_training_blocks(int two_level) {
    return Foundation::PT::TrainingPathsBlocksPerSm(two_level != 0);
}

// Copies an uploaded scene's array to (write 0) or from (write 1) the host:
// part 0 the wide nodes (node_bytes), 1 the triangle records (tri_bytes).
extern "C" int product_scene_bytes(fnd_rt_scene* scene, int part, int write, void* host) {
    void* d = part == 0 ? scene->d_nodes : scene->d_tris;
    const size_t bytes = part == 0 ? scene->info.node_bytes : scene->info.tri_bytes;
    if (cudaDeviceSynchronize() != cudaSuccess) return 1;
    const cudaError_t e = write ? cudaMemcpy(d, host, bytes, cudaMemcpyHostToDevice)
                                : cudaMemcpy(host, d, bytes, cudaMemcpyDeviceToHost);
    return e == cudaSuccess ? 0 : 1;
}

// The persistent kernels over a hand-made scene of triangle records (three
// float4 each), as every uploaded scene is laid out. The same ray n times;
// hits: n (id, t bits) pairs, or (any) n occlusion bytes.
extern "C" int product_trace_records(const void* nodes, uint32_t num_nodes, const float* tris, uint32_t num_tris,
                                     const float* rays, uint32_t n, int any, void* hits, uint32_t* status_out) {
    using namespace Foundation::RT;
    const size_t nb = 80 * (size_t)num_nodes, tb = 48 * (size_t)num_tris, rb = 32 * (size_t)n;
    const size_t hb = (any ? 1 : 8) * (size_t)n;
    unsigned char* d = nullptr;
    if (cudaMalloc(&d, 256 + nb + tb + rb + hb) != cudaSuccess) return 1;
    unsigned char* p = d + 256;
    int sms = 0, blocks = 0;
    bool ok = cudaMemset(d, 0, 256) == cudaSuccess && cudaMemcpy(p, nodes, nb, cudaMemcpyHostToDevice) == cudaSuccess &&
              (tb == 0 || cudaMemcpy(p + nb, tris, tb, cudaMemcpyHostToDevice) == cudaSuccess) &&
              cudaMemcpy(p + nb + tb, rays, rb, cudaMemcpyHostToDevice) == cudaSuccess &&
              cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, 0) == cudaSuccess &&
              TraceOccupancy(any ? 1 : 0, &blocks) == cudaSuccess;
    if (ok) {
        TraceLaunch L{};
        L.scene.nodes = reinterpret_cast<const uint4*>(p);
        L.scene.num_nodes = num_nodes;
        Foundation::CApi::ViewTriangles(L.scene, p + nb, num_tris);
        L.rays = reinterpret_cast<const float4*>(p + nb + tb);
        L.n = n;
        L.hits = p + nb + tb + rb;
        L.occluded = p + nb + tb + rb;
        L.counter = reinterpret_cast<uint32_t*>(d);
        L.status = L.counter + 1;
        L.refill_min = 8;
        ok = LaunchTrace(L, any != 0, false, sms * (blocks > 0 ? blocks : 1), nullptr) == cudaSuccess &&
             cudaDeviceSynchronize() == cudaSuccess &&
             cudaMemcpy(hits, p + nb + tb + rb, hb, cudaMemcpyDeviceToHost) == cudaSuccess &&
             cudaMemcpy(status_out, d + 4, 4, cudaMemcpyDeviceToHost) == cudaSuccess;
    }
    cudaFree(d);
    return ok ? 0 : 1;
}
