// product_check.cu — TEST HARNESS: reaches into a live context of the library,
// for states that no call of the API produces by itself. Links libfnd_rt.so.
#include <cuda_runtime.h>

#include <cstdint>

#include "../../foundation_gb300/csrc/capi/context.hpp"

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
