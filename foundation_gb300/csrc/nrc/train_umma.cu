// train_umma.cu — one optimiser step of the radiance cache's MLP on the
// fifth-generation tensor cores (tcgen05, sm_103a): input encoding, forward,
// relative-L2 loss, backward and weight gradients of 128-row tiles, fused in
// one kernel.
//
// A CTA takes one tile of kRows = 128 samples, the M of one tcgen05 MMA:
//  * the tcgen05 weight images (nrc.hpp) arrive in shared memory by two bulk
//    copies (TMA) that run under the input encoding; the encoded inputs X, the
//    five hidden activations H1..H5 and two gradient buffers dZ stay there in
//    the core-matrix layout of umma.cuh, so every GEMM of the step reads its
//    operands from shared memory;
//  * forward: Z_l = H_l W_l (H_0 = X) accumulates in tensor memory; the
//    epilogue (8 warps, each a quarter of the lanes and half the columns)
//    applies ReLU, rounds to BF16 and writes H_{l+1};
//  * loss: the 3 outputs of each row, relative L2 (y - t)^2 / (y^2 + eps)
//    with the denominator held constant (Müller et al. 2021), give dZ_5;
//  * backward, per layer l = 5 .. 0, two GEMMs:
//      dH_l    = dZ_l W_l^T   (M = 128 rows), and the epilogue masks dH_l by
//                             H_l > 0 into dZ_{l-1} (BF16);
//      dW_l^T  = dZ_l^T H_l   (M = outputs padded to 128, K = the 128 rows:
//                             both operands MN-major, the transposed reads of
//                             the same shared arrays), under that epilogue;
//  * the weight gradients go from tensor memory to shared memory under the next
//    layer's GEMM and are added to the global FP32 gradient by the TMA.
//
// What bounds it: the chain. Twelve dependent GEMMs of a few hundred cycles, one
// tile per CTA, so what counts is the latency around them. Cycles of a CTA at
// each form:
//   MMAs issued by thread 0 under a plain branch: 4 take 850 cycles, 1,550 a
//     phase; gradients by vector atomics, a row per lane: 13,500 of 40,600;
//   an elected lane, unrolled: 270, 960 a forward phase; gradients through
//     shared memory and one bulk reduction at the end: 8,500 of 31,000;
//   this form, a warp of its own for the MMAs (they and the tensor-memory
//     set-up run beside the other warps), dW behind dH in the queue, gradients
//     out layer by layer, the encoding's two halves in different warps: 27,400.
// (Six steps on 65,536 paths' samples, paths included: 527, 483, 465 us.)
// Features that the host holds are bound by the link (6.3 MB at 205 GB/s, 31 us).
// One elected lane issues every MMA and commits it to an mbarrier; each wait for
// one is bounded and, when it runs out, the step latches the timeout bit of the
// status word, stops, and still releases its tensor memory. Adam (mlp.cu) then
// applies the gradient.
//
// Tensor memory (512 columns): Z / dH at column 0 (64), dW_0^T at 64 (96), the
// others at 160 + 64 (l - 1).
#include <cuda_bf16.h>

#include <type_traits>

#include "../rt/device_scene.hpp"
#include "mlp_common.cuh"
#include "nrc.hpp"
#include "umma.cuh"

namespace Foundation {
namespace NRC {
namespace {

using namespace Umma;

constexpr uint32_t kRows = 128;
constexpr uint32_t kEpilogueWarps = 8, kEpilogueThreads = 32 * kEpilogueWarps, kThreads = kEpilogueThreads + 32;
constexpr uint32_t kTmemCols = 512;
constexpr uint32_t kColZ = 0;  // Z_l, then dH_l
__host__ __device__ constexpr uint32_t ColDW(int l) { return l == 0 ? 64 : 160 + 64 * (l - 1); }
constexpr uint32_t kWaitLimit = 1u << 22;

// shared-memory map (bytes, each region 1024-aligned)
constexpr uint32_t kSmWf = 0;                                 // forward images, layers 0..5
constexpr uint32_t kSmWb = kSmWf + 2 * kUFwdElems;            // backward images, layers 1..5
constexpr uint32_t kSmX = kSmWb + 2 * kUBwdElems;             // X [128][96]
constexpr uint32_t kSmH = kSmX + 2 * kRows * kIn;             // H1..H5 [128][64]
constexpr uint32_t kHBytes = 2 * kRows * kWidth;
constexpr uint32_t kSmDz = kSmH + 5 * kHBytes;                // dZ [128][64] (layer 5: [128][16]), two buffers
__host__ __device__ constexpr uint32_t DzBuffer(int l) { return kSmDz + (l & 1) * kHBytes; }
constexpr uint32_t kSmTgt = kSmDz + 2 * kHBytes;              // float4 per row
constexpr uint32_t kSmBytes = kSmTgt + 16 * kRows;
static_assert(kSmWb % 1024 == 0 && kSmX % 1024 == 0 && kSmH % 1024 == 0 && kSmDz % 1024 == 0, "alignment");
// the padded M = 128 reads of the weight-gradient GEMMs run past a dZ buffer by
// 1024 bytes (into the other one or the targets); what they give is not used
static_assert(kSmBytes <= 227 * 1024, "shared memory");

// layer l's gradient (FP32, in the order of the parameters) takes the place of
// that layer's inputs
static_assert(4 * ParamOffset(1) == kSmH - kSmX && 4 * (ParamOffset(2) - ParamOffset(1)) == kHBytes, "in place");

struct TrainArgs {
    Net net;
    const TrainSample* samples;  // sampled mode
    const float4* targets;
    const uint32_t* count;
    const float* raw_feats;      // raw mode (tests): n x 96 features
    const float* raw_targets;    // n x 3
    float* out_grad;             // raw mode: where the last CTA copies the gradient (16-byte aligned), or null
    double* out_loss;
    uint32_t rows;               // rows of this step (batch)
    uint32_t seed;
    float inv_norm;              // 1 / (3 * rows)
    uint32_t* status;            // timeout bit on a wait that ran out
};

__device__ __forceinline__ uint32_t bf16x2(float lo, float hi) {
    __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<uint32_t*>(&v);
}
__device__ __forceinline__ float bf16_lo(uint32_t u) { return __uint_as_float(u << 16); }
__device__ __forceinline__ float bf16_hi(uint32_t u) { return __uint_as_float(u & 0xFFFF0000u); }

// K-major operand of a row-group-major [rows][cols] array: K steps of 16
// are 256 bytes apart.
__device__ __forceinline__ uint64_t kmajor(uint32_t saddr, uint32_t cols) {
    return smem_desc(saddr, 128u, cols / 8u * 128u);
}
// MN-major operand (the transposed read): the K (row) steps of 16 are
// 2 * cols / 8 * 128 bytes apart.
__device__ __forceinline__ uint64_t mnmajor(uint32_t saddr, uint32_t cols) {
    return smem_desc(saddr, cols / 8u * 128u, 128u);
}

// Explicit features (host or device memory): a row's 96 floats are contiguous,
// so the tile is read as one run of float4.
__device__ __forceinline__ void stage_raw(const TrainArgs& A, unsigned char* smem, uint32_t tile, uint32_t tid) {
    const uint32_t rows = min(kRows, A.rows - tile * kRows);
    const float4* src = reinterpret_cast<const float4*>(A.raw_feats + (size_t)tile * kRows * kIn);
    float4 v[kRows * kIn / 4 / kEpilogueThreads];
#pragma unroll
    for (uint32_t i = 0; i < kRows * kIn / 4 / kEpilogueThreads; ++i) {
        const uint32_t e = tid + kEpilogueThreads * i;
        v[i] = e < rows * (kIn / 4) ? __ldcs(src + e) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    float4 tg = make_float4(0.f, 0.f, 0.f, 0.f);
    if (tid < rows) {
        const float* t = A.raw_targets + 3 * ((size_t)tile * kRows + tid);
        tg = make_float4(t[0], t[1], t[2], 1.0f);
    }
#pragma unroll
    for (uint32_t i = 0; i < kRows * kIn / 4 / kEpilogueThreads; ++i) {
        const uint32_t e = tid + kEpilogueThreads * i, r = e / (kIn / 4), c = e % (kIn / 4) * 4;
        *reinterpret_cast<uint2*>(smem + kSmX + canon_offset(r, c, kIn)) =
            make_uint2(bf16_bits(v[i].x) | (uint32_t)bf16_bits(v[i].y) << 16,
                       bf16_bits(v[i].z) | (uint32_t)bf16_bits(v[i].w) << 16);
    }
    if (tid < kRows) reinterpret_cast<float4*>(smem + kSmTgt)[tid] = tg;
}

// Row r's 48 features of one half (uniform in a warp: the halves differ in code)
// into the X array.
__device__ __forceinline__ void stage_inputs(const TrainArgs& A, unsigned char* smem, uint32_t tile, uint32_t count,
                                             uint32_t tid) {
    const uint32_t r = tid % kRows, half = tid / kRows;
    const uint32_t b = tile * kRows + r;
    uint16_t f[96];
    float4 tg = make_float4(0.f, 0.f, 0.f, 0.f);
    if (b < A.rows && count > 0) {
        const uint32_t si = pcg_hash(A.seed ^ pcg_hash(b)) % count;
        const CachePoint pt = A.samples[si].pt;
        encode_half(pt, A.net.lo, A.net.hi, (int)half, f);
        if (half == 0) tg = A.targets[si];
    } else {
#pragma unroll
        for (int i = 0; i < 96; ++i) f[i] = 0;
    }
    unsigned char* x = smem + kSmX;
    if (half == 0) {
#pragma unroll
        for (int j = 0; j < 6; ++j) {
            uint4 v;
            v.x = (uint32_t)f[8 * j] | ((uint32_t)f[8 * j + 1] << 16);
            v.y = (uint32_t)f[8 * j + 2] | ((uint32_t)f[8 * j + 3] << 16);
            v.z = (uint32_t)f[8 * j + 4] | ((uint32_t)f[8 * j + 5] << 16);
            v.w = (uint32_t)f[8 * j + 6] | ((uint32_t)f[8 * j + 7] << 16);
            *reinterpret_cast<uint4*>(x + canon_offset(r, 8 * j, kIn)) = v;
        }
        reinterpret_cast<float4*>(smem + kSmTgt)[r] = tg;
    } else {
#pragma unroll
        for (int j = 6; j < 12; ++j) {
            uint4 v;
            v.x = (uint32_t)f[8 * j] | ((uint32_t)f[8 * j + 1] << 16);
            v.y = (uint32_t)f[8 * j + 2] | ((uint32_t)f[8 * j + 3] << 16);
            v.z = (uint32_t)f[8 * j + 4] | ((uint32_t)f[8 * j + 5] << 16);
            v.w = (uint32_t)f[8 * j + 6] | ((uint32_t)f[8 * j + 7] << 16);
            *reinterpret_cast<uint4*>(x + canon_offset(r, 8 * j, kIn)) = v;
        }
    }
}

// Shared-memory writes -> visible to the next MMAs and bulk operations; true in
// every thread when `ok` is true in every thread.
__device__ __forceinline__ bool publish_smem(bool ok) {
    fence_smem_to_async();
    fence_before_sync();
    const bool bad = __syncthreads_or(!ok) != 0;
    fence_after_sync();
    return !bad;
}

// dW_l^T from tensor memory (lane = output, column = input) into its place in
// the parameters' order. Four warps: lanes 0..63 hold outputs, and each half of
// the warps takes half of the columns; a store's lanes are consecutive words.
template <int l>
__device__ __forceinline__ void flush_gradient(unsigned char* smem, uint32_t tmem, uint32_t quarter, uint32_t chalf,
                                               uint32_t row) {
    constexpr uint32_t F = LayerK(l), N = LayerN(l), kCols = F / 2;
    if (32 * quarter >= N) return;  // whole warp: lanes past the outputs are padding
    uint32_t v[kCols];
    const uint32_t at = tmem_addr(tmem, 32 * quarter, ColDW(l) + kCols * chalf);
#pragma unroll
    for (uint32_t j = 0; j < kCols; j += 16) tmem_ld16(at + j, v + j);
    tmem_ld_wait();
    float* G = reinterpret_cast<float*>(smem + kSmX) + ParamOffset(l) + kCols * chalf * N + row;
    if (row < N)
#pragma unroll
        for (uint32_t j = 0; j < kCols; ++j) G[j * N] = __uint_as_float(v[j]);
}

template <int l>
__device__ __forceinline__ void reduce_gradient(const TrainArgs& A, unsigned char* smem) {
    const uint32_t at = ParamOffset(l);
    bulk_reduce_add(A.net.grad + at, smem + kSmX + 4 * at, 4 * LayerK(l) * LayerN(l));
}

// One CTA, one tile: warps 0..7 stage the inputs and run the epilogues, warp 8
// issues the MMAs.
template <bool kRaw>
__global__ void __launch_bounds__(kThreads, 1) train_umma_kernel(const TrainArgs A) {
    extern __shared__ __align__(1024) unsigned char smem[];
    __shared__ uint64_t s_chain;  // Z_l and dH_l are complete
    __shared__ uint64_t s_dw;     // dW_l is complete
    __shared__ uint64_t s_mbar_w; // weight images in shared memory
    __shared__ uint32_t s_tmem, s_last;
    const uint32_t tid = threadIdx.x, lane = tid & 31;
    const uint32_t warp = __shfl_sync(0xFFFFFFFFu, tid >> 5, 0);  // (uniform for the compiler too)
    const bool issuer = warp == kEpilogueWarps;
    const uint32_t quarter = warp & 3, chalf = warp >> 2;
    const uint32_t row = 32 * quarter + lane;  // the tile row (tensor-memory lane) of this thread's epilogue
    const uint32_t sbase = smem_u32(smem);
    const uint32_t tile = blockIdx.x;
    double loss = 0.0;

    if (issuer) {
        if (lane == 0) {
            mbar_init(&s_chain, 1);
            mbar_init(&s_dw, 1);
            mbar_init(&s_mbar_w, 1);
            mbar_expect_tx(&s_mbar_w, 2 * (kUFwdElems + kUBwdElems));
            bulk_g2s(smem + kSmWf, A.net.ufwd, 2 * kUFwdElems, &s_mbar_w);
            bulk_g2s(smem + kSmWb, A.net.ubwd, 2 * kUBwdElems, &s_mbar_w);
        }
        __syncwarp();
        tmem_alloc(&s_tmem, kTmemCols);
    } else if constexpr (kRaw) {
        stage_raw(A, smem, tile, tid);
    } else {
        stage_inputs(A, smem, tile, A.count ? *A.count : 0u, tid);
    }
    publish_smem(true);
    const uint32_t tmem = s_tmem;
    // warp 0..7: waits for commit i of a barrier, at most kWaitLimit polls
    bool ok = true;
    auto wait = [&](uint64_t* mbar, uint32_t i) {
        if (!mbar_wait(mbar, i & 1u, kWaitLimit)) ok = false;
        fence_after_sync();
    };
    bool alive = true;
    uint32_t chain = 0, dws = 0;  // commits so far
    if (issuer) {
        ok = __all_sync(0xFFFFFFFFu, mbar_wait(&s_mbar_w, 0, kWaitLimit));
        if (!ok && lane == 0) mbar_arrive(&s_chain);  // the copies never landed: complete phase 0 without an MMA
    }
    // ---- forward ------------------------------------------------------------
#pragma unroll
    for (int l = 0; l < kLayers; ++l) {
        const uint32_t K = LayerK(l), N = UmmaN(l);
        if (issuer) {
            if (ok && elect_one()) {
                const uint32_t a0 = sbase + (l == 0 ? kSmX : kSmH + (l - 1) * kHBytes);
                const uint32_t b0 = sbase + kSmWf + 2 * UFwdOffset(l);
                const uint32_t idesc = instr_desc_bf16(128, N, false, false);
#pragma unroll
                for (uint32_t k = 0; k < K / 16; ++k)
                    mma_bf16(tmem + kColZ, kmajor(a0 + 256 * k, K), kmajor(b0 + 256 * k, K), idesc, k > 0);
                mma_commit(&s_chain);
            }
            __syncwarp();
        } else {
            wait(&s_chain, l);
            if (l + 1 < kLayers) {
                uint32_t v[32];
                tmem_ld16(tmem_addr(tmem, 32 * quarter, kColZ + 32 * chalf), v);
                tmem_ld16(tmem_addr(tmem, 32 * quarter, kColZ + 32 * chalf + 16), v + 16);
                tmem_ld_wait();
                unsigned char* h = smem + kSmH + l * kHBytes;
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    uint4 o;
                    o.x = bf16x2(fmaxf(__uint_as_float(v[8 * j]), 0.f), fmaxf(__uint_as_float(v[8 * j + 1]), 0.f));
                    o.y = bf16x2(fmaxf(__uint_as_float(v[8 * j + 2]), 0.f), fmaxf(__uint_as_float(v[8 * j + 3]), 0.f));
                    o.z = bf16x2(fmaxf(__uint_as_float(v[8 * j + 4]), 0.f), fmaxf(__uint_as_float(v[8 * j + 5]), 0.f));
                    o.w = bf16x2(fmaxf(__uint_as_float(v[8 * j + 6]), 0.f), fmaxf(__uint_as_float(v[8 * j + 7]), 0.f));
                    *reinterpret_cast<uint4*>(h + canon_offset(row, 32 * chalf + 8 * j, kWidth)) = o;
                }
            } else if (chalf == 0) {
                // outputs -> loss and its gradient dZ_5 ([128][16], columns 3.. zero)
                uint32_t v[16];
                tmem_ld16(tmem_addr(tmem, 32 * quarter, kColZ), v);
                tmem_ld_wait();
                const float4 tg = reinterpret_cast<const float4*>(smem + kSmTgt)[row];
                float g[3] = {0.f, 0.f, 0.f};
                if (tg.w > 0.0f) {
                    const float t3[3] = {tg.x, tg.y, tg.z};
#pragma unroll
                    for (int c = 0; c < 3; ++c) {
                        const float y = __uint_as_float(v[c]);
                        const float den = y * y + kLossEps;
                        const float d = y - t3[c];
                        loss += (double)(d * d / den);
                        g[c] = 2.0f * d / den * A.inv_norm;
                    }
                }
                unsigned char* dz = smem + DzBuffer(kLayers - 1);
                *reinterpret_cast<uint4*>(dz + canon_offset(row, 0, 16)) =
                    make_uint4(bf16x2(g[0], g[1]), bf16x2(g[2], 0.f), 0u, 0u);
                *reinterpret_cast<uint4*>(dz + canon_offset(row, 8, 16)) = make_uint4(0u, 0u, 0u, 0u);
            }
        }
        chain++;
        alive = publish_smem(ok);
        if (!alive) break;
    }
    // ---- backward -----------------------------------------------------------
    // Layer l's weight gradient is computed under the epilogue of its dH and
    // leaves under the next layer's GEMM: its copy overwrites the activations
    // it came from (the same place, kSmX + 4 * ParamOffset), which nothing
    // reads any more.
    auto backward = [&](auto layer) {
        constexpr int l = decltype(layer)::value;
        constexpr uint32_t F = LayerK(l), Nb = UmmaN(l);
        if (issuer) {
            if (elect_one()) {
                const uint32_t h0 = sbase + (l == 0 ? kSmX : kSmH + (l - 1) * kHBytes);
                const uint32_t dz0 = sbase + DzBuffer(l);
                if constexpr (l > 0) {
                    // dH_l = dZ_l W_l^T
                    const uint32_t b0 = sbase + kSmWb + 2 * UBwdOffset(l);
                    const uint32_t idesc_a = instr_desc_bf16(128, kWidth, false, false);
#pragma unroll
                    for (uint32_t k = 0; k < Nb / 16; ++k)
                        mma_bf16(tmem + kColZ, kmajor(dz0 + 256 * k, Nb), kmajor(b0 + 256 * k, Nb), idesc_a, k > 0);
                    mma_commit(&s_chain);
                }
                // dW_l^T = dZ_l^T H_l over the tile's rows
                const uint32_t idesc_w = instr_desc_bf16(128, F, true, true);
#pragma unroll
                for (uint32_t k = 0; k < kRows / 16; ++k)
                    mma_bf16(tmem + ColDW(l), mnmajor(dz0 + 2 * (Nb / 8 * 128) * k, Nb),
                             mnmajor(h0 + 2 * (F / 8 * 128) * k, F), idesc_w, k > 0);
                mma_commit(&s_dw);
            }
            __syncwarp();
        } else {
            if constexpr (l + 1 < kLayers) flush_gradient<l + 1>(smem, tmem, quarter, chalf, row);
            if constexpr (l > 0) {
                // dZ_{l-1} = dH_l masked by H_l > 0 (BF16)
                wait(&s_chain, 2 * kLayers - 1 - l);
                uint32_t v[32];
                tmem_ld16(tmem_addr(tmem, 32 * quarter, kColZ + 32 * chalf), v);
                tmem_ld16(tmem_addr(tmem, 32 * quarter, kColZ + 32 * chalf + 16), v + 16);
                tmem_ld_wait();
                const unsigned char* h = smem + kSmH + (l - 1) * kHBytes;
                unsigned char* dz = smem + DzBuffer(l - 1);
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const uint32_t off = canon_offset(row, 32 * chalf + 8 * j, kWidth);
                    const uint4 a = *reinterpret_cast<const uint4*>(h + off);
                    const uint32_t aw[4] = {a.x, a.y, a.z, a.w};
                    uint32_t o[4];
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        const float d0 = bf16_lo(aw[e]) > 0.f ? __uint_as_float(v[8 * j + 2 * e]) : 0.f;
                        const float d1 = bf16_hi(aw[e]) > 0.f ? __uint_as_float(v[8 * j + 2 * e + 1]) : 0.f;
                        o[e] = bf16x2(d0, d1);
                    }
                    *reinterpret_cast<uint4*>(dz + off) = make_uint4(o[0], o[1], o[2], o[3]);
                }
            }
            // (every commit is waited for before the barrier that lets the next
            // one be issued: a parity tells only neighbours apart)
            wait(&s_dw, kLayers - 1 - l);
            if constexpr (l == 0) flush_gradient<0>(smem, tmem, quarter, chalf, row);
        }
        alive = publish_smem(ok);
        if (alive && tid == 0) {
            if constexpr (l + 1 < kLayers) reduce_gradient<l + 1>(A, smem);
            if constexpr (l == 0) reduce_gradient<0>(A, smem);
        }
    };
    if (alive) backward(std::integral_constant<int, 5>{}), chain++, dws++;
    if (alive) backward(std::integral_constant<int, 4>{}), chain++, dws++;
    if (alive) backward(std::integral_constant<int, 3>{}), chain++, dws++;
    if (alive) backward(std::integral_constant<int, 2>{}), chain++, dws++;
    if (alive) backward(std::integral_constant<int, 1>{}), chain++, dws++;
    if (alive) backward(std::integral_constant<int, 0>{}), dws++;
    static_assert(kLayers == 6, "one call per layer");
    if (tid == 0) bulk_reduce_wait();
    if (!alive) {
        if (lane == 0 && A.status) atomicOr(A.status, Foundation::RT::kStatusTimeout);
        // let the MMAs of the unfinished phase and the weight copies drain
        // (bounded) before the tensor memory is released
        if (tid == 0) {
            (void)mbar_wait(&s_chain, (chain - 1) & 1u, kWaitLimit);
            if (dws) (void)mbar_wait(&s_dw, (dws - 1) & 1u, kWaitLimit);
            (void)mbar_wait(&s_mbar_w, 0, kWaitLimit);
        }
    }
    for (int o = 16; o > 0; o >>= 1) loss += __shfl_down_sync(0xFFFFFFFFu, loss, o);
    if (lane == 0 && A.net.loss && loss != 0.0) atomicAdd(A.net.loss, loss);
    fence_before_sync();
    __syncthreads();
    if (issuer) tmem_dealloc(tmem, kTmemCols);
    if constexpr (kRaw) {
        // The CTA that finishes last copies the sums out. (A call for 16,384 /
        // 1,000 samples with two copies after the kernel 77.4 / 48.7 us, with
        // this 70.6 / 39.8; with one load and store at a time 87.2 / 57.0.)
        if (A.out_grad) {
            if (tid == 0) {
                fence_proxies();
                __threadfence();
                s_last = atomicAdd(reinterpret_cast<uint32_t*>(A.net.loss + 1), 1u) + 1u == gridDim.x;
            }
            __syncthreads();
            if (s_last) {
                __threadfence();
                fence_proxies();
                // all of a thread's loads before its first store
                constexpr uint32_t kVecs = kNumParams / 4, kEach = (kVecs + kThreads - 1) / kThreads;
                float4 g[kEach];
#pragma unroll
                for (uint32_t i = 0; i < kEach; ++i)
                    if (tid + kThreads * i < kVecs)
                        g[i] = __ldcg(reinterpret_cast<const float4*>(A.net.grad) + tid + kThreads * i);
                if (tid == 0) *A.out_loss = __ldcg(A.net.loss);
#pragma unroll
                for (uint32_t i = 0; i < kEach; ++i)
                    if (tid + kThreads * i < kVecs)
                        __stcs(reinterpret_cast<float4*>(A.out_grad) + tid + kThreads * i, g[i]);
            }
        }
    }
}

template <typename K>
cudaError_t allow_smem(K kernel) {
    return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmBytes);
}

}  // namespace

size_t TrainSmemBytes() { return kSmBytes; }

// One CTA per 128-row tile (a single wave for the 16,384-sample batches).
static int train_grid(uint32_t rows) { return (int)((rows + kRows - 1) / kRows); }

cudaError_t LaunchTrainUmma(const Net& net, const TrainSample* smp, const float4* targets, const uint32_t* count,
                            uint32_t batch, uint64_t seed, uint32_t* status, cudaStream_t s) {
    cudaError_t e = allow_smem(train_umma_kernel<false>);
    if (e != cudaSuccess) return e;
    e = cudaMemsetAsync(net.loss, 0, sizeof(double), s);
    if (e != cudaSuccess) return e;
    if (batch == 0) return cudaSuccess;
    TrainArgs A{};
    A.net = net;
    A.samples = smp;
    A.targets = targets;
    A.count = count;
    A.rows = batch;
    A.seed = (uint32_t)(seed ^ (seed >> 32));
    A.inv_norm = 1.0f / (3.0f * (float)batch);
    A.status = status;
    train_umma_kernel<false><<<train_grid(batch), kThreads, kSmBytes, s>>>(A);
    return cudaGetLastError();
}

cudaError_t GradRaw(Net& net, const float* feats, const float* targets, uint32_t n, float* out_grad,
                    double* out_loss, uint32_t* status, cudaStream_t s) {
    cudaError_t e = allow_smem(train_umma_kernel<true>);
    if (e != cudaSuccess) return e;
    net.grad_left = true;
    // (the loss may lie directly behind the gradient: one launch clears both)
    const bool one = reinterpret_cast<char*>(net.loss) == reinterpret_cast<char*>(net.grad + kNumParams);
    const size_t sums = 2 * sizeof(double);  // loss and CTA count
    e = cudaMemsetAsync(net.grad, 0, sizeof(float) * kNumParams + (one ? sums : 0), s);
    if (e == cudaSuccess && !one) e = cudaMemsetAsync(net.loss, 0, sums, s);
    if (e != cudaSuccess || n == 0) return e;
    TrainArgs A{};
    A.net = net;
    A.raw_feats = feats;
    A.raw_targets = targets;
    A.out_grad = out_grad;
    A.out_loss = out_loss;
    A.rows = n;
    A.inv_norm = 1.0f / (3.0f * (float)n);
    A.status = status;
    train_umma_kernel<true><<<train_grid(n), kThreads, kSmBytes, s>>>(A);
    return cudaGetLastError();
}

}  // namespace NRC
}  // namespace Foundation
