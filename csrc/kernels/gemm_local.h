// Argument blocks of the fused linear layer for ranks that share one GPU (gemm_local.cu).
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "../comm/layout.h"

namespace yali {

constexpr uint32_t kLocalGemmPairCols = 256;   // columns of an item: rows of W on the M side of the MMA, 128 per CTA
constexpr uint32_t kLocalGemmUnitCols = 128;   // columns of one CTA, announced together
constexpr uint32_t kLocalGemmMaxTokens = 256;  // rows of x on the N side
constexpr uint32_t kLocalGemmMaxSplit = 8;
constexpr int kLocalGemmThreads = 384;         // eight epilogue warps, TMA, MMA, announcer, one idle
constexpr int kLocalLinearNormThreads = 256;   // one row; up to two 16-byte vectors per thread: N <= 4096

// T rows in `tiles` token tiles of `tokens` (a multiple of 32, at most 256), the k-blocks of all ranks (one after the
// other) in `nsplit` runs of `kper`.
struct LocalGemmShape {
    uint32_t tiles, tokens, nsplit, kper;
};

struct alignas(64) LocalGemmArgs {
    CUtensorMap tmap_x[kMaxRanks];  // x_r [T, K] bf16, box 64 x tokens / 2, 128-byte swizzle
    CUtensorMap tmap_w[kMaxRanks];  // W_r [N, K] bf16, box 64 x 128, 128-byte swizzle
    CommView cv;                    // rank 0's
    char* sums;                     // [nsplit][T, N] bf16
    uint32_t T, N;
    uint32_t kb_rank;               // k-blocks (of 64) of one rank
    uint32_t kb_total;              // of all ranks
    LocalGemmShape s;
};

struct LocalLinearNormArgs {
    CommView cv;
    const char* sums;
    const void* residual[kMaxRanks];  // [T, N]; entries may be nullptr
    void* residual_out[kMaxRanks];    // [T, N]; entries may be nullptr
    const void* weight[kMaxRanks];    // [N]
    void* out[kMaxRanks];             // [T, N]
    uint32_t T, N, world;
    LocalGemmShape s;
    float eps;
};

const void* LocalGemmKernel();
uint32_t LocalGemmSmemBytes();
// `ranks_per_cta`: 1, 2 or 4.
const void* LocalLinearNormKernel(uint32_t N, int ranks_per_cta);

}  // namespace yali
