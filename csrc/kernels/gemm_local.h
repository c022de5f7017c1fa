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
constexpr int kLocalGemmThreads = 384;         // eight epilogue warps, TMA, MMA, announcer, prefetch
// Elements of all ranks' outputs up to which the rows of a call release the kernel behind it when they start.  With more, the rows keep
// HBM busy by themselves and W on its way only delays them.  Back to back, without / with, us: 2 ranks, K = 2048, N = 4096: T =
// 400 26.0 / 24.0, T = 1400 (11 Mi) 60.1 / 61.0, T = 2048 (16 Mi) 77.7 / 78.7; 4 ranks: K = 1024, N = 2048, T = 1024 (8 Mi)
// 33.2 / 32.8, K = 2048, N = 4096, T = 600 (9.4 Mi) 61.4 / 60.0; 8 ranks, N = 4096: K = 512, T = 256 (8 Mi) 27.7 / 28.2, K = 1792,
// T = 300 (9.4 Mi) 60.5 / 59.5, T = 350 (11 Mi) 67.3 / 66.2.  The kernel behind asks for its W whatever its own size: large calls
// behind small ones 80.2 / 78.0, 68.6 / 67.9, 90.6 / 91.3 with / without such a limit, large behind large level.
constexpr uint64_t kLocalLinearEarly = 12ull << 20;
constexpr int kLocalLinearNormThreads = 256;   // at most; one row, one or two 16-byte vectors per thread: N <= 4096
constexpr int LocalLinearNormVectors(uint32_t N) { return N <= 8u * kLocalLinearNormThreads ? 1 : 2; }
// No more warps than a row needs.  A unit of the row kernel is a chain of latencies, so what counts is how many are in flight.
constexpr int LocalLinearNormThreads(uint32_t N) {
    const uint32_t per_warp = 32u * 8u * LocalLinearNormVectors(N);
    return 32 * static_cast<int>((N + per_warp - 1) / per_warp);
}

// T rows in `tiles` token tiles of `tokens` (a multiple of 32, at most 256), the k-blocks of all ranks (one rank after the
// other) in `nsplit` runs of `kper`.
struct LocalGemmShape {
    uint32_t tiles, tokens, nsplit, kper;
};

struct alignas(64) LocalGemmArgs {
    CUtensorMap tmap_x[kMaxRanks];  // x_r [T, K] bf16, box 64 x tokens / 2, 128-byte swizzle
    CUtensorMap tmap_w[kMaxRanks];  // W_r [N, K] bf16, box 64 x 128, 128-byte swizzle
    CommView cv;                    // rank 0's
    char* sums;                     // [nsplit][T, N] bf16, or lines of twice the size
    uint32_t lines;                 // 1: flag-in-data lines {2 bf16, call, 2 bf16, ~call} instead of plain sums and flags
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
    uint32_t by_groups;  // ceil(2^32 / groups of ranks): the row of a unit without a division
    uint32_t early;  // at most kLocalLinearEarly elements: the next kernel may start under these rows
    float eps;
};

// Registers per thread of the row kernel.  Up to 72, two CTAs of 256 threads fit beside the GEMM's, so that up to two units per SM are there,
// with their residuals, when the sums come; CTAs that start when the GEMM's have left are 2.5 us later (8 ranks, 32 x 1792 x 4096 31.0
// with 128 registers, 26.9 with 72).  `slim`, where there are two instances: one rank, the other one asks for the lines of four K
// splits at a time; two ranks, two vectors, one split: the other one, with three CTAs per SM instead of four, asks for the weights at once.
// Two vectors of two ranks and several splits do not fit 72 (spills: 50 -> 55 us).
constexpr int LocalLinearNormRegs(int vectors, int ranks_per_cta, bool split, bool slim) {
    if (ranks_per_cta == 1) return slim ? 72 : vectors == 1 ? 104 : 144;
    if (ranks_per_cta == 2) return !split ? (vectors == 1 || slim ? 64 : 72) : vectors == 1 ? 72 : 96;
    return !split ? 72 : 96;
}

const void* LocalGemmKernel();
uint32_t LocalGemmSmemBytes();
// `ranks_per_cta`: 1, 2 or (rows of one vector per thread) 4; `split`: more than one K split; `lines` (one rank per CTA, split):
// flag-in-data sums.
const void* LocalLinearNormKernel(uint32_t N, int ranks_per_cta, bool split, bool lines, bool slim);

}  // namespace yali
