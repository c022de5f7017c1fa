// Argument block and host entry points of the fused row-parallel GEMM +
// all-reduce + residual + RMSNorm kernel (gemm_ar_rmsnorm.cu).
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "../comm/layout.h"

namespace yali {

// The tile that FusedLinearTileSplit and FusedLinearCounts count in.
constexpr int kGemmTileM = 128;
constexpr int kGemmTileN = 256;
// Tile of the kernel: 256 columns of the output (the M side of the MMA: rows of W, 128 per CTA of a pair) x up to
// 256 tokens (the N side: rows of x, half of them per CTA).
constexpr uint32_t kGemmPairCols = 256;
constexpr uint32_t kGemmUnitCols = 128;    // columns of one CTA: the unit in which partial sums are announced
constexpr uint32_t kGemmMaxTokens = 256;   // tokens of a tile
constexpr int kGemmThreads = 640;          // eight epilogue warps, eight row warps, TMA, MMA, announcer and row-producer warp
constexpr uint32_t kGemmMaxRowVecs = 512;  // 16-byte vectors of a row: N <= 4096

// How the T rows are cut into token tiles: `domains` runs of `span` rows (one per row owner, or one run of all
// rows), each cut into `tiles` tiles of `tokens` rows (a multiple of 32; the last ones may be short or empty).
// A pair of CTAs walks the items (token tile, 256 columns, K split) of its rank; `group` token tiles are
// walked together column by column, so that they read a slice of W at about the same time.
struct GemmTiling {
    uint32_t span, domains, tiles, tokens, group;
};

// One work item of a pair.
struct GemmItem {
    uint32_t tile;    // token tile, numbered alike on every rank
    uint32_t t0, nt;  // its rows [t0, t0 + nt); nt = 0: nothing to do
    uint32_t col_tile, split;
};
// Items of a rank in walking order: groups of token tiles, in a group column tile by column tile, token tile by
// token tile, split by split.  With one domain per owner the k-th tile of every owner comes before the
// (k+1)-th, starting with the right-hand neighbour's: at any moment the ranks push to different owners, and
// every owner's rows complete bit by bit.  (The host-thread model walks them, too.)
__host__ __device__ inline GemmItem GemmItemAt(const GemmTiling& t, uint32_t T, uint32_t rank, uint32_t i, uint32_t ncol,
                                               uint32_t ks_shift) {
    GemmItem it;
    it.split = i & ((1u << ks_shift) - 1u);
    i >>= ks_shift;
    const uint32_t ntt = t.domains * t.tiles, per_group = t.group * ncol;
    const uint32_t g = i / per_group, in_g = i - g * per_group;
    const uint32_t left = ntt - g * t.group, here = t.group < left ? t.group : left;  // the last group may be smaller
    it.col_tile = in_g / here;
    const uint32_t pos = g * t.group + in_g % here;
    const uint32_t b = pos / t.domains;
    uint32_t dom = pos - b * t.domains;
    if (t.domains > 1) dom = (dom + rank + 1) % t.domains;
    it.tile = dom * t.tiles + b;
    it.t0 = dom * t.span + b * t.tokens;
    uint32_t end = (dom + 1) * t.span;
    end = end < T ? end : T;
    end = end < it.t0 + t.tokens ? end : it.t0 + t.tokens;
    it.nt = end > it.t0 ? end - it.t0 : 0u;
    return it;
}
// The token tile of a row.
__host__ __device__ inline uint32_t GemmTileOfRow(const GemmTiling& t, uint32_t row) {
    const uint32_t dom = t.domains > 1 ? row / t.span : 0u;
    return dom * t.tiles + (row - dom * t.span) / t.tokens;
}

struct alignas(64) GemmArArgs {
    CUtensorMap tmap_x;  // x  [T, K] bf16, box 64 x tokens / 2, 128-byte swizzle (rows beyond T read as zeros)
    CUtensorMap tmap_w;  // W  [N, K] bf16, box 64 x 128, 128-byte swizzle (rows beyond N read as zeros)
    CommView cv;
    const void* residual;     // [T, N] bf16 or nullptr
    void* residual_out;       // [T, N] bf16 or nullptr (sum + residual), this rank's copy
    void* residual_out_all[kMaxRanks];  // two-shot: every rank's residual_out (the row owner writes all copies)
    const void* norm_weight;  // [N] bf16
    void* out[kMaxRanks];     // every rank's output [T, N] (two-shot writes all, one-shot only its own)
    uint32_t T, N, K;
    GemmTiling tl;
    uint32_t rows_per_owner;  // two-shot: rows normalised by each rank
    uint32_t oneshot;         // 1: every rank receives all partial rows and normalises all of them
    uint32_t ksplit;          // one-shot, few tiles: pairs that share the K extent of a tile (1, 2 or 4; world x ksplit <= 8)
    uint32_t kper;            // k-blocks (of 64) per split
    uint32_t one_gpu;         // all ranks' heaps are this GPU's memory: announcements need GPU scope only
    uint32_t done_inc[kMaxRanks];  // per owner: rows it delivers to every rank's output in this call
    float eps;
    // NVLS form of the two-shot (nvls != 0): every rank keeps its partial rows in its OWN landing
    // zone, the owner of a row sums all ranks' copies in the switch (multimem.ld_reduce) and
    // writes the normalised row to every rank with one multimem.st through these addresses.
    // out_mc alone (nvls == 0) keeps the peer pushes of phase 1 and only delivers through the switch.
    uint32_t nvls;
    char* out_mc;           // multicast address of out, or nullptr: write every rank's copy with peer stores
    char* residual_out_mc;  // multicast address of residual_out, or nullptr
    unsigned long long* trace;  // optional: 8 x %globaltimer of CTA 0 at the phase boundaries (debugging aid)
};

struct GemmArEmuArgs {
    GemmArArgs r[kMaxRanks];
};

const void* GemmArKernel(bool emu);
uint32_t GemmArSmemBytes();

// ---- few-token form (gemm_ar_decode.cu): 128 x 256 tiles with the K extent split over CTAs, partial rows
// travel as flag-in-data lines in landing tiles of 32 columns
constexpr int kGemmDecodeTileN = 32;
constexpr int kGemmDecodeMmaN = 256;
constexpr uint32_t kGemmDecodeMaxSplit = 8;   // K splits per tile (sources per rank of the reduction)
constexpr int kGemmDecodeThreads = 512;       // TMA warp, MMA warp, eight epilogue warps; all 16 warps reduce rows
constexpr int kGemmDecodeVecPerThread = 1;    // N <= 512 threads * 8 bf16 = 4096
constexpr uint32_t kGemmDecodeMaxRows = 64;   // two TMEM lane quarters

struct alignas(64) GemmDecodeArgs {
    CUtensorMap tmap_a;  // x  [T, K] bf16, box 64 x a_box_rows (rows beyond T read as zeros), 128-byte swizzle
    CUtensorMap tmap_b;  // W  [N, K] bf16, box 64 x tile_n (rows beyond N read as zeros), 128-byte swizzle
    CommView cv;
    const void* residual;     // [T, N] bf16 or nullptr
    void* residual_out;       // [T, N] bf16 or nullptr
    const void* norm_weight;  // [N] bf16
    void* out;                // [T, N] bf16, this rank's
    uint32_t T, N, K;
    uint32_t a_box_rows;  // rows of x one TMA copy brings in: 8, 16, 32 or 64 (the smallest that holds T)
    uint32_t tile_n;      // columns of a tile = N of the MMA and rows of the box of W: 128 or 256
    uint32_t ksplit;      // CTAs that share the K extent of one tile (1, 2, 4 or 8)
    uint32_t kper;        // k-blocks (of 64) per split: split ks takes [ks * kper, min(K / 64, (ks + 1) * kper))
    float eps;
    unsigned long long* trace;  // optional: %globaltimer of CTA 0 at the phase boundaries
};
struct GemmDecodeEmuArgs {
    GemmDecodeArgs r[kMaxRanks];
};
const void* GemmDecodeKernel(bool emu);
uint32_t GemmDecodeSmemBytes();

}  // namespace yali
