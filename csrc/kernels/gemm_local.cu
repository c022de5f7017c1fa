// The fused linear layer of a group whose ranks all live on ONE GPU (emulated ranks):
//
//     out_r = RMSNorm(residual_r + sum_q x_q @ W_q^T) * norm_weight_r          for every rank r
//
// One launch sees every rank's operands, so the sum over the ranks is a sum over k-blocks: the GEMM runs once over the
// concatenated K extent of all ranks and adds in the fp32 accumulator of the tensor cores.  No partial rows travel
// between ranks, no rank waits for another one.  Two kernels:
//
//   local_gemm_kernel          persistent pairs of CTAs (tcgen05.mma.cta_group::2), one CTA per SM; an item is (token
//                              tile, 256 columns, K split) and leaves bf16 sums [split][T, N] in memory;
//   local_linear_norm_kernel   one CTA per row (and group of ranks): adds the splits and the residual, normalises, writes
//                              out and residual_out.
//
// The second kernel starts while the first one runs (griddepcontrol.launch_dependents, issued by every CTA of the first
// one when it starts: all of them are resident by then, so whoever waits for them here waits for running CTAs),
// and its CTAs wait for the flags of their token tile: rows are finished under the GEMM of later tiles.
//
// The pair computes the transposed tile, W on the M side: a tile can then be any multiple of 32 tokens wide, and each CTA
// loads 128 rows of W and half of the tokens per 64-deep k-block.  The threads that issue TMA and MMA are picked
// by elect.sync (behind a lane test the compiler wraps each of these instructions in a loop over the active
// threads: 540 instead of 390 cycles per k-block of 160 tokens).
//
// Calls that follow one another overlap: the row kernel lets the kernel behind it start when all of its own CTAs have, and where that
// is the next call's GEMM, it sets up and asks L2 for its first k-blocks of W before it waits for the rows.  In a graph, weights beyond
// L2, without / with, us: 2 ranks: K = 1024, N = 3072, T = 45 10.8 / 8.3; K = 2048, N = 4096: T = 8 12.3 / 10.1, T = 64 14.7 / 12.7,
// T = 400 26.0 / 23.4.  kLocalLinearEarly says up to where.
//
// Bound by the tensor cores at the clock they leave (2 ranks, T = 2048, K = 2048: the GEMM takes 55 us in the profiler, 1.24
// PFLOP/s), and by writing the rows that complete with the last tiles (4.6 - 5.3 TB/s of stores); by reading W from HBM
// for few tokens.  Measured per call, ranks on one B200, N = 4096, inputs beyond L2, against the exchange of bf16 partial
// rows in one cooperative launch (gemm_ar_rmsnorm.cu, gemm_ar_decode.cu), us back to back / in single bursts of 20 calls,
// where the clock stays up: 2 ranks, K = 2048: T = 8 16.4 -> 12.0 / 15.3 -> 11.9, T = 128 26.7 -> 17.3 / 24.9 -> 17.3,
// T = 2048 85 -> 76 / 75 -> 66; 8 ranks: K = 1792, T = 300 69 -> 57 / 67 -> 53; K = 512, T = 2048 179 -> 130 / 177 -> 112.
//
// Parity: none in the reference (it has no GEMM, no fused op and no tensor-core code).
#include <cuda.h>

#include "gemm_local.h"
#include "tc_common.cuh"

namespace yali {

namespace {

constexpr int BK = 64;                        // BK bf16 = one 128-byte swizzle row
constexpr uint32_t kWBytes = 128 * BK * 2;    // one CTA's half of the W operand of a stage
constexpr uint32_t kRingBytes = 192 * 1024;   // operand stages: 6 of 32 KB (256 tokens) to 10 of 18 KB (32 tokens)
constexpr int kMaxStages = 12;
constexpr uint32_t kSmemBytes = kRingBytes + 1024;  // + slack to align the base
constexpr uint32_t kTmemCols = 2 * kLocalGemmMaxTokens;  // two accumulators: all of TMEM
constexpr uint32_t kEpiChunk = 32;                              // tokens an epilogue group moves at a time
constexpr uint32_t kEpiBufBytes = kEpiChunk * 64;  // 2 KiB per warp: 32 columns of a chunk
constexpr int kEpiGroups = 2, kEpilogueWarps = 4 * kEpiGroups;
constexpr int kTmaWarp = 8, kMmaWarp = 9, kAnnounceWarp = 10, kPrefetchWarp = 11;
constexpr uint32_t kNumberBarrier = 1;  // named barrier: the announcer has read the call number, the epilogue warps use it
constexpr uint32_t kPrefetchBlocks = 8;  // how far the prefetch warp runs ahead of the loads, in k-blocks
static_assert(kTmemCols == 512 && kLocalGemmThreads == 32 * (kPrefetchWarp + 1), "one CTA per SM");
static_assert(kSmemBytes + kEpilogueWarps * kEpiBufBytes + 1024 <= 216 * 1024, "leaves room for CTAs of the second kernel");

struct Item {
    uint32_t tile;  // token tile
    uint32_t col_tile, split;
    uint32_t kb_begin, kb_end;
};
// The k-th item of a pair; false: no more.  Token tile by token tile, so that rows complete early; items in flight together
// read the same stretch of K.
__device__ __forceinline__ bool item_at(const LocalGemmArgs& a, uint32_t k, uint32_t pair, uint32_t npairs, uint32_t ncol, Item* it) {
    const uint32_t i = pair + k * npairs, per_tile = ncol * a.s.nsplit;
    if (i >= a.s.tiles * per_tile) return false;
    it->tile = i / per_tile;
    const uint32_t in_tile = i - it->tile * per_tile;
    it->split = in_tile / ncol;
    it->col_tile = in_tile - it->split * ncol;
    it->kb_begin = it->split * a.s.kper;
    it->kb_end = min(a.kb_total, it->kb_begin + a.s.kper);
    return true;
}

struct Shared {
    __align__(8) uint64_t full_bar[kMaxStages], empty_bar[kMaxStages], tmem_full_bar[2], tmem_empty_bar[2];
    __align__(8) uint64_t stored_bar[2], announced_bar[2];  // epilogue warps -> announcer warp and back
    __align__(8) uint64_t drain_bar;  // all MMAs have finished
    uint32_t tmem, epoch;      // epoch: this call's number
    volatile uint32_t loaded;  // k-blocks whose loads have been issued
    volatile int abort;
};

}  // namespace

__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kLocalGemmThreads, 1)
    local_gemm_kernel(const __grid_constant__ LocalGemmArgs a) {
    extern __shared__ uint8_t smem_raw[];
    __shared__ Shared s;
    __shared__ __align__(128) uint8_t s_epi[kEpilogueWarps][kEpiBufBytes];

    const CommView& cv = a.cv;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t cta = blockIdx.x, half = ptx::cluster_cta_rank();
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    const uint32_t ncol = (a.N + kLocalGemmPairCols - 1) / kLocalGemmPairCols;
    const uint32_t pair = cta >> 1, npairs = gridDim.x >> 1;
    const uint32_t xbytes = a.s.tokens / 2 * (BK * 2);  // one CTA's half of the token operand of a stage: whole KiB
    const uint32_t stage_bytes = kWBytes + xbytes;
    const uint32_t stages = min(kRingBytes / stage_bytes, static_cast<uint32_t>(kMaxStages));
    // Nothing up to the wait depends on earlier kernels: it runs under the end of the one in front.
    uint32_t fetched = 0;  // prefetch warp: k-blocks of W that are on their way into L2 already
    if (warp == kPrefetchWarp) {
        // The rows of the call in front leave HBM time, and what this call waits for first is W.  It is no more than asked for
        // here: should the kernel in front still be writing it, the loads behind the wait see that.  Beside the set-up and not
        // in front of it: this warp has nothing to set up, arrives at once and does not hold up the others.  Graph of calls, 2
        // ranks, T = 8, K = 2048, N = 4096, W in L2 / partly / beyond it, us: no overlap of calls 8.7 / 11.6 / 12.3, without
        // this 7.65 / 10.1 / 10.75, in front of the set-up 8.7 / 9.7 / 9.95, behind it 7.9 / 9.8 / 10.35, here 7.7 / 9.3 /
        // 10.1.  One call after which the host waits, in that order: 21.9, 22.0, 23.3, 22.5, 22.25.
        ptx::cluster_arrive();
        if (ptx::elect_one()) {
            Item it;
            if (item_at(a, 0, pair, npairs, ncol, &it) && it.tile == 0) {
                const int wrow = it.col_tile * kLocalGemmPairCols + half * kLocalGemmUnitCols;
                uint32_t rank = it.kb_begin / a.kb_rank, kb = it.kb_begin - rank * a.kb_rank;
                for (uint32_t g = it.kb_begin; g < it.kb_end && fetched < stages + kPrefetchBlocks; ++g, ++fetched) {
                    ptx::tma_prefetch_2d(&a.tmap_w[rank], kb * BK, wrow);
                    if (++kb == a.kb_rank) kb = 0, ++rank;
                }
            }
        }
        __syncwarp();
    } else {
        if (tid == 64) {
            s.abort = 0;
            s.loaded = 0;
            for (int i = 0; i < kMaxStages; ++i) {
                ptx::mbar_init(&s.full_bar[i], 1);
                ptx::mbar_init(&s.empty_bar[i], 1);
            }
            for (int b = 0; b < 2; ++b) {
                ptx::mbar_init(&s.tmem_full_bar[b], 1);
                ptx::mbar_init(&s.tmem_empty_bar[b], 2 * kEpilogueWarps);  // the epilogue warps of both CTAs
                ptx::mbar_init(&s.stored_bar[b], kEpilogueWarps);
                ptx::mbar_init(&s.announced_bar[b], 1);
            }
            ptx::mbar_init(&s.drain_bar, 1);
            ptx::mbar_fence_init();
            ptx::tma_prefetch_desc(&a.tmap_w[0]);
            ptx::tma_prefetch_desc(&a.tmap_x[0]);
        }
        if (warp == kMmaWarp) {
            ptx::tmem_alloc_pair(&s.tmem, kTmemCols);
            ptx::tmem_relinquish_pair();
        }
        ptx::tc_fence_before_sync();
        __syncwarp();
        ptx::cluster_arrive();
    }
    ptx::cluster_wait();  // barriers and TMEM are ready, in both CTAs
    ptx::tc_fence_after_sync();
    const uint32_t tmem = s.tmem;
    // In this order: the row kernel behind does not wait for the kernels in front of this one.  It reads its call number, the unit counter
    // and the call's inputs as soon as it starts, which is right because some thread of every CTA here has been through its wait.
    ptx::grid_dependency_wait();
    ptx::grid_launch_dependents();
    const uint64_t deadline = ptx::globaltimer() + cv.timeout_ns;

    if (warp == kTmaWarp) {
        if (ptx::elect_one()) {
            uint32_t st = 0, round = 0, loaded = 0;
            Item it;
            for (uint32_t i = 0; !s.abort && item_at(a, i, pair, npairs, ncol, &it); ++i) {
                const int wrow = it.col_tile * kLocalGemmPairCols + half * kLocalGemmUnitCols;
                const int xrow = it.tile * a.s.tokens + half * (a.s.tokens / 2);
                uint32_t rank = it.kb_begin / a.kb_rank, kb = it.kb_begin - rank * a.kb_rank;  // k-block of that rank
                for (uint32_t g = it.kb_begin; g < it.kb_end; ++g) {
                    if (!wait_bar(&s.empty_bar[st], (round & 1u) ^ 1u, deadline, &s.abort)) {
                        if (!s.abort) report_timeout(cv, kSiteMbar, rank, cta, 1, g);
                        s.abort = 1;
                        break;
                    }
                    // Both halves are counted on the leader's barrier, which its own producer arms.
                    if (half == 0) ptx::mbar_expect_tx(&s.full_bar[st], 2 * stage_bytes);
                    const uint32_t bar = ptx::mapa_u32(&s.full_bar[st], 0);
                    uint8_t* stage = smem + st * stage_bytes;
                    ptx::tma_load_2d_pair(stage, &a.tmap_w[rank], kb * BK, wrow, bar);
                    ptx::tma_load_2d_pair(stage + kWBytes, &a.tmap_x[rank], kb * BK, xrow, bar);
                    s.loaded = ++loaded;
                    if (++kb == a.kb_rank) kb = 0, ++rank;
                    if (++st == stages) st = 0, ++round;
                }
            }
            s.loaded = 0x7fffffffu;  // nothing left to run ahead of
            // The MMAs' releases of the last stages arrive here from the leader: none may be under way when this CTA
            // leaves.
            bool up = !s.abort;
            for (uint32_t k = 0; k < stages && up; ++k) {
                up = wait_bar(&s.empty_bar[st], (round & 1u) ^ 1u, deadline, &s.abort);
                if (++st == stages) st = 0, ++round;
            }
            if (!up) {
                // The time ran out in mid-work.  The leader's barriers count the loads of both CTAs; what this one
                // has issued beyond the leader, nobody counts.
                s.abort = 1;
                if (half == 0) mbar_drain_ring(s.full_bar, stages, loaded);
                else
                    for (const uint64_t until = ptx::globaltimer() + kDrainNs; ptx::globaltimer() < until;) ptx::nanosleep(1000);
            }
            if (loaded > 0) mbar_drain(&s.drain_bar, 0);
        }
    } else if (warp == kMmaWarp) {
        if (half == 0 && ptx::elect_one()) {
            const uint32_t idesc = mma_idesc_bf16(kLocalGemmPairCols, a.s.tokens);
            uint32_t st = 0, round = 0, n = 0;
            Item it;
            for (; !s.abort && item_at(a, n, pair, npairs, ncol, &it); ++n) {
                const uint32_t b = n & 1u;
                if (!wait_bar(&s.tmem_empty_bar[b], ((n >> 1) & 1u) ^ 1u, deadline, &s.abort)) {
                    if (!s.abort) report_timeout(cv, kSiteMbar, 0, cta, 4, n);
                    s.abort = 1;
                    break;
                }
                ptx::tc_fence_after_sync();
                const uint32_t d_tmem = tmem + b * kLocalGemmMaxTokens;
                for (uint32_t g = it.kb_begin; g < it.kb_end; ++g) {
                    if (!wait_bar(&s.full_bar[st], round & 1u, deadline, &s.abort)) {
                        if (!s.abort) report_timeout(cv, kSiteMbar, 0, cta, 2, g);
                        s.abort = 1;
                        break;
                    }
                    ptx::tc_fence_after_sync();
                    const uint32_t addr = ptx::smem_u32(smem + st * stage_bytes);
                    const uint64_t dw = smem_desc_sw128(addr), dx = smem_desc_sw128(addr + kWBytes);
#pragma unroll
                    for (int k = 0; k < BK / 16; ++k)
                        // 16 bf16 = 32 bytes further along K inside the swizzle row: +2 in the address field
                        ptx::tc_mma_f16_pair(d_tmem, dw + 2 * k, dx + 2 * k, idesc, (g != it.kb_begin || k != 0) ? 1u : 0u);
                    ptx::tc_commit_pair(&s.empty_bar[st]);  // frees the stage in both CTAs when these MMAs have read it
                    if (++st == stages) st = 0, ++round;
                }
                if (s.abort) break;
                ptx::tc_commit_pair(&s.tmem_full_bar[b]);  // accumulator complete
            }
            if (n > 0 || s.abort) {  // a pair without items leaves at once
                ptx::tc_commit_pair(&s.drain_bar);
                mbar_drain(&s.drain_bar, 0);
            }
        }
    } else if (warp == kAnnounceWarp) {
        // When the epilogue warps have stored their part of a unit: publish the call number in its flag.  The release orders
        // the stores (made visible to this warp by the mbarrier) before the flag; it waits for them to arrive, so it
        // sits in a warp of its own.
        // It also reads this call's number; the epilogue warps need it where the sums are lines.
        uint32_t epoch = 0;
        if (lane == 0) epoch = *reinterpret_cast<volatile uint32_t*>(flag_word(cv, 0, kCallLocalGemm)) + 1u;
        if (a.lines) {
            if (lane == 0) s.epoch = epoch;
            ptx::named_barrier(kNumberBarrier, 32 * (kEpilogueWarps + 1));
        }
        if (lane == 0) {
            // The last CTA that has read the number advances it for the next call.  The row kernel keeps a count of its own:
            // it runs at the same time and, where the sums are lines, is done with its count before any of them is here.
            auto check_in = [&] {
                uint32_t* const in = flag_word(cv, 0, kCallLocalGemmIn);
                if (atomicAdd(in, 1u) != gridDim.x - 1) return;
                *reinterpret_cast<volatile uint32_t*>(in) = 0u;
                *reinterpret_cast<volatile uint32_t*>(flag_word(cv, 0, kCallLocalGemm)) = epoch;
            };
            if (a.lines) check_in();  // nothing to announce: now rather than at the end
            const uint32_t units = a.N / kLocalGemmUnitCols;
            Item it;
            for (uint32_t n = 0; item_at(a, n, pair, npairs, ncol, &it); ++n) {
                const uint32_t b = n & 1u, unit = it.col_tile * 2 + half;
                if (!wait_bar(&s.stored_bar[b], (n >> 1) & 1u, deadline, &s.abort)) {
                    if (!s.abort) report_timeout(cv, kSiteMbar, 0, cta, 5, n);
                    s.abort = 1;
                    break;
                }
                if (unit < units && !a.lines)
                    ptx::st_release_gpu(flag_word(cv, 0, kLocalGemmFlagOff + (it.tile * a.s.nsplit + it.split) * units + unit), epoch);
                ptx::mbar_arrive(&s.announced_bar[b]);
            }
            if (!a.lines) check_in();  // the rows take longer
        }
    } else if (warp == kPrefetchWarp) {
        // Brings the operands into L2 ahead of the loads: what a CTA has in flight in its stages does not cover the latency of
        // HBM.  One item of those that use a slice fetches it: of W those of the first token tile, of x those of
        // the first columns.
        if (ptx::elect_one()) {
            uint32_t ahead = 0;
            Item it;
            for (uint32_t i = 0; item_at(a, i, pair, npairs, ncol, &it); ++i) {
                const bool w_here = it.tile == 0, x_here = it.col_tile == 0;
                const int wrow = it.col_tile * kLocalGemmPairCols + half * kLocalGemmUnitCols;
                const int xrow = it.tile * a.s.tokens + half * (a.s.tokens / 2);
                uint32_t rank = it.kb_begin / a.kb_rank, kb = it.kb_begin - rank * a.kb_rank;
                for (uint32_t g = it.kb_begin; g < it.kb_end; ++g, ++ahead) {
                    while (static_cast<int32_t>(ahead - s.loaded) > static_cast<int32_t>(stages + kPrefetchBlocks)) ptx::nanosleep(40);
                    if (w_here && ahead >= fetched) ptx::tma_prefetch_2d(&a.tmap_w[rank], kb * BK, wrow);
                    if (x_here) ptx::tma_prefetch_2d(&a.tmap_x[rank], kb * BK, xrow);
                    if (++kb == a.kb_rank) kb = 0, ++rank;
                }
            }
        }
    } else if (warp < kEpilogueWarps) {
        const int q = warp & 3;   // TMEM lane quarter this warp may read: columns 32q .. 32q+31 of the CTA's 128
        const int g = warp >> 2;  // takes every second chunk of 32 tokens
        // A chunk is transposed through 2 KiB of this warp's own, [32 tokens][64 bytes] with the 16-byte pieces swizzled: no
        // barrier with other warps.  stmatrix: this thread's row of the transposed matrices is token lane % 8 of an
        // 8-token group; matrix lane / 8 holds 8 of the warp's 32 columns.
        uint8_t* const stage = s_epi[warp];
        uint8_t* const st_row = stage + (lane & 7) * 64 + (((lane >> 3) ^ ((lane >> 1) & 3)) << 4);
        const uint32_t token = lane >> 2;  // stores: token of a group of 8, 16-byte piece lane % 4
        const uint8_t* const ld_row = stage + token * 64 + (((lane & 3) ^ ((token >> 1) & 3)) << 4);
        const uint64_t rowbytes = static_cast<uint64_t>(a.N) * 2;
        uint32_t epoch = 0;
        if (a.lines) {
            ptx::named_barrier(kNumberBarrier, 32 * (kEpilogueWarps + 1));
            epoch = s.epoch;
        }
        Item it;
        for (uint32_t n = 0; item_at(a, n, pair, npairs, ncol, &it); ++n) {
            const uint32_t b = n & 1u, t0 = it.tile * a.s.tokens, nt = min(a.T - t0, a.s.tokens);
            const uint32_t col = it.col_tile * kLocalGemmPairCols + half * kLocalGemmUnitCols;
            // The second half of the last column tile may lie beyond N.
            const uint32_t chunks = col < a.N ? (nt + kEpiChunk - 1) / kEpiChunk : 0u;
            const uint64_t first = (static_cast<uint64_t>(it.split) * a.T + t0) * rowbytes + (col + q * 32 + (lane & 3) * 8) * 2;
            char* const dst0 = a.sums + (a.lines ? 2 * first : first);
            if (!wait_bar(&s.tmem_full_bar[b], (n >> 1) & 1u, deadline, &s.abort)) {
                if (lane == 0 && !s.abort) report_timeout(cv, kSiteMbar, 0, cta, 3, n);
                s.abort = 1;
                break;
            }
            __syncwarp();
            ptx::tc_fence_after_sync();
            for (uint32_t ch = g; ch < chunks; ch += kEpiGroups) {
                uint32_t v[2][16];  // lanes 0..15 and 16..31 of the quarter
                const uint32_t src = tmem + b * kLocalGemmMaxTokens + (static_cast<uint32_t>(q * 32) << 16) + ch * kEpiChunk;
                ptx::tmem_ld_16x256b_x4(src, v[0]);
                ptx::tmem_ld_16x256b_x4(src + (16u << 16), v[1]);
                ptx::tmem_ld_wait();
#pragma unroll
                for (int k = 0; k < 4; ++k) {  // 8 tokens each: four matrices of 8 columns x 8 tokens
                    uint32_t m[4];
#pragma unroll
                    for (int h = 0; h < 4; ++h) {  // columns 8h .. 8h+7 of the warp's 32
                        const __nv_bfloat162 p = __floats2bfloat162_rn(__uint_as_float(v[h >> 1][4 * k + 2 * (h & 1)]),
                                                                       __uint_as_float(v[h >> 1][4 * k + 2 * (h & 1) + 1]));
                        m[h] = *reinterpret_cast<const uint32_t*>(&p);
                    }
                    ptx::stmatrix_x4_trans(st_row + k * 8 * 64, m[0], m[1], m[2], m[3]);
                }
                __syncwarp();
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const uint4 x = *reinterpret_cast<const uint4*>(ld_row + k * 8 * 64);
                    const uint32_t tok = ch * kEpiChunk + k * 8 + token;
                    if (tok >= nt) continue;
                    if (a.lines) {  // {2 bf16, call, 2 bf16, ~call} per four columns: the flag is in the data
                        ptx::st_v4(dst0 + tok * 2 * rowbytes, make_uint4(x.x, epoch, x.y, ~epoch));
                        ptx::st_v4(dst0 + tok * 2 * rowbytes + 16, make_uint4(x.z, epoch, x.w, ~epoch));
                    } else {
                        ptx::st_v4(dst0 + tok * rowbytes, x);
                    }
                }
                __syncwarp();
            }
            // Out of the accumulator: hand it back.
            ptx::tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) {
                ptx::mbar_arrive_cluster(ptx::mapa_u32(&s.tmem_empty_bar[b], 0));
                // Hand the unit to the announcer, which has to be done with the one before last.
                if (n < 2 || wait_bar(&s.announced_bar[b], ((n >> 1) - 1u) & 1u, deadline, &s.abort)) {
                    ptx::mbar_arrive(&s.stored_bar[b]);
                } else {
                    if (!s.abort) report_timeout(cv, kSiteMbar, 0, cta, 6, n);
                    s.abort = 1;
                }
            }
            __syncwarp();
        }
    }
    __syncwarp();
    ptx::tc_fence_before_sync();
    __syncthreads();
    // Nobody leaves (or gives TMEM back) while the other CTA's MMAs, loads or arrivals may still reach this one.
    ptx::cluster_arrive();
    ptx::cluster_wait();
    if (warp == kMmaWarp) ptx::tmem_dealloc_pair(tmem, kTmemCols);
}

namespace {

// Pauses between two looks at a flag and at a line.  Polling costs the GEMM more than a late look costs the row: with 50 ns
// and all lines asked for on every look, us: 2 ranks, K = 2048: T = 8 10.0 -> 9.8, T = 64 17.3 -> 14.6, T = 128 18.3 -> 16.5
// (flags, 3000 ns level, 600 ns 16.8); 4 ranks, K = 1792, T = 100 20.4 -> 18.5 (3000 ns 20.5, 1000 ns 19.1).  Lines: 0 to 100 ns
// are level.  Once one of a warp's flags is set, the others are not far: kFlagNearNs from then on against 1500 ns always / 400 ns always, us: 2 ranks,
// 182 x 832 x 3072 10.6 / 10.8 / 11.4, 96 x 2048 x 2048 10.5 / 10.6 / 11.3, 300 x 2048 x 4096 19.7 / 20.4 / 19.9; 4 ranks, 1500 x 640 x 1536 26.1
// / 26.6 / 26.3; 8 ranks, 678 x 640 x 1664 28.9 / 29.4 / 29.1, 418 x 704 x 1152 18.7 / 18.7 / 19.5; of 25 sizes 1.2 % and 1.6 % in the mean.
constexpr uint32_t kFlagSleepNs = 1500, kFlagNearNs = 400, kLineSleepNs = 40;

// A unit of work is a row for G ranks (unit u: row u / ngroups, ranks from (u % ngroups) * G); a thread holds NV 16-byte
// vectors of the row.  SPLIT: more than one K split; LINES: the sums come as flag-in-data lines; SLIM: of two instances for
// the same, the one that takes fewer registers.
//
// Bound by memory once enough is in flight, and before that by the chain of a unit: residuals and sums, two barriers, weights, stores.
// So a unit waits for memory as seldom as it can (the sums of a complete tile are asked for with the residuals, the weights of all its
// ranks at once), a CTA has no more warps than a row needs, and instructions that do no arithmetic are kept out (no division, no
// branch or zeros for the threads beyond the row's end).  Registers are capped so that 16 to 32 warps share an SM, and none is spilled:
// 16 bytes of it cost 1 us of 23 (8 ranks, 4 x 1728 x 4096).  A grid with fewer CTAs than units takes them in row order from a
// counter, the residuals of the next unit on their way into L2: rows as CTAs of their own came in waves, each a chain of
// launch, residual, sums and stores (8 ranks, 300 rows: 600 CTAs on 444 places took two of them).
//
// In a graph, W from HBM, before these measures / with them, us: 8 ranks: 1000 x 256 x 1024 35.1 / 22.5, 2048 x 256 x 1024 47.9 / 32.6,
// 1500 x 512 x 2304 68.9 / 53.4, 678 x 640 x 1664 33.4 / 29.0, 688 x 1792 x 2816 72.9 / 65.4, 300 x 1792 x 4096 51.0 / 49.0, 32 x 1792 x 4096
// 31.0 / 26.9, 21 x 384 x 3328 11.9 / 9.4; 4 ranks: 300 x 512 x 1024 14.7 / 10.4, 512 x 2048 x 4096 41.7 / 40.2, 60 x 256 x 3072 10.5 / 8.4;
// 2 ranks: 188 x 1024 x 2944 13.5 / 11.9, 2048 x 2048 x 4096 level.  Of the 16 us that the rows of 8 x 300 x 4096 take behind the GEMM
// for 59 MB, 2 go by before the first row is complete and 3 while the last CTAs finish (1200 units on 296 places, two CTAs of 96 registers per SM:
// 16 units are left for a fifth round).
template <int NV, int G, bool SPLIT, bool LINES, bool SLIM>
__global__ void __maxnreg__(LocalLinearNormRegs(NV, G, SPLIT, SLIM))
    local_linear_norm_kernel(const __grid_constant__ LocalLinearNormArgs a) {
    constexpr int VEC = 8, kMostWarps = kLocalLinearNormThreads / 32;
    __shared__ __align__(16) float s_red[G][kMostWarps];
    __shared__ uint32_t s_next;
    const CommView& cv = a.cv;
    const uint32_t ngroups = (a.world + G - 1) / G, units = a.T * ngroups, flags_per_split = a.N / kLocalGemmUnitCols;
    const uint32_t tid = threadIdx.x, nthreads = blockDim.x, nvec = a.N / VEC, rowbytes = a.N * 2;
    const bool taking = gridDim.x < units;  // from the counter
    uint32_t* const counter = flag_word(cv, 0, kCallLocalRows);
    // The next kernel may set up, and ask for its weights, under this one.  Whatever it is, it waits for the end of this kernel, and with
    // it of the GEMM (see the last line), before it touches memory.
    if (a.early) ptx::grid_launch_dependents();
    const uint32_t epoch = *reinterpret_cast<volatile uint32_t*>(flag_word(cv, 0, kCallLocalRowCalls)) + 1u;
    const uint64_t deadline = ptx::globaltimer() + cv.timeout_ns;
    // A thread without a vector of the row (the last ones of a CTA) loads the row's last one, which costs no branch and no zeros,
    // and keeps it out of the sum of squares and of memory.
    bool have[NV];
    uint32_t at[NV];  // byte in the row
#pragma unroll
    for (int j = 0; j < NV; ++j) {
        have[j] = tid + j * nthreads < nvec;
        at[j] = min(tid + j * nthreads, nvec - 1) * 16;
    }
    uint32_t unit = blockIdx.x;
    uint32_t tile = 0, tile_end = 0;  // the tile in front of row tile_end is complete (a CTA's rows only go up)
    if (tid < G * kMostWarps) (&s_red[0][0])[tid] = 0.f;  // those of warps that a CTA of this size has not
    if (taking) {
        if (tid == 0) s_next = atomicAdd(counter, 1u);
        __syncthreads();
        unit = s_next;
        __syncthreads();
    }
    auto check_in = [&] {
        if (check_in_last(cv, 3, gridDim.x)) {
            *reinterpret_cast<volatile uint32_t*>(counter) = 0u;
            advance_call_word(cv, kCallLocalRowCalls, 1);
        }
    };
    if (unit >= units && tid == 0) check_in();  // nothing was left for this CTA
    const float inv_n = 1.f / static_cast<float>(a.N);
    bool late = false;
    // When a step asks for its weights (plain loads: the rows of an SM share them in L1).  One by one behind the stores and the barrier
    // each rank's is a latency of its own, so: 0 with the residuals, 1 ahead of the stores, 2 all at once behind the barrier, 3 one by
    // one where registers are short and there are enough rows to hide it.
    constexpr int kWeights = G == 1 ? 0 : NV * G == 2 ? 1 : NV == 2 && !SPLIT && SLIM ? 3 : 2;
    uint4 w1[NV][G];
    auto load_weight = [&](int g, int j, uint32_t q) { w1[j][g] = ptx::ld_v4(static_cast<const char*>(a.weight[q]) + at[j]); };
    const uint32_t most = a.world - 1;  // a group beyond the last rank computes that one again and stores nothing
    auto load_weights = [&](uint32_t q0) {
#pragma unroll
        for (int g = 0; g < G; ++g)
#pragma unroll
            for (int j = 0; j < NV; ++j) load_weight(g, j, min(q0 + g, most));
    };
    while (unit < units) {
        const uint32_t row = ngroups == 1 ? unit : __umulhi(unit, a.by_groups), q0 = (unit - row * ngroups) * G;
        const uint32_t off0 = row * rowbytes;
        if (taking && tid == 0) s_next = atomicAdd(counter, 1u);
        // Residuals and weights are inputs of the call: complete since before the first kernel passed its own wait.
        uint4 res[NV][G];
        if (kWeights == 0) load_weights(q0);
#pragma unroll
        for (int g = 0; g < G; ++g) {
            const char* const r = static_cast<const char*>(a.residual[min(q0 + g, most)]);
            if (r) {
#pragma unroll
                for (int j = 0; j < NV; ++j) res[j][g] = ptx::ld_cg_v4(r + off0 + at[j]);
            } else {
#pragma unroll
                for (int j = 0; j < NV; ++j) res[j][g] = make_uint4(0, 0, 0, 0);
            }
        }
        const uint32_t nsplit = a.s.nsplit;
        const uint64_t split_stride = static_cast<uint64_t>(a.T) * a.N * (LINES ? 4 : 2);
        // Splits in flight together, added in order.
        constexpr int kFly = !SPLIT ? 1 : G > 1 ? 2 : SLIM ? (NV == 2 ? 1 : LINES ? 2 : 4) : 4;
        uint4 x[NV][kFly];
        auto load_sums = [&](uint32_t k0) {
#pragma unroll
            for (int k = 0; k < kFly; ++k)
                if (k0 + k < nsplit) {
#pragma unroll
                    for (int j = 0; j < NV; ++j) x[j][k] = ptx::ld_cg_v4(a.sums + (k0 + k) * split_stride + off0 + at[j]);
                }
        };
        // The first sums of a tile that is known to be complete are asked for together with the residuals.
        const bool asked = !LINES && row < tile_end;
        if (asked) load_sums(0);
        if (!LINES && !asked) {
            // The flags of this row's token tile, a few per thread.
            while (row >= tile_end) tile_end += a.s.tokens, ++tile;
            const uint32_t first = kLocalGemmFlagOff + (tile - 1) * nsplit * flags_per_split;
            static_assert(kLocalGemmMaxSplit * VEC * NV <= kLocalGemmUnitCols, "a thread waits for one flag: a split's columns / kLocalGemmUnitCols");
            bool there = tid >= nsplit * flags_per_split || late;
            const uint32_t mine = __ballot_sync(0xffffffffu, !there);  // lanes that have a flag
            for (uint32_t polls = 1;; ++polls) {
                uint32_t seen = 0;
                if (!there) there = ptx::seq_reached(seen = ptx::ld_acquire_gpu(flag_word(cv, 0, first + tid)), epoch);
                const uint32_t waiting = __ballot_sync(0xffffffffu, !there);
                if (waiting == 0) break;
                // This CTA shares the SM with the GEMM, and hundreds of them poll; but once the first of a warp's units is there, the
                // last one is not far.
                if (polls > 2) ptx::nanosleep(waiting == mine ? kFlagSleepNs : kFlagNearNs);
                if ((polls & 7u) == 0 && __any_sync(0xffffffffu, ptx::globaltimer() > deadline)) {
                    if (!there) report_timeout(cv, kSiteGemmPartials, 0, blockIdx.x, epoch, seen);
                    late = true;
                    break;
                }
            }
        }
        // After a wait that ran out the rows are not worth anything, but the CTA goes on, without waiting: every unit is taken,
        // every CTA checks in and the two counts of calls stay alike.
        __syncthreads();
        if (taking) {
            unit = s_next;
            if (unit < units) {
                const uint32_t nrow = ngroups == 1 ? unit : __umulhi(unit, a.by_groups), nq = (unit - nrow * ngroups) * G;
                // One 128-byte line per eight vectors.
                if ((tid & 7) == 0) {
#pragma unroll
                    for (int g = 0; g < G; ++g) {
                        const char* const r = static_cast<const char*>(a.residual[min(nq + g, most)]);
                        if (r)
#pragma unroll
                            for (int j = 0; j < NV; ++j) ptx::prefetch_l2(r + nrow * rowbytes + at[j]);
                    }
                }
            }
        } else {
            unit = units;
        }
        // Once every CTA has read the call number and taken its last unit, both counters may move on: the next call reads
        // them, nothing in this one does.  Done here, under the work of the last unit.
        if (unit >= units && tid == nthreads - 1) check_in();

        float sum[SPLIT ? NV : 1][VEC];
        if constexpr (!SPLIT) {
            if (!asked) load_sums(0);
        } else {
            for (uint32_t k0 = 0; k0 < nsplit && !late; k0 += kFly) {
                if constexpr (LINES) {
                    const char* const src = a.sums + 2 * static_cast<uint64_t>(off0);
                    uint4 y[NV][kFly];
                    uint32_t polls = 0;
                    bool missing;
                    // One lane of a warp waits for one of its lines of the last split: asking for all lines again and
                    // again (64 KiB per CTA) holds up the GEMM that writes them.
                    if (k0 == 0 && (tid & 31) == 0) {
                        uint4 l;
                        while ((l = ptx::ld_volatile_v4(src + 2 * at[0] + (nsplit - 1) * split_stride)).y != epoch || l.w != ~epoch) {
                            ptx::nanosleep(kLineSleepNs);
                            if ((++polls & 63u) == 0 && ptx::globaltimer() > deadline) break;  // the loop below reports it
                        }
                    }
                    __syncwarp();
                    do {
                        missing = false;
#pragma unroll
                        for (int k = 0; k < kFly; ++k)
                            if (k0 + k < nsplit) {
#pragma unroll
                                for (int j = 0; j < NV; ++j) {
                                    const char* p = src + (k0 + k) * split_stride + 2 * at[j];
                                    x[j][k] = ptx::ld_volatile_v4(p);
                                    y[j][k] = ptx::ld_volatile_v4(p + 16);
                                }
                            }
#pragma unroll
                        for (int k = 0; k < kFly; ++k)
#pragma unroll
                            for (int j = 0; j < NV; ++j)
                                if (k0 + k < nsplit)
                                    missing |= x[j][k].y != epoch || x[j][k].w != ~epoch || y[j][k].y != epoch || y[j][k].w != ~epoch;
                        if (missing && (++polls & 63u) == 0 && ptx::globaltimer() > deadline) {
                            report_timeout(cv, kSiteGemmPartials, 0, blockIdx.x, epoch, 0u);
                            late = true;
                        }
                    } while (missing && !late);
#pragma unroll
                    for (int k = 0; k < kFly; ++k)
#pragma unroll
                        for (int j = 0; j < NV; ++j) x[j][k] = make_uint4(x[j][k].x, x[j][k].z, y[j][k].x, y[j][k].z);
                } else {
                    if (k0 > 0 || !asked) load_sums(k0);
                }
#pragma unroll
                for (int k = 0; k < kFly; ++k)
#pragma unroll
                    for (int j = 0; j < NV; ++j) {
                        if (k == 0 && k0 == 0) unpack16<__nv_bfloat16>(sum[j], x[j][0]);
                        else if (k0 + k < nsplit) accumulate<__nv_bfloat16>(sum[j], x[j][k]);
                    }
            }
            if (late) {
#pragma unroll
                for (int j = 0; j < NV; ++j)
#pragma unroll
                    for (int i = 0; i < VEC; ++i) sum[j][i] = 0.f;
            }
        }
        if (kWeights == 1) load_weights(q0);
        // sum + residual of rank q0 + g, vector j.
        auto row_of = [&](int j, int g, float (&p)[VEC]) {
            if constexpr (SPLIT) {
#pragma unroll
                for (int i = 0; i < VEC; ++i) p[i] = sum[j][i];
            } else {
                unpack16<__nv_bfloat16>(p, x[j][0]);
            }
            accumulate<__nv_bfloat16>(p, res[j][g]);
        };
#pragma unroll
        for (int g = 0; g < G; ++g) {
            float ss = 0.f;
            char* const ro = q0 + g <= most ? static_cast<char*>(a.residual_out[q0 + g]) : nullptr;
#pragma unroll
            for (int j = 0; j < NV; ++j) {
                float p[VEC];
                row_of(j, g, p);
                if (ro && have[j]) ptx::st_v4(ro + off0 + at[j], pack16<__nv_bfloat16>(p));
                float sq = p[0] * p[0];
#pragma unroll
                for (int i = 1; i < VEC; ++i) sq += p[i] * p[i];
                ss += have[j] ? sq : 0.f;
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
            if ((tid & 31) == 0) s_red[g][tid >> 5] = ss;
        }
        __syncthreads();
        if (kWeights == 2) load_weights(q0);
#pragma unroll
        for (int g = 0; g < G; ++g) {
            if (q0 + g > most) break;
            float t = 0.f;
#pragma unroll
            for (int w = 0; w < kMostWarps; w += 4) {
                const float4 part = *reinterpret_cast<const float4*>(&s_red[g][w]);
                t += (part.x + part.y) + (part.z + part.w);
            }
            const float inv_rms = rsqrtf(t * inv_n + a.eps);
            char* const out = static_cast<char*>(a.out[q0 + g]) + off0;
#pragma unroll
            for (int j = 0; j < NV; ++j) {
                if (!have[j]) continue;
                float p[VEC], w[VEC];
                row_of(j, g, p);
                if (kWeights == 3) load_weight(g, j, q0 + g);
                unpack16<__nv_bfloat16>(w, w1[j][g]);
#pragma unroll
                for (int i = 0; i < VEC; ++i) p[i] = p[i] * inv_rms * w[i];
                ptx::st_v4(out + at[j], pack16<__nv_bfloat16>(p));
            }
        }
    }
    // The call is over when both kernels are.
    ptx::grid_dependency_wait();
}

template <int NV, int G>
const void* pick_linear_norm(bool split) {
    return split ? (const void*)local_linear_norm_kernel<NV, G, true, false, true>
                 : (const void*)local_linear_norm_kernel<NV, G, false, false, true>;
}

}  // namespace

const void* LocalGemmKernel() { return reinterpret_cast<const void*>(local_gemm_kernel); }
uint32_t LocalGemmSmemBytes() { return kSmemBytes; }

const void* LocalLinearNormKernel(uint32_t N, int ranks_per_cta, bool split, bool lines, bool slim) {
    const bool wide = LocalLinearNormVectors(N) == 2;
    if (lines) {
        if (wide) return slim ? (const void*)local_linear_norm_kernel<2, 1, true, true, true> : (const void*)local_linear_norm_kernel<2, 1, true, true, false>;
        return slim ? (const void*)local_linear_norm_kernel<1, 1, true, true, true> : (const void*)local_linear_norm_kernel<1, 1, true, true, false>;
    }
    if (ranks_per_cta == 4) return pick_linear_norm<1, 4>(split);
    if (ranks_per_cta == 2 && wide && !split && !slim) return (const void*)local_linear_norm_kernel<2, 2, false, false, false>;
    if (ranks_per_cta == 2) return wide ? pick_linear_norm<2, 2>(split) : pick_linear_norm<1, 2>(split);
    return wide ? pick_linear_norm<2, 1>(split) : pick_linear_norm<1, 1>(split);
}

}  // namespace yali
