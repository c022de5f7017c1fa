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
// Bound by the tensor cores from about 200 tokens on, by reading W below.
//
// Parity: none in the reference (it has no GEMM, no fused op and no tensor-core code).
#include <cuda.h>

#include "coll_common.cuh"
#include "gemm_local.h"

namespace yali {

namespace {

constexpr int BK = 64;                        // BK bf16 = one 128-byte swizzle row
constexpr uint32_t kWBytes = 128 * BK * 2;    // one CTA's half of the W operand of a stage
constexpr uint32_t kRingBytes = 192 * 1024;   // operand stages: 6 of 32 KB (256 tokens) to 10 of 18 KB (32 tokens)
constexpr int kMaxStages = 12;
constexpr uint32_t kSmemBytes = kRingBytes + 1024;  // + slack to align the base
constexpr uint32_t kTmemCols = 2 * kLocalGemmMaxTokens;  // two accumulators: all of TMEM
constexpr uint32_t kEpiChunk = 32;                              // tokens an epilogue group moves at a time
constexpr uint32_t kEpiRowBytes = kLocalGemmUnitCols * 2;       // 256 bytes per token
constexpr uint32_t kEpiBufBytes = kEpiChunk * kEpiRowBytes;     // 8 KiB per group of four warps
constexpr int kEpiGroups = 2, kEpilogueWarps = 4 * kEpiGroups;
constexpr int kTmaWarp = 8, kMmaWarp = 9, kAnnounceWarp = 10;
static_assert(kTmemCols == 512 && kLocalGemmThreads >= 32 * (kAnnounceWarp + 1), "one CTA per SM");
static_assert(kSmemBytes + kEpiGroups * kEpiBufBytes + 1024 <= 216 * 1024, "leaves room for CTAs of the second kernel");

// tcgen05 instruction descriptor: D = fp32, A = B = bf16, both K-major, N at bit 17 (>>3), M at bit 24 (>>4).
__device__ __forceinline__ uint32_t pair_idesc(uint32_t n) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((n >> 3) << 17) | ((kLocalGemmPairCols >> 4) << 24);
}

// Shared-memory matrix descriptor of a K-major operand tile stored by TMA with 128-byte
// swizzle: rows of 128 bytes, groups of 8 rows 1024 bytes apart.
__device__ __forceinline__ uint64_t smem_desc_sw128(uint32_t smem_addr) {
    uint64_t d = 0;
    d |= static_cast<uint64_t>((smem_addr & 0x3ffffu) >> 4);  // start address
    d |= static_cast<uint64_t>(1) << 16;                      // leading byte offset (unused with swizzle)
    d |= static_cast<uint64_t>(1024 >> 4) << 32;              // stride byte offset: next 8-row group
    d |= static_cast<uint64_t>(1) << 46;                      // descriptor version of sm_100
    d |= static_cast<uint64_t>(2) << 61;                      // SWIZZLE_128B
    return d;
}

struct Item {
    uint32_t tile, t0, nt;       // token tile, its rows [t0, t0 + nt)
    uint32_t col_tile, split;
    uint32_t kb_begin, kb_end;
};
// Token tile by token tile, so that rows complete early; the items in flight together read the same stretch of K.
__device__ __forceinline__ Item item_at(const LocalGemmArgs& a, uint32_t i, uint32_t ncol) {
    Item it;
    const uint32_t per_tile = ncol * a.s.nsplit;
    it.tile = i / per_tile;
    const uint32_t in_tile = i - it.tile * per_tile;
    it.split = in_tile / ncol;
    it.col_tile = in_tile - it.split * ncol;
    it.t0 = it.tile * a.s.tokens;
    it.nt = min(a.T - it.t0, a.s.tokens);
    it.kb_begin = it.split * a.s.kper;
    it.kb_end = min(a.kb_total, it.kb_begin + a.s.kper);
    return it;
}

struct Shared {
    __align__(8) uint64_t full_bar[kMaxStages], empty_bar[kMaxStages], tmem_full_bar[2], tmem_empty_bar[2];
    __align__(8) uint64_t stored_bar[2], announced_bar[2];  // epilogue warps -> announcer warp and back
    uint32_t tmem;
    volatile int abort;
};

// Bounded waits: give up at the deadline or when another role of this CTA has.
__device__ __forceinline__ bool wait_bar(uint64_t* bar, uint32_t parity, uint64_t deadline, volatile int* abort) {
    uint32_t tries = 0;
    while (!ptx::mbar_try_wait_cluster(bar, parity)) {
        if ((++tries & 15u) == 0 && (*abort || ptx::globaltimer() > deadline)) return false;
    }
    return true;
}

}  // namespace

__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kLocalGemmThreads, 1)
    local_gemm_kernel(const __grid_constant__ LocalGemmArgs a) {
    extern __shared__ uint8_t smem_raw[];
    __shared__ Shared s;
    __shared__ __align__(16) uint8_t s_epi[kEpiGroups][kEpiBufBytes];

    const CommView& cv = a.cv;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t cta = blockIdx.x, half = ptx::cluster_cta_rank();
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    // Nothing up to the wait depends on earlier kernels: it runs under the end of the one in front.
    if (tid == 64) {
        s.abort = 0;
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
        ptx::mbar_fence_init();
        ptx::tma_prefetch_desc(&a.tmap_w[0]);
        ptx::tma_prefetch_desc(&a.tmap_x[0]);
    }
    if (warp == kMmaWarp) {
        ptx::tmem_alloc_pair(&s.tmem, kTmemCols);
        ptx::tmem_relinquish_pair();
    }
    ptx::tc_fence_before_sync();
    __syncthreads();
    ptx::cluster_arrive();  // the other CTA's barriers and TMEM are ready, too
    ptx::cluster_wait();
    ptx::tc_fence_after_sync();
    const uint32_t tmem = s.tmem;
    ptx::grid_dependency_wait();
    ptx::grid_launch_dependents();
    const uint64_t deadline = ptx::globaltimer() + cv.timeout_ns;

    const uint32_t ncol = (a.N + kLocalGemmPairCols - 1) / kLocalGemmPairCols;
    const uint32_t nitems = a.s.tiles * ncol * a.s.nsplit;
    const uint32_t pair = cta >> 1, npairs = gridDim.x >> 1;
    const uint32_t xbytes = a.s.tokens / 2 * (BK * 2);  // one CTA's half of the token operand of a stage: whole KiB
    const uint32_t stage_bytes = kWBytes + xbytes;
    const uint32_t stages = min(kRingBytes / stage_bytes, static_cast<uint32_t>(kMaxStages));

    if (warp == kTmaWarp) {
        if (ptx::elect_one()) {
            uint32_t st = 0, round = 0;
            for (uint32_t i = pair; i < nitems && !s.abort; i += npairs) {
                const Item it = item_at(a, i, ncol);
                const int wrow = it.col_tile * kLocalGemmPairCols + half * kLocalGemmUnitCols;
                const int xrow = it.t0 + half * (a.s.tokens / 2);
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
                    if (++kb == a.kb_rank) kb = 0, ++rank;
                    if (++st == stages) st = 0, ++round;
                }
            }
            // The MMAs' releases of the last stages arrive here from the leader: none may be under way when this CTA
            // leaves.
            for (uint32_t k = 0; k < stages && !s.abort; ++k) {
                if (!wait_bar(&s.empty_bar[st], (round & 1u) ^ 1u, deadline, &s.abort)) s.abort = 1;
                if (++st == stages) st = 0, ++round;
            }
        }
    } else if (warp == kMmaWarp) {
        if (half == 0 && ptx::elect_one()) {
            const uint32_t idesc = pair_idesc(a.s.tokens);
            uint32_t st = 0, round = 0, n = 0;
            for (uint32_t i = pair; i < nitems && !s.abort; i += npairs, ++n) {
                const Item it = item_at(a, i, ncol);
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
        }
    } else if (warp == kAnnounceWarp) {
        // When the eight epilogue warps have stored their part of a unit: publish the call number in its flag.  The release
        // orders the stores (made visible to this warp by the mbarrier) before the flag; it waits for them to
        // arrive, so it sits in a warp of its own.
        const uint32_t epoch = *reinterpret_cast<volatile uint32_t*>(flag_word(cv, 0, kCallLocalGemm)) + 1u;
        const uint32_t units = a.N / kLocalGemmUnitCols;
        uint32_t n = 0;
        for (uint32_t i = pair; i < nitems; i += npairs, ++n) {
            const Item it = item_at(a, i, ncol);
            const uint32_t b = n & 1u, unit = it.col_tile * 2 + half;
            if (!wait_bar(&s.stored_bar[b], (n >> 1) & 1u, deadline, &s.abort)) {
                if (lane == 0 && !s.abort) report_timeout(cv, kSiteMbar, 0, cta, 5, n);
                s.abort = 1;
                break;
            }
            if (lane == 0) {
                if (unit < units)
                    ptx::st_release_gpu(flag_word(cv, 0, kLocalGemmFlagOff + (it.tile * a.s.nsplit + it.split) * units + unit), epoch);
                ptx::mbar_arrive(&s.announced_bar[b]);
            }
            __syncwarp();
        }
    } else if (warp < kEpilogueWarps) {
        const int q = warp & 3;   // TMEM lane quarter this warp may read: columns 32q .. 32q+31 of the CTA's 128
        const int g = warp >> 2;  // its group takes every second chunk of 32 tokens
        const int gt = tid & 127;
        const uint32_t c16 = gt & 15, rsub = gt >> 4;  // stores: 16-byte piece of a token's 256 bytes, token % 8
        const uint64_t rowbytes = static_cast<uint64_t>(a.N) * 2;
        uint8_t* const stage = s_epi[g];
        uint32_t n = 0;
        for (uint32_t i = pair; i < nitems; i += npairs, ++n) {
            const Item it = item_at(a, i, ncol);
            const uint32_t b = n & 1u;
            const uint32_t col = it.col_tile * kLocalGemmPairCols + half * kLocalGemmUnitCols;
            // The second half of the last column tile may lie beyond N.
            const uint32_t chunks = col < a.N ? (it.nt + kEpiChunk - 1) / kEpiChunk : 0u;
            char* const dst0 = a.sums + (static_cast<uint64_t>(it.split) * a.T + it.t0) * rowbytes +
                               static_cast<uint64_t>(col) * 2 + c16 * 16;
            // Every warp of a group has to take the same way through the chunks (they share a barrier).
            const bool up = wait_bar(&s.tmem_full_bar[b], (n >> 1) & 1u, deadline, &s.abort);
            if (!up) {
                if (lane == 0 && !s.abort) report_timeout(cv, kSiteMbar, 0, cta, 3, n);
                s.abort = 1;
            }
            if (ptx::named_barrier_or(1 + g, 128, !up)) break;
            ptx::tc_fence_after_sync();
            bool released = false;
            for (uint32_t ch = g; ch < chunks; ch += kEpiGroups) {
                uint32_t v[32];
                ptx::tmem_ld_32x32(tmem + b * kLocalGemmMaxTokens + (static_cast<uint32_t>(q * 32) << 16) + ch * kEpiChunk, v);
                ptx::tmem_ld_wait();
                if (ch + kEpiGroups >= chunks) {  // this warp's last read of the accumulator: hand it back
                    ptx::tc_fence_before_sync();
                    __syncwarp();
                    if (lane == 0) ptx::mbar_arrive_cluster(ptx::mapa_u32(&s.tmem_empty_bar[b], 0));
                    released = true;
                }
                // Thread = column, register = token: token t's 128 columns become 256 contiguous bytes (32 lanes
                // write 64 of them at once: no bank conflict).
                if (ch != static_cast<uint32_t>(g)) ptx::named_barrier(1 + g, 128);  // the chunk before has been read
#pragma unroll
                for (int t = 0; t < 32; ++t)
                    *reinterpret_cast<__nv_bfloat16*>(stage + t * kEpiRowBytes + q * 64 + lane * 2) =
                        __float2bfloat16_rn(__uint_as_float(v[t]));
                ptx::named_barrier(1 + g, 128);
                const uint32_t tok0 = ch * kEpiChunk + rsub;  // 16 lanes cover a token's 256 bytes
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const uint4 x = *reinterpret_cast<const uint4*>(stage + (rsub + 8 * k) * kEpiRowBytes + c16 * 16);
                    if (tok0 + 8 * k < it.nt) ptx::st_v4(dst0 + (tok0 + 8 * k) * rowbytes, x);
                }
            }
            if (!released) {  // no chunk for this group
                ptx::tc_fence_before_sync();
                __syncwarp();
                if (lane == 0) ptx::mbar_arrive_cluster(ptx::mapa_u32(&s.tmem_empty_bar[b], 0));
            }
            // Hand the unit to the announcer warp, which has to be done with the one before last.
            const bool free = n < 2 || wait_bar(&s.announced_bar[b], ((n >> 1) - 1u) & 1u, deadline, &s.abort);
            if (!free) {
                if (lane == 0 && !s.abort) report_timeout(cv, kSiteMbar, 0, cta, 6, n);
                s.abort = 1;
            }
            ptx::named_barrier(1 + g, 128);  // the staging buffer may be written again, and all four warps have stored
            if (lane == 0 && free) ptx::mbar_arrive(&s.stored_bar[b]);
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

// NV 16-byte vectors of a row per thread, G ranks per CTA.  CTA b: row b / ngroups, ranks from (b % ngroups) * G.
template <int NV, int G>
__global__ void __launch_bounds__(kLocalLinearNormThreads) local_linear_norm_kernel(const __grid_constant__ LocalLinearNormArgs a) {
    constexpr int VEC = 8, kThreads = kLocalLinearNormThreads, kWarps = kThreads / 32;
    __shared__ float s_red[G][kWarps];
    const CommView& cv = a.cv;
    const uint32_t ngroups = (a.world + G - 1) / G;
    const uint32_t row = blockIdx.x / ngroups, q0 = (blockIdx.x % ngroups) * G;
    const uint32_t tid = threadIdx.x, nvec = a.N / VEC;
    const uint64_t row_off = static_cast<uint64_t>(row) * a.N * 2;
    const uint32_t epoch = *reinterpret_cast<volatile uint32_t*>(flag_word(cv, 0, kCallLocalGemm)) + 1u;

    // Residuals are inputs of the call: complete since before the first kernel passed its own wait.
    uint4 res[NV][G];
#pragma unroll
    for (int j = 0; j < NV; ++j) {
        const uint32_t c = min(tid + j * kThreads, nvec - 1);
#pragma unroll
        for (int g = 0; g < G; ++g) {
            const char* r = q0 + g < a.world ? static_cast<const char*>(a.residual[q0 + g]) : nullptr;
            res[j][g] = r ? ptx::ld_cg_v4(r + row_off + c * 16ull) : make_uint4(0, 0, 0, 0);
        }
    }
    // The flags of this row's token tile, a few per thread.
    const uint32_t tile = row / a.s.tokens, per_tile = a.s.nsplit * (a.N / kLocalGemmUnitCols);
    bool late = false;
    if (tid < per_tile) {
        const uint64_t deadline = ptx::globaltimer() + cv.timeout_ns;
        for (uint32_t e = tid; e < per_tile && !late; e += kThreads) {
            const uint32_t* flag = flag_word(cv, 0, kLocalGemmFlagOff + tile * per_tile + e);
            uint32_t polls = 0, seen;
            while (!ptx::seq_reached(seen = ptx::ld_acquire_gpu(flag), epoch)) {
                ptx::nanosleep(40);  // this CTA shares the SM with the GEMM
                if ((++polls & 63u) == 0 && ptx::globaltimer() > deadline) {
                    report_timeout(cv, kSiteGemmPartials, 0, blockIdx.x, epoch, seen);
                    late = true;
                    break;
                }
            }
        }
    }
    if (__syncthreads_or(late)) return;
    // Everybody has read the call number; the last CTA of the call advances it.
    if (tid == kThreads - 1 && check_in_last(cv, 3, gridDim.x)) advance_call_word(cv, kCallLocalGemm, 1);

    float f[NV][VEC];
#pragma unroll
    for (int j = 0; j < NV; ++j)
#pragma unroll
        for (int i = 0; i < VEC; ++i) f[j][i] = 0.f;
    const uint64_t split_stride = static_cast<uint64_t>(a.T) * a.N * 2;
    const char* const src = a.sums + row_off;
    for (uint32_t k0 = 0; k0 < a.s.nsplit; k0 += 4) {  // four splits in flight, added in order
        uint4 x[NV][4];
#pragma unroll
        for (int k = 0; k < 4; ++k)
#pragma unroll
            for (int j = 0; j < NV; ++j)
                if (k0 + k < a.s.nsplit && tid + j * kThreads < nvec)
                    x[j][k] = ptx::ld_cg_v4(src + (k0 + k) * split_stride + (tid + j * kThreads) * 16ull);
#pragma unroll
        for (int k = 0; k < 4; ++k)
#pragma unroll
            for (int j = 0; j < NV; ++j)
                if (k0 + k < a.s.nsplit && tid + j * kThreads < nvec) accumulate<__nv_bfloat16>(f[j], x[j][k]);
    }
    float ss[G];
#pragma unroll
    for (int g = 0; g < G; ++g) {
        ss[g] = 0.f;
        char* const ro = q0 + g < a.world ? static_cast<char*>(a.residual_out[q0 + g]) : nullptr;
#pragma unroll
        for (int j = 0; j < NV; ++j) {
            if (tid + j * kThreads >= nvec) continue;
            float p[VEC];
#pragma unroll
            for (int i = 0; i < VEC; ++i) p[i] = f[j][i];
            accumulate<__nv_bfloat16>(p, res[j][g]);
            if (ro) ptx::st_v4(ro + row_off + (tid + j * kThreads) * 16ull, pack16<__nv_bfloat16>(p));
#pragma unroll
            for (int i = 0; i < VEC; ++i) ss[g] += p[i] * p[i];
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) ss[g] += __shfl_xor_sync(0xffffffffu, ss[g], o);
        if ((tid & 31) == 0) s_red[g][tid >> 5] = ss[g];
    }
    __syncthreads();
    const float inv_n = 1.f / static_cast<float>(a.N);
#pragma unroll
    for (int g = 0; g < G; ++g) {
        if (q0 + g >= a.world) break;
        float t = 0.f;
#pragma unroll
        for (int w = 0; w < kWarps; ++w) t += s_red[g][w];
        const float inv_rms = rsqrtf(t * inv_n + a.eps);
#pragma unroll
        for (int j = 0; j < NV; ++j) {
            const uint32_t c = tid + j * kThreads;
            if (c >= nvec) continue;
            float p[VEC], w[VEC];
#pragma unroll
            for (int i = 0; i < VEC; ++i) {
                p[i] = f[j][i];
                w[i] = 0.f;
            }
            accumulate<__nv_bfloat16>(p, res[j][g]);
            accumulate<__nv_bfloat16>(w, ptx::ld_cg_v4(static_cast<const char*>(a.weight[q0 + g]) + c * 16ull));
#pragma unroll
            for (int i = 0; i < VEC; ++i) p[i] = p[i] * inv_rms * w[i];
            ptx::st_v4(static_cast<char*>(a.out[q0 + g]) + row_off + c * 16ull, pack16<__nv_bfloat16>(p));
        }
    }
    // The call is over when both kernels are: the CTAs of the last token tile stay for the GEMM's end.
    if (tile + 1 == a.s.tiles) ptx::grid_dependency_wait();
}

}  // namespace

const void* LocalGemmKernel() { return reinterpret_cast<const void*>(local_gemm_kernel); }
uint32_t LocalGemmSmemBytes() { return kSmemBytes; }

const void* LocalLinearNormKernel(uint32_t N, int g) {
    const bool one = N / 8 <= static_cast<uint32_t>(kLocalLinearNormThreads);
    switch (g) {
        case 1: return one ? (const void*)local_linear_norm_kernel<1, 1> : (const void*)local_linear_norm_kernel<2, 1>;
        case 2: return one ? (const void*)local_linear_norm_kernel<1, 2> : (const void*)local_linear_norm_kernel<2, 2>;
        default: return one ? (const void*)local_linear_norm_kernel<1, 4> : (const void*)local_linear_norm_kernel<2, 4>;
    }
}

}  // namespace yali
