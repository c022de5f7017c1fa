// Tensor-parallel output projection fused with its all-reduce, residual add and
// RMSNorm in ONE kernel per rank:
//
//     out = RMSNorm(residual + sum_r x_r @ W_r^T) * norm_weight
//
// x_r is [T, K] (this rank's slice of the attention / MLP activations), W_r is
// [N, K] (this rank's slice of the row-parallel weight, K contiguous, the layout of
// torch.nn.Linear.weight), both bf16; the sum runs over the ranks.
//
// The grid is persistent, one CTA per SM, in clusters of two.  A pair of CTAs computes the transposed tile
// W[256 columns] x x[up to 256 tokens]^T with tcgen05.mma.cta_group::2 (M = 256, N = tokens): each CTA loads 128
// rows of W and half of the tokens' rows, 32 KB per 64-deep k-block for its 128 x 256 outputs, where a CTA on its
// own loads 48 KB.  W is on the M side because a tile can then be any multiple of 32 tokens wide: 300 tokens are
// two tiles of 160, not three of 128.
//
// Roles of a CTA's warps, all running at the same time:
//   0..7    epilogue: read the finished accumulator (tcgen05.ld; thread = column, so 32 tokens at a time are
//           transposed through shared memory), round to bf16 and PUSH every token's 256 bytes into the landing
//           zone of the rank that owns the row (peer stores over NVLink); two TMEM accumulators alternate, so
//           the MMAs of the next tile run meanwhile;
//   8..15   rows, two groups that take turns: add the ranks' partial rows in fp32 in rank order, add the residual, normalise and write the bf16
//           row into EVERY rank's output (two-shot: rows are sharded over the ranks), or, for few rows, every
//           rank owns all rows and writes only its own output (one-shot);
//   16      TMA producer of the GEMM (cp.async.bulk.tensor, 128-byte swizzle, no multicast);
//   17      MMA issuer (leader CTA only);
//   18      announcer: writes the call number into the owners' flag word of the tile unit once its pushes
//           are out.  The release in front of it waits for the peer stores to land (an NVLink round trip), so
//           it sits in a warp of its own;
//   19      row producer: waits (bounded) until all ranks' partial sums of a token tile have landed and streams this
//           CTA's rows of it into a shared-memory ring (cp.async.bulk), several rows ahead of the row warps.
// Rows are therefore finished under the GEMM of the later tiles; only those of the last tiles come after it.
// Bound by the tensor cores (their clock falls to about 1.5 GHz under this load) for 256-token tiles, by the writes of
// the outputs (4.6-5.3 TB/s of stores is what an idle B200 takes) at the end.  Measured in a CUDA graph, ranks
// emulated on one B200, against one-CTA 128 x 256 tiles with a separate row phase: 2 ranks, T = 2048, K = 2048:
// 125 -> 73 us; 8 ranks, T = 300, K = 1792: 98 -> 67 us.
// NVLS form of the two-shot (ranks joined by an NVSwitch multicast object): the
// epilogue keeps the partial rows in this rank's OWN landing zone, so the GEMM has no
// peer stores at all; the owner of a row reads the sum over all ranks with one
// multimem.ld_reduce per 16 bytes (fp32 accumulation in the switch) and delivers the
// normalised row to every rank with one multimem.st.  An SM then issues 1/W of the
// loads and stores; on the links the switch still pulls (W-1)/W * T*N*2 bytes out of
// every rank for the sums, while delivery sends only T*N*2/W per rank.  A third form
// keeps the peer pushes and uses the switch for delivery alone.
//
// Parity: none in the reference (it has no GEMM, no fused op and no tensor-core
// code; see its src/kernels and src/all_reduce).  The unfused composition (library
// GEMM, all-reduce, separate norm kernel) is kept in Python as the baseline.
#include <cuda.h>

#include "gemm_ar_rmsnorm.h"
#include "tc_common.cuh"

namespace yali {

namespace {

constexpr int BK = 64;                      // BK bf16 = one 128-byte swizzle row
constexpr uint32_t kWBytes = 128 * BK * 2;  // one CTA's half of the W operand of a stage
// Shared memory: the GEMM ran 7 % faster with five 32 KB stages than with four (loads take 1.5-2 us under load, and
// that is what the stages have to cover), so the rows get what is left.
constexpr uint32_t kRingBytes = 160 * 1024;  // operand stages of the GEMM: 5 of 32 KB (256 tokens) to 8 of 18 KB (32)
constexpr int kMaxStages = 8;
constexpr uint32_t kRowRingBytes = 48 * 1024;  // rows on their way to the row warps: 3 of 8 KB (N = 4096) per row group
constexpr int kMaxRowSlots = 8;  // per row group
constexpr uint32_t kEpiChunk = 32;                           // tokens an epilogue group moves at a time
constexpr uint32_t kEpiRowBytes = kGemmUnitCols * 2;         // 256 bytes per token
constexpr uint32_t kEpiBufBytes = kEpiChunk * kEpiRowBytes;  // 8 KiB; one per group of four warps
constexpr uint32_t kSmemBytes = kRingBytes + kRowRingBytes + 1024;  // + slack to align the base
constexpr uint32_t kTmemCols = 2 * kGemmMaxTokens;                  // two accumulators: all of TMEM
constexpr int kEpiGroups = 2, kEpilogueWarps = 4 * kEpiGroups;
constexpr int kRowGroups = 2, kRowWarps = 4;  // warps of a group
constexpr int kTmaWarp = 16, kMmaWarp = 17, kAnnounceWarp = 18, kRowTmaWarp = 19;
constexpr uint32_t kRowBarrier = 1 + kEpiGroups;  // named barriers: 1.. epilogue groups, then the row warps
static_assert(kRowGroups == 2 && kRowRingBytes / kRowGroups >= 2 * kGemmMaxRowVecs * 16, "two rows at least");
static_assert(kTmemCols == 512 && kGemmThreads == 32 * (kRowTmaWarp + 1), "one CTA per SM");
static_assert(kSmemBytes + kEpiGroups * kEpiBufBytes + 1024 <= 227 * 1024, "shared memory of one SM");

// Landing zone of the partial rows of source `src` on a rank, relative to that rank's heap base.
__device__ __forceinline__ uint64_t landing_off(const GemmArArgs& a, int src, uint32_t parity) {
    return a.cv.lay.gemm_off + (static_cast<uint64_t>(parity) * a.cv.world + src) * a.cv.lay.gemm_cap;
}

// NVLS form: one [T, N] bf16 image per call parity at the same offset of every rank's heap.
__device__ __forceinline__ uint64_t landing_nvls_off(const GemmArArgs& a, uint32_t parity) {
    return a.cv.lay.gemm_off + static_cast<uint64_t>(parity) * a.cv.world * a.cv.lay.gemm_cap;
}

using Item = GemmItem;
__device__ __forceinline__ Item item_at(const GemmArArgs& a, uint32_t i, uint32_t ncol, uint32_t ks_shift) {
    return GemmItemAt(a.tl, a.T, static_cast<uint32_t>(a.cv.rank), i, ncol, ks_shift);
}

// State the roles share.
struct Shared {
    __align__(8) uint64_t full_bar[kMaxStages], empty_bar[kMaxStages], tmem_full_bar[2], tmem_empty_bar[2];
    __align__(8) uint64_t pushed_bar[2], announced_bar[2];  // epilogue warps -> announcer warp and back
    __align__(8) uint64_t drain_bar;  // all MMAs have finished
    __align__(8) uint64_t row_full[kRowGroups][kMaxRowSlots], row_empty[kRowGroups][kMaxRowSlots];
    uint32_t tmem, row_armed[kRowGroups];  // row_armed: pieces of rows that have been asked for
    char* heap[kMaxRanks];  // the heap bases: read with a run-time rank
    volatile int abort;
    uint32_t call[1 + kMaxRanks];
    float red[kRowGroups][2][kRowWarps];  // sums of squares of the row warps, two rows alternating
};

// The rows this rank normalises (CTA c takes rows c, c + nctas, ...) and how they travel through the row ring.
struct MyRows {
    uint32_t lo, n;           // first of them in the [T, N] images, their number
    uint32_t nsrc, ks_shift;  // partial rows per row: source q = (rank q >> ks_shift, K split), at most kMaxRanks
    uint32_t chunks;          // pieces of a row in the ring: partial rows in source order, then the residual
    uint32_t slots;           // of a group's ring
};
__device__ __forceinline__ MyRows my_rows(const GemmArArgs& a) {
    MyRows m;
    m.lo = a.oneshot ? 0u : min(a.T, static_cast<uint32_t>(a.cv.rank) * a.rows_per_owner);
    m.n = (a.oneshot ? a.T : min(a.T, m.lo + a.rows_per_owner)) - m.lo;
    m.ks_shift = 31 - __clz(a.ksplit);
    m.nsrc = static_cast<uint32_t>(a.cv.world) << m.ks_shift;
    m.chunks = (a.nvls ? 0u : m.nsrc) + (a.residual ? 1u : 0u);
    m.slots = min(kRowRingBytes / kRowGroups / (a.N * 2), static_cast<uint32_t>(kMaxRowSlots));
    return m;
}

// Row producer (one warp).
__device__ __forceinline__ void row_producer(const GemmArArgs& a, Shared& s, uint8_t* ring, uint32_t cta, uint32_t nctas,
                                             uint32_t epoch, uint64_t deadline) {
    const CommView& cv = a.cv;
    const int r = cv.rank;
    const uint32_t lane = threadIdx.x & 31, W = cv.world;
    const MyRows m = my_rows(a);
    const uint32_t per_tile = (a.N / kGemmUnitCols) << m.ks_shift;  // announcements of a source per token tile
    const uint32_t rowbytes = a.N * 2;
    const uint64_t split_cap = cv.lay.gemm_cap >> m.ks_shift;
    const char* const landing = s.heap[r] + landing_off(a, 0, epoch & 1u);
    uint32_t ready = ~0u, group = 0;
    uint32_t slots[kRowGroups] = {}, rounds[kRowGroups] = {};
    for (uint32_t lr = cta; lr < m.n; lr += nctas, group ^= 1u) {
        uint64_t* const full = s.row_full[group];
        uint64_t* const empty = s.row_empty[group];
        uint8_t* const mine = ring + group * (kRowRingBytes / kRowGroups);
        uint32_t slot = group ? slots[1] : slots[0], round = group ? rounds[1] : rounds[0];
        const uint32_t grow = m.lo + lr;
        const uint32_t tile = GemmTileOfRow(a.tl, grow);
        bool late = false;
        if (tile != ready) {
            // The flags of all (128-column unit, K split, source) of the row's token tile, a few per lane.
            for (uint32_t e = lane; e < per_tile * W && !late; e += 32) {
                const uint32_t src = e % W, word = kGemmTileFlagOff + (tile * per_tile + e / W) * kMaxRanks + src;
                uint32_t seen;
                if (!ptx::wait_flag_reached(flag_word(cv, r, word), epoch, deadline, &seen)) {
                    if (!s.abort) report_timeout(cv, kSiteGemmPartials, src, cta, epoch, seen);
                    s.abort = 1;
                    late = true;
                }
            }
            if (a.trace && cta == 0 && lane == 0 && ready == ~0u) a.trace[5] = ptx::globaltimer();
            ready = tile;
        }
        if (__any_sync(0xffffffffu, late)) break;
        // The acquires above, ordered before the whole warp, cover the partial rows; the bulk copies read them
        // through the async proxy.
        ptx::fence_proxy_async();
        const char* const part = landing + static_cast<uint64_t>(lr) * rowbytes;
        for (uint32_t k = 0; k < max(m.chunks, 1u); ++k) {
            late = !wait_bar(&empty[slot], (round & 1u) ^ 1u, deadline, &s.abort);
            if (__any_sync(0xffffffffu, late)) {
                s.abort = 1;
                break;
            }
            if (ptx::elect_one()) {
                if (m.chunks == 0) {
                    ptx::mbar_arrive(&full[slot]);  // nothing to copy: only "the row is there"
                } else {
                    const bool is_res = a.residual && k == m.chunks - 1;
                    const char* src = is_res ? static_cast<const char*>(a.residual) + static_cast<uint64_t>(grow) * rowbytes
                                             : part + (k >> m.ks_shift) * cv.lay.gemm_cap + (k & (a.ksplit - 1)) * split_cap;
                    ptx::mbar_expect_tx(&full[slot], rowbytes);
                    ptx::bulk_g2s(mine + slot * rowbytes, src, rowbytes, &full[slot]);
                }
            }
            __syncwarp();
            if (++slot == m.slots) slot = 0, ++round;
        }
        slots[0] = group ? slots[0] : slot;
        rounds[0] = group ? rounds[0] : round;
        slots[1] = group ? slot : slots[1];
        rounds[1] = group ? round : rounds[1];
        if (__any_sync(0xffffffffu, late)) break;
    }
    if (lane == 0) {
        s.row_armed[0] = rounds[0] * m.slots + slots[0];
        s.row_armed[1] = rounds[1] * m.slots + slots[1];
    }
}

// The four warps of row group `group`: every second of this CTA's rows (two groups, because a row is a chain of latencies:
// 0.3 us per chunk, 0.3 us for the reduction, 1 us of stores).  Returns the rows written.  All threads of a group
// leave the loop at the same place: a wait that ran out is carried to the row's barrier.
__device__ __forceinline__ uint32_t row_consumers(const GemmArArgs& a, Shared& s, const uint8_t* ring, uint32_t group,
                                                  uint32_t cta, uint32_t nctas, uint32_t epoch, uint64_t deadline) {
    constexpr int VEC = 8, NV = kGemmMaxRowVecs / (32 * kRowWarps);  // a thread holds four 16-byte vectors of a row
    constexpr uint32_t kStep = 32 * kRowWarps;
    const CommView& cv = a.cv;
    const int W = cv.world, r = cv.rank;
    const uint32_t t = threadIdx.x % kStep, lane = t & 31;
    const MyRows m = my_rows(a);
    const uint32_t rowbytes = a.N * 2, nvec = a.N / VEC, chunks = max(m.chunks, 1u);
    const char* const mc_in = cv.mc_heap + landing_nvls_off(a, epoch & 1u);
    const char* const wgt = static_cast<const char*>(a.norm_weight);
    char* res_out = static_cast<char*>(a.residual_out);
    const float inv_n = 1.f / static_cast<float>(a.N);
    uint32_t slot = 0, round = 0, done = 0;
    ring += group * (kRowRingBytes / kRowGroups);  // a ring of its own
    for (uint32_t lr = cta + group * nctas; lr < m.n; lr += kRowGroups * nctas) {
        const uint64_t goff0 = static_cast<uint64_t>(m.lo + lr) * rowbytes;  // this row in [T, N] images
        float f[NV][VEC];
#pragma unroll
        for (int j = 0; j < NV; ++j)
#pragma unroll
            for (int i = 0; i < VEC; ++i) f[j][i] = 0.f;
        bool late = false;
        for (uint32_t k = 0; k < chunks; ++k) {
            if (!wait_bar(&s.row_full[group][slot], round & 1u, deadline, &s.abort)) {
                if (lane == 0 && !s.abort) report_timeout(cv, kSiteMbar, r, cta, 7, done);
                s.abort = 1;
                late = true;
                break;
            }
            if (a.nvls && k == 0) {  // the switch adds the copies of all ranks
#pragma unroll
                for (int j = 0; j < NV; ++j)
                    if (t + j * kStep < nvec)
                        accumulate<__nv_bfloat16>(f[j], ptx::multimem_ld_reduce_bf16x8(mc_in + goff0 + (t + j * kStep) * 16ull));
            }
            if (m.chunks != 0) {
                const uint4* const src = reinterpret_cast<const uint4*>(ring + slot * rowbytes);
                uint4 x[NV];
#pragma unroll
                for (int j = 0; j < NV; ++j) x[j] = t + j * kStep < nvec ? src[t + j * kStep] : make_uint4(0, 0, 0, 0);
#pragma unroll
                for (int j = 0; j < NV; ++j) accumulate<__nv_bfloat16>(f[j], x[j]);
            }
            __syncwarp();
            if (lane == 0) ptx::mbar_arrive(&s.row_empty[group][slot]);
            if (++slot == m.slots) slot = 0, ++round;
        }
        float ss = 0.f;
#pragma unroll
        for (int j = 0; j < NV; ++j) {
#pragma unroll
            for (int i = 0; i < VEC; ++i) ss += f[j][i] * f[j][i];
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
        float* const red = s.red[group][done & 1u];
        if (lane == 0) red[t >> 5] = ss;
        if (ptx::named_barrier_or(kRowBarrier + group, kStep, late)) break;
        const float inv_rms = rsqrtf((red[0] + red[1] + red[2] + red[3]) * inv_n + a.eps);
#pragma unroll
        for (int j = 0; j < NV; ++j) {
            if (t + j * kStep >= nvec) continue;
            const uint64_t goff = goff0 + (t + j * kStep) * 16ull;
            const uint4 pre = pack16<__nv_bfloat16>(f[j]);
            float w[VEC];
#pragma unroll
            for (int i = 0; i < VEC; ++i) w[i] = 0.f;
            accumulate<__nv_bfloat16>(w, *reinterpret_cast<const uint4*>(wgt + (t + j * kStep) * 16ull));
#pragma unroll
            for (int i = 0; i < VEC; ++i) w[i] = f[j][i] * inv_rms * w[i];
            const uint4 y = pack16<__nv_bfloat16>(w);
            if (a.oneshot) {
                if (res_out) ptx::st_v4(res_out + goff, pre);
                ptx::st_v4(static_cast<char*>(a.out[r]) + goff, y);
                continue;
            }
            if (a.residual_out_mc) {  // one store through the switch fills every rank's copy
                ptx::multimem_st_v4(a.residual_out_mc + goff, pre);
            } else if (res_out) {  // the owner of the row fills every rank's copy
                for (int k = 0, d = r; k < W; ++k) {
                    char* dst = static_cast<char*>(a.residual_out_all[d]);
                    if (dst) ptx::st_v4(dst + goff, pre);
                    if (++d == W) d = 0;
                }
            }
            if (a.out_mc) {
                ptx::multimem_st_v4(a.out_mc + goff, y);
            } else {
                for (int k = 0, d = r; k < W; ++k) {
                    ptx::st_v4(static_cast<char*>(a.out[d]) + goff, y);
                    if (++d == W) d = 0;
                }
            }
        }
        ++done;
    }
    return done;
}

__device__ __forceinline__ void gemm_ar_body(const GemmArArgs& a, uint32_t cta, uint32_t nctas) {
    extern __shared__ uint8_t smem_raw[];
    __shared__ Shared s;
    __shared__ __align__(16) uint8_t s_epi[kEpiGroups][kEpiBufBytes];

    const CommView& cv = a.cv;
    const int W = cv.world, r = cv.rank;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t half = ptx::cluster_cta_rank();  // which 128 of the pair's 256 columns, which half of its tokens
    ptx::grid_dependency_wait();
    const uint64_t deadline = ptx::globaltimer() + cv.timeout_ns;
    // Optional timeline of CTA 0 (a.trace != nullptr): %globaltimer at the phase boundaries.
#define YALI_STAMP(slot, who)                                                              \
    do {                                                                                   \
        if (a.trace && cta == 0 && tid == (who)) a.trace[slot] = ptx::globaltimer();       \
    } while (0)
    YALI_STAMP(0, 0);  // entry
    // Call number and counter targets come from this rank's call words (advanced by the last
    // CTA of the previous launch), so the launch itself carries no per-call state.
    if (tid >= 32 && tid < 32 + kMaxRanks) s.heap[tid - 32] = cv.heap[tid - 32];
    if (tid < 1 + W) {
        const uint32_t word = tid == 0 ? kCallGemmEpoch : kCallGemmDone + (tid - 1);
        s.call[tid] = *reinterpret_cast<volatile uint32_t*>(flag_word(cv, r, word));
    }
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint8_t* row_ring = smem + kRingBytes;
    if (tid == 64) {
        s.abort = 0;
        for (int i = 0; i < kMaxStages; ++i) {
            ptx::mbar_init(&s.full_bar[i], 1);
            ptx::mbar_init(&s.empty_bar[i], 1);
        }
        for (int b = 0; b < 2; ++b) {
            ptx::mbar_init(&s.tmem_full_bar[b], 1);
            ptx::mbar_init(&s.tmem_empty_bar[b], 2 * kEpilogueWarps);  // the epilogue warps of both CTAs
            ptx::mbar_init(&s.pushed_bar[b], kEpilogueWarps);
            ptx::mbar_init(&s.announced_bar[b], 1);
        }
        ptx::mbar_init(&s.drain_bar, 1);
        for (int i = 0; i < kRowGroups * kMaxRowSlots; ++i) {
            ptx::mbar_init(&s.row_full[0][0] + i, 1);
            ptx::mbar_init(&s.row_empty[0][0] + i, kRowWarps);
        }
        ptx::mbar_fence_init();
        ptx::tma_prefetch_desc(&a.tmap_w);
        ptx::tma_prefetch_desc(&a.tmap_x);
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
    if (tid == 32 * kRowTmaWarp && check_in_last(cv, 3, nctas)) {
        advance_call_word(cv, kCallGemmEpoch, 1);
        for (int q = 0; q < W; ++q) advance_call_word(cv, kCallGemmDone + q, a.done_inc[q]);
    }
    const uint32_t tmem = s.tmem;
    const uint32_t epoch = s.call[0] + 1u, parity = epoch & 1u;
    YALI_STAMP(1, 0);  // barriers initialised, TMEM allocated

    const uint32_t ncol = (a.N + kGemmPairCols - 1) / kGemmPairCols, kblocks = a.K / BK;
    const uint32_t ks_shift = 31 - __clz(a.ksplit), kper = a.kper;
    const uint32_t nitems = (a.tl.domains * a.tl.tiles * ncol) << ks_shift;
    const uint32_t pair = cta >> 1, npairs = nctas >> 1;
    const uint32_t xbytes = a.tl.tokens / 2 * (BK * 2);  // one CTA's half of the token operand of a stage: whole KiB
    const uint32_t stage_bytes = kWBytes + xbytes;
    const uint32_t stages = min(kRingBytes / stage_bytes, static_cast<uint32_t>(kMaxStages));

    // The issuing thread of a role is picked by elect.sync, not by its lane number: with it the compiler knows that one
    // thread runs, and issues TMA and MMA instructions straight; behind a lane test it wraps each of them in
    // a loop over the active threads.  Measured per 64-deep k-block (wait, 4 MMAs of N = 160, commit):
    // 540 cycles with the lane test, 390 with elect.sync; the MMAs alone take 320.
    if (warp == kTmaWarp) {
        if (ptx::elect_one()) {
            uint32_t st = 0, round = 0;
            for (uint32_t i = pair; i < nitems && !s.abort; i += npairs) {
                const Item it = item_at(a, i, ncol, ks_shift);
                if (it.nt == 0) continue;
                const int wrow = it.col_tile * kGemmPairCols + half * kGemmUnitCols, xrow = it.t0 + half * (a.tl.tokens / 2);
                const uint32_t kb_end = min(kblocks, (it.split + 1) * kper);
                for (uint32_t kb = it.split * kper; kb < kb_end; ++kb) {
                    if (!wait_bar(&s.empty_bar[st], (round & 1u) ^ 1u, deadline, &s.abort)) {
                        if (!s.abort) report_timeout(cv, kSiteMbar, r, cta, 1, kb);
                        s.abort = 1;
                        break;
                    }
                    // Both halves are counted on the leader's barrier, which its own producer arms.
                    if (half == 0) ptx::mbar_expect_tx(&s.full_bar[st], 2 * stage_bytes);
                    const uint32_t bar = ptx::mapa_u32(&s.full_bar[st], 0);
                    uint8_t* stage = smem + st * stage_bytes;
                    ptx::tma_load_2d_pair(stage, &a.tmap_w, kb * BK, wrow, bar);
                    ptx::tma_load_2d_pair(stage + kWBytes, &a.tmap_x, kb * BK, xrow, bar);
                    if (++st == stages) st = 0, ++round;
                }
            }
            // The MMAs' releases of the last stages arrive here from the leader: none may be under way when this CTA
            // leaves.
            bool up = !s.abort;
            const uint32_t loaded = round * stages + st;
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
            const uint32_t idesc = mma_idesc_bf16(kGemmPairCols, a.tl.tokens);
            uint32_t st = 0, round = 0, n = 0;
            for (uint32_t i = pair; i < nitems && !s.abort; i += npairs) {
                const Item it = item_at(a, i, ncol, ks_shift);
                if (it.nt == 0) continue;
                const uint32_t kb_begin = it.split * kper, kb_end = min(kblocks, (it.split + 1) * kper);
                const uint32_t b = n & 1u;
                if (!wait_bar(&s.tmem_empty_bar[b], ((n >> 1) & 1u) ^ 1u, deadline, &s.abort)) {
                    if (!s.abort) report_timeout(cv, kSiteMbar, r, cta, 4, n);
                    s.abort = 1;
                    break;
                }
                ptx::tc_fence_after_sync();
                const uint32_t d_tmem = tmem + b * kGemmMaxTokens;
                for (uint32_t kb = kb_begin; kb < kb_end; ++kb) {
                    if (!wait_bar(&s.full_bar[st], round & 1u, deadline, &s.abort)) {
                        if (!s.abort) report_timeout(cv, kSiteMbar, r, cta, 2, kb);
                        s.abort = 1;
                        break;
                    }
                    ptx::tc_fence_after_sync();
                    const uint32_t addr = ptx::smem_u32(smem + st * stage_bytes);
                    const uint64_t dw = smem_desc_sw128(addr), dx = smem_desc_sw128(addr + kWBytes);
#pragma unroll
                    for (int k = 0; k < BK / 16; ++k)
                        // 16 bf16 = 32 bytes further along K inside the swizzle row: +2 in the address field
                        ptx::tc_mma_f16_pair(d_tmem, dw + 2 * k, dx + 2 * k, idesc, (kb != kb_begin || k != 0) ? 1u : 0u);
                    ptx::tc_commit_pair(&s.empty_bar[st]);  // frees the stage in both CTAs when these MMAs have read it
                    if (++st == stages) st = 0, ++round;
                }
                if (s.abort) break;
                ptx::tc_commit_pair(&s.tmem_full_bar[b]);  // accumulator complete
                ++n;
            }
            if (n > 0 || s.abort) {  // a pair without items leaves at once
                ptx::tc_commit_pair(&s.drain_bar);
                mbar_drain(&s.drain_bar, 0);
            }
        }
    } else if (warp == kAnnounceWarp) {
        // When the eight epilogue warps have issued the pushes of a tile unit, tell every owner of rows of it.
        // The release orders the pushes (made visible to this warp by the mbarrier) before the flag.
        uint32_t n = 0;
        for (uint32_t i = pair; i < nitems; i += npairs) {
            const Item it = item_at(a, i, ncol, ks_shift);
            if (it.nt == 0) continue;
            const uint32_t b = n & 1u, unit = it.col_tile * 2 + half;
            if (!wait_bar(&s.pushed_bar[b], (n >> 1) & 1u, deadline, &s.abort)) {
                if (lane == 0 && !s.abort) report_timeout(cv, kSiteMbar, r, cta, 5, n);
                s.abort = 1;
                break;
            }
            if (lane < W && unit * kGemmUnitCols < a.N) {
                const uint32_t Rs = a.rows_per_owner, q = lane;
                const bool touched = a.oneshot || (q * Rs < it.t0 + it.nt && (q + 1) * Rs > it.t0);
                const uint32_t idx = ((it.tile * (a.N / kGemmUnitCols) + unit) << ks_shift) + it.split;
                uint32_t* flag = flag_word(cv, q, kGemmTileFlagOff + idx * kMaxRanks + r);
                if (touched) {
                    if (a.one_gpu) ptx::st_release_gpu(flag, epoch);
                    else ptx::st_release_sys(flag, epoch);
                }
            }
            __syncwarp();
            if (lane == 0) ptx::mbar_arrive(&s.announced_bar[b]);
            if (n == 0) YALI_STAMP(3, kAnnounceWarp * 32);  // first tile pushed and announced
            ++n;
        }
    } else if (warp < kEpilogueWarps) {
        const int q = warp & 3;   // TMEM lane quarter this warp may read: columns 32q .. 32q+31 of the CTA's 128
        const int g = warp >> 2;  // its group takes every second chunk of 32 tokens
        const int gt = tid & 127;
        const uint32_t c16 = gt & 15, rsub = gt >> 4;  // pushes: 16-byte piece of a token's 256 bytes, token % 8
        const uint64_t rowbytes = static_cast<uint64_t>(a.N) * 2, split_cap = cv.lay.gemm_cap >> ks_shift;
        const uint32_t Rs = a.rows_per_owner;
        const uint64_t land = landing_off(a, r, parity);  // where this rank's partial rows go on every owner
        uint8_t* const stage = s_epi[g];
        uint32_t n = 0;
        for (uint32_t i = pair; i < nitems; i += npairs) {
            const Item it = item_at(a, i, ncol, ks_shift);
            if (it.nt == 0) continue;
            const uint32_t b = n & 1u;
            const uint32_t col = it.col_tile * kGemmPairCols + half * kGemmUnitCols;
            const uint64_t col_off = static_cast<uint64_t>(col) * 2 + c16 * 16;
            // The second half of the last column tile may lie beyond N.
            const uint32_t chunks = col < a.N ? (it.nt + kEpiChunk - 1) / kEpiChunk : 0u;
            // Owner and local row of this thread's first token (one division, while the MMAs of the tile run).
            uint32_t grow0 = it.t0 + g * kEpiChunk + rsub;
            uint32_t d = 0, local = grow0;
            if (!a.nvls && !a.oneshot) {
                d = grow0 / Rs;
                local = grow0 - d * Rs;
            }
            // Every warp of a group has to take the same way through the chunks (they share a barrier).
            const bool up = wait_bar(&s.tmem_full_bar[b], (n >> 1) & 1u, deadline, &s.abort);
            if (!up) {
                if (lane == 0 && !s.abort) report_timeout(cv, kSiteMbar, r, cta, 3, n);
                s.abort = 1;
            }
            if (ptx::named_barrier_or(1 + g, 128, !up)) break;
            ptx::tc_fence_after_sync();
            if (n == 0) YALI_STAMP(2, 0);  // first accumulator complete
            bool released = false;
            for (uint32_t ch = g; ch < chunks; ch += kEpiGroups) {
                uint32_t v[32];
                ptx::tmem_ld_32x32(tmem + b * kGemmMaxTokens + (static_cast<uint32_t>(q * 32) << 16) + ch * kEpiChunk, v);
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
                uint4 x[4];
#pragma unroll
                for (int k = 0; k < 4; ++k)
                    x[k] = *reinterpret_cast<const uint4*>(stage + (rsub + 8 * k) * kEpiRowBytes + c16 * 16);
                // Push: 16 lanes cover a token's 256 bytes.
                const uint32_t tok0 = ch * kEpiChunk + rsub;
                if (a.nvls) {
                    char* p = s.heap[r] + landing_nvls_off(a, parity) + static_cast<uint64_t>(it.t0 + tok0) * rowbytes + col_off;
#pragma unroll
                    for (int k = 0; k < 4; ++k)
                        if (tok0 + 8 * k < it.nt) ptx::st_v4(p + static_cast<uint64_t>(8 * k) * rowbytes, x[k]);
                } else if (a.oneshot) {
                    const uint64_t off = land + it.split * split_cap + static_cast<uint64_t>(it.t0 + tok0) * rowbytes + col_off;
                    for (int k = 0, dst = r; k < W; ++k) {
                        if (++dst == W) dst = 0;  // the peers first, the own copy last
                        char* p = s.heap[dst] + off;
#pragma unroll
                        for (int k4 = 0; k4 < 4; ++k4)
                            if (tok0 + 8 * k4 < it.nt) ptx::st_v4(p + static_cast<uint64_t>(8 * k4) * rowbytes, x[k4]);
                    }
                } else {
                    // Tokens 8 apart, then on to this group's next chunk; rows run on into the next owner's.
#pragma unroll
                    for (int k = 0; k < 4 + 4; ++k) {
                        while (local >= Rs && d + 1 < static_cast<uint32_t>(W)) {
                            local -= Rs;
                            ++d;
                        }
                        if (k < 4 && tok0 + 8 * k < it.nt)
                            ptx::st_v4(s.heap[d] + land + static_cast<uint64_t>(local) * rowbytes + col_off, x[k < 4 ? k : 0]);
                        local += 8;
                    }
                }
            }
            if (!released) {  // no chunk for this group
                ptx::tc_fence_before_sync();
                __syncwarp();
                if (lane == 0) ptx::mbar_arrive_cluster(ptx::mapa_u32(&s.tmem_empty_bar[b], 0));
            }
            // This warp's pushes of the tile are issued: hand it to the announcer warp, which has to be done with the
            // tile before last (it is, unless it lags two tiles behind).
            const bool free = n < 2 || wait_bar(&s.announced_bar[b], ((n >> 1) - 1u) & 1u, deadline, &s.abort);
            if (!free) {
                if (lane == 0 && !s.abort) report_timeout(cv, kSiteMbar, r, cta, 6, n);
                s.abort = 1;
            }
            __syncwarp();
            if (lane == 0 && free) ptx::mbar_arrive(&s.pushed_bar[b]);
            ++n;
        }
        YALI_STAMP(4, 0);  // all tiles of this CTA pushed
    } else if (warp == kRowTmaWarp) {
        row_producer(a, s, row_ring, cta, nctas, epoch, deadline);
    } else {
        const uint32_t group = (warp - kEpilogueWarps) / kRowWarps;
        const uint32_t rows_done = row_consumers(a, s, row_ring, group, cta, nctas, epoch, deadline);
        // Two-shot: tell every rank how many of its output rows this group delivered.
        ptx::named_barrier(kRowBarrier + group, 32 * kRowWarps);
        const int t = tid % (32 * kRowWarps);
        // (Where one launch on one GPU runs all ranks, its end delivers them.)
        if (!a.oneshot && !a.one_gpu && t < W && rows_done > 0) ptx::red_release_sys_add(flag_word(cv, t, kGemmDoneOff + r), rows_done);
    }
    __syncwarp();
    ptx::tc_fence_before_sync();
    __syncthreads();
    YALI_STAMP(6, 0);  // own rows reduced and written
    // Row warps that stop early leave copies on their way into the ring.
    if (s.abort && warp == kRowTmaWarp && lane < kRowGroups) mbar_drain_ring(s.row_full[lane], my_rows(a).slots, s.row_armed[lane]);
    __syncwarp();
    // Nobody leaves (or gives TMEM back) while the other CTA's MMAs, loads or arrivals may still reach this one.
    ptx::cluster_arrive();
    ptx::cluster_wait();
    if (warp == kMmaWarp) ptx::tmem_dealloc_pair(tmem, kTmemCols);
    if (s.abort) return;
    // Two-shot: this rank's output is complete when every owner's rows have landed.  One CTA
    // waits; the kernel cannot finish before it does.
    if (!a.oneshot && !a.one_gpu && cta == 0) {
        if (tid < W) {
            uint32_t seen;
            const uint32_t want = s.call[1 + tid] + a.done_inc[tid];
            if (!ptx::wait_flag_reached(flag_word(cv, r, kGemmDoneOff + tid), want, deadline, &seen)) {
                report_timeout(cv, kSiteGemmDone, tid, cta, want, seen);
                s.abort = 1;
            }
        }
        __syncthreads();
        if (s.abort) return;
    }
    YALI_STAMP(7, 0);  // output complete
#undef YALI_STAMP
}

}  // namespace

__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kGemmThreads, 1)
    gemm_ar_rmsnorm_kernel(const __grid_constant__ GemmArArgs a) {
    gemm_ar_body(a, blockIdx.x, gridDim.x);
}

// All ranks of an emulated communicator in one cooperative launch (ranks = blockIdx.y).
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kGemmThreads, 1)
    gemm_ar_rmsnorm_kernel_emu(const __grid_constant__ GemmArEmuArgs e) {
    gemm_ar_body(e.r[blockIdx.y], blockIdx.x, gridDim.x);
}

const void* GemmArKernel(bool emu) {
    return emu ? reinterpret_cast<const void*>(gemm_ar_rmsnorm_kernel_emu)
               : reinterpret_cast<const void*>(gemm_ar_rmsnorm_kernel);
}
uint32_t GemmArSmemBytes() { return kSmemBytes; }

}  // namespace yali
