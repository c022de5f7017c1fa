#include "fused_linear.h"

#include "../core/env.h"
#include "../core/nvtx.h"

#include <algorithm>
#include <atomic>
#include <cstring>
#include <map>
#include <mutex>
#include <set>

#include "../comm/cuda_driver.h"
#include "../kernels/gemm_ar_rmsnorm.h"
#include "../kernels/launch.h"

namespace yali {

namespace {

bool EncodeTileMap(const DriverApi* d, CUtensorMap* map, const void* base, uint64_t rows, uint64_t cols_k,
                   uint32_t box_rows, std::string* err);

// Few-token form: one launch of gemm_ar_decode.cu per rank.
Result LaunchDecode(Communicator& comm, const DriverApi* drv, const FusedLinearDesc* descs, uint32_t T, uint32_t N,
                    uint32_t K, const FusedLinearOptions& opt, const cudaStream_t* streams) {
    const int W = comm.world(), nlocal = comm.nlocal();
    auto fail = [&](Result r, const std::string& what) {
        comm.set_error(what);
        return r;
    };
    const void* fn = GemmDecodeKernel(comm.emulated());
    const uint32_t smem = GemmDecodeSmemBytes();
    static std::mutex attr_mu;
    static std::set<std::pair<int, int>> attr_done;
    {
        std::lock_guard<std::mutex> lock(attr_mu);
        for (int i = 0; i < nlocal; ++i) {
            const std::pair<int, int> key(comm.emulated() ? 1 : 0, comm.device_of(i));
            if (attr_done.count(key)) continue;
            if (nlocal > 1) cudaSetDevice(comm.device_of(i));
            cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
            if (e != cudaSuccess) return fail(Result::CudaError, std::string("cudaFuncSetAttribute: ") + cudaGetErrorString(e));
            attr_done.insert(key);
        }
    }
    int sms = 0;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, comm.device_of(0));
    // One CTA per SM (160 KiB of stages each); emulated ranks share the GPU.
    uint32_t resident = static_cast<uint32_t>(std::max(1, sms));
    if (comm.emulated()) resident = std::max<uint32_t>(1, resident / W);
    const uint32_t kblocks = K / 64;
    static const long long forced = env::GetInt("YALI_GEMM_DECODE_KSPLIT", 0);  // measurements only
    static const long long forced_tile = env::GetInt("YALI_GEMM_DECODE_TILE", 0);
    const uint32_t ksplit = FusedLinearDecodeSplit(T, N, K, W, resident, comm.layout().gemm_ll_cap,
                                                   forced > 0 ? static_cast<uint32_t>(forced) : 0u);
    uint32_t tile_n = FusedLinearDecodeTile(N, ksplit, resident);
    if (forced_tile == 128 || forced_tile == 256) tile_n = static_cast<uint32_t>(forced_tile);
    const uint32_t ntn = (N + tile_n - 1) / tile_n;
    const uint32_t kper = (kblocks + ksplit - 1) / ksplit;
    uint32_t ctas = std::min<uint32_t>(resident, ntn * ksplit);
    ctas = std::max<uint32_t>(ctas, std::min<uint32_t>(resident, T));  // CTA t normalises row t
    if (opt.ctas > 0) ctas = std::min<uint32_t>(ctas, opt.ctas);
    std::string derr;
    std::vector<GemmDecodeArgs> args(nlocal);
    for (int i = 0; i < nlocal; ++i) {
        GemmDecodeArgs& a = args[i];
        std::memset(&a, 0, sizeof(a));
        const FusedLinearDesc& d = descs[i];
        if (nlocal > 1) cudaSetDevice(comm.device_of(i));
        const uint32_t a_box_rows = T <= 8 ? 8u : T <= 16 ? 16u : T <= 32 ? 32u : 64u;
        if (!EncodeTileMap(drv, &a.tmap_a, d.x, T, K, a_box_rows, &derr) ||
            !EncodeTileMap(drv, &a.tmap_b, d.w, N, K, tile_n, &derr))
            return fail(Result::CudaError, derr);
        a.a_box_rows = a_box_rows;
        a.tile_n = tile_n;
        a.ksplit = ksplit;
        a.kper = kper;
        a.cv = comm.View(i);
        a.residual = d.residual;
        a.residual_out = d.residual_out;
        a.norm_weight = d.norm_weight;
        a.out = d.out;
        a.T = T;
        a.N = N;
        a.K = K;
        a.eps = opt.eps;
        a.trace = opt.trace ? opt.trace[i] : nullptr;
    }
    if (comm.emulated()) {
        GemmDecodeEmuArgs* e = new GemmDecodeEmuArgs();
        std::memset(e, 0, sizeof(*e));
        for (int i = 0; i < nlocal; ++i) e->r[comm.rank_of(i)] = args[i];
        cudaStream_t s = streams && streams[0] ? streams[0] : comm.default_stream(0);
        void* params[] = {e};
        cudaError_t ce = cudaLaunchCooperativeKernel(fn, dim3(ctas, W), dim3(kGemmDecodeThreads), params, smem, s);
        delete e;
        if (ce != cudaSuccess) {
            (void)cudaGetLastError();
            return fail(Result::CudaError, std::string("cooperative launch failed: ") + cudaGetErrorString(ce));
        }
        comm.CountLaunch(1);
        return Result::Success;
    }
    for (int i = 0; i < nlocal; ++i) {
        if (nlocal > 1) cudaSetDevice(comm.device_of(i));
        cudaStream_t s = streams && streams[i] ? streams[i] : comm.default_stream(i);
        void* params[] = {&args[i]};
        cudaError_t ce = LaunchInStream(fn, dim3(ctas), dim3(kGemmDecodeThreads), params, smem, s);
        if (ce != cudaSuccess) {
            (void)cudaGetLastError();
            return fail(Result::CudaError, std::string("kernel launch failed: ") + cudaGetErrorString(ce));
        }
        comm.CountLaunch(1);
    }
    return Result::Success;
}

bool EncodeTileMap(const DriverApi* d, CUtensorMap* map, const void* base, uint64_t rows, uint64_t cols_k,
                   uint32_t box_rows, std::string* err) {
    const cuuint64_t dims[2] = {cols_k, rows};             // innermost first
    const cuuint64_t strides[1] = {cols_k * 2};            // bytes between rows
    const cuuint32_t box[2] = {64, box_rows};              // 64 bf16 = 128 bytes = one swizzle row
    const cuuint32_t estr[2] = {1, 1};
    CUresult r = d->TensorMapEncodeTiled(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims,
                                         strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                                         CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                                         CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) {
        if (err) *err = "cuTensorMapEncodeTiled: " + d->ErrorText(r);
        return false;
    }
    return true;
}

}  // namespace

// Up to how many rows every rank receives all partial rows and normalises all of them itself (one NVLink
// phase instead of two, (W - 1) times the bytes).  Measured with one CTA per 128 x 256 tile, us one-shot / two-shot:
// 2 ranks T = 128: 25.3 / 30.8, T = 512: 35.0 / 36.5; 4 ranks T = 128: 25.0 / 27.5, T = 512: 42.3 / 33.6.
uint32_t FusedLinearOneShotMaxRows(int world) { return world <= 2 ? 256u : world <= 4 ? 128u : 32u; }

// K splits per 256-column tile of the few-token form.  An MMA of K = 16 costs about 90 ns whatever its
// width, so the k-blocks a CTA walks set the length of the GEMM phase (0.36 us each); every split is one more
// source for the reduction, which takes its sources eight at a time (about 1.8 us per eight, measured).  So:
// world x ksplit = 8 sources where K allows (2 x B200, K = 2048, T = 1: 12.7 us with 4 splits, 13.2 with 8,
// 15.5 with 2, 20.6 with 1), as long as the landing zone holds T rows per split, the work items fit the
// resident CTAs and no split is empty.  `want` > 0 replaces the first rule (measurements).
// Width of a tile of the few-token form: an MMA costs the same for 128 and for 256 columns, so the narrower
// tile is free for the GEMM and halves what an epilogue warp has to convert and push (32 columns instead of
// 64, to every rank); the wide one is for GPUs that hold fewer CTAs than there are narrow work items
// (several emulated ranks on one GPU).
uint32_t FusedLinearDecodeTile(uint32_t N, uint32_t ksplit, uint32_t resident_ctas) {
    return ((N + 127) / 128) * ksplit <= resident_ctas ? 128u : 256u;
}

uint32_t FusedLinearDecodeSplit(uint32_t T, uint32_t N, uint32_t K, int world, uint32_t resident_ctas, uint64_t ll_cap,
                                uint32_t want) {
    const uint32_t ntn = (N + kGemmDecodeMmaN - 1) / kGemmDecodeMmaN, kblocks = K / 64;
    if (want == 0) want = std::max<uint32_t>(1, std::min<uint32_t>(kblocks / 4, 8u / static_cast<uint32_t>(std::max(world, 1))));
    uint32_t ksplit = 1;
    while (ksplit * 2 <= std::min<uint32_t>(want, kGemmDecodeMaxSplit)) ksplit *= 2;
    auto fits = [&](uint32_t ks) {
        const uint32_t kper = (kblocks + ks - 1) / ks;
        return static_cast<uint64_t>(T) * N * 4 * ks <= ll_cap && ntn * ks <= resident_ctas &&
               static_cast<uint64_t>(ks - 1) * kper < kblocks;
    };
    while (ksplit > 1 && !fits(ksplit)) ksplit /= 2;
    return ksplit;
}

uint32_t FusedLinearDecodeMaxRows(const HeapLayout& lay, uint32_t N, int world) {
    if (world < 2 || N == 0 || N % kGemmDecodeTileN != 0 ||
        N > static_cast<uint32_t>(kGemmDecodeThreads) * kGemmDecodeVecPerThread * 8 || lay.gemm_ll_cap == 0)
        return 0;
    // Payload bytes double as flag-in-data lines.
    const uint64_t rows = lay.gemm_ll_cap / (static_cast<uint64_t>(N) * 4);
    return static_cast<uint32_t>(std::min<uint64_t>(rows, kGemmDecodeMaxRows));
}

// Rows that every owner delivers to every rank in one call: the targets of the delivered-row counters.
void FusedLinearRows(uint32_t T, int W, bool oneshot, uint32_t* rows_of) {
    const uint32_t Rs = (T + W - 1) / W;
    for (int q = 0; q < W; ++q) rows_of[q] = oneshot ? 0u : std::min<uint32_t>(Rs, T - std::min<uint32_t>(T, q * Rs));
}

// The same, and how many 128 x 256 tiles of the partial sums hold rows of every owner (one-shot: all of them).  For the
// C API: no kernel counts such tiles any more, a unit of sums is announced by the call's number.
void FusedLinearCounts(uint32_t T, uint32_t N, int W, bool oneshot, uint32_t* arrivals, uint32_t* rows_of) {
    const uint32_t ntm = (T + kGemmTileM - 1) / kGemmTileM, ntn = (N + kGemmTileN - 1) / kGemmTileN, Rs = (T + W - 1) / W;
    FusedLinearRows(T, W, oneshot, rows_of);
    for (int q = 0; q < W; ++q) {
        const uint32_t lo = q * Rs, hi = lo + rows_of[q];
        arrivals[q] = oneshot ? ntm * ntn : rows_of[q] ? ((hi - 1) / kGemmTileM - lo / kGemmTileM + 1) * ntn : 0u;
    }
}

// K splits per tile of a one-shot call of the tile form: powers of two while world x ksplit <= 8 (the flags and the row
// producer count sources by rank and split), every split keeps at least four k-blocks, as many 128 x 256 tiles fit the
// resident pairs (each of which now works on 256 x 256, so this errs on the side of fewer splits), a split's
// partial rows fit its share of the landing zone, and the partial rows a rank sends to its peers (every split sends
// its own) stay within 2 MiB (4 MiB for two splits).  The limits come from the form with one CTA per 128 x 256 tile, on 2 x
// B200 with K = 2048, us with 1 / 2 / 4 splits: T = 128: 25.0 / 21.1 / 23.4; T = 256: - / 27.2 / 32.3 (two-shot: 30.8);
// pairs of CTAs have not been measured on several GPUs.  `want` > 0 replaces the k-block and traffic rules
// (measurements).
uint32_t FusedLinearTileSplit(uint32_t T, uint32_t N, uint32_t K, int world, uint32_t resident_ctas, uint64_t gemm_cap,
                              uint32_t want) {
    const uint32_t ntiles = ((T + kGemmTileM - 1) / kGemmTileM) * ((N + kGemmTileN - 1) / kGemmTileN), kblocks = K / 64;
    uint32_t ks = 1;
    auto fits = [&](uint32_t s) {
        const uint32_t kper = (kblocks + s - 1) / s;
        const uint64_t sent = static_cast<uint64_t>(T) * N * 2 * s * static_cast<uint64_t>(std::max(world - 1, 1));
        const bool by_rule = kblocks / s >= 4 && sent <= (s == 2 ? (4ull << 20) : (2ull << 20));
        return static_cast<uint32_t>(world) * s <= static_cast<uint32_t>(kMaxRanks) && (want > 0 ? s <= want : by_rule) &&
               ntiles * s <= resident_ctas && static_cast<uint64_t>(T) * N * 2 * s <= gemm_cap &&
               static_cast<uint64_t>(s - 1) * kper < kblocks;
    };
    while (ks < 4 && fits(ks * 2)) ks *= 2;
    return ks;
}

// How the rows are cut into token tiles.  Candidates: one run of tiles per row owner (two-shot; rows then complete
// owner by owner and pushes spread over the owners) or one run over all rows, each with the fewest tiles that
// hold 256 tokens and a few more.  The time of a k-block grows with the tile's tokens above a part that does not
// (measured 519 cycles with 256 tokens, about 340 with 160 or fewer, where issue and operand fill set the
// pace), taken as max(340, 2 tokens + 6); the cost of a candidate is that times the rounds its items take on
// the resident pairs.  All inputs are alike on all ranks.
GemmTiling FusedLinearTiling(uint32_t T, uint32_t N, int world, bool oneshot, uint32_t ksplit, uint32_t pairs) {
    const uint32_t ncol = (N + kGemmPairCols - 1) / kGemmPairCols, Rs = oneshot ? T : (T + world - 1) / world;
    GemmTiling best{};
    uint64_t best_cost = ~0ull;
    auto consider = [&](uint32_t span, uint32_t domains) {
        const uint32_t fewest = (span + kGemmMaxTokens - 1) / kGemmMaxTokens;
        for (uint32_t n = fewest; n < fewest + 4; ++n) {
            GemmTiling t;
            t.span = span;
            t.domains = domains;
            t.tokens = ((span + n - 1) / n + 31) / 32 * 32;
            t.tiles = (span + t.tokens - 1) / t.tokens;
            const uint64_t items = static_cast<uint64_t>(domains) * t.tiles * ncol * ksplit;
            uint64_t cost = (items + pairs - 1) / pairs * std::max<uint32_t>(340, 2 * t.tokens + 6) * 100;
            // Without several tiles per owner no row completes before the end, and the row phase follows the GEMM instead
            // of running under it (2 ranks, T = 2048, K = 2048 on 37 pairs each: 73 us with, 91 us without).
            if (!oneshot && world > 1 && (domains == 1 || t.tiles == 1)) cost = cost * 5 / 4;
            if (cost >= best_cost) continue;
            best_cost = cost;
            // Column by column over all tiles (a slice of W is then read from HBM once, by neighbours) unless rows can
            // complete early: then the owners' k-th tiles together.
            t.group = domains > 1 && t.tiles > 1 ? domains : domains * t.tiles;
            best = t;
        }
    };
    if (!oneshot && world > 1) consider(Rs, static_cast<uint32_t>(world));
    consider(T, 1);
    return best;
}

// Which multicast form the two-shot takes by default (0 none, 1 in-switch reduce + multicast store,
// 2 peer pushes + multicast store), from measurements on 2, 4 and 8 B200.
// 8 x B200, K = 512 per rank, N = 4096, CUDA-graph timing (us, modes 0 / 1 / 2): T = 128: 31.4 / 28.9 /
// 29.5; T = 512: 37.4 / 36.0 / 35.6; T = 2048: 80.1 / 78.7 / 78.1.  2 x B200 (K = 2048): mode 1 loses
// (109 against 90 us at T = 2048, the switch adds a hop and saves no bytes), mode 2 ties with mode 0.
// 4 x B200 (K = 1024, 128 x 256 tiles): T = 512: 33.6 / 35.4 / 33.9; T = 2048: 65.9 / 73.0 / 68.6: the peer
// pushes win or tie, so the switch is used from 8 ranks on.  8 x B200 with 128 x 256 tiles: T = 128: 28.2 /
// 28.4 / 27.2; T = 512: 36.5 / 35.5 / 35.9; T = 2048: 73.6 / 77.1 / 72.7: pushes + multicast delivery throughout.
int FusedLinearAutoMulticastMode(int world, uint32_t /*T*/) {
    return world < 8 ? 0 : 2;
}

// Tries the cuts and takes the one with the lowest estimate, in cycles of an SM:
//   * a k-block of an item takes 2 cycles per token on the tensor cores, at least 350 for its instructions, and an item
//     1500 more; every pair has the same number of items, up to one;
//   * no run is shorter than reading all of W and x from HBM (3440 bytes per cycle, 15 % lost), by the pairs that are busy;
//   * with more than one token tile, a twelfth of reading W from HBM on top: tiles that run together ask for the same W at
//     slightly different times, and part of it comes twice.  The same for two tiles and for eight: it decides between one tile and
//     several (T <= 256) and never makes more tiles the cheaper cut;
//   * the sums are written and read again (1600 bytes per cycle): why splitting K costs more than cutting the tokens finer;
//   * the last item's read-out (10 per token), 60 per pair that has nothing to do (its SMs load nothing), and 2200 for
//     the fence and the flag of plain sums (`lines`: the splits travel as flag-in-data lines).
// Fitted to sweeps on B200 (in a graph, short bursts; back to back the long ones take 10-20 % more), us: 2 ranks, K = 2048,
// N = 4096: T = 256: 2 tiles of 128 x 2 splits 20.5, 1 of 256 x 4 23.2, 2 of 128 unsplit 24.8; T = 512: 4 of 128 27.5, 2 of
// 256 x 2 30.0; T = 2048: 8 of 256 65, 11 of 192 72; T = 8: 4 splits 10.6, 3 11.6.  8 ranks, K = 1792, T = 300: 2 of 160 x 2
// 54, unsplit 71.  One tile or several, W beyond / in L2: 8 ranks: N = 4096, K = 1792: T = 64: 2 tiles of 32 x 2 34.6 / 33.6, 1 of
// 64 x 4 32.5 / 32.5, T = 33: 32 x 2 32.9 / 32.9, 64 x 4 31.5 / 31.6; N = 2816, K = 1728, T = 57: 32 x 3 26.1 / 26.8, 64 x 6 24.2 / 18.1;
// 4 ranks, N = 3840, K = 1600, T = 65: 64 x 2 18.6 / 17.6, 96 x 4 17.4 / 14.1; 2 ranks, N = 3584, K = 1408, T = 66: 64 x 2 12.4 / 11.5,
// 96 x 5 10.6 / 10.5.  Of 310 sizes timed with the cuts of both the term changes 51, to 0.90 of the time in the mean; three of
// them, with little of W per pair, lose 4 - 10 % (8 ranks, K = 256, N = 2432, T = 40: 32 x 3 12.2 / 10.5, 64 x 7 12.5 / 12.6).
// A tenth to a sixteenth rank much alike; with an eighth eight of 83 lose.
// The whole ranks shapes and is no prediction: rows that become ready with the last items, and so cannot run under the
// GEMM, have no term, and where all items fit one round it comes out far too low (T = 300: 28-33 of 49 us).  Timed again when the row kernel
// changed: 0.6 % above the best of up to nine cuts in the mean of 14 sizes, 4 % at worst.
LocalGemmShape LocalGemmShapeFor(uint32_t T, uint32_t N, uint32_t kb_total, uint64_t room, uint32_t pairs, bool lines) {
    const uint32_t ncol = (N + kLocalGemmPairCols - 1) / kLocalGemmPairCols, units = N / kLocalGemmUnitCols;
    const uint32_t fewest = (T + kLocalGemmMaxTokens - 1) / kLocalGemmMaxTokens;
    const uint64_t hbm = static_cast<uint64_t>(kb_total) * (N + T) * 128 / 3440 * 115 / 100 + 1500;
    const uint64_t again = static_cast<uint64_t>(kb_total) * N * 128 / 3440 / 12;
    LocalGemmShape best{};
    uint64_t best_cost = ~0ull;
    for (uint32_t n = fewest; n < fewest + 4; ++n) {
        LocalGemmShape s;
        s.tokens = ((T + n - 1) / n + 31) / 32 * 32;
        s.tiles = (T + s.tokens - 1) / s.tokens;
        const uint64_t block = std::max<uint64_t>(350, 2ull * s.tokens + 8);
        for (uint32_t split = 1; split <= std::min(kLocalGemmMaxSplit, kb_total); ++split) {
            s.kper = (kb_total + split - 1) / split;
            s.nsplit = (kb_total + s.kper - 1) / s.kper;
            const uint64_t sums = static_cast<uint64_t>(T) * N * 2 * s.nsplit;
            if (s.nsplit != split) continue;
            if (split > 1 && sums > room) break;
            if (static_cast<uint64_t>(s.tiles) * units * s.nsplit > kLocalGemmFlags) break;
            const uint64_t items = static_cast<uint64_t>(s.tiles) * ncol * s.nsplit;
            const uint64_t rounds = (items + pairs - 1) / pairs, used = std::min<uint64_t>(items, pairs);
            uint64_t cost = std::max(rounds * (s.kper * block + 1500), hbm * (rounds * used) / items) + 2 * sums / 1600 +
                            10 * s.tokens + 60 * (pairs - used);
            if (!(lines && split > 1)) cost += 2200;
            if (s.tiles > 1) cost += again;
            if (cost < best_cost) {
                best_cost = cost;
                best = s;
            }
        }
    }
    return best;
}

namespace {

// Ranks that share this GPU: a GEMM over all ranks' K extents and a row kernel that starts under it (gemm_local.cu).
// The second kernel runs while the first still reads x and W, so no output may lie on an input, except that a
// rank's residual may be updated in place.
bool CanRunLocal(Communicator& comm, const FusedLinearDesc* descs, uint32_t T, uint32_t N, uint32_t K,
                 const FusedLinearOptions& opt) {
    static const bool measuring = env::GetInt("YALI_GEMM_DECODE", -1) >= 0 || env::GetInt("YALI_GEMM_KSPLIT", 0) > 0 ||
                                  env::GetInt("YALI_GEMM_DECODE_KSPLIT", 0) > 0 || env::GetInt("YALI_GEMM_DECODE_TILE", 0) > 0;
    if (!comm.emulated() || comm.world() < 2 || opt.force_oneshot >= 0 || opt.decode >= 0 || opt.nvls > 0 || opt.ctas > 0 ||
        opt.trace || measuring)
        return false;
    const uint64_t rows = static_cast<uint64_t>(T) * N * 2, xb = static_cast<uint64_t>(T) * K * 2, wb = static_cast<uint64_t>(N) * K * 2;
    // What the multi-GPU forms take (one landing zone per source): no more, so that the two agree on what is too large.
    const uint64_t share = static_cast<uint64_t>((T + comm.world() - 1) / comm.world()) * N * 2;
    if (share > comm.layout().gemm_cap || rows > 2ull * comm.world() * comm.layout().gemm_cap) return false;
    auto overlap = [](const void* a, uint64_t an, const void* b, uint64_t bn) {
        const char *p = static_cast<const char*>(a), *q = static_cast<const char*>(b);
        return p && q && p < q + bn && q < p + an;
    };
    for (int j = 0; j < comm.nlocal(); ++j) {
        const void* const outs[2] = {descs[j].out, descs[j].residual_out};
        for (int i = 0; i < comm.nlocal(); ++i) {
            for (const void* o : outs)
                if (overlap(o, rows, descs[i].x, xb) || overlap(o, rows, descs[i].w, wb) ||
                    overlap(o, rows, descs[i].norm_weight, static_cast<uint64_t>(N) * 2) ||
                    (overlap(o, rows, descs[i].residual, rows) && !(i == j && o == descs[i].residual)))
                    return false;
            // Two outputs on one another: which of them is left depends on the order of the writes.
            if (overlap(descs[j].out, rows, descs[i].residual_out, rows) ||
                (i != j && (overlap(descs[j].out, rows, descs[i].out, rows) || overlap(descs[j].residual_out, rows, descs[i].residual_out, rows))))
                return false;
        }
    }
    return true;
}

Result LaunchLocal(Communicator& comm, const DriverApi* drv, const FusedLinearDesc* descs, uint32_t T, uint32_t N,
                   uint32_t K, const FusedLinearOptions& opt, const cudaStream_t* streams) {
    auto fail = [&](Result r, const std::string& what) {
        comm.set_error(what);
        return r;
    };
    const int W = comm.world();
    const void* fn = LocalGemmKernel();
    const uint32_t smem = LocalGemmSmemBytes();
    static std::mutex mu;
    static std::map<int, uint32_t> pairs_of;  // resident pairs of CTAs per device; the shared-memory limit is raised with it
    uint32_t pairs = 0;
    {
        std::lock_guard<std::mutex> lock(mu);
        uint32_t& p = pairs_of[comm.device_of(0)];
        if (p == 0) {
            cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
            cudaLaunchConfig_t cfg;
            std::memset(&cfg, 0, sizeof(cfg));
            cfg.gridDim = dim3(2);
            cfg.blockDim = dim3(kLocalGemmThreads);
            cfg.dynamicSmemBytes = smem;
            int n = 0;
            if (e == cudaSuccess) e = cudaOccupancyMaxActiveClusters(&n, fn, &cfg);
            if (e != cudaSuccess || n < 1) return fail(Result::CudaError, std::string("fused linear: ") + cudaGetErrorString(e));
            p = static_cast<uint32_t>(n);
        }
        pairs = p;
    }
    const uint32_t sms = 2 * pairs;
    const HeapLayout& lay = comm.layout();
    LocalGemmArgs g;
    std::memset(&g, 0, sizeof(g));
    g.cv = comm.View(0);
    g.sums = g.cv.heap[0] + lay.gemm_off;
    g.T = T;
    g.N = N;
    g.kb_rank = K / 64;
    g.kb_total = g.kb_rank * W;
    const bool few = static_cast<uint64_t>(T) * W <= 2 * sms;
    g.s = LocalGemmShapeFor(T, N, g.kb_total, 2ull * W * lay.gemm_cap, pairs, few && T <= 64);
    LocalLinearNormArgs n;
    std::memset(&n, 0, sizeof(n));
    n.early = static_cast<uint64_t>(T) * N * W <= kLocalLinearEarly;
    n.cv = g.cv;
    n.sums = g.sums;
    n.T = T;
    n.N = N;
    n.world = static_cast<uint32_t>(W);
    n.s = g.s;
    n.eps = opt.eps;
    std::string derr;
    for (int i = 0; i < W; ++i) {
        const int r = comm.rank_of(i);
        const FusedLinearDesc& d = descs[i];
        if (!EncodeTileMap(drv, &g.tmap_x[r], d.x, T, K, g.s.tokens / 2, &derr) ||
            !EncodeTileMap(drv, &g.tmap_w[r], d.w, N, K, kLocalGemmUnitCols, &derr))
            return fail(Result::CudaError, derr);
        n.residual[r] = d.residual;
        n.residual_out[r] = d.residual_out;
        n.weight[r] = d.norm_weight;
        n.out[r] = d.out;
    }
    const uint32_t items = g.s.tiles * ((N + kLocalGemmPairCols - 1) / kLocalGemmPairCols) * g.s.nsplit;
    // With few rows the sums travel as flag-in-data lines, which saves the fence and the flag at the price of twice the bytes.
    // (In a graph, short bursts, us.  2 ranks, K = 2048: T = 16 13.1 -> 12.1, T = 64 16.1 -> 15.1; 8 ranks, K = 1792, two splits:
    // T = 36 34.6 -> 33.4; but 2 ranks T = 96 16.0 -> 16.9, T = 128 16.5 -> 18.4.)
    const uint64_t line_bytes = static_cast<uint64_t>(T) * N * 4 * g.s.nsplit;
    const bool lines = few && T <= 64 && g.s.nsplit > 1 && line_bytes <= 2ull * W * lay.gemm_ll_cap;
    if (lines) {
        g.lines = 1;
        n.sums = g.sums = g.cv.heap[0] + lay.gemm_ll_off;
    }
    const uint32_t threads = LocalLinearNormThreads(N);
    const bool split = g.s.nsplit > 1;
    const bool narrow = LocalLinearNormVectors(N) == 1;
    auto units_of = [&](int gr) { return static_cast<uint32_t>(T * ((W + gr - 1) / gr)); };
    // Lines of one rank: the instance that is not slim asks for the lines of four splits at a time instead of one or two, in registers that leave
    // no room for a second CTA beside the GEMM's.  Wide rows: with six to eight splits that pays while every SM has one unit and a few have a second one
    // (slim / not, us: 8 ranks, 17 x 256 x 2176, 136 units 9.4 / 7.8; 6 ranks, 26 x 1792 x 2432, 156 units 15.5 / 14.2, 28 x 768 x 2816, 168 units 10.8 /
    // 12.4; 8 ranks, 35 x 1536 x 3072, 280 units 20.0 / 23.7), with fewer while there are few threads per SM (2 ranks, 40 x 512 x 2176, 86 threads 7.1 /
    // 6.7; 4 ranks, 12 x 1024 x 3328, 73 10.1 / 9.3; 4 ranks, 17 x 1536 x 3584, 103 12.2 / 12.9; 2 ranks, 64 x 1024 x 3328, 194 9.7 / 10.4; 5 ranks, 30 x 1280 x
    // 3200, 227 12.1 / 15.7).  Of 129 sizes the worst loses 7 %, the mean 0.3 %.  Narrow rows: 8 ranks, 24 x 512 x 1024 7.2 / 6.9, 30 x 1024 x 2048 11.7 /
    // 13.6.
    bool slim = narrow ? units_of(1) * threads > 256 * sms : g.s.nsplit > 5 ? units_of(1) > sms + sms / 18 : units_of(1) * threads > 100 * sms;
    cudaError_t asked = cudaSuccess;
    auto places_of = [&](int gr, bool slim) {
        uint32_t n = 1;
        const cudaError_t e = FusedLinearRowPlaces(comm.device_of(0), N, gr, split, lines, slim, &n);
        if (e != cudaSuccess) asked = e;
        return sms * n;
    };
    // Ranks that a CTA serves, each CTA adding the splits again: one while that needs no more than two CTAs of 256 threads per SM and four
    // of any size (one / two / four ranks, us: 8 ranks, 40 x 256 x 512 7.1 / 8.4 / 8.4, 60 x 512 x 1024 9.7 / 10.2 / 10.3; 4 ranks, 76 x 1024 x
    // 2048 10.9 / 10.5 / 12.3; 2 ranks, 1000 x 256 x 128 13.2 / 9.7).  Above, two for wide rows (four, which spill: 8 ranks, 2048 x 512 x 4096
    // 120 / 105, 1500 x 512 x 2304 61.7 / 53.1; one, 300 x 1792 x 4096 51.6 / 50.4).  For narrow rows two while they leave half of the places
    // free, else four, which read the sums less often (two / four: 8 ranks, 40 x 1024 x 2048 14.5 / 15.3, 133 x 448 x 1152 12.3 / 11.6, 1000 x 256
    // x 1024 23.2 / 21.1; 4 ranks, 200 x 1024 x 2048 14.3 / 13.8), unless the last group would hold one or two ranks (6 ranks, 300 x 1024 x
    // 2048 21.2 / 21.8).
    int group = 1;
    if (!few && !(narrow && units_of(1) <= 4 * sms && units_of(1) * threads <= 512 * sms))
        group = !narrow || (W & 3) == 1 || (W & 3) == 2 || 2 * units_of(2) <= places_of(2, true) ? 2 : 4;
    // Four CTAs per SM with the weights one by one while they take all units at once, else three that ask for them together (four / three:
    // 2 ranks, N = 4096, K = 2048: T = 512 24.6 / 25.9, T = 700 30.1 / 29.4; 1000 x 512 x 3072 25.8 / 24.8; 4 ranks, 1000 x 512 x 4096 41.1 / 38.0).
    if (group == 2) slim = units_of(2) <= places_of(2, true);
    const uint32_t ngroups = (W + group - 1) / group, units = units_of(group), places = places_of(group, slim);
    if (asked != cudaSuccess) return fail(Result::CudaError, std::string("fused linear: ") + cudaGetErrorString(asked));
    n.by_groups = static_cast<uint32_t>(((1ull << 32) + ngroups - 1) / ngroups);
    const void* const fn2 = LocalLinearNormKernel(N, group, split, lines, slim);
    const cudaStream_t s = streams && streams[0] ? streams[0] : comm.default_stream(0);
    void* gp[] = {&g};
    void* np[] = {&n};
    cudaError_t e = LaunchInStream(fn, dim3(2 * std::min(items, pairs)), dim3(kLocalGemmThreads), gp, smem, s);
    if (e == cudaSuccess)
        e = LaunchInStream(fn2, dim3(std::min(units, places)), dim3(threads), np, 0, s);
    if (e != cudaSuccess) {
        (void)cudaGetLastError();
        return fail(Result::CudaError, std::string("kernel launch failed: ") + cudaGetErrorString(e));
    }
    comm.CountLaunch(2);
    return Result::Success;
}

}  // namespace

cudaError_t FusedLinearRowPlaces(int device, uint32_t N, int ranks_per_cta, bool split, bool lines, bool slim, uint32_t* places) {
    constexpr int kDevices = 32;  // beyond: asked for on every call
    static std::atomic<int> known[kDevices][5][3][2][kLocalLinearNormThreads / 32 + 1];
    const int threads = LocalLinearNormThreads(N);
    std::atomic<int>* const k = device < 0 || device >= kDevices ? nullptr
                                : &known[device][slim && ranks_per_cta < 4 ? 3 + ranks_per_cta / 2 : ranks_per_cta / 2]
                                        [lines ? 2 : split ? 1 : 0][LocalLinearNormVectors(N) - 1][threads / 32];
    int n = k ? k->load(std::memory_order_relaxed) : 0;
    if (n == 0) {
        const cudaError_t e =
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, LocalLinearNormKernel(N, ranks_per_cta, split, lines, slim), threads, 0);
        if (e != cudaSuccess || n < 1) {
            (void)cudaGetLastError();
            return e != cudaSuccess ? e : cudaErrorLaunchOutOfResources;
        }
        if (k) k->store(n, std::memory_order_relaxed);
    }
    *places = static_cast<uint32_t>(n);
    return cudaSuccess;
}

Result FusedLinearAllReduceRmsNorm(Communicator& comm, const FusedLinearDesc* descs, uint32_t T, uint32_t N,
                                   uint32_t K, const FusedLinearOptions& opt, const cudaStream_t* streams) {
    YALI_NVTX_RANGE("yali::FusedLinear");
    auto fail = [&](Result r, const std::string& what) {
        comm.set_error(what);
        return r;
    };
    if (comm.poisoned()) return fail(Result::Timeout, "communicator is poisoned by an earlier timeout; call Reset()");
    if (T == 0) return Result::Success;
    if (N % 128 != 0 || N > 4096 || K % 64 != 0 || K == 0)
        return fail(Result::Unsupported, "fused linear needs N a multiple of 128 (at most 4096) and K a multiple of 64");
    const int W = comm.world(), nlocal = comm.nlocal();
    for (int i = 0; i < nlocal; ++i) {
        const FusedLinearDesc& d = descs[i];
        if (!d.x || !d.w || !d.norm_weight || !d.out) return fail(Result::InvalidArg, "null tensor");
        if ((reinterpret_cast<uintptr_t>(d.x) | reinterpret_cast<uintptr_t>(d.w) | reinterpret_cast<uintptr_t>(d.out) |
             reinterpret_cast<uintptr_t>(d.norm_weight) | reinterpret_cast<uintptr_t>(d.residual) |
             reinterpret_cast<uintptr_t>(d.residual_out)) & 15u)
            return fail(Result::InvalidArg, "tensors must be 16-byte aligned");
    }
    std::string derr;
    const DriverApi* drv = DriverApi::Get(&derr);
    if (!drv) return fail(Result::CudaError, derr);

    if (CanRunLocal(comm, descs, T, N, K, opt)) return LaunchLocal(comm, drv, descs, T, N, K, opt, streams);

    const HeapLayout& lay = comm.layout();
    const uint64_t row_bytes = static_cast<uint64_t>(N) * 2;
    {
        // Few tokens: the latency form (every rank normalises all rows; nothing else to decide).
        const uint32_t decode_max = FusedLinearDecodeMaxRows(lay, N, W);
        static const long long decode_env = env::GetInt("YALI_GEMM_DECODE", -1);
        const int want = opt.decode >= 0 ? opt.decode : static_cast<int>(decode_env);
        if (want == 1 && T > decode_max)
            return fail(Result::Unsupported, "the few-token form of the fused linear takes at most " +
                                                 std::to_string(decode_max) + " rows of this width");
        if (want != 0 && T <= decode_max && (want == 1 || (opt.force_oneshot != 0 && opt.nvls <= 0)))
            return LaunchDecode(comm, drv, descs, T, N, K, opt, streams);
    }
    bool oneshot = opt.force_oneshot >= 0 ? opt.force_oneshot != 0 : T <= FusedLinearOneShotMaxRows(W);
    if (W == 1) oneshot = true;
    // Two-shot writes into every rank's output: those must be addressable from here.
    bool outs_addressable = nlocal == W;
    uint64_t out_off = 0;
    if (!outs_addressable) {
        outs_addressable = comm.IsSymmetric(0, descs[0].out, static_cast<uint64_t>(T) * row_bytes);
        if (outs_addressable) out_off = static_cast<const char*>(descs[0].out) - comm.View(0).heap[comm.rank_of(0)];
    }
    uint64_t res_out_off = 0;
    if (nlocal != W && descs[0].residual_out) {
        // One GPU per process, two-shot: the owner of a row also writes every rank's residual_out.
        if (comm.IsSymmetric(0, descs[0].residual_out, static_cast<uint64_t>(T) * row_bytes))
            res_out_off = static_cast<const char*>(descs[0].residual_out) - comm.View(0).heap[comm.rank_of(0)];
        else
            outs_addressable = false;
    }
    if (!oneshot && !outs_addressable) {
        if (opt.force_oneshot == 0)
            return fail(Result::Unsupported, "two-shot fused linear needs out (and residual_out) in symmetric memory");
        oneshot = true;
    }
    uint32_t Rs = oneshot ? T : (T + W - 1) / W;
    if (static_cast<uint64_t>(Rs) * row_bytes > lay.gemm_cap) {
        if (oneshot && outs_addressable && static_cast<uint64_t>((T + W - 1) / W) * row_bytes <= lay.gemm_cap &&
            opt.force_oneshot != 1) {
            oneshot = false;
            Rs = (T + W - 1) / W;
        } else {
            return fail(Result::Unsupported, "rows do not fit the landing zone of the fused linear (" +
                                                 std::to_string(lay.gemm_cap) + " bytes per source)");
        }
    }

    // Forms of the two-shot that go through the NVSwitch multicast object: they need the multicast
    // mapping and out / residual_out at one common heap offset on every rank (tensors from SymmAlloc
    // are); the in-switch reduce also needs the [T, N] image to fit the landing region of one call
    // parity.  Mode 1: in-switch reduce + multicast store; mode 2: peer pushes + multicast store.
    int mc_mode = 0;
    uint64_t mc_out_off = 0, mc_res_out_off = 0;
    {
        const long long nvls_env = env::GetInt("YALI_GEMM_NVLS", -1);
        const int want = opt.nvls >= 0 ? opt.nvls : (nvls_env >= 0 ? static_cast<int>(nvls_env) : -1);
        bool possible = !oneshot && !comm.emulated() && W > 1 && want != 0 && comm.View(0).mc_heap != nullptr;
        for (int i = 0; i < nlocal && possible; ++i) {
            const char* base = comm.View(i).heap[comm.rank_of(i)];
            if (!comm.IsSymmetric(i, descs[i].out, static_cast<uint64_t>(T) * row_bytes)) possible = false;
            const uint64_t off = static_cast<const char*>(descs[i].out) - base;
            if (i == 0) mc_out_off = off;
            else if (off != mc_out_off) possible = false;
            if (descs[i].residual_out) {
                if (!comm.IsSymmetric(i, descs[i].residual_out, static_cast<uint64_t>(T) * row_bytes)) possible = false;
                const uint64_t roff = static_cast<const char*>(descs[i].residual_out) - base;
                if (i == 0) mc_res_out_off = roff;
                else if (roff != mc_res_out_off) possible = false;
            }
        }
        const bool image_fits = static_cast<uint64_t>(T) * row_bytes <= lay.gemm_cap * W;
        if (want > 0) {
            if (!possible || (want == 1 && !image_fits))
                return fail(Result::Unsupported,
                            "the multicast forms of the fused linear need two-shot, the multicast mapping and symmetric out tensors");
            mc_mode = want == 1 ? 1 : 2;
        } else if (possible) {
            mc_mode = FusedLinearAutoMulticastMode(W, T);
            if (mc_mode == 1 && !image_fits) mc_mode = 2;
        }
    }
    const bool nvls = mc_mode == 1;

    // Rows every owner delivers in this call.
    uint32_t rows_of[kMaxRanks] = {};
    FusedLinearRows(T, W, oneshot, rows_of);
    const void* fn = GemmArKernel(comm.emulated());
    const uint32_t smem = GemmArSmemBytes();
    // The dynamic shared-memory limit is a per-device property of the kernel: raise it once for every
    // (kernel flavour, device) this process launches on, and ask once how many pairs of CTAs are resident (all
    // GPUs of a group are alike).
    static std::mutex attr_mu;
    static std::set<std::pair<int, int>> attr_done;
    static int cached_pairs[2] = {0, 0};
    const int flavour = comm.emulated() ? 1 : 0;
    uint32_t pairs = 0;
    {
        std::lock_guard<std::mutex> lock(attr_mu);
        for (int i = 0; i < nlocal; ++i) {
            const std::pair<int, int> key(flavour, comm.device_of(i));
            if (attr_done.count(key)) continue;
            if (nlocal > 1) cudaSetDevice(comm.device_of(i));
            cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
            if (e != cudaSuccess) return fail(Result::CudaError, std::string("cudaFuncSetAttribute: ") + cudaGetErrorString(e));
            attr_done.insert(key);
        }
        if (cached_pairs[flavour] == 0) {
            cudaLaunchConfig_t cfg;
            std::memset(&cfg, 0, sizeof(cfg));
            cfg.gridDim = dim3(2);
            cfg.blockDim = dim3(kGemmThreads);
            cfg.dynamicSmemBytes = smem;
            int n = 0;
            cudaError_t e = cudaOccupancyMaxActiveClusters(&n, fn, &cfg);
            if (e != cudaSuccess || n < 1)
                return fail(Result::CudaError, std::string("cudaOccupancyMaxActiveClusters: ") + cudaGetErrorString(e));
            cached_pairs[flavour] = n;
        }
        pairs = static_cast<uint32_t>(cached_pairs[flavour]);
    }
    if (comm.emulated()) {
        if (pairs < static_cast<uint32_t>(W)) return fail(Result::Unsupported, "the GPU holds fewer pairs of CTAs than ranks");
        pairs /= W;
    }
    // One-shot calls split the K extent of their tiles while that shortens the GEMM phase (see FusedLinearTileSplit).
    static const long long forced_split = env::GetInt("YALI_GEMM_KSPLIT", 0);  // measurements only
    uint32_t ksplit = oneshot && mc_mode == 0 && W > 1
                          ? FusedLinearTileSplit(T, N, K, W, pairs, lay.gemm_cap, forced_split > 0 ? static_cast<uint32_t>(forced_split) : 0u)
                          : 1u;
    const uint32_t kper = (K / 64 + ksplit - 1) / ksplit;
    const GemmTiling tiling = FusedLinearTiling(T, N, W, oneshot, ksplit, pairs);
    const uint32_t tiles = tiling.domains * tiling.tiles;
    if (static_cast<uint64_t>(tiles) * (N / kGemmUnitCols) * ksplit > kGemmTileFlags)
        return fail(Result::Unsupported, "too many tiles for the fused linear");
    const uint32_t items = tiles * ((N + kGemmPairCols - 1) / kGemmPairCols) * ksplit;
    const uint32_t work = std::max<uint32_t>(2 * items, oneshot ? T : Rs);
    uint32_t ctas = std::min<uint32_t>(2 * pairs, work);
    if (opt.ctas > 0) ctas = std::min<uint32_t>(ctas, opt.ctas);
    ctas = (ctas + 1) / 2 * 2;

    std::vector<GemmArArgs> args(nlocal);
    for (int i = 0; i < nlocal; ++i) {
        GemmArArgs& a = args[i];
        std::memset(&a, 0, sizeof(a));
        const FusedLinearDesc& d = descs[i];
        const int rank = comm.rank_of(i);
        if (nlocal > 1) cudaSetDevice(comm.device_of(i));
        if (!EncodeTileMap(drv, &a.tmap_x, d.x, T, K, tiling.tokens / 2, &derr) ||
            !EncodeTileMap(drv, &a.tmap_w, d.w, N, K, kGemmUnitCols, &derr))
            return fail(Result::CudaError, derr);
        a.cv = comm.View(i);
        a.residual = d.residual;
        a.residual_out = d.residual_out;
        a.norm_weight = d.norm_weight;
        for (int q = 0; q < W; ++q) a.out[q] = a.residual_out_all[q] = nullptr;
        a.out[rank] = d.out;
        a.residual_out_all[rank] = d.residual_out;
        if (!oneshot) {
            if (nlocal == W) {
                for (int j = 0; j < nlocal; ++j) {
                    a.out[comm.rank_of(j)] = descs[j].out;
                    a.residual_out_all[comm.rank_of(j)] = descs[j].residual_out;
                }
            } else {
                for (int q = 0; q < W; ++q) {
                    a.out[q] = a.cv.heap[q] + out_off;
                    if (d.residual_out) a.residual_out_all[q] = a.cv.heap[q] + res_out_off;
                }
            }
        }
        a.T = T;
        a.N = N;
        a.K = K;
        a.tl = tiling;
        a.rows_per_owner = Rs;
        a.one_gpu = comm.emulated() || W == 1 ? 1u : 0u;
        a.oneshot = oneshot ? 1u : 0u;
        a.ksplit = ksplit;
        a.kper = kper;
        for (int q = 0; q < W; ++q) a.done_inc[q] = rows_of[q];
        a.eps = opt.eps;
        a.nvls = nvls ? 1u : 0u;
        if (mc_mode != 0) {
            a.out_mc = a.cv.mc_heap + mc_out_off;
            a.residual_out_mc = d.residual_out ? a.cv.mc_heap + mc_res_out_off : nullptr;
        }
        a.trace = opt.trace ? opt.trace[i] : nullptr;
    }
    if (comm.emulated()) {
        GemmArEmuArgs* e = new GemmArEmuArgs();
        std::memset(e, 0, sizeof(*e));
        for (int i = 0; i < nlocal; ++i) e->r[comm.rank_of(i)] = args[i];
        cudaStream_t s = streams && streams[0] ? streams[0] : comm.default_stream(0);
        void* params[] = {e};
        cudaError_t ce = cudaLaunchCooperativeKernel(fn, dim3(ctas, W), dim3(kGemmThreads), params, smem, s);
        delete e;
        if (ce != cudaSuccess) {
            (void)cudaGetLastError();
            return fail(Result::CudaError, std::string("cooperative launch failed: ") + cudaGetErrorString(ce));
        }
        comm.CountLaunch(1);
        return Result::Success;
    }
    for (int i = 0; i < nlocal; ++i) {
        if (nlocal > 1) cudaSetDevice(comm.device_of(i));
        cudaStream_t s = streams && streams[i] ? streams[i] : comm.default_stream(i);
        void* params[] = {&args[i]};
        cudaError_t ce = LaunchInStream(fn, dim3(ctas), dim3(kGemmThreads), params, smem, s);
        if (ce != cudaSuccess) {
            (void)cudaGetLastError();
            return fail(Result::CudaError, std::string("kernel launch failed: ") + cudaGetErrorString(ce));
        }
        comm.CountLaunch(1);
    }
    return Result::Success;
}

}  // namespace yali
