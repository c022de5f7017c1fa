// Argument block and geometry of the kernels for groups whose ranks share one GPU and one launch
// (local_group.cu).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "../comm/layout.h"

namespace yali {

constexpr int kLocalThreads = 512;
constexpr int kLocalNormHeld = 8;  // packed residual vectors a thread of the norm kernel keeps (vectors x ranks)

enum class LocalKind : int { Sum = 0, ReduceScatter = 1, AllGather = 2 };

struct LocalArgs {
    const void* send[kMaxRanks];
    void* recv[kMaxRanks];
    const void* residual[kMaxRanks];  // norm kernel only; entries may be nullptr
    void* residual_out[kMaxRanks];    // norm kernel only; entries may be nullptr
    const void* weight[kMaxRanks];    // norm kernel only
    uint32_t* ctl[kMaxRanks];         // flag region of every rank (timeline of traced calls)
    uint64_t count;                   // elements of the message
    uint64_t shard_elems;             // reduce-scatter / all-gather: elements a rank owns
    EpilogueParams ep;                // scale, eps, hidden
    uint32_t world;
    uint32_t flags;                   // kFlagVecOk, kFlagTrace
};

constexpr int kLocalHostThreads = 256;
constexpr int kLocalHostCtas = 64;

// How the norm kernel cuts its work: threads of a CTA (one row), vectors per thread, and for how many ranks
// a CTA normalises the row.
struct LocalNormShape {
    int threads;
    int vec_per_thread;  // 1, 2 or 4
    int ranks_per_cta;
};
// One vector per thread while a row fits 512 threads.  With few rows the ranks are spread over CTAs (each adds the
// row's inputs again, which stay in L2); from `rows * world` >= 2 CTAs per SM on, one CTA serves as many
// ranks as its registers hold, so that every input is read once.
inline LocalNormShape LocalNormShapeFor(uint64_t rows, uint32_t vec_per_row, int world, uint32_t sm_count) {
    LocalNormShape s;
    const uint32_t want = vec_per_row < static_cast<uint32_t>(kLocalThreads) ? vec_per_row : static_cast<uint32_t>(kLocalThreads);
    s.threads = static_cast<int>((want + 31) / 32 * 32);
    const uint32_t nv = (vec_per_row + s.threads - 1) / s.threads;
    s.vec_per_thread = nv <= 1 ? 1 : nv <= 2 ? 2 : 4;
    const int most = kLocalNormHeld / s.vec_per_thread;
    s.ranks_per_cta = rows * static_cast<uint64_t>(world) < 2ull * sm_count ? 1 : (world < most ? world : most);
    // Worlds without an instance of their own run the generic kernel, which holds `most` ranks.
    if (s.ranks_per_cta > 1 && world != 2 && world != 4 && world != 8) s.ranks_per_cta = most;
    return s;
}

// nullptr when the combination is not built.
const void* LocalKernelFor(Dtype in, Dtype out, int world, LocalKind kind);
// Sum of buffers in host memory that the GPU can address; any number of CTAs.
const void* LocalHostKernelFor(Dtype dt, int world);
const void* LocalNormKernelFor(Dtype dt, int world, const LocalNormShape& shape);

}  // namespace yali
