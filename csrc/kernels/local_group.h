// Argument block and geometry of the kernels for groups whose ranks share one GPU and one launch
// (local_group.cu).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "../comm/layout.h"

namespace yali {

constexpr int kLocalThreads = 512;

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

// How the norm kernel cuts its work: threads of a CTA (one row), vectors per thread, for how many ranks a CTA normalises
// the row, and whether it asks for the weights behind the barrier, which takes fewer registers.
struct LocalNormShape {
    int threads;
    int vec_per_thread;  // 1, 2 or 4
    int ranks_per_cta;   // 1, 2 or 4
    bool late;
};
// One vector per thread while a row fits 512 threads.  Up to what runs together (32 warps per SM; twice that for the largest choice) the ranks
// are spread over CTAs as far as possible: each adds the row's inputs again, which stay in L2.  us for one / two / four ranks per CTA, bf16:
// 8 ranks: 16 x 4096 2.2 / 2.6 / 3.5, 64 x 4096 6.3 / 4.8 / 5.5, 256 x 4096 19.0 / 14.9 / 14.1; 4 ranks: 256 x 1024 3.1 / 3.2 / 4.1, 256 x
// 4096 8.5 / 8.2 / 7.6; 2 ranks: 64 x 8192 2.9 / 3.6, 256 x 4096 5.0 / 4.4.  Beyond, two ranks per CTA in as few registers as that takes,
// with the weights behind the barrier (late / early: 2 ranks 1024 x 4096 13.1 / 13.3, 4000 x 4096 41.4 / 43.2, but 512 x 4096 8.7 / 7.6; 8 ranks
// 1000 x 2944 35.0 / 41.1; four ranks 37.4), at 4 ranks ahead of it (1000 x 2944 19.1 / 17.7).  Rows of two vectors per thread: one rank,
// early, up to four rounds (8 ranks 100 x 8192 13.0, two late 13.6; 500 x 8192 56.8, 48.2), but fp32 on 2 ranks two, early, from one
// round on (500 x 4096 12.3 / 12.1, late 12.8).  Of four: the same, but on 2 ranks one rank late (fp32 1024 x 8192 42.5; two 45.3).
inline LocalNormShape LocalNormShapeFor(uint64_t rows, uint32_t vec_per_row, int elem_bytes, int world, uint32_t sm_count) {
    LocalNormShape s;
    const uint32_t want = vec_per_row < static_cast<uint32_t>(kLocalThreads) ? vec_per_row : static_cast<uint32_t>(kLocalThreads);
    s.threads = static_cast<int>((want + 31) / 32 * 32);
    const uint32_t nv = (vec_per_row + s.threads - 1) / s.threads;
    s.vec_per_thread = nv <= 1 ? 1 : nv <= 2 ? 2 : 4;
    s.ranks_per_cta = 1;
    s.late = false;
    if (world == 1) return s;
    auto warps = [&](int g) { return rows * ((world + g - 1) / g) * (s.threads / 32); };
    const uint64_t round = 32ull * sm_count;  // warps that run together
    if (s.vec_per_thread == 1) {
        const int most = world < 4 ? 2 : 4;
        while (s.ranks_per_cta < most && warps(s.ranks_per_cta) > round) s.ranks_per_cta *= 2;
        if (warps(s.ranks_per_cta) > 2 * round) {
            s.ranks_per_cta = 2;
            s.late = world != 4;
        }
    } else if (s.vec_per_thread == 2 && elem_bytes == 4 && world == 2) {
        if (warps(1) > round) s.ranks_per_cta = 2;
    } else if (warps(1) > 4 * round) {
        s.late = true;
        s.ranks_per_cta = s.vec_per_thread == 4 && world == 2 ? 1 : 2;
    }
    return s;
}

// CTAs: one per row and group of ranks.  A launch takes up to kMostLocalCtas.
constexpr uint64_t kMostLocalCtas = 0x7fffffff;
inline uint64_t LocalNormCtas(uint64_t rows, int world, const LocalNormShape& s) {
    return rows * ((world + s.ranks_per_cta - 1) / s.ranks_per_cta);
}

// nullptr when the combination is not built.  `wide`: every output starts on a 32-byte
// boundary (sums to a type of twice the width store 32 bytes at a time).
const void* LocalKernelFor(Dtype in, Dtype out, int world, LocalKind kind, bool wide);
// Sum of buffers in host memory that the GPU can address; any number of CTAs.
const void* LocalHostKernelFor(Dtype dt, int world);
const void* LocalNormKernelFor(Dtype dt, int world, const LocalNormShape& shape);

}  // namespace yali
