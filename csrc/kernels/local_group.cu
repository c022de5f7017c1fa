// Collectives of a group whose ranks all live on ONE GPU and run in one launch (emulated ranks, or a
// group of one).  Nothing has to be exchanged there: every rank's input is complete when the launch
// starts (stream order) and every rank's output counts as delivered when it ends, so the barriers, flags
// and staging copies of the multi-GPU kernels carry no information.  What is left is the arithmetic:
// read every rank's input once, add in fp32 in rank order, apply the epilogue, write every rank's output
// once.  No CTA waits for another one, so the launch is an ordinary one, not a cooperative one.
//
// The planner picks these kernels for automatically chosen calls only (PlanCaps::one_launch); a forced
// mode, a forced geometry or a tuning table still runs the multi-GPU kernel it names.
//
// Bound by HBM: bytes of all inputs plus all outputs.  One 16-byte unit per thread and a grid as large as
// the message measured best on B200: two ranks x 128 MiB fp32 80.3 us (6.69 TB/s) with 512 threads,
// against 81-84 us with 2 or 4 units per thread and 92-94 us with a persistent grid-stride loop; the
// pipelined two-shot kernel (TMA stages, two cross-rank barriers) takes 97 us for the same call.  Whole calls
// from Python, back to back, multi-GPU kernel / this one: 4 ranks x 6 MB fp16 18.7 / 8.7 us, 8 ranks x 25 MiB fp32 -> bf16
// 61.1 / 48.4 us, reduce-scatter + all-gather of 64 MiB over 4 ranks 201 / 103 us, all-reduce + residual +
// RMSNorm of 2048 x 4096 bf16 over 2 ranks 49.3 / 23.1 us.
//
// Parity: none in the reference (it always drives two GPUs).
#include "coll_common.cuh"
#include "launch.h"
#include "local_group.h"

namespace yali {

namespace {

// Timeline of a traced call (kFlagTrace): one launch serves every rank, so the first CTA stamps the start
// and the last one the end into the ring of each of them.
__device__ __forceinline__ void local_trace_begin(const LocalArgs& a) {
    if (!(a.flags & kFlagTrace) || blockIdx.x != 0 || blockIdx.y != 0) return;
    if (threadIdx.x < a.world) {
        uint32_t* ctl = a.ctl[threadIdx.x];
        const uint32_t idx = *reinterpret_cast<volatile uint32_t*>(ctl + kCallTraceIdx);
        reinterpret_cast<volatile uint64_t*>(ctl + kTraceOff)[(idx % kTraceCap) * 2] = ptx::globaltimer();
    }
}
__device__ __forceinline__ void local_trace_end(const LocalArgs& a) {
    if (!(a.flags & kFlagTrace)) return;
    __syncthreads();
    if (threadIdx.x != 0) return;
    uint32_t* done = a.ctl[0] + kCallDoneCtas;
    __threadfence();
    if (atomicAdd(done, 1u) != gridDim.x * gridDim.y - 1) return;
    *reinterpret_cast<volatile uint32_t*>(done) = 0u;
    for (uint32_t q = 0; q < a.world; ++q) {
        volatile uint32_t* iw = a.ctl[q] + kCallTraceIdx;
        const uint32_t idx = *iw;
        reinterpret_cast<volatile uint64_t*>(a.ctl[q] + kTraceOff)[(idx % kTraceCap) * 2 + 1] = ptx::globaltimer();
        *iw = idx + 1;
    }
}

// The E elements at element offset e of `base`, as 16-byte vectors.
template <typename Tin, int E>
__device__ __forceinline__ void load_unit(uint4 (&x)[E * sizeof(Tin) / 16], const void* base, uint64_t e) {
#pragma unroll
    for (int i = 0; i < static_cast<int>(E * sizeof(Tin) / 16); ++i)
        x[i] = ptx::ld_cg_v4(static_cast<const char*>(base) + e * sizeof(Tin) + i * 16);
}
// WIDE: a unit of two vectors in one access, on a 32-byte boundary.  Sums to a type of twice the width: a warp that stores 16 bytes at a
// 32-byte stride leaves every sector half written.  In a graph, us, 16 / 32 bytes: bf16 -> fp32: 2 ranks x 1000003 3.9 / 3.4, 6000017 14.8 /
// 12.4; 4 ranks x 1000003 7.0 / 5.2, 6000017 30.2 / 23.2; 8 ranks x 6000017 59.6 / 46.0 (floor 44.1).  Loads of 32 bytes (fp32 ->
// bf16) gain where the inputs are in L2 and lose where they are not: 8 ranks x 250000 3.6 / 3.4 and 5.6 / 6.2, x 6553600 47.2 / 47.8; units
// of 32 bytes for equal types lose (8 ranks x 1000003 bf16 6.5 / 7.1).
template <bool WIDE, int N>
__device__ __forceinline__ void store_vectors(void* base, uint64_t byte, const uint4 (&y)[N]) {
    char* const p = static_cast<char*>(base) + byte;
    if constexpr (N == 2 && WIDE) {
        ptx::st_v8(p, y[0], y[1]);
    } else {
#pragma unroll
        for (int i = 0; i < N; ++i) ptx::st_v4(p + i * 16, y[i]);
    }
}

// KIND: what the grid covers.  Sum: units of the whole message (grid.x).  ReduceScatter / AllGather: units of
// shard blockIdx.y (a shard is a multiple of 16 elements, so it consists of whole units up to the message's
// end); the owner's buffer starts at the shard.
template <typename Tin, typename Tout, int WORLD, LocalKind KIND, bool WIDE>
__global__ void __launch_bounds__(kLocalThreads) local_kernel(const __grid_constant__ LocalArgs a) {
    // Elements of a unit: 16 bytes of the narrower type, so that neither side moves less than 16 bytes.
    constexpr int E = 16 / (sizeof(Tin) < sizeof(Tout) ? sizeof(Tin) : sizeof(Tout));
    constexpr int NIN = E * sizeof(Tin) / 16, NOUT = E * sizeof(Tout) / 16, VOUT = 16 / sizeof(Tout);
    constexpr int kMaxW = WORLD ? WORLD : kMaxRanks;
    const uint32_t W = WORLD ? WORLD : a.world;
    ptx::grid_dependency_wait();
    local_trace_begin(a);
    const EpiScale epi(a.ep);
    const uint32_t owner = KIND == LocalKind::Sum ? 0u : blockIdx.y;
    const uint64_t lo = KIND == LocalKind::Sum ? 0ull : min(a.count, static_cast<uint64_t>(owner) * a.shard_elems);
    const uint64_t hi = KIND == LocalKind::Sum ? a.count : min(a.count, lo + a.shard_elems);
    const uint64_t in_off = KIND == LocalKind::AllGather ? lo : 0ull;      // the owner's input starts at its shard
    const uint64_t out_off = KIND == LocalKind::ReduceScatter ? lo : 0ull;  // the owner's output starts at its shard
    const uint64_t u = static_cast<uint64_t>(blockIdx.x) * kLocalThreads + threadIdx.x;
    const uint64_t e0 = lo + u * E;
    if (a.flags & kFlagVecOk) {
        if (e0 + E <= hi) {
            uint4 x[kMaxW][NIN];
            if constexpr (KIND == LocalKind::AllGather) {
                load_unit<Tin, E>(x[0], a.send[owner], e0 - in_off);
#pragma unroll
                for (int q = 0; q < kMaxW; ++q)
                    if (q < W) store_vectors<WIDE>(a.recv[q], e0 * sizeof(Tout), x[0]);
            } else {
                float f[E];
#pragma unroll
                for (int i = 0; i < E; ++i) f[i] = 0.f;
#pragma unroll
                for (int q = 0; q < kMaxW; ++q)
                    if (q < W) load_unit<Tin, E>(x[q], a.send[q], e0);
#pragma unroll
                for (int q = 0; q < kMaxW; ++q)
                    if (q < W) {
#pragma unroll
                        for (int i = 0; i < NIN; ++i) accumulate<Tin>(f + i * (16 / sizeof(Tin)), x[q][i]);
                    }
#pragma unroll
                for (int i = 0; i < E; ++i) f[i] = epi(f[i]);
                uint4 y[NOUT];
#pragma unroll
                for (int i = 0; i < NOUT; ++i) y[i] = pack16<Tout>(f + i * VOUT);
                if constexpr (KIND == LocalKind::ReduceScatter) {
                    store_vectors<WIDE>(a.recv[owner], (e0 - out_off) * sizeof(Tout), y);
                } else {
#pragma unroll
                    for (int q = 0; q < kMaxW; ++q)
                        if (q < W) store_vectors<WIDE>(a.recv[q], e0 * sizeof(Tout), y);
                }
            }
        }
    }
    // Elements one by one: the remainder behind the last whole unit, or all of them when some buffer is
    // aligned to its element type only.  Every element is read and written by one thread alone, after that
    // thread has read it from every rank: buffers may be used in place.
    uint64_t eb, ee, step;
    if (a.flags & kFlagVecOk) {
        eb = lo + (hi - lo) / E * E + threadIdx.x;
        ee = blockIdx.x == 0 ? hi : 0;
        step = kLocalThreads;
    } else {
        eb = lo + u;
        ee = hi;
        step = static_cast<uint64_t>(gridDim.x) * kLocalThreads;
    }
    for (uint64_t e = eb; e < ee; e += step) {
        Tout o;
        if constexpr (KIND == LocalKind::AllGather) {
            o = static_cast<const Tout*>(a.send[owner])[e - in_off];
        } else {
            float s = 0.f;
#pragma unroll
            for (int q = 0; q < kMaxW; ++q)
                if (q < W) s += to_f32<Tin>(__ldcg(static_cast<const Tin*>(a.send[q]) + e));
            o = from_f32<Tout>(epi(s));
        }
        if constexpr (KIND == LocalKind::ReduceScatter) {
            static_cast<Tout*>(a.recv[owner])[e - out_off] = o;
        } else {
#pragma unroll
            for (int q = 0; q < kMaxW; ++q)
                if (q < W) static_cast<Tout*>(a.recv[q])[e] = o;
        }
    }
    local_trace_end(a);
}

// The sum of buffers in pinned host memory, read and written where they are: both directions of the host link run from the
// first to the last byte, without staging copies, chunks or events.  Bound by that link.  Measured on B200 (PCIe 5),
// 2 ranks x 32 MiB fp32: 1.66-1.70 ms with 16-148 CTAs, 1.94 ms with one 16-byte unit per thread (8192 CTAs), against
// 1.80-2.46 ms for the chunked copies of ops/host_pipeline.cc; copy engines moving the same bytes both ways 1.55 ms.
template <typename T, int WORLD>
__global__ void __launch_bounds__(kLocalHostThreads) local_host_kernel(const __grid_constant__ LocalArgs a) {
    constexpr int VEC = TypeTraits<T>::kVec;
    constexpr int kMaxW = WORLD ? WORLD : kMaxRanks;
    const uint32_t W = WORLD ? WORLD : a.world;
    ptx::grid_dependency_wait();
    local_trace_begin(a);
    const EpiScale epi(a.ep);
    const uint64_t first = static_cast<uint64_t>(blockIdx.x) * kLocalHostThreads + threadIdx.x;
    const uint64_t step = static_cast<uint64_t>(gridDim.x) * kLocalHostThreads;
    const uint64_t nvec = (a.flags & kFlagVecOk) ? a.count / VEC : 0;
    for (uint64_t v = first; v < nvec; v += step) {
        uint4 x[kMaxW];
#pragma unroll
        for (int q = 0; q < kMaxW; ++q)
            if (q < W) x[q] = ptx::ld_cv_v4(static_cast<const char*>(a.send[q]) + v * 16);
        float f[VEC];
#pragma unroll
        for (int i = 0; i < VEC; ++i) f[i] = 0.f;
#pragma unroll
        for (int q = 0; q < kMaxW; ++q)
            if (q < W) accumulate<T>(f, x[q]);
#pragma unroll
        for (int i = 0; i < VEC; ++i) f[i] = epi(f[i]);
        const uint4 y = pack16<T>(f);
#pragma unroll
        for (int q = 0; q < kMaxW; ++q)
            if (q < W) ptx::st_v4(static_cast<char*>(a.recv[q]) + v * 16, y);
    }
    for (uint64_t e = nvec * VEC + first; e < a.count; e += step) {
        float s = 0.f;
#pragma unroll
        for (int q = 0; q < kMaxW; ++q)
            if (q < W) s += to_f32<T>(__ldcv(static_cast<const T*>(a.send[q]) + e));
        const T o = from_f32<T>(epi(s));
#pragma unroll
        for (int q = 0; q < kMaxW; ++q)
            if (q < W) static_cast<T*>(a.recv[q])[e] = o;
    }
    local_trace_end(a);
}

// CTAs of 512 threads of the norm kernel that share an SM, which caps their registers at 32, 40, 64 or 128.  What counts is the warps that share an
// SM: 2 ranks, 2048 x 4096 bf16 22.9 us with 40 registers, 23.4 with 64; 2 ranks, 1024 x 8192 fp32 43.2 with 64, 47.7 with the 72 that it
// takes by itself.  13 instances spill 4 to 12 bytes under it: four ranks per CTA in bf16 and fp16, and three of seven ranks behind the barrier.
// One CTA per SM less and no spills cost more (us, as it is / without): 8 ranks, 256 x 4096 bf16 14.2 / 17.9, 180 x 4096 11.3 / 13.3; 4 ranks, 256 x 4096
// bf16 7.9 / 9.7, 300 x 4096 fp16 10.6 / 12.0, but 512 x 2944 11.6 / 11.2; 5 ranks, 300 x 4096 fp16 level; 7 ranks, 1000 x 4096 bf16 45.6 / 51.1,
// 300 x 8192 fp16 29.2 / 36.8.
constexpr int norm_ctas(int world, int nv, bool late, int elem_bytes) {
    if (nv == 1) return world == 1 ? 4 : late ? 3 : 2;
    return nv == 2 || (world == 2 && late && elem_bytes == 4) ? 2 : 1;
}

// Sum + residual + RMSNorm of one row for the ranks [g * G, g * G + G) of the group; CTA b handles row
// b / ngroups, group b % ngroups (the groups of a row are neighbours, so the second one finds the row in
// L2).  A thread holds NV vectors of the row: it reads them from every rank once, adds in fp32, and keeps
// the packed residuals of its G ranks until the G sums of squares are known (one block reduction for all).
//
// Bound by HBM with many rows, where the phases of a CTA (loads, barrier, stores) have to run under those of others: few registers, so
// that two or more CTAs of 512 threads share an SM, and for that two ranks at a time (LATE asks for their weights behind the barrier).
// Bound by the chain of latencies with few, where it helps to have the weights before the barrier (one by one behind the stores each
// rank's is a latency) and ranks spread over CTAs.  LocalNormShapeFor has the lines.  In a graph, inputs from HBM, all ranks of a row in a
// CTA and weights one by one / now, us (floor): bf16, 8 ranks: 64 x 4096 9.5 / 4.9 (2.6), 256 x 4096 19.4 / 14.0 (10.3), 512 x 4096 33.2 / 25.5
// (20.6), 1000 x 2944 44.7 / 34.9 (28.9), 500 x 8192 59.8 / 48.5 (40.2); 4 ranks: 256 x 1024 4.7 / 3.1, 1024 x 8192 57.3 / 46.7 (41.1);
// 2 ranks: 64 x 8192 4.1 / 2.9, 2000 x 8192 44.6 / 41.7 (40.2), 2048 x 4096 22.9 / 22.8 (20.6); 3 ranks, 1500 x 4096 45 / 27.4 (22.6); one rank,
// 8192 x 8192 83.6 / 82.2 (82.2); fp32, 8 ranks, 250 x 8192 71.8 / 49.6 (40.2).
template <typename T, int WORLD, int NV, int G, bool LATE>
__global__ void __launch_bounds__(kLocalThreads, norm_ctas(WORLD, NV, LATE, sizeof(T))) local_norm_kernel(const __grid_constant__ LocalArgs a) {
    constexpr int VEC = TypeTraits<T>::kVec, kMostWarps = kLocalThreads / 32;
    constexpr uint32_t W = WORLD;
    __shared__ __align__(16) float s_red[G][kMostWarps];
    const int tid = threadIdx.x, nt = blockDim.x;
    if (nt < kLocalThreads)  // those of warps that a CTA of this size has not
        for (int i = tid; i < G * kMostWarps; i += nt) (&s_red[0][0])[i] = 0.f;
    const uint32_t ngroups = (W + G - 1) / G;
    const uint32_t row = ngroups == 1 ? blockIdx.x : blockIdx.x / ngroups, q0 = (blockIdx.x - row * ngroups) * G;
    const uint32_t vec_per_row = a.ep.hidden / VEC;
    const uint64_t row_off = static_cast<uint64_t>(row) * vec_per_row * 16;
    // A thread without a vector of the row (the last ones of a CTA) loads the row's last one, which costs no branch and no zeros, and
    // keeps it out of the sum of squares and of memory.
    bool have[NV];
    uint32_t at[NV];  // byte in the row
#pragma unroll
    for (int j = 0; j < NV; ++j) {
        have[j] = tid + j * nt < vec_per_row;
        at[j] = min(static_cast<uint32_t>(tid + j * nt), vec_per_row - 1) * 16;
    }
    if (nt < kLocalThreads) __syncthreads();
    ptx::grid_dependency_wait();
    local_trace_begin(a);

    uint4 res[NV][G], wgt[NV][LATE ? 1 : G];
    float f[NV][VEC];
    auto load_residuals = [&](int j) {
#pragma unroll
        for (int g = 0; g < G; ++g) {
            const char* const r = q0 + g < W ? static_cast<const char*>(a.residual[q0 + g]) : nullptr;
            res[j][g] = r ? ptx::ld_cg_v4(r + row_off + at[j]) : make_uint4(0, 0, 0, 0);
        }
    };
    // Residuals ahead of all inputs or with the inputs of their vector: how many loads the compiler leaves in flight under its cap depends on it (us,
    // ahead / with: fp32, 3 ranks 300 x 8192 23.2 / 26.1, 5 ranks 40 x 8192 8.1 / 8.6, 7 ranks 60 x 4096 8.1 / 10.3; but 6 ranks 300 x 8192 46.7 / 44.0,
    // 8 ranks 120 x 4096 15.9 / 15.5, bf16 500 x 8192 49.8 / 48.3).
    constexpr bool kResidualsFirst = sizeof(T) == 4 && WORLD > 1 && (WORLD & 1);
    if constexpr (kResidualsFirst) {
#pragma unroll
        for (int j = 0; j < NV; ++j) load_residuals(j);
    }
#pragma unroll
    for (int j = 0; j < NV; ++j) {
        uint4 x[W];
#pragma unroll
        for (int q = 0; q < WORLD; ++q) x[q] = ptx::ld_cg_v4(static_cast<const char*>(a.send[q]) + row_off + at[j]);
        if constexpr (!kResidualsFirst) load_residuals(j);
        unpack16<T>(f[j], x[0]);
#pragma unroll
        for (int q = 1; q < WORLD; ++q) accumulate<T>(f[j], x[q]);
    }
    auto load_weight = [&](int j, int g) { return ptx::ld_v4(static_cast<const char*>(a.weight[min(q0 + g, W - 1)]) + at[j]); };
    if constexpr (!LATE) {
#pragma unroll
        for (int g = 0; g < G; ++g)
#pragma unroll
            for (int j = 0; j < NV; ++j) wgt[j][g] = load_weight(j, g);
    }
#pragma unroll
    for (int g = 0; g < G; ++g) {
        float ss = 0.f;
        char* const ro = q0 + g < W ? static_cast<char*>(a.residual_out[q0 + g]) : nullptr;
#pragma unroll
        for (int j = 0; j < NV; ++j) {
            float p[VEC];
#pragma unroll
            for (int i = 0; i < VEC; ++i) p[i] = f[j][i];
            accumulate<T>(p, res[j][g]);
            if (ro && have[j]) ptx::st_v4(ro + row_off + at[j], pack16<T>(p));
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
    const float inv_h = 1.f / static_cast<float>(a.ep.hidden);
#pragma unroll
    for (int g = 0; g < G; ++g) {
        if (q0 + g >= W) break;
        if constexpr (LATE) {
#pragma unroll
            for (int j = 0; j < NV; ++j) wgt[j][0] = load_weight(j, g);
        }
        float t = 0.f;
#pragma unroll
        for (int w = 0; w < kMostWarps; w += 4) {
            const float4 part = *reinterpret_cast<const float4*>(&s_red[g][w]);
            t += (part.x + part.y) + (part.z + part.w);
        }
        const float inv_rms = rsqrtf(t * inv_h + a.ep.eps);
#pragma unroll
        for (int j = 0; j < NV; ++j) {
            if (!have[j]) continue;
            float p[VEC], w[VEC];
#pragma unroll
            for (int i = 0; i < VEC; ++i) p[i] = f[j][i];
            accumulate<T>(p, res[j][g]);
            unpack16<T>(w, wgt[j][LATE ? 0 : g]);
#pragma unroll
            for (int i = 0; i < VEC; ++i) p[i] = p[i] * inv_rms * w[i];
            ptx::st_v4(static_cast<char*>(a.recv[q0 + g]) + row_off + at[j], pack16<T>(p));
        }
    }
    local_trace_end(a);
}

template <typename Tin, typename Tout, LocalKind KIND, bool WIDE = false>
const void* pick_world(int world) {
    switch (world) {
        case 1: return (const void*)local_kernel<Tin, Tout, 1, KIND, WIDE>;
        case 2: return (const void*)local_kernel<Tin, Tout, 2, KIND, WIDE>;
        case 4: return (const void*)local_kernel<Tin, Tout, 4, KIND, WIDE>;
        case 8: return (const void*)local_kernel<Tin, Tout, 8, KIND, WIDE>;
        default: return (const void*)local_kernel<Tin, Tout, 0, KIND, WIDE>;
    }
}
template <typename Tin, typename Tout>
const void* pick_mixed(int world, bool wide) {
    if constexpr (sizeof(Tout) > sizeof(Tin)) {
        if (wide) return pick_world<Tin, Tout, LocalKind::Sum, true>(world);
    }
    return pick_world<Tin, Tout, LocalKind::Sum>(world);
}
template <typename T>
const void* pick_host(int world) {
    switch (world) {
        case 1: return (const void*)local_host_kernel<T, 1>;
        case 2: return (const void*)local_host_kernel<T, 2>;
        case 4: return (const void*)local_host_kernel<T, 4>;
        case 8: return (const void*)local_host_kernel<T, 8>;
        default: return (const void*)local_host_kernel<T, 0>;
    }
}
template <LocalKind KIND>
const void* pick_same(Dtype dt, int world) {
    switch (dt) {
        case Dtype::FP32: return pick_world<float, float, KIND>(world);
        case Dtype::FP16: return pick_world<__half, __half, KIND>(world);
        case Dtype::BF16: return pick_world<__nv_bfloat16, __nv_bfloat16, KIND>(world);
    }
    return nullptr;
}
// The instances that LocalNormShapeFor asks for; nullptr for others.
template <typename T, int WORLD, int NV, int G>
const void* pick_norm_late(bool late) {
    constexpr bool kPairEarly = sizeof(T) == 4 && WORLD == 2 && NV == 2;
    constexpr bool kEarly = NV == 1 || G == 1 || kPairEarly;
    constexpr bool kLate = WORLD > 1 && (NV == 1 ? G == 2 && WORLD != 4 : NV == 2 ? G == 2 && !kPairEarly : G == (WORLD == 2 ? 1 : 2));
    if constexpr (kLate) {
        if (late) return (const void*)local_norm_kernel<T, WORLD, NV, G, true>;
    }
    if constexpr (kEarly) {
        if (!late) return (const void*)local_norm_kernel<T, WORLD, NV, G, false>;
    }
    return nullptr;
}
template <typename T, int WORLD, int NV>
const void* pick_norm_g(const LocalNormShape& s) {
    if constexpr (NV == 1 && WORLD >= 4) {
        if (s.ranks_per_cta == 4) return pick_norm_late<T, WORLD, NV, 4>(s.late);
    }
    if constexpr (WORLD >= 2) {
        if (s.ranks_per_cta == 2) return pick_norm_late<T, WORLD, NV, 2>(s.late);
    }
    return pick_norm_late<T, WORLD, NV, 1>(s.late);
}
template <typename T, int WORLD>
const void* pick_norm_nv(const LocalNormShape& s) {
    return s.vec_per_thread == 1   ? pick_norm_g<T, WORLD, 1>(s)
           : s.vec_per_thread == 2 ? pick_norm_g<T, WORLD, 2>(s)
                                   : pick_norm_g<T, WORLD, 4>(s);
}
template <typename T>
const void* pick_norm(int world, const LocalNormShape& s) {
    static_assert(kMaxRanks == 8, "one instance per group size");
    switch (world) {
        case 1: return pick_norm_nv<T, 1>(s);
        case 2: return pick_norm_nv<T, 2>(s);
        case 3: return pick_norm_nv<T, 3>(s);
        case 4: return pick_norm_nv<T, 4>(s);
        case 5: return pick_norm_nv<T, 5>(s);
        case 6: return pick_norm_nv<T, 6>(s);
        case 7: return pick_norm_nv<T, 7>(s);
        case 8: return pick_norm_nv<T, 8>(s);
    }
    return nullptr;
}

}  // namespace

const void* LocalKernelFor(Dtype in, Dtype out, int world, LocalKind kind, bool wide) {
    using bf16 = __nv_bfloat16;
    if (kind == LocalKind::ReduceScatter) return in == out ? pick_same<LocalKind::ReduceScatter>(in, world) : nullptr;
    if (kind == LocalKind::AllGather) return in == out ? pick_same<LocalKind::AllGather>(in, world) : nullptr;
    constexpr LocalKind S = LocalKind::Sum;
    if (in == out) return pick_same<S>(in, world);
    if (in == Dtype::FP32 && out == Dtype::BF16) return pick_mixed<float, bf16>(world, wide);
    if (in == Dtype::FP32 && out == Dtype::FP16) return pick_mixed<float, __half>(world, wide);
    if (in == Dtype::BF16 && out == Dtype::FP32) return pick_mixed<bf16, float>(world, wide);
    if (in == Dtype::FP16 && out == Dtype::FP32) return pick_mixed<__half, float>(world, wide);
    return nullptr;
}

const void* LocalHostKernelFor(Dtype dt, int world) {
    switch (dt) {
        case Dtype::FP32: return pick_host<float>(world);
        case Dtype::FP16: return pick_host<__half>(world);
        case Dtype::BF16: return pick_host<__nv_bfloat16>(world);
    }
    return nullptr;
}

const void* LocalNormKernelFor(Dtype dt, int world, const LocalNormShape& s) {
    switch (dt) {
        case Dtype::FP32: return pick_norm<float>(world, s);
        case Dtype::FP16: return pick_norm<__half>(world, s);
        case Dtype::BF16: return pick_norm<__nv_bfloat16>(world, s);
    }
    return nullptr;
}

}  // namespace yali
