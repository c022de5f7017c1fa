// Host-side entry points of the kernel translation units.  Each returns the
// __global__ function for a (dtype, epilogue, world) combination so that the
// dispatcher can launch it with LaunchInStream below (one rank per launch) or, for
// an emulated communicator whose ranks share one GPU, with a cooperative launch
// of the *_emu twin (ranks = blockIdx.y), which guarantees that all CTAs that
// wait on one another are resident together.
//
// Parity: src/all_reduce/kernels.cuh:41-55 (LaunchFlashKernel) and the
// extern "C" YaliKernel symbols of src/kernels/stream.cu:104-111.
#pragma once

#include <cuda_runtime.h>

#include <cstring>

#include "../comm/layout.h"

namespace yali {

constexpr int kFlashThreads = 512;
constexpr int kStreamThreads = 512;
constexpr int kNvlsThreads = 512;
constexpr int kDirectThreads = 288;   // one producer warp + eight consumer warps
constexpr int kDirectMaxStages = kMaxPipelineStages;

// Ordinary (not cooperative) launch.  Programmatic stream serialization lets the launch overlap the end of the kernel in
// front of it in the stream, whose end the kernel waits for with ptx::grid_dependency_wait() before it reads or writes memory
// (prefetches into L2 aside).  Every kernel launched here has to: the row kernel of the fused layer for one GPU releases
// the kernel behind it when it starts.  That row kernel itself is the one exception.  It waits only at its end, and may run
// because the GEMM in front of it releases it behind its own wait.  Without the attribute back-to-back launches on B200 take
// turns on a 2.05 us grid: a 5.2 us kernel came every 8.2 us, with it every 5.9 us.
inline cudaError_t LaunchInStream(const void* fn, dim3 grid, dim3 block, void** params, size_t smem, cudaStream_t s) {
    cudaLaunchConfig_t cfg;
    std::memset(&cfg, 0, sizeof(cfg));
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute at;
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelExC(&cfg, fn, params);
}

// nullptr when the combination is not built.
const void* FlashKernelFor(Dtype in, Dtype out, int epilogue, int world, bool emu);
// Flag-in-data form of the one-shot kernel (equal in/out type, scale epilogue only).
const void* FlashLLKernelFor(Dtype dt, int world, bool emu);
const void* StreamKernelFor(Dtype in, Dtype out, int epilogue, int world, bool emu);
const void* NvlsKernelFor(Dtype dt, int world, bool two_shot);
// Pipelined direct kernel (all buffers peer-addressable): one-shot pull or two-shot pull + push.
const void* DirectKernelFor(Dtype in, Dtype out, int world, bool one_shot, bool emu);

}  // namespace yali
