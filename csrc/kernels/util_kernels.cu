// Buffer utilities: seeded fills, conversion to fp32 and on-device validation of
// an all-reduce result against the sum recomputed from the generators in fp64.
//
// Parity: seed_buffer_kernel / SeedBufferSync / ZeroBuffer / AllocAndSeed
// (src/common/buffer_ops.cuh:16-59) fill with one constant per rank, and
// convert_to_float_kernel / VerifyAllReduceSum / ValidateRankResult
// (src/common/validation.cuh:18-115) copy the result to the host and expect
// N(N+1)/2 everywhere.  Constant fills are kept; in addition a counter-based
// generator (Philox4x32-10, identical on host and device) gives every element of
// every rank its own U(-1,1) or N(0,1) value, so a missing, duplicated or
// misplaced contribution changes the numbers.
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "../ops/buffer_ops.h"
#include "launch.h"
#include "type_ops.cuh"

namespace yali {

namespace {

template <typename T>
__global__ void fill_constant_kernel(T* p, uint64_t n, float v) {
    const T x = from_f32<T>(v);
    for (uint64_t i = blockIdx.x * static_cast<uint64_t>(blockDim.x) + threadIdx.x; i < n;
         i += static_cast<uint64_t>(gridDim.x) * blockDim.x)
        p[i] = x;
}

template <typename T>
__global__ void fill_random_kernel(T* p, uint64_t n, int dist, uint64_t seed) {
    for (uint64_t i = blockIdx.x * static_cast<uint64_t>(blockDim.x) + threadIdx.x; i < n;
         i += static_cast<uint64_t>(gridDim.x) * blockDim.x)
        p[i] = from_f32<T>(RandomValue(dist, seed, i));
}

template <typename T>
__global__ void to_float_kernel(const T* src, float* dst, uint64_t n) {
    for (uint64_t i = blockIdx.x * static_cast<uint64_t>(blockDim.x) + threadIdx.x; i < n;
         i += static_cast<uint64_t>(gridDim.x) * blockDim.x)
        dst[i] = to_f32<T>(src[i]);
}

// expected[i] = scale * sum_r round_to_Tin(gen(seed_base + r, i)) in fp64.
template <typename Tin, typename Tout>
__global__ void validate_sum_kernel(const Tout* out, uint64_t n, uint64_t index_offset, int dist, uint64_t seed_base,
                                    int world, float scale, double rtol, double atol, ValidateReport* rep) {
    unsigned long long bad = 0;
    double worst = 0.0;
    unsigned long long first = ~0ull;
    for (uint64_t i = blockIdx.x * static_cast<uint64_t>(blockDim.x) + threadIdx.x; i < n;
         i += static_cast<uint64_t>(gridDim.x) * blockDim.x) {
        double e = 0.0;
        for (int r = 0; r < world; ++r)
            e += static_cast<double>(to_f32<Tin>(from_f32<Tin>(RandomValue(dist, seed_base + r, index_offset + i))));
        e *= static_cast<double>(scale);
        const double got = static_cast<double>(to_f32<Tout>(out[i]));
        const double err = fabs(got - e);
        if (!(err <= atol + rtol * fabs(e))) {
            ++bad;
            if (i < first) first = i;
        }
        if (err > worst || err != err) worst = (err != err) ? 1e300 : err;
    }
    if (bad) {
        atomicAdd(&rep->mismatches, bad);
        atomicMin(&rep->first_mismatch, first);
    }
    // max of non-negative doubles == max of their bit patterns
    atomicMax(reinterpret_cast<unsigned long long*>(&rep->max_abs_err),
              static_cast<unsigned long long>(__double_as_longlong(worst)));
}

// In-place residual add + RMSNorm over rows of `hidden` elements, one CTA per row.
// Used when a message is too large for the one-shot kernel that fuses this step: the all-reduce
// runs first, then this kernel normalises the local result.  (Ranks that share one GPU have local_group.cu, except for what that does not take.)
// Bound by HBM (three or four row images in and out).  A thread keeps its NV vectors of the row in registers
// between the sum of squares and the store, so the row is read once; 16-byte accesses.
template <typename T, int NV>
__global__ void __launch_bounds__(512) residual_rmsnorm_kernel(T* x, const T* residual, T* residual_out, const T* weight,
                                                               uint32_t hidden, float eps, bool store_rows) {
    constexpr int VEC = TypeTraits<T>::kVec;
    __shared__ float s_part[16];
    ptx::grid_dependency_wait();
    const int tid = threadIdx.x, nt = blockDim.x;
    const uint32_t vec_per_row = hidden / VEC;
    const uint64_t row_off = static_cast<uint64_t>(blockIdx.x) * hidden;
    float f[NV][VEC];
    float ss = 0.f;
#pragma unroll
    for (int j = 0; j < NV; ++j) {
        const uint32_t c = tid + j * nt;
#pragma unroll
        for (int i = 0; i < VEC; ++i) f[j][i] = 0.f;
        if (c < vec_per_row) {
            const uint64_t e = row_off + static_cast<uint64_t>(c) * VEC;
            const uint4 xv = ptx::ld_cg_v4(x + e);
            const uint4 rv = residual ? ptx::ld_cg_v4(residual + e) : make_uint4(0, 0, 0, 0);
            accumulate<T>(f[j], xv);
            if (residual) accumulate<T>(f[j], rv);
            if (residual_out) ptx::st_v4(residual_out + e, pack16<T>(f[j]));
        }
#pragma unroll
        for (int i = 0; i < VEC; ++i) ss += f[j][i] * f[j][i];
    }
    for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
    if ((tid & 31) == 0) s_part[tid >> 5] = ss;
    __syncthreads();
    float tot = 0.f;
    for (int w = 0; w < (nt + 31) / 32; ++w) tot += s_part[w];
    const float inv = rsqrtf(tot / static_cast<float>(hidden) + eps);
#pragma unroll
    for (int j = 0; j < NV; ++j) {
        const uint32_t c = tid + j * nt;
        if (c < vec_per_row && store_rows) {
            float w[VEC];
#pragma unroll
            for (int i = 0; i < VEC; ++i) w[i] = 0.f;
            accumulate<T>(w, *reinterpret_cast<const uint4*>(weight + static_cast<uint64_t>(c) * VEC));
#pragma unroll
            for (int i = 0; i < VEC; ++i) f[j][i] = f[j][i] * inv * w[i];
            ptx::st_v4(x + row_off + static_cast<uint64_t>(c) * VEC, pack16<T>(f[j]));
        }
    }
}

// The same element by element: rows that are no whole number of 16-byte vectors, are longer than 2048 of
// them, or start on an address that is aligned to the element only.  A row is read twice, so nothing is stored before the second time:
// the residual may be updated in place.
template <typename T>
__global__ void residual_rmsnorm_elems_kernel(T* x, const T* residual, T* residual_out, const T* weight, uint64_t rows,
                                              uint32_t hidden, float eps, bool store_rows) {
    __shared__ float s_part[32];
    const int tid = threadIdx.x, nt = blockDim.x;
    for (uint64_t row = blockIdx.x; row < rows; row += gridDim.x) {
        T* xr = x + row * hidden;
        float ss = 0.f;
        for (uint32_t c = tid; c < hidden; c += nt) {
            float v = to_f32<T>(xr[c]);
            if (residual) v += to_f32<T>(residual[row * hidden + c]);
            ss += v * v;
        }
        for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
        __syncthreads();
        if ((tid & 31) == 0) s_part[tid >> 5] = ss;
        __syncthreads();
        float tot = 0.f;
        for (int w = 0; w < (nt + 31) / 32; ++w) tot += s_part[w];
        const float inv = rsqrtf(tot / static_cast<float>(hidden) + eps);
        for (uint32_t c = tid; c < hidden; c += nt) {
            float v = to_f32<T>(xr[c]);
            if (residual) v += to_f32<T>(residual[row * hidden + c]);
            if (residual_out) residual_out[row * hidden + c] = from_f32<T>(v);
            if (store_rows) xr[c] = from_f32<T>(v * inv * to_f32<T>(weight[c]));
        }
    }
}

int GridFor(uint64_t n) {
    uint64_t b = (n + 255) / 256;
    if (b < 1) b = 1;
    if (b > 148 * 8) b = 148 * 8;
    return static_cast<int>(b);
}

template <typename Tin>
cudaError_t ValidateOut(const void* out, Dtype out_dt, uint64_t n, uint64_t off, int dist, uint64_t seed, int world,
                        float scale, double rtol, double atol, ValidateReport* d_rep, cudaStream_t s) {
    switch (out_dt) {
        case Dtype::FP32:
            validate_sum_kernel<Tin, float><<<GridFor(n), 256, 0, s>>>(static_cast<const float*>(out), n, off, dist,
                                                                       seed, world, scale, rtol, atol, d_rep);
            break;
        case Dtype::FP16:
            validate_sum_kernel<Tin, __half><<<GridFor(n), 256, 0, s>>>(static_cast<const __half*>(out), n, off, dist,
                                                                        seed, world, scale, rtol, atol, d_rep);
            break;
        case Dtype::BF16:
            validate_sum_kernel<Tin, __nv_bfloat16><<<GridFor(n), 256, 0, s>>>(
                static_cast<const __nv_bfloat16*>(out), n, off, dist, seed, world, scale, rtol, atol, d_rep);
            break;
    }
    return cudaGetLastError();
}

}  // namespace

cudaError_t FillConstant(void* p, uint64_t n, Dtype dt, float v, cudaStream_t s) {
    if (n == 0) return cudaSuccess;
    switch (dt) {
        case Dtype::FP32: fill_constant_kernel<<<GridFor(n), 256, 0, s>>>(static_cast<float*>(p), n, v); break;
        case Dtype::FP16: fill_constant_kernel<<<GridFor(n), 256, 0, s>>>(static_cast<__half*>(p), n, v); break;
        case Dtype::BF16: fill_constant_kernel<<<GridFor(n), 256, 0, s>>>(static_cast<__nv_bfloat16*>(p), n, v); break;
    }
    return cudaGetLastError();
}

cudaError_t FillRandom(void* p, uint64_t n, Dtype dt, int dist, uint64_t seed, cudaStream_t s) {
    if (n == 0) return cudaSuccess;
    switch (dt) {
        case Dtype::FP32: fill_random_kernel<<<GridFor(n), 256, 0, s>>>(static_cast<float*>(p), n, dist, seed); break;
        case Dtype::FP16: fill_random_kernel<<<GridFor(n), 256, 0, s>>>(static_cast<__half*>(p), n, dist, seed); break;
        case Dtype::BF16:
            fill_random_kernel<<<GridFor(n), 256, 0, s>>>(static_cast<__nv_bfloat16*>(p), n, dist, seed);
            break;
    }
    return cudaGetLastError();
}

cudaError_t ConvertToFloat(const void* src, float* dst, uint64_t n, Dtype dt, cudaStream_t s) {
    if (n == 0) return cudaSuccess;
    switch (dt) {
        case Dtype::FP32: to_float_kernel<<<GridFor(n), 256, 0, s>>>(static_cast<const float*>(src), dst, n); break;
        case Dtype::FP16: to_float_kernel<<<GridFor(n), 256, 0, s>>>(static_cast<const __half*>(src), dst, n); break;
        case Dtype::BF16:
            to_float_kernel<<<GridFor(n), 256, 0, s>>>(static_cast<const __nv_bfloat16*>(src), dst, n);
            break;
    }
    return cudaGetLastError();
}

cudaError_t ValidateSumAsync(const void* out, uint64_t n, uint64_t index_offset, Dtype in_dt, Dtype out_dt, int dist,
                             uint64_t seed_base, int world, float scale, double rtol, double atol,
                             ValidateReport* d_rep, cudaStream_t s) {
    if (n == 0) return cudaSuccess;
    switch (in_dt) {
        case Dtype::FP32:
            return ValidateOut<float>(out, out_dt, n, index_offset, dist, seed_base, world, scale, rtol, atol, d_rep, s);
        case Dtype::FP16:
            return ValidateOut<__half>(out, out_dt, n, index_offset, dist, seed_base, world, scale, rtol, atol, d_rep,
                                       s);
        case Dtype::BF16:
            return ValidateOut<__nv_bfloat16>(out, out_dt, n, index_offset, dist, seed_base, world, scale, rtol, atol,
                                              d_rep, s);
    }
    return cudaErrorInvalidValue;
}

namespace {
template <typename T>
void LaunchResidualRmsNorm(void* x, const void* residual, void* residual_out, const void* weight, uint64_t rows,
                           uint32_t hidden, float eps, cudaStream_t s, bool store_rows) {
    constexpr uint32_t VEC = TypeTraits<T>::kVec;
    T* xt = static_cast<T*>(x);
    const T* rt = static_cast<const T*>(residual);
    T* ot = static_cast<T*>(residual_out);
    const T* wt = static_cast<const T*>(weight);
    const uint32_t vec_per_row = hidden / VEC;
    const bool aligned = ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(residual) |
                           reinterpret_cast<uintptr_t>(residual_out) | reinterpret_cast<uintptr_t>(weight)) & 15u) == 0;
    if (hidden % VEC != 0 || vec_per_row > 2048 || !aligned || rows > 0x7fffffffull) {
        const int grid = static_cast<int>(rows < 148 * 8 ? rows : 148 * 8);
        residual_rmsnorm_elems_kernel<<<grid, 256, 0, s>>>(xt, rt, ot, wt, rows, hidden, eps, store_rows);
        return;
    }
    // Two vectors per thread from 256 vectors on: enough loads in flight, and four or more rows per SM.
    const uint32_t nv = vec_per_row <= 128 ? 1 : vec_per_row <= 1024 ? 2 : 4;
    const uint32_t threads = ((vec_per_row + nv - 1) / nv + 31) / 32 * 32;
    const uint32_t grid = static_cast<uint32_t>(rows);
    const void* fn = nv == 1   ? (const void*)residual_rmsnorm_kernel<T, 1>
                     : nv == 2 ? (const void*)residual_rmsnorm_kernel<T, 2>
                               : (const void*)residual_rmsnorm_kernel<T, 4>;
    void* params[] = {&xt, &rt, &ot, &wt, &hidden, &eps, &store_rows};
    (void)LaunchInStream(fn, dim3(grid), dim3(threads), params, 0, s);
}
}  // namespace

cudaError_t ResidualRmsNormInPlace(void* x, const void* residual, void* residual_out, const void* weight, uint64_t rows,
                                   uint32_t hidden, float eps, Dtype dt, cudaStream_t s, bool store_rows) {
    if (rows == 0) return cudaSuccess;
    switch (dt) {
        case Dtype::FP32: LaunchResidualRmsNorm<float>(x, residual, residual_out, weight, rows, hidden, eps, s, store_rows); break;
        case Dtype::FP16: LaunchResidualRmsNorm<__half>(x, residual, residual_out, weight, rows, hidden, eps, s, store_rows); break;
        case Dtype::BF16: LaunchResidualRmsNorm<__nv_bfloat16>(x, residual, residual_out, weight, rows, hidden, eps, s, store_rows); break;
    }
    return cudaGetLastError();
}

}  // namespace yali
