// Layer norm with a gain and no bias, in the two forms a decoder step needs, and the cast of
// the 32-bit residual stream to the storage type of the matrix products.
//
//   plain        y[r] = T( LN(src[s]) * gain )            s = rows ? rows[r] : r, src is 32-bit
//   accumulate   x[r] += LN(src[r]) * gain;  y[r] = T(x[r])   src is a sublayer's output (type T)
//
// LN(v) = (v - mean(v)) / sqrt(mean((v - mean(v))^2) + eps): the variance is the mean of the
// squared deviations, taken in a second pass over the row (kept in shared memory).  Statistics,
// the gain and the residual sum are 32-bit whatever T is.
#include "common.cuh"

namespace fsie {

template <typename S, typename T>
__global__ void add_layernorm_kernel(const S* __restrict__ src, const int* __restrict__ rows,
                                     const float* __restrict__ gain, float* __restrict__ x,
                                     T* __restrict__ y, int width, float eps) {
    extern __shared__ float row_cache[];
    __shared__ float scratch[32];
    grid_dependency_wait();
    grid_dependents_go();
    const int r = blockIdx.x;
    const size_t s = rows ? (size_t)rows[r] : (size_t)r;
    const S* in = src + s * width;
    float sum = 0.f;
    for (int c = threadIdx.x; c < width; c += blockDim.x) {
        const float v = to_float(in[c]);
        row_cache[c] = v;
        sum += v;
    }
    const float mean = block_sum(sum, scratch) / (float)width;
    float sq = 0.f;
    for (int c = threadIdx.x; c < width; c += blockDim.x) {
        const float d = row_cache[c] - mean;
        sq += d * d;
    }
    const float inv = 1.0f / sqrtf(block_sum(sq, scratch) / (float)width + eps);
    float* xr = x ? x + (size_t)r * width : nullptr;
    T* yr = y ? y + (size_t)r * width : nullptr;
    for (int c = threadIdx.x; c < width; c += blockDim.x) {
        float v = (row_cache[c] - mean) * inv * gain[c];
        if (xr) {
            v += xr[c];
            xr[c] = v;
        }
        if (yr) yr[c] = from_float<T>(v);
    }
}

// The same, to the bit, with the row in registers (at most PER values of a thread, all asked for at once): a step of few
// tokens is a chain of such rows, each two sums over a block, and nothing but their trips to memory and barriers bounds it
// (4 rows of 2,048 took 6.9 us of the step's chain, a turn through shared memory for each value, and 3.7 now); the gain, a
// constant, is asked for before the kernel before has finished.  A thread keeps the values that it has above, neighbours apart by
// the block: eight neighbours of a thread would be one load, but another order of the sums.
template <typename S, typename T, int PER>
__global__ void __launch_bounds__(512) add_layernorm_regs_kernel(const S* __restrict__ src, const int* __restrict__ rows,
                                                                 const float* __restrict__ gain, float* __restrict__ x,
                                                                 T* __restrict__ y, int width, float eps) {
    __shared__ float scratch[32];
    const int r = blockIdx.x;
    float g[PER], v[PER], old[PER];
#pragma unroll
    for (int i = 0; i < PER; ++i) {
        const int c = threadIdx.x + i * blockDim.x;
        g[i] = c < width ? gain[c] : 0.f;
    }
    grid_dependency_wait();
    grid_dependents_go();
    const size_t s = rows ? (size_t)rows[r] : (size_t)r;
    const S* in = src + s * width;
    float* xr = x ? x + (size_t)r * width : nullptr;
    T* yr = y ? y + (size_t)r * width : nullptr;
#pragma unroll
    for (int i = 0; i < PER; ++i) {
        const int c = threadIdx.x + i * blockDim.x;
        v[i] = c < width ? to_float(in[c]) : 0.f;
    }
#pragma unroll
    for (int i = 0; i < PER; ++i) {
        const int c = threadIdx.x + i * blockDim.x;
        old[i] = xr && c < width ? xr[c] : 0.f;
    }
    float sum = 0.f;
#pragma unroll
    for (int i = 0; i < PER; ++i)
        if (threadIdx.x + i * blockDim.x < width) sum += v[i];
    const float mean = block_sum(sum, scratch) / (float)width;
    float sq = 0.f;
#pragma unroll
    for (int i = 0; i < PER; ++i)
        if (threadIdx.x + i * blockDim.x < width) {
            const float d = v[i] - mean;
            sq += d * d;
        }
    const float inv = 1.0f / sqrtf(block_sum(sq, scratch) / (float)width + eps);
#pragma unroll
    for (int i = 0; i < PER; ++i) {
        const int c = threadIdx.x + i * blockDim.x;
        if (c >= width) break;
        float n = (v[i] - mean) * inv * g[i];
        if (xr) {
            n = fmaf((v[i] - mean) * inv, g[i], old[i]);        // (written out: the general kernel's product is not rounded before)
            xr[c] = n;
        }
        if (yr) yr[c] = from_float<T>(n);
    }
}

template <typename T>
__global__ void cast_rows_kernel(const float* __restrict__ x, T* __restrict__ y, long long count) {
    grid_dependency_wait();
    grid_dependents_go();
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < count;
         i += (long long)gridDim.x * blockDim.x)
        y[i] = from_float<T>(x[i]);
}

}  // namespace fsie

using namespace fsie;

extern "C" {

// accumulate = 0: src is float [*, width] (read at `rows` if given), y gets the normed rows.
// accumulate = 1: src is of the storage type, x (float) += LN(src) * gain, y (optional) = T(x).
// general != 0: the kernel for rows of any width, whatever the width.
int fsie_add_layernorm(const void* src, const int* rows, const float* gain, float* x, void* y,
                       int num_rows, int width, float eps, int accumulate, int dtype,
                       int general, int early, cudaStream_t stream) {
    if (num_rows <= 0) return 0;
    if (width <= 0 || (!accumulate && !y) || (accumulate && !x)) return ERR_BAD_ARGUMENT;
    const size_t smem = (size_t)width * sizeof(float);
    if (smem > 200 * 1024) return ERR_UNSUPPORTED;
    const int threads = width >= 2048 ? 512 : (width >= 512 ? 256 : 128);
    const int values = (width + threads - 1) / threads;
    // (longer rows would spill: they stay in shared memory.  So do many plain ones of five to seven values a thread: us in
    // shared memory and in registers, 2,048 rows of 2,304 14.6 and 15.9, of 3,072 16.4 and 17.6, of 1,536 8.2 and 8.4; of 2,048 values,
    // four a thread, 10.3 and 9.4, of 4,096 24.2 and 23.7; with the sum, which reads a row more, of 2,304 17.8 and 16.6; and of 8,192 rows
    // of 3,072, more than L2 holds, 83 and 71)
    const bool shared = !accumulate && values >= 5 && values <= 7 && many_rows(num_rows, threads) && (long long)num_rows * width < 16 << 20;
    if (!general && values <= 8 && !shared) {
#define FSIE_LN_REGS(S, T, PER)                                                                                               \
        launch_dependent_if(early, add_layernorm_regs_kernel<S, T, PER>, num_rows, threads, 0, stream, (const S*)src, rows, gain, \
                            accumulate ? x : nullptr, (T*)y, width, eps)
#define FSIE_LN_F32(PER) FSIE_LN_REGS(float, float, PER)
#define FSIE_LN_SUM(PER) FSIE_LN_REGS(bf16, bf16, PER)
#define FSIE_LN_BF16(PER) FSIE_LN_REGS(float, bf16, PER)
        if (dtype == DTYPE_F32) return FSIE_BY_VALUES(values, FSIE_LN_F32);
        return accumulate ? FSIE_BY_VALUES(values, FSIE_LN_SUM) : FSIE_BY_VALUES(values, FSIE_LN_BF16);
#undef FSIE_LN_F32
#undef FSIE_LN_SUM
#undef FSIE_LN_BF16
#undef FSIE_LN_REGS
    }
    int code = 0;
#define FSIE_LN(S, T)                                                                           \
    do {                                                                                        \
        if (smem > 48 * 1024)                                                                   \
            cudaFuncSetAttribute(add_layernorm_kernel<S, T>,                                    \
                                 cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);      \
        code = launch_dependent(add_layernorm_kernel<S, T>, num_rows, threads, smem, stream,    \
                                (const S*)src, rows, gain, accumulate ? x : nullptr, (T*)y,      \
                                width, eps);                                                     \
    } while (0)
    if (dtype == DTYPE_F32) {
        FSIE_LN(float, float);
    } else if (accumulate) {
        FSIE_LN(bf16, bf16);
    } else {
        FSIE_LN(float, bf16);
    }
#undef FSIE_LN
    return code;
}

int fsie_cast_rows(const float* x, void* y, long long count, int dtype, cudaStream_t stream) {
    if (count <= 0) return 0;
    const int threads = 256;
    const long long wanted = (count + threads - 1) / threads;
    const unsigned blocks = (unsigned)(wanted > 4096 ? 4096 : wanted);
    if (dtype == DTYPE_F32)
        return launch_dependent(cast_rows_kernel<float>, blocks, threads, 0, stream, x, (float*)y, count);
    return launch_dependent(cast_rows_kernel<bf16>, blocks, threads, 0, stream, x, (bf16*)y, count);
}

}  // extern "C"
