// Shared helpers of the sm_100a kernels: storage types, conversions, reductions.
#pragma once

#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace fsie {

typedef __nv_bfloat16 bf16;

__device__ __forceinline__ float to_float(float v) { return v; }
__device__ __forceinline__ float to_float(bf16 v) { return __bfloat162float(v); }

template <typename T> __device__ __forceinline__ T from_float(float v);
template <> __device__ __forceinline__ float from_float<float>(float v) { return v; }
template <> __device__ __forceinline__ bf16 from_float<bf16>(float v) { return __float2bfloat16_rn(v); }

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}

// Sum over the block in a fixed order (the same bits on every run); `scratch` holds 32 floats.
__device__ __forceinline__ float block_sum(float v, float* scratch) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int warps = (blockDim.x + 31) >> 5;
    v = warp_sum(v);
    __syncthreads();
    if (lane == 0) scratch[warp] = v;
    __syncthreads();
    float total = 0.f;
    for (int w = 0; w < warps; ++w) total += scratch[w];
    return total;
}

__device__ __forceinline__ float block_max(float v, float* scratch) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int warps = (blockDim.x + 31) >> 5;
    v = warp_max(v);
    __syncthreads();
    if (lane == 0) scratch[warp] = v;
    __syncthreads();
    float total = scratch[0];
    for (int w = 1; w < warps; ++w) total = fmaxf(total, scratch[w]);
    return total;
}

// ---- 8 consecutive elements at once (16 bytes of bf16, 32 bytes of float); p is aligned to that
__device__ __forceinline__ void load8(const float* p, float (&v)[8]) {
    const float4 a = *reinterpret_cast<const float4*>(p);
    const float4 b = *reinterpret_cast<const float4*>(p + 4);
    v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
}
__device__ __forceinline__ void load8(const bf16* p, float (&v)[8]) {
    const uint4 raw = *reinterpret_cast<const uint4*>(p);
    const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&raw);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const float2 f = __bfloat1622float2(h[i]);
        v[2 * i] = f.x; v[2 * i + 1] = f.y;
    }
}
__device__ __forceinline__ void store8(float* p, const float (&v)[8]) {
    *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
    *reinterpret_cast<float4*>(p + 4) = make_float4(v[4], v[5], v[6], v[7]);
}
__device__ __forceinline__ void store8(bf16* p, const float (&v)[8]) {
    uint4 raw;
    __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&raw);
#pragma unroll
    for (int i = 0; i < 4; ++i) h[i] = __floats2bfloat162_rn(v[2 * i], v[2 * i + 1]);
    *reinterpret_cast<uint4*>(p) = raw;
}

// dtype tags of the C entry points
enum { DTYPE_F32 = 0, DTYPE_BF16 = 1 };

// Return codes of the C entry points beyond cudaError_t values.
enum { ERR_BAD_ARGUMENT = -1, ERR_UNSUPPORTED = -2 };

// ---- programmatic dependent launch
// A kernel launched with launch_dependent() may be scheduled while the kernel before it in the
// stream is still running; it must call grid_dependency_wait() before it touches anything that
// kernel wrote (and before it writes anything that kernel may read).  A kernel that calls
// grid_dependents_go() lets the kernel after it be scheduled from that point on.  Both are
// no-ops for kernels launched the ordinary way.
//
// A kernel may read in front of its wait what is older than the kernel before it: what that kernel did not write, and what was
// complete when that kernel's own wait returned.  The second holds behind a kernel whose blocks all call grid_dependents_go()
// after their wait and leave after it, as all here do but one: attn_tc_decode_kernel (attention_tcgen05.cu) lets the next kernel
// go before it waits, so that one may still overlap the kernel in front of it.  Behind it only merges and products run, which
// read nothing early but weights and lists.
// Whether its operands are that old a kernel's caller knows: launch_dependent_if() with `early` = 0 launches the ordinary way.
__device__ __forceinline__ void grid_dependency_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void grid_dependents_go() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

template <typename... Params, typename... Args>
inline int launch_dependent_if(int early, void (*kernel)(Params...), dim3 grid, dim3 block, size_t smem,
                               cudaStream_t stream, Args... args) {
    cudaLaunchConfig_t config = {};
    config.gridDim = grid;
    config.blockDim = block;
    config.dynamicSmemBytes = smem;
    config.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    config.attrs = attr;
    config.numAttrs = early ? 1 : 0;
    return (int)cudaLaunchKernelEx(&config, kernel, static_cast<Params>(args)...);
}

template <typename... Params, typename... Args>
inline int launch_dependent(void (*kernel)(Params...), dim3 grid, dim3 block, size_t smem,
                            cudaStream_t stream, Args... args) {
    return launch_dependent_if(1, kernel, grid, block, smem, stream, args...);
}

// ---- rows of a norm in registers
// Blocks of a row each that are many: a third more threads than 148 SMs hold at once.  Beyond, rows in registers pay where the
// kernel stays small enough for as many of its blocks on an SM (the rules at each launch).
inline bool many_rows(long long blocks, int threads) { return blocks * threads > 400000; }

}  // namespace fsie

// CALL(n) for the number of values (1 to 8) that a thread of a row's block holds.  As many as there are and no more: 2,304
// values of 512 threads in registers for eight each took a prompt's 2,048 rows 8 to 31 % longer than rows in shared memory.
#define FSIE_BY_VALUES(values, CALL)                                                                          \
    ((values) == 1 ? CALL(1) : (values) == 2 ? CALL(2) : (values) == 3 ? CALL(3) : (values) == 4 ? CALL(4)    \
     : (values) == 5 ? CALL(5) : (values) == 6 ? CALL(6) : (values) == 7 ? CALL(7) : CALL(8))

#define FSIE_LAUNCH_CHECK() ((int)cudaGetLastError())
