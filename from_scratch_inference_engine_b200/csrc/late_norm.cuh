// RMS norm without a launch of its own, for steps of few tokens: the product before it leaves what is needed, the product
// behind it does the rest.
//
//   v = x + product (rounded to bfloat16)        the residual stream, 32-bit, written back
//   z = bfloat16(v * gain)                       what the next product multiplies
//   parts[t][n / 16] = sum of v^2 over 16 neighbouring columns
//   next product, on its sums: z w^T / sqrt(sum of parts[t] / width + eps)
//
// The norm's factor is one number per row, so it may follow the product: z is rounded to bfloat16 with the same relative
// error as the normed row would be.  The parts are added in a fixed order.
#pragma once

#include "common.cuh"

namespace fsie {

constexpr int LATE_COLS = 16;          // columns of one part

// What a product reads beside z (parts == nullptr: nothing).
struct LateNorm {
    const float* parts; int count; int width; float eps;     // parts [tokens][count]
};
// Where a product leaves its result (x == nullptr: in y).
struct LateResidual {
    float* x; long long ldx; const void* gain; int gain_f32; bf16* z; long long ldz; float* parts; int count;
};

// A token's factor from its parts, by one warp (all lanes get it); lane l reads parts l, l + 32, ...
__device__ __forceinline__ float late_factor(const float* parts, const LateNorm& n, int lane) {
    float sum = 0.f;
    for (int i = lane; i < n.count; i += 32) sum += parts[i];
    return 1.0f / sqrtf(warp_sum(sum) / (float)n.width + n.eps);
}

// What the residual stream holds at column n of token t, and the gain there: asked for before the sums are done.
__device__ __forceinline__ void late_fetch(const LateResidual& r, int t, int n, bool in, float& old, float& gain) {
    old = gain = 0.f;
    if (in) {
        old = r.x[(size_t)t * r.ldx + n];
        gain = r.gain_f32 ? reinterpret_cast<const float*>(r.gain)[n] : __bfloat162float(reinterpret_cast<const bf16*>(r.gain)[n]);
    }
}

// One output, column n of token t, into the residual stream; the 16 lanes with the columns of one part call it together (in
// whole warps), `in` false where there is no such output.
__device__ __forceinline__ void late_store(const LateResidual& r, float out, float old, float gain, int t, int n, bool in, int lane) {
    const float v = in ? old + __bfloat162float(__float2bfloat16_rn(out)) : 0.f;
    if (in) {
        r.x[(size_t)t * r.ldx + n] = v;
        r.z[(size_t)t * r.ldz + n] = __float2bfloat16_rn(v * gain);
    }
    float sq = v * v;
#pragma unroll
    for (int o = LATE_COLS / 2; o > 0; o >>= 1) sq += __shfl_xor_sync(0xffffffffu, sq, o);
    if (in && (lane & (LATE_COLS - 1)) == 0) r.parts[(size_t)t * r.count + n / LATE_COLS] = sq;
}

}  // namespace fsie
