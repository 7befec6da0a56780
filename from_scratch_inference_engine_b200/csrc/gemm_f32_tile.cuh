// The tiled FFMA product of the float32 path: 128 x 128 outputs per block, k in steps of 16 through
// shared memory, each output one thread's sum over k in ascending order.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace fsie {

constexpr int TM = 128, TN = 128, TK = 16;      // block tile; 256 threads, 8 x 8 outputs each

// The 128 x 128 outputs from (m0, n0) on, by a block of 256 threads.  REPAIR: of those only the ones that y holds no
// finite number for.
template <bool REPAIR = false>
__device__ __forceinline__ void f32_tile(const float* __restrict__ x, const float* __restrict__ w,
                                         const float* __restrict__ bias, float* __restrict__ y,
                                         int M, int N, int K, int ldx, int ldy, int m0, int n0) {
    // k-major in shared memory, so that a thread's 8 rows (columns) are two 16-byte reads
    __shared__ __align__(16) float xs[2][TK][TM + 4];      // + 4: the four k of a thread's load fall into other banks
    __shared__ __align__(16) float ws[2][TK][TN + 4];
    const int tid = threadIdx.x;
    const int tx = tid & 15, ty = tid >> 4;           // tx -> columns (N), ty -> rows (M)
    // loads: 128 rows x 16 k per operand = 512 float4; thread t takes rows t / 4 and t / 4 + 64,
    // k offset (t % 4) * 4
    const int lrow = tid >> 2, lk = (tid & 3) * 4;
    float acc[8][8];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[i][j] = 0.f;

    float4 xr[2], wr[2];
    auto fetch = [&](int k0) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int m = m0 + lrow + h * 64, n = n0 + lrow + h * 64, k = k0 + lk;
            xr[h] = (m < M && k < K) ? *reinterpret_cast<const float4*>(x + (size_t)m * ldx + k)
                                     : make_float4(0.f, 0.f, 0.f, 0.f);
            wr[h] = (n < N && k < K) ? __ldg(reinterpret_cast<const float4*>(w + (size_t)n * K + k))
                                     : make_float4(0.f, 0.f, 0.f, 0.f);
        }
    };
    auto stash = [&](int buf) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int r = lrow + h * 64;
            xs[buf][lk + 0][r] = xr[h].x; xs[buf][lk + 1][r] = xr[h].y;
            xs[buf][lk + 2][r] = xr[h].z; xs[buf][lk + 3][r] = xr[h].w;
            ws[buf][lk + 0][r] = wr[h].x; ws[buf][lk + 1][r] = wr[h].y;
            ws[buf][lk + 2][r] = wr[h].z; ws[buf][lk + 3][r] = wr[h].w;
        }
    };
    fetch(0);
    stash(0);
    __syncthreads();
    int buf = 0;
    for (int k0 = 0; k0 < K; k0 += TK) {
        const bool more = k0 + TK < K;
        if (more) fetch(k0 + TK);                 // the next step's operands travel while this one computes
#pragma unroll
        for (int c = 0; c < TK; ++c) {
            // rows ty*4 .. +3 and 64 + ty*4 .. +3, columns tx*4 .. +3 and 64 + tx*4 .. +3:
            // consecutive threads read consecutive 16 bytes, no bank conflicts
            const float4 a0 = *reinterpret_cast<const float4*>(&xs[buf][c][ty * 4]);
            const float4 a1 = *reinterpret_cast<const float4*>(&xs[buf][c][64 + ty * 4]);
            const float4 b0 = *reinterpret_cast<const float4*>(&ws[buf][c][tx * 4]);
            const float4 b1 = *reinterpret_cast<const float4*>(&ws[buf][c][64 + tx * 4]);
            const float a[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
            const float b[8] = {b0.x, b0.y, b0.z, b0.w, b1.x, b1.y, b1.z, b1.w};
#pragma unroll
            for (int i = 0; i < 8; ++i)
#pragma unroll
                for (int j = 0; j < 8; ++j) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
        }
        if (more) {
            stash(buf ^ 1);
            __syncthreads();
            buf ^= 1;
        }
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int m = m0 + (i < 4 ? ty * 4 + i : 64 + ty * 4 + i - 4);
        if (m >= M) continue;
#pragma unroll
        for (int jh = 0; jh < 2; ++jh) {
            const int n = n0 + jh * 64 + tx * 4;
            float v[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) v[j] = acc[i][jh * 4 + j] + ((bias && n + j < N) ? bias[n + j] : 0.f);
            float* out = y + (size_t)m * ldy + n;
            if (REPAIR) {
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    if (n + j < N && !(fabsf(out[j]) <= 3.402823466e38f)) out[j] = v[j];
            } else if (n + 3 < N && (((size_t)out) & 15) == 0) {
                *reinterpret_cast<float4*>(out) = make_float4(v[0], v[1], v[2], v[3]);
            } else {
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    if (n + j < N) out[j] = v[j];
            }
        }
    }
}

}  // namespace fsie
