// True 32-bit matrix products for the float32 path: y[M,N] = x[M,K] * w[N,K]^T (+ bias[N]).
// Plain FFMA on CUDA cores (the reference instead asks its library for strict fp32,
// src/cuda/device.cu:322-357); steps of many tokens take the product that splits its operands into three
// bfloat16 parts, exactly (gemm_f32_tcgen05.cu), unless k is short.  Three kernels:
//
//  * gemm_f32_rows_kernel - steps of few tokens (M <= 48, in tiles of up to 16 rows).  The
//    product is bound by reading w once from HBM, so a warp owns R rows of w and streams them
//    16 bytes per lane, its 32 lanes side by side along k; the step's rows of x wait in shared
//    memory and every x value read from there is used for R rows of w.  A lane's partial sums
//    run over k in ascending order and the 32 lanes are then added in a fixed tree, so an
//    output does not depend on how many other rows share the launch.
//  * gemm_f32_tiles_kernel - more rows than that, k below about 128: tiles of 128 x 128 outputs, k in steps of 16 through
//    shared memory, 8 x 8 outputs per thread in registers.  Each output is one thread's sum over
//    k in ascending order.
//  * gemm_f32_plain_kernel - any sizes and alignments (k no multiple of 4, unaligned rows).
//
// An output of the rows kernel and the same output of the tiles kernel differ in the order of
// their sums, that is by rounding; within one kernel a row's result does not depend on the batch.
#include "common.cuh"
#include "gemm_f32_tile.cuh"

namespace fsie {

// ------------------------------------------------------------------------- few rows
// 16 bytes from global to shared memory without passing through registers; src_bytes = 0 writes zeros.
__device__ __forceinline__ void copy16_async(void* dst, const void* src, int src_bytes) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(src_bytes) : "memory");
}
__device__ __forceinline__ void copies_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void copies_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// MT rows of x per block, R rows of w per warp.  A warp walks k in passes of 128 elements (16 bytes
// per lane and row of w).  What bounds the product is how many bytes of w are on their way, so every warp keeps
// DEPTH passes of its rows in a ring of its own in shared memory (cp.async; a lane reads back only the 16 bytes
// that it asked for itself, so no barrier guards the ring), and the ring runs on into the warp's next rows of
// w: one block per SM stays for all of the matrix that falls to it.
// The step's rows of x come through shared memory in chunks of XC elements, the next chunk copied while the
// current one is used: one barrier per chunk, none but the first where a row of x is one chunk.
// Launched as a programmatic dependent (where the caller knows that kernel not to write w): the first rows of w are
// asked for before the kernel that produces x has finished.
constexpr int ROWS_MAX_WARPS = 16;
template <int MT, int R> struct RowsShape {
    static constexpr int XC = MT >= 16 ? 512 : (MT >= 8 ? 1024 : 2048);
    static constexpr int PER_CHUNK = XC / 128;
    // 6 to 8 KB per warp, and not more passes than a chunk has, so that a chunk of x asked for at the start of the one before
    // it has landed when its first pass has: that leaves 4 KB of one row of w from 5 rows of x on, 2 from 9 on, and 4 of two rows from 9 on
    static constexpr int DEEP = R == 1 ? 12 : (R == 2 ? 8 : 4);
    static constexpr int DEPTH = DEEP < PER_CHUNK ? DEEP : PER_CHUNK;
    static constexpr int WARP_BYTES = DEPTH * R * 512;
};

template <int MT, int R>
__global__ void __launch_bounds__(ROWS_MAX_WARPS * 32, 1)
gemm_f32_rows_kernel(const float* __restrict__ x, const float* __restrict__ w,
                     const float* __restrict__ bias, float* __restrict__ y,
                     int M, int N, int K, int ldx, int ldy) {
    using S = RowsShape<MT, R>;
    constexpr int XC = S::XC, PER_CHUNK = S::PER_CHUNK, D = S::DEPTH;
    extern __shared__ __align__(16) float xs_raw[];                  // [1 or 2][MT][XC] of x, then the warps' rings
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, warps = blockDim.x >> 5;
    const int passes = (K + 127) / 128, chunks = (K + XC - 1) / XC;
    // the tiles of rows of x are the fast grid dimension: blocks that read the same rows of w
    // run side by side and share them through L2
    const int m0 = blockIdx.x * MT;
    const int block_rows = warps * R, step = gridDim.y * block_rows;
    const int rounds = ((N + block_rows - 1) / block_rows - (int)blockIdx.y + (int)gridDim.y - 1) / (int)gridDim.y;
    int n0 = (int)blockIdx.y * block_rows + warp * R;
    unsigned char* ring = reinterpret_cast<unsigned char*>(xs_raw + (size_t)(chunks > 1 ? 2 : 1) * MT * XC)
                          + (size_t)warp * S::WARP_BYTES + lane * 16;

    // the next pass of the warp's rows that nobody has asked for yet (rows from N on and elements from K on are zeros)
    int ask_n = n0, ask_pass = 0, ask_round = 0;
    const float* ask_w = w + (size_t)n0 * K + lane * 4;
    auto ask = [&](int slot) {
        if (ask_round < rounds) {
            const bool in_row = ask_pass * 128 + lane * 4 < K;
#pragma unroll
            for (int r = 0; r < R; ++r) {
                const bool valid = in_row && ask_n + r < N;
                copy16_async(ring + (slot * R + r) * 512, valid ? ask_w + (size_t)r * K + ask_pass * 128 : w, valid ? 16 : 0);
            }
            if (++ask_pass == passes) {
                ask_pass = 0; ++ask_round; ask_n += step;
                ask_w += (size_t)step * K;
            }
        }
        copies_commit();                  // one group per pass, also when empty
    };
#pragma unroll
    for (int d = 0; d < D; ++d) ask(d);     // w does not depend on the kernel before
    grid_dependency_wait();
    grid_dependents_go();

    // the first chunk of the step's rows of x (zeros beyond M and K), through registers; the later ones by cp.async
    for (int e = tid; e < MT * (XC / 4); e += blockDim.x) {
        const int m = e / (XC / 4), c = (e - m * (XC / 4)) * 4;
        if (c >= passes * 128) continue;                             // never read
        const bool valid = m0 + m < M && c < K;
        *reinterpret_cast<float4*>(xs_raw + m * XC + c) =
            valid ? *reinterpret_cast<const float4*>(x + (size_t)(m0 + m) * ldx + c) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    auto stage_x = [&](int chunk, int half) {
        float* to = xs_raw + (size_t)half * MT * XC;
        for (int e = tid; e < MT * (XC / 4); e += blockDim.x) {
            const int m = e / (XC / 4), c = (e - m * (XC / 4)) * 4, k = chunk * XC + c;
            const bool valid = m0 + m < M && k < K;
            copy16_async(to + m * XC + c, valid ? x + (size_t)(m0 + m) * ldx + k : x, valid ? 16 : 0);
        }
    };
    __syncthreads();

    int slot = 0, half = 0;
    for (int round = 0; round < rounds; ++round, n0 += step) {
        float acc[R][MT];
#pragma unroll
        for (int r = 0; r < R; ++r)
#pragma unroll
            for (int m = 0; m < MT; ++m) acc[r][m] = 0.f;
        for (int chunk = 0; chunk < chunks; ++chunk) {
            const int first = chunk * PER_CHUNK, last = min(passes, first + PER_CHUNK);
            if (chunks > 1) {
                if (round + chunk > 0) {
                    // this chunk's x was asked for in the group of the first pass of the chunk before it: as many
                    // passes ago as that chunk has, which is enough unless it was a short one at a row's end
                    if (chunk == 0 && passes - (chunks - 1) * PER_CHUNK < D) copies_wait<0>(); else copies_wait<D - 1>();
                    __syncthreads();      // it has landed for every thread, and the other half is no longer read
                    half ^= 1;
                }
                if (chunk + 1 < chunks) stage_x(chunk + 1, half ^ 1);
                else if (round + 1 < rounds) stage_x(0, half ^ 1);
            }
            const float* xrow = xs_raw + (size_t)half * MT * XC + lane * 4;
            for (int pass = first; pass < last; ++pass, xrow += 128) {
                copies_wait<D - 1>();     // the oldest group - this slot - has landed
                float4 wv[R];
#pragma unroll
                for (int r = 0; r < R; ++r) wv[r] = *reinterpret_cast<const float4*>(ring + (slot * R + r) * 512);
#pragma unroll
                for (int m = 0; m < MT; ++m) {
                    const float4 xv = *reinterpret_cast<const float4*>(xrow + m * XC);
#pragma unroll
                    for (int r = 0; r < R; ++r) {
                        float a = acc[r][m];
                        a = fmaf(xv.x, wv[r].x, a);
                        a = fmaf(xv.y, wv[r].y, a);
                        a = fmaf(xv.z, wv[r].z, a);
                        a = fmaf(xv.w, wv[r].w, a);
                        acc[r][m] = a;
                    }
                }
                ask(slot);                // refill what has just been used
                slot = slot + 1 == D ? 0 : slot + 1;
            }
        }
        // The 32 lanes' parts, added in the tree of lane distances 16, 8, 4, 2, 1.  An exchange hands over half of the
        // sums that a lane still holds (the other half goes to its partner), so lane l ends up with
        // the sums whose number has the bits of l: 16 exchanges for 16 sums instead of 80.
        constexpr int SUMS = R * MT;
        float part[SUMS];
#pragma unroll
        for (int r = 0; r < R; ++r)
#pragma unroll
            for (int m = 0; m < MT; ++m) part[r * MT + m] = acc[r][m];
        int held = SUMS, mine = 0;         // this lane holds sums mine .. mine + held - 1 of the SUMS
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            if (held > 1) {
                held >>= 1;
                const bool upper = lane & o;
#pragma unroll
                for (int i = 0; i < SUMS / 2; ++i) {
                    if (i < held) {
                        const float give = upper ? part[i] : part[i + held];
                        const float keep = upper ? part[i + held] : part[i];
                        part[i] = keep + __shfl_xor_sync(0xffffffffu, give, o);
                    }
                }
                mine += upper ? held : 0;
            } else {
                part[0] += __shfl_xor_sync(0xffffffffu, part[0], o);
            }
        }
        // lanes that differ only in distances below the last halving hold the same sums: one of them stores
        constexpr int REPEATED = SUMS >= 32 ? 1 : 32 / SUMS;
        if ((lane & (REPEATED - 1)) == 0) {
#pragma unroll
            for (int i = 0; i < (SUMS >= 32 ? SUMS / 32 : 1); ++i) {
                const int r = (mine + i) / MT, m = (mine + i) % MT;
                if (n0 + r < N && m0 + m < M)
                    y[(size_t)(m0 + m) * ldy + n0 + r] = part[i] + (bias ? bias[n0 + r] : 0.f);
            }
        }
    }
}

template <int MT, int R> static size_t rows_smem(int warps, int K) {
    using S = RowsShape<MT, R>;
    return sizeof(float) * (K > S::XC ? 2 : 1) * MT * S::XC + (size_t)warps * S::WARP_BYTES;
}

template <int MT, int R>
static int launch_rows_as(const float* x, const float* w, const float* bias, float* y, int M, int N,
                          int K, int ldx, int ldy, int m_tiles, int sms, int warps, int early, cudaStream_t stream) {
    static bool raised = false;          // per instantiation: the limit of dynamic shared memory
    if (!raised) {
        const cudaError_t e = cudaFuncSetAttribute(gemm_f32_rows_kernel<MT, R>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                   (int)rows_smem<MT, R>(ROWS_MAX_WARPS, 1 << 30));
        if (e != cudaSuccess) return (int)e;
        raised = true;
    }
    const int blocks = (N + warps * R - 1) / (warps * R), most = sms / m_tiles > 0 ? sms / m_tiles : 1;
    return launch_dependent_if(early, gemm_f32_rows_kernel<MT, R>, dim3(m_tiles, blocks < most ? blocks : most), dim3(warps * 32),
                            rows_smem<MT, R>(warps, K), stream, x, w, bias, y, M, N, K, ldx, ldy);
}

// How long the SM with most rows of w is busy, in clocks per pass: what is least decides the rows per warp and
// the warps per block.  Of a pass of one row (512 bytes) an SM takes in 27 bytes a clock; shared memory moves 128
// bytes a clock, the row in and out and MT rows of x for R rows of w; an instruction per clock and scheduler
// gives 4 MT products for 32 lanes.  Fewer than 48 KB on their way leave the SM waiting.  A block that stays for many
// rounds has 12 or 16 warps: the last round's idle warps are few against what an uneven share of the four schedulers and
// fewer warps to switch between cost (8 rows, 151,936 x 1,536: 6 warps 223 us, 12 171; 2 rows: 13 warps 147 to 167, 12 135).
template <int MT, int R>
static float rows_cost(int N, int sms, int m_tiles, int& warps) {
    using S = RowsShape<MT, R>;
    const int most = sms / m_tiles > 0 ? sms / m_tiles : 1;
    const float shared = 4.f * (2.f + (float)MT / R), issue = 0.3f * (4.f * MT + (float)MT / R + 8.f);
    const float clocks = fmaxf(19.f, fmaxf(shared, issue));
    float best = 1e30f;
    for (int count = ROWS_MAX_WARPS; count >= 4; --count) {
        const int blocks = (N + count * R - 1) / (count * R), grid = blocks < most ? blocks : most;
        const int rounds = (blocks + grid - 1) / grid;
        if (rounds > 4 && count != 12 && count != 16) continue;       // (see above)
        const float wait = fmaxf(1.f, 48.f * 1024.f / ((float)count * S::WARP_BYTES));
        const float cost = (float)rounds * count * R * clocks * wait;
        if (cost < best) { best = cost; warps = count; }
    }
    return best;
}

template <int MT>
static int launch_rows(const float* x, const float* w, const float* bias, float* y, int M, int N,
                       int K, int ldx, int ldy, int sms, int rows_per_warp, int early, cudaStream_t stream) {
    const int m_tiles = (M + MT - 1) / MT;
    int w1 = 1, w2 = 1, w4 = 1;
    const float c1 = rows_cost<MT, 1>(N, sms, m_tiles, w1), c2 = rows_cost<MT, 2>(N, sms, m_tiles, w2),
                c4 = rows_cost<MT, 4>(N, sms, m_tiles, w4);
    int r = c4 <= c2 && c4 <= c1 ? 4 : (c2 <= c1 ? 2 : 1);
    // where not even every SM has four rows of w, a warp's own chain from pass to pass is what takes the time, and it is
    // shorter for one row than for two (8 rows of x, 256 x 1,536: 6.6 us with two, 5.8; 512 x 4,096 11.7 and 10.7; a row of one
    // chunk is over before that shows: 256 x 256 2.6 and 3.5)
    if (MT == 8 && N <= 4 * sms && K > RowsShape<MT, 1>::XC) { r = 1; w1 = 8; }
    if (rows_per_warp == 1 || rows_per_warp == 2 || rows_per_warp == 4) r = rows_per_warp;
    if (r == 4) return launch_rows_as<MT, 4>(x, w, bias, y, M, N, K, ldx, ldy, m_tiles, sms, w4, early, stream);
    if (r == 2) return launch_rows_as<MT, 2>(x, w, bias, y, M, N, K, ldx, ldy, m_tiles, sms, w2, early, stream);
    return launch_rows_as<MT, 1>(x, w, bias, y, M, N, K, ldx, ldy, m_tiles, sms, w1, early, stream);
}

// ---------------------------------------------------------------------------- tiles
__global__ void __launch_bounds__(256, 2)
gemm_f32_tiles_kernel(const float* __restrict__ x, const float* __restrict__ w,
                      const float* __restrict__ bias, float* __restrict__ y,
                      int M, int N, int K, int ldx, int ldy) {
    f32_tile(x, w, bias, y, M, N, K, ldx, ldy, blockIdx.y * TM, blockIdx.x * TN);
}

// ---------------------------------------------------------------------------- plain
constexpr int GM = 64, GN = 64, GK = 16;   // block tile; 256 threads, 4x4 outputs each

__global__ void __launch_bounds__(256)
gemm_f32_plain_kernel(const float* __restrict__ x, const float* __restrict__ w,
                      const float* __restrict__ bias, float* __restrict__ y,
                      int M, int N, int K, int ldx, int ldy) {
    __shared__ float xs[GK][GM + 4];
    __shared__ float ws[GK][GN + 4];
    const int tid = threadIdx.x;
    const int tx = tid & 15, ty = tid >> 4;           // tx -> columns (N), ty -> rows (M)
    const int m0 = blockIdx.y * GM, n0 = blockIdx.x * GN;
    float acc[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;

    for (int k0 = 0; k0 < K; k0 += GK) {
        // 64x16 elements per operand, 256 threads -> 4 each; consecutive threads walk k
        for (int e = tid; e < GM * GK; e += 256) {
            const int r = e / GK, c = e - r * GK;
            const int m = m0 + r, n = n0 + r, k = k0 + c;
            xs[c][r] = (m < M && k < K) ? x[(size_t)m * ldx + k] : 0.f;
            ws[c][r] = (n < N && k < K) ? w[(size_t)n * K + k] : 0.f;
        }
        __syncthreads();
#pragma unroll
        for (int c = 0; c < GK; ++c) {
            float a[4], b[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) a[i] = xs[c][ty * 4 + i];
#pragma unroll
            for (int j = 0; j < 4; ++j) b[j] = ws[c][tx * 4 + j];
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int m = m0 + ty * 4 + i;
        if (m >= M) continue;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int n = n0 + tx * 4 + j;
            if (n < N) y[(size_t)m * ldy + n] = acc[i][j] + (bias ? bias[n] : 0.f);
        }
    }
}

}  // namespace fsie

// Rows of a step that still take the few-rows kernel (in tiles of 16).  Measured on the
// 37,888 x 3,584 matrix: 32 rows 0.46 ms against 0.79 ms for the tiles kernel, 64 rows 0.88
// against 0.79 - the tiles kernel's time does not depend on the rows below 128.
extern "C" int fsie_gemm_f32_rows_limit() { return 48; }

// kind: 0 = choose by size and alignment, 1 = few-rows kernel, 2 = tiles kernel, 3 = plain kernel
// (the tests ask for each by name; a kind that cannot take the operands is refused).
// rows_per_warp: 0 = chosen by size; 1, 2 or 4 fix it for the few-rows kernel (tests, measurements).
extern "C" int fsie_gemm_f32(const float* x, const float* w, const float* bias, float* y, int M,
                             int N, int K, int ldx, int ldy, int kind, int rows_per_warp,
                             int early, cudaStream_t stream) {
    using namespace fsie;
    if (M <= 0 || N <= 0) return 0;
    if (K <= 0 || kind < 0 || kind > 3) return ERR_BAD_ARGUMENT;
    // 16-byte loads need k in steps of 4 and rows that start on 16 bytes
    const bool aligned = (K % 4 == 0) && (ldx % 4 == 0) && ((((size_t)x) | ((size_t)w)) & 15) == 0;
    if ((kind == 1 || kind == 2) && !aligned) return ERR_UNSUPPORTED;
    if (kind == 1 && M > fsie_gemm_f32_rows_limit()) return ERR_UNSUPPORTED;
    if (kind == 0) kind = !aligned ? 3 : (M <= fsie_gemm_f32_rows_limit() ? 1 : 2);
    if (kind == 3) {
        dim3 grid((N + GN - 1) / GN, (M + GM - 1) / GM);
        gemm_f32_plain_kernel<<<grid, 256, 0, stream>>>(x, w, bias, y, M, N, K, ldx, ldy);
        return FSIE_LAUNCH_CHECK();
    }
    if (kind == 2) {
        dim3 grid((N + TN - 1) / TN, (M + TM - 1) / TM);
        gemm_f32_tiles_kernel<<<grid, 256, 0, stream>>>(x, w, bias, y, M, N, K, ldx, ldy);
        return FSIE_LAUNCH_CHECK();
    }
    int device = 0, sms = 148;
    if (cudaGetDevice(&device) == cudaSuccess)
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
    if (M == 1) return launch_rows<1>(x, w, bias, y, M, N, K, ldx, ldy, sms, rows_per_warp, early, stream);
    if (M == 2) return launch_rows<2>(x, w, bias, y, M, N, K, ldx, ldy, sms, rows_per_warp, early, stream);
    if (M <= 4) return launch_rows<4>(x, w, bias, y, M, N, K, ldx, ldy, sms, rows_per_warp, early, stream);
    if (M <= 8) return launch_rows<8>(x, w, bias, y, M, N, K, ldx, ldy, sms, rows_per_warp, early, stream);
    return launch_rows<16>(x, w, bias, y, M, N, K, ldx, ldy, sms, rows_per_warp, early, stream);
}
