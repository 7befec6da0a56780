// 32-bit matrix products for steps of many tokens on the 5th-generation tensor cores, without giving
// up precision: y[M, N] = x[M, K] * w[N, K]^T (+ bias[N]), everything float32.
//
// A float32 number times 2^40 is exactly the sum of three bfloat16 numbers (8 bits of the significand each, rounded
// to nearest, what is left goes to the next): x = x0 + x1 + x2, w = w0 + w1 + w2.  Without the factor the third
// part of a number below 2^-109 would fall under bfloat16's smallest step; with it the last bit of the smallest
// float32 number is 2^-109, and numbers from 2^88 and sums from 2^48 on, which overflow, go the way of infinities (below).
// Sums are multiplied by 2^-80 when their tile is complete.  Products of bfloat16 numbers are exact in the tensor cores, so
//     x w = x0 w0 + (x0 w1 + x1 w0) + (x1 w1 + x0 w2 + x2 w0) + ...
// and what the six products leave out is below 2^-24 of |x w|.  The tensor cores round their running sums
// towards zero at every step, which over a long k would cost more than float32 does: the accumulator is
// therefore read back and added up in registers (rounding to nearest) after every 64 k-elements, and
// within those the small products come first.  Errors against 64-bit products (2-norm, normal inputs, here /
// in the FFMA kernel): k = 64 7.8e-8 / 1.5e-7, 1,536 1.2e-7 / 7.0e-7, 8,960 2.3e-7 / 1.7e-6, 18,944 3.2e-7 / 2.5e-6.
//
// What bounds it: six tensor-core products, so at best a sixth of the bfloat16 rate (1,396 TFLOP/s
// sustained: 233), where FFMA gives 74.  Measured, us (TFLOP/s) here and in the tiled FFMA kernel: 1,668 rows of
// 17,920 x 1,536 376 (244) and 2,258 (41); of 1,536 x 8,960 304 and 1,856 (42 tiles for 74 pairs); 512 rows of
// 37,888 x 3,584 514 (270) and 3,379.  Where all numbers of w in a stage are bfloat16 numbers (a checkpoint stored
// as such), the second and third part of w are zero and the three products with them are left out: 295 to 310 us
// instead of 362 to 386; every stage finds that out for itself.
//
// x is split by a kernel of its own into three planes (it is small and every tile of columns reads it); w,
// which would be 1.5 times itself as planes, is split on its way into shared memory.  Two blocks (a
// cluster of two) share a 256 x 256 tile as in the bfloat16 product: per 64 k-elements a block gets the
// planes of its 128 rows of x by TMA; eight warps take 16 of its rows of w each (float32, by TMA, asked for as
// soon as the rows before them are in registers: loads straight into registers took 440 us instead of 376,
// since beside 128 sums a thread's rows in flight were spilled and waited for), write their planes
// into the 128-byte swizzle and add up the previous stage's accumulator (2 x 256 columns of tensor memory,
// one per stage).  One barrier per stage says "filled, and its accumulator is free", one says "multiplied".
// While the warps store a finished tile the tensor cores have the next tile's first stage to work on.
//
// One thread of the first block issues the products, which read planes that warps of both blocks wrote with
// ordinary stores.  Every lane fences its stores for the tensor cores, and a warp's arrival at the issuer's barrier
// releases them at cluster scope, which the issuer acquires.  Both fences are restricted to shared memory and
// cost nothing that could be measured; general releases at cluster scope took 1,000 cycles a stage, and
// a single one per block and stage by a warp of its own 420 us instead of 380 (1,668 rows of 17,920 x 1,536).
//
// A sum with an infinite or NaN input, or one that overflows, would come out as NaN where FFMA gives an
// infinity (0 * inf among the planes): tiles with such a result are noted, and a launch of one block per SM behind this
// one, which finds nothing to do otherwise, computes them by FFMA and replaces the results that are not finite.
//
// An output does not depend on the other rows of the launch: which of the two kernels it comes from is decided by
// itself.  Every wait on an mbarrier is bounded.
#include "common.cuh"
#include "gemm_f32_tile.cuh"
#include "tcgen05_pair.cuh"
#include "tma.cuh"

namespace fsie {

constexpr int F3_HALF = 128, F3_TILE = 256;          // rows of a block, of the pair's tile
constexpr int F3_K = 64;                             // k-elements per stage: 128 bytes of a plane, one swizzle row
constexpr int F3_STAGES = 2;
constexpr uint32_t F3_BOX = F3_HALF * F3_K * 2;      // one plane of 128 rows: 16 KB
constexpr uint32_t F3_STAGE = 6 * F3_BOX;            // planes of x, planes of w
constexpr int F3_WORKERS = 8;                        // warps
constexpr int F3_THREADS = 128 + 32 * F3_WORKERS;    // and a warp for the planes of x, one for the MMAs, two that keep the warpgroup whole
constexpr uint32_t F3_OUT_BOX = 32 * 128;            // a warp's 4 KB: 16 rows of w (64 k-elements), or 32 rows x 32 outputs on their way out
constexpr uint32_t F3_SMEM = 1024 + F3_STAGES * F3_STAGE + F3_WORKERS * F3_OUT_BOX;
constexpr uint32_t F3_TMEM = 512;                    // an accumulator of 256 columns per stage
constexpr float F3_UP = 0x1p40f, F3_DOWN = 0x1p-80f; // of the operands, of their products
constexpr int F3_RASTER = 8;                         // tiles of rows that run side by side (they share w in L2)

enum { ERR_F3_TMA_WAIT = 41, ERR_F3_MMA_WAIT = 42, ERR_F3_WORKER_WAIT = 43 };

struct SplitGemmParams {
    const float* bias; float* y;
    long long ldy;
    int M, N, K, m_tiles, n_tiles;
    int tma_store;
    int* odd;                       // [tiles]: set for a tile with a result that is not finite
    int* error;
};

// tile -> (row tile, column tile): bands of F3_RASTER row tiles, inside a band the rows run fastest
__device__ __forceinline__ void f3_place(int tile, int m_tiles, int n_tiles, int& m, int& n) {
    const int band = tile / (F3_RASTER * n_tiles), first = band * F3_RASTER;
    const int height = min(F3_RASTER, m_tiles - first), in_band = tile - band * F3_RASTER * n_tiles;
    m = first + in_band % height;
    n = in_band / height;
}

// four floats as they are split: exact, and so are the three parts then
__device__ __forceinline__ void scale_up(float4& v) { v.x *= F3_UP; v.y *= F3_UP; v.z *= F3_UP; v.w *= F3_UP; }

// the three bfloat16 parts of four floats, as 8 bytes per plane
__device__ __forceinline__ void split3(const float4& v, uint2 (&plane)[3]) {
    float a[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int p = 0; p < 3; ++p) {
        const __nv_bfloat162 lo = __floats2bfloat162_rn(a[0], a[1]), hi = __floats2bfloat162_rn(a[2], a[3]);
        plane[p].x = *reinterpret_cast<const uint32_t*>(&lo);
        plane[p].y = *reinterpret_cast<const uint32_t*>(&hi);
        a[0] -= __uint_as_float(plane[p].x << 16);
        a[1] -= __uint_as_float(plane[p].x & 0xffff0000u);
        a[2] -= __uint_as_float(plane[p].y << 16);
        a[3] -= __uint_as_float(plane[p].y & 0xffff0000u);
    }
}

// planes[p][m][0 .. K) = part p of x[m] * F3_UP; also clears the notes of the tiles to come
__global__ void __launch_bounds__(256)
gemm_f32_split_rows_kernel(const float* __restrict__ x, long long ldx, bf16* __restrict__ planes, int M, int K,
                           int plane_ld, int* __restrict__ odd, int tiles) {
    grid_dependency_wait();
    grid_dependents_go();
    const long long quads = (long long)M * (K / 4), step = (long long)gridDim.x * blockDim.x;
    const long long first = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    for (long long t = first; t < tiles; t += step) odd[t] = 0;
    for (long long q = first; q < quads; q += step) {
        const int m = (int)(q / (K / 4)), k = (int)(q - (long long)m * (K / 4)) * 4;
        uint2 plane[3];
        float4 v = *reinterpret_cast<const float4*>(x + m * ldx + k);
        scale_up(v);
        split3(v, plane);
#pragma unroll
        for (int p = 0; p < 3; ++p)
            *reinterpret_cast<uint2*>(planes + ((size_t)p * M + m) * plane_ld + k) = plane[p];
    }
}

__device__ __forceinline__ void tma_load_3d_pair(void* dst, const CUtensorMap* map, int c0, int c1, int c2, uint64_t* bar) {
    asm volatile("cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];"
                 ::"r"(smem_addr(dst)), "l"(map), "r"(c0), "r"(c1), "r"(c2), "r"(smem_addr(bar) & FIRST_BLOCK_MASK) : "memory");
}
// Four bytes into the first block's shared memory, counted by a barrier there.
__device__ __forceinline__ void store_first_block_async(int* p, int v, uint64_t* bar) {
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.u32 [%0], %1, [%2];"
                 ::"r"(smem_addr(p) & FIRST_BLOCK_MASK), "r"(v), "r"(smem_addr(bar) & FIRST_BLOCK_MASK) : "memory");
}

__global__ void __launch_bounds__(F3_THREADS, 1)
gemm_f32_split_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x,
                      const __grid_constant__ CUtensorMap map_y, const SplitGemmParams p) {
    extern __shared__ unsigned char smem_raw[];
    unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    __shared__ uint64_t full_bar[F3_STAGES], done_bar[F3_STAGES], raw_bar[F3_WORKERS];
    __shared__ uint32_t tmem_base_slot;
    __shared__ int abort_flag;
    // first block, one per worker of the pair: some number of w in its rows of the stage has more than one part
    __shared__ __align__(16) int fine[F3_STAGES][2 * F3_WORKERS];

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int rank = (int)cluster_rank();
    const int pair = blockIdx.x >> 1, pairs = gridDim.x >> 1;
    const int kblocks = (p.K + F3_K - 1) / F3_K, tiles = p.m_tiles * p.n_tiles;
    const int items = pair < tiles ? (tiles - pair + pairs - 1) / pairs : 0;
    const int total = items * kblocks;               // stages this pair goes through (the host bounds it)

    if (threadIdx.x == 0) {
        for (int s = 0; s < F3_STAGES; ++s) {
            mbar_init(&full_bar[s], 1 + 2 * F3_WORKERS);      // the copies of x, and the workers of both blocks
            mbar_init(&done_bar[s], 1);
        }
        for (int w = 0; w < F3_WORKERS; ++w) mbar_init(&raw_bar[w], 1);
        abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(&tmem_base_slot)), "r"(F3_TMEM) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    cluster_sync_all();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = tmem_base_slot;
    grid_dependency_wait();
    grid_dependents_go();

    // a worker's sums and rows of w fill 224 registers: 256 x 224 + 128 x 40 <= the 384 x 168 of the launch
    if (warp >= 4) {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 224;");
        // ------------------------------------------------------------ w into planes, sums into registers, results out
        const int worker = warp - 4;
        // as loader: 16 rows of w, the warp's own 4 KB (by TMA, one stage ahead); a lane splits 8 k-elements
        // of rows r, r + 4, r + 8, r + 12.  Half of the lanes read their second 16 bytes first: no bank
        // is asked for twice.
        const int r = lane >> 3, c8 = lane & 7, swap = (lane >> 2) & 1;
        const uint32_t place = 3 * F3_BOX + (worker * 16 + r) * 128 + ((c8 ^ r) << 4);
        unsigned char* raw = smem + F3_STAGES * F3_STAGE + worker * F3_OUT_BOX;
        // as reader: rows of a quarter of the tensor-memory lanes, half of the columns
        const int quarter = warp & 3, half = worker >> 2;
        const bool vector_ok = (p.ldy & 3) == 0 && (reinterpret_cast<uintptr_t>(p.y) & 15) == 0;

        int load_item = 0, load_kb = 0, load_n = 0, loads = 0;
        bool ok = true;
        auto load = [&]() {                          // by lane 0: the next stage's rows of w (zeros beyond N and K)
            if (load_kb == 0) {
                int mt, nt;
                f3_place(pair + load_item * pairs, p.m_tiles, p.n_tiles, mt, nt);
                load_n = nt * F3_TILE + rank * F3_HALF + worker * 16;
            }
            mbar_expect_tx(&raw_bar[worker], F3_OUT_BOX);
            tma_load_2d(raw, &map_w, load_kb * F3_K, load_n, &raw_bar[worker]);
            ++loads;
            if (++load_kb == kblocks) { load_kb = 0; ++load_item; }
        };
        float sum[128];
#pragma unroll
        for (int j = 0; j < 128; ++j) sum[j] = 0.f;
        int sum_kb = 0, sum_item = 0;
        if (total > 0 && lane == 0) load();
        for (int it = 0; it < total + F3_STAGES; ++it) {
            const int s = it & 1;
            // (a warp goes on or gives up as one: the votes and shared reads below wait for all of its lanes)
            if (it >= F3_STAGES) {
                // ---- stage it - 2 has been multiplied: add its accumulator up
                if (__any_sync(0xffffffffu, *(volatile int*)&abort_flag)) { ok = false; break; }
                if (!__all_sync(0xffffffffu, mbar_wait(&done_bar[s], ((it >> 1) - 1) & 1))) {
                    atomicExch(p.error, ERR_F3_WORKER_WAIT); atomicExch(&abort_flag, 1); ok = false; break;
                }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t from_tmem = tmem + ((uint32_t)(quarter * 32) << 16) + s * F3_TILE + half * F3_HALF;
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    float v[32];
                    tmem_load_32(from_tmem + q * 32, v);
                    tmem_load_wait();
#pragma unroll
                    for (int j = 0; j < 32; ++j) sum[q * 32 + j] += v[j];
                }
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            }
            if (it < total) {
                if (!__all_sync(0xffffffffu, mbar_wait(&raw_bar[worker], it & 1))) {
                    atomicExch(p.error, ERR_F3_WORKER_WAIT); atomicExch(&abort_flag, 1); ok = false; break;
                }
                unsigned char* to = smem + s * F3_STAGE;
                float4 f[4][2];
                uint32_t bits = 0;
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const float4* from = reinterpret_cast<const float4*>(raw + (r + 4 * i) * 256 + c8 * 32);
                    f[i][0] = from[swap];
                    f[i][1] = from[1 - swap];
                }
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    float4& v = f[i >> 1][i & 1];
                    scale_up(v);
                    bits |= __float_as_uint(v.x) | __float_as_uint(v.y) | __float_as_uint(v.z) | __float_as_uint(v.w);
                }
                // A number whose lower half is zero is a bfloat16 number.  The vote needs every lane's numbers, so
                // behind it all of them have arrived in registers and the copy may overwrite them.
                const bool more = __any_sync(0xffffffffu, (bits & 0xffffu) != 0);
                // the rows after these, unless a finished tile is stored from there first
                if (lane == 0 && it + 1 < total && !(it >= F3_STAGES && sum_kb + 1 == kblocks)) load();
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    uint2 a[3], b[3];
                    split3(swap ? f[i][1] : f[i][0], a);
                    split3(swap ? f[i][0] : f[i][1], b);
#pragma unroll
                    for (int q = 0; q < 3; ++q)      // (row & 7 is r or r + 4)
                        *reinterpret_cast<uint4*>(to + q * F3_BOX + ((place + i * 512) ^ ((i & 1) << 6))) =
                            make_uint4(a[q].x, a[q].y, b[q].x, b[q].y);
                }
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                __syncwarp();
                if (lane == 0) {
                    store_first_block_async(&fine[s][rank * F3_WORKERS + worker], more, &full_bar[s]);
                    mbar_release_first_block(&full_bar[s]);
                }
            }
            if (it >= F3_STAGES && ++sum_kb == kblocks) {
                // ---- the tile is complete (the tensor cores are at the next one's first stages)
                const int tile = pair + sum_item * pairs;
                int mt, nt;
                f3_place(tile, p.m_tiles, p.n_tiles, mt, nt);
                const int row0 = mt * F3_TILE + rank * F3_HALF + quarter * 32;
                bool finite = true;
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const int n = nt * F3_TILE + half * F3_HALF + q * 32;
                    if (n < p.N) {
                        float* v = sum + q * 32;
#pragma unroll
                        for (int j = 0; j < 32; ++j) v[j] *= F3_DOWN;
                        if (p.bias) {
#pragma unroll
                            for (int j = 0; j < 32; ++j) if (n + j < p.N) v[j] += p.bias[n + j];
                        }
#pragma unroll
                        for (int j = 0; j < 32; ++j) finite = finite && fabsf(v[j]) <= 3.402823466e38f;
                        if (p.tma_store) {
                            if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
                            __syncwarp();
#pragma unroll
                            for (int j = 0; j < 8; ++j)
                                *reinterpret_cast<float4*>(raw + lane * 128 + ((j ^ (lane & 7)) << 4)) =
                                    make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
                            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                            __syncwarp();
                            if (lane == 0) {         // rows beyond M and columns beyond N are clipped by the copy engine
                                asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%2, %3}], [%1];"
                                             ::"l"(&map_y), "r"(smem_addr(raw)), "r"(n), "r"(row0) : "memory");
                                asm volatile("cp.async.bulk.commit_group;" ::: "memory");
                            }
                        } else if (row0 + lane < p.M) {
                            float* dst = p.y + (size_t)(row0 + lane) * p.ldy + n;
                            if (vector_ok && n + 32 <= p.N) {
#pragma unroll
                                for (int j = 0; j < 32; j += 4)
                                    *reinterpret_cast<float4*>(dst + j) = make_float4(v[j], v[j + 1], v[j + 2], v[j + 3]);
                            } else {
#pragma unroll
                                for (int j = 0; j < 32; ++j) if (n + j < p.N) dst[j] = v[j];
                            }
                        }
                    }
                }
                if (lane == 0 && it + 1 < total) {   // the warp's 4 KB are free for rows of w again
                    asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
                    load();
                }
                if (!finite) p.odd[tile] = 1;
#pragma unroll
                for (int j = 0; j < 128; ++j) sum[j] = 0.f;
                sum_kb = 0;
                ++sum_item;
            }
        }
        if (!ok && loads > 0) mbar_wait(&raw_bar[worker], (loads - 1) & 1);      // giving up: the last copy lands first
        if (lane == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
    } else {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 40;");
        if (warp == 0 && lane == 0) {
            // ------------------------------------------------------------ the planes of x (both blocks)
            int it = 0, issued = 0;
            bool ok = true;
            for (int item = 0; ok && item < items; ++item) {
                int mt, nt;
                f3_place(pair + item * pairs, p.m_tiles, p.n_tiles, mt, nt);
                const int m0 = mt * F3_TILE + rank * F3_HALF;
                for (int kb = 0; kb < kblocks; ++kb, ++it) {
                    const int s = it & 1;
                    if (it >= F3_STAGES && !mbar_wait(&done_bar[s], ((it >> 1) - 1) & 1)) {
                        atomicExch(p.error, ERR_F3_TMA_WAIT); atomicExch(&abort_flag, 1);
                    }
                    if (*(volatile int*)&abort_flag) { ok = false; break; }
                    // both blocks' boxes and their workers' notes
                    if (rank == 0) mbar_expect_tx(&full_bar[s], 2 * 3 * F3_BOX + (uint32_t)sizeof(fine[s]));
#pragma unroll
                    for (int plane = 0; plane < 3; ++plane)
                        tma_load_3d_pair(smem + s * F3_STAGE + plane * F3_BOX, &map_x, kb * F3_K, m0, plane, &full_bar[s]);
                    issued = it + 1;
                }
            }
            if (!ok) {      // giving up: let the copies already issued land before the block's memory is released
                if (rank == 0) {
                    for (int j = max(0, issued - F3_STAGES); j < issued; ++j) mbar_wait(&full_bar[j & 1], (j >> 1) & 1);
                } else {
                    for (int i = 0; i < 1000; ++i) __nanosleep(1000);
                }
            }
        } else if (warp == 1 && lane == 0 && rank == 0) {
            // ------------------------------------------------------------ MMA issuer (first block)
            const uint32_t idesc = umma_idesc(F3_TILE, F3_TILE);
            for (int it = 0; it < total; ++it) {
                const int s = it & 1;
                if (*(volatile int*)&abort_flag) break;
                if (!mbar_wait_cluster(&full_bar[s], (it >> 1) & 1)) {
                    atomicExch(p.error, ERR_F3_MMA_WAIT); atomicExch(&abort_flag, 1); break;
                }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const unsigned char* stage = smem + s * F3_STAGE;
                int any = 0;
                for (int i = 0; i < 2 * F3_WORKERS; ++i) any |= *(volatile int*)&fine[s][i];
                const bool whole = any != 0;
                constexpr int X[6] = {0, 1, 0, 2, 1, 0}, W[6] = {2, 1, 1, 0, 0, 0};        // small products first
#pragma unroll
                for (int t = 0; t < 6; ++t) {
                    if (t < 3 && !whole) continue;   // products with parts of w that are all zero
                    const uint64_t a = umma_desc(stage + X[t] * F3_BOX), b = umma_desc(stage + (3 + W[t]) * F3_BOX);
#pragma unroll
                    for (int k = 0; k < F3_K / 16; ++k)
                        umma_bf16_pair(tmem + s * F3_TILE, a + 2 * k, b + 2 * k, idesc, (k > 0 || t > (whole ? 0 : 3)) ? 1u : 0u);
                }
                umma_commit_pair(&done_bar[s]);
            }
        }
    }

    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    cluster_sync_all();     // neither block frees tensor memory or leaves while the other may still signal it
    if (warp == 1) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(F3_TMEM) : "memory");
    }
}

// In tiles with results that are not finite those results, computed by FFMA.
__global__ void __launch_bounds__(256, 2)
gemm_f32_odd_tiles_kernel(const float* __restrict__ x, const float* __restrict__ w, const float* __restrict__ bias,
                          float* __restrict__ y, int M, int N, int K, int ldx, int ldy, int m_tiles, int n_tiles,
                          const int* __restrict__ odd) {
    grid_dependency_wait();
    grid_dependents_go();
    constexpr int PER = (F3_TILE / TM) * (F3_TILE / TN);
    for (int t = blockIdx.x; t < m_tiles * n_tiles * PER; t += gridDim.x) {
        if (!odd[t / PER]) continue;
        int mt, nt;
        f3_place(t / PER, m_tiles, n_tiles, mt, nt);
        const int m0 = mt * F3_TILE + (t & 1) * TM, n0 = nt * F3_TILE + ((t >> 1) & 1) * TN;
        if (m0 >= M || n0 >= N) continue;
        __syncthreads();
        f32_tile<true>(x, w, bias, y, M, N, K, ldx, ldy, m0, n0);
    }
}

static int f3_pairs(int* out) {
    static int max_pairs = 0;
    if (max_pairs == 0) {
        cudaError_t e = cudaFuncSetAttribute(gemm_f32_split_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)F3_SMEM);
        if (e != cudaSuccess) return (int)e;
        int device = 0, sms = 0, clusters = 0;
        cudaGetDevice(&device);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
        cudaLaunchConfig_t config = {};
        config.gridDim = dim3(sms & ~1, 1, 1);
        config.blockDim = dim3(F3_THREADS, 1, 1);
        config.dynamicSmemBytes = F3_SMEM;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = 2;
        attr[0].val.clusterDim.y = 1;
        attr[0].val.clusterDim.z = 1;
        config.attrs = attr;
        config.numAttrs = 1;
        e = cudaOccupancyMaxActiveClusters(&clusters, gemm_f32_split_kernel, &config);
        if (e != cudaSuccess) return (int)e;
        if (clusters <= 0) return ERR_UNSUPPORTED;
        max_pairs = clusters;
    }
    *out = max_pairs;
    return 0;
}

static int f3_map(CUtensorMap* map, CUtensorMapDataType type, int rank, const void* base, const cuuint64_t* dims,
                  const cuuint64_t* strides, const cuuint32_t* box, CUtensorMapL2promotion promotion,
                  CUtensorMapSwizzle swizzle = CU_TENSOR_MAP_SWIZZLE_128B) {
    EncodeTiled encode = encode_tiled();
    if (!encode) return ERR_UNSUPPORTED;
    const cuuint32_t elem[3] = {1, 1, 1};
    return encode(map, type, rank, const_cast<void*>(base), dims, strides, box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE,
                  swizzle, promotion, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS
               ? 0 : ERR_BAD_ARGUMENT;
}

static int f3_plane_ld(int K) { return (K + 7) / 8 * 8; }      // rows of a plane start on 16 bytes

}  // namespace fsie

using namespace fsie;

extern "C" {

// How many pairs of blocks run at the same time (also sets the kernel up, outside any stream capture).
int fsie_gemm_f32_split_pairs() {
    int pairs = 0;
    const int rc = f3_pairs(&pairs);
    return rc != 0 ? (rc > 0 ? -rc : rc) : pairs;
}

// Room the launch needs: bfloat16 elements of planes and ints of notes.
int fsie_gemm_f32_split_room(int M, int N, int K, long long* plane_elements, int* notes) {
    if (M <= 0 || N <= 0 || K <= 0) return ERR_BAD_ARGUMENT;
    *plane_elements = 3LL * M * f3_plane_ld(K);
    const long long tiles = (long long)((M + F3_TILE - 1) / F3_TILE) * ((N + F3_TILE - 1) / F3_TILE);
    if (tiles > 0x1fffffff || tiles * ((K + F3_K - 1) / F3_K) > 0x3fffffff) return ERR_UNSUPPORTED;
    *notes = (int)tiles;
    return 0;
}

// y = x w^T (+ bias), all float32; K and ldx multiples of 4, x and w on 16 bytes.
int fsie_gemm_f32_split(const float* x, long long ldx, const float* w, const float* bias, float* y, long long ldy, int M,
                        int N, int K, void* planes, long long plane_elements, int* notes, int notes_len, int blocks,
                        int* error, cudaStream_t stream) {
    if (M <= 0 || N <= 0) return 0;
    if (K <= 0 || K % 4 || ldx % 4 || ldx < K || ldx > 0x7fffffff || ldy < N || ldy > 0x7fffffff || blocks < 2 || !error ||
        ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(w) | reinterpret_cast<uintptr_t>(planes)) & 15))
        return ERR_BAD_ARGUMENT;
    long long need_planes = 0;
    int tiles = 0, pairs = 0;
    int rc = fsie_gemm_f32_split_room(M, N, K, &need_planes, &tiles);
    if (rc != 0) return rc;
    if (!planes || !notes || plane_elements < need_planes || notes_len < tiles) return ERR_BAD_ARGUMENT;
    rc = f3_pairs(&pairs);
    if (rc != 0) return rc;
    if (pairs > blocks / 2) pairs = blocks / 2;
    if (tiles < pairs) pairs = tiles;
    const int plane_ld = f3_plane_ld(K);

    CUtensorMap map_w, map_x, map_y;
    {
        const cuuint64_t dims[2] = {(cuuint64_t)K, (cuuint64_t)N};
        const cuuint64_t strides[1] = {(cuuint64_t)K * 4};
        const cuuint32_t box[2] = {F3_K, 16};
        rc = f3_map(&map_w, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, w, dims, strides, box, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                    CU_TENSOR_MAP_SWIZZLE_NONE);
        if (rc != 0) return rc;
    }
    {
        const cuuint64_t dims[3] = {(cuuint64_t)K, (cuuint64_t)M, 3};
        const cuuint64_t strides[2] = {(cuuint64_t)plane_ld * 2, (cuuint64_t)M * plane_ld * 2};
        const cuuint32_t box[3] = {F3_K, F3_HALF, 1};
        rc = f3_map(&map_x, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, planes, dims, strides, box, CU_TENSOR_MAP_L2_PROMOTION_L2_256B);
        if (rc != 0) return rc;
    }
    SplitGemmParams p;
    p.bias = bias; p.y = y; p.ldy = ldy; p.M = M; p.N = N; p.K = K;
    p.m_tiles = (M + F3_TILE - 1) / F3_TILE;
    p.n_tiles = (N + F3_TILE - 1) / F3_TILE;
    // the copy engine clips a box at 16 bytes: rows of y that end elsewhere are stored by the lanes
    p.tma_store = N % 4 == 0 && ldy % 4 == 0 && (reinterpret_cast<uintptr_t>(y) & 15) == 0;
    p.odd = notes; p.error = error;
    map_y = map_x;
    if (p.tma_store) {
        const cuuint64_t dims[2] = {(cuuint64_t)N, (cuuint64_t)M};
        const cuuint64_t strides[1] = {(cuuint64_t)ldy * 4};
        const cuuint32_t box[2] = {32, 32};
        rc = f3_map(&map_y, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, y, dims, strides, box, CU_TENSOR_MAP_L2_PROMOTION_NONE);
        if (rc != 0) return rc;
    }
    const long long quads = (long long)M * (K / 4);
    const int split_blocks = (int)(quads / 1024 + 1 < 4LL * blocks ? quads / 1024 + 1 : 4LL * blocks);
    rc = launch_dependent(gemm_f32_split_rows_kernel, dim3(split_blocks), dim3(256), 0, stream, x, ldx, (bf16*)planes, M, K,
                          plane_ld, notes, tiles);
    if (rc != 0) return rc;
    cudaLaunchConfig_t config = {};
    config.gridDim = dim3(2 * pairs, 1, 1);
    config.blockDim = dim3(F3_THREADS, 1, 1);
    config.dynamicSmemBytes = F3_SMEM;
    config.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    config.attrs = attr;
    config.numAttrs = 2;
    rc = (int)cudaLaunchKernelEx(&config, gemm_f32_split_kernel, map_w, map_x, map_y, p);
    if (rc != 0) return rc;
    const int odd_blocks = 4 * tiles < blocks ? 4 * tiles : blocks;
    return launch_dependent(gemm_f32_odd_tiles_kernel, dim3(odd_blocks), dim3(256), 0, stream, x, w, bias, y, M, N, K,
                            (int)ldx, (int)ldy, p.m_tiles, p.n_tiles, (const int*)notes);
}

}  // extern "C"
