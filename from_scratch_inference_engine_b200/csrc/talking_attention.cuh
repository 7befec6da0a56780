// Softmax attention whose normalised weights are mixed across heads before they meet the
// values, over a sliding window that also keeps the first tokens of the sequence.
//
//   s_h(i, j) = (q_h,i . k_g(h),j) * scale   for visible j:
//                   j <= i and (window == 0 or i - j < window or j < keep_first)
//   p_h = softmax_j s_h            p'_h = sum_h' talk[h, h'] p_h'
//   o_h,i = sum_j p'_h(i, j) v_g(h),j                      g(h) = h / (heads / kv_heads)
//
// The mixing needs every head's FINISHED softmax at the same (i, j), so one block takes a tile of
// consecutive tokens of one request with all heads and walks the visible keys twice: once for
// every row's maximum and sum, once to form the weights, mix them and apply them to the values.
// Scores, softmax, mixed weights and outputs are 32-bit arithmetic on the CUDA cores whatever the
// storage type T of the pages.  A tile whose keys are many and whose tokens are few (decoding)
// is split over several blocks by key range: a first launch leaves every range's maximum and
// sum, a second combines them, applies its own range and leaves a partial output, a third adds
// the partial outputs in a fixed order.
//
// Included by one source file per storage type, which instantiates `talking_attention_launch`.
#pragma once

#include "common.cuh"

namespace fsie {

constexpr int TA_WARPS = 8;
constexpr int TA_ROWS = 64;        // (token, head) rows a block holds at most: 8 per warp

struct TalkingArgs {
    const float* q; const void* k_pages; const void* v_pages; long long page_stride; int page_size;
    const int* block_tables; int table_stride; const int* tile_item; const int* tile_row0;
    const int* item_qstart; const int* item_qlen; const int* item_pos0; const int* item_slots;
    const float* talk; void* out;
    int heads, kv_heads, dim, vdim, window, keep_first, tile_tokens;
    float scale; int* error;
    int nsplit, mode;              // mode 0: both walks, out; 1: first walk, part_stats; 2: second walk, part_out
    float* part_stats;             // [tiles][nsplit][TA_ROWS][2]
    float* part_out;               // [nsplit][tokens][heads * vdim]
    int tokens, early;             // early: the mixing matrix and the lists are older than the kernel before the first walk
};

__device__ __forceinline__ void load2(const float* p, float& a, float& b) {
    const float2 v = *reinterpret_cast<const float2*>(p);
    a = v.x; b = v.y;
}
__device__ __forceinline__ void load2(const bf16* p, float& a, float& b) {
    const float2 v = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(p));
    a = v.x; b = v.y;
}

// sizes of the shared-memory layout, the same on host and device
struct TalkingLayout {
    int dim8, vdim8, q_ld, kv_ld;
    size_t q_bytes, kv_bytes, p_bytes, talk_bytes, total;
    __host__ __device__ TalkingLayout(int heads, int kv_heads, int dim, int vdim, int key_tile,
                                      int elem_bytes, int rows = TA_ROWS) {
        dim8 = (dim + 7) & ~7;
        vdim8 = (vdim + 7) & ~7;
        q_ld = dim8 + 4;
        kv_ld = (dim8 > vdim8 ? dim8 : vdim8) + 16 / elem_bytes;     // rows 16 bytes apart in banks
        q_bytes = (size_t)rows * q_ld * sizeof(float);
        kv_bytes = (size_t)kv_heads * key_tile * kv_ld * elem_bytes;
        p_bytes = (size_t)rows * key_tile * sizeof(float);
        talk_bytes = (((size_t)heads * heads * sizeof(float)) + 15) & ~(size_t)15;
        total = q_bytes + kv_bytes + 2 * p_bytes + talk_bytes + 2 * key_tile * sizeof(int);
    }
};

// One tile of keys (or values) of every key/value head from the pages into shared memory
// [g][key][ld], zero beyond `width` and for keys without a page: asynchronous copies of 16 bytes
// where the rows allow it, all of a tile's on their way together (a warp that copied a row at a time
// through registers waited for memory once a row, 32 times for 4 heads of 64 keys).
__device__ __forceinline__ void talking_copy16(void* to, const void* from, int bytes) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((unsigned)__cvta_generic_to_shared(to)), "l"(from), "r"(bytes)
                 : "memory");
}
template <typename T>
__device__ __forceinline__ void copy_tile(T* __restrict__ dst, const T* __restrict__ pages,
                                          const int* key_page, const int* key_off, int G, int keys,
                                          int width, int width8, int ld, long long page_stride,
                                          int page_size, int warp, int lane) {
    constexpr int PER = 16 / (int)sizeof(T);                 // elements of one 16-byte piece
    const bool wide = width % PER == 0 && page_stride % PER == 0 &&
                      (reinterpret_cast<uintptr_t>(pages) & 15) == 0;
    if (wide) {
        const int pieces = width8 / PER, total = G * keys * pieces;
        for (int i = warp * 32 + lane; i < total; i += TA_WARPS * 32) {
            const int row = i / pieces, d = (i - row * pieces) * PER, g = row / keys, jj = row - g * keys;
            const int page = key_page[jj];
            const bool there = page >= 0 && d < width;
            talking_copy16(dst + (size_t)row * ld + d,
                           there ? pages + page * page_stride + ((size_t)g * page_size + key_off[jj]) * width + d : pages,
                           there ? 16 : 0);
        }
    } else {
        for (int row = warp; row < G * keys; row += TA_WARPS) {
            const int g = row / keys, jj = row - g * keys;
            const int page = key_page[jj];
            T* to = dst + (size_t)row * ld;
            const T* from = page < 0 ? nullptr :
                pages + page * page_stride + ((size_t)g * page_size + key_off[jj]) * width;
            for (int d = lane; d < width8; d += 32)
                to[d] = (from && d < width) ? from[d] : from_float<T>(0.f);
        }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
}
__device__ __forceinline__ void talking_copies_done() { asm volatile("cp.async.wait_group 0;" ::: "memory"); }

// Warp w owns heads w, w + 8, ... (HS of them at most: 8 / TOK, two where 16 heads of single tokens need no more code and registers) and, of each, the tile's TOK
// tokens: rows that share their keys and values, so one load of a key or value serves TOK rows.
// Lane l owns keys l (+ 32) of a tile for the scores and value columns 2 l, 2 l + 1 (+ 64 c).
// A split tile's block has one or two tiles of keys: it is a chain of trips to memory.  The lists, the first tile's pages
// and the mixing matrix are read before the kernel before has finished, and the second walk gets as far as its first tile's
// scores and values then: the first walk only read the queries, keys and values.  Shared memory is laid out for the
// tile's own rows, so that blocks of both walks fit an SM (4 requests of 1,024 keys, the three launches: 56 us, 20 now; code for
// 64 heads where there are 16 alone cost 20 us, 10 a walk, most of it the fetch of instructions).
template <typename T, int TOK, int VC2, int KPL, int HS>
__global__ void __launch_bounds__(TA_WARPS * 32) talking_attention_kernel(const TalkingArgs a) {
    constexpr int TK = 32 * KPL;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int H = a.heads, G = a.kv_heads, dim = a.dim, vdim = a.vdim;
    const int group = H / G;
    const int tile = blockIdx.x, split = blockIdx.y;
    const int item = a.tile_item[tile], tok0 = a.tile_row0[tile];
    const int n_tok = min(TOK, a.item_qlen[item] - tok0);
    if (a.item_slots[item] < 0 || n_tok <= 0) {         // a padding entry of a fixed-size batch
        grid_dependency_wait();
        return;
    }
    const int R = n_tok * H;
    const int p_first = a.item_pos0[item] + tok0, p_last = p_first + n_tok - 1;
    const int lo = a.window > 0 ? max(0, p_first - a.window + 1) : 0;
    const int kept = min(a.keep_first, lo);             // kept first tokens that lie below the window
    const int n_keys = kept + (p_last - lo + 1);
    const int key_tiles = (n_keys + TK - 1) / TK;
    const int per_split = (key_tiles + a.nsplit - 1) / a.nsplit;
    const int u_begin = min(n_keys, split * per_split * TK);
    const int u_end = min(n_keys, (split + 1) * per_split * TK);

    const TalkingLayout L(H, G, dim, vdim, TK, (int)sizeof(T), TOK * H);
    float* qs = reinterpret_cast<float*>(smem_raw);
    T* kv = reinterpret_cast<T*>(smem_raw + L.q_bytes);
    float* P = reinterpret_cast<float*>(smem_raw + L.q_bytes + L.kv_bytes);
    float* P2 = P + TOK * H * TK;
    float* talk = P2 + TOK * H * TK;
    int* key_page = reinterpret_cast<int*>(reinterpret_cast<unsigned char*>(talk) + L.talk_bytes);
    int* key_off = key_page + TK;

    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const T* k_pages = reinterpret_cast<const T*>(a.k_pages);
    const T* v_pages = reinterpret_cast<const T*>(a.v_pages);
    const int* table = a.block_tables + (size_t)item * a.table_stride;
    const int token0 = a.item_qstart[item] + tok0;

    bool gone = false;                                  // a visible key's page was given back
    const auto find_keys = [&](int u0) {
        if ((int)threadIdx.x >= TK) return;
        int page = -1, off = 0;
        if (u0 + (int)threadIdx.x < u_end) {
            const int u = u0 + threadIdx.x;
            const int j = u < kept ? u : lo + (u - kept);
            page = table[j / a.page_size];
            off = j - (j / a.page_size) * a.page_size;
            gone |= page < 0;
        }
        key_page[threadIdx.x] = page;
        key_off[threadIdx.x] = off;
    };
    // keys or values of every key/value head: [g][key][dim8], zero beyond dim and beyond the tile
    const auto copy_keys = [&]() {
        copy_tile<T>(kv, k_pages, key_page, key_off, G, TK, dim, L.dim8, L.kv_ld, a.page_stride, a.page_size, warp, lane);
    };
    const auto copy_values = [&]() {
        copy_tile<T>(kv, v_pages, key_page, key_off, G, TK, vdim, L.vdim8, L.kv_ld, a.page_stride, a.page_size, warp, lane);
    };
    const bool early = a.mode == 2;                     // what the keys' writer left is older than the kernel before
    for (int idx = threadIdx.x; idx < H * H; idx += blockDim.x) talk[idx] = a.talk[idx];
    if (u_begin < u_end) find_keys(u_begin);
    if (!early) {
        grid_dependency_wait();
        grid_dependents_go();                           // (not before the wait: the second walk's early reads rest on it)
    } else {
        __syncthreads();                                // the first tile's pages
        if (u_begin < u_end) copy_keys();
    }
    // q rows [tok * H + h], zero beyond dim and beyond the tile's tokens
    for (int idx = threadIdx.x; idx < TOK * H * L.dim8; idx += blockDim.x) {
        const int r = idx / L.dim8, d = idx - r * L.dim8;
        qs[r * L.q_ld + d] = (r < R && d < dim) ? a.q[((size_t)token0 * H + r) * dim + d] : 0.f;
    }
    float row_max[HS][TOK], row_sum[HS][TOK], acc[HS][TOK][VC2][2];
#pragma unroll
    for (int hs = 0; hs < HS; ++hs)
#pragma unroll
        for (int t = 0; t < TOK; ++t) {
            row_max[hs][t] = -INFINITY;
            row_sum[hs][t] = 0.f;
#pragma unroll
            for (int c = 0; c < VC2; ++c) acc[hs][t][c][0] = acc[hs][t][c][1] = 0.f;
        }

    const auto read_statistics = [&]() {
        // maximum and sum over all key ranges, from what the first launch left: a lane reads a range's, the sum is
        // taken range by range
        const float* stats = a.part_stats + (size_t)tile * a.nsplit * TA_ROWS * 2;
        float range_max[HS][TOK], range_sum[HS][TOK];
        const auto read_ranges = [&](int s0) {
#pragma unroll
            for (int hs = 0; hs < HS; ++hs)
#pragma unroll
                for (int t = 0; t < TOK; ++t) {
                    const int h = warp + TA_WARPS * hs, s = s0 + lane;
                    const bool in = h < H && t < n_tok && s < a.nsplit;
                    const float2 v = in ? *reinterpret_cast<const float2*>(stats + ((size_t)s * TA_ROWS + t * H + h) * 2)
                                        : make_float2(-INFINITY, 0.f);
                    range_max[hs][t] = v.x;
                    range_sum[hs][t] = v.y;
                }
        };
        for (int s0 = 0; s0 < a.nsplit; s0 += 32) {
            read_ranges(s0);
#pragma unroll
            for (int hs = 0; hs < HS; ++hs)
#pragma unroll
                for (int t = 0; t < TOK; ++t) row_max[hs][t] = fmaxf(row_max[hs][t], warp_max(range_max[hs][t]));
        }
        for (int s0 = 0; s0 < a.nsplit; s0 += 32) {
            if (a.nsplit > 32) read_ranges(s0);
#pragma unroll
            for (int hs = 0; hs < HS; ++hs)
#pragma unroll
                for (int t = 0; t < TOK; ++t) {
                    if (warp + TA_WARPS * hs >= H || t >= n_tok) continue;
                    const float factor = expf(range_max[hs][t] - row_max[hs][t]);
                    for (int s = 0; s < min(32, a.nsplit - s0); ++s) {
                        const float ms = __shfl_sync(0xffffffffu, range_max[hs][t], s);
                        const float sum = __shfl_sync(0xffffffffu, range_sum[hs][t], s);
                        const float e = __shfl_sync(0xffffffffu, factor, s);
                        if (ms > -INFINITY) row_sum[hs][t] += sum * e;
                    }
                }
        }
    };

    const int first_pass = a.mode == 2 ? 1 : 0, last_pass = a.mode == 1 ? 0 : 1;
    // whether the tile's token t sees this lane's key in the tile of n keys from u0
    const auto sees = [&](int u0, int n, int t, int kp) {
        const int u = u0 + lane + 32 * kp, j = u < kept ? u : lo + (u - kept), p_i = p_first + t;
        return lane + 32 * kp < n && j <= p_i && (a.window <= 0 || p_i - j < a.window || j < a.keep_first);
    };
    for (int pass = first_pass; pass <= last_pass; ++pass) {
        for (int u0 = u_begin; u0 < u_end; u0 += TK) {
            const int n = min(TK, u_end - u0);
            if (!(early && u0 == u_begin)) {
                __syncthreads();                         // the tile before is done with kv, P, P2
                if (u0 != u_begin || pass != first_pass) find_keys(u0);
                __syncthreads();
                copy_keys();
            }
            talking_copies_done();
            __syncthreads();
#pragma unroll
            for (int hs = 0; hs < HS; ++hs) {
                const int h = warp + TA_WARPS * hs;
                if (h >= H) continue;
                const int g = h / group;
                float s[TOK][KPL];
#pragma unroll
                for (int t = 0; t < TOK; ++t)
#pragma unroll
                    for (int kp = 0; kp < KPL; ++kp) s[t][kp] = 0.f;
                for (int d = 0; d < L.dim8; d += 8) {
                    float kk[KPL][8];
#pragma unroll
                    for (int kp = 0; kp < KPL; ++kp)
                        load8(kv + ((size_t)g * TK + lane + 32 * kp) * L.kv_ld + d, kk[kp]);
#pragma unroll
                    for (int t = 0; t < TOK; ++t) {
                        float qq[8];
                        load8(qs + (t * H + h) * L.q_ld + d, qq);
#pragma unroll
                        for (int kp = 0; kp < KPL; ++kp)
#pragma unroll
                            for (int e = 0; e < 8; ++e) s[t][kp] += qq[e] * kk[kp][e];
                    }
                }
#pragma unroll
                for (int t = 0; t < TOK; ++t) {
                    if (t >= n_tok) continue;
                    bool see[KPL];
                    float tile_max = -INFINITY;
#pragma unroll
                    for (int kp = 0; kp < KPL; ++kp) {
                        see[kp] = sees(u0, n, t, kp);
                        s[t][kp] = see[kp] ? s[t][kp] * a.scale : -INFINITY;
                        tile_max = fmaxf(tile_max, s[t][kp]);
                    }
                    if (pass == 0) {
                        const float m_new = fmaxf(row_max[hs][t], warp_max(tile_max));
                        if (m_new > -INFINITY) {
                            float e = 0.f;
#pragma unroll
                            for (int kp = 0; kp < KPL; ++kp) e += see[kp] ? expf(s[t][kp] - m_new) : 0.f;
                            row_sum[hs][t] = row_sum[hs][t] * expf(row_max[hs][t] - m_new) + warp_sum(e);
                            row_max[hs][t] = m_new;
                        }
                    } else {
#pragma unroll
                        for (int kp = 0; kp < KPL; ++kp) P[(t * H + h) * TK + lane + 32 * kp] = s[t][kp];
                    }
                }
            }
            if (pass == 0) continue;
            __syncthreads();                             // everybody is done with the keys
            copy_values();
            if (early && u0 == u_begin) {
                grid_dependency_wait();
                grid_dependents_go();
                read_statistics();
            }
            // weights from the scores that this lane has just left there
#pragma unroll
            for (int hs = 0; hs < HS; ++hs) {
                const int h = warp + TA_WARPS * hs;
                if (h >= H) continue;
#pragma unroll
                for (int t = 0; t < TOK; ++t) {
                    if (t >= n_tok) continue;
                    const float inv = 1.0f / row_sum[hs][t];
#pragma unroll
                    for (int kp = 0; kp < KPL; ++kp) {
                        float* at = P + (t * H + h) * TK + lane + 32 * kp;
                        *at = sees(u0, n, t, kp) ? expf(*at - row_max[hs][t]) * inv : 0.f;
                    }
                }
            }
            __syncthreads();                             // P holds every head's weights of this tile
            for (int idx = threadIdx.x; idx < R * TK; idx += blockDim.x) {
                const int r = idx / TK, jj = idx - r * TK;
                const int t = r / H, h = r - t * H;
                const float* mix = talk + h * H;
                const float* col = P + (size_t)t * H * TK + jj;
                float m = 0.f;
                for (int h2 = 0; h2 < H; ++h2) m += mix[h2] * col[h2 * TK];
                P2[idx] = m;
            }
            talking_copies_done();
            __syncthreads();
#pragma unroll
            for (int hs = 0; hs < HS; ++hs) {
                const int h = warp + TA_WARPS * hs;
                if (h >= H) continue;
                const T* vg = kv + (size_t)(h / group) * TK * L.kv_ld;
                for (int jj = 0; jj < TK; jj += 4) {
                    if (jj >= n) break;
                    float4 p[TOK];
#pragma unroll
                    for (int t = 0; t < TOK; ++t)
                        p[t] = t < n_tok ? *reinterpret_cast<const float4*>(P2 + (t * H + h) * TK + jj)
                                         : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
                    for (int c = 0; c < VC2; ++c) {
                        const int col = 2 * lane + 64 * c;
                        if (col >= L.vdim8) continue;
                        float v[4][2];
#pragma unroll
                        for (int x = 0; x < 4; ++x) load2(vg + (size_t)(jj + x) * L.kv_ld + col, v[x][0], v[x][1]);
#pragma unroll
                        for (int t = 0; t < TOK; ++t) {
                            acc[hs][t][c][0] += p[t].x * v[0][0] + p[t].y * v[1][0] + p[t].z * v[2][0] + p[t].w * v[3][0];
                            acc[hs][t][c][1] += p[t].x * v[0][1] + p[t].y * v[1][1] + p[t].z * v[2][1] + p[t].w * v[3][1];
                        }
                    }
                }
            }
        }
    }

    if (early && u_begin >= u_end) {                    // a range without keys
        grid_dependency_wait();
        grid_dependents_go();
    }
    if (gone) atomicExch(a.error, 3);
    if (a.mode == 1) {
        float* stats = a.part_stats + ((size_t)tile * a.nsplit + split) * TA_ROWS * 2;
#pragma unroll
        for (int hs = 0; hs < HS; ++hs) {
            const int h = warp + TA_WARPS * hs;
#pragma unroll
            for (int t = 0; t < TOK; ++t) {
                if (h >= H || t >= n_tok || lane != 0) continue;
                stats[(t * H + h) * 2] = row_max[hs][t];
                stats[(t * H + h) * 2 + 1] = row_sum[hs][t];
            }
        }
        return;
    }
#pragma unroll
    for (int hs = 0; hs < HS; ++hs) {
        const int h = warp + TA_WARPS * hs;
        if (h >= H) continue;
#pragma unroll
        for (int t = 0; t < TOK; ++t) {
            if (t >= n_tok) continue;
            const size_t at = ((size_t)(token0 + t) * H + h) * vdim;
#pragma unroll
            for (int c = 0; c < VC2; ++c)
#pragma unroll
                for (int x = 0; x < 2; ++x) {
                    const int col = 2 * lane + 64 * c + x;
                    if (col >= vdim) continue;
                    if (a.mode == 0) reinterpret_cast<T*>(a.out)[at + col] = from_float<T>(acc[hs][t][c][x]);
                    else a.part_out[(size_t)split * a.tokens * H * vdim + at + col] = acc[hs][t][c][x];
                }
        }
    }
}

// out = the partial outputs of the key ranges added in order
template <typename T>
__global__ void talking_attention_merge_kernel(const float* __restrict__ part, T* __restrict__ out,
                                               long long count, int nsplit) {
    grid_dependency_wait();
    grid_dependents_go();
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < count;
         i += (long long)gridDim.x * blockDim.x) {
        float v = 0.f;
#pragma unroll 16
        for (int s = 0; s < nsplit; ++s) v += part[(size_t)s * count + i];
        out[i] = from_float<T>(v);
    }
}

// keys of one tile (64 or 32) that fit the shared memory for these sizes; 0: none does
inline int talking_key_tile(int heads, int kv_heads, int dim, int vdim, int elem_bytes) {
    const size_t limits[2] = {110 * 1024, 220 * 1024};   // two blocks on an SM, else one
    for (size_t limit : limits)
        for (int tile = 64; tile >= 32; tile /= 2)
            if (TalkingLayout(heads, kv_heads, dim, vdim, tile, elem_bytes).total <= limit) return tile;
    return 0;
}

template <typename T, int TOK, int VC2>
int talking_attention_launch_tile(const TalkingArgs& a, int num_tiles, int key_tile, size_t smem,
                                  cudaStream_t stream) {
    const dim3 grid(num_tiles, a.nsplit);
    const auto go = [&](auto kernel) {
        cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        return launch_dependent_if(a.early || a.mode == 2, kernel, grid, TA_WARPS * 32, smem, stream, a);
    };
    if constexpr (TOK == 1) {
        if (a.heads <= 2 * TA_WARPS)
            return key_tile == 64 ? go(talking_attention_kernel<T, TOK, VC2, 2, 2>) : go(talking_attention_kernel<T, TOK, VC2, 1, 2>);
    }
    return key_tile == 64 ? go(talking_attention_kernel<T, TOK, VC2, 2, 8 / TOK>) : go(talking_attention_kernel<T, TOK, VC2, 1, 8 / TOK>);
}

template <typename T, int TOK>
int talking_attention_launch_tok(const TalkingArgs& a, int num_tiles, int key_tile, size_t smem,
                                 cudaStream_t stream) {
    const int pairs = (a.vdim + 63) / 64;
    if (pairs <= 1) return talking_attention_launch_tile<T, TOK, 1>(a, num_tiles, key_tile, smem, stream);
    if (pairs <= 2) return talking_attention_launch_tile<T, TOK, 2>(a, num_tiles, key_tile, smem, stream);
    return talking_attention_launch_tile<T, TOK, 4>(a, num_tiles, key_tile, smem, stream);
}

template <typename T>
int talking_attention_launch(TalkingArgs a, int num_tiles, cudaStream_t stream) {
    if (num_tiles <= 0) return 0;
    if (a.heads <= 0 || a.kv_heads <= 0 || a.heads % a.kv_heads || a.window < 0 || a.keep_first < 0 ||
        a.nsplit < 1 || a.nsplit > 65535 ||
        (a.tile_tokens != 1 && a.tile_tokens != 2 && a.tile_tokens != 4 && a.tile_tokens != 8) ||
        a.tile_tokens * ((a.heads + TA_WARPS - 1) / TA_WARPS) > 8)
        return ERR_BAD_ARGUMENT;
    if (a.vdim > 256) return ERR_UNSUPPORTED;
    const int key_tile = talking_key_tile(a.heads, a.kv_heads, a.dim, a.vdim, (int)sizeof(T));
    if (key_tile == 0) return ERR_UNSUPPORTED;
    const size_t smem = TalkingLayout(a.heads, a.kv_heads, a.dim, a.vdim, key_tile, (int)sizeof(T),
                                      a.tile_tokens * a.heads).total;
    if (a.nsplit > 1 && (!a.part_stats || !a.part_out)) return ERR_BAD_ARGUMENT;
    const int first = a.nsplit > 1 ? 1 : 0, last = a.nsplit > 1 ? 2 : 0;
    for (int mode = first; mode <= last; ++mode) {
        a.mode = mode;
        int code;
        switch (a.tile_tokens) {
            case 1: code = talking_attention_launch_tok<T, 1>(a, num_tiles, key_tile, smem, stream); break;
            case 2: code = talking_attention_launch_tok<T, 2>(a, num_tiles, key_tile, smem, stream); break;
            case 4: code = talking_attention_launch_tok<T, 4>(a, num_tiles, key_tile, smem, stream); break;
            default: code = talking_attention_launch_tok<T, 8>(a, num_tiles, key_tile, smem, stream); break;
        }
        if (code) return code;
    }
    if (a.nsplit > 1) {
        const long long count = (long long)a.tokens * a.heads * a.vdim;
        const long long wanted = (count + 255) / 256;
        return launch_dependent(talking_attention_merge_kernel<T>, (unsigned)(wanted > 2048 ? 2048 : wanted), 256, 0, stream,
                                a.part_out, reinterpret_cast<T*>(a.out), count, a.nsplit);
    }
    return 0;
}

}  // namespace fsie
