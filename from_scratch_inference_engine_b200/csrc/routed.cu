// A feed-forward of routed experts: every token chooses `top` of `experts` small gated
// feed-forwards and adds their outputs with weights.
//
//   route      z = W_r y (32-bit), s = sigmoid(z) (or softmax over the experts), choice = s + correction;
//              experts form `groups` equal groups of neighbours, a group's score is the sum of its two
//              largest choices, only experts of the `keep` best groups can be chosen (the others
//              count as minus infinity); the `top` largest choices are taken; their weights are
//              s / (sum of the chosen s + 1e-20) * scale (normalise = 0: s * scale).  With a router
//              bias z = W_r y + bias.  Scores over the chosen alone: s = z for the choice, and the
//              weights are softmax(z) over the chosen experts * scale
//   align      (token, choice) pairs sorted by expert, cut into tiles of rows that share an expert
//   gate_up    act[r] = f(W_gate[e] y[t(r)]) * (W_up[e] y[t(r)])       r in sorted order
//   down       out[pair(r)] = W_down[e] act[r]
//   combine    y_out[t] = sum_j weight[t, j] * out[t, j] (+ what a shared expert gave for t)
//
// The number of rows per expert is known only on the device, so the grids are sized for the worst
// case (pairs / tile + experts tiles) and blocks beyond the tile count leave at once: a step
// launches the same kernels whatever the routing says.  The router, its scores, the choice and the
// weights are 32-bit; the products add in 32-bit.
#include "common.cuh"
#include <math.h>

namespace fsie {

constexpr int MOE_TILE = 64;          // rows (and output columns) per tile of the tiled products
constexpr int MOE_FEW_TILE = 16;      // rows per tile of the products that stream the experts' matrices

// what a router's logits become: sigmoid, softmax over all experts, softmax over the chosen ones
enum { SCORES_SIGMOID = 0, SCORES_SOFTMAX = 1, SCORES_CHOSEN_SOFTMAX = 2 };

// -------------------------------------------------------------------------------- router
// (value, index) maximum over a shared array by one warp; ties go to the lower index.
__device__ __forceinline__ int warp_argmax(const float* v, const unsigned char* taken, int n, int lane) {
    float best = -INFINITY;
    int at = -1;
    for (int i = lane; i < n; i += 32) {
        if (taken[i]) continue;
        if (at < 0 || v[i] > best) { best = v[i]; at = i; }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const float ob = __shfl_xor_sync(0xffffffffu, best, o);
        const int oa = __shfl_xor_sync(0xffffffffu, at, o);
        if (oa >= 0 && (at < 0 || ob > best || (ob == best && oa < at))) { best = ob; at = oa; }
    }
    return at;
}

// y == nullptr: the router's logits were computed by a matrix product and wait in `logits`
// [tokens, experts]; the block (one warp then) only scores, chooses and weighs.
template <typename T>
__global__ void moe_route_kernel(const T* __restrict__ y, int y_ld, const float* __restrict__ w_router,
                                 const float* __restrict__ logits,
                                 const float* __restrict__ bias, const float* __restrict__ correction,
                                 int* __restrict__ ids, float* __restrict__ weights, int width, int experts,
                                 int top, int groups, int keep, float scale, int score_kind, int normalise,
                                 int group_max) {
    extern __shared__ float route_smem[];
    float* row = route_smem;                       // [width]
    float* score = row + width;                    // [experts] s
    float* choice = score + experts;               // [experts] s + correction
    float* group_score = choice + experts;         // [groups]
    unsigned char* taken = reinterpret_cast<unsigned char*>(group_score + groups);   // [experts]
    unsigned char* group_taken = taken + experts;                                     // [groups]
    const int t = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
    grid_dependency_wait();
    grid_dependents_go();
    if (y) {
        const T* yr = y + (size_t)t * y_ld;
        for (int c = threadIdx.x; c < width; c += blockDim.x) row[c] = to_float(yr[c]);
        __syncthreads();
        for (int e = warp; e < experts; e += warps) {
            const float* wr = w_router + (size_t)e * width;
            float acc = 0.f;
            for (int c = lane; c < width; c += 32) acc = fmaf(wr[c], row[c], acc);
            acc = warp_sum(acc);
            if (lane == 0) score[e] = acc + (bias ? bias[e] : 0.f);
        }
    } else {
        for (int e = threadIdx.x; e < experts; e += blockDim.x) score[e] = logits[(size_t)t * experts + e] + (bias ? bias[e] : 0.f);
    }
    __syncthreads();
    if (warp != 0) return;
    if (score_kind == SCORES_SOFTMAX) {
        float m = -INFINITY;
        for (int e = lane; e < experts; e += 32) m = fmaxf(m, score[e]);
        m = warp_max(m);
        float sum = 0.f;
        for (int e = lane; e < experts; e += 32) sum += expf(score[e] - m);
        sum = warp_sum(sum);
        for (int e = lane; e < experts; e += 32) score[e] = expf(score[e] - m) / sum;
    } else if (score_kind == SCORES_SIGMOID) {
        for (int e = lane; e < experts; e += 32) score[e] = 1.0f / (1.0f + expf(-score[e]));
    }
    for (int e = lane; e < experts; e += 32) {
        choice[e] = score[e] + (correction ? correction[e] : 0.f);
        taken[e] = 0;
    }
    __syncwarp();
    if (groups > 1 && keep < groups) {
        const int per = experts / groups;
        for (int g = lane; g < groups; g += 32) {
            float first = -INFINITY, second = -INFINITY;
            for (int i = 0; i < per; ++i) {
                const float v = choice[g * per + i];
                if (v > first) { second = first; first = v; }
                else if (v > second) second = v;
            }
            group_score[g] = (per > 1 && !group_max) ? first + second : first;
            group_taken[g] = 0;
        }
        __syncwarp();
        for (int k = 0; k < keep; ++k) {
            const int g = warp_argmax(group_score, group_taken, groups, lane);
            if (lane == 0 && g >= 0) group_taken[g] = 1;
            __syncwarp();
        }
        for (int e = lane; e < experts; e += 32)
            if (!group_taken[e / per]) taken[e] = 1;       // outside the kept groups: never chosen
        __syncwarp();
    }
    float sum = 0.f, largest = -INFINITY;
    for (int k = 0; k < top; ++k) {
        const int e = warp_argmax(choice, taken, experts, lane);
        if (lane == 0) {
            ids[(size_t)t * top + k] = e < 0 ? 0 : e;
            if (e >= 0) taken[e] = 1;
        }
        sum += e < 0 ? 0.f : score[e];
        if (e >= 0) largest = fmaxf(largest, score[e]);
        __syncwarp();
    }
    if (score_kind == SCORES_CHOSEN_SOFTMAX) {
        if (lane != 0) return;
        float total = 0.f;
        for (int k = 0; k < top; ++k) total += expf(score[ids[(size_t)t * top + k]] - largest);
        for (int k = 0; k < top; ++k)
            weights[(size_t)t * top + k] = expf(score[ids[(size_t)t * top + k]] - largest) / total * scale;
    } else if (lane == 0) {
        for (int k = 0; k < top; ++k) {
            const float s = score[ids[(size_t)t * top + k]];
            weights[(size_t)t * top + k] = normalise ? s / (sum + 1e-20f) * scale : s * scale;
        }
    }
}

// ------------------------------------------------------------------- pairs sorted by expert
// By one warp, from the rows of every expert: start[e], the expert's first row (start[experts]: their number; `padded`:
// every expert's rows start on a multiple of `tile`), and tile_start[e], its first tile.  Returns the number of tiles.
__device__ __forceinline__ int expert_starts(const int* count, int experts, int tile, int padded, int* start, int* tile_start) {
    const int lane = threadIdx.x & 31;
    int rows_before = 0, tiles_before = 0;
    for (int e0 = 0; e0 < experts; e0 += 32) {
        const int e = e0 + lane, n = e < experts ? count[e] : 0;
        int rows = n, tiles = (n + tile - 1) / tile;
        const int own_tiles = tiles;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int r = __shfl_up_sync(0xffffffffu, rows, o), t = __shfl_up_sync(0xffffffffu, tiles, o);
            if (lane >= o) { rows += r; tiles += t; }
        }
        if (e < experts) {
            tile_start[e] = tiles_before + tiles - own_tiles;
            start[e] = padded ? tile_start[e] * tile : rows_before + rows - n;
        }
        rows_before += __shfl_sync(0xffffffffu, rows, 31);
        tiles_before += __shfl_sync(0xffffffffu, tiles, 31);
    }
    if (lane == 0) {
        start[experts] = padded ? tiles_before * tile : rows_before;
        tile_start[experts] = tiles_before;
    }
    return tiles_before;
}

// One block.  Compact layout: offsets[e] .. offsets[e + 1] are the rows of expert e in `sorted`
// (pair = token * top + choice); tiles: (expert, first row) of every tile of `tile` rows; meta[0] =
// their number.  Padded layout (`padded`): every expert's rows start on a multiple of `tile`, rows
// that no pair owns hold -1, offsets[e] is the expert's first row, and place[pair] is the pair's row.
__global__ void moe_align_kernel(const int* __restrict__ ids, int pairs, int experts, int tile, int padded,
                                 int* __restrict__ offsets, int* __restrict__ sorted, int* __restrict__ tile_expert,
                                 int* __restrict__ tile_row0, int* __restrict__ meta, int* __restrict__ place) {
    extern __shared__ int align_smem[];
    int* count = align_smem;                    // [experts]
    int* start = count + experts;               // [experts + 1]
    int* tile_start = start + experts + 1;      // [experts + 1]
    grid_dependency_wait();
    grid_dependents_go();
    for (int e = threadIdx.x; e < experts; e += blockDim.x) count[e] = 0;
    __syncthreads();
    for (int p = threadIdx.x; p < pairs; p += blockDim.x) {
        const int e = ids[p];
        if (e >= 0 && e < experts) atomicAdd(&count[e], 1);
    }
    __syncthreads();
    if (threadIdx.x < 32) {
        const int tiles = expert_starts(count, experts, tile, padded, start, tile_start);
        if (threadIdx.x == 0) meta[0] = tiles;
    }
    __syncthreads();
    for (int e = threadIdx.x; e <= experts; e += blockDim.x) offsets[e] = start[e];
    for (int e = threadIdx.x; e < experts; e += blockDim.x) {
        const int n = tile_start[e + 1] - tile_start[e];
        for (int i = 0; i < n; ++i) {
            tile_expert[tile_start[e] + i] = e;
            tile_row0[tile_start[e] + i] = start[e] + i * tile;
        }
        count[e] = 0;                           // from here on: how many rows of e are placed
    }
    if (padded)
        for (int r = threadIdx.x; r < start[experts]; r += blockDim.x) sorted[r] = -1;
    __syncthreads();
    // a pair's place among its expert's rows: in the order the threads arrive.  Each row of a
    // product is summed on its own, so the order of an expert's rows changes no result.
    for (int p = threadIdx.x; p < pairs; p += blockDim.x) {
        const int e = ids[p];
        if (e < 0 || e >= experts) continue;
        const int at = start[e] + atomicAdd(&count[e], 1);
        sorted[at] = p;
        if (place) place[p] = at;
    }
}

// ------------------------------------------------- choice and lists of a step in one launch
// The choice of one token by one warp, its experts' scores in registers (expert lane + 32 j in the lane's j-th): what
// moe_route_kernel computes from the router's logits, the same bits.  Lane k < top receives choice k and its weight.
// `choice_smem`: room of this warp for `experts` floats.
template <int EPL>
__device__ __forceinline__ int lane_argmax(const float (&v)[EPL], unsigned taken, int lane) {
    float best = -INFINITY;
    int at = -1;
#pragma unroll
    for (int j = 0; j < EPL; ++j)
        if (!(taken >> j & 1) && (at < 0 || v[j] > best)) { best = v[j]; at = lane + 32 * j; }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const float ob = __shfl_xor_sync(0xffffffffu, best, o);
        const int oa = __shfl_xor_sync(0xffffffffu, at, o);
        if (oa >= 0 && (at < 0 || ob > best || (ob == best && oa < at))) { best = ob; at = oa; }
    }
    return __shfl_sync(0xffffffffu, at, 0);
}

template <int EPL>
__device__ __forceinline__ void choose_experts(const float* __restrict__ logits, const float* __restrict__ bias,
                                               const float* __restrict__ correction, float* choice_smem, int experts,
                                               int top, int groups, int keep, float scale, int score_kind, int normalise,
                                               int group_max, int lane, int& my_expert, float& my_weight) {
    float s[EPL], c[EPL];
    unsigned taken = 0;
#pragma unroll
    for (int j = 0; j < EPL; ++j) {
        const int e = lane + 32 * j;
        s[j] = e < experts ? logits[e] + (bias ? bias[e] : 0.f) : -INFINITY;
        if (e >= experts) taken |= 1u << j;
    }
    if (score_kind == SCORES_SOFTMAX) {
        float m = -INFINITY, sum = 0.f;
#pragma unroll
        for (int j = 0; j < EPL; ++j) if (lane + 32 * j < experts) m = fmaxf(m, s[j]);
        m = warp_max(m);
#pragma unroll
        for (int j = 0; j < EPL; ++j) if (lane + 32 * j < experts) sum += expf(s[j] - m);
        sum = warp_sum(sum);
#pragma unroll
        for (int j = 0; j < EPL; ++j) s[j] = expf(s[j] - m) / sum;
    } else if (score_kind == SCORES_SIGMOID) {
#pragma unroll
        for (int j = 0; j < EPL; ++j) s[j] = 1.0f / (1.0f + expf(-s[j]));
    }
#pragma unroll
    for (int j = 0; j < EPL; ++j) {
        const int e = lane + 32 * j;
        c[j] = s[j] + (correction && e < experts ? correction[e] : 0.f);
    }
    if (groups > 1 && keep < groups) {
        const int per = experts / groups;
#pragma unroll
        for (int j = 0; j < EPL; ++j) if (lane + 32 * j < experts) choice_smem[lane + 32 * j] = c[j];
        __syncwarp();
        float score[EPL];
        unsigned kept = 0;                               // of the groups lane + 32 j
        unsigned none = 0;                               // ... those that do not exist
#pragma unroll
        for (int j = 0; j < EPL; ++j) {
            const int g = lane + 32 * j;
            float first = -INFINITY, second = -INFINITY;
            if (g < groups)
                for (int i = 0; i < per; ++i) {
                    const float v = choice_smem[g * per + i];
                    if (v > first) { second = first; first = v; }
                    else if (v > second) second = v;
                }
            else none |= 1u << j;
            score[j] = (per > 1 && !group_max) ? first + second : first;
        }
        for (int k = 0; k < keep; ++k) {
            const int g = lane_argmax<EPL>(score, kept | none, lane);
            if (g >= 0 && (g & 31) == lane) kept |= 1u << (g >> 5);
        }
        __syncwarp();                                    // every lane has read the choices: the room holds marks now
#pragma unroll
        for (int j = 0; j < EPL; ++j) if (lane + 32 * j < groups) choice_smem[lane + 32 * j] = kept >> j & 1 ? 1.f : 0.f;
        __syncwarp();
#pragma unroll
        for (int j = 0; j < EPL; ++j)
            if (lane + 32 * j < experts && choice_smem[(lane + 32 * j) / per] == 0.f) taken |= 1u << j;
    }
    float sum = 0.f, largest = -INFINITY, my_score = 0.f;
    my_expert = 0;
    for (int k = 0; k < top; ++k) {
        const int found = lane_argmax<EPL>(c, taken, lane), e = found < 0 ? 0 : found;
        float v = 0.f;
#pragma unroll
        for (int j = 0; j < EPL; ++j) if (j == e >> 5) v = s[j];
        v = __shfl_sync(0xffffffffu, v, e & 31);
        if (found >= 0) {
            sum += v;
            largest = fmaxf(largest, v);
            if ((e & 31) == lane) taken |= 1u << (e >> 5);
        }
        if (lane == k) { my_expert = e; my_score = v; }
    }
    if (score_kind == SCORES_CHOSEN_SOFTMAX) {
        const float part = expf(my_score - largest);
        float total = 0.f;
        for (int k = 0; k < top; ++k) total += __shfl_sync(0xffffffffu, part, k);
        my_weight = part / total * scale;
    } else {
        my_weight = normalise ? my_score / (sum + 1e-20f) * scale : my_score * scale;
    }
}

// One block, a warp per token: the choice from the router's logits, then the lists of moe_align_kernel (compact layout) from
// the choices in shared memory.  Nothing here is more than a chain of dependent steps, so what
// counts is their number: as two launches that met in global memory, with the scores in shared memory and one
// thread walking the experts' counts, 8 tokens of 64 experts in 8 groups took 16 us of a decode step's layer.
constexpr int CHOOSE_TOKENS = 32;
template <int EPL>
__global__ void __launch_bounds__(32 * CHOOSE_TOKENS)
moe_route_align_kernel(const float* __restrict__ logits, const float* __restrict__ bias,
                       const float* __restrict__ correction, int* __restrict__ ids,
                       float* __restrict__ weights, int routed, int top, int groups, int keep,
                       float scale, int score_kind, int normalise, int group_max, int experts, int tile,
                       int* __restrict__ offsets, int* __restrict__ sorted, int* __restrict__ tile_expert,
                       int* __restrict__ tile_row0, int* __restrict__ meta) {
    extern __shared__ float choose_smem[];
    const int t = threadIdx.x >> 5, lane = threadIdx.x & 31, tokens = blockDim.x >> 5;
    float* room = choose_smem + (size_t)t * routed;                                    // [tokens][routed]
    int* count = reinterpret_cast<int*>(choose_smem + (size_t)tokens * routed);         // [experts]
    int* start = count + experts;                                                      // [experts + 1]
    int* tile_start = start + experts + 1;                                             // [experts + 1]
    for (int e = threadIdx.x; e < experts; e += blockDim.x) count[e] = 0;
    grid_dependency_wait();
    grid_dependents_go();
    int expert;
    float weight;
    choose_experts<EPL>(logits + (size_t)t * routed, bias, correction, room, routed, top, groups, keep, scale, score_kind,
                        normalise, group_max, lane, expert, weight);
    __syncthreads();                                     // the counts are zero
    // choices at or beyond `experts` are identity experts: no rows.  A pair's place among its expert's rows is the
    // order the lanes arrive in: each row of a product is summed on its own, so it changes no result.
    const bool chosen = lane < top, listed = chosen && expert < experts;
    int place = 0;
    if (chosen) {
        ids[t * top + lane] = expert;
        weights[t * top + lane] = weight;
    }
    if (listed) place = atomicAdd(&count[expert], 1);
    __syncthreads();
    if (t == 0) {
        const int tiles = expert_starts(count, experts, tile, 0, start, tile_start);
        if (lane == 0) meta[0] = tiles;
    }
    __syncthreads();
    if (listed) sorted[start[expert] + place] = t * top + lane;
    for (int e = threadIdx.x; e <= experts; e += blockDim.x) {
        offsets[e] = start[e];
        if (e == experts) break;
        for (int i = tile_start[e]; i < tile_start[e + 1]; ++i) {
            tile_expert[i] = e;
            tile_row0[i] = start[e] + (i - tile_start[e]) * tile;
        }
    }
}

// x_sorted[r] = x[sorted[r] / top] for the rows of the used tiles (zeros where no pair owns the row):
// the rows of the step's tokens in the padded order, for a product that reads whole tiles.
__global__ void moe_gather_kernel(const bf16* __restrict__ x, long long x_ld, const int* __restrict__ sorted,
                                  const int* __restrict__ meta, int tile, int top, bf16* __restrict__ out, int k) {
    grid_dependency_wait();
    grid_dependents_go();
    const int r = blockIdx.x;
    if (r >= meta[0] * tile) return;
    const int pair = sorted[r];
    uint4* dst = reinterpret_cast<uint4*>(out + (size_t)r * k);
    if (pair < 0) {
        for (int c = threadIdx.x; c < k / 8; c += blockDim.x) dst[c] = make_uint4(0, 0, 0, 0);
        return;
    }
    const uint4* src = reinterpret_cast<const uint4*>(x + (size_t)(pair / top) * x_ld);
    for (int c = threadIdx.x; c < k / 8; c += blockDim.x) dst[c] = src[c];
}

// --------------------------------------------------------------- tiled products, any type
// A block owns one tile (expert e, 64 rows) x 64 output columns; a thread 4 x 4 of them; k in
// steps of 16 through shared memory.  GATED: the 64 columns are 32 of the gate and the same 32 of
// the up projection (a thread holds two of each), the result is f(gate) * up, rows are read at
// token = pair / top and written in sorted order.  Not GATED: rows are read in sorted order and
// written at their pair.
__device__ __forceinline__ float gate_fn(float g, int kind) {
    if (kind == 2) { const float r = fmaxf(g, 0.f); return r * r; }      // the square of relu
    if (kind == 1) return 0.5f * g * (1.0f + tanhf(0.7978845608028654f * (g + 0.044715f * g * g * g)));
    return g / (1.0f + expf(-g));
}

template <typename T, int MODE>
__global__ void __launch_bounds__(256) moe_product_kernel(
        const T* __restrict__ x, long long x_ld, const T* __restrict__ w, T* __restrict__ out, long long out_ld,
        const int* __restrict__ offsets, const int* __restrict__ sorted, const int* __restrict__ tile_expert,
        const int* __restrict__ tile_row0, const int* __restrict__ meta, int top, int n, int k, int gate_kind) {
    constexpr bool GATED = MODE == 1, FIRST = MODE != 0;
    __shared__ float xs[16][MOE_TILE + 4];
    __shared__ float ws[16][MOE_TILE + 4];
    __shared__ int src[MOE_TILE], dst[MOE_TILE];
    grid_dependency_wait();
    grid_dependents_go();
    const int tile = blockIdx.x;
    if (tile >= meta[0]) return;
    const int e = tile_expert[tile], r0 = tile_row0[tile];
    const int rows = min(MOE_TILE, offsets[e + 1] - r0);
    constexpr int COLS = GATED ? MOE_TILE / 2 : MOE_TILE;     // distinct outputs per block
    const int n0 = blockIdx.y * COLS;
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    if (threadIdx.x < MOE_TILE) {
        const int r = threadIdx.x;
        const int pair = r < rows ? sorted[r0 + r] : -1;
        src[r] = pair < 0 ? -1 : (FIRST ? pair / top : r0 + r);
        dst[r] = pair < 0 ? -1 : (FIRST ? r0 + r : pair);
    }
    __syncthreads();
    const T* we = w + (size_t)e * (GATED ? 2 : 1) * n * k;
    float acc[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;
    for (int k0 = 0; k0 < k; k0 += 16) {
        for (int idx = threadIdx.x; idx < MOE_TILE * 16; idx += 256) {
            const int r = idx / 16, kk = idx - r * 16, kc = k0 + kk;
            const int s = src[r];
            xs[kk][r] = (s >= 0 && kc < k) ? to_float(x[(size_t)s * x_ld + kc]) : 0.f;
            // column r of the tile: which row of the expert's matrix
            int wrow;
            if (GATED) {
                const int c = n0 + (r >> 2) * 2 + (r & 1);
                wrow = c < n ? ((r & 2) ? n + c : c) : -1;
            } else {
                wrow = n0 + r < n ? n0 + r : -1;
            }
            ws[kk][r] = (wrow >= 0 && kc < k) ? to_float(we[(size_t)wrow * k + kc]) : 0.f;
        }
        __syncthreads();
#pragma unroll
        for (int kk = 0; kk < 16; ++kk) {
            const float4 a = *reinterpret_cast<const float4*>(&xs[kk][ty * 4]);
            const float4 b = *reinterpret_cast<const float4*>(&ws[kk][tx * 4]);
            const float av[4] = {a.x, a.y, a.z, a.w}, bv[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(av[i], bv[j], acc[i][j]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int d = dst[ty * 4 + i];
        if (d < 0) continue;
        T* o = out + (size_t)d * out_ld;
        if (GATED) {
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                const int c = n0 + tx * 2 + j;
                // gate and up are rounded to the storage type before the activation, as a product
                // that stored them in between would have
                const float g = to_float(from_float<T>(acc[i][j])), u = to_float(from_float<T>(acc[i][2 + j]));
                if (c < n) o[c] = from_float<T>(gate_fn(g, gate_kind) * u);
            }
        } else {
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int c = n0 + tx * 4 + j;
                if (c < n) o[c] = MODE == 2 ? from_float<T>(gate_fn(to_float(from_float<T>(acc[i][j])), gate_kind))
                                            : from_float<T>(acc[i][j]);
            }
        }
    }
}

// ------------------------------------------------- the same on the tensor cores (bfloat16)
// mma.sync m16n8k16: a block of four warps owns a tile of 64 rows x 64 columns (GATED: 32 of the
// gate, then the same 32 of the up projection; a thread's fragments j and j + 4 are a gate and its
// up), a warp 16 rows; x and w travel by cp.async in chunks of 64 k-elements into two slots.
constexpr int MM_K = 64, MM_LD = MM_K + 8;

__device__ __forceinline__ uint32_t mm_smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mm_ldsm_x4(uint32_t (&r)[4], const void* p) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(mm_smem_u32(p)));
}
__device__ __forceinline__ void mm_mma(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void mm_cp16(void* dst, const void* src, bool valid) {
    const int bytes = valid ? 16 : 0;
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" :: "r"(mm_smem_u32(dst)), "l"(src), "r"(bytes) : "memory");
}

template <int MODE>
__global__ void __launch_bounds__(128) moe_product_mma_kernel(
        const bf16* __restrict__ x, long long x_ld, const bf16* __restrict__ w, bf16* __restrict__ out,
        long long out_ld, const int* __restrict__ offsets, const int* __restrict__ sorted,
        const int* __restrict__ tile_expert, const int* __restrict__ tile_row0, const int* __restrict__ meta,
        int top, int n, int k, int gate_kind) {
    constexpr bool GATED = MODE == 1, FIRST = MODE != 0;
    __shared__ __align__(16) bf16 xs[2][MOE_TILE][MM_LD];
    __shared__ __align__(16) bf16 ws[2][MOE_TILE][MM_LD];
    __shared__ int src[MOE_TILE], dst[MOE_TILE];
    grid_dependency_wait();
    grid_dependents_go();
    const int tile = blockIdx.x;
    if (tile >= meta[0]) return;
    const int e = tile_expert[tile], r0 = tile_row0[tile];
    const int rows = min(MOE_TILE, offsets[e + 1] - r0);
    constexpr int COLS = GATED ? MOE_TILE / 2 : MOE_TILE;
    const int n0 = blockIdx.y * COLS;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int g = lane >> 2, t = lane & 3;
    if (tid < MOE_TILE) {
        const int pair = tid < rows ? sorted[r0 + tid] : -1;
        src[tid] = pair < 0 ? -1 : (FIRST ? pair / top : r0 + tid);
        dst[tid] = pair < 0 ? -1 : (FIRST ? r0 + tid : pair);
    }
    __syncthreads();
    const bf16* we = w + (size_t)e * (GATED ? 2 : 1) * n * k;
    // a thread copies half a row (four 16-byte pieces) of x and of w per chunk
    const int cr = tid >> 1, c0 = (tid & 1) * 4;
    const int xrow = src[cr];
    int wrow;
    if (GATED) {
        const int c = n0 + (cr & 31);
        wrow = c < n ? (cr >= 32 ? n + c : c) : -1;
    } else {
        wrow = n0 + cr < n ? n0 + cr : -1;
    }
    auto issue = [&](int stage, int k0) {
#pragma unroll
        for (int c = c0; c < c0 + 4; ++c) {
            const int kc = k0 + c * 8;
            const bool xin = xrow >= 0 && kc < k, win = wrow >= 0 && kc < k;
            mm_cp16(&xs[stage][cr][c * 8], x + (xin ? (size_t)xrow * x_ld + kc : 0), xin);
            mm_cp16(&ws[stage][cr][c * 8], we + (win ? (size_t)wrow * k + kc : 0), win);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    float acc[8][4];
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[j][0] = acc[j][1] = acc[j][2] = acc[j][3] = 0.f;
    issue(0, 0);
    int it = 0;
    for (int k0 = 0; k0 < k; k0 += MM_K, ++it) {
        const int stage = it & 1;
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();
        if (k0 + MM_K < k) issue(stage ^ 1, k0 + MM_K);
        if (warp * 16 < rows) {
            const bf16* xa = &xs[stage][warp * 16 + (lane & 15)][(lane >> 4) * 8];
            const bf16* wb = &ws[stage][(lane & 7) + (lane >> 4) * 8][((lane >> 3) & 1) * 8];
#pragma unroll
            for (int kk = 0; kk < MM_K; kk += 16) {
                uint32_t a[4];
                mm_ldsm_x4(a, xa + kk);
#pragma unroll
                for (int nb = 0; nb < 4; ++nb) {
                    uint32_t b[4];
                    mm_ldsm_x4(b, wb + nb * 16 * MM_LD + kk);
                    mm_mma(acc[2 * nb], a, b[0], b[1]);
                    mm_mma(acc[2 * nb + 1], a, b[2], b[3]);
                }
            }
        }
    }
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        const int d = dst[warp * 16 + g + 8 * i];
        if (d < 0) continue;
        bf16* o = out + (size_t)d * out_ld;
        if (GATED) {
#pragma unroll
            for (int j = 0; j < 4; ++j) {
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int c = n0 + j * 8 + 2 * t + h;
                    const float gt = __bfloat162float(__float2bfloat16_rn(acc[j][2 * i + h]));
                    const float up = __bfloat162float(__float2bfloat16_rn(acc[j + 4][2 * i + h]));
                    if (c < n) o[c] = __float2bfloat16_rn(gate_fn(gt, gate_kind) * up);
                }
            }
        } else {
#pragma unroll
            for (int j = 0; j < 8; ++j) {
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int c = n0 + j * 8 + 2 * t + h;
                    if (c < n)
                        o[c] = MODE == 2 ? __float2bfloat16_rn(gate_fn(__bfloat162float(__float2bfloat16_rn(acc[j][2 * i + h])), gate_kind))
                                         : __float2bfloat16_rn(acc[j][2 * i + h]);
                }
            }
        }
    }
}

// ------------------------------------------------ few rows per expert: the matrices streamed once
// A decode step gives an expert one to a few rows, so the product is the time its matrices take to come
// in.  The tiled kernel above waits for every 64 k-elements with one chunk asked for ahead and keeps 18 KB
// per block on the way.  Here blocks stay (three of 256 threads per SM) and walk items of (tile of up to 16
// rows, 32 rows of w - GATED: 16 of the gate and the same 16 of the up projection) in slots of 128 k-elements:
// all threads ask for a slot's 8 KB of w and its rows of x with cp.async, five slots ahead (40 KB of w per
// block on the way), and the slots run on into the next items.  One barrier per slot: three blocks with 6
// slots hide it from each other (64 experts of 1,408 x 2,048, 8 tokens x 6, 36 experts met, us for gate-up + down:
// 69 + 38, floor 64 + 32; two blocks with 8 slots 81 + 44; the tiled kernel 124 + 85).  Up to four warps
// multiply, 16 rows of w by 8 rows of x (the N side of mma.sync m16n8k16) each; GATED: 8 gate rows and their 8
// up rows, so that a lane ends with both.  A warp's sum runs over k in steps of 16 in ascending order, as
// in the tiled kernel: the results are the same to the bit.
constexpr int FEW_THREADS = 256, FEW_K = 128, FEW_SLOTS = 6, FEW_ROWS = 32;
constexpr int FEW_CHUNK = 32;                                                // k comes in these: two steps of 16
constexpr int FEW_PIECES = FEW_K / 8;                                        // 16-byte pieces of a slot's row
constexpr int FEW_SLOT = (FEW_ROWS + MOE_FEW_TILE) * FEW_K * 2;              // rows of w, rows of x
constexpr size_t FEW_SMEM = (size_t)FEW_SLOTS * FEW_SLOT;

// a piece's place in its slot: moved by the row, so that eight rows' pieces lie in different banks
__device__ __forceinline__ int few_place(int row, int piece) { return row * (FEW_K * 2) + ((piece ^ (row & 7)) << 4); }

template <int MODE>
__global__ void __launch_bounds__(FEW_THREADS, 3) moe_product_few_kernel(
        const bf16* __restrict__ x, long long x_ld, const bf16* __restrict__ w, bf16* __restrict__ out,
        long long out_ld, const int* __restrict__ offsets, const int* __restrict__ sorted,
        const int* __restrict__ tile_expert, const int* __restrict__ tile_row0, const int* __restrict__ meta,
        int top, int n, int k, int gate_kind, int early) {
    constexpr bool GATED = MODE == 1, FIRST = MODE != 0;
    constexpr int COLS = GATED ? 16 : 32;                    // outputs per row and item
    extern __shared__ __align__(128) unsigned char few_smem[];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    // the second product, early: the lists are older than the kernel before (else it is not launched as a dependent), and the
    // first slots of w are asked for while that one still runs.  (Without `early` the wait has nothing to wait for, but with both
    // orders in the code it comes out faster: 12 tokens in a step 63.0 and 61.9 us.)
    if (MODE != 0 || !early) {
        grid_dependency_wait();
        grid_dependents_go();
    }
    const int tiles = meta[0];
    // neighbouring items are the tiles of the same columns: an expert's further tiles find its rows in L2
    const int items = tiles * ((n + COLS - 1) / COLS);
    if ((int)blockIdx.x >= items) {
        if (MODE == 0 && early) grid_dependency_wait();
        return;
    }
    const int per = (k + FEW_K - 1) / FEW_K;                 // slots per item
    const int step_tile = gridDim.x % tiles, step_n0 = (gridDim.x / tiles) * COLS;
    auto advance = [&](int& tile, int& n0) {                 // the block's next item
        tile += step_tile;
        n0 += step_n0;
        if (tile >= tiles) { tile -= tiles; n0 += COLS; }
    };

    // ---- asking: a thread's two pieces of w (rows `row` and row + 16 of the slot) and its piece of x (row `row`)
    const int row = tid / FEW_PIECES, piece = tid % FEW_PIECES;
    int ask_tile = blockIdx.x % tiles, ask_n0 = (blockIdx.x / tiles) * COLS, ask_j = 0, ask_slot = 0;
    const bf16 *wr[2], *xr = nullptr;
    auto point = [&]() {
        if (ask_n0 >= n) return;
        const int e = tile_expert[ask_tile], r0 = tile_row0[ask_tile];
        const bf16* we = w + (size_t)e * (GATED ? 2 : 1) * n * k + piece * 8;
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            // GATED: rows 0-7 of every 16 are gate rows, rows 8-15 the up rows of the same outputs
            const int at = GATED ? ((row & 8) ? n : 0) + min(ask_n0 + 8 * i + (row & 7), n - 1) : min(ask_n0 + 16 * i + row, n - 1);
            wr[i] = we + (size_t)at * k;
        }
        const bool met = row < min(MOE_FEW_TILE, offsets[e + 1] - r0);
        xr = met ? x + (size_t)(FIRST ? sorted[r0 + row] / top : r0 + row) * x_ld + piece * 8 : nullptr;
    };
    auto ask = [&](bool of_w = true, bool of_x = true) {
        const int k0 = ask_j * FEW_K;
        if (ask_n0 < n && k0 + piece * 8 < k) {
            unsigned char* slot = few_smem + ask_slot * FEW_SLOT;
            if (of_w) {
#pragma unroll
                for (int i = 0; i < 2; ++i) mm_cp16(slot + few_place(16 * i + row, piece), wr[i] + k0, true);
            }
            if (of_x && xr) mm_cp16(slot + few_place(FEW_ROWS + row, piece), xr + k0, true);
        }
        if (of_x) asm volatile("cp.async.commit_group;" ::: "memory");  // one group per slot, also when empty
        ask_slot = ask_slot + 1 == FEW_SLOTS ? 0 : ask_slot + 1;
        if (++ask_j == per) {
            ask_j = 0;
            advance(ask_tile, ask_n0);
            point();
        }
    };
    static_assert(FEW_THREADS == MOE_FEW_TILE * FEW_PIECES && FEW_ROWS == 2 * MOE_FEW_TILE, "a thread's pieces");
    point();
    if (MODE == 0 && early) {
#pragma unroll
        for (int j = 0; j < FEW_SLOTS - 1; ++j) ask(true, false);
        grid_dependency_wait();
        grid_dependents_go();
        ask_tile = blockIdx.x % tiles; ask_n0 = (blockIdx.x / tiles) * COLS; ask_j = ask_slot = 0;     // once more for x
        point();
    }
#pragma unroll
    for (int j = 0; j < FEW_SLOTS - 1; ++j) ask(MODE != 0 || !early, true);

    // ---- multiplying: warp = (16 rows of w, 8 rows of x)
    const int half = warp & 1, eight = warp >> 1;
    const int a_row = half * 16 + (lane & 15), a_piece = lane >> 4;
    const int b_row = FEW_ROWS + eight * 8 + (lane & 7), b_piece = lane >> 3;          // two steps of 16 at a time
    int slot = 0;
    for (int tile = blockIdx.x % tiles, n0 = (blockIdx.x / tiles) * COLS; n0 < n; advance(tile, n0)) {
        const int r0 = tile_row0[tile], rows = min(MOE_FEW_TILE, offsets[tile_expert[tile] + 1] - r0);
        const bool mine = eight * 8 < rows;                  // (warps 4 to 7 never)
        float acc[4] = {0.f, 0.f, 0.f, 0.f};
        for (int j = 0; j < per; ++j) {
            asm volatile("cp.async.wait_group %0;" ::"n"(FEW_SLOTS - 2) : "memory");   // the oldest slot has landed
            __syncthreads();                                 // for all threads; and the slot before it is no longer read
            ask();
            if (mine) {
                const unsigned char* at = few_smem + slot * FEW_SLOT;
                const int end = min(FEW_K, k - j * FEW_K) / 8;       // pieces, a multiple of 4
                uint32_t a[FEW_PIECES / 2][4], b[FEW_PIECES / 4][4];
#pragma unroll
                for (int q = 0; q < FEW_PIECES; q += 2) mm_ldsm_x4(a[q / 2], at + few_place(a_row, q + a_piece));
#pragma unroll
                for (int q = 0; q < FEW_PIECES; q += 4) mm_ldsm_x4(b[q / 4], at + few_place(b_row, q + b_piece));
#pragma unroll
                for (int q = 0; q < FEW_PIECES; q += 4) {
                    if (q >= end) break;
                    mm_mma(acc, a[q / 2], b[q / 4][0], b[q / 4][1]);
                    mm_mma(acc, a[q / 2 + 1], b[q / 4][2], b[q / 4][3]);
                }
            }
            slot = slot + 1 == FEW_SLOTS ? 0 : slot + 1;
        }
        if (!mine) continue;
        // acc: rows g (0, 1) and g + 8 (2, 3) of the 16 of w, rows 2 t and 2 t + 1 of the 8 of x
        const int g = lane >> 2, t = lane & 3;
#pragma unroll
        for (int v = 0; v < 2; ++v) {
            const int r = eight * 8 + 2 * t + v;
            if (r >= rows) continue;
            bf16* o = out + (size_t)(FIRST ? r0 + r : sorted[r0 + r]) * out_ld;
            // rounded as a product that stored its result in between would have
            const float lo = __bfloat162float(__float2bfloat16_rn(acc[v])), hi = __bfloat162float(__float2bfloat16_rn(acc[2 + v]));
            if (GATED) {
                const int c = n0 + half * 8 + g;
                if (c < n) o[c] = __float2bfloat16_rn(gate_fn(lo, gate_kind) * hi);
            } else {
                const int c = n0 + half * 16 + g;
                if (c < n) o[c] = __float2bfloat16_rn(MODE == 2 ? gate_fn(lo, gate_kind) : lo);
                if (c + 8 < n) o[c + 8] = __float2bfloat16_rn(MODE == 2 ? gate_fn(hi, gate_kind) : hi);
            }
        }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
}

// The same in 32 bits: a warp owns two rows of w (GATED: a gate row and its up row), its lanes lie side by side
// along k, the rows of w of the next three passes of 128 elements are on their way into registers, and
// the tile's rows of x wait in shared memory, where every value read serves both rows of w.  8 tokens x 6 of 64
// experts of 1,408 x 2,048: 164 + 92 us (floor 124 + 62; the tiled kernel 1,220 + 596: its blocks multiply 64 rows
// whatever the tile holds).
constexpr int FEW32_WARPS = 8, FEW32_XC = 512, FEW32_DEPTH = 4;
constexpr size_t FEW32_SMEM = 2 * MOE_FEW_TILE * FEW32_XC * sizeof(float);

template <int MODE>
__global__ void __launch_bounds__(32 * FEW32_WARPS, 2) moe_product_few_f32_kernel(
        const float* __restrict__ x, long long x_ld, const float* __restrict__ w, float* __restrict__ out,
        long long out_ld, const int* __restrict__ offsets, const int* __restrict__ sorted,
        const int* __restrict__ tile_expert, const int* __restrict__ tile_row0, const int* __restrict__ meta,
        int top, int n, int k, int gate_kind) {
    constexpr bool GATED = MODE == 1, FIRST = MODE != 0;
    constexpr int PER_CHUNK = FEW32_XC / 128, D = FEW32_DEPTH;
    extern __shared__ __align__(16) float few32_smem[];
    float (*xs)[MOE_FEW_TILE][FEW32_XC] = reinterpret_cast<float (*)[MOE_FEW_TILE][FEW32_XC]>(few32_smem);
    __shared__ int src[MOE_FEW_TILE], dst[MOE_FEW_TILE];
    grid_dependency_wait();
    grid_dependents_go();
    const int tile = blockIdx.x;
    if (tile >= meta[0]) return;
    const int e = tile_expert[tile], r0 = tile_row0[tile], rows = min(MOE_FEW_TILE, offsets[e + 1] - r0);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (tid < rows) {
        const int pair = sorted[r0 + tid];
        src[tid] = FIRST ? pair / top : r0 + tid;
        dst[tid] = FIRST ? r0 + tid : pair;
    }
    const int c0 = (blockIdx.y * FEW32_WARPS + warp) * (GATED ? 1 : 2);
    const float* we = w + (size_t)e * (GATED ? 2 : 1) * n * k + lane * 4;
    const int row0 = min(c0, n - 1);
    const float* wrow[2] = {we + (size_t)row0 * k, we + (size_t)(GATED ? n + row0 : min(c0 + 1, n - 1)) * k};
    const int passes = (k + 127) / 128;
    float4 ring[D][2];
    auto load_w = [&](int pass, float4 (&to)[2]) {
        const bool in_range = pass < passes && pass * 128 + lane * 4 < k;
#pragma unroll
        for (int r = 0; r < 2; ++r)
            to[r] = in_range ? __ldg(reinterpret_cast<const float4*>(wrow[r] + pass * 128)) : make_float4(0.f, 0.f, 0.f, 0.f);
    };
#pragma unroll
    for (int d = 0; d < D - 1; ++d) load_w(d, ring[d]);
    __syncthreads();
    auto stage_x = [&](int chunk) {
        const int k0 = chunk * FEW32_XC;
        for (int i = tid; i < rows * (FEW32_XC / 4); i += 32 * FEW32_WARPS) {
            const int m = i / (FEW32_XC / 4), c = (i - m * (FEW32_XC / 4)) * 4;
            const bool in = k0 + c < k;
            mm_cp16(&xs[chunk & 1][m][c], x + (in ? (size_t)src[m] * x_ld + k0 + c : 0), in);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    stage_x(0);
    float acc[2][MOE_FEW_TILE];
#pragma unroll
    for (int m = 0; m < MOE_FEW_TILE; ++m) acc[0][m] = acc[1][m] = 0.f;
    for (int base = 0; base < passes; base += D) {
#pragma unroll
        for (int u = 0; u < D; ++u) {
            const int pass = base + u;
            load_w(pass + D - 1, ring[(u + D - 1) % D]);
            if (pass >= passes) continue;
            const int chunk = pass / PER_CHUNK, within = pass - chunk * PER_CHUNK;
            if (within == 0) {
                asm volatile("cp.async.wait_group 0;" ::: "memory");
                __syncthreads();              // this chunk's x has landed, the other half is no longer read
                if ((chunk + 1) * FEW32_XC < k) stage_x(chunk + 1);
            }
            const float* xrow = &xs[chunk & 1][0][within * 128 + lane * 4];
#pragma unroll
            for (int m = 0; m < MOE_FEW_TILE; ++m) {
                if (m >= rows) break;
                const float4 xv = *reinterpret_cast<const float4*>(xrow + m * FEW32_XC);
#pragma unroll
                for (int r = 0; r < 2; ++r)
                    acc[r][m] = fmaf(xv.w, ring[u][r].w, fmaf(xv.z, ring[u][r].z,
                                fmaf(xv.y, ring[u][r].y, fmaf(xv.x, ring[u][r].x, acc[r][m]))));
            }
        }
    }
#pragma unroll
    for (int m = 0; m < MOE_FEW_TILE; ++m) {
        if (m >= rows) break;
        const float lo = warp_sum(acc[0][m]), hi = warp_sum(acc[1][m]);
        float* o = out + (size_t)dst[m] * out_ld + c0;
        if (lane != 0 || c0 >= n) continue;
        if (GATED) {
            o[0] = gate_fn(lo, gate_kind) * hi;
        } else {
            o[0] = MODE == 2 ? gate_fn(lo, gate_kind) : lo;
            if (c0 + 1 < n) o[1] = MODE == 2 ? gate_fn(hi, gate_kind) : hi;
        }
    }
}

template <typename F>
static int allow_smem(F* kernel, size_t bytes, bool& done) {
    if (done) return 0;
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    if (e == cudaSuccess) done = true;
    return (int)e;
}

template <int MODE>
static int launch_few(const void* x, long long x_ld, const void* w, void* out, long long out_ld, const int* offsets,
                      const int* sorted, const int* tile_expert, const int* tile_row0, const int* meta, int tiles,
                      int top, int n, int k, int gate_kind, int dtype, int early, cudaStream_t stream) {
    static bool allowed[2] = {false, false};
    if (dtype == DTYPE_F32) {
        if (int e = allow_smem(moe_product_few_f32_kernel<MODE>, FEW32_SMEM, allowed[0])) return e;
        const int cols = FEW32_WARPS * (MODE == 1 ? 1 : 2);
        const dim3 grid(tiles, (n + cols - 1) / cols);
        if (grid.y > 65535) return ERR_UNSUPPORTED;
        return launch_dependent(moe_product_few_f32_kernel<MODE>, grid, dim3(32 * FEW32_WARPS), FEW32_SMEM, stream,
                                (const float*)x, x_ld, (const float*)w, (float*)out, out_ld, offsets, sorted,
                                tile_expert, tile_row0, meta, top, n, k, gate_kind);
    }
    if (int e = allow_smem(moe_product_few_kernel<MODE>, FEW_SMEM, allowed[1])) return e;
    int device = 0, sms = 148;
    if (cudaGetDevice(&device) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
    const int cols = MODE == 1 ? FEW_ROWS / 2 : FEW_ROWS;
    const long long most = (long long)tiles * ((n + cols - 1) / cols);
    return launch_dependent_if(MODE != 0 || early, moe_product_few_kernel<MODE>, dim3((unsigned)(most < 3 * sms ? most : 3 * sms)),
                            dim3(FEW_THREADS), FEW_SMEM, stream, (const bf16*)x, x_ld, (const bf16*)w, (bf16*)out,
                            out_ld, offsets, sorted, tile_expert, tile_row0, meta, top, n, k, gate_kind, early);
}

// -------------------------------------------------------------------------------- combine
// VEC: eight columns per thread, 16-byte accesses; the sums run in the same order.  AHEAD > 0: so many choices' rows travel together (a
// last one again where there are fewer), where one after the other, each behind its id and place, they were the launch's time
// (8 tokens of 8 choices of 4,096 5.6 -> 3.2 us).
template <typename T, bool VEC, int AHEAD>
__global__ void moe_combine_kernel(const T* __restrict__ expert_out, const float* __restrict__ weights,
                                   const T* __restrict__ shared, const int* __restrict__ place,
                                   T* __restrict__ out, int width, int top, const int* __restrict__ ids,
                                   int experts, const T* __restrict__ y, long long y_ld) {
    grid_dependency_wait();
    grid_dependents_go();
    const size_t t = blockIdx.x;
    // a choice at or beyond `experts` is an identity expert: its output is the token's input row
    if constexpr (VEC && AHEAD > 0) {
        for (int c = threadIdx.x * 8; c < width; c += blockDim.x * 8) {
            float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f}, v[8];
            for (int j0 = 0; j0 < top; j0 += AHEAD) {
                const T* src[AHEAD];
                float w[AHEAD], rows[AHEAD][8];
#pragma unroll
                for (int j = 0; j < AHEAD; ++j) {
                    const size_t at = t * top + min(j0 + j, top - 1);
                    const bool own = ids && ids[at] >= experts;
                    w[j] = weights[at];
                    src[j] = own ? y + t * y_ld : expert_out + (place ? (own ? 0 : (size_t)place[at]) : at) * width;
                }
#pragma unroll
                for (int j = 0; j < AHEAD; ++j) load8(src[j] + c, rows[j]);
#pragma unroll
                for (int j = 0; j < AHEAD; ++j)
                    if (j0 + j < top) {
#pragma unroll
                        for (int i = 0; i < 8; ++i) acc[i] = fmaf(w[j], rows[j][i], acc[i]);
                    }
            }
            if (shared) {
                load8(shared + t * width + c, v);
#pragma unroll
                for (int i = 0; i < 8; ++i) acc[i] += v[i];
            }
            store8(out + t * width + c, acc);
        }
        return;
    }
    if constexpr (VEC) {
        for (int c = threadIdx.x * 8; c < width; c += blockDim.x * 8) {
            float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f}, v[8];
            for (int j = 0; j < top; ++j) {
                const float w = weights[t * top + j];
                if (ids && ids[t * top + j] >= experts) {
                    load8(y + t * y_ld + c, v);
                } else {
                    const size_t row = place ? (size_t)place[t * top + j] : t * top + j;
                    load8(expert_out + row * width + c, v);
                }
#pragma unroll
                for (int i = 0; i < 8; ++i) acc[i] = fmaf(w, v[i], acc[i]);
            }
            if (shared) {
                load8(shared + t * width + c, v);
#pragma unroll
                for (int i = 0; i < 8; ++i) acc[i] += v[i];
            }
            store8(out + t * width + c, acc);
        }
        return;
    }
    for (int c = threadIdx.x; c < width; c += blockDim.x) {
        float acc = 0.f;
        for (int j = 0; j < top; ++j) {
            if (ids && ids[t * top + j] >= experts) {
                acc = fmaf(weights[t * top + j], to_float(y[t * y_ld + c]), acc);
                continue;
            }
            const size_t row = place ? (size_t)place[t * top + j] : t * top + j;
            acc = fmaf(weights[t * top + j], to_float(expert_out[row * width + c]), acc);
        }
        if (shared) acc += to_float(shared[t * width + c]);
        out[t * width + c] = from_float<T>(acc);
    }
}

}  // namespace fsie

using namespace fsie;

extern "C" {

int fsie_moe_tile_rows() { return MOE_TILE; }
int fsie_moe_few_tile_rows() { return MOE_FEW_TILE; }

// y [tokens, y_ld] of the storage type; w_router float32 [experts, width]; bias and correction float32
// [experts] or null; ids int32 / weights float32 [tokens, top].
int fsie_moe_route(const void* y, int y_ld, const float* w_router, const float* logits, const float* bias,
                   const float* correction, int* ids, float* weights, int tokens, int width, int experts, int top,
                   int groups, int keep, float scale, int score_kind, int normalise, int group_max, int dtype,
                   cudaStream_t stream) {
    if (tokens <= 0) return 0;
    if ((y && width <= 0) || experts <= 0 || top <= 0 || top > experts || groups <= 0 || experts % groups ||
        score_kind < SCORES_SIGMOID || score_kind > SCORES_CHOSEN_SOFTMAX || keep <= 0 || keep > groups || top > keep * (experts / groups))
        return ERR_BAD_ARGUMENT;
    if (!y && !logits) return ERR_BAD_ARGUMENT;
    if (!y) width = 0;
    const int threads = y ? 128 : 32;
    const size_t smem = ((size_t)width + 2 * experts + groups) * sizeof(float) + experts + groups + 8;
    if (smem > 200 * 1024) return ERR_UNSUPPORTED;
    if (dtype == DTYPE_F32) {
        if (smem > 48 * 1024)
            cudaFuncSetAttribute(moe_route_kernel<float>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        return launch_dependent(moe_route_kernel<float>, tokens, threads, smem, stream, (const float*)y, y_ld, w_router,
                                logits, bias, correction, ids, weights, width, experts, top, groups, keep, scale,
                                score_kind, normalise, group_max);
    }
    if (smem > 48 * 1024)
        cudaFuncSetAttribute(moe_route_kernel<bf16>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    return launch_dependent(moe_route_kernel<bf16>, tokens, threads, smem, stream, (const bf16*)y, y_ld, w_router,
                            logits, bias, correction, ids, weights, width, experts, top, groups, keep, scale, score_kind,
                            normalise, group_max);
}

// offsets [experts + 1], sorted [pairs] (padded: [(pairs / tile + experts) * tile]), tile_expert /
// tile_row0 [pairs / tile + experts], meta [1], place [pairs] or null
int fsie_moe_align(const int* ids, int pairs, int experts, int tile, int padded, int* offsets, int* sorted,
                   int* tile_expert, int* tile_row0, int* meta, int* place, cudaStream_t stream) {
    if (pairs <= 0) return 0;
    if (experts <= 0 || tile <= 0 || (!padded && tile != MOE_TILE && tile != MOE_FEW_TILE)) return ERR_BAD_ARGUMENT;
    const size_t smem = (3 * (size_t)experts + 2) * sizeof(int);
    if (smem > 40 * 1024) return ERR_UNSUPPORTED;
    const int threads = pairs >= 4096 ? 1024 : (pairs >= 512 ? 256 : 64);
    return launch_dependent(moe_align_kernel, 1, threads, smem, stream, ids, pairs, experts, tile, padded, offsets,
                            sorted, tile_expert, tile_row0, meta, place);
}

// The choice from the router's logits [tokens, routed] and the lists of the compact layout in one launch (arguments as above;
// experts <= routed: choices from `experts` on are identity experts).  Up to CHOOSE_TOKENS tokens, 256
// experts and 32 choices.
int fsie_moe_route_align_tokens() { return CHOOSE_TOKENS; }

int fsie_moe_route_align(const float* logits, const float* bias, const float* correction, int* ids, float* weights, int tokens,
                         int routed, int top, int groups, int keep, float scale, int score_kind, int normalise,
                         int group_max, int experts, int tile, int* offsets, int* sorted, int* tile_expert,
                         int* tile_row0, int* meta, cudaStream_t stream) {
    if (tokens <= 0) return 0;
    if (!logits || routed <= 0 || top <= 0 || top > routed || groups <= 0 || routed % groups || experts <= 0 || experts > routed ||
        score_kind < SCORES_SIGMOID || score_kind > SCORES_CHOSEN_SOFTMAX || keep <= 0 || keep > groups ||
        top > keep * (routed / groups) || (tile != MOE_TILE && tile != MOE_FEW_TILE))
        return ERR_BAD_ARGUMENT;
    if (tokens > CHOOSE_TOKENS || routed > 256 || top > 32) return ERR_UNSUPPORTED;
    const size_t smem = ((size_t)tokens * routed + 3 * (size_t)experts + 2) * 4;     // 35 KB at most
#define FSIE_ROUTE_ALIGN(EPL)                                                                                       \
    launch_dependent(moe_route_align_kernel<EPL>, 1, 32 * tokens, smem, stream, logits, bias, correction, ids, weights, \
                     routed, top, groups, keep, scale, score_kind, normalise, group_max, experts, tile, offsets, sorted, \
                     tile_expert, tile_row0, meta)
    if (routed <= 32) return FSIE_ROUTE_ALIGN(1);
    if (routed <= 64) return FSIE_ROUTE_ALIGN(2);
    if (routed <= 128) return FSIE_ROUTE_ALIGN(4);
    return FSIE_ROUTE_ALIGN(8);
#undef FSIE_ROUTE_ALIGN
}

// out [rows of the padded layout, k] bf16 = the tokens' rows of x in that order; `rows` is the room
// there is (pairs / tile + experts tiles).
int fsie_moe_gather(const void* x, long long x_ld, const int* sorted, const int* meta, int tile, int top,
                    void* out, int rows, int k, cudaStream_t stream) {
    if (rows <= 0) return 0;
    if (k <= 0 || k % 8 || x_ld % 8 || ((((size_t)x) | ((size_t)out)) & 15)) return ERR_BAD_ARGUMENT;
    return launch_dependent(moe_gather_kernel, rows, k >= 2048 ? 256 : 128, 0, stream, (const bf16*)x, x_ld, sorted,
                            meta, tile, top, (bf16*)out, k);
}

// gated = 1: x [tokens, x_ld] read at pair / top, w [experts, 2 n, k] (gate rows, then up rows), out
// [pairs, out_ld] in sorted order.  gated = 2: the same rows in and out, w [experts, n, k], out = f(x w^T)
// (an expert without a gate: gate_kind names f).  gated = 0: x [pairs, x_ld] in sorted order, w [experts, n, k], out
// written at the pair's own row.  `tile`: the rows per tile that the lists were made with; MOE_FEW_TILE takes
// the kernels that stream the matrices (k a multiple of 32 in bfloat16 and of 4 in float32, rows on 16 bytes).
int fsie_moe_product(const void* x, long long x_ld, const void* w, void* out, long long out_ld,
                     const int* offsets, const int* sorted, const int* tile_expert, const int* tile_row0,
                     const int* meta, int pairs, int experts, int top, int n, int k, int gated, int gate_kind,
                     int dtype, int tile, int early, cudaStream_t stream) {
    if (pairs <= 0 || n <= 0) return 0;
    if (k <= 0 || experts <= 0 || top <= 0 || gated < 0 || gated > 2) return ERR_BAD_ARGUMENT;
    if (tile == MOE_FEW_TILE) {
        const int step = dtype == DTYPE_F32 ? 4 : 8;                 // elements in 16 bytes
        if (k % (dtype == DTYPE_F32 ? 4 : FEW_CHUNK) || x_ld % step || ((((size_t)x) | ((size_t)w)) & 15))
            return ERR_BAD_ARGUMENT;
#define FSIE_MOE_FEW(M)                                                                                           \
        launch_few<M>(x, x_ld, w, out, out_ld, offsets, sorted, tile_expert, tile_row0, meta, pairs / tile + experts, \
                      top, n, k, gate_kind, dtype, early, stream)
        return gated == 1 ? FSIE_MOE_FEW(1) : (gated == 2 ? FSIE_MOE_FEW(2) : FSIE_MOE_FEW(0));
#undef FSIE_MOE_FEW
    }
    if (tile != MOE_TILE) return ERR_BAD_ARGUMENT;
    const int cols = gated == 1 ? MOE_TILE / 2 : MOE_TILE;
    const dim3 grid(pairs / MOE_TILE + experts, (n + cols - 1) / cols);
    if (grid.y > 65535) return ERR_UNSUPPORTED;
    if (dtype == DTYPE_BF16 && k % 8 == 0 && x_ld % 8 == 0 && ((((size_t)x) | ((size_t)w)) & 15) == 0) {
#define FSIE_MOE_MMA(M)                                                                                      \
        launch_dependent(moe_product_mma_kernel<M>, grid, dim3(128), 0, stream, (const bf16*)x, x_ld,              \
                         (const bf16*)w, (bf16*)out, out_ld, offsets, sorted, tile_expert, tile_row0, meta, top, n, \
                         k, gate_kind)
        return gated == 1 ? FSIE_MOE_MMA(1) : (gated == 2 ? FSIE_MOE_MMA(2) : FSIE_MOE_MMA(0));
#undef FSIE_MOE_MMA
    }
#define FSIE_MOE(T, G)                                                                                      \
    launch_dependent(moe_product_kernel<T, G>, grid, dim3(256), 0, stream, (const T*)x, x_ld, (const T*)w, \
                     (T*)out, out_ld, offsets, sorted, tile_expert, tile_row0, meta, top, n, k, gate_kind)
    if (dtype == DTYPE_F32) return gated == 1 ? FSIE_MOE(float, 1) : (gated == 2 ? FSIE_MOE(float, 2) : FSIE_MOE(float, 0));
    return gated == 1 ? FSIE_MOE(bf16, 1) : (gated == 2 ? FSIE_MOE(bf16, 2) : FSIE_MOE(bf16, 0));
#undef FSIE_MOE
}

// ids [tokens, top] with `experts` and y [tokens, y_ld] (or all null): a choice at or beyond `experts` is an
// identity expert, whose output is the token's row of y.
// expert_out [tokens * top, width] at the pairs' rows (or, with `place`, pair p at row place[p]);
// weights float32 [tokens, top]; shared [tokens, width] or null; out [tokens, width].
int fsie_moe_combine(const void* expert_out, const float* weights, const void* shared, const int* place, void* out,
                     int tokens, int width, int top, const int* ids, int experts, const void* y, long long y_ld,
                     int dtype, cudaStream_t stream) {
    if (tokens <= 0 || width <= 0) return 0;
    if (ids && !y) return ERR_BAD_ARGUMENT;
    const bool vec = width % 8 == 0 && (!ids || y_ld % 8 == 0) &&
        (((size_t)expert_out | (size_t)shared | (size_t)out | (size_t)y) & 15) == 0;
    const int threads = vec ? (width >= 2048 ? 256 : (width >= 1024 ? 128 : 64)) : (width >= 1024 ? 256 : 128);
    // Many tokens: one choice's row after the other where places are looked up, and for a medium number of them where a fourth row
    // or more would be asked for twice.  us one after the other and together: 2,048 tokens of 2,048, 4 choices 7.3 and 6.1, 6 10.1
    // and 9.0, with places 7.0 and 8.9; 512 tokens of 6 choices 3.9 and 4.1, of 4 3.3 and 3.0, of 2 2.7 and 2.8; 4,096 of 6 32 and 24.
    // One choice or two have no more rows: 2,048 tokens of one choice 4.3 and 3.8, and 5.6 with four.
    const bool in_turn = tokens > 256 && (place || (tokens <= 1024 && (top % 4 == 1 || top % 4 == 2)));
    const int ahead = in_turn ? 0 : (top < 3 ? top : 4);
#define FSIE_COMBINE(T, V, A) launch_dependent(moe_combine_kernel<T, V, A>, tokens, threads, 0, stream, (const T*)expert_out, \
                                            weights, (const T*)shared, place, (T*)out, width, top, ids, experts, \
                                            (const T*)y, y_ld)
#define FSIE_COMBINE_AS(T)                                                                                          \
    (!vec ? FSIE_COMBINE(T, false, 0) : ahead == 0 ? FSIE_COMBINE(T, true, 0) : ahead == 1 ? FSIE_COMBINE(T, true, 1) \
     : ahead == 2 ? FSIE_COMBINE(T, true, 2) : FSIE_COMBINE(T, true, 4))
    return dtype == DTYPE_F32 ? FSIE_COMBINE_AS(float) : FSIE_COMBINE_AS(bf16);
#undef FSIE_COMBINE_AS
#undef FSIE_COMBINE
}

}  // extern "C"
