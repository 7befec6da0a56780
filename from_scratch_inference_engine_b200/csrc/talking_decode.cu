// Attention with mixed heads (talking_attention.cuh) for steps of one token per request, in two launches.
//
//   scores   s[h, j] = (q_h . k_g(h),j) * scale, 32-bit, to memory, and of every range of 64 keys each head's
//            maximum and sum of exponentials
//   values   from those every head's softmax p_h, the mixed weights p'_h = sum_h' talk[h, h'] p_h' of one group of heads,
//            and o_h = sum_j p'_h(j) v_g(h),j
//
// The tiled kernel keeps all heads of a range of keys in one block because the mixing needs them together, so a step of
// few requests has few blocks, and it walks the keys twice, each time through shared memory behind barriers.
// A token's scores are few numbers: written once, they let every group of heads have blocks of its own for the keys
// (scores) and for 32 columns of the values (values), whose loads wait for nothing but the list of pages.
// What bounds both is the chain of dependent trips to memory.
#include "common.cuh"

namespace fsie {

constexpr int TD_KEYS = 64;          // keys of a block of the first launch
constexpr int TD_GROUP = 8;          // query heads per key/value head at most
constexpr int TD_TILE = 256;         // keys whose mixed weights a block of the second launch holds at once
constexpr int TD_COLS = 32;          // value columns of such a block

struct TalkingDecodeArgs {
    const float* q; const void* k_pages; const void* v_pages; long long page_stride; int page_size;
    const int* block_tables; int table_stride;
    const int* item_qstart; const int* item_qlen; const int* item_pos0; const int* item_slots;
    const float* talk; void* out;
    int heads, kv_heads, dim, vdim, window, keep_first, nsplit;
    float scale; int* error;
    float* scores;                   // [items][heads][nsplit * TD_KEYS]
    float* stats;                    // [items][nsplit][heads][2]
};

__device__ __forceinline__ void load_pair(const float* p, float& a, float& b) {
    const float2 v = *reinterpret_cast<const float2*>(p);
    a = v.x; b = v.y;
}
__device__ __forceinline__ void load_pair(const bf16* p, float& a, float& b) {
    const float2 v = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(p));
    a = v.x; b = v.y;
}

// The keys that the token of a request sees, numbered from 0: first the kept ones below the window, then the window's.
struct SeenKeys {
    int lo, kept, count;
    __device__ __forceinline__ SeenKeys(const TalkingDecodeArgs& a, int item) {
        const int p = a.item_pos0[item];
        lo = a.window > 0 ? max(0, p - a.window + 1) : 0;
        kept = min(a.keep_first, lo);
        count = min(kept + (p - lo + 1), a.nsplit * TD_KEYS);
    }
    __device__ __forceinline__ int key(int u) const { return u < kept ? u : lo + (u - kept); }
};

// Element offset of a key's row for key/value head g and rows of `width`, or -1 where its page was given back.
__device__ __forceinline__ long long row_offset(const TalkingDecodeArgs& a, const int* table, int j, int g, int width) {
    const int block = j / a.page_size, page = table[block];
    if (page < 0) return -1;
    return page * a.page_stride + ((long long)g * a.page_size + (j - block * a.page_size)) * width;
}

// grid (ranges of 64 keys, key/value heads, requests), 128 threads: eight lanes share a key, each with 8 of every 64
// columns (16 bytes of bfloat16); DIT: columns in 64s.
template <typename T, int DIT>
__global__ void __launch_bounds__(128) talking_scores_kernel(const TalkingDecodeArgs a) {
    __shared__ __align__(16) float qs[TD_GROUP][DIT * 64];
    __shared__ float sc[TD_GROUP][TD_KEYS];
    const int split = blockIdx.x, g = blockIdx.y, item = blockIdx.z;
    const int group = a.heads / a.kv_heads, tid = threadIdx.x, sub = tid & 7;
    const int slot = a.item_slots[item];
    const bool padding = slot < 0 || a.item_qlen[item] <= 0;      // a padding entry of a fixed-size batch
    const SeenKeys seen(a, item);
    const int u0 = split * TD_KEYS, n = padding ? 0 : min(TD_KEYS, seen.count - u0);
    const int* table = a.block_tables + (size_t)item * a.table_stride;
    // lists and tables were staged before the step: read while the kernel before still runs
    long long row[TD_KEYS / 16];
#pragma unroll
    for (int i = 0; i < TD_KEYS / 16; ++i) {
        const int u = i * 16 + (tid >> 3);
        row[i] = -1;
        if (u < n) {
            row[i] = row_offset(a, table, seen.key(u0 + u), g, a.dim);
            if (row[i] < 0 && sub == 0) atomicExch(a.error, 3);      // a visible key's page was given back
        }
    }
    grid_dependency_wait();
    grid_dependents_go();
    if (n <= 0) return;
    const T* pages = reinterpret_cast<const T*>(a.k_pages);
    float k[TD_KEYS / 16][DIT][8];
#pragma unroll
    for (int i = 0; i < TD_KEYS / 16; ++i)
#pragma unroll
        for (int x = 0; x < DIT; ++x) {
            const int d = x * 64 + sub * 8;
            if (row[i] >= 0 && d < a.dim) load8(pages + row[i] + d, k[i][x]);
            else {
#pragma unroll
                for (int e = 0; e < 8; ++e) k[i][x][e] = 0.f;
            }
        }
    const float* q = a.q + ((size_t)a.item_qstart[item] * a.heads + g * group) * a.dim;
    for (int idx = tid; idx < group * DIT * 64; idx += 128) {
        const int h = idx / (DIT * 64), d = idx - h * (DIT * 64);
        qs[h][d] = d < a.dim ? q[(size_t)h * a.dim + d] : 0.f;
    }
    __syncthreads();
    for (int h = 0; h < group; ++h) {
        float s[TD_KEYS / 16];
#pragma unroll
        for (int i = 0; i < TD_KEYS / 16; ++i) s[i] = 0.f;
#pragma unroll
        for (int x = 0; x < DIT; ++x) {
            float qq[8];
            load8(&qs[h][x * 64 + sub * 8], qq);
#pragma unroll
            for (int i = 0; i < TD_KEYS / 16; ++i)
#pragma unroll
                for (int e = 0; e < 8; ++e) s[i] = fmaf(qq[e], k[i][x][e], s[i]);
        }
#pragma unroll
        for (int i = 0; i < TD_KEYS / 16; ++i) {
#pragma unroll
            for (int o = 1; o < 8; o <<= 1) s[i] += __shfl_xor_sync(0xffffffffu, s[i], o);
            if (sub == 0) sc[h][i * 16 + (tid >> 3)] = s[i] * a.scale;
        }
    }
    __syncthreads();
    const int lane = tid & 31;
    for (int h = tid >> 5; h < group; h += 4) {
        const int head = g * group + h;
        float* to = a.scores + ((size_t)item * a.heads + head) * a.nsplit * TD_KEYS + u0;
        const float s0 = lane < n ? sc[h][lane] : -INFINITY, s1 = lane + 32 < n ? sc[h][lane + 32] : -INFINITY;
        if (lane < n) to[lane] = s0;
        if (lane + 32 < n) to[lane + 32] = s1;
        const float m = warp_max(fmaxf(s0, s1));
        const float l = warp_sum((s0 > -INFINITY ? expf(s0 - m) : 0.f) + (s1 > -INFINITY ? expf(s1 - m) : 0.f));
        if (lane == 0) {
            float* stats = a.stats + (((size_t)item * a.nsplit + split) * a.heads + head) * 2;
            stats[0] = m;
            stats[1] = l;
        }
    }
}

// grid (32 value columns, key/value heads, requests), 256 threads.
template <typename T>
__global__ void __launch_bounds__(256) talking_values_kernel(const TalkingDecodeArgs a) {
    extern __shared__ __align__(16) float td_smem[];
    const int group = a.heads / a.kv_heads, H = a.heads;
    float* talk = td_smem;                                  // [group][H]
    float* top = talk + group * H;                          // [H] maximum
    float* inv = top + H;                                   // [H] 1 / sum
    float* weight = inv + H;                                // [group][TD_TILE]
    __shared__ long long row[TD_TILE];
    const int c0 = blockIdx.x * TD_COLS, g = blockIdx.y, item = blockIdx.z;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const bool padding = a.item_slots[item] < 0 || a.item_qlen[item] <= 0;
    const SeenKeys seen(a, item);
    const int* table = a.block_tables + (size_t)item * a.table_stride;
    for (int i = tid; i < group * H; i += 256) talk[i] = a.talk[(size_t)g * group * H + i];
    grid_dependency_wait();
    grid_dependents_go();
    if (padding) return;
    const int splits = (seen.count + TD_KEYS - 1) / TD_KEYS;
    for (int h = warp; h < H; h += 8) {
        const float* stats = a.stats + ((size_t)item * a.nsplit * H + h) * 2;
        float m = -INFINITY, l = 0.f;
        for (int s = lane; s < splits; s += 32) m = fmaxf(m, stats[(size_t)s * H * 2]);
        m = warp_max(m);
        for (int s = lane; s < splits; s += 32) {
            const float ms = stats[(size_t)s * H * 2];
            if (ms > -INFINITY) l += stats[(size_t)s * H * 2 + 1] * expf(ms - m);
        }
        l = warp_sum(l);
        if (lane == 0) { top[h] = m; inv[h] = 1.0f / l; }
    }
    const float* scores = a.scores + (size_t)item * H * a.nsplit * TD_KEYS;
    const size_t head_ld = (size_t)a.nsplit * TD_KEYS;
    const T* pages = reinterpret_cast<const T*>(a.v_pages);
    const int col = c0 + 2 * (lane & 15), slice = warp * 2 + (lane >> 4);
    float acc[TD_GROUP][2];
#pragma unroll
    for (int h = 0; h < TD_GROUP; ++h) acc[h][0] = acc[h][1] = 0.f;
    for (int t0 = 0; t0 < seen.count; t0 += TD_TILE) {
        const int n = min(TD_TILE, seen.count - t0);
        __syncthreads();                                    // maxima and sums are there; the tile before is done with
        if (tid < n) {
            row[tid] = row_offset(a, table, seen.key(t0 + tid), g, a.vdim);
            float mix[TD_GROUP];
#pragma unroll
            for (int h = 0; h < TD_GROUP; ++h) mix[h] = 0.f;
#pragma unroll 8
            for (int h2 = 0; h2 < H; ++h2) {
                const float p = expf(scores[h2 * head_ld + t0 + tid] - top[h2]) * inv[h2];
#pragma unroll
                for (int h = 0; h < TD_GROUP; ++h) if (h < group) mix[h] += talk[h * H + h2] * p;
            }
#pragma unroll
            for (int h = 0; h < TD_GROUP; ++h) if (h < group) weight[h * TD_TILE + tid] = mix[h];
        }
        __syncthreads();
        if (col < a.vdim) {
#pragma unroll 8
            for (int j = slice; j < n; j += 16) {
                const long long at = row[j];
                float v0, v1;
                load_pair(pages + (at < 0 ? 0 : at) + col, v0, v1);
                if (at < 0) v0 = v1 = 0.f;                  // its page was given back: a row of zeros
#pragma unroll
                for (int h = 0; h < TD_GROUP; ++h)
                    if (h < group) {
                        const float p = weight[h * TD_TILE + j];
                        acc[h][0] = fmaf(p, v0, acc[h][0]);
                        acc[h][1] = fmaf(p, v1, acc[h][1]);
                    }
            }
        }
    }
    // the 16 slices' sums, added in order: [slice][group][32 columns] over the weights
    __syncthreads();
    float* parts = weight;                                  // 16 x group x 32 floats: room for 512 per head of the group
#pragma unroll
    for (int h = 0; h < TD_GROUP; ++h)
        if (h < group) {
            float* to = parts + (size_t)(slice * group + h) * TD_COLS + 2 * (lane & 15);
            to[0] = acc[h][0];
            to[1] = acc[h][1];
        }
    __syncthreads();
    for (int i = tid; i < group * TD_COLS; i += 256) {
        const int h = i / TD_COLS, c = c0 + i % TD_COLS;
        if (c >= a.vdim) continue;
        float sum = 0.f;
#pragma unroll
        for (int s = 0; s < 16; ++s) sum += parts[(size_t)s * group * TD_COLS + i];
        reinterpret_cast<T*>(a.out)[((size_t)a.item_qstart[item] * H + g * group + h) * a.vdim + c] = from_float<T>(sum);
    }
}

template <typename T>
static int launch_talking_decode(const TalkingDecodeArgs& a, int items, cudaStream_t stream) {
    const int group = a.heads / a.kv_heads;
    const dim3 grid(a.nsplit, a.kv_heads, items);
    int code;
    if (a.dim <= 64) code = launch_dependent(talking_scores_kernel<T, 1>, grid, 128, 0, stream, a);
    else if (a.dim <= 128) code = launch_dependent(talking_scores_kernel<T, 2>, grid, 128, 0, stream, a);
    else code = launch_dependent(talking_scores_kernel<T, 4>, grid, 128, 0, stream, a);
    if (code) return code;
    const size_t smem = ((size_t)group * a.heads + 2 * a.heads + (size_t)group * 16 * TD_COLS) * sizeof(float);
    return launch_dependent(talking_values_kernel<T>, dim3((a.vdim + TD_COLS - 1) / TD_COLS, a.kv_heads, items), 256, smem,
                            stream, a);
}

}  // namespace fsie

using namespace fsie;

extern "C" {

int fsie_talking_decode_keys() { return TD_KEYS; }

// One token per request: q [items, heads * dim] float, out [items, heads * vdim] of the storage type, both at item_qstart;
// scores [items, heads, nsplit * 64] and stats [items, nsplit, heads, 2] float, nsplit * 64 at least the
// keys that any of the tokens sees.  dim and vdim multiples of 8, up to 256 columns and 8 query heads per
// key/value head, rows of the pages on 16 bytes.
int fsie_talking_decode(const float* q, const void* k_pages, const void* v_pages, long long page_stride, int page_size,
                        const int* block_tables, int table_stride, const int* item_qstart, const int* item_qlen,
                        const int* item_pos0, const int* item_slots, int items, const float* talk, void* out, int heads,
                        int kv_heads, int dim, int vdim, int window, int keep_first, float scale, int* error, int nsplit,
                        float* scores, float* stats, int dtype, cudaStream_t stream) {
    if (items <= 0) return 0;
    if (heads <= 0 || kv_heads <= 0 || heads % kv_heads || window < 0 || keep_first < 0 || nsplit < 1 || page_size <= 0 ||
        !scores || !stats || items > 65535 || kv_heads > 65535)
        return ERR_BAD_ARGUMENT;
    const int per = dtype == DTYPE_F32 ? 4 : 8;
    if (heads / kv_heads > TD_GROUP || heads > 64 || dim <= 0 || vdim <= 0 || dim % 8 || vdim % 8 || dim > 256 || vdim > 256 ||
        page_stride % per || ((((size_t)k_pages) | ((size_t)v_pages)) & 15))
        return ERR_UNSUPPORTED;
    TalkingDecodeArgs a;
    a.q = q; a.k_pages = k_pages; a.v_pages = v_pages; a.page_stride = page_stride; a.page_size = page_size;
    a.block_tables = block_tables; a.table_stride = table_stride; a.item_qstart = item_qstart; a.item_qlen = item_qlen;
    a.item_pos0 = item_pos0; a.item_slots = item_slots; a.talk = talk; a.out = out; a.heads = heads; a.kv_heads = kv_heads;
    a.dim = dim; a.vdim = vdim; a.window = window; a.keep_first = keep_first; a.nsplit = nsplit; a.scale = scale;
    a.error = error; a.scores = scores; a.stats = stats;
    return dtype == DTYPE_F32 ? launch_talking_decode<float>(a, items, stream) : launch_talking_decode<bf16>(a, items, stream);
}

}  // extern "C"
