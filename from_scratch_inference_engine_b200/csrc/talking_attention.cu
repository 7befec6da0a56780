// Attention whose softmax weights are mixed across heads ("talking heads"), over a sliding
// window that also keeps the first tokens of the sequence, fed by projections that pass a
// short causal convolution, whole-projection RMS norms and an interleaved rotation.
//
//   prepare   u = conv(projected q | k | v)              y_t = sum_j w[:, j] u_{t - taps + 1 + j}
//             q = rot(rms(u_q) * w_q)   k = rot(rms(u_k) * w_k)     rms over the WHOLE projection
//             v_head = u_v,head / sqrt(mean(u_v,head^2) + eps)
//             q -> a 32-bit buffer; k, v -> the pages of the cache
//   tails     the last taps - 1 projected rows of every request -> its state slot
//   attend    (talking_attention.cuh)  s_h(i, j) = (q_h,i . k_g(h),j) * scale  for visible j:
//                 j <= i and (window == 0 or i - j < window or j < keep_first)
//             p_h = softmax_j s_h          p'_h = sum_h' talk[h, h'] p_h'
//             o_h,i = sum_j p'_h(i, j) v_g(h),j
//
// Positions, norms, scores, softmax and the mixed weights are 32-bit whatever the storage type
// T of the projections and the pages.  Page layout: keys [kv_head][slot][dim] at k_pages +
// page * page_stride, values [kv_head][slot][vdim] at v_pages + page * page_stride.
#include "common.cuh"

namespace fsie {

// index of the request that token t belongs to: item_qstart is ascending, requests are packed
__device__ __forceinline__ int item_of_token(const int* __restrict__ item_qstart, int items, int t) {
    int lo = 0, hi = items - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (item_qstart[mid] <= t) lo = mid; else hi = mid - 1;
    }
    return lo;
}

// ------------------------------------------------------------------------------ prepare
// One block per token.  `proj` [tokens, ld] holds q (wq columns), then k (wk), then v (wv);
// wk = wv = 0 for a layer that reads another layer's keys.  `tails` [slots, taps - 1, wq + wk +
// wv] holds the projected rows of the taps - 1 positions before the step's first token.
template <typename T>
__global__ void conv_norm_rotate_kernel(const T* __restrict__ proj, int ld, int items,
                                        const int* __restrict__ item_qstart,
                                        const int* __restrict__ item_pos0,
                                        const int* __restrict__ item_slots,
                                        const float* __restrict__ tails,
                                        const float* __restrict__ conv_w, int taps,
                                        const float* __restrict__ q_gain,
                                        const float* __restrict__ k_gain,
                                        const float* __restrict__ cos_sin, int table_len, int rot_dims,
                                        const int* __restrict__ slot_of, T* __restrict__ k_pages,
                                        T* __restrict__ v_pages, long long page_stride, int page_size,
                                        float* __restrict__ q_out, int heads, int kv_heads, int dim,
                                        int vdim, int has_kv, float eps, int* error) {
    extern __shared__ float y[];                       // the convolved row, then per-head value scales
    __shared__ float scratch[32];
    grid_dependency_wait();
    grid_dependents_go();
    const int t = blockIdx.x;
    const int item = item_of_token(item_qstart, items, t);
    const int slot = item_slots[item];
    if (slot < 0) return;                               // a padding entry of a fixed-size batch
    const int start = item_qstart[item], pos0 = item_pos0[item];
    const int pos = pos0 + (t - start);
    const int wq = heads * dim, wk = has_kv ? kv_heads * dim : 0, wv = has_kv ? kv_heads * vdim : 0;
    const int width = wq + wk + wv;
    const float* tail = tails ? tails + (size_t)slot * (taps - 1) * width : nullptr;
    float* v_scale = y + width;

    for (int c = threadIdx.x; c < width; c += blockDim.x) {
        float acc = 0.f;
        for (int j = 0; j < taps; ++j) {
            const int p = pos - taps + 1 + j;
            if (p < 0) continue;
            float u;
            if (p >= pos0) u = to_float(proj[(size_t)(start + p - pos0) * ld + c]);
            else u = tail[(size_t)(p - pos0 + taps - 1) * width + c];
            acc += conv_w[(size_t)c * taps + j] * u;
        }
        y[c] = acc;
    }
    __syncthreads();
    float sq = 0.f;
    for (int c = threadIdx.x; c < wq; c += blockDim.x) sq += y[c] * y[c];
    const float q_inv = 1.0f / sqrtf(block_sum(sq, scratch) / (float)wq + eps);
    float k_inv = 0.f;
    if (has_kv) {
        sq = 0.f;
        for (int c = threadIdx.x; c < wk; c += blockDim.x) sq += y[wq + c] * y[wq + c];
        k_inv = 1.0f / sqrtf(block_sum(sq, scratch) / (float)wk + eps);
        const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
        for (int g = warp; g < kv_heads; g += warps) {
            const float* head = y + wq + wk + g * vdim;
            float s = 0.f;
            for (int c = lane; c < vdim; c += 32) s += head[c] * head[c];
            s = warp_sum(s);
            if (lane == 0) v_scale[g] = 1.0f / sqrtf(s / (float)vdim + eps);
        }
    }
    __syncthreads();

    int table_pos = pos;
    if (rot_dims > 0 && (pos < 0 || pos >= table_len)) {
        if (threadIdx.x == 0) atomicExch(error, 2);
        table_pos = 0;
    }
    const int half = rot_dims / 2;
    const float* cs = cos_sin + (size_t)table_pos * rot_dims;      // [cos (half) | sin (half)]
    const int slot_kv = has_kv ? slot_of[t] : -1;
    const long long page = slot_kv >= 0 ? slot_kv / page_size : 0;
    const int offset = slot_kv >= 0 ? slot_kv - (int)page * page_size : 0;

    // q and k: normed with their gains, pairs (2i, 2i + 1) of the first rot_dims of a head turned
    for (int c = threadIdx.x; c < wq + wk; c += blockDim.x) {
        const bool is_q = c < wq;
        const int local = is_q ? c : c - wq;
        const int h = local / dim, d = local - h * dim;
        const float inv = is_q ? q_inv : k_inv;
        const float* gain = is_q ? q_gain : k_gain;
        float value = y[c] * inv * gain[local];
        if (d < rot_dims) {
            const int partner = (d & 1) ? c - 1 : c + 1;
            const int plocal = (d & 1) ? local - 1 : local + 1;
            const float other = y[partner] * inv * gain[plocal];
            const float co = cs[d >> 1], si = cs[half + (d >> 1)];
            value = (d & 1) ? value * co + other * si : value * co - other * si;
        }
        if (is_q) {
            q_out[(size_t)t * wq + c] = value;
        } else if (slot_kv >= 0) {
            k_pages[page * page_stride + ((size_t)h * page_size + offset) * dim + d] = from_float<T>(value);
        }
    }
    if (slot_kv >= 0) {
        for (int c = threadIdx.x; c < wv; c += blockDim.x) {
            const int g = c / vdim, d = c - g * vdim;
            v_pages[page * page_stride + ((size_t)g * page_size + offset) * vdim + d] =
                from_float<T>(y[wq + wk + c] * v_scale[g]);
        }
    }
}

// The same with eight neighbouring channels per thread, all of a row in one go (up to CONV_VEC_WIDTH channels): 16-byte loads,
// everything a row needs on its way at once (weights, gains, angles and lists before the kernel that makes
// the projection has finished).  A decode step's rows are few, so the chain of trips to memory is what it takes: with a
// channel per thread and turn, and the tails in a launch behind it, 4 tokens of 3,072 channels took 22 + 10 us of
// the step's chain, 6.8 now.  The squares are added up from shared memory as the general kernel's threads and warps
// do it, so that both leave the same bits.
// FOLD (every request brings one token): the row's own channels move the request's tail on as well, which conv_tails
// does otherwise (a longer portion's first tokens still read the old tail when its last one is done).
// Rows of up to 6,144 channels fit a block of 768 threads with the registers that eight channels of four taps take.  A prompt's rows are
// many, and there the chain counts less than how many rows an SM holds: two blocks of up to 384 threads, one of more.  With the
// tails' launch, general kernel and this one, us: 2,048 tokens of 3,072 channels 69 and 58, of 3,584 77 and 88, of 5,120 102
// and 108, of 6,144 121 and 122 to 130; 1,300 of 3,584 55 and 59, of 6,144 85 and 81; 700 of 3,584 37 and 37, of 6,144 58 and 51.
constexpr int CONV_VEC_WIDTH = 6144;
constexpr int CONV_VEC_SHARED = 3072;    // channels up to which two rows share an SM
constexpr int CONV_VEC_TOKENS = 1024;    // tokens up to which longer rows take this kernel all the same
__host__ __device__ constexpr int conv_threads(int width) { return width >= 1024 ? 512 : 256; }     // of the general kernel
template <typename T, int TAPS, bool FOLD>
__global__ void __launch_bounds__(CONV_VEC_WIDTH / 8)
conv_norm_rotate_vec_kernel(const T* __restrict__ proj, int ld, int items, const int* __restrict__ item_qstart,
                            const int* __restrict__ item_pos0, const int* __restrict__ item_slots,
                            float* tails, const float* __restrict__ conv_w,
                            const float* __restrict__ q_gain, const float* __restrict__ k_gain,
                            const float* __restrict__ cos_sin, int table_len, int rot_dims,
                            const int* __restrict__ slot_of, T* __restrict__ k_pages, T* __restrict__ v_pages,
                            long long page_stride, int page_size, float* __restrict__ q_out, int heads, int kv_heads,
                            int dim, int vdim, int has_kv, float eps, int* error) {
    __shared__ __align__(16) float all[CONV_VEC_WIDTH]; // the convolved row
    __shared__ float sums[2][16];                       // squares of q, of k: one for each warp of the general kernel
    extern __shared__ float v_scale[];                  // of every head's values
    const int t = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
    const int wq = heads * dim, wk = has_kv ? kv_heads * dim : 0, wv = has_kv ? kv_heads * vdim : 0;
    const int width = wq + wk + wv, c0 = threadIdx.x * 8;
    const bool active = c0 < width, is_q = c0 < wq, is_k = !is_q && c0 < wq + wk, is_v = active && !is_q && !is_k;
    // neither the lists nor the constants come from the kernel before
    const int item = item_of_token(item_qstart, items, t);
    const int slot = item_slots[item], start = item_qstart[item], pos0 = item_pos0[item], pos = pos0 + (t - start);
    const int slot_kv = has_kv && slot >= 0 ? slot_of[t] : -1;
    float w[TAPS * 8];                                  // [channel][tap]
    float gain[8], co[4], si[4];
    const int local = is_q ? c0 : c0 - wq, head = is_v ? (local - wk) / vdim : local / dim;
    const int d0 = is_v ? local - wk - head * vdim : local - head * dim;
    const bool refused = rot_dims > 0 && (pos < 0 || pos >= table_len);
    if (active) {
#pragma unroll
        for (int i = 0; i < TAPS; ++i) {
            float part[8];
            load8(conv_w + (size_t)c0 * TAPS + 8 * i, part);
#pragma unroll
            for (int e = 0; e < 8; ++e) w[8 * i + e] = part[e];
        }
        if (!is_v) {
            load8((is_q ? q_gain : k_gain) + local, gain);
            const float* cs = cos_sin + (size_t)(refused ? 0 : pos) * rot_dims;      // [cos (half) | sin (half)]
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const bool turned = d0 + 2 * i < rot_dims;
                co[i] = turned ? cs[d0 / 2 + i] : 1.f;
                si[i] = turned ? cs[rot_dims / 2 + d0 / 2 + i] : 0.f;
            }
        }
    }
    grid_dependency_wait();
    grid_dependents_go();
    if (slot < 0) return;                               // a padding entry of a fixed-size batch
    if (refused && threadIdx.x == 0) atomicExch(error, 2);
    float* tail = tails + (size_t)slot * (TAPS - 1) * width + c0;
    float u[TAPS][8], y[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) y[e] = 0.f;
    if (active) {
#pragma unroll
        for (int j = 0; j < TAPS; ++j) {
            const int p = pos - TAPS + 1 + j;
            if (p >= pos0) load8(proj + (size_t)(start + p - pos0) * ld + c0, u[j]);
            else load8(tail + (size_t)(p - pos0 + TAPS - 1) * width, u[j]);
        }
#pragma unroll
        for (int j = 0; j < TAPS; ++j) {
            if (pos - TAPS + 1 + j < 0) continue;       // before the sequence starts
#pragma unroll
            for (int e = 0; e < 8; ++e) y[e] += w[e * TAPS + j] * u[j][e];
        }
        if (FOLD) {
#pragma unroll
            for (int j = 1; j < TAPS; ++j) store8(tail + (size_t)(j - 1) * width, u[j]);
        }
        store8(all + c0, y);
    }
    __syncthreads();
    const int stride = conv_threads(width);
    for (int g = warp; g < stride / 32; g += warps) {
        float sq = 0.f;
        for (int c = g * 32 + lane; c < wq; c += stride) sq += all[c] * all[c];
        sq = warp_sum(sq);
        float sk = 0.f;
        for (int c = g * 32 + lane; c < wk; c += stride) sk += all[wq + c] * all[wq + c];
        sk = warp_sum(sk);
        if (lane == 0) { sums[0][g] = sq; sums[1][g] = sk; }
    }
    for (int g = warp; g < (has_kv ? kv_heads : 0); g += warps) {
        const float* values = all + wq + wk + g * vdim;
        float s = 0.f;
        for (int c = lane; c < vdim; c += 32) s += values[c] * values[c];
        s = warp_sum(s);
        if (lane == 0) v_scale[g] = 1.0f / sqrtf(s / (float)vdim + eps);
    }
    __syncthreads();
    if (!active) return;
    float inv;
    if (is_v) {
        inv = v_scale[head];
    } else {
        float total = 0.f;
        for (int i = 0; i < stride / 32; ++i) total += sums[is_k ? 1 : 0][i];
        inv = 1.0f / sqrtf(total / (float)(is_q ? wq : wk) + eps);
    }
    if (!is_v) {
#pragma unroll
        for (int e = 0; e < 8; ++e) y[e] = y[e] * inv * gain[e];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            if (d0 + 2 * i >= rot_dims) continue;
            const float a = y[2 * i], b = y[2 * i + 1];
            // which product is rounded is written out: the general kernel's, and so its bits
            y[2 * i] = fmaf(a, co[i], -__fmul_rn(b, si[i]));
            y[2 * i + 1] = fmaf(b, co[i], __fmul_rn(a, si[i]));
        }
        if (is_q) {
            store8(q_out + (size_t)t * wq + c0, y);
            return;
        }
    } else {
#pragma unroll
        for (int e = 0; e < 8; ++e) y[e] *= inv;
    }
    if (slot_kv < 0) return;
    const long long page = slot_kv / page_size;
    const int offset = slot_kv - (int)page * page_size, row = is_v ? vdim : dim;
    store8((is_v ? v_pages : k_pages) + page * page_stride + ((size_t)head * page_size + offset) * row + d0, y);
}

// ------------------------------------------------------------------------------- tails
// One block per request: row r of its new tail is the projected row of position
// end - (taps - 1) + r, which is a row of this step or, when the step brought fewer than
// taps - 1 tokens, row r + count of the old tail (read before anything overwrites it: a thread
// owns a channel and moves upwards).
template <typename T>
__global__ void conv_tails_kernel(const T* __restrict__ proj, int ld, const int* __restrict__ item_qstart,
                                  const int* __restrict__ item_qlen, const int* __restrict__ item_slots,
                                  float* __restrict__ tails, int taps, int width) {
    grid_dependency_wait();
    grid_dependents_go();
    const int item = blockIdx.x;
    const int slot = item_slots[item];
    if (slot < 0) return;
    const int start = item_qstart[item], count = item_qlen[item], keep = taps - 1;
    float* tail = tails + (size_t)slot * keep * width;
    for (int c = threadIdx.x; c < width; c += blockDim.x) {
        for (int r = 0; r < keep; ++r) {
            const int back = keep - r;                  // how far before the end this row lies
            float u;
            if (back <= count) u = to_float(proj[(size_t)(start + count - back) * ld + c]);
            else u = tail[(size_t)(r + count) * width + c];
            tail[(size_t)r * width + c] = u;
        }
    }
}

}  // namespace fsie

using namespace fsie;

extern "C" {

// fold_tails != 0 (every request brings one token): the kernel also moves the requests' tails on where it can; *folded
// (host memory) says whether it does, else conv_tails has to follow.
int fsie_conv_norm_rotate(const void* proj, int ld, int tokens, int items, const int* item_qstart,
                          const int* item_pos0, const int* item_slots, float* tails,
                          const float* conv_w, int taps, const float* q_gain, const float* k_gain,
                          const float* cos_sin, int table_len, int rot_dims, const int* slot_of,
                          void* k_pages, void* v_pages, long long page_stride, int page_size,
                          float* q_out, int heads, int kv_heads, int dim, int vdim, int has_kv,
                          float eps, int dtype, int* error, int fold_tails, int* folded, int early, cudaStream_t stream) {
    if (folded) *folded = 0;
    if (tokens <= 0) return 0;
    if (items <= 0 || taps <= 0 || (taps > 1 && !tails) || rot_dims < 0 || rot_dims > dim || (rot_dims & 1) ||
        (fold_tails && (tokens != items || !folded)))
        return ERR_BAD_ARGUMENT;
    const int width = heads * dim + (has_kv ? kv_heads * (dim + vdim) : 0);
    const int per = dtype == DTYPE_F32 ? 4 : 8;
    const bool vec = taps >= 2 && taps <= 4 && dim % 8 == 0 && vdim % 8 == 0 && width <= CONV_VEC_WIDTH && ld % per == 0 &&
        (!has_kv || !k_pages || (page_stride % per == 0 && ((((size_t)k_pages) | ((size_t)v_pages)) & 15) == 0)) &&
        ((((size_t)proj) | ((size_t)tails) | ((size_t)conv_w) | ((size_t)q_gain) | ((size_t)k_gain) | ((size_t)q_out)) & 15) == 0;
    if (vec && (fold_tails || tokens <= CONV_VEC_TOKENS || width <= CONV_VEC_SHARED)) {
        const int threads = ((width / 8 + 31) / 32) * 32;
        if (folded) *folded = fold_tails;
#define FSIE_PREPARE_VEC(T, N, F)                                                                                       \
        launch_dependent_if(early, conv_norm_rotate_vec_kernel<T, N, F>, tokens, threads, kv_heads * sizeof(float), stream, (const T*)proj, ld, items, \
                         item_qstart, item_pos0, item_slots, tails, conv_w, q_gain, k_gain, cos_sin, table_len, rot_dims, \
                         slot_of, (T*)k_pages, (T*)v_pages, page_stride, page_size, q_out, heads, kv_heads, dim, vdim, \
                         has_kv, eps, error)
#define FSIE_PREPARE_TAPS(T)                                                                                            \
        switch (taps) {                                                                                                 \
            case 2: return fold_tails ? FSIE_PREPARE_VEC(T, 2, true) : FSIE_PREPARE_VEC(T, 2, false);                    \
            case 3: return fold_tails ? FSIE_PREPARE_VEC(T, 3, true) : FSIE_PREPARE_VEC(T, 3, false);                    \
            default: return fold_tails ? FSIE_PREPARE_VEC(T, 4, true) : FSIE_PREPARE_VEC(T, 4, false);                   \
        }
        if (dtype == DTYPE_F32) FSIE_PREPARE_TAPS(float)
        FSIE_PREPARE_TAPS(bf16)
#undef FSIE_PREPARE_TAPS
#undef FSIE_PREPARE_VEC
    }
    const size_t smem = (size_t)(width + kv_heads) * sizeof(float);
    if (smem > 200 * 1024) return ERR_UNSUPPORTED;
    const int threads = conv_threads(width);
    int code = 0;
#define FSIE_PREPARE(T)                                                                          \
    do {                                                                                         \
        if (smem > 48 * 1024)                                                                    \
            cudaFuncSetAttribute(conv_norm_rotate_kernel<T>,                                     \
                                 cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);       \
        code = launch_dependent(conv_norm_rotate_kernel<T>, tokens, threads, smem, stream,       \
            (const T*)proj, ld, items, item_qstart, item_pos0, item_slots, tails, conv_w, taps,  \
            q_gain, k_gain, cos_sin, table_len, rot_dims, slot_of, (T*)k_pages, (T*)v_pages,     \
            page_stride, page_size, q_out, heads, kv_heads, dim, vdim, has_kv, eps, error);      \
    } while (0)
    if (dtype == DTYPE_F32) FSIE_PREPARE(float);
    else FSIE_PREPARE(bf16);
#undef FSIE_PREPARE
    return code;
}

int fsie_conv_tails(const void* proj, int ld, const int* item_qstart, const int* item_qlen,
                    const int* item_slots, int items, float* tails, int taps, int width, int dtype,
                    cudaStream_t stream) {
    if (items <= 0 || taps <= 1) return 0;
    if (dtype == DTYPE_F32)
        return launch_dependent(conv_tails_kernel<float>, items, 256, 0, stream, (const float*)proj, ld,
                                item_qstart, item_qlen, item_slots, tails, taps, width);
    return launch_dependent(conv_tails_kernel<bf16>, items, 256, 0, stream, (const bf16*)proj, ld,
                            item_qstart, item_qlen, item_slots, tails, taps, width);
}

}  // extern "C"
