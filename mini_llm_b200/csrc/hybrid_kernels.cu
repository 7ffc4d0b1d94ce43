// Kernels of layers that run a softmax attention beside a linear recurrence, and of routed
// feed-forwards:
//   rotary_store      rotary positions (interleaved pairs, a frequency table, an amplitude) on the
//                     step's queries and keys, and the keys and values into their cache pages
//   capped_attention  causal attention over the paged cache with keys and values of different
//                     sizes, a tanh cap on the scores and query heads that share a key/value head;
//                     scores, softmax and the weighted sum of values in 32-bit
//   linear_recurrence S <- a_t S + k_t u_t^T per head with a_t and the write strength b_t per token:
//                     u_t = b_t v_t (state-space form) or u_t = b_t (v_t - (a_t S)^T k_t) (delta rule);
//                     read out after the write; gates, decays and the state in 32-bit
//   route / expert_up / expert_down   a router with sigmoid scores and the largest few experts per
//                     token, gated experts fed the token times its score, a shared expert with an
//                     output gate
//   scaled_add        x += a * u + b * v on the 32-bit residual stream
//   head_norm_store   queries and keys divided by their root mean square per head (no gain), and the
//                     keys and values into their cache pages
// capped_attention also takes a chunked mask (a query sees the keys of its own block of `chunk`
// positions only), a number of first keys that stay visible behind a window, and a gate per (token, head) whose sigmoid multiplies the head's result;
// linear_recurrence also takes a decay per key channel instead of one per head.
// Every kernel is templated on the element type of the activations (float: the true 32-bit path;
// bfloat16: the serving path) and is launched as a programmatic dependent of the kernel before it.
#include "common.cuh"
#include <type_traits>

#include "mma_tiles.cuh"

MLLM_DEFINE_ERROR_API(mllm_hybrid)

__device__ __forceinline__ float sigmoid_f(float z) { return 1.0f / (1.0f + expf(-z)); }
__device__ __forceinline__ float silu_f(float z) { return z / (1.0f + expf(-z)); }
__device__ __forceinline__ float softplus_f(float z) { return fmaxf(z, 0.0f) + log1pf(expf(-fabsf(z))); }

// ---------------------------------------------------------------------------
// Rotary positions and the cache store.  A row of `qkv` holds [q: heads * dim | k: kv_heads * dim |
// v: kv_heads * vdim] at the given column offsets.  Among the first rot_dims entries of every
// query and key head, (x[2i], x[2i+1]) turns by position * inv_freq[i]; cosine and sine are
// multiplied by `amplitude`.  Angles are taken in 64-bit, once per token and pair.  Queries and
// keys are rotated in place; keys and values then go to the token's place in the pages.
// ---------------------------------------------------------------------------
template <typename T>
__global__ void rotary_store_kernel(T* __restrict__ qkv, long ld, int k_off, int v_off, int heads, int kv_heads, int dim,
                                    int vdim, int rot_dims, const double* __restrict__ inv_freq, double amplitude,
                                    const int* __restrict__ positions, const int* __restrict__ token_item,
                                    const int* __restrict__ block_table, int max_blocks, int page_size,
                                    T* __restrict__ k_pages, T* __restrict__ v_pages, int writes) {
    // the angles and the token's place ahead of the wait: they come with the step's arrays
    dependents_may_start();
    extern __shared__ float turn[];              // [rot_dims / 2][2]: cosine, sine
    const int t = blockIdx.x;
    const int p = positions[t];
    const int half = rot_dims / 2;
    for (int i = threadIdx.x; i < half; i += blockDim.x) {
        double s, c;
        sincos((double)p * inv_freq[i], &s, &c);
        turn[2 * i] = (float)(c * amplitude);
        turn[2 * i + 1] = (float)(s * amplitude);
    }
    const int page = block_table[(long)token_item[t] * max_blocks + p / page_size];
    const long slot = (long)page * page_size + (p % page_size);
    wait_for_earlier_kernels();
    __syncthreads();
    T* row = behind_the_wait(qkv) + (long)t * ld;
    const int first = blockIdx.y * blockDim.x + threadIdx.x, step = gridDim.y * blockDim.x;      // (blockIdx.y: a share of the token's row)
    // queries and keys: pairs of the rotated part, then what passes unchanged
    const int pairs_per_head = dim / 2 + (dim & 1);
    for (int u = first; u < (heads + kv_heads) * pairs_per_head; u += step) {
        const int head = u / pairs_per_head, i = u % pairs_per_head;
        const bool is_key = head >= heads;
        T* x = is_key ? row + k_off + (long)(head - heads) * dim : row + (long)head * dim;
        float a = to_f32(x[2 * i]);
        float b = 2 * i + 1 < dim ? to_f32(x[2 * i + 1]) : 0.0f;
        if (i < half) {
            const float c = turn[2 * i], s = turn[2 * i + 1];
            const float ra = a * c - b * s, rb = b * c + a * s;
            a = ra, b = rb;
            x[2 * i] = from_f32<T>(a);
            x[2 * i + 1] = from_f32<T>(b);
        }
        if (is_key && writes) {
            T* dst = k_pages + (slot * kv_heads + (head - heads)) * dim;
            dst[2 * i] = from_f32<T>(a);
            if (2 * i + 1 < dim) dst[2 * i + 1] = from_f32<T>(b);
        }
    }
    if (writes)
        for (int c = first; c < kv_heads * vdim; c += step)
            v_pages[slot * kv_heads * vdim + c] = row[v_off + c];
}

extern "C" int mllm_hybrid_rotary_store(void* qkv, long ld, int k_off, int v_off, int heads, int kv_heads, int dim, int vdim,
                                        int rot_dims, const double* inv_freq, double amplitude, const int* positions,
                                        const int* token_item, const int* block_table, int max_blocks, int page_size,
                                        void* k_pages, void* v_pages, int writes, int n_tokens, int dtype, void* stream) {
    if (n_tokens <= 0) return 0;
    if (rot_dims < 0 || rot_dims % 2 != 0 || rot_dims > dim) return fail("rotary_store: an even number of at most dim entries is rotated");
    cudaStream_t s = (cudaStream_t)stream;
    const size_t shared = (size_t)(rot_dims + 2) * sizeof(float);
    // few tokens: a thread a pair (16 heads of 64 by one block of 128 threads are four trips to L2 one after the other, as a
    // store may be what the next load reads)
    const int shares = n_tokens <= 64 ? ((heads + kv_heads) * ((dim + 1) / 2) + 127) / 128 : 1;
    const dim3 grid(n_tokens, shares < 64 ? shares : 64);
    if (dtype == DT_F32)
        launch_kernel(g_dependent_launch != 0, rotary_store_kernel<float>, grid, dim3(128), shared, s, (float*)qkv, ld,
                      k_off, v_off, heads, kv_heads, dim, vdim, rot_dims, inv_freq, amplitude, positions, token_item, block_table,
                      max_blocks, page_size, (float*)k_pages, (float*)v_pages, writes);
    else if (dtype == DT_BF16)
        launch_kernel(g_dependent_launch != 0, rotary_store_kernel<bf16>, grid, dim3(128), shared, s, (bf16*)qkv, ld,
                      k_off, v_off, heads, kv_heads, dim, vdim, rot_dims, inv_freq, amplitude, positions, token_item, block_table,
                      max_blocks, page_size, (bf16*)k_pages, (bf16*)v_pages, writes);
    else
        return fail("rotary_store: unknown dtype");
    return check_launch("rotary_store_kernel");
}

// ---------------------------------------------------------------------------
// Queries and keys over their root mean square, per head and without a gain:
// x / sqrt(mean(x^2) + eps) over the head's `dim` entries, in place; the normed keys and the values
// then go to the token's place in the pages.  A row of `qkv` is laid out as for rotary_store.  One
// block per token, a warp per head in turn; sums in 32-bit.
// ---------------------------------------------------------------------------
template <typename T>
__global__ void __launch_bounds__(128)
head_norm_store_kernel(T* __restrict__ qkv, long ld, int k_off, int v_off, int heads, int kv_heads, int dim, int vdim,
                       float eps, const int* __restrict__ positions, const int* __restrict__ token_item,
                       const int* __restrict__ block_table, int max_blocks, int page_size, T* __restrict__ k_pages,
                       T* __restrict__ v_pages, int writes) {
    dependents_may_start();
    const int t = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int p = positions[t];
    long slot = 0;
    if (writes) slot = (long)block_table[(long)token_item[t] * max_blocks + p / page_size] * page_size + (p % page_size);
    wait_for_earlier_kernels();                      // (the token's place comes with the step's arrays)
    T* row = behind_the_wait(qkv) + (long)t * ld;
    for (int head = blockIdx.y * 4 + warp; head < heads + kv_heads; head += gridDim.y * 4) {
        const bool is_key = head >= heads;
        T* x = is_key ? row + k_off + (long)(head - heads) * dim : row + (long)head * dim;
        float sq = 0.0f;
        for (int d = lane; d < dim; d += 32) {
            const float v = to_f32(x[d]);
            sq = fmaf(v, v, sq);
        }
        const float inv = eps >= 0.0f ? 1.0f / sqrtf(warp_sum(sq) / (float)dim + eps) : 1.0f;      // (eps < 0: stored as they are)
        T* dst = k_pages + (slot * kv_heads + (head - heads)) * dim;
        for (int d = lane; d < dim; d += 32) {
            const T v = from_f32<T>(to_f32(x[d]) * inv);
            x[d] = v;
            if (is_key && writes) dst[d] = v;
        }
    }
    if (writes)
        for (int c = blockIdx.y * blockDim.x + threadIdx.x; c < kv_heads * vdim; c += gridDim.y * blockDim.x) v_pages[slot * kv_heads * vdim + c] = row[v_off + c];
}

extern "C" int mllm_hybrid_head_norm_store(void* qkv, long ld, int k_off, int v_off, int heads, int kv_heads, int dim, int vdim,
                                           float eps, const int* positions, const int* token_item, const int* block_table,
                                           int max_blocks, int page_size, void* k_pages, void* v_pages, int writes, int n_tokens,
                                           int dtype, void* stream) {
    if (n_tokens <= 0) return 0;
    if (heads <= 0 || kv_heads <= 0 || dim <= 0 || vdim <= 0) return fail("head_norm_store: sizes must be positive");
    cudaStream_t s = (cudaStream_t)stream;
    // few tokens: a warp a head (the heads of one token one after the other took 5.9 us in a decode step of one token)
    const int shares = n_tokens <= 64 ? (heads + kv_heads + 3) / 4 : 1;
    const dim3 grid(n_tokens, shares < 64 ? shares : 64);
    if (dtype == DT_F32)
        launch_kernel(g_dependent_launch != 0, head_norm_store_kernel<float>, grid, dim3(128), 0, s, (float*)qkv, ld, k_off,
                      v_off, heads, kv_heads, dim, vdim, eps, positions, token_item, block_table, max_blocks, page_size,
                      (float*)k_pages, (float*)v_pages, writes);
    else if (dtype == DT_BF16)
        launch_kernel(g_dependent_launch != 0, head_norm_store_kernel<bf16>, grid, dim3(128), 0, s, (bf16*)qkv, ld, k_off,
                      v_off, heads, kv_heads, dim, vdim, eps, positions, token_item, block_table, max_blocks, page_size,
                      (bf16*)k_pages, (bf16*)v_pages, writes);
    else
        return fail("head_norm_store: unknown dtype");
    return check_launch("head_norm_store_kernel");
}

// ---------------------------------------------------------------------------
// Causal attention with capped scores, one block per (token, head): the plain form, which takes
// every size.  score = cap * tanh((q . k) * scale / cap) (cap <= 0: no cap); the query at position
// p sees keys max(0, p - window + 1) .. p (window <= 0: all) and those below `keep`.  With `slopes` [heads] a bias
// by distance comes off the (capped) score: slopes[h] * (p - j) for key j.  `gate` opens the result by a sigmoid: one number per head
// (gate[t, h]) or, with gate_wide, one per entry (gate[t, h * vdim + d]).  Four warps take the keys in turn,
// each with an online softmax; their states are merged in a fixed order.
// ---------------------------------------------------------------------------
constexpr int CAP_MAX_HEAD = 256;

__device__ __forceinline__ float capped(float s, float cap, float inv_cap) { return cap > 0.0f ? cap * tanhf(s * inv_cap) : s; }

// The first key the query at position p sees: the last `window` positions (window <= 0: all), and
// within its own block of `chunk` positions counted from 0 (chunk <= 0: no blocks).
__device__ __forceinline__ int first_visible(int p, int window, int chunk) {
    int lo = (window > 0 && p - window + 1 > 0) ? p - window + 1 : 0;
    if (chunk > 0) lo = max(lo, (p / chunk) * chunk);
    return lo;
}

// Keys below `keep` stay visible to every query after them, whatever the window.  A tile walk over a run's keys
// [0, keep) and [lo, p_last] starts at tile 0 if anything is kept and leaps from the kept tiles to the one that holds lo.
__device__ __forceinline__ bool key_visible(int j, int lo, int keep) { return j >= lo || j < keep; }
__device__ __forceinline__ int first_tile(int first_base, int keep) { return keep > 0 ? 0 : first_base; }
__device__ __forceinline__ int next_tile(int base, int step, int first_base, int keep) {
    base += step;
    return base >= keep && base < first_base ? first_base : base;
}

template <typename T>
__global__ void __launch_bounds__(128)
capped_attention_plain_kernel(T* __restrict__ out, long ld_out, const T* __restrict__ q, long ld_q,
                              const T* __restrict__ k_pages, const T* __restrict__ v_pages,
                              const int* __restrict__ block_table, int max_blocks, const int* __restrict__ positions,
                              const int* __restrict__ token_item, int n_heads, int n_kv_heads, int dim, int vdim,
                              int page_size, float scale, float cap, int window, int chunk, int keep,
                              const float* __restrict__ gate, long ld_gate, int gate_wide, const float* __restrict__ sink,
                              const float* __restrict__ slopes) {
    dependents_may_start();
    wait_for_earlier_kernels();
    constexpr int R = CAP_MAX_HEAD / 32;
    const int t = blockIdx.x, h = blockIdx.y;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int p = positions[t];
    const int* bt = block_table + (long)token_item[t] * max_blocks;
    const int hk = h / (n_heads / n_kv_heads);
    const float inv_cap = cap > 0.0f ? 1.0f / cap : 0.0f;
    float qr[R], acc[R];
#pragma unroll
    for (int i = 0; i < R; i++) {
        const int d = lane + 32 * i;
        qr[i] = d < dim ? to_f32(q[(long)t * ld_q + (long)h * dim + d]) : 0.0f;
        acc[i] = 0.0f;
    }
    float m = -INFINITY, l = 0.0f;
    const float slope = slopes != nullptr ? slopes[h] : 0.0f;
    const int lo = first_visible(p, window, chunk);
    const int n_kept = min(keep, lo);                        // kept keys ahead of the window, then the window's
    for (int i = warp; i <= p - lo + n_kept; i += 4) {
        const int j = i < n_kept ? i : i - n_kept + lo;
        const long slot = (long)bt[j / page_size] * page_size + (j % page_size);
        const T* kr = k_pages + (slot * n_kv_heads + hk) * dim;
        const T* vr = v_pages + (slot * n_kv_heads + hk) * vdim;
        float s = 0.0f;
#pragma unroll
        for (int i = 0; i < R; i++) {
            const int d = lane + 32 * i;
            if (d < dim) s = fmaf(qr[i], to_f32(kr[d]), s);
        }
        s = capped(warp_sum(s) * scale, cap, inv_cap) - slope * (float)(p - j);
        const float m_new = fmaxf(m, s);
        const float c = expf(m - m_new), e = expf(s - m_new);
        l = l * c + e;
#pragma unroll
        for (int i = 0; i < R; i++) {
            const int d = lane + 32 * i;
            if (d < vdim) acc[i] = acc[i] * c + e * to_f32(vr[d]);
        }
        m = m_new;
    }
    __shared__ float sm_m[4], sm_l[4];
    __shared__ float sm_acc[4][CAP_MAX_HEAD];
    if (lane == 0) sm_m[warp] = m, sm_l[warp] = l;
#pragma unroll
    for (int i = 0; i < R; i++) {
        const int d = lane + 32 * i;
        if (d < vdim) sm_acc[warp][d] = acc[i];
    }
    __syncthreads();
    float big = fmaxf(fmaxf(sm_m[0], sm_m[1]), fmaxf(sm_m[2], sm_m[3]));
    // a sink: one more term exp(sink[h]) in the denominator, with no key and no value
    if (sink != nullptr) big = fmaxf(big, sink[h]);
    float total = sink != nullptr ? expf(sink[h] - big) : 0.0f, wgt[4];
#pragma unroll
    for (int w = 0; w < 4; w++) {
        wgt[w] = sm_m[w] == -INFINITY ? 0.0f : expf(sm_m[w] - big);
        total += sm_l[w] * wgt[w];
    }
    for (int d = threadIdx.x; d < vdim; d += blockDim.x) {
        const float open = gate != nullptr ? sigmoid_f(gate[(long)t * ld_gate + (gate_wide ? h * vdim + d : h)]) : 1.0f;
        float o = 0.0f;
#pragma unroll
        for (int w = 0; w < 4; w++) o += sm_acc[w][d] * wgt[w];
        out[(long)t * ld_out + (long)h * vdim + d] = from_f32<T>(o / total * open);
    }
}

// ---------------------------------------------------------------------------
// The same attention in tiles, for steps with prompt portions.  A block takes consecutive tokens
// of the step and up to HC query heads of one key/value head: 8 * R (token, head) rows, R a warp
// (R = 2 or 4: a step with many rows lets more of them share a block's keys).  Tokens of
// one request that lie side by side share every block of 32 cached keys and values, which the
// block brings into shared memory once, in 32-bit, as 16-byte vectors asked for a block ahead.
// Within a warp the lanes take the 32 keys of a block for the scores (a key's entries are read
// once for all R rows) and the value entries for the weighted sum (a value's entry is read once
// for all R rows); scores, maxima, sums and weights are 32-bit.  A tile whose tokens belong to
// several requests takes the requests one after the other.
// ---------------------------------------------------------------------------
constexpr int TILE_KEYS = 32;
constexpr int TILE_WARPS = 8;

// sixteen bytes of activations as 32-bit floats into shared memory
template <typename T> __device__ __forceinline__ void widen(const uint4& v, float* dst);
template <> __device__ __forceinline__ void widen<float>(const uint4& v, float* dst) {
    *reinterpret_cast<float4*>(dst) = make_float4(__uint_as_float(v.x), __uint_as_float(v.y), __uint_as_float(v.z), __uint_as_float(v.w));
}
template <> __device__ __forceinline__ void widen<bf16>(const uint4& v, float* dst) {
    // a bfloat16 is the upper half of the float it stands for
    *reinterpret_cast<float4*>(dst) = make_float4(__uint_as_float(v.x << 16), __uint_as_float(v.x & 0xffff0000u),
                                                  __uint_as_float(v.y << 16), __uint_as_float(v.y & 0xffff0000u));
    *reinterpret_cast<float4*>(dst + 4) = make_float4(__uint_as_float(v.z << 16), __uint_as_float(v.z & 0xffff0000u),
                                                      __uint_as_float(v.w << 16), __uint_as_float(v.w & 0xffff0000u));
}

template <typename T, int R, int SIZE>      // rows a warp; the least of 64, 128, 256 that holds the key and the value size
__global__ void __launch_bounds__(TILE_WARPS * 32, R <= 4 && SIZE <= 128 ? 2 : 1)
capped_attention_tiled_kernel(T* __restrict__ out, long ld_out, const T* __restrict__ q, long ld_q,
                              const T* __restrict__ k_pages, const T* __restrict__ v_pages,
                              const int* __restrict__ block_table, int max_blocks, const int* __restrict__ positions,
                              const int* __restrict__ token_item, int n_tokens, int n_heads, int n_kv_heads, int dim,
                              int vdim, int page_size, float scale, float cap, int window, int chunk, int keep,
                              const float* __restrict__ gate, long ld_gate, int gate_wide, const float* __restrict__ sink,
                              const float* __restrict__ slopes, int tokens_per_block, int heads_per_block) {
    dependents_may_start();
    wait_for_earlier_kernels();
    constexpr int ROWS = TILE_WARPS * R;
    constexpr int VPL = SIZE / 32;                           // value entries a lane
    extern __shared__ float shared[];
    const int kd = dim + 4;                                  // padded key row: lanes read rows, four entries at a time
    float* q_rows = shared;                                  // [ROWS][dim]
    float* keys = q_rows + ROWS * dim;                       // [TILE_KEYS][kd]
    float* values = keys + TILE_KEYS * kd;                   // [TILE_KEYS][vdim]
    float* weights = values + TILE_KEYS * vdim;              // [TILE_WARPS][TILE_KEYS][R]
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int group = n_heads / n_kv_heads;
    const int chunks = (group + heads_per_block - 1) / heads_per_block;
    const int hk = blockIdx.y / chunks;
    const int first_head = hk * group + (blockIdx.y % chunks) * heads_per_block;
    const int n_heads_here = min(heads_per_block, hk * group + group - first_head);
    const int first_token = blockIdx.x * tokens_per_block;
    const int n_tok = min(tokens_per_block, n_tokens - first_token);
    const int n_rows = n_tok * n_heads_here;
    const float inv_cap = cap > 0.0f ? 1.0f / cap : 0.0f;

    // this warp's rows: r = warp + s * TILE_WARPS; row r = (token r / heads, head r % heads)
    int row_pos[R], row_item[R];
    float m[R], l[R], acc[R][VPL], slope[R];
#pragma unroll
    for (int s = 0; s < R; s++) {
        const int r = warp + s * TILE_WARPS;
        const bool live = r < n_rows;
        const int token = live ? first_token + r / n_heads_here : 0;
        row_pos[s] = live ? positions[token] : -1;
        row_item[s] = live ? token_item[token] : -1;
        slope[s] = live && slopes != nullptr ? slopes[first_head + r % n_heads_here] : 0.0f;
        m[s] = -INFINITY, l[s] = 0.0f;
#pragma unroll
        for (int i = 0; i < VPL; i++) acc[s][i] = 0.0f;
    }
    for (int u = threadIdx.x; u < n_rows * dim; u += blockDim.x) {
        const int r = u / dim, d = u % dim;
        q_rows[r * dim + d] = to_f32(q[(long)(first_token + r / n_heads_here) * ld_q + (long)(first_head + r % n_heads_here) * dim + d]);
    }

    // A block of 32 keys and values comes in 16-byte vectors, up to MAXV of each per thread; which
    // (key, column) a thread's vectors are is fixed for the kernel, so no division is left in the loop.
    constexpr int VEC = 16 / (int)sizeof(T);
    constexpr int MAXV = TILE_KEYS * SIZE / VEC / (TILE_WARPS * 32);
    uint4 key_vec[MAXV], value_vec[MAXV];
    int key_row[MAXV], key_col[MAXV], value_row[MAXV], value_col[MAXV];
#pragma unroll
    for (int i = 0; i < MAXV; i++) {
        const int u = threadIdx.x + i * TILE_WARPS * 32;
        key_row[i] = u < TILE_KEYS * (dim / VEC) ? u / (dim / VEC) : -1;
        key_col[i] = (u % (dim / VEC)) * VEC;
        value_row[i] = u < TILE_KEYS * (vdim / VEC) ? u / (vdim / VEC) : -1;
        value_col[i] = (u % (vdim / VEC)) * VEC;
        key_vec[i] = value_vec[i] = make_uint4(0, 0, 0, 0);
    }
    const int page_shift = (page_size & (page_size - 1)) == 0 ? 31 - __clz(page_size) : -1;
    auto fetch = [&](const int* bt, int base, int p_last, int p_lo) {
#pragma unroll
        for (int i = 0; i < MAXV; i++) {
            const int kp = base + key_row[i], vp = base + value_row[i];
            if (key_row[i] >= 0 && kp <= p_last && key_visible(kp, p_lo, keep)) {
                const int block = page_shift >= 0 ? kp >> page_shift : kp / page_size;
                const long slot = (long)bt[block] * page_size + (kp - block * page_size);
                key_vec[i] = *reinterpret_cast<const uint4*>(k_pages + (slot * n_kv_heads + hk) * dim + key_col[i]);
            }
            if (value_row[i] >= 0 && vp <= p_last && key_visible(vp, p_lo, keep)) {
                const int block = page_shift >= 0 ? vp >> page_shift : vp / page_size;
                const long slot = (long)bt[block] * page_size + (vp - block * page_size);
                value_vec[i] = *reinterpret_cast<const uint4*>(v_pages + (slot * n_kv_heads + hk) * vdim + value_col[i]);
            }
        }
    };

    float* my_weights = weights + warp * TILE_KEYS * R;
    int run_first = 0;
    while (run_first < n_tok) {
        // a run: consecutive tokens of the tile that belong to one request
        const int item = token_item[first_token + run_first];
        int run_last = run_first;
        while (run_last + 1 < n_tok && token_item[first_token + run_last + 1] == item) run_last++;
        const int p_first = positions[first_token + run_first], p_last = positions[first_token + run_last];
        const int lo = first_visible(p_first, window, chunk);
        const int* bt = block_table + (long)item * max_blocks;
        const int first_base = (lo / TILE_KEYS) * TILE_KEYS;
        int base = first_tile(first_base, keep), next = 0;
        fetch(bt, base, p_last, lo);                // (pages before the first visible key may be gone)
        for (; base <= p_last; base = next) {
            next = next_tile(base, TILE_KEYS, first_base, keep);
            __syncthreads();                                  // the block before has been read; q_rows are written
            const int n_keys = min(TILE_KEYS, p_last + 1 - base);
#pragma unroll
            for (int i = 0; i < MAXV; i++) {
                if (key_row[i] >= 0 && key_row[i] < n_keys) widen<T>(key_vec[i], keys + key_row[i] * kd + key_col[i]);
                if (value_row[i] >= 0 && value_row[i] < n_keys) widen<T>(value_vec[i], values + value_row[i] * vdim + value_col[i]);
            }
            __syncthreads();
            // the next block's rows are asked for now and arrive while this one is worked on
            if (next <= p_last) fetch(bt, next, p_last, lo);
            // which of the warp's rows see a key of this block at all
            bool any = false, seen[R];
            int first_seen[R];
#pragma unroll
            for (int s = 0; s < R; s++) {
                first_seen[s] = first_visible(row_pos[s], window, chunk);
                seen[s] = row_item[s] == item && base <= row_pos[s] && (base + TILE_KEYS > first_seen[s] || base < keep);
                any = any || seen[s];
            }
            if (!any) continue;                               // (uniform in the warp; the barriers are at the loop's head)
            // scores: this lane's key against the warp's rows, four entries at a time
            float dot[R];
#pragma unroll
            for (int s = 0; s < R; s++) dot[s] = 0.0f;
            const float* kr = keys + lane * kd;
#pragma unroll 2
            for (int d = 0; d < dim; d += 4) {
                const float4 b = *reinterpret_cast<const float4*>(kr + d);
#pragma unroll
                for (int s = 0; s < R; s++) {
                    const float4 a = *reinterpret_cast<const float4*>(q_rows + (warp + s * TILE_WARPS) * dim + d);
                    dot[s] = fmaf(a.x, b.x, dot[s]);
                    dot[s] = fmaf(a.y, b.y, dot[s]);
                    dot[s] = fmaf(a.z, b.z, dot[s]);
                    dot[s] = fmaf(a.w, b.w, dot[s]);
                }
            }
            const int pos = base + lane;
#pragma unroll
            for (int s = 0; s < R; s++) {
                const bool mine = seen[s] && lane < n_keys && pos <= row_pos[s] && key_visible(pos, first_seen[s], keep);
                const float score = mine ? capped(dot[s] * scale, cap, inv_cap) - slope[s] * (float)(row_pos[s] - pos) : -INFINITY;
                const float block_max = warp_max(score);
                float rescale = 1.0f, e = 0.0f;
                if (block_max != -INFINITY) {
                    const float m_new = fmaxf(m[s], block_max);
                    rescale = expf(m[s] - m_new);
                    e = mine ? expf(score - m_new) : 0.0f;
                    m[s] = m_new;
                }
                l[s] = l[s] * rescale + warp_sum(e);
#pragma unroll
                for (int i = 0; i < VPL; i++) acc[s][i] *= rescale;
                my_weights[lane * R + s] = e;
            }
            __syncwarp();
#pragma unroll 4
            for (int j = 0; j < n_keys; j++) {
                float w[R];
#pragma unroll
                for (int s = 0; s < R; s += 2) {
                    const float2 pair = *reinterpret_cast<const float2*>(my_weights + j * R + s);
                    w[s] = pair.x, w[s + 1] = pair.y;
                }
                const float* vr = values + j * vdim;
#pragma unroll
                for (int i = 0; i < VPL; i++) {
                    const int d = lane + 32 * i;
                    if (i + 1 < VPL || d < vdim) {
                        const float v = d < vdim ? vr[d] : 0.0f;
#pragma unroll
                        for (int s = 0; s < R; s++) acc[s][i] = fmaf(w[s], v, acc[s][i]);
                    }
                }
            }
            __syncwarp();
        }
        run_first = run_last + 1;
    }
#pragma unroll
    for (int s = 0; s < R; s++) {
        const int r = warp + s * TILE_WARPS;
        if (r >= n_rows) continue;
        const int token = first_token + r / n_heads_here, head = first_head + r % n_heads_here;
        float sum = l[s], shrink = 1.0f;
        if (sink != nullptr) {
            // the sink's term joins the denominator; the sums are rescaled if it is the largest
            const float top = fmaxf(m[s], sink[head]);
            shrink = expf(m[s] - top);
            sum = sum * shrink + expf(sink[head] - top);
        }
        const float inv = (gate != nullptr && !gate_wide ? sigmoid_f(gate[(long)token * ld_gate + head]) : 1.0f) * shrink / sum;
#pragma unroll
        for (int i = 0; i < VPL; i++) {
            const int d = lane + 32 * i;
            if (d >= vdim) continue;
            const float open = gate != nullptr && gate_wide ? sigmoid_f(gate[(long)token * ld_gate + (long)head * vdim + d]) : 1.0f;
            out[(long)token * ld_out + (long)head * vdim + d] = from_f32<T>(acc[s][i] * inv * open);
        }
    }
}

// ---------------------------------------------------------------------------
// The same attention as register tiles, for the common sizes (keys and values of up to 128 entries, no
// mask of blocks).  A block of 256 threads takes 64 (token, head) rows of one key/value head and walks
// the keys 64 at a time.  Thread (ty, tx) of a 16 x 16 grid holds the scores of rows 4 ty .. 4 ty + 3 against keys
// tx, tx + 16, tx + 32, tx + 48 (sixteen sums, fed by 16-byte reads of q and k rows along the head: eight FMAs a
// read), then, after the block's softmax step, the sums of those rows' values for columns 4 tx .. 4 tx + 3 (and
// 64 + 4 tx .. for values of 128): again sixteen (thirty-two) sums fed by 16-byte reads of the weights' rows and
// of the values' rows.  The sixteen threads of a row lie in one half of a warp: a row's maximum and sum are four
// shuffles, and its weights pass through shared memory between threads of one warp.  Scores, maxima, sums and
// weights are 32-bit.  Tokens of several requests in a tile are taken request by request, as in the kernel above.
// ---------------------------------------------------------------------------
constexpr int BLOCK_ROWS = 64, BLOCK_KEYS = 64;
constexpr int BLOCK_RT = 4;                                   // rows a thread (eight measured slower: 255 registers, one block fewer an SM)
constexpr int BLOCK_THREADS = 16 * BLOCK_ROWS / BLOCK_RT;

template <typename T, int VG>          // VG: 64-entry groups that hold a value (1 or 2; the last may be filled in part)
__global__ void __launch_bounds__(BLOCK_THREADS)
capped_attention_block_kernel(T* __restrict__ out, long ld_out, const T* __restrict__ q, long ld_q,
                              const T* __restrict__ k_pages, const T* __restrict__ v_pages,
                              const int* __restrict__ block_table, int max_blocks, const int* __restrict__ positions,
                              const int* __restrict__ token_item, int n_tokens, int n_heads, int n_kv_heads, int dim,
                              int vdim, int page_size, float scale, float cap, int window, int keep,
                              const float* __restrict__ gate, long ld_gate, int gate_wide, const float* __restrict__ sink,
                              const float* __restrict__ slopes, int tokens_per_block, int heads_per_block) {
    dependents_may_start();
    wait_for_earlier_kernels();
    constexpr int VDIM = 64 * VG;
    extern __shared__ float shared[];
    const int kd = dim + 4, vd = VDIM + 4, pd = BLOCK_KEYS + 4;
    float* q_rows = shared;                                  // [64][kd]
    float* keys = q_rows + BLOCK_ROWS * kd;                  // [64][kd]
    float* values = keys + BLOCK_KEYS * kd;                  // [64][vd]
    float* weights = values + BLOCK_KEYS * vd;               // [64][pd]
    int* row_pos = reinterpret_cast<int*>(weights + BLOCK_ROWS * pd);     // [64]
    int* row_item = row_pos + BLOCK_ROWS;                    // [64]
    float* row_slope = reinterpret_cast<float*>(row_item + BLOCK_ROWS);   // [64]
    const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
    const int group = n_heads / n_kv_heads;
    const int chunks = (group + heads_per_block - 1) / heads_per_block;
    const int hk = blockIdx.y / chunks;
    const int first_head = hk * group + (blockIdx.y % chunks) * heads_per_block;
    const int n_heads_here = min(heads_per_block, hk * group + group - first_head);
    // the step's last tokens first: within a request they see the most keys, and a long block that starts last would
    // leave the other SMs idle at the end
    const int first_token = (gridDim.x - 1 - blockIdx.x) * tokens_per_block;
    const int n_tok = min(tokens_per_block, n_tokens - first_token);
    const int n_rows = n_tok * n_heads_here;
    const float inv_cap = cap > 0.0f ? 1.0f / cap : 0.0f;
    constexpr int VEC = 16 / (int)sizeof(T);

    for (int r = tid; r < BLOCK_ROWS; r += blockDim.x) {
        const bool live = r < n_rows;
        const int token = live ? first_token + r / n_heads_here : 0;
        row_pos[r] = live ? positions[token] : -1;
        row_item[r] = live ? token_item[token] : -1;
        row_slope[r] = live && slopes != nullptr ? slopes[first_head + r % n_heads_here] : 0.0f;
    }
    for (int u = tid; u < BLOCK_ROWS * (dim / VEC); u += blockDim.x) {
        const int r = u / (dim / VEC), d = (u % (dim / VEC)) * VEC;
        uint4 v = make_uint4(0u, 0u, 0u, 0u);
        if (r < n_rows)
            v = *reinterpret_cast<const uint4*>(q + (long)(first_token + r / n_heads_here) * ld_q + (long)(first_head + r % n_heads_here) * dim + d);
        widen<T>(v, q_rows + r * kd + d);
    }
    __syncthreads();
    constexpr int RT = BLOCK_RT;
    int my_pos[RT], my_item[RT], my_first[RT];
    float m[RT], l[RT], o[RT][4 * VG];
#pragma unroll
    for (int i = 0; i < RT; i++) {
        my_pos[i] = row_pos[ty * RT + i], my_item[i] = row_item[ty * RT + i];
        my_first[i] = first_visible(my_pos[i], window, 0);
        m[i] = -INFINITY, l[i] = 0.0f;
#pragma unroll
        for (int c = 0; c < 4 * VG; c++) o[i][c] = 0.0f;
    }
    const int page_shift = (page_size & (page_size - 1)) == 0 ? 31 - __clz(page_size) : -1;
    // A tile of 64 keys and values comes in 16-byte vectors, a fixed few of each per thread, asked for a tile ahead;
    // which (key, column) a thread's vectors are is fixed for the kernel.
    constexpr int MAXK = BLOCK_KEYS * 128 / VEC / BLOCK_THREADS, MAXV = BLOCK_KEYS * VDIM / VEC / BLOCK_THREADS;
    uint4 key_vec[MAXK], value_vec[MAXV];
    int key_row[MAXK], key_col[MAXK], value_row[MAXV], value_col[MAXV];
#pragma unroll
    for (int i = 0; i < MAXK; i++) {
        const int u = tid + i * BLOCK_THREADS;
        key_row[i] = u < BLOCK_KEYS * (dim / VEC) ? u / (dim / VEC) : -1;
        key_col[i] = (u % (dim / VEC)) * VEC;
        key_vec[i] = make_uint4(0u, 0u, 0u, 0u);
    }
#pragma unroll
    for (int i = 0; i < MAXV; i++) {
        const int u = tid + i * BLOCK_THREADS;
        value_row[i] = u / (VDIM / VEC);
        value_col[i] = (u % (VDIM / VEC)) * VEC;             // (columns from vdim on stay zero)
        value_vec[i] = make_uint4(0u, 0u, 0u, 0u);
    }
    auto fetch = [&](const int* bt, int base, int p_last, int p_lo) {
#pragma unroll
        for (int i = 0; i < MAXK; i++) {
            const int kp = base + key_row[i];
            key_vec[i] = make_uint4(0u, 0u, 0u, 0u);
            if (key_row[i] >= 0 && kp <= p_last && key_visible(kp, p_lo, keep)) {      // (pages before the first visible key may be gone)
                const int block = page_shift >= 0 ? kp >> page_shift : kp / page_size;
                const long slot = (long)bt[block] * page_size + (kp - block * page_size);
                key_vec[i] = *reinterpret_cast<const uint4*>(k_pages + (slot * n_kv_heads + hk) * dim + key_col[i]);
            }
        }
#pragma unroll
        for (int i = 0; i < MAXV; i++) {
            const int vp = base + value_row[i];
            value_vec[i] = make_uint4(0u, 0u, 0u, 0u);
            if (value_col[i] < vdim && vp <= p_last && key_visible(vp, p_lo, keep)) {
                const int block = page_shift >= 0 ? vp >> page_shift : vp / page_size;
                const long slot = (long)bt[block] * page_size + (vp - block * page_size);
                value_vec[i] = *reinterpret_cast<const uint4*>(v_pages + (slot * n_kv_heads + hk) * vdim + value_col[i]);
            }
        }
    };

    int run_first = 0;
    while (run_first < n_tok) {
        const int item = token_item[first_token + run_first];
        int run_last = run_first;
        while (run_last + 1 < n_tok && token_item[first_token + run_last + 1] == item) run_last++;
        const int p_first = positions[first_token + run_first], p_last = positions[first_token + run_last];
        const int lo = first_visible(p_first, window, 0);
        const int* bt = block_table + (long)item * max_blocks;
        const int first_base = (lo / BLOCK_KEYS) * BLOCK_KEYS;
        int base = first_tile(first_base, keep), next = 0;
        fetch(bt, base, p_last, lo);
        for (; base <= p_last; base = next) {
            next = next_tile(base, BLOCK_KEYS, first_base, keep);
            __syncthreads();                                  // the tile before has been read
#pragma unroll
            for (int i = 0; i < MAXK; i++)
                if (key_row[i] >= 0) widen<T>(key_vec[i], keys + key_row[i] * kd + key_col[i]);
#pragma unroll
            for (int i = 0; i < MAXV; i++) widen<T>(value_vec[i], values + value_row[i] * vd + value_col[i]);
            __syncthreads();
            // the next tile's rows are asked for now and arrive while this one is worked on
            if (next <= p_last) fetch(bt, next, p_last, lo);
            // does any row of this warp see a key of this tile?
            bool any = false;
#pragma unroll
            for (int i = 0; i < RT; i++)
                any = any || (my_item[i] == item && base <= my_pos[i] && (base + BLOCK_KEYS > my_first[i] || base < keep));
            if (!__any_sync(0xffffffffu, any)) continue;      // (uniform in the warp; the barriers are at the loop's head)
            float acc[RT][4];
#pragma unroll
            for (int i = 0; i < RT; i++)
#pragma unroll
                for (int j = 0; j < 4; j++) acc[i][j] = 0.0f;
#pragma unroll 2
            for (int d = 0; d < dim; d += 4) {
                float4 a[RT], b[4];
#pragma unroll
                for (int i = 0; i < RT; i++) a[i] = *reinterpret_cast<const float4*>(q_rows + (ty * RT + i) * kd + d);
#pragma unroll
                for (int j = 0; j < 4; j++) b[j] = *reinterpret_cast<const float4*>(keys + (tx + 16 * j) * kd + d);
#pragma unroll
                for (int i = 0; i < RT; i++)
#pragma unroll
                    for (int j = 0; j < 4; j++) {
                        acc[i][j] = fmaf(a[i].x, b[j].x, acc[i][j]);
                        acc[i][j] = fmaf(a[i].y, b[j].y, acc[i][j]);
                        acc[i][j] = fmaf(a[i].z, b[j].z, acc[i][j]);
                        acc[i][j] = fmaf(a[i].w, b[j].w, acc[i][j]);
                    }
            }
#pragma unroll
            for (int i = 0; i < RT; i++) {
                const bool row_here = my_item[i] == item;
                const float slope = row_slope[ty * RT + i];
                float score[4], top = -INFINITY;
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    const int pos = base + tx + 16 * j;
                    const bool seen = row_here && pos <= my_pos[i] && key_visible(pos, my_first[i], keep);
                    score[j] = seen ? capped(acc[i][j] * scale, cap, inv_cap) - slope * (float)(my_pos[i] - pos) : -INFINITY;
                    top = fmaxf(top, score[j]);
                }
#pragma unroll
                for (int step = 8; step > 0; step >>= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, step));
                float rescale = 1.0f, e[4] = {0.0f, 0.0f, 0.0f, 0.0f}, sum = 0.0f;
                if (top != -INFINITY) {
                    const float m_new = fmaxf(m[i], top);
                    rescale = expf(m[i] - m_new);
#pragma unroll
                    for (int j = 0; j < 4; j++) {
                        e[j] = score[j] == -INFINITY ? 0.0f : expf(score[j] - m_new);
                        sum += e[j];
                    }
                    m[i] = m_new;
                }
#pragma unroll
                for (int step = 8; step > 0; step >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, step);
                l[i] = l[i] * rescale + sum;
#pragma unroll
                for (int c = 0; c < 4 * VG; c++) o[i][c] *= rescale;
#pragma unroll
                for (int j = 0; j < 4; j++) weights[(ty * RT + i) * pd + tx + 16 * j] = e[j];
            }
            __syncwarp();                                     // a row's sixteen threads lie in this warp
#pragma unroll 2
            for (int j = 0; j < BLOCK_KEYS; j += 4) {
                float4 w[RT];
#pragma unroll
                for (int i = 0; i < RT; i++) w[i] = *reinterpret_cast<const float4*>(weights + (ty * RT + i) * pd + j);
#pragma unroll
                for (int jj = 0; jj < 4; jj++) {
#pragma unroll
                    for (int g = 0; g < VG; g++) {
                        const float4 v = *reinterpret_cast<const float4*>(values + (j + jj) * vd + 64 * g + tx * 4);
#pragma unroll
                        for (int i = 0; i < RT; i++) {
                            const float p = jj == 0 ? w[i].x : (jj == 1 ? w[i].y : (jj == 2 ? w[i].z : w[i].w));
                            o[i][4 * g] = fmaf(p, v.x, o[i][4 * g]);
                            o[i][4 * g + 1] = fmaf(p, v.y, o[i][4 * g + 1]);
                            o[i][4 * g + 2] = fmaf(p, v.z, o[i][4 * g + 2]);
                            o[i][4 * g + 3] = fmaf(p, v.w, o[i][4 * g + 3]);
                        }
                    }
                }
            }
            __syncwarp();                                     // the weights are read before the next tile's are written
        }
        run_first = run_last + 1;
    }
#pragma unroll
    for (int i = 0; i < RT; i++) {
        const int r = ty * RT + i;
        if (r >= n_rows) continue;
        const int token = first_token + r / n_heads_here, head = first_head + r % n_heads_here;
        float sum = l[i], shrink = 1.0f;
        if (sink != nullptr) {
            const float top = fmaxf(m[i], sink[head]);
            shrink = expf(m[i] - top);
            sum = sum * shrink + expf(sink[head] - top);
        }
        const float inv = (gate != nullptr && !gate_wide ? sigmoid_f(gate[(long)token * ld_gate + head]) : 1.0f) * shrink / sum;
        const float* open = gate != nullptr && gate_wide ? gate + (long)token * ld_gate + (long)head * vdim : nullptr;
#pragma unroll
        for (int g = 0; g < VG; g++)
#pragma unroll
            for (int c = 0; c < 4; c++) {
                const int d = 64 * g + tx * 4 + c;
                if (d < vdim)
                    out[(long)token * ld_out + (long)head * vdim + d] =
                        from_f32<T>(o[i][4 * g + c] * inv * (open != nullptr ? sigmoid_f(open[d]) : 1.0f));
            }
    }
}

// ---------------------------------------------------------------------------
// The same attention on tensor-core tiles, bfloat16, keys and values of up to 128 entries (multiples of 8).  A block of eight
// warps takes 64 (token, head) rows of one key/value head and walks the keys 64 at a time, keys and values copied a tile ahead;
// warp w has rows 16 (w % 4) .. and keys 32 (w / 4) .. of every tile, and the two warps of a row group are merged at the end (four warps
// with all 64 keys left a scheduler one warp, whose products, exponentials and exchanges then stood one behind the other).  Scores are products of bfloat16 operands with 32-bit sums; the weights stay 32-bit: each goes into the
// second product as three bfloat16 terms, which hold all 24 bits of it, against the values as they are.  Maxima, sums,
// weights and results are 32-bit in the rows' threads, four threads a row; cap, slopes, masks, sink and gate as above.
// The products no longer bound it: a tile of 16 x 64 takes 128 of them (KEY 64, VALUE 64, three terms a weight) against 131,072 FMAs,
// 4,096 instructions of a warp, on register tiles, and the exponentials and masks stand beside them.
// Three prompts of 640, 1,200 and 2,048 tokens (12 heads over 4, sizes 64, capped): 480 us a launch on register tiles, 175 here (four warps 210).
// A tile's product is added with a rounded FMA: left in the tensor cores' accumulators, whose sums are cut off, the error against 64 bits
// was twice the register tiles'; so it is two thirds of theirs.
// ---------------------------------------------------------------------------
template <int KEY, int VALUE>          // entries of a key and of a value: 64 or 128, zeros past dim and vdim
__global__ void __launch_bounds__(256, KEY + VALUE == 128 ? 2 : 1)
capped_attention_mma_kernel(bf16* __restrict__ out, long ld_out, const bf16* q, long ld_q, const bf16* k_pages, const bf16* v_pages,
                            const int* block_table, int max_blocks, const int* positions, const int* token_item, int n_tokens,
                            int n_heads, int n_kv_heads, int dim, int vdim, int page_size, float scale, float cap, int window, int chunk,
                            int keep, const float* gate, long ld_gate, int gate_wide, const float* sink, const float* slopes,
                            int tokens_per_block, int heads_per_block) {
    constexpr int KEYS = 64, LDK = KEY + 8, LDV = VALUE + 8;           // rows an odd number of 16 bytes apart: no bank twice
    extern __shared__ __align__(16) unsigned char mma_shared[];
    bf16* q_rows = reinterpret_cast<bf16*>(mma_shared);               // [64][LDK]
    bf16* keys = q_rows + 64 * LDK;                                    // [2][64][LDK]
    bf16* values = keys + 2 * KEYS * LDK;                              // [2][64][LDV]
    __shared__ int row_pos[64], row_item[64];
    dependents_may_start();
    wait_for_earlier_kernels();
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, tq = lane & 3;
    const int quarter = warp & 3, half = warp >> 2;
    const int group = n_heads / n_kv_heads, chunks = (group + heads_per_block - 1) / heads_per_block;
    const int hk = blockIdx.y / chunks, first_head = hk * group + (blockIdx.y % chunks) * heads_per_block;
    const int n_heads_here = min(heads_per_block, hk * group + group - first_head);
    // (the step's last tokens first, as above)
    const int first_token = (gridDim.x - 1 - blockIdx.x) * tokens_per_block;
    const int n_tok = min(tokens_per_block, n_tokens - first_token), n_rows = n_tok * n_heads_here;
    const float inv_cap = cap > 0.0f ? 1.0f / cap : 0.0f;
    if (tid < 64) {
        const int token = tid < n_rows ? first_token + tid / n_heads_here : -1;
        row_pos[tid] = token >= 0 ? positions[token] : -1;
        row_item[tid] = token >= 0 ? token_item[token] : -1;
    }
    for (int u = tid; u < 64 * (KEY / 8); u += 256) {
        const int r = u / (KEY / 8), d = (u % (KEY / 8)) * 8;
        const bool there = r < n_rows && d < dim;
        const bf16* from = there ? q + (long)(first_token + r / n_heads_here) * ld_q + (long)(first_head + r % n_heads_here) * dim + d : q;
        copy_16(q_rows + r * LDK + d, from, there);
    }
    copies_end();
    copies_landed<0>();
    __syncthreads();
    uint32_t qa[KEY / 16][4];
#pragma unroll
    for (int k = 0; k < KEY / 16; k++) load_blocks(qa[k], q_rows + (quarter * 16 + (lane & 15)) * LDK + k * 16 + (lane >> 4) * 8);
    int my_pos[2], my_item[2], my_first[2];
    float my_slope[2], m[2] = {-INFINITY, -INFINITY}, l[2] = {0.0f, 0.0f}, o[VALUE / 8][4];
#pragma unroll
    for (int h = 0; h < 2; h++) {
        const int r = quarter * 16 + h * 8 + g;
        my_pos[h] = row_pos[r], my_item[h] = row_item[r], my_first[h] = first_visible(my_pos[h], window, chunk);
        my_slope[h] = r < n_rows && slopes != nullptr ? slopes[first_head + r % n_heads_here] : 0.0f;
    }
#pragma unroll
    for (int j = 0; j < VALUE / 8; j++) o[j][0] = o[j][1] = o[j][2] = o[j][3] = 0.0f;
    const int page_shift = (page_size & (page_size - 1)) == 0 ? 31 - __clz(page_size) : -1;

    int run_first = 0;
    while (run_first < n_tok) {
        const int item = token_item[first_token + run_first];
        int run_last = run_first;
        while (run_last + 1 < n_tok && token_item[first_token + run_last + 1] == item) run_last++;
        const int p_first = positions[first_token + run_first], p_last = positions[first_token + run_last];
        const int lo = first_visible(p_first, window, chunk);
        const int* bt = block_table + (long)item * max_blocks;
        const int first_base = (lo / KEYS) * KEYS;
        auto ask = [&](int base, int buffer) {
            bf16* into_k = keys + buffer * KEYS * LDK;
            bf16* into_v = values + buffer * KEYS * LDV;
            for (int u = tid; u < KEYS * (KEY / 8 + VALUE / 8); u += 256) {
                const bool value = u >= KEYS * (KEY / 8);
                const int v = value ? u - KEYS * (KEY / 8) : u, pieces = value ? VALUE / 8 : KEY / 8;
                const int j = v / pieces, d = (v % pieces) * 8, kp = base + j, size = value ? vdim : dim;
                // (pages before the first visible key may be gone)
                const bool there = d < size && kp <= p_last && key_visible(kp, lo, keep);
                const bf16* from = k_pages;
                if (there) {
                    const int block = page_shift >= 0 ? kp >> page_shift : kp / page_size;
                    const long slot = (long)bt[block] * page_size + (kp - block * page_size);
                    from = (value ? v_pages : k_pages) + (slot * n_kv_heads + hk) * size + d;
                }
                copy_16(value ? into_v + j * LDV + d : into_k + j * LDK + d, from, there);
            }
            copies_end();
        };
        int base = first_tile(first_base, keep), next = 0, buffer = 0;
        ask(base, 0);
        for (; base <= p_last; base = next, buffer ^= 1) {
            next = next_tile(base, KEYS, first_base, keep);
            // (the other buffer was left by every warp before the barrier that ended the last round)
            if (next <= p_last) ask(next, buffer ^ 1);
            else copies_end();
            copies_landed<1>();
            __syncthreads();
            const int key0 = base + half * 32;
            bool any = false;
#pragma unroll
            for (int h = 0; h < 2; h++)
                any = any || (my_item[h] == item && key0 <= my_pos[h] && (key0 + 32 > my_first[h] || key0 < keep));
            if (__any_sync(0xffffffffu, any)) {
                const bf16* kt = keys + (buffer * KEYS + half * 32) * LDK;
                const bf16* vt = values + (buffer * KEYS + half * 32) * LDV;
                float s[4][4];
#pragma unroll
                for (int j = 0; j < 4; j++) s[j][0] = s[j][1] = s[j][2] = s[j][3] = 0.0f;
#pragma unroll
                for (int k = 0; k < KEY / 16; k++)
#pragma unroll
                    for (int j = 0; j < 4; j += 2) {
                        uint32_t b[4];
                        load_blocks(b, kt + (j * 8 + (lane & 7) + ((lane >> 4) & 1) * 8) * LDK + k * 16 + ((lane >> 3) & 1) * 8);
                        mma_added(s[j], qa[k], b[0], b[1]);
                        mma_added(s[j + 1], qa[k], b[2], b[3]);
                    }
                float corr[2];
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    const bool row_here = my_item[h] == item;
                    float top = -INFINITY;
#pragma unroll
                    for (int j = 0; j < 4; j++)
#pragma unroll
                        for (int e = 0; e < 2; e++) {
                            const int pos = key0 + j * 8 + 2 * tq + e;
                            const bool seen = row_here && pos <= my_pos[h] && key_visible(pos, my_first[h], keep);
                            float& x = s[j][2 * h + e];
                            x = seen ? capped(x * scale, cap, inv_cap) - my_slope[h] * (float)(my_pos[h] - pos) : -INFINITY;
                            top = fmaxf(top, x);
                        }
                    top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 1));
                    top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 2));
                    const float m_new = fmaxf(m[h], top), from = m_new == -INFINITY ? 0.0f : m_new;
                    corr[h] = expf(m[h] - from);
                    float sum = 0.0f;
#pragma unroll
                    for (int j = 0; j < 4; j++)
#pragma unroll
                        for (int e = 0; e < 2; e++) {
                            s[j][2 * h + e] = expf(s[j][2 * h + e] - from);
                            sum += s[j][2 * h + e];
                        }
                    l[h] = l[h] * corr[h] + sum;             // this thread's share of the row
                    m[h] = m_new;
                }
                uint32_t a[2][3][4];
#pragma unroll
                for (int k = 0; k < 2; k++) weight_terms_of(a[k], s[2 * k], s[2 * k + 1]);
#pragma unroll
                for (int j = 0; j < VALUE / 8; j += 2) {
                    uint32_t b[2][4];
                    float x[2][4];
#pragma unroll
                    for (int k = 0; k < 2; k++)
                        load_blocks_turned(b[k], vt + (k * 16 + (lane & 7) + ((lane >> 3) & 1) * 8) * LDV + j * 8 + ((lane >> 4) & 1) * 8);
                    weighted_rows(x, a, b);
                    // (a row of another request keeps what it has: its weights of zero would carry a value that is no finite number into it)
#pragma unroll
                    for (int e = 0; e < 4; e++) {
                        if (my_item[e >> 1] != item) continue;
                        o[j][e] = fmaf(o[j][e], corr[e >> 1], x[0][e]);
                        o[j + 1][e] = fmaf(o[j + 1][e], corr[e >> 1], x[1][e]);
                    }
                }
            }
            __syncthreads();
        }
        copies_landed<0>();
        run_first = run_last + 1;
    }
    // the second half's states go through shared memory (the tiles are used up) to the first half's warps
    float* other = reinterpret_cast<float*>(mma_shared) + (quarter * 32 + lane) * (VALUE / 2 + 8);
#pragma unroll
    for (int h = 0; h < 2; h++) {
        l[h] += __shfl_xor_sync(0xffffffffu, l[h], 1);
        l[h] += __shfl_xor_sync(0xffffffffu, l[h], 2);
    }
    if (half == 1) {
#pragma unroll
        for (int j = 0; j < VALUE / 8; j++) *reinterpret_cast<float4*>(other + 4 * j) = make_float4(o[j][0], o[j][1], o[j][2], o[j][3]);
        *reinterpret_cast<float4*>(other + VALUE / 2) = make_float4(m[0], m[1], l[0], l[1]);
    }
    __syncthreads();
    if (half == 1) return;
    {
        const float4 state = *reinterpret_cast<const float4*>(other + VALUE / 2);
        const float m_other[2] = {state.x, state.y}, l_other[2] = {state.z, state.w};
        float mine[2], theirs[2];
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const float big = fmaxf(m[h], m_other[h]), from = big == -INFINITY ? 0.0f : big;
            mine[h] = expf(m[h] - from), theirs[h] = expf(m_other[h] - from);
            l[h] = fmaf(l[h], mine[h], l_other[h] * theirs[h]);
            m[h] = big;
        }
#pragma unroll
        for (int j = 0; j < VALUE / 8; j++) {
            const float4 x = *reinterpret_cast<const float4*>(other + 4 * j);
            o[j][0] = fmaf(o[j][0], mine[0], x.x * theirs[0]), o[j][1] = fmaf(o[j][1], mine[0], x.y * theirs[0]);
            o[j][2] = fmaf(o[j][2], mine[1], x.z * theirs[1]), o[j][3] = fmaf(o[j][3], mine[1], x.w * theirs[1]);
        }
    }
#pragma unroll
    for (int h = 0; h < 2; h++) {
        float sum = l[h];
        const int r = quarter * 16 + h * 8 + g;
        if (r >= n_rows) continue;
        const int token = first_token + r / n_heads_here, head = first_head + r % n_heads_here;
        float shrink = 1.0f;
        if (sink != nullptr) {
            const float top = fmaxf(m[h], sink[head]);
            shrink = expf(m[h] - top);
            sum = sum * shrink + expf(sink[head] - top);
        }
        const float inv = (gate != nullptr && !gate_wide ? sigmoid_f(gate[(long)token * ld_gate + head]) : 1.0f) * shrink / sum;
        const float* open = gate != nullptr && gate_wide ? gate + (long)token * ld_gate + (long)head * vdim : nullptr;
#pragma unroll
        for (int j = 0; j < VALUE / 8; j++)
#pragma unroll
            for (int e = 0; e < 2; e++) {
                const int d = j * 8 + 2 * tq + e;
                if (d < vdim)
                    out[(long)token * ld_out + (long)head * vdim + d] =
                        __float2bfloat16_rn(o[j][2 * h + e] * inv * (open != nullptr ? sigmoid_f(open[d]) : 1.0f));
            }
    }
}

// (rows of queries, keys and values in whole 16-byte pieces)
static bool capped_mma_takes(const void* q, long ld_q, const void* k_pages, const void* v_pages, int dim, int vdim) {
    return dim % 8 == 0 && vdim % 8 == 0 && dim <= 128 && vdim <= 128 && ld_q % 8 == 0 &&
           ((reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(k_pages) | reinterpret_cast<uintptr_t>(v_pages)) & 15) == 0;
}

static size_t capped_block_shared(int dim, int vdim) {
    return sizeof(float) * ((size_t)2 * BLOCK_ROWS * (dim + 4) + (size_t)BLOCK_KEYS * (vdim + 4) + (size_t)BLOCK_ROWS * (BLOCK_KEYS + 4)) +
           (2 * sizeof(int) + sizeof(float)) * BLOCK_ROWS;
}

// (keys and values in whole 16-byte vectors; values narrower than half their groups go to the tiles of few rows)
static bool capped_block_takes(int dim, int vdim, int vec) {
    return dim > 0 && dim <= 128 && dim % vec == 0 && dim % 4 == 0 && vdim > 32 && vdim <= 128 && vdim % vec == 0 && vdim % 4 == 0;
}

template <typename T, int VG>
static int launch_capped_block(void* out, long ld_out, const void* q, long ld_q, const void* k_pages, const void* v_pages,
                               const int* block_table, int max_blocks, const int* positions, const int* token_item, int n_tokens,
                               int n_heads, int n_kv_heads, int dim, int vdim, int page_size, float scale, float cap, int window,
                               int keep, const float* gate, long ld_gate, int gate_wide, const float* sink, const float* slopes,
                               cudaStream_t s) {
    const int group = n_heads / n_kv_heads;
    const int heads_per_block = group < BLOCK_ROWS ? group : BLOCK_ROWS;
    const int tokens_per_block = BLOCK_ROWS / heads_per_block;
    const int chunks = (group + heads_per_block - 1) / heads_per_block;
    const size_t shared = capped_block_shared(dim, 64 * VG);
    cudaError_t e = cudaFuncSetAttribute(capped_attention_block_kernel<T, VG>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)shared);
    if (e != cudaSuccess) return fail("capped_attention: the register tiles' shared memory was refused");
    cudaFuncSetAttribute(capped_attention_block_kernel<T, VG>, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
    dim3 grid((n_tokens + tokens_per_block - 1) / tokens_per_block, n_kv_heads * chunks);
    launch_kernel(AFTER_THE_KERNELS_AHEAD, capped_attention_block_kernel<T, VG>, grid, dim3(BLOCK_THREADS), shared, s, (T*)out, ld_out, (const T*)q,
                  ld_q, (const T*)k_pages, (const T*)v_pages, block_table, max_blocks, positions, token_item, n_tokens, n_heads,
                  n_kv_heads, dim, vdim, page_size, scale, cap, window, keep, gate, ld_gate, gate_wide, sink, slopes,
                  tokens_per_block, heads_per_block);
    return check_launch("capped_attention_block_kernel");
}

static size_t capped_tiled_shared(int dim, int vdim, int rows_per_warp) {
    return sizeof(float) * ((size_t)TILE_WARPS * rows_per_warp * dim + (size_t)TILE_KEYS * (dim + 4) + (size_t)TILE_KEYS * vdim +
                            (size_t)TILE_WARPS * TILE_KEYS * rows_per_warp);
}

// (keys and values in whole 16-byte vectors: sizes that are multiples of `vec` elements)
extern "C" int mllm_hybrid_capped_attention_tiled_takes(int dim, int vdim, int vec) {
    return dim > 0 && vdim > 0 && dim % vec == 0 && vdim % vec == 0 && dim % 4 == 0 && vdim % 4 == 0 && dim <= CAP_MAX_HEAD &&
           vdim <= CAP_MAX_HEAD && capped_tiled_shared(dim, vdim, 2) <= 160 * 1024;
}

template <typename T, int R, int SIZE>
static int launch_capped_tiles(void* out, long ld_out, const void* q, long ld_q, const void* k_pages, const void* v_pages,
                               const int* block_table, int max_blocks, const int* positions, const int* token_item, int n_tokens,
                               int n_heads, int n_kv_heads, int dim, int vdim, int page_size, float scale, float cap, int window,
                               int chunk, int keep, const float* gate, long ld_gate, int gate_wide, const float* sink,
                               const float* slopes, cudaStream_t s) {
    constexpr int ROWS = TILE_WARPS * R;
    const int group = n_heads / n_kv_heads;
    const int heads_per_block = group < ROWS ? group : ROWS;
    const int tokens_per_block = ROWS / heads_per_block;
    const int chunks = (group + heads_per_block - 1) / heads_per_block;
    const size_t shared = capped_tiled_shared(dim, vdim, R);
    cudaError_t e = cudaFuncSetAttribute(capped_attention_tiled_kernel<T, R, SIZE>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)shared);
    if (e != cudaSuccess) return fail("capped_attention: the tiles' shared memory was refused");
    // several blocks an SM: as much of the SM's memory as shared memory as they need
    cudaFuncSetAttribute(capped_attention_tiled_kernel<T, R, SIZE>, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
    dim3 grid((n_tokens + tokens_per_block - 1) / tokens_per_block, n_kv_heads * chunks);
    launch_kernel(AFTER_THE_KERNELS_AHEAD, capped_attention_tiled_kernel<T, R, SIZE>, grid, dim3(TILE_WARPS * 32), shared, s, (T*)out,
                  ld_out, (const T*)q, ld_q, (const T*)k_pages, (const T*)v_pages, block_table, max_blocks, positions, token_item,
                  n_tokens, n_heads, n_kv_heads, dim, vdim, page_size, scale, cap, window, chunk, keep, gate, ld_gate, gate_wide, sink,
                  slopes, tokens_per_block, heads_per_block);
    return check_launch("capped_attention_tiled_kernel");
}

template <typename T>
static int launch_capped_attention(bool tiled, void* out, long ld_out, const void* q, long ld_q, const void* k_pages,
                                   const void* v_pages, const int* block_table, int max_blocks, const int* positions,
                                   const int* token_item, int n_tokens, int n_heads, int n_kv_heads, int dim, int vdim,
                                   int page_size, float scale, float cap, int window, int chunk, int keep, const float* gate,
                                   long ld_gate, int gate_wide, const float* sink, const float* slopes, cudaStream_t s) {
    if (!tiled) {
        launch_kernel(g_dependent_launch != 0, capped_attention_plain_kernel<T>, dim3(n_tokens, n_heads), dim3(128), 0, s, (T*)out,
                      ld_out, (const T*)q, ld_q, (const T*)k_pages, (const T*)v_pages, block_table, max_blocks, positions,
                      token_item, n_heads, n_kv_heads, dim, vdim, page_size, scale, cap, window, chunk, keep, gate, ld_gate, gate_wide,
                      sink, slopes);
        return check_launch("capped_attention_plain_kernel");
    }
    // bfloat16 of the common sizes goes to the tensor-core tiles
    if constexpr (sizeof(T) == 2) {
        if (capped_mma_takes(q, ld_q, k_pages, v_pages, dim, vdim)) {
            // A block walks the keys of every request among its tokens, one request behind the other: fewer tokens a block while the
            // blocks are no more than half the SMs, or tokens that stand alone beside a short portion wait for one another (20 of 600
            // keys beside a portion of 60, 12 heads over 4: 631 us with 21 tokens a block, 78 with 2; a prompt of 300 23.1 and 22.0).
            const int group = n_heads / n_kv_heads, heads_per_block = group < 64 ? group : 64;
            const int head_blocks = n_kv_heads * ((group + heads_per_block - 1) / heads_per_block);
            int tokens_per_block = 64 / heads_per_block;
            while (tokens_per_block > 1 && (long)((n_tokens + tokens_per_block - 1) / tokens_per_block) * head_blocks * 2 <= 148) tokens_per_block /= 2;
            const int key = dim <= 64 ? 64 : 128, value = vdim <= 64 ? 64 : 128;
            const size_t shared = sizeof(bf16) * (size_t)(192 * (key + 8) + 128 * (value + 8));
            const dim3 grid((n_tokens + tokens_per_block - 1) / tokens_per_block, head_blocks);
#define CAPPED_MMA(KEY, VALUE)                                                                                                    \
    do {                                                                                                                          \
        if (cudaFuncSetAttribute(capped_attention_mma_kernel<KEY, VALUE>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)shared) !=  \
            cudaSuccess)                                                                                                          \
            return fail("capped_attention: the tiles' shared memory was refused");                                               \
        cudaFuncSetAttribute(capped_attention_mma_kernel<KEY, VALUE>, cudaFuncAttributePreferredSharedMemoryCarveout,             \
                             cudaSharedmemCarveoutMaxShared);                                                                     \
        launch_kernel(AFTER_THE_KERNELS_AHEAD, capped_attention_mma_kernel<KEY, VALUE>, grid, dim3(256), shared, s, (bf16*)out, ld_out,  \
                      (const bf16*)q, ld_q, (const bf16*)k_pages, (const bf16*)v_pages, block_table, max_blocks, positions, token_item, \
                      n_tokens, n_heads, n_kv_heads, dim, vdim, page_size, scale, cap, window, chunk, keep, gate, ld_gate, gate_wide, sink, \
                      slopes, tokens_per_block, heads_per_block);                                                                 \
        return check_launch("capped_attention_mma_kernel");                                                                       \
    } while (0)
            if (key == 64 && value == 64) CAPPED_MMA(64, 64);
            if (key == 64) CAPPED_MMA(64, 128);
            if (value == 64) CAPPED_MMA(128, 64);
            CAPPED_MMA(128, 128);
#undef CAPPED_MMA
        }
    }
    // 32-bit rows of the common sizes go to the register tiles
    if constexpr (sizeof(T) == 4) if (chunk == 0 && n_tokens * (long)n_heads >= 2048 && capped_block_takes(dim, vdim, 16 / (int)sizeof(T)) &&
        (ld_q * sizeof(T)) % 16 == 0) {
        if (vdim <= 64)
            return launch_capped_block<T, 1>(out, ld_out, q, ld_q, k_pages, v_pages, block_table, max_blocks, positions, token_item,
                                             n_tokens, n_heads, n_kv_heads, dim, vdim, page_size, scale, cap, window, keep, gate, ld_gate,
                                             gate_wide, sink, slopes, s);
        return launch_capped_block<T, 2>(out, ld_out, q, ld_q, k_pages, v_pages, block_table, max_blocks, positions, token_item,
                                         n_tokens, n_heads, n_kv_heads, dim, vdim, page_size, scale, cap, window, keep, gate, ld_gate,
                                             gate_wide, sink, slopes, s);
    }
    // rows a warp: four where the step has rows enough for the blocks to fill the GPU all the same
    // (and their shared memory fits), else two
    const long rows = (long)n_tokens * n_heads;
    int per_warp = rows >= 8192 ? 4 : 2;
    if (capped_tiled_shared(dim, vdim, per_warp) > 160 * 1024) per_warp = 2;
#define TILES(R, SIZE)                                                                                                        \
    return launch_capped_tiles<T, R, SIZE>(out, ld_out, q, ld_q, k_pages, v_pages, block_table, max_blocks, positions, token_item, \
                                           n_tokens, n_heads, n_kv_heads, dim, vdim, page_size, scale, cap, window, chunk, keep, gate, ld_gate, gate_wide, \
                                           sink, slopes, s)
    const int size = (dim > vdim ? dim : vdim) <= 64 ? 64 : ((dim > vdim ? dim : vdim) <= 128 ? 128 : 256);
    if (per_warp == 4) { if (size == 64) TILES(4, 64); if (size == 128) TILES(4, 128); TILES(4, 256); }
    if (size == 64) TILES(2, 64);
    if (size == 128) TILES(2, 128);
    TILES(2, 256);
#undef TILES
}

extern "C" int mllm_hybrid_capped_attention(void* out, long ld_out, const void* q, long ld_q, const void* k_pages,
                                            const void* v_pages, const int* block_table, int max_blocks, const int* positions,
                                            const int* token_item, int n_tokens, int n_heads, int n_kv_heads, int dim, int vdim,
                                            int page_size, float scale, float cap, int window, int chunk, int keep, const float* gate,
                                            long ld_gate, int gate_wide, const float* sink, const float* slopes, int tiled, int dtype,
                                            void* stream) {
    if (n_tokens <= 0) return 0;
    if (dim <= 0 || dim > CAP_MAX_HEAD || vdim <= 0 || vdim > CAP_MAX_HEAD) return fail("capped_attention: key and value sizes must be in 1..256");
    if (n_kv_heads <= 0 || n_heads % n_kv_heads != 0) return fail("capped_attention: heads must be a multiple of the key/value heads");
    if (n_heads > 65535) return fail("capped_attention: too many heads for one launch");
    if (keep < 0 || (keep > 0 && chunk > 0)) return fail("capped_attention: kept first keys go with a window, not with blocks of positions");
    if (tiled && !mllm_hybrid_capped_attention_tiled_takes(dim, vdim, dtype == DT_F32 ? 4 : 8)) return fail("capped_attention: the tiles do not take these sizes");
    cudaStream_t s = (cudaStream_t)stream;
    if (dtype == DT_F32)
        return launch_capped_attention<float>(tiled != 0, out, ld_out, q, ld_q, k_pages, v_pages, block_table, max_blocks, positions,
                                              token_item, n_tokens, n_heads, n_kv_heads, dim, vdim, page_size, scale, cap, window, chunk, keep,
                                              gate, ld_gate, gate_wide, sink, slopes, s);
    if (dtype == DT_BF16)
        return launch_capped_attention<bf16>(tiled != 0, out, ld_out, q, ld_q, k_pages, v_pages, block_table, max_blocks, positions,
                                             token_item, n_tokens, n_heads, n_kv_heads, dim, vdim, page_size, scale, cap, window, chunk, keep,
                                             gate, ld_gate, gate_wide, sink, slopes, s);
    return fail("capped_attention: unknown dtype");
}

// ---------------------------------------------------------------------------
// Linear recurrence with a matrix state per head, S [dim, vdim] in 32-bit:
//   a_t = exp(-exp(log_rate[h]) * step_t),  step_t = softplus(gate_a[t, h] + step_bias[h])
//   state-space form:  b_t = step_t;               u_t = b_t v_t
//   delta rule:        b_t = sigmoid(gate_b[t, h]); u_t = b_t (v_t - (a_t S)^T k_t)
//   S <- a_t S + k_t u_t^T;   out_t = S^T q_t (+ skip[h] v_t)
// Query/key head of head h: h / (heads / qk_heads).  With unit_norm, q and k are divided by
// sqrt(sum(x^2) + 1e-6) per head first; q is multiplied by q_scale.
// With channel_decay the decay is one per key channel instead: gate_a [T, heads * dim] and step_bias
// [heads * dim], a_t[i] = exp(-exp(log_rate[h]) * softplus(gate_a[t, h, i] + step_bias[h, i])), and row i of S
// is multiplied by a_t[i] before the old column is read: S <- diag(a_t) S; u_t = b_t (v_t - S^T k_t);
// S <- S + k_t u_t^T.
// One block per (entry, head, slice of the value entries): a column of S belongs to LANES threads
// of one warp, each with DPT rows in registers; both sums over the old column (with k and with q)
// are taken in one pass, and the read-out follows from them: S_new^T q = a S^T q + u (k . q).
// The entry's tokens are taken in order, TOK at a time through shared memory, by four warps; four others
// ask for the chunk after next into registers and prepare the next one (decays, gates, unit vectors) meanwhile.  What bounds it are
// instructions, some 180 a token for the walk and 2,000 a chunk for what comes before: 700 tokens of 6 heads of 128 x 128 with a decay per
// channel 319 us when the same four warps did both in turn, 239 so; 2 x 350 163 and 124; 100 tokens in 32 bits 42 and 36.
// ---------------------------------------------------------------------------
struct RecurrenceParams {
    float* out; long ld_out;
    const void* q; const void* k; const void* v; long ld_q, ld_k, ld_v;
    const float* gate_a; const float* gate_b; long ld_gate_a, ld_gate_b;
    const float* log_rate; const float* step_bias; const float* skip;
    float* state; long state_stride;
    const int* item_slot; const int* item_offset; const int* item_count;
    int heads, qk_heads, dim, vdim;
    float q_scale;
    int delta, unit_norm, writes;
    int channel_decay;
    int state_ahead;               // recurrence_few_kernel: no kernel that may still run writes the states
};

template <typename T, int DPT, int LANES, int TOK, int CPT, bool CHANNEL>      // CPT: columns of the state a thread takes
__global__ void __launch_bounds__(256) linear_recurrence_kernel(RecurrenceParams pp) {
    dependents_may_start();
    wait_for_earlier_kernels();
    constexpr int GROUPS = 128 / LANES;                    // groups of lanes; each takes CPT columns of the state,
    constexpr int COLS = GROUPS * CPT;                     // GROUPS apart, whose chains of sums run side by side
    constexpr int PAD = DPT + 4;                           // a lane's DPT entries of a staged row, 16 bytes apart from the
    constexpr int ROW = LANES * PAD;                       // next lane's in the banks: four entries are read at a time
    constexpr int TPR = 128 / (2 * TOK);                   // threads that bring one staged row (k or q of a token)
    constexpr int PER = (DPT * LANES + TPR - 1) / TPR;     // entries of that row a thread brings
    constexpr int VPER = (TOK * COLS + 127) / 128;         // values a thread brings
    extern __shared__ float shared[];
    const int dim = pp.dim, vdim = pp.vdim;
    // Four warps take the tokens one by one; four others bring the next chunk meanwhile, into the other of two buffers.
    constexpr int CHUNK = (CHANNEL ? 3 : 2) * TOK * ROW + TOK * COLS + 3 * TOK;
    const bool brings = threadIdx.x >= 128;
    const int tid = threadIdx.x & 127;
    float *ks, *qs, *vs, *as, *bs, *kq, *gs;
    auto buffer = [&](int which) {
        ks = shared + which * CHUNK;            // [TOK][ROW]: entry i of a row at (i / DPT) * PAD + i % DPT, zero past dim
        qs = ks + TOK * ROW;                    // [TOK][ROW]
        vs = qs + TOK * ROW;                    // [TOK][COLS]
        as = vs + TOK * COLS;                   // [TOK] the step's gate, then the decay
        bs = as + TOK;                          // [TOK] the write gate, then the write strength
        kq = bs + TOK;                          // [TOK] k . q
        gs = kq + TOK;                          // [TOK][ROW] (CHANNEL only): the decay of every key channel, laid out as ks
    };
    constexpr int GPER = CHANNEL ? (TOK * DPT * LANES + 127) / 128 : 1;     // decays a thread brings
    const int item = blockIdx.x, head = blockIdx.y;
    const int count = pp.item_count[item];
    if (count <= 0) return;
    const long first = pp.item_offset[item];
    const int qk_head = head / (pp.heads / pp.qk_heads);
    const int lane_in = tid % LANES, col_local = tid / LANES;
    // this thread's columns: col_local, col_local + GROUPS, ... of the block's COLS
    // this thread's part of its column of the state: rows lane_in * DPT .. + DPT - 1 (zero past dim, and it stays zero)
    float* S = pp.state + (long)pp.item_slot[item] * pp.state_stride + (long)head * dim * vdim;
    // (the block's slice of the state goes through shared memory both ways, so that the global
    // reads and writes run along the rows of S, whatever the lanes' share of a column is)
    float s[CPT][DPT];
    for (int u = threadIdx.x; u < dim * COLS; u += 256) {
        const int i = u / COLS, c = blockIdx.z * COLS + u % COLS;
        shared[u] = c < vdim ? S[(long)i * vdim + c] : 0.0f;
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < DPT; r++) {
        const int i = lane_in * DPT + r;
#pragma unroll
        for (int c = 0; c < CPT; c++) s[c][r] = i < dim ? shared[i * COLS + col_local + c * GROUPS] : 0.0f;
    }
    __syncthreads();
    const float rate = expf(pp.log_rate[head]);
    const float bias = CHANNEL ? 0.0f : pp.step_bias[head];
    const float skip = pp.skip != nullptr ? pp.skip[head] : 0.0f;
    const T* q = (const T*)pp.q;
    const T* k = (const T*)pp.k;
    const T* v = (const T*)pp.v;
    const int warp = tid >> 5, lane = tid & 31;

    // What a thread brings of every chunk of TOK tokens: PER entries of one row (the k or the q of one
    // token), VPER values, and (the first threads) a token's gates.  The next chunk is asked for
    // before the current one is worked on, so its way through the memory lies under the sums.
    const int row = tid / TPR, row_sub = tid % TPR;
    const int row_token = row >> 1;
    const T* row_base = (row & 1) ? q : k;
    const long row_ld = (row & 1) ? pp.ld_q : pp.ld_k;
    T raw[PER], raw_v[VPER];
    float raw_a = 0.0f, raw_b = 0.0f;
    float raw_g[GPER];
    // (the channel's bias is the same in every chunk: it is read once here, and added when the chunk is staged,
    // so that asking for a chunk waits for nothing)
    float bias_g[GPER];
    if (CHANNEL) {
#pragma unroll
        for (int i = 0; i < GPER; i++) {
            const int d = (tid + 128 * i) % (DPT * LANES);
            bias_g[i] = d < dim ? pp.step_bias[(long)head * dim + d] : 0.0f;
        }
    }
    auto ask = [&](int start) {
        const int n = min(TOK, count - start);
        const long t0 = first + start;
#pragma unroll
        for (int i = 0; i < PER; i++) {
            const int d = row_sub + TPR * i;
            raw[i] = (row_token < n && d < dim) ? row_base[(t0 + row_token) * row_ld + (long)qk_head * dim + d] : from_f32<T>(0.0f);
        }
#pragma unroll
        for (int i = 0; i < VPER; i++) {
            const int u = tid + 128 * i, tt = u / COLS, c = blockIdx.z * COLS + u % COLS;
            raw_v[i] = (tt < n && c < vdim) ? v[(t0 + tt) * pp.ld_v + (long)head * vdim + c] : from_f32<T>(0.0f);
        }
        if (tid < n) {
            if (!CHANNEL) raw_a = pp.gate_a[(t0 + tid) * pp.ld_gate_a + head];
            if (pp.delta) raw_b = pp.gate_b[(t0 + tid) * pp.ld_gate_b + head];
        }
        if (CHANNEL) {
#pragma unroll
            for (int i = 0; i < GPER; i++) {
                const int u = tid + 128 * i, tt = u / (DPT * LANES), d = u % (DPT * LANES);
                raw_g[i] = (tt < n && d < dim) ? pp.gate_a[(t0 + tt) * pp.ld_gate_a + (long)head * dim + d] : 0.0f;
            }
        }
    };
    // (the bringing warps alone) the chunk that was asked for, from token `start` on, into the current buffer
    auto stage = [&](int start) {
        const int n = min(TOK, count - start);
        float* row_smem = ((row & 1) ? qs : ks) + row_token * ROW;
#pragma unroll
        for (int i = 0; i < PER; i++) {
            const int d = row_sub + TPR * i;
            if (d < DPT * LANES) row_smem[(d / DPT) * PAD + d % DPT] = to_f32(raw[i]);       // (zero past dim)
        }
#pragma unroll
        for (int i = 0; i < VPER; i++) {
            const int u = tid + 128 * i;
            if (u < TOK * COLS) vs[u] = to_f32(raw_v[i]);
        }
        if (tid < TOK) {
            // a thread a token: the step, the decay, the write strength
            const float step = softplus_f(raw_a + bias);
            as[tid] = CHANNEL ? 1.0f : expf(-rate * step);
            bs[tid] = pp.delta ? sigmoid_f(raw_b) : step;
        }
        if (CHANNEL) {
#pragma unroll
            for (int i = 0; i < GPER; i++) {
                const int u = tid + 128 * i, tt = u / (DPT * LANES), d = u % (DPT * LANES);
                if (tt < TOK) gs[tt * ROW + (d / DPT) * PAD + d % DPT] = expf(-rate * softplus_f(raw_g[i] + bias_g[i]));
            }
        }
        asm volatile("bar.sync 1, 128;" ::: "memory");
        // a warp finishes TOK / 4 tokens: unit vectors if asked, and k . q; the sums of its tokens are
        // taken side by side, so that their exchanges between the lanes lie under one another
        {
            constexpr int MINE = TOK / 4;
            float sk[MINE], sq[MINE], sd[MINE];
#pragma unroll
            for (int j = 0; j < MINE; j++) {
                const int tt = warp + 4 * j;
                sk[j] = sq[j] = sd[j] = 0.0f;
                if (tt < n)
                    for (int d = lane; d < DPT * LANES; d += 32) {
                        const int at = tt * ROW + (d / DPT) * PAD + d % DPT;
                        const float kv = ks[at], qv = qs[at];
                        sk[j] = fmaf(kv, kv, sk[j]), sq[j] = fmaf(qv, qv, sq[j]), sd[j] = fmaf(kv, qv, sd[j]);
                    }
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1)
#pragma unroll
                for (int j = 0; j < MINE; j++) {
                    sk[j] += __shfl_xor_sync(0xffffffffu, sk[j], o);
                    sq[j] += __shfl_xor_sync(0xffffffffu, sq[j], o);
                    sd[j] += __shfl_xor_sync(0xffffffffu, sd[j], o);
                }
#pragma unroll
            for (int j = 0; j < MINE; j++) {
                const int tt = warp + 4 * j;
                if (tt >= n) continue;
                const float fk = pp.unit_norm ? 1.0f / sqrtf(sk[j] + 1e-6f) : 1.0f;
                const float fq = pp.unit_norm ? pp.q_scale / sqrtf(sq[j] + 1e-6f) : pp.q_scale;
                if (pp.unit_norm || fq != 1.0f)
                    for (int d = lane; d < DPT * LANES; d += 32) {
                        const int at = tt * ROW + (d / DPT) * PAD + d % DPT;
                        ks[at] *= fk, qs[at] *= fq;
                    }
                if (lane == 0) kq[tt] = sd[j] * fk * fq;
            }
        }
    };
    buffer(0);
    if (brings) {
        ask(0);
        stage(0);
        if (TOK < count) ask(TOK);
    }
    __syncthreads();
    for (int start = 0, which = 0; start < count; start += TOK, which ^= 1) {
        const int n = min(TOK, count - start);
        if (brings) {
            buffer(which ^ 1);
            if (start + TOK < count) stage(start + TOK);
            if (start + 2 * TOK < count) ask(start + 2 * TOK);
        } else {
            buffer(which);
        }
        for (int tt = 0; tt < (brings ? 0 : n); tt++) {
            const float* kr = ks + tt * ROW + lane_in * PAD;
            const float* qr = qs + tt * ROW + lane_in * PAD;
            float kreg[DPT];
            float dk[CPT][2], dq[CPT][2];                      // two chains each: half the latency
#pragma unroll
            for (int c = 0; c < CPT; c++) dk[c][0] = dk[c][1] = dq[c][0] = dq[c][1] = 0.0f;
#pragma unroll
            for (int r = 0; r < DPT; r += 4) {
                const float4 k4 = *reinterpret_cast<const float4*>(kr + r);
                const float4 q4 = *reinterpret_cast<const float4*>(qr + r);
                kreg[r] = k4.x, kreg[r + 1] = k4.y, kreg[r + 2] = k4.z, kreg[r + 3] = k4.w;
                if (CHANNEL) {
                    // every row of the state decays by its own factor first; the sums then read the decayed rows
                    const float4 g4 = *reinterpret_cast<const float4*>(gs + tt * ROW + lane_in * PAD + r);
#pragma unroll
                    for (int c = 0; c < CPT; c++) s[c][r] *= g4.x, s[c][r + 1] *= g4.y, s[c][r + 2] *= g4.z, s[c][r + 3] *= g4.w;
                }
#pragma unroll
                for (int c = 0; c < CPT; c++) {
                    dk[c][0] = fmaf(s[c][r], k4.x, dk[c][0]), dq[c][0] = fmaf(s[c][r], q4.x, dq[c][0]);
                    dk[c][1] = fmaf(s[c][r + 1], k4.y, dk[c][1]), dq[c][1] = fmaf(s[c][r + 1], q4.y, dq[c][1]);
                    dk[c][0] = fmaf(s[c][r + 2], k4.z, dk[c][0]), dq[c][0] = fmaf(s[c][r + 2], q4.z, dq[c][0]);
                    dk[c][1] = fmaf(s[c][r + 3], k4.w, dk[c][1]), dq[c][1] = fmaf(s[c][r + 3], q4.w, dq[c][1]);
                }
            }
            float sum_k[CPT], sum_q[CPT];
#pragma unroll
            for (int c = 0; c < CPT; c++) sum_k[c] = dk[c][0] + dk[c][1], sum_q[c] = dq[c][0] + dq[c][1];
#pragma unroll
            for (int o = LANES / 2; o > 0; o >>= 1)
#pragma unroll
                for (int c = 0; c < CPT; c++) {
                    sum_k[c] += __shfl_xor_sync(0xffffffffu, sum_k[c], o);
                    sum_q[c] += __shfl_xor_sync(0xffffffffu, sum_q[c], o);
                }
            // (with a decay per key channel the rows have decayed already: a factor of one, known when compiled)
            const float a = CHANNEL ? 1.0f : as[tt], b = bs[tt], both = kq[tt];
#pragma unroll
            for (int c = 0; c < CPT; c++) {
                const float value = vs[tt * COLS + col_local + c * GROUPS];
                const float u = pp.delta ? b * (value - a * sum_k[c]) : b * value;
#pragma unroll
                for (int r = 0; r < DPT; r++) s[c][r] = fmaf(kreg[r], u, a * s[c][r]);
                const int col = blockIdx.z * COLS + col_local + c * GROUPS;
                if (col < vdim && lane_in == 0)
                    pp.out[(first + start + tt) * pp.ld_out + (long)head * vdim + col] = fmaf(u, both, a * sum_q[c]) + skip * value;
            }
        }
        __syncthreads();                                      // this chunk has been read, the next one is there
    }
    if (pp.writes) {
#pragma unroll
        for (int r = 0; r < DPT; r++) {
            const int i = lane_in * DPT + r;
#pragma unroll
            for (int c = 0; c < CPT; c++)
                if (i < dim && !brings) shared[i * COLS + col_local + c * GROUPS] = s[c][r];
        }
        __syncthreads();
        for (int u = threadIdx.x; u < dim * COLS; u += 256) {
            const int i = u / COLS, c = blockIdx.z * COLS + u % COLS;
            if (c < vdim) S[(long)i * vdim + c] = shared[u];
        }
    }
}

template <typename T, int DPT, int LANES, int TOK, int CPT, bool CHANNEL>
static int launch_recurrence_as(const RecurrenceParams& pp, int n_items, cudaStream_t s) {
    constexpr int COLS = 128 / LANES * CPT;
    // the staged chunk, or the block's slice of the state on its way in and out, whichever is larger
    const size_t staged = 2 * ((size_t)(CHANNEL ? 3 : 2) * TOK * LANES * (DPT + 4) + TOK * COLS + 3 * TOK), slice = (size_t)DPT * LANES * COLS;
    const size_t shared = sizeof(float) * (staged > slice ? staged : slice);
    dim3 grid(n_items, pp.heads, (pp.vdim + COLS - 1) / COLS);
    if (shared > 48 * 1024 &&
        cudaFuncSetAttribute(linear_recurrence_kernel<T, DPT, LANES, TOK, CPT, CHANNEL>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)shared) != cudaSuccess)
        return fail("linear_recurrence: the staged rows' shared memory was refused");
    launch_kernel(AFTER_THE_KERNELS_AHEAD, linear_recurrence_kernel<T, DPT, LANES, TOK, CPT, CHANNEL>, grid, dim3(256), shared, s, pp);
    return check_launch("linear_recurrence_kernel");
}

// ---- one token an entry ----------------------------------------------------------------------------
// Keys of up to 128 entries.  One token's update reads and writes the state once (0.3 us of HBM time for an entry of six heads of
// 128 x 128), so what it takes is the way there and back: a block takes 32 columns of a head, a lane a column and a warp 16 rows,
// all asked for at once and kept in registers, and both sums over the old state meet in shared memory once.  Staging the
// state and 16 tokens' places as the walk above does took 10.3 us for two entries (11.4 for one with a decay a channel); here 4.4 and 4.3.
template <typename T, bool CHANNEL>
__global__ void __launch_bounds__(256) recurrence_few_kernel(RecurrenceParams pp) {
    dependents_may_start();
    if (!pp.state_ahead) wait_for_earlier_kernels();
    constexpr int ROWS = 16, WARPS = 8;
    __shared__ float ks[ROWS * WARPS], qs[ROWS * WARPS], gs[CHANNEL ? ROWS * WARPS : 1], sums[3][4], part_k[WARPS][32], part_q[WARPS][32];
    const int item = blockIdx.x, head = blockIdx.y, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int count = pp.item_count[item];
    if (count <= 0) return;
    const long first = pp.item_offset[item];
    const int dim = pp.dim, vdim = pp.vdim, col = blockIdx.z * 32 + lane;
    const long qk_at = (long)(head / (pp.heads / pp.qk_heads)) * dim;
    float* S = pp.state + (long)pp.item_slot[item] * pp.state_stride + (long)head * dim * vdim;
    float s[ROWS];
#pragma unroll
    for (int r = 0; r < ROWS; r++) {
        const int d = warp * ROWS + r;
        s[r] = d < dim && col < vdim ? S[(long)d * vdim + col] : 0.0f;
    }
    const float rate = expf(pp.log_rate[head]), skip = pp.skip != nullptr ? pp.skip[head] : 0.0f;
    const float bias = CHANNEL ? (tid < dim ? pp.step_bias[(long)head * dim + tid] : 0.0f) : pp.step_bias[head];
    if (pp.state_ahead) wait_for_earlier_kernels();          // (the state is asked for; what the kernels ahead write follows)
    for (int i = 0; i < count; i++) {
        const long t = first + i;
        const float value = col < vdim ? to_f32(((const T*)pp.v)[t * pp.ld_v + (long)head * vdim + col]) : 0.0f;
        float a = 1.0f, b = pp.delta ? sigmoid_f(pp.gate_b[t * pp.ld_gate_b + head]) : 0.0f;
        if (!CHANNEL) {
            const float step = softplus_f(pp.gate_a[t * pp.ld_gate_a + head] + bias);
            a = expf(-rate * step);
            if (!pp.delta) b = step;
        }
        if (tid < ROWS * WARPS) {
            const float k = tid < dim ? to_f32(((const T*)pp.k)[t * pp.ld_k + qk_at + tid]) : 0.0f;
            const float q = tid < dim ? to_f32(((const T*)pp.q)[t * pp.ld_q + qk_at + tid]) : 0.0f;
            if (CHANNEL) gs[tid] = tid < dim ? expf(-rate * softplus_f(pp.gate_a[t * pp.ld_gate_a + (long)head * dim + tid] + bias)) : 1.0f;
            ks[tid] = k, qs[tid] = q;
            const float kk = warp_sum(k * k), qq = warp_sum(q * q), kq = warp_sum(k * q);
            if (lane == 0) sums[0][warp] = kk, sums[1][warp] = qq, sums[2][warp] = kq;
        }
        __syncthreads();
        const float kk = (sums[0][0] + sums[0][1]) + (sums[0][2] + sums[0][3]), qq = (sums[1][0] + sums[1][1]) + (sums[1][2] + sums[1][3]);
        const float fk = pp.unit_norm ? 1.0f / sqrtf(kk + 1e-6f) : 1.0f, fq = pp.unit_norm ? pp.q_scale / sqrtf(qq + 1e-6f) : pp.q_scale;
        const float both = ((sums[2][0] + sums[2][1]) + (sums[2][2] + sums[2][3])) * fk * fq;
        float dk[2] = {0.0f, 0.0f}, dq[2] = {0.0f, 0.0f};
#pragma unroll
        for (int r = 0; r < ROWS; r++) {
            const int d = warp * ROWS + r;
            if (CHANNEL) s[r] *= gs[d];
            dk[r & 1] = fmaf(s[r], ks[d], dk[r & 1]), dq[r & 1] = fmaf(s[r], qs[d], dq[r & 1]);
        }
        part_k[warp][lane] = dk[0] + dk[1], part_q[warp][lane] = dq[0] + dq[1];
        __syncthreads();
        float sum_k = 0.0f, sum_q = 0.0f;
#pragma unroll
        for (int w = 0; w < WARPS; w++) sum_k += part_k[w][lane], sum_q += part_q[w][lane];
        const float u = pp.delta ? b * (value - a * sum_k * fk) : b * value;
#pragma unroll
        for (int r = 0; r < ROWS; r++) s[r] = fmaf(ks[warp * ROWS + r] * fk, u, a * s[r]);
        if (warp == 0 && col < vdim) pp.out[t * pp.ld_out + (long)head * vdim + col] = fmaf(u, both, a * sum_q * fq) + skip * value;
        if (i + 1 < count) __syncthreads();
    }
    if (!pp.writes) return;
#pragma unroll
    for (int r = 0; r < ROWS; r++) {
        const int d = warp * ROWS + r;
        if (d < dim && col < vdim) S[(long)d * vdim + col] = s[r];
    }
}

template <typename T>
static int launch_recurrence_few(const RecurrenceParams& pp, int n_items, cudaStream_t s) {
    const dim3 grid(n_items, pp.heads, (pp.vdim + 31) / 32);
    if (pp.channel_decay) launch_kernel(g_dependent_launch != 0, recurrence_few_kernel<T, true>, grid, dim3(256), 0, s, pp);
    else launch_kernel(g_dependent_launch != 0, recurrence_few_kernel<T, false>, grid, dim3(256), 0, s, pp);
    return check_launch("recurrence_few_kernel");
}

// ---- prompt portions, 16 tokens at a time --------------------------------------------------------
// bfloat16 rows, one decay per head.  The walk above is a chain of one token after the other; over a chunk of 16 tokens the
// same sums are products of small matrices.  With S the state before the chunk, G(t) the product of the decays up to token t, R(t, s) that of
// the decays after s up to t, and k, q normed:
//   delta rule:  M u = b (v - G S^T k),  M(t, s) = b_t R(t, s) (k_t . k_s) below a diagonal of ones  (else u = b v)
//   out_t = G(t) S^T q_t + sum over s <= t of R(t, s) (q_t . k_s) u_s (+ skip v_t)
//   S <- G(15) S + sum over s of R(15, s) k_s u_s^T
// A block takes 16 columns of a head's state, transposed, in the accumulators of four warps, a quarter of the key entries each: as
// the first operand of the next product the accumulators of m16n8k16 tiles need no exchange.  Those warps are the chain; what does not read the
// state is prepared by six more while the chunk before is worked on: four bring the rows and take k . k and q . k, one solves
// M T = 1 row by row, one makes the gates and the products of the decays (as products: no difference of logarithms).  Decays, S, u, T and
// every sum are 32-bit: 32-bit operands enter a product as three bfloat16 terms that hold all their bits, the rows are bfloat16 as they
// come and their norms are factors of the sums.  T is bounded: with |k| = 1 and b <= 1 every factor of the recurrence shrinks.
// What bounds it: issue slots (4,900 warp instructions a chunk, a quarter of them splitting operands) and the chain from S to S.  Two portions of
// 1,024 tokens, 6 heads of 128 x 128: 513 us a launch token by token, 107 here; 24 heads of 128 x 64 without the delta rule, whose
// 192 blocks take two passes over the SMs, 662 and 173 (6 such heads 88).
// Errors against 64 bits (relative): 1,000 + 777 tokens 2.83e-7 token by token, 2.43e-7 here, without the delta rule 1.0e-7 and 8.3e-8; 1,000
// tokens under faster decays 1.29e-7 and 1.43e-7, without the delta rule 1.06e-7 and 1.19e-7.
constexpr int REC_TOKENS = 16, REC_ROW_SLOTS = 6, REC_SLOTS = 4, REC_LD = 24;     // (rows of 16 terms, 48 bytes apart: no bank twice)

template <int DIM> struct RecurrenceRows {
    bf16 k[REC_TOKENS * (DIM + 8)], q[REC_TOKENS * (DIM + 8)], v[REC_TOKENS * REC_LD];
};
struct RecurrenceChunk {
    bf16 solve[3][REC_TOKENS * REC_LD], read[3][REC_TOKENS * REC_LD];             // T and R (q . k), [term][t][s]
    float below[REC_TOKENS * 20];                                                 // M below the diagonal, [s][t]
    float rest[REC_TOKENS * 17];                                                  // R(t, s), [t][s]
    float until[REC_TOKENS];                                                      // G(t)
    float strength[REC_TOKENS], old_k[REC_TOKENS], old_q[REC_TOKENS], write[REC_TOKENS];      // b, b G |k|, G |q|, R(15, s) |k|
};
template <int DIM> struct RecurrenceShared {
    RecurrenceRows<DIM> rows[REC_ROW_SLOTS];
    RecurrenceChunk chunk[REC_SLOTS];
    float4 sums[4][4][32];                                                        // [quarter][k or q, 8 tokens][lane]
    float unit[2][REC_TOKENS];                                                    // 1 / |k|, q_scale / |q|
};

__device__ __forceinline__ void barrier_of_128(int id) { asm volatile("bar.sync %0, 128;" ::"r"(id) : "memory"); }

// c = a b, both 32-bit as three terms; the product of the two smallest, 2^-28 of the largest at most, is left out.
__device__ __forceinline__ void mma_terms(float (&c)[4], const uint32_t (&a)[3][4], const uint32_t (&b)[3][4], int half) {
    c[0] = c[1] = c[2] = c[3] = 0.0f;
#pragma unroll
    for (int order = 3; order >= 1; order--)
#pragma unroll
        for (int i = order == 3 ? 1 : 0; i <= order && i < 3; i++) mma_tile(c, a[i], half ? b[order - i][2] : b[order - i][0], half ? b[order - i][3] : b[order - i][1]);
    mma_added(c, a[0], half ? b[0][2] : b[0][0], half ? b[0][3] : b[0][1]);
}

template <int DIM, bool DELTA>
__global__ void __launch_bounds__(320, 1) recurrence_chunks_kernel(RecurrenceParams pp) {
    extern __shared__ __align__(16) unsigned char recurrence_shared[];
    RecurrenceShared<DIM>& sh = *reinterpret_cast<RecurrenceShared<DIM>*>(recurrence_shared);
    constexpr int LD = DIM + 8, QUARTER = DIM / 4, TILES = QUARTER / 8;
    dependents_may_start();
    wait_for_earlier_kernels();
    const int item = blockIdx.x, head = blockIdx.y, col0 = blockIdx.z * 16;
    const int count = pp.item_count[item];
    if (count <= 0) return;
    const long first = pp.item_offset[item];
    const int dim = pp.dim, vdim = pp.vdim, chunks = (count + REC_TOKENS - 1) / REC_TOKENS;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, tq = lane & 3;
    const long qk_at = (long)(head / (pp.heads / pp.qk_heads)) * dim, v_at = (long)head * vdim + col0;
    float* S = pp.state + (long)pp.item_slot[item] * pp.state_stride + (long)head * dim * vdim;

    // the state's warps
    float s[TILES][4];
    if (warp < 4) {
#pragma unroll
        for (int j = 0; j < TILES; j++)
#pragma unroll
            for (int e = 0; e < 4; e++) {
                const int d = warp * QUARTER + j * 8 + 2 * tq + (e & 1), c = col0 + g + 8 * (e >> 1);
                s[j][e] = d < dim && c < vdim ? S[(long)d * vdim + c] : 0.0f;
            }
    }
    const float skip = pp.skip != nullptr ? pp.skip[head] : 0.0f;
    // y(t) = the sum over s <= t of L(t, s) x(s), one product after the other: where an x is no finite number, the zeros that
    // the tensor cores take in place of the L(t, s) of later tokens would carry it into earlier ones.
    auto lower_product = [&](const bf16 (&terms)[3][REC_TOKENS * REC_LD], const float (&x)[2][4], float (&y)[2][4]) {
#pragma unroll
        for (int e = 0; e < 8; e++) y[e / 4][e % 4] = 0.0f;
#pragma unroll
        for (int s_ = 0; s_ < REC_TOKENS; s_++) {
            const int from = g * 4 + s_ % 8 / 2;
            const float left = __shfl_sync(0xffffffffu, x[s_ / 8][s_ % 2], from), right = __shfl_sync(0xffffffffu, x[s_ / 8][2 + s_ % 2], from);
#pragma unroll
            for (int e = 0; e < 8; e++) {
                const int t = e / 4 * 8 + 2 * tq + (e & 1), at = t * REC_LD + s_;
                const float l = to_f32(terms[0][at]) + (to_f32(terms[1][at]) + to_f32(terms[2][at]));
                if (s_ <= t) y[e / 4][e % 4] = fmaf(l, (e & 2) ? right : left, y[e / 4][e % 4]);
            }
        }
    };
    auto all_finite = [&](const float (&x)[2][4]) {
        bool finite = true;
#pragma unroll
        for (int e = 0; e < 8; e++) finite = finite && fabsf(x[e / 4][e % 4]) < INFINITY;
        return __all_sync(0xffffffffu, finite) != 0;
    };
    auto walk = [&](int i) {
        const RecurrenceRows<DIM>& rows = sh.rows[i % REC_ROW_SLOTS];
        const RecurrenceChunk& ch = sh.chunk[i % REC_SLOTS];
        float sums[4][4];                                                         // S^T k of 2 x 8 tokens, S^T q
#pragma unroll
        for (int j = 0; j < 4; j++) sums[j][0] = sums[j][1] = sums[j][2] = sums[j][3] = 0.0f;
        const int at = ((lane & 7) + ((lane >> 4) & 1) * 8) * LD + warp * QUARTER + ((lane >> 3) & 1) * 8;
#pragma unroll
        for (int j = 0; j < TILES; j += 2) {
            uint32_t a[3][4], bk[4], bq[4];
            float x[4][4] = {};
            terms_of(a, s[j], s[j + 1]);
            if (DELTA) load_blocks(bk, rows.k + at + j * 8);
            load_blocks(bq, rows.q + at + j * 8);
#pragma unroll
            for (int term = 2; term >= 0; term--) {
                if (DELTA) mma_tile(x[0], a[term], bk[0], bk[1]), mma_tile(x[1], a[term], bk[2], bk[3]);
                mma_tile(x[2], a[term], bq[0], bq[1]), mma_tile(x[3], a[term], bq[2], bq[3]);
            }
#pragma unroll
            for (int e = 0; e < 16; e++) sums[e / 4][e % 4] += x[e / 4][e % 4];
        }
#pragma unroll
        for (int j = DELTA ? 0 : 2; j < 4; j++) sh.sums[warp][j][lane] = make_float4(sums[j][0], sums[j][1], sums[j][2], sums[j][3]);
        float v[2][4], u[2][4];
#pragma unroll
        for (int j = 0; j < 2; j++)
#pragma unroll
            for (int e = 0; e < 4; e++) v[j][e] = to_f32(rows.v[(j * 8 + 2 * tq + (e & 1)) * REC_LD + g + 8 * (e >> 1)]);
        barrier_of_128(1);
        if (DELTA) {
            float r[2][4];
#pragma unroll
            for (int j = 0; j < 2; j++) {
                const float4 x = sh.sums[0][j][lane], y = sh.sums[1][j][lane], z = sh.sums[2][j][lane], w = sh.sums[3][j][lane];
                const float old[4] = {(x.x + y.x) + (z.x + w.x), (x.y + y.y) + (z.y + w.y), (x.z + y.z) + (z.z + w.z), (x.w + y.w) + (z.w + w.w)};
#pragma unroll
                for (int e = 0; e < 4; e++) {
                    const int t = j * 8 + 2 * tq + (e & 1);
                    r[j][e] = ch.strength[t] * v[j][e] - ch.old_k[t] * old[e];
                }
            }
            uint32_t a[3][4], b[3][4];
            terms_of(a, r[0], r[1]);
#pragma unroll
            for (int term = 0; term < 3; term++) load_blocks(b[term], ch.solve[term] + ((lane & 7) + ((lane >> 4) & 1) * 8) * REC_LD + ((lane >> 3) & 1) * 8);
            mma_terms(u[0], a, b, 0);
            mma_terms(u[1], a, b, 1);
            if (!all_finite(r)) lower_product(ch.solve, r, u);
        } else {
#pragma unroll
            for (int j = 0; j < 2; j++)
#pragma unroll
                for (int e = 0; e < 4; e++) u[j][e] = ch.strength[j * 8 + 2 * tq + (e & 1)] * v[j][e];
        }
        // the state moves on first: it is what the next chunk waits for
        {
            float w[2][4];
            uint32_t a[3][4];
#pragma unroll
            for (int j = 0; j < 2; j++)
#pragma unroll
                for (int e = 0; e < 4; e++) w[j][e] = ch.write[j * 8 + 2 * tq + (e & 1)] * u[j][e];
            terms_of(a, w[0], w[1]);
            const float whole = ch.until[REC_TOKENS - 1];
#pragma unroll
            for (int j = 0; j < TILES; j += 2) {
                uint32_t b[4];
                load_blocks_turned(b, rows.k + ((lane & 7) + ((lane >> 3) & 1) * 8) * LD + warp * QUARTER + j * 8 + ((lane >> 4) & 1) * 8);
                float x[2][4] = {};
#pragma unroll
                for (int term = 2; term >= 0; term--) mma_tile(x[0], a[term], b[0], b[1]), mma_tile(x[1], a[term], b[2], b[3]);
#pragma unroll
                for (int e = 0; e < 4; e++) s[j][e] = fmaf(s[j][e], whole, x[0][e]), s[j + 1][e] = fmaf(s[j + 1][e], whole, x[1][e]);
            }
        }
        if (warp < 2) {                                                           // eight tokens' results a warp
            uint32_t a[3][4], b[3][4];
            terms_of(a, u[0], u[1]);
#pragma unroll
            for (int term = 0; term < 3; term++) load_blocks(b[term], ch.read[term] + ((lane & 7) + ((lane >> 4) & 1) * 8) * REC_LD + ((lane >> 3) & 1) * 8);
            float o[4];
            mma_terms(o, a, b, warp);
            if (!all_finite(u)) {
                float y[2][4];
                lower_product(ch.read, u, y);
#pragma unroll
                for (int e = 0; e < 4; e++) o[e] = warp == 0 ? y[0][e] : y[1][e];
            }
            const float4 x = sh.sums[0][2 + warp][lane], y = sh.sums[1][2 + warp][lane], z = sh.sums[2][2 + warp][lane], w = sh.sums[3][2 + warp][lane];
            const float old[4] = {(x.x + y.x) + (z.x + w.x), (x.y + y.y) + (z.y + w.y), (x.z + y.z) + (z.z + w.z), (x.w + y.w) + (z.w + w.w)};
#pragma unroll
            for (int e = 0; e < 4; e++) {
                const int t = warp * 8 + 2 * tq + (e & 1), c = g + 8 * (e >> 1);
                const float value = warp == 0 ? v[0][e] : v[1][e];
                if (i * REC_TOKENS + t < count && col0 + c < vdim)
                    pp.out[(first + i * REC_TOKENS + t) * pp.ld_out + v_at + c] = fmaf(ch.old_q[t], old[e], o[e]) + skip * value;
            }
        }
    };

    // the rows' warps
    const int p = tid - 128, rows_warp = warp - 4;
    // (a thread's pieces of a chunk lie where those of the chunk before lay, 16 rows on)
    constexpr int PIECES = DIM / 8, STEP = 128 / PIECES;
    const int piece_t = p / PIECES, piece_d = p % PIECES * 8, value_t = (p >> 1) & (REC_TOKENS - 1), value_c = (p & 1) * 8;
    const bf16* k_from = (const bf16*)pp.k + (first + piece_t) * pp.ld_k + qk_at + piece_d;
    const bf16* q_from = (const bf16*)pp.q + (first + piece_t) * pp.ld_q + qk_at + piece_d;
    const bf16* v_from = (const bf16*)pp.v + (first + value_t) * pp.ld_v + v_at + value_c;
    auto bring = [&](int i) {
        if (i < chunks) {
            RecurrenceRows<DIM>& rows = sh.rows[i % REC_ROW_SLOTS];
            const int n = count - i * REC_TOKENS;
#pragma unroll
            for (int j = 0; j < REC_TOKENS / STEP; j++) {
                const bool there = piece_t + j * STEP < n && piece_d < dim;
                const int to = (piece_t + j * STEP) * LD + piece_d;
                copy_16(rows.k + to, there ? k_from + j * STEP * pp.ld_k : (const bf16*)pp.k, there);
                copy_16(rows.q + to, there ? q_from + j * STEP * pp.ld_q : (const bf16*)pp.q, there);
            }
            if (p < 2 * REC_TOKENS) {
                const bool there = value_t < n && col0 + value_c < vdim;
                copy_16(rows.v + value_t * REC_LD + value_c, there ? v_from : (const bf16*)pp.v, there);
            }
            k_from += REC_TOKENS * pp.ld_k, q_from += REC_TOKENS * pp.ld_q, v_from += REC_TOKENS * pp.ld_v;
        }
        copies_end();
    };
    auto pairs = [&](int i) {
        bring(i + 3);
        copies_landed<3>();
        barrier_of_128(2);                                                        // the rows of chunk i are there
        const RecurrenceRows<DIM>& rows = sh.rows[i % REC_ROW_SLOTS];
        RecurrenceChunk& ch = sh.chunk[i % REC_SLOTS];
        {
            const int row = p >> 2, t = row & (REC_TOKENS - 1);
            const bf16* x = (row < REC_TOKENS ? rows.k : rows.q) + t * LD + (p & 3) * QUARTER;
            float sum = 0.0f;
            if (pp.unit_norm) {
#pragma unroll
                for (int d = 0; d < QUARTER; d += 8) {
                    const uint4 eight = *reinterpret_cast<const uint4*>(x + d);
                    const uint32_t twos[4] = {eight.x, eight.y, eight.z, eight.w};
#pragma unroll
                    for (int r = 0; r < 4; r++) {
                        const float2 f = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&twos[r]));
                        sum = fmaf(f.x, f.x, fmaf(f.y, f.y, sum));
                    }
                }
                sum += __shfl_xor_sync(0xffffffffu, sum, 1);
                sum += __shfl_xor_sync(0xffffffffu, sum, 2);
            }
            const float scale = row < REC_TOKENS ? 1.0f : pp.q_scale;
            if ((p & 3) == 0) sh.unit[row >> 4][t] = pp.unit_norm ? scale / sqrtf(sum + 1e-6f) : scale;
        }
        // warps 0 and 1: k . k with tokens s of 0..7, 8..15; warps 2 and 3: q . k
        const bool is_q = rows_warp >= 2;
        float even[4] = {0.0f, 0.0f, 0.0f, 0.0f}, odd[4] = {0.0f, 0.0f, 0.0f, 0.0f};
        if (DELTA || is_q) {
            const bf16* a_at = (is_q ? rows.q : rows.k) + (lane & 15) * LD + (lane >> 4) * 8;
            const bf16* b_at = rows.k + ((rows_warp & 1) * 8 + (lane & 7)) * LD + (lane >> 3) * 8;
#pragma unroll
            for (int d = 0; d < DIM; d += 32) {
                uint32_t a[4], b[4];
                load_blocks(b, b_at + d);
                load_blocks(a, a_at + d);
                mma_added(even, a, b[0], b[1]);
                load_blocks(a, a_at + d + 16);
                mma_added(odd, a, b[2], b[3]);
            }
        }
        barrier_of_128(2);                                                        // the norms are written
        if (DELTA || is_q) {
            const int s0 = (rows_warp & 1) * 8 + 2 * tq;
#pragma unroll
            for (int h = 0; h < 2; h++) {
                const int t = g + 8 * h;
                const float left = sh.unit[is_q][t];
                float x[2];
#pragma unroll
                for (int e = 0; e < 2; e++) {
                    const int s_ = s0 + e;
                    x[e] = (is_q ? s_ <= t : s_ < t) ? (even[2 * h + e] + odd[2 * h + e]) * (left * sh.unit[0][s_]) * ch.rest[t * 17 + s_] : 0.0f;
                    if (!is_q) ch.below[s_ * 20 + t] = ch.strength[t] * x[e];
                }
                if (is_q) {
                    uint32_t terms[3];
                    three_terms(x[0], x[1], terms[0], terms[1], terms[2]);
#pragma unroll
                    for (int term = 0; term < 3; term++) *reinterpret_cast<uint32_t*>(ch.read[term] + t * REC_LD + s0) = terms[term];
                }
            }
        }
        if (p < REC_TOKENS) {
            const float unit_k = sh.unit[0][p], until = ch.until[p];
            ch.old_k[p] = ch.strength[p] * until * unit_k;
            ch.old_q[p] = until * sh.unit[1][p];
            ch.write[p] = ch.rest[(REC_TOKENS - 1) * 17 + p] * unit_k;
        }
    };
    // T: lane l has column l mod 16
    auto solve = [&](int i) {
        RecurrenceChunk& ch = sh.chunk[i % REC_SLOTS];
        const int column = lane & 15;
        float x[REC_TOKENS];
#pragma unroll
        for (int t = 0; t < REC_TOKENS; t++) x[t] = t == column ? 1.0f : 0.0f;
#pragma unroll
        for (int s_ = 0; s_ < REC_TOKENS - 1; s_++) {
            const float* below = ch.below + s_ * 20;
#pragma unroll
            for (int t4 = (s_ + 1) / 4 * 4; t4 < REC_TOKENS; t4 += 4) {
                const float4 m = *reinterpret_cast<const float4*>(below + t4);
                const float f[4] = {m.x, m.y, m.z, m.w};
#pragma unroll
                for (int r = 0; r < 4; r++)
                    if (t4 + r > s_) x[t4 + r] = fmaf(-f[r], x[s_], x[t4 + r]);
            }
        }
        if (lane < REC_TOKENS) {
#pragma unroll
            for (int t = 0; t < REC_TOKENS; t += 2) {
                uint32_t terms[3];
                three_terms(x[t], x[t + 1], terms[0], terms[1], terms[2]);
#pragma unroll
                for (int j = 0; j < 3; j++) {
                    const __nv_bfloat162 two = *reinterpret_cast<const __nv_bfloat162*>(&terms[j]);
                    ch.solve[j][t * REC_LD + column] = two.x;
                    ch.solve[j][(t + 1) * REC_LD + column] = two.y;
                }
            }
        }
    };
    // the gates of a chunk, asked for a chunk ahead: a lane a token, and then a lane an s
    const float rate = expf(pp.log_rate[head]), bias = pp.step_bias[head];
    float raw_a = 0.0f, raw_b = 0.0f;
    auto ask_gates = [&](int i) {
        const int t = i * REC_TOKENS + lane;
        if (lane < REC_TOKENS && t < count) {
            raw_a = pp.gate_a[(first + t) * pp.ld_gate_a + head];
            if (DELTA) raw_b = pp.gate_b[(first + t) * pp.ld_gate_b + head];
        }
    };
    auto gates = [&](int i) {
        RecurrenceChunk& ch = sh.chunk[i % REC_SLOTS];
        const bool there = lane < REC_TOKENS && i * REC_TOKENS + lane < count;
        const float step = softplus_f(raw_a + bias), decay = there ? expf(-rate * step) : 1.0f;
        if (lane < REC_TOKENS) ch.strength[lane] = there ? (DELTA ? sigmoid_f(raw_b) : step) : 0.0f;
        if (i + 1 < chunks) ask_gates(i + 1);
        float run = 1.0f;
#pragma unroll
        for (int t = 0; t < REC_TOKENS; t++) {
            const float a = __shfl_sync(0xffffffffu, decay, t);
            if (lane == REC_TOKENS || t > lane) run *= a;
            if (t >= lane) ch.rest[t * 17 + lane] = run;
            if (lane == REC_TOKENS) ch.until[t] = run;
        }
    };

    if (warp >= 4 && warp < 8)
        for (int i = 0; i < 3; i++) bring(i);
    if (warp == 9) ask_gates(0);
    // chunk i's gates are made three rounds before it is walked, its pairs two, its T one
    for (int i = -3; i < chunks; i++) {
        if (warp < 4) {
            if (i >= 0) walk(i);
        } else if (warp < 8) {
            if (i >= -2 && i + 2 < chunks) pairs(i + 2);
        } else if (warp == 8) {
            if (DELTA && i >= -1 && i + 1 < chunks) solve(i + 1);
        } else if (i + 3 < chunks) gates(i + 3);
        __syncthreads();
    }
    if (warp < 4 && pp.writes) {
#pragma unroll
        for (int j = 0; j < TILES; j++)
#pragma unroll
            for (int e = 0; e < 4; e++) {
                const int d = warp * QUARTER + j * 8 + 2 * tq + (e & 1), c = col0 + g + 8 * (e >> 1);
                if (d < dim && c < vdim) S[(long)d * vdim + c] = s[j][e];
            }
    }
}

// Portions of bfloat16 rows in whole 16-byte pieces; the delta rule with normed keys (what bounds T).  The walk above takes 250 ns
// a token, a chunk of 16 here 1.7 us and its first three rounds of preparation as long as one chunk more: from some 16 tokens an entry on.
static bool recurrence_chunks_take(const RecurrenceParams& pp, int n_items, int n_tokens) {
    auto on_16 = [](const void* x, long ld) { return ((reinterpret_cast<uintptr_t>(x) | (uintptr_t)(ld * 2)) & 15) == 0; };
    return !pp.channel_decay && n_tokens >= 32 + 2 * n_items && pp.dim % 8 == 0 && pp.dim > 32 && pp.dim <= 128 && pp.vdim % 8 == 0 &&
           (!pp.delta || pp.unit_norm) && on_16(pp.q, pp.ld_q) && on_16(pp.k, pp.ld_k) && on_16(pp.v, pp.ld_v);
}

template <int DIM, bool DELTA>
static int launch_recurrence_chunks(const RecurrenceParams& pp, int n_items, cudaStream_t s) {
    const int shared = (int)sizeof(RecurrenceShared<DIM>);
    if (cudaFuncSetAttribute(recurrence_chunks_kernel<DIM, DELTA>, cudaFuncAttributeMaxDynamicSharedMemorySize, shared) != cudaSuccess)
        return fail("linear_recurrence: the chunks' shared memory was refused");
    const dim3 grid(n_items, pp.heads, (pp.vdim + 15) / 16);
    launch_kernel(AFTER_THE_KERNELS_AHEAD, recurrence_chunks_kernel<DIM, DELTA>, grid, dim3(320), shared, s, pp);
    return check_launch("recurrence_chunks_kernel");
}

template <typename T, int DPT, int LANES, int TOK, int CPT>
static int launch_recurrence(const RecurrenceParams& pp, int n_items, cudaStream_t s) {
    if (pp.channel_decay) return launch_recurrence_as<T, DPT, LANES, TOK, CPT, true>(pp, n_items, s);
    return launch_recurrence_as<T, DPT, LANES, TOK, CPT, false>(pp, n_items, s);
}

// A column of the state lies in the registers of 4 to 32 lanes of a warp.  Prompt portions: eight
// rows a lane up to a key size of 256 (short sums).  Steps of few tokens per entry: as many rows a
// lane as registers hold, so that the blocks, each of which pays the same chain of loads for its
// few tokens, are few.  Steps of one token an entry (or two more in all) have a kernel of their own, which asks for a token's
// values when the one before is done: beside them an entry of many tokens would wait for each (63 entries of one token and one of 95, 6 heads of
// 128 x 128: 155 us, 80 on the walk; one entry of four, heads of 64 x 64: 7.8 and 5.9).
template <typename T>
static int pick_recurrence(const RecurrenceParams& pp, int n_items, int n_tokens, cudaStream_t s) {
    if (pp.dim <= 32) return launch_recurrence<T, 8, 4, 16, 1>(pp, n_items, s);
    if (pp.dim <= 128 && n_tokens <= n_items + 2) return launch_recurrence_few<T>(pp, n_items, s);
    if (n_tokens <= 4 * n_items) {
        if (pp.dim <= 64) return launch_recurrence<T, 16, 4, 16, 1>(pp, n_items, s);
        if (pp.dim <= 128) return launch_recurrence<T, 32, 4, 16, 1>(pp, n_items, s);
    } else if (pp.dim <= 128) {
        // Prompt portions.  The walk from token to token is a chain of dependent sums and exchanges
        // between lanes; a thread takes two columns, whose chains run in one another's gaps, or four
        // where two would leave the busy entries' blocks more than one an SM (entries of a step that
        // is filled up to a round shape may be empty: portions are taken to hold 1,024 tokens).
        // Eight columns a thread measured slower: every column has its own exchanges.
        const int groups = pp.dim <= 64 ? 16 : 8;
        int busy = (n_tokens + 1023) / 1024;
        if (busy > n_items) busy = n_items;
        const bool four = (long)busy * pp.heads * ((pp.vdim + groups * 2 - 1) / (groups * 2)) > 148;
        if (pp.dim <= 64) {
            if (four) return launch_recurrence<T, 8, 8, 16, 4>(pp, n_items, s);
            return launch_recurrence<T, 8, 8, 16, 2>(pp, n_items, s);
        }
        if (four) return launch_recurrence<T, 8, 16, 16, 4>(pp, n_items, s);
        return launch_recurrence<T, 8, 16, 16, 2>(pp, n_items, s);
    }
    if (pp.dim <= 256) return launch_recurrence<T, 8, 32, 16, 2>(pp, n_items, s);
    return launch_recurrence<T, 32, 32, 4, 1>(pp, n_items, s);
}

extern "C" int mllm_hybrid_linear_recurrence(const RecurrenceParams* params, int n_items, int n_tokens, int dtype, void* stream) {
    if (n_items <= 0) return 0;
    const RecurrenceParams& pp = *params;
    if (pp.dim <= 0 || pp.dim > 1024 || pp.vdim <= 0) return fail("linear_recurrence: the key size must be in 1..1024");
    if (pp.qk_heads <= 0 || pp.heads % pp.qk_heads != 0) return fail("linear_recurrence: heads must be a multiple of the query/key heads");
    if (pp.heads > 65535) return fail("linear_recurrence: too many heads for one launch");
    if (pp.delta && pp.gate_b == nullptr) return fail("linear_recurrence: the delta rule needs its write gates");
    if (pp.channel_decay && pp.skip != nullptr) return fail("linear_recurrence: a decay per key channel goes with no skip");
    cudaStream_t s = (cudaStream_t)stream;
    if (dtype == DT_F32) return pick_recurrence<float>(pp, n_items, n_tokens, s);
    if (dtype == DT_BF16 && recurrence_chunks_take(pp, n_items, n_tokens)) {
        if (pp.dim <= 64) return pp.delta ? launch_recurrence_chunks<64, true>(pp, n_items, s) : launch_recurrence_chunks<64, false>(pp, n_items, s);
        return pp.delta ? launch_recurrence_chunks<128, true>(pp, n_items, s) : launch_recurrence_chunks<128, false>(pp, n_items, s);
    }
    if (dtype == DT_BF16) return pick_recurrence<bf16>(pp, n_items, n_tokens, s);
    return fail("linear_recurrence: unknown dtype");
}

// ---------------------------------------------------------------------------
// Routed feed-forward, the plain form: every (token, chosen expert) pair by itself.
//   route        per token: z = W_router x in 32-bit, s = sigmoid(z); the `top` experts with the
//                largest s (the lower index wins a tie) with s as the weight of their INPUT; if
//                there is a shared expert, one more pair: expert `n_experts`, input weight 1,
//                output weight sigmoid(w_shared_gate . x) (or 1 for a shared expert without a gate).
//                ROUTE_SOFTMAX_OF_CHOSEN: z (+ a bias per expert) itself ranks the experts, the
//                chosen ones' OUTPUTS are weighed by the softmax over the chosen logits only, and
//                their inputs by 1.  ROUTE_SOFTMAX_OF_ALL: s = the softmax over all outputs; s plus a
//                correction per output ranks them, the chosen ones' outputs are weighed by s over
//                the chosen ones' sum (+ 1e-20), times `scale`.  ROUTE_SIGMOID: s = sigmoid(z); s plus a
//                correction ranks, the chosen ones' outputs are weighed by s itself, times `scale`.  With
//                `groups` the experts form that many equal runs of neighbours, of which only the `keep`
//                best can be chosen from; a group's score is the sum of its two largest ranking scores.
//                The last `n_identity` outputs are
//                identity experts, whose output is the token itself: such a choice becomes -1 and
//                its weight goes into the token's identity weight
//   expert_up    act[pair, f] = silu(W_gate[e] x') * (W_up[e] x') with x' = weight * x (or another form of
//                an expert, see ExpertForm)
//   expert_down  hidden[t] += sum over the token's pairs of out_weight * W_down[e] act[pair] (or, with `assign`,
//                hidden[t] = that sum)
// Experts are named by a table of pointers (gate, up, down) and inner sizes, so that experts of
// different sizes (the shared one) go through the same kernels; the down matrices are column
// ranges of one matrix [width, all inner sizes], so their rows lie ld_down apart.
//
// For many tokens the same sum runs as two products over ALL experts: gates and ups of every
// expert as one matrix, the down matrices side by side as another.  An expert a token did not
// choose gets the input weight 0, and expert(0) = W_down (silu(0) * 0) = 0 exactly; the input
// weight multiplies the product's result instead of its input (W (s x) = s (W x)):
//   expert_combine   act[t, c] = silu(s G[t, c]) * (s U[t, c]) * out_weight for column c of expert e,
//                    s = the token's input weight for e, or 0
// ---------------------------------------------------------------------------
// Sixteen bytes of a row as 32-bit floats in registers: 8 bfloat16 or 4 floats.
template <typename T> struct Vec16;
template <> struct Vec16<float> {
    static constexpr int N = 4;
    static __device__ __forceinline__ void unpack(const uint4& v, float* out) {
        out[0] = __uint_as_float(v.x), out[1] = __uint_as_float(v.y), out[2] = __uint_as_float(v.z), out[3] = __uint_as_float(v.w);
    }
    static __device__ __forceinline__ void load(const float* p, float* out) { unpack(*reinterpret_cast<const uint4*>(p), out); }
};
template <> struct Vec16<bf16> {
    static constexpr int N = 8;
    static __device__ __forceinline__ void unpack(const uint4& v, float* out) {
        out[0] = __uint_as_float(v.x << 16), out[1] = __uint_as_float(v.x & 0xffff0000u);
        out[2] = __uint_as_float(v.y << 16), out[3] = __uint_as_float(v.y & 0xffff0000u);
        out[4] = __uint_as_float(v.z << 16), out[5] = __uint_as_float(v.z & 0xffff0000u);
        out[6] = __uint_as_float(v.w << 16), out[7] = __uint_as_float(v.w & 0xffff0000u);
    }
    static __device__ __forceinline__ void load(const bf16* p, float* out) { unpack(*reinterpret_cast<const uint4*>(p), out); }
};
__device__ __forceinline__ bool aligned16(const void* p) { return (reinterpret_cast<unsigned long long>(p) & 15ull) == 0; }
static bool aligned_host(const void* p) { return (reinterpret_cast<unsigned long long>(p) & 15ull) == 0; }

// How a token's experts are chosen and weighed (the launcher's `rule`).
enum RouteRule { ROUTE_SIGMOID_ON_INPUT = 0, ROUTE_SOFTMAX_OF_CHOSEN = 1, ROUTE_SOFTMAX_OF_ALL = 2, ROUTE_SIGMOID = 3 };

// A block takes TOKENS consecutive tokens (four in long steps: a router row that is read serves all of them) and deals
// the outputs out to its warps; then a warp a token ranks.
template <typename T, int TOKENS>
__global__ void __launch_bounds__(512)
route_kernel(const T* __restrict__ x, long ld_x, const T* __restrict__ router, const float* __restrict__ router_bias,
             const float* __restrict__ correction, const T* __restrict__ shared_gate, int shared_plain, int rule, float scale,
             int width, int n_outputs, int n_identity, int groups, int keep_groups, int top, int pairs, int n_tokens,
             int* __restrict__ choice, float* __restrict__ in_weight, float* __restrict__ out_weight, float* __restrict__ identity_weight) {
    dependents_may_start();
    wait_for_earlier_kernels();
    extern __shared__ __align__(16) float shared[];
    float* rows = shared;                                  // [TOKENS][width]
    float* scores = rows + TOKENS * width;                 // [TOKENS][n_outputs + 1]: what ranks the experts
    float* shares = scores + TOKENS * (n_outputs + 1);     // [TOKENS][n_outputs]: what weighs them where that is something else
    float* group_scores = shares + TOKENS * n_outputs;     // [TOKENS][groups]
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, n_warps = blockDim.x >> 5;
    const int t0 = blockIdx.x * TOKENS, n_here = min(TOKENS, n_tokens - t0);
    constexpr int N = Vec16<T>::N;
    const bool vectors = width % N == 0 && aligned16(x) && ld_x % N == 0 && aligned16(router);
    for (int g = 0; g < TOKENS; g++) {
        const T* row = x + (long)(t0 + g) * ld_x;
        if (g >= n_here) {
            for (int c = threadIdx.x; c < width; c += blockDim.x) rows[g * width + c] = 0.0f;
        } else if (vectors) {
            for (int c = threadIdx.x * N; c < width; c += blockDim.x * N) Vec16<T>::load(row + c, rows + g * width + c);
        } else {
            for (int c = threadIdx.x; c < width; c += blockDim.x) rows[g * width + c] = to_f32(row[c]);
        }
    }
    __syncthreads();
    for (int e = warp; e < n_outputs + (shared_gate != nullptr ? 1 : 0); e += n_warps) {
        const T* w = e < n_outputs ? router + (long)e * width : shared_gate;
        float z[TOKENS];
#pragma unroll
        for (int g = 0; g < TOKENS; g++) z[g] = 0.0f;
        if (vectors && aligned16(w)) {
#pragma unroll 2
            for (int c = lane * N; c < width; c += 32 * N) {
                float a[N];
                Vec16<T>::load(w + c, a);
#pragma unroll
                for (int g = 0; g < TOKENS; g++)
#pragma unroll
                    for (int i = 0; i < N; i += 4) {
                        const float4 b = *reinterpret_cast<const float4*>(rows + g * width + c + i);
                        z[g] = fmaf(a[i], b.x, fmaf(a[i + 1], b.y, fmaf(a[i + 2], b.z, fmaf(a[i + 3], b.w, z[g]))));
                    }
            }
        } else {
            for (int c = lane; c < width; c += 32)
#pragma unroll
                for (int g = 0; g < TOKENS; g++) z[g] = fmaf(to_f32(w[c]), rows[g * width + c], z[g]);
        }
#pragma unroll
        for (int g = 0; g < TOKENS; g++) {
            float sum = warp_sum(z[g]);
            if (e < n_outputs && router_bias != nullptr) sum += router_bias[e];
            // (a softmax needs the logits themselves)
            const bool logit = (rule == ROUTE_SOFTMAX_OF_CHOSEN || rule == ROUTE_SOFTMAX_OF_ALL) && e < n_outputs;
            if (lane == 0) scores[g * (n_outputs + 1) + e] = logit ? sum : sigmoid_f(sum);
        }
    }
    __syncthreads();
    if (warp >= n_here) return;
    const int t = t0 + warp;
    float *score = scores + warp * (n_outputs + 1), *share = shares + warp * n_outputs;
    // one warp ranks: lane l looks at outputs l, l + 32, ...
    if (rule == ROUTE_SOFTMAX_OF_ALL) {
        float most = -INFINITY, sum = 0.0f;
        for (int e = lane; e < n_outputs; e += 32) most = fmaxf(most, score[e]);
        most = warp_max(most);
        for (int e = lane; e < n_outputs; e += 32) {
            share[e] = expf(score[e] - most);
            sum += share[e];
        }
        sum = warp_sum(sum);
        for (int e = lane; e < n_outputs; e += 32) {
            share[e] /= sum;
            score[e] = share[e] + (correction != nullptr ? correction[e] : 0.0f);
        }
        __syncwarp();
    }
    if (rule == ROUTE_SIGMOID) {
        for (int e = lane; e < n_outputs; e += 32) {
            share[e] = score[e];
            score[e] += correction != nullptr ? correction[e] : 0.0f;
        }
        __syncwarp();
    }
    if (groups > 0) {
        // a lane sums its groups' two best; then the groups that keep_groups others beat (the lower index wins a tie) drop out
        float* group_score = group_scores + warp * groups;
        const int size = n_outputs / groups;
        for (int g = lane; g < groups; g += 32) {
            float first = -INFINITY, second = -INFINITY;
            for (int e = g * size; e < (g + 1) * size; e++) {
                const float v = score[e];
                if (v > first) second = first, first = v;
                else if (v > second) second = v;
            }
            group_score[g] = size > 1 ? first + second : first;
        }
        __syncwarp();
        for (int e = lane; e < n_outputs; e += 32) {
            const int mine = e / size;
            int ahead = 0;
            for (int g = 0; g < groups; g++)
                ahead += group_score[g] > group_score[mine] || (group_score[g] == group_score[mine] && g < mine) ? 1 : 0;
            if (ahead >= keep_groups) score[e] = -INFINITY;
        }
        __syncwarp();
    }
    const int n_real = n_outputs - n_identity;
    float largest = 0.0f, total = 0.0f;
    for (int k = 0; k < top; k++) {
        int best = n_outputs;
        float best_score = -INFINITY;
        for (int e = lane; e < n_outputs; e += 32)
            if (score[e] > best_score) best = e, best_score = score[e];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const float other_score = __shfl_xor_sync(0xffffffffu, best_score, o);
            const int other = __shfl_xor_sync(0xffffffffu, best, o);
            if (other_score > best_score || (other_score == best_score && other < best)) best = other, best_score = other_score;
        }
        if (best >= n_outputs) best = 0, best_score = score[0];      // (scores that are no numbers)
        if (k == 0) largest = best_score;                            // (the first is the largest)
        float weight = best_score;
        if (rule == ROUTE_SOFTMAX_OF_CHOSEN) weight = expf(best_score - largest);
        if (rule == ROUTE_SOFTMAX_OF_ALL || rule == ROUTE_SIGMOID) weight = share[best];
        total += weight;
        if (lane == 0) {
            const long pair = (long)t * pairs + k;
            choice[pair] = best;
            in_weight[pair] = rule == ROUTE_SIGMOID_ON_INPUT ? weight : 1.0f;
            out_weight[pair] = rule == ROUTE_SIGMOID_ON_INPUT ? 1.0f : weight;
            score[best] = -INFINITY;
        }
        __syncwarp();
    }
    if (lane != 0) return;
    if (rule != ROUTE_SIGMOID_ON_INPUT) {
        // the chosen experts' weights over their own sum; an identity expert's goes to the token's input itself
        float passed = 0.0f;
        for (int k = 0; k < top; k++) {
            const long pair = (long)t * pairs + k;
            const float over = rule == ROUTE_SIGMOID ? 1.0f : (rule == ROUTE_SOFTMAX_OF_ALL ? total + 1e-20f : total);
            const float weight = out_weight[pair] / over * (rule == ROUTE_SOFTMAX_OF_CHOSEN ? 1.0f : scale);
            const bool identity = choice[pair] >= n_real;
            if (identity) passed += weight, choice[pair] = -1;
            out_weight[pair] = identity ? 0.0f : weight;
        }
        if (identity_weight != nullptr) identity_weight[t] = passed;
    }
    if (shared_gate != nullptr || shared_plain) {
        choice[(long)t * pairs + top] = n_real;
        in_weight[(long)t * pairs + top] = 1.0f;
        out_weight[(long)t * pairs + top] = shared_gate != nullptr ? score[n_outputs] : 1.0f;
    }
}

// The SM count of the current device (asked once per device).
static int sm_count() {
    static int counts[64] = {0};
    int device = 0;
    if (cudaGetDevice(&device) != cudaSuccess || device < 0 || device >= 64) return 148;
    if (counts[device] == 0) {
        int sms = 0;
        if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess || sms <= 0) sms = 148;
        counts[device] = sms;
    }
    return counts[device];
}

// What an expert applies between its two products: silu(gate) * up; (no gate matrix) the square of relu(up); or, with
// both products clamped, g' * sigmoid(alpha g') * (u' + 1) for g' = min(gate, limit), u' = clamp(up, -limit, limit).
enum ExpertForm { EXPERT_GATED_SILU = 0, EXPERT_RELU_SQUARED = 1, EXPERT_CLAMPED_GLU = 2 };

template <int FORM> __device__ __forceinline__ float expert_form(float g, float u, float limit, float alpha) {
    if (FORM == EXPERT_RELU_SQUARED) {
        const float r = fmaxf(u, 0.0f);
        return r * r;
    }
    if (FORM == EXPERT_CLAMPED_GLU) {
        g = fminf(g, limit), u = fminf(fmaxf(u, -limit), limit);
        return g * sigmoid_f(alpha * g) * (u + 1.0f);
    }
    return silu_f(g) * u;
}

// A warp takes F inner features of a pair at once: their rows' loads do not wait on one another.
// (the routed experts share one limit; expert `n_experts`, the shared one, has its own)
template <typename T, int FORM, int F>
__global__ void __launch_bounds__(256)
expert_up_kernel(T* __restrict__ act, long ld_act, const T* __restrict__ x, long ld_x, const int* __restrict__ choice,
                 const float* __restrict__ in_weight, const long long* __restrict__ gate_of, const long long* __restrict__ up_of,
                 const int* __restrict__ inner_of, int width, int pairs, float limit, float shared_limit, float alpha,
                 int n_experts) {
    constexpr bool GATED = FORM != EXPERT_RELU_SQUARED;
    dependents_may_start();
    wait_for_earlier_kernels();
    extern __shared__ __align__(16) float row[];             // [width]: the token times its weight, rounded as an activation
    const int pair = blockIdx.x, t = pair / pairs;
    const int e = choice[pair];
    if (e < 0) return;                         // (an identity expert: expert_down passes the input on)
    const int inner = inner_of[e];
    const int first = blockIdx.y * 8 * F;
    if (first >= inner) return;
    const float weight = in_weight[pair];
    for (int c = threadIdx.x; c < width; c += blockDim.x)
        row[c] = to_f32(from_f32<T>(weight * to_f32(x[(long)t * ld_x + c])));
    __syncthreads();
    const T* up = (const T*)up_of[e];
    const T* gate = GATED ? (const T*)gate_of[e] : up;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int f0 = first + warp * F;
    if (f0 >= inner) return;
    float zg[F], zu[F];
#pragma unroll
    for (int k = 0; k < F; k++) zg[k] = zu[k] = 0.0f;
    constexpr int N = Vec16<T>::N;
    if (width % N == 0 && aligned16(gate) && aligned16(up)) {
        for (int c = lane * N; c < width; c += 32 * N) {
            uint4 vg[F], vu[F];
#pragma unroll
            for (int k = 0; k < F; k++) {
                const long r = (long)min(f0 + k, inner - 1) * width + c;       // (past the end: the last row once more)
                if (GATED) vg[k] = *reinterpret_cast<const uint4*>(gate + r);
                vu[k] = *reinterpret_cast<const uint4*>(up + r);
            }
#pragma unroll
            for (int k = 0; k < F; k++) {
                float a[N], b[N];
                if (GATED) Vec16<T>::unpack(vg[k], a);
                Vec16<T>::unpack(vu[k], b);
#pragma unroll
                for (int i = 0; i < N; i++) {
                    if (GATED) zg[k] = fmaf(a[i], row[c + i], zg[k]);
                    zu[k] = fmaf(b[i], row[c + i], zu[k]);
                }
            }
        }
    } else {
        for (int c = lane; c < width; c += 32)
#pragma unroll
            for (int k = 0; k < F; k++) {
                const long r = (long)min(f0 + k, inner - 1) * width + c;
                if (GATED) zg[k] = fmaf(to_f32(gate[r]), row[c], zg[k]);
                zu[k] = fmaf(to_f32(up[r]), row[c], zu[k]);
            }
    }
#pragma unroll
    for (int k = 0; k < F; k++) {
        const float g = GATED ? warp_sum(zg[k]) : 0.0f, u = warp_sum(zu[k]);
        if (lane == 0 && f0 + k < inner)
            act[(long)pair * ld_act + f0 + k] = from_f32<T>(expert_form<FORM>(g, u, e == n_experts ? shared_limit : limit, alpha));
    }
}

// A warp takes C columns of a token's sum: every pair's loads of all of them are asked for together.
template <typename T, int C>
__global__ void __launch_bounds__(256)
expert_down_kernel(float* __restrict__ hidden, long ld_hidden, const T* __restrict__ act, long ld_act,
                   const int* __restrict__ choice, const float* __restrict__ out_weight, const long long* __restrict__ down_of,
                   const int* __restrict__ inner_of, long ld_down, int width, int pairs, int assign, const T* __restrict__ x,
                   long ld_x, const float* __restrict__ identity_weight) {
    dependents_may_start();
    wait_for_earlier_kernels();
    const int t = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int c0 = (blockIdx.y * 8 + warp) * C;
    if (c0 >= width) return;
    constexpr int N = Vec16<T>::N;
    float total[C];
#pragma unroll
    for (int q = 0; q < C; q++) total[q] = 0.0f;
#pragma unroll 2
    for (int k = 0; k < pairs; k++) {
        const long pair = (long)t * pairs + k;
        const int e = choice[pair];
        if (e < 0) continue;
        const int inner = inner_of[e];
        const T* w = (const T*)down_of[e];
        const T* a = act + pair * ld_act;
        float z[C];
#pragma unroll
        for (int q = 0; q < C; q++) z[q] = 0.0f;
        if (inner % N == 0 && ld_down % N == 0 && aligned16(w) && aligned16(a)) {
#pragma unroll 2
            for (int f = lane * N; f < inner; f += 32 * N) {
                uint4 v[C];
#pragma unroll
                for (int q = 0; q < C; q++) v[q] = *reinterpret_cast<const uint4*>(w + (long)min(c0 + q, width - 1) * ld_down + f);
                float y[N];
                Vec16<T>::load(a + f, y);
#pragma unroll
                for (int q = 0; q < C; q++) {
                    float b[N];
                    Vec16<T>::unpack(v[q], b);
#pragma unroll
                    for (int i = 0; i < N; i++) z[q] = fmaf(b[i], y[i], z[q]);
                }
            }
        } else {
            for (int f = lane; f < inner; f += 32)
#pragma unroll
                for (int q = 0; q < C; q++) z[q] = fmaf(to_f32(w[(long)min(c0 + q, width - 1) * ld_down + f]), to_f32(a[f]), z[q]);
        }
#pragma unroll
        for (int q = 0; q < C; q++) total[q] = fmaf(out_weight[pair], warp_sum(z[q]), total[q]);
    }
#pragma unroll
    for (int q = 0; q < C; q++) {
        const int c = c0 + q;
        if (lane != 0 || c >= width) continue;
        // identity experts hand the token on as it came
        if (identity_weight != nullptr) total[q] = fmaf(identity_weight[t], to_f32(x[(long)t * ld_x + c]), total[q]);
        float* h = hidden + (long)t * ld_hidden + c;
        *h = assign ? total[q] : *h + total[q];
    }
}

// ---- the pairs of few tokens, by expert ----------------------------------------------------------
// Up to EXPERT_TILE_TOKENS tokens, bfloat16, inner sizes and the width multiples of 8: the pairs of one expert go through mma.sync tiles
// (m16n8k16) together, so that an expert's weights cross the chip once however many tokens chose it, and the sums are the tensor
// cores', every product added by a rounded addition.  What bounds the two kernels are the weights' way from HBM (35 MB at 8 experts of 768 and a shared one of
// 1,536 with a width of 768: 5.4 us) and the chain of choice, lists, operands and sums behind the router.  So all of a block's
// weights are asked for at once, ahead of the wait for the kernels ahead where the tokens choose half as many experts as there are, and the
// first kernel's idle lanes bring the second one's into L2.  Both kernels, 1, 2, 8, 16, 31 tokens of such experts, replayed back to back:
// 14.2, 17.0, 18.0, 19.8, 24.5 us (16.1, 21.4, 24.3, 26.1, 32.3 by the kernels for wide rows below); in a decode step of 16 requests 17.8 us a
// layer where it was 25.4.
constexpr int EXPERT_TILE_TOKENS = 31, EXPERT_TABLES = 64, EXPERT_UNITS = 64, EXPERT_UNIT_K = 256;

// The pairs that chose expert e, in their order, by one warp: the list gets those from number `begin` on, 32 at most, and `place`
// (if there is one) a pair's place in it, -1 for those that found none.  Returns how many chose the expert in all: more than 32
// only where a token names an expert more than once, as the router does for a token whose scores are no numbers.
__device__ __forceinline__ int pairs_of_expert(const int* choice, int n_pairs, int e, int begin, int* list, int* place) {
    const int lane = threadIdx.x & 31;
    int count = 0;
    for (int first = 0; first < n_pairs; first += 32) {
        const int pair = first + lane;
        const bool mine = pair < n_pairs && choice[pair] == e;
        const unsigned all = __ballot_sync(0xffffffffu, mine);
        const int at = count + __popc(all & ((1u << lane) - 1u)) - begin;
        const bool listed = at >= 0 && at < 32;
        if (mine && listed) list[at] = pair;
        if (mine && place != nullptr) place[pair] = listed ? at : -1;
        count += __popc(all);
    }
    return count;
}

// Whether the weights of all experts are asked for ahead of the wait, before their tokens are known: where the tokens choose half as many
// experts as there are or more, a token's last pair not counted (where there is a shared expert it is that one's; where there is none, two tokens of 8
// experts, two each, are the faster behind the wait, too: 15.5 us ahead and 14.3).  What is read in vain costs less than the wait for what is
// not: the router's kernel runs meanwhile.  With a shared expert one token of 8, two each: 15.4 us behind the wait, 16.7 ahead; two: 18.4 and 17.7.
__device__ __forceinline__ bool experts_ahead(int n_tokens, int pairs, int n_experts) {
    return n_tokens * (pairs > 1 ? pairs - 1 : 1) * 2 >= n_experts;
}

// By one warp, two experts a lane: where the parts of the experts that `has` names begin, expert e's `parts_of(e)` of them, in
// first_part[0 .. n_tables]; returns their number.
template <typename Has, typename Parts>
__device__ __forceinline__ int parts_of_experts(int n_tables, int* first_part, Has has, Parts parts_of) {
    const int lane = threadIdx.x & 31;
    int mine[2];
#pragma unroll
    for (int h = 0; h < 2; h++) mine[h] = 2 * lane + h < n_tables && has(2 * lane + h) ? parts_of(2 * lane + h) : 0;
    int sum = mine[0] + mine[1];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int before = __shfl_up_sync(0xffffffffu, sum, o);
        if (lane >= o) sum += before;
    }
    const int total = __shfl_sync(0xffffffffu, sum, 31), start = sum - mine[0] - mine[1];
    if (2 * lane < n_tables) first_part[2 * lane] = start;
    if (2 * lane + 1 < n_tables) first_part[2 * lane + 1] = start + mine[0];
    if (lane == 0) first_part[n_tables] = total;
    return total;
}

// The expert of part number `part` (parts begin where parts_of_experts wrote), by one warp.
__device__ __forceinline__ int expert_of_part(const int* first_part, int n_tables, int part) {
    const int lane = threadIdx.x & 31;
    int e = 0;
    for (int first = 0; first < n_tables; first += 32) {
        const int at = first + lane;
        const unsigned here = __ballot_sync(0xffffffffu, at < n_tables && first_part[at] <= part && part < first_part[at + 1]);
        if (here != 0u) e = first + 31 - __clz(here);
    }
    return e;
}

// A warp: eight inner features of an expert with a gate (16 without): its tile's 16 rows are the gates and the ups of the same features,
// so that a lane holds both of a result; the tile's columns are pairs, eight at a time.  The weights lie in a ring of the lane's own
// in shared memory (`depth` blocks of 32 of K: all of them at a width of 768), the tokens beside them.
constexpr int EXPERT_UP_WARPS = 8, EXPERT_UP_SHARED = 224 * 1024, EXPERT_UP_BLOCK = EXPERT_UP_WARPS * 2 * 32 * 16;     // (bytes of a block of 32 of K)
constexpr int EXPERT_UP_STATIC = (EXPERT_UP_WARPS * 32 + EXPERT_TABLES + 1) * 4 + EXPERT_TABLES * 28 + 64;

template <int FORM>
__global__ void __launch_bounds__(EXPERT_UP_WARPS * 32, 1)
expert_up_tiles_kernel(bf16* __restrict__ act, long ld_act, const bf16* x, long ld_x, const int* choice, const float* in_weight,
                       const long long* __restrict__ gate_of, const long long* __restrict__ up_of, const long long* __restrict__ down_of,
                       const int* __restrict__ inner_of, int n_tables, long ld_down, int width, int pairs, int n_tokens, float limit,
                       float shared_limit, float alpha, int n_experts, int depth) {
    constexpr bool GATED = FORM != EXPERT_RELU_SQUARED;
    constexpr int FEATURES = GATED ? 8 : 16, THREADS = EXPERT_UP_WARPS * 32;
    __shared__ int lists[EXPERT_UP_WARPS][32], first_part[EXPERT_TABLES + 1], inner_here[EXPERT_TABLES];
    __shared__ long long gate_here[EXPERT_TABLES], up_here[EXPERT_TABLES], down_here[EXPERT_TABLES];
    extern __shared__ __align__(16) unsigned char up_shared[];
    uint4* ring = reinterpret_cast<uint4*>(up_shared);                        // [block of K][row of a lane][thread]
    const int n_pairs = n_tokens * pairs, pieces = width / 8, all = (width + 31) / 32;
    const int ld_held = width * 2 + (width % 64 == 0 ? 64 : 16);              // bytes: neighbouring rows in other banks
    unsigned char* held = up_shared + (size_t)depth * EXPERT_UP_BLOCK;
    int* chosen = reinterpret_cast<int*>(held + (size_t)n_tokens * ld_held);
    float* scales = reinterpret_cast<float*>(chosen + n_pairs);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, tq = lane & 3;
    const int half = depth / 2;
    dependents_may_start();
    for (int e = threadIdx.x; e < n_tables; e += THREADS) {
        inner_here[e] = __ldg(inner_of + e);
        gate_here[e] = GATED ? __ldg(gate_of + e) : 0;
        up_here[e] = __ldg(up_of + e);
        down_here[e] = __ldg(down_of + e);
    }
    __syncthreads();
    auto parts_of = [&](int e) { return (inner_here[e] + FEATURES - 1) / FEATURES; };
    const bool early = experts_ahead(n_tokens, pairs, n_experts);
    if (early) {
        if (warp == 0) parts_of_experts(n_tables, first_part, [](int) { return true; }, parts_of);
        __syncthreads();
    }
    const bf16 *low, *high;                                                   // this lane's rows of weights
    auto rows_of = [&](int e, int f0) {
        const int inner = inner_here[e];
        const bf16* up = reinterpret_cast<const bf16*>(up_here[e]);
        low = (GATED ? reinterpret_cast<const bf16*>(gate_here[e]) : up) + (long)min(f0 + g, inner - 1) * width + tq * 8;
        high = up + (long)min(f0 + (GATED ? 0 : 8) + g, inner - 1) * width + tq * 8;
    };
    auto ask = [&](int which, int first) {                                    // half the ring: blocks of K from `first` on
        for (int i = 0; i < half; i++) {
            const bool there = first + i < all && (first + i) * 4 + tq < pieces;
            uint4* to = ring + (size_t)(which * half + i) * 2 * THREADS + threadIdx.x;
            if (first + i < all) {
                copy_16(to, there ? low + (first + i) * 32 : low - tq * 8, there);
                copy_16(to + THREADS, there ? high + (first + i) * 32 : high - tq * 8, there);
            }
        }
        copies_end();
    };
    const int walker = warp * gridDim.x + blockIdx.x, walkers = EXPERT_UP_WARPS * gridDim.x;     // neighbouring parts on different SMs
    auto begin_part = [&](int part, int& e, int& f0) {
        e = expert_of_part(first_part, n_tables, part);
        f0 = (part - first_part[e]) * FEATURES;
        rows_of(e, f0);
        ask(0, 0);
        ask(1, half);
    };
    // the other kernel's weights come into L2 meanwhile, an expert's piece of a row at a time (the launcher sees to width <= walkers; with a
    // division to find each piece's expert, those without a token cost as much as those with one: one token of 60 experts 21.4 us, 18.5 so)
    auto down_ahead = [&](auto has) {
        int at_row = walker;
        for (int e = 0; e < n_tables; e++) {
            if (at_row < width && has(e)) {
                const char* row = reinterpret_cast<const char*>(down_here[e]) + (long)at_row * ld_down * 2;
                const int bytes = inner_here[e] * 2;
                for (int at = lane * 128; at < bytes; at += 32 * 128) asm volatile("prefetch.global.L2 [%0];" ::"l"(row + at));
            }
            at_row -= width;
            if (at_row < 0) at_row += walkers;
        }
    };
    int part = walker, e = 0, f0 = 0;
    if (early) {
        if (part < first_part[n_tables]) begin_part(part, e, f0);
        down_ahead([](int) { return true; });
    }
    wait_for_earlier_kernels();
    choice = behind_the_wait(choice);
    x = behind_the_wait(x);
    in_weight = behind_the_wait(in_weight);
    for (int t = warp; t < n_tokens; t += EXPERT_UP_WARPS)
        for (int c = lane; c < pieces; c += 32) copy_16(held + (size_t)t * ld_held + c * 16, x + (long)t * ld_x + c * 8, true);
    copies_end();
    for (int i = threadIdx.x; i < n_pairs; i += THREADS) {
        chosen[i] = choice[i];
        scales[i] = in_weight[i];
    }
    __syncthreads();
    if (!early) {
        // only the experts that have a pair
        auto has = [&](int expert) {
            bool found = false;
            for (int i = 0; i < n_pairs; i++) found |= chosen[i] == expert;
            return found;
        };
        if (warp == 0) parts_of_experts(n_tables, first_part, has, parts_of);
        __syncthreads();
        if (part < first_part[n_tables]) begin_part(part, e, f0);
        down_ahead([&](int expert) { return first_part[expert] < first_part[expert + 1]; });
    }
    copies_landed<0>();
    __syncthreads();                                                          // the tokens are there, whoever copied them
    // the listed pairs, eight a tile, times the weights in the ring
    auto multiply = [&](auto tiles, int here, int e, int f0, const int* list) {
        constexpr int TILES = decltype(tiles)::value;
        const uint4 none = make_uint4(0u, 0u, 0u, 0u);
        const unsigned char* row[TILES];
        float scale[TILES];
        bool scaled = false;
#pragma unroll
        for (int t = 0; t < TILES; t++) {
            // (a column without a pair repeats the first one's and is not stored)
            const int pair = list[t * 8 + g < here ? t * 8 + g : 0], token = pair / pairs;
            row[t] = held + (size_t)token * ld_held;
            scale[t] = scales[pair];
            scaled |= scale[t] != 1.0f;
        }
        scaled = __any_sync(0xffffffffu, scaled);
        float sums[TILES][4][4];                                              // [tile of pairs][in turn][entry]
#pragma unroll
        for (int t = 0; t < TILES; t++)
#pragma unroll
            for (int i = 0; i < 16; i++) sums[t][i / 4][i % 4] = 0.0f;
        for (int first = 0, which = 0; first < all; first += half, which ^= 1) {
            copies_landed<1>();
            const uint4* mine = ring + (size_t)which * half * 2 * THREADS + threadIdx.x;
            const int here_blocks = min(half, all - first);
            // four blocks of K at a time: their loads do not wait on one another
            for (int i = 0; i < here_blocks; i += 4) {
                uint4 a[4], b[4], v[4][TILES];
#pragma unroll
                for (int u = 0; u < 4; u++) {
                    const int c = (first + i + u) * 4 + tq;
                    const bool there = i + u < here_blocks;
                    a[u] = there ? mine[(size_t)(i + u) * 2 * THREADS] : none;
                    b[u] = there ? mine[(size_t)(i + u) * 2 * THREADS + THREADS] : none;
#pragma unroll
                    for (int t = 0; t < TILES; t++) v[u][t] = there && c < pieces ? *reinterpret_cast<const uint4*>(row[t] + c * 16) : none;
                }
                if (scaled)                                                   // the inputs' weights, rounded as activations
#pragma unroll
                    for (int u = 0; u < 4; u++)
#pragma unroll
                        for (int t = 0; t < TILES; t++) {
                            float y[8];
                            Vec16<bf16>::unpack(v[u][t], y);
                            __nv_bfloat162 two[4];
#pragma unroll
                            for (int k = 0; k < 4; k++) two[k] = __floats2bfloat162_rn(scale[t] * y[2 * k], scale[t] * y[2 * k + 1]);
                            v[u][t] = *reinterpret_cast<const uint4*>(two);
                        }
#pragma unroll
                for (int u = 0; u < 4; u++) {
                    const uint32_t even[4] = {a[u].x, b[u].x, a[u].y, b[u].y}, odd[4] = {a[u].z, b[u].z, a[u].w, b[u].w};
#pragma unroll
                    for (int t = 0; t < TILES; t++) {
                        mma_added(sums[t][2 * (u & 1)], even, v[u][t].x, v[u][t].y);
                        mma_added(sums[t][2 * (u & 1) + 1], odd, v[u][t].z, v[u][t].w);
                    }
                }
            }
            ask(which, first + 2 * half);
        }
        float z[TILES][2][2];                                                 // [tile][pair][row]
#pragma unroll
        for (int t = 0; t < TILES; t++)
#pragma unroll
            for (int i = 0; i < 4; i++) z[t][i & 1][i >> 1] = (sums[t][0][i] + sums[t][1][i]) + (sums[t][2][i] + sums[t][3][i]);
        const int inner = inner_here[e];
        const float most = e == n_experts ? shared_limit : limit;
#pragma unroll
        for (int t = 0; t < TILES; t++)
#pragma unroll
            for (int j = 0; j < 2; j++) {
                const int at = t * 8 + 2 * tq + j;
                if (at >= here) continue;
                bf16* to = act + (long)list[at] * ld_act + f0 + g;
                if (GATED) {
                    if (f0 + g < inner) *to = __float2bfloat16_rn(expert_form<FORM>(z[t][j][0], z[t][j][1], most, alpha));
                } else {
                    if (f0 + g < inner) to[0] = __float2bfloat16_rn(expert_form<FORM>(0.0f, z[t][j][0], most, alpha));
                    if (f0 + 8 + g < inner) to[8] = __float2bfloat16_rn(expert_form<FORM>(0.0f, z[t][j][1], most, alpha));
                }
            }
    };
    const int parts = first_part[n_tables];
    for (; part < parts; part += walkers) {
        if (part != walker) begin_part(part, e, f0);
        int* list = lists[warp];
        int m0 = 0, count;
        do {
            // up to 32 pairs at a time
            __syncwarp();
            count = pairs_of_expert(chosen, n_pairs, e, m0, list, nullptr);
            __syncwarp();
            const int here = min(32, count - m0);
            if (m0 > 0) {
                ask(0, 0);
                ask(1, half);
            }
            if (here > 0 && here <= 8) multiply(std::integral_constant<int, 1>(), here, e, f0, list);
            else if (here > 8 && here <= 16) multiply(std::integral_constant<int, 2>(), here, e, f0, list);
            else if (here > 16) multiply(std::integral_constant<int, 4>(), here, e, f0, list);
            m0 += 32;
        } while (m0 < count);
        copies_landed<0>();
    }
}

// A block: eight columns of the sum, all tokens.  A unit is an expert's pairs and EXPERT_UNIT_K of its inner size (all of it
// where the experts would bring more units than there is room for); sixteen warps take the units in turn, whose weights they ask
// for two units ahead, and a token's column adds its pairs' units in their order.
constexpr int EXPERT_DOWN_AHEAD = 2, EXPERT_DOWN_SUMS = EXPERT_UNITS * 32 * 8 * 4, EXPERT_DOWN_RING = 16 * EXPERT_DOWN_AHEAD * EXPERT_UNIT_K * 8 * 2;
constexpr size_t EXPERT_DOWN_SHARED = 215 * 1024;
__global__ void __launch_bounds__(512)
expert_down_tiles_kernel(float* hidden, long ld_hidden, const bf16* act, long ld_act, const int* choice, const float* out_weight,
                         const long long* __restrict__ down_of, const int* __restrict__ inner_of, int n_tables, long ld_down,
                         int width, int pairs, int n_tokens, int assign, const bf16* x, long ld_x, const float* identity_weight,
                         int n_experts, int ahead, int held_pairs) {
    constexpr int BLOCKS = EXPERT_UNIT_K / 32;
    __shared__ int list[EXPERT_TABLES][32], count_of[EXPERT_TABLES], first_unit[EXPERT_TABLES + 1], inner_here[EXPERT_TABLES], unit_k;
    __shared__ long long down_here[EXPERT_TABLES];
    extern __shared__ __align__(16) float down_shared[];     // [units][32 rows][8 columns], the weights asked for ahead, the pairs' places, (held_pairs) choices and weights
    uint4* ring = reinterpret_cast<uint4*>(down_shared + EXPERT_UNITS * 32 * 8);                  // [ahead][block of K][thread]
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, tq = lane & 3;
    const int c0 = blockIdx.x * 8, n_pairs = n_tokens * pairs;
    int* place = reinterpret_cast<int*>(ring + ahead * BLOCKS * 512);
    dependents_may_start();
    for (int e = threadIdx.x; e < n_tables; e += 512) {
        inner_here[e] = __ldg(inner_of + e);
        down_here[e] = __ldg(down_of + e);
    }
    __syncthreads();
    // how many units every expert has, and where they begin
    auto plan = [&](auto has) {
        if (warp == 0) {
            int size = EXPERT_UNIT_K;
            if (parts_of_experts(n_tables, first_unit, has, [&](int e) { return (inner_here[e] + EXPERT_UNIT_K - 1) / EXPERT_UNIT_K; }) > EXPERT_UNITS) {
                parts_of_experts(n_tables, first_unit, has, [](int) { return 1; });
                size = 0;
            }
            if (lane == 0) unit_k = size;
        }
        __syncthreads();
    };
    auto row_of = [&](int e) { return reinterpret_cast<const bf16*>(down_here[e]) + (long)min(c0 + g, width - 1) * ld_down; };
    auto ask = [&]() {                                       // the weights of this warp's first units
        for (int a = 0; a < ahead; a++) {
            const int unit = warp + 16 * a;
            if (unit_k == 0 || unit >= first_unit[n_tables]) break;
            const int e = expert_of_part(first_unit, n_tables, unit);
            const int k_first = (unit - first_unit[e]) * EXPERT_UNIT_K, k_end = min(inner_here[e], k_first + EXPERT_UNIT_K);
            const bf16* w = row_of(e);
#pragma unroll
            for (int i = 0; i < BLOCKS; i++) {
                const int k = k_first + i * 32 + tq * 8;
                copy_16(ring + (a * BLOCKS + i) * 512 + threadIdx.x, k < k_end ? w + k : w, k < k_end);
            }
        }
        copies_end();
    };
    // (all experts may be more units than there is room for where the chosen ones are not: planning again for those behind the wait was slower, 24 experts
    // of 768, 16 and 31 tokens 31.5 and 35.8 us so, 33.7 and 37.1 then)
    const bool early = experts_ahead(n_tokens, pairs, n_experts);
    if (early) {
        plan([](int) { return true; });
        ask();
    }
    wait_for_earlier_kernels();
    choice = behind_the_wait(choice);
    act = behind_the_wait(act);
    out_weight = behind_the_wait(out_weight);
    x = behind_the_wait(x);
    const int* chosen = choice;
    const float* scales = out_weight;
    if (held_pairs) {
        int* to = place + n_pairs;
        for (int i = threadIdx.x; i < n_pairs; i += 512) {
            to[i] = choice[i];
            to[n_pairs + i] = __float_as_int(out_weight[i]);
        }
        chosen = to;
        scales = reinterpret_cast<const float*>(to + n_pairs);
    }
    // the sum that the first result of this thread joins
    const int t_mine = threadIdx.x / 8, c_mine = c0 + threadIdx.x % 8;
    const bool mine = t_mine < n_tokens && c_mine < width;
    const float hidden_mine = mine && !assign ? hidden[(long)t_mine * ld_hidden + c_mine] : 0.0f;
    __syncthreads();
    for (int e = warp; e < n_tables; e += 16) {
        const int count = pairs_of_expert(chosen, n_pairs, e, 0, list[e], place);
        if (lane == 0) count_of[e] = min(count, 32);
    }
    __syncthreads();
    if (!early) {
        plan([&](int e) { return count_of[e] > 0; });
        ask();
    }
    const int units = first_unit[n_tables];
    const uint4 none = make_uint4(0u, 0u, 0u, 0u);
    copies_landed<0>();
    for (int unit = warp, turn = 0; unit < units; unit += 16, turn++) {
        const int e = expert_of_part(first_unit, n_tables, unit);
        const int inner = inner_here[e], count = count_of[e];
        const int k_first = unit_k > 0 ? (unit - first_unit[e]) * unit_k : 0, k_end = unit_k > 0 ? min(inner, k_first + unit_k) : inner;
        const uint4* w = reinterpret_cast<const uint4*>(row_of(e));
        const bool asked = unit_k > 0 && turn < ahead;
        for (int m0 = 0; m0 < count; m0 += 16) {
            const uint4* ar[2];
#pragma unroll
            for (int r = 0; r < 2; r++)
                ar[r] = m0 + r * 8 + g < count ? reinterpret_cast<const uint4*>(act + (long)list[e][m0 + r * 8 + g] * ld_act) : nullptr;
            float z[4] = {0.0f, 0.0f, 0.0f, 0.0f};
            for (int k0 = k_first; k0 < k_end; k0 += EXPERT_UNIT_K) {
                uint4 wv[BLOCKS], av[BLOCKS][2];
#pragma unroll
                for (int i = 0; i < BLOCKS; i++) {
                    const int c = k0 / 8 + i * 4 + tq;
                    const bool there = c * 8 < k_end;
                    wv[i] = asked ? ring[(turn * BLOCKS + i) * 512 + threadIdx.x] : there ? __ldg(w + c) : none;
#pragma unroll
                    for (int r = 0; r < 2; r++) av[i][r] = there && ar[r] != nullptr ? ar[r][c] : none;
                }
#pragma unroll
                for (int i = 0; i < BLOCKS; i++) {
                    const uint32_t first_half[4] = {av[i][0].x, av[i][1].x, av[i][0].y, av[i][1].y};
                    const uint32_t second_half[4] = {av[i][0].z, av[i][1].z, av[i][0].w, av[i][1].w};
                    mma_added(z, first_half, wv[i].x, wv[i].y);
                    mma_added(z, second_half, wv[i].z, wv[i].w);
                }
            }
            float* to = down_shared + (unit * 32 + m0 + g) * 8 + 2 * tq;
            to[0] = z[0], to[1] = z[1];
            to[64] = z[2], to[65] = z[3];
        }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < n_tokens * 8; i += 512) {
        const int t = i / 8, c = c0 + i % 8;
        if (c >= width) continue;
        float total = 0.0f;
        for (int k = 0; k < pairs; k++) {
            const int pair = t * pairs + k, e = chosen[pair];
            if (e < 0 || e >= n_tables) continue;
            if (place[pair] < 0) {                           // beyond an expert's 32 (a token that named it more than once): by itself
                const bf16* row = act + (long)pair * ld_act;
                const bf16* w = reinterpret_cast<const bf16*>(down_here[e]) + (long)c * ld_down;
                float z = 0.0f;
                for (int f = 0; f < inner_here[e]; f++) z = fmaf(to_f32(row[f]), to_f32(w[f]), z);
                total = fmaf(scales[pair], z, total);
                continue;
            }
            float z = 0.0f;
            for (int u = first_unit[e]; u < first_unit[e + 1]; u++) z += down_shared[(u * 32 + place[pair]) * 8 + i % 8];
            total = fmaf(scales[pair], z, total);
        }
        if (identity_weight != nullptr) total = fmaf(behind_the_wait(identity_weight)[t], to_f32(x[(long)t * ld_x + c]), total);
        float* h = hidden + (long)t * ld_hidden + c;
        *h = assign ? total : (i == (int)threadIdx.x ? hidden_mine : *h) + total;
    }
}

// Rows wider than the second kernel above has blocks for at once (eight columns each, one an SM): the same by more and smaller blocks, weights
// in registers, two and more of them an SM.  8 experts of 1,024, two a token, 16 tokens, these kernels against those: width 1,024 25.3
// and 23.2 us, 1,280 29.3 and 32.3, 2,048 34.5 and 43.1.
// A block: 16 inner features of an expert, in two tiles of 8 whose K four warps share.
template <int FORM>
__global__ void __launch_bounds__(256, 2)
expert_up_blocks_kernel(bf16* __restrict__ act, long ld_act, const bf16* x, long ld_x, const int* choice, const float* in_weight,
                       const long long* __restrict__ gate_of, const long long* __restrict__ up_of, const int* __restrict__ inner_of,
                       int width, int pairs, int n_tokens, float limit, float shared_limit, float alpha, int n_experts) {
    constexpr bool GATED = FORM != EXPERT_RELU_SQUARED;
    constexpr int AHEAD = 4;
    __shared__ int list[32], found;                          // (32 pairs at a time)
    __shared__ float sums[2][8][16][9];                      // [gate, up][warp][row][feature]
    const int e = blockIdx.y, inner = __ldg(inner_of + e);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, tq = lane & 3;
    const int f_block = blockIdx.x * 16, f0 = f_block + (warp >> 2) * 8;
    dependents_may_start();
    if (f_block >= inner) return;
    const int pieces = width / 8, all = (width + 31) / 32, each = (all + 3) / 4;
    const int begin = (warp & 3) * each, end = f0 < inner ? min(all, begin + each) : begin;
    const long row = (long)min(f0 + g, inner - 1) * pieces;
    const uint4* up = reinterpret_cast<const uint4*>(__ldg(up_of + e)) + row;
    const uint4* gate = GATED ? reinterpret_cast<const uint4*>(__ldg(gate_of + e)) + row : up;
    const uint4 none = make_uint4(0u, 0u, 0u, 0u);
    uint4 wu[AHEAD], wg[AHEAD];
    auto weights = [&](int i, int block) {
        const int c = block * 4 + tq;
        const bool there = block < end && c < pieces;
        wu[i] = there ? __ldg(up + c) : none;
        if (GATED) wg[i] = there ? __ldg(gate + c) : none;
    };
    // (ahead of the wait only where nearly every expert will have a token: a step of one reads four of eight)
    const bool early = n_tokens * (pairs > 1 ? pairs - 1 : 1) >= n_experts;
    if (early)
#pragma unroll
        for (int i = 0; i < AHEAD; i++) weights(i, begin + i);
    wait_for_earlier_kernels();
    choice = behind_the_wait(choice);
    x = behind_the_wait(x);
    in_weight = behind_the_wait(in_weight);
    if (warp == 0) {
        const int count = pairs_of_expert(choice, n_tokens * pairs, e, 0, list, nullptr);
        if (lane == 0) found = count;
    }
    __syncthreads();
    const int count = found;
    for (int m0 = 0; m0 < count; m0 += 16) {
        if (m0 > 0 && m0 % 32 == 0) {                        // (every thread left the list before the barrier that ended the last tile)
            if (warp == 0) pairs_of_expert(choice, n_tokens * pairs, e, m0, list, nullptr);
            __syncthreads();
        }
        const int* listed = list + m0 % 32;
        if (m0 > 0 || !early)
#pragma unroll
            for (int i = 0; i < AHEAD; i++) weights(i, begin + i);
        // rows g and g + 8 of the tile: the tokens of two pairs and the weight their entries get
        const uint4* xr[2];
        float scale[2];
#pragma unroll
        for (int r = 0; r < 2; r++) {
            const bool there = m0 + r * 8 + g < count;
            const int pair = there ? listed[r * 8 + g] : 0;
            xr[r] = there ? reinterpret_cast<const uint4*>(x + (long)(pair / pairs) * ld_x) : nullptr;
            scale[r] = there ? in_weight[pair] : 1.0f;
        }
        float zg[4] = {0.0f, 0.0f, 0.0f, 0.0f}, zu[4] = {0.0f, 0.0f, 0.0f, 0.0f};
        for (int first = begin; first < end; first += AHEAD) {
            uint4 xv[AHEAD][2];
#pragma unroll
            for (int i = 0; i < AHEAD; i++)
#pragma unroll
                for (int r = 0; r < 2; r++) {
                    const int c = (first + i) * 4 + tq;
                    xv[i][r] = xr[r] != nullptr && first + i < end && c < pieces ? xr[r][c] : none;
                }
#pragma unroll
            for (int i = 0; i < AHEAD; i++) {
                const uint4 u = wu[i], v = GATED ? wg[i] : none;
                weights(i, first + AHEAD + i);
#pragma unroll
                for (int r = 0; r < 2; r++)
                    if (scale[r] != 1.0f) {                  // the input's weight, rounded as an activation
                        float y[8];
                        Vec16<bf16>::unpack(xv[i][r], y);
                        __nv_bfloat162 two[4];
#pragma unroll
                        for (int k = 0; k < 4; k++) two[k] = __floats2bfloat162_rn(scale[r] * y[2 * k], scale[r] * y[2 * k + 1]);
                        xv[i][r] = *reinterpret_cast<const uint4*>(two);
                    }
                const uint32_t first_half[4] = {xv[i][0].x, xv[i][1].x, xv[i][0].y, xv[i][1].y}, second_half[4] = {xv[i][0].z, xv[i][1].z, xv[i][0].w, xv[i][1].w};
                mma_added(zu, first_half, u.x, u.y);
                mma_added(zu, second_half, u.z, u.w);
                if (GATED) {
                    mma_added(zg, first_half, v.x, v.y);
                    mma_added(zg, second_half, v.z, v.w);
                }
            }
        }
#pragma unroll
        for (int i = 0; i < 4; i++) {
            sums[1][warp][g + (i >> 1) * 8][2 * tq + (i & 1)] = zu[i];
            if (GATED) sums[0][warp][g + (i >> 1) * 8][2 * tq + (i & 1)] = zg[i];
        }
        __syncthreads();
        const int f = threadIdx.x & 15, r = threadIdx.x >> 4;
        if (m0 + r < count && f_block + f < inner) {
            float a = 0.0f, b = 0.0f;
            for (int s = 0; s < 4; s++) {
                if (GATED) a += sums[0][(f >> 3) * 4 + s][r][f & 7];
                b += sums[1][(f >> 3) * 4 + s][r][f & 7];
            }
            act[(long)listed[r] * ld_act + f_block + f] =
                __float2bfloat16_rn(expert_form<FORM>(a, b, e == n_experts ? shared_limit : limit, alpha));
        }
        __syncthreads();
    }
}

// A block: eight columns of the sum, all tokens.  A unit is an expert's pairs and EXPERT_UNIT_K of its inner size (all of it
// where the chosen experts would bring more units than there is room for); sixteen warps take the units in turn, and a
// token's column adds its pairs' units in their order.
__global__ void __launch_bounds__(512)
expert_down_blocks_kernel(float* hidden, long ld_hidden, const bf16* act, long ld_act, const int* choice, const float* out_weight,
                         const long long* __restrict__ down_of, const int* __restrict__ inner_of, int n_tables, long ld_down,
                         int width, int pairs, int n_tokens, int assign, const bf16* x, long ld_x, const float* identity_weight) {
    constexpr int BLOCKS = EXPERT_UNIT_K / 32;
    __shared__ int list[EXPERT_TABLES][32], count_of[EXPERT_TABLES], first_unit[EXPERT_TABLES + 1], unit_k;
    extern __shared__ float down_shared[];                   // [units][32 rows][8 columns], then the pairs' places as ints
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, tq = lane & 3;
    const int c0 = blockIdx.x * 8, n_pairs = n_tokens * pairs;
    int* place = reinterpret_cast<int*>(down_shared + EXPERT_UNITS * 32 * 8);
    dependents_may_start();
    wait_for_earlier_kernels();
    choice = behind_the_wait(choice);
    act = behind_the_wait(act);
    out_weight = behind_the_wait(out_weight);
    x = behind_the_wait(x);
    for (int e = warp; e < n_tables; e += 16) {
        const int count = pairs_of_expert(choice, n_pairs, e, 0, list[e], place);
        if (lane == 0) count_of[e] = min(count, 32);
    }
    __syncthreads();
    if (warp == 0) {
        // how many units every expert has, and where they begin: two experts a lane
        int size = EXPERT_UNIT_K, total = 0;
        for (int attempt = 0; attempt < 2; attempt++) {
            int mine[2];
#pragma unroll
            for (int h = 0; h < 2; h++) {
                const int e = 2 * lane + h;
                mine[h] = e < n_tables && count_of[e] > 0 ? (attempt == 0 ? (__ldg(inner_of + e) + EXPERT_UNIT_K - 1) / EXPERT_UNIT_K : 1) : 0;
            }
            int sum = mine[0] + mine[1];
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int before = __shfl_up_sync(0xffffffffu, sum, o);
                if (lane >= o) sum += before;
            }
            total = __shfl_sync(0xffffffffu, sum, 31);
            const int start = sum - mine[0] - mine[1];
            if (2 * lane < n_tables) first_unit[2 * lane] = start;
            if (2 * lane + 1 < n_tables) first_unit[2 * lane + 1] = start + mine[0];
            size = attempt == 0 ? EXPERT_UNIT_K : 0;
            if (total <= EXPERT_UNITS) break;
        }
        if (lane == 0) {
            first_unit[n_tables] = total;
            unit_k = size;
        }
    }
    __syncthreads();
    const int units = first_unit[n_tables];
    const uint4 none = make_uint4(0u, 0u, 0u, 0u);
    for (int unit = warp; unit < units; unit += 16) {
        int e = 0;                                           // the last expert that begins at or before this unit and has units
        for (int first = 0; first < n_tables; first += 32) {
            const int at = first + lane;
            const unsigned here = __ballot_sync(0xffffffffu, at < n_tables && count_of[at] > 0 && first_unit[at] <= unit);
            if (here != 0u) e = first + 31 - __clz(here);
        }
        const int inner = __ldg(inner_of + e), count = count_of[e];
        const int k_first = unit_k > 0 ? (unit - first_unit[e]) * unit_k : 0, k_end = unit_k > 0 ? min(inner, k_first + unit_k) : inner;
        const uint4* w = reinterpret_cast<const uint4*>(reinterpret_cast<const bf16*>(__ldg(down_of + e)) + (long)min(c0 + g, width - 1) * ld_down);
        for (int m0 = 0; m0 < count; m0 += 16) {
            const uint4* ar[2];
#pragma unroll
            for (int r = 0; r < 2; r++)
                ar[r] = m0 + r * 8 + g < count ? reinterpret_cast<const uint4*>(act + (long)list[e][m0 + r * 8 + g] * ld_act) : nullptr;
            float z[4] = {0.0f, 0.0f, 0.0f, 0.0f};
            for (int k0 = k_first; k0 < k_end; k0 += EXPERT_UNIT_K) {
                uint4 wv[BLOCKS], av[BLOCKS][2];
#pragma unroll
                for (int i = 0; i < BLOCKS; i++) {
                    const int c = k0 / 8 + i * 4 + tq;
                    const bool there = c * 8 < k_end;
                    wv[i] = there ? __ldg(w + c) : none;
#pragma unroll
                    for (int r = 0; r < 2; r++) av[i][r] = there && ar[r] != nullptr ? ar[r][c] : none;
                }
#pragma unroll
                for (int i = 0; i < BLOCKS; i++) {
                    const uint32_t first_half[4] = {av[i][0].x, av[i][1].x, av[i][0].y, av[i][1].y};
                    const uint32_t second_half[4] = {av[i][0].z, av[i][1].z, av[i][0].w, av[i][1].w};
                    mma_added(z, first_half, wv[i].x, wv[i].y);
                    mma_added(z, second_half, wv[i].z, wv[i].w);
                }
            }
            float* mine = down_shared + (unit * 32 + m0 + g) * 8 + 2 * tq;
            mine[0] = z[0], mine[1] = z[1];
            mine[64] = z[2], mine[65] = z[3];
        }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < n_tokens * 8; i += 512) {
        const int t = i / 8, c = c0 + i % 8;
        if (c >= width) continue;
        float total = 0.0f;
        for (int k = 0; k < pairs; k++) {
            const int pair = t * pairs + k, e = choice[pair];
            if (e < 0 || e >= n_tables) continue;
            if (place[pair] < 0) {                           // beyond an expert's 32 (a token that named it more than once): by itself
                const bf16* row = act + (long)pair * ld_act;
                const bf16* w = reinterpret_cast<const bf16*>(__ldg(down_of + e)) + (long)c * ld_down;
                float z = 0.0f;
                for (int f = 0; f < __ldg(inner_of + e); f++) z = fmaf(to_f32(row[f]), to_f32(w[f]), z);
                total = fmaf(out_weight[pair], z, total);
                continue;
            }
            const int last = unit_k > 0 ? first_unit[e] + (__ldg(inner_of + e) + EXPERT_UNIT_K - 1) / EXPERT_UNIT_K : first_unit[e] + 1;
            float z = 0.0f;
            for (int u = first_unit[e]; u < last; u++) z += down_shared[(u * 32 + place[pair]) * 8 + i % 8];
            total = fmaf(out_weight[pair], z, total);
        }
        if (identity_weight != nullptr) total = fmaf(behind_the_wait(identity_weight)[t], to_f32(x[(long)t * ld_x + c]), total);
        float* h = hidden + (long)t * ld_hidden + c;
        *h = assign ? total : *h + total;
    }
}

// gu: [T, 2 * total] = [gates of all experts | ups of all experts]; act: [T, total].  Columns
// [e * inner, (e + 1) * inner) belong to routed expert e, columns from n_experts * inner on to the
// shared expert (pair index `top` of every token, if there is one).
// (VEC: a thread takes the 16 bytes of columns that lie side by side, all of one expert: inner sizes that are
// multiples of a vector's elements.  The token's weights per expert lie in shared memory, 0 for an expert it
// did not choose, whose columns are written as zeros without reading the products.)
// (EXPERT_RELU_SQUARED: experts without a gate matrix; gu holds the ups alone, [T, total], and act is the square of relu.
// With `identity_weight` the block's share of the token's columns of `hidden` also gets identity_weight[t] * x[t]:
// set to it with `assign`, else added.)
template <typename T, bool VEC, int FORM>
__global__ void __launch_bounds__(256)
expert_combine_kernel(T* __restrict__ act, long ld_act, const T* __restrict__ gu, long ld_gu, const int* __restrict__ choice,
                      const float* __restrict__ in_weight, const float* __restrict__ out_weight, int n_experts, int inner,
                      int total, int top, int pairs, float* __restrict__ hidden, long ld_hidden, const T* __restrict__ x,
                      long ld_x, const float* __restrict__ identity_weight, int width, int assign, float limit,
                      float shared_limit, float alpha) {
    constexpr bool GATED = FORM != EXPERT_RELU_SQUARED;
    dependents_may_start();
    wait_for_earlier_kernels();
    extern __shared__ float weights[];             // [n_experts + 1][2]: input weight, output weight
    const int t = blockIdx.x;
    for (int e = threadIdx.x; e <= n_experts; e += blockDim.x) {
        float s = 0.0f, o = 1.0f;
        if (e == n_experts) {
            if (pairs > top) s = in_weight[(long)t * pairs + top], o = out_weight[(long)t * pairs + top];
        } else {
            for (int k = 0; k < top; k++)
                if (choice[(long)t * pairs + k] == e) s = in_weight[(long)t * pairs + k], o = out_weight[(long)t * pairs + k];
        }
        weights[2 * e] = s, weights[2 * e + 1] = o;
    }
    __syncthreads();
    constexpr int N = VEC ? Vec16<T>::N : 1;
    const T* row = gu + (long)t * ld_gu;
    T* dst = act + (long)t * ld_act;
    for (int c = (blockIdx.y * blockDim.x + threadIdx.x) * N; c < total; c += gridDim.y * blockDim.x * N) {
        const int e = c < n_experts * inner ? c / inner : n_experts;
        const float s = weights[2 * e], o = weights[2 * e + 1];
        const float most = e == n_experts ? shared_limit : limit;
        if (VEC) {
            uint4 packed = make_uint4(0u, 0u, 0u, 0u);
            if (s != 0.0f) {
                float g[N], u[N];
                if (GATED) Vec16<T>::load(row + c, g);
                Vec16<T>::load(row + (GATED ? total : 0) + c, u);
                T* lanes = reinterpret_cast<T*>(&packed);
#pragma unroll
                for (int i = 0; i < N; i++)
                    lanes[i] = from_f32<T>(expert_form<FORM>(GATED ? s * g[i] : 0.0f, s * u[i], most, alpha) * o);
            }
            *reinterpret_cast<uint4*>(dst + c) = packed;
        } else {
            float v = 0.0f;
            if (s != 0.0f)
                v = expert_form<FORM>(GATED ? s * to_f32(row[c]) : 0.0f, s * to_f32(row[(GATED ? total : 0) + c]), most, alpha) * o;
            dst[c] = from_f32<T>(v);
        }
    }
    if (identity_weight != nullptr) {
        const float passed = identity_weight[t];
        if (assign || passed != 0.0f)
            for (int c = blockIdx.y * blockDim.x + threadIdx.x; c < width; c += gridDim.y * blockDim.x) {
                const float v = passed * to_f32(x[(long)t * ld_x + c]);
                float* h = hidden + (long)t * ld_hidden + c;
                *h = assign ? v : *h + v;
            }
    }
}

extern "C" int mllm_hybrid_expert_combine(void* act, long ld_act, const void* gu, long ld_gu, const int* choice,
                                          const float* in_weight, const float* out_weight, int n_experts, int inner, int total,
                                          int top, int pairs, int form, float limit, float shared_limit, float alpha, float* hidden, long ld_hidden, const void* x, long ld_x,
                                          const float* identity_weight, int width, int assign, int n_tokens, int dtype,
                                          void* stream) {
    if (n_tokens <= 0) return 0;
    if (dtype != DT_F32 && dtype != DT_BF16) return fail("expert_combine: unknown dtype");
    cudaStream_t s = (cudaStream_t)stream;
    const int n = dtype == DT_F32 ? 4 : 8;
    const bool vec = inner % n == 0 && total % n == 0 && ld_act % n == 0 && ld_gu % n == 0 && aligned_host(act) && aligned_host(gu);
    const int per_block = 256 * (vec ? n : 1);
    int y = (total + per_block - 1) / per_block;
    if (y > 64) y = 64;
    dim3 grid(n_tokens, y);
    const size_t shared = sizeof(float) * 2 * ((size_t)n_experts + 1);
    if (shared > 48 * 1024) return fail("expert_combine: too many experts for the table of weights");
    if (form < EXPERT_GATED_SILU || form > EXPERT_CLAMPED_GLU) return fail("expert_combine: unknown form of an expert");
#define RUN(T, VEC, FORM)                                                                                                       \
    launch_kernel(g_dependent_launch != 0, expert_combine_kernel<T, VEC, FORM>, grid, dim3(256), shared, s, (T*)act, ld_act,    \
                  (const T*)gu, ld_gu, choice, in_weight, out_weight, n_experts, inner, total, top, pairs, hidden, ld_hidden,    \
                  (const T*)x, ld_x, identity_weight, width, assign, limit, shared_limit, alpha)
#define PICK(T, VEC)                                                                                                            \
    do {                                                                                                                        \
        if (form == EXPERT_GATED_SILU) RUN(T, VEC, EXPERT_GATED_SILU);                                                          \
        else if (form == EXPERT_RELU_SQUARED) RUN(T, VEC, EXPERT_RELU_SQUARED);                                                 \
        else RUN(T, VEC, EXPERT_CLAMPED_GLU);                                                                                   \
    } while (0)
#define RUN_AS(T)                                                                                                               \
    do {                                                                                                                        \
        if (vec) PICK(T, true);                                                                                                 \
        else PICK(T, false);                                                                                                    \
    } while (0)
    if (dtype == DT_F32) RUN_AS(float);
    else RUN_AS(bf16);
#undef RUN_AS
#undef PICK
#undef RUN
    return check_launch("expert_combine_kernel");
}

extern "C" int mllm_hybrid_route(const void* x, long ld_x, const void* router, const float* router_bias, const float* correction,
                                 const void* shared_gate, int shared_plain, int rule, float scale, int width, int n_outputs,
                                 int n_identity, int groups, int keep_groups, int top, int* choice, float* in_weight,
                                 float* out_weight, float* identity_weight, int n_tokens, int dtype, void* stream) {
    if (n_tokens <= 0) return 0;
    if (top <= 0 || top > n_outputs) return fail("route: every token takes between one and all experts");
    if (shared_plain && shared_gate != nullptr) return fail("route: the shared expert has a gate or none");
    if (rule < ROUTE_SIGMOID_ON_INPUT || rule > ROUTE_SIGMOID) return fail("route: unknown rule");
    if (groups < 0 || (groups > 0 && (n_outputs % groups != 0 || keep_groups < 1 || keep_groups > groups || keep_groups * (n_outputs / groups) < top)))
        return fail("route: equal groups of experts, and enough of them kept to choose from");
    if (n_identity < 0 || n_identity > n_outputs) return fail("route: more identity experts than experts");
    if (n_identity > 0 && (identity_weight == nullptr || rule == ROUTE_SIGMOID_ON_INPUT))
        return fail("route: identity experts need weights on the outputs and room for the token's sum of them");
    cudaStream_t s = (cudaStream_t)stream;
    const int pairs = top + (shared_gate != nullptr || shared_plain ? 1 : 0);
    const size_t one = sizeof(float) * ((size_t)width + 2 * (size_t)n_outputs + 1 + (size_t)groups);
    if (one > 48 * 1024) return fail("route: the token and the scores do not fit shared memory");
    const bool four = n_tokens >= 512 && 4 * one <= 48 * 1024;
    // a warp for every output in steps of few tokens, four to sixteen of them
    const int warps = four ? 8 : (n_tokens >= 512 || n_outputs <= 4 ? 4 : (n_outputs < 16 ? n_outputs : 16));
#define RUN(T, TOKENS)                                                                                                          \
    launch_kernel(g_dependent_launch != 0, route_kernel<T, TOKENS>, dim3((n_tokens + TOKENS - 1) / TOKENS), dim3(32 * warps),   \
                  TOKENS * one, s, (const T*)x, ld_x, (const T*)router, router_bias, correction, (const T*)shared_gate,         \
                  shared_plain, rule, scale, width, n_outputs, n_identity, groups, keep_groups, top, pairs, n_tokens, choice,  \
                  in_weight, out_weight, identity_weight)
    if (dtype == DT_F32) { if (four) RUN(float, 4); else RUN(float, 1); }
    else if (dtype == DT_BF16) { if (four) RUN(bf16, 4); else RUN(bf16, 1); }
    else return fail("route: unknown dtype");
#undef RUN
    return check_launch("route_kernel");
}

// (form: an ExpertForm, with its constants; EXPERT_RELU_SQUARED has no gate matrices; expert `n_experts` is the shared one;
// identity_weight: see expert_down)
extern "C" int mllm_hybrid_experts(float* hidden, long ld_hidden, void* act, long ld_act, const void* x, long ld_x,
                                   const int* choice, const float* in_weight, const float* out_weight,
                                   const long long* gate_of, const long long* up_of, const long long* down_of,
                                   const int* inner_of, long ld_down, int max_inner, int width, int pairs,
                                   const float* identity_weight, int form, float limit, float shared_limit, float alpha,
                                   int n_experts, int n_tokens, int assign, int n_tables, int dtype, void* stream) {
    if (n_tokens <= 0) return 0;
    if (form < EXPERT_GATED_SILU || form > EXPERT_CLAMPED_GLU || (form != EXPERT_RELU_SQUARED && gate_of == nullptr))
        return fail("experts: unknown form of an expert, or one without its gate matrices");
    cudaStream_t s = (cudaStream_t)stream;
    const size_t shared = sizeof(float) * (size_t)width;
    if (shared > 48 * 1024) return fail("experts: the token does not fit shared memory");
    if (n_tables > 0) {
        // the caller's word that every inner size is a multiple of 8; what else the tiles need is looked at here
        auto on_16 = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; };
        if (dtype != DT_BF16 || n_tokens > EXPERT_TILE_TOKENS || n_tables > EXPERT_TABLES || width % 8 != 0 || ld_x % 8 != 0 ||
            ld_act % 8 != 0 || ld_down % 8 != 0 || !on_16(x) || !on_16(act))
            return fail("experts: the tiles take up to 31 bfloat16 tokens, 64 experts, rows on 16-byte boundaries");
        const size_t n_pairs = (size_t)n_tokens * pairs;
        if (n_pairs > 16384) return fail("experts: too many pairs for the tiles");
        const bf16* xb = (const bf16*)x;
        bf16* ab = (bf16*)act;
        // the first kernel's shared memory: the tokens, the pairs' choices and weights, and as much again or more for the ring of weights
        const size_t room = EXPERT_UP_SHARED - EXPERT_UP_STATIC;
        const size_t beside = n_pairs * 8 + (size_t)n_tokens * (width * 2 + (width % 64 == 0 ? 64 : 16));
        // (widths of two rounds of the second kernel's blocks, and tokens of more than some 150 pairs)
        if ((width + 7) / 8 > sm_count() || beside > room / 2) {
            const dim3 tiles((max_inner + 15) / 16, n_tables);
#define UP_BLOCKS(FORM)                                                                                                          \
    launch_kernel(g_dependent_launch != 0, expert_up_blocks_kernel<FORM>, tiles, dim3(256), 0, s, ab, ld_act, xb, ld_x, choice, in_weight, \
                  gate_of, up_of, inner_of, width, pairs, n_tokens, limit, shared_limit, alpha, n_experts)
            if (form == EXPERT_GATED_SILU) UP_BLOCKS(EXPERT_GATED_SILU);
            else if (form == EXPERT_RELU_SQUARED) UP_BLOCKS(EXPERT_RELU_SQUARED);
            else UP_BLOCKS(EXPERT_CLAMPED_GLU);
#undef UP_BLOCKS
            // (at every launch, as the limit is a device's own)
            if (cudaFuncSetAttribute(expert_down_blocks_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 128 * 1024) != cudaSuccess)
                return fail("experts: cannot raise the shared memory limit");
            launch_kernel(AFTER_THE_KERNELS_AHEAD, expert_down_blocks_kernel, dim3((width + 7) / 8), dim3(512),
                          sizeof(float) * EXPERT_UNITS * 32 * 8 + sizeof(int) * n_pairs, s, hidden, ld_hidden, (const bf16*)act, ld_act, choice,
                          out_weight, down_of, inner_of, n_tables, ld_down, width, pairs, n_tokens, assign, xb, ld_x, identity_weight);
            return check_launch("expert blocks");
        }
        int depth = (int)((room - beside) / EXPERT_UP_BLOCK) / 2 * 2;
        const int blocks_of_k = (width + 31) / 32;
        if (depth > (blocks_of_k + 1) / 2 * 2) depth = (blocks_of_k + 1) / 2 * 2;
        const size_t up_bytes = (size_t)depth * EXPERT_UP_BLOCK + beside;
        const dim3 walkers(sm_count());
        // (the limits at every launch, as they are a device's own)
#define UP_TILES(FORM)                                                                                                           \
    do {                                                                                                                         \
        if (cudaFuncSetAttribute(expert_up_tiles_kernel<FORM>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)room) != cudaSuccess) \
            return fail("experts: cannot raise the shared memory limit");                                                        \
        launch_kernel(g_dependent_launch != 0, expert_up_tiles_kernel<FORM>, walkers, dim3(EXPERT_UP_WARPS * 32), up_bytes, s, ab, ld_act, xb, ld_x, \
                      choice, in_weight, gate_of, up_of, down_of, inner_of, n_tables, ld_down, width, pairs, n_tokens, limit, shared_limit, alpha, \
                      n_experts, depth);                                                                                         \
    } while (0)
        if (form == EXPERT_GATED_SILU) UP_TILES(EXPERT_GATED_SILU);
        else if (form == EXPERT_RELU_SQUARED) UP_TILES(EXPERT_RELU_SQUARED);
        else UP_TILES(EXPERT_CLAMPED_GLU);
#undef UP_TILES
        if (cudaFuncSetAttribute(expert_down_tiles_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)EXPERT_DOWN_SHARED) != cudaSuccess)
            return fail("experts: cannot raise the shared memory limit");
        // the second kernel's: the sums, the pairs' places, and as far as they fit the weights that are asked for ahead and the pairs' choices
        const size_t least = EXPERT_DOWN_SUMS + 4 * n_pairs;
        const int ahead = least + 8 * n_pairs + EXPERT_DOWN_RING <= EXPERT_DOWN_SHARED ? EXPERT_DOWN_AHEAD : 0;
        const int held_pairs = least + 8 * n_pairs <= EXPERT_DOWN_SHARED;
        const size_t down_bytes = least + (ahead > 0 ? EXPERT_DOWN_RING : 0) + (held_pairs ? 8 * n_pairs : 0);
        launch_kernel(g_dependent_launch != 0, expert_down_tiles_kernel, dim3((width + 7) / 8), dim3(512), down_bytes, s, hidden, ld_hidden,
                      (const bf16*)act, ld_act, choice, out_weight, down_of, inner_of, n_tables, ld_down, width, pairs, n_tokens, assign, xb,
                      ld_x, identity_weight, n_experts, ahead, held_pairs);
        return check_launch("expert tiles");
    }
    constexpr int F = 4, C = 2;
    dim3 up_grid(n_tokens * pairs, (max_inner + 8 * F - 1) / (8 * F)), down_grid(n_tokens, (width + 8 * C - 1) / (8 * C));
    if (up_grid.y > 65535 || down_grid.y > 65535) return fail("experts: the sizes are too large for one launch");
#define UP(T, FORM)                                                                                                             \
    launch_kernel(g_dependent_launch != 0, expert_up_kernel<T, FORM, F>, up_grid, dim3(256), shared, s, (T*)act, ld_act,        \
                  (const T*)x, ld_x, choice, in_weight, gate_of, up_of, inner_of, width, pairs, limit, shared_limit, alpha, n_experts)
#define RUN(T)                                                                                                                  \
    do {                                                                                                                        \
        if (form == EXPERT_GATED_SILU) UP(T, EXPERT_GATED_SILU);                                                                \
        else if (form == EXPERT_RELU_SQUARED) UP(T, EXPERT_RELU_SQUARED);                                                       \
        else UP(T, EXPERT_CLAMPED_GLU);                                                                                         \
        launch_kernel(g_dependent_launch != 0, expert_down_kernel<T, C>, down_grid, dim3(256), 0, s, hidden, ld_hidden,         \
                      (const T*)act, ld_act, choice, out_weight, down_of, inner_of, ld_down, width, pairs, assign, (const T*)x, \
                      ld_x, identity_weight);                                                                                   \
    } while (0)
    if (dtype == DT_F32) RUN(float);
    else if (dtype == DT_BF16) RUN(bf16);
    else return fail("experts: unknown dtype");
#undef RUN
#undef UP
    return check_launch("expert kernels");
}

// ---------------------------------------------------------------------------
// x[r, c] += a * u[r, c] + b * v[r, c]  (32-bit; v may be null; with `assign` x is set to the sum instead)
// ---------------------------------------------------------------------------
__global__ void scaled_add_kernel(float* __restrict__ x, const float* __restrict__ u, float a, const float* __restrict__ v,
                                  float b, long n, int assign) {
    dependents_may_start();
    wait_for_earlier_kernels();
    for (long i = (long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x) {
        float sum = a * u[i];
        if (v != nullptr) sum = fmaf(b, v[i], sum);
        x[i] = assign ? sum : x[i] + sum;
    }
}

extern "C" int mllm_hybrid_scaled_add(float* x, const float* u, float a, const float* v, float b, long n, int assign, void* stream) {
    if (n <= 0) return 0;
    long blocks = (n + 255) / 256;
    if (blocks > 4096) blocks = 4096;
    launch_kernel(g_dependent_launch != 0, scaled_add_kernel, dim3((unsigned)blocks), dim3(256), 0, (cudaStream_t)stream, x, u, a, v, b, n, assign);
    return check_launch("scaled_add_kernel");
}
