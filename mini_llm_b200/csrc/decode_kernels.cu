// Kernels for steps of few tokens (decoding, short prompt portions), bfloat16.
//
// With a handful of rows every matrix product is a stream of the weights
// through the SMs, bound by HBM bandwidth and by launch latency, as in the
// reference's batched matrix-vector kernel (engine/src/matvec_batch.cu:148-261:
// rows staged in shared memory, weights streamed once, bias / gelu / residual
// in the epilogue).  Here:
//
//   skinny_linear   out = epilogue(norm?(x) W^T + bias) for up to 16 rows per
//                   CTA; mma.sync tiles, fp32 accumulation; optional
//                   layer-norm prologue (the norm never round-trips through
//                   memory), optional epilogue that scatters key and value
//                   columns straight into the cache pages.
//   layernorm       one warp per row, the row read once (the norm of long steps, and of
//                   steps whose products do not take the norm on the way in).
//   split_attention one CTA per (token, head, chunk of keys); partial softmax
//                   states go to scratch memory and the CTA that finishes
//                   last for its (token, head) merges them in chunk order, so
//                   the result does not depend on which CTA came last.
#include "mma_tiles.cuh"

MLLM_DEFINE_ERROR_API(mllm_decode)

// ---------------------------------------------------------------------------
// skinny_linear
// ---------------------------------------------------------------------------
struct SkinnyParams {
    void* out;                 // bf16 [M, ldo] / fp32 [M, ldo] (EPI_ADD, or out_f32)
    const void* x;             // bf16 [M, ldx], or fp32 [*, K] with the norm prologue
    const bf16* w;             // [N, K], K contiguous
    const float* bias;         // [N] or null
    const float* gamma;        // norm prologue: gain and shift [K], else null
    const float* beta;
    const int* rows;           // norm prologue: source row of each output row, or null
    float eps;
    int M, N, K;
    long ldx, ldo;
    int epilogue;
    int out_f32;               // EPI_STORE into fp32 (logits)
    // scatter of key / value columns into pages (null k_pages: off)
    bf16* k_pages;
    bf16* v_pages;
    const int* positions;
    const int* token_item;
    const int* block_table;
    int max_blocks, page_size, q_width, kv_width;
    // a batch of products of one shape (no norm, no scatter): product b reads x + b * x_step and w + b * w_step and
    // writes out + b * out_step (elements); batch 0 or 1: one product
    int batch;
    long x_step, w_step, out_step;
};

// A tile is 8 output features by up to 16 rows of x on mma.sync m16n8k16 (the rows of x are the tile's rows: with a handful of
// tokens a tcgen05 tile of 128 rows would be padding and its way through tensor memory longer than the product).  What bounds such a
// product is latency: the weights' way from HBM, then x's from L2, the sums between warps, the store.  So
//   - `split` warps of a block share a tile's K, their sums meet in shared memory in warp order;
//   - a lane's first AHEAD pieces of weights (all of them at K = 768) are asked for before the kernels ahead of this one have
//     ended (no kernel of a step writes weights), x, bias and residual right behind that wait;
//   - both operands come straight into registers, 16 bytes a lane: the entries of a block of 32 of K are taken in the order
//     0-1, 8-9, 16-17, 24-25 | 2-3, ... by both, so that a lane's piece of 8 feeds two products.
// Replayed back to back, against a warp a feature that unpacked x from shared memory for every one: 8 x 768 x 768 3.8 -> 2.3 us,
// 8 x 768 x 3072 7.7 -> 3.0, 16 x 3072 x 768 10.8 -> 3.9, 1 x 50257 x 768 15.2 -> 14.2 (floor 11.9).  Errors against 64 bits (operands
// of one sign in brackets): 6.6e-8 (3.6e-8) -> 7.4e-8 (5.0e-8) at K = 768, 1.1e-7 (3.9e-8) -> 9.7e-8 (5.0e-8) at 6,400.
template <int ROWS, int WARPS, bool NORM>     // rows of x of a tile: 8 (half of the tensor core's) or 16
__global__ void __launch_bounds__(WARPS * 32, 16 / WARPS)
skinny_linear_kernel(const SkinnyParams p, int split) {
    extern __shared__ __align__(16) unsigned char smem_raw[];             // the sums, then, if there is a norm, normed rows [ROWS or M][K]
    constexpr int AHEAD = 8, STEP = ROWS == 8 ? 8 : 4, STRIDE = ROWS + 1;  // (partial sums: [warp][feature][row])
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, tq = lane & 3;
    const int m0 = blockIdx.y * ROWS;
    const int m_count = min(ROWS, p.M - m0);
    const int K = p.K, pieces = K / 8;
    const int features = WARPS / split * 8, n_first = blockIdx.x * features;          // of this block
    const int part = warp % split, n0 = n_first + warp / split * 8;
    const int all = (K + 31) / 32, each = (all + split - 1) / split;      // blocks of 32 of K: all, and this warp's
    const int begin = part * each, end = n0 < p.N ? min(all, begin + each) : begin;
    const uint4 none = make_uint4(0u, 0u, 0u, 0u);
    const uint4* w_row = reinterpret_cast<const uint4*>(p.w + (long)blockIdx.z * p.w_step + (long)min(n0 + g, p.N - 1) * K);
    const long out_first = (long)blockIdx.z * p.out_step;
    uint4 wv[AHEAD];
    dependents_may_start();
#pragma unroll
    for (int i = 0; i < AHEAD; i++) {
        const int c = (begin + i) * 4 + tq;
        wv[i] = begin + i < end && c < pieces ? __ldg(w_row + c) : none;
    }
    wait_for_earlier_kernels();

    const bf16* x = behind_the_wait(reinterpret_cast<const bf16*>(p.x)) + (long)blockIdx.z * p.x_step + (long)m0 * p.ldx;
    long ldx = p.ldx;
    float* partial = reinterpret_cast<float*>(smem_raw);                  // [WARPS][8][STRIDE]
    if (NORM) {
        // The rows are normed on the way in, into shared memory: as many warps share a row as there are, whose first KEPT entries a
        // thread stay in registers through both sums.  One row of 768
        // with 2,304 features took 8.7 us with a warp a row, 4.1 so.
        constexpr int KEPT = 4;
        bf16* xs = reinterpret_cast<bf16*>(smem_raw + sizeof(float) * (WARPS * 8 * STRIDE));
        const float* src = behind_the_wait(reinterpret_cast<const float*>(p.x));
        const int group = m_count <= 1 ? WARPS : (m_count <= 2 ? WARPS / 2 : (m_count <= 4 ? WARPS / 4 : WARPS / 8));      // warps of a row
        const int team = warp / group, teams = WARPS / group, threads = group * 32, mine = threadIdx.x - team * threads;
        auto row_sum = [&](float v, float* slots) {                       // (two uses in turn, each with slots of its own)
            v = warp_sum(v);
            if (lane == 0) slots[warp] = v;
            __syncthreads();
            float total = 0.0f;
            for (int w = 0; w < group; w++) total += slots[team * group + w];
            return total;
        };
        for (int first = 0; first < m_count; first += teams) {
            const int m = min(first + team, m_count - 1);                 // (a team without a row does the last one again)
            const float* row = src + (long)(p.rows ? p.rows[m0 + m] : m0 + m) * K;
            float held[KEPT], sum = 0.0f, sq = 0.0f;
#pragma unroll
            for (int i = 0; i < KEPT; i++) {
                held[i] = mine + i * threads < K ? row[mine + i * threads] : 0.0f;
                sum += held[i];
            }
#pragma unroll 4
            for (int k = mine + KEPT * threads; k < K; k += threads) sum += row[k];
            const float mean = row_sum(sum, partial) / (float)K;
#pragma unroll
            for (int i = 0; i < KEPT; i++) {
                held[i] -= mean;
                if (mine + i * threads < K) sq = fmaf(held[i], held[i], sq);
            }
#pragma unroll 4
            for (int k = mine + KEPT * threads; k < K; k += threads) {
                const float c = row[k] - mean;
                sq = fmaf(c, c, sq);
            }
            const float inv = 1.0f / sqrtf(row_sum(sq, partial + WARPS) / (float)K + p.eps);
            if (first + team >= m_count) continue;
#pragma unroll
            for (int i = 0; i < KEPT; i++) {
                const int k = mine + i * threads;
                if (k < K) xs[m * K + k] = __float2bfloat16_rn(held[i] * inv * p.gamma[k] + p.beta[k]);
            }
#pragma unroll 4
            for (int k = mine + KEPT * threads; k < K; k += threads)
                xs[m * K + k] = __float2bfloat16_rn((row[k] - mean) * inv * p.gamma[k] + p.beta[k]);
        }
        __syncthreads();
        x = xs;
        ldx = K;
    }
    // the first result this thread will write: its bias and residual are on their way during the product
    const int outputs = features * ROWS;
    auto place = [&](int i, int& n, int& m) {                             // neighbouring threads: neighbouring features
        n = n_first + i % features;
        m = i / features;
        return m < m_count && n < p.N;
    };
    auto bias = [&](int n) { return p.bias ? p.bias[n] : 0.0f; };
    auto residual = [&](int n, int m) {
        return p.epilogue == EPI_ADD ? reinterpret_cast<const float*>(p.out)[out_first + (long)(m0 + m) * p.ldo + n] : 0.0f;
    };
    int n_mine, m_mine;
    float bias_mine = 0.0f, residual_mine = 0.0f;
    if ((int)threadIdx.x < outputs && place(threadIdx.x, n_mine, m_mine)) {
        bias_mine = bias(n_mine);
        residual_mine = residual(n_mine, m_mine);
    }

    // Every product of 16 entries of K is added by a rounded addition, in turn to one of four sums: left in the tensor cores'
    // accumulators, whose sums are cut off, the error against 64 bits was up to ten times that of rounded FMAs.
    float sums_of[4][4] = {};
    const bool low_there = g < m_count, high_there = ROWS > 8 && g + 8 < m_count;
    const uint4* x_low = reinterpret_cast<const uint4*>(x + (long)g * ldx);
    const uint4* x_high = reinterpret_cast<const uint4*>(x + (long)(g + 8) * ldx);
    for (int first = begin; first < end; first += AHEAD) {
#pragma unroll
        for (int half = 0; half < AHEAD; half += STEP) {
            uint4 xl[STEP], xh[STEP];
#pragma unroll
            for (int i = 0; i < STEP; i++) {
                const int c = (first + half + i) * 4 + tq;
                const bool there = first + half + i < end && c < pieces;
                xl[i] = there && low_there ? x_low[c] : none;
                xh[i] = there && high_there ? x_high[c] : none;
            }
#pragma unroll
            for (int i = 0; i < STEP; i++) {
                // this block of weights is used up, the one AHEAD blocks on asked for into its place
                const uint4 w = wv[half + i];
                const int c = (first + AHEAD + half + i) * 4 + tq;
                wv[half + i] = first + AHEAD + half + i < end && c < pieces ? __ldg(w_row + c) : none;
                const uint32_t first_half[4] = {xl[i].x, xh[i].x, xl[i].y, xh[i].y}, second_half[4] = {xl[i].z, xh[i].z, xl[i].w, xh[i].w};
                mma_added(sums_of[2 * (i & 1)], first_half, w.x, w.y);
                mma_added(sums_of[2 * (i & 1) + 1], second_half, w.z, w.w);
            }
        }
    }
    float acc[4];
#pragma unroll
    for (int e = 0; e < 4; e++) acc[e] = (sums_of[0][e] + sums_of[1][e]) + (sums_of[2][e] + sums_of[3][e]);
    float* sums = partial + (warp * 8 + 2 * tq) * STRIDE + g;
    sums[0] = acc[0];
    sums[STRIDE] = acc[1];
    if (ROWS > 8) {
        sums[8] = acc[2];
        sums[STRIDE + 8] = acc[3];
    }
    __syncthreads();
    for (int i = threadIdx.x; i < outputs; i += WARPS * 32) {
        int n, m;
        if (!place(i, n, m)) continue;
        const int f = n - n_first;
        float v = 0.0f;
        for (int s = 0; s < split; s++) v += partial[((f / 8 * split + s) * 8 + f % 8) * STRIDE + m];
        v += i == threadIdx.x ? bias_mine : bias(n);
        if (p.epilogue == EPI_GELU_TANH) v = gelu_tanh_f(v);
        else if (p.epilogue == EPI_GELU_ERF) v = gelu_erf_f(v);
        else if (p.epilogue == EPI_RELU_SQ) v = v > 0.0f ? v * v : 0.0f;
        else if (p.epilogue == EPI_SILU) v = v / (1.0f + expf(-v));
        const int row = m0 + m;
        if (p.k_pages != nullptr && n >= p.q_width) {
            int pos = p.positions[row];
            int page = p.block_table[(long)p.token_item[row] * p.max_blocks + pos / p.page_size];
            long slot = ((long)page * p.page_size + pos % p.page_size) * p.kv_width;
            if (n < p.q_width + p.kv_width) p.k_pages[slot + (n - p.q_width)] = __float2bfloat16_rn(v);
            else p.v_pages[slot + (n - p.q_width - p.kv_width)] = __float2bfloat16_rn(v);
        } else if (p.epilogue == EPI_ADD) {
            reinterpret_cast<float*>(p.out)[out_first + (long)row * p.ldo + n] = (i == threadIdx.x ? residual_mine : residual(n, m)) + v;
        } else if (p.out_f32) {
            reinterpret_cast<float*>(p.out)[out_first + (long)row * p.ldo + n] = v;
        } else {
            reinterpret_cast<bf16*>(p.out)[out_first + (long)row * p.ldo + n] = __float2bfloat16_rn(v);
        }
    }
}

static int g_smem_optin = -1;

template <int ROWS, int WARPS, bool NORM>
static int launch_skinny(const SkinnyParams& p, int split, cudaStream_t s) {
    const size_t sums = sizeof(float) * WARPS * 8 * (ROWS + 1);
    // (normed rows: those there are, so that one row may be as long as the sizes that are taken say)
    const size_t smem = sums + (NORM ? (size_t)(p.M < ROWS ? p.M : ROWS) * p.K * sizeof(bf16) : 0);
    if (g_smem_optin < 0) {
        int dev = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&g_smem_optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    }
    if (smem > (size_t)g_smem_optin) return fail("skinny_linear: the rows do not fit shared memory");
    static bool configured = false;               // per instantiation
    if (smem > 48 * 1024 && !configured) {
        cudaError_t e = cudaFuncSetAttribute(skinny_linear_kernel<ROWS, WARPS, NORM>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             g_smem_optin);
        if (e != cudaSuccess) return fail("skinny_linear: cannot raise the shared memory limit");
        configured = true;
    }
    const int features = WARPS / split * 8;
    dim3 grid((p.N + features - 1) / features, (p.M + ROWS - 1) / ROWS, p.batch);
    return launched(launch_kernel(g_dependent_launch != 0, skinny_linear_kernel<ROWS, WARPS, NORM>, grid, dim3(WARPS * 32), smem, s, p, split),
                    "skinny_linear_kernel");
}

// Warps that share a tile's K: all eight of a block while the tiles' blocks run side by side (two an SM), fewer where the
// features alone bring enough warps (a vocabulary: one warp a tile; with eight it took 25.3 us in place of 14.3, as every block's
// sums meet); sixteen for a long K of few features, so that each warp's share is asked for ahead as a whole.
template <int ROWS, bool NORM>
static int launch_skinny_rows(const SkinnyParams& p, cudaStream_t s) {
    const long tiles = (long)((p.N + 7) / 8) * p.batch;
    if (p.K > 2048 && tiles <= 148) return launch_skinny<ROWS, 16, NORM>(p, 16, s);
    return launch_skinny<ROWS, 8, NORM>(p, tiles <= 296 ? 8 : tiles <= 592 ? 4 : tiles <= 1184 ? 2 : 1, s);
}

extern "C" int mllm_decode_skinny_linear(const SkinnyParams* params, void* stream) {
    SkinnyParams p = *params;
    if (p.batch == 0) p.batch = 1;
    if (p.M <= 0 || p.N <= 0) return 0;
    if (p.K <= 0 || p.K % 8 != 0) return fail("skinny_linear: K must be a positive multiple of 8");
    if (p.gamma == nullptr && p.ldx % 8 != 0) return fail("skinny_linear: the row stride of x must be a multiple of 8");
    if (p.epilogue == EPI_ADD && p.k_pages != nullptr) return fail("skinny_linear: no scatter with the residual sum");
    if (p.batch < 0 || p.batch > 65535) return fail("skinny_linear: a batch has up to 65535 products");
    if (p.batch > 1 && (p.gamma != nullptr || p.k_pages != nullptr || p.x_step % 8 != 0 || p.w_step % 8 != 0))
        return fail("skinny_linear: a batch takes no norm and no scatter, and its products start on 16-byte boundaries");
    cudaStream_t s = (cudaStream_t)stream;
    if (p.gamma != nullptr) return p.M <= 8 ? launch_skinny_rows<8, true>(p, s) : launch_skinny_rows<16, true>(p, s);
    return p.M <= 8 ? launch_skinny_rows<8, false>(p, s) : launch_skinny_rows<16, false>(p, s);
}

__device__ __forceinline__ void cp_async_16(void* smem, const void* global) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(smem)), "l"(global)
                 : "memory");
}

// ---------------------------------------------------------------------------
// split_attention
// ---------------------------------------------------------------------------
// Scratch layout (fp32): for every (token, head, chunk):
//   acc  [tokens, heads, max_chunks, head_size]   un-normalised weighted values
//   ml   [tokens, heads, max_chunks, 2]           running maximum, running sum
// and one int32 counter per (token, head), zero between launches.
// The keys a token sees are numbered without gaps: the kept first ones (those below `keep` that the window has
// passed), then the window's; chunks are ranges of these numbers, so a chunk is full whatever lies between.
// FULL: keys and values have D entries; else key rows have `dim` and value rows `vdim` entries (multiples of 8 up
// to D; scratch keeps its stride D), and a lane past a row's end copies nothing and holds zeros.
// A tile of 16 keys goes through m16n8k16 products: keys times the query (which stands in all eight columns), then values, turned, times the
// weights, which enter as three bfloat16 terms in three columns and so keep all 24 bits; a tile's product is added with a rounded FMA.
// What bounds it: few keys a pair, the chain of position, block table, keys and merge; many, the copies' way from HBM.  One lane a key's
// 16 bytes with FMAs took 50 instructions a key and pair and was bound by their issue (60 % of all cycles); now some 13.  Heads of 64, before
// and now: 64 x 12 pairs of 110 keys 11.2 -> 8.0 us, 24 x 16 of 112 to 778 22.3 -> 15.5, 64 x 25 of 264 31.1 -> 24.4, 2 x 12 of 1,000 13.6 -> 7.9.
template <int D, bool FULL, int WARPS, int STAGES>       // head size: 16, 32, 64, 128 or 256
__global__ void __launch_bounds__(WARPS * 32)
split_attention_kernel(bf16* __restrict__ out, long ld_out, const bf16* q, long ld_q,
                       const bf16* __restrict__ k_pages, const bf16* __restrict__ v_pages,
                       const int* __restrict__ block_table, int max_blocks, const int* __restrict__ positions,
                       const int* __restrict__ token_item, int n_heads, int n_kv_heads, int dim, int vdim, int page_size,
                       float scale, float cap, int window, int block, int keep, const float* gate, long ld_gate,
                       int gate_wide, const float* __restrict__ sink, const float* __restrict__ slopes, int chunk, int max_chunks, float* __restrict__ part_acc,
                       float* __restrict__ part_ml, int* __restrict__ counters, const int* records, const int* first_new) {
    if (FULL) dim = vdim = D;
    constexpr int LD = D + 8, STEPS = D / 16;              // rows of a tile an odd number of 16 bytes apart: no bank twice
    dependents_may_start();
    if (first_new == nullptr) wait_for_earlier_kernels();
    const int h = blockIdx.y, c = blockIdx.z;
    const long pair = (long)blockIdx.x * n_heads + h;          // whose scratch this is
    // (a record of the step's work list: entry, row, rows, position)
    const int* record = records + (long)blockIdx.x * 8;
    const int t = records != nullptr ? record[1] : blockIdx.x;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int g = lane >> 2, tq = lane & 3;
    const int p = records != nullptr ? record[3] : positions[t], item = records != nullptr ? record[0] : token_item[t];
    // the first key seen: the window's, and with a mask of blocks of positions the first of the query's block
    int lo = (window > 0 && p - window + 1 > 0) ? p - window + 1 : 0;
    if (block > 0) lo = max(lo, p - p % block);
    const int n_kept = min(keep, lo), gap = lo - n_kept;        // key number i is position i (i < n_kept) or i + gap
    const int n_seen = n_kept + p - lo + 1;
    // the chunk that is asked for, or what makes the launch's chunks cover this token's keys (a multiple of 32 then)
    if ((long)chunk * max_chunks < n_seen) chunk = ((n_seen + max_chunks - 1) / max_chunks + 31) / 32 * 32;
    const int c_last = (n_seen - 1) / chunk;
    if (c > c_last) return;
    const int begin = c * chunk, end = min(n_seen, begin + chunk) - 1;             // key numbers, inclusive
    const int* bt = block_table + (long)item * max_blocks;
    const int hk = h / (n_heads / n_kv_heads);
    const long k_width = (long)n_kv_heads * dim, v_width = (long)n_kv_heads * vdim;

    // Keys from this position on are written by kernels of the step that may still run (`first_new`, one position an entry; without it
    // nothing is read ahead of the wait): the first tiles of the others are asked for ahead of the wait.
    const int limit = first_new != nullptr ? first_new[item] : p + 1;
    // scores are kept in units of log2(e): exp(x) = 2^(x log2 e) costs one instruction then
    const float scale_log2 = scale * 1.4426950408889634f;
    // a cap on the scores, cap * tanh(score / cap), in the same units (cap <= 0: none)
    const float cap_log2 = cap * 1.4426950408889634f, inv_cap_log2 = cap > 0.0f ? 1.0f / cap_log2 : 0.0f;
    // a bias by distance, taken off the (capped) score, in the same units
    const float slope_log2 = slopes != nullptr ? slopes[h] * 1.4426950408889634f : 0.0f;
    float m = -INFINITY, l = 0.0f, acc[STEPS][4];        // m in log2 units; l: of this lane's keys
#pragma unroll
    for (int j = 0; j < STEPS; j++) acc[j][0] = acc[j][1] = acc[j][2] = acc[j][3] = 0.0f;
    // A warp's tiles are 16 keys each, every WARPS-th of the chunk; STAGES - 1 are on their way while one is worked on, and
    // where the next one's keys lie is asked for a tile before its copies (lane l mod 16 has key l).
    extern __shared__ uint4 split_shared[];
    bf16* ring = reinterpret_cast<bf16*>(split_shared) + warp * (STAGES * 2 * 16 * LD);
    const int first_key = begin + warp * 16, tiles = (end - first_key) / (WARPS * 16) + (end >= first_key);
    // pages of a power of two are the rule: shift and mask instead of a division per key
    const int page_shift = (page_size & (page_size - 1)) == 0 ? 31 - __clz(page_size) : -1;
    const bf16* k_head = k_pages + (long)hk * dim;
    const bf16* v_head = v_pages + (long)hk * vdim;
    long row = -1;                                        // (-1: no such key, -2: left for a second look)
    auto find = [&](int i, int from, int to) {            // positions [from, to)
        const int number = first_key + i * (WARPS * 16) + (lane & 15);
        const int j = number < n_kept ? number : number + gap;
        const int block = page_shift >= 0 ? j >> page_shift : j / page_size;
        const int within = page_shift >= 0 ? j & (page_size - 1) : j % page_size;
        row = number > end ? (from == 0 ? -1 : -2) : j < from || j >= to ? -2 : ((long)bt[block] * page_size + within) * (FULL ? k_width : 1);
    };
    auto copy_rows = [&](int i) {
        bf16* kt = ring + (i % STAGES) * (2 * 16 * LD);
#pragma unroll
        for (int u = 0; u < STEPS; u++) {
            const int key = (lane + 32 * u) / (D / 8), d = (lane + 32 * u) % (D / 8) * 8;
            const long at = __shfl_sync(0xffffffffu, row, key);
            const bool k_there = at >= 0 && (FULL || d < dim), v_there = at >= 0 && (FULL || d < vdim);
            if (at != -2) {
                copy_16(kt + key * LD + d, k_there ? k_head + (FULL ? at : at * k_width) + d : k_head, k_there);
                copy_16(kt + (16 + key) * LD + d, v_there ? v_head + (FULL ? at : at * v_width) + d : v_head, v_there);
            }
        }
    };
    auto issue = [&](int i, int to) {
        if (i < tiles) {
            copy_rows(i);
            find(i + 1, 0, to);
        }
        copies_end();
    };
    const int ahead = first_new != nullptr ? limit : p + 1;
    if (tiles > 0) find(0, 0, ahead);
#pragma unroll
    for (int i = 0; i < STAGES - 1; i++) issue(i, ahead);
    if (first_new != nullptr) {
        wait_for_earlier_kernels();
        // the step's own keys among those tiles' (a key below the window that stays visible may be one)
        bool left = false;
#pragma unroll
        for (int i = 0; i < STAGES - 1; i++)
            if (i < tiles) {
                find(i, limit, p + 1);
                if (__any_sync(0xffffffffu, row >= 0)) {
                    copy_rows(i);
                    left = true;
                }
            }
        if (left) {
            copies_end();
            copies_landed<0>();
        }
        if (STAGES - 1 < tiles) find(STAGES - 1, 0, p + 1);
    }
    // The query stands in all eight columns of the second operand, so that every lane has the scores of its two keys.
    q = behind_the_wait(q);
    uint32_t qb[STEPS][2];
#pragma unroll
    for (int k = 0; k < STEPS; k++)
#pragma unroll
        for (int u = 0; u < 2; u++) {
            const int d = k * 16 + u * 8 + 2 * tq;
            qb[k][u] = FULL || d < dim ? *reinterpret_cast<const uint32_t*>(q + (long)t * ld_q + (long)h * dim + d) : 0u;
        }
    gate = behind_the_wait(gate);
    for (int i = 0; i < tiles; i++) {
        issue(i + STAGES - 1, p + 1);
        copies_landed<STAGES - 1>();
        __syncwarp();
        const bf16* kt = ring + (i % STAGES) * (2 * 16 * LD);
        const bf16* vt = kt + 16 * LD;
        float c[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
        for (int k = 0; k < STEPS; k++) {
            uint32_t a[4];
            load_blocks(a, kt + (lane & 15) * LD + k * 16 + (lane >> 4) * 8);
            mma_added(c, a, qb[k][0], qb[k][1]);
        }
        float x[2];                                       // keys g and g + 8
#pragma unroll
        for (int u = 0; u < 2; u++) {
            const int number = first_key + i * (WARPS * 16) + g + 8 * u;
            x[u] = c[2 * u] * scale_log2;
            if (cap > 0.0f) x[u] = cap_log2 * tanhf(x[u] * inv_cap_log2);
            if (slopes != nullptr) x[u] = fmaf(-slope_log2, (float)(p - (number < n_kept ? number : number + gap)), x[u]);
            if (number > end) x[u] = -INFINITY;
        }
        float m_new = fmaxf(x[0], x[1]);
#pragma unroll
        for (int o = 4; o < 32; o <<= 1) m_new = fmaxf(m_new, __shfl_xor_sync(0xffffffffu, m_new, o));
        m_new = fmaxf(m_new, m);
        const float from = m_new == -INFINITY ? 0.0f : m_new;
        const float corr = exp2f(m - from);
        x[0] = exp2f(x[0] - from), x[1] = exp2f(x[1] - from);
        l = fmaf(l, corr, x[0] + x[1]);
        m = m_new;
        // the weights, 16 keys in the rows, their three bfloat16 terms (all 24 bits) in the first three columns
        uint32_t low[3], high[3];
        three_weight_terms(__shfl_sync(0xffffffffu, x[0], 8 * tq), __shfl_sync(0xffffffffu, x[0], 8 * tq + 4), low[0], low[1], low[2]);
        three_weight_terms(__shfl_sync(0xffffffffu, x[1], 8 * tq), __shfl_sync(0xffffffffu, x[1], 8 * tq + 4), high[0], high[1], high[2]);
        const uint32_t b0 = g == 0 ? low[0] : (g == 1 ? low[1] : (g == 2 ? low[2] : 0u));
        const uint32_t b1 = g == 0 ? high[0] : (g == 1 ? high[1] : (g == 2 ? high[2] : 0u));
#pragma unroll
        for (int j = 0; j < STEPS; j++) {
            uint32_t a[4];
            float y[4] = {0.0f, 0.0f, 0.0f, 0.0f};
            load_blocks_turned(a, vt + ((lane & 7) + ((lane >> 4) & 1) * 8) * LD + j * 16 + ((lane >> 3) & 1) * 8);
            mma_tile(y, a, b0, b1);
#pragma unroll
            for (int e = 0; e < 4; e++) acc[j][e] = fmaf(acc[j][e], corr, y[e]);       // (rounded: what a tile adds is cut off)
        }
        __syncwarp();                                     // the tile is copied over in the next round
    }
    copies_landed<0>();

    // a lane's keys into the warp's sum, the terms' columns (of lanes tq 0 and 1) into one, then the warps through shared
    // memory, always in the same order
#pragma unroll
    for (int o = 4; o < 32; o <<= 1) l += __shfl_xor_sync(0xffffffffu, l, o);
    __syncthreads();                                  // the tiles are used up: what follows lies in their memory
    float (*sm_acc)[D] = reinterpret_cast<float (*)[D]>(split_shared);
    float* sm_m = &sm_acc[WARPS][0];
    float* sm_l = sm_m + WARPS;
    float* sm_top = sm_l + WARPS;
    float* sm_sum = sm_top + WARPS;
    float* weight = sm_sum + WARPS;                   // [threads]
    float* spread = weight + WARPS * 32;              // [threads]
    if (lane == 0) sm_m[warp] = m, sm_l[warp] = l;
#pragma unroll
    for (int j = 0; j < STEPS; j++)
#pragma unroll
        for (int u = 0; u < 2; u++) {
            float value = tq == 0 ? acc[j][2 * u] + acc[j][2 * u + 1] : acc[j][2 * u];
            value += __shfl_xor_sync(0xffffffffu, value, 1);
            if (tq == 0) sm_acc[warp][j * 16 + u * 8 + g] = value;
        }
    __syncthreads();
    float top = -INFINITY, total = 0.0f, share[WARPS];
#pragma unroll
    for (int w = 0; w < WARPS; w++) top = fmaxf(top, sm_m[w]);
    const float from = top == -INFINITY ? 0.0f : top;
#pragma unroll
    for (int w = 0; w < WARPS; w++) share[w] = exp2f(sm_m[w] - from), total = fmaf(sm_l[w], share[w], total);
    auto sum_of = [&](int d) {
        float o = 0.0f;
#pragma unroll
        for (int w = 0; w < WARPS; w++) o = fmaf(sm_acc[w][d], share[w], o);
        return o;
    };
    // a sink: one more term exp(sink[h]) in the denominator, with no key and no value (scores are in units of log2 e)
    const float sink_log2 = sink != nullptr ? sink[h] * 1.4426950408889634f : -INFINITY;
    // a gate per (token, head), or per entry of the head's result, opens it by its sigmoid
    auto open = [&](int d) {
        return gate != nullptr ? 1.0f / (1.0f + __expf(-gate[(long)t * ld_gate + (gate_wide ? h * vdim + d : h)])) : 1.0f;
    };
    if (c_last == 0) {                               // one chunk: nothing to merge with
        const float above = fmaxf(top, sink_log2);
        const float shrink = exp2f(top - above), denom = total * shrink + (sink != nullptr ? exp2f(sink_log2 - above) : 0.0f);
        for (int d = threadIdx.x; d < vdim; d += WARPS * 32)
            out[(long)t * ld_out + (long)h * vdim + d] = __float2bfloat16_rn(sum_of(d) * shrink / denom * open(d));
        return;
    }
    const long cell = pair * max_chunks + c;
    for (int d = threadIdx.x; d < vdim; d += WARPS * 32) part_acc[cell * D + d] = sum_of(d);
    if (threadIdx.x == 0) part_ml[cell * 2] = top, part_ml[cell * 2 + 1] = total;

    // the CTA that arrives last for this (token, head) merges the chunks: as many threads share an entry of the result as
    // there are, each with every so many chunks, and what a thread reads is asked for eight chunks at a time
    __shared__ int is_last;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) {
        int ticket = atomicAdd(&counters[pair], 1);
        is_last = (ticket == c_last);
        if (is_last) counters[pair] = 0;       // ready for the next launch
    }
    __syncthreads();
    if (!is_last) return;
    __threadfence();
    constexpr int THREADS = WARPS * 32, SPREAD = D >= THREADS ? 1 : THREADS / D, ENTRIES = D > THREADS ? D / THREADS : 1, BATCH = THREADS;
    const long first = pair * max_chunks;
    const int d0 = threadIdx.x % (D < THREADS ? D : THREADS), turn = threadIdx.x / (D < THREADS ? D : THREADS);
    float o[ENTRIES], denom = 0.0f;
#pragma unroll
    for (int e = 0; e < ENTRIES; e++) o[e] = 0.0f;
    top = sink_log2;
    if (sink != nullptr) denom = 1.0f;
    for (int base = 0; base <= c_last; base += BATCH) {
        const int mine = base + threadIdx.x, here = min(BATCH, c_last + 1 - base);
        const float m_part = mine <= c_last ? __ldcg(part_ml + (first + mine) * 2) : -INFINITY;
        const float l_part = mine <= c_last ? __ldcg(part_ml + (first + mine) * 2 + 1) : 0.0f;
        float big = warp_max(m_part);
        if (lane == 0) sm_top[warp] = big;
        __syncthreads();
        big = top;
#pragma unroll
        for (int w = 0; w < WARPS; w++) big = fmaxf(big, sm_top[w]);
        const float over = big == -INFINITY ? 0.0f : big;
        const float w = exp2f(m_part - over), sum = warp_sum(l_part * w), shrink = exp2f(top - over);
        weight[threadIdx.x] = w;
        if (lane == 0) sm_sum[warp] = sum;
        __syncthreads();
        denom *= shrink;
#pragma unroll
        for (int w = 0; w < WARPS; w++) denom += sm_sum[w];
        top = big;
#pragma unroll
        for (int e = 0; e < ENTRIES; e++) {
            o[e] *= shrink;
#pragma unroll 8
            for (int cc = turn; cc < here; cc += SPREAD) o[e] = fmaf(__ldcg(part_acc + (first + base + cc) * D + d0 + e * THREADS), weight[cc], o[e]);
        }
        __syncthreads();
    }
    if (SPREAD > 1) {
        spread[threadIdx.x] = o[0];
        __syncthreads();
        if (turn > 0) return;
        float x = 0.0f;
#pragma unroll
        for (int r = 0; r < SPREAD; r++) x += spread[r * D + d0];
        o[0] = x;
    }
#pragma unroll
    for (int e = 0; e < ENTRIES; e++) {
        const int d = d0 + e * THREADS;
        if (d < vdim) out[(long)t * ld_out + (long)h * vdim + d] = __float2bfloat16_rn(o[e] / denom * open(d));
    }
}

// (with a cap on the scores: score <- cap * tanh(score / cap); cap <= 0: none; with a mask of blocks of
// positions: block > 0, a query sees only keys of its own block, counted from position 0; with a gate:
// fp32 [tokens, >= heads], head h's result times sigmoid(gate[t, h]), or with gate_wide [tokens, >= heads * vdim], entry d
// of it times sigmoid(gate[t, h * vdim + d]); with slopes: fp32 [heads], slopes[h] * (distance) comes off the score; with a sink: fp32 [heads], exp(sink[h]) joins
// head h's softmax denominator)
// The widest form: key rows of `dim` and value rows of `vdim` entries (equal and one of 16, 32, 64, 128, 256, or
// any multiples of 8 up to 256; the scratch's rows then have the least of those sizes that holds both), and the keys
// below `keep` stay visible behind a window.  max_chunks * chunk covers the most keys a token of the step sees.
// (with `records`, 8 numbers each: the single tokens that n_tokens records of a step's work list name,
// entry, row, rows, position first; scratch is theirs in the list's order)
// (with `first_new`, a position an entry: kernels that may still run write no key or value before it, so those are read ahead of the wait
// for them.  Positions, block table and records are read there too: they come with the step's arrays)
extern "C" int mllm_decode_split_attention_records(void* out, long ld_out, const void* q, long ld_q, const void* k_pages,
                                                const void* v_pages, const int* block_table, int max_blocks,
                                                const int* positions, const int* token_item, int n_tokens, int n_heads,
                                                int n_kv_heads, int dim, int vdim, int page_size, float scale, float cap,
                                                int window, int block, int keep, const float* gate, long ld_gate,
                                                int gate_wide, const float* sink, const float* slopes, int chunk, int max_chunks, float* part_acc,
                                                float* part_ml, int* counters, const int* records, const int* first_new, void* stream) {
    if (n_tokens <= 0) return 0;
    if (n_kv_heads <= 0 || n_heads % n_kv_heads != 0)
        return fail("split_attention: heads must be a multiple of key/value heads");
    if (chunk <= 0 || max_chunks <= 0 || max_chunks > 65535 || n_heads > 65535)
        return fail("split_attention: bad chunking");
    if (ld_q % 8 != 0) return fail("split_attention: the row stride of q must be a multiple of 8");
    if (keep < 0 || (keep > 0 && block > 0)) return fail("split_attention: kept first keys go with a window, not with blocks of positions");
    if (dim <= 0 || vdim <= 0 || dim % 8 != 0 || vdim % 8 != 0 || dim > 256 || vdim > 256)
        return fail("split_attention: key and value sizes are multiples of 8 up to 256");
    const int most = dim > vdim ? dim : vdim;
    const int size = most <= 16 ? 16 : (most <= 32 ? 32 : (most <= 64 ? 64 : (most <= 128 ? 128 : 256)));
    const bool full = dim == size && vdim == size;
    cudaStream_t s = (cudaStream_t)stream;
    // Chunks a (token, head) pair is launched with.  max_chunks follows the block table's reach, which without a limit on
    // positions is the whole cache: 65,536 keys are 256 to 1,024 chunks a pair, nearly all of which have no keys and only come
    // and go (16 tokens x 12 heads at 120 keys: 51 us for 49,152 blocks, 7.6 us for 1,536).  A wave of 1,184 blocks (8 an SM) is shared among
    // the pairs, at least 4 each; a token that sees more keys than so many chunks hold takes longer chunks (in the kernel).
    const long pairs = (long)n_tokens * n_heads;
    const long share = (1184 + pairs - 1) / pairs;
    if (max_chunks > share && max_chunks > 4) max_chunks = (int)(share > 4 ? share : 4);
    dim3 grid(n_tokens, n_heads, max_chunks);
    // Heads of up to 64: eight warps a block where three such blocks an SM hold the launch, so that a long request's keys are half as many
    // tiles one after the other; else four warps, with three stages of the ring where a wave of blocks holds the launch all the same, else
    // two, of which six blocks of heads of 64 fit an SM.  At heads of 64, four warps of three stages against eight: 24 x 16 pairs of 114 to 780
    // keys 17.4 and 14.0 us, 20 x 12 of 500 11.8 and 9.3, 32 x 12 of 30 to 960 19.6 and 15.1, 3 x 12 of 800 in chunks of 128 6.6 and 6.1; three
    // stages against two: 24 x 16 pairs of 112 to 778 15.1 and 16.2 us, 64 x 12 of 1,000 38.9 and 50.4; 64 x 12 of 110 (five blocks an SM are
    // needed for one wave) 10.9 and 8.0.
    const long blocks = pairs * max_chunks;
    const bool wide = blocks <= 444 && size <= 64, deep = blocks <= 592 && size <= 64;
#define LAUNCH_SPLIT(D, FULL, WARPS, STAGES)                                                                             \
    do {                                                                                                                 \
        constexpr int ring = WARPS * STAGES * 2 * 16 * (D + 8) * 2;                                                      \
        if (ring > 48 * 1024 && cudaFuncSetAttribute(split_attention_kernel<D, FULL, WARPS, STAGES>,                     \
                                                     cudaFuncAttributeMaxDynamicSharedMemorySize, ring) != cudaSuccess)  \
            return fail("split_attention: the ring's shared memory was refused");                                        \
        launch_kernel(g_dependent_launch != 0, split_attention_kernel<D, FULL, WARPS, STAGES>, grid, dim3(WARPS * 32), ring, s, (bf16*)out, ld_out, \
                      (const bf16*)q, ld_q, (const bf16*)k_pages, (const bf16*)v_pages, block_table, max_blocks,         \
                      positions, token_item, n_heads, n_kv_heads, dim, vdim, page_size, scale, cap, window, block, keep, \
                      gate, ld_gate, gate_wide, sink, slopes, chunk, max_chunks, part_acc, part_ml, counters, records, first_new); \
    } while (0)
#define PICK_SPLIT_SMALL(D)                                                       \
    do {                                                                          \
        if (full && wide) LAUNCH_SPLIT(D, true, 8, 2);                            \
        else if (wide) LAUNCH_SPLIT(D, false, 8, 2);                              \
        else if (full && deep) LAUNCH_SPLIT(D, true, 4, 3);                       \
        else if (full) LAUNCH_SPLIT(D, true, 4, 2);                               \
        else if (deep) LAUNCH_SPLIT(D, false, 4, 3);                              \
        else LAUNCH_SPLIT(D, false, 4, 2);                                        \
    } while (0)
#define PICK_SPLIT(D)                                                             \
    do {                                                                          \
        if (full) LAUNCH_SPLIT(D, true, 4, 2);                                    \
        else LAUNCH_SPLIT(D, false, 4, 2);                                        \
    } while (0)
    switch (size) {
    case 16: PICK_SPLIT_SMALL(16); break;
    case 32: PICK_SPLIT_SMALL(32); break;
    case 64: PICK_SPLIT_SMALL(64); break;
    case 128: PICK_SPLIT(128); break;
    default: PICK_SPLIT(256); break;
    }
#undef PICK_SPLIT
#undef PICK_SPLIT_SMALL
#undef LAUNCH_SPLIT
    return check_launch("split_attention_kernel");
}

extern "C" int mllm_decode_split_attention_kept(void* out, long ld_out, const void* q, long ld_q, const void* k_pages,
                                                const void* v_pages, const int* block_table, int max_blocks,
                                                const int* positions, const int* token_item, int n_tokens, int n_heads,
                                                int n_kv_heads, int dim, int vdim, int page_size, float scale, float cap,
                                                int window, int block, int keep, const float* gate, long ld_gate,
                                                int gate_wide, const float* sink, const float* slopes, int chunk, int max_chunks, float* part_acc,
                                                float* part_ml, int* counters, void* stream) {
    return mllm_decode_split_attention_records(out, ld_out, q, ld_q, k_pages, v_pages, block_table, max_blocks, positions, token_item,
                                               n_tokens, n_heads, n_kv_heads, dim, vdim, page_size, scale, cap, window, block, keep,
                                               gate, ld_gate, gate_wide, sink, slopes, chunk, max_chunks, part_acc, part_ml, counters,
                                               nullptr, nullptr, stream);
}

extern "C" int mllm_decode_split_attention_sink(void* out, long ld_out, const void* q, long ld_q, const void* k_pages,
                                                const void* v_pages, const int* block_table, int max_blocks,
                                                const int* positions, const int* token_item, int n_tokens, int n_heads,
                                                int n_kv_heads, int head_size, int page_size, float scale, float cap,
                                                int window, int block, const float* gate, long ld_gate, const float* sink,
                                                int chunk, int max_chunks, float* part_acc, float* part_ml, int* counters,
                                                void* stream) {
    switch (head_size) {
    case 16: case 32: case 64: case 128: case 256: break;
    default: return fail("split_attention: head size must be 16, 32, 64, 128 or 256");
    }
    return mllm_decode_split_attention_kept(out, ld_out, q, ld_q, k_pages, v_pages, block_table, max_blocks, positions,
                                            token_item, n_tokens, n_heads, n_kv_heads, head_size, head_size, page_size, scale,
                                            cap, window, block, 0, gate, ld_gate, 0, sink, nullptr, chunk, max_chunks, part_acc,
                                            part_ml, counters, stream);
}

extern "C" int mllm_decode_split_attention_masked(void* out, long ld_out, const void* q, long ld_q, const void* k_pages,
                                                  const void* v_pages, const int* block_table, int max_blocks,
                                                  const int* positions, const int* token_item, int n_tokens, int n_heads,
                                                  int n_kv_heads, int head_size, int page_size, float scale, float cap,
                                                  int window, int block, const float* gate, long ld_gate, int chunk,
                                                  int max_chunks, float* part_acc, float* part_ml, int* counters,
                                                  void* stream) {
    return mllm_decode_split_attention_sink(out, ld_out, q, ld_q, k_pages, v_pages, block_table, max_blocks, positions,
                                            token_item, n_tokens, n_heads, n_kv_heads, head_size, page_size, scale, cap, window,
                                            block, gate, ld_gate, nullptr, chunk, max_chunks, part_acc, part_ml, counters, stream);
}

extern "C" int mllm_decode_split_attention_capped(void* out, long ld_out, const void* q, long ld_q, const void* k_pages,
                                                  const void* v_pages, const int* block_table, int max_blocks,
                                                  const int* positions, const int* token_item, int n_tokens, int n_heads,
                                                  int n_kv_heads, int head_size, int page_size, float scale, float cap,
                                                  int window, int chunk, int max_chunks, float* part_acc, float* part_ml,
                                                  int* counters, void* stream) {
    return mllm_decode_split_attention_masked(out, ld_out, q, ld_q, k_pages, v_pages, block_table, max_blocks, positions,
                                              token_item, n_tokens, n_heads, n_kv_heads, head_size, page_size, scale, cap,
                                              window, 0, nullptr, 0, chunk, max_chunks, part_acc, part_ml, counters, stream);
}

extern "C" int mllm_decode_split_attention(void* out, long ld_out, const void* q, long ld_q, const void* k_pages,
                                           const void* v_pages, const int* block_table, int max_blocks,
                                           const int* positions, const int* token_item, int n_tokens, int n_heads,
                                           int n_kv_heads, int head_size, int page_size, float scale, int window,
                                           int chunk, int max_chunks, float* part_acc, float* part_ml, int* counters,
                                           void* stream) {
    return mllm_decode_split_attention_capped(out, ld_out, q, ld_q, k_pages, v_pages, block_table, max_blocks, positions,
                                              token_item, n_tokens, n_heads, n_kv_heads, head_size, page_size, scale, 0.0f,
                                              window, chunk, max_chunks, part_acc, part_ml, counters, stream);
}

// Whether split_attention takes a head size (the others run the plain kernel).
extern "C" int mllm_decode_split_attention_takes(int head_size) {
    return head_size == 16 || head_size == 32 || head_size == 64 || head_size == 128 || head_size == 256;
}

// ---------------------------------------------------------------------------
// group_attention: the same split-key attention with the products on mma.sync tiles.
//
// One CTA per (token, key/value head, chunk of keys); its four warps take tiles of 16 keys in
// turn.  The query heads that share the key/value head (1 to 8) are the rows of the tiles:
//   S[heads x 8 keys]  = Q[heads x dims] K^T      m16n8k16, A = Q (kept in registers), B = K
//   O[heads x 8 dims] += P[heads x 16 keys] V     A = P (the registers S came in), B = V
// Keys and values stream through a cp.async ring in shared memory (a warp's own slots); the
// key rows are read back as 16-byte chunks, the value tiles with ldmatrix.trans.  The dims of
// a row are taken in a permuted order that is the same for Q and K, so that a lane reads whole
// 16-byte chunks; both tiles are swizzled so that the reads have no bank conflicts.  The
// softmax is the online one of split_attention, per 16 keys, in 32-bit, in exp2 units; the
// partial states and their merge by the last CTA of a pair use split_attention's scratch
// layout.  Against one key per eight lanes this needs about a tenth of the instructions.
// ---------------------------------------------------------------------------
__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
    __nv_bfloat162 two = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<uint32_t*>(&two);
}

template <int D>       // head size: 64 or 128
__global__ void __launch_bounds__(128)
group_attention_kernel(bf16* __restrict__ out, long ld_out, const bf16* __restrict__ q, long ld_q,
                       const bf16* __restrict__ k_pages, const bf16* __restrict__ v_pages,
                       const int* __restrict__ block_table, int max_blocks, const int* __restrict__ positions,
                       const int* __restrict__ token_item, int n_heads, int n_kv_heads, int page_size, float scale,
                       int window, int chunk, int max_chunks, float* __restrict__ part_acc,
                       float* __restrict__ part_ml, int* __restrict__ counters) {
    constexpr int CH = D / 8;              // 16-byte chunks of a key or value row
    constexpr int PAIRS = D / 32;          // chunks a lane reads of a key row (each serves two k steps)
    constexpr int NT = D / 8;              // 8-dim tiles of the output
    constexpr int RING = 256 / D;          // tiles of 16 keys in flight per warp: 4 (D = 64) or 2
    constexpr int TILE_BYTES = 16 * D * 2; // one tile of keys (or values)
    extern __shared__ __align__(16) unsigned char ga_smem[];
    dependents_may_start();
    wait_for_earlier_kernels();
    const int t = blockIdx.x, hk = blockIdx.y, c = blockIdx.z;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int g = lane >> 2, tq = lane & 3;
    const int heads = n_heads / n_kv_heads;            // 1..8: rows of the tiles
    const int p = positions[t];
    const int lo = (window > 0 && p - window + 1 > 0) ? p - window + 1 : 0;
    const int c_first = lo / chunk, c_last = p / chunk;
    if (c < c_first || c > c_last) return;
    const int begin = max(lo, c * chunk), end = min(p, c * chunk + chunk - 1);     // inclusive
    const int* bt = block_table + (long)token_item[t] * max_blocks;
    const long kv_width = (long)n_kv_heads * D;
    const float scale_log2 = scale * 1.4426950408889634f;
    unsigned char* ring_k = ga_smem + (size_t)warp * RING * 2 * TILE_BYTES;
    unsigned char* ring_v = ring_k + RING * TILE_BYTES;

    // the queries of this lane's row: chunk 4u + tq serves k steps 2u (words 0, 1) and 2u + 1 (words 2, 3)
    uint32_t qa[PAIRS][4];
#pragma unroll
    for (int u = 0; u < PAIRS; u++) {
        uint4 v = make_uint4(0, 0, 0, 0);
        if (g < heads) v = *reinterpret_cast<const uint4*>(q + (long)t * ld_q + (long)(hk * heads + g) * D + (4 * u + tq) * 8);
        qa[u][0] = v.x; qa[u][1] = v.y; qa[u][2] = v.z; qa[u][3] = v.w;
    }
    float o[NT][2];
#pragma unroll
    for (int j = 0; j < NT; j++) o[j][0] = o[j][1] = 0.0f;
    float m = -INFINITY, l = 0.0f;         // of row g; l is this lane's share of the sum

    const int n_tiles = (end - begin) / 16 + 1;                         // of the chunk
    const int my_tiles = n_tiles > warp ? (n_tiles - warp + 3) / 4 : 0; // tiles warp, warp + 4, ...
    auto issue = [&](int i) {
        if (i < my_tiles) {
            const int first = begin + (warp + 4 * i) * 16;
            unsigned char* tk = ring_k + (i % RING) * TILE_BYTES;
            unsigned char* tv = ring_v + (i % RING) * TILE_BYTES;
#pragma unroll
            for (int r = 0; r < CH / 2; r++) {
                const int idx = lane + 32 * r, key = idx / CH, ch = idx % CH;
                const int j = first + key;
                // keys: chunk position xor 4 on odd rows; values: xor the row's low three bits
                unsigned char* dk = tk + key * (D * 2) + ((ch & ~7) | ((ch ^ ((key & 1) << 2)) & 7)) * 16;
                unsigned char* dv = tv + key * (D * 2) + ((ch & ~7) | ((ch ^ key) & 7)) * 16;
                if (j <= end) {
                    const long base = ((long)bt[j / page_size] * page_size + (j % page_size)) * kv_width + (long)hk * D + ch * 8;
                    cp_async_16(dk, k_pages + base);
                    cp_async_16(dv, v_pages + base);
                } else {
                    *reinterpret_cast<uint4*>(dv) = make_uint4(0, 0, 0, 0);     // a value that is never weighted must not be NaN
                    *reinterpret_cast<uint4*>(dk) = make_uint4(0, 0, 0, 0);
                }
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    for (int i = 0; i < RING - 1; i++) issue(i);
    for (int i = 0; i < my_tiles; i++) {
        issue(i + RING - 1);
        asm volatile("cp.async.wait_group %0;" ::"n"(RING - 1) : "memory");
        __syncwarp();                                   // every lane's copies of this tile have landed
        const int first = begin + (warp + 4 * i) * 16;
        const unsigned char* tk = ring_k + (i % RING) * TILE_BYTES;
        const uint32_t tv = (uint32_t)__cvta_generic_to_shared(ring_v + (i % RING) * TILE_BYTES);
        // scores of row g against keys 2 tq, 2 tq + 1 of both halves of the tile
        float s[2][4];
#pragma unroll
        for (int h = 0; h < 2; h++) {
            s[h][0] = s[h][1] = s[h][2] = s[h][3] = 0.0f;
            const int key = 8 * h + g;
#pragma unroll
            for (int u = 0; u < PAIRS; u++) {
                const int ch = 4 * u + tq;
                const uint4 kb = *reinterpret_cast<const uint4*>(tk + key * (D * 2) + ((ch & ~7) | ((ch ^ ((key & 1) << 2)) & 7)) * 16);
                mma_bf16_16816(s[h][0], s[h][1], s[h][2], s[h][3], qa[u][0], 0u, qa[u][1], 0u, kb.x, kb.y);
                mma_bf16_16816(s[h][0], s[h][1], s[h][2], s[h][3], qa[u][2], 0u, qa[u][3], 0u, kb.z, kb.w);
            }
        }
        float tile_max = -INFINITY;
#pragma unroll
        for (int h = 0; h < 2; h++)
#pragma unroll
            for (int e = 0; e < 2; e++) {
                const int j = first + 8 * h + 2 * tq + e;
                s[h][e] = j <= end ? s[h][e] * scale_log2 : -INFINITY;
                tile_max = fmaxf(tile_max, s[h][e]);
            }
        tile_max = fmaxf(tile_max, __shfl_xor_sync(0xffffffffu, tile_max, 1));
        tile_max = fmaxf(tile_max, __shfl_xor_sync(0xffffffffu, tile_max, 2));
        const float m_new = fmaxf(m, tile_max);           // finite: the tile's first key is never past the end
        const float corr = exp2f(m - m_new);
        const float p00 = exp2f(s[0][0] - m_new), p01 = exp2f(s[0][1] - m_new);
        const float p10 = exp2f(s[1][0] - m_new), p11 = exp2f(s[1][1] - m_new);
        const uint32_t pa0 = pack_bf16(p00, p01), pa1 = pack_bf16(p10, p11);
        // the sum uses the rounded weights the product below sees
        const __nv_bfloat162 r0 = *reinterpret_cast<const __nv_bfloat162*>(&pa0), r1 = *reinterpret_cast<const __nv_bfloat162*>(&pa1);
        l = l * corr + (__low2float(r0) + __high2float(r0)) + (__low2float(r1) + __high2float(r1));
        m = m_new;
        float unused0 = 0.0f, unused1 = 0.0f;             // rows 8..15 of the tiles
#pragma unroll
        for (int j = 0; j < NT; j += 2) {
            // four 8 x 8 blocks of the value tile, transposed: (keys 0-7 | 8-15) x (dims 8j.. | 8(j+1)..)
            const int key = (lane & 7) + ((lane >> 3) & 1) * 8, ch = j + (lane >> 4);
            uint32_t b0, b1, b2, b3;
            asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
                         : "=r"(b0), "=r"(b1), "=r"(b2), "=r"(b3)
                         : "r"(tv + key * (D * 2) + ((ch & ~7) | ((ch ^ key) & 7)) * 16));
            o[j][0] *= corr; o[j][1] *= corr; o[j + 1][0] *= corr; o[j + 1][1] *= corr;
            mma_bf16_16816(o[j][0], o[j][1], unused0, unused1, pa0, 0u, pa1, 0u, b0, b1);
            mma_bf16_16816(o[j + 1][0], o[j + 1][1], unused0, unused1, pa0, 0u, pa1, 0u, b2, b3);
        }
        __syncwarp();                                   // the slot is copied into again two issues from now
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    l += __shfl_xor_sync(0xffffffffu, l, 1);
    l += __shfl_xor_sync(0xffffffffu, l, 2);

    // merge the four warps (through the ring, free by now), always in the same order
    __syncthreads();
    float* sm_m = reinterpret_cast<float*>(ga_smem);           // [4][8]
    float* sm_l = sm_m + 32;                                   // [4][8]
    float* sm_acc = sm_l + 32;                                 // [4][8][D]
    if (tq == 0) {
        sm_m[warp * 8 + g] = m;
        sm_l[warp * 8 + g] = l;
    }
#pragma unroll
    for (int j = 0; j < NT; j++) {
        sm_acc[(warp * 8 + g) * D + 8 * j + 2 * tq] = o[j][0];
        sm_acc[(warp * 8 + g) * D + 8 * j + 2 * tq + 1] = o[j][1];
    }
    __syncthreads();
    __shared__ int is_last[8];
    for (int row = 0; row < heads; row++) {
        const int h = hk * heads + row;
        float big = -INFINITY;
        for (int w = 0; w < 4; w++) big = fmaxf(big, sm_m[w * 8 + row]);
        const long cell = (((long)t * n_heads + h) * max_chunks + c);
        for (int d = threadIdx.x; d < D; d += 128) {
            float acc = 0.0f;
            for (int w = 0; w < 4; w++) {
                const float mw = sm_m[w * 8 + row];
                if (mw != -INFINITY) acc += sm_acc[(w * 8 + row) * D + d] * exp2f(mw - big);
            }
            part_acc[cell * D + d] = acc;
        }
        if (threadIdx.x == 0) {
            float total = 0.0f;
            for (int w = 0; w < 4; w++) {
                const float mw = sm_m[w * 8 + row];
                if (mw != -INFINITY) total += sm_l[w * 8 + row] * exp2f(mw - big);
            }
            part_ml[cell * 2] = big;
            part_ml[cell * 2 + 1] = total;
        }
    }
    // the CTA that arrives last for a (token, head) merges the chunks
    __threadfence();
    __syncthreads();
    if (threadIdx.x < heads) {
        const int h = hk * heads + threadIdx.x;
        const int ticket = atomicAdd(&counters[t * n_heads + h], 1);
        is_last[threadIdx.x] = (ticket == c_last - c_first);
        if (is_last[threadIdx.x]) counters[t * n_heads + h] = 0;      // ready for the next launch
    }
    __syncthreads();
    for (int row = 0; row < heads; row++) {
        if (!is_last[row]) continue;
        __threadfence();
        const int h = hk * heads + row;
        const long first_cell = ((long)t * n_heads + h) * max_chunks;
        float top = -INFINITY;
        for (int cc = c_first; cc <= c_last; cc++) top = fmaxf(top, __ldcg(part_ml + (first_cell + cc) * 2));
        float denom = 0.0f;
        for (int cc = c_first; cc <= c_last; cc++)
            denom += __ldcg(part_ml + (first_cell + cc) * 2 + 1) * exp2f(__ldcg(part_ml + (first_cell + cc) * 2) - top);
        for (int d = threadIdx.x; d < D; d += 128) {
            float acc = 0.0f;
            for (int cc = c_first; cc <= c_last; cc++)
                acc += __ldcg(part_acc + (first_cell + cc) * D + d) * exp2f(__ldcg(part_ml + (first_cell + cc) * 2) - top);
            out[(long)t * ld_out + (long)h * D + d] = __float2bfloat16_rn(acc / denom);
        }
    }
}

// Whether group_attention takes a layout: head size 64 or 128, at most eight query heads per
// key/value head, rows of q on 16-byte boundaries.
extern "C" int mllm_decode_group_attention_takes(int head_size, int n_heads, int n_kv_heads, long ld_q, const void* q) {
    return (head_size == 64 || head_size == 128) && n_kv_heads > 0 && n_heads % n_kv_heads == 0 &&
           n_heads / n_kv_heads <= 8 && ld_q % 8 == 0 && (reinterpret_cast<uintptr_t>(q) & 15) == 0;
}

// Same arguments and scratch as mllm_decode_split_attention; chunk must be a multiple of 16.
extern "C" int mllm_decode_group_attention(void* out, long ld_out, const void* q, long ld_q, const void* k_pages,
                                           const void* v_pages, const int* block_table, int max_blocks,
                                           const int* positions, const int* token_item, int n_tokens, int n_heads,
                                           int n_kv_heads, int head_size, int page_size, float scale, int window,
                                           int chunk, int max_chunks, float* part_acc, float* part_ml, int* counters,
                                           void* stream) {
    if (n_tokens <= 0) return 0;
    if (!mllm_decode_group_attention_takes(head_size, n_heads, n_kv_heads, ld_q, q))
        return fail("group_attention: head size 64 or 128, at most 8 query heads per key/value head, q 16-byte aligned");
    if (chunk <= 0 || chunk % 16 != 0 || max_chunks <= 0 || max_chunks > 65535 || n_kv_heads > 65535)
        return fail("group_attention: bad chunking");
    cudaStream_t s = (cudaStream_t)stream;
    dim3 grid(n_tokens, n_kv_heads, max_chunks);
    const size_t smem = (size_t)4 * (256 / head_size) * 2 * 16 * head_size * 2;       // 64 KB
    static bool configured = false;
    if (!configured) {
        if (cudaFuncSetAttribute(group_attention_kernel<64>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess ||
            cudaFuncSetAttribute(group_attention_kernel<128>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess)
            return fail("group_attention: cannot raise the shared memory limit");
        configured = true;
    }
#define LAUNCH_GROUP(D)                                                                                              \
    launch_kernel(g_dependent_launch != 0, group_attention_kernel<D>, grid, dim3(128), smem, s, (bf16*)out, ld_out,  \
                  (const bf16*)q, ld_q, (const bf16*)k_pages, (const bf16*)v_pages, block_table, max_blocks,         \
                  positions, token_item, n_heads, n_kv_heads, page_size, scale, window, chunk, max_chunks, part_acc, \
                  part_ml, counters)
    if (head_size == 64) LAUNCH_GROUP(64);
    else LAUNCH_GROUP(128);
#undef LAUNCH_GROUP
    return check_launch("group_attention_kernel");
}

// ---------------------------------------------------------------------------
// Layer norm, one warp per row, the row read once.  Each lane keeps up to HELD chunks of
// four values in registers (eight: rows up to 1024 wide; sixteen: up to 2048; measured at
// 2048 x 1600: 5.6 us with the row re-read for each pass); a wider row is re-read.
// Same arithmetic as the plain kernel: mean, variance of the centred values, then
// (x - mean) / sqrt(var + eps) * gain + shift, all in 32-bit; the output is bfloat16.
// ---------------------------------------------------------------------------
template <int HELD>
__global__ void __launch_bounds__(256)
layernorm_warp_kernel(bf16* __restrict__ out, const float* __restrict__ x, const float* __restrict__ gamma,
                      const float* __restrict__ beta, const int* __restrict__ rows, int n_rows, int width, float eps) {
    dependents_may_start();
    wait_for_earlier_kernels();
    const int lane = threadIdx.x & 31;
    const int r = blockIdx.x * 8 + (threadIdx.x >> 5);
    if (r >= n_rows) return;
    const float4* row = reinterpret_cast<const float4*>(x + (long)(rows ? rows[r] : r) * width);
    const int quads = width / 4;
    const bool held = quads <= 32 * HELD;
    float4 keep[HELD];
    float sum = 0.0f;
#pragma unroll
    for (int i = 0; i < HELD; i++) {
        keep[i] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (held && lane + 32 * i < quads) keep[i] = row[lane + 32 * i];
        sum += keep[i].x + keep[i].y + keep[i].z + keep[i].w;
    }
    if (!held)
        for (int q = lane; q < quads; q += 32) {
            const float4 v = row[q];
            sum += v.x + v.y + v.z + v.w;
        }
    const float mean = warp_sum(sum) / (float)width;
    float sq = 0.0f;
    if (held) {
#pragma unroll
        for (int i = 0; i < HELD; i++)
            if (lane + 32 * i < quads) {
                const float a = keep[i].x - mean, b = keep[i].y - mean, c = keep[i].z - mean, d = keep[i].w - mean;
                sq += a * a + b * b + c * c + d * d;
            }
    } else {
        for (int q = lane; q < quads; q += 32) {
            const float4 v = row[q];
            const float a = v.x - mean, b = v.y - mean, c = v.z - mean, d = v.w - mean;
            sq += a * a + b * b + c * c + d * d;
        }
    }
    const float inv = 1.0f / sqrtf(warp_sum(sq) / (float)width + eps);
    auto emit = [&](int q, const float4& v) {
        const float4 g = __ldg(reinterpret_cast<const float4*>(gamma) + q);
        const float4 b = __ldg(reinterpret_cast<const float4*>(beta) + q);
        __nv_bfloat162 lo = __floats2bfloat162_rn((v.x - mean) * inv * g.x + b.x, (v.y - mean) * inv * g.y + b.y);
        __nv_bfloat162 hi = __floats2bfloat162_rn((v.z - mean) * inv * g.z + b.z, (v.w - mean) * inv * g.w + b.w);
        *reinterpret_cast<uint2*>(out + (long)r * width + q * 4) =
            make_uint2(*reinterpret_cast<uint32_t*>(&lo), *reinterpret_cast<uint32_t*>(&hi));
    };
    if (held) {
#pragma unroll
        for (int i = 0; i < HELD; i++)
            if (lane + 32 * i < quads) emit(lane + 32 * i, keep[i]);
    } else {
        for (int q = lane; q < quads; q += 32) emit(q, row[q]);
    }
}

// A block a row, 16 bytes of it a thread: gain and shift are there before the kernels ahead have ended (no kernel of a step
// writes them), and the row takes one pass of loads, two sums with one barrier each and the store.  A warp a row walked up to
// thirteen dependent pieces of it: 64 rows of 768 2.2 -> 1.8 us, of 1,600 3.6 -> 2.1 (replayed back to back).
__global__ void __launch_bounds__(1024)
layernorm_block_kernel(bf16* __restrict__ out, const float* __restrict__ x, const float* __restrict__ gamma,
                       const float* __restrict__ beta, const int* __restrict__ rows, int width, float eps) {
    __shared__ float slots[2][32];
    const int q = threadIdx.x;
    const bool there = q < width / 4;
    const float4 none = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    dependents_may_start();
    const float4 g = there ? __ldg(reinterpret_cast<const float4*>(gamma) + q) : none;
    const float4 b = there ? __ldg(reinterpret_cast<const float4*>(beta) + q) : none;
    wait_for_earlier_kernels();
    x = behind_the_wait(x);
    const int r = blockIdx.x;
    float4 v = there ? reinterpret_cast<const float4*>(x + (long)(rows ? rows[r] : r) * width)[q] : none;
    const float mean = block_sum_once(v.x + v.y + v.z + v.w, slots[0]) / (float)width;
    v.x -= mean; v.y -= mean; v.z -= mean; v.w -= mean;
    const float sq = there ? v.x * v.x + v.y * v.y + v.z * v.z + v.w * v.w : 0.0f;
    const float inv = 1.0f / sqrtf(block_sum_once(sq, slots[1]) / (float)width + eps);
    if (!there) return;
    __nv_bfloat162 lo = __floats2bfloat162_rn(v.x * inv * g.x + b.x, v.y * inv * g.y + b.y);
    __nv_bfloat162 hi = __floats2bfloat162_rn(v.z * inv * g.z + b.z, v.w * inv * g.w + b.w);
    *reinterpret_cast<uint2*>(out + (long)r * width + q * 4) =
        make_uint2(*reinterpret_cast<uint32_t*>(&lo), *reinterpret_cast<uint32_t*>(&hi));
}

// x fp32 [*, width] (width a multiple of 4), out bfloat16 [n_rows, width]; rows: optional gather.
extern "C" int mllm_decode_layernorm(void* out, const float* x, const float* gamma, const float* beta, const int* rows,
                                     int n_rows, int width, float eps, void* stream) {
    if (n_rows <= 0) return 0;
    if (width <= 0 || width % 4 != 0) return fail("layernorm: the width must be a multiple of 4");
    // few rows wait for one row's passes; many are bound by instructions, where a warp a row needs fewer (2,048 x 768: 2.7
    // against 4.2 us; 64 x 768: 2.2 against 1.8)
    if (width <= 4096 && n_rows <= 256)
        return launched(launch_kernel(g_dependent_launch != 0, layernorm_block_kernel, dim3(n_rows), dim3((width / 4 + 31) / 32 * 32), 0,
                                      (cudaStream_t)stream, (bf16*)out, x, gamma, beta, rows, width, eps),
                        "layernorm_block_kernel");
    if (width <= 1024)
        return launched(launch_kernel(g_dependent_launch != 0, layernorm_warp_kernel<8>, dim3((n_rows + 7) / 8), dim3(256), 0,
                                      (cudaStream_t)stream, (bf16*)out, x, gamma, beta, rows, n_rows, width, eps),
                        "layernorm_warp_kernel");
    return launched(launch_kernel(g_dependent_launch != 0, layernorm_warp_kernel<16>, dim3((n_rows + 7) / 8), dim3(256), 0,
                                  (cudaStream_t)stream, (bf16*)out, x, gamma, beta, rows, n_rows, width, eps),
                    "layernorm_warp_kernel");
}

// ---------------------------------------------------------------------------
// split_attention with built-in scratch, for callers that cannot allocate
// (see split_attention_static.h for who they are and what the limits mean).
// ---------------------------------------------------------------------------
#include "split_attention_static.h"

// Device memory.  In host code this name is only a handle for the symbol, not an address a
// kernel could use: the address is asked for once per device, below.
static __device__ __align__(256) unsigned char
    g_static_scratch[(MLLM_STATIC_ACC_FLOATS + MLLM_STATIC_ML_FLOATS) * sizeof(float) +
                     MLLM_STATIC_COUNTERS * sizeof(int)];

constexpr int STATIC_MAX_DEVICES = 64;
static unsigned char* g_static_address[STATIC_MAX_DEVICES] = {nullptr};

extern "C" int mllm_decode_split_attention_static(void* out, long ld_out, const void* q, long ld_q,
                                                  const void* k_pages, const void* v_pages, const int* block_table,
                                                  int max_blocks, const int* positions, const int* token_item,
                                                  int n_tokens, int n_heads, int n_kv_heads, int head_size,
                                                  int page_size, float scale, int window, int chunk, void* stream) {
    if (n_tokens <= 0) return 0;
    if (n_heads <= 0 || chunk <= 0 || page_size <= 0 || max_blocks <= 0 || head_size <= 0)
        return fail("split_attention_static: sizes must be positive");
    const long chunks = ((long)max_blocks * page_size + chunk - 1) / chunk;
    const long pairs = (long)n_tokens * n_heads;
    if (pairs > MLLM_STATIC_COUNTERS || pairs * chunks * 2 > MLLM_STATIC_ML_FLOATS ||
        pairs * chunks * head_size > MLLM_STATIC_ACC_FLOATS) {
        snprintf(g_error_text, MLLM_ERROR_BUFFER,
                 "split_attention_static: %d tokens x %d heads x %ld chunks x head size %d exceed the built-in scratch "
                 "(%d partial floats, %d max/sum floats, %d counters); use mllm_decode_split_attention with your own",
                 n_tokens, n_heads, chunks, head_size, MLLM_STATIC_ACC_FLOATS, MLLM_STATIC_ML_FLOATS,
                 MLLM_STATIC_COUNTERS);
        return 1;
    }
    int device = -1;
    if (cudaGetDevice(&device) != cudaSuccess || device < 0 || device >= STATIC_MAX_DEVICES)
        return fail("split_attention_static: cannot tell the current device");
    if (g_static_address[device] == nullptr) {
        // set-up, once per device, with that device current
        void* address = nullptr;
        cudaError_t e = cudaGetSymbolAddress(&address, g_static_scratch);
        if (e != cudaSuccess || address == nullptr) {
            snprintf(g_error_text, MLLM_ERROR_BUFFER, "split_attention_static: cudaGetSymbolAddress failed: %s",
                     cudaGetErrorString(e));
            return 2;
        }
        g_static_address[device] = static_cast<unsigned char*>(address);
    }
    float* part_acc = reinterpret_cast<float*>(g_static_address[device]);
    float* part_ml = part_acc + MLLM_STATIC_ACC_FLOATS;
    int* counters = reinterpret_cast<int*>(part_ml + MLLM_STATIC_ML_FLOATS);
    // The array keeps the last call's contents; the counters must start at zero.
    cudaError_t e = cudaMemsetAsync(counters, 0, (size_t)pairs * sizeof(int), (cudaStream_t)stream);
    if (e != cudaSuccess) {
        snprintf(g_error_text, MLLM_ERROR_BUFFER, "split_attention_static: clearing the counters failed: %s",
                 cudaGetErrorString(e));
        return 2;
    }
    return mllm_decode_split_attention(out, ld_out, q, ld_q, k_pages, v_pages, block_table, max_blocks, positions,
                                       token_item, n_tokens, n_heads, n_kv_heads, head_size, page_size, scale, window,
                                       chunk, (int)chunks, part_acc, part_ml, counters, stream);
}
