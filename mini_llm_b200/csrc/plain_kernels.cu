// Plain kernels: one straightforward SIMT kernel for every operation of a
// step.  With 32-bit element types they are the true 32-bit path of the whole
// model (scalar fp32 FMA, no tensor cores, no reduced-precision matrix mode);
// with bfloat16 element types they are the twin each fast kernel is checked
// against, and the kernel of last resort for sizes a fast kernel refuses.
// Sums, softmax and norm statistics are always 32-bit.
//
// Operations and their formulas follow the reference's CPU operators:
//   embedding   engine/src/embedding.c:9-15
//   layer norm  engine/src/layernorm.c:12-33
//   linear      engine/src/linear.c:5-19
//   attention   engine/src/attention.c:24-49 with the causal softmax of
//               engine/src/softmax.c:29-55, in the online form of
//               engine/src/attention.cu:98-123
#include <cooperative_groups.h>

#include "common.cuh"

MLLM_DEFINE_ERROR_API(mllm_plain)

// ---------------------------------------------------------------------------
// Embedding: out[t, :] = scale * table[id[t], :] (+ position_table[pos[t], :])
// ---------------------------------------------------------------------------
template <typename W>
__global__ void embed_kernel(float* __restrict__ out, const int* __restrict__ ids,
                             const int* __restrict__ positions, const W* __restrict__ table,
                             const W* __restrict__ position_table, int width, float scale) {
    dependents_may_start();
    wait_for_earlier_kernels();
    int t = blockIdx.x;
    long row = (long)ids[t] * width;
    if (position_table != nullptr) {
        long prow = (long)positions[t] * width;
        for (int d = threadIdx.x; d < width; d += blockDim.x)
            out[(long)t * width + d] = to_f32(table[row + d]) * scale + to_f32(position_table[prow + d]);
    } else {
        for (int d = threadIdx.x; d < width; d += blockDim.x)
            out[(long)t * width + d] = to_f32(table[row + d]) * scale;
    }
}

// hidden[t, :] += position_table[pos[t], :]   (position encoding applied alone)
template <typename W>
__global__ void add_rows_kernel(float* __restrict__ hidden, const int* __restrict__ positions,
                                const W* __restrict__ table, int width) {
    int t = blockIdx.x;
    long prow = (long)positions[t] * width;
    for (int d = threadIdx.x; d < width; d += blockDim.x)
        hidden[(long)t * width + d] += to_f32(table[prow + d]);
}

extern "C" int mllm_plain_embed(float* out, const int* ids, const int* positions, const void* table,
                                const void* position_table, int n_tokens, int width, float scale, int table_dtype,
                                void* stream) {
    if (n_tokens <= 0) return 0;
    cudaStream_t s = (cudaStream_t)stream;
    int threads = width >= 256 ? 256 : 64;
    if (table_dtype == DT_F32)
        launch_kernel(AFTER_THE_KERNELS_AHEAD, embed_kernel<float>, dim3(n_tokens), dim3(threads), 0, s, out, ids, positions,
                      (const float*)table, (const float*)position_table, width, scale);
    else if (table_dtype == DT_BF16)
        launch_kernel(AFTER_THE_KERNELS_AHEAD, embed_kernel<bf16>, dim3(n_tokens), dim3(threads), 0, s, out, ids, positions,
                      (const bf16*)table, (const bf16*)position_table, width, scale);
    else
        return fail("embed: unknown table dtype");
    return check_launch("embed_kernel");
}

extern "C" int mllm_plain_add_rows(float* hidden, const int* positions, const void* table, int n_tokens,
                                   int width, int table_dtype, void* stream) {
    if (n_tokens <= 0) return 0;
    cudaStream_t s = (cudaStream_t)stream;
    int threads = width >= 256 ? 256 : 64;
    if (table_dtype == DT_F32)
        add_rows_kernel<float><<<n_tokens, threads, 0, s>>>(hidden, positions, (const float*)table, width);
    else if (table_dtype == DT_BF16)
        add_rows_kernel<bf16><<<n_tokens, threads, 0, s>>>(hidden, positions, (const bf16*)table, width);
    else
        return fail("add_rows: unknown table dtype");
    return check_launch("add_rows_kernel");
}

// ---------------------------------------------------------------------------
// Layer norm, one block per row.  mean, then the variance of the centred
// values (biased), then (x - mean) * (1 / sqrt(var + eps)) * gamma + beta.
// `rows` (may be null) gathers: output row r is computed from input row
// rows[r].
// ---------------------------------------------------------------------------
template <typename O>
__global__ void layernorm_kernel(O* __restrict__ out, const float* __restrict__ x,
                                 const float* __restrict__ gamma, const float* __restrict__ beta,
                                 const int* __restrict__ rows, int width, float eps) {
    __shared__ float scratch[33];
    int r = blockIdx.x;
    const float* row = x + (long)(rows ? rows[r] : r) * width;
    float sum = 0.0f;
    for (int d = threadIdx.x; d < width; d += blockDim.x) sum += row[d];
    float mean = block_sum(sum, scratch) / (float)width;
    float sq = 0.0f;
    for (int d = threadIdx.x; d < width; d += blockDim.x) {
        float c = row[d] - mean;
        sq += c * c;
    }
    float var = block_sum(sq, scratch) / (float)width;
    float inv = 1.0f / sqrtf(var + eps);
    for (int d = threadIdx.x; d < width; d += blockDim.x) {
        float n = (row[d] - mean) * inv;
        out[(long)r * width + d] = from_f32<O>(n * gamma[d] + beta[d]);
    }
}

// 32-bit rows whose width is a multiple of 4 (up to 4,096): the row is read once, 16 bytes a lane, and stays in registers
// through both sums.  A few rows are bound by the latency of their dependent passes (loads, two sums over the block,
// store), not by bytes: three passes over memory cost 5.7 us at 4 x 768, one costs 3.
__global__ void __launch_bounds__(256)
layernorm_float_kernel(float* __restrict__ out, const float* __restrict__ x, const float* __restrict__ gamma,
                       const float* __restrict__ beta, const int* __restrict__ rows, int width, float eps) {
    __shared__ float scratch[33];
    dependents_may_start();
    wait_for_earlier_kernels();
    x = behind_the_wait(x);
    rows = behind_the_wait(rows);
    const int r = blockIdx.x, quads = width / 4;
    const float4* row = reinterpret_cast<const float4*>(x + (long)(rows ? rows[r] : r) * width);
    float4 v[4];
    float sum = 0.0f;
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const int c = threadIdx.x + i * 256;
        v[i] = c < quads ? row[c] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        sum += (v[i].x + v[i].y) + (v[i].z + v[i].w);
    }
    const float mean = block_sum(sum, scratch) / (float)width;
    float sq = 0.0f;
#pragma unroll
    for (int i = 0; i < 4; i++) {
        if (threadIdx.x + i * 256 < quads) {
            v[i].x -= mean; v[i].y -= mean; v[i].z -= mean; v[i].w -= mean;
            sq += (v[i].x * v[i].x + v[i].y * v[i].y) + (v[i].z * v[i].z + v[i].w * v[i].w);
        }
    }
    const float inv = 1.0f / sqrtf(block_sum(sq, scratch) / (float)width + eps);
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const int c = threadIdx.x + i * 256;
        if (c < quads) {
            const float4 g = reinterpret_cast<const float4*>(gamma)[c], b = reinterpret_cast<const float4*>(beta)[c];
            reinterpret_cast<float4*>(out + (long)r * width)[c] =
                make_float4(v[i].x * inv * g.x + b.x, v[i].y * inv * g.y + b.y, v[i].z * inv * g.z + b.z, v[i].w * inv * g.w + b.w);
        }
    }
}

static bool on_16_bytes(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

extern "C" int mllm_plain_layernorm(void* out, const float* x, const float* gamma, const float* beta,
                                    const int* rows, int n_rows, int width, float eps, int out_dtype,
                                    void* stream) {
    if (n_rows <= 0) return 0;
    cudaStream_t s = (cudaStream_t)stream;
    int threads = width >= 1024 ? 256 : (width >= 256 ? 128 : 64);
    if (out_dtype == DT_F32 && width % 4 == 0 && width <= 4096 && on_16_bytes(out) && on_16_bytes(x) && on_16_bytes(gamma) &&
        on_16_bytes(beta))
        return launched(launch_kernel(g_dependent_launch != 0, layernorm_float_kernel, dim3(n_rows), dim3(256), 0, s, (float*)out,
                                      x, gamma, beta, rows, width, eps), "layernorm_float_kernel");
    if (out_dtype == DT_F32)
        layernorm_kernel<float><<<n_rows, threads, 0, s>>>((float*)out, x, gamma, beta, rows, width, eps);
    else if (out_dtype == DT_BF16)
        layernorm_kernel<bf16><<<n_rows, threads, 0, s>>>((bf16*)out, x, gamma, beta, rows, width, eps);
    else
        return fail("layernorm: unknown output dtype");
    return check_launch("layernorm_kernel");
}

// ---------------------------------------------------------------------------
// Linear: out[m, n] = epilogue(sum_k a[m, k] * w[n, k] + bias[n]).
// `w` is [N, K] with K contiguous.  64x64 tile, 256 threads, each 4x4
// outputs; the sum over k runs in order with fp32 FMA.
// ---------------------------------------------------------------------------
template <typename AT, typename WT, typename OT, int EPI>
__global__ void __launch_bounds__(256)
linear_plain_kernel(OT* __restrict__ out, const AT* __restrict__ a, const WT* __restrict__ w,
                    const float* __restrict__ bias, int M, int N, int K, long lda, long ldo) {
    constexpr int BM = 64, BN = 64, BK = 16;
    __shared__ float As[BK][BM + 4];
    __shared__ float Ws[BK][BN + 4];
    int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
    float acc[4][4];
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
        for (int j = 0; j < 4; j++) acc[i][j] = 0.0f;

    for (int k0 = 0; k0 < K; k0 += BK) {
        for (int i = threadIdx.x; i < BM * BK; i += 256) {
            int r = i / BK, c = i % BK;
            int gm = m0 + r, gn = n0 + r, gk = k0 + c;
            As[c][r] = (gm < M && gk < K) ? to_f32(a[(long)gm * lda + gk]) : 0.0f;
            Ws[c][r] = (gn < N && gk < K) ? to_f32(w[(long)gn * K + gk]) : 0.0f;
        }
        __syncthreads();
#pragma unroll
        for (int kk = 0; kk < BK; kk++) {
            float av[4], wv[4];
#pragma unroll
            for (int i = 0; i < 4; i++) av[i] = As[kk][ty * 4 + i];
#pragma unroll
            for (int j = 0; j < 4; j++) wv[j] = Ws[kk][tx * 4 + j];
#pragma unroll
            for (int i = 0; i < 4; i++)
#pragma unroll
                for (int j = 0; j < 4; j++) acc[i][j] = fmaf(av[i], wv[j], acc[i][j]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 4; i++) {
        int gm = m0 + ty * 4 + i;
        if (gm >= M) continue;
#pragma unroll
        for (int j = 0; j < 4; j++) {
            int gn = n0 + tx * 4 + j;
            if (gn >= N) continue;
            float v = acc[i][j] + (bias ? bias[gn] : 0.0f);
            long o = (long)gm * ldo + gn;
            if (EPI == EPI_ADD)
                out[o] = from_f32<OT>(to_f32(out[o]) + v);
            else
                out[o] = from_f32<OT>(apply_activation<EPI>(v));
        }
    }
}

__device__ __forceinline__ float activate(int epilogue, float v) {
    switch (epilogue) {
    case EPI_GELU_TANH: return gelu_tanh_f(v);
    case EPI_GELU_ERF: return gelu_erf_f(v);
    case EPI_RELU_SQ: return apply_activation<EPI_RELU_SQ>(v);
    case EPI_SILU: return apply_activation<EPI_SILU>(v);
    default: return v;
    }
}

// 32-bit operands, up to 8 rows: the product is a stream of the weights, bound by HBM and by the latency of one pass.
// The rows of `a` lie in shared memory; `split` warps share the inner size of F output features between them (their sums meet
// in shared memory in warp order), so that a product of 768 features still brings 3,072 warps.  The first four
// 16-byte pieces of each feature are asked for before the kernels ahead have ended: no kernel writes weights.
// 4 x 768 x 3072: 300 us with the 64-wide tiles below (12 blocks, 94 % of the rows padding), under 10 us so.
template <int MT, int F>
__global__ void __launch_bounds__(256)
linear_float_rows_kernel(float* __restrict__ out, const float* __restrict__ a, const float* __restrict__ w,
                         const float* __restrict__ bias, int M, int N, int K, long lda, long ldo, int epilogue, int split) {
    extern __shared__ __align__(16) float rows_shared[];                  // [MT][K]
    __shared__ float partial[8][F][MT];
    constexpr int AHEAD = F == 1 ? 4 : 2;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int quads = K / 4, part = warp % split;
    const int per_part = ((quads + split - 1) / split + 31) / 32 * 32;
    const int begin = part * per_part, end = min(quads, begin + per_part);
    const int n0 = (blockIdx.x * (8 / split) + warp / split) * F;
    const float4* wrow[F];
#pragma unroll
    for (int f = 0; f < F; f++) wrow[f] = reinterpret_cast<const float4*>(w + (long)min(n0 + f, N - 1) * K);
    float4 ahead[F][AHEAD];
    dependents_may_start();
#pragma unroll
    for (int i = 0; i < AHEAD; i++)
#pragma unroll
        for (int f = 0; f < F; f++) {
            const int c = begin + lane + 32 * i;
            ahead[f][i] = c < end ? __ldg(wrow[f] + c) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        }
    wait_for_earlier_kernels();
    a = behind_the_wait(a);
    for (int m = 0; m < MT; m++)
        for (int c = threadIdx.x; c < quads; c += 256)
            reinterpret_cast<float4*>(rows_shared + (long)m * K)[c] =
                m < M ? reinterpret_cast<const float4*>(a + (long)m * lda)[c] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    __syncthreads();
    float acc[F][MT];
#pragma unroll
    for (int f = 0; f < F; f++)
#pragma unroll
        for (int m = 0; m < MT; m++) acc[f][m] = 0.0f;
    for (int first = begin + lane; first < end; first += 32 * AHEAD) {
        float4 now[F][AHEAD];
#pragma unroll
        for (int i = 0; i < AHEAD; i++)
#pragma unroll
            for (int f = 0; f < F; f++) {
                now[f][i] = ahead[f][i];
                const int c = first + 32 * (AHEAD + i);
                ahead[f][i] = c < end ? __ldg(wrow[f] + c) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            }
#pragma unroll
        for (int i = 0; i < AHEAD; i++) {
            const int c = first + 32 * i;
            if (c >= end) break;
#pragma unroll
            for (int m = 0; m < MT; m++) {
                const float4 x = reinterpret_cast<const float4*>(rows_shared + (long)m * K)[c];
#pragma unroll
                for (int f = 0; f < F; f++) {
                    acc[f][m] = fmaf(now[f][i].x, x.x, acc[f][m]);
                    acc[f][m] = fmaf(now[f][i].y, x.y, acc[f][m]);
                    acc[f][m] = fmaf(now[f][i].z, x.z, acc[f][m]);
                    acc[f][m] = fmaf(now[f][i].w, x.w, acc[f][m]);
                }
            }
        }
    }
#pragma unroll
    for (int f = 0; f < F; f++)
#pragma unroll
        for (int m = 0; m < MT; m++) {
            const float total = warp_sum(acc[f][m]);
            if (lane == 0) partial[warp][f][m] = total;
        }
    __syncthreads();
    // one thread per (feature of the block, row)
    for (int i = threadIdx.x; i < (8 / split) * F * MT; i += 256) {
        const int m = i % MT, f = (i / MT) % F, group = i / (MT * F);
        const int n = (blockIdx.x * (8 / split) + group) * F + f;
        if (m >= M || n >= N) continue;
        float v = 0.0f;
        for (int s = 0; s < split; s++) v += partial[group * split + s][f][m];
        v += bias ? bias[n] : 0.0f;
        float* o = out + (long)m * ldo + n;
        *o = epilogue == EPI_ADD ? *o + v : activate(epilogue, v);
    }
}

// 32-bit operands, more rows: tiles of BM x 64 by 128 threads, BM / 16 x 8 sums a thread out of 16-byte reads of shared memory
// (a step of K of 128 rows: 64 FMAs for 16 values read), the next step's values and the next 16 entries of K in registers while
// these are multiplied.  Where the tiles are fewer than the SMs a cluster of 2, 4 or 8 blocks shares a tile's K: every
// block leaves its sums in its shared memory, and block r finishes rows r * BM / blocks and up, adding the parts in block order
// (the order is the tile's, never timing).  Scalar FMA.
// 256 rows: 35 us at 768 x 768 (73 as tiles of 64 rows launched early, 41 launched late), 38 at 2,304 x 768.
constexpr int FLOAT_BN = 64, FLOAT_K = 16;
template <int BM>
__global__ void __launch_bounds__(128)
linear_float_tile_kernel(float* __restrict__ out, const float* a, const float* __restrict__ w,
                         const float* __restrict__ bias, int M, int N, int K, long lda, long ldo, int epilogue, int per_block) {
    constexpr int TM = BM / 16, LDA = BM + 4, LDW = FLOAT_BN + 4, LDS = FLOAT_BN + 4;
    constexpr int STAGED = 2 * FLOAT_K * (LDA + LDW), SUMS = BM * LDS;
    __shared__ __align__(16) float staged[STAGED > SUMS ? STAGED : SUMS];     // [buffer][k][row] of a, then of w; the sums at the end
    dependents_may_start();
    wait_for_earlier_kernels();
    const int tid = threadIdx.x, tx = tid & 7, ty = tid >> 3;
    const int m0 = blockIdx.y * BM, n0 = blockIdx.x * FLOAT_BN;
    const int blocks = gridDim.z, rank = blockIdx.z;
    const int k_begin = rank * per_block, k_end = min(K, k_begin + per_block);
    // what this thread copies of 16 entries of K: four of them (a quad) of rows row, row + 32, ...
    const int row = tid >> 2, quad = (tid & 3) * 4;
    constexpr int AR = BM / 32, WR = FLOAT_BN / 32;
    const float4 none = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    float4 ra[AR], rw[WR];
    auto fetch = [&](int k0) {
        const int k = k0 + quad;
#pragma unroll
        for (int i = 0; i < AR; i++) {
            const int r = m0 + row + 32 * i;
            ra[i] = r < M && k < k_end ? *reinterpret_cast<const float4*>(a + (long)r * lda + k) : none;
        }
#pragma unroll
        for (int i = 0; i < WR; i++) {
            const int r = n0 + row + 32 * i;
            rw[i] = r < N && k < k_end ? __ldg(reinterpret_cast<const float4*>(w + (long)r * K + k)) : none;
        }
    };
    auto stage = [&](int buffer) {
        float* as = staged + buffer * FLOAT_K * LDA;
        float* ws = staged + 2 * FLOAT_K * LDA + buffer * FLOAT_K * LDW;
#pragma unroll
        for (int i = 0; i < AR; i++) {
            float* to = as + quad * LDA + row + 32 * i;
            to[0] = ra[i].x; to[LDA] = ra[i].y; to[2 * LDA] = ra[i].z; to[3 * LDA] = ra[i].w;
        }
#pragma unroll
        for (int i = 0; i < WR; i++) {
            float* to = ws + quad * LDW + row + 32 * i;
            to[0] = rw[i].x; to[LDW] = rw[i].y; to[2 * LDW] = rw[i].z; to[3 * LDW] = rw[i].w;
        }
    };
    // a thread's rows: 4 ty .. and (of 128) 64 + 4 ty ..; its columns: 4 tx .. and 32 + 4 tx ..
    float acc[TM][8];
#pragma unroll
    for (int i = 0; i < TM; i++)
#pragma unroll
        for (int j = 0; j < 8; j++) acc[i][j] = 0.0f;
    auto load = [&](int buffer, int kk, float (&x)[TM], float (&y)[8]) {
        const float* as = staged + (buffer * FLOAT_K + kk) * LDA;
        const float* ws = staged + 2 * FLOAT_K * LDA + (buffer * FLOAT_K + kk) * LDW;
#pragma unroll
        for (int i = 0; i < TM / 4; i++) *reinterpret_cast<float4*>(x + 4 * i) = *reinterpret_cast<const float4*>(as + 64 * i + 4 * ty);
#pragma unroll
        for (int j = 0; j < 2; j++) *reinterpret_cast<float4*>(y + 4 * j) = *reinterpret_cast<const float4*>(ws + 32 * j + 4 * tx);
    };
    if (k_begin < k_end) {
        fetch(k_begin);
        stage(0);
    }
    __syncthreads();
    int buffer = 0;
    for (int k0 = k_begin; k0 < k_end; k0 += FLOAT_K) {
        const bool more = k0 + FLOAT_K < k_end;
        if (more) fetch(k0 + FLOAT_K);
        alignas(16) float x[2][TM], y[2][8];
        load(buffer, 0, x[0], y[0]);
#pragma unroll
        for (int kk = 0; kk < FLOAT_K; kk++) {
            if (kk + 1 < FLOAT_K) load(buffer, kk + 1, x[(kk + 1) & 1], y[(kk + 1) & 1]);
#pragma unroll
            for (int i = 0; i < TM; i++)
#pragma unroll
                for (int j = 0; j < 8; j++) acc[i][j] = fmaf(x[kk & 1][i], y[kk & 1][j], acc[i][j]);
        }
        if (more) stage(buffer ^ 1);           // the other buffer: every thread left it before the barrier below, a trip ago
        __syncthreads();
        buffer ^= 1;
    }
    auto finish = [&](int m, int n, float v) {
        if (m >= M || n >= N) return;
        v += bias ? bias[n] : 0.0f;
        float* o = out + (long)m * ldo + n;
        *o = epilogue == EPI_ADD ? *o + v : activate(epilogue, v);
    };
    if (blocks == 1) {
#pragma unroll
        for (int i = 0; i < TM; i++)
#pragma unroll
            for (int j = 0; j < 8; j++) finish(m0 + i / 4 * 64 + 4 * ty + i % 4, n0 + j / 4 * 32 + 4 * tx + j % 4, acc[i][j]);
        return;
    }
#pragma unroll
    for (int i = 0; i < TM; i++)
#pragma unroll
        for (int j = 0; j < 8; j += 4)
            *reinterpret_cast<float4*>(staged + (i / 4 * 64 + 4 * ty + i % 4) * LDS + j / 4 * 32 + 4 * tx) =
                make_float4(acc[i][j], acc[i][j + 1], acc[i][j + 2], acc[i][j + 3]);
    cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
    cluster.sync();
    const int mine = BM / blocks;
    for (int i = tid; i < mine * FLOAT_BN; i += 128) {
        const int r = rank * mine + i / FLOAT_BN, c = i % FLOAT_BN;
        float v = 0.0f;
        for (int b = 0; b < blocks; b++) v += cluster.map_shared_rank(staged, b)[r * LDS + c];
        finish(m0 + r, n0 + c, v);
    }
    cluster.sync();                                                       // no block leaves while another reads its sums
}

template <int BM>
static int launch_float_tiles(float* out, const float* a, const float* w, const float* bias, int M, int N, int K, long lda, long ldo,
                              int epilogue, cudaStream_t s) {
    const dim3 tiles((N + FLOAT_BN - 1) / FLOAT_BN, (M + BM - 1) / BM);
    // blocks that share a tile's K: while they stay within three to an SM and each has 64 entries of K or more
    int blocks = 1;
    while (blocks < 8 && (long)tiles.x * tiles.y * blocks * 2 <= 444 && K >= blocks * 2 * 64) blocks *= 2;
    const int per_block = ((K + blocks - 1) / blocks + FLOAT_K - 1) / FLOAT_K * FLOAT_K;
    return launched(launch_kernel_in_clusters(AFTER_THE_KERNELS_AHEAD, blocks > 1 ? dim3(1, 1, blocks) : dim3(0, 1, 1),
                                              linear_float_tile_kernel<BM>, dim3(tiles.x, tiles.y, blocks), dim3(128), 0, s, out, a, w, bias, M,
                                              N, K, lda, ldo, epilogue, per_block), "linear_float_tile_kernel");
}

template <int MT, int F>
static int launch_float_rows(float* out, const float* a, const float* w, const float* bias, int M, int N, int K, long lda, long ldo,
                             int epilogue, int split, cudaStream_t s) {
    const size_t shared = (size_t)MT * K * sizeof(float);
    if (shared > 40 * 1024) {
        cudaError_t e = cudaFuncSetAttribute(linear_float_rows_kernel<MT, F>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)shared);
        if (e != cudaSuccess) return fail("linear: cannot raise the shared memory limit");
    }
    const int per_block = 8 / split * F;
    return launched(launch_kernel(g_dependent_launch != 0, linear_float_rows_kernel<MT, F>, dim3((N + per_block - 1) / per_block),
                                  dim3(256), shared, s, out, a, w, bias, M, N, K, lda, ldo, epilogue, split),
                    "linear_float_rows_kernel");
}

// Whether the two kernels above take the operands: rows on 16-byte boundaries (K and the stride of `a` multiples of 4).
static bool linear_float_takes(const void* a, const void* w, int K, long lda) {
    return K % 4 == 0 && lda % 4 == 0 && on_16_bytes(a) && on_16_bytes(w);
}

static int launch_linear_float(float* out, const float* a, const float* w, const float* bias, int M, int N, int K, long lda, long ldo,
                               int epilogue, cudaStream_t s) {
    // up to 8 rows that fit 128 KB of shared memory stream the weights; more rows reuse them in tiles
    if (M <= 8 && (size_t)(M <= 1 ? 1 : M <= 2 ? 2 : M <= 4 ? 4 : 8) * K * sizeof(float) <= 128 * 1024) {
        // wide products (a vocabulary) take four features a warp, so that a row read from shared memory serves four; narrow
        // ones share a feature's K among up to four warps, while each still has 128 pieces of 16 bytes
        const bool wide = N >= 16384;
        int split = 1;
        while (!wide && split < 4 && N * split < 3072 && K / 4 >= split * 2 * 64) split *= 2;
#define FLOAT_ROWS(MT) (wide ? launch_float_rows<MT, 4>(out, a, w, bias, M, N, K, lda, ldo, epilogue, 1, s) \
                             : launch_float_rows<MT, 1>(out, a, w, bias, M, N, K, lda, ldo, epilogue, split, s))
        if (M <= 1) return FLOAT_ROWS(1);
        if (M <= 2) return FLOAT_ROWS(2);
        if (M <= 4) return FLOAT_ROWS(4);
        return FLOAT_ROWS(8);
#undef FLOAT_ROWS
    }
    return M <= 64 ? launch_float_tiles<64>(out, a, w, bias, M, N, K, lda, ldo, epilogue, s)
                   : launch_float_tiles<128>(out, a, w, bias, M, N, K, lda, ldo, epilogue, s);
}

template <typename AT, typename WT, typename OT>
static int launch_linear_plain(void* out, const void* a, const void* w, const float* bias, int M, int N, int K,
                               long lda, long ldo, int epilogue, cudaStream_t s) {
    dim3 grid((N + 63) / 64, (M + 63) / 64);
    OT* o = (OT*)out;
    const AT* ap = (const AT*)a;
    const WT* wp = (const WT*)w;
    switch (epilogue) {
    case EPI_STORE: linear_plain_kernel<AT, WT, OT, EPI_STORE><<<grid, 256, 0, s>>>(o, ap, wp, bias, M, N, K, lda, ldo); break;
    case EPI_GELU_TANH: linear_plain_kernel<AT, WT, OT, EPI_GELU_TANH><<<grid, 256, 0, s>>>(o, ap, wp, bias, M, N, K, lda, ldo); break;
    case EPI_GELU_ERF: linear_plain_kernel<AT, WT, OT, EPI_GELU_ERF><<<grid, 256, 0, s>>>(o, ap, wp, bias, M, N, K, lda, ldo); break;
    case EPI_ADD: linear_plain_kernel<AT, WT, OT, EPI_ADD><<<grid, 256, 0, s>>>(o, ap, wp, bias, M, N, K, lda, ldo); break;
    case EPI_RELU_SQ: linear_plain_kernel<AT, WT, OT, EPI_RELU_SQ><<<grid, 256, 0, s>>>(o, ap, wp, bias, M, N, K, lda, ldo); break;
    case EPI_SILU: linear_plain_kernel<AT, WT, OT, EPI_SILU><<<grid, 256, 0, s>>>(o, ap, wp, bias, M, N, K, lda, ldo); break;
    default: return fail("linear: unknown epilogue");
    }
    return check_launch("linear_plain_kernel");
}

// in_dtype: element type of `a` and `w`; out_dtype: element type of `out`
// (EPI_ADD needs a 32-bit `out`).  lda / ldo are row strides in elements.
extern "C" int mllm_plain_linear(void* out, const void* a, const void* w, const float* bias, int M, int N,
                                 int K, long lda, long ldo, int in_dtype, int out_dtype, int epilogue,
                                 void* stream) {
    if (M <= 0 || N <= 0) return 0;
    if (K <= 0) return fail("linear: K must be positive");
    if ((M + 63) / 64 > 65535) return fail("linear: too many rows for one launch");
    if (epilogue == EPI_ADD && out_dtype != DT_F32) return fail("linear: the residual sum is kept in 32-bit");
    cudaStream_t s = (cudaStream_t)stream;
    if (in_dtype == DT_F32 && out_dtype == DT_F32 && linear_float_takes(a, w, K, lda))
        return launch_linear_float((float*)out, (const float*)a, (const float*)w, bias, M, N, K, lda, ldo, epilogue, s);
    if (in_dtype == DT_F32 && out_dtype == DT_F32)
        return launch_linear_plain<float, float, float>(out, a, w, bias, M, N, K, lda, ldo, epilogue, s);
    if (in_dtype == DT_BF16 && out_dtype == DT_BF16)
        return launch_linear_plain<bf16, bf16, bf16>(out, a, w, bias, M, N, K, lda, ldo, epilogue, s);
    if (in_dtype == DT_BF16 && out_dtype == DT_F32)
        return launch_linear_plain<bf16, bf16, float>(out, a, w, bias, M, N, K, lda, ldo, epilogue, s);
    return fail("linear: unsupported combination of element types");
}

// ---------------------------------------------------------------------------
// Store this step's keys and values into their pages.
// pages: [n_pages, page_size, width] per tensor, width = kv_heads * head_size.
// ---------------------------------------------------------------------------
template <typename T>
__global__ void kv_store_kernel(T* __restrict__ k_pages, T* __restrict__ v_pages, const T* __restrict__ k_src,
                                const T* __restrict__ v_src, long ld_src, const int* __restrict__ positions,
                                const int* __restrict__ token_item, const int* __restrict__ block_table,
                                int max_blocks, int page_size, int width) {
    int t = blockIdx.x;
    int p = positions[t];
    int page = block_table[(long)token_item[t] * max_blocks + p / page_size];
    long dst = ((long)page * page_size + (p % page_size)) * width;
    for (int d = threadIdx.x; d < width; d += blockDim.x) {
        k_pages[dst + d] = k_src[(long)t * ld_src + d];
        v_pages[dst + d] = v_src[(long)t * ld_src + d];
    }
}

extern "C" int mllm_plain_kv_store(void* k_pages, void* v_pages, const void* k_src, const void* v_src,
                                   long ld_src, const int* positions, const int* token_item,
                                   const int* block_table, int max_blocks, int page_size, int width,
                                   int n_tokens, int dtype, void* stream) {
    if (n_tokens <= 0) return 0;
    cudaStream_t s = (cudaStream_t)stream;
    int threads = width >= 256 ? 256 : 64;
    if (dtype == DT_F32)
        kv_store_kernel<float><<<n_tokens, threads, 0, s>>>((float*)k_pages, (float*)v_pages, (const float*)k_src,
                                                            (const float*)v_src, ld_src, positions, token_item,
                                                            block_table, max_blocks, page_size, width);
    else if (dtype == DT_BF16)
        kv_store_kernel<bf16><<<n_tokens, threads, 0, s>>>((bf16*)k_pages, (bf16*)v_pages, (const bf16*)k_src,
                                                           (const bf16*)v_src, ld_src, positions, token_item,
                                                           block_table, max_blocks, page_size, width);
    else
        return fail("kv_store: unknown dtype");
    return check_launch("kv_store_kernel");
}

// ---------------------------------------------------------------------------
// Causal attention over the paged cache, one block per (token, head).
// The query at absolute position p sees the keys at positions
// max(0, p - window + 1) .. p of its own request (window <= 0: all of them),
// read from the pages its block table names.  Four warps take the keys in
// turn, each with an online softmax; their states are merged at the end in a
// fixed order, so a token's result does not depend on the rest of the batch.
// ---------------------------------------------------------------------------
constexpr int ATT_PLAIN_MAX_HEAD = 256;

template <typename T>
__global__ void __launch_bounds__(128)
attention_plain_kernel(T* __restrict__ out, long ld_out, const T* __restrict__ q, long ld_q,
                       const T* __restrict__ k_pages, const T* __restrict__ v_pages,
                       const int* __restrict__ block_table, int max_blocks, const int* __restrict__ positions,
                       const int* __restrict__ token_item, int n_heads, int n_kv_heads, int head_size,
                       int page_size, float scale, int window) {
    constexpr int R = ATT_PLAIN_MAX_HEAD / 32;
    int t = blockIdx.x, h = blockIdx.y;
    int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    int p = positions[t];
    const int* bt = block_table + (long)token_item[t] * max_blocks;
    int hk = h / (n_heads / n_kv_heads);
    int kv_width = n_kv_heads * head_size;

    float qr[R], acc[R];
#pragma unroll
    for (int i = 0; i < R; i++) {
        int d = lane + 32 * i;
        qr[i] = d < head_size ? to_f32(q[(long)t * ld_q + (long)h * head_size + d]) : 0.0f;
        acc[i] = 0.0f;
    }
    float m = -INFINITY, l = 0.0f;
    int lo = (window > 0 && p - window + 1 > 0) ? p - window + 1 : 0;
    for (int j = lo + warp; j <= p; j += 4) {
        int page = bt[j / page_size];
        long base = ((long)page * page_size + (j % page_size)) * kv_width + (long)hk * head_size;
        float s = 0.0f;
#pragma unroll
        for (int i = 0; i < R; i++) {
            int d = lane + 32 * i;
            if (d < head_size) s = fmaf(qr[i], to_f32(k_pages[base + d]), s);
        }
        s = warp_sum(s) * scale;
        float m_new = fmaxf(m, s);
        float c = expf(m - m_new);
        float e = expf(s - m_new);
        l = l * c + e;
#pragma unroll
        for (int i = 0; i < R; i++) {
            int d = lane + 32 * i;
            if (d < head_size) acc[i] = acc[i] * c + e * to_f32(v_pages[base + d]);
        }
        m = m_new;
    }

    __shared__ float sm_m[4], sm_l[4];
    __shared__ float sm_acc[4][ATT_PLAIN_MAX_HEAD];
    if (lane == 0) {
        sm_m[warp] = m;
        sm_l[warp] = l;
    }
#pragma unroll
    for (int i = 0; i < R; i++) {
        int d = lane + 32 * i;
        if (d < head_size) sm_acc[warp][d] = acc[i];
    }
    __syncthreads();
    float big = fmaxf(fmaxf(sm_m[0], sm_m[1]), fmaxf(sm_m[2], sm_m[3]));
    float total = 0.0f;
    float wgt[4];
#pragma unroll
    for (int w = 0; w < 4; w++) {
        wgt[w] = sm_m[w] == -INFINITY ? 0.0f : expf(sm_m[w] - big);
        total += sm_l[w] * wgt[w];
    }
    for (int d = threadIdx.x; d < head_size; d += blockDim.x) {
        float o = 0.0f;
#pragma unroll
        for (int w = 0; w < 4; w++) o += sm_acc[w][d] * wgt[w];
        out[(long)t * ld_out + (long)h * head_size + d] = from_f32<T>(o / total);
    }
}

// 32-bit queries, keys and values whose head size is a multiple of 4 up to 128: a lane owns four of the head's entries, LPK
// lanes own a key, and a warp has four keys a lane group in flight before it uses the first (one key at a time, each with its own
// block-table look-up and a reduction over 32 lanes, waited 1.4 us a key: 21 us for 60 keys of 4 tokens).  Eight warps a
// block; their states are merged in warp and group order.
template <int LPK>
__global__ void __launch_bounds__(256)
attention_float_kernel(float* __restrict__ out, long ld_out, const float* __restrict__ q, long ld_q, const float* __restrict__ k_pages,
                       const float* __restrict__ v_pages, const int* __restrict__ block_table, int max_blocks,
                       const int* __restrict__ positions, const int* __restrict__ token_item, int n_heads, int n_kv_heads,
                       int head_size, int page_size, float scale, int window) {
    constexpr int KPW = 32 / LPK, STATES = 8 * KPW, DEEP = 4;
    __shared__ float state_m[STATES], state_l[STATES];
    __shared__ __align__(16) float state_acc[STATES][LPK * 4];
    dependents_may_start();
    wait_for_earlier_kernels();
    q = behind_the_wait(q);
    k_pages = behind_the_wait(k_pages);
    v_pages = behind_the_wait(v_pages);
    const int t = blockIdx.x, h = blockIdx.y;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, sub = lane % LPK, group = lane / LPK;
    const int p = positions[t];
    const int* bt = block_table + (long)token_item[t] * max_blocks;
    const long width = (long)n_kv_heads * head_size, column = (long)(h / (n_heads / n_kv_heads)) * head_size + sub * 4;
    const bool there = sub * 4 < head_size;
    const float4 none = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    const float4 mine = there ? *reinterpret_cast<const float4*>(q + (long)t * ld_q + (long)h * head_size + sub * 4) : none;
    float4 acc = none;
    float m = -INFINITY, l = 0.0f;
    const int lo = (window > 0 && p - window + 1 > 0) ? p - window + 1 : 0;
    // every lane of a warp runs the same trips (the shuffles need all of them)
    for (int base = lo + warp * KPW * DEEP; base <= p; base += STATES * DEEP) {
        float4 k[DEEP], v[DEEP];
        float s[DEEP];
#pragma unroll
        for (int i = 0; i < DEEP; i++) {
            const int j = base + i * KPW + group;
            k[i] = v[i] = none;
            if (j <= p && there) {
                const long at = ((long)bt[j / page_size] * page_size + j % page_size) * width + column;
                k[i] = *reinterpret_cast<const float4*>(k_pages + at);
                v[i] = *reinterpret_cast<const float4*>(v_pages + at);
            }
        }
        float top = m;
#pragma unroll
        for (int i = 0; i < DEEP; i++) {
            float dot = fmaf(mine.x, k[i].x, fmaf(mine.y, k[i].y, fmaf(mine.z, k[i].z, mine.w * k[i].w)));
#pragma unroll
            for (int o = LPK / 2; o > 0; o >>= 1) dot += __shfl_xor_sync(0xffffffffu, dot, o);
            s[i] = base + i * KPW + group <= p ? dot * scale : -INFINITY;
            top = fmaxf(top, s[i]);
        }
        if (top != -INFINITY) {
            const float keep = expf(m - top);
            l *= keep;
            acc.x *= keep; acc.y *= keep; acc.z *= keep; acc.w *= keep;
#pragma unroll
            for (int i = 0; i < DEEP; i++) {
                const float e = expf(s[i] - top);
                l += e;
                acc.x = fmaf(e, v[i].x, acc.x); acc.y = fmaf(e, v[i].y, acc.y);
                acc.z = fmaf(e, v[i].z, acc.z); acc.w = fmaf(e, v[i].w, acc.w);
            }
            m = top;
        }
    }
    const int cell = warp * KPW + group;
    if (sub == 0) {
        state_m[cell] = m;
        state_l[cell] = l;
    }
    *reinterpret_cast<float4*>(&state_acc[cell][sub * 4]) = acc;
    __syncthreads();
    float big = -INFINITY, total = 0.0f;
    for (int c = 0; c < STATES; c++) big = fmaxf(big, state_m[c]);
    for (int c = 0; c < STATES; c++) total += state_m[c] == -INFINITY ? 0.0f : state_l[c] * expf(state_m[c] - big);
    for (int d = threadIdx.x; d < head_size; d += 256) {
        float o = 0.0f;
        for (int c = 0; c < STATES; c++) o += state_m[c] == -INFINITY ? 0.0f : state_acc[c][d] * expf(state_m[c] - big);
        out[(long)t * ld_out + (long)h * head_size + d] = o / total;
    }
}

extern "C" int mllm_plain_attention(void* out, long ld_out, const void* q, long ld_q, const void* k_pages,
                                    const void* v_pages, const int* block_table, int max_blocks,
                                    const int* positions, const int* token_item, int n_tokens, int n_heads,
                                    int n_kv_heads, int head_size, int page_size, float scale, int window,
                                    int dtype, void* stream) {
    if (n_tokens <= 0) return 0;
    if (head_size <= 0 || head_size > ATT_PLAIN_MAX_HEAD) return fail("attention: head size must be in 1..256");
    if (n_kv_heads <= 0 || n_heads % n_kv_heads != 0)
        return fail("attention: the number of heads must be a multiple of the number of key/value heads");
    if (n_heads > 65535) return fail("attention: too many heads for one launch");
    cudaStream_t s = (cudaStream_t)stream;
    dim3 grid(n_tokens, n_heads);
    if (dtype == DT_F32 && head_size % 4 == 0 && head_size <= 128 && ld_q % 4 == 0 && on_16_bytes(q) && on_16_bytes(k_pages) &&
        on_16_bytes(v_pages)) {
#define FLOAT_ATTENTION(LPK)                                                                                                     \
    return launched(launch_kernel(g_dependent_launch != 0, attention_float_kernel<LPK>, grid, dim3(256), 0, s, (float*)out, ld_out, \
                                  (const float*)q, ld_q, (const float*)k_pages, (const float*)v_pages, block_table, max_blocks,  \
                                  positions, token_item, n_heads, n_kv_heads, head_size, page_size, scale, window),              \
                    "attention_float_kernel")
        if (head_size <= 16) FLOAT_ATTENTION(4);
        if (head_size <= 32) FLOAT_ATTENTION(8);
        if (head_size <= 64) FLOAT_ATTENTION(16);
        FLOAT_ATTENTION(32);
#undef FLOAT_ATTENTION
    }
    if (dtype == DT_F32)
        attention_plain_kernel<float><<<grid, 128, 0, s>>>((float*)out, ld_out, (const float*)q, ld_q,
                                                           (const float*)k_pages, (const float*)v_pages, block_table,
                                                           max_blocks, positions, token_item, n_heads, n_kv_heads,
                                                           head_size, page_size, scale, window);
    else if (dtype == DT_BF16)
        attention_plain_kernel<bf16><<<grid, 128, 0, s>>>((bf16*)out, ld_out, (const bf16*)q, ld_q,
                                                          (const bf16*)k_pages, (const bf16*)v_pages, block_table,
                                                          max_blocks, positions, token_item, n_heads, n_kv_heads,
                                                          head_size, page_size, scale, window);
    else
        return fail("attention: unknown dtype");
    return check_launch("attention_plain_kernel");
}

// The current device, for a benchmark's record: name, compute capability, SM count, memory,
// runtime and driver versions (the reference's gpt2_gpu_device_info, engine/src/gpt2_gpu.cu:369-383).
// values: [major, minor, SMs, runtime version, driver version]; memory in bytes.
extern "C" int mllm_plain_device_info(char* name, int name_bytes, int* values, long* memory_bytes) {
    int device = 0;
    cudaDeviceProp properties;
    if (cudaGetDevice(&device) != cudaSuccess || cudaGetDeviceProperties(&properties, device) != cudaSuccess)
        return fail("device_info: no CUDA device");
    snprintf(name, (size_t)name_bytes, "%s", properties.name);
    values[0] = properties.major;
    values[1] = properties.minor;
    values[2] = properties.multiProcessorCount;
    *memory_bytes = (long)properties.totalGlobalMem;
    if (cudaRuntimeGetVersion(&values[3]) != cudaSuccess || cudaDriverGetVersion(&values[4]) != cudaSuccess)
        return fail("device_info: cannot read the versions");
    return 0;
}
