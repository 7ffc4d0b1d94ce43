// Products of up to 64 tokens on mma.sync tiles, out = epilogue(x W^T + bias): part of the library of gemm_tcgen05.cu.
//
// What bounds such a product in a step of single tokens is latency, not its 1 to 20 MB of weights: with a tcgen05 tile of 128
// features there are 6 to 50 tiles, each a chain of barrier set-up, TMA, product, commit, tensor memory, shared memory, two
// cluster barriers and loads from the other CTAs of its cluster.  Here a block takes 16, 32 or 48 features, whose K its eight warps
// share: both operands come straight into the fragments, 16 bytes a lane, the weights through a ring in shared memory that is asked
// for ahead of the wait for the kernels ahead, x from L2 two or four blocks of 32 of K early.  What bounds it then is x's way from L2,
// once a block, and with 64 tokens the products themselves (about 500 multiply-adds a clock and SM in this form); see narrow_plan.
#pragma once

#include "mma_tiles.cuh"

namespace {

constexpr int NARROW_WARPS = 8, NARROW_THREADS = NARROW_WARPS * 32, NARROW_AHEAD = 4, NARROW_PAD = 4;

// Shared memory: the ring of weights, over it (when all are used) the warps' sums; behind them the tokens' slots in the cache pages
// and what the other blocks of the cluster send.
template <int NT, int FT> struct NarrowShared {
    static constexpr int F = FT * 16, M = NT * 8, LD = F + NARROW_PAD;
    static constexpr size_t RING = (size_t)NARROW_AHEAD * 2 * FT * NARROW_THREADS * 16;
    static constexpr size_t SUMS = (size_t)NARROW_WARPS * M * LD * 4;
    static constexpr size_t MAIN = RING > SUMS ? RING : SUMS;
    static constexpr size_t bytes(int splits) { return MAIN + 64 * sizeof(long) + (splits > 1 ? (size_t)(M + 4) * F * 4 : 0); }
};

// NT: tiles of eight tokens, FT: tiles of 16 features a block; blockIdx.y: which NT tiles of tokens.
template <int NT, int FT>
__global__ void __launch_bounds__(NARROW_THREADS, NT * FT <= 6 ? 2 : 1)
narrow_product_kernel(const GemmParams p, const bf16* x, long ldx, const bf16* __restrict__ w) {
    using Shared = NarrowShared<NT, FT>;
    constexpr int F = Shared::F, LD = Shared::LD, HELD = NT <= 4 ? 4 : 2;      // HELD: blocks of x on their way
    extern __shared__ __align__(16) unsigned char smem_raw[];
    uint4* ring = reinterpret_cast<uint4*>(smem_raw);
    float* sums = reinterpret_cast<float*>(smem_raw);                                      // [warp][token][LD]
    long* kv_off = reinterpret_cast<long*>(smem_raw + Shared::MAIN);
    float* sent = reinterpret_cast<float*>(smem_raw + Shared::MAIN + 64 * sizeof(long));   // [rank][own outputs]
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, tq = lane & 3;
    const int rank = p.splits > 1 ? (int)cluster_rank() : 0;
    const int n0 = (int)blockIdx.x / p.splits * F;
    const int t0 = (int)blockIdx.y * NT * 8, M = min(NT * 8, p.M - t0);        // this block's tokens
    const int K = p.K, pieces = K / 8;
    // blocks of 32 of K: this block's share, dealt out to the warps in turn (the warps' 64 bytes a row then lie side by side)
    const int all = (K + 31) / 32, each = (all + p.splits - 1) / p.splits;
    const int begin = rank * each + warp, end = min(all, (rank + 1) * each);
    const bf16* rows[2 * FT];
#pragma unroll
    for (int j = 0; j < 2 * FT; j++) rows[j] = w + (long)min(n0 + j * 8 + g, p.N - 1) * K + tq * 8;
    dependents_may_start();
    if (p.splits > 1) asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");      // (this block runs: others may write to it)
    // a lane copies what it will read itself: no barrier between the copy and the product
    auto ask = [&](int block, int slot) {
        const bool there = block < end && block * 4 + tq < pieces;
#pragma unroll
        for (int j = 0; j < 2 * FT; j++)
            copy_16(ring + (slot * 2 * FT + j) * NARROW_THREADS + threadIdx.x, there ? rows[j] + (long)block * 32 : w, there);
        copies_end();
    };
#pragma unroll
    for (int s = 0; s < NARROW_AHEAD; s++) ask(begin + s * NARROW_WARPS, s);
    wait_for_earlier_kernels();
    x = behind_the_wait(x) + (long)(t0 + g) * ldx + tq * 8;
    uint4 held[HELD][NT];
    auto tokens = [&](int block, uint4 (&v)[NT]) {
        const bool there = block < end && block * 4 + tq < pieces;
#pragma unroll
        for (int t = 0; t < NT; t++)
            v[t] = there && t * 8 + g < M ? *reinterpret_cast<const uint4*>(x + (long)t * 8 * ldx + (long)block * 32)
                                            : make_uint4(0u, 0u, 0u, 0u);
    };
#pragma unroll
    for (int u = 0; u < HELD; u++) tokens(begin + u * NARROW_WARPS, held[u]);
    if (p.k_pages != nullptr && (int)threadIdx.x < M) {
        const int pos = p.positions[t0 + threadIdx.x];
        const int page = p.block_table[(long)p.token_item[t0 + threadIdx.x] * p.max_blocks + pos / p.page_size];
        kv_off[threadIdx.x] = ((long)page * p.page_size + pos % p.page_size) * p.kv_width;
    }
    float acc[FT][NT][4];
#pragma unroll
    for (int f = 0; f < FT; f++)
#pragma unroll
        for (int t = 0; t < NT; t++)
#pragma unroll
            for (int e = 0; e < 4; e++) acc[f][t][e] = 0.0f;
    int slot = 0;
    for (int first = begin; first < end; first += HELD * NARROW_WARPS) {
#pragma unroll
        for (int u = 0; u < HELD; u++) {
            const int block = first + u * NARROW_WARPS;
            if (block >= end) break;
            // one block of 32 of K: the weights are rows g and g + 8 of a tile, its eight entries of K feed two products
            copies_landed<NARROW_AHEAD - 1>();
            const uint4* mine = ring + slot * 2 * FT * NARROW_THREADS + threadIdx.x;
#pragma unroll
            for (int f = 0; f < FT; f++) {
                const uint4 low = mine[2 * f * NARROW_THREADS], high = mine[(2 * f + 1) * NARROW_THREADS];
                const uint32_t even[4] = {low.x, high.x, low.y, high.y}, odd[4] = {low.z, high.z, low.w, high.w};
#pragma unroll
                for (int t = 0; t < NT; t++) mma_tile(acc[f][t], even, held[u][t].x, held[u][t].y);
#pragma unroll
                for (int t = 0; t < NT; t++) mma_tile(acc[f][t], odd, held[u][t].z, held[u][t].w);
            }
            tokens(block + HELD * NARROW_WARPS, held[u]);
            ask(block + NARROW_AHEAD * NARROW_WARPS, slot);
            slot = (slot + 1) % NARROW_AHEAD;
        }
    }
    copies_landed<0>();
    __syncthreads();                                         // every warp's weights are used up: the sums lie over them
#pragma unroll
    for (int f = 0; f < FT; f++)
#pragma unroll
        for (int t = 0; t < NT; t++)
#pragma unroll
            for (int e = 0; e < 4; e++)
                sums[(warp * Shared::M + t * 8 + 2 * tq + (e & 1)) * LD + f * 16 + g + (e >> 1) * 8] = acc[f][t][e];
    __syncthreads();
    auto finish = [&](int t, int r, float v) {
        if (r >= p.N) return;
        if (p.bias != nullptr) v += p.bias[r];
        if (p.k_pages != nullptr && r >= p.q_width) {
            if (r < p.q_width + p.kv_width) p.k_pages[kv_off[t] + r - p.q_width] = __float2bfloat16_rn(v);
            else p.v_pages[kv_off[t] + r - p.q_width - p.kv_width] = __float2bfloat16_rn(v);
            return;
        }
        const long at = (long)(t0 + t) * p.ldo + r;
        // (the residual sum as one addition at the memory: nothing else adds to the element in this launch)
        if (p.epilogue == EPI_ADD) atomicAdd(reinterpret_cast<float*>(p.out) + at, v);
        else if (p.out_f32) reinterpret_cast<float*>(p.out)[at] = v;
        else reinterpret_cast<bf16*>(p.out)[at] = __float2bfloat16_rn(activate(v, p.epilogue));
    };
    auto of_warps = [&](int t, int f) {
        float v = 0.0f;
#pragma unroll
        for (int s = 0; s < NARROW_WARPS; s++) v += sums[(s * Shared::M + t) * LD + f];
        return v;
    };
    if (p.splits <= 1) {
        for (int i = threadIdx.x; i < M * F; i += NARROW_THREADS) finish(i / F, n0 + i % F, of_warps(i / F, i % F));
        return;
    }
    // Token t is finished by the block of rank t % splits: every other block stores its part there (stores wait for no answer),
    // and behind the barrier the parts are added in the ranks' order.
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    const int most = (M + p.splits - 1) / p.splits * F;
    for (int i = threadIdx.x; i < M * F; i += NARROW_THREADS) {
        const int t = i / F, f = i % F, owner = t % p.splits;
        uint32_t to;
        asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(to) : "r"(smem_u32(sent + rank * most + t / p.splits * F + f)), "r"(owner));
        asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(to), "f"(of_warps(t, f)) : "memory");
    }
    cluster_sync();
    for (int i = threadIdx.x; i < most; i += NARROW_THREADS) {
        const int t = i / F * p.splits + rank;
        if (t >= M) continue;
        float v = 0.0f;
        for (int z = 0; z < p.splits; z++) v += sent[z * most + i];
        finish(t, n0 + i % F, v);
    }
}

template <int NT, int FT>
int launch_narrow(const GemmParams& p, const bf16* x, long ldx, const bf16* w, cudaStream_t s) {
    using Shared = NarrowShared<NT, FT>;
    // (at every launch, as the limit is a device's own)
    if (cudaFuncSetAttribute(narrow_product_kernel<NT, FT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)Shared::bytes(2)) != cudaSuccess)
        return fail("gemm: cannot raise the shared memory limit");
    const int tiles = (p.N + Shared::F - 1) / Shared::F;
    return launched(launch_kernel_in_clusters(g_dependent_launch != 0, dim3(p.splits > 1 ? p.splits : 0, 1, 1), narrow_product_kernel<NT, FT>,
                                              dim3(tiles * p.splits, (p.M + NT * 8 - 1) / (NT * 8)), dim3(NARROW_THREADS), Shared::bytes(p.splits), s, p, x, ldx, w),
                    "narrow_product_kernel");
}

// How a product is split: tiles of 16 features a block, blocks that share K, and blocks that share the tokens, as
// 100 * (blocks - 1) + 10 * tiles + blocks; the plan with the least expected time, in us.  Fitted to products of 12 to 64 tokens, 768 to
// 6,400 features and 768 to 6,400 of K, and its rounds of blocks: a block's way in and out, its loop over K (x's way from L2, then the products), blocks that
// wait for others to end, a cluster's exchange, and the weights' way from HBM.
static int narrow_token_tiles(int M) { return M <= 16 ? 2 : M <= 24 ? 3 : M <= 32 ? 4 : M <= 48 ? 6 : 8; }
int narrow_plan(int M, int N, int K, int sms, int* rounds_of_plan) {
    int best = 11;
    double least = -1.0;
    for (int shares = 1; shares <= (M > 16 ? 2 : 1); shares++)
        for (int ft = 1; ft <= 3; ft++)
            for (int splits = 1; splits <= 4; splits *= 2) {
                const int nt = narrow_token_tiles((M + shares - 1) / shares);
                const long blocks = (long)((N + 16 * ft - 1) / (16 * ft)) * splits * shares;
                if (splits > 1 && (K < 512 * splits || blocks > (splits == 2 ? sms : 13 * sms / 16))) continue;
                const int at_once = nt * ft <= 6 ? 2 * sms : sms;
                const long waves = (blocks + at_once - 1) / at_once;
                const double rounds = blocks > sms && waves == 1 ? 1.2 : (double)waves;
                const double loop = (double)K / splits * 1e-3 * (0.45 + 0.07 * nt + (nt > 4 ? 0.25 : 0.0) + 0.1 * ft * nt);
                const double cost = 2.0 + rounds * loop + (double)(waves - 1) + (splits > 1 ? 1.2 : 0.0) + (double)N * K * 2.0 / 6.5e6;
                if (least < 0.0 || cost < least) {
                    least = cost;
                    best = 100 * (shares - 1) + 10 * ft + splits;
                    *rounds_of_plan = (int)waves;
                }
            }
    return best;
}

int launch_narrow_plan(GemmParams p, int plan, const void* x, long ldx, const void* w, cudaStream_t s) {
    const bf16 *xb = (const bf16*)x, *wb = (const bf16*)w;
    const int shares = plan / 100 + 1, ft = plan / 10 % 10, nt = narrow_token_tiles((p.M + shares - 1) / shares);
    p.splits = plan % 10;
    if (p.M > 64 || shares > 2 || ft < 1 || ft > 3 || !(p.splits == 1 || p.splits == 2 || p.splits == 4))
        return fail("gemm: narrow tiles take up to 64 tokens, shared by up to 2 blocks, 16 to 48 features, 1, 2 or 4 blocks along K");
#define NARROW(NT)                                                                                                  \
    (ft == 1 ? launch_narrow<NT, 1>(p, xb, ldx, wb, s) : ft == 2 ? launch_narrow<NT, 2>(p, xb, ldx, wb, s)          \
                                                                 : launch_narrow<NT, 3>(p, xb, ldx, wb, s))
    if (nt == 2) return NARROW(2);
    if (nt == 3) return NARROW(3);
    if (nt == 4) return NARROW(4);
    if (nt == 6) return NARROW(6);
    return NARROW(8);
#undef NARROW
}

}  // namespace
