// Pieces of attention kernels on mma.sync m16n8k16 tiles: operands from shared memory, asynchronous copies into it, and a
// 32-bit operand as three bfloat16 terms.
#pragma once

#include "common.cuh"

// Four 8 x 8 blocks of 16-bit entries; lane l names row l % 8 of block l / 8.
__device__ __forceinline__ void load_blocks(uint32_t (&r)[4], const void* row) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"((uint32_t)__cvta_generic_to_shared(row))
                 : "memory");
}
__device__ __forceinline__ void load_blocks_turned(uint32_t (&r)[4], const void* row) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"((uint32_t)__cvta_generic_to_shared(row))
                 : "memory");
}

__device__ __forceinline__ void mma_tile(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    mma_bf16_16816(c[0], c[1], c[2], c[3], a[0], a[1], a[2], a[3], b0, b1);
}

// 16 bytes to shared memory, zeros where there is nothing to copy.
__device__ __forceinline__ void copy_16(void* to, const void* from, bool there) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(to)), "l"(from),
                 "r"(there ? 16 : 0)
                 : "memory");
}
__device__ __forceinline__ void copies_end() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int LEFT> __device__ __forceinline__ void copies_landed() { asm volatile("cp.async.wait_group %0;" ::"n"(LEFT) : "memory"); }

// Two 32-bit numbers as three pairs of bfloat16 whose sums they are: 8 bits of the significand a term, all 24 in three.  A
// product of such an operand with a bfloat16 one is three products with 32-bit sums, and rounds where those sums do.
// The terms are cut off, not rounded, so that they have the number's sign, and a term is 2^-126 rather than zero where the number
// is not: times an infinity all three are the infinity that the number times it is (with a rounded term of the other sign, or
// a zero, their sum would be no number), and times anything else 2^-126 is nothing beside the first term.
__device__ __forceinline__ uint32_t upper_halves(float low, float high) { return __byte_perm(__float_as_uint(low), __float_as_uint(high), 0x7632); }
__device__ __forceinline__ float upper_half(float x) { return __uint_as_float(__float_as_uint(x) & 0xffff0000u); }
__device__ __forceinline__ void three_terms(float x, float y, uint32_t& first, uint32_t& second, uint32_t& third) {
    constexpr float LEAST = 1.1754943508222875e-38f;                      // 2^-126
    const float least_x = fminf(fabsf(x), LEAST), least_y = fminf(fabsf(y), LEAST);
    first = upper_halves(x, y);
    // (of an infinity nothing is left that is a number: fmaxf takes the other)
    const float x2 = x - upper_half(x), y2 = y - upper_half(y);
    second = upper_halves(copysignf(fmaxf(fabsf(upper_half(x2)), least_x), x), copysignf(fmaxf(fabsf(upper_half(y2)), least_y), y));
    const float x3 = x2 - upper_half(x2), y3 = y2 - upper_half(y2);
    third = upper_halves(copysignf(fmaxf(fabsf(x3), least_x), x), copysignf(fmaxf(fabsf(y3), least_y), y));
}
// The same for numbers that are not negative (an attention's weights).
__device__ __forceinline__ void three_weight_terms(float x, float y, uint32_t& first, uint32_t& second, uint32_t& third) {
    constexpr float LEAST = 1.1754943508222875e-38f;
    const float least_x = fminf(x, LEAST), least_y = fminf(y, LEAST);
    first = upper_halves(x, y);
    const float x2 = x - upper_half(x), y2 = y - upper_half(y);
    second = upper_halves(fmaxf(upper_half(x2), least_x), fmaxf(upper_half(y2), least_y));
    third = upper_halves(fmaxf(x2 - upper_half(x2), least_x), fmaxf(y2 - upper_half(y2), least_y));
}

// The accumulators of two tiles, 16 rows by 16, as the first operand of the next product.
__device__ __forceinline__ void terms_of(uint32_t (&a)[3][4], const float (&x)[4], const float (&y)[4]) {
    three_terms(x[0], x[1], a[0][0], a[1][0], a[2][0]);
    three_terms(x[2], x[3], a[0][1], a[1][1], a[2][1]);
    three_terms(y[0], y[1], a[0][2], a[1][2], a[2][2]);
    three_terms(y[2], y[3], a[0][3], a[1][3], a[2][3]);
}

// A tile's sum is cut off at 24 bits when it is added to what the accumulators held: over a long row of products that adds up.
// The product by itself, added with a rounded addition, keeps a sum as near as a chain of FMAs does.
__device__ __forceinline__ void mma_added(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    float x[4];
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%10, %10, %10, %10};"
        : "=f"(x[0]), "=f"(x[1]), "=f"(x[2]), "=f"(x[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(0.0f));
#pragma unroll
    for (int e = 0; e < 4; e++) c[e] += x[e];
}

__device__ __forceinline__ void weight_terms_of(uint32_t (&a)[3][4], const float (&x)[4], const float (&y)[4]) {
    three_weight_terms(x[0], x[1], a[0][0], a[1][0], a[2][0]);
    three_weight_terms(x[2], x[3], a[0][1], a[1][1], a[2][1]);
    three_weight_terms(y[0], y[1], a[0][2], a[1][2], a[2][2]);
    three_weight_terms(y[2], y[3], a[0][3], a[1][3], a[2][3]);
}

// x = the weights of 16 rows and 32 keys, as three terms, times two tiles of eight value columns: the small terms first.
__device__ __forceinline__ void weighted_rows(float (&x)[2][4], const uint32_t (&a)[2][3][4], const uint32_t (&b)[2][4]) {
#pragma unroll
    for (int e = 0; e < 8; e++) x[e / 4][e % 4] = 0.0f;
#pragma unroll
    for (int term = 2; term >= 0; term--)
#pragma unroll
        for (int k = 0; k < 2; k++) {
            mma_tile(x[0], a[k][term], b[k][0], b[k][1]);
            mma_tile(x[1], a[k][term], b[k][2], b[k][3]);
        }
}
