// 32-bit products on the tensor cores by operands split in two: x = hi + lo, a leading and a
// trailing part of 11 bits each (exact up to 2^-22), and hi hi + hi lo + lo hi with 32-bit sums:
// 32-bit products up to about 2^-21 of their size.
//
// Fragments are those of mma.sync m16n8k8.  The eight k places of a step are taken in the order
// (0, 2, 4, 6, 1, 3, 5, 7), the same for both operands, which changes no sum's terms: thread j of
// a row's four then holds the neighbouring elements 2 j and 2 j + 1 (one 8-byte load), and an
// accumulator tile's registers are the left operand of a next product.
#pragma once

#include <stdint.h>

namespace rfx {

struct Split {
    uint32_t hi, lo;
};
__device__ __forceinline__ Split split(float x) {
    const uint32_t h = __float_as_uint(x) & 0xffffe000u;
    return {h, __float_as_uint(x - __uint_as_float(h))};
}
__device__ __forceinline__ void mma_tf32(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm(
        "mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
        "{%0, %1, %2, %3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// The left operand of a k-step, split.
struct Left {
    uint32_t hi[4], lo[4];
};
// from elements (row, k) = (l4, 2 j), (l4 + 8, 2 j), (l4, 2 j + 1), (l4 + 8, 2 j + 1)
__device__ __forceinline__ Left left_from(float a, float b, float c, float d) {
    Left l;
    const float t[4] = {a, b, c, d};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const Split s = split(t[i]);
        l.hi[i] = s.hi;
        l.lo[i] = s.lo;
    }
    return l;
}
// from an accumulator tile (columns 2 j and 2 j + 1 are its k places)
__device__ __forceinline__ Left left_of(const float (&t)[4]) { return left_from(t[0], t[2], t[1], t[3]); }
// d[n] += a b[n]^T for N right operands, pass by pass so that the products of different n
// follow one another, not those of one sum.
template <int N>
__device__ __forceinline__ void product3(float (&d)[N][4], const Left& a, const float2 (&b)[N]) {
    Split x[N], y[N];
#pragma unroll
    for (int n = 0; n < N; ++n) {
        x[n] = split(b[n].x);
        y[n] = split(b[n].y);
    }
#pragma unroll
    for (int n = 0; n < N; ++n) mma_tf32(d[n], a.lo, x[n].hi, y[n].hi);
#pragma unroll
    for (int n = 0; n < N; ++n) mma_tf32(d[n], a.hi, x[n].lo, y[n].lo);
#pragma unroll
    for (int n = 0; n < N; ++n) mma_tf32(d[n], a.hi, x[n].hi, y[n].hi);
}

}  // namespace rfx
