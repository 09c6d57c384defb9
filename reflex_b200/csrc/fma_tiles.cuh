// Products of small tiles in shared memory by 32-bit multiply-adds.  A thread owns four rows (4 ty ..) by
// four neighbouring columns (4 tx ..) of a tile, 16 bytes an access.  Sums of sixteen terms are added
// up, not one chain of all terms: a chain of 128 is off by twice as much as short ones.
#pragma once

#include "common.cuh"

namespace rfx {

__device__ __forceinline__ void outer4(float (&acc)[4][4], const float4& a, const float4& b) {
    const float x[4] = {a.x, a.y, a.z, a.w}, y[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(x[i], y[j], acc[i][j]);
}
// acc += (or, NEG, -=) part
template <bool NEG = false>
__device__ __forceinline__ void add4(float (&acc)[4][4], const float (&part)[4][4]) {
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] += NEG ? -part[i][j] : part[i][j];
}

// acc += a b^T over n16 sixteens, both read along their rows: `a` the thread's first row, its columns'
// rows `apart` floats from one another from `b` on (eight threads' rows side by side, an odd number of
// 16 bytes each, meet all banks).
template <int COLS>
__device__ __forceinline__ void product_along(float (&acc)[4][COLS], const float* a, int ald, const float* b, int apart,
                                              int n16) {
    for (int s = 0; s < n16; ++s, a += 16, b += 16) {
        float part[4][COLS] = {};
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            float4 x[4], y[COLS];
#pragma unroll
            for (int i = 0; i < 4; ++i) x[i] = load4(a + i * ald + 4 * q);
#pragma unroll
            for (int j = 0; j < COLS; ++j) y[j] = load4(b + j * apart + 4 * q);
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < COLS; ++j) {
                    part[i][j] = fmaf(x[i].x, y[j].x, part[i][j]);
                    part[i][j] = fmaf(x[i].y, y[j].y, part[i][j]);
                    part[i][j] = fmaf(x[i].z, y[j].z, part[i][j]);
                    part[i][j] = fmaf(x[i].w, y[j].w, part[i][j]);
                }
        }
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < COLS; ++j) acc[i][j] += part[i][j];
    }
}

// acc += w v for the rows 4 ty .. 4 ty + 3 of w and v's rows s no later than each (STRICT: before each)
// alone: a later row's v is never multiplied, so what is not finite there does not reach an earlier
// result.  `w` the thread's first row, `v` its first column.
template <bool STRICT, bool NEG = false>
__device__ __forceinline__ void product_below(float (&acc)[4][4], const float* w, int wld, const float* v, int vld, int ty) {
    for (int b0 = 0; b0 <= ty; b0 += 4) {  // fours of rows, sixteen of them a sum
        float part[4][4] = {};
        for (int b = b0; b < min(b0 + 4, ty); ++b, w += 4, v += 4 * vld) {
            float4 x[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) x[i] = load4(w + i * wld);
            outer4(part, make_float4(x[0].x, x[1].x, x[2].x, x[3].x), load4(v));
            outer4(part, make_float4(x[0].y, x[1].y, x[2].y, x[3].y), load4(v + vld));
            outer4(part, make_float4(x[0].z, x[1].z, x[2].z, x[3].z), load4(v + 2 * vld));
            outer4(part, make_float4(x[0].w, x[1].w, x[2].w, x[3].w), load4(v + 3 * vld));
        }
        if (ty < b0 + 4) {  // the rows' own four
#pragma unroll
            for (int s = 0; s < 4; ++s) {
                const float4 y = load4(v + s * vld);
#pragma unroll
                for (int i = s + STRICT; i < 4; ++i) {
                    const float x = w[i * wld + s];
                    part[i][0] = fmaf(x, y.x, part[i][0]);
                    part[i][1] = fmaf(x, y.y, part[i][1]);
                    part[i][2] = fmaf(x, y.z, part[i][2]);
                    part[i][3] = fmaf(x, y.w, part[i][3]);
                }
            }
        }
        add4<NEG>(acc, part);
    }
}

// acc += (NEG: -=) a^T b over `rows` rows (a multiple of sixteen), both read down the rows: left columns
// 4 ty .. and `second` further, right columns 4 tx ..
template <bool NEG = false>
__device__ __forceinline__ void product_down(float (&acc)[2][4][4], const float* a, int ald, int second, const float* b,
                                             int bld, int rows) {
    for (int s0 = 0; s0 < rows; s0 += 16) {
        float part[2][4][4] = {};
#pragma unroll 4
        for (int s = 0; s < 16; ++s, a += ald, b += bld) {
            const float4 y = load4(b);
            outer4(part[0], load4(a), y);
            outer4(part[1], load4(a + second), y);
        }
        add4<NEG>(acc[0], part[0]);
        add4<NEG>(acc[1], part[1]);
    }
}

}  // namespace rfx
