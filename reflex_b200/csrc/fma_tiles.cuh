// Products of small tiles in shared memory by 32-bit multiply-adds, two an instruction (fma.rn.f32x2: no
// more of them a second than one by one, half as many instructions, whose issue the reads of shared
// memory share).  A thread owns four rows (4 ty ..) by four neighbouring columns (4 tx ..) of a tile, 16
// bytes an access.  Sums of sixteen terms are added up, not one chain of all terms: a chain of 128 is off
// by twice as much as short ones.
#pragma once

#include "common.cuh"

namespace rfx {

// Two 32-bit numbers in a register pair.
typedef unsigned long long Pair;
__device__ __forceinline__ Pair pair_of(float a, float b) {
    Pair p;
    asm("mov.b64 %0, {%1, %2};" : "=l"(p) : "f"(a), "f"(b));
    return p;
}
__device__ __forceinline__ float2 floats_of(Pair p) {
    float2 f;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(f.x), "=f"(f.y) : "l"(p));
    return f;
}
__device__ __forceinline__ void fma2(Pair& d, Pair a, Pair b) { asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b)); }
__device__ __forceinline__ ulonglong2 load_pairs(const float* p) { return *reinterpret_cast<const ulonglong2*>(p); }

// part += x y^T: four numbers by four, pairs along y
__device__ __forceinline__ void outer4(Pair (&part)[4][2], const float4& x, const ulonglong2& y) {
    const float a[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const Pair w = pair_of(a[i], a[i]);
        fma2(part[i][0], w, y.x);
        fma2(part[i][1], w, y.y);
    }
}
// acc += (or, NEG, -=) part
template <bool NEG = false>
__device__ __forceinline__ void add4(float (&acc)[4][4], const Pair (&part)[4][2]) {
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            const float2 p = floats_of(part[i][j]);
            acc[i][2 * j] += NEG ? -p.x : p.x;
            acc[i][2 * j + 1] += NEG ? -p.y : p.y;
        }
}

// acc += a b^T over n16 sixteens, both read along their rows: the thread's rows of `a` `a_apart` floats from
// one another, its columns' rows of `b` `b_apart` (eight threads' rows side by side, an odd number of 16
// bytes each, meet all banks).  Even and odd terms in sums of their own, sixteen terms each.
template <int COLS>
__device__ __forceinline__ void product_along(float (&acc)[4][COLS], const float* a, int a_apart, const float* b,
                                              int b_apart, int n16) {
    for (int s = 0; s < n16; s += 2) {
        Pair part[4][COLS] = {};
        for (int t = min(2, n16 - s); t > 0; --t, a += 16, b += 16) {
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                ulonglong2 x[4], y[COLS];
#pragma unroll
                for (int i = 0; i < 4; ++i) x[i] = load_pairs(a + i * a_apart + 4 * q);
#pragma unroll
                for (int j = 0; j < COLS; ++j) y[j] = load_pairs(b + j * b_apart + 4 * q);
#pragma unroll
                for (int i = 0; i < 4; ++i)
#pragma unroll
                    for (int j = 0; j < COLS; ++j) {
                        fma2(part[i][j], x[i].x, y[j].x);
                        fma2(part[i][j], x[i].y, y[j].y);
                    }
            }
        }
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < COLS; ++j) {
                const float2 p = floats_of(part[i][j]);
                acc[i][j] += p.x + p.y;
            }
    }
}

// acc += w v for the rows 4 ty .. 4 ty + 3 of w and v's rows s no later than each (STRICT: before each)
// alone: a later row's v is never multiplied, so what is not finite there does not reach an earlier
// result.  `w` the thread's first row, the others `apart` floats from one another, `v` its first column.
template <bool STRICT, bool NEG = false>
__device__ __forceinline__ void product_below(float (&acc)[4][4], const float* w, int apart, const float* v, int vld, int ty) {
    for (int b0 = 0; b0 <= ty; b0 += 4) {  // fours of rows, sixteen of them a sum
        Pair part[4][2] = {};
        for (int b = b0; b < min(b0 + 4, ty); ++b, w += 4, v += 4 * vld) {
            float4 x[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) x[i] = load4(w + i * apart);
            outer4(part, make_float4(x[0].x, x[1].x, x[2].x, x[3].x), load_pairs(v));
            outer4(part, make_float4(x[0].y, x[1].y, x[2].y, x[3].y), load_pairs(v + vld));
            outer4(part, make_float4(x[0].z, x[1].z, x[2].z, x[3].z), load_pairs(v + 2 * vld));
            outer4(part, make_float4(x[0].w, x[1].w, x[2].w, x[3].w), load_pairs(v + 3 * vld));
        }
        if (ty < b0 + 4) {  // the rows' own four
#pragma unroll
            for (int s = 0; s < 4; ++s) {
                const ulonglong2 y = load_pairs(v + s * vld);
#pragma unroll
                for (int i = s + STRICT; i < 4; ++i) {
                    const float x = w[i * apart + s];
                    const Pair xx = pair_of(x, x);
                    fma2(part[i][0], xx, y.x);
                    fma2(part[i][1], xx, y.y);
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
        Pair part[2][2][4] = {};  // pairs along the left columns
#pragma unroll 4
        for (int s = 0; s < 16; ++s, a += ald, b += bld) {
            const float4 y = load4(b);
            const ulonglong2 x[2] = {load_pairs(a), load_pairs(a + second)};
            const Pair yy[4] = {pair_of(y.x, y.x), pair_of(y.y, y.y), pair_of(y.z, y.z), pair_of(y.w, y.w)};
#pragma unroll
            for (int t = 0; t < 2; ++t)
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    fma2(part[t][0][j], x[t].x, yy[j]);
                    fma2(part[t][1][j], x[t].y, yy[j]);
                }
        }
#pragma unroll
        for (int t = 0; t < 2; ++t)
#pragma unroll
            for (int i = 0; i < 2; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const float2 p = floats_of(part[t][i][j]);
                    acc[t][2 * i][j] += NEG ? -p.x : p.x;
                    acc[t][2 * i + 1][j] += NEG ? -p.y : p.y;
                }
    }
}

}  // namespace rfx
