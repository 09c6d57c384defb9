// 32-bit products on the tcgen05 tensor cores by operands split in three: x = h + m + l, bfloat16 each,
// exactly (24 bits as 6, 8 and 8, rounded to nearest, so that the parts' signs vary and give the other two).  All
// products but l l, which is 2^-30 of the whole: h h in sums of two or three steps, the others in one or two more.
//
// The tensor core cuts every step of a sum off instead of rounding it.  A product of six bits by six takes twelve, so
// a sum of two or three steps of terms of like size fits 24 bits and next to nothing is cut off it, and what is cut
// off the others is 2^-6 of that; sums that 32 bits hold come out exact.  (With h of eight bits about half a unit in
// the last place went at every step; an average of that given back made 1.0 of one live term 1.0000001.)
// The state-space recurrence of 64 x 128 and the mLSTM of 128 x 256, 331 rows, 2-norm error against 64 bits, and by
// multiply-adds in chains of sixteen:
//                                   results                                    memories
//   normal numbers                  8.9e-8 and 1.06e-7   (1.35e-7, 1.40e-7)    7.7e-8 and 1.13e-7   (9.5e-8, 1.25e-7)
//   of one sign                     4.6e-8 and 8.0e-8    (5.6e-8, 8.5e-8)      4.7e-8 and 8.6e-8    (5.5e-8, 9.7e-8)
//   decays of e^-8 a row and less   6.4e-8 and 6.5e-8    (1.05e-7, 9.7e-8)     5.0e-8 and 8.1e-8    (4.9e-8, 6.5e-8)
//   e^(2 normal) times normal       1.8e-7 and 1.6e-7    (1.6e-7, 1.35e-7)     7.9e-8 and 1.13e-7   (9.3e-8, 1.31e-7)
// (Where one term outweighs all others and those are 2^-12 of it, a cut is half a unit on average and shows.)
//
// Operands lie in shared memory as tiles of 64 rows of 64 numbers, 128 bytes a row and part with the 128-byte
// swizzle, three parts one behind the other (24 KB), each on a 1,024-byte boundary.  A tile is K-major or
// MN-major as the descriptor says.
//
// "Odd" numbers, not finite or so large (2^60) that a sum of products might not be, count as zero here; who makes a
// tile learns that it held some and adds their products by multiply-adds (`is_odd`).  Of numbers below 2^-110 the
// last bits are beyond bfloat16's range.
#pragma once

#include "common.cuh"
#include "sm100.cuh"

namespace rfx {
namespace split3 {

constexpr int PART = 64 * 128, TILE = 3 * PART;  // bytes

__device__ __forceinline__ bool is_odd(float x) { return !(fabsf(x) < 0x1p60f); }
// h is rounded to six bits: half a unit is added, and bfloat16's last two bits go (of two neighbours at once)
constexpr uint32_t H_HALF = 1u << 17, H_MASK = 0xfffcfffcu;

// What one of THREADS threads makes of a tile: rows tid / 8 and THREADS / 8 further, columns 8 (tid % 8) on.
template <int THREADS>
struct Own {
    static constexpr int ROWS = 512 / THREADS;
    float x[ROWS][8];
    static __device__ __forceinline__ int row(int i) { return (threadIdx.x >> 3) + THREADS / 8 * i; }
    static __device__ __forceinline__ int col() { return 8 * (threadIdx.x & 7); }
    // from 32-bit rows `ld` apart; rows from `rows` on and columns from `cols` (in fours) on as zeros
    __device__ __forceinline__ void load(const float* src, size_t ld, int rows, int cols) {
#pragma unroll
        for (int i = 0; i < ROWS; ++i) {
            const float* s = src + (size_t)row(i) * ld + col();
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                if (row(i) < rows && col() + 4 * j < cols) v = load4(s + 4 * j);
                float* to = x[i] + 4 * j;
                to[0] = v.x; to[1] = v.y; to[2] = v.z; to[3] = v.w;
            }
        }
    }
    __device__ __forceinline__ bool put(char* tile) const;  // true if some were odd
};

__device__ __forceinline__ uint32_t pack(float a, float b) {
    const __nv_bfloat162 t = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<const uint32_t*>(&t);
}
// the pair's rounded values taken off, and the rest rounded in turn
__device__ __forceinline__ uint32_t rest(float& a, float& b, uint32_t part) {
    a -= __uint_as_float(part << 16);
    b -= __uint_as_float(part & 0xffff0000u);
    return pack(a, b);
}
// the larger size; a NaN stays
__device__ __forceinline__ float larger(float a, float b) {
    float r;
    asm("max.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(fabsf(b)));
    return r;
}
// eight numbers into a tile's three parts at row r, 16-byte place c; true if some were odd
__device__ __forceinline__ bool put8(const float* in, char* tile, int r, int c) {
    float x[8], top = 0.0f;
    uint32_t h[4];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        x[i] = in[i];
        top = larger(top, x[i]);
    }
    const bool odd = is_odd(top);
    if (odd)
#pragma unroll
        for (int i = 0; i < 8; ++i) x[i] = is_odd(x[i]) ? 0.0f : x[i];
#pragma unroll
    for (int i = 0; i < 4; ++i)
        h[i] = __byte_perm(__float_as_uint(x[2 * i]) + H_HALF, __float_as_uint(x[2 * i + 1]) + H_HALF, 0x7632) & H_MASK;
    char* to = tile + r * 128 + ((c ^ (r & 7)) << 4);
    *reinterpret_cast<uint4*>(to) = make_uint4(h[0], h[1], h[2], h[3]);
#pragma unroll
    for (int p = 1; p < 3; ++p) {
#pragma unroll
        for (int i = 0; i < 4; ++i) h[i] = rest(x[2 * i], x[2 * i + 1], h[i]);
        *reinterpret_cast<uint4*>(to + p * PART) = make_uint4(h[0], h[1], h[2], h[3]);
    }
    return odd;
}
template <int THREADS>
__device__ __forceinline__ bool Own<THREADS>::put(char* tile) const {
    bool odd = false;
#pragma unroll
    for (int i = 0; i < ROWS; ++i) odd |= put8(x[i], tile, row(i), threadIdx.x & 7);
    return odd;
}
// what the threads wrote, for the tensor core; before the barrier that its issuing thread passes
__device__ __forceinline__ void tiles_written() {
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    sm100::tc_fence_before_sync();
}

// Descriptors of a tile's first part and first sixteen; of the part after it, of the sixteen after it (within a
// tile) and of the next tile, in 16 bytes.
__device__ __forceinline__ uint64_t k_major(uint32_t tile) { return sm100::umma_desc_k_sw128(tile); }
// `block`: from 64 elements along MN to the next (a tile further, or a part)
__device__ __forceinline__ uint64_t mn_major(uint32_t tile, int block) {
    return (uint64_t)((tile & 0x3FFFF) >> 4) | (uint64_t)(block >> 4) << 16 | (uint64_t)(1024 >> 4) << 32 |
           (uint64_t)1 << 46 | (uint64_t)2 << 61;
}
constexpr int NEXT_PART = PART >> 4, NEXT_TILE = TILE >> 4, K_STEP = 2, MN_STEP = 16 * 128 >> 4;
constexpr uint32_t A_MN = 1u << 15, B_MN = 1u << 16;  // of the instruction's descriptor

// Products of a left side of 64 or 128 rows with a right side of 64 over up to eight `steps` of sixteen, four a tile,
// by one thread.  A left row is a lane of tensor memory; from column `to` on the h parts' sums, two steps each (three
// where there are more than six), then SMALL (one or two) sums of all other products, 64 columns each; with two an
// instruction takes two of the right side's parts, which lie one behind the other.  (Of 64 rows too products are made
// as of 128: what lies behind a part gives lanes 64 on, which are left alone.)
__host__ __device__ constexpr int steps_a_set(int steps) { return steps > 6 ? 3 : 2; }
__host__ __device__ constexpr int sets_of(int steps) { return (steps + steps_a_set(steps) - 1) / steps_a_set(steps); }
template <int SMALL, int A_STEP, int B_STEP>
__device__ __forceinline__ void issue(uint32_t to, uint32_t majors, int steps, uint64_t a, uint64_t b) {
    const uint32_t one = sm100::umma_idesc_bf16(128, 64) | majors, two = sm100::umma_idesc_bf16(128, 128) | majors;
    const uint32_t small = to + 64 * sets_of(steps);
    const int every = steps_a_set(steps);
    int done = 0;  // steps of the set
    for (int k0 = 0; k0 < steps; k0 += 4, a += NEXT_TILE, b += NEXT_TILE) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            if (k0 + i >= steps) break;
            const uint64_t ah = a + i * A_STEP, am = ah + NEXT_PART, al = am + NEXT_PART;
            const uint64_t bh = b + i * B_STEP, bm = bh + NEXT_PART, bl = bm + NEXT_PART;
            const uint32_t add = k0 + i > 0;
            if (SMALL == 2) {
                sm100::umma_bf16(small, ah, bm, two, add);  // h [m l]
                sm100::umma_bf16(small, am, bm, two, 1);    // m [m l]
                sm100::umma_bf16(small, al, bh, two, 1);    // l [h m]
            } else {
                sm100::umma_bf16(small, am, bl, one, add);
                sm100::umma_bf16(small, al, bm, one, 1);
                sm100::umma_bf16(small, ah, bl, one, 1);
                sm100::umma_bf16(small, al, bh, one, 1);
                sm100::umma_bf16(small, am, bm, one, 1);
                sm100::umma_bf16(small, ah, bm, one, 1);
            }
            sm100::umma_bf16(small, am, bh, one, 1);
            if (done == every) {
                done = 0;
                to += 64;
            }
            sm100::umma_bf16(to, ah, bh, one, done++ > 0);
        }
    }
}

// Eight columns of the thread's lane of what these left from `at` on.
template <int SMALL>
__device__ __forceinline__ void sums_of(float (&y)[8], uint32_t at, int steps) {
    uint32_t h[8], r[8], r2[8];
    const uint32_t small = at + 64 * sets_of(steps);
    __syncwarp();  // (the warp's lanes load together, and what came before may have parted them)
    sm100::tmem_ld_8_nowait(small, r);
    if (SMALL == 2) sm100::tmem_ld_8_nowait(small + 64, r2);
    sm100::tmem_ld_8_nowait(at, h);
    sm100::tmem_ld_wait_8(h);
    sm100::tmem_loaded_8(r);
    if (SMALL == 2) sm100::tmem_loaded_8(r2);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        const float s = __uint_as_float(r[j]);
        y[j] = __uint_as_float(h[j]) + (SMALL == 2 ? s + __uint_as_float(r2[j]) : s);
    }
    for (at += 64; at != small; at += 64) {
        sm100::tmem_ld_8_nowait(at, h);
        sm100::tmem_ld_wait_8(h);
#pragma unroll
        for (int j = 0; j < 8; ++j) y[j] += __uint_as_float(h[j]);
    }
}

}  // namespace split3
}  // namespace rfx
