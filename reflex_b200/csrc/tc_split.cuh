// 32-bit products on the tcgen05 tensor cores by operands split in three: x = h + m + l, bfloat16 each,
// exactly (24 bits of 8 each, rounded to nearest, so that the parts' signs vary), and of the nine products the
// six that 32 bits can see: h h in one sum, h m + m h + h l + l h + m m in another.  The tensor core cuts
// every step of a sum off instead of rounding it; two sums keep that out of the result, since the second is
// 2^-8 of the first and the first takes 16-bit products whose sum of sixteen mostly needs no more than 24 bits.
// 2-norm error of products of normal numbers against 64 bits, 64 terms: 5.1e-8, 5.4e-8 and 7.0e-8 with the
// first sum begun anew every 16, 32 and 64 terms, of which the cuts' common part (CUT, given back) is 1.2e-8,
// 2.5e-8 and 4.9e-8; 3.9e-7 with all six products in one sum; 32-bit multiply-adds in chains of sixteen 8.4e-8.
//
// Operands lie in shared memory as tiles of 64 rows of 64 numbers, 128 bytes a row and part with the 128-byte
// swizzle, three parts one behind the other (24 KB), each on a 1,024-byte boundary.  A tile is K-major or
// MN-major as the descriptor says.
//
// What three parts cannot hold, "odd" numbers (not finite, or so large that bfloat16 is not), counts as zero
// here; who makes a tile learns that it held some and adds their products by multiply-adds (`is_odd`).
#pragma once

#include "common.cuh"
#include "sm100.cuh"

namespace rfx {
namespace split3 {

// What the cuts take off a sum of the h parts a step, of its size: on average 1.2e-8 where terms are of either
// sign, 1.6e-8 to 2.5e-8 where they are not or fall off.  Who takes a sum adds so much back.
constexpr float CUT = 1.5e-8f;

constexpr int PART = 64 * 128, TILE = 3 * PART;  // bytes

// what bfloat16 rounds to an exponent of all ones
__device__ __forceinline__ bool is_odd(float x) { return (__float_as_uint(x) & 0x7fffffffu) >= 0x7f7f8000u; }

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
// eight numbers into a tile's three parts at row r, 16-byte place c; true if some were odd
__device__ __forceinline__ bool put8(const float* in, char* tile, int r, int c) {
    float x[8];
    uint32_t h[4], top = 0;
#pragma unroll
    for (int i = 0; i < 8; ++i) x[i] = in[i];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        h[i] = pack(x[2 * i], x[2 * i + 1]);
        top |= (h[i] & 0x7f807f80u) + 0x00800080u;  // an exponent of all ones runs over
    }
    const bool odd = (top & 0x80008000u) != 0;
    if (odd) {
#pragma unroll
        for (int i = 0; i < 8; ++i) x[i] = is_odd(x[i]) ? 0.0f : x[i];
#pragma unroll
        for (int i = 0; i < 4; ++i) h[i] = pack(x[2 * i], x[2 * i + 1]);
    }
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

// Products with a right side of 64 over `steps` sixteens, four a tile.  In tensor memory from `to` on, 64 columns
// each: the h parts' sums, EVERY steps each; two sums of small products.  By one thread.  B's parts lie one
// behind the other, so that one instruction takes two of them (N = 128).
template <int EVERY>
__host__ __device__ constexpr int sets(int steps) { return (steps + EVERY - 1) / EVERY; }
// A has 128 rows: a lane's result is all of its sums.
template <int EVERY, int A_STEP, int B_STEP>
__device__ __forceinline__ void issue128(uint32_t to, uint32_t majors, int steps, uint64_t a, uint64_t b) {
    const uint32_t one = sm100::umma_idesc_bf16(128, 64) | majors, two = sm100::umma_idesc_bf16(128, 128) | majors;
    const uint32_t small = to + 64 * sets<EVERY>(steps);
    for (int k0 = 0; k0 < steps; k0 += 4, a += NEXT_TILE, b += NEXT_TILE) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int k = k0 + i;
            if (k >= steps) break;
            const uint64_t ah = a + i * A_STEP, bh = b + i * B_STEP;
            sm100::umma_bf16(small, ah, bh + NEXT_PART, two, k > 0);             // h [m l]
            sm100::umma_bf16(small, ah + NEXT_PART, bh, two, 1);                 // m [h m]
            sm100::umma_bf16(small, ah + 2 * NEXT_PART, bh, one, 1);             // l h
            sm100::umma_bf16(to + 64 * (k / EVERY), ah, bh, one, k % EVERY > 0);
        }
    }
}
// A has 64 rows, whose m part, behind the h part, takes the lower 64 lanes: row t's result is lane t's sums and,
// of lane 64 + t, all but the last.  (Behind the l part lies something else, and so does its product.)
template <int EVERY, int A_STEP, int B_STEP>
__device__ __forceinline__ void issue64(uint32_t to, uint32_t majors, int steps, uint64_t a, uint64_t b) {
    const uint32_t one = sm100::umma_idesc_bf16(128, 64) | majors, two = sm100::umma_idesc_bf16(128, 128) | majors;
    const uint32_t small = to + 64 * sets<EVERY>(steps);
    for (int k0 = 0; k0 < steps; k0 += 4, a += NEXT_TILE, b += NEXT_TILE) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int k = k0 + i;
            if (k >= steps) break;
            const uint64_t ah = a + i * A_STEP, bh = b + i * B_STEP;
            sm100::umma_bf16(small, ah, bh + NEXT_PART, two, k > 0);             // [h; m] [m l]
            sm100::umma_bf16(small + 64, ah + 2 * NEXT_PART, bh, one, 1);        // [l; ..] h
            sm100::umma_bf16(to + 64 * (k / EVERY), ah, bh, one, k % EVERY > 0);  // [h; m] h
        }
    }
}

// Eight columns of the thread's lane of what these left from `at` on, the last of the h parts' sums added to
// all others.  `second`: a lane of the m part.
template <int EVERY>
__device__ __forceinline__ void sums_of(float (&y)[8], uint32_t at, int sets, bool second = false) {
    float x[8], z[8];
    __syncwarp();  // (the warp's lanes load together, and what came before may have parted them)
    sm100::tmem_ld_8(at + 64 * sets, x);
    if (!second) {
        sm100::tmem_ld_8(at + 64 * sets + 64, z);
#pragma unroll
        for (int j = 0; j < 8; ++j) x[j] += z[j];
    }
    const float cut = second ? 0.0f : CUT * EVERY;
    for (int i = 0; i < sets - 1; ++i) {
        sm100::tmem_ld_8(at + 64 * i, z);
#pragma unroll
        for (int j = 0; j < 8; ++j) x[j] = z[j] + fmaf(cut, z[j], x[j]);
    }
    sm100::tmem_ld_8(at + 64 * (sets - 1), y);
#pragma unroll
    for (int j = 0; j < 8; ++j) y[j] += fmaf(cut, y[j], x[j]);
}

}  // namespace split3
}  // namespace rfx
