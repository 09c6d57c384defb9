// Matrix products  y[r, n] = sum_k x[r, k] * W[n, k]   (W row-major [out, in],
// the layout of the reference's linear layers: src/kernels_cuda/gemv.cu:1-4).
//
//  * rfx_gemm_f32: the true 32-bit product.  CUDA-core fused multiply-adds
//    only; each output element is reduced over k = 0..K-1 in index order by one
//    thread, so its value does not depend on how many rows the call has or on
//    where the row sits in the batch, nor on which form (tile) runs.
//  * rfx_gemv_bf16: bfloat16 weights and activations for a few rows (decode),
//    32-bit accumulation; a pure weight-streaming kernel with 16-byte loads.
#include "common.cuh"

namespace {

using namespace rfx;

constexpr int TM = 64, TN = 64, TK = 16;

__global__ void __launch_bounds__(256)
gemm_f32_kernel(const float* __restrict__ x, const float* __restrict__ W, float* __restrict__ y,
                int R, int N, int K) {
    __shared__ float xs[TK][TM + 1];
    __shared__ float ws[TK][TN + 1];
    pdl_prologue();
    const int r0 = blockIdx.y * TM, n0 = blockIdx.x * TN;
    const int tx = threadIdx.x % 16, ty = threadIdx.x / 16;  // 16 x 16 threads, 4 x 4 outputs
    float acc[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = 0.0f;

    for (int k0 = 0; k0 < K; k0 += TK) {
        // 64 rows x 16 k per operand = 1024 elements, 4 per thread
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int e = threadIdx.x + i * 256;
            const int row = e / TK, kk = e % TK;
            const int k = k0 + kk;
            xs[kk][row] = (r0 + row < R && k < K) ? x[(size_t)(r0 + row) * K + k] : 0.0f;
            ws[kk][row] = (n0 + row < N && k < K) ? W[(size_t)(n0 + row) * K + k] : 0.0f;
        }
        __syncthreads();
#pragma unroll
        for (int kk = 0; kk < TK; ++kk) {
            float a[4], b[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) a[i] = xs[kk][ty * 4 + i];
#pragma unroll
            for (int j = 0; j < 4; ++j) b[j] = ws[kk][tx * 4 + j];
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int r = r0 + ty * 4 + i;
        if (r >= R) continue;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int n = n0 + tx * 4 + j;
            if (n < N) y[(size_t)r * N + n] = acc[i][j];
        }
    }
}

// The forms below read both operands 16 bytes an access through rings of asynchronous copies (K a
// multiple of four, both matrices on 16 bytes; other products take the form above).
__device__ __forceinline__ void copy16(float* dst, const float* src, bool valid) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src),
                 "r"(valid ? 16 : 0)
                 : "memory");
}
__device__ __forceinline__ void copies_done() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void wait_copies() {
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// A block owns BM rows by BN columns, a thread TM rows (BM / TM apart) by TN columns (BN / TN apart:
// the reads of eight neighbours then meet all banks).  An element's sum is one chain over k, so neither
// tensor cores nor a split of k may serve, and the chip is filled by elements alone.  What bounds it:
// with one or two rows the weights (4,096 x 4,096: 3.3 TB/s, 24,576 x 4,096: 5.9); with few rows the
// chain of K dependent multiply-adds beside the reads of shared memory, so threads have few elements and
// stages are long (one barrier for 128 steps of the chain); with many rows the registers' banks, as a
// multiply-add whose sum and weight share one takes two cycles, and columns side by side in K alternate
// with it: 48 of 72 TFLOP/s at most, 47 reached (24,576 columns, 1,024 rows).  Packed pairs of columns (one
// instruction, no such meeting) were slower, the pairs' x being read twice from shared memory.
template <int BM, int BN, int TM, int TN, int BK, int STAGES_>
struct Tile {
    static constexpr int ACROSS = BN / TN, THREADS = BM / TM * ACROSS, LD = BK + 4, STAGE = (BM + BN) * LD;
    static constexpr int STAGES = STAGES_, RS = THREADS / (BK / 4);  // rows a pass of the block's copies covers
    static constexpr int XC = (BM + RS - 1) / RS, WC = (BN + RS - 1) / RS;
    static constexpr size_t SMEM = (size_t)STAGES * STAGE * sizeof(float);
    static_assert(THREADS % (BK / 4) == 0 && BN % RS == 0, "whole passes");
};

template <class T, int BM, int BN, int TM, int TN, int BK>
__global__ void __launch_bounds__(T::THREADS)
gemm_f32_tile_kernel(const float* __restrict__ x, const float* __restrict__ W, float* __restrict__ y, int R, int N,
                     int K) {
    constexpr int STAGES = T::STAGES, LD = T::LD, RS = T::RS;
    extern __shared__ __align__(16) float sm[];
    pdl_prologue();
    const int tx = threadIdx.x % T::ACROSS, ty = threadIdx.x / T::ACROSS;
    const int r0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
    const int tiles = (K + BK - 1) / BK;
    const int crow = threadIdx.x / (BK / 4), cc = 4 * (threadIdx.x % (BK / 4));
    const float* xsrc = x + (size_t)(r0 + crow) * K + cc;
    const float* wsrc = W + (size_t)(n0 + crow) * K + cc;
    int to = 0;  // the stage the next tile goes to
    auto fetch = [&](int t) {
        if (t < tiles) {
            const bool in = t * BK + cc < K;
            float* d = sm + to * T::STAGE + crow * LD + cc;
#pragma unroll
            for (int i = 0; i < T::WC; ++i) {
                const bool ok = in && n0 + crow + i * RS < N;
                copy16(d + (BM + i * RS) * LD, ok ? wsrc + (size_t)(i * RS) * K : W, ok);
            }
#pragma unroll
            for (int i = 0; i < T::XC; ++i) {
                if (BM % RS && crow + i * RS >= BM) continue;
                const bool ok = in && r0 + crow + i * RS < R;
                copy16(d + i * RS * LD, ok ? xsrc + (size_t)(i * RS) * K : x, ok);
            }
            xsrc += BK;
            wsrc += BK;
        }
        copies_done();
        to = to + 1 == STAGES ? 0 : to + 1;
    };
#pragma unroll
    for (int t = 0; t < STAGES - 1; ++t) fetch(t);
    float acc[TM][TN];
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = 0.0f;
    int at = 0;
    for (int t = 0; t < tiles; ++t) {
        wait_copies<STAGES - 2>();
        __syncthreads();  // tile t has landed, and every warp is done with the tile before
        fetch(t + STAGES - 1);
        const float* a = sm + at * T::STAGE + ty * LD;
        const float* b = sm + at * T::STAGE + (BM + tx) * LD;
        at = at + 1 == STAGES ? 0 : at + 1;
#pragma unroll
        for (int k = 0; k < BK; k += 4) {
            float4 av[TM], bv[TN];
#pragma unroll
            for (int i = 0; i < TM; ++i) av[i] = *reinterpret_cast<const float4*>(a + i * (BM / TM) * LD + k);
#pragma unroll
            for (int j = 0; j < TN; ++j) bv[j] = *reinterpret_cast<const float4*>(b + j * T::ACROSS * LD + k);
#pragma unroll
            for (int i = 0; i < TM; ++i)
#pragma unroll
                for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(av[i].x, bv[j].x, acc[i][j]);
#pragma unroll
            for (int i = 0; i < TM; ++i)
#pragma unroll
                for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(av[i].y, bv[j].y, acc[i][j]);
#pragma unroll
            for (int i = 0; i < TM; ++i)
#pragma unroll
                for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(av[i].z, bv[j].z, acc[i][j]);
#pragma unroll
            for (int i = 0; i < TM; ++i)
#pragma unroll
                for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(av[i].w, bv[j].w, acc[i][j]);
        }
    }
#pragma unroll
    for (int i = 0; i < TM; ++i) {
        const int r = r0 + ty + BM / TM * i;
        if (r >= R) continue;
#pragma unroll
        for (int j = 0; j < TN; ++j) {
            const int n = n0 + tx + T::ACROSS * j;
            if (n < N) y[(size_t)r * N + n] = acc[i][j];
        }
    }
}

template <int BM, int BN, int TM, int TN, int BK, int STAGES>
int launch_tiles(const float* x, const float* W, float* y, int R, int N, int K, cudaStream_t s) {
    using T = Tile<BM, BN, TM, TN, BK, STAGES>;
    auto kernel = gemm_f32_tile_kernel<T, BM, BN, TM, TN, BK>;
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)T::SMEM);
    if (e != cudaSuccess) return (int)e;
    RFX_LAUNCH(kernel, dim3((N + BN - 1) / BN, (R + BM - 1) / BM), T::THREADS, T::SMEM, s, x, W, y, R, N, K);
    return 0;
}

// One warp per output column n; RT rows of x per pass.  K must be a multiple
// of 8 (16-byte loads); the host refuses other K.
template <int RT, typename TO>
__global__ void __launch_bounds__(256)
gemv_bf16_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ W,
                 TO* __restrict__ y, int R, int N, int K) {
    pdl_prologue();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int n = blockIdx.x * 8 + warp;
    if (n >= N) return;
    const uint4* wrow = reinterpret_cast<const uint4*>(W + (size_t)n * K);
    const int kv = K / 8;
    for (int r0 = 0; r0 < R; r0 += RT) {
        float acc[RT];
#pragma unroll
        for (int i = 0; i < RT; ++i) acc[i] = 0.0f;
        for (int c = lane; c < kv; c += 32) {
            const uint4 wv = wrow[c];
            const __nv_bfloat162* w2 = reinterpret_cast<const __nv_bfloat162*>(&wv);
            float wf[8];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float2 f = __bfloat1622float2(w2[j]);
                wf[2 * j] = f.x;
                wf[2 * j + 1] = f.y;
            }
#pragma unroll
            for (int i = 0; i < RT; ++i) {
                if (r0 + i < R) {
                    const uint4 xv = reinterpret_cast<const uint4*>(x + (size_t)(r0 + i) * K)[c];
                    const __nv_bfloat162* x2 = reinterpret_cast<const __nv_bfloat162*>(&xv);
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const float2 f = __bfloat1622float2(x2[j]);
                        acc[i] = fmaf(wf[2 * j], f.x, acc[i]);
                        acc[i] = fmaf(wf[2 * j + 1], f.y, acc[i]);
                    }
                }
            }
        }
#pragma unroll
        for (int i = 0; i < RT; ++i) {
            const float total = warp_sum(acc[i]);
            if (lane == 0 && r0 + i < R) st<TO>(y, (size_t)(r0 + i) * N + n, total);
        }
    }
}

// y[j] = x[j, :] . W[ids[j], :]: the head's rows of a handful of token ids only,
// for scoring given continuations (the reference's gathered product,
// src/kernels_cuda/gemv_gather.cu:10-51): kilobytes of the head are read, not
// the whole vocabulary.  One warp per pair.  32-bit: the lanes stage the two
// rows in shared memory, a chunk at a time, and lane 0 runs one fused
// multiply-add chain over k in index order, which gives the bits of
// `gemm_f32_kernel` for the same row and column.  An id outside [0, V) gives
// NaN and sets the error word (the host checks ids before it launches).
constexpr int GATHER_WARPS = 4, GATHER_CHUNK = 512;

__global__ void __launch_bounds__(GATHER_WARPS * 32)
gather_dot_f32_kernel(const float* __restrict__ x, const float* __restrict__ W, const int* __restrict__ ids,
                      float* __restrict__ y, int P, int K, int V, int* __restrict__ err) {
    __shared__ float xs[GATHER_WARPS][GATHER_CHUNK];
    __shared__ float ws[GATHER_WARPS][GATHER_CHUNK];
    pdl_prologue();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int j = blockIdx.x * GATHER_WARPS + warp;
    if (j >= P) return;
    const int id = ids[j];
    if (id < 0 || id >= V) {
        if (lane == 0) {
            y[j] = __int_as_float(0x7fc00000);
            atomicExch(err, 1 + j);
        }
        return;
    }
    const float* xr = x + (size_t)j * K;
    const float* wr = W + (size_t)id * K;
    float acc = 0.0f;
    for (int k0 = 0; k0 < K; k0 += GATHER_CHUNK) {
        const int n = min(GATHER_CHUNK, K - k0);
        for (int i = lane; i < n; i += 32) {
            xs[warp][i] = xr[k0 + i];
            ws[warp][i] = wr[k0 + i];
        }
        __syncwarp();
        if (lane == 0)
            for (int i = 0; i < n; ++i) acc = fmaf(xs[warp][i], ws[warp][i], acc);
        __syncwarp();
    }
    if (lane == 0) y[j] = acc;
}

// bfloat16 rows, 32-bit accumulation: 16-byte loads when K is a multiple of 8.
__global__ void __launch_bounds__(GATHER_WARPS * 32)
gather_dot_bf16_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ W,
                       const int* __restrict__ ids, float* __restrict__ y, int P, int K, int V,
                       int* __restrict__ err) {
    pdl_prologue();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int j = blockIdx.x * GATHER_WARPS + warp;
    if (j >= P) return;
    const int id = ids[j];
    if (id < 0 || id >= V) {
        if (lane == 0) {
            y[j] = __int_as_float(0x7fc00000);
            atomicExch(err, 1 + j);
        }
        return;
    }
    const __nv_bfloat16* xr = x + (size_t)j * K;
    const __nv_bfloat16* wr = W + (size_t)id * K;
    float acc = 0.0f;
    if ((K & 7) == 0) {
        const uint4* x4 = reinterpret_cast<const uint4*>(xr);
        const uint4* w4 = reinterpret_cast<const uint4*>(wr);
        for (int c = lane; c < K / 8; c += 32) {
            const uint4 xv = x4[c], wv = w4[c];
            const __nv_bfloat162* x2 = reinterpret_cast<const __nv_bfloat162*>(&xv);
            const __nv_bfloat162* w2 = reinterpret_cast<const __nv_bfloat162*>(&wv);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const float2 a = __bfloat1622float2(x2[i]), b = __bfloat1622float2(w2[i]);
                acc = fmaf(a.x, b.x, acc);
                acc = fmaf(a.y, b.y, acc);
            }
        }
    } else {
        for (int i = lane; i < K; i += 32) acc = fmaf(__bfloat162float(xr[i]), __bfloat162float(wr[i]), acc);
    }
    acc = warp_sum(acc);
    if (lane == 0) y[j] = acc;
}

}  // namespace

extern "C" int rfx_gather_dot(const void* x, const void* W, int dt, const int* ids, float* y, int P, int K,
                              int V, int* err, void* stream) {
    if (P <= 0) return 0;
    if (K <= 0 || V <= 0) return RFX_ERR_BAD_ARG;
    const int blocks = (P + GATHER_WARPS - 1) / GATHER_WARPS;
    cudaStream_t s = (cudaStream_t)stream;
    if (dt == RFX_DT_F32)
        RFX_LAUNCH(gather_dot_f32_kernel, blocks, GATHER_WARPS * 32, 0, s, (const float*)x, (const float*)W, ids,
                   y, P, K, V, err);
    else if (dt == RFX_DT_BF16) {
        if ((K & 7) == 0 && ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(W)) & 15))
            return RFX_ERR_BAD_ARG;
        RFX_LAUNCH(gather_dot_bf16_kernel, blocks, GATHER_WARPS * 32, 0, s, (const __nv_bfloat16*)x,
                   (const __nv_bfloat16*)W, ids, y, P, K, V, err);
    } else
        return RFX_ERR_BAD_ARG;
    return 0;
}

extern "C" int rfx_gemm_f32(const float* x, const float* W, float* y, int R, int N, int K,
                            void* stream) {
    if (R <= 0 || N <= 0) return 0;
    if (K <= 0) return RFX_ERR_BAD_ARG;
    dim3 grid((N + TN - 1) / TN, (R + TM - 1) / TM);
    if (grid.y > 65535) return RFX_ERR_UNSUPPORTED;
    cudaStream_t st = (cudaStream_t)stream;
    if (K % 4 == 0 && ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(W)) & 15) == 0) {
        // measured for N = K = 4,096 (and N = 24,576) against the 32-column form next to it in the list
        const bool few = N <= 32 * sm_count();  // 32 columns a block do not fill the chip
        if (R <= 1) return launch_tiles<1, 32, 1, 1, 128, 6>(x, W, y, R, N, K, st);  // 20 (69) us
        if (R <= 2) return launch_tiles<2, 32, 2, 1, 128, 6>(x, W, y, R, N, K, st);  // 25 (74)
        if (R <= 4) return launch_tiles<4, 16, 2, 1, 128, 6>(x, W, y, R, N, K, st);  // 28 (99), by 32 columns 33 (102)
        if (R <= 8) return launch_tiles<8, 16, 2, 1, 128, 5>(x, W, y, R, N, K, st);  // 37 (128), by 32: 43 (130)
        if (R <= 16)  // 44 (240) and 62 (147)
            return few ? launch_tiles<16, 16, 2, 2, 128, 5>(x, W, y, R, N, K, st)
                       : launch_tiles<16, 32, 4, 2, 64, 5>(x, W, y, R, N, K, st);
        if (R <= 32)  // 61 (347) and 94 (229)
            return few ? launch_tiles<32, 32, 4, 2, 128, 4>(x, W, y, R, N, K, st)
                       : launch_tiles<32, 32, 4, 4, 64, 4>(x, W, y, R, N, K, st);
        if (R <= 64 && few) return launch_tiles<64, 32, 4, 2, 128, 3>(x, W, y, R, N, K, st);  // 92 (533), below 127 (376)
        // Waves of blocks times a tile's work; small tiles do 6 % less a cycle, large ones a third less
        // while an SM has three or fewer.  6,144 columns, K = 4,096, small and large: 300 rows 418 and 446
        // us, 1,024 rows 1,234 and 1,177; 1,536 columns, K = 1,024, 701 rows: 66 and 103.
        const int sms = sm_count();
        const auto blocks = [&](int bm, int bn) { return (long long)((R + bm - 1) / bm) * ((N + bn - 1) / bn); };
        const long long per_small = (blocks(32, 64) + sms - 1) / sms, per_large = (blocks(64, 64) + sms - 1) / sms;
        if (per_small >= 2 && blocks(64, 32) <= 2 * sms)  // two a SM, a longer stage: 200 rows of N = 1,536 41 us, not 49
            return launch_tiles<64, 32, 4, 4, 64, 4>(x, W, y, R, N, K, st);
        if (per_small * 106 <= per_large * (per_large <= 3 ? 260 : 200) && (R + 31) / 32 <= 65535)  // (a grid's limit)
            return launch_tiles<32, 64, 4, 4, 32, 4>(x, W, y, R, N, K, st);
        return launch_tiles<64, 64, 8, 4, 32, 3>(x, W, y, R, N, K, st);
    }
    RFX_LAUNCH(gemm_f32_kernel, grid, 256, 0, (cudaStream_t)stream, x, W, y, R, N, K);
    return 0;
}

extern "C" int rfx_gemv_bf16(const void* x, const void* W, void* y, int y_dt, int R, int N, int K,
                             void* stream) {
    if (R <= 0 || N <= 0) return 0;
    if (K <= 0 || K % 8 != 0) return RFX_ERR_UNSUPPORTED;
    if ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(W)) & 15) return RFX_ERR_BAD_ARG;
    cudaStream_t s = (cudaStream_t)stream;
    const int blocks = (N + 7) / 8;
    const __nv_bfloat16* xb = (const __nv_bfloat16*)x;
    const __nv_bfloat16* wb = (const __nv_bfloat16*)W;
#define RFX_GEMV(RT)                                                                             \
    do {                                                                                         \
        if (y_dt == RFX_DT_F32)                                                                  \
            RFX_LAUNCH((gemv_bf16_kernel<RT, float>), blocks, 256, 0, s, xb, wb, (float*)y, R, N, K); \
        else if (y_dt == RFX_DT_BF16)                                                            \
            RFX_LAUNCH((gemv_bf16_kernel<RT, __nv_bfloat16>), blocks, 256, 0, s, xb, wb,         \
                       (__nv_bfloat16*)y, R, N, K);                                              \
        else                                                                                     \
            return RFX_ERR_BAD_ARG;                                                              \
    } while (0)
    if (R == 1) RFX_GEMV(1);
    else if (R == 2) RFX_GEMV(2);
    else if (R <= 4) RFX_GEMV(4);
    else RFX_GEMV(8);
#undef RFX_GEMV
    return 0;
}
