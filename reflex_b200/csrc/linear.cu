// Matrix products  y[r, n] = sum_k x[r, k] * W[n, k]   (W row-major [out, in],
// the layout of the reference's linear layers: src/kernels_cuda/gemv.cu:1-4).
//
//  * rfx_gemm_f32: the true 32-bit product.  CUDA-core fused multiply-adds
//    only; each output element is reduced over k = 0..K-1 in index order by one
//    thread, so its value does not depend on how many rows the call has or on
//    where the row sits in the batch, nor on which of the three forms runs.
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

// Up to 64 rows: the weights are streamed once.  A block owns 32 columns, a lane a column, a warp RPW
// rows; what bounds it is one element's chain of K dependent multiply-adds (four cycles each), beside
// which the weights of a square matrix arrive at about the memory's rate, so the chains of different
// rows run in different warps, few to a warp.
constexpr int KT = 64, WLD = KT + 4;  // columns of a stage; row stride: eight lanes' 16-byte reads meet all banks

template <int RPW>
__global__ void __launch_bounds__(512)
gemm_f32_rows_kernel(const float* __restrict__ x, const float* __restrict__ W, float* __restrict__ y, int R, int N,
                     int K, int stages) {
    extern __shared__ __align__(16) float sm[];
    pdl_prologue();
    const int warps = blockDim.x >> 5, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int rows = warps * RPW, r0 = blockIdx.y * rows, n0 = blockIdx.x * 32;
    const int stage = 32 * WLD + rows * KT;  // [32][WLD] of W, [rows][KT] of x
    const int tiles = (K + KT - 1) / KT;
    auto fetch = [&](int t) {
        if (t < tiles) {
            float* to = sm + (t % stages) * stage;
            for (int e = threadIdx.x; e < (32 + rows) * (KT / 4); e += blockDim.x) {
                const int i = e / (KT / 4), c = 4 * (e % (KT / 4)), k = t * KT + c;
                if (i < 32) copy16(to + i * WLD + c, W + (size_t)(n0 + i < N ? n0 + i : 0) * K + (k < K ? k : 0), n0 + i < N && k < K);
                else {
                    const int r = r0 + i - 32;
                    copy16(to + 32 * WLD + (i - 32) * KT + c, x + (size_t)(r < R ? r : 0) * K + (k < K ? k : 0), r < R && k < K);
                }
            }
        }
        copies_done();
    };
    for (int t = 0; t < stages - 1; ++t) fetch(t);
    float acc[RPW];
#pragma unroll
    for (int i = 0; i < RPW; ++i) acc[i] = 0.0f;
    for (int t = 0; t < tiles; ++t) {
        switch (stages) {  // the group of tile t is the oldest of stages - 1 in flight
            case 8: wait_copies<6>(); break;
            case 6: wait_copies<4>(); break;
            default: wait_copies<2>(); break;
        }
        __syncthreads();  // tile t has landed, and every warp is done with the tile before
        fetch(t + stages - 1);
        const float* w = sm + (t % stages) * stage + lane * WLD;
        const float* xs = sm + (t % stages) * stage + 32 * WLD + warp * RPW * KT;
#pragma unroll
        for (int k = 0; k < KT; k += 4) {
            const float4 b = *reinterpret_cast<const float4*>(w + k);
#pragma unroll
            for (int i = 0; i < RPW; ++i) {
                const float4 a = *reinterpret_cast<const float4*>(xs + i * KT + k);
                acc[i] = fmaf(a.x, b.x, acc[i]);
                acc[i] = fmaf(a.y, b.y, acc[i]);
                acc[i] = fmaf(a.z, b.z, acc[i]);
                acc[i] = fmaf(a.w, b.w, acc[i]);
            }
        }
    }
#pragma unroll
    for (int i = 0; i < RPW; ++i) {
        const int r = r0 + warp * RPW + i;
        if (r < R && n0 + lane < N) y[(size_t)r * N + n0 + lane] = acc[i];
    }
}

// More rows: BM x BN tiles, a thread 8 rows by TN columns (rows ty + BM / 8 i, columns tx + 16 j: the
// reads of a quarter warp then meet all banks), both operands as they lie, sixteen k a stage.
constexpr int BK = 16, BLD = BK + 4, BSTAGES = 4;

template <int BM, int BN>
__global__ void __launch_bounds__(BM * 2)
gemm_f32_tile_kernel(const float* __restrict__ x, const float* __restrict__ W, float* __restrict__ y, int R, int N,
                     int K) {
    constexpr int THREADS = BM * 2, TN = BN / 16, STAGE = (BM + BN) * BLD;
    extern __shared__ __align__(16) float sm[];
    pdl_prologue();
    const int tx = threadIdx.x % 16, ty = threadIdx.x / 16;
    const int r0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
    const int tiles = (K + BK - 1) / BK;
    auto fetch = [&](int t) {
        if (t < tiles) {
            float* to = sm + (t % BSTAGES) * STAGE;
#pragma unroll
            for (int e = threadIdx.x; e < (BM + BN) * (BK / 4); e += THREADS) {
                const int i = e / (BK / 4), c = 4 * (e % (BK / 4)), k = t * BK + c;
                const int row = i < BM ? r0 + i : n0 + i - BM;
                const bool ok = row < (i < BM ? R : N) && k < K;
                const float* src = i < BM ? x : W;
                copy16(to + i * BLD + c, ok ? src + (size_t)row * K + k : src, ok);
            }
        }
        copies_done();
    };
#pragma unroll
    for (int t = 0; t < BSTAGES - 1; ++t) fetch(t);
    float acc[8][TN];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = 0.0f;
    for (int t = 0; t < tiles; ++t) {
        wait_copies<BSTAGES - 2>();
        __syncthreads();
        fetch(t + BSTAGES - 1);
        const float* a = sm + (t % BSTAGES) * STAGE + ty * BLD;
        const float* b = sm + (t % BSTAGES) * STAGE + (BM + tx) * BLD;
#pragma unroll
        for (int k = 0; k < BK; k += 4) {
            float4 av[8], bv[TN];
#pragma unroll
            for (int i = 0; i < 8; ++i) av[i] = *reinterpret_cast<const float4*>(a + i * (BM / 8) * BLD + k);
#pragma unroll
            for (int j = 0; j < TN; ++j) bv[j] = *reinterpret_cast<const float4*>(b + j * 16 * BLD + k);
#pragma unroll
            for (int i = 0; i < 8; ++i)
#pragma unroll
                for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(av[i].x, bv[j].x, acc[i][j]);
#pragma unroll
            for (int i = 0; i < 8; ++i)
#pragma unroll
                for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(av[i].y, bv[j].y, acc[i][j]);
#pragma unroll
            for (int i = 0; i < 8; ++i)
#pragma unroll
                for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(av[i].z, bv[j].z, acc[i][j]);
#pragma unroll
            for (int i = 0; i < 8; ++i)
#pragma unroll
                for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(av[i].w, bv[j].w, acc[i][j]);
        }
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int r = r0 + ty + (BM / 8) * i;
        if (r >= R) continue;
#pragma unroll
        for (int j = 0; j < TN; ++j) {
            const int n = n0 + tx + 16 * j;
            if (n < N) y[(size_t)r * N + n] = acc[i][j];
        }
    }
}

template <int RPW>
int launch_rows(const float* x, const float* W, float* y, int R, int N, int K, cudaStream_t s) {
    int warps = (R + RPW - 1) / RPW;
    if (warps < 4) warps = 4;  // enough threads to issue the copies
    const size_t stage = (size_t)(32 * WLD + warps * RPW * KT) * sizeof(float);
    const int stages = stage * 8 <= 100 * 1024 ? 8 : stage * 6 <= 110 * 1024 ? 6 : 4;
    cudaError_t e = cudaFuncSetAttribute(gemm_f32_rows_kernel<RPW>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)(stage * stages));
    if (e != cudaSuccess) return (int)e;
    RFX_LAUNCH(gemm_f32_rows_kernel<RPW>, dim3((N + 31) / 32, 1), warps * 32, stage * stages, s, x, W, y, R, N, K, stages);
    return 0;
}

template <int BM, int BN>
int launch_tiles(const float* x, const float* W, float* y, int R, int N, int K, cudaStream_t s) {
    constexpr size_t smem = (size_t)BSTAGES * (BM + BN) * BLD * sizeof(float);
    cudaError_t e = cudaFuncSetAttribute(gemm_f32_tile_kernel<BM, BN>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return (int)e;
    RFX_LAUNCH((gemm_f32_tile_kernel<BM, BN>), dim3((N + BN - 1) / BN, (R + BM - 1) / BM), BM * 2, smem, s, x, W, y, R, N, K);
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
        if (R <= 8) return launch_rows<1>(x, W, y, R, N, K, st);
        if (R <= 32) return launch_rows<2>(x, W, y, R, N, K, st);
        if (R <= 64) return launch_rows<4>(x, W, y, R, N, K, st);
        // the larger tile reads shared memory half as often a multiply-add; it needs two tiles an SM
        if ((long long)((R + 127) / 128) * ((N + 127) / 128) >= 2LL * sm_count())
            return launch_tiles<128, 128>(x, W, y, R, N, K, st);
        return launch_tiles<64, 64>(x, W, y, R, N, K, st);
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
