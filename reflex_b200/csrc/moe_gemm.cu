// The experts' products of a decode step: for every expert with rows, y[rows] = act(x[rows] W_e^T),
// each expert's weights read once, however many of the (at most 64) rows chose it.
//
// As in gemm_tc.cu the weights are the M operand of tcgen05.mma (128 weight rows a CTA, streamed by
// TMA into an mbarrier ring) and the expert's rows its N operand: they lie side by side (moe.cu places
// the (row, choice) pairs expert by expert), so one TMA box of 16, 32 or 64 rows from the expert's
// first one brings them, and the rows behind them are not stored.  (An expert that a row names several
// times can have more rows than the step: its CTAs go over the weights again for every further box.)
// A gated expert ([gate rows | up rows]) gives a CTA 64 gate rows and the 64 up rows that belong to
// them; its epilogue writes the activation of the pair, so the up product's 2 ff columns never go to
// memory.
//
// Memory bounds it: a CTA's ring is filled with weights before the wait on the kernel before where
// most experts have rows (the weights do not depend on the routing; an expert without rows then drops
// what it brought).  Eight rows, four of sixteen experts of 3 x 2,048 x 2,048 (363 MB on average): the
// library's grouped products took 89 us, their preparation and the activation 7 more; these two launches
// take 60 (the whole layer 121 us, now 80).
#include "common.cuh"
#include "sm100.cuh"
#include "tma_host.cuh"

namespace {

using namespace sm100;

constexpr int BM = 128, BK = 64, THREADS = 192, MAX_STAGES = 8;
constexpr int A_BYTES = BM * BK * 2;

enum Act { PLAIN = 0, RELU2 = 1, SILU = 2, GLU_CLAMPED = 3, SWIGLU = 4 };

template <int ACT>
__device__ __forceinline__ float activation(float g, float u, float alpha, float limit) {
    if constexpr (ACT == RELU2) {
        g = fmaxf(g, 0.0f);
        return g * g;
    }
    if constexpr (ACT == SILU) return g / (1.0f + expf(-g));
    if constexpr (ACT == GLU_CLAMPED) {
        g = fminf(g, limit);
        u = fminf(fmaxf(u, -limit), limit);
        return (g / (1.0f + expf(-alpha * g))) * (u + 1.0f);
    }
    if constexpr (ACT == SWIGLU) return (g / (1.0f + expf(-g))) * u;
    return g;
}

template <int BN, int ACT, typename TO>
__global__ void __launch_bounds__(THREADS)
moe_gemm_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x,
                const int* __restrict__ offsets, TO* __restrict__ y, int N, int K, int stages, int ahead, float alpha,
                float limit, int* __restrict__ err) {
    constexpr bool GATED = ACT >= GLU_CLAMPED;
    constexpr int COLS = GATED ? BM / 2 : BM;   // output columns a CTA makes
    constexpr int B_BYTES = BN * BK * 2, STAGE = A_BYTES + B_BYTES;
    constexpr uint32_t TMEM_COLS = BN < 32 ? 32 : BN;
    extern __shared__ uint8_t smem_raw[];
    __shared__ __align__(8) uint64_t full_bar[MAX_STAGES], empty_bar[MAX_STAGES], done_bar, read_bar;
    __shared__ uint32_t tmem_base;
    __shared__ float ups[GATED ? BN * (BM / 2) : 1];
    uint8_t* tiles = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int n0 = blockIdx.x * COLS, e = blockIdx.y;
    const int nkb = (K + BK - 1) / BK;
    // the tile's two halves of 64 weight rows
    const int w0 = GATED ? e * 2 * N + n0 : e * N + n0, w1 = GATED ? w0 + N : w0 + 64;
    if (threadIdx.x == 0) {
        for (int s = 0; s < stages; ++s) {
            mbar_init(&full_bar[s], 2);  // the weights' bytes and the rows' are announced apart
            mbar_init(&empty_bar[s], 1);
        }
        mbar_init(&done_bar, 1);
        mbar_init(&read_bar, 4);
        fence_barrier_init();
        prefetch_tensormap(&map_w);
        prefetch_tensormap(&map_x);
    }
    if (warp == 1) {
        tmem_alloc(&tmem_base, TMEM_COLS);
        tmem_relinquish();
    }
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem = tmem_base;
    rfx::pdl_launch_dependents();
    auto load_w = [&](int i, int s) {
        uint8_t* a = tiles + (size_t)s * STAGE;
        mbar_expect_tx(&full_bar[s], A_BYTES);
        tma_load_2d(a, &map_w, &full_bar[s], i * BK, w0);
        tma_load_2d(a + A_BYTES / 2, &map_w, &full_bar[s], i * BK, w1);
    };
    if (warp == 0) {
        if (elect_one()) {
            const int pre = min(nkb, ahead);
            for (int i = 0; i < pre; ++i) load_w(i, i);
            rfx::pdl_wait();
            const int first = offsets[e], rows = offsets[e + 1] - first;
            if (rows > 0) {
                bool ok = true;
                for (int r = 0, it = 0; r < rows && ok; r += BN)
                    for (int i = 0; i < nkb; ++i, ++it) {
                        const int s = it % stages;
                        const uint32_t ph = (it / stages) & 1;
                        if (it >= pre) {
                            if (!mbar_wait(&empty_bar[s], ph ^ 1)) {
                                atomicExch(err, 51);
                                ok = false;
                                break;
                            }
                            load_w(i, s);
                        }
                        mbar_expect_tx(&full_bar[s], B_BYTES);
                        tma_load_2d(tiles + (size_t)s * STAGE + A_BYTES, &map_x, &full_bar[s], i * BK, first + r);
                    }
            } else {
                // nothing to do: what was brought ahead has to land before the CTA leaves
                for (int i = 0; i < pre; ++i) mbar_arrive(&full_bar[i]);
                for (int i = 0; i < pre; ++i)
                    if (!mbar_wait(&full_bar[i], 0)) atomicExch(err, 52);
            }
        }
        __syncwarp();
    } else if (warp == 1) {
        rfx::pdl_wait();
        const int rows = offsets[e + 1] - offsets[e];
        if (rows > 0 && elect_one()) {
            constexpr uint32_t idesc = umma_idesc_bf16(BM, BN);
            bool ok = true;
            for (int box = 0, it = 0; box * BN < rows && ok; ++box) {
                if (box && !mbar_wait(&read_bar, (box - 1) & 1)) {  // the sums of the box before have been read
                    atomicExch(err, 55);
                    break;
                }
                tc_fence_after_sync();
                for (int i = 0; i < nkb; ++i, ++it) {
                    const int s = it % stages;
                    if (!mbar_wait(&full_bar[s], (it / stages) & 1)) {
                        atomicExch(err, 53);
                        ok = false;
                        break;
                    }
                    tc_fence_after_sync();
                    const uint32_t a = smem_u32(tiles + (size_t)s * STAGE);
                    const uint64_t da = umma_desc_k_sw128(a), db = umma_desc_k_sw128(a + A_BYTES);
#pragma unroll
                    for (int k = 0; k < BK / 16; ++k) umma_bf16(tmem, da + 2 * k, db + 2 * k, idesc, (i > 0 || k > 0) ? 1u : 0u);
                    umma_commit(&empty_bar[s]);
                }
                if (ok) umma_commit(&done_bar);
            }
        }
        __syncwarp();
    } else {
        rfx::pdl_wait();
        const int first = offsets[e], rows = offsets[e + 1] - first;
        const int q = warp & 3, m = q * 32 + lane;  // this warp may read TMEM lanes [32 q, 32 q + 32)
        const uint32_t base = tmem + ((uint32_t)(q * 32) << 16);
        for (int box = 0; box * BN < rows; ++box) {  // (all boxes, also after a wait that gave up: the warps meet below)
            const bool have = mbar_wait(&done_bar, box & 1);
            if (!have && lane == 0) atomicExch(err, 54);
            tc_fence_after_sync();
            if constexpr (GATED) {
                if (q >= 2) {
#pragma unroll 1
                    for (int c = 0; c < BN / 16; ++c) {
                        float v[16];
                        tmem_ld_16(base + c * 16, v);
#pragma unroll
                        for (int j = 0; j < 16; ++j) ups[(c * 16 + j) * (BM / 2) + m - BM / 2] = v[j];
                    }
                }
                asm volatile("bar.sync 1, 128;" ::: "memory");
            }
            if (!GATED || q < 2) {
                const int n = n0 + m, here = rows - box * BN;
#pragma unroll 1
                for (int c = 0; c < BN / 16; ++c) {
                    float v[16];
                    tmem_ld_16(base + c * 16, v);
                    if (c * 16 >= here) break;
                    if (n < N && have) {
#pragma unroll
                        for (int j = 0; j < 16; ++j) {
                            const int r = c * 16 + j;
                            const float u = GATED ? ups[r * (BM / 2) + m] : 0.0f;
                            if (r < here)
                                rfx::st<TO>(y, (size_t)(first + box * BN + r) * N + n, activation<ACT>(v[j], u, alpha, limit));
                        }
                    }
                }
            }
            tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) mbar_arrive(&read_bar);
        }
    }
    __syncthreads();
    if (warp == 1) {
        tc_fence_after_sync();
        tmem_dealloc(tmem, TMEM_COLS);
    }
}

template <int BN, int ACT, typename TO>
int launch(const void* x, const void* W, const int* offsets, void* y, int n_pairs, int E, int N, int K, float alpha,
           float limit, int* err, cudaStream_t s) {
    constexpr bool GATED = ACT >= GLU_CLAMPED;
    CUtensorMap mw, mx;
    if (!rfx::tma::make_map_rows64(&mw, W, (long long)E * N * (GATED ? 2 : 1), K, BM / 2) ||
        !rfx::tma::make_map_rows64(&mx, x, n_pairs, K, BN))
        return RFX_ERR_UNSUPPORTED;
    constexpr int STAGE = A_BYTES + BN * BK * 2;
    // two CTAs an SM, about 100 KB each; gated ones for 33 to 64 rows have 16 KB of up values beside the ring and
    // an SM to themselves
    int stages = 98 * 1024 / STAGE;
    if (stages > MAX_STAGES) stages = MAX_STAGES;
    const int nkb = (K + BK - 1) / BK;
    // on average an expert has rows with 1 - (1 - 1/E)^pairs: from pairs = 1.25 E on 7 of 10
    const int ahead = 4LL * n_pairs >= 5LL * E ? (stages < nkb ? stages : nkb) : 0;
    const size_t smem = (size_t)stages * STAGE + 1024;
    auto kernel = moe_gemm_kernel<BN, ACT, TO>;
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return (int)e;
    const int cols = GATED ? BM / 2 : BM;
    RFX_LAUNCH(kernel, dim3((N + cols - 1) / cols, E), THREADS, smem, s, mw, mx, offsets, (TO*)y, N, K, stages, ahead,
               alpha, limit, err);
    return 0;
}

template <int ACT, typename TO>
int by_rows(int max_rows, const void* x, const void* W, const int* offsets, void* y, int n_pairs, int E, int N, int K,
            float alpha, float limit, int* err, cudaStream_t s) {
    if (max_rows <= 16) return launch<16, ACT, TO>(x, W, offsets, y, n_pairs, E, N, K, alpha, limit, err, s);
    if (max_rows <= 32) return launch<32, ACT, TO>(x, W, offsets, y, n_pairs, E, N, K, alpha, limit, err, s);
    return launch<64, ACT, TO>(x, W, offsets, y, n_pairs, E, N, K, alpha, limit, err, s);
}

}  // namespace

// y[p, :] = act(x[p, :] W_e^T) for the rows p in [offsets[e], offsets[e + 1]) of every expert e: x bfloat16
// [n_pairs, K], W bfloat16 [E, N, K] (gated activations: [E, 2 N, K], gate rows first), offsets int32
// [E + 1] on the device.  max_rows <= 64: the most rows an expert has as a rule (more are right, at the
// price of reading its weights again).  act 0 none (y float32), 1 relu^2, 2 silu,
// 3 the clamped gated form with alpha and limit, 4 silu(gate) * up (y bfloat16).  K in eights, x and W on
// 16 bytes.
extern "C" int rfx_moe_gemm(const void* x, const void* W, const int* offsets, void* y, int n_pairs, int max_rows, int E,
                            int N, int K, int act, float alpha, float limit, int* err, void* stream) {
    if (n_pairs <= 0) return 0;
    if (E <= 0 || N <= 0 || K <= 0 || max_rows <= 0 || act < 0 || act > 4) return RFX_ERR_BAD_ARG;
    if (max_rows > 64 || K % 8 || E > 65535 || ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(W)) & 15))
        return RFX_ERR_UNSUPPORTED;
    cudaStream_t s = (cudaStream_t)stream;
#define RFX_GO(A, T) return by_rows<A, T>(max_rows, x, W, offsets, y, n_pairs, E, N, K, alpha, limit, err, s)
    switch (act) {
        case PLAIN: RFX_GO(PLAIN, float);
        case RELU2: RFX_GO(RELU2, __nv_bfloat16);
        case SILU: RFX_GO(SILU, __nv_bfloat16);
        case GLU_CLAMPED: RFX_GO(GLU_CLAMPED, __nv_bfloat16);
        default: RFX_GO(SWIGLU, __nv_bfloat16);
    }
#undef RFX_GO
}
