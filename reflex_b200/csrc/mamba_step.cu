// A decode step of the selective-scan mixer between its first and last product, for a few sequences:
// the short filter over x, the product [dt | B | C] = W_x u, the step sizes' second product and the
// scan's one step, in one launch (rfx_short_conv_act, rfx_gemm_bf16_tc and rfx_mamba_scan are three).
//
// Such a step has next to no work (width 1,024, one sequence: 0.6 MB of weights and state); what it
// costs is launches, one after the other.  A thread-block cluster takes a sequence: a CTA owns a slice of
// the channels, filters them, multiplies them with its columns of W_x, and sends the R + 2 N partial sums
// to every CTA of the cluster (distributed shared memory, one cluster barrier); each adds them in rank
// order and then steps its channels' states.  The weights' slices come to shared memory before the wait
// on the kernel before.  Every cluster reads all of W_x (from L2), so this form is for a few sequences.
//
// Types as in the three launches: u 32-bit, rounded to bfloat16 for the product, 32-bit sums, the low-rank
// vector rounded to bfloat16, everything else 32-bit.
#include <cooperative_groups.h>

#include "attn_mma.cuh"
#include "common.cuh"
#include "short_conv.cuh"

namespace cg = cooperative_groups;

namespace {

using namespace rfx;

constexpr int THREADS = 512, WARPS = THREADS / 32, LPC = 4;  // four lanes share a channel's states
constexpr float LOG2E = 1.4426950408889634f;
constexpr size_t MAX_SMEM = 200 * 1024;

__device__ __forceinline__ float softplus_f(float v) { return fmaxf(v, 0.0f) + log1pf(expf(-fabsf(v))); }
__device__ __forceinline__ float decay2(float v) {
    float r;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(v));
    return r;
}

struct Args {
    const float* xz;  // [R][ld]: x at column 0, z at column C
    int ld, C, N, rank, taps, outs;  // outs = rank + 2 N
    const float *filters, *conv_bias;
    const __nv_bfloat16 *w_x, *w_dt;  // [outs][C], [C][rank]
    const float *dt_bias, *A, *D;
    float* state;
    long long stride;  // a slot's floats: the filter's last taps - 1 inputs, then S [C][N]
    const int* row_slot;
    __nv_bfloat16* out;
    int keep_dt;  // whether W_dt's slice fits shared memory beside W_x's
};

// shared memory: W_x's slice [outs][CB + 8] and W_dt's [CB][rank + 8] in bfloat16, u [CB], u rounded [CB],
// partial sums [ranks][outs], their sums [outs]
inline size_t step_smem(int CB, int outs, int rank, int ranks, int keep_dt) {
    return ((size_t)outs * (CB + 8) + (keep_dt ? (size_t)CB * (rank + 8) : 0) + CB) * 2 +
           ((size_t)CB + (size_t)(ranks + 1) * outs) * 4;
}

template <int NPL>  // states a lane holds: N = 4 NPL
__global__ void __launch_bounds__(THREADS) mamba_step_kernel(Args a) {
    extern __shared__ __align__(16) uint8_t smem_raw[];
    cg::cluster_group cluster = cg::this_cluster();
    const int ranks = gridDim.z, rank = blockIdx.z, r = blockIdx.y;
    const int CB = a.C / ranks, c0 = rank * CB, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int WLD = CB + 8, DLD = a.rank + 8;
    __nv_bfloat16* Wx = reinterpret_cast<__nv_bfloat16*>(smem_raw);
    __nv_bfloat16* Wd = Wx + (size_t)a.outs * WLD;
    __nv_bfloat16* us = Wd + (a.keep_dt ? (size_t)CB * DLD : 0);
    float* u = reinterpret_cast<float*>(us + CB);
    float* recv = u + CB;
    float* sums = recv + ranks * a.outs;
    pdl_launch_dependents();
    cluster.barrier_arrive();  // met below: every CTA runs before another writes into its memory
    for (int e = tid; e < a.outs * (CB / 8); e += THREADS) {
        const int o = e / (CB / 8), c = 8 * (e - o * (CB / 8));
        attn::cp_async_16(Wx + o * WLD + c, a.w_x + (size_t)o * a.C + c0 + c, true);
    }
    for (int e = tid; a.keep_dt && e < CB * (a.rank / 8); e += THREADS) {
        const int c = e / (a.rank / 8), j = 8 * (e - c * (a.rank / 8));
        attn::cp_async_16(Wd + c * DLD + j, a.w_dt + (size_t)(c0 + c) * a.rank + j, true);
    }
    attn::cp_async_commit();
    pdl_wait();
    float* slot = a.state + (size_t)a.row_slot[r] * a.stride;
    const int T = a.taps - 1;
    for (int c = 4 * tid; c < CB; c += 4 * THREADS) {
        const int ch = c0 + c;
        float4 y = conv::conv4_at(a.xz, a.ld, 0, ch, nullptr, a.filters, a.taps, slot, a.C, r, 0);
        const float4 b = load4(a.conv_bias + ch);
        y = make_float4(conv::silu_of(y.x + b.x), conv::silu_of(y.y + b.y), conv::silu_of(y.z + b.z), conv::silu_of(y.w + b.w));
        store4(u + c, y);
        store4(us + c, y);
        for (int i = 0; i + 1 < T; ++i) store4(slot + (size_t)i * a.C + ch, load4(slot + (size_t)(i + 1) * a.C + ch));
        if (T > 0) store4(slot + (size_t)(T - 1) * a.C + ch, load4(a.xz + (size_t)r * a.ld + ch));
    }
    attn::cp_async_wait<0>();
    __syncthreads();
    cluster.barrier_wait();
    // this slice's share of W_x u, four outputs a warp at a time
    for (int o0 = 4 * warp; o0 < a.outs; o0 += 4 * WARPS) {
        float acc[4] = {};
        for (int c = 8 * lane; c < CB; c += 256) {
            const uint4 x = *reinterpret_cast<const uint4*>(us + c);
            const __nv_bfloat162* xp = reinterpret_cast<const __nv_bfloat162*>(&x);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                if (o0 + i >= a.outs) break;
                const uint4 w = *reinterpret_cast<const uint4*>(Wx + (o0 + i) * WLD + c);
                const __nv_bfloat162* wp = reinterpret_cast<const __nv_bfloat162*>(&w);
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const float2 p = __bfloat1622float2(xp[k]), q = __bfloat1622float2(wp[k]);
                    acc[i] = fmaf(p.x, q.x, acc[i]);
                    acc[i] = fmaf(p.y, q.y, acc[i]);
                }
            }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
#pragma unroll
            for (int i = 0; i < 4; ++i) acc[i] += __shfl_xor_sync(0xffffffffu, acc[i], o);
        // lane d sends to rank d
        if (lane < ranks) {
            float* to = cluster.map_shared_rank(recv, lane) + rank * a.outs;
#pragma unroll
            for (int i = 0; i < 4; ++i)
                if (o0 + i < a.outs) to[o0 + i] = acc[i];
        }
    }
    cluster.sync();  // every rank's sums are here; nobody reads another's memory after this
    for (int o = tid; o < a.outs; o += THREADS) {
        float s = 0.0f;
        for (int k = 0; k < ranks; ++k) s += recv[k * a.outs + o];
        sums[o] = s;
    }
    __syncthreads();
    const int sub = tid % LPC;
    float B[NPL], Cc[NPL];
#pragma unroll
    for (int i = 0; i < NPL; ++i) {
        B[i] = sums[a.rank + sub + LPC * i];
        Cc[i] = sums[a.rank + a.N + sub + LPC * i];
    }
    for (int c = tid / LPC; c < CB; c += THREADS / LPC) {  // CB a multiple of the warp's channels: whole warps
        const int ch = c0 + c;
        float* Sg = slot + (size_t)T * a.C + (size_t)ch * a.N;
        float S[NPL], al[NPL];
#pragma unroll
        for (int i = 0; i < NPL; ++i) {
            S[i] = Sg[sub + LPC * i];
            al[i] = a.A[(size_t)ch * a.N + sub + LPC * i] * LOG2E;
        }
        const float z = a.xz[(size_t)r * a.ld + a.C + ch], bias = a.dt_bias[ch], d = a.D[ch];
        float dt = 0.0f;
        const __nv_bfloat16* wrow = a.keep_dt ? Wd + c * DLD : a.w_dt + (size_t)ch * a.rank;
        for (int j = 8 * sub; j < a.rank; j += 8 * LPC) {
            const uint4 w = *reinterpret_cast<const uint4*>(wrow + j);
            const __nv_bfloat162* wp = reinterpret_cast<const __nv_bfloat162*>(&w);
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const float2 q = __bfloat1622float2(wp[k]);
                dt = fmaf(q.x, __bfloat162float(__float2bfloat16_rn(sums[j + 2 * k])), dt);
                dt = fmaf(q.y, __bfloat162float(__float2bfloat16_rn(sums[j + 2 * k + 1])), dt);
            }
        }
#pragma unroll
        for (int o = 1; o < LPC; o <<= 1) dt += __shfl_xor_sync(0xffffffffu, dt, o);
        dt = softplus_f(dt + bias);
        const float xv = u[c], dx = dt * xv;
        float y = 0.0f;
#pragma unroll
        for (int i = 0; i < NPL; ++i) {
            S[i] = fmaf(decay2(dt * al[i]), S[i], dx * B[i]);
            y = fmaf(S[i], Cc[i], y);
            Sg[sub + LPC * i] = S[i];
        }
#pragma unroll
        for (int o = 1; o < LPC; o <<= 1) y += __shfl_xor_sync(0xffffffffu, y, o);
        if (sub == 0) a.out[(size_t)r * a.C + ch] = __float2bfloat16_rn(fmaf(d, xv, y) * conv::silu_of(z));
    }
}

template <int NPL>
int launch(Args a, int R, cudaStream_t s) {
    auto kernel = mamba_step_kernel<NPL>;
    // sixteen CTAs a sequence where the device holds such a cluster for each at a time, else eight; not in two
    // waves (width 2,048: 24.7 us for the layer with six sequences and 35.1 with eight, 29.5 and 28.9 with
    // three launches; width 1,024: 20.0 with eight and 27.0 with sixteen, 21.3 and 22.6)
    for (int ranks = 16; ranks >= 8; ranks /= 2) {
        if (a.C % (ranks * 8 * (32 / LPC))) continue;  // slices of whole warps' channels, 16 bytes a copy
        a.keep_dt = step_smem(a.C / ranks, a.outs, a.rank, ranks, 1) <= MAX_SMEM;
        const size_t smem = step_smem(a.C / ranks, a.outs, a.rank, ranks, a.keep_dt);
        if (smem > MAX_SMEM) continue;
        cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return (int)e;
        if (ranks > 8 && cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess) {
            cudaGetLastError();
            continue;
        }
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(1, 1, ranks);
        cfg.blockDim = dim3(THREADS);
        cfg.dynamicSmemBytes = smem;
        cudaLaunchAttribute at[1];
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = 1;
        at[0].val.clusterDim.y = 1;
        at[0].val.clusterDim.z = ranks;
        cfg.attrs = at;
        cfg.numAttrs = 1;
        int n = 0;  // clusters the device holds at a time
        const bool fits = cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) == cudaSuccess && n >= R;
        cudaGetLastError();  // a refusal is an answer, not an error to carry on
        if (!fits) continue;
        e = rfx::launch(kernel, dim3(1, R, ranks), dim3(THREADS), smem, s, ranks, a);
        return e == cudaSuccess ? 0 : (int)e;
    }
    return RFX_ERR_UNSUPPORTED;
}

}  // namespace

// One row a sequence: xz float32 [R][ld] = [x | z | ..], filters [taps][C], w_x bfloat16 [rank + 2 N][C] (rows
// dt, B, C), w_dt bfloat16 [C][rank], A [C][N] (negative), state [slots][stride]: the filter's last taps - 1
// inputs, oldest first, then S [C][N]; both move on.  out bfloat16 [R][C] = y * silu(z).  N 4, 8, 16 or 32;
// RFX_ERR_UNSUPPORTED, before anything has run, for other sizes, more sequences than the device holds clusters
// at a time, and what is not on 16 bytes.
extern "C" int rfx_mamba_step(const float* xz, int ld, int C, int N, int rank, int taps, const float* filters,
                              const float* conv_bias, const void* w_x, const void* w_dt, const float* dt_bias,
                              const float* A, const float* D, float* state, long long stride, const int* row_slot, int R,
                              void* out, void* stream) {
    if (R <= 0) return 0;
    if (C <= 0 || N <= 0 || rank <= 0 || taps <= 0 || ld < 2 * C) return RFX_ERR_BAD_ARG;
    if (rank % 8 || ld % 4 || stride % 4 || C % 8 || taps > conv::MAX_TAPS || R > 65535 || !conv_bias || !dt_bias || !D ||
        ((reinterpret_cast<uintptr_t>(xz) | reinterpret_cast<uintptr_t>(filters) | reinterpret_cast<uintptr_t>(conv_bias) |
          reinterpret_cast<uintptr_t>(w_x) | reinterpret_cast<uintptr_t>(w_dt) | reinterpret_cast<uintptr_t>(state)) & 15))
        return RFX_ERR_UNSUPPORTED;
    Args a{xz, ld, C, N, rank, taps, rank + 2 * N, filters, conv_bias, (const __nv_bfloat16*)w_x,
           (const __nv_bfloat16*)w_dt, dt_bias, A, D, state, stride, row_slot, (__nv_bfloat16*)out, 0};
    cudaStream_t s = (cudaStream_t)stream;
    if (N == 4) return launch<1>(a, R, s);
    if (N == 8) return launch<2>(a, R, s);
    if (N == 16) return launch<4>(a, R, s);
    if (N == 32) return launch<8>(a, R, s);
    return RFX_ERR_UNSUPPORTED;
}
