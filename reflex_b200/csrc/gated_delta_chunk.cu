// The gated delta rule (gated_delta.cu) for steps that bring a sequence many rows: sixteen
// rows at a time, as products on the tensor cores.
//
// With S0 the memory before a chunk of rows, c_i the product of the chunk's decays up to
// row i, r_ij that of the rows after j up to i, and L_ij = r_ij (k_i.k_j) for j < i,
//     u = T (v - c * (K S0)),     T = (I + diag(beta) L)^-1 diag(beta)
//     o = c * (Q S0) + M u,       M_ij = r_ij (q_i.k_j) for j <= i
//     S0 <- c_last S0 + K^T (r_last * u)
// which is the row-by-row rule with the rows' dependence on one another solved once per
// chunk and head (T, by forward substitution), independently of the memory and of every other
// chunk: rfx_gated_delta_chunk_prep does that for all chunks side by side, and
// rfx_gated_delta_chunk walks the chunks with the products.
//
// The memory stays 32-bit (the products' accumulators are the memory itself); products are
// those of split_mma.cuh.  The true 32-bit path takes the row-by-row kernel instead.
//
// S^T [16 columns x channels] of a warp is an accumulator tile row of mma.sync m16n8k8, and the
// same registers are the left operand of the next chunk's products; likewise u^T.
#include "attn_mma.cuh"
#include "common.cuh"
#include "fma_tiles.cuh"
#include "split_mma.cuh"

namespace {

constexpr int CH = 16;            // rows of a chunk
constexpr int TLD = 24;           // row stride of T and M: a fragment's 8-byte loads meet all banks
// per chunk and head: T [16][TLD], M [16][TLD], c [16], r_last [16], c_last and padding
constexpr int COEF = 2 * CH * TLD + 2 * CH + 4;

using rfx::Left;
using rfx::left_of;
using rfx::product3;

// Chunk c of sequence `seq`, whose first row of the step is row0: its place among all chunks
// (a sequence of n rows has ceil(n / 16), so no two places meet; at most R / 16 + sequences).
__device__ __forceinline__ size_t chunk_place(int row0, int seq, int c) { return (size_t)row0 / CH + seq + c; }

// A block a (chunk, query/key head): the products between the chunk's rows once, by 32-bit multiply-adds,
// each warp some of the channels (four by four results a lane, of [k; q] by k); then per value head of
// the group (eight at a time) T, M and the decays' products.  Bound by the steps' latencies: 45 us for 4,096
// rows of 16 heads of 128 with two value heads each (53 with the decays' products by pairs of rows).  (A thread a pair of rows, bound by its reads of shared
// memory: 66; on the tensor cores with operands split in two 51, and the results 1.4 times as far from 64 bits.)
constexpr int PREP_WARPS = CH * CH / 32, PREP_HEADS = 8;
__host__ __device__ constexpr int prep_ld(int d) { return (d + 15) / 16 * 16 + 4; }  // an odd number of 16 bytes
__global__ void __launch_bounds__(CH * CH, 3)
gated_delta_chunk_prep_kernel(const float* __restrict__ qkv, const float* __restrict__ gates,
                              const int* __restrict__ seq_row0, float* __restrict__ coef, int H, int G, int d, int dv) {
    extern __shared__ __align__(16) float sm[];
    __shared__ float L[PREP_HEADS][CH][CH + 1], bs[PREP_HEADS][CH];  // L: the decays' products until it is made
    rfx::pdl_prologue();
    const int seq = blockIdx.y, kvh = blockIdx.z;
    const int row0 = seq_row0[seq], row1 = seq_row0[seq + 1];
    const int first = row0 + blockIdx.x * CH, n = min(CH, row1 - first);
    if (n <= 0) return;
    const int C = 2 * G * d + H * dv, LD = prep_ld(d), c4 = (LD - 4) / 4;
    float *ks = sm, *qs = sm + CH * LD;
    float4* part = reinterpret_cast<float4*>(sm + 2 * CH * LD);  // [warp][four rows][lane]
    const int tid = threadIdx.x, i = tid / CH, j = tid % CH;
    const int warp = tid >> 5, lane = tid & 31;
    for (int r = warp; r < CH; r += PREP_WARPS) {  // rows and channels that are not there as zeros
        const float* src = qkv + (size_t)(first + r) * C + kvh * d;
        for (int c = lane; c < c4; c += 32) {
            const bool ok = r < n && 4 * c < d;
            attn::cp_async_16(qs + r * LD + 4 * c, ok ? src + 4 * c : qkv, ok);
            attn::cp_async_16(ks + r * LD + 4 * c, ok ? src + G * d + 4 * c : qkv, ok);
        }
    }
    attn::cp_async_commit();
    const int per = H / G;
    auto place = [&](int h) { return coef + (chunk_place(row0, seq, blockIdx.x) * H + kvh * per + h) * COEF; };
    // A warp a head: lane j has the product of the decays after row j, down the rows, lane CH that of all
    auto decays = [&](int h0) {
        const int h = h0 + warp;
        if (h >= per) return;
        const float* src = gates + (size_t)(first + lane) * 2 * H + kvh * per + h;
        const float g = lane < n ? src[0] : 1.0f;
        if (lane < CH) bs[warp][lane] = lane < n ? src[H] : 0.0f;
        float* o = place(h) + 2 * CH * TLD;
        float r = 1.0f;
#pragma unroll
        for (int a = 0; a < CH; ++a) {
            const float next = __shfl_sync(0xffffffffu, g, a);
            if (lane == CH || a > lane) r *= next;
            if (lane < CH) L[warp][a][lane] = r;
            if (lane == CH) o[a] = r;
        }
        if (lane < CH) o[CH + lane] = r;
        if (lane == CH) o[2 * CH] = r;
    };
    decays(0);
    attn::cp_async_wait<0>();
    __syncthreads();
    float acc[4][4] = {};  // rows lane / 4 + 8 i of [k; q], columns lane % 4 + 4 j
    for (int s = warp; s < c4 / 4; s += PREP_WARPS)
        rfx::product_along<4>(acc, ks + (lane >> 2) * LD + 16 * s, 8 * LD, ks + (lane & 3) * LD + 16 * s, 4 * LD, 1);
#pragma unroll
    for (int t = 0; t < 4; ++t) part[(warp * 4 + t) * 32 + lane] = make_float4(acc[t][0], acc[t][1], acc[t][2], acc[t][3]);
    __syncthreads();
    float kk = 0.0f, qk = 0.0f;
    {
        const float* p = reinterpret_cast<const float*>(part) + 4 * ((i / 8) * 32 + (i % 8) * 4 + j % 4) + j / 4;
#pragma unroll
        for (int w = 0; w < PREP_WARPS; ++w) {
            kk += p[w * 4 * 128];
            qk += p[(w * 4 + 2) * 128];
        }
    }
    for (int h0 = 0; h0 < per; h0 += PREP_HEADS) {
        const int heads = min(PREP_HEADS, per - h0);
        if (h0) {
            __syncthreads();  // L and bs of the heads before have been read
            decays(h0);
            __syncthreads();
        }
        float* out = place(h0);
        for (int hh = 0; hh < heads; ++hh) {
            const float r = L[hh][i][j];
            L[hh][i][j] = j < i ? bs[hh][i] * (r * kk) : 0.0f;
            out[(size_t)hh * COEF + CH * TLD + i * TLD + j] = j <= i ? r * qk : 0.0f;
        }
        __syncthreads();
        if (warp < heads && lane < CH) {  // a warp a head: column `lane` of T, row by row
            float t[CH];  // (each row known is taken off all later ones: fifteen multiply-adds deep, not 120)
#pragma unroll
            for (int a = 0; a < CH; ++a) t[a] = a == lane ? bs[warp][a] : 0.0f;
#pragma unroll
            for (int l = 0; l < CH; ++l) {
                out[(size_t)warp * COEF + l * TLD + lane] = t[l];
#pragma unroll
                for (int a = l + 1; a < CH; ++a) t[a] = fmaf(-L[warp][a][l], t[l], t[a]);
            }
        }
    }
}

// u = T w for the sixteen columns of a fragment's rows, w = v - c (K S0).  A sum's three passes go to
// places of their own and meet at the end: nothing else runs beside this chain.
struct Solved {
    float u[2][4];
};
template <typename Total>
__device__ __forceinline__ Solved solve(const float* cf, const float* v, int VLD, int l4, int j, const float2 (&ci)[2],
                                        Total&& total) {
    Left a[2];
#pragma unroll
    for (int t = 0; t < 2; ++t) {
        float x[4];
        total(t, x);
        const float* vt = v + 8 * t * VLD;
        x[0] = fmaf(-ci[t].x, x[0], vt[0]);
        x[1] = fmaf(-ci[t].y, x[1], vt[VLD]);
        x[2] = fmaf(-ci[t].x, x[2], vt[8]);
        x[3] = fmaf(-ci[t].y, x[3], vt[VLD + 8]);
        a[t] = left_of(x);
    }
    // T is lower triangular: its rows 0..7 meet rows 0..7 alone
    const float2 b00 = *reinterpret_cast<const float2*>(cf + l4 * TLD + 2 * j);
    const float2 b10 = *reinterpret_cast<const float2*>(cf + (8 + l4) * TLD + 2 * j);
    const float2 b11 = *reinterpret_cast<const float2*>(cf + (8 + l4) * TLD + 8 + 2 * j);
    float part[3][2][4] = {};
    auto passes = [&](int n, const Left& l, const float2& b) {
        const rfx::Split x = rfx::split(b.x), y = rfx::split(b.y);
        rfx::mma_tf32(part[0][n], l.lo, x.hi, y.hi);
        rfx::mma_tf32(part[1][n], l.hi, x.lo, y.lo);
        rfx::mma_tf32(part[2][n], l.hi, x.hi, y.hi);
    };
    passes(1, a[0], b10);
    passes(0, a[0], b00);
    passes(1, a[1], b11);
    Solved r;
#pragma unroll
    for (int n = 0; n < 2; ++n)
#pragma unroll
        for (int i = 0; i < 4; ++i) r.u[n][i] = (part[0][n][i] + part[1][n][i]) + part[2][n][i];
    return r;
}

// Four warps own sixteen value columns, a quarter of the key channels each (NT eights; channels
// beyond d are zeros); a block has up to four such groups, and helpers that bring the chunks, of whom
// the first ones, one a group, also make and write its results.  The four quarters' partial sums of
// K S0 and Q S0 meet in shared memory in their order; u is solved by every warp of the group (each of
// the four needs it for its channels, the helper for o).
//
// What bounds the walk is a chunk's chain: K S0, the partial sums' way through shared memory, u, the
// memory's step (4,096 rows of 32 heads of 128 x 128: 440 us, 1.7 us a chunk; 507 with the copies and
// the results in the same warps).  Helpers copy asynchronously, 16 bytes a lane, two chunks ahead; a
// warp alone issues such copies slowly, so there are several.  The one barrier a chunk that the partial
// sums need also says that the next chunk has landed and that the last one's buffer is free.
template <int NT>
__global__ void __launch_bounds__(768)
gated_delta_chunk_kernel(const float* __restrict__ qkv, const float* __restrict__ coef, float* __restrict__ state,
                         long long state_stride, long long state_off, const int* __restrict__ seq_slot,
                         const int* __restrict__ seq_row0, float* __restrict__ out, int H, int G, int d, int dv,
                         int cols, int stages) {
    constexpr int DP = 32 * NT, LDK = DP + 8;
    extern __shared__ __align__(16) float sm[];
    const int seq = blockIdx.x, h = blockIdx.y, c_first = blockIdx.z * cols;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int groups = cols / 16, n_warps = groups * 4;  // (the helpers come after these)
    const int l4 = lane >> 2, j = lane & 3;
    const int VLD = cols + 4, buf_floats = 2 * CH * LDK + COEF + CH * VLD;
    const int C = 2 * G * d + H * dv, kvh = h / (H / G);
    const bool helps = warp >= n_warps;
    const int helper = warp - n_warps, helpers = (blockDim.x >> 5) - n_warps;
    const int grp = helps ? helper : warp >> 2, quarter = warp & 3;
    // partial sums: [parity][group][tile of D][quarter][lane] four floats
    float4* red = reinterpret_cast<float4*>(sm + stages * buf_floats);
    // everything a copy does not reach stays zero: channels beyond d, rows beyond the first chunks'
    for (int e = threadIdx.x; e < stages * buf_floats; e += blockDim.x) sm[e] = 0.0f;
    __syncthreads();
    rfx::pdl_prologue();
    const int row0 = seq_row0[seq], row1 = seq_row0[seq + 1];
    const int n_chunks = (row1 - row0 + CH - 1) / CH;
    const int d4 = d / 4, v4 = min(cols, dv - c_first) / 4;
    const int cl = grp * 16, col = c_first + cl;
    const bool live = col < dv;  // dv is a multiple of sixteen: a group's columns all or none
    const auto sums = [&](int c) {  // of chunk c, this group's
        return red + (size_t)((c & 1) * groups + grp) * 4 * 4 * 32 + lane;
    };
    const auto total = [&](const float4* all4, int n, float (&t)[4]) {
        const float4 p0 = all4[n * 128], p1 = all4[n * 128 + 32], p2 = all4[n * 128 + 64], p3 = all4[n * 128 + 96];
        t[0] = (p0.x + p1.x) + (p2.x + p3.x);
        t[1] = (p0.y + p1.y) + (p2.y + p3.y);
        t[2] = (p0.z + p1.z) + (p2.z + p3.z);
        t[3] = (p0.w + p1.w) + (p2.w + p3.w);
    };
    const auto next = [&](int b) { return b + 1 == stages ? 0 : b + 1; };
    // of all warps, from either side's code
    const auto meet = [&]() { asm volatile("barrier.cta.sync 1, %0;" ::"r"((int)blockDim.x) : "memory"); };
    if (helps) {
        int to = 0;  // the buffer the next chunk goes to
        auto fetch = [&](int c) {
            if (c < n_chunks) {
                float* base = sm + to * buf_floats;
                const int first = row0 + c * CH, n = min(CH, row1 - first);
                const float* src = qkv + (size_t)(first + helper) * C + 4 * lane;
                for (int r = helper; r < n; r += helpers, src += (size_t)helpers * C) {
                    for (int e = lane; e < d4; e += 32) {
                        attn::cp_async_16(base + r * LDK + 4 * e, src + G * d + kvh * d + 4 * (e - lane), true);
                        attn::cp_async_16(base + (CH + r) * LDK + 4 * e, src + kvh * d + 4 * (e - lane), true);
                    }
                    if (lane < v4)
                        attn::cp_async_16(base + 2 * CH * LDK + COEF + r * VLD + 4 * lane, src + 2 * G * d + h * dv + c_first, true);
                }
                const float* cf = coef + (chunk_place(row0, seq, c) * H + h) * COEF;
                for (int e = helper * 32 + lane; e < COEF / 4; e += helpers * 32)
                    attn::cp_async_16(base + 2 * CH * LDK + 4 * e, cf + 4 * e, true);
            }
            attn::cp_async_commit();
            to = next(to);
        };
        for (int c = 0; c < stages - 1; ++c) fetch(c);
        if (stages == 4) attn::cp_async_wait<2>();
        else attn::cp_async_wait<1>();
        meet();  // the first chunk
        int buf = 0;
        for (int c = 0; c < n_chunks; ++c) {
            const float *cf = sm + buf * buf_floats + 2 * CH * LDK, *vs = cf + COEF;
            buf = next(buf);
            if (stages == 4) attn::cp_async_wait<1>();
            else attn::cp_async_wait<0>();
            meet();  // the group's sums; the next chunk; the last chunk's buffer is free
            fetch(c + stages - 1);
            if (grp >= groups || !live) continue;
            const float4* all4 = sums(c);
            const float2 ci[2] = {*reinterpret_cast<const float2*>(cf + 2 * CH * TLD + 2 * j),
                                  *reinterpret_cast<const float2*>(cf + 2 * CH * TLD + 8 + 2 * j)};
            const Solved u = solve(cf, vs + 2 * j * VLD + cl + l4, VLD, l4, j, ci,
                                   [&](int t, float (&x)[4]) { total(all4, t, x); });
            float O[2][4];
#pragma unroll
            for (int t = 0; t < 2; ++t) {
                total(all4, 2 + t, O[t]);
                O[t][0] *= ci[t].x;
                O[t][1] *= ci[t].y;
                O[t][2] *= ci[t].x;
                O[t][3] *= ci[t].y;
            }
#pragma unroll
            for (int t = 0; t < 2; ++t) {
                const Left a = left_of(u.u[t]);
                float2 b[2];
#pragma unroll
                for (int n = 0; n < 2; ++n)
                    b[n] = *reinterpret_cast<const float2*>(cf + CH * TLD + (8 * n + l4) * TLD + 8 * t + 2 * j);
                if (t == 0) product3<2>(O, a, b);
                else product3<1>(*reinterpret_cast<float(*)[1][4]>(&O[1]), a, *reinterpret_cast<const float2(*)[1]>(&b[1]));
            }
            const int left = row1 - row0 - c * CH;
            const size_t ld = (size_t)H * dv;
            float* o = out + (size_t)(row0 + c * CH) * ld + (size_t)h * dv + col + l4;
#pragma unroll
            for (int t = 0; t < 2; ++t) {
                const int r = 8 * t + 2 * j;
                if (r < left) {
                    o[r * ld] = O[t][0];
                    o[r * ld + 8] = O[t][2];
                }
                if (r + 1 < left) {
                    o[(r + 1) * ld] = O[t][1];
                    o[(r + 1) * ld + 8] = O[t][3];
                }
            }
        }
        return;
    }
    const int ch0 = quarter * 8 * NT;  // the warp's first channel
    float* Sg = state + (size_t)seq_slot[seq] * state_stride + state_off + ((size_t)h * dv + (live ? col : 0)) * d + ch0;
    float S[NT][4];
#pragma unroll
    for (int s = 0; s < NT; ++s) {
        float2 x = make_float2(0.0f, 0.0f), y = x;
        if (live && ch0 + 8 * s < d) {
            x = *reinterpret_cast<const float2*>(Sg + (size_t)l4 * d + 8 * s + 2 * j);
            y = *reinterpret_cast<const float2*>(Sg + (size_t)(l4 + 8) * d + 8 * s + 2 * j);
        }
        S[s][0] = x.x; S[s][1] = x.y; S[s][2] = y.x; S[s][3] = y.y;
    }
    meet();  // the first chunk
    int buf = 0;
    for (int c = 0; c < n_chunks; ++c) {
        const float* base = sm + buf * buf_floats;
        buf = next(buf);
        const float *ks = base + ch0, *cf = base + 2 * CH * LDK, *vs = cf + COEF;
        // this quarter's K S0 and Q S0, transposed: [0], [1] the k rows 0..7 and 8..15, [2], [3] the q rows
        float D[4][4] = {};
#pragma unroll
        for (int s = 0; s < NT; ++s) {
            const Left a = left_of(S[s]);
            float2 b[4];
#pragma unroll
            for (int n = 0; n < 4; ++n)
                b[n] = *reinterpret_cast<const float2*>(ks + (8 * n + l4) * LDK + 8 * s + 2 * j);
            product3<4>(D, a, b);
        }
        const float4* all4 = sums(c);
        float4* mine = const_cast<float4*>(all4) + quarter * 32;
#pragma unroll
        for (int n = 0; n < 4; ++n) mine[n * 4 * 32] = make_float4(D[n][0], D[n][1], D[n][2], D[n][3]);
        const float2 ci[2] = {*reinterpret_cast<const float2*>(cf + 2 * CH * TLD + 2 * j),
                              *reinterpret_cast<const float2*>(cf + 2 * CH * TLD + 8 + 2 * j)};
        const float all = cf[2 * CH * TLD + 2 * CH];
#pragma unroll
        for (int s = 0; s < NT; ++s)
#pragma unroll
            for (int i = 0; i < 4; ++i) S[s][i] *= all;
        meet();  // the group's sums; the next chunk; the last chunk's buffer is free
        const Solved u = solve(cf, vs + 2 * j * VLD + cl + l4, VLD, l4, j, ci,
                               [&](int t, float (&x)[4]) { total(all4, t, x); });
        // the memory's step: K^T (r_last * u)
#pragma unroll
        for (int t = 0; t < 2; ++t) {
            const float2 rl = *reinterpret_cast<const float2*>(cf + 2 * CH * TLD + CH + 8 * t + 2 * j);
            const float w[4] = {u.u[t][0] * rl.x, u.u[t][1] * rl.y, u.u[t][2] * rl.x, u.u[t][3] * rl.y};
            const Left a = left_of(w);
            const float* k = ks + (8 * t + 2 * j) * LDK + l4;
            float2 b[NT];
#pragma unroll
            for (int s = 0; s < NT; ++s) b[s] = make_float2(k[8 * s], k[LDK + 8 * s]);
            product3<NT>(S, a, b);
        }
    }
    if (!live) return;
#pragma unroll
    for (int s = 0; s < NT; ++s)
        if (ch0 + 8 * s < d) {
            *reinterpret_cast<float2*>(Sg + (size_t)l4 * d + 8 * s + 2 * j) = make_float2(S[s][0], S[s][1]);
            *reinterpret_cast<float2*>(Sg + (size_t)(l4 + 8) * d + 8 * s + 2 * j) = make_float2(S[s][2], S[s][3]);
        }
}

template <int NT>
int launch_chunk(const float* qkv, const float* coef, float* state, long long state_stride, long long state_off,
                 const int* seq_slot, const int* seq_row0, int n_seq, float* out, int H, int G, int d, int dv,
                 cudaStream_t s) {
    // value columns a block owns, sixteen a group of four warps; fewer while the blocks do not fill the SMs
    int cols = 64;
    while (cols > 16 && (cols / 2 >= dv ||
                         (long long)n_seq * H * ((dv + cols - 1) / cols) < rfx::sm_count() * 3LL / 4))
        cols /= 2;
    const size_t stage = (size_t)(2 * CH * (32 * NT + 8) + COEF + CH * (cols + 4)) * sizeof(float);
    const size_t red = (size_t)2 * (cols / 16) * 4 * 4 * 32 * sizeof(float4);
    // four buffers (the chunk in use, the next, two on their way) where a block has its SM to itself,
    // else three
    int stages = (long long)n_seq * H * ((dv + cols - 1) / cols) <= rfx::sm_count() ? 4 : 3;
    if (stages * stage + red > 220 * 1024) stages = 3;
    const size_t smem = stages * stage + red;
    if (smem > 220 * 1024) return RFX_ERR_UNSUPPORTED;
    auto kernel = gated_delta_chunk_kernel<NT>;
    if (smem > 48 * 1024) {
        cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return (int)e;
    }
    dim3 grid(n_seq, H, (dv + cols - 1) / cols);
    // (two helpers for 32 columns: 582 us for 4,096 rows of 32 heads of 128, four 464, eight 440, sixteen 444)
    const int helpers = cols == 16 ? 4 : 8;
    RFX_LAUNCH(kernel, grid, cols * 8 + helpers * 32, smem, s, qkv, coef, state, state_stride, state_off, seq_slot, seq_row0,
               out, H, G, d, dv, cols, stages);
    return 0;
}

}  // namespace

// Floats of `coef` that steps of R rows in n_seq sequences need.
extern "C" long long rfx_gated_delta_chunk_floats(int R, int n_seq, int H) {
    return (long long)(R / CH + n_seq) * H * COEF;
}

// T, M and the decays' products of every chunk (chunks counted from each sequence's first row of the
// step).  `max_rows`: the most rows any sequence brings.  d a multiple of 4, `qkv` 16-byte aligned.
extern "C" int rfx_gated_delta_chunk_prep(const float* qkv, const float* gates, const int* seq_row0, int n_seq,
                                          float* coef, int H, int G, int d, int dv, int max_rows, void* stream) {
    if (n_seq <= 0 || max_rows <= 0) return 0;
    if (H <= 0 || G <= 0 || H % G || d <= 0 || dv <= 0) return RFX_ERR_BAD_ARG;
    const size_t smem = (size_t)2 * CH * prep_ld(d) * sizeof(float) + PREP_WARPS * 4 * 32 * sizeof(float4);
    if (d % 4 || dv % 4 || (size_t)2 * CH * (d + 4) * sizeof(float) > 48 * 1024 || n_seq > 65535 || G > 65535) return RFX_ERR_UNSUPPORTED;
    dim3 grid((max_rows + CH - 1) / CH, n_seq, G);
    if (smem + 12 * 1024 > 48 * 1024) {
        cudaError_t e = cudaFuncSetAttribute(gated_delta_chunk_prep_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return (int)e;
    }
    RFX_LAUNCH(gated_delta_chunk_prep_kernel, grid, CH * CH, smem, (cudaStream_t)stream, qkv, gates, seq_row0, coef, H,
               G, d, dv);
    return 0;
}

// The recurrence over the step's rows, chunk by chunk.  d a multiple of 8 up to 256, dv of 16;
// the running state as rfx_gated_delta_scan keeps it.
extern "C" int rfx_gated_delta_chunk(const float* qkv, const float* coef, float* state, long long state_stride,
                                     long long state_off, const int* seq_slot, const int* seq_row0, int n_seq,
                                     float* out, int H, int G, int d, int dv, void* stream) {
    if (n_seq <= 0) return 0;
    if (H <= 0 || G <= 0 || H % G || d <= 0 || dv <= 0) return RFX_ERR_BAD_ARG;
    if ((state_stride | state_off) & 3 || (reinterpret_cast<uintptr_t>(state) & 15)) return RFX_ERR_BAD_ARG;
    if (d % 8 || dv % 16 || d > 256 || H > 65535 ||
        ((reinterpret_cast<uintptr_t>(qkv) | reinterpret_cast<uintptr_t>(coef)) & 15))
        return RFX_ERR_UNSUPPORTED;
    cudaStream_t s = (cudaStream_t)stream;
#define RFX_CHUNK(N)                                                                                              \
    return launch_chunk<N>(qkv, coef, state, state_stride, state_off, seq_slot, seq_row0, n_seq, out, H, G, d, dv, \
                           s)
    if (d <= 32) RFX_CHUNK(1);
    if (d <= 64) RFX_CHUNK(2);
    if (d <= 96) RFX_CHUNK(3);
    if (d <= 128) RFX_CHUNK(4);
    if (d <= 192) RFX_CHUNK(6);
    RFX_CHUNK(8);
#undef RFX_CHUNK
}
