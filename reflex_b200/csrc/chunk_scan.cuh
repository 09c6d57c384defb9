// Recurrences S <- decay S + weight k v^T, y = S^T q with one decay and one weight a head and
// row (ssd.cu, mlstm.cu) over the many rows of a prompt, 64 rows at a time and all chunks side by
// side, as products of 32-bit multiply-adds.
//
//   chunk_state_kernel   what each chunk adds to the memory, from zero: sum_s W_s k_s v_s^T
//   chunk_carry_kernel   the memory before each chunk, chunk after chunk, element by element; the
//                        running state's start and end
//   chunk_out_kernel     a chunk's rows: alpha_t (q_t . S) + sum_{s<=t} w_ts (q_t . k_s) v_s; the policy's
//                        running number after a sequence's last chunk (every block of the carry reads the
//                        number before the first one, and nothing orders those blocks)
//
// W, alpha and w come from the policy (which recurrence): products of decays as exponentials of
// differences of their running logarithms.  Those are summed in 64 bits from the chunk's first row
// and kept as two 32-bit numbers each, so that the difference of neighbours is as exact as 32 bits
// allow however far the sum has run.
//
// A walk through the rows has one chain of dependent steps a head and leaves most SMs without
// work; chunks cost the memory's way out and back (heads x N x P floats each) and about twice the
// arithmetic.  A prompt of 2,048 rows: 1.2 ms walking and 0.14 ms in chunks for 32 heads of 64 x 128
// (42 us the chunks' sums, 20 the carry, 80 the rows), 0.76 and 0.15 ms for 8 of 128 x 256 (49, 30 and
// 73); the carry is bound by L2, the other two issue on half of the cycles (sixteen warps an SM, shared
// memory half busy).  64 rows: with 32 the memories' traffic doubles, with 128 the products inside the
// chunk do and a block no longer shares its SM.
//
// The same products on the tensor cores, operands split in two parts of 11 bits, took 30 + 20 + 75 and
// 35 + 27 + 65 us, but are 3 to 15 times as far from 64 bits as the walk (1.5e-6 against 1.1e-7 for the
// first shape's results, 3.8e-7 against 7e-8 for its state): 1.2e-7 and 7e-8 here, 1.2e-7 and 7e-8 to
// 1.1e-7 for the second shape, whose chunkwise form on CUDA cores stands at 6e-7 and 1e-6.
//
// A policy `Pol` gives: q, k, v rows (float32, 16-byte aligned, counts in fours), `heads`, `per`
// (heads per q/k head), N (elements of q and k, at most 128), P (elements of v) and the functions
// named below.  A long step goes through a bounded scratch in several rounds (chunk_plan.cuh).
#pragma once

#include "attn_mma.cuh"
#include "chunk_plan.cuh"
#include "common.cuh"
#include "fma_tiles.cuh"

namespace chunk {

using namespace rfx;

constexpr int L = 64;     // rows of a chunk
constexpr int PT = 64;    // elements of v a block takes at a time
constexpr int VLD = PT + 4, WLD = L + 4;  // row strides of v's tile and of the rows' weights
constexpr int THREADS = 256;

struct Step {
    const int* seq_slot;
    const int* seq_row0;
    Round round;
    float* scratch;  // [place][head][P][N] (+ [N] with a normaliser): a chunk's own sum, then the memory before it
    float4* aux;     // [place][head]: what the carry needs of a chunk
    float* before;   // [place][head]: the policy's running number before the chunk
    float4* rows;    // [place][head][L][RECORDS]: the policy's records of the chunk's rows
};

struct Rows {
    int first, n;  // the chunk's first row and how many it has
    bool last;     // of its sequence's in the launch's round
    size_t place;
};
__device__ __forceinline__ Rows rows_of(const Step& s, int seq, int c) {
    const int row0 = s.seq_row0[seq], from = row0 + s.round.seg * s.round.seg_rows;
    const int to = min(s.seq_row0[seq + 1], from + s.round.seg_rows);
    const int first = from + c * L;
    return {first, min(L, to - first), to - first <= L, place_in(s.round, L, row0, seq, c)};
}

// A tile of 64 rows of 4 * c4 floats, rows from n on and columns from n4 (in fours) on zero.  SPREAD: row
// r lies at 16 (r % 4) + r / 4, so that the threads that own four neighbouring rows each read, row by
// row, rows side by side (an odd number of 16 bytes apart: eight of them meet all banks).
template <bool SPREAD>
__device__ __forceinline__ void load_tile(float* dst, int ld, const float* src, size_t src_ld, int n, int c4, int n4) {
    auto at = [&](int r) { return dst + (SPREAD ? (r & 3) * 16 + (r >> 2) : r) * ld; };
    if (THREADS % c4 == 0) {  // a thread keeps its column: no division a piece
        const int c = threadIdx.x % c4, step = THREADS / c4;
        int r = threadIdx.x / c4;
        const float* s = src + (size_t)r * src_ld + 4 * c;
        const int live = c < n4 ? n : 0;
        for (; r < 64; r += step, s += (size_t)step * src_ld) attn::cp_async_16(at(r) + 4 * c, r < live ? s : src, r < live);
    } else {
        for (int e = threadIdx.x; e < 64 * c4; e += THREADS) {
            const int r = e / c4, c = e - r * c4;
            const bool ok = r < n && c < n4;
            attn::cp_async_16(at(r) + 4 * c, ok ? src + (size_t)r * src_ld + 4 * c : src, ok);
        }
    }
}

// A block a (chunk, head, PT elements of v): the chunk's own sum, [P][N].
template <class Pol>
__global__ void __launch_bounds__(THREADS, 2) chunk_state_kernel(Pol pol, Step st) {
    extern __shared__ __align__(16) float sm[];
    __shared__ float wl[L];
    rfx::pdl_prologue();
    const int seq = st.round.seq0 + blockIdx.y;
    const Rows ch = rows_of(st, seq, blockIdx.x);
    if (ch.n <= 0) return;
    const int ptiles = (pol.P + PT - 1) / PT, h = blockIdx.z / ptiles, p0 = (blockIdx.z - h * ptiles) * PT;
    const bool wide = pol.N > 64;
    const int ldk = wide ? 132 : 68;
    float *Vs = sm, *Ks = sm + L * VLD;
    const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
    load_tile<false>(Vs, VLD, pol.v_row(ch.first, h) + p0, pol.ldv, ch.n, PT / 4, min(PT, pol.P - p0) / 4);
    load_tile<false>(Ks, ldk, pol.k_row(ch.first, h), pol.ldk, ch.n, wide ? 32 : 16, pol.N / 4);
    attn::cp_async_commit();
    const size_t at = ch.place * pol.heads + h;
    if (tid < 32) {
        const float4 a = pol.state_weights(wl, p0 == 0 ? st.rows + at * L * Pol::RECORDS : nullptr, h, ch.first, ch.n, tid);
        if (p0 == 0 && tid == 0) st.aux[at] = a;
    }
    attn::cp_async_wait<0>();
    __syncthreads();
    for (int e = tid; e < L * PT / 4; e += THREADS) {  // the weights go into v
        float* v = Vs + (e >> 4) * VLD + 4 * (e & 15);
        const float4 x = load4(v);
        const float w = wl[e >> 4];
        store4(v, make_float4(x.x * w, x.y * w, x.z * w, x.w * w));
    }
    __syncthreads();
    const size_t E = (size_t)pol.P * pol.N + (Pol::NORMALISER ? pol.N : 0);
    float* out = st.scratch + at * E;
    const int p = p0 + 4 * ty;
    if (p < pol.P) {
        float acc[2][4][4] = {};  // [half of k's elements][element of k][of v]
        const int rows = (ch.n + 15) / 16 * 16;
        product_down(acc, Ks + 4 * tx, ldk, wide ? 64 : 0, Vs + 4 * ty, VLD, rows);
#pragma unroll
        for (int t = 0; t < 2; ++t) {
            const int n = 64 * t + 4 * tx;
            if (n < pol.N)
#pragma unroll
                for (int i = 0; i < 4; ++i)  // (P is a multiple of four)
                    store4(out + (size_t)(p + i) * pol.N + n, make_float4(acc[t][0][i], acc[t][1][i], acc[t][2][i], acc[t][3][i]));
        }
    }
    if (Pol::NORMALISER && p0 == 0)
        for (int n = tid; n < pol.N; n += THREADS) {
            float a[4] = {};
#pragma unroll 4
            for (int s = 0; s < L; ++s) a[s & 3] = fmaf(wl[s], Ks[s * ldk + n], a[s & 3]);  // rows from n on: zeros
            out[(size_t)pol.P * pol.N + n] = (a[0] + a[1]) + (a[2] + a[3]);
        }
}

// Four neighbouring elements of a head's memory a thread; eight chunks' sums are fetched ahead.
template <class Pol>
__global__ void __launch_bounds__(128) chunk_carry_kernel(Pol pol, Step st) {
    constexpr int AHEAD = 8;
    rfx::pdl_prologue();
    const int seq = st.round.seq0 + blockIdx.y, h = blockIdx.z;
    const int e = 4 * (blockIdx.x * 128 + threadIdx.x);
    const int E = pol.P * pol.N + (Pol::NORMALISER ? pol.N : 0);
    if (e >= E) return;
    const int row0 = st.seq_row0[seq], from = row0 + st.round.seg * st.round.seg_rows;
    const int rows = min(st.seq_row0[seq + 1] - from, st.round.seg_rows);
    const int n = (rows + L - 1) / L;
    if (rows <= 0) return;
    const int slot = st.seq_slot[seq];
    float4 S = pol.load_state(slot, h, e);
    float m = pol.load_number(slot, h);
    const size_t at = place_in(st.round, L, row0, seq, 0) * pol.heads + h;
    float* sc = st.scratch + at * E + e;
    const size_t step = (size_t)pol.heads * E;
    for (int c0 = 0; c0 < n; c0 += AHEAD) {
        float4 d[AHEAD], a[AHEAD];
#pragma unroll
        for (int i = 0; i < AHEAD; ++i)
            if (c0 + i < n) {
                d[i] = *reinterpret_cast<const float4*>(sc + (c0 + i) * step);
                a[i] = st.aux[at + (size_t)(c0 + i) * pol.heads];
            }
#pragma unroll
        for (int i = 0; i < AHEAD; ++i)
            if (c0 + i < n) {
                *reinterpret_cast<float4*>(sc + (c0 + i) * step) = S;
                if (e == 0) st.before[at + (size_t)(c0 + i) * pol.heads] = m;
                const float2 f = pol.carry(a[i], m);
                S.x = fmaf(f.x, S.x, f.y * d[i].x);
                S.y = fmaf(f.x, S.y, f.y * d[i].y);
                S.z = fmaf(f.x, S.z, f.y * d[i].z);
                S.w = fmaf(f.x, S.w, f.y * d[i].w);
            }
    }
    pol.store_state(slot, h, e, S);
}

// Inclusive sums (or maxima) over the chunk's 64 rows, lane i holding rows i and i + 32.
__device__ __forceinline__ void scan_sum(double& a, double& b, int lane) {
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const double x = __shfl_up_sync(0xffffffffu, a, o), y = __shfl_up_sync(0xffffffffu, b, o);
        if (lane >= o) {
            a += x;
            b += y;
        }
    }
    b += __shfl_sync(0xffffffffu, a, 31);
}
__device__ __forceinline__ void scan_max(double& a, double& b, int lane) {
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const double x = __shfl_up_sync(0xffffffffu, a, o), y = __shfl_up_sync(0xffffffffu, b, o);
        if (lane >= o) {
            a = fmax(a, x);
            b = fmax(b, y);
        }
    }
    b = fmax(b, __shfl_sync(0xffffffffu, a, 31));
}
__device__ __forceinline__ void two_parts(double v, float* hi, float* lo) {
    const float h = (float)v;
    *hi = h;
    *lo = isinf(h) ? 0.0f : (float)(v - (double)h);
}

// What a row t brings to its results: w_ts = exp((g_s + e_t)) * w_s with e in two parts, the factor of
// q . S, and a number for the policy's store.
struct RowTerms {
    float e_hi, e_lo, alpha, extra;
};

// A block a (chunk, q/k head, some of that head's items); an item is a (head, PT elements of v).  The
// rows' products with the chunk's k, once, stay in registers; then head by head they become the rows'
// weights in shared memory, and item by item the memory's tile and v's come and meet q and the weights.
// A row never multiplies a later row's v, so what is not finite there does not reach it.
template <class Pol>
__global__ void __launch_bounds__(THREADS, 2) chunk_out_kernel(Pol pol, Step st, int items_a_block) {
    extern __shared__ __align__(16) float sm[];
    __shared__ __align__(16) float4 rec[L * Pol::RECORDS];
    __shared__ float nv[128];
    rfx::pdl_prologue();
    const int seq = st.round.seq0 + blockIdx.y;
    const Rows ch = rows_of(st, seq, blockIdx.x);
    if (ch.n <= 0) return;
    const int ptiles = (pol.P + PT - 1) / PT, items = pol.per * ptiles;
    const int sets = (items + items_a_block - 1) / items_a_block;
    const int kvh = blockIdx.z / sets, i0 = (blockIdx.z - kvh * sets) * items_a_block;
    const int i1 = min(items, i0 + items_a_block);
    const int n16 = (pol.N + 15) / 16, ld = 16 * n16 + 4;
    float *Qs = sm, *Bs = sm + L * ld, *Vs = Bs + L * ld, *Ws = Vs + L * VLD;
    const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4, t0 = 4 * ty;
    load_tile<false>(Qs, ld, pol.q_row(ch.first, kvh * pol.per), pol.ldq, ch.n, 4 * n16, pol.N / 4);
    load_tile<true>(Bs, ld, pol.k_row(ch.first, kvh * pol.per), pol.ldk, ch.n, 4 * n16, pol.N / 4);
    attn::cp_async_commit();
    attn::cp_async_wait<0>();
    __syncthreads();
    const float *qa = Qs + t0 * ld, *ba = Bs + tx * ld;
    float G[4][4] = {};  // rows t0 .. by rows 4 tx .. of k, where any of those is no later
    if (tx <= ty) product_along<4>(G, qa, ld, ba, 16 * ld, n16);
    int head = -1;
    for (int item = i0; item < i1; ++item) {
        const int h = kvh * pol.per + item / ptiles, p0 = (item % ptiles) * PT;
        const size_t at = ch.place * pol.heads + h;
        const size_t E = (size_t)pol.P * pol.N + (Pol::NORMALISER ? pol.N : 0);
        const float* S = st.scratch + at * E;
        const float before = st.before[at];
        __syncthreads();  // k, or the item before, has been read by every warp
        if (h != head) {
            for (int i = tid; i < L * Pol::RECORDS; i += THREADS)
                attn::cp_async_16(&rec[i], st.rows + at * L * Pol::RECORDS + i, true);
            if (Pol::NORMALISER)
                for (int n = tid; n < pol.N; n += THREADS) nv[n] = S[(size_t)pol.P * pol.N + n];
        }
        attn::cp_async_commit();
        load_tile<true>(Bs, ld, S + (size_t)p0 * pol.N, pol.N, min(PT, pol.P - p0), 4 * n16, pol.N / 4);
        load_tile<false>(Vs, VLD, pol.v_row(ch.first, h) + p0, pol.ldv, ch.n, PT / 4, min(PT, pol.P - p0) / 4);
        attn::cp_async_commit();
        if (h != head) {
            attn::cp_async_wait<1>();
            __syncthreads();
            if (tx <= ty) {
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const RowTerms r = pol.row_terms(rec + (t0 + i) * Pol::RECORDS, before);
                    float w[4];
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const float4 k = rec[(4 * tx + j) * Pol::RECORDS];
                        w[j] = 4 * tx + j <= t0 + i
                                   ? G[i][j] * (Pol::weight(k) * expf((Pol::g_hi(k) + r.e_hi) + (Pol::g_lo(k) + r.e_lo)))
                                   : 0.0f;
                    }
                    store4(Ws + (t0 + i) * WLD + 4 * tx, make_float4(w[0], w[1], w[2], w[3]));
                }
            }
            head = h;
        }
        if constexpr (Pol::NORMALISER) {
            if (ch.last && p0 == 0 && tid == 0) {
                float m = before;
                pol.carry(st.aux[at], m);
                pol.store_number(st.seq_slot[seq], h, m);
            }
        }
        attn::cp_async_wait<0>();
        __syncthreads();
        float acc[4][4] = {};
        product_along<4>(acc, qa, ld, ba, 16 * ld, n16);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float alpha = pol.row_terms(rec + (t0 + i) * Pol::RECORDS, before).alpha;
#pragma unroll
            for (int j = 0; j < 4; ++j) acc[i][j] *= alpha;
        }
        product_below<false>(acc, Ws + t0 * WLD, WLD, Vs + 4 * tx, VLD, ty);
        if constexpr (Pol::NORMALISER) {
            if (p0 == 0) {  // four threads a row
                const int t = tid >> 2, j = tid & 3;
                const RowTerms r = pol.row_terms(rec + t * Pol::RECORDS, before);
                float sum = 0.0f, qn = 0.0f;
                for (int s = j; s <= t; s += 4) sum += Ws[t * WLD + s];
                for (int n = j; n < pol.N; n += 4) qn = fmaf(Qs[t * ld + n], nv[n], qn);
                sum = fmaf(r.alpha, qn, sum);
                sum += __shfl_xor_sync(0xffffffffu, sum, 1);
                sum += __shfl_xor_sync(0xffffffffu, sum, 2);
                if (j == 0 && t < ch.n) pol.store_sum(ch.first + t, h, sum, r.extra);
            }
        }
        const int p = p0 + 4 * tx;
        if (p < pol.P)  // (P is a multiple of four)
#pragma unroll
            for (int i = 0; i < 4; ++i)
                if (t0 + i < ch.n)
                    pol.store_row(ch.first + t0 + i, h, p, make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]),
                                  load4(Vs + (t0 + i) * VLD + 4 * tx));
    }
}

// Floats of scratch a chunk needs: its memories and what the other kernels read beside them.
inline long long chunk_floats(int heads, long long E, int records) { return heads * (E + 8 + 4 * L * records); }

template <class Pol>
int run(const Pol& pol, const int* seq_slot, const int* seq_row0, int n_seq, int R, int max_rows, float* scratch,
        cudaStream_t s) {
    const long long E = (long long)pol.P * pol.N + (Pol::NORMALISER ? pol.N : 0);
    const Plan plan = plan_rounds(R, n_seq, max_rows, L, chunk_floats(pol.heads, E, Pol::RECORDS));
    Step st;
    st.seq_slot = seq_slot;
    st.seq_row0 = seq_row0;
    const long long n_places = plan.places;
    st.scratch = scratch;
    st.aux = reinterpret_cast<float4*>(scratch + n_places * pol.heads * E);  // E is a multiple of four
    st.rows = st.aux + n_places * pol.heads;
    st.before = reinterpret_cast<float*>(st.rows + n_places * pol.heads * L * Pol::RECORDS);
    const int ptiles = (pol.P + PT - 1) / PT;
    const int chunks = plan.seg_rows / L;
    const size_t sm_state = (size_t)L * (VLD + (pol.N > 64 ? 132 : 68)) * sizeof(float);
    const size_t sm_out = (size_t)L * (VLD + WLD + 2 * ((pol.N + 15) / 16 * 16 + 4)) * sizeof(float);
    const int qk_heads = pol.heads / pol.per, items = pol.per * ptiles;
    // items a block: the rows' products with k, which serve them all, cost about as much as one item; two
    // blocks share an SM
    int ipb = items;
    long long least = -1;
    for (int i = items; i >= 1; --i) {
        const long long blocks = (long long)chunks * plan.group * qk_heads * ((items + i - 1) / i);
        const long long cost = (blocks + 2 * sm_count() - 1) / (2 * sm_count()) * (1 + i);
        if (least < 0 || cost < least) {
            least = cost;
            ipb = i;
        }
    }
    const int sets = (items + ipb - 1) / ipb;
    if (n_seq > 65535 || (long long)pol.heads * ptiles > 65535 || (long long)qk_heads * sets > 65535)
        return RFX_ERR_UNSUPPORTED;
    cudaError_t e = cudaFuncSetAttribute(chunk_state_kernel<Pol>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm_state);
    if (e != cudaSuccess) return (int)e;
    e = cudaFuncSetAttribute(chunk_out_kernel<Pol>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm_out);
    if (e != cudaSuccess) return (int)e;
    for (int seq0 = 0; seq0 < n_seq; seq0 += plan.group)
        for (int seg = 0; seg < plan.n_segs; ++seg) {
            const int seqs = min(plan.group, n_seq - seq0);
            st.round = Round{plan.seg_rows, seg, seq0, plan.whole};
            RFX_LAUNCH(chunk_state_kernel<Pol>, dim3(chunks, seqs, pol.heads * ptiles), THREADS, sm_state, s, pol, st);
            RFX_LAUNCH(chunk_carry_kernel<Pol>, dim3((unsigned)((E / 4 + 127) / 128), seqs, pol.heads), 128, 0, s, pol, st);
            RFX_LAUNCH(chunk_out_kernel<Pol>, dim3(chunks, seqs, qk_heads * sets), THREADS, sm_out, s, pol, st, ipb);
        }
    return 0;
}

}  // namespace chunk
