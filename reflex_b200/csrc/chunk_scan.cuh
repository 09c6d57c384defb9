// Recurrences S <- decay S + weight k v^T, y = S^T q with one decay and one weight a head and
// row (ssd.cu, mlstm.cu) over the many rows of a prompt, 64 rows at a time and all chunks side by
// side, as products on the tensor cores of operands split in two (split_mma.cuh).
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
// arithmetic.  A prompt of 2,048 rows: 1.2 ms walking and 0.12 ms in chunks for 32 heads of 64 x 128
// (30 us the chunks' sums, 19 the carry, 75 the rows), 0.76 and 0.13 ms for 8 of 128 x 256 (35, 27 and
// 65); the carry is bound by L2, the other two by the latency of tiles and fragments on the way to
// the tensor pipe (28 % busy).  64 rows: with 32 the memories' traffic doubles, with 128 the products
// inside the chunk do and a block no longer shares its SM.
//
// A policy `Pol` gives: q, k, v rows (float32, 16-byte aligned, counts in fours), `heads`, `per`
// (heads per q/k head), N (elements of q and k, at most 128), P (elements of v) and the functions
// named below.  A long step goes through a bounded scratch in several rounds (chunk_plan.cuh).
#pragma once

#include <type_traits>

#include "attn_mma.cuh"
#include "chunk_plan.cuh"
#include "common.cuh"
#include "split_mma.cuh"

namespace chunk {

using namespace rfx;

constexpr int L = 64;     // rows of a chunk
constexpr int PT = 64;    // elements of v a block takes at a time
constexpr int VLD = PT + 4;  // row stride of v's tile: 2 VLD = 8 mod 32, four rows' reads meet all banks

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
    bool last;     // of its sequence's in this round
    size_t place;
};
__device__ __forceinline__ Rows rows_of(const Step& s, int seq, int c) {
    const int row0 = s.seq_row0[seq], from = row0 + s.round.seg * s.round.seg_rows;
    const int to = min(s.seq_row0[seq + 1], from + s.round.seg_rows);
    const int first = from + c * L;
    return {first, min(L, to - first), to - first <= L, place_in(s.round, L, row0, seq, c)};
}

// A tile of `rows` rows of 4 * c4 floats, rows from n on and columns from n4 (in fours) on zero.
template <int THREADS>
__device__ __forceinline__ void load_tile(float* dst, int ld, const float* src, size_t src_ld, int rows, int n, int c4,
                                          int n4) {
    if (THREADS % c4 == 0) {  // a thread keeps its column: no division a piece
        const int c = threadIdx.x % c4, step = THREADS / c4;
        int r = threadIdx.x / c4;
        float* d = dst + r * ld + 4 * c;
        const float* s = src + (size_t)r * src_ld + 4 * c;
        const int live = c < n4 ? n : 0;
        for (; r < rows; r += step, d += step * ld, s += (size_t)step * src_ld) attn::cp_async_16(d, r < live ? s : src, r < live);
    } else {
        for (int e = threadIdx.x; e < rows * c4; e += THREADS) {
            const int r = e / c4, c = e - r * c4;
            const bool ok = r < n && c < n4;
            attn::cp_async_16(dst + r * ld + 4 * c, ok ? src + (size_t)r * src_ld + 4 * c : src, ok);
        }
    }
}

// A block a (chunk, head, PT elements of v): the chunk's own sum, [P][N].  Warps: 16 of v's elements
// by 64 of k's.
template <class Pol>
__global__ void __launch_bounds__(256) chunk_state_kernel(Pol pol, Step st) {
    extern __shared__ __align__(16) float sm[];
    __shared__ __align__(8) float wl[L];
    rfx::pdl_prologue();
    const int seq = st.round.seq0 + blockIdx.y;
    const Rows ch = rows_of(st, seq, blockIdx.x);
    if (ch.n <= 0) return;
    const int ptiles = (pol.P + PT - 1) / PT, h = blockIdx.z / ptiles, p0 = (blockIdx.z - h * ptiles) * PT;
    const int N8 = (pol.N + 7) / 8 * 8, ldk = N8 + 4;
    float *Vs = sm, *Ks = sm + L * VLD;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, j = lane & 3;
    load_tile<256>(Vs, VLD, pol.v_row(ch.first, h) + p0, pol.ldv, L, ch.n, PT / 4, min(PT, pol.P - p0) / 4);
    load_tile<256>(Ks, ldk, pol.k_row(ch.first, h), pol.ldk, L, ch.n, N8 / 4, pol.N / 4);
    attn::cp_async_commit();
    const size_t at = ch.place * pol.heads + h;
    if (warp == 0) {
        const float4 a = pol.state_weights(wl, p0 == 0 ? st.rows + at * L * Pol::RECORDS : nullptr, h, ch.first, ch.n, lane);
        if (p0 == 0 && lane == 0) st.aux[at] = a;
    }
    attn::cp_async_wait<0>();
    __syncthreads();
    const int pm = (warp & 3) * 16, n0 = (warp >> 2) * 64;
    const size_t E = (size_t)pol.P * pol.N + (Pol::NORMALISER ? pol.N : 0);
    float* out = st.scratch + at * E;
    if (n0 < N8 && p0 + pm < pol.P) {
        float acc[8][4] = {};
#pragma unroll 2
        for (int s = 0; s < L / 8; ++s) {
            const float2 w = *reinterpret_cast<const float2*>(wl + 8 * s + 2 * j);
            const float* v = Vs + (8 * s + 2 * j) * VLD + pm + g;
            const Left a = left_from(v[0] * w.x, v[8] * w.x, v[VLD] * w.y, v[VLD + 8] * w.y);
            const float* k = Ks + (8 * s + 2 * j) * ldk + g;
            float2 b[8];
#pragma unroll
            for (int t = 0; t < 8; ++t) {
                const int c = n0 + 8 * t < N8 ? n0 + 8 * t : 0;  // a tile beyond N: any column, not stored
                b[t] = make_float2(k[c], k[ldk + c]);
            }
            product3<8>(acc, a, b);
        }
#pragma unroll
        for (int t = 0; t < 8; ++t) {
            const int n = n0 + 8 * t + 2 * j, p = p0 + pm + g;
            if (n < pol.N) {
                if (p < pol.P) store2(out + (size_t)p * pol.N + n, acc[t][0], acc[t][1]);
                if (p + 8 < pol.P) store2(out + (size_t)(p + 8) * pol.N + n, acc[t][2], acc[t][3]);
            }
        }
    }
    if (Pol::NORMALISER && p0 == 0)
        for (int n = threadIdx.x; n < pol.N; n += 256) {
            float a = 0.0f;
            for (int s = 0; s < ch.n; ++s) a = fmaf(wl[s], Ks[s * ldk + n], a);
            out[(size_t)pol.P * pol.N + n] = a;
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

// A block a (chunk, q/k head, some of that head's items); an item is a (head, PT elements of v).
// Two warps take sixteen rows, half an item's columns each: the rows' products with the chunk's k, once,
// stay in registers; then item by item the memory's tile and v's replace k's in shared memory.  Eight
// warps, although two then make the same products with k: at 87 KB a block two share an SM, and four
// warps each leave too few to cover the tiles' arrival, the exponentials and the fragments' splitting
// (96 and 74 us for the two shapes above, now 75 and 65).
template <class Pol>
__global__ void __launch_bounds__(256, 2) chunk_out_kernel(Pol pol, Step st, int items_a_block) {
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
    const int N8 = (pol.N + 7) / 8 * 8, ld = N8 + 8;
    float *Qs = sm, *Bs = sm + L * ld, *Vs = Bs + L * ld;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, j = lane & 3;
    const int rw = warp & 3, c0 = (warp >> 2) * (PT / 2);  // the warp's rows (sixteen) and columns of a tile
    load_tile<256>(Qs, ld, pol.q_row(ch.first, kvh * pol.per), pol.ldq, L, ch.n, N8 / 4, pol.N / 4);
    load_tile<256>(Bs, ld, pol.k_row(ch.first, kvh * pol.per), pol.ldk, L, ch.n, N8 / 4, pol.N / 4);
    attn::cp_async_commit();
    attn::cp_async_wait<0>();
    __syncthreads();
    const float* qa = Qs + (16 * rw + g) * ld + 2 * j;
    const int tiles = 2 * rw + 2;  // of eight rows s <= the warp's last row
    float G[8][4] = {};
    auto scores = [&](auto& acc, auto count) {
        constexpr int T = decltype(count)::value;
        for (int s = 0; s < N8 / 8; ++s) {
            const float2 x = *reinterpret_cast<const float2*>(qa + 8 * s);
            const float2 y = *reinterpret_cast<const float2*>(qa + 8 * ld + 8 * s);
            const Left a = left_from(x.x, y.x, x.y, y.y);
            float2 b[T];
#pragma unroll
            for (int t = 0; t < T; ++t) b[t] = *reinterpret_cast<const float2*>(Bs + (8 * t + g) * ld + 8 * s + 2 * j);
            product3<T>(acc, a, b);
        }
    };
    if (rw >= 2) scores(G, std::integral_constant<int, 8>{});
    else scores(*reinterpret_cast<float(*)[4][4]>(&G), std::integral_constant<int, 4>{});
    const int ra = 16 * rw + g, rb = ra + 8;
    int head = -1;
    for (int item = i0; item < i1; ++item) {
        const int h = kvh * pol.per + item / ptiles, p0 = (item % ptiles) * PT;
        const size_t at = ch.place * pol.heads + h;
        const size_t E = (size_t)pol.P * pol.N + (Pol::NORMALISER ? pol.N : 0);
        const float* S = st.scratch + at * E;
        __syncthreads();  // k, or the item before, has been read by every warp
        load_tile<256>(Bs, ld, S + (size_t)p0 * pol.N, pol.N, PT, min(PT, pol.P - p0), N8 / 4, pol.N / 4);
        load_tile<256>(Vs, VLD, pol.v_row(ch.first, h) + p0, pol.ldv, L, ch.n, PT / 4, min(PT, pol.P - p0) / 4);
        if (h != head) {
            for (int i = threadIdx.x; i < L * Pol::RECORDS; i += 256)
                attn::cp_async_16(&rec[i], st.rows + at * L * Pol::RECORDS + i, true);
            if (Pol::NORMALISER)
                for (int n = threadIdx.x; n < pol.N; n += 256) nv[n] = S[(size_t)pol.P * pol.N + n];
            head = h;
        }
        attn::cp_async_commit();
        const float before = st.before[at];
        if constexpr (Pol::NORMALISER) {
            if (ch.last && p0 == 0 && threadIdx.x == 0) {
                float m = before;
                pol.carry(st.aux[at], m);
                pol.store_number(st.seq_slot[seq], h, m);
            }
        }
        attn::cp_async_wait<0>();
        __syncthreads();
        float acc[4][4] = {};
        for (int s = 0; s < N8 / 8; ++s) {
            const float2 x = *reinterpret_cast<const float2*>(qa + 8 * s);
            const float2 y = *reinterpret_cast<const float2*>(qa + 8 * ld + 8 * s);
            const Left a = left_from(x.x, y.x, x.y, y.y);
            float2 b[4];
#pragma unroll
            for (int t = 0; t < 4; ++t)
                b[t] = *reinterpret_cast<const float2*>(Bs + (c0 + 8 * t + g) * ld + 8 * s + 2 * j);
            product3<4>(acc, a, b);
        }
        const RowTerms ta = pol.row_terms(rec + ra * Pol::RECORDS, before), tb = pol.row_terms(rec + rb * Pol::RECORDS, before);
#pragma unroll
        for (int t = 0; t < 4; ++t) {
            acc[t][0] *= ta.alpha;
            acc[t][1] *= ta.alpha;
            acc[t][2] *= tb.alpha;
            acc[t][3] *= tb.alpha;
        }
        float sum_a = 0.0f, sum_b = 0.0f;
#pragma unroll
        for (int t = 0; t < 8; ++t) {
            if (t < tiles) {
                float p[4];
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    const int s = 8 * t + 2 * j + i;
                    const float4 r = rec[s * Pol::RECORDS];
                    const float gh = Pol::g_hi(r), gl = Pol::g_lo(r), w = Pol::weight(r);
                    p[i] = s <= ra ? G[t][i] * (w * expf((gh + ta.e_hi) + (gl + ta.e_lo))) : 0.0f;
                    p[2 + i] = s <= rb ? G[t][2 + i] * (w * expf((gh + tb.e_hi) + (gl + tb.e_lo))) : 0.0f;
                }
                if (Pol::NORMALISER) {
                    sum_a += p[0] + p[1];
                    sum_b += p[2] + p[3];
                }
                const Left a = left_of(p);
                const float* v = Vs + (8 * t + 2 * j) * VLD + c0 + g;
                float2 b[4];
#pragma unroll
                for (int c = 0; c < 4; ++c) b[c] = make_float2(v[8 * c], v[VLD + 8 * c]);
                product3<4>(acc, a, b);
            }
        }
        if constexpr (Pol::NORMALISER) {
            if (p0 == 0 && c0 == 0) {
                float qa_n = 0.0f, qb_n = 0.0f;
                for (int n = j; n < pol.N; n += 4) {
                    qa_n = fmaf(Qs[ra * ld + n], nv[n], qa_n);
                    qb_n = fmaf(Qs[rb * ld + n], nv[n], qb_n);
                }
                sum_a = fmaf(ta.alpha, qa_n, sum_a);
                sum_b = fmaf(tb.alpha, qb_n, sum_b);
#pragma unroll
                for (int o = 1; o < 4; o <<= 1) {
                    sum_a += __shfl_xor_sync(0xffffffffu, sum_a, o);
                    sum_b += __shfl_xor_sync(0xffffffffu, sum_b, o);
                }
                if (j == 0) {
                    if (ra < ch.n) pol.store_sum(ch.first + ra, h, sum_a, ta.extra);
                    if (rb < ch.n) pol.store_sum(ch.first + rb, h, sum_b, tb.extra);
                }
            }
        }
#pragma unroll
        for (int t = 0; t < 4; ++t) {
            const int c = c0 + 8 * t + 2 * j, p = p0 + c;
            if (p < pol.P) {
                const float2 va = *reinterpret_cast<const float2*>(Vs + ra * VLD + c);
                const float2 vb = *reinterpret_cast<const float2*>(Vs + rb * VLD + c);
                if (ra < ch.n) pol.store_row(ch.first + ra, h, p, acc[t][0], acc[t][1], va.x, va.y);
                if (rb < ch.n) pol.store_row(ch.first + rb, h, p, acc[t][2], acc[t][3], vb.x, vb.y);
            }
        }
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
    const int N8 = (pol.N + 7) / 8 * 8, ptiles = (pol.P + PT - 1) / PT;
    const int chunks = plan.seg_rows / L;
    const size_t sm_state = (size_t)L * (VLD + N8 + 4) * sizeof(float);
    const size_t sm_out = (size_t)L * (VLD + 2 * (N8 + 8)) * sizeof(float);
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
            RFX_LAUNCH(chunk_state_kernel<Pol>, dim3(chunks, seqs, pol.heads * ptiles), 256, sm_state, s, pol, st);
            RFX_LAUNCH(chunk_carry_kernel<Pol>, dim3((unsigned)((E / 4 + 127) / 128), seqs, pol.heads), 128, 0, s, pol, st);
            RFX_LAUNCH(chunk_out_kernel<Pol>, dim3(chunks, seqs, qk_heads * sets), 256, sm_out, s, pol, st, ipb);
        }
    return 0;
}

}  // namespace chunk
