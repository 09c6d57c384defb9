// Recurrences S <- decay S + weight k v^T, y = S^T q with one decay and one weight a head and
// row (ssd.cu, mlstm.cu) over the many rows of a prompt, 64 rows at a time and all chunks side by
// side, as 32-bit products on the tcgen05 tensor cores (tc_split.cuh).
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
// arithmetic.  64 rows: with 32 the memories' traffic doubles, with 128 the products inside the chunk do.
// A prompt of 2,048 rows, us: for 32 heads of 64 x 128 21 the chunks' sums, 13.5 the carry, 58 the rows (1,200
// walking), for 8 of 128 x 256 24, 17 and 57 (760).  With the products by 32-bit multiply-adds, whose reads of
// shared memory and whose latencies bound them, 42, 12 and 76, and 49, 18 and 65.  What bounds these now is a block's
// stages, which wait for one another: numbers taken apart, eight products a sixteen, sums out of tensor memory (1.5 of
// four instructions issued a cycle, the tensor cores busy a quarter of the time); the carry is bound by L2.
//
// 2-norm errors against 64 bits, the same shapes, normal numbers: results 9.1e-8 and 1.07e-7 (1.36e-7 and 1.40e-7 by
// multiply-adds), states 7.4e-8 and 1.18e-7 (9.5e-8 and 1.39e-7); other numbers in tc_split.cuh.
//
// A policy `Pol` gives: q, k, v rows (float32, 16-byte aligned, counts in fours), `heads`, `per`
// (heads per q/k head), N (elements of q and k, at most 128), P (elements of v) and the functions
// named below.  A long step goes through a bounded scratch in several rounds (chunk_plan.cuh).
#pragma once

#include "chunk_plan.cuh"
#include "common.cuh"
#include "tc_split.cuh"

namespace chunk {

using namespace rfx;

constexpr int L = 64;     // rows of a chunk
constexpr int PT = 64;    // elements of v a block takes at a time
constexpr int STATE_THREADS = 256, WARPS = STATE_THREADS / 32, OUT_THREADS = 512;
constexpr int OLD = 68;   // row stride of results in shared memory
constexpr uint32_t TMEM_COLS = 256;  // two blocks share an SM
constexpr size_t SMEM = 4 * split3::TILE + 1024;  // (aligned by the kernels)

struct Step {
    const int* seq_slot;
    const int* seq_row0;
    Round round;
    float* scratch;  // [place][head][P][N] (+ [N] with a normaliser): a chunk's own sum, then the memory before it
    float4* aux;     // [place][head]: what the carry needs of a chunk
    float* before;   // [place][head]: the policy's running number before the chunk
    float4* rows;    // [place][head][L][RECORDS]: the policy's records of the chunk's rows
    int* err;        // where a wait that ran out is reported
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

// What both tensor-core kernels of a block hold: the barrier its products arrive at, the tensor memory, and
// whether a wait ran out (reported; nothing is multiplied or waits after that, and the block ends with what is there).
struct Core {
    uint32_t tmem;
    uint64_t* done;
    uint32_t phase;  // of either barrier, in a bit each
    bool waits;
    int* err;

    // Every thread, first of all: the products' barriers and the tensor memory, before the next kernels are let in
    // (their blocks could otherwise hold columns while they wait for this grid, and a block of this grid wait for
    // those columns); then the wait for the kernels before.
    __device__ __forceinline__ void open(uint64_t* bars, uint32_t* slot, int* error) {
        done = bars;
        phase = 0;
        waits = true;
        err = error;
        if (threadIdx.x == 0) {
            sm100::mbar_init(done, 1);
            sm100::mbar_init(done + 1, 1);
            sm100::fence_barrier_init();
        }
        if (threadIdx.x < 32) {
            __syncwarp();
            sm100::tmem_alloc(slot, TMEM_COLS);
            sm100::tmem_relinquish();
        }
        sm100::tc_fence_before_sync();
        __syncthreads();
        sm100::tc_fence_after_sync();
        tmem = *slot;
        rfx::pdl_prologue();
    }
    // Products that one thread issues once all have passed this barrier; true if any thread saw odd numbers.
    template <class Issue>
    __device__ __forceinline__ bool start(int bar, bool odd, Issue&& issue) {
        split3::tiles_written();
        const bool any = __syncthreads_or(odd);
        if (threadIdx.x < 32) {
            sm100::tc_fence_after_sync();
            if (sm100::elect_one() && waits) {
                issue();
                sm100::umma_commit(done + bar);
            }
            __syncwarp();
        }
        return any;
    }
    __device__ __forceinline__ void wait(int bar) {
        if (waits && !sm100::mbar_wait(done + bar, phase >> bar & 1)) {
            waits = false;
            if (err) atomicExch(err, 42);
            sm100::mbar_wait(done + bar, phase >> bar & 1);  // as long again for what is still being multiplied
        }
        phase ^= 1u << bar;
        sm100::tc_fence_after_sync();
    }
    __device__ __forceinline__ void close() {
        sm100::tc_fence_before_sync();
        __syncthreads();
        if (threadIdx.x < 32) {
            sm100::tc_fence_after_sync();
            sm100::tmem_dealloc(tmem, TMEM_COLS);
        }
    }
};
__device__ __forceinline__ char* tiles_of(char* sm) {  // shared memory from a boundary of 1,024 bytes on
    return sm + (-(int)sm100::smem_u32(sm) & 1023);
}
// A block a (chunk, q/k head, some of that head's items); an item is a (head, PT elements of v): the
// chunk's own sums, [P][N], as k's elements (128 lanes) by v's.  k is split once, the heads' weights come from
// a warp each; an item's product runs while the one before is stored and the next one's v is on its way.
template <class Pol>
__global__ void __launch_bounds__(STATE_THREADS, 2) chunk_state_kernel(Pol pol, Step st, int items_a_block) {
    extern __shared__ __align__(16) char sm_raw[];
    __shared__ float wl[WARPS][L];
    __shared__ uint64_t bars[2];
    __shared__ uint32_t tmem_slot;
    Core core;
    core.open(bars, &tmem_slot, st.err);
    const int seq = st.round.seq0 + blockIdx.y;
    const Rows ch = rows_of(st, seq, blockIdx.x);
    if (ch.n <= 0) {
        core.close();
        return;
    }
    const int ptiles = (pol.P + PT - 1) / PT, items = pol.per * ptiles;
    const int sets = (items + items_a_block - 1) / items_a_block;
    const int kvh = blockIdx.z / sets, i0 = (blockIdx.z - kvh * sets) * items_a_block;
    const int i1 = min(items, i0 + items_a_block), h0 = kvh * pol.per + i0 / ptiles;
    char *Ks = tiles_of(sm_raw), *Vs = Ks + 2 * split3::TILE;  // k's two tiles of 64 elements, v of two items
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const size_t E = (size_t)pol.P * pol.N + (Pol::NORMALISER ? pol.N : 0);
    using Own = split3::Own<STATE_THREADS>;
    auto bring = [&](Own& v, int item) {
        const int p0 = (item % ptiles) * PT;
        v.load(pol.v_row(ch.first, kvh * pol.per + item / ptiles) + p0, pol.ldv, ch.n, pol.P - p0);
    };
    Own v, k0, k1;
    k0.load(pol.k_row(ch.first, kvh * pol.per), pol.ldk, ch.n, pol.N);
    k1.load(pol.k_row(ch.first, kvh * pol.per) + 64, pol.ldk, ch.n, pol.N - 64);
    bring(v, i0);
    {
        const int h = h0 + warp;
        if (h <= kvh * pol.per + (i1 - 1) / ptiles) {
            const size_t to = ch.place * pol.heads + h;
            const bool first = warp || i0 % ptiles == 0;  // the head's first item is this block's
            const float4 a = pol.state_weights(wl[warp], first ? st.rows + to * L * Pol::RECORDS : nullptr, h, ch.first, ch.n, lane);
            if (first && lane == 0) st.aux[to] = a;
        }
    }
    bool odd_k = k0.put(Ks);
    odd_k |= k1.put(Ks + split3::TILE);
    __syncthreads();  // the weights are there
    if (Pol::NORMALISER && i0 % ptiles == 0) {  // the head's sum of k (it is the block's only head), a thread's rows first
        float* part = reinterpret_cast<float*>(Vs + split3::TILE);
        float* mine = part + (tid >> 3) * 128 + Own::col();
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            float a = 0.0f, b = 0.0f;
#pragma unroll
            for (int i = 0; i < Own::ROWS; ++i) {
                a = fmaf(wl[0][Own::row(i)], k0.x[i][j], a);
                b = fmaf(wl[0][Own::row(i)], k1.x[i][j], b);
            }
            mine[j] = a;
            mine[64 + j] = b;
        }
        __syncthreads();
        if (tid < pol.N) {
            float a[4] = {};
#pragma unroll
            for (int i = 0; i < STATE_THREADS / 8; ++i) a[i & 3] += part[i * 128 + tid];
            st.scratch[(ch.place * pol.heads + h0) * E + (size_t)pol.P * pol.N + tid] = (a[0] + a[1]) + (a[2] + a[3]);
        }
    }
    const uint32_t k_at = sm100::smem_u32(Ks);
    const int n = 32 * (warp & 3) + lane, half = 32 * (warp >> 2);  // the thread's element of k and 32 of v's
    bool any_odd = false;  // in the item that is being multiplied
    auto store = [&](int item) {
        const int h = kvh * pol.per + item / ptiles;
        core.wait(0);
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            const int p0 = (item % ptiles) * PT + half + 8 * c;
            float y[8];
            split3::sums_of<2>(y, core.tmem + ((uint32_t)(32 * (warp & 3)) << 16) + half + 8 * c, L / 16);
            const bool live = n < pol.N;
            if (live && any_odd) {  // the odd numbers' products
                const float *k = pol.k_row(ch.first, h) + n, *x = pol.v_row(ch.first, h);
                for (int s = 0; s < ch.n; ++s) {
                    const float ks = k[(size_t)s * pol.ldk];
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        const float vs = x[(size_t)s * pol.ldv + min(p0 + i, pol.P - 1)] * wl[h - h0][s];
                        if (split3::is_odd(ks) || split3::is_odd(vs)) y[i] = fmaf(ks, vs, y[i]);
                    }
                }
            }
            float* to = st.scratch + (ch.place * pol.heads + h) * E + (size_t)p0 * pol.N + n;
            const int left = pol.P - p0;
#pragma unroll
            for (int i = 0; i < 8; ++i, to += pol.N)
                if (live && i < left) *to = y[i];
        }
    };
    for (int item = i0; item < i1; ++item) {
        const int h = kvh * pol.per + item / ptiles;
        const float* weights = wl[h - h0];
        char* V = Vs + ((item - i0) & 1) * split3::TILE;  // (the product that read it two items ago has been waited for)
#pragma unroll
        for (int i = 0; i < Own::ROWS; ++i)
#pragma unroll
            for (int j = 0; j < 8; ++j) v.x[i][j] *= weights[Own::row(i)];
        const bool odd = v.put(V) || odd_k;
        if (item + 1 < i1) bring(v, item + 1);
        if (item > i0) store(item - 1);
        any_odd = core.start(0, odd, [&] {
            split3::issue<2, split3::MN_STEP, split3::MN_STEP>(core.tmem, split3::A_MN | split3::B_MN, L / 16,
                                                               split3::mn_major(k_at, split3::TILE),
                                                               split3::mn_major(sm100::smem_u32(V), split3::PART));
        });
    }
    store(i1 - 1);
    core.close();
}

// Four neighbouring elements of a head's memory a thread; eight chunks' sums are fetched ahead.
template <class Pol>
__global__ void __launch_bounds__(128, 4) chunk_carry_kernel(Pol pol, Step st) {
    constexpr int AHEAD = 8;
    rfx::pdl_wait();
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
    // the next kernel's blocks are let in as these end: before, they crowd on the SMs that these leave free (48 rows of 32
    // heads of 64 x 128: 29 us all three launches, 24 so)
    rfx::pdl_launch_dependents();
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
__device__ __forceinline__ float exp_of(float hi, float lo) {
    const float e = expf(hi);
    return isinf(e) ? e : fmaf(e, lo, e);
}
// e^v as exactly as expf has it, where a v rounded to 32 bits would be off by 2^-25 v
__device__ __forceinline__ float exp_of(double v) {
    float hi, lo;
    two_parts(v, &hi, &lo);
    return exp_of(hi, lo);
}

// (in a chain of eight the first numbers are rounded seven times)
__device__ __forceinline__ float sum8(const float (&x)[8]) {
    return ((x[0] + x[1]) + (x[2] + x[3])) + ((x[4] + x[5]) + (x[6] + x[7]));
}

// What a row t brings to its results: w_ts = exp((g_s + e_t)) * w_s with e in two parts, the factor of
// q . S, and a number for the policy's store.
struct RowTerms {
    float e_hi, e_lo, alpha, extra;
};

// A block a (chunk, q/k head, some of that head's items).  The rows' products with the chunk's k, once,
// stay in registers.  Item by item q meets the memory's tile; meanwhile head by head the products become the
// rows' weights, which then meet v.  A warp has the weights of sixteen rows by sixteen, a thread those of a row
// by eight; results as it has v (split3::Own).
//
// A row's weights of later rows are zero, and a number that is not finite is no operand of the tensor core
// (tc_split.cuh): its products are added afterwards to the rows it may reach, so that it does not reach others.
template <class Pol>
__global__ void __launch_bounds__(OUT_THREADS, 2) chunk_out_kernel(Pol pol, Step st, int items_a_block) {
    extern __shared__ __align__(16) char sm_raw[];
    __shared__ __align__(16) float4 rec[L * Pol::RECORDS];
    __shared__ float row_sum[Pol::NORMALISER ? 8 : 1][L];
    __shared__ uint64_t bars[2];
    __shared__ uint32_t tmem_slot;
    Core core;
    core.open(bars, &tmem_slot, st.err);
    const int seq = st.round.seq0 + blockIdx.y;
    const Rows ch = rows_of(st, seq, blockIdx.x);
    if (ch.n <= 0) {
        core.close();
        return;
    }
    const int ptiles = (pol.P + PT - 1) / PT, items = pol.per * ptiles;
    const int sets = (items + items_a_block - 1) / items_a_block;
    const int kvh = blockIdx.z / sets, i0 = (blockIdx.z - kvh * sets) * items_a_block;
    const int i1 = min(items, i0 + items_a_block);
    // q's two tiles of 64 elements; two tiles of k, then an item's two of the memory, then its weights and v;
    // between them 32-bit results.  (The products of 64 rows are made as of 128, whose other half reads what lies
    // behind a tile and is left where it is.)
    char *Qs = tiles_of(sm_raw), *Bs = Qs + 2 * split3::TILE, *Ws = Bs, *Vs = Bs + split3::TILE;
    float* res = reinterpret_cast<float*>(Bs);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int blocks = pol.N > 64 ? 2 : 1, t = 16 * (warp >> 2) + (lane & 15), sb = (warp + (warp >> 2)) & 3, s0 = 16 * sb + 8 * (lane >> 4);
    const size_t E = (size_t)pol.P * pol.N + (Pol::NORMALISER ? pol.N : 0);
    const float *q = pol.q_row(ch.first, kvh * pol.per), *k = pol.k_row(ch.first, kvh * pol.per);
    using Own = split3::Own<OUT_THREADS>;
    bool odd_qk = false;
#pragma unroll
    for (int b = 0; b < 2; ++b)
        if (b < blocks) {
            Own x, y;
            x.load(q + 64 * b, pol.ldq, ch.n, pol.N - 64 * b);
            y.load(k + 64 * b, pol.ldk, ch.n, pol.N - 64 * b);
            odd_qk |= x.put(Qs + b * split3::TILE);
            odd_qk |= y.put(Bs + b * split3::TILE);
        }
    const int q_steps = (pol.N + 15) / 16;
    const uint32_t q_at = sm100::smem_u32(Qs), b_at = sm100::smem_u32(Bs);
    // q by the two tiles at b_at
    auto q_products = [&] {
        split3::issue<1, split3::K_STEP, split3::K_STEP>(core.tmem, 0, q_steps, split3::k_major(q_at), split3::k_major(b_at));
    };
    // results lie in lanes 0 to 63, which two warps of four can read, sixteen columns each
    const bool reads = !(warp & 2);
    const int row = 32 * (warp & 1) + lane, c0 = 16 * (warp >> 2);
    const uint32_t lanes = core.tmem + ((uint32_t)(32 * (warp & 3)) << 16) + c0;
    auto spread = [&](const float (&y)[8], int c) {  // for every thread to read
        float* to = res + row * OLD + c0 + c;
#pragma unroll
        for (int i = 0; i < 2; ++i) store4(to + 4 * i, make_float4(y[4 * i], y[4 * i + 1], y[4 * i + 2], y[4 * i + 3]));
    };
    auto read8 = [&](float (&y)[8], const float* from) {
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const float4 r = load4(from + 4 * i);
            y[4 * i] = r.x; y[4 * i + 1] = r.y; y[4 * i + 2] = r.z; y[4 * i + 3] = r.w;
        }
    };
    odd_qk = core.start(0, odd_qk, q_products);
    core.wait(0);
    if (reads)
#pragma unroll
        for (int c = 0; c < 16; c += 8) {
            float y[8];
            split3::sums_of<1>(y, lanes + c, q_steps);
            spread(y, c);
        }
    sm100::tc_fence_before_sync();
    __syncthreads();
    float G[8];  // row t by rows s0 .. of k
    read8(G, res + t * OLD + s0);
    if (odd_qk && t < ch.n)
        for (int e = 0; e < pol.N; ++e) {
            const float qe = q[(size_t)t * pol.ldq + e];
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const float ke = s0 + i <= t ? k[(size_t)(s0 + i) * pol.ldk + e] : 0.0f;
                if (split3::is_odd(qe) || split3::is_odd(ke)) G[i] = fmaf(qe, ke, G[i]);
            }
        }
    __syncthreads();  // the results have been read
    auto weights = [&](float (&w)[8], const RowTerms& r) {
        if (16 * sb > t) {
#pragma unroll
            for (int i = 0; i < 8; ++i) w[i] = 0.0f;
        } else {
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const float4 c = rec[(s0 + i) * Pol::RECORDS];
                w[i] = s0 + i <= t ? G[i] * (Pol::weight(c) * expf((Pol::g_hi(c) + r.e_hi) + (Pol::g_lo(c) + r.e_lo))) : 0.0f;
            }
        }
    };
    auto begin_head = [&](int h) {
        const float4* rows = st.rows + (ch.place * pol.heads + h) * L * Pol::RECORDS;
        if (tid < L * Pol::RECORDS) rec[tid] = rows[tid];
    };
    if constexpr (!Pol::SHARED) {  // one head a block: its weights stand where the products stood
        const float before = st.before[ch.place * pol.heads + kvh];
        begin_head(kvh);
        __syncthreads();
        float w[8];
        weights(w, pol.row_terms(rec + t * Pol::RECORDS, before));
#pragma unroll
        for (int i = 0; i < 8; ++i) G[i] = w[i];
    }
    for (int item = i0; item < i1; ++item) {
        const int h = kvh * pol.per + item / ptiles, p0 = (item % ptiles) * PT;
        const size_t at = ch.place * pol.heads + h;
        const float *S = st.scratch + at * E, *vr = pol.v_row(ch.first, h) + p0;
        Own v, m;
        v.load(S + (size_t)p0 * pol.N, pol.N, pol.P - p0, pol.N);
        m.load(S + (size_t)p0 * pol.N + 64, pol.N, pol.P - p0, pol.N - 64);
        const float before = st.before[at];
        if constexpr (Pol::SHARED) begin_head(h);
        bool odd = v.put(Bs) || odd_qk;
        if (blocks == 2) odd |= m.put(Bs + split3::TILE);
        odd = core.start(0, odd, q_products);
        v.load(vr, pol.ldv, ch.n, pol.P - p0);
        float w[8];
        auto make_weights = [&] {
            if constexpr (Pol::SHARED) weights(w, pol.row_terms(rec + t * Pol::RECORDS, before));
            else
#pragma unroll
                for (int i = 0; i < 8; ++i) w[i] = G[i];
        };
        make_weights();
        if constexpr (Pol::NORMALISER) {
            if (p0 == 0) {  // eight threads a row
                const RowTerms terms = pol.row_terms(rec + t * Pol::RECORDS, before);
                const float* n = S + (size_t)pol.P * pol.N;
                const float sum = sum8(w);
                float qn = 0.0f;
                if (t < ch.n)
                    for (int e = s0 / 2; e < pol.N; e += 32) {
                        const float4 a = load4(q + (size_t)t * pol.ldq + e), b = load4(n + e);
                        qn = fmaf(a.x, b.x, fmaf(a.y, b.y, fmaf(a.z, b.z, fmaf(a.w, b.w, qn))));
                    }
                row_sum[s0 / 8][t] = fmaf(terms.alpha, qn, sum);
                if (ch.last && tid == 0) {
                    float m = before;
                    pol.carry(st.aux[at], m);
                    pol.store_number(st.seq_slot[seq], h, m);
                }
            }
        }
        core.wait(0);
        if (reads) {  // times alpha (if that is all of it), and out of the way of the next products' sums
            const float alpha = odd ? 1.0f : pol.row_terms(rec + row * Pol::RECORDS, before).alpha;
#pragma unroll
            for (int c = 0; c < 16; c += 8) {
                float y[8];
                split3::sums_of<1>(y, lanes + c, q_steps);
#pragma unroll
                for (int i = 0; i < 8; ++i) y[i] *= alpha;
                sm100::tmem_st_8(lanes + 192 + c, y);
            }
            sm100::tmem_st_wait();
        }
        const bool odd_q = odd;
        odd |= split3::put8(w, Ws, t, s0 / 8);
        odd |= v.put(Vs);
        odd = core.start(1, odd, [&] {
            split3::issue<1, split3::K_STEP, split3::MN_STEP>(core.tmem, split3::B_MN, L / 16, split3::k_major(sm100::smem_u32(Ws)),
                                                              split3::mn_major(sm100::smem_u32(Vs), split3::PART));
        });
        if constexpr (Pol::NORMALISER)
            if (p0 == 0 && s0 == 0 && t < ch.n) {
                float parts[8];
#pragma unroll
                for (int i = 0; i < 8; ++i) parts[i] = row_sum[i][t];
                const float sum = sum8(parts);
                pol.store_sum(ch.first + t, h, sum, pol.row_terms(rec + t * Pol::RECORDS, before).extra);
            }
        core.wait(1);
        auto first8 = [&](float (&y)[8], int c) {
            uint32_t first[8];
            __syncwarp();
            sm100::tmem_ld_8_nowait(lanes + 192 + c, first);
            sm100::tmem_ld_wait_8(first);
#pragma unroll
            for (int i = 0; i < 8; ++i) y[i] = __uint_as_float(first[i]);
        };
        if (reads)
#pragma unroll
            for (int c = 0; c < 16; c += 8) {
                float y[8], first[8];
                split3::sums_of<1>(y, lanes + c, L / 16);
                first8(first, c);
                if (!odd_q)
#pragma unroll
                    for (int i = 0; i < 8; ++i) y[i] += first[i];
                spread(y, c);
            }
        const int r = Own::row(0), p = p0 + Own::col();
        float4 gate[2];
#pragma unroll
        for (int i = 0; i < 2; ++i) gate[i] = pol.gate(min(r, ch.n - 1) + ch.first, h, min(p + 4 * i, pol.P - 4));
        sm100::tc_fence_before_sync();
        __syncthreads();
        float y[8];
        read8(y, res + r * OLD + Own::col());
        __syncthreads();  // the results have been read
        if (odd) {  // the odd numbers' products
            float* weight = reinterpret_cast<float*>(Vs);
            if (odd_q && reads)
#pragma unroll 1
                for (int c = 0; c < 16; c += 8) {
                    float first[8];
                    first8(first, c);
                    spread(first, c);
                }
            make_weights();
#pragma unroll
            for (int i = 0; i < 8; ++i) weight[t * OLD + s0 + i] = w[i];
            __syncthreads();
            if (r < ch.n)
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    const int c = min(p + j, pol.P - 1) - p0;
                    if (odd_q) {
                        float a = res[r * OLD + Own::col() + j];
                        for (int e = 0; e < pol.N; ++e) {
                            const float x = q[(size_t)r * pol.ldq + e], m = S[(size_t)(p0 + c) * pol.N + e];
                            if (split3::is_odd(x) || split3::is_odd(m)) a = fmaf(x, m, a);
                        }
                        y[j] += __fmul_rn(pol.row_terms(rec + r * Pol::RECORDS, before).alpha, a);  // (rounded as without odd numbers)
                    }
                    for (int s = 0; s <= r; ++s) {
                        const float x = weight[r * OLD + s], m = vr[(size_t)s * pol.ldv + c];
                        if (split3::is_odd(x) || split3::is_odd(m)) y[j] = fmaf(x, m, y[j]);
                    }
                }
            __syncthreads();
        }
#pragma unroll
        for (int i = 0; i < 2; ++i)  // (P is a multiple of four)
            if (r < ch.n && p + 4 * i < pol.P)
                pol.store_row(ch.first + r, h, p + 4 * i, gate[i], make_float4(y[4 * i], y[4 * i + 1], y[4 * i + 2], y[4 * i + 3]),
                              make_float4(v.x[0][4 * i], v.x[0][4 * i + 1], v.x[0][4 * i + 2], v.x[0][4 * i + 3]));
    }
    core.close();
}

// Floats of scratch a chunk needs: its memories and what the other kernels read beside them.
inline long long chunk_floats(int heads, long long E, int records) { return heads * (E + 8 + 4 * L * records); }

template <class Pol>
int run(const Pol& pol, const int* seq_slot, const int* seq_row0, int n_seq, int R, int max_rows, float* scratch,
        int* err, cudaStream_t s) {
    const long long E = (long long)pol.P * pol.N + (Pol::NORMALISER ? pol.N : 0);
    const Plan plan = plan_rounds(R, n_seq, max_rows, L, chunk_floats(pol.heads, E, Pol::RECORDS));
    Step st;
    st.seq_slot = seq_slot;
    st.seq_row0 = seq_row0;
    st.err = err;
    const long long n_places = plan.places;
    st.scratch = scratch;
    st.aux = reinterpret_cast<float4*>(scratch + n_places * pol.heads * E);  // E is a multiple of four
    st.rows = st.aux + n_places * pol.heads;
    st.before = reinterpret_cast<float*>(st.rows + n_places * pol.heads * L * Pol::RECORDS);
    const int ptiles = (pol.P + PT - 1) / PT;
    const int chunks = plan.seg_rows / L;
    const int qk_heads = pol.heads / pol.per, items = pol.per * ptiles;
    // items a block: k (its products with the rows) and the weights, which serve them all, cost about as much as
    // one item; two blocks share an SM
    auto items_a_block = [&](int most) {
        int ipb = most;
        long long least = -1;
        for (int i = most; i >= 1; --i) {
            const long long blocks = (long long)chunks * plan.group * qk_heads * ((items + i - 1) / i);
            const long long cost = (blocks + 2 * sm_count() - 1) / (2 * sm_count()) * (1 + i);
            if (least < 0 || cost < least) {
                least = cost;
                ipb = i;
            }
        }
        return ipb;
    };
    const int ipb_state = items_a_block(min(items, (WARPS - 1) * ptiles));  // (a warp a head at most)
    const int ipb_out = items_a_block(items);
    const int sets_state = (items + ipb_state - 1) / ipb_state, sets_out = (items + ipb_out - 1) / ipb_out;
    if (n_seq > 65535 || (long long)pol.heads * ptiles > 65535) return RFX_ERR_UNSUPPORTED;
    cudaError_t e = cudaFuncSetAttribute(chunk_state_kernel<Pol>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SMEM);
    if (e != cudaSuccess) return (int)e;
    e = cudaFuncSetAttribute(chunk_out_kernel<Pol>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SMEM);
    if (e != cudaSuccess) return (int)e;
    for (int seq0 = 0; seq0 < n_seq; seq0 += plan.group)
        for (int seg = 0; seg < plan.n_segs; ++seg) {
            const int seqs = min(plan.group, n_seq - seq0);
            st.round = Round{plan.seg_rows, seg, seq0, plan.whole};
            RFX_LAUNCH(chunk_state_kernel<Pol>, dim3(chunks, seqs, qk_heads * sets_state), STATE_THREADS, SMEM, s, pol, st, ipb_state);
            RFX_LAUNCH(chunk_carry_kernel<Pol>, dim3((unsigned)((E / 4 + 127) / 128), seqs, pol.heads), 128, 0, s, pol, st);
            RFX_LAUNCH(chunk_out_kernel<Pol>, dim3(chunks, seqs, qk_heads * sets_out), OUT_THREADS, SMEM, s, pol, st, ipb_out);
        }
    return 0;
}

}  // namespace chunk
