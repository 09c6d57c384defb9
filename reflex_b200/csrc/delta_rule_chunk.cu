// The generalized delta rule (delta_rule.cu) for steps that bring a sequence many rows: 32 rows at a
// time, as products of 32-bit multiply-adds.  Heads of 64.
//
// With W_t the product of the decays from the chunk's first row to t (per key channel), z_t = S^T u_t
// what row t removes, S0 the memory before the chunk, and
//     A_ts = (u_t W_{t-1}) . (k_s / W_s),   B_ts = (u_t W_{t-1}) . (p_s / W_s)   for s < t, p = a * u,
//     C_ts = (r_t W_t) . (k_s / W_s),       E_ts = (r_t W_t) . (p_s / W_s)       for s <= t,
// the rows depend on one another through (I + B) Z = (u W) S0 + A V alone.  Solved for both right
// sides at once, Z = Y S0 + Zl, and then, with k', p' = k, p times W_last / W_s,
//     o      = (r W - E Y) S0 + (C V - E Zl)
//     S_last = (diag(W_last) - p'^T Y) S0 + (k'^T V - p'^T Zl).
// Everything but S0 is the chunk's own: delta_chunk_prep_kernel makes the four factors for all chunks
// side by side (C V - E Zl straight into the results), and delta_chunk_walk_kernel is left with one
// product of 96 x 64 with the memory a chunk, a chain of about 1.4 us instead of 32 rows' walk of 0.35 us
// each.
//
// As products on the tensor cores of operands split in two parts of 11 bits both kernels were about 60 us
// faster for 2,048 rows of 32 heads, and eleven times as far from 64 bits as the walk (1.1e-6 against
// 9.7e-8); these are 1.3e-7 off, the state 9.8e-8 (7e-8 walking).
//
// The factors W_t and 1 / W_s lie within e^(rate 32) of one (their products are what counts and keep
// their relative precision); rates for which that leaves 32 bits' range take the row-by-row walk.
// The memory itself stays 32-bit from chunk to chunk.
#include "attn_mma.cuh"
#include "chunk_plan.cuh"
#include "common.cuh"
#include "fma_tiles.cuh"
#include "sm100.cuh"

namespace {

using namespace rfx;

constexpr int L = 32, D = 64;
constexpr int LD = D + 4;   // an odd number of 16 bytes: eight rows side by side meet all banks
constexpr int SLD = L + 4;  // the rows' products with one another
// per (chunk, head): M [64][LD] and R [32][LD] in one piece, then the chunk's own sum [key][value]
constexpr int MR = (D + L) * LD, PLACE = MR + D * D;
constexpr int PREP_FLOATS = 6 * L * LD + 4 * L * SLD;  // 70 KB
constexpr int STAGES = 3;

struct Step {
    const int* seq_slot;
    const int* seq_row0;
    chunk::Round round;
    float* scratch;
};

__device__ __forceinline__ float sigmoid_f(float t) { return 1.0f / (1.0f + expf(-t)); }

// A block a (chunk, head), eight warps; two halves of them where there are two things to do.  What
// is not finite in a row reaches that row's results and later ones alone: products between rows take
// the rows that count, not zeros for the others.
__global__ void __launch_bounds__(256, 2)
delta_chunk_prep_kernel(const float* __restrict__ proj, int ld, int r_off, int k_off, int v_off, int a_off,
                        const float* __restrict__ wpre, const float* __restrict__ w_bias,
                        const float* __restrict__ a_bias, float rate, float unit_eps, Step st, float* __restrict__ out,
                        int heads) {
    extern __shared__ __align__(16) float sm[];
    float *Us = sm, *Rs = Us + L * LD, *Ks = Rs + L * LD, *Ps = Ks + L * LD, *Vs = Ps + L * LD, *Zs = Vs + L * LD;
    float *As = Zs + L * LD, *Bs = As + L * SLD, *Cs = Bs + L * SLD, *Es = Cs + L * SLD;
    __shared__ __align__(16) float wl[D];
    pdl_prologue();
    const int seq = st.round.seq0 + blockIdx.y, h = blockIdx.z;
    const int row0 = st.seq_row0[seq], from = row0 + st.round.seg * st.round.seg_rows;
    const int first = from + blockIdx.x * L, n = min(L, min(st.seq_row0[seq + 1], from + st.round.seg_rows) - first);
    if (n <= 0) return;
    const int hd = heads * D, tid = threadIdx.x;
    float* ws = Zs;  // the rows' decays, until the right sides take their place
#pragma unroll
    for (int i = 0; i < L * (D / 4) / 256; ++i) {
        const int e = tid + 256 * i, t = e / (D / 4), c = 4 * (e % (D / 4));
        float4 r = make_float4(0.0f, 0.0f, 0.0f, 0.0f), k = r, v = r, a = r, w = make_float4(1.0f, 1.0f, 1.0f, 1.0f);
        if (t < n) {
            const float* pr = proj + (size_t)(first + t) * ld + h * D + c;
            r = load4(pr + r_off);
            k = load4(pr + k_off);
            v = load4(pr + v_off);
            const float4 ap = load4(pr + a_off), ab = load4(a_bias + h * D + c);
            const float4 wp = load4(wpre + (size_t)(first + t) * hd + h * D + c), wb = load4(w_bias + h * D + c);
            a = make_float4(sigmoid_f(ap.x + ab.x), sigmoid_f(ap.y + ab.y), sigmoid_f(ap.z + ab.z), sigmoid_f(ap.w + ab.w));
            w = make_float4(expf(-rate * sigmoid_f(wp.x + wb.x)), expf(-rate * sigmoid_f(wp.y + wb.y)),
                            expf(-rate * sigmoid_f(wp.z + wb.z)), expf(-rate * sigmoid_f(wp.w + wb.w)));
        }
        // the unit key: a row's sixteen threads are neighbours
        float kk = fmaf(k.x, k.x, fmaf(k.y, k.y, fmaf(k.z, k.z, k.w * k.w)));
#pragma unroll
        for (int o = 1; o < 16; o <<= 1) kk += __shfl_xor_sync(0xffffffffu, kk, o);
        const float inv = t < n ? 1.0f / sqrtf(kk + unit_eps) : 0.0f;  // (no row, no unit key, whatever unit_eps is)
        const float4 u = make_float4(k.x * inv, k.y * inv, k.z * inv, k.w * inv);
        store4(Us + t * LD + c, u);
        store4(Rs + t * LD + c, r);
        store4(Ks + t * LD + c, k);
        store4(Ps + t * LD + c, make_float4(a.x * u.x, a.y * u.y, a.z * u.z, a.w * u.w));
        store4(Vs + t * LD + c, v);
        store4(ws + t * LD + c, w);
    }
    __syncthreads();
    // the decays' products, multiplied row by row (neighbouring rows' ratios are then exact to the
    // last bit but one); a channel a thread, one array of u, r, k and p each to two warps
    {
        const int c = tid & (D - 1), part = tid >> 6;
        float W = 1.0f;
        float* x = sm + part * L * LD + c;
        if (part == 0) {
#pragma unroll 8
            for (int t = 0; t < L; ++t) {
                x[t * LD] *= W;
                W *= ws[t * LD + c];
            }
            wl[c] = W;
        } else if (part == 1) {
#pragma unroll 8
            for (int t = 0; t < L; ++t) {
                W *= ws[t * LD + c];
                x[t * LD] *= W;
            }
        } else {
#pragma unroll 8
            for (int t = 0; t < L; ++t) {
                W *= ws[t * LD + c];
                x[t * LD] *= 1.0f / W;
            }
        }
    }
    __syncthreads();
    // [u; r] [k; p]^T, rows s <= t (r) or s < t (u) alone: a thread four rows of u or r by rows tx, tx + 16
    // of k and p
    {
        const int tx = tid & 15, m0 = 4 * (tid >> 4), t0 = m0 & (L - 1), own = m0 >= L;
        const float *a = Us + m0 * LD, *b = Ks + tx * LD;  // Rs follows Us, Ps Ks
        float* to = As + 2 * own * L * SLD + t0 * SLD + tx;  // As, Bs, Cs, Es
        auto store = [&](int to_p, int s, const float (&v)[4]) {
            const float sign = own && to_p ? -1.0f : 1.0f;  // E is only ever taken off
#pragma unroll
            for (int i = 0; i < 4; ++i) to[to_p * L * SLD + i * SLD + 16 * s] = tx + 16 * s < t0 + i + own ? sign * v[i] : 0.0f;
        };
        if (t0 < 16) {
            float acc[4][2] = {};
            product_along<2>(acc, a, LD, b, L * LD, D / 16);
            const float k[4] = {acc[0][0], acc[1][0], acc[2][0], acc[3][0]}, p[4] = {acc[0][1], acc[1][1], acc[2][1], acc[3][1]};
            store(0, 0, k);
            store(1, 0, p);
        } else {
            float acc[4][4] = {};
            product_along<4>(acc, a, LD, b, 16 * LD, D / 16);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float v[4] = {acc[0][j], acc[1][j], acc[2][j], acc[3][j]};
                store(j >> 1, j & 1, v);
            }
        }
    }
    __syncthreads();
    const int u = tid & 127, tx = u & 15, ty = u >> 4;  // 4 rows (8 for a 64 x 64 result) by 4 columns
    const bool upper = tid >= 128;
    for (int e = tid; e < 2 * L * (D / 4); e += 256) {  // k and p to the chunk's last row
        float* x = Ks + (e / (D / 4)) * LD + 4 * (e % (D / 4));
        const float4 v = load4(x), w = load4(wl + 4 * (e % (D / 4)));
        store4(x, make_float4(v.x * w.x, v.y * w.y, v.z * w.z, v.w * w.w));
    }
    float acc[4][4] = {};  // upper: C V - E Zl, the chunk's own results; lower: A V, the right side beside u W
    if (upper) {
        product_below<false>(acc, Cs + 4 * ty * SLD, SLD, Vs + 4 * tx, LD, ty);
    } else {
        product_below<true>(acc, As + 4 * ty * SLD, SLD, Vs + 4 * tx, LD, ty);
#pragma unroll
        for (int i = 0; i < 4; ++i) store4(Zs + (4 * ty + i) * LD + 4 * tx, make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]));
    }
    __syncthreads();
    // upper: the chunk's own sum [key 4 ty .., 32 + 4 ty ..][value 4 tx ..]; lower: M
    float total[2][4][4] = {};
    if (!upper) {  // (I + B) [Zl | Y] = [A V | u W], a column a thread, in place
        float* col = u < D ? Zs + u : Us + u - D;
        float x[L];
#pragma unroll
        for (int t = 0; t < L; ++t) {
            float v = col[t * LD], v1 = 0.0f;
#pragma unroll
            for (int l = 0; l + 3 < t; l += 4) {
                const float4 b = load4(Bs + t * SLD + l);
                v = fmaf(-b.x, x[l], v);
                v1 = fmaf(-b.y, x[l + 1], v1);
                v = fmaf(-b.z, x[l + 2], v);
                v1 = fmaf(-b.w, x[l + 3], v1);
            }
#pragma unroll
            for (int l = t / 4 * 4; l < t; ++l) {
                if (l & 1) v1 = fmaf(-Bs[t * SLD + l], x[l], v1);
                else v = fmaf(-Bs[t * SLD + l], x[l], v);
            }
            x[t] = v + v1;
            col[t * LD] = x[t];
        }
    } else {
        product_down(total, Ks + 4 * ty, LD, L, Vs + 4 * tx, LD, L);
    }
    __syncthreads();
    float* place = st.scratch + (chunk::place_in(st.round, L, row0, seq, blockIdx.x) * heads + h) * PLACE;
    // r W - E Y for the walk (lower), C V - E Zl into the results (upper)
    if (!upper) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float4 r = load4(Rs + (4 * ty + i) * LD + 4 * tx);
            acc[i][0] = r.x; acc[i][1] = r.y; acc[i][2] = r.z; acc[i][3] = r.w;
        }
    }
    product_below<false>(acc, Es + 4 * ty * SLD, SLD, (upper ? Zs : Us) + 4 * tx, LD, ty);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int t = 4 * ty + i;
        const float4 v = make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
        if (!upper) store4(place + (D + t) * LD + 4 * tx, v);
        else if (t < n) store4(out + (size_t)(first + t) * hd + h * D + 4 * tx, v);
    }
    // the chunk's own sum - p'^T Zl (upper), M = diag(W_last) - p'^T Y (lower)
    product_down<true>(total, Ps + 4 * ty, LD, L, (upper ? Zs : Us) + 4 * tx, LD, L);
    float* to = (upper ? place + MR : place) + 4 * tx;
    const int ld_to = upper ? D : LD;
#pragma unroll
    for (int half = 0; half < 2; ++half)
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int key = 32 * half + 4 * ty + i;
            if (!upper) {
                const float w = wl[key];
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    if (key == 4 * tx + j) total[half][i][j] += w;
            }
            store4(to + key * ld_to, make_float4(total[half][i][0], total[half][i][1], total[half][i][2], total[half][i][3]));
        }
}

// A block a (sequence, head, COLS value columns) walks the chunks: [M; R] S, 96 rows by COLS columns over 64
// key channels.  Four lanes make a tile of 4 x 4, each a quarter of the channels (four of each
// sixteen), whose parts meet by shuffles, so that a chunk has one barrier.  (The quarters in warps of
// their own, meeting in shared memory: no faster; a thread a row and eight columns, all channels:
// 121 us in place of 99 for 64 chunks of 32 heads.)  M and R of the next chunks arrive meanwhile, a
// chunk's by one bulk copy (by all threads, 16 bytes each, a quarter of a step's time went into issuing
// the copies).  What bounds a step is the latency of its reads of shared memory.  Four sequences of 571, 714, 428
// and 286 rows of 32 heads: 75 us; 105 with copies by all threads and sequences in their own order.  Sixteen columns a block, eight where
// that leaves SMs without a block: both kernels take 224 and 282 us for 2,048 rows of 32 heads with
// eight and sixteen, 441 and 412 for 64 heads.
constexpr int TLD = D + 16;  // sixteen floats more: two columns' sixteens meet all banks
template <int COLS>
__global__ void __launch_bounds__(COLS * (D + L) / 4)
delta_chunk_walk_kernel(Step st, float* __restrict__ state, long long state_stride, long long state_off,
                        float* __restrict__ out, int heads, int* err) {
    constexpr int CG = COLS / 4, THREADS = CG * (D + L);
    extern __shared__ __align__(16) float sm[];
    __shared__ __align__(16) float Ss[2][COLS * TLD];  // S^T, column 4 c + j at row CG j + c
    __shared__ uint64_t full[STAGES];
    if (threadIdx.x == 0) {
        for (int i = 0; i < STAGES; ++i) sm100::mbar_init(&full[i], 1);
        sm100::fence_barrier_init();
    }
    pdl_prologue();
    // the longest sequences' blocks first (up to 32 of them are put in order)
    auto rows_of = [&](int s) {
        const int from = st.seq_row0[s] + st.round.seg * st.round.seg_rows;
        return min(st.seq_row0[s + 1] - from, st.round.seg_rows);
    };
    int seq = st.round.seq0 + blockIdx.z;
    if (gridDim.z > 1 && gridDim.z <= 32) {
        const int lane = threadIdx.x & 31, n = gridDim.z, mine = lane < n ? rows_of(st.round.seq0 + lane) : 0;
        int longer = 0;
        for (int i = 0; i < n; ++i) {
            const int other = __shfl_sync(0xffffffffu, mine, i);
            longer += other > mine || (other == mine && i < lane);
        }
        seq = st.round.seq0 + __ffs(__ballot_sync(0xffffffffu, lane < n && longer == blockIdx.z)) - 1;
    }
    const int h = blockIdx.y, c0 = COLS * blockIdx.x;
    const int row0 = st.seq_row0[seq], from = row0 + st.round.seg * st.round.seg_rows, rows = rows_of(seq);
    if (rows <= 0) return;
    const int chunks = (rows + L - 1) / L, hd = heads * D, tid = threadIdx.x;
    const int quarter = tid & 3, cg = tid >> 2 & (CG - 1), first_row = 4 * (tid / COLS);  // the tile's first row
    const int row = first_row + quarter, c = c0 + 4 * cg;  // whose results the lane ends up with, and their columns
    const float* base = st.scratch + (chunk::place_in(st.round, L, row0, seq, 0) * heads + h) * PLACE;
    const size_t step = (size_t)heads * PLACE;
    // a chunk's factors lie in one piece: one copy of 26 KB, issued by one thread
    auto fetch = [&](int k, int to) {
        if (k < chunks) {
            sm100::mbar_expect_tx(&full[to], MR * sizeof(float));
            sm100::bulk_load(sm + to * MR, base + k * step, MR * sizeof(float), &full[to]);
        }
    };
    if (tid == 0)
        for (int k = 0; k < STAGES; ++k) fetch(k, k);
    float* Sg = state + (size_t)st.seq_slot[seq] * state_stride + state_off + (size_t)h * D * D;
    for (int e = tid; e < COLS * D / 4; e += THREADS) {
        const int col = e / (D / 4), k = 4 * (e % (D / 4));
        store4(Ss[0] + (CG * (col % 4) + col / 4) * TLD + k, load4(Sg + (size_t)(c0 + col) * D + k));
    }
    float4 own = make_float4(0.0f, 0.0f, 0.0f, 0.0f), next = own;  // what the products are added to: the chunk's
    auto ahead = [&](int k) {                                       // own sum, or its own results
        if (row < D) next = load4(base + k * step + MR + row * D + c);
        else if (row - D < rows - k * L) next = load4(out + (size_t)(from + k * L + row - D) * hd + h * D + c);
    };
    ahead(0);
    __syncthreads();
    int at = 0, round = 0;
    bool waits = true;  // a wait that ran out is reported, and the walk ends with whatever is there
    for (int k = 0; k < chunks; ++k) {
        const int now = at;
        if (waits && !sm100::mbar_wait(&full[now], round & 1)) {
            waits = false;
            if (err) atomicExch(err, 43);
            if (tid == 0)  // no copy is begun any more; those on their way get as long again each
                for (int i = k; i < min(chunks, k + STAGES); ++i) sm100::mbar_wait(&full[i % STAGES], i / STAGES & 1);
        }
        const float* m = sm + at * MR + first_row * LD + 4 * quarter;
        const float* S = Ss[k & 1] + cg * TLD + 4 * quarter;
        float* Sn = Ss[(k + 1) & 1];
        if (++at == STAGES) {
            at = 0;
            ++round;
        }
        own = next;
        if (k + 1 < chunks) ahead(k + 1);
        float acc[4][4] = {};
#pragma unroll
        for (int s = 0; s < D; s += 16) {
            float4 x[4], y[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) x[i] = load4(m + i * LD + s);
#pragma unroll
            for (int j = 0; j < 4; ++j) y[j] = load4(S + CG * j * TLD + s);
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    acc[i][j] = fmaf(x[i].x, y[j].x, acc[i][j]);
                    acc[i][j] = fmaf(x[i].y, y[j].y, acc[i][j]);
                    acc[i][j] = fmaf(x[i].z, y[j].z, acc[i][j]);
                    acc[i][j] = fmaf(x[i].w, y[j].w, acc[i][j]);
                }
        }
        // row i's four parts to lane i of the four
        const bool odd = quarter & 1, high = quarter & 2;
        float half[2][4], sum[4];
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float give = odd ? acc[2 * i][j] : acc[2 * i + 1][j];
                half[i][j] = (odd ? acc[2 * i + 1][j] : acc[2 * i][j]) + __shfl_xor_sync(0xffffffffu, give, 1);
            }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const float give = high ? half[0][j] : half[1][j];
            sum[j] = (high ? half[1][j] : half[0][j]) + __shfl_xor_sync(0xffffffffu, give, 2);
        }
        own.x += sum[0];
        own.y += sum[1];
        own.z += sum[2];
        own.w += sum[3];
        if (row < D) {
            Sn[cg * TLD + row] = own.x;
            Sn[(CG + cg) * TLD + row] = own.y;
            Sn[(2 * CG + cg) * TLD + row] = own.z;
            Sn[(3 * CG + cg) * TLD + row] = own.w;
        } else if (row - D < rows - k * L) {
            store4(out + (size_t)(from + k * L + row - D) * hd + h * D + c, own);
        }
        __syncthreads();  // the next S is there; this chunk's factors have been read
        if (tid == 0 && waits) fetch(k + STAGES, now);
    }
    if (row < D) {
        float* s = Sg + (size_t)c * D + row;
        s[0] = own.x;
        s[D] = own.y;
        s[2 * D] = own.z;
        s[3 * D] = own.w;
    }
}

inline chunk::Plan plan_of(int R, int n_seq, int max_rows, int heads) {
    return chunk::plan_rounds(R, n_seq, max_rows, L, (long long)heads * PLACE);
}

}  // namespace

// Floats of scratch rfx_delta_rule_chunk needs for a step of R rows in n_seq sequences of at most max_rows.
extern "C" long long rfx_delta_rule_chunk_floats(int R, int n_seq, int max_rows, int heads) {
    return plan_of(R, n_seq, max_rows, heads).places * heads * PLACE;
}

// As rfx_delta_rule with 32-bit results and the state [heads][value column][key channel].  d 64, rates
// from 0 to 2; rows, biases, state, results and `scratch` on 16 bytes.  RFX_ERR_UNSUPPORTED otherwise.
extern "C" int rfx_delta_rule_chunk(const float* proj, int ld, int r_off, int k_off, int v_off, int a_off,
                                    const float* wpre, const float* w_bias, const float* a_bias, float rate,
                                    float unit_eps, float* state, long long state_stride, long long state_off,
                                    const int* seq_slot, const int* seq_row0, int n_seq, int R, int max_rows, float* out,
                                    float* scratch, int heads, int d, int* err, void* stream) {
    if (n_seq <= 0 || R <= 0 || max_rows <= 0) return 0;
    if (heads <= 0 || d <= 0) return RFX_ERR_BAD_ARG;
    if (d != D || !(rate >= 0.0f && rate <= 2.0f) || n_seq > 65535 || heads > 65535 ||
        ((ld | r_off | k_off | v_off | a_off) & 3) || ((state_stride | state_off) & 3) ||
        ((reinterpret_cast<uintptr_t>(proj) | reinterpret_cast<uintptr_t>(wpre) | reinterpret_cast<uintptr_t>(w_bias) |
          reinterpret_cast<uintptr_t>(a_bias) | reinterpret_cast<uintptr_t>(state) | reinterpret_cast<uintptr_t>(out) |
          reinterpret_cast<uintptr_t>(scratch)) & 15))
        return RFX_ERR_UNSUPPORTED;
    cudaStream_t s = (cudaStream_t)stream;
    Step st;
    st.seq_slot = seq_slot;
    st.seq_row0 = seq_row0;
    st.scratch = scratch;
    const chunk::Plan plan = plan_of(R, n_seq, max_rows, heads);
    const int chunks = plan.seg_rows / L;
    constexpr size_t sm_prep = PREP_FLOATS * sizeof(float), sm_walk = (size_t)STAGES * MR * sizeof(float);
    cudaError_t e = cudaFuncSetAttribute(delta_chunk_prep_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm_prep);
    if (e != cudaSuccess) return (int)e;
    const bool narrow = (long long)plan.group * heads * (D / 16) <= sm_count();
    e = narrow ? cudaFuncSetAttribute(delta_chunk_walk_kernel<8>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm_walk)
               : cudaFuncSetAttribute(delta_chunk_walk_kernel<16>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm_walk);
    if (e != cudaSuccess) return (int)e;
    for (int seq0 = 0; seq0 < n_seq; seq0 += plan.group)
        for (int seg = 0; seg < plan.n_segs; ++seg) {
            const int seqs = min(plan.group, n_seq - seq0);
            st.round = chunk::Round{plan.seg_rows, seg, seq0, plan.whole};
            RFX_LAUNCH(delta_chunk_prep_kernel, dim3(chunks, seqs, heads), 256, sm_prep, s, proj, ld, r_off, k_off, v_off,
                       a_off, wpre, w_bias, a_bias, rate, unit_eps, st, out, heads);
            if (narrow)
                RFX_LAUNCH(delta_chunk_walk_kernel<8>, dim3(D / 8, heads, seqs), 2 * (D + L), sm_walk, s, st, state,
                           state_stride, state_off, out, heads, err);
            else
                RFX_LAUNCH(delta_chunk_walk_kernel<16>, dim3(D / 16, heads, seqs), 4 * (D + L), sm_walk, s, st, state,
                           state_stride, state_off, out, heads, err);
        }
    return 0;
}
