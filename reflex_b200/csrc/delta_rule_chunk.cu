// The generalized delta rule (delta_rule.cu) for steps that bring a sequence many rows: 32 rows at a
// time, as products on the tensor cores of operands split in two (split_mma.cuh).  Heads of 64.
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
// 64 x 64 product a chunk and 16 value columns, a chain of about 0.7 us instead of 32 rows' walk of
// 0.35 us each.
//
// The factors W_t and 1 / W_s lie within e^(rate 32) of one (their products are what counts and keep
// their relative precision); rates for which that leaves 32 bits' range take the row-by-row walk.
// The memory itself stays 32-bit from chunk to chunk.
#include "attn_mma.cuh"
#include "chunk_plan.cuh"
#include "common.cuh"
#include "split_mma.cuh"

namespace {

using namespace rfx;

constexpr int L = 32, D = 64;
constexpr int LD = D + 8;   // rows read 8 bytes a lane along the channels
constexpr int VLD = D + 4;  // rows read down the rows
constexpr int SLD = L + 8;  // the rows' products with one another
// per (chunk, head): M [64][LD] and R [32][LD] in one piece, then the chunk's own sum [value][key]
constexpr int MR = (D + L) * LD, PLACE = MR + D * D;
constexpr int PREP_FLOATS = 4 * L * LD + 2 * L * VLD + 4 * L * SLD;  // 75 KB: three blocks an SM
constexpr int STAGES = 3;

struct Step {
    const int* seq_slot;
    const int* seq_row0;
    chunk::Round round;
    float* scratch;
};

__device__ __forceinline__ float sigmoid_f(float t) { return 1.0f / (1.0f + expf(-t)); }

// acc [16 rows m0 ..][8 N columns n0 ..] += sign * left^T right over the chunk's rows, both read down
// the rows (eight at a time from row 8 s on)
template <int N>
__device__ __forceinline__ void down_step(float (&acc)[N][4], const float* left, int lld, float sign,
                                          const float* right, int rld, int s, int g, int j) {
    const float* l = left + (8 * s + 2 * j) * lld + g;
    const Left a = left_from(sign * l[0], sign * l[8], sign * l[lld], sign * l[lld + 8]);
    const float* r = right + (8 * s + 2 * j) * rld + g;
    float2 b[N];
#pragma unroll
    for (int t = 0; t < N; ++t) b[t] = make_float2(r[8 * t], r[rld + 8 * t]);
    product3<N>(acc, a, b);
}
// acc += S right, S [t][s] read along s
template <int N>
__device__ __forceinline__ void along_step(float (&acc)[N][4], const float* S, const float* right, int rld, int s,
                                           int g, int j) {
    const float2 x = *reinterpret_cast<const float2*>(S + g * SLD + 8 * s + 2 * j);
    const float2 y = *reinterpret_cast<const float2*>(S + (g + 8) * SLD + 8 * s + 2 * j);
    const Left a = left_from(x.x, y.x, x.y, y.y);
    const float* r = right + (8 * s + 2 * j) * rld + g;
    float2 b[N];
#pragma unroll
    for (int t = 0; t < N; ++t) b[t] = make_float2(r[8 * t], r[rld + 8 * t]);
    product3<N>(acc, a, b);
}

// A block a (chunk, head); eight warps, since what bounds it is how many warps an SM holds to issue
// the short phases' instructions (with four warps and two blocks an SM 130 us for 2,000 rows of 32 heads).
__global__ void __launch_bounds__(256, 3)
delta_chunk_prep_kernel(const float* __restrict__ proj, int ld, int r_off, int k_off, int v_off, int a_off,
                        const float* __restrict__ wpre, const float* __restrict__ w_bias,
                        const float* __restrict__ a_bias, float rate, float unit_eps, Step st, float* __restrict__ out,
                        int heads) {
    extern __shared__ __align__(16) float sm[];
    float *Us = sm, *Rs = Us + L * LD, *Ks = Rs + L * LD, *Ps = Ks + L * LD, *Vs = Ps + L * LD, *Zs = Vs + L * VLD;
    float *As = Zs + L * VLD, *Bs = As + L * SLD, *Cs = Bs + L * SLD, *Es = Cs + L * SLD;
    __shared__ float wl[D];
    pdl_prologue();
    const int seq = st.round.seq0 + blockIdx.y, h = blockIdx.z;
    const int row0 = st.seq_row0[seq], from = row0 + st.round.seg * st.round.seg_rows;
    const int first = from + blockIdx.x * L, n = min(L, min(st.seq_row0[seq + 1], from + st.round.seg_rows) - first);
    if (n <= 0) return;
    const int hd = heads * D, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, j = lane & 3;
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
        store4(Vs + t * VLD + c, v);
        store4(ws + t * VLD + c, w);
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
                W *= ws[t * VLD + c];
            }
            wl[c] = W;
        } else if (part == 1) {
#pragma unroll 8
            for (int t = 0; t < L; ++t) {
                W *= ws[t * VLD + c];
                x[t * LD] *= W;
            }
        } else {
#pragma unroll 8
            for (int t = 0; t < L; ++t) {
                W *= ws[t * VLD + c];
                x[t * LD] *= 1.0f / W;
            }
        }
    }
    __syncthreads();
    // [u; r] [k; p]^T: a warp sixteen rows of u or r by the rows of k or p
    {
        const int m = warp & 3, to_p = warp >> 2, m0 = 16 * (m & 1);
        const float* left = sm + (16 * m + g) * LD + 2 * j;  // Rs follows Us
        const float* right = Ks + to_p * L * LD;
        float acc[4][4] = {};
#pragma unroll 2
        for (int s = 0; s < D / 8; ++s) {
            const float2 x = *reinterpret_cast<const float2*>(left + 8 * s);
            const float2 y = *reinterpret_cast<const float2*>(left + 8 * LD + 8 * s);
            const Left a = left_from(x.x, y.x, x.y, y.y);
            float2 b[4];
#pragma unroll
            for (int t = 0; t < 4; ++t) b[t] = *reinterpret_cast<const float2*>(right + (8 * t + g) * LD + 8 * s + 2 * j);
            product3<4>(acc, a, b);
        }
        const int own = m >> 1, ta = m0 + g, tb = ta + 8;      // rows of r meet their own row too
        float* to = As + (2 * own + to_p) * L * SLD;           // As, Bs, Cs, Es
        const float sign = own && to_p ? -1.0f : 1.0f;         // E is only ever taken off
#pragma unroll
        for (int t = 0; t < 4; ++t) {
            const int s = 8 * t + 2 * j;
            store2(to + ta * SLD + s, s < ta + own ? sign * acc[t][0] : 0.0f, s + 1 < ta + own ? sign * acc[t][1] : 0.0f);
            store2(to + tb * SLD + s, s < tb + own ? sign * acc[t][2] : 0.0f, s + 1 < tb + own ? sign * acc[t][3] : 0.0f);
        }
    }
    __syncthreads();
    {   // A V, the right side beside u W
        const int m0 = 16 * (warp & 1), n0 = 16 * (warp >> 1);
        float acc[2][4] = {};
        const int ks = m0 ? 4 : 2;
        for (int s = 0; s < ks; ++s) along_step<2>(acc, As + m0 * SLD, Vs + n0, VLD, s, g, j);
#pragma unroll
        for (int t = 0; t < 2; ++t) {
            store2(Zs + (m0 + g) * VLD + n0 + 8 * t + 2 * j, acc[t][0], acc[t][1]);
            store2(Zs + (m0 + g + 8) * VLD + n0 + 8 * t + 2 * j, acc[t][2], acc[t][3]);
        }
    }
    __syncthreads();
    if (tid < 2 * D) {  // (I + B) [Zl | Y] = [A V | u W], a column a thread, in place
        float* col = tid < D ? Zs + tid : Us + tid - D;
        const int cld = tid < D ? VLD : LD;
        float x[L];
#pragma unroll
        for (int t = 0; t < L; ++t) {
            float v = col[t * cld], v1 = 0.0f;
#pragma unroll
            for (int l = 0; l + 1 < t; l += 2) {
                const float2 b = *reinterpret_cast<const float2*>(Bs + t * SLD + l);
                v = fmaf(-b.x, x[l], v);
                v1 = fmaf(-b.y, x[l + 1], v1);
            }
            if (t & 1) v = fmaf(-Bs[t * SLD + t - 1], x[t - 1], v);
            x[t] = v + v1;
            col[t * cld] = x[t];
        }
    } else {  // k and p to the chunk's last row
        const int c = tid & (D - 1);
        const float w = wl[c];
        float* x = (tid < 3 * D ? Ks : Ps) + c;
#pragma unroll 8
        for (int t = 0; t < L; ++t) x[t * LD] *= w;
    }
    __syncthreads();
    float* place = st.scratch + (chunk::place_in(st.round, L, row0, seq, blockIdx.x) * heads + h) * PLACE;
    {   // C V - E Zl into the results, r W - E Y for the walk: sixteen rows by 32 columns a warp
        const int m0 = 16 * (warp & 1), half = (warp >> 1) & 1, n0 = 32 * (warp >> 2);
        const int ta = m0 + g, tb = ta + 8;
        float acc[4][4] = {};
        if (half) {
#pragma unroll
            for (int t = 0; t < 4; ++t) {
                const float2 x = *reinterpret_cast<const float2*>(Rs + ta * LD + n0 + 8 * t + 2 * j);
                const float2 y = *reinterpret_cast<const float2*>(Rs + tb * LD + n0 + 8 * t + 2 * j);
                acc[t][0] = x.x; acc[t][1] = x.y; acc[t][2] = y.x; acc[t][3] = y.y;
            }
        }
        const int ks = m0 ? 4 : 2;  // rows s <= t alone
        if (half) {
            for (int s = 0; s < ks; ++s) along_step<4>(acc, Es + m0 * SLD, Us + n0, LD, s, g, j);
        } else {
            for (int s = 0; s < ks; ++s) along_step<4>(acc, Es + m0 * SLD, Zs + n0, VLD, s, g, j);
            for (int s = 0; s < ks; ++s) along_step<4>(acc, Cs + m0 * SLD, Vs + n0, VLD, s, g, j);
        }
#pragma unroll
        for (int t = 0; t < 4; ++t) {
            const int c = n0 + 8 * t + 2 * j;
            if (half) {
                store2(place + (D + ta) * LD + c, acc[t][0], acc[t][1]);
                store2(place + (D + tb) * LD + c, acc[t][2], acc[t][3]);
            } else {
                if (ta < n) store2(out + (size_t)(first + ta) * hd + h * D + c, acc[t][0], acc[t][1]);
                if (tb < n) store2(out + (size_t)(first + tb) * hd + h * D + c, acc[t][2], acc[t][3]);
            }
        }
    }
    {   // the chunk's own sum [value][key] and M, sixteen rows by 32 key channels a warp each
        const int m0 = 16 * (warp & 3), n0 = 32 * (warp >> 2);
        float acc[4][4] = {};
#pragma unroll 1
        for (int s = 0; s < L / 8; ++s) {
            down_step<4>(acc, Vs + m0, VLD, 1.0f, Ks + n0, LD, s, g, j);
            down_step<4>(acc, Zs + m0, VLD, -1.0f, Ps + n0, LD, s, g, j);
        }
        float* sum = place + MR + (m0 + g) * D + n0 + 2 * j;
#pragma unroll
        for (int t = 0; t < 4; ++t) {
            store2(sum + 8 * t, acc[t][0], acc[t][1]);
            store2(sum + 8 * D + 8 * t, acc[t][2], acc[t][3]);
        }
#pragma unroll
        for (int t = 0; t < 4; ++t)
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int row = m0 + g + (i & 2 ? 8 : 0), c = n0 + 8 * t + 2 * j + (i & 1);
                acc[t][i] = row == c ? wl[c] : 0.0f;
            }
#pragma unroll 1
        for (int s = 0; s < L / 8; ++s) down_step<4>(acc, Ps + m0, LD, -1.0f, Us + n0, LD, s, g, j);
        float* M = place + (m0 + g) * LD + n0 + 2 * j;
#pragma unroll
        for (int t = 0; t < 4; ++t) {
            store2(M + 8 * t, acc[t][0], acc[t][1]);
            store2(M + 8 * LD + 8 * t, acc[t][2], acc[t][3]);
        }
    }
}

// A block a (sequence, head, 16 value columns) walks the chunks.  S^T is the left operand of both
// products, held whole (split) by each of the four warps; a warp makes sixteen key channels of the
// next S^T and eight of the chunk's rows, and the warps exchange their parts through shared memory,
// one barrier a chunk.  M and R of the next chunks arrive meanwhile.
__global__ void __launch_bounds__(128)
delta_chunk_walk_kernel(Step st, float* __restrict__ state, long long state_stride, long long state_off,
                        float* __restrict__ out, int heads) {
    extern __shared__ __align__(16) float sm[];
    __shared__ __align__(16) float4 part[2][D / 8][32];
    pdl_prologue();
    const int seq = st.round.seq0 + blockIdx.x, h = blockIdx.y, c0 = 16 * blockIdx.z;
    const int row0 = st.seq_row0[seq], from = row0 + st.round.seg * st.round.seg_rows;
    const int rows = min(st.seq_row0[seq + 1] - from, st.round.seg_rows);
    if (rows <= 0) return;
    const int chunks = (rows + L - 1) / L, hd = heads * D;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, j = lane & 3;
    const float* base = st.scratch + (chunk::place_in(st.round, L, row0, seq, 0) * heads + h) * PLACE;
    const size_t step = (size_t)heads * PLACE;
    auto fetch = [&](int c) {
        if (c < chunks) {
            const float* src = base + c * step;
            float* dst = sm + (c % STAGES) * MR;
            for (int e = tid; e < MR / 4; e += 128) attn::cp_async_16(dst + 4 * e, src + 4 * e, true);
        }
        attn::cp_async_commit();
    };
#pragma unroll
    for (int c = 0; c < STAGES; ++c) fetch(c);
    float* Sg = state + (size_t)st.seq_slot[seq] * state_stride + state_off + ((size_t)h * D + c0) * D;
    Left S[D / 8];
#pragma unroll
    for (int s = 0; s < D / 8; ++s) {
        const float2 x = *reinterpret_cast<const float2*>(Sg + (size_t)g * D + 8 * s + 2 * j);
        const float2 y = *reinterpret_cast<const float2*>(Sg + (size_t)(g + 8) * D + 8 * s + 2 * j);
        S[s] = left_from(x.x, y.x, x.y, y.y);
    }
    float own[2][4], next[2][4];  // the warp's tiles of S^T, and the chunk's own sum they start from
    auto sums = [&](int c) {
        const float* d = base + c * step + MR + (c0 + g) * D + 16 * warp + 2 * j;
#pragma unroll
        for (int t = 0; t < 2; ++t) {
            const float2 x = *reinterpret_cast<const float2*>(d + 8 * t);
            const float2 y = *reinterpret_cast<const float2*>(d + 8 * D + 8 * t);
            next[t][0] = x.x; next[t][1] = x.y; next[t][2] = y.x; next[t][3] = y.y;
        }
    };
    sums(0);
    attn::cp_async_wait<STAGES - 1>();
    __syncthreads();
    for (int c = 0; c < chunks; ++c) {
        const float* M = sm + (c % STAGES) * MR;
        const float* R = M + D * LD;
        const int first = from + c * L, t0 = 8 * warp + 2 * j;
        float* o = out + (size_t)(first + t0) * hd + h * D + c0 + g;
        const bool la = t0 < rows - c * L, lb = t0 + 1 < rows - c * L;
        float O[4] = {};
        if (la) {
            O[0] = o[0];
            O[2] = o[8];
        }
        if (lb) {
            O[1] = o[hd];
            O[3] = o[hd + 8];
        }
#pragma unroll
        for (int t = 0; t < 2; ++t)
#pragma unroll
            for (int i = 0; i < 4; ++i) own[t][i] = next[t][i];
        if (c + 1 < chunks) sums(c + 1);
        float Q[1][4] = {};
#pragma unroll
        for (int s = 0; s < D / 8; ++s) {
            float2 b[2], r[1];
#pragma unroll
            for (int t = 0; t < 2; ++t)
                b[t] = *reinterpret_cast<const float2*>(M + (16 * warp + 8 * t + g) * LD + 8 * s + 2 * j);
            r[0] = *reinterpret_cast<const float2*>(R + (8 * warp + g) * LD + 8 * s + 2 * j);
            product3<2>(own, S[s], b);
            product3<1>(Q, S[s], r);
        }
#pragma unroll
        for (int t = 0; t < 2; ++t)
            part[c & 1][2 * warp + t][lane] = make_float4(own[t][0], own[t][1], own[t][2], own[t][3]);
        if (la) {
            o[0] = O[0] + Q[0][0];
            o[8] = O[2] + Q[0][2];
        }
        if (lb) {
            o[hd] = O[1] + Q[0][1];
            o[hd + 8] = O[3] + Q[0][3];
        }
        attn::cp_async_wait<STAGES - 2>();
        __syncthreads();  // the parts and the next chunk's factors are there; this chunk's have been read
        fetch(c + STAGES);
#pragma unroll
        for (int s = 0; s < D / 8; ++s) {
            const float4 p = part[c & 1][s][lane];
            S[s] = left_from(p.x, p.z, p.y, p.w);
        }
    }
#pragma unroll
    for (int t = 0; t < 2; ++t) {
        float* to = Sg + (size_t)g * D + 16 * warp + 8 * t + 2 * j;
        store2(to, own[t][0], own[t][1]);
        store2(to + 8 * D, own[t][2], own[t][3]);
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
                                    float* scratch, int heads, int d, void* stream) {
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
    e = cudaFuncSetAttribute(delta_chunk_walk_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm_walk);
    if (e != cudaSuccess) return (int)e;
    for (int seq0 = 0; seq0 < n_seq; seq0 += plan.group)
        for (int seg = 0; seg < plan.n_segs; ++seg) {
            const int seqs = min(plan.group, n_seq - seq0);
            st.round = chunk::Round{plan.seg_rows, seg, seq0, plan.whole};
            RFX_LAUNCH(delta_chunk_prep_kernel, dim3(chunks, seqs, heads), 256, sm_prep, s, proj, ld, r_off, k_off, v_off,
                       a_off, wpre, w_bias, a_bias, rate, unit_eps, st, out, heads);
            RFX_LAUNCH(delta_chunk_walk_kernel, dim3(seqs, heads, D / 16), 128, sm_walk, s, st, state, state_stride,
                       state_off, out, heads);
        }
    return 0;
}
