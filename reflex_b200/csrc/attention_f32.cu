// The plain attention (attention_plain.cu) of the true 32-bit path, 32 keys and up to sixteen queries
// at a time: the same operations on the same numbers in the same order, so the same bits, for head
// sizes of 32, 64, 128 and 256.
//
// The plain kernel's warp walks the keys one after another; every key costs it a butterfly, two
// exponentials and two loads' latency in a chain (a query of 300 keys: 0.2 ms).  Here the queries of
// up to four rows and the query heads of one key/value head form a block, and 32 keys' rows come to
// shared memory once for all of them:
//   scores      a lane a key.  What the plain kernel's lane l sums over elements l, l + 32, .. is a
//               chain of this lane's; the 32 chains meet in the butterfly's order, so the sum's bits do.
//   softmax     running maxima by a scan (a maximum has no rounding), then both exponentials of all
//               keys side by side.
//   values      the lanes over a head's elements, key after key: l = fma(l, corr, p),
//               acc = fma(acc, corr, p * v).
// Reads of shared memory and a tile's chain of steps bound it (9,000 cycles a tile of 32 keys with two blocks an
// SM).  8 heads of 128 for prompts of 155, 311 and 235 rows: 50 us; 65 with the early rows' blocks first and a
// page looked up by every copying thread for each of its rows.  24 heads, 8 prompts of 709 rows in all: 53 (65).
#include "attn_mma.cuh"
#include "common.cuh"
#include "exact_math.cuh"
#include "paged.cuh"

namespace {

using namespace rfx;

constexpr int KEYS = 32, WARPS = 8, QUERIES = 2 * WARPS;

// The score of a lane's key with U queries (`q` of them `step` apart): 32 chains over d / 32 elements,
// met as a butterfly over lanes meets them.
template <int NI, int U>
__device__ __forceinline__ void dots(const float* k, const float* q, int step, float (&s)[U]) {
    constexpr int d = 32 * NI;
    float4 t4[U];
#pragma unroll
    for (int a = 0; a < 2; ++a) {
        float4 t8[U];
#pragma unroll
        for (int b = 0; b < 2; ++b) {
            float4 t16[U];
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                const int l0 = 4 * a + 8 * b + 16 * c;
                float4 p[U];
#pragma unroll
                for (int u = 0; u < U; ++u) p[u] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll
                for (int i = 0; i < NI; ++i) {
                    const float4 x = *reinterpret_cast<const float4*>(k + l0 + 32 * i);
#pragma unroll
                    for (int u = 0; u < U; ++u) {
                        const float4 y = *reinterpret_cast<const float4*>(q + u * step * d + l0 + 32 * i);
                        p[u].x = fmaf(y.x, x.x, p[u].x);
                        p[u].y = fmaf(y.y, x.y, p[u].y);
                        p[u].z = fmaf(y.z, x.z, p[u].z);
                        p[u].w = fmaf(y.w, x.w, p[u].w);
                    }
                }
#pragma unroll
                for (int u = 0; u < U; ++u)
                    t16[u] = c ? make_float4(t16[u].x + p[u].x, t16[u].y + p[u].y, t16[u].z + p[u].z, t16[u].w + p[u].w) : p[u];
            }
#pragma unroll
            for (int u = 0; u < U; ++u)
                t8[u] = b ? make_float4(t8[u].x + t16[u].x, t8[u].y + t16[u].y, t8[u].z + t16[u].z, t8[u].w + t16[u].w) : t16[u];
        }
#pragma unroll
        for (int u = 0; u < U; ++u)
            t4[u] = a ? make_float4(t4[u].x + t8[u].x, t4[u].y + t8[u].y, t4[u].z + t8[u].z, t4[u].w + t8[u].w) : t8[u];
    }
#pragma unroll
    for (int u = 0; u < U; ++u) s[u] = (t4[u].x + t4[u].z) + (t4[u].y + t4[u].w);
}

// elements NI lane .. of a row
template <int NI>
__device__ __forceinline__ void load_own(const float* row, int lane, float (&v)[NI]) {
    if constexpr (NI == 1) v[0] = row[lane];
    else if constexpr (NI == 2) {
        const float2 x = *reinterpret_cast<const float2*>(row + 2 * lane);
        v[0] = x.x;
        v[1] = x.y;
    } else {
#pragma unroll
        for (int i = 0; i < NI / 4; ++i) {
            const float4 x = *reinterpret_cast<const float4*>(row + 4 * (lane + 32 * i));
            v[4 * i] = x.x;
            v[4 * i + 1] = x.y;
            v[4 * i + 2] = x.z;
            v[4 * i + 3] = x.w;
        }
    }
}
template <int NI>
__device__ __forceinline__ int own_element(int lane, int i) {
    return NI <= 2 ? NI * lane + i : 4 * (lane + 32 * (i / 4)) + i % 4;
}

struct Args {
    const float *q, *k_pages, *v_pages;
    PagedKV cache;
    const int *seq_slot, *seq_start, *seq_new, *seq_row0;
    float* out;
    int nq, heads, rows;  // query heads and rows a block takes
    int seqs;
    int window, keep_first;
    float scale;
    const float *sink, *slopes;
    float softcap;
};

template <int NI>
__global__ void __launch_bounds__(WARPS * 32, NI > 4 ? 1 : 2) attention_f32_kernel(Args A) {
    constexpr int d = 32 * NI, KLD = d + 4, d4 = d / 4;
    extern __shared__ __align__(16) float sm[];
    float *Qs = sm, *Ks = Qs + QUERIES * d, *Vs = Ks + 2 * KEYS * KLD;
    float2* Ws = reinterpret_cast<float2*>(Vs + 2 * KEYS * d);  // [WARPS][2][KEYS]: corr, p
    pdl_prologue();
    const int group = A.nq / A.cache.n_kv_heads, parts = (group + A.heads - 1) / A.heads, sets = A.cache.n_kv_heads * parts;
    // late rows have many keys, early ones few: the latest ones first
    const int set = blockIdx.x % sets, seq = blockIdx.x / sets % A.seqs;
    const int n_new = A.seq_new[seq], row_first = (int)((gridDim.x - 1 - blockIdx.x) / (sets * A.seqs)) * A.rows;
    if (row_first >= n_new) return;
    const int n_rows = min(A.rows, n_new - row_first);
    const int kvh = set / parts, h0 = kvh * group + (set - kvh * parts) * A.heads;
    const int n_heads = min(A.heads, (kvh + 1) * group - h0);
    const int slot = A.seq_slot[seq], p_first = A.seq_start[seq] + row_first, p_last = p_first + n_rows - 1;
    const int row0 = A.seq_row0[seq] + row_first;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    auto low = [&](int pos) { return A.window > 0 && pos + 1 > A.window ? pos + 1 - A.window : 0; };
    const int lo_first = low(p_first), kept_last = min(A.keep_first, low(p_last));
    // keys some row of the block sees: those before kept_last, and lo_first .. p_last
    auto next = [&](int t) {
        ++t;
        return KEYS * t >= kept_last && KEYS * t + KEYS - 1 < lo_first ? lo_first / KEYS : t;
    };
    // a page holds whole tiles (or not: then every row looks its place up); a tile's page is asked for a tile ahead
    const bool whole = A.cache.page_size % KEYS == 0;
    auto place = [&](int t) { return whole && t <= p_last / KEYS ? kv_offset(A.cache, slot, KEYS * t, kvh) : 0; };
    auto fetch = [&](int t, int buf, size_t base) {
#pragma unroll
        for (int e = tid; e < KEYS * d4; e += WARPS * 32) {
            const int i = e / d4, c = 4 * (e - i * d4), j = KEYS * t + i;
            const bool ok = j <= p_last && (j < kept_last || j >= lo_first);
            const size_t at = !ok ? 0 : whole ? base + i * d + c : kv_offset(A.cache, slot, j, kvh) + c;
            attn::cp_async_16(Ks + (buf * KEYS + i) * KLD + c, A.k_pages + at, ok);
            attn::cp_async_16(Vs + (buf * KEYS + i) * d + c, A.v_pages + at, ok);
        }
        attn::cp_async_commit();
    };
    const int t_end = p_last / KEYS;
    int t = next(-1);
    fetch(t, 0, place(t));
    size_t base = place(next(t));
    for (int e = tid; e < QUERIES * d4; e += WARPS * 32) {
        const int i = e / d4, c = 4 * (e - i * d4), r = i / A.heads, h = i - r * A.heads;
        const bool ok = r < n_rows && h < n_heads;
        *reinterpret_cast<float4*>(Qs + i * d + c) =
            ok ? *reinterpret_cast<const float4*>(A.q + ((size_t)(row0 + r) * A.nq + h0 + h) * d + c)
               : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    }
    // the warp's two queries: warp and warp + 8
    int pos[2], lo[2], kept[2], head[2];
    bool live[2];
    float m[2], l[2], acc[2][NI], slope[2];
#pragma unroll
    for (int u = 0; u < 2; ++u) {
        const int i = warp + WARPS * u, r = i / A.heads, h = i - r * A.heads;
        live[u] = r < n_rows && h < n_heads;
        pos[u] = live[u] ? p_first + r : -1;
        lo[u] = low(pos[u]);
        kept[u] = min(A.keep_first, lo[u]);
        head[u] = h0 + h;
        slope[u] = A.slopes && live[u] ? A.slopes[head[u]] : 0.0f;
        m[u] = -INFINITY;
        l[u] = 0.0f;
#pragma unroll
        for (int i2 = 0; i2 < NI; ++i2) acc[u][i2] = 0.0f;
    }
    float2* mine = Ws + warp * 2 * KEYS;
    for (int buf = 0; t <= t_end; buf ^= 1) {
        const int t_next = next(t);
        if (t_next <= t_end) {
            fetch(t_next, buf ^ 1, base);
            base = place(next(t_next));
            attn::cp_async_wait<1>();
        } else {
            attn::cp_async_wait<0>();
        }
        __syncthreads();
        const int j = KEYS * t + lane;
        uint32_t see[2];
#pragma unroll
        for (int u = 0; u < 2; ++u)
            see[u] = __ballot_sync(0xffffffffu, j <= pos[u] && (j < kept[u] || j >= lo[u]));
        if (see[0] | see[1]) {
            const float* k = Ks + (buf * KEYS + lane) * KLD;
            float s[2] = {0.0f, 0.0f};
            if (see[0] && see[1]) {
                dots<NI, 2>(k, Qs + warp * d, WARPS, s);
            } else {
                float one[1];
                const int u = see[0] ? 0 : 1;
                dots<NI, 1>(k, Qs + (warp + WARPS * u) * d, 0, one);
                s[0] = s[1] = one[0];
            }
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                if (!see[u]) continue;
                const bool ok = see[u] >> lane & 1;
                float x = s[u] * A.scale;
                if (A.slopes) x = fmaf(-slope[u], (float)(pos[u] - j), x);
                if (A.softcap > 0.0f) x = A.softcap * tanhf(x / A.softcap);
                float M = ok ? x : -INFINITY;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const float other = __shfl_up_sync(0xffffffffu, M, o);
                    if (lane >= o) M = fmaxf(other, M);
                }
                M = fmaxf(m[u], M);
                const float up = __shfl_up_sync(0xffffffffu, M, 1), before = lane ? up : m[u];
                mine[u * KEYS + lane] = make_float2(exact_expf(before - M), exact_expf(x - M));
                m[u] = __shfl_sync(0xffffffffu, M, 31);
            }
            __syncwarp();
            const float* v = Vs + buf * KEYS * d;
            if ((see[0] & see[1]) == 0xffffffffu) {
#pragma unroll 4
                for (int i = 0; i < KEYS; ++i) {
                    float e[NI];
                    load_own<NI>(v + i * d, lane, e);
#pragma unroll
                    for (int u = 0; u < 2; ++u) {
                        const float2 w = mine[u * KEYS + i];
                        l[u] = fmaf(l[u], w.x, w.y);
#pragma unroll
                        for (int c = 0; c < NI; ++c) acc[u][c] = fmaf(acc[u][c], w.x, __fmul_rn(w.y, e[c]));
                    }
                }
            } else {
                for (uint32_t left = see[0] | see[1]; left; left &= left - 1) {
                    const int i = __ffs(left) - 1;
                    float e[NI];
                    load_own<NI>(v + i * d, lane, e);
#pragma unroll
                    for (int u = 0; u < 2; ++u) {
                        if (!(see[u] >> i & 1)) continue;
                        const float2 w = mine[u * KEYS + i];
                        l[u] = fmaf(l[u], w.x, w.y);
#pragma unroll
                        for (int c = 0; c < NI; ++c) acc[u][c] = fmaf(acc[u][c], w.x, __fmul_rn(w.y, e[c]));
                    }
                }
            }
        }
        __syncthreads();  // the tile's buffer is the target of the copies after next
        t = t_next;
    }
#pragma unroll
    for (int u = 0; u < 2; ++u) {
        if (!live[u]) continue;
        if (A.sink) {
            const float sv = A.sink[head[u]], M = fmaxf(m[u], sv), corr = exact_expf(m[u] - M);
            l[u] = fmaf(l[u], corr, exact_expf(sv - M));
#pragma unroll
            for (int c = 0; c < NI; ++c) acc[u][c] *= corr;
        }
        float* o = A.out + ((size_t)(row0 + pos[u] - p_first) * A.nq + head[u]) * d;
#pragma unroll
        for (int c = 0; c < NI; ++c) o[own_element<NI>(lane, c)] = acc[u][c] / l[u];
    }
}

}  // namespace

// As rfx_attention_plain with 32-bit rows, sequence by sequence (rows packed from seq_row0, positions from
// seq_start); at most max_new rows a sequence.  `longest_blocks`: the blocks' work in blocks as long as the longest, 0
// where the caller does not know it.  head_dim 32, 64, 128 or 256, everything on 16 bytes;
// RFX_ERR_UNSUPPORTED otherwise.
extern "C" int rfx_attention_f32(const float* q, const float* k_pages, const float* v_pages, const int* page_table,
                                 int max_pages, int page_size, const int* seq_slot, const int* seq_start,
                                 const int* seq_new, const int* seq_row0, float* out, int S, int max_new, int nq, int nkv,
                                 int head_dim, int window, int keep_first, float scale, const float* sink,
                                 const float* slopes, float softcap, float longest_blocks, void* stream) {
    if (S <= 0 || max_new <= 0) return 0;
    if (softcap < 0.0f || nkv <= 0 || nq % nkv != 0) return RFX_ERR_BAD_ARG;
    if (((reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(k_pages) | reinterpret_cast<uintptr_t>(v_pages) |
          reinterpret_cast<uintptr_t>(out)) & 15) || S > 65535)
        return RFX_ERR_UNSUPPORTED;
    const int group = nq / nkv;
    Args a{q, k_pages, v_pages, PagedKV{page_table, max_pages, page_size, nkv, head_dim}, seq_slot, seq_start, seq_new,
           seq_row0, out, nq, 0, 0, S, window, window > 0 ? keep_first : 0, scale, sink, slopes, softcap};
    // sixteen queries: all heads of the group that fit, then rows (a row alone: half the warps idle at worst)
    a.heads = group < QUERIES ? group : QUERIES;
    a.rows = QUERIES / a.heads;
    if (a.rows > max_new) a.rows = max_new;
    const int parts = (group + a.heads - 1) / a.heads;
    const long long blocks = ((long long)max_new + a.rows - 1) / a.rows * S * nkv * parts;
    if ((long long)nkv * parts > 65535 || blocks > 2147483647LL) return RFX_ERR_UNSUPPORTED;
    dim3 grid((unsigned)blocks);
    // Two blocks an SM, or one: then a block has the SM's shared memory to itself and ends in 1/1.15 of the time.  That
    // wins where the longest block decides, the longest ones being taken first: as long as all blocks are no more
    // work than one as long as the longest an SM.  us with one and with two, 8 query heads and 2 others of 128, new
    // prompts of 512 rows (0.86 of that work) 68 and 80, of 600 (1.01) 88 and 96, of 155, 311 and 235 (0.98) 55 and 66,
    // of 700 (1.18) 121 and 113; 512 rows after 800 others (1.39) 240 and 205; where blocks are of like length, as in
    // a decode step of 64 sequences with 8 key/value heads after 1,000 tokens, 488 and 291.
    const bool alone = longest_blocks > 0.0f && longest_blocks <= 1.02f * sm_count();
#define RFX_GO(NI)                                                                                                 \
    do {                                                                                                           \
        constexpr size_t need = (QUERIES * 32 * NI + 2 * KEYS * (64 * NI + 4) + WARPS * 2 * KEYS * 2) * sizeof(float); \
        constexpr size_t most = need < 120 * 1024 ? 120 * 1024 : need;                                                \
        const size_t smem = alone ? most : need;                                                                    \
        cudaError_t e = cudaFuncSetAttribute(attention_f32_kernel<NI>, cudaFuncAttributeMaxDynamicSharedMemorySize,  \
                                             (int)most);                                                            \
        if (e != cudaSuccess) return (int)e;                                                                        \
        RFX_LAUNCH(attention_f32_kernel<NI>, grid, WARPS * 32, smem, (cudaStream_t)stream, a);                        \
        return 0;                                                                                                   \
    } while (0)
    if (head_dim == 32) RFX_GO(1);
    if (head_dim == 64) RFX_GO(2);
    if (head_dim == 128) RFX_GO(4);
    if (head_dim == 256) RFX_GO(8);
#undef RFX_GO
    return RFX_ERR_UNSUPPORTED;
}
