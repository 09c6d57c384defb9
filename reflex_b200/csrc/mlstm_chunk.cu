// The mLSTM matrix memory (mlstm.cu) for steps that bring a sequence many rows: 64 rows at a time,
// all chunks side by side (chunk_scan.cuh).
//
// With F_t the sum of the log forget gates from the chunk's first row to t, g_s = i_s - F_s and
// M_t = max(m_prev, max_{s<=t} g_s), the walk gives m_t = F_t + M_t and
//   S_t^T q_t = e^(m_prev - M_t) S_prev^T q_t + sum_{s<=t} e^(g_s - M_t) (q_t . k_s) v_s
// and the same for n with v = 1.  A chunk's own sum is taken relative to its largest g (every
// exponent is <= 0); the carry meets it with the memory before.
#include "chunk_scan.cuh"

namespace {

struct Mlstm {
    static constexpr bool NORMALISER = true;
    static constexpr bool SHARED = false;  // every head has its own q and k
    static constexpr int RECORDS = 2;  // g and its running maximum, F, each in two parts
    const float *proj, *bias_i, *bias_f;
    float cap, q_scale;
    float *state, *num, *den;
    int q_off, k_off, v_off, i_off, f_off, heads, per, N, P;  // N: dim, P: vdim
    int ldq, ldk, ldv;

    __device__ __forceinline__ const float* q_row(int r, int h) const { return proj + (size_t)r * ldq + q_off + h * N; }
    __device__ __forceinline__ const float* k_row(int r, int h) const { return proj + (size_t)r * ldq + k_off + h * N; }
    __device__ __forceinline__ const float* v_row(int r, int h) const { return proj + (size_t)r * ldq + v_off + h * P; }
    // F and g of rows lane and lane + 32; rows from n on: F stays, g is -inf
    __device__ __forceinline__ void gates(int h, int first, int n, int lane, double (&F)[2], double (&gg)[2]) const {
        const float bi = bias_i[h], bf = bias_f[h];
        const float* row = proj + (size_t)first * ldq + h;
        float gi[2];
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const int r = lane + 32 * i;
            gi[i] = -INFINITY;
            F[i] = 0.0;
            if (r < n) {
                gi[i] = cap * tanhf((row[(size_t)r * ldq + i_off] + bi) / cap);
                const float z = cap * tanhf((row[(size_t)r * ldq + f_off] + bf) / cap);
                F[i] = (double)(fminf(z, 0.0f) - log1pf(expf(-fabsf(z))));
            }
        }
        chunk::scan_sum(F[0], F[1], lane);
        gg[0] = (double)gi[0] - F[0];
        gg[1] = (double)gi[1] - F[1];
    }
    __device__ __forceinline__ float4 state_weights(float* wl, float4* rows, int h, int first, int n, int lane) const {
        double F[2], gg[2];
        gates(h, first, n, lane, F, gg);
        double M[2] = {gg[0], gg[1]};
        chunk::scan_max(M[0], M[1], lane);
        const double G = __shfl_sync(0xffffffffu, M[1], 31), all = __shfl_sync(0xffffffffu, F[1], 31);
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const int r = lane + 32 * i;
            wl[r] = chunk::exp_of(gg[i] - G);
            if (rows) {
                float4 a, b = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                chunk::two_parts(gg[i], &a.x, &a.y);
                chunk::two_parts(M[i], &a.z, &a.w);
                chunk::two_parts(F[i], &b.x, &b.y);
                rows[2 * r] = a;
                rows[2 * r + 1] = b;
            }
        }
        float4 a;
        chunk::two_parts(all, &a.x, &a.y);
        chunk::two_parts(G, &a.z, &a.w);
        return a;
    }
    static __device__ __forceinline__ float g_hi(const float4& r) { return r.x; }
    static __device__ __forceinline__ float g_lo(const float4& r) { return r.y; }
    static __device__ __forceinline__ float weight(const float4&) { return 1.0f; }
    // M_t = max(m_prev, the rows' maximum so far)
    __device__ __forceinline__ chunk::RowTerms row_terms(const float4* r, float m_prev) const {
        const bool prev = m_prev > r->z || (m_prev == r->z && r->w < 0.0f);
        const float hi = prev ? m_prev : r->z, lo = prev ? 0.0f : r->w;
        return {-hi, -lo, expf((m_prev - hi) - lo), expf(-((r[1].x + hi) + (r[1].y + lo)))};
    }
    __device__ __forceinline__ float* head_state(int slot, int h) const {
        return state + ((size_t)slot * heads + h) * ((size_t)N * P + N + (P + 63) / 64);
    }
    // elements e .. e + 3 of [P][N | n]; the state keeps S as [N][P], then n, then m once per 64 columns
    __device__ __forceinline__ size_t at(int e, int i) const {
        const int p = e / N, n = e - p * N + i;
        return p < P ? (size_t)n * P + p : (size_t)N * P + n;
    }
    __device__ __forceinline__ float4 load_state(int slot, int h, int e) const {
        const float* s = head_state(slot, h);
        return make_float4(s[at(e, 0)], s[at(e, 1)], s[at(e, 2)], s[at(e, 3)]);
    }
    __device__ __forceinline__ float load_number(int slot, int h) const { return head_state(slot, h)[(size_t)N * P + N]; }
    __device__ __forceinline__ float2 carry(const float4& a, float& m) const {
        const double F = (double)a.x + a.y, G = (double)a.z + a.w, old = m;
        m = (float)(F + fmax(old, G));
        // relative to the number as it is kept, so that its rounding is no error of the memory
        return make_float2(chunk::exp_of(F + old - m), chunk::exp_of(F + G - m));
    }
    __device__ __forceinline__ void store_state(int slot, int h, int e, const float4& S) const {
        float* s = head_state(slot, h);
        s[at(e, 0)] = S.x;
        s[at(e, 1)] = S.y;
        s[at(e, 2)] = S.z;
        s[at(e, 3)] = S.w;
    }
    __device__ __forceinline__ void store_number(int slot, int h, float m) const {
        float* s = head_state(slot, h) + (size_t)N * P + N;
        for (int i = 0; i < (P + 63) / 64; ++i) s[i] = m;
    }
    __device__ __forceinline__ float4 gate(int, int, int) const { return make_float4(0.0f, 0.0f, 0.0f, 0.0f); }
    __device__ __forceinline__ void store_row(int r, int h, int p, const float4&, const float4& y, const float4&) const {
        rfx::store4(num + ((size_t)r * heads + h) * P + p,
                    make_float4(y.x * q_scale, y.y * q_scale, y.z * q_scale, y.w * q_scale));
    }
    __device__ __forceinline__ void store_sum(int r, int h, float nq, float floor) const {
        den[(size_t)r * heads + h] = fmaxf(fabsf(nq * q_scale), floor) + 1e-6f;
    }
};

}  // namespace

// Floats of scratch rfx_mlstm_chunks needs for a step of R rows in S sequences of at most max_rows.
extern "C" long long rfx_mlstm_chunks_floats(int R, int S, int max_rows, int heads, int dim, int vdim) {
    const long long one = chunk::chunk_floats(heads, (long long)vdim * dim + dim, Mlstm::RECORDS);
    return chunk::plan_rounds(R, S, max_rows, chunk::L, one).places * one;
}

// As rfx_mlstm_scan.  dim in fours up to 128, vdim in fours; rows, results and `scratch` on 16 bytes.
// RFX_ERR_UNSUPPORTED otherwise.
extern "C" int rfx_mlstm_chunks(const float* proj, int ld, int q_off, int k_off, int v_off, int i_off, int f_off,
                                const float* bias_i, const float* bias_f, float cap, float q_scale,
                                const int* seq_slot, const int* seq_row0, int S, int R, int max_rows, float* state,
                                float* num, float* den, float* scratch, int heads, int dim, int vdim, int* err, void* stream) {
    if (S <= 0 || R <= 0 || max_rows <= 0) return 0;
    if (heads <= 0 || dim <= 0 || vdim <= 0 || cap <= 0.0f) return RFX_ERR_BAD_ARG;
    if (dim % 4 || vdim % 4 || dim > 128 || ((ld | q_off | k_off | v_off) & 3) ||
        ((reinterpret_cast<uintptr_t>(proj) | reinterpret_cast<uintptr_t>(num) | reinterpret_cast<uintptr_t>(scratch)) & 15))
        return RFX_ERR_UNSUPPORTED;
    Mlstm p{proj, bias_i, bias_f, cap, q_scale, state, num, den, q_off, k_off, v_off, i_off, f_off, heads, 1, dim,
            vdim, ld, ld, ld};
    return chunk::run(p, seq_slot, seq_row0, S, R, max_rows, scratch, err, (cudaStream_t)stream);
}
