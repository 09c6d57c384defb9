// The state-space recurrence with one decay a head (ssd.cu) for steps that bring a sequence many
// rows: 64 rows at a time, all chunks side by side (chunk_scan.cuh).
//
//     dt = softplus(dt_pre[h] + dt_bias[h]),  S <- exp(A[h] dt) S + dt B x^T,  y = S^T C + D[h] x
//     out = y * silu(z)
// with q = C, k = B, v = x, the weight dt and the running logarithm A[h] (dt_1 + .. + dt_t).  The
// heads of a group share C and B, and so the products between a chunk's rows.
#include "chunk_scan.cuh"

namespace {

struct Ssd {
    static constexpr bool NORMALISER = false;
    static constexpr bool SHARED = true;  // several heads have the same q and k
    static constexpr int RECORDS = 1;  // running logarithm in two parts, step size, its exponential
    const float *xbc, *proj, *dt_bias, *A, *D;
    float *state, *out;
    long long state_stride, state_off;
    int ldx, ldp, z_off, dt_off, heads, per, N, P, inner, groups;
    int ldq, ldk, ldv;

    __device__ __forceinline__ const float* q_row(int r, int h) const {
        return xbc + (size_t)r * ldx + inner + groups * N + (h / per) * N;
    }
    __device__ __forceinline__ const float* k_row(int r, int h) const {
        return xbc + (size_t)r * ldx + inner + (h / per) * N;
    }
    __device__ __forceinline__ const float* v_row(int r, int h) const { return xbc + (size_t)r * ldx + h * P; }
    // step sizes and running logarithms of rows lane and lane + 32; rows from n on: zero step sizes
    __device__ __forceinline__ void logs(int h, int first, int n, int lane, float& da, float& db, double& ca,
                                         double& cb) const {
        const float bias = dt_bias ? dt_bias[h] : 0.0f;
        const float* pre = proj + (size_t)first * ldp + dt_off + h;
        auto step = [&](int r) {
            if (r >= n) return 0.0f;
            const float v = pre[(size_t)r * ldp] + bias;
            return fmaxf(v, 0.0f) + log1pf(expf(-fabsf(v)));
        };
        da = step(lane);
        db = step(lane + 32);
        ca = (double)A[h] * da;
        cb = (double)A[h] * db;
        chunk::scan_sum(ca, cb, lane);
    }
    __device__ __forceinline__ float4 state_weights(float* wl, float4* rows, int h, int first, int n, int lane) const {
        float d[2];
        double c[2];
        logs(h, first, n, lane, d[0], d[1], c[0], c[1]);
        const double all = __shfl_sync(0xffffffffu, c[1], 31);
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const int r = lane + 32 * i;
            wl[r] = d[i] * chunk::exp_of(all - c[i]);
            if (rows) {
                float hi, lo;
                chunk::two_parts(c[i], &hi, &lo);
                rows[r] = make_float4(hi, lo, d[i], chunk::exp_of(hi, lo));
            }
        }
        return make_float4(chunk::exp_of(all), 0.0f, 0.0f, 0.0f);
    }
    static __device__ __forceinline__ float g_hi(const float4& r) { return -r.x; }
    static __device__ __forceinline__ float g_lo(const float4& r) { return -r.y; }
    static __device__ __forceinline__ float weight(const float4& r) { return r.z; }
    __device__ __forceinline__ chunk::RowTerms row_terms(const float4* r, float) const { return {r->x, r->y, r->w, 0.0f}; }
    __device__ __forceinline__ float* memory(int slot, int h, int e) const {
        return state + (size_t)slot * state_stride + state_off + (size_t)h * P * N + e;
    }
    __device__ __forceinline__ float4 load_state(int slot, int h, int e) const {
        return *reinterpret_cast<const float4*>(memory(slot, h, e));
    }
    __device__ __forceinline__ float load_number(int, int) const { return 0.0f; }
    __device__ __forceinline__ float2 carry(const float4& a, float&) const { return make_float2(a.x, 1.0f); }
    __device__ __forceinline__ void store_state(int slot, int h, int e, const float4& S) const {
        *reinterpret_cast<float4*>(memory(slot, h, e)) = S;
    }
    static __device__ __forceinline__ float silu(float z) { return z / (1.0f + expf(-z)); }
    __device__ __forceinline__ float4 gate(int r, int h, int p) const {
        return rfx::load4(proj + (size_t)r * ldp + z_off + h * P + p);
    }
    __device__ __forceinline__ void store_row(int r, int h, int p, const float4& z, const float4& y, const float4& x) const {
        const float d = D ? D[h] : 0.0f;
        rfx::store4(out + (size_t)r * inner + h * P + p,
                    make_float4(fmaf(d, x.x, y.x) * silu(z.x), fmaf(d, x.y, y.y) * silu(z.y), fmaf(d, x.z, y.z) * silu(z.z),
                                fmaf(d, x.w, y.w) * silu(z.w)));
    }
};

}  // namespace

// Floats of scratch rfx_ssd_chunk needs for a step of R rows in n_seq sequences of at most max_rows.
extern "C" long long rfx_ssd_chunk_floats(int R, int n_seq, int max_rows, int heads, int P, int N) {
    const long long one = chunk::chunk_floats(heads, (long long)P * N, Ssd::RECORDS);
    return chunk::plan_rounds(R, n_seq, max_rows, chunk::L, one).places * one;
}

// As rfx_ssd_scan with 32-bit results, the state [heads][P][N].  P and N in fours, N up to 128; rows and
// state on 16 bytes; `scratch` on 16 bytes too.  RFX_ERR_UNSUPPORTED otherwise.
extern "C" int rfx_ssd_chunk(const float* xbc, int ldx, const float* proj, int ldp, int z_off, int dt_off,
                             const float* dt_bias, const float* A, const float* D, float* state,
                             long long state_stride, long long state_off, const int* seq_slot, const int* seq_row0,
                             int n_seq, int R, int max_rows, float* out, float* scratch, int heads, int P, int N,
                             int groups, int* err, void* stream) {
    if (n_seq <= 0 || R <= 0 || max_rows <= 0) return 0;
    if (heads <= 0 || groups <= 0 || heads % groups || P <= 0 || N <= 0) return RFX_ERR_BAD_ARG;
    if (P % 4 || N % 4 || N > 128 || ((ldx | ldp | z_off) & 3) || ((state_stride | state_off) & 3) ||
        ((reinterpret_cast<uintptr_t>(xbc) | reinterpret_cast<uintptr_t>(proj) | reinterpret_cast<uintptr_t>(state) |
          reinterpret_cast<uintptr_t>(out) | reinterpret_cast<uintptr_t>(scratch)) & 15))
        return RFX_ERR_UNSUPPORTED;
    Ssd p{xbc, proj, dt_bias, A, D, state, out, state_stride, state_off, ldx, ldp, z_off, dt_off, heads,
          heads / groups, N, P, heads * P, groups, ldx, ldx, ldx};
    return chunk::run(p, seq_slot, seq_row0, n_seq, R, max_rows, scratch, err, (cudaStream_t)stream);
}
