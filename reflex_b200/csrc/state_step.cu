// A decode step of the recurrences with a matrix memory a head, where every sequence has one row: the
// state-space recurrence (ssd.cu), the mLSTM (mlstm.cu), the generalized delta rule (delta_rule.cu) and the
// gated delta rule (gated_delta.cu), the same functions of the same states.
//
// A row reads and writes its head's whole memory, 16 to 128 KB, so memory bounds the step.  The walks there
// serve any number of rows: a warp has a column or four, and waits for the row, staged in shared memory
// behind one or two barriers.  Here (but for the mLSTM's k and q) nothing is staged: a thread's share of the memory, up
// to eight 16-byte loads (one to four where heads are few or small), is on its way at once with what it needs of the
// row.  A block has 64 columns of a head, 32 or 16 where few heads leave SMs without one.
//
// us walking and now: state-space of 64 heads of 64 x 128, 59 sequences (247 MB) 127 and 48; mLSTM of 16 heads of
// 128 x 256, 40 sequences (168 MB) 85 and 30; delta rule of 64 heads of 64, 40 sequences (84 MB) 59 and 19; gated
// delta rule of 48 heads of 128 x 128, 26 sequences (164 MB) 50 and 25.5.  One sequence of width 1,024: all four
// layers 1 to 2 us less.
#include "common.cuh"

namespace {

using namespace rfx;

constexpr int THREADS = 256, WARPS = THREADS / 32;

__device__ __forceinline__ float softplus_f(float v) { return fmaxf(v, 0.0f) + log1pf(expf(-fabsf(v))); }
__device__ __forceinline__ float sigmoid_f(float t) { return 1.0f / (1.0f + expf(-t)); }
__device__ __forceinline__ float dot4(const float4& a, const float4& b) {
    return fmaf(a.x, b.x, a.y * b.y) + fmaf(a.z, b.z, a.w * b.w);
}
template <int LANES>
__device__ __forceinline__ float lanes_sum(float v) {
#pragma unroll
    for (int o = LANES / 2; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// ---- state-space: S [channel][state], LANES lanes a channel, four states each, COLS channels a lane ----
template <int LANES, int COLS>
__global__ void __launch_bounds__(THREADS, 3)
ssd_step_kernel(const float* __restrict__ xbc, int ldx, const float* __restrict__ proj, int ldp, int z_off, int dt_off,
                const float* __restrict__ dt_bias, const float* __restrict__ A, const float* __restrict__ D,
                float* __restrict__ state, long long state_stride, long long state_off,
                const int* __restrict__ seq_slot, float* __restrict__ out, int heads, int P, int N, int groups) {
    constexpr int SIDE = 32 / LANES;  // channels side by side in a warp
    pdl_prologue();
    const int seq = blockIdx.x, h = blockIdx.y, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int n = 4 * (lane % LANES), grp = h / (heads / groups), inner = heads * P;
    const int p0 = (blockIdx.z * WARPS + warp) * SIDE * COLS + lane / LANES;  // the lane's channels, SIDE apart
    const bool live = n < N;
    const float *row = xbc + (size_t)seq * ldx, *pr = proj + (size_t)seq * ldp;
    float* S = state + (size_t)seq_slot[seq] * state_stride + state_off + ((size_t)h * P + p0) * N + n;
    const float4 none = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    float4 s[COLS];
    float x[COLS];
#pragma unroll
    for (int i = 0; i < COLS; ++i) {
        const int p = p0 + SIDE * i;
        s[i] = live && p < P ? load4(S + (size_t)SIDE * i * N) : none;
        x[i] = p < P ? row[h * P + p] : 0.0f;
    }
    const float4 b = live ? load4(row + inner + grp * N + n) : none;
    const float4 c = live ? load4(row + inner + (groups + grp) * N + n) : none;
    const float dt = softplus_f(pr[dt_off + h] + (dt_bias ? dt_bias[h] : 0.0f)), decay = expf(A[h] * dt);
    const float d = D ? D[h] : 0.0f;
    float y[COLS];
#pragma unroll
    for (int i = 0; i < COLS; ++i) {
        const float dx = dt * x[i];
        s[i].x = fmaf(s[i].x, decay, b.x * dx);
        s[i].y = fmaf(s[i].y, decay, b.y * dx);
        s[i].z = fmaf(s[i].z, decay, b.z * dx);
        s[i].w = fmaf(s[i].w, decay, b.w * dx);
        if (live && p0 + SIDE * i < P) store4(S + (size_t)SIDE * i * N, s[i]);
        y[i] = live ? dot4(s[i], c) : 0.0f;  // (an infinite x leaves NaN in lanes beyond N)
    }
#pragma unroll
    for (int i = 0; i < COLS; ++i) y[i] = fmaf(d, x[i], lanes_sum<LANES>(y[i]));
#pragma unroll
    for (int i = 0; i < COLS; ++i)  // a lane of the channel's a result
        if (lane % LANES == i) {
            const int p = p0 + SIDE * i;
            if (p < P) {
                const float z = pr[z_off + h * P + p];
                out[(size_t)seq * inner + h * P + p] = y[i] * (z / (1.0f + expf(-z)));
            }
        }
}

// ---- delta rules: S [value column][key channel], LANES lanes a column, four channels each ----
// The generalized one: rows [r | k | v | a] and the decays' pre-activations, a channel each.
template <int LANES, int COLS>
__global__ void __launch_bounds__(THREADS, 4)
delta_step_kernel(const float* __restrict__ proj, int ld, int r_off, int k_off, int v_off, int a_off,
                  const float* __restrict__ wpre, const float* __restrict__ w_bias, const float* __restrict__ a_bias,
                  float rate, float unit_eps, float* __restrict__ state, long long state_stride, long long state_off,
                  const int* __restrict__ seq_slot, float* __restrict__ out, int heads, int d) {
    constexpr int SIDE = 32 / LANES;
    pdl_prologue();
    const int seq = blockIdx.x, h = blockIdx.y, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int c = 4 * (lane % LANES), hd = heads * d;
    const int j0 = (blockIdx.z * WARPS + warp) * SIDE * COLS + lane / LANES;
    const bool live = c < d;
    const float* pr = proj + (size_t)seq * ld + h * d;
    float* S = state + (size_t)seq_slot[seq] * state_stride + state_off + ((size_t)h * d + j0) * d + c;
    const float4 none = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    float4 s[COLS];
    float v[COLS];
#pragma unroll
    for (int i = 0; i < COLS; ++i) {
        const int j = j0 + SIDE * i;
        s[i] = live && j < d ? load4(S + (size_t)SIDE * i * d) : none;
        v[i] = j < d ? pr[v_off + j] : 0.0f;
    }
    float4 k = none, r = none, a = none, w = none;
    if (live) {
        k = load4(pr + k_off + c);
        r = load4(pr + r_off + c);
        const float4 ap = load4(pr + a_off + c), ab = load4(a_bias + h * d + c);
        const float4 wp = load4(wpre + (size_t)seq * hd + h * d + c), wb = load4(w_bias + h * d + c);
        a = make_float4(sigmoid_f(ap.x + ab.x), sigmoid_f(ap.y + ab.y), sigmoid_f(ap.z + ab.z), sigmoid_f(ap.w + ab.w));
        w = make_float4(expf(-rate * sigmoid_f(wp.x + wb.x)), expf(-rate * sigmoid_f(wp.y + wb.y)),
                        expf(-rate * sigmoid_f(wp.z + wb.z)), expf(-rate * sigmoid_f(wp.w + wb.w)));
    }
    const float inv = 1.0f / sqrtf(lanes_sum<LANES>(dot4(k, k)) + unit_eps);
    const float4 u = make_float4(k.x * inv, k.y * inv, k.z * inv, k.w * inv);
    const float4 au = make_float4(a.x * u.x, a.y * u.y, a.z * u.z, a.w * u.w);
    float seen[COLS], o[COLS];
#pragma unroll
    for (int i = 0; i < COLS; ++i) seen[i] = dot4(u, s[i]);
#pragma unroll
    for (int i = 0; i < COLS; ++i) seen[i] = lanes_sum<LANES>(seen[i]);
#pragma unroll
    for (int i = 0; i < COLS; ++i) {
        s[i].x = fmaf(k.x, v[i], fmaf(w.x, s[i].x, -au.x * seen[i]));
        s[i].y = fmaf(k.y, v[i], fmaf(w.y, s[i].y, -au.y * seen[i]));
        s[i].z = fmaf(k.z, v[i], fmaf(w.z, s[i].z, -au.z * seen[i]));
        s[i].w = fmaf(k.w, v[i], fmaf(w.w, s[i].w, -au.w * seen[i]));
        if (live && j0 + SIDE * i < d) store4(S + (size_t)SIDE * i * d, s[i]);
        o[i] = live ? dot4(s[i], r) : 0.0f;
    }
#pragma unroll
    for (int i = 0; i < COLS; ++i) o[i] = lanes_sum<LANES>(o[i]);
#pragma unroll
    for (int i = 0; i < COLS; ++i)
        if (lane % LANES == i && j0 + SIDE * i < d) out[(size_t)seq * hd + h * d + j0 + SIDE * i] = o[i];
}

// The gated one: rows [q | k | v] as gated_delta_prep leaves them, a decay and a write rate a head.
template <int LANES, int COLS>
__global__ void __launch_bounds__(THREADS)
gated_delta_step_kernel(const float* __restrict__ qkv, const float* __restrict__ gates, float* __restrict__ state,
                        long long state_stride, long long state_off, const int* __restrict__ seq_slot,
                        float* __restrict__ out, int H, int G, int d, int dv) {
    constexpr int SIDE = 32 / LANES;
    pdl_prologue();
    const int seq = blockIdx.x, h = blockIdx.y, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int c = 4 * (lane % LANES), kvh = h / (H / G);
    const int j0 = (blockIdx.z * WARPS + warp) * SIDE * COLS + lane / LANES;
    const bool live = c < d;
    const float* row = qkv + (size_t)seq * (2 * G * d + H * dv);
    float* S = state + (size_t)seq_slot[seq] * state_stride + state_off + ((size_t)h * dv + j0) * d + c;
    const float4 none = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    float4 s[COLS];
    float v[COLS];
#pragma unroll
    for (int i = 0; i < COLS; ++i) {
        const int j = j0 + SIDE * i;
        s[i] = live && j < dv ? load4(S + (size_t)SIDE * i * d) : none;
        v[i] = j < dv ? row[2 * G * d + h * dv + j] : 0.0f;
    }
    const float4 q = live ? load4(row + kvh * d + c) : none, k = live ? load4(row + G * d + kvh * d + c) : none;
    const float g = gates[(size_t)seq * 2 * H + h], beta = gates[(size_t)seq * 2 * H + H + h];
    float u[COLS], o[COLS];
#pragma unroll
    for (int i = 0; i < COLS; ++i) u[i] = dot4(k, s[i]);
#pragma unroll
    for (int i = 0; i < COLS; ++i) u[i] = beta * fmaf(-g, lanes_sum<LANES>(u[i]), v[i]);
#pragma unroll
    for (int i = 0; i < COLS; ++i) {
        s[i].x = fmaf(k.x, u[i], g * s[i].x);
        s[i].y = fmaf(k.y, u[i], g * s[i].y);
        s[i].z = fmaf(k.z, u[i], g * s[i].z);
        s[i].w = fmaf(k.w, u[i], g * s[i].w);
        if (live && j0 + SIDE * i < dv) store4(S + (size_t)SIDE * i * d, s[i]);
        o[i] = dot4(s[i], q);
    }
#pragma unroll
    for (int i = 0; i < COLS; ++i) o[i] = lanes_sum<LANES>(o[i]);
#pragma unroll
    for (int i = 0; i < COLS; ++i)
        if (lane % LANES == i && j0 + SIDE * i < dv) out[(size_t)seq * H * dv + (size_t)h * dv + j0 + SIDE * i] = o[i];
}

// ---- mLSTM: S [element of k][element of v], then n, then m once per 64 elements of v ----
// A block a (sequence, head, 64 elements of v): a thread four of them and every sixteenth element of k, whose
// partial sums of S^T q meet in shared memory; the first block also has n.
constexpr int VT = 64, KSETS = THREADS / (VT / 4), MAX_DIM = 128, ROWS = MAX_DIM / KSETS;
__global__ void __launch_bounds__(THREADS)
mlstm_step_kernel(const float* __restrict__ proj, int ld, int q_off, int k_off, int v_off, int i_off, int f_off,
                  const float* __restrict__ bias_i, const float* __restrict__ bias_f, float cap, float q_scale,
                  const int* __restrict__ seq_slot, float* __restrict__ state, float* __restrict__ num,
                  float* __restrict__ den, int heads, int dim, int vdim) {
    __shared__ float ks[MAX_DIM], qs[MAX_DIM];
    __shared__ __align__(16) float4 part[KSETS][VT / 4];
    __shared__ float dots[WARPS];
    pdl_prologue();
    const int seq = blockIdx.x, h = blockIdx.y, tid = threadIdx.x, lane = tid & 31;
    const int c = 4 * (tid % (VT / 4)), set = tid / (VT / 4), j = blockIdx.z * VT + c;
    float* head = state + ((size_t)seq_slot[seq] * heads + h) * ((size_t)dim * vdim + dim + gridDim.z);
    const float* row = proj + (size_t)seq * ld;
    const bool live = j < vdim;
    const float4 none = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    float4 s[ROWS];
#pragma unroll
    for (int i = 0; i < ROWS; ++i) {
        const int e = set + KSETS * i;
        s[i] = live && e < dim ? load4(head + (size_t)e * vdim + j) : none;
    }
    const float4 v = live ? load4(row + v_off + h * vdim + j) : none;
    const bool has_n = blockIdx.z == 0;
    const float nn = has_n && tid < dim ? head[(size_t)dim * vdim + tid] : 0.0f;
    float* mp = head + (size_t)dim * vdim + dim + blockIdx.z;
    const float m = *mp;
    if (tid < dim) {
        ks[tid] = row[k_off + h * dim + tid];
        qs[tid] = row[q_off + h * dim + tid];
    }
    const float gi = cap * tanhf((row[i_off + h] + bias_i[h]) / cap), z = cap * tanhf((row[f_off + h] + bias_f[h]) / cap);
    const float fm = (fminf(z, 0.0f) - log1pf(expf(-fabsf(z)))) + m, m_new = fmaxf(fm, gi);
    const float a = expf(fm - m_new), b = expf(gi - m_new);
    const float4 bv = make_float4(b * v.x, b * v.y, b * v.z, b * v.w);
    __syncthreads();  // (m has been read by every thread, too)
    float4 acc = none;
#pragma unroll
    for (int i = 0; i < ROWS; ++i) {
        const int e = set + KSETS * i;
        if (e < dim) {
            const float k = ks[e], q = qs[e];
            s[i].x = fmaf(a, s[i].x, bv.x * k);
            s[i].y = fmaf(a, s[i].y, bv.y * k);
            s[i].z = fmaf(a, s[i].z, bv.z * k);
            s[i].w = fmaf(a, s[i].w, bv.w * k);
            if (live) store4(head + (size_t)e * vdim + j, s[i]);
            acc.x = fmaf(s[i].x, q, acc.x);
            acc.y = fmaf(s[i].y, q, acc.y);
            acc.z = fmaf(s[i].z, q, acc.z);
            acc.w = fmaf(s[i].w, q, acc.w);
        }
    }
    part[set][tid % (VT / 4)] = acc;
    if (has_n) {  // n as a column whose v is 1
        float nq = 0.0f;
        if (tid < dim) {
            const float n2 = fmaf(a, nn, b * ks[tid]);
            head[(size_t)dim * vdim + tid] = n2;
            nq = n2 * qs[tid];
        }
        nq = warp_sum(nq);
        if (lane == 0) dots[tid >> 5] = nq;
    }
    if (tid == 0) *mp = m_new;
    __syncthreads();
    if (tid < VT && blockIdx.z * VT + tid < vdim) {
        const float* p = reinterpret_cast<const float*>(part) + tid;
        float t[4] = {};
#pragma unroll
        for (int i = 0; i < KSETS; ++i) t[i & 3] += p[i * VT];
        num[((size_t)seq * heads + h) * vdim + blockIdx.z * VT + tid] = ((t[0] + t[1]) + (t[2] + t[3])) * q_scale;
    }
    if (has_n && tid == 0) {
        float t = 0.0f;
#pragma unroll
        for (int i = 0; i < MAX_DIM / 32; ++i) t += dots[i];
        den[(size_t)seq * heads + h] = fmaxf(fabsf(t * q_scale), expf(-m_new)) + 1e-6f;
    }
}

inline bool on16(const void* a, const void* b = nullptr, const void* c = nullptr, const void* d = nullptr) {
    return ((reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(b) | reinterpret_cast<uintptr_t>(c) |
             reinterpret_cast<uintptr_t>(d)) & 15) == 0;
}

// blocks that `cols` columns or channels take
inline int blocks_of(int cols, int lanes, int a_lane) {
    const int block = WARPS * (32 / lanes) * a_lane;
    return (cols + block - 1) / block;
}
// so few heads that a block each leaves SMs idle: then more blocks a head, fewer loads a thread
inline bool few_heads(int n_seq, int heads) { return (long long)n_seq * heads < 2LL * sm_count(); }

}  // namespace

// As rfx_ssd_scan with 32-bit results in a step whose row i is sequence i's only one.  P and N in fours, N up to 128,
// everything on 16 bytes; RFX_ERR_UNSUPPORTED otherwise.
extern "C" int rfx_ssd_step(const float* xbc, int ldx, const float* proj, int ldp, int z_off, int dt_off,
                            const float* dt_bias, const float* A, const float* D, float* state, long long state_stride,
                            long long state_off, const int* seq_slot, int n_seq, float* out, int heads, int P, int N,
                            int groups, void* stream) {
    if (n_seq <= 0) return 0;
    if (heads <= 0 || groups <= 0 || heads % groups || P <= 0 || N <= 0) return RFX_ERR_BAD_ARG;
    if (P % 4 || N % 4 || N > 128 || ((ldx | ldp | z_off) & 3) || ((state_stride | state_off) & 3) || heads > 65535 ||
        !on16(xbc, proj, state))
        return RFX_ERR_UNSUPPORTED;
#define RFX_GO(LANES, COLS)                                                                                        \
    RFX_LAUNCH((ssd_step_kernel<LANES, COLS>), dim3(n_seq, heads, blocks_of(P, LANES, COLS)), THREADS, 0,            \
               (cudaStream_t)stream, xbc, ldx, proj, ldp, z_off, dt_off, dt_bias, A, D, state, state_stride,       \
               state_off, seq_slot, out, heads, P, N, groups)
    const bool few = few_heads(n_seq, heads);
    if (N <= 32) RFX_GO(8, 2);
    else if (N <= 64 && few) RFX_GO(16, 2);
    else if (N <= 64) RFX_GO(16, 4);
    else if (few) RFX_GO(32, 2);
    else RFX_GO(32, 8);
#undef RFX_GO
    return 0;
}

// As rfx_delta_rule with 32-bit results, likewise.  d in fours up to 64 (beyond that some sizes' walk keeps the memory
// the other way round).
extern "C" int rfx_delta_step(const float* proj, int ld, int r_off, int k_off, int v_off, int a_off, const float* wpre,
                              const float* w_bias, const float* a_bias, float rate, float unit_eps, float* state,
                              long long state_stride, long long state_off, const int* seq_slot, int n_seq, float* out,
                              int heads, int d, void* stream) {
    if (n_seq <= 0) return 0;
    if (heads <= 0 || d <= 0) return RFX_ERR_BAD_ARG;
    if (d % 4 || d > 64 || ((ld | r_off | k_off | v_off | a_off) & 3) || ((state_stride | state_off) & 3) || heads > 65535 ||
        !on16(proj, wpre, w_bias, a_bias) || !on16(state))
        return RFX_ERR_UNSUPPORTED;
#define RFX_GO(LANES, COLS)                                                                                        \
    RFX_LAUNCH((delta_step_kernel<LANES, COLS>), dim3(n_seq, heads, blocks_of(d, LANES, COLS)), THREADS, 0,          \
               (cudaStream_t)stream, proj, ld, r_off, k_off, v_off, a_off, wpre, w_bias, a_bias, rate, unit_eps,   \
               state, state_stride, state_off, seq_slot, out, heads, d)
    if (d <= 32) RFX_GO(8, 1);
    else if (few_heads(n_seq, heads)) RFX_GO(16, 1);
    else RFX_GO(16, 4);
#undef RFX_GO
    return 0;
}

// As rfx_gated_delta_scan, likewise.  d and dv in fours, d up to 128.
extern "C" int rfx_gated_delta_step(const float* qkv, const float* gates, float* state, long long state_stride,
                                    long long state_off, const int* seq_slot, int n_seq, float* out, int H, int G,
                                    int d, int dv, void* stream) {
    if (n_seq <= 0) return 0;
    if (H <= 0 || G <= 0 || H % G || d <= 0 || dv <= 0) return RFX_ERR_BAD_ARG;
    if (d % 4 || dv % 4 || d > 128 || ((state_stride | state_off) & 3) || H > 65535 || !on16(qkv, state)) return RFX_ERR_UNSUPPORTED;
#define RFX_GO(LANES, COLS)                                                                                        \
    RFX_LAUNCH((gated_delta_step_kernel<LANES, COLS>), dim3(n_seq, H, blocks_of(dv, LANES, COLS)), THREADS, 0,       \
               (cudaStream_t)stream, qkv, gates, state, state_stride, state_off, seq_slot, out, H, G, d, dv)
    const bool few = few_heads(n_seq, H);
    if (d <= 32) RFX_GO(8, 2);
    else if (d <= 64 && few) RFX_GO(16, 2);
    else if (d <= 64) RFX_GO(16, 4);
    else if (few) RFX_GO(32, 2);
    else RFX_GO(32, 8);
#undef RFX_GO
    return 0;
}

// As rfx_mlstm_scan, likewise.  dim and vdim in fours, dim up to 128, a head's state a multiple of 16 bytes.
extern "C" int rfx_mlstm_step(const float* proj, int ld, int q_off, int k_off, int v_off, int i_off, int f_off,
                              const float* bias_i, const float* bias_f, float cap, float q_scale, const int* seq_slot,
                              int S, float* state, float* num, float* den, int heads, int dim, int vdim, void* stream) {
    if (S <= 0) return 0;
    if (heads <= 0 || dim <= 0 || vdim <= 0 || cap <= 0.0f) return RFX_ERR_BAD_ARG;
    const int tiles = (vdim + VT - 1) / VT;
    if (dim % 4 || vdim % 4 || dim > MAX_DIM || ((dim * vdim + dim + tiles) & 3) || ((ld | v_off) & 3) || heads > 65535 ||
        tiles > 65535 || !on16(proj, state))
        return RFX_ERR_UNSUPPORTED;
    RFX_LAUNCH(mlstm_step_kernel, dim3(S, heads, tiles), THREADS, 0, (cudaStream_t)stream, proj, ld, q_off, k_off, v_off,
               i_off, f_off, bias_i, bias_f, cap, q_scale, seq_slot, state, num, den, heads, dim, vdim);
    return 0;
}
