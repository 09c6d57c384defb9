// Device functions of the short causal convolutions (short_conv.cu has the layout and the
// rules), shared by the kernels that do something with the convolved rows in the same launch.
#pragma once

#include <cuda_runtime.h>

namespace rfx {
namespace conv {

constexpr int MAX_TAPS = 16;

// rows of this step that precede row r in its sequence, up to `cap`; the slots of
// the rows before are loaded side by side, not one after the other's answer
__device__ __forceinline__ int rows_before(const int* __restrict__ row_slot, int r, int cap) {
    const int slot = row_slot[r];
    int t = cap;  // the nearest row back that is not this sequence's ends the count (no early exit: no chain)
#pragma unroll
    for (int j = cap - 1; j >= 0; --j) {
        const bool same = r - j - 1 >= 0 && row_slot[r - j - 1] == slot;
        if (!same) t = j;
    }
    return t;
}

// the convolution of channel c (column col0 + c of proj) at row r
__device__ __forceinline__ float conv_at(const float* __restrict__ proj, int ld, int col0, int c,
                                         const float* __restrict__ bias, const float* __restrict__ w,
                                         int taps, const float* __restrict__ state_slot, int C, int r,
                                         int before) {
    const int T = taps - 1;
    const float b = bias ? bias[c] : 0.0f;
    float y = 0.0f;
    for (int j = 0; j < taps; ++j) {
        const int back = T - j;  // tap j meets the input `back` tokens ago
        float u;
        if (back <= before) u = proj[(size_t)(r - back) * ld + col0 + c] + b;
        else u = state_slot[(size_t)(T + before - back) * C + c];
        y = fmaf(w[(size_t)j * C + c], u, y);
    }
    return y;
}

// the same for channels c .. c + 3 (every offset a multiple of four floats)
__device__ __forceinline__ float4 conv4_at(const float* __restrict__ proj, int ld, int col0, int c,
                                           const float* __restrict__ bias, const float* __restrict__ w,
                                           int taps, const float* __restrict__ state_slot, int C, int r,
                                           int before) {
    const int T = taps - 1;
    const float4 b = bias ? *reinterpret_cast<const float4*>(bias + c) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    float4 y = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll
    for (int j = 0; j < taps; ++j) {
        const int back = T - j;
        const bool here = back <= before;  // one load from either place: no branch between the taps' loads
        float4 u = *reinterpret_cast<const float4*>(here ? proj + (size_t)(r - back) * ld + col0 + c
                                                         : state_slot + (size_t)(T + before - back) * C + c);
        if (here) { u.x += b.x; u.y += b.y; u.z += b.z; u.w += b.w; }
        const float4 f = *reinterpret_cast<const float4*>(w + (size_t)j * C + c);
        y.x = fmaf(f.x, u.x, y.x);
        y.y = fmaf(f.y, u.y, y.y);
        y.z = fmaf(f.z, u.z, y.z);
        y.w = fmaf(f.w, u.w, y.w);
    }
    return y;
}

// Four channels through several neighbouring rows: the last TAPS - 1 inputs in registers, oldest first, so
// that a prompt's input is loaded once and not by every row that it reaches.  `at(r)`, `tail(slot)`: where
// row r's and a slot's four channels lie (the state's rows `C` apart).
template <int TAPS>
struct Window {
    float4 u[TAPS - 1];
    template <class At, class Tail>
    __device__ __forceinline__ void begin(const int* __restrict__ row_slot, int r, int C, const float4& b, At&& at, Tail&& tail) {
        const int before = rows_before(row_slot, r, TAPS - 1);
        const float* t = tail(row_slot[r]);
#pragma unroll
        for (int j = 0; j < TAPS - 1; ++j) {
            const int back = TAPS - 1 - j;
            const bool here = back <= before;
            u[j] = *reinterpret_cast<const float4*>(here ? at(r - back) : t + (size_t)(j + before) * C);
            if (here) { u[j].x += b.x; u[j].y += b.y; u[j].z += b.z; u[j].w += b.w; }
        }
    }
    // the row's results (taps summed oldest first, as conv4_at), and its input into the window
    __device__ __forceinline__ float4 step(const float4 (&f)[TAPS], const float4& now) {
        float4 y = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll
        for (int j = 0; j < TAPS; ++j) {
            const float4 x = j < TAPS - 1 ? u[j < TAPS - 1 ? j : 0] : now;
            y.x = fmaf(f[j].x, x.x, y.x);
            y.y = fmaf(f[j].y, x.y, y.y);
            y.z = fmaf(f[j].z, x.z, y.z);
            y.w = fmaf(f[j].w, x.w, y.w);
        }
#pragma unroll
        for (int j = 0; j + 1 < TAPS - 1; ++j) u[j] = u[j + 1];
        u[TAPS - 2] = now;
        return y;
    }
};

// y / (1 + e^-y), 32-bit
__device__ __forceinline__ float silu_of(float y) { return y / (1.0f + expf(-y)); }

}  // namespace conv
}  // namespace rfx
