// Forward scans of a few rows (decoding steps): FSS_ALGO_AUTO takes this path up to kMaxRows rows.
// One thread owns one vector of channels for all rows, loads them at once and walks them; no tiles, no
// descriptors, no TMA maps, no workspace.  Bound: the launch and one memory round trip.  Kernel time against
// the look-back kernel (whose tiles are 64 rows and more, mostly past the end here), bf16 / fp32: B16 T1 D2560 2.1 /
// 1.9 us against 5.4 / 6.9, B128 T4 D5120 3.8 / 5.1 against 31 / 48, B128 T8 D5120 4.8 / 7.0 against 31 / 49.
#pragma once

#include "fss_common.cuh"

namespace fss {
namespace brief {

// Rows that a thread holds in registers, two tensors at once.  Not a crossover: the first lengths past it still take the
// look-back kernel mostly empty tiles (9 rows of B128 D2560 bf16 18 us, 8 rows 3.6).
constexpr int kMaxRows = 8;
constexpr int kThreads = 128;

// Views are in scan order; state vectors 16-byte aligned when V > 1.
template <typename T, int V>
__global__ void __launch_bounds__(kThreads)
scan_forward(int64_t B, int rows, int64_t D, View<const T> alpha, View<const T> beta, View<T> h, const float *__restrict__ state_in,
             float *__restrict__ state_out, bool continuation) {
    const int64_t nvec = D / V, idx = (int64_t)blockIdx.x * kThreads + threadIdx.x;
    if (idx >= B * nvec) return;
    const int64_t b = idx / nvec, d0 = (idx - b * nvec) * V;
    typename Frag<T, V>::Raw ra[kMaxRows], rx[kMaxRows];
#pragma unroll
    for (int t = 0; t < kMaxRows; ++t) {
        if (t < rows) {
            ra[t] = Frag<T, V>::load_raw(alpha.row(b, t) + d0);
            rx[t] = Frag<T, V>::load_raw(beta.row(b, t) + d0);
        }
    }
    float st[V];
#pragma unroll
    for (int v = 0; v < V; ++v) st[v] = 0.0f;
    if (state_in) {
        if constexpr (V == 1) st[0] = state_in[b * D + d0];
        else {
#pragma unroll
            for (int v = 0; v < V; v += 4) {
                const float4 q = *reinterpret_cast<const float4 *>(state_in + b * D + d0 + v);
                st[v] = q.x; st[v + 1] = q.y; st[v + 2] = q.z; st[v + 3] = q.w;
            }
        }
    }
#pragma unroll
    for (int t = 0; t < kMaxRows; ++t) {
        if (t < rows) {
            float a[V], x[V];
            Frag<T, V>::unpack(ra[t], a);
            Frag<T, V>::unpack(rx[t], x);
            const bool head = t == 0 && !continuation;      // the first alpha is not part of the recurrence
#pragma unroll
            for (int v = 0; v < V; ++v) st[v] = fmaf(head ? 0.0f : a[v], st[v], x[v]);
            Frag<T, V>::store(h.row(b, t) + d0, st);
        }
    }
    if (state_out) {
        if constexpr (V == 1) state_out[b * D + d0] = st[0];
        else {
#pragma unroll
            for (int v = 0; v < V; v += 4)
                *reinterpret_cast<float4 *>(state_out + b * D + d0 + v) = make_float4(st[v], st[v + 1], st[v + 2], st[v + 3]);
        }
    }
}

}  // namespace brief
}  // namespace fss
