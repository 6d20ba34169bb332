// The any-layout single-pass path (odd widths, unaligned views): what FSS_ALGO_AUTO takes when TMA
// cannot address the tensors.  One launch; every tensor element is read once.
//
// A CTA owns a tile of 128 rows x 32 channels: eight warps of 16 rows, one channel per lane, the rows
// of all tensors held in registers from the first load to the last store.  Tiles are taken from a
// counter, row-block-major in scan order, so a tile only waits for tiles that some CTA already works
// on.  Its entering state comes from a decoupled look-back over the descriptor cells of the eight
// tiles before it (one per warp, one round trip): the nearest final state among them is carried
// forward through the summaries in between, tile by tile.  That is the order in which those tiles
// compute their own final states, so the result does not depend on who was first.
//
// Bound: the launch and memory latency for small problems, then the rate of 2- and 4-byte accesses
// (16 loads per tensor in flight per thread, three CTAs per SM).  Against the chunked kernels with one
// element per access, which read every input twice and compose the chunks' states in one thread per
// column (forward / backward): B4 T1000 D1001 bf16 46 / 50 -> 18 / 26 us, B8 T2048 D2049 bf16 276 / 320 ->
// 126 / 187 us (1.6 / 1.8 TB/s), B1 T65536 D515 bf16 1687 / 1703 -> 142 / 205 us, B2 T8192 D2051 fp32 439 / 517 ->
// 111 / 160 us (3.6 / 4.2 TB/s).
#pragma once

#include "fss_common.cuh"
#include "fss_lookback.cuh"

namespace fss {
namespace ragged {

constexpr int kWarps = 8;             // also the width of the look-back window
constexpr int kRows = 16;             // rows per warp
constexpr int kTileRows = kWarps * kRows;
constexpr int kChannels = 32;         // one per lane
constexpr int kThreads = kWarps * 32;
// descriptor cells of a tile: (product, state from zero) and final state per channel
constexpr int64_t kAggBytes = kChannels * 16, kTileBytes = kAggBytes + kChannels * 8;

struct Params {
    int64_t T, D;
    int64_t S;                // row blocks
    uint32_t ncg, ncols;      // channel groups per row; columns = batch rows * groups
    char *cells;
    lookback::Header *hdr;
    int32_t *status;
    const float *state_in;    // [B, D] or null
    float *state_out;
    const float *h_prev;      // backward only
    int continuation;
    uint32_t max_spins;
};

// P * s + c where a state of exactly zero also absorbs a product that has overflowed
__device__ __forceinline__ float apply(float P, float s, float c) { return s == 0.0f ? c : fmaf(P, s, c); }

template <typename T> struct Scalar;
template <> struct Scalar<bf16> {
    static __device__ __forceinline__ float get(bf16 x) { return __bfloat162float(x); }
    static __device__ __forceinline__ bf16 put(float x) { return __float2bfloat16_rn(x); }
};
template <> struct Scalar<float> {
    static __device__ __forceinline__ float get(float x) { return x; }
    static __device__ __forceinline__ float put(float x) { return x; }
};

__device__ __forceinline__ unsigned long long load_cell(const char *p) {
    unsigned long long c;
    asm volatile("ld.global.cg.b64 %0, [%1];" : "=l"(c) : "l"(p) : "memory");
    return c;
}
__device__ __forceinline__ void store_cell(char *p, float x, uint32_t tag) {
    asm volatile("st.global.cg.b64 [%0], %1;" ::"l"(p), "l"(lookback::make_cell(x, tag)) : "memory");
}

// All views are in scan order (row 0 is the first one the scan visits): the host flips those of a
// scan that runs from the last row.  Forward: x = beta, out0 = h.  Backward: x = the gradient of h,
// the row after the current one in scan order holds h_{t-1}; out0 = dalpha, out1 = dbeta.
template <typename T, bool kBackward>
__global__ void __launch_bounds__(kThreads, 3)
scan_kernel(View<const T> alpha, View<const T> x, View<const T> h, View<T> out0, View<T> out1, const Params p) {
    __shared__ uint32_t s_tile, s_epoch, s_abort;
    __shared__ float sP[kWarps][32], sC[kWarps][32];
    __shared__ float wP[kWarps][32], wC[kWarps][32];      // window: summary, or final state in wC
    __shared__ int w_kind[kWarps];                         // 0 nothing yet, 1 summary, 2 final state
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        s_tile = atomicAdd(&p.hdr->ticket, 1u);
        s_epoch = lookback::ld_volatile(&p.hdr->epoch) + 1u;
        s_abort = 0;
    }
    __syncthreads();
    const uint32_t tile = s_tile, epoch = s_epoch;
    const int64_t s = tile / p.ncols;
    const uint32_t col = tile - (uint32_t)s * p.ncols, cg = col % p.ncg;
    const int64_t b = col / p.ncg, d = (int64_t)cg * kChannels + lane;
    const bool ch_ok = d < p.D;
    const int64_t i0 = s * kTileRows + warp * kRows;
    const int n = !ch_ok || i0 >= p.T ? 0 : (p.T - i0 < kRows ? (int)(p.T - i0) : kRows);      // this thread's rows

    // ---- everything this thread will read, in flight at once
    T ra[kRows], rx[kRows], rh[kBackward ? kRows : 1];
    {
        const T *pa = alpha.row(b, i0) + d, *px = x.row(b, i0) + d, *ph = kBackward ? h.row(b, i0 + 1) + d : nullptr;
        const int nh = i0 + kRows < p.T ? n : n - 1;       // the last row of the scan has no row after it
#pragma unroll
        for (int j = 0; j < kRows; ++j) {
            ra[j] = j < n ? __ldg(pa + j * alpha.st) : Scalar<T>::put(1.0f);      // rows after the end hand the state on
            rx[j] = j < n ? __ldg(px + j * x.st) : Scalar<T>::put(0.0f);
            if (kBackward) rh[j] = j < nh ? __ldg(ph + j * h.st) : Scalar<T>::put(0.0f);
        }
    }
    // The sequence's first row (in time): its alpha is not part of the recurrence unless continued.
    // Forward: scan row 0; backward: scan row T-1.
    const int64_t head_off = (kBackward ? p.T - 1 : 0) - i0;
    const int head = head_off >= 0 && head_off < n ? (int)head_off : -1;
    if (head >= 0) {
        const T prev = kBackward && p.continuation && p.h_prev ? Scalar<T>::put(p.h_prev[b * p.D + d]) : Scalar<T>::put(0.0f);
#pragma unroll
        for (int j = 0; j < kRows; ++j)
            if (j == head) {
                if (!p.continuation) ra[j] = Scalar<T>::put(0.0f);
                if (kBackward) rh[j] = prev;
            }
    }

    // ---- summaries: this warp's rows, the rows of the warps before it, the tile
    float P = 1.0f, C = 0.0f;
#pragma unroll
    for (int j = 0; j < kRows; ++j) {
        const float a = Scalar<T>::get(ra[j]), v = Scalar<T>::get(rx[j]);
        C = kBackward ? a * (v + C) : fmaf(a, C, v);
        P *= a;
    }
    sP[warp][lane] = P;
    sC[warp][lane] = C;
    __syncthreads();
    float tP = 1.0f, tC = 0.0f;
    if (warp == kWarps - 1) {
#pragma unroll
        for (int w = 0; w < kWarps; ++w) {
            tC = apply(sP[w][lane], tC, sC[w][lane]);
            tP *= sP[w][lane];
        }
    }
    const uint32_t tag_agg = (epoch << 2) | lookback::kStateAggregate, tag_inc = (epoch << 2) | lookback::kStateInclusive;
    auto agg_cells = [&](uint32_t k) { return p.cells + (int64_t)k * kTileBytes + lane * 16; };
    auto inc_cell = [&](uint32_t k) { return p.cells + (int64_t)k * kTileBytes + kAggBytes + lane * 8; };
    const bool last_block = s + 1 == p.S;
    if (warp == kWarps - 1 && !last_block && s > 0) {       // (the first block publishes its final state right below)
        store_cell(agg_cells(tile), tP, tag_agg);
        store_cell(agg_cells(tile) + 8, tC, tag_agg);
    }

    // ---- the state that enters the tile
    float cin = p.state_in && ch_ok ? p.state_in[b * p.D + d] : 0.0f;      // ... and the scan
    if (s > 0) {
        const int64_t m = s - 1 - warp;        // row block this warp looks at; -1: the state before the first one
        const float before = cin;
        uint32_t spins = 0;
        for (;;) {
            int kind = 0;
            float vP = 1.0f, vC = before;
            if (m == -1) {
                kind = 2;
            } else if (m >= 0) {
                const uint32_t k = (uint32_t)(m * p.ncols) + col;
                const unsigned long long inc = load_cell(inc_cell(k)), a0 = load_cell(agg_cells(k)), a1 = load_cell(agg_cells(k) + 8);
                if (__all_sync(0xffffffffu, (uint32_t)(inc >> 32) == tag_inc)) {
                    kind = 2;
                    vC = __uint_as_float((uint32_t)inc);
                } else if (__all_sync(0xffffffffu, (uint32_t)(a0 >> 32) == tag_agg && (uint32_t)(a1 >> 32) == tag_agg)) {
                    kind = 1;
                    vP = __uint_as_float((uint32_t)a0);
                    vC = __uint_as_float((uint32_t)a1);
                }
            }
            wP[warp][lane] = vP;
            wC[warp][lane] = vC;
            if (lane == 0) w_kind[warp] = kind;
            if (threadIdx.x == 0 && (++spins & 15u) == 0u) {
                if (spins >= p.max_spins) {
                    atomicExch(&p.hdr->abort, 1u);
                    report_status(p.status, FSS_STATUS_LOOKBACK_TIMEOUT);
                }
                if (lookback::ld_volatile(&p.hdr->abort)) s_abort = 1;
            }
            __syncthreads();
            int from = -1;                     // nearest final state with nothing missing before it
#pragma unroll
            for (int w = kWarps - 1; w >= 0; --w) from = w_kind[w] == 2 ? w : w_kind[w] == 1 ? from : -1;
            const bool stop = s_abort != 0;
            if (from >= 0) {
                cin = wC[from][lane];
                for (int w = from - 1; w >= 0; --w) cin = apply(wP[w][lane], cin, wC[w][lane]);
            }
            __syncthreads();                   // the window may be written again
            if (from >= 0 || stop) {
                if (from < 0) goto leave;      // (the same decision in every thread)
                break;
            }
        }
    }
    {
        const float tile_out = apply(tP, cin, tC);
        if (warp == kWarps - 1) {
            if (!last_block) store_cell(inc_cell(tile), tile_out, tag_inc);
            else if (p.state_out && ch_ok) p.state_out[b * p.D + d] = tile_out;
        }
    }

    // ---- results
    {
        float st = cin;
        for (int w = 0; w < warp; ++w) st = apply(sP[w][lane], st, sC[w][lane]);
        T *p0 = out0.row(b, i0) + d, *p1 = kBackward ? out1.row(b, i0) + d : nullptr;
#pragma unroll
        for (int j = 0; j < kRows; ++j) {
            const float a = Scalar<T>::get(ra[j]), v = Scalar<T>::get(rx[j]);
            if (!kBackward) {
                st = fmaf(a, st, v);
                if (j < n) p0[j * out0.st] = Scalar<T>::put(st);
            } else {
                const float dh = v + st;
                const float da = j == head && !p.continuation ? 0.0f : dh * Scalar<T>::get(rh[j]);
                st = a * dh;
                if (j < n) { p0[j * out0.st] = Scalar<T>::put(da); p1[j * out1.st] = Scalar<T>::put(dh); }
            }
        }
    }
leave:
    // the last CTA advances the epoch, which invalidates every descriptor of this launch
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        if (atomicAdd(&p.hdr->done, 1u) + 1 == gridDim.x) {
            p.hdr->done = 0;
            p.hdr->ticket = 0;
            p.hdr->abort = 0;
            __threadfence();
            p.hdr->epoch = epoch;
        }
    }
}

// ------------------------------------------------------------------ host side
inline int64_t tiles(int64_t B, int64_t T, int64_t D) { return B * ceil_div(D, kChannels) * ceil_div(T, kTileRows); }
// tile numbers are 32-bit (checked without overflow)
inline bool fits(int64_t B, int64_t T, int64_t D) {
    const int64_t lim = 0x7fffffffLL, ncg = ceil_div(D, kChannels), S = ceil_div(T, kTileRows);
    if (ncg > lim || S > lim || B > lim / ncg) return false;
    return S <= lim / (B * ncg);
}
inline size_t workspace_bytes(int64_t B, int64_t T, int64_t D) { return (size_t)tiles(B, T, D) * kTileBytes; }

template <typename T, bool kBackward>
inline int launch(const fss_scan_ctx *ctx, const WsPlan &ws, int64_t B, int64_t Tn, int64_t D, const View<const T> &alpha,
                  const View<const T> &x, const View<const T> &h, const View<T> &out0, const View<T> &out1, Params p,
                  std::string *err_text) {
    if (workspace_bytes(B, Tn, D) > ws.packet_bytes) return FSS_E_WORKSPACE;
    p.T = Tn; p.D = D;
    p.S = ceil_div(Tn, kTileRows);
    p.ncg = (uint32_t)ceil_div(D, kChannels);
    p.ncols = (uint32_t)(B * p.ncg);
    p.cells = ws.packets;
    p.hdr = reinterpret_cast<lookback::Header *>(ws.hdr);
    p.status = ctx->status;
    p.continuation = (ctx->flags & FSS_FLAG_CONTINUATION) ? 1 : 0;
    p.max_spins = (ctx->flags & FSS_FLAG_TEST_SHORT_WAITS) ? 4096u : lookback::kMaxSpins / 4;      // (a round of the window takes several times a poll)
    scan_kernel<T, kBackward><<<(unsigned)tiles(B, Tn, D), kThreads, 0, (cudaStream_t)ctx->stream>>>(alpha, x, h, out0, out1, p);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) { *err_text = std::string("any-layout launch: ") + cudaGetErrorString(e); return FSS_E_LAUNCH; }
    return FSS_OK;
}

}  // namespace ragged
}  // namespace fss
