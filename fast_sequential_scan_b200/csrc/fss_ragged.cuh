// The any-layout single-pass path (odd widths, unaligned views): what FSS_ALGO_AUTO takes when TMA
// cannot address the tensors.  One launch; every tensor element is read once.
//
// A CTA owns a tile of 128 rows x 32 channels (64 where bf16 rows allow 4-byte accesses: even width and
// strides, 4-byte aligned bases): eight warps of 16 rows, one or two channels per lane, the rows
// of all tensors held in registers from the first load to the last store.  Tiles are taken from a
// counter, row-block-major in scan order, so a tile only waits for tiles that some CTA already works
// on.  Its entering state comes from a decoupled look-back over the descriptor cells of the eight
// tiles before it (one per warp, one round trip): the nearest final state among them is carried
// forward through the summaries in between, tile by tile.  That is the order in which those tiles
// compute their own final states, so the result does not depend on who was first.
//
// Bound: the launch and memory latency for small problems, then the rate of 2- and 4-byte accesses
// (16 loads per tensor in flight per thread, two or three CTAs per SM).  Against the chunked kernels with
// one element per access, which read every input twice and compose the chunks' states in one thread
// per column (forward / backward): B4 T1000 D1001 bf16 46 / 50 -> 15 / 24 us, B8 T2048 D2049 bf16 276 / 320 ->
// 87 / 161 us (2.3 / 2.1 TB/s), D2052 76 / 104 us, B1 T65536 D515 bf16 1687 / 1703 -> 113 / 196 us, B2 T8192 D2051 fp32
// 439 / 517 -> 99 / 152 us (4.1 / 4.4 TB/s).  A few rows of many columns are the chunked kernels' (rows_for_chunks).
#pragma once

#include "fss_common.cuh"
#include "fss_lookback.cuh"

namespace fss {
namespace ragged {

constexpr int kWarps = 8;             // also the width of the look-back window
constexpr int kRows = 16;             // rows per warp
constexpr int kTileRows = kWarps * kRows;
constexpr int kThreads = kWarps * 32;
// descriptor cells of a channel and tile: product, state from zero, final state
constexpr int64_t kCellBytes = 24;

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
    int mute_first_block;     // test hook: row block 0 publishes no descriptors (its successors' waits run out)
};

// P * s + c where a state of exactly zero also absorbs a product that has overflowed
__device__ __forceinline__ float apply(float P, float s, float c) { return s == 0.0f ? c : fmaf(P, s, c); }

// V adjacent channels of a row as one access
template <typename T, int V> struct Lot;
template <> struct Lot<bf16, 1> {
    using Raw = bf16;
    static __device__ __forceinline__ void get(const Raw &r, float (&x)[1]) { x[0] = __bfloat162float(r); }
    static __device__ __forceinline__ Raw put(const float (&x)[1]) { return __float2bfloat16_rn(x[0]); }
};
template <> struct Lot<bf16, 2> {
    using Raw = uint32_t;
    static __device__ __forceinline__ void get(const Raw &r, float (&x)[2]) {
        x[0] = __uint_as_float(r << 16);
        x[1] = __uint_as_float(r & 0xffff0000u);
    }
    static __device__ __forceinline__ Raw put(const float (&x)[2]) {
        __nv_bfloat162 v = __floats2bfloat162_rn(x[0], x[1]);
        return *reinterpret_cast<uint32_t *>(&v);
    }
};
template <> struct Lot<float, 1> {
    using Raw = float;
    static __device__ __forceinline__ void get(const Raw &r, float (&x)[1]) { x[0] = r; }
    static __device__ __forceinline__ Raw put(const float (&x)[1]) { return x[0]; }
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
// CTAs per SM the registers are cut for.  A third one pays where it costs no spills: fp32 backward 152
// us with three against 177 with two (B2 T8192 D2051), bf16 backward 207 against 171 (B8 T2048 D2049), pairs 118
// against 104 (D2052).
template <typename T, bool kBackward, int V> constexpr int kMinCtas = V == 2 || (kBackward && sizeof(T) == 2) ? 2 : 3;
// kEarly: a first look at the tile before this one, ahead of the loads.  With more columns than a wave of
// CTAs takes, that tile is long finished and its final state is here before this tile's rows are: B8 T2048
// D2049 bf16 forward / backward 95 / 171 -> 87 / 161 us, B16 T512 D4093 91 / 166 -> 86 / 157.  With fewer columns it
// finds nothing and costs 1-2 % (B4 T1000 D1001), and the fp32 kernels have no registers left for it.
template <typename T, bool kBackward, int V, bool kEarly>
__global__ void __launch_bounds__(kThreads, kMinCtas<T, kBackward, V>)
scan_kernel(View<const T> alpha, View<const T> x, View<const T> h, View<T> out0, View<T> out1, const Params p) {
    using L = Lot<T, V>;
    using Raw = typename L::Raw;
    __shared__ uint32_t s_tile, s_epoch, s_abort, s_early;
    __shared__ float sP[V][kWarps][32], sC[V][kWarps][32];
    __shared__ float wP[V][kWarps][32], wC[V][kWarps][32];      // window: summary, or final state in wC
    __shared__ int w_kind[kWarps];                               // 0 nothing yet, 1 summary, 2 final state
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        s_tile = atomicAdd(&p.hdr->ticket, 1u);
        s_epoch = lookback::ld_volatile(&p.hdr->epoch) + 1u;
        s_abort = 0;
        s_early = 0;
    }
    __syncthreads();
    const uint32_t tile = s_tile, epoch = s_epoch;
    const int64_t s = tile / p.ncols;
    const uint32_t col = tile - (uint32_t)s * p.ncols, cg = col % p.ncg;
    const int64_t b = col / p.ncg, d = ((int64_t)cg * 32 + lane) * V;
    const bool ch_ok = d < p.D;                                  // (V divides D)
    const int64_t i0 = s * kTileRows + warp * kRows;
    const int n = !ch_ok || i0 >= p.T ? 0 : (p.T - i0 < kRows ? (int)(p.T - i0) : kRows);      // this thread's rows

    const uint32_t tag_agg = (epoch << 2) | lookback::kStateAggregate, tag_inc = (epoch << 2) | lookback::kStateInclusive;
    auto agg_cells = [&](uint32_t k, int v) { return p.cells + (int64_t)k * (32 * V * kCellBytes) + (v * 32 + lane) * 16; };
    auto inc_cell = [&](uint32_t k, int v) { return p.cells + (int64_t)k * (32 * V * kCellBytes) + 32 * V * 16 + (v * 32 + lane) * 8; };

    const bool early_look = kEarly && warp == 0 && s > 0;
    unsigned long long early[V];
    if (early_look) {
#pragma unroll
        for (int v = 0; v < V; ++v) early[v] = load_cell(inc_cell(tile - p.ncols, v));
    }

    // ---- everything this thread will read, in flight at once
    float ones[V], zeros[V];
#pragma unroll
    for (int v = 0; v < V; ++v) { ones[v] = 1.0f; zeros[v] = 0.0f; }
    const Raw one = L::put(ones), zero = L::put(zeros);
    Raw ra[kRows], rx[kRows], rh[kBackward ? kRows : 1];
    {
        const T *pa = alpha.row(b, i0) + d, *px = x.row(b, i0) + d, *ph = kBackward ? h.row(b, i0 + 1) + d : nullptr;
        const int nh = i0 + kRows < p.T ? n : n - 1;       // the last row of the scan has no row after it
#pragma unroll
        for (int j = 0; j < kRows; ++j) {
            ra[j] = j < n ? __ldg(reinterpret_cast<const Raw *>(pa + j * alpha.st)) : one;      // rows after the end hand the state on
            rx[j] = j < n ? __ldg(reinterpret_cast<const Raw *>(px + j * x.st)) : zero;
            if (kBackward) rh[j] = j < nh ? __ldg(reinterpret_cast<const Raw *>(ph + j * h.st)) : zero;
        }
    }
    // The sequence's first row (in time): its alpha is not part of the recurrence unless continued.
    // Forward: scan row 0; backward: scan row T-1.
    const int64_t head_off = (kBackward ? p.T - 1 : 0) - i0;
    const int head = head_off >= 0 && head_off < n ? (int)head_off : -1;
    // the state before that row (backward), in 32 bits: fp32 rows have a place for it, bf16 rows get it at their end
    const bool has_prev = kBackward && head >= 0 && p.continuation && p.h_prev;
    if (head >= 0) {
        float prev[V];
#pragma unroll
        for (int v = 0; v < V; ++v) prev[v] = sizeof(T) == 4 && has_prev ? p.h_prev[b * p.D + d + v] : 0.0f;
#pragma unroll
        for (int j = 0; j < kRows; ++j)
            if (j == head) {
                if (!p.continuation) ra[j] = zero;
                if (kBackward && sizeof(T) == 4) rh[j] = L::put(prev);
            }
    }

    if (early_look) {
        bool ok = true;
#pragma unroll
        for (int v = 0; v < V; ++v) {
            ok &= (uint32_t)(early[v] >> 32) == tag_inc;
            wC[v][0][lane] = __uint_as_float((uint32_t)early[v]);
        }
        ok = __all_sync(0xffffffffu, ok);
        if (lane == 0) s_early = ok;
    }

    // ---- summaries: this warp's rows, the rows of the warps before it, the tile
    {
        float P[V], C[V];
#pragma unroll
        for (int v = 0; v < V; ++v) { P[v] = 1.0f; C[v] = 0.0f; }
#pragma unroll
        for (int j = 0; j < kRows; ++j) {
            float a[V], y[V];
            L::get(ra[j], a);
            L::get(rx[j], y);
#pragma unroll
            for (int v = 0; v < V; ++v) {
                C[v] = kBackward ? a[v] * (y[v] + C[v]) : fmaf(a[v], C[v], y[v]);
                P[v] *= a[v];
            }
        }
#pragma unroll
        for (int v = 0; v < V; ++v) { sP[v][warp][lane] = P[v]; sC[v][warp][lane] = C[v]; }
    }
    __syncthreads();
    const bool last_block = s + 1 == p.S;
    float tP[V], tC[V];                                          // the tile's summary, in the last warp
    if (warp == kWarps - 1) {
#pragma unroll
        for (int v = 0; v < V; ++v) {
            tP[v] = 1.0f;
            tC[v] = 0.0f;
#pragma unroll
            for (int w = 0; w < kWarps; ++w) {
                tC[v] = apply(sP[v][w][lane], tC[v], sC[v][w][lane]);
                tP[v] *= sP[v][w][lane];
            }
            if (!last_block && s > 0) {       // (the first block publishes its final state right below)
                store_cell(agg_cells(tile, v), tP[v], tag_agg);
                store_cell(agg_cells(tile, v) + 8, tC[v], tag_agg);
            }
        }
    }

    // ---- the state that enters the tile
    bool gave_up = false;
    float cin[V];
#pragma unroll
    for (int v = 0; v < V; ++v) cin[v] = p.state_in && ch_ok ? p.state_in[b * p.D + d + v] : 0.0f;      // ... and the scan
    if (kEarly && s > 0 && s_early) {
#pragma unroll
        for (int v = 0; v < V; ++v) cin[v] = wC[v][0][lane];
    } else if (s > 0) {
        const int64_t m = s - 1 - warp;        // row block this warp looks at; -1: the state before the first one
        uint32_t spins = 0;
        float before[V];
#pragma unroll
        for (int v = 0; v < V; ++v) before[v] = cin[v];
        for (;;) {
            int kind = 0;
            float vP[V], vC[V];
#pragma unroll
            for (int v = 0; v < V; ++v) { vP[v] = 1.0f; vC[v] = before[v]; }
            if (m == -1) {
                kind = 2;
            } else if (m >= 0) {
                const uint32_t k = (uint32_t)(m * p.ncols) + col;
                unsigned long long inc[V], a0[V], a1[V];
#pragma unroll
                for (int v = 0; v < V; ++v) {
                    inc[v] = load_cell(inc_cell(k, v));
                    a0[v] = load_cell(agg_cells(k, v));
                    a1[v] = load_cell(agg_cells(k, v) + 8);
                }
                bool inc_ok = true, agg_ok = true;
#pragma unroll
                for (int v = 0; v < V; ++v) {
                    inc_ok &= (uint32_t)(inc[v] >> 32) == tag_inc;
                    agg_ok &= (uint32_t)(a0[v] >> 32) == tag_agg && (uint32_t)(a1[v] >> 32) == tag_agg;
                }
                if (__all_sync(0xffffffffu, inc_ok)) {
                    kind = 2;
#pragma unroll
                    for (int v = 0; v < V; ++v) vC[v] = __uint_as_float((uint32_t)inc[v]);
                } else if (__all_sync(0xffffffffu, agg_ok)) {
                    kind = 1;
#pragma unroll
                    for (int v = 0; v < V; ++v) { vP[v] = __uint_as_float((uint32_t)a0[v]); vC[v] = __uint_as_float((uint32_t)a1[v]); }
                }
            }
#pragma unroll
            for (int v = 0; v < V; ++v) { wP[v][warp][lane] = vP[v]; wC[v][warp][lane] = vC[v]; }
            if (lane == 0) w_kind[warp] = kind;
            if (threadIdx.x == 0 && (++spins & 15u) == 0u) {
                if (spins >= p.max_spins) {
                    atomicExch(&p.hdr->abort, 1u);
                    __threadfence();           // ahead of this CTA's count, so that the last CTA's reset comes after it
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
#pragma unroll
                for (int v = 0; v < V; ++v) {
                    cin[v] = wC[v][from][lane];
                    for (int w = from - 1; w >= 0; --w) cin[v] = apply(wP[v][w][lane], cin[v], wC[v][w][lane]);
                }
            }
            __syncthreads();                   // the window may be written again
            if (from >= 0 || stop) {
                gave_up = from < 0;            // (the same decision in every thread)
                break;
            }
        }
    }
    if (warp == kWarps - 1 && !gave_up) {
#pragma unroll
        for (int v = 0; v < V; ++v) {
            const float tile_out = apply(tP[v], cin[v], tC[v]);
            if (last_block) {
                if (p.state_out && ch_ok) p.state_out[b * p.D + d + v] = tile_out;
            } else if (s > 0 || !p.mute_first_block) {
                store_cell(inc_cell(tile, v), tile_out, tag_inc);
            }
        }
    }
    // counted here, so that the answer arrives while the results are written (with a fence at the CTA's end
    // B8 T2048 D2049 bf16 forward took 126 us instead of 95)
    const uint32_t finished = threadIdx.x == 0 ? atomicAdd(&p.hdr->done, 1u) : 0u;

    // ---- results
    if (!gave_up) {
        float st[V];
#pragma unroll
        for (int v = 0; v < V; ++v) {
            st[v] = cin[v];
            for (int w = 0; w < warp; ++w) st[v] = apply(sP[v][w][lane], st[v], sC[v][w][lane]);
        }
        float prev[V];
#pragma unroll
        for (int v = 0; v < V; ++v) prev[v] = sizeof(T) == 2 && has_prev ? p.h_prev[b * p.D + d + v] : 0.0f;
        T *p0 = out0.row(b, i0) + d, *p1 = kBackward ? out1.row(b, i0) + d : nullptr;
#pragma unroll
        for (int j = 0; j < kRows; ++j) {
            float a[V], y[V], hp[V], da[V], dh[V];
            L::get(ra[j], a);
            L::get(rx[j], y);
            if (kBackward) L::get(rh[j], hp);
#pragma unroll
            for (int v = 0; v < V; ++v) {
                if (!kBackward) {
                    st[v] = fmaf(a[v], st[v], y[v]);
                } else {
                    dh[v] = y[v] + st[v];
                    da[v] = j == head && !p.continuation ? 0.0f : dh[v] * (j == head && sizeof(T) == 2 ? prev[v] : hp[v]);
                    st[v] = a[v] * dh[v];
                }
            }
            if (j < n) {
                *reinterpret_cast<Raw *>(p0 + j * out0.st) = L::put(kBackward ? da : st);
                if (kBackward) *reinterpret_cast<Raw *>(p1 + j * out1.st) = L::put(dh);
            }
        }
    }
    // the CTA that finished its look-back last advances the epoch, which invalidates every descriptor of
    // this launch: nobody needs the header any more
    if (threadIdx.x == 0 && finished + 1 == gridDim.x) {
        p.hdr->done = 0;
        p.hdr->ticket = 0;
        p.hdr->abort = 0;
        p.hdr->epoch = epoch;
    }
}

// ------------------------------------------------------------------ host side
// rows that 4-byte accesses can address
inline bool pair_aligned(const View<const bf16> &v) { return !(reinterpret_cast<uintptr_t>(v.ptr) & 3u) && !(v.sb & 1) && !(v.st & 1); }
inline bool pairs_ok(int64_t D, std::initializer_list<View<const bf16>> views) {
    if (D % 2) return false;
    for (const auto &v : views)
        if (!pair_aligned(v)) return false;
    return true;
}
inline int64_t tiles(int64_t B, int64_t T, int64_t D, int V) { return B * ceil_div(D, 32 * V) * ceil_div(T, kTileRows); }
// tile numbers are 32-bit (checked without overflow)
inline bool fits(int64_t B, int64_t T, int64_t D) {
    const int64_t lim = 0x7fffffffLL, ncg = ceil_div(D, 32), S = ceil_div(T, kTileRows);
    if (ncg > lim || S > lim || B > lim / ncg) return false;
    return S <= lim / (B * ncg);
}
inline size_t workspace_bytes(int64_t B, int64_t T, int64_t D) { return (size_t)(tiles(B, T, D, 2) * 64 * kCellBytes); }

// Up to how many rows the chunked kernels are faster.  A tile costs its CTA much the same whether its 128
// rows are there or not, which nobody notices while the CTAs fit the GPU at once (some 300 of them); the
// chunked kernels do little for few rows.  With more columns of tiles the line rises to the rows of a tile that
// pay for its launch, look-back and stores.  Any-layout against chunked, B128 D1001 bf16 forward / backward (4,096
// columns): 9 rows 33 / 57 us against 13 / 14, 32 rows 35 / 63 against 26 / 30, 64 rows 37 / 68 against 40 / 54, 100 rows 40 /
// 78 against 68 / 101; fp32 32 rows 34 / 52 against 24 / 32, 64 rows 39 / 58 against 42 / 66; by pairs (B128 D5002) 32 rows
// 134 / 176 against 116 / 144, 48 rows 137 / 183 against 196 / 231.  B16 D1001 (512 columns): backward 9 rows 9.6 against
// 8.0, 24 rows 10.4 against 11.5.  Measured over 64 to 10,048 columns and 1 to 520 rows; near the line, and for bf16
// backwards of 129 to 150 rows, the two lie within 7 % of each other.
template <typename T, bool kBackward> inline int64_t rows_for_chunks(int64_t cols, bool pairs) {
    const bool wide = sizeof(T) == 4;
    const int64_t cap = kBackward ? (wide ? 54 : pairs ? 38 : 84) : (wide ? 50 : pairs ? 36 : 54);
    const int64_t step = kBackward ? (wide ? 17 : 12) : (wide ? 25 : pairs ? 55 : 45);
    const int64_t rows = (cols - 300) / step;
    return rows < cap ? rows : cap;
}

template <typename T, bool kBackward, int V>
inline int launch_lots(const fss_scan_ctx *ctx, const WsPlan &ws, int64_t B, int64_t Tn, int64_t D, const View<const T> &alpha,
                       const View<const T> &x, const View<const T> &h, const View<T> &out0, const View<T> &out1, Params p,
                       std::string *err_text) {
    if (workspace_bytes(B, Tn, D) > ws.packet_bytes) return FSS_E_WORKSPACE;
    p.T = Tn; p.D = D;
    p.S = ceil_div(Tn, kTileRows);
    p.ncg = (uint32_t)ceil_div(D, 32 * V);
    p.ncols = (uint32_t)(B * p.ncg);
    p.cells = ws.packets;
    p.hdr = reinterpret_cast<lookback::Header *>(ws.hdr);
    p.status = ctx->status;
    p.continuation = (ctx->flags & FSS_FLAG_CONTINUATION) ? 1 : 0;
    p.max_spins = (ctx->flags & FSS_FLAG_TEST_SHORT_WAITS) ? 4096u : lookback::kMaxSpins / 4;      // (a round of the window takes several times a poll)
    p.mute_first_block = (ctx->flags & FSS_FLAG_TEST_MUTE_FIRST_BLOCK) ? 1 : 0;
    const unsigned grid = (unsigned)tiles(B, Tn, D, V);
    const cudaStream_t stream = (cudaStream_t)ctx->stream;
    if (sizeof(T) == 2 && p.ncols >= 2 * 148)      // (a wave: two CTAs on each of the 148 SMs)
        scan_kernel<T, kBackward, V, sizeof(T) == 2><<<grid, kThreads, 0, stream>>>(alpha, x, h, out0, out1, p);
    else
        scan_kernel<T, kBackward, V, false><<<grid, kThreads, 0, stream>>>(alpha, x, h, out0, out1, p);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) { *err_text = std::string("any-layout launch: ") + cudaGetErrorString(e); return FSS_E_LAUNCH; }
    return FSS_OK;
}
template <typename T, bool kBackward>
inline int launch(const fss_scan_ctx *ctx, const WsPlan &ws, int64_t B, int64_t Tn, int64_t D, const View<const T> &alpha,
                  const View<const T> &x, const View<const T> &h, const View<T> &out0, const View<T> &out1, const Params &p,
                  std::string *err_text) {
    if constexpr (sizeof(T) == 2) {
        auto in = [](const View<T> &v) { return View<const T>{v.ptr, v.sb, v.st}; };
        if (pairs_ok(D, {alpha, x, h, in(out0), in(out1)}))
            return launch_lots<T, kBackward, 2>(ctx, ws, B, Tn, D, alpha, x, h, out0, out1, p, err_text);
    }
    return launch_lots<T, kBackward, 1>(ctx, ws, B, Tn, D, alpha, x, h, out0, out1, p, err_text);
}

}  // namespace ragged
}  // namespace fss
