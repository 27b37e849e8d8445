// The llama.cpp bridge's entry points (integration/polarquant-kv.patch of the reference,
// decoded lines 695-763) for sm_100a: the per-vector-radius codec with nibble-packed
// indices, as kernels laid out for a 148-SM part instead of one CTA per vector / per head.
//
//   compress   below 4096 vectors, and for other head dims than 64 and 128, a CTA takes one vector (four from 768 vectors
//              on) and streams R from L2; above that an FP32 kernel with R^T in shared memory, and for buffers on 16-byte
//              boundaries and more than a wave of its CTAs pq_bridge_compress.cu (tensor cores).
//   attention  head dims 64 and 128: pq_bridge_attn.cu.  Other head dims: CTAs own (kv head, query group, slice of S); a
//              warp takes 32 tokens at a time, each lane holds D/32 (rounded up) dims, the 32 partial dot products are
//              transposed and summed with 31 shuffles so that lane t ends with token t's score; online softmax; the
//              slices are merged by the last CTA to finish.
//   rotate / inverse rotate: one CTA per row (a few dozen rows per call).
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstdlib>

#include "polarquant_llama_abi.h"
#include "pq_bridge.cuh"
#include "pq_common.cuh"

namespace {

thread_local int t_last_error = 0;

enum { kErrNull = 1, kErrDim = 2, kErrLevels = 3, kErrHeads = 4, kErrCuda = 5 };

constexpr int kMaxDim = 1024;
constexpr unsigned kFull = 0xffffffffu;

bool fail(int code, const char* what) {
    t_last_error = code;
    fprintf(stderr, "PolarQuant: %s\n", what);
    return false;
}

bool dim_ok(int D) { return D > 0 && D <= kMaxDim && (D & 1) == 0; }

bool launched() {
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) {
        t_last_error = kErrCuda;
        fprintf(stderr, "PolarQuant: %s\n", cudaGetErrorString(e));
        return false;
    }
    return true;
}

// ---------------------------------------------------------------------------------------------
// rows · Rᵀ and rows · R
// ---------------------------------------------------------------------------------------------

int device_sms() {
    int dev = 0, sms = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    return sms;
}

// These run over a few dozen rows per call and are bound by the latency of R's loads from L2, so what counts is how many
// of them a warp has in flight: a warp takes kRowBatch rows of R at once (a row per loop step, as a first version did,
// is one round trip after another: 6 us instead of 2.5 for a token's eight vectors of 128).
constexpr int kRowBatch = 8;

// dot[v][u] = sum_k xs[v][k] * R[j0 + u][k] over the warp's lanes (every lane gets the sums); rows past D read row D - 1.
template <int V>
__device__ __forceinline__ void dot_rows(const float (*xs)[kMaxDim], const float* __restrict__ R, int D, int j0, int lane,
                                         float (&dot)[V][kRowBatch]) {
#pragma unroll
    for (int v = 0; v < V; ++v)
#pragma unroll
        for (int u = 0; u < kRowBatch; ++u) dot[v][u] = 0.0f;
#pragma unroll (V == 1 ? 4 : 2)
    for (int k = lane; k < D; k += 32) {
        float r[kRowBatch];
#pragma unroll
        for (int u = 0; u < kRowBatch; ++u) r[u] = __ldg(R + (size_t)min(j0 + u, D - 1) * D + k);
#pragma unroll
        for (int v = 0; v < V; ++v) {
            const float x = xs[v][k];
#pragma unroll
            for (int u = 0; u < kRowBatch; ++u) dot[v][u] = fmaf(x, r[u], dot[v][u]);
        }
    }
#pragma unroll
    for (int o = 16; o; o >>= 1)
#pragma unroll
        for (int v = 0; v < V; ++v)
#pragma unroll
            for (int u = 0; u < kRowBatch; ++u) dot[v][u] += __shfl_xor_sync(kFull, dot[v][u], o);
}

// out[n][j] = sum_k in[n][k] * R[j][k]: lanes along k (coalesced).
__global__ void __launch_bounds__(512) rotate_rows_kernel(const float* in, const float* __restrict__ R, float* out, int D) {
    __shared__ float xs[1][kMaxDim];
    const int n = blockIdx.x;
    for (int k = threadIdx.x; k < D; k += blockDim.x) xs[0][k] = in[(size_t)n * D + k];
    __syncthreads();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int j0 = warp * kRowBatch; j0 < D; j0 += (blockDim.x >> 5) * kRowBatch) {
        float dot[1][kRowBatch];
        dot_rows<1>(xs, R, D, j0, lane, dot);
#pragma unroll
        for (int u = 0; u < kRowBatch; ++u)
            if (lane == u && j0 + u < D) out[(size_t)n * D + j0 + u] = dot[0][u];
    }
}

// out[n][j] = sum_k in[n][k] * R[k][j] for the COLS columns from blockIdx.y * COLS, k dealt to PARTS threads of a column.
// Latency again: a thread's loads of R are independent, and with 1024 threads a row takes one to eight round trips.
template <int COLS, int PARTS>
__global__ void __launch_bounds__(COLS * PARTS) inverse_rotate_split_kernel(const float* __restrict__ in, const float* __restrict__ R,
                                                                            float* __restrict__ out, int D) {
    __shared__ float xs[kMaxDim];
    __shared__ float part[PARTS][COLS];
    const int n = blockIdx.x, c = threadIdx.x, y = threadIdx.y, j = blockIdx.y * COLS + c;
    for (int k = y * COLS + c; k < D; k += COLS * PARTS) xs[k] = in[(size_t)n * D + k];
    __syncthreads();
    const float* col = R + min(j, D - 1);
    float s = 0.0f;
#pragma unroll 16
    for (int k = y; k < D; k += PARTS) s = fmaf(xs[k], __ldg(col + (size_t)k * D), s);
    part[y][c] = s;
    __syncthreads();
    if (y == 0 && j < D) {
        float t = 0.0f;
#pragma unroll
        for (int u = 0; u < PARTS; ++u) t += part[u][c];
        out[(size_t)n * D + j] = t;
    }
}

// The same by one CTA per row, a thread per column, which reads its input before it writes: `output` may be `input`.  Also
// the faster one for many rows, whose CTAs fill the card by themselves.  Split / one CTA per row: 32 rows of 128 2.9 / 4.8 us,
// of 1024 16 / 108; 200 rows of 256 7.9 / 8.7, of 1024 80 / 111; 512 rows of 128 6.2 / 5.2, of 256 16 / 9.8, of 1024 201 / 125.
__global__ void __launch_bounds__(256) inverse_rotate_rows_kernel(const float* __restrict__ in,
                                                                  const float* __restrict__ R,
                                                                  float* __restrict__ out, int D) {
    __shared__ float xs[kMaxDim];
    const int n = blockIdx.x;
    for (int k = threadIdx.x; k < D; k += blockDim.x) xs[k] = in[(size_t)n * D + k];
    __syncthreads();
    for (int j = threadIdx.x; j < D; j += blockDim.x) {
        float s = 0.0f;
        for (int k = 0; k < D; ++k) s = fmaf(xs[k], R[(size_t)k * D + j], s);
        out[(size_t)n * D + j] = s;
    }
}

// ---------------------------------------------------------------------------------------------
// compress
// ---------------------------------------------------------------------------------------------

__device__ __forceinline__ int nearest_level(float v, const float* cb, int n_levels) {
    int best = 0;
    float dist = 1e30f;
    for (int i = 0; i < n_levels; ++i) {
        const float d = fabsf(v - cb[i]);
        if (d < dist) { dist = d; best = i; }
    }
    return best;
}

constexpr int kCmpWarps = 8;
constexpr int kCmpVecs = 4;      // vectors a warp carries through the rotation together
constexpr int kCmpMin = 4096;

// Head dims 64 and 128, whatever the alignment.  R^T sits in shared memory once per CTA, a warp carries four vectors, lane l
// owns rotated elements l + 32 i; the sum of squares is combined in the order of the reference's shared-memory tree.  The
// tensor-core kernel stores the same bytes and is the faster one once there is more than a wave of this one's CTAs (Lloyd-Max
// table, this kernel / that one: 9472 vectors of 128 22.6 / 22.8 us, 18 944 39 / 23; 18 944 vectors of 64 15.3 / 16.5 us,
// 40 000 29 / 21).
template <int D>
__global__ void __launch_bounds__(kCmpWarps * 32) compress_kernel(const float* __restrict__ input,
                                                                   const float* __restrict__ R,
                                                                   const float* __restrict__ codebook,
                                                                   float* __restrict__ radius_out,
                                                                   uint8_t* __restrict__ packed_out,
                                                                   int N, int n_levels) {
    constexpr int DPL = D / 32;
    constexpr int kPitch = D + 1;                       // transposed fill and row reads both conflict-free
    extern __shared__ __align__(16) float smem[];
    float* Rt = smem;                                   // Rt[k][j] = R[j][k]
    float* xs = smem + D * kPitch;                      // [warp][k][kCmpVecs]
    __shared__ float cb[16];
    if (threadIdx.x < n_levels) cb[threadIdx.x] = codebook[threadIdx.x];
    for (int e = threadIdx.x; e < D * D; e += blockDim.x) {
        const int j = e / D, k = e - j * D;
        Rt[k * kPitch + j] = R[e];
    }
    __syncthreads();

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    float4* xw = reinterpret_cast<float4*>(xs + warp * D * kCmpVecs);
    const int n_groups = (N + kCmpVecs - 1) / kCmpVecs;
    for (int grp = blockIdx.x * kCmpWarps + warp; grp < n_groups; grp += gridDim.x * kCmpWarps) {
        const int v0 = grp * kCmpVecs;
        // stage the four inputs interleaved: xw[k] = {x0[k], x1[k], x2[k], x3[k]}
        for (int k = lane; k < D; k += 32) {
            float4 x;
            x.x = input[(size_t)v0 * D + k];
            x.y = v0 + 1 < N ? input[(size_t)(v0 + 1) * D + k] : 0.0f;
            x.z = v0 + 2 < N ? input[(size_t)(v0 + 2) * D + k] : 0.0f;
            x.w = v0 + 3 < N ? input[(size_t)(v0 + 3) * D + k] : 0.0f;
            xw[k] = x;
        }
        __syncwarp();
        float acc[kCmpVecs][DPL];
#pragma unroll
        for (int v = 0; v < kCmpVecs; ++v)
#pragma unroll
            for (int i = 0; i < DPL; ++i) acc[v][i] = 0.0f;
#pragma unroll 4
        for (int k = 0; k < D; ++k) {
            const float4 x = xw[k];
#pragma unroll
            for (int i = 0; i < DPL; ++i) {
                const float r = Rt[k * kPitch + lane + 32 * i];
                acc[0][i] = fmaf(x.x, r, acc[0][i]);
                acc[1][i] = fmaf(x.y, r, acc[1][i]);
                acc[2][i] = fmaf(x.z, r, acc[2][i]);
                acc[3][i] = fmaf(x.w, r, acc[3][i]);
            }
        }
        __syncwarp();
#pragma unroll
        for (int v = 0; v < kCmpVecs; ++v) {
            // sum of squares: element t pairs with t + D/2, then + D/4, ... down to + 1
            float sq[DPL];
#pragma unroll
            for (int i = 0; i < DPL; ++i) sq[i] = __fmul_rn(acc[v][i], acc[v][i]);   // no contraction into the adds
#pragma unroll
            for (int h = DPL / 2; h; h >>= 1)
#pragma unroll
                for (int i = 0; i < h; ++i) sq[i] = __fadd_rn(sq[i], sq[i + h]);
            float s = sq[0];
#pragma unroll
            for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(kFull, s, o);
            const float radius = sqrtf(s);
            const bool live = v0 + v < N;
            if (live && lane == 0) radius_out[v0 + v] = radius;
#pragma unroll
            for (int i = 0; i < DPL; ++i) {
                const float dir = radius > 1e-30f ? acc[v][i] / radius : 0.0f;
                const int idx = nearest_level(dir, cb, n_levels);
                const int up = __shfl_down_sync(kFull, idx, 1);
                if (live && !(lane & 1))
                    packed_out[(size_t)(v0 + v) * (D / 2) + (lane >> 1) + 16 * i] = (uint8_t)(idx | (up << 4));
            }
        }
    }
}

template <int D>
cudaError_t launch_compress(int ctas, const float* input, const float* R, const float* codebook, float* radius_out,
                            uint8_t* packed_out, int N, int n_levels, cudaStream_t stream) {
    constexpr size_t smem = ((size_t)D * (D + 1) + (size_t)kCmpWarps * D * kCmpVecs) * sizeof(float);
    static std::atomic<uint64_t> allowed{0};
    const cudaError_t e = pq::allow_shared(compress_kernel<D>, smem, allowed);
    if (e != cudaSuccess) return e;
    compress_kernel<D><<<ctas, kCmpWarps * 32, smem, stream>>>(input, R, codebook, radius_out, packed_out, N, n_levels);
    return cudaGetLastError();
}

// Any even head dim up to 1024: V vectors per CTA.  One, so that a token's few vectors spread over the SMs; four once L2,
// which every CTA streams the whole of R from, is what counts (one / four: 511 vectors of 128 7.8 / 9.3 us, of 256 15 / 22, of
// 1024 125 / 254; 1000 of 128 14 / 11.6, of 256 30 / 25, of 1024 245 / 254).
constexpr int kCmpFour = 768;
constexpr int kSmallWarps = 16;
template <int V>
__global__ void __launch_bounds__(kSmallWarps * 32) compress_any_dim_kernel(const float* __restrict__ input,
                                                               const float* __restrict__ R,
                                                               const float* __restrict__ codebook,
                                                               float* __restrict__ radius_out,
                                                               uint8_t* __restrict__ packed_out,
                                                               int N, int D, int n_levels) {
    __shared__ float xs[V][kMaxDim];
    __shared__ float rot[V][kMaxDim];
    __shared__ float cb[16];
    __shared__ float part[V][8];
    const int n0 = blockIdx.x * V;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x < n_levels) cb[threadIdx.x] = codebook[threadIdx.x];
#pragma unroll
    for (int v = 0; v < V; ++v)
        for (int k = threadIdx.x; k < D; k += blockDim.x) xs[v][k] = input[(size_t)min(n0 + v, N - 1) * D + k];
    __syncthreads();
    for (int j0 = warp * kRowBatch; j0 < D; j0 += kSmallWarps * kRowBatch) {
        float dot[V][kRowBatch];
        dot_rows<V>(xs, R, D, j0, lane, dot);
#pragma unroll
        for (int u = 0; u < kRowBatch; ++u)
#pragma unroll
            for (int v = 0; v < V; ++v)
                if (lane == u && j0 + u < D) rot[v][j0 + u] = dot[v][u];
    }
    __syncthreads();
    // squares in eight chains (j mod 8), added in order: stored indices at a decision point depend on the order
    if (threadIdx.x < 8 * V) {
        const int v = threadIdx.x >> 3, w = threadIdx.x & 7;
        float sq = 0.0f;
#pragma unroll 8
        for (int j = w; j < D; j += 8) sq = fmaf(rot[v][j], rot[v][j], sq);
        part[v][w] = sq;
    }
    __syncthreads();
#pragma unroll
    for (int v = 0; v < V; ++v) {
        if (n0 + v >= N) break;
        float total = 0.0f;
#pragma unroll
        for (int w = 0; w < 8; ++w) total += part[v][w];
        const float radius = sqrtf(total);
        if (threadIdx.x == 0) radius_out[n0 + v] = radius;
        // a quarter of the threads per vector when there are four
        for (int b = (int)threadIdx.x - v * (kSmallWarps * 32 / V); b < D / 2; b += kSmallWarps * 32) {
            if (b < 0) continue;
            const float d0 = radius > 1e-30f ? rot[v][2 * b] / radius : 0.0f;
            const float d1 = radius > 1e-30f ? rot[v][2 * b + 1] / radius : 0.0f;
            packed_out[(size_t)(n0 + v) * (D / 2) + b] =
                (uint8_t)(nearest_level(d0, cb, n_levels) | (nearest_level(d1, cb, n_levels) << 4));
        }
    }
}

// ---------------------------------------------------------------------------------------------
// attention
// ---------------------------------------------------------------------------------------------

constexpr int kAttWarps = 4;
constexpr int kTile = 32;                     // tokens a warp takes at a time (lane t <-> token t)
constexpr float kLowest = -1e30f;

using AttnParams = pq::BridgeAttnParams;

// DPL/2 packed bytes of one row for this lane, zero beyond the row.
template <int DPL>
__device__ __forceinline__ void load_row_bytes(const uint8_t* row, int row_bytes, int lane, bool vec,
                                               uint32_t (&w)[(DPL + 7) / 8]) {
    constexpr int BPL = DPL / 2;
    constexpr int W = (DPL + 7) / 8;
    const int b0 = lane * BPL;
#pragma unroll
    for (int i = 0; i < W; ++i) w[i] = 0;
    if (vec && b0 + BPL <= row_bytes) {
        if constexpr (BPL == 1) w[0] = row[b0];
        else if constexpr (BPL == 2) w[0] = *reinterpret_cast<const uint16_t*>(row + b0);
        else if constexpr (BPL == 4) w[0] = *reinterpret_cast<const uint32_t*>(row + b0);
        else if constexpr (BPL == 8) {
            const uint2 t = *reinterpret_cast<const uint2*>(row + b0);
            w[0] = t.x; w[1] = t.y;
        } else {
            const uint4 t = *reinterpret_cast<const uint4*>(row + b0);
            w[0] = t.x; w[1] = t.y; w[2] = t.z; w[3] = t.w;
        }
    } else {
#pragma unroll
        for (int b = 0; b < BPL; ++b)
            if (b0 + b < row_bytes) w[b >> 2] |= (uint32_t)row[b0 + b] << (8 * (b & 3));
    }
}

// Centroid pairs of a stored byte: entry (byte, copy) = {codebook[byte & mask], codebook[(byte >> 4) & mask]},
// kPairCopies copies side by side (a lane uses copy lane % kPairCopies, which thins out bank conflicts).
constexpr int kPairCopies = 4;

template <int DPL>
__device__ __forceinline__ void decode_row(const uint32_t (&w)[(DPL + 7) / 8], uint32_t pair_lane, float (&v)[DPL]) {
#pragma unroll
    for (int i = 0; i < DPL / 2; ++i) {
        const uint32_t byte = (w[i >> 2] >> (8 * (i & 3))) & 0xFFu;
        float2 c;
        asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];\n" : "=f"(c.x), "=f"(c.y) : "r"(pair_lane + byte * (kPairCopies * 8)));
        v[2 * i] = c.x;
        v[2 * i + 1] = c.y;
    }
}

// A warp fetches the packed words of `kChunk` consecutive tokens before it touches any of them, so
// that the loads are in flight together: 32 tokens when a lane's share of a row is one word,
// fewer for the wide head dims.
template <int DPL>
struct Chunk {
    static constexpr int W = (DPL + 7) / 8;
    static constexpr int kTokens = 32 / W;
    static constexpr int kLevel = W == 1 ? 5 : (W == 2 ? 4 : 3);
};

// Rows past `valid` repeat the last valid row: their scores and weights are masked by the caller.
template <int DPL>
__device__ __forceinline__ void load_chunk(const uint8_t* rows, int row_bytes, int first, int valid, int lane, bool vec,
                                           uint32_t (&w)[Chunk<DPL>::kTokens][Chunk<DPL>::W]) {
#pragma unroll
    for (int t = 0; t < Chunk<DPL>::kTokens; ++t)
        load_row_bytes<DPL>(rows + (uint32_t)(min(first + t, valid - 1) * row_bytes), row_bytes, lane, vec, w[t]);
}

template <int DPL, int G>
struct TileScores {
    using C = Chunk<DPL>;
    const uint8_t* rows;      // first row of the tile
    int row_bytes, valid, lane;
    bool vec;
    uint32_t pair_lane;       // shared address of this lane's copy of the pair table
    const float (*q)[DPL];

    // Sums over the 32 lanes of `1 << L` fetched tokens starting at chunk position t; afterwards
    // lane l holds the token t + (l mod 2^L) in out[].
    template <int L>
    __device__ __forceinline__ void reduce(const uint32_t (&w)[C::kTokens][C::W], int t, float (&out)[G]) const {
        if constexpr (L == 0) {
            float kv[DPL];
            decode_row<DPL>(w[t], pair_lane, kv);
#pragma unroll
            for (int h = 0; h < G; ++h) {
                float s = 0.0f;
#pragma unroll
                for (int i = 0; i < DPL; ++i) s = fmaf(q[h][i], kv[i], s);
                out[h] = s;
            }
        } else {
            float a[G], b[G];
            reduce<L - 1>(w, t, a);
            reduce<L - 1>(w, t + (1 << (L - 1)), b);
            combine<L>(a, b, out);
        }
    }

    template <int L>
    __device__ __forceinline__ void combine(const float (&a)[G], const float (&b)[G], float (&out)[G]) const {
        const bool upper = lane & (1 << (L - 1));
#pragma unroll
        for (int h = 0; h < G; ++h) {
            const float send = upper ? a[h] : b[h];
            const float keep = upper ? b[h] : a[h];
            out[h] = keep + __shfl_xor_sync(kFull, send, 1 << (L - 1));
        }
    }

    // The same over `1 << L` tokens of the tile starting at token t, chunk by chunk.
    template <int L>
    __device__ __forceinline__ void run(int t, float (&out)[G]) const {
        if constexpr (L == C::kLevel) {
            uint32_t w[C::kTokens][C::W];
            load_chunk<DPL>(rows, row_bytes, t, valid, lane, vec, w);
            reduce<L>(w, 0, out);
        } else {
            float a[G], b[G];
            run<L - 1>(t, a);
            run<L - 1>(t + (1 << (L - 1)), b);
            combine<L>(a, b, out);
        }
    }
};

// Workspace of the sliced launches: records of the slices and one arrival counter per (kv head,
// query group); the last slice to arrive puts its counter back to zero.  The one below is part of
// the module, so that the bridge's own entry point allocates nothing: launches that use it have to be
// ordered with respect to each other, which the bridge's single compute stream gives.  Callers with
// several streams bring their own (polarquant_fused_attention_ws_cuda_c): counters in its first
// kWsCounterBytes, records behind them.
constexpr size_t kWsFloats = size_t(1) << 20;
constexpr int kWsTickets = 4096;
constexpr size_t kWsCounterBytes = POLARQUANT_ATTENTION_COUNTER_BYTES;
static_assert(kWsTickets * sizeof(unsigned) <= kWsCounterBytes, "the counters fit their region");
__device__ float g_partials[kWsFloats];
__device__ unsigned g_tickets[kWsTickets];

template <int DPL, int G>
__global__ void __launch_bounds__(kAttWarps * 32, 3) attention_kernel(const AttnParams p) {
    constexpr int DP = 32 * DPL;                      // padded head dim
    constexpr int REC = DP + 2;                       // partial record: m, l, acc[DP]
    __shared__ __align__(16) float2 pair_tab[256 * kPairCopies];
    __shared__ float sm_m[kAttWarps][G], sm_l[kAttWarps][G];
    __shared__ float sm_acc[kAttWarps][G][DP];
    __shared__ unsigned sm_last;

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int split = blockIdx.x, group = blockIdx.y, hkv = blockIdx.z;
    const int hq0 = hkv * p.gqa + group * G;
    const int row_bytes = p.D >> 1;
    const uint32_t mask = (uint32_t)(p.n_levels - 1);
    for (int e = threadIdx.x; e < 256 * kPairCopies; e += blockDim.x) {
        const uint32_t byte = (uint32_t)e / kPairCopies;
        pair_tab[e] = make_float2(p.codebook[byte & mask], p.codebook[(byte >> 4) & mask]);
    }
    __syncthreads();
    const uint32_t pair_lane = (uint32_t)__cvta_generic_to_shared(pair_tab) + (lane % kPairCopies) * 8;

    float q[G][DPL];
#pragma unroll
    for (int h = 0; h < G; ++h)
#pragma unroll
        for (int i = 0; i < DPL; ++i) {
            const int d = lane * DPL + i;
            q[h][i] = d < p.D ? p.q[(size_t)(hq0 + h) * p.D + d] : 0.0f;
        }

    float m[G], l[G], acc[G][DPL];
#pragma unroll
    for (int h = 0; h < G; ++h) {
        m[h] = kLowest;
        l[h] = 0.0f;
#pragma unroll
        for (int i = 0; i < DPL; ++i) acc[h][i] = 0.0f;
    }

    const int n_tiles = (p.S + kTile - 1) / kTile;
    const int tile_lo = split * p.tiles_per_split;
    const int tile_hi = min(n_tiles, tile_lo + p.tiles_per_split);
    const size_t kv_row0 = (size_t)hkv * p.S;
    for (int tile = tile_lo + warp; tile < tile_hi; tile += kAttWarps) {
        const int s0 = tile * kTile;
        const int valid = min(kTile, p.S - s0);
        const float kr = lane < valid ? p.kr[kv_row0 + s0 + lane] : 0.0f;
        const float vr = lane < valid ? p.vr[kv_row0 + s0 + lane] : 0.0f;

        TileScores<DPL, G> ts{p.pk + (kv_row0 + s0) * row_bytes, row_bytes, valid, lane, p.vector_loads != 0,
                              pair_lane, q};
        float sc[G];
        ts.template run<5>(0, sc);

        float w[G];
#pragma unroll
        for (int h = 0; h < G; ++h) {
            const float s = lane < valid ? sc[h] * kr * p.scale : kLowest;
            float tmax = s;
#pragma unroll
            for (int o = 16; o; o >>= 1) tmax = fmaxf(tmax, __shfl_xor_sync(kFull, tmax, o));
            const float m_new = fmaxf(m[h], tmax);
            const float corr = __expf(m[h] - m_new);
            const float pr = lane < valid ? __expf(s - m_new) : 0.0f;
            m[h] = m_new;
            l[h] = l[h] * corr + pr;                   // lane-private share of the denominator
            w[h] = pr * vr;
#pragma unroll
            for (int i = 0; i < DPL; ++i) acc[h][i] *= corr;
        }

        const uint8_t* vrows = p.pv + (kv_row0 + s0) * row_bytes;
        using C = Chunk<DPL>;
#pragma unroll 1
        for (int c0 = 0; c0 < valid; c0 += C::kTokens) {
            uint32_t vw[C::kTokens][C::W];
            load_chunk<DPL>(vrows, row_bytes, c0, valid, lane, p.vector_loads != 0, vw);
#pragma unroll
            for (int t = 0; t < C::kTokens; ++t) {
                float vv[DPL];
                decode_row<DPL>(vw[t], pair_lane, vv);
#pragma unroll
                for (int h = 0; h < G; ++h) {
                    const float wt = __shfl_sync(kFull, w[h], c0 + t);     // 0 for tokens past `valid`
#pragma unroll
                    for (int i = 0; i < DPL; ++i) acc[h][i] = fmaf(wt, vv[i], acc[h][i]);
                }
            }
        }
    }

    // the CTA's four warps -> one (m, l, acc) per head
#pragma unroll
    for (int h = 0; h < G; ++h) {
        float lt = l[h];
#pragma unroll
        for (int o = 16; o; o >>= 1) lt += __shfl_xor_sync(kFull, lt, o);
        if (lane == 0) { sm_m[warp][h] = m[h]; sm_l[warp][h] = lt; }
#pragma unroll
        for (int i = 0; i < DPL; ++i) sm_acc[warp][h][lane * DPL + i] = acc[h][i];
    }
    __syncthreads();

    const bool single = p.n_split == 1;
    for (int e = threadIdx.x; e < G * DP; e += blockDim.x) {
        const int h = e / DP, d = e - h * DP;
        float mm = sm_m[0][h];
#pragma unroll
        for (int wv = 1; wv < kAttWarps; ++wv) mm = fmaxf(mm, sm_m[wv][h]);
        float ll = 0.0f, aa = 0.0f;
#pragma unroll
        for (int wv = 0; wv < kAttWarps; ++wv) {
            const float c = __expf(sm_m[wv][h] - mm);
            ll = fmaf(sm_l[wv][h], c, ll);
            aa = fmaf(sm_acc[wv][h][d], c, aa);
        }
        if (single) {
            if (d < p.D) p.out[(size_t)(hq0 + h) * p.D + d] = ll > 0.0f ? aa / ll : 0.0f;
        } else {
            float* rec = p.partials + ((size_t)(hq0 + h) * p.n_split + split) * REC;
            if (d == 0) { rec[0] = mm; rec[1] = ll; }
            rec[2 + d] = aa;
        }
    }
    if (single) return;

    // the last slice to finish merges the records of its heads
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) {
        const unsigned done = atomicAdd(p.tickets + hkv * gridDim.y + group, 1u);
        sm_last = done == (unsigned)p.n_split - 1;
        if (sm_last) p.tickets[hkv * gridDim.y + group] = 0;
    }
    __syncthreads();
    if (!sm_last) return;
    __threadfence();
    for (int e = threadIdx.x; e < G * DP; e += blockDim.x) {
        const int h = e / DP, d = e - h * DP;
        if (d >= p.D) continue;
        const float* rec = p.partials + (size_t)(hq0 + h) * p.n_split * REC;
        // eight records per round trip to L2: the loads of a round do not depend on each other
        float mm = kLowest, ll = 0.0f, aa = 0.0f;
        for (int s0 = 0; s0 < p.n_split; s0 += 8) {
            float ms[8], ls[8], as[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                const float* r = rec + (size_t)min(s0 + u, p.n_split - 1) * REC;
                ms[u] = __ldcg(r);
                ls[u] = __ldcg(r + 1);
                as[u] = __ldcg(r + 2 + d);
            }
            float m_new = mm;
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                if (s0 + u >= p.n_split) { ms[u] = kLowest; ls[u] = 0.0f; as[u] = 0.0f; }
                m_new = fmaxf(m_new, ms[u]);
            }
            const float c = __expf(mm - m_new);
            ll *= c;
            aa *= c;
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                const float cu = __expf(ms[u] - m_new);
                ll = fmaf(ls[u], cu, ll);
                aa = fmaf(as[u], cu, aa);
            }
            mm = m_new;
        }
        p.out[(size_t)(hq0 + h) * p.D + d] = ll > 0.0f ? aa / ll : 0.0f;
    }
}

// Whether pq_bridge_attn.cu serves the call.  Its CTA has an SM to itself, so very many heads over a tile or two of tokens
// are left to the general kernel, more so while its three CTAs per SM hold all of them (512 kv heads of 64, 33 tokens: 10.8 us,
// general 9.8; of 128 12.0 and 12.5; 320 of 128 9.2 and 7.2).
bool tuned_attention(const AttnParams& p, int total_kv_heads, const void* packed_k, const void* packed_v) {
    const int sms = device_sms();
    const long long little = total_kv_heads <= 2 * sms ? 0 : total_kv_heads <= 3 * sms ? 8192 : 4096;
    return pq::bridge_attention_fits(p.D, packed_k, packed_v) && (long long)p.S * p.D > little;
}

// How a call is cut: which kernel, and over how many slices (p.n_split, p.tiles_per_split).
struct AttnPlan {
    bool tuned;               // pq_bridge_attn.cu
    int DPL, G, groups;       // of the general kernel (DPL, G); groups of either
};
AttnPlan plan_attention(AttnParams& p, bool tuned, int total_q_heads, int total_kv_heads, int sms, size_t ws_floats) {
    AttnPlan a{};
    a.tuned = tuned;
    if (tuned) {
        a.groups = pq::bridge_attention_plan(p, total_kv_heads, sms, ws_floats, kWsTickets, total_q_heads);
        return a;
    }
    a.DPL = 2;
    while (32 * a.DPL < p.D) a.DPL *= 2;
    a.G = 8;
    while (a.G > 1 && (p.gqa % a.G || a.G * a.DPL > 32)) a.G >>= 1;
    a.groups = p.gqa / a.G;
    const int n_tiles = (p.S + kTile - 1) / kTile;
    const int base = total_kv_heads * a.groups;
    // two CTAs per SM with at least two tiles per warp (three CTAs per SM measured slower)
    int n_split = std::max(1, std::min((2 * sms + base - 1) / base, n_tiles / (2 * kAttWarps)));
    int tiles_per_split = (n_tiles + n_split - 1) / n_split;
    n_split = (n_tiles + tiles_per_split - 1) / tiles_per_split;
    if (n_split > 1) {
        const size_t per_split = (size_t)total_q_heads * (32 * a.DPL + 2);
        if (base > kWsTickets || per_split * 2 > ws_floats) {
            n_split = 1;
        } else {
            n_split = (int)std::min<size_t>(n_split, ws_floats / per_split);
        }
        tiles_per_split = (n_tiles + n_split - 1) / n_split;
        n_split = (n_tiles + tiles_per_split - 1) / tiles_per_split;
    }
    p.n_split = n_split;
    p.tiles_per_split = tiles_per_split;
    return a;
}

// The records and counters of a sliced call: the caller's workspace, or the module's own on the current device.
bool workspace(AttnParams& p, void* given) {
    if (given) {
        p.tickets = static_cast<unsigned*>(given);
        p.partials = reinterpret_cast<float*>(static_cast<uint8_t*>(given) + kWsCounterBytes);
        return true;
    }
    if (cudaGetSymbolAddress((void**)&p.partials, g_partials) == cudaSuccess &&
        cudaGetSymbolAddress((void**)&p.tickets, g_tickets) == cudaSuccess)
        return true;
    fail(kErrCuda, "attention: workspace symbol lookup failed");
    cudaGetLastError();
    return false;
}

template <int DPL, int G>
bool launch_attention(const AttnParams& p, dim3 grid, cudaStream_t stream) {
    attention_kernel<DPL, G><<<grid, kAttWarps * 32, 0, stream>>>(p);
    return launched();
}

template <int DPL>
bool dispatch_group(int G, const AttnParams& p, dim3 grid, cudaStream_t stream) {
    if constexpr (DPL * 8 <= 32) if (G == 8) return launch_attention<DPL, 8>(p, grid, stream);
    if constexpr (DPL * 4 <= 32) if (G == 4) return launch_attention<DPL, 4>(p, grid, stream);
    if constexpr (DPL * 2 <= 32) if (G == 2) return launch_attention<DPL, 2>(p, grid, stream);
    return launch_attention<DPL, 1>(p, grid, stream);
}

// Built-in tables of the bridge (patch 985-1003): centroids for head dim 128.
const float kCodebook4[16] = {-0.1547f, -0.1175f, -0.0928f, -0.0722f, -0.0537f, -0.0363f, -0.0193f, -0.0024f,
                              0.0145f,  0.0318f,  0.0498f,  0.0692f,  0.0907f,  0.1157f,  0.1467f,  0.1947f};
const float kCodebook3[8] = {-0.1350f, -0.0820f, -0.0440f, -0.0110f, 0.0220f, 0.0560f, 0.0950f, 0.1500f};
const float kCodebook2[4] = {-0.1050f, -0.0280f, 0.0400f, 0.1200f};

// Uniform(-1, 1) entries from the C library generator, rows orthonormalised in order
// (patch 556-579).
void seeded_rotation(float* R, int D, int seed) {
    srand(seed);
    for (int i = 0; i < D * D; ++i) R[i] = ((float)rand() / RAND_MAX) * 2.0f - 1.0f;
    for (int i = 0; i < D; ++i) {
        float* ri = R + (size_t)i * D;
        for (int j = 0; j < i; ++j) {
            const float* rj = R + (size_t)j * D;
            float dot = 0.0f;
            for (int k = 0; k < D; ++k) dot += ri[k] * rj[k];
            for (int k = 0; k < D; ++k) ri[k] -= dot * rj[k];
        }
        float nn = 0.0f;
        for (int k = 0; k < D; ++k) nn += ri[k] * ri[k];
        nn = sqrtf(nn);
        if (nn > 1e-10f)
            for (int k = 0; k < D; ++k) ri[k] /= nn;
    }
}

}  // namespace

extern "C" {

int polarquant_last_error_c(void) {
    const int e = t_last_error;
    t_last_error = 0;
    return e;
}

void polarquant_rotate_query_cuda_c(const float* q_input, const float* rotation, float* q_rotated,
                                    int total_q_heads, int D, void* stream) {
    if (total_q_heads <= 0 || D <= 0) return;
    if (!q_input || !rotation || !q_rotated) { fail(kErrNull, "rotate_query: NULL pointer"); return; }
    if (D > kMaxDim) { fail(kErrDim, "rotate_query: head dim above 1024"); return; }
    rotate_rows_kernel<<<total_q_heads, 512, 0, (cudaStream_t)stream>>>(q_input, rotation, q_rotated, D);
    launched();
}

void polarquant_inverse_rotate_cuda_c(const float* input, const float* rotation, float* output,
                                      int total_q_heads, int D, void* stream) {
    if (total_q_heads <= 0 || D <= 0) return;
    if (!input || !rotation || !output) { fail(kErrNull, "inverse_rotate: NULL pointer"); return; }
    if (D > kMaxDim) { fail(kErrDim, "inverse_rotate: head dim above 1024"); return; }
    cudaStream_t st = (cudaStream_t)stream;
    const int blocks = (D + 127) / 128;
    if (input == output || total_q_heads > device_sms() * 4 / 3)
        inverse_rotate_rows_kernel<<<total_q_heads, 256, 0, st>>>(input, rotation, output, D);
    else if (D <= 64)
        inverse_rotate_split_kernel<64, 16><<<total_q_heads, dim3(64, 16), 0, st>>>(input, rotation, output, D);
    else
        inverse_rotate_split_kernel<128, 8><<<dim3(total_q_heads, blocks), dim3(128, 8), 0, st>>>(input, rotation, output, D);
    launched();
}

void polarquant_compress_cuda_c(const float* input, const float* rotation, const float* codebook,
                                float* radius_out, uint8_t* packed_out,
                                int N, int D, int n_levels, void* stream) {
    if (N <= 0 || D <= 0) return;
    if (!input || !rotation || !codebook || !radius_out || !packed_out) { fail(kErrNull, "compress: NULL pointer"); return; }
    if (!dim_ok(D)) { fail(kErrDim, "compress: head dim must be even and at most 1024"); return; }
    if (n_levels < 1 || n_levels > 16) { fail(kErrLevels, "compress: n_levels outside [1, 16]"); return; }
    cudaStream_t st = (cudaStream_t)stream;
    // The shared-memory transpose of R costs 13 us per launch (7 at D = 64); below a few thousand vectors the kernel that
    // streams R from L2 finishes first.
    if ((D == 64 || D == 128) && N >= kCmpMin) {
        const int sms = device_sms();
        const int wave = (D == 64 ? 4 : 2) * sms;
        cudaError_t e;
        if (N > wave * kCmpWarps * kCmpVecs && pq::bridge_compress_fits(D, input, rotation, packed_out)) {
            e = pq::bridge_compress_launch(input, rotation, codebook, radius_out, packed_out, N, D, n_levels, sms, st);
        } else {
            const int ctas = std::min(((N + kCmpVecs - 1) / kCmpVecs + kCmpWarps - 1) / kCmpWarps, wave);
            e = D == 64 ? launch_compress<64>(ctas, input, rotation, codebook, radius_out, packed_out, N, n_levels, st)
                        : launch_compress<128>(ctas, input, rotation, codebook, radius_out, packed_out, N, n_levels, st);
        }
        if (e != cudaSuccess) fail(kErrCuda, cudaGetErrorString(e));
        return;
    }
    if (N < kCmpFour)
        compress_any_dim_kernel<1><<<N, kSmallWarps * 32, 0, st>>>(input, rotation, codebook, radius_out, packed_out, N, D, n_levels);
    else
        compress_any_dim_kernel<4><<<(N + 3) / 4, kSmallWarps * 32, 0, st>>>(input, rotation, codebook, radius_out, packed_out, N, D, n_levels);
    launched();
}

size_t polarquant_fused_attention_ws_bytes_c(int total_q_heads, int total_kv_heads, int S, int D) {
    if (total_q_heads <= 0 || total_kv_heads <= 0 || total_q_heads % total_kv_heads || S <= 0 || !dim_ok(D)) return 0;
    size_t floats = 0;
    for (const bool tuned : {false, true}) {                   // which of the two depends on the buffers' alignment
        AttnParams p{};
        p.gqa = total_q_heads / total_kv_heads; p.S = S; p.D = D;
        if (tuned && !tuned_attention(p, total_kv_heads, nullptr, nullptr)) continue;
        const AttnPlan a = plan_attention(p, tuned, total_q_heads, total_kv_heads, device_sms(), kWsFloats);
        if (p.n_split > 1) floats = std::max(floats, (size_t)p.n_split * total_q_heads * ((tuned ? D : 32 * a.DPL) + 2));
    }
    return floats ? kWsCounterBytes + floats * sizeof(float) : 0;
}

void polarquant_fused_attention_ws_cuda_c(const float* q_rotated, const uint8_t* packed_k,
                                          const float* k_radius, const uint8_t* packed_v,
                                          const float* v_radius, const float* codebook, float* output,
                                          int total_q_heads, int total_kv_heads,
                                          int S, int D, int n_levels, float scale,
                                          void* ws, size_t ws_bytes, void* stream) {
    if (total_q_heads <= 0 || S <= 0 || D <= 0) return;
    if (!q_rotated || !packed_k || !k_radius || !packed_v || !v_radius || !codebook || !output) {
        fail(kErrNull, "attention: NULL pointer");
        return;
    }
    if (!dim_ok(D)) { fail(kErrDim, "attention: head dim must be even and at most 1024"); return; }
    if (n_levels < 1 || n_levels > 16) { fail(kErrLevels, "attention: n_levels outside [1, 16]"); return; }
    if (total_kv_heads <= 0 || total_q_heads % total_kv_heads) {
        fail(kErrHeads, "attention: total_q_heads is not a multiple of total_kv_heads");
        return;
    }
    cudaStream_t st = (cudaStream_t)stream;
    AttnParams p{};
    p.q = q_rotated; p.pk = packed_k; p.kr = k_radius; p.pv = packed_v; p.vr = v_radius;
    p.codebook = codebook; p.out = output;
    p.gqa = total_q_heads / total_kv_heads; p.S = S; p.D = D; p.n_levels = n_levels; p.scale = scale;

    // Head dims 64 and 128 on 16-byte boundaries (the bridge's own buffers are) have a kernel of their own.  It masks
    // indices with n_levels - 1 like the general one, so other table sizes than powers of two behave alike.
    const bool tuned = tuned_attention(p, total_kv_heads, packed_k, packed_v) && (reinterpret_cast<uintptr_t>(q_rotated) & 7) == 0;
    size_t floats = kWsFloats;
    if (ws) floats = ws_bytes <= kWsCounterBytes ? 0 : std::min(kWsFloats, (ws_bytes - kWsCounterBytes) / sizeof(float));
    const AttnPlan a = plan_attention(p, tuned, total_q_heads, total_kv_heads, device_sms(), floats);
    if (p.n_split > 1 && !workspace(p, ws)) return;
    if (tuned) {
        const cudaError_t e = pq::bridge_attention_launch(p, total_kv_heads, a.groups, st);
        if (e != cudaSuccess) fail(kErrCuda, cudaGetErrorString(e));
        return;
    }
    const int bpl = a.DPL / 2;
    p.vector_loads = ((D / 2) % bpl == 0) && (reinterpret_cast<uintptr_t>(packed_k) % bpl == 0) &&
                     (reinterpret_cast<uintptr_t>(packed_v) % bpl == 0);
    const dim3 grid(p.n_split, a.groups, total_kv_heads);
    switch (a.DPL) {
        case 2:  dispatch_group<2>(a.G, p, grid, st); break;
        case 4:  dispatch_group<4>(a.G, p, grid, st); break;
        case 8:  dispatch_group<8>(a.G, p, grid, st); break;
        case 16: dispatch_group<16>(a.G, p, grid, st); break;
        default: dispatch_group<32>(a.G, p, grid, st); break;
    }
}

void polarquant_fused_attention_cuda_c(const float* q_rotated, const uint8_t* packed_k,
                                       const float* k_radius, const uint8_t* packed_v,
                                       const float* v_radius, const float* codebook, float* output,
                                       int total_q_heads, int total_kv_heads,
                                       int S, int D, int n_levels, float scale, void* stream) {
    polarquant_fused_attention_ws_cuda_c(q_rotated, packed_k, k_radius, packed_v, v_radius, codebook, output, total_q_heads,
                                         total_kv_heads, S, D, n_levels, scale, nullptr, 0, stream);
}

struct polarquant_state* polarquant_init_c(int head_dim, int n_kv_heads, int n_q_heads,
                                           int n_layers, int n_kv_max, int n_bits) {
    if (head_dim <= 0 || (head_dim & 1) || head_dim > kMaxDim || n_kv_heads <= 0 || n_layers < 0 || n_kv_max <= 0) {
        fail(kErrDim, "init: bad shape");
        return nullptr;
    }
    const float* cb_host = kCodebook4;
    if (n_bits == 3) cb_host = kCodebook3;
    else if (n_bits == 2) cb_host = kCodebook2;
    else if (n_bits != 4) {
        fprintf(stderr, "PolarQuant: unsupported n_bits=%d, using 4\n", n_bits);
        n_bits = 4;
    }
    polarquant_state* st = new polarquant_state();
    st->enabled = true;
    st->n_bits = n_bits;
    st->n_levels = 1 << n_bits;
    st->head_dim = head_dim;
    st->n_kv_heads = n_kv_heads;
    st->n_q_heads = n_q_heads;
    st->n_layers = n_layers;
    st->n_kv_max = n_kv_max;
    st->codebook = nullptr;
    st->rotation = nullptr;
    st->layers = new polarquant_kv_layer[n_layers > 0 ? n_layers : 1]();

    bool ok = cudaMalloc(&st->codebook, st->n_levels * sizeof(float)) == cudaSuccess &&
              cudaMemcpy(st->codebook, cb_host, st->n_levels * sizeof(float), cudaMemcpyHostToDevice) == cudaSuccess;
    if (ok) {
        float* R = new float[(size_t)head_dim * head_dim];
        seeded_rotation(R, head_dim, 42);
        const size_t bytes = (size_t)head_dim * head_dim * sizeof(float);
        ok = cudaMalloc(&st->rotation, bytes) == cudaSuccess &&
             cudaMemcpy(st->rotation, R, bytes, cudaMemcpyHostToDevice) == cudaSuccess;
        delete[] R;
    }
    const size_t packed_bytes = (size_t)n_kv_heads * n_kv_max * (head_dim / 2);
    const size_t radius_bytes = (size_t)n_kv_heads * n_kv_max * sizeof(float);
    for (int l = 0; ok && l < n_layers; ++l) {
        polarquant_kv_layer& L = st->layers[l];
        ok = cudaMalloc(&L.k_packed, packed_bytes) == cudaSuccess && cudaMalloc(&L.k_radius, radius_bytes) == cudaSuccess &&
             cudaMalloc(&L.v_packed, packed_bytes) == cudaSuccess && cudaMalloc(&L.v_radius, radius_bytes) == cudaSuccess &&
             cudaMemset(L.k_packed, 0, packed_bytes) == cudaSuccess && cudaMemset(L.k_radius, 0, radius_bytes) == cudaSuccess &&
             cudaMemset(L.v_packed, 0, packed_bytes) == cudaSuccess && cudaMemset(L.v_radius, 0, radius_bytes) == cudaSuccess;
    }
    if (!ok) {
        cudaGetLastError();
        fail(kErrCuda, "init: device allocation failed");
        polarquant_free_c(st);
        return nullptr;
    }
    const double compressed = 2.0 * n_layers * (double)n_kv_heads * n_kv_max * (head_dim / 2 + sizeof(float));
    const double original = 2.0 * n_layers * (double)n_kv_heads * n_kv_max * head_dim * sizeof(float);
    fprintf(stderr, "PolarQuant-KV initialized: head_dim=%d n_kv_heads=%d n_q_heads=%d n_layers=%d n_bits=%d n_kv_max=%d; "
                    "compressed cache %.2f MB (fp32 %.2f MB, %.1fx)\n",
            head_dim, n_kv_heads, n_q_heads, n_layers, n_bits, n_kv_max, compressed / 1048576.0, original / 1048576.0,
            compressed > 0 ? original / compressed : 0.0);
    return st;
}

void polarquant_free_c(struct polarquant_state* state) {
    if (!state) return;
    if (state->codebook) cudaFree(state->codebook);
    if (state->rotation) cudaFree(state->rotation);
    if (state->layers) {
        for (int l = 0; l < state->n_layers; ++l) {
            polarquant_kv_layer& L = state->layers[l];
            if (L.k_packed) cudaFree(L.k_packed);
            if (L.k_radius) cudaFree(L.k_radius);
            if (L.v_packed) cudaFree(L.v_packed);
            if (L.v_radius) cudaFree(L.v_radius);
        }
        delete[] state->layers;
    }
    delete state;
}

}  // extern "C"
