// pq_dequant: stored block_pq4 blocks -> centroid[idx] * float(d) (rotated space) -> inverse rotation v @ R -> float32
// or float16.
//
// Follows dequantize_with_codebook (src/polarquant_kv_cuda/lloyd_max.py:93-98), the radius restore of
// quantizer.decompress (python/polarquant_kv/quantizer.py:151) and inverse_rotate (python/polarquant_kv/rotation.py:61);
// the float16 output is clamped to +-65504 like decompress_gpu (src/polarquant_kv_cuda/decompress_kernel.py:47-51).
//
// The inverse rotation is a [vectors x D] . [D x D] contraction on the 5th-generation tensor cores (tcgen05.mma kind::f16,
// M = 128) with both operands as two float16 terms and three product terms (lo*hi, hi*lo, then hi*hi into the same
// float32 accumulator), which keeps float32-level accuracy (2e-6 of a vector's largest component).
//
// Bound: HBM, 72 bytes in and 256 or 512 out per vector of 128 (4-bit).  A persistent CTA owns 128 vectors at a time:
//   copy warp     the tile's stored bytes (contiguous), by bulk copy, four tiles in flight (the last one, if partial, by
//                 4-byte asynchronous copies);
//   worker warps  (4 per 32-dim block) a thread owns one vector x one block: a stored byte is one lookup of its centroids'
//                 hi and lo float16 terms (256-byte table rows at a fixed shared address, 16 private copies, so a byte
//                 becomes an address with one byte-permute and lookups never conflict), times the radius as an error-free
//                 float16 product (hi = h x d, lo = l x d + (h x d - hi)), and goes into tensor memory as the A operand
//                 (two buffers) - nothing is staged through shared memory;
//   MMA warp      3 x D/16 MMAs per tile (1.5 K cycles at D = 128; HBM needs 1.8 K for the float16 output);
//   the same worker warps, one tile behind, read their vector's 32 accumulator columns, scale, and send the results off
//                 through swizzled shared memory by TMA (stores straight from the threads, one vector's 32 bytes per lane,
//                 took two thirds of the load-store pipe: 136 us against 118).
// A power of two per vector keeps the largest radius in [1, 2) inside, so tiny vectors keep their precision.
// Error against 64 bits: 4e-8 of a vector's largest component rms, 7e-7 at most over 400 000 vectors (8e-8 and 2e-6 with
// float32 products split afterwards and the cross term in an accumulator of its own).
// Measured: 2^20 vectors of 128 at 4 bits to float16 118 us (181 with operands staged through shared memory).
// All waits are bounded (a lost completion sets an error flag instead of hanging).
#include <atomic>

#include "pq_common.cuh"
#include "pq_tcgen05.cuh"

namespace pq {

constexpr int kDqVecs = 128;
constexpr float kDqCbScale = 64.0f;          // centroids sit x64 in the table (keeps the lo terms normal)

// bit 0: a bounded wait gave up; bit 1: shared-memory window unusable (pq_poll_device_errors, bits 6 and 12 there)
static __device__ unsigned int g_dequant_error = 0;

struct DequantParams {
    const uint8_t* blocks;
    const float* rot;
    void* out;
    int64_t n_vec;
    int64_t n_items;             // tiles of 128 vectors
    int out_is_fp16;
    float cb[16];
};

template <int D>
struct DequantCfg {
    static constexpr int NBLK = D / 32;
    static constexpr int kWorkers = 128 * NBLK;                   // one thread per (vector, block)
    static constexpr int kThreads = kWorkers + 64;                // + MMA warp + copy warp
    static constexpr int kRing = 4;                               // tiles of stored bytes in flight or in use
    static constexpr uint32_t kSlot = kDqVecs * NBLK * 18;        // stored bytes of a tile at 4 bits
    // [window start: ring, barriers][0x10000: table rows of 256 bytes, their upper halves hold the core matrices of R_hi]
    // [0x20000: R_lo][results on their way out]
    static constexpr uint32_t kTabAddr = 0x10000u, kBLoAddr = 0x20000u, kBTerm = 2u * D * D;
    static constexpr uint32_t kOutAddr = kBLoAddr + kBTerm, kOutBytes = kDqVecs * D * 4;
    static constexpr uint32_t kLow = kRing * kSlot + 256 + 128;
    static constexpr size_t smem_bytes() { return (size_t)kOutAddr + kOutBytes; }
    static constexpr uint32_t kTmemCols = 4 * D;                  // A 2 x D, accumulators 2 x D
};

__device__ __forceinline__ void dq_tmem_st16(uint32_t taddr, const uint32_t (&v)[16]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};\n" ::"r"(taddr),
                 "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]),
                 "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15])
                 : "memory");
}
// Two float16 terms of (h + l) x d per half: the product h x d is split without error.
__device__ __forceinline__ void dq_scaled(uint32_t h, uint32_t l, __half2 d, uint32_t& hi, uint32_t& lo) {
    const __half2 H = *reinterpret_cast<const __half2*>(&h), L = *reinterpret_cast<const __half2*>(&l);
    const __half2 p = __hmul2(H, d);
    const __half2 q = __hfma2(L, d, __hfma2(H, d, __hneg2(p)));
    hi = *reinterpret_cast<const uint32_t*>(&p);
    lo = *reinterpret_cast<const uint32_t*>(&q);
}
__device__ __forceinline__ uint32_t dq_lds_u16(uint32_t a) {
    uint32_t v;
    asm volatile("{ .reg .u16 t; ld.shared.u16 t, [%1]; cvt.u32.u16 %0, t; }\n" : "=r"(v) : "r"(a));
    return v;
}
// float16 bits: the larger of m and |x|, NaN if either is
__device__ __forceinline__ unsigned short dq_max_abs(unsigned short m, uint32_t x) {
    asm("{ .reg .f16 a; abs.f16 a, %1; max.NaN.f16 %0, %0, a; }\n" : "+h"(m) : "h"((unsigned short)x));
    return m;
}
__device__ __forceinline__ uint32_t dq_lds_u32(uint32_t a) {
    uint32_t v;
    asm volatile("ld.shared.u32 %0, [%1];\n" : "=r"(v) : "r"(a));
    return v;
}
// pack two floats as float16, values outside the range clamped to +-65504
__device__ __forceinline__ uint32_t dq_pack_sat(float lo, float hi) {
    uint32_t w;
    asm("cvt.rn.satfinite.f16x2.f32 %0, %1, %2;\n" : "=r"(w) : "f"(hi), "f"(lo));
    return w;
}
__device__ __forceinline__ float2 dq_mul2(float2 a, float2 b) {
    float2 d;
    asm("mul.rn.f32x2 %0, %1, %2;\n"
        : "=l"(*reinterpret_cast<unsigned long long*>(&d))
        : "l"(*reinterpret_cast<unsigned long long*>(&a)), "l"(*reinterpret_cast<unsigned long long*>(&b)));
    return d;
}
__device__ __forceinline__ void dq_sts4(uint32_t a, uint32_t x, uint32_t y, uint32_t z, uint32_t w) {
    asm volatile("st.shared.v4.u32 [%0], {%1,%2,%3,%4};\n" ::"r"(a), "r"(x), "r"(y), "r"(z), "r"(w) : "memory");
}

template <int D, int BITS>
__global__ void __launch_bounds__(DequantCfg<D>::kThreads, 1) pq_dequant_kernel(const DequantParams p, const __grid_constant__ CUtensorMap out_map) {
    using C = DequantCfg<D>;
    constexpr int NBLK = C::NBLK, WORKERS = C::kWorkers, RING = C::kRing;
    constexpr int BB = block_bytes(BITS), VB = NBLK * BB;
    extern __shared__ __align__(128) uint8_t smem_raw[];
    const uint32_t base = (sm_addr(smem_raw) + 127u) & ~127u;
    uint8_t* zero = smem_raw - sm_addr(smem_raw);                  // generic address of shared address 0
    if (base + C::kLow > C::kTabAddr) {
        if (threadIdx.x == 0) atomicOr(&g_dequant_error, 2u);
        return;
    }
    const uint32_t ring = base;
    uint64_t* mbar = reinterpret_cast<uint64_t*>(zero + base + RING * C::kSlot);
    // stored bytes landed / read, per ring slot; A buffer written; its MMAs done (A free, accumulator complete);
    // accumulator read out
    uint64_t *in_full = mbar, *in_free = mbar + RING, *a_full = mbar + 2 * RING, *mma_done = a_full + 2, *acc_free = a_full + 4;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(a_full + 6);
    volatile uint32_t* abort_s = tmem_slot + 1;
    uint32_t* cs = tmem_slot + 4;                                  // 16 split centroids
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;

    // ---- set-up
    if (tid == 0) {
        for (int i = 0; i < RING; ++i) {
            mbar_init(sm_addr(in_full + i), 32);                   // every lane of the copy warp
            mbar_init(sm_addr(in_free + i), WORKERS);
        }
        for (int i = 0; i < 2; ++i) {
            mbar_init(sm_addr(a_full + i), WORKERS);
            mbar_init(sm_addr(mma_done + i), 1);
            mbar_init(sm_addr(acc_free + i), WORKERS);
        }
        *abort_s = 0u;
    }
    if (tid < 16) {
        __half h, l;
        split_half(p.cb[tid] * kDqCbScale, h, l);
        cs[tid] = (uint32_t)__half_as_ushort(h) | ((uint32_t)__half_as_ushort(l) << 16);
    }
    // B terms, K-major core matrices: B[n][k] = 4096 R[k][n]  (out[v][n] = sum_k x[v][k] R[k][n]); lanes along n
    for (int e = tid; e < D * (D / 8); e += C::kThreads) {
        const int n = e % D, kc = e / D;
        uint32_t h[4], l[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const float x0 = __ldg(p.rot + (size_t)(kc * 8 + 2 * u) * D + n) * 4096.f;
            const float x1 = __ldg(p.rot + (size_t)(kc * 8 + 2 * u + 1) * D + n) * 4096.f;
            const __half2 hh = __floats2half2_rn(x0, x1);
            const float2 f = __half22float2(hh);
            h[u] = *reinterpret_cast<const uint32_t*>(&hh);
            l[u] = pack_half2(x0 - f.x, x1 - f.y);
        }
        const uint32_t m = (uint32_t)(kc * (D / 8) + (n >> 3)), in = (uint32_t)(n & 7) * 16;     // core matrix, row
        *reinterpret_cast<uint4*>(zero + C::kTabAddr + m * 256 + 128 + in) = make_uint4(h[0], h[1], h[2], h[3]);
        *reinterpret_cast<uint4*>(zero + C::kBLoAddr + m * 128 + in) = make_uint4(l[0], l[1], l[2], l[3]);
    }
    if (warp == 0) tmem_alloc(sm_addr(tmem_slot), C::kTmemCols);
    __syncthreads();
    // table: row r (256 bytes) = the centroid pairs of byte r, {hi pair, lo pair}
    if (BITS == 4) {
        for (int e = tid; e < 256 * 16; e += C::kThreads) {
            const int b = e >> 4;
            const uint32_t c0 = cs[b & 15], c1 = cs[b >> 4];
            *reinterpret_cast<uint2*>(zero + C::kTabAddr + b * 256 + (e & 15) * 8) =
                make_uint2(__byte_perm(c0, c1, 0x5410), __byte_perm(c0, c1, 0x7632));
        }
    } else {
        for (int e = tid; e < 256 * 8; e += C::kThreads) {
            const int b = e >> 3;
            const uint32_t c0 = cs[b & 3], c1 = cs[(b >> 2) & 3], c2 = cs[(b >> 4) & 3], c3 = cs[b >> 6];
            *reinterpret_cast<uint4*>(zero + C::kTabAddr + b * 256 + (e & 7) * 16) =
                make_uint4(__byte_perm(c0, c1, 0x5410), __byte_perm(c0, c1, 0x7632),
                           __byte_perm(c2, c3, 0x5410), __byte_perm(c2, c3, 0x7632));
        }
    }
    fence_async_smem();                                            // B is read by the tensor core through the async proxy
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    const int n_my = (int)((p.n_items - blockIdx.x + gridDim.x - 1) / gridDim.x);
    bool ok = true;
    // first vector of the i-th tile of this CTA
    auto first = [&](int i) -> int64_t { return ((int64_t)blockIdx.x + (int64_t)i * gridDim.x) * kDqVecs; };

    if (warp == WORKERS / 32) {
        // ---- MMA warp: every lane runs the loop, lane 0 issues
        constexpr uint32_t idesc = umma_idesc_f16(D);
        // no swizzle; core matrices 256 B apart (R_hi, between the table rows) or 128 B (R_lo), K chunks D / 8 of them
        constexpr uint32_t hi_step = (D / 8) * 256, lo_step = (D / 8) * 128;
        constexpr uint32_t hi_d = (256u >> 4) | (1u << 14), lo_d = (128u >> 4) | (1u << 14);
        const uint32_t hi0 = (((C::kTabAddr + 128) >> 4) & 0x3FFFu) | ((hi_step >> 4) << 16);
        const uint32_t lo0 = ((C::kBLoAddr >> 4) & 0x3FFFu) | ((lo_step >> 4) << 16);
        const uint32_t issue = lane == 0 ? 1u : 0u;
        for (int i = 0; i < n_my && ok; ++i) {
            const uint32_t b = i & 1, use = (uint32_t)i >> 1;
            ok = mbar_wait(sm_addr(a_full + b), use & 1u, abort_s, 32) && ok;
            if (i >= 2) ok = mbar_wait(sm_addr(acc_free + b), (use - 1u) & 1u, abort_s, 32) && ok;
            if (!ok) break;
            tc_fence_after();
            const uint32_t a = tmem_base + b * D, acc = tmem_base + 2 * D + b * D;
#pragma unroll
            for (int t = 0; t < 3; ++t)                            // lo x hi, hi x lo, hi x hi
#pragma unroll
                for (int ks = 0; ks < D / 16; ++ks)
                    umma_f16_ts_pred(acc, a + (t == 0 ? D / 2 : 0) + ks * 8,
                                     t == 1 ? lo0 + ((2 * ks * lo_step) >> 4) : hi0 + ((2 * ks * hi_step) >> 4),
                                     t == 1 ? lo_d : hi_d, idesc, (t || ks) ? 1u : 0u, issue);
            umma_commit_pred(sm_addr(mma_done + b), issue);
            __syncwarp();
        }
    } else if (warp == WORKERS / 32 + 1) {
        // ---- copy warp
        int slot = 0;
        uint32_t round = 0;
        for (int i = 0; i < n_my && ok; ++i) {
            if (round) ok = mbar_wait(sm_addr(in_free + slot), (round - 1u) & 1u, abort_s, 32) && ok;
            if (!ok) break;
            const int64_t v0 = first(i);
            const int n = (int)min((int64_t)kDqVecs, p.n_vec - v0);
            const uint8_t* src = p.blocks + v0 * VB;
            const uint32_t dst = ring + slot * C::kSlot, bar = sm_addr(in_full + slot);
            if (n == kDqVecs) {
                if (lane == 0) {
                    mbar_expect_tx(bar, kDqVecs * VB);
                    bulk_load(dst, src, kDqVecs * VB, bar);
                } else {
                    mbar_arrive(bar);
                }
            } else {
                // 4-byte asynchronous copies (vectors are multiples of 4 bytes); the barrier counts every lane's
                for (int c = lane; c < n * VB / 4; c += 32)
                    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(dst + 4 * c), "l"(src + 4 * c));
                asm volatile("cp.async.mbarrier.arrive.noinc.shared.b64 [%0];\n" ::"r"(bar) : "memory");
            }
            __syncwarp();
            if (++slot == RING) { slot = 0; ++round; }
        }
    } else {
        // ---- workers: vector `row` of the tile (= TMEM lane), block `wg`
        const int wg = warp >> 2, q = warp & 3, row = 32 * q + lane;
        const uint32_t tmem_lane = tmem_base + ((uint32_t)(32 * q) << 16);
        const uint32_t tab_lane = C::kTabAddr | (BITS == 4 ? (lane & 15) * 8 : (lane & 7) * 16);
        float scale = 0.f;                                         // of the tile produced last
        auto produce = [&](int i) {
            const int slot = i % RING;
            ok = mbar_wait(sm_addr(in_full + slot), (uint32_t)(i / RING) & 1u, abort_s) && ok;
            const uint32_t vec = ring + slot * C::kSlot + row * VB, blk = vec + wg * BB;
            uint32_t words[BITS], dbits;
            unsigned short dmax = 0;
            {
                uint32_t w[BITS + 1];
                const uint32_t a = blk & ~3u;
#pragma unroll
                for (int k = 0; k <= BITS; ++k) w[k] = dq_lds_u32(a + 4 * k);
                if (wg & 1) {                                      // the block starts in the upper half of a word
                    dbits = w[0] >> 16;
#pragma unroll
                    for (int k = 0; k < BITS; ++k) words[k] = w[k + 1];
                } else {
                    dbits = w[0] & 0xFFFFu;
#pragma unroll
                    for (int k = 0; k < BITS; ++k) words[k] = __funnelshift_r(w[k], w[k + 1], 16);
                }
            }
#pragma unroll
            for (int j = 0; j < NBLK; ++j) dmax = dq_max_abs(dmax, dq_lds_u16(vec + j * BB));
            mbar_arrive(sm_addr(in_free + slot));
            // largest radius -> [1, 2)
            const uint32_t be = __float_as_uint(__half2float(__ushort_as_half(dmax))) >> 23;
            const bool normal = be > 0 && be < 255;
            scale = normal ? __uint_as_float(be << 23) : be ? __int_as_float(0x7FFFFFFF) : 1.0f;      // NaN: no finite vector
            const float ds = __half2float(__ushort_as_half((unsigned short)dbits)) * (normal ? __uint_as_float((254u - be) << 23) : 1.0f);
            const __half2 d2 = __float2half2_rn(ds);               // exact but for radii 2^-14 below the largest
            uint32_t hi[16], lo[16];
#pragma unroll
            for (int k = 0; k < BITS; ++k)
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const uint32_t a = __byte_perm(words[k], tab_lane, 0x7604u | (j << 4));
                    if (BITS == 4) {
                        uint32_t h, l;
                        asm volatile("ld.shared.v2.u32 {%0,%1}, [%2];\n" : "=r"(h), "=r"(l) : "r"(a));
                        dq_scaled(h, l, d2, hi[4 * k + j], lo[4 * k + j]);
                    } else {
                        uint32_t h0, l0, h1, l1;
                        asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];\n" : "=r"(h0), "=r"(l0), "=r"(h1), "=r"(l1) : "r"(a));
                        dq_scaled(h0, l0, d2, hi[8 * k + 2 * j], lo[8 * k + 2 * j]);
                        dq_scaled(h1, l1, d2, hi[8 * k + 2 * j + 1], lo[8 * k + 2 * j + 1]);
                    }
                }
            const uint32_t b = i & 1;
            if (i >= 2) {                                          // the A buffer's MMAs (tile i - 2) are done
                ok = mbar_wait(sm_addr(mma_done + b), (uint32_t)((i >> 1) - 1) & 1u, abort_s) && ok;
                tc_fence_after();
            }
            dq_tmem_st16(tmem_lane + b * D + wg * 16, hi);
            dq_tmem_st16(tmem_lane + b * D + D / 2 + wg * 16, lo);
            asm volatile("tcgen05.wait::st.sync.aligned;\n" ::: "memory");
            tc_fence_before();
            mbar_arrive(sm_addr(a_full + b));
        };
        auto epilogue = [&](int i, float sc) {                     // (every thread of the warp runs all of it)
            const uint32_t b = i & 1;
            ok = mbar_wait(sm_addr(mma_done + b), (uint32_t)(i >> 1) & 1u, abort_s) && ok;
            tc_fence_after();
            float2 v[16];
            tmem_ld32(v, tmem_lane + 2 * D + b * D + wg * 32);
            tc_fence_before();
            mbar_arrive(sm_addr(acc_free + b));
            const float s = sc * (1.0f / (kDqCbScale * 4096.f));
            float2 s2 = make_float2(s, s);
            const int64_t v0 = first(i) + 32 * q;
            // 32 vectors: rows of 128 bytes, 16-byte chunks swizzled as the tensor map says
            if (p.out_is_fp16) {
                // 64 dims = rows of 128 bytes, shared by two warps (boxes of 64-byte rows are limited by the number of
                // rows a TMA unit stores)
                const uint32_t piece = C::kOutAddr + b * (C::kOutBytes / 2) + (uint32_t)((wg >> 1) * kDqVecs + 32 * q) * 128;
                const bool leader = !(wg & 1) && lane == 0;
                if (s != s) {                                  // clamped like a value below the range
#pragma unroll
                    for (int k = 0; k < 16; ++k) v[k] = make_float2(-65504.f, -65504.f);
                    s2 = make_float2(1.f, 1.f);
                }
                const uint32_t bar = 1u + (uint32_t)(q * (D / 64) + (wg >> 1));
                // (the pair's barrier of the tile in between orders this wait before the partner's writes too)
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    uint32_t w[4];
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        const float2 x = dq_mul2(v[4 * c + u], s2);
                        w[u] = dq_pack_sat(x.x, x.y);
                    }
                    dq_sts4(piece + lane * 128 + ((((wg & 1) * 4 + c) ^ (lane & 7)) << 4), w[0], w[1], w[2], w[3]);
                }
                fence_async_smem();
                if (leader) bulk_wait_read();                  // the store of the other buffer: free for the next tile
                asm volatile("bar.sync %0, 64;\n" ::"r"(bar) : "memory");
                if (leader && v0 < p.n_vec) tma_store_2d(&out_map, (wg >> 1) * 64, (int)v0, piece);
            } else {
                const uint32_t piece = C::kOutAddr + (uint32_t)(wg * kDqVecs + 32 * q) * 128;
                if (lane == 0) bulk_wait_read();
                __syncwarp();
#pragma unroll
                for (int c = 0; c < 8; ++c) {
                    const float2 x = dq_mul2(v[2 * c], s2), y = dq_mul2(v[2 * c + 1], s2);
                    dq_sts4(piece + lane * 128 + ((c ^ (lane & 7)) << 4), __float_as_uint(x.x), __float_as_uint(x.y),
                            __float_as_uint(y.x), __float_as_uint(y.y));
                }
                fence_async_smem();
                __syncwarp();
                if (lane == 0 && v0 < p.n_vec) tma_store_2d(&out_map, wg * 32, (int)v0, piece);
            }
        };
        float before = 0.f;                                        // scale of the tile in the epilogue
        // (a wait that gave up lets the rest of the loop run through on garbage, waits returning at once, so that the two
        // warps of a barrier stay together)
        for (int i = 0; i < n_my; ++i) {
            before = scale;
            produce(i);
            if (i >= 1) epilogue(i - 1, before);
            if (!ok && lane == 0) *abort_s = 1u;
        }
        if (n_my >= 1) epilogue(n_my - 1, scale);
        if (lane == 0) bulk_wait_all();                            // stores in flight read shared memory
    }
    if (!ok && lane == 0) { *abort_s = 1u; atomicOr(&g_dequant_error, 1u); }
    if (*abort_s && tid == 0) {                                    // give copies still in flight time to land
        const long long t0 = clock64();
        while (clock64() - t0 < (1ll << 20)) {}
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) tmem_dealloc(tmem_base, C::kTmemCols);
}

// Read and clear this file's device error flag (for pq_poll_device_errors).
int dequant_error_flags(unsigned int* flags) {
    unsigned int v = 0, zero = 0;
    if (cudaMemcpyFromSymbol(&v, g_dequant_error, sizeof(v)) != cudaSuccess) return PQ_ERR_CUDA;
    if (v && cudaMemcpyToSymbol(g_dequant_error, &zero, sizeof(zero)) != cudaSuccess) return PQ_ERR_CUDA;
    *flags = v;
    return PQ_OK;
}

template <int D, int BITS>
static int launch_dequant(const DequantParams& p, cudaStream_t st) {
    using C = DequantCfg<D>;
    auto kern = pq_dequant_kernel<D, BITS>;
    static std::atomic<uint64_t> allowed{0};
    if (allow_shared(kern, C::smem_bytes(), allowed) != cudaSuccess) return PQ_ERR_CUDA;
    int dev = 0, sms = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
        return PQ_ERR_CUDA;
    const int grid = (int)(p.n_items < sms ? p.n_items : sms);      // persistent: one CTA per SM (tensor memory)
    CUtensorMap map;
    const cuuint64_t dims[2] = {(cuuint64_t)D, (cuuint64_t)p.n_vec}, strides[1] = {(cuuint64_t)D * (p.out_is_fp16 ? 2 : 4)};
    const cuuint32_t box[2] = {p.out_is_fp16 ? 64u : 32u, 32u};
    if (!encode_tensor_map_2d(&map, p.out_is_fp16 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT32, p.out,
                              dims, strides, box))
        return PQ_ERR_CUDA;
    kern<<<grid, C::kThreads, C::smem_bytes(), st>>>(p, map);
    return cudaGetLastError() == cudaSuccess ? PQ_OK : PQ_ERR_CUDA;
}

}  // namespace pq

extern "C" int pq_dequant(const void* blocks, int64_t n_vec, int head_dim, int n_bits,
                          const float* codebook, const float* rot, void* out, int out_is_fp16,
                          void* stream) {
    using namespace pq;
    if (n_vec < 0) return PQ_ERR_BAD_SHAPE;
    if (head_dim != 64 && head_dim != 128) return PQ_ERR_BAD_HEAD_DIM;
    if (n_bits != 2 && n_bits != 4) return PQ_ERR_BAD_BITS;
    if (n_vec == 0) return PQ_OK;
    if (n_vec > (int64_t)0x7FFFFF00) return PQ_ERR_TOO_LARGE;      // tile coordinates are 32-bit
    if (!blocks || !codebook || !rot || !out) return PQ_ERR_NULL_POINTER;
    if ((reinterpret_cast<uintptr_t>(blocks) & 15) || (reinterpret_cast<uintptr_t>(rot) & 15) ||
        (reinterpret_cast<uintptr_t>(out) & 31))
        return PQ_ERR_MISALIGNED;
    DequantParams p{};
    p.blocks = static_cast<const uint8_t*>(blocks);
    p.n_items = (n_vec + kDqVecs - 1) / kDqVecs;
    p.rot = rot;
    p.out = out;
    p.n_vec = n_vec;
    p.out_is_fp16 = out_is_fp16;
    for (int i = 0; i < 16; ++i) p.cb[i] = i < (1 << n_bits) ? codebook[i] : 0.f;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (head_dim == 64) return n_bits == 4 ? launch_dequant<64, 4>(p, st) : launch_dequant<64, 2>(p, st);
    return n_bits == 4 ? launch_dequant<128, 4>(p, st) : launch_dequant<128, 2>(p, st);
}
