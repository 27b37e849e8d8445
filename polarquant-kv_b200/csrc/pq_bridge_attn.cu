// Attention of the llama.cpp bridge's codec (one float32 radius per vector, nibble-packed indices) for head dims 64
// and 128: score = dot(q, codebook[k idx]) * k_radius * scale, softmax, sum of weight * codebook[v idx] * v_radius.
// Operands, products and sums are float32 throughout, as the interface's are.
//
// Bound.  A stored byte (two elements) costs a table lookup and one packed float32x2 multiply-add per query head:
// for four query heads about 30 warp instructions per token against 136 stored bytes, so the kernel is bound by
// instruction issue and the shared-memory pipe, not by HBM.  What the layout does about it:
//   * centroid pairs come from a table with one 256-byte row per byte value at a fixed shared address (16 private
//     8-byte copies: a warp's lookup is two conflict-free wavefronts); a byte is dropped into the address with one
//     byte-permute;
//   * keys: four lanes share a token (a quarter of the row each) and a lane carries four tokens, so one load of the
//     query serves four tokens and the cross-lane sum is 12 shuffles per 32 tokens and head quadruple;
//   * values: a lane owns eight (four heads) or four (eight heads) dims of every second token, weights are broadcast
//     from shared memory;
//   * the running maximum moves only when a score exceeds it by 16 (log2): weights stay below 2^16 in float32;
//   * packed rows of a 32-token tile are contiguous and arrive by bulk copy, one tile ahead.
// Measured (D = 128, 8 kv heads, input sets in turn): 32 query heads x 32768 tokens 29 us (general kernel 68), x 65536 47
// (119); 64 query heads x 65536 80 (164); 8 query heads x 65536 31 (89) = 2.3 TB/s of the stored bytes.
// One CTA of 16 or 12 warps per SM; a (kv head, query group) is cut into slices over CTAs, merged by the last to arrive.
#include "pq_bridge.cuh"
#include "pq_tcgen05.cuh"

namespace pq {

static __device__ unsigned int g_bridge_error = 0;

constexpr int kBaTile = 32;                   // tokens a warp takes at a time
constexpr float kBaLowest = -1e30f;
constexpr float kBaGap = 16.0f;               // log2 units a scaled score may exceed the maximum in use
constexpr uint32_t kBaTab = 0x10000u;         // shared address of the pair table (bits 8..15 select its row)

template <int D, int G>
struct BridgeAttnCfg {
    static constexpr int WARPS = G <= 4 ? 16 : 12;            // eight heads need more than 128 registers
    static constexpr int ROWB = D / 2;                        // packed bytes per token
    static constexpr int KT = G <= 4 ? 4 : 2;                 // tokens a lane scores together
    static constexpr int VD = G <= 4 ? 8 : 4;                 // dims of a value a lane accumulates
    static constexpr bool kDup = G <= 4;                      // weights stored as (w, w) pairs
    static constexpr int kStage = 2 * kBaTile * ROWB;         // K rows, V rows
    static constexpr int kWts = kBaTile * G * (kDup ? 8 : 4);
    static constexpr int kWarpBytes = 2 * kStage + kWts;      // two stages; the warp's record reuses them at the end
    static constexpr int kQPad = 16;                          // bytes between the four quarters of the query rows
    static constexpr int kQBytes = D / 2 * G * 8 + 4 * kQPad;
    static constexpr int kFixed = kQBytes + WARPS * 16;    // + mbarriers
    static constexpr int kLowWarps = (65536 - 2048 - kFixed) / kWarpBytes < WARPS
                                         ? (65536 - 2048 - kFixed) / kWarpBytes : WARPS;
    static constexpr size_t smem_bytes() { return 2 * 65536 + (size_t)(WARPS - kLowWarps) * kWarpBytes; }
    static_assert(G * (D + 2) * 4 <= 2 * kStage, "a warp's record fits its stages");
};

__device__ __forceinline__ float2 ba_fma2(float2 a, float2 b, float2 c) {
    float2 d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;\n"
        : "=l"(*reinterpret_cast<unsigned long long*>(&d))
        : "l"(*reinterpret_cast<unsigned long long*>(&a)), "l"(*reinterpret_cast<unsigned long long*>(&b)),
          "l"(*reinterpret_cast<unsigned long long*>(&c)));
    return d;
}
__device__ __forceinline__ float2 ba_lds_f2(uint32_t a) {
    float2 v;
    asm volatile("ld.shared.v2.f32 {%0,%1}, [%2];\n" : "=f"(v.x), "=f"(v.y) : "r"(a));
    return v;
}
__device__ __forceinline__ float4 ba_lds_f4(uint32_t a) {
    float4 v;
    asm volatile("ld.shared.v4.f32 {%0,%1,%2,%3}, [%4];\n" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(a));
    return v;
}
// centroid pair of byte J of w
template <int J>
__device__ __forceinline__ float2 ba_pair(uint32_t w, uint32_t lane_const) {
    return ba_lds_f2(__byte_perm(w, lane_const, 0x7604u | (J << 4)));
}
__device__ __forceinline__ float2 ba_pair_at(uint32_t w, uint32_t lane_const, int j) {   // j known at compile time
    return j == 0 ? ba_pair<0>(w, lane_const) : j == 1 ? ba_pair<1>(w, lane_const)
         : j == 2 ? ba_pair<2>(w, lane_const) : ba_pair<3>(w, lane_const);
}
// `count` consecutive float2 (1, 2, 4 or 8) at a 16-byte boundary
template <int COUNT>
__device__ __forceinline__ void ba_lds_pairs(float2 (&v)[COUNT], uint32_t a) {
    if constexpr (COUNT == 1) {
        v[0] = ba_lds_f2(a);
    } else {
#pragma unroll
        for (int i = 0; i < COUNT / 2; ++i) {
            const float4 t = ba_lds_f4(a + 16 * i);
            v[2 * i] = make_float2(t.x, t.y);
            v[2 * i + 1] = make_float2(t.z, t.w);
        }
    }
}

template <int D, int G>
__global__ void __launch_bounds__(BridgeAttnCfg<D, G>::WARPS * 32, 1) bridge_attn_kernel(const BridgeAttnParams p) {
    using C = BridgeAttnCfg<D, G>;
    constexpr int WARPS = C::WARPS, ROWB = C::ROWB, KT = C::KT, VD = C::VD;
    constexpr int QB = ROWB / 4, QW = QB / 4;                  // bytes and words of a row per lane (a quarter)
    constexpr unsigned kAll = 0xffffffffu;
    extern __shared__ __align__(128) uint8_t smem[];
    __shared__ unsigned s_last;
    const uint32_t base = sm_addr(smem);
    if (base + C::kFixed + C::kLowWarps * C::kWarpBytes > kBaTab) {
        if (threadIdx.x == 0) atomicOr(&g_bridge_error, 2u);
        return;
    }
    uint8_t* zero = smem - base;                               // generic address of shared address 0
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int split = blockIdx.x, group = blockIdx.y, hkv = blockIdx.z;
    const int hq0 = hkv * p.gqa + group * G;
    const int n_heads = min(G, p.gqa - group * G);             // query heads of this CTA that exist
    const uint32_t q_addr = base, bar0 = base + C::kQBytes + warp * 16;
    auto warp_area = [&](int w) -> uint8_t* {
        return w < C::kLowWarps ? smem + C::kFixed + w * C::kWarpBytes
                                : zero + 0x20000 + (w - C::kLowWarps) * C::kWarpBytes;
    };
    const uint32_t area = sm_addr(warp_area(warp));
    const uint32_t wts = area + 2 * C::kStage;

    const int n_tiles = (p.S + kBaTile - 1) / kBaTile;
    const int tile_hi = min(n_tiles, (split + 1) * p.tiles_per_split);
    const size_t row0 = (size_t)hkv * p.S;
    auto issue = [&](int tile, int slot) {                     // lane 0: the packed rows of a tile
        if (tile >= tile_hi || lane != 0) return;
        const uint32_t bytes = (uint32_t)min(kBaTile, p.S - tile * kBaTile) * ROWB, mb = bar0 + 8 * slot;
        const size_t off = (row0 + (size_t)tile * kBaTile) * ROWB;
        mbar_expect_tx(mb, 2 * bytes);
        bulk_load(area + slot * C::kStage, p.pk + off, bytes, mb);
        bulk_load(area + slot * C::kStage + kBaTile * ROWB, p.pv + off, bytes, mb);
    };
    // lane <-> token of the tile: four lanes score tokens 8 i + lane / 4 together, lane t of them keeps i = t
    const int tk = 8 * (lane & 3) + (lane >> 2);
    int tile = split * p.tiles_per_split + warp;
    float kr = 0.f, vr = 0.f;
    auto fetch_radii = [&](int t) {
        const int s = t * kBaTile + tk;
        const bool in = t < tile_hi && s < p.S;
        kr = in ? __ldg(p.kr + row0 + s) : 0.f;
        vr = in ? __ldg(p.vr + row0 + s) : 0.f;
    };
    if (lane == 0) {
        mbar_init(bar0, 1);
        mbar_init(bar0 + 8, 1);
    }
    __syncwarp();
    issue(tile, 0);
    fetch_radii(tile);
    // ---- the pair table and the query, [quarter][byte][head] -> the two query elements the byte multiplies
    {
        const uint32_t mask = (uint32_t)(p.n_levels - 1);
        for (int e = tid; e < 256 * 16; e += WARPS * 32) {
            const uint32_t byte = (uint32_t)e >> 4;
            *reinterpret_cast<float2*>(zero + kBaTab + byte * 256 + (e & 15) * 8) =
                make_float2(__ldg(p.codebook + (byte & mask)), __ldg(p.codebook + ((byte >> 4) & mask)));
        }
        for (int e = tid; e < (D / 2) * G; e += WARPS * 32) {
            const int h = e / (D / 2), b = e % (D / 2);
            float2 v = make_float2(0.f, 0.f);
            if (h < n_heads) v = __ldg(reinterpret_cast<const float2*>(p.q + (size_t)(hq0 + h) * D) + b);
            *reinterpret_cast<float2*>(smem + (b * G + h) * 8 + (b / QB) * C::kQPad) = v;
        }
    }
    __syncthreads();
    const uint32_t tab_lane = kBaTab | ((lane & 15) * 8);
    const uint32_t q_lane = q_addr + (lane & 3) * (QB * G * 8 + C::kQPad);
    // Scores are kept as dot x radius, rounded once, and scaled after the maximum is taken off, where they are small if the
    // weight is not (with radii scaled beforehand the results were 4 % further from 64 bits
    // than the general kernel's, now they are 2 % closer).  A negative scale's sign
    // goes with the radii.
    const float scale2 = fabsf(p.scale) * 1.4426950408889634f, sign = p.scale < 0.f ? -1.f : 1.f;

    float m[G], l[G];
    float2 acc[G][VD / 2];
#pragma unroll
    for (int h = 0; h < G; ++h) {
        m[h] = kBaLowest;
        l[h] = 0.f;
#pragma unroll
        for (int i = 0; i < VD / 2; ++i) acc[h][i] = make_float2(0.f, 0.f);
    }
    constexpr int LPR = D / VD, TPI = 32 / LPR;                // lanes per value row, rows per step
    const int sub = lane / LPR, li = lane % LPR;
    bool dead = false;
    uint32_t slot = 0, phase = 0;
    for (; tile < tile_hi; tile += WARPS) {
        issue(tile + WARPS, slot ^ 1);
        const float kr_t = kr * sign, vr_t = vr;
        fetch_radii(tile + WARPS);
        const int valid = min(kBaTile, p.S - tile * kBaTile);
        if (!dead && !mbar_wait(bar0 + 8 * slot, (phase >> slot) & 1u)) {
            dead = true;
            atomicOr(&g_bridge_error, 1u);
        }
        phase ^= 1u << slot;
        const uint32_t ks = area + slot * C::kStage, vs = ks + kBaTile * ROWB;
        // ---- scores
        float s[G];
        // (a real loop: unrolled, the compiler keeps all of the query in registers between the passes and spills)
#pragma unroll 1
        for (int pass = 0; pass < 4 / KT; ++pass) {
            uint32_t w[KT][QW];
            float2 a[KT][G];
#pragma unroll
            for (int i = 0; i < KT; ++i) {
                const uint32_t r = ks + (8 * (pass * KT + i) + (lane >> 2)) * ROWB + (lane & 3) * QB;
                if constexpr (QW == 4) {
                    const float4 v = ba_lds_f4(r);
                    w[i][0] = __float_as_uint(v.x); w[i][1] = __float_as_uint(v.y);
                    w[i][QW - 2] = __float_as_uint(v.z); w[i][QW - 1] = __float_as_uint(v.w);
                } else {
                    const float2 v = ba_lds_f2(r);
                    w[i][0] = __float_as_uint(v.x); w[i][1] = __float_as_uint(v.y);
                }
#pragma unroll
                for (int h = 0; h < G; ++h) a[i][h] = make_float2(0.f, 0.f);
            }
#pragma unroll
            for (int b = 0; b < QB; ++b) {
                float2 qv[G];
                ba_lds_pairs<G>(qv, q_lane + b * G * 8);
#pragma unroll
                for (int i = 0; i < KT; ++i) {
                    const float2 c = ba_pair_at(w[i][b >> 2], tab_lane, b & 3);
#pragma unroll
                    for (int h = 0; h < G; ++h) a[i][h] = ba_fma2(qv[h], c, a[i][h]);
                }
            }
            // sums over the four lanes of a token; lane t ends with token i = t
            const bool up1 = lane & 1, up2 = lane & 2;
#pragma unroll
            for (int h = 0; h < G; ++h) {
                float v[KT];
#pragma unroll
                for (int i = 0; i < KT; ++i) v[i] = a[i][h].x + a[i][h].y;
                if constexpr (KT == 4) {
                    const float k0 = up2 ? v[2] : v[0], k1 = up2 ? v[3] : v[1];
                    const float x0 = k0 + __shfl_xor_sync(kAll, up2 ? v[0] : v[2], 2);
                    const float x1 = k1 + __shfl_xor_sync(kAll, up2 ? v[1] : v[3], 2);
                    s[h] = (up1 ? x1 : x0) + __shfl_xor_sync(kAll, up1 ? x0 : x1, 1);
                } else {
                    const float x = (up1 ? v[1] : v[0]) + __shfl_xor_sync(kAll, up1 ? v[0] : v[1], 1);
                    const float y = x + __shfl_xor_sync(kAll, x, 2);
                    s[h] = (pass == 0 || up2) ? y : s[h];      // pass 0 serves lanes with t < 2, pass 1 the others
                }
            }
        }
        // ---- online softmax
        const bool in = tk < valid;
        bool grow = false;
#pragma unroll
        for (int h = 0; h < G; ++h) {
            s[h] = in ? s[h] * kr_t : kBaLowest;
            grow |= (s[h] - m[h]) * scale2 > kBaGap;
        }
        if (__any_sync(kAll, grow)) {
#pragma unroll
            for (int h = 0; h < G; ++h) {
                float t = s[h];
#pragma unroll
                for (int o = 16; o; o >>= 1) t = fmaxf(t, __shfl_xor_sync(kAll, t, o));
                const float m_new = fmaxf(m[h], t), c = fast_exp2((m[h] - m_new) * scale2);
                m[h] = m_new;
                l[h] *= c;
#pragma unroll
                for (int i = 0; i < VD / 2; ++i) { acc[h][i].x *= c; acc[h][i].y *= c; }
            }
        }
        float wt[G];
#pragma unroll
        for (int h = 0; h < G; ++h) {
            const float pr = in ? fast_exp2((s[h] - m[h]) * scale2) : 0.f;
            l[h] += pr;                                        // this lane's share of the denominator
            wt[h] = pr * vr_t;
        }
        if constexpr (C::kDup) {
#pragma unroll
            for (int h = 0; h < G; ++h)
                asm volatile("st.shared.v2.f32 [%0], {%1,%1};\n" ::"r"(wts + (tk * G + h) * 8), "f"(wt[h]) : "memory");
        } else {
#pragma unroll
            for (int h = 0; h < G; h += 4)
                asm volatile("st.shared.v4.f32 [%0], {%1,%2,%3,%4};\n" ::"r"(wts + (tk * G + h) * 4), "f"(wt[h]),
                             "f"(wt[h + 1]), "f"(wt[h + 2]), "f"(wt[h + 3])
                             : "memory");
        }
        __syncwarp();
        // ---- values: rows past the end carry weight zero (whatever bytes the stage holds there decode to centroids)
#pragma unroll 4
        for (int it = 0; it < kBaTile / TPI; ++it) {
            const int t = it * TPI + sub;
            uint32_t w;
            if constexpr (VD == 8)
                asm volatile("ld.shared.u32 %0, [%1];\n" : "=r"(w) : "r"(vs + t * ROWB + li * 4));
            else
                asm volatile("{ .reg .u16 t; ld.shared.u16 t, [%1]; cvt.u32.u16 %0, t; }\n" : "=r"(w) : "r"(vs + t * ROWB + li * 2));
            float2 wv[G];
            if constexpr (C::kDup) {
                ba_lds_pairs<G>(wv, wts + t * G * 8);
            } else {
                float2 half[G / 2];
                ba_lds_pairs<G / 2>(half, wts + t * G * 4);
#pragma unroll
                for (int h = 0; h < G; ++h) {
                    const float x = (h & 1) ? half[h / 2].y : half[h / 2].x;
                    wv[h] = make_float2(x, x);
                }
            }
#pragma unroll
            for (int i = 0; i < VD / 2; ++i) {
                const float2 c = ba_pair_at(w, tab_lane, i);
#pragma unroll
                for (int h = 0; h < G; ++h) acc[h][i] = ba_fma2(wv[h], c, acc[h][i]);
            }
        }
        __syncwarp();
        slot ^= 1;
    }

    // ---- warp record over its stages: m, l, o[D] per head
    float* rec = reinterpret_cast<float*>(warp_area(warp));
#pragma unroll
    for (int h = 0; h < G; ++h) {
        float lt = l[h];
#pragma unroll
        for (int o = 16; o; o >>= 1) lt += __shfl_xor_sync(kAll, lt, o);
#pragma unroll
        for (int i = 0; i < VD / 2; ++i) {
#pragma unroll
            for (int o = LPR; o < 32; o <<= 1) {
                acc[h][i].x += __shfl_xor_sync(kAll, acc[h][i].x, o);
                acc[h][i].y += __shfl_xor_sync(kAll, acc[h][i].y, o);
            }
        }
        if (lane == 0) { rec[h * (D + 2)] = m[h]; rec[h * (D + 2) + 1] = lt; }
        if (sub == 0) {
#pragma unroll
            for (int i = 0; i < VD / 2; ++i) {
                rec[h * (D + 2) + 2 + li * VD + 2 * i] = acc[h][i].x;
                rec[h * (D + 2) + 3 + li * VD + 2 * i] = acc[h][i].y;
            }
        }
    }
    __syncthreads();
    constexpr int REC = D + 2;
    const bool single = p.n_split == 1;
    for (int e = tid; e < n_heads * D; e += WARPS * 32) {
        const int h = e / D, d = e - h * D;
        float ms[WARPS], mm = kBaLowest, ll = 0.f, aa = 0.f;
#pragma unroll
        for (int w = 0; w < WARPS; ++w) {
            ms[w] = reinterpret_cast<const float*>(warp_area(w))[h * REC];
            mm = fmaxf(mm, ms[w]);
        }
#pragma unroll
        for (int w = 0; w < WARPS; ++w) {
            const float* r = reinterpret_cast<const float*>(warp_area(w)) + h * REC;
            const float c = fast_exp2((ms[w] - mm) * scale2);
            ll = fmaf(r[1], c, ll);
            aa = fmaf(r[2 + d], c, aa);
        }
        if (single) {
            p.out[(size_t)(hq0 + h) * D + d] = ll > 0.f ? aa / ll : 0.f;
        } else {
            float* o = p.partials + ((size_t)(hq0 + h) * p.n_split + split) * REC;
            if (d == 0) { __stcg(o, mm); __stcg(o + 1, ll); }
            __stcg(o + 2 + d, aa);
        }
    }
    if (single) return;
    // ---- the last slice to finish merges the records of its heads
    __threadfence();
    __syncthreads();
    if (tid == 0) {
        unsigned* ticket = p.tickets + hkv * gridDim.y + group;
        s_last = atomicAdd(ticket, 1u) == (unsigned)p.n_split - 1;
        if (s_last) *ticket = 0;
    }
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    for (int e = tid; e < n_heads * D; e += WARPS * 32) {
        const int h = e / D, d = e - h * D;
        const float* r0 = p.partials + (size_t)(hq0 + h) * p.n_split * REC;
        float mm = kBaLowest, ll = 0.f, aa = 0.f;
        for (int s0 = 0; s0 < p.n_split; s0 += 8) {            // eight records per round trip to L2
            float ms[8], ls[8], as[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                const float* r = r0 + (size_t)min(s0 + u, p.n_split - 1) * REC;
                ms[u] = __ldcg(r);
                ls[u] = __ldcg(r + 1);
                as[u] = __ldcg(r + 2 + d);
            }
            float m_new = mm;
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                if (s0 + u >= p.n_split) { ms[u] = kBaLowest; ls[u] = 0.f; as[u] = 0.f; }
                m_new = fmaxf(m_new, ms[u]);
            }
            const float c = fast_exp2((mm - m_new) * scale2);
            ll *= c;
            aa *= c;
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                const float cu = fast_exp2((ms[u] - m_new) * scale2);
                ll = fmaf(ls[u], cu, ll);
                aa = fmaf(as[u], cu, aa);
            }
            mm = m_new;
        }
        p.out[(size_t)(hq0 + h) * D + d] = ll > 0.f ? aa / ll : 0.f;
    }
}

// ------------------------------------------------------------------ host side
bool bridge_attention_fits(int D, const void* packed_k, const void* packed_v) {
    return (D == 64 || D == 128) && ((reinterpret_cast<uintptr_t>(packed_k) | reinterpret_cast<uintptr_t>(packed_v)) & 15) == 0;
}

// Query heads per CTA: the smallest of 1, 2, 4, 8 that holds the group (a missing head costs its multiply-adds, a
// second CTA over the same keys would repeat the lookups too); groups above eight heads are cut into eights.  Short calls,
// where a CTA's latency counts, take fours unless eights come out even (14 query / 2 kv heads of 128, 200 tokens: eights
// 10.6 us, fours 8.5, the general kernel 9.8).
static int bridge_heads(int gqa, int S) {
    if (gqa >= 5) return gqa % 8 && S <= 512 ? 4 : 8;
    return gqa >= 3 ? 4 : gqa;
}

int bridge_attention_plan(BridgeAttnParams& p, int total_kv_heads, int sms, size_t ws_floats, int ws_tickets,
                          int total_q_heads) {
    const int G = bridge_heads(p.gqa, p.S), groups = (p.gqa + G - 1) / G;
    const int n_tiles = (p.S + kBaTile - 1) / kBaTile, rows = total_kv_heads * groups;
    // one CTA per SM; a slice has at least four tiles (four warps already keep an SM's schedulers busy, and a tile takes
    // an SM 250 cycles of issue, about what merging one more slice costs)
    int n_split = sms / rows;
    const int most = (n_tiles + 3) / 4;
    if (n_split > most) n_split = most;
    const size_t per_split = (size_t)total_q_heads * (p.D + 2);
    if (rows > ws_tickets) n_split = 1;
    if (n_split > 1 && (size_t)n_split * per_split > ws_floats) n_split = (int)(ws_floats / per_split);
    if (n_split < 1) n_split = 1;
    p.tiles_per_split = (n_tiles + n_split - 1) / n_split;
    p.n_split = (n_tiles + p.tiles_per_split - 1) / p.tiles_per_split;
    return groups;
}

template <int D, int G>
static cudaError_t launch_bridge(const BridgeAttnParams& p, int total_kv_heads, int groups, cudaStream_t st) {
    auto kern = bridge_attn_kernel<D, G>;
    const size_t smem = BridgeAttnCfg<D, G>::smem_bytes();
    static std::atomic<uint64_t> allowed{0};
    const cudaError_t e = allow_shared(kern, smem, allowed);
    if (e != cudaSuccess) return e;
    kern<<<dim3(p.n_split, groups, total_kv_heads), BridgeAttnCfg<D, G>::WARPS * 32, smem, st>>>(p);
    return cudaGetLastError();
}

cudaError_t bridge_attention_launch(const BridgeAttnParams& p, int total_kv_heads, int groups, cudaStream_t st) {
    const int G = bridge_heads(p.gqa, p.S);
#define PQ_BA(DD, GG) if (p.D == DD && G == GG) return launch_bridge<DD, GG>(p, total_kv_heads, groups, st);
    PQ_BA(128, 1) PQ_BA(128, 2) PQ_BA(128, 4) PQ_BA(128, 8)
    PQ_BA(64, 1) PQ_BA(64, 2) PQ_BA(64, 4) PQ_BA(64, 8)
#undef PQ_BA
    return cudaErrorInvalidValue;
}

int bridge_error_flags(unsigned int* flags) {
    unsigned int v = 0, zero = 0;
    if (cudaMemcpyFromSymbol(&v, g_bridge_error, sizeof(v)) != cudaSuccess) return PQ_ERR_CUDA;
    if (v && cudaMemcpyToSymbol(g_bridge_error, &zero, sizeof(zero)) != cudaSuccess) return PQ_ERR_CUDA;
    *flags = v;
    return PQ_OK;
}

}  // namespace pq
