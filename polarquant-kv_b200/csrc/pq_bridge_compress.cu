// Compress of the llama.cpp bridge's codec for head dims 64 and 128 and many vectors: rotate,
// Euclidean norm, divide, nearest level of a device-side codebook, pack two indices per byte.
//
// The rotation is a [N x D] . [D x D] product of float32 operands.  On CUDA cores it is the bound (34 GFLOP at 2^20
// vectors of 128: 0.5 ms at the FP32 peak); here it runs on the 5th-generation tensor cores with both operands as the
// sum of three bfloat16 terms.  The tensor core cuts off what falls below its accumulator's last bit at every step, always
// towards zero, which took 1.4e-7 off every radius while all products shared one accumulator and the leading terms were the
// operands rounded to bfloat16.  Therefore
//   * the leading term of a row (of x, of R) is the row in whole units of 2^-8 of its largest element's power of two:
//     integers up to 256, whose products add up to at most 2^23 units at D = 128, exactly;
//   * their sum has an accumulator to itself.  The five correction products (the three left out are below 2^-25 of the
//     largest one) go into a second one, whose cuts are 2^-8 as large, and the two are added in float32.
// The error of a coordinate is then a third of an FP32 chain's, that of the radius four fifths (3.3e-8 against 4.2e-8 rms).
//
// A persistent CTA owns 128 vectors at a time:
//   copy warp    boxes of 128 vectors x 32 floats by TMA (128-byte swizzle), a ring of them in flight;
//   worker warps (4 per 32 dims) one thread = one vector x 32 dims: reads its row of the box, writes the three terms
//                into tensor memory as the A operand; one tile behind, reads its 32 columns of both accumulators
//                and runs the float32 epilogue, under which the MMAs of the next tile go on;
//   MMA warp     6 x D/16 MMAs per tile (A from tensor memory, B = the three terms of R in shared memory), 3.1 K
//                cycles at D = 128.
// Index search: the reference scans the levels and keeps the first of the closest.  For levels in ascending order that is
// "how many decision points lie below", with the decision points found once per CTA by bisection over the float32 numbers;
// a coordinate's bucket (1/128 wide) holds at most one of them.  Where two fall into one bucket, or the levels come in
// another order or repeat themselves, a search tree of the sorted decision points takes four lookups instead of one; levels
// closer than 1e-5, or outside (-1, 1), are scanned as the reference does.
// Measured (16 levels, second pass included): 131 072 vectors of 128 49 us, 2^20 of them 244 (R^T in shared memory on CUDA
// cores: 238 and 1835); of 64: 30 and 125 us (80 and 595).  One accumulator and plain bfloat16 terms: 45.5, 230, 27, 117.
// By the search tree 2^20 vectors of 128 take 340 us and of 64 184 (level by level: 805 and 625).
// The rotation's last bits depend on the order of its additions, and a coordinate within them of a decision point gets one
// index or the other.  So that stored bytes do not depend on which of the two kernels for many vectors wrote them (the one
// below 4096 vectors adds in another order, and may differ there), a block with a coordinate closer
// than kBcNear to a decision point (one in 500 at 16 levels) is put on a list and done again at the end in the order of
// an FP32 chain, k ascending per output, with R copied over the boxes, which are free by then.  The same goes for whole vectors whose radius is not a number,
// infinite, or so small that its squares are subnormal: there too the stored values are the chain's.
// All waits are bounded (bit 10 of pq_poll_device_errors).
#include <cstring>

#include "pq_bridge.cuh"
#include "pq_tcgen05.cuh"

namespace pq {

static __device__ unsigned int g_bridge_compress_error = 0;

constexpr int kBcVecs = 128;
constexpr float kBcNear = 6e-7f;               // ten times the typical difference between two summation orders
constexpr uint32_t kBcScan = 0, kBcTree = 1, kBcBuckets = 2;    // how indices are found
constexpr int kBcList = 480;                   // (vector, block) entries a CTA keeps for the second pass

template <int D>
struct BridgeCompressCfg {
    static constexpr int WG = D / 32;
    static constexpr int WORKERS = 128 * WG;                       // one thread per (vector, 32 dims)
    static constexpr int THREADS = WORKERS + 64;                   // + MMA warp + copy warp
    static constexpr uint32_t kBTerm = D * D * 2;                  // one bfloat16 term of R
    static constexpr uint32_t kBox = kBcVecs * 32 * 4;             // 128 vectors x 32 floats
    // A slot of the ring always serves the same 32 dims (a multiple of WG): its next box can then not be waited for
    // before every thread that reads the slot has seen the previous one, which the parity waits rely on.
    static constexpr int kBoxes = D == 128 ? 4 : 6;
    static_assert(kBoxes % WG == 0, "a box slot belongs to one group of worker warps");
    // Layout by absolute shared address: index table (257 buckets x 16 copies x 8 bytes; its address is an immediate of
    // the lookups) | three terms of R | boxes | small buffers
    static constexpr uint32_t kTabAddr = 4096;
    static constexpr uint32_t kTabRows = 258;
    static constexpr uint32_t kBAddr = (kTabAddr + kTabRows * 128 + 1023) & ~1023u;
    static constexpr uint32_t kBoxAddr = (kBAddr + 3 * kBTerm + 1023) & ~1023u;
    static constexpr uint32_t kSmallAddr = kBoxAddr + kBoxes * kBox;
    static constexpr uint32_t kATerm = D / 2;                      // tensor-memory columns of one term
    static constexpr uint32_t kAcc = 2 * D;                        // leading products; the corrections D columns further
    static constexpr uint32_t kTmemCols = 4 * D;
    // norms and largest elements [2][128][WG] each, four arrays of 16 around the codebook, barriers, tensor-memory slot,
    // flags, list
    static constexpr uint32_t kSmall = 4 * kBcVecs * WG * 4 + 4 * 16 * 4 + (2 * kBoxes + 6) * 8 + 32 + kBcList * 4;
    static constexpr size_t smem_bytes() { return kSmallAddr + kSmall; }
};

// kind::f16 instruction descriptor with bfloat16 operands (both K-major), float32 accumulator, M = 128
__host__ __device__ constexpr uint32_t umma_idesc_bf16(int n) { return umma_idesc_f16(n) | (1u << 7) | (1u << 10); }

__device__ __forceinline__ float2 bc_mul2(float2 a, float2 b) {
    float2 d;
    asm("mul.rn.f32x2 %0, %1, %2;\n"
        : "=l"(*reinterpret_cast<unsigned long long*>(&d))
        : "l"(*reinterpret_cast<unsigned long long*>(&a)), "l"(*reinterpret_cast<unsigned long long*>(&b)));
    return d;
}
__device__ __forceinline__ float2 bc_fma2(float2 a, float2 b, float2 c) {
    float2 d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;\n"
        : "=l"(*reinterpret_cast<unsigned long long*>(&d))
        : "l"(*reinterpret_cast<unsigned long long*>(&a)), "l"(*reinterpret_cast<unsigned long long*>(&b)),
          "l"(*reinterpret_cast<unsigned long long*>(&c)));
    return d;
}
__device__ __forceinline__ float2 bc_add2(float2 a, float2 b) {
    float2 d;
    asm("add.rn.f32x2 %0, %1, %2;\n"
        : "=l"(*reinterpret_cast<unsigned long long*>(&d))
        : "l"(*reinterpret_cast<unsigned long long*>(&a)), "l"(*reinterpret_cast<unsigned long long*>(&b)));
    return d;
}
// 1.5 x 2^23 units, for a row whose largest element is `most` and whose unit is 2^-8 of the power of two above it: adding
// and taking it off again rounds to whole units.  From 2^112 on it is not a number, and then the whole row becomes none.
__device__ __forceinline__ float bc_unit_magic(float most) {
    return __uint_as_float((min((__float_as_uint(most) >> 23) + 16u, 255u) << 23) | 0x400000u);
}
// leading term of two elements, packed bfloat16 (exact), and what it leaves (exact)
__device__ __forceinline__ uint32_t bc_lead(float2& x, float magic) {
    const float2 h = bc_add2(bc_add2(x, make_float2(magic, magic)), make_float2(-magic, -magic));
    uint32_t w;
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;\n" : "=r"(w) : "f"(h.y), "f"(h.x));
    x = bc_fma2(h, make_float2(-1.f, -1.f), x);
    return w;
}
// two floats -> packed bfloat16 (first in the low half), and what the rounding left
__device__ __forceinline__ uint32_t bc_term(float2& x) {
    uint32_t w;
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;\n" : "=r"(w) : "f"(x.y), "f"(x.x));
    const float2 neg = make_float2(__uint_as_float((w << 16) ^ 0x80000000u), __uint_as_float((w & 0xFFFF0000u) ^ 0x80000000u));
    x = bc_add2(x, neg);                                            // exact
    return w;
}
__device__ __forceinline__ void bc_tmem_st16(uint32_t taddr, const uint32_t (&v)[16]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};\n" ::"r"(taddr),
                 "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]),
                 "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15])
                 : "memory");
}
// Bucket of a coordinate in bits 7..15: the unit in the last place of 128 v + 98432 is 2^-7, so those bits hold
// floor(128 v + 128 + shift) after rounding to 1/128.  Monotone in v.  `magic` = 98432 + shift; the shift (below 1) keeps
// every decision point away from the edges of its bucket, so that a coordinate near one shares its bucket.
__device__ __forceinline__ uint32_t bc_bucket_bits(float v, float magic) { return __float_as_uint(fmaf(v, 128.f, magic)) & 0xFF80u; }
// order-preserving integer image of a float and back
__device__ __forceinline__ int bc_key(float x) {
    const int b = __float_as_int(x);
    return b >= 0 ? b : -(b & 0x7FFFFFFF);
}
__device__ __forceinline__ float bc_unkey(int k) {
    return k >= 0 ? __int_as_float(k) : __uint_as_float((uint32_t)(-k) | 0x80000000u);
}

struct BridgeCompressParams {
    const float* R;
    const float* codebook;
    float* radius_out;
    uint8_t* packed_out;
    const float* x;
    int N, n_levels;
};

// Byte offset of R[n][k] in the second pass's copy: consecutive n at one k, and consecutive k at one n, are in different banks.
template <int D>
__device__ __forceinline__ uint32_t bc_staged(int n, int k) { return (uint32_t)(k * D + (n ^ (k & 31))) * 4; }

// One block of one vector once more, by a whole warp (lane l: elements l + 32 i): k ascending per output as on CUDA cores,
// squares as a tree over i and the lanes, then level by level; block 0 brings the radius along.  What it overwrites was
// stored by this warp, or before a barrier.  (Out of line and with real loops: it runs for a few blocks per CTA, and
// straight-line code would spend its time on instruction fetches.)  SHARED: R is where the second pass put it, else in L2,
// whose lines every lane of a load would hit one of (ten times the time).
template <int D, bool SHARED>
__device__ __noinline__ void bc_again(const BridgeCompressParams& p, const float* cb, int vec, int block) {
    using C = BridgeCompressCfg<D>;
    constexpr int WG = C::WG;
    const int lane = threadIdx.x & 31;
    const float* x = p.x + (size_t)vec * D;
    float acc[WG], xl[WG];
#pragma unroll
    for (int m = 0; m < WG; ++m) { xl[m] = __ldg(x + lane + 32 * m); acc[m] = 0.f; }
#pragma unroll 1
    for (int kc = 0; kc < D / 8; ++kc) {
        float xv[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) xv[k] = __shfl_sync(0xffffffffu, xl[0], ((kc & 3) * 8 + k) & 31);
        if ((kc & 3) == 3) {
#pragma unroll
            for (int m = 0; m + 1 < WG; ++m) xl[m] = xl[m + 1];
        }
#pragma unroll
        for (int i = 0; i < WG; ++i) {
            float r[8];                                        // R[lane + 32 i][8 kc .. 8 kc + 7]
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                if constexpr (SHARED)
                    asm volatile("ld.shared.f32 %0, [%1];\n" : "=f"(r[k]) : "r"(C::kBoxAddr + bc_staged<D>(lane + 32 * i, 8 * kc + k)));
                else
                    r[k] = __ldg(p.R + (size_t)(lane + 32 * i) * D + 8 * kc + k);
            }
#pragma unroll
            for (int k = 0; k < 8; ++k) acc[i] = fmaf(xv[k], r[k], acc[i]);
        }
    }
    float sq[WG];
#pragma unroll
    for (int i = 0; i < WG; ++i) sq[i] = __fmul_rn(acc[i], acc[i]);
#pragma unroll
    for (int h = WG / 2; h; h >>= 1)
#pragma unroll
        for (int i = 0; i < h; ++i) sq[i] = __fadd_rn(sq[i], sq[i + h]);
    float t = sq[0];
#pragma unroll
    for (int o = 16; o; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    const float radius = __fsqrt_rn(t);
    float v = acc[0];
#pragma unroll
    for (int i = 1; i < WG; ++i)
        if (i == block) v = acc[i];
    const float dir = radius > 1e-30f ? __fdiv_rn(v, radius) : 0.f;
    uint32_t best = 0;
    float dist = 1e30f;
#pragma unroll 1
    for (int l = 0; l < p.n_levels; ++l) {
        const float d = fabsf(dir - cb[l]);
        if (d < dist) { dist = d; best = l; }
    }
    const uint32_t up = __shfl_down_sync(0xffffffffu, best, 1);
    __syncwarp();
    if (!(lane & 1)) p.packed_out[(size_t)vec * (D / 2) + block * 16 + (lane >> 1)] = (uint8_t)(best | (up << 4));
    if (block == 0 && lane == 0) p.radius_out[vec] = radius;
}

template <int D>
__global__ void __launch_bounds__(BridgeCompressCfg<D>::THREADS, 1)
bridge_compress_kernel(const __grid_constant__ BridgeCompressParams p, const __grid_constant__ CUtensorMap x_map) {
    using C = BridgeCompressCfg<D>;
    constexpr int WG = C::WG, WORKERS = C::WORKERS, NB = C::kBoxes;
    extern __shared__ __align__(128) uint8_t smem[];
    const uint32_t base = sm_addr(smem);
    if (base > C::kTabAddr) {                                  // the window starts too high for the fixed layout
        if (threadIdx.x == 0) atomicOr(&g_bridge_compress_error, 2u);
        return;
    }
    uint8_t* zero = smem - base;                               // generic address of shared address 0
    uint8_t* Bt = zero + C::kBAddr;
    float* norm_s = reinterpret_cast<float*>(zero + C::kSmallAddr);          // [tile parity][vector][WG]
    float* most_s = norm_s + 2 * kBcVecs * WG;                               // the same
    float* cb = most_s + 2 * kBcVecs * WG;
    float* thr = cb + 16;
    float* sorted = thr + 16;
    int* which = reinterpret_cast<int*>(sorted + 16);
    uint64_t* mbar = reinterpret_cast<uint64_t*>(which + 16);
    // [0, NB) box landed; [NB, 2 NB) box read; then, per parity of the tile: A written; its MMAs done (A free, the
    // accumulators complete); accumulators read out
    uint64_t* box_full = mbar;
    uint64_t* box_free = mbar + NB;
    uint64_t* a_full = mbar + 2 * NB;
    uint64_t* mma_done = a_full + 2;
    uint64_t* acc_free = a_full + 4;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(a_full + 6);
    volatile uint32_t* abort_s = tmem_slot + 1;
    uint32_t* kind_s = tmem_slot + 2;
    float* magic_s = reinterpret_cast<float*>(tmem_slot + 3);
    int* n_list = reinterpret_cast<int*>(tmem_slot + 4);
    int* list = reinterpret_cast<int*>(tmem_slot + 8);          // vector * WG + block

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    // ---- set-up
    if (tid == 0) {
        for (int i = 0; i < NB; ++i) {
            mbar_init(sm_addr(box_full + i), 1);
            mbar_init(sm_addr(box_free + i), 128);
        }
        for (int i = 0; i < 2; ++i) {
            mbar_init(sm_addr(a_full + i), WORKERS);
            mbar_init(sm_addr(mma_done + i), 1);
            mbar_init(sm_addr(acc_free + i), WORKERS);
        }
        *abort_s = 0u;
        *n_list = 0;
    }
    if (tid < 16) cb[tid] = __ldg(p.codebook + min(tid, p.n_levels - 1));
    // B: three bfloat16 terms of R, K-major core matrices (8 rows x 16 bytes), K chunks D / 8 * 128 bytes apart.  A thread's
    // pieces (8 elements of a row) are all in flight at once; the largest element of a row comes from its pieces' threads.
    {
        constexpr int PIECES = D * (D / 8), MINE = (PIECES + C::THREADS - 1) / C::THREADS;
        auto row = [](int e) { return (e & 7) + 8 * (e / D); };
        auto chunk = [](int e) { return (e >> 3) % (D / 8); };
        float2 x[MINE][4];
#pragma unroll
        for (int j = 0; j < MINE; ++j) {
            const int e = min(tid + j * C::THREADS, PIECES - 1);
#pragma unroll
            for (int i = 0; i < 4; ++i) x[j][i] = __ldg(reinterpret_cast<const float2*>(p.R + (size_t)row(e) * D + chunk(e) * 8) + i);
        }
        if (tid < D) most_s[tid] = 0.f;
        __syncthreads();
#pragma unroll
        for (int j = 0; j < MINE; ++j) {
            float most = 0.f;
#pragma unroll
            for (int i = 0; i < 4; ++i) most = fmaxf(most, fmaxf(fabsf(x[j][i].x), fabsf(x[j][i].y)));
            // (the bits of floats that are not negative are in their order)
            atomicMax(reinterpret_cast<int*>(most_s) + row(min(tid + j * C::THREADS, PIECES - 1)), __float_as_int(most));
        }
        __syncthreads();
#pragma unroll
        for (int j = 0; j < MINE; ++j) {
            const int e = tid + j * C::THREADS;
            if (e >= PIECES) break;
            const int n = row(e);
            const uint32_t off = (uint32_t)(chunk(e) * (D / 8) * 128 + (n >> 3) * 128 + (n & 7) * 16);
            const float unit = bc_unit_magic(most_s[n]);
#pragma unroll
            for (int t = 0; t < 3; ++t) {
                uint32_t w[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) w[i] = t == 0 ? bc_lead(x[j][i], unit) : bc_term(x[j][i]);
                *reinterpret_cast<uint4*>(Bt + t * C::kBTerm + off) = make_uint4(w[0], w[1], w[2], w[3]);
            }
        }
    }
    if (warp == 0) tmem_alloc(sm_addr(tmem_slot), C::kTmemCols);
    __syncthreads();
    if (warp == 0) {
        // The different levels in ascending order (of equal ones the first counts), and between neighbours the decision
        // point: the largest v for which the lower one is taken, both distances rounded to float32 as a scan rounds them;
        // equally close, the scan keeps the one it meets first.
        const int n_levels = p.n_levels;
        const float v = cb[lane & 15];
        float other[16];                                           // (entries past the last level repeat it)
#pragma unroll
        for (int j = 0; j < 16; ++j) other[j] = cb[j];
        bool first = lane < n_levels;
#pragma unroll
        for (int j = 0; j < 16; ++j) first = first && !(j < lane && other[j] == v);
        const uint32_t firsts = __ballot_sync(0xffffffffu, first);
        const int n = __popc(firsts);
        int rank = 0;
#pragma unroll
        for (int j = 0; j < 16; ++j) rank += (firsts >> j & 1u) && other[j] < v ? 1 : 0;
        if (first) { sorted[rank] = v; which[rank] = lane; }
        __syncwarp();
        bool good = lane >= n_levels || (v > -1.f && v < 1.f);     // (a NaN is not)
        if (lane < n - 1) good = good && sorted[lane + 1] - sorted[lane] > 1e-5f;
        const bool all_good = __all_sync(0xffffffffu, good), straight = __all_sync(0xffffffffu, !first || rank == lane) && n == n_levels;
        float t = 3.0e38f;                                         // no coordinate reaches it
        if (all_good && lane < n - 1) {
            const float a = sorted[lane], b = sorted[lane + 1];
            const bool lower_first = which[lane] < which[lane + 1];
            int lo = bc_key(a), hi = bc_key(b);                    // the lower level is taken at a, not at b
            while (hi - lo > 1) {
                const int mid = lo + (hi - lo) / 2;
                const float x = bc_unkey(mid), da = x - a, db = b - x;
                if (da < db || (lower_first && da == db)) lo = mid; else hi = mid;
            }
            t = bc_unkey(lo);
        }
        if (lane < 16) thr[lane] = t;
        uint32_t kind = all_good ? kBcTree : kBcScan;
        float magic = 98432.f;
        if (all_good && straight) {
            // the first shift for which every decision point lies alone in its bucket and off its edges
            const bool mine = lane < n - 1;
            bool found = false;
            for (int k = 0; k < 16 && !found; ++k) {
                magic = 98432.f + (float)k * 0.0625f;
                const float at = mine ? t : 0.f;
                const uint32_t b = bc_bucket_bits(at, magic);
                const uint32_t next = __shfl_down_sync(0xffffffffu, b, 1);
                const bool bad = mine && (bc_bucket_bits(at - 4e-6f, magic) != b || bc_bucket_bits(at + 4e-6f, magic) != b ||
                                          (lane + 1 < n - 1 && next == b));
                found = !__any_sync(0xffffffffu, bad);
            }
            if (found) kind = kBcBuckets;
        }
        if (lane == 0) { *kind_s = kind; *magic_s = magic; }
    }
    __syncthreads();
    const float magic1 = *magic_s;
    const uint32_t kind = *kind_s;
    if (kind == kBcBuckets) {
        // a bucket's entry: its decision point (or a number no coordinate reaches) and the count of lower ones,
        // replicated into every index field of a word
        for (int e = tid; e < (int)C::kTabRows * 16; e += C::THREADS) {
            const uint32_t bits = (uint32_t)(e >> 4) << 7;
            float t = 3.0e38f;
            uint32_t cnt = 0;
            for (int i = 0; i < p.n_levels - 1; ++i) {
                const uint32_t tb = bc_bucket_bits(thr[i], magic1);
                if (tb == bits) t = thr[i];
                cnt += tb < bits ? 1u : 0u;
            }
            *reinterpret_cast<uint2*>(zero + C::kTabAddr + (e >> 4) * 128 + (e & 15) * 8) =
                make_uint2(__float_as_uint(t), cnt * 0x11111111u);
        }
    } else if (kind == kBcTree) {
        // row i of 32 copies: 1 to 15 the search tree (children of i: 2 i and 2 i + 1), 16 to 31 the levels' indices
        for (int e = tid; e < 32 * 32; e += C::THREADS) {
            const int i = e >> 5, depth = 31 - __clz(i | 1);
            const uint32_t entry = i >= 16 ? (uint32_t)which[i - 16]
                                           : __float_as_uint(thr[i ? ((2 * (i - (1 << depth)) + 1) << (3 - depth)) - 1 : 0]);
            *reinterpret_cast<uint32_t*>(zero + C::kTabAddr + i * 128 + (e & 31) * 4) = entry;
        }
    }
    fence_async_smem();                                        // B is read by the tensor core through the async proxy
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    const int n_tiles = (p.N + kBcVecs - 1) / kBcVecs;
    const int n_my = (n_tiles - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x;
    bool ok = true;

    if (warp == WORKERS / 32) {
        // ---- MMA warp: every lane runs the loop, lane 0 issues
        constexpr uint32_t idesc = umma_idesc_bf16(D);
        constexpr uint32_t kLbo = (D / 8) * 128;
        constexpr uint32_t b_hi = (128u >> 4) | (1u << 14);    // 8-row groups 128 B apart, no swizzle
        const uint32_t b0 = ((C::kBAddr >> 4) & 0x3FFFu) | ((kLbo >> 4) << 16);
        const uint32_t issue = lane == 0 ? 1u : 0u, acc = tmem_base + C::kAcc;
        for (int i = 0; i < n_my && ok; ++i) {
            const uint32_t b = i & 1, use = (uint32_t)i >> 1;
            ok = mbar_wait(sm_addr(a_full + b), use & 1u, abort_s, 32) && ok;
            if (i >= 1) ok = mbar_wait(sm_addr(acc_free + (b ^ 1)), (uint32_t)((i - 1) >> 1) & 1u, abort_s, 32) && ok;
            if (!ok) break;
            tc_fence_after();
            // (term of x, term of R): the leading products, then the corrections, smallest first
            constexpr int ta[6] = {0, 2, 0, 1, 1, 0}, tb[6] = {0, 0, 2, 1, 0, 1};
#pragma unroll
            for (int t = 0; t < 6; ++t)
#pragma unroll
                for (int ks = 0; ks < D / 16; ++ks)
                    umma_f16_ts_pred(acc + (t ? D : 0), tmem_base + ta[t] * C::kATerm + ks * 8,
                                     b0 + (uint32_t)((tb[t] * C::kBTerm + 2 * ks * kLbo) >> 4), b_hi, idesc,
                                     (t > 1 || ks) ? 1u : 0u, issue);
            umma_commit_pred(sm_addr(mma_done + b), issue);
            __syncwarp();
        }
    } else if (warp == WORKERS / 32 + 1) {
        // ---- copy warp
        int slot = 0;
        uint32_t round = 0;
        for (int i = 0; i < n_my && ok; ++i) {
            const int v0 = ((int)blockIdx.x + i * (int)gridDim.x) * kBcVecs;
            for (int g = 0; g < WG && ok; ++g) {
                if (round) ok = mbar_wait(sm_addr(box_free + slot), (round - 1u) & 1u, abort_s, 32) && ok;
                if (!ok) break;
                if (lane == 0) {
                    mbar_expect_tx(sm_addr(box_full + slot), C::kBox);
                    tma_load_2d(C::kBoxAddr + slot * C::kBox, &x_map, g * 32, v0, sm_addr(box_full + slot));
                }
                __syncwarp();
                if (++slot == NB) { slot = 0; ++round; }
            }
        }
    } else {
        // ---- workers: vector `row` of the tile (= TMEM lane), dims 32 wg .. 32 wg + 31
        const int wg = warp >> 2, q = warp & 3, row = 32 * q + lane;
        const uint32_t tmem_lane = tmem_base + ((uint32_t)(32 * q) << 16);
        const uint32_t lane_copy = (uint32_t)(lane & 15) * 8;
        auto produce = [&](int i) {
            const int n = i * WG + wg, slot = n % NB;
            ok = mbar_wait(sm_addr(box_full + slot), (uint32_t)(n / NB) & 1u, abort_s) && ok;
            float2 x[16];
            const uint32_t r = C::kBoxAddr + slot * C::kBox + row * 128;
#pragma unroll
            for (int c = 0; c < 8; ++c) {
                float4 v;
                asm volatile("ld.shared.v4.f32 {%0,%1,%2,%3}, [%4];\n" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(r + ((c ^ (row & 7)) << 4)));
                x[2 * c] = make_float2(v.x, v.y);
                x[2 * c + 1] = make_float2(v.z, v.w);
            }
            mbar_arrive(sm_addr(box_free + slot));
            // the vector's largest element, from its WG threads (infinities and NaN turn up in the radius)
            float most = fmaxf(fabsf(x[0].x), fabsf(x[0].y));
#pragma unroll
            for (int k = 1; k < 16; ++k) most = fmaxf(most, fmaxf(fabsf(x[k].x), fabsf(x[k].y)));
            float* ms = most_s + (i & 1) * kBcVecs * WG + row * WG;
            ms[wg] = most;
            asm volatile("bar.sync %0, %1;\n" ::"r"(1 + q), "r"(32 * WG) : "memory");
#pragma unroll
            for (int k = 0; k < WG; ++k) most = fmaxf(most, ms[k]);
            const float unit = bc_unit_magic(most);
            if (i >= 1) {                                      // the MMAs of the tile before are done with A
                ok = mbar_wait(sm_addr(mma_done + ((i - 1) & 1)), (uint32_t)((i - 1) >> 1) & 1u, abort_s) && ok;
                tc_fence_after();
            }
#pragma unroll
            for (int t = 0; t < 3; ++t) {
                uint32_t w[16];
#pragma unroll
                for (int k = 0; k < 16; ++k) w[k] = t == 0 ? bc_lead(x[k], unit) : bc_term(x[k]);
                bc_tmem_st16(tmem_lane + t * C::kATerm + wg * 16, w);
            }
            asm volatile("tcgen05.wait::st.sync.aligned;\n" ::: "memory");
            tc_fence_before();
            mbar_arrive(sm_addr(a_full + (i & 1)));
        };
        auto epilogue = [&](int i) -> bool {
            const uint32_t b = i & 1;
            ok = mbar_wait(sm_addr(mma_done + b), (uint32_t)(i >> 1) & 1u, abort_s) && ok;
            tc_fence_after();
            float2 v2[16];
            {
                float2 low[16];
                tmem_ld32(v2, tmem_lane + C::kAcc + wg * 32);
                tmem_ld32(low, tmem_lane + C::kAcc + D + wg * 32);
                tc_fence_before();
                mbar_arrive(sm_addr(acc_free + b));
#pragma unroll
                for (int k = 0; k < 16; ++k) v2[k] = bc_add2(v2[k], low[k]);
            }
            // squares: this thread's 32 as a tree, then the vector's WG parts
            float2 s2[16];
#pragma unroll
            for (int k = 0; k < 16; ++k) s2[k] = bc_mul2(v2[k], v2[k]);
#pragma unroll
            for (int h = 8; h; h >>= 1)
#pragma unroll
                for (int k = 0; k < h; ++k) { s2[k].x = __fadd_rn(s2[k].x, s2[k + h].x); s2[k].y = __fadd_rn(s2[k].y, s2[k + h].y); }
            float* ns = norm_s + (i & 1) * kBcVecs * WG + row * WG;
            ns[wg] = __fadd_rn(s2[0].x, s2[0].y);
            // the barrier also votes: a wait that gave up in one of the group's warps stops all of them here
            if (group_barrier_any(1u + q, 32u * WG, !ok || *abort_s != 0u)) {
                ok = false;
                *abort_s = 1u;
                return false;
            }
            float ss;
            if constexpr (WG == 4) {
                const float4 t = *reinterpret_cast<const float4*>(ns);
                ss = __fadd_rn(__fadd_rn(t.x, t.z), __fadd_rn(t.y, t.w));
            } else {
                const float2 t = *reinterpret_cast<const float2*>(ns);
                ss = __fadd_rn(t.x, t.y);
            }
            const float radius = __fsqrt_rn(ss);
            const int vec = ((int)blockIdx.x + i * (int)gridDim.x) * kBcVecs + row;
            // radii that the FP32 chain has to give: its infinities and NaN are others, and subnormal squares lose bits
            bool odd = !(radius >= 1e-17f && radius <= 1.8e19f);
            if (odd) {
                const float* ms = most_s + (i & 1) * kBcVecs * WG + row * WG;
                float most = ms[0];
#pragma unroll
                for (int k = 1; k < WG; ++k) most = fmaxf(most, ms[k]);
                odd = !(radius == 0.f && most == 0.f);              // (rows of zeros are common)
            }
            const bool live = radius > 1e-30f && radius < 3.4e38f;      // otherwise every direction is 0
            const float dsafe = live ? radius : 1.f;
            // IEEE-rounded quotient from the correctly rounded reciprocal and one residual step (Markstein 1990)
            const float rinv = __frcp_rn(dsafe);
            const float2 rinv2 = make_float2(rinv, rinv), negd2 = make_float2(-dsafe, -dsafe);
            uint32_t packed[4] = {0u, 0u, 0u, 0u};
            float near = 1.f;                              // smallest distance of a coordinate to a decision point
            if (!live) {
#pragma unroll
                for (int k = 0; k < 16; ++k) v2[k] = make_float2(0.f, 0.f);
            }
            if (kind == kBcBuckets) {
                const float2 c128 = make_float2(128.f, 128.f), magic = make_float2(magic1, magic1);
#pragma unroll
                for (int k = 0; k < 16; ++k) {
                    const float2 y = bc_mul2(v2[k], rinv2);
                    const float2 dir = bc_fma2(bc_fma2(y, negd2, v2[k]), rinv2, y);
                    const float2 u = bc_fma2(dir, c128, magic);
#pragma unroll
                    for (int e = 0; e < 2; ++e) {
                        const int j = 2 * k + e, sh = (j * 4) & 31;
                        const uint32_t a = (__float_as_uint(e ? u.y : u.x) & 0xFF80u) | lane_copy;
                        uint2 be;
                        asm volatile("ld.shared.v2.u32 {%0, %1}, [%2 + %3];\n" : "=r"(be.x), "=r"(be.y) : "r"(a), "n"(C::kTabAddr));
                        uint32_t& pw = packed[j >> 3];
                        pw |= be.y & (0xFu << sh);
                        const float off = (e ? dir.y : dir.x) - __uint_as_float(be.x);       // its sign is exact
                        near = fminf(near, fabsf(off));
                        asm("{\n\t.reg .pred p;\n\t"
                            "setp.gt.f32 p, %1, 0f00000000;\n\t"
                            "@p add.u32 %0, %0, %2;\n\t}\n"
                            : "+r"(pw)
                            : "f"(off), "r"(1u << sh));
                    }
                }
            } else if (kind == kBcTree) {
                const uint32_t lane4 = (uint32_t)lane * 4;
#pragma unroll
                for (int k = 0; k < 16; ++k) {
                    const float2 y = bc_mul2(v2[k], rinv2);
                    const float2 dir = bc_fma2(bc_fma2(y, negd2, v2[k]), rinv2, y);
#pragma unroll
                    for (int e = 0; e < 2; ++e) {
                        uint32_t row = 128u, best;
#pragma unroll
                        for (int step = 0; step < 4; ++step) {
                            float t;
                            asm volatile("ld.shared.f32 %0, [%1 + %2];\n" : "=f"(t) : "r"(row | lane4), "n"(C::kTabAddr));
                            const float off = (e ? dir.y : dir.x) - t;                        // its sign is exact
                            near = fminf(near, fabsf(off));
                            row = 2u * row + (off > 0.f ? 128u : 0u);
                        }
                        asm volatile("ld.shared.u32 %0, [%1 + %2];\n" : "=r"(best) : "r"(row | lane4), "n"(C::kTabAddr));
                        packed[k >> 2] |= best << (((2 * k + e) * 4) & 31);
                    }
                }
            } else {
#pragma unroll
                for (int k = 0; k < 16; ++k) {
                    const float dir[2] = {__fdiv_rn(v2[k].x, dsafe), __fdiv_rn(v2[k].y, dsafe)};
#pragma unroll
                    for (int e = 0; e < 2; ++e) {
                        uint32_t best = 0;
                        float dist = 1e30f, second = 1e30f;
                        for (int l = 0; l < p.n_levels; ++l) {
                            const float d = fabsf(dir[e] - cb[l]);
                            if (d < dist) { second = dist; dist = d; best = l; } else { second = fminf(second, d); }
                        }
                        near = fminf(near, 0.5f * (second - dist));
                        packed[k >> 2] |= best << (((2 * k + e) * 4) & 31);
                    }
                }
            }
            if (vec < p.N) {
                if (wg == 0) p.radius_out[vec] = radius;
                *reinterpret_cast<uint4*>(p.packed_out + (size_t)vec * (D / 2) + wg * 16) =
                    make_uint4(packed[0], packed[1], packed[2], packed[3]);
            }
            uint32_t todo = __ballot_sync(0xffffffffu, ((near < kBcNear && live) || odd) && vec < p.N);
            if (todo) {
                int at = 0;
                if (lane == 0) at = atomicAdd(n_list, __popc(todo));
                at = __shfl_sync(0xffffffffu, at, 0);
                const int mine = at + __popc(todo & ((1u << lane) - 1u));
                if ((todo >> lane & 1u) && mine < kBcList) list[mine] = vec * WG + wg;
                todo = __ballot_sync(0xffffffffu, (todo >> lane & 1u) && mine >= kBcList);
                while (todo) {                                 // the list is full: at once
                    const int v = __ffs(todo) - 1;
                    todo &= todo - 1;
                    bc_again<D, false>(p, cb, vec - lane + v, wg);
                }
            }
            return true;
        };
        bool going = true;
        for (int i = 0; i < n_my && going; ++i) {
            produce(i);
            if (i >= 1) going = epilogue(i - 1);
        }
        if (going && n_my >= 1) epilogue(n_my - 1);
        // the second pass: the list is complete, its blocks are stored, and every box has been read
        static_assert((uint32_t)D * D * 4 <= NB * C::kBox, "R fits the boxes");
        const bool stop = group_barrier_any(9u, WORKERS, !ok || *abort_s != 0u);
        const int n = min(*n_list, kBcList);
        if (n > 0 && !stop) {
#pragma unroll 8
            for (int e = tid; e < D * D; e += WORKERS)
                *reinterpret_cast<float*>(zero + C::kBoxAddr + bc_staged<D>(e / D, e % D)) = __ldg(p.R + e);
            asm volatile("bar.sync 9, %0;\n" ::"r"(WORKERS) : "memory");
            for (int e = warp; e < n; e += WORKERS / 32) bc_again<D, true>(p, cb, list[e] / WG, list[e] % WG);
        }
    }
    if (!ok && lane == 0) { *abort_s = 1u; atomicOr(&g_bridge_compress_error, 1u); }
    if (*abort_s && tid == 0) {                                // give box copies still in flight time to land
        const long long t0 = clock64();
        while (clock64() - t0 < (1ll << 20)) {}
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) tmem_dealloc(tmem_base, C::kTmemCols);
}

// ------------------------------------------------------------------ host side
bool bridge_compress_fits(int D, const float* input, const float* rotation, const uint8_t* packed) {
    // a tensor map's base and 16-byte stores; the rotation is read in pairs
    return (D == 64 || D == 128) && (reinterpret_cast<uintptr_t>(input) & 15) == 0 &&
           (reinterpret_cast<uintptr_t>(rotation) & 7) == 0 && (reinterpret_cast<uintptr_t>(packed) & 15) == 0;
}

template <int D>
static cudaError_t launch_bridge_compress(const float* input, const BridgeCompressParams& p, int sms, cudaStream_t st) {
    using C = BridgeCompressCfg<D>;
    CUtensorMap map;
    const cuuint64_t dims[2] = {(cuuint64_t)D, (cuuint64_t)p.N}, strides[1] = {(cuuint64_t)D * 4};
    const cuuint32_t box[2] = {32u, (cuuint32_t)kBcVecs};
    if (!encode_tensor_map_2d(&map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, input, dims, strides, box)) return cudaErrorInvalidValue;
    auto kern = bridge_compress_kernel<D>;
    static std::atomic<uint64_t> allowed{0};
    const cudaError_t e = allow_shared(kern, C::smem_bytes(), allowed);
    if (e != cudaSuccess) return e;
    const int n_tiles = (p.N + kBcVecs - 1) / kBcVecs;
    kern<<<n_tiles < sms ? n_tiles : sms, C::THREADS, C::smem_bytes(), st>>>(p, map);
    return cudaGetLastError();
}

cudaError_t bridge_compress_launch(const float* input, const float* rotation, const float* codebook, float* radius_out,
                                   uint8_t* packed_out, int N, int D, int n_levels, int sms, cudaStream_t st) {
    BridgeCompressParams p{rotation, codebook, radius_out, packed_out, input, N, n_levels};
    return D == 64 ? launch_bridge_compress<64>(input, p, sms, st) : launch_bridge_compress<128>(input, p, sms, st);
}

int bridge_compress_error_flags(unsigned int* flags) {
    unsigned int v = 0, zero = 0;
    if (cudaMemcpyFromSymbol(&v, g_bridge_compress_error, sizeof(v)) != cudaSuccess) return PQ_ERR_CUDA;
    if (v && cudaMemcpyToSymbol(g_bridge_compress_error, &zero, sizeof(zero)) != cudaSuccess) return PQ_ERR_CUDA;
    *flags = v;
    return PQ_OK;
}

}  // namespace pq
