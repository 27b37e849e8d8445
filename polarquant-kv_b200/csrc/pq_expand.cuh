// The expanded form of a stored cache that the prefill kernel contracts: one record per (kv row, 64-token tile).
#pragma once

#include "pq_common.cuh"

namespace pq {

constexpr int kExpTok = 64;                                  // tokens per record

// A record: K hi | K lo rows stacked per 64 dims (128 rows of 128 bytes), V hi tile, V lo tile (64 rows of 128 bytes per
// 64 dims) - float16 terms of keys and values in the ORIGINAL space (rotated back), 128-byte-swizzled as they sit in
// shared memory; then per token: the factor of its score column, the factor of its weight (a power of two), and the
// largest weight factor of each half of the tile.
template <int D>
struct ExpandRec {
    static constexpr uint32_t kTerm = kExpTok * D * 2;       // one term of K or V
    static constexpr uint32_t kFactors = 4 * kTerm;          // 64 score factors, 64 weight factors, 4 floats (2 used)
    static constexpr uint32_t kBytes = 4 * kTerm + 2 * kExpTok * 4 + 32;
};
constexpr float kExpScale = 1024.0f;                         // terms hold 1024 * value / weight factor

struct ExpandArgs {
    const uint8_t* kb;
    const uint8_t* vb;
    const float* rot;
    uint8_t* ws;
    int64_t S, Scap;
    int rows;
    float score_scale;                                       // softmax scale * log2(e)
    const float* codebook_k;                                 // HOST tables
    const float* codebook_v;
};
// Both operands; one launch when their widths agree, two otherwise.  Returns a pq_status.
int expand_launch(const ExpandArgs& a, int head_dim, int k_bits, int v_bits, cudaStream_t st);

}  // namespace pq
