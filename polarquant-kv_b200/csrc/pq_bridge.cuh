// What the files behind the llama.cpp bridge's entry points share.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace pq {

// Arguments of the bridge's attention kernels (see polarquant_fused_attention_cuda_c).
struct BridgeAttnParams {
    const float* q;
    const uint8_t* pk;
    const float* kr;
    const uint8_t* pv;
    const float* vr;
    const float* codebook;
    float* out;
    float* partials;          // records of the slices, [total_q_heads][n_split][2 + padded D], used when n_split > 1
    unsigned* tickets;        // [total_kv_heads * groups], zero between launches
    int gqa, S, D, n_levels, n_split, tiles_per_split;
    float scale;
    int vector_loads;         // rows start on a multiple of the lane's byte count
};

// pq_bridge_attn.cu: head dims 64 and 128, packed rows on 16-byte boundaries.
bool bridge_attention_fits(int D, const void* packed_k, const void* packed_v);
// Splits every (kv head, query group) over CTAs; fills p.n_split, p.tiles_per_split.  Returns the number of groups.
int bridge_attention_plan(BridgeAttnParams& p, int total_kv_heads, int sms, size_t ws_floats, int ws_tickets,
                          int total_q_heads);
cudaError_t bridge_attention_launch(const BridgeAttnParams& p, int total_kv_heads, int groups, cudaStream_t st);
// bit 0: a bounded wait for a tile copy gave up; bit 1: the shared-memory window started too high
int bridge_error_flags(unsigned int* flags);

// pq_bridge_compress.cu: head dims 64 and 128, aligned buffers.
bool bridge_compress_fits(int D, const float* input, const float* rotation, const uint8_t* packed);
cudaError_t bridge_compress_launch(const float* input, const float* rotation, const float* codebook, float* radius_out,
                                   uint8_t* packed_out, int N, int D, int n_levels, int sms, cudaStream_t st);
// the same bits as bridge_error_flags
int bridge_compress_error_flags(unsigned int* flags);

}  // namespace pq
