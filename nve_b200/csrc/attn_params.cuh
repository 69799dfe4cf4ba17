// Launch parameters of the decode attention kernels (attn_decode.cu, attn_decode_mma.cu, attn_stream_mma.cu, attn_prefill_mma.cu, attn_prefill_tc.cu).
#pragma once
#include "common.cuh"
#include "gemm_w4a16.cuh"

namespace nve {

struct AttnParams {
    const uint16_t* q;        // [nh, hd]
    const uint16_t* k_new;    // [nkv, hd] (fused form)
    const uint16_t* v_new;    // [nkv, hd]
    uint16_t* k_cache;        // [nkv, kv_stride, hd]
    uint16_t* v_cache;
    const uint16_t* cos_tab;  // [max_seq, hd/2]
    const uint16_t* sin_tab;
    const int* d_pos;         // fused form: position of the new token
    const int* d_seq_len;     // valid length (device scalar) or NULL
    int seq_len;              // valid length when d_seq_len == NULL
    uint16_t* out;            // [nh, hd] f16
    int8_t* out_q;            // optional int8 codes of out, group 32
    float* out_scales;        // [nh*hd/32]
    int num_heads, num_kv_heads, kv_stride;
    float scale;
    // un-fused form only: blockIdx.y selects one of `rows` query rows; row r reads q + r * row_stride, writes
    // out + r * row_stride and attends to seq_len + r positions (causal attention over a block of new positions)
    int rows, row_stride;
    // batched fused form, streaming kernel: q, k and v may be a product whose segments are not summed yet
    PairLeft left;
    // batched fused form: `rows` independent sequences; elements between consecutive K (or V) caches
    long long cache_stride;
};

// attn_stream_mma.cu: fused (`rows` independent sequences with RoPE and the K/V write inside) or plain form, positions split
// over clusters chosen for the grid; false when the shape is not covered (the caller then uses another kernel).
bool attn_stream_mma_try(const AttnParams& p, int head_dim, cudaStream_t st, cudaError_t& err, bool fused = true);

// attn_prefill_mma.cu: the causal block described above, in tiles of query rows; false when the shape is not covered.
bool attn_prefill_mma_try(const AttnParams& p, int head_dim, cudaStream_t st, cudaError_t& err);

// attn_prefill_tc.cu: the same in tiles of 128 query rows on tcgen05; false: not its shapes, or too few of them.
bool attn_prefill_tc_try(const AttnParams& p, int head_dim, cudaStream_t st, cudaError_t& err);

// attn_decode_mma.cu: decode attention of one sequence (or query row) on the tensor cores, built for latency; false when the
// shape is not covered.
bool attn_decode_mma_try(const AttnParams& p, int head_dim, cudaStream_t st, cudaError_t& err, bool fused = true);

}  // namespace nve
