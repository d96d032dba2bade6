// Dense f32 attention in tiles (attention_f32.cu).
#pragma once

#include <type_traits>

#include "common.cuh"

namespace singe {

// Queries [batch, heads, query_len, head_dim] and keys, values [batch, kv_heads, key_len, head_dim] under any strides of
// batch, head and row; `out` has the queries' strides, `lse` is [batch, heads, query_len].
struct DenseF32 {
    const float *query;
    float *out;
    float *lse;          // or nullptr
    const float *key;
    const float *value;
    const float *sinks;  // [heads] or nullptr
    int heads, kv_heads, query_len, key_len, head_dim, causal;
    long long window;
    long long q_batch, q_head, q_row, k_batch, k_head, k_row;
    float scale, softcap;
};

// Fewer rows a head than this leave most of a tile empty: one warp per row is the better split then (512 heads of 64:
// 8 rows 8.6 us against 15.8, 16 rows 23.3 against 16.1).
constexpr int kDenseF32LeastRows = 16;

bool dense_attention_f32_takes(const DenseF32 &p, size_t batch);
int dense_attention_f32(cudaStream_t stream, const DenseF32 &p, size_t batch);

}  // namespace singe
