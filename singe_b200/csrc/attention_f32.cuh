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
// 8 rows 8.6 us against 15.8).  16 rows over 256 keys take a fifth of its time or less at 4 - 512 heads of 4 - 128 columns;
// over 16 keys the two are near each other (us in tiles and by warps, 4 - 128 heads: of 4 columns 8.0 - 8.2 and 9.1 - 12.8, of 64
// 8.0 - 8.2 and 13.3 - 15.1; 512 heads: of 4 26.3 and 23.6, of 64 26.1 and 29.0, of 96 40.1 and 32.9), over 24 no longer.
constexpr int kDenseF32LeastRows = 16;

bool dense_attention_f32_takes(const DenseF32 &p, size_t batch);
int dense_attention_f32(cudaStream_t stream, const DenseF32 &p, size_t batch);

}  // namespace singe
