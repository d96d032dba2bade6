// What the flash-decode kernels over paged caches share: their parameters, the rotation of query fragments and the view a
// query has of its chunk.
#pragma once

#include "common.cuh"

namespace singe {

constexpr int kPageTokens = 16;
constexpr int kHalfBytes = kPageTokens * 128;  // one TMA box: 16 rows x 128 bytes

struct DecodeParams {
    void *out;            // [batch, heads, head_dim] in the cache dtype, or nullptr (partials only)
    float *attn_partial;  // [batch, heads, max_splits, head_dim]
    float *lse_partial;   // [batch, heads, max_splits]
    const void *query;    // [batch, heads, head_dim]
    const int32_t *lens;
    const uint32_t *table;
    int batch;
    int heads;
    int kv_heads;
    int group;
    int physical_blocks;
    int table_stride;
    int split_tokens;  // multiple of 16
    int max_splits;
    int partials_only;  // 1: every split slot is written, nothing goes to `out`
    float scale_log2;   // scale * log2(e)
    uint32_t *status;
};

// What only a decode step passes (the EXTRAS forms of the kernel).  It is a kernel argument of its own: the plain and
// ragged kernels do not carry it, and measurably so -- with these fields inside DecodeParams the plain kernel's
// registers were allotted differently and config 2 took 0.6 us longer.
struct StepExtras {
    int stable_paging;  // 1: lengths, block table and every cached row but each sequence's last key position are not
                        //    written by work still in flight (SINGE_HINT_STABLE_PAGING): they are read ahead of the
                        //    wait on the preceding kernels
    int early_release;  // 1: the grid fits the machine in one wave, so the next kernel may become resident at once
    int prefetch_pages; // with stable_paging: pages beyond the ring pulled into L2 ahead of the wait
    WarmRange warm;     // pulled into L2 beside the kernel's own work (classic form only)
    // Fused step form (FUSED): the kernel reads the step's un-rotated projections itself, rotates Q and the new K row,
    // writes the new K/V rows into the cache and attends over the cached keys plus the new one.
    const void *qkv;          // [batch, qkv_stride]: heads*D query | kv_heads*D key | kv_heads*D value projections
    long long qkv_stride;     // elements
    void *key_rows;           // the caches as plain pointers, for the one row this step adds per sequence and KV head
    void *value_rows;
    const void *write_pages;  // [batch] int32 / int64 (rope_index_width)
    const void *write_slots;
    uint32_t *tickets;  // [batch, kv_heads], zero between launches, or nullptr.  With tickets the split that finishes
                        // a row last folds the row's partials itself and no combine kernel follows (classic form)
    // Rotation of the queries inside the kernel (rope_cos == nullptr: the queries arrive rotated)
    const void *rope_cos;        // [capacity, head_dim / 2] in the cache dtype
    const void *rope_sin;
    const void *rope_positions;  // [batch] position of each sequence's query token, int32 or int64
    int rope_index_width;        // 4 or 8
    int rope_capacity;
    const void *query_gain;      // per-head RMSNorm before the rotation: gain [head_dim] or nullptr
    int query_norm;              // 1: normalise
    float query_norm_eps;
};

__device__ __forceinline__ float fast_tanh(float x) {
    float y;
    asm("tanh.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

__device__ __forceinline__ float fast_exp2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// Rotates (and first, if asked, RMS-normalises) the query fragments a lane holds, in registers.  A lane of row
// `row` (a query head of the group) and quad q holds, for every 16-wide k step ks, the elements ks*16 + 2q, +1
// (qa[ks][0]) and ks*16 + 8 + 2q, +1 (qa[ks][1]): an element of the head's first half and its partner half a head
// further on sit in the same slot of steps ks and ks + KSTEPS/2, so the half-split rotation needs no exchange.
// Rounding follows the tensor-op chain of the separate kernel (singe_rotary_cache_write_bf16): every product and every
// sum is rounded to the cache dtype, so attention over queries rotated here equals attention over queries rotated there.
// Replaces the query stage of singe_rotary_paged_attention
// (singe/src/backend/cuda/kernel_plan/source/paged_attention.rs:881-977, QueryRotation).
template <typename T, int HD>
__device__ __forceinline__ void rotate_query_fragments(uint32_t (&qa)[HD / 16][2], const DecodeParams &p,
                                                       const StepExtras &x, int b, int row,
                                                       int quad, bool may_normalise = true) {
    constexpr int KSTEPS = HD / 16;
    constexpr int HALF_STEPS = KSTEPS / 2;
    long long position = x.rope_index_width == 8 ? static_cast<const long long *>(x.rope_positions)[b]
                                                 : static_cast<long long>(static_cast<const int *>(x.rope_positions)[b]);
    if (position < 0) position += x.rope_capacity;
    if (position < 0 || position >= x.rope_capacity) {
        report_status(p.status, kStatusIndexOutOfBounds);
        position = 0;
    }
    auto low = [](uint32_t word) {
        T value;
        *reinterpret_cast<uint16_t *>(&value) = static_cast<uint16_t>(word & 0xffffu);
        return to_float<T>(value);
    };
    auto high = [](uint32_t word) {
        T value;
        *reinterpret_cast<uint16_t *>(&value) = static_cast<uint16_t>(word >> 16);
        return to_float<T>(value);
    };
    auto rounded = [](float value) { return to_float<T>(from_float<T>(value)); };
    if (x.query_norm && may_normalise) {
        float squares = 0.0f;
#pragma unroll
        for (int ks = 0; ks < KSTEPS; ++ks) {
#pragma unroll
            for (int j = 0; j < 2; ++j) squares += low(qa[ks][j]) * low(qa[ks][j]) + high(qa[ks][j]) * high(qa[ks][j]);
        }
        squares += __shfl_xor_sync(0xffffffffu, squares, 1);
        squares += __shfl_xor_sync(0xffffffffu, squares, 2);
        const float scale = 1.0f / sqrtf(squares / static_cast<float>(HD) + x.query_norm_eps);
        const uint32_t *gain = static_cast<const uint32_t *>(x.query_gain);
#pragma unroll
        for (int ks = 0; ks < KSTEPS; ++ks) {
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                const uint32_t g = gain != nullptr ? gain[ks * 8 + j * 4 + quad] : 0u;
                const float g_low = gain != nullptr ? low(g) : 1.0f;
                const float g_high = gain != nullptr ? high(g) : 1.0f;
                qa[ks][j] = pack2<T>(low(qa[ks][j]) * scale * g_low, high(qa[ks][j]) * scale * g_high);
            }
        }
    }
    const uint32_t *cos_row = static_cast<const uint32_t *>(x.rope_cos) + position * (HD / 4);
    const uint32_t *sin_row = static_cast<const uint32_t *>(x.rope_sin) + position * (HD / 4);
    (void)row;
#pragma unroll
    for (int ks = 0; ks < HALF_STEPS; ++ks) {
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            const uint32_t c = cos_row[ks * 8 + j * 4 + quad];   // pairs ks*16 + 8j + 2q, +1
            const uint32_t s = sin_row[ks * 8 + j * 4 + quad];
            const uint32_t first = qa[ks][j], second = qa[ks + HALF_STEPS][j];
            const float f0 = low(first), f1 = high(first), s0 = low(second), s1 = high(second);
            qa[ks][j] = pack2<T>(rounded(f0 * low(c)) - rounded(s0 * low(s)), rounded(f1 * high(c)) - rounded(s1 * high(s)));
            qa[ks + HALF_STEPS][j] =
                pack2<T>(rounded(s0 * low(c)) + rounded(f0 * low(s)), rounded(s1 * high(c)) + rounded(f1 * high(s)));
        }
    }
}

// FUSED: the key and value a step adds to sequence b, KV head g: rotates K, puts both rows into the cache and attends the new
// key.  One warp, whose lanes hold the query fragments and the accumulator.
template <typename T, int HD>
__device__ __forceinline__ void add_new_key(const DecodeParams &p, const StepExtras &x, const uint32_t (&qa)[HD / 16][2],
                                            float (&o)[HD / 8][4], float &run_max, float &run_sum, int b, int g, int row, int quad,
                                            int lane) {
    constexpr int KSTEPS = HD / 16;
    constexpr int NTILES = HD / 8;
    const T *projections = static_cast<const T *>(x.qkv) + static_cast<size_t>(b) * x.qkv_stride;
    const uint32_t *k32 = reinterpret_cast<const uint32_t *>(projections + static_cast<size_t>(p.heads + g) * HD);
    const uint32_t *v32 =
        reinterpret_cast<const uint32_t *>(projections + static_cast<size_t>(p.heads + p.kv_heads + g) * HD);
    long long page = x.rope_index_width == 8 ? static_cast<const long long *>(x.write_pages)[b]
                                             : static_cast<long long>(static_cast<const int *>(x.write_pages)[b]);
    long long slot = x.rope_index_width == 8 ? static_cast<const long long *>(x.write_slots)[b]
                                             : static_cast<long long>(static_cast<const int *>(x.write_slots)[b]);
    if (page < 0) page += p.physical_blocks;
    if (slot < 0) slot += kPageTokens;
    const bool slot_ok = page >= 0 && page < p.physical_blocks && slot >= 0 && slot < kPageTokens;
    if (!slot_ok && lane == 0) report_status(p.status, kStatusIndexOutOfBounds);
    const size_t cache_row = ((static_cast<size_t>(slot_ok ? page : 0) * kPageTokens + (slot_ok ? slot : 0)) *
                                  p.kv_heads + g) * HD;
    uint32_t *k_out = reinterpret_cast<uint32_t *>(static_cast<T *>(x.key_rows) + cache_row);
    uint32_t *v_out = reinterpret_cast<uint32_t *>(static_cast<T *>(x.value_rows) + cache_row);
    uint32_t kf[KSTEPS][2];
#pragma unroll
    for (int ks = 0; ks < KSTEPS; ++ks) {
        kf[ks][0] = k32[ks * 8 + quad];
        kf[ks][1] = k32[ks * 8 + 4 + quad];
    }
    rotate_query_fragments<T, HD>(kf, p, x, b, row, quad, false);   // the same rotation, without the query's norm
    auto low = [](uint32_t word) {
        T value;
        *reinterpret_cast<uint16_t *>(&value) = static_cast<uint16_t>(word & 0xffffu);
        return to_float<T>(value);
    };
    auto high = [](uint32_t word) {
        T value;
        *reinterpret_cast<uint16_t *>(&value) = static_cast<uint16_t>(word >> 16);
        return to_float<T>(value);
    };
    float dot = 0.0f;
#pragma unroll
    for (int ks = 0; ks < KSTEPS; ++ks) {
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            dot = fmaf(low(qa[ks][j]), low(kf[ks][j]), dot);
            dot = fmaf(high(qa[ks][j]), high(kf[ks][j]), dot);
            if (row == 0 && slot_ok) k_out[ks * 8 + j * 4 + quad] = kf[ks][j];   // lanes 0-3 hold the whole row
        }
    }
    dot += __shfl_xor_sync(0xffffffffu, dot, 1);
    dot += __shfl_xor_sync(0xffffffffu, dot, 2);
    if (slot_ok && lane < HD / 2) v_out[lane] = v32[lane];   // HD / 2 words
    if (HD / 2 > 32 && slot_ok) v_out[lane + 32] = v32[lane + 32];
    const float score = dot * p.scale_log2;
    const float next_max = fmaxf(run_max, score);
    const float correction = fast_exp2(run_max - next_max);
    const float weight = fast_exp2(score - next_max);
    run_max = next_max;
    run_sum = run_sum * correction + (quad == 0 ? weight : 0.0f);   // the quad's sums are added up below
    // the weight takes the rounding the split grid's tensor-core path gives P (the even form's cached keys have two terms)
    T packed_weight = from_float<T>(weight);
    const float rounded_weight = to_float<T>(packed_weight);
#pragma unroll
    for (int nt = 0; nt < NTILES; ++nt) {
        const uint32_t value = v32[nt * 4 + quad];   // columns nt*8 + 2*quad, +1
        o[nt][0] = o[nt][0] * correction + rounded_weight * low(value);
        o[nt][1] = o[nt][1] * correction + rounded_weight * high(value);
    }
}

// What a query of the chunked form reads: the sequence's pages from first_page on, `keys` of them counted from that page's
// first slot, of which the first `hidden` belong to the chunk before.
struct ChunkView {
    int sequence, first_page, keys, hidden;
};

__device__ __forceinline__ ChunkView chunk_view(const ChunkedDecode &chunked, int query, int len, int table_stride, uint32_t *status) {
    ChunkView view = {chunked.sequence_of[query], 0, 0, 0};
    if (view.sequence < 0 || view.sequence >= chunked.sequences || len > table_stride * kPageTokens) {
        if (threadIdx.x == 0) report_status(status, kStatusIndexOutOfBounds);
        view.sequence = 0;
        return view;
    }
    if (len <= 0) return view;
    const int start = (len - 1) / chunked.size * chunked.size;
    view.first_page = start / kPageTokens;
    view.hidden = start - view.first_page * kPageTokens;
    view.keys = len - view.first_page * kPageTokens;
    return view;
}

// paged_decode_even.cu
size_t paged_decode_even_slots(size_t batch, size_t heads, size_t kv_heads, size_t head_dim, size_t bound);
int paged_decode_even(cudaStream_t stream, int element, const DecodeParams &params, const StepExtras &extras, const void *key_cache,
                      const void *value_cache, size_t head_dim, size_t slots);
int paged_decode_even_chunked(cudaStream_t stream, const DecodeParams &params, const ChunkedDecode &chunked, const void *key_cache,
                              const void *value_cache, size_t head_dim, size_t slots);

}  // namespace singe
