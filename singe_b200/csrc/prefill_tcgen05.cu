// Packed variable-length flash-attention prefill on the tcgen05 tensor core (bf16 or f16, head_dim 128, GQA).
//
// Meaning: ragged_kv_prefill_attention (singe-kernel/src/cpu/attention.rs:1343-1420): sequence b owns query
// tokens [offsets[b], offsets[b] + lens_q[b]) and key rows [offsets[b], offsets[b] + lens_kv[b]) of the packed
// tensors; causal hides key_index > query_index (sequence-local); out [T, H, D] and a natural-log LSE [T, H],
// -1.0e20 for a row that sees no key.  Replaces singe_tcgen05_attention
// (singe/src/backend/cuda/kernel_plan/source/tcgen05_attention.rs:76-258), which is single-stage, cp.async-fed and
// rescales the output through tensor memory on every tile.
//
// One CTA = 256 consecutive query rows of one (sequence, head), handled as two 128-row tiles A and B that take
// turns on the tensor core, so the softmax of one tile runs while the other tile's MMAs execute.  Roles:
//   warps 0-3  softmax of tile A, one thread per query row (= tensor-memory lane); warps 4-7 the same for tile B.
//              The softmax is the bottleneck next to the MMAs (instruction issue and the 16 exp2 per clock of the
//              special-function unit), so its steady state is a single pass with as few instructions per score as
//              possible: scores come out of tensor memory 32 columns at a time (the next load in flight while the
//              current chunk is processed), p = exp2(s * scale - base) as packed f32x2 arithmetic, the row sum,
//              the bf16 pack, and P goes back over S with tcgen05.st.  No row maximum is taken: `base` only has to
//              keep the numbers in range, the result does not depend on it (out = O / sum, LSE = base +
//              log2(sum)).  The first key tile takes the exact row maximum as base (a two-pass tile); afterwards
//              the row is re-based by an exact power of two whenever its running sum passes 2^16 (O in tensor
//              memory and the sum are scaled, at the start of the next tile, when the previous P V has retired).
//              A row whose scores jump by more than ~2^64 from one key tile to the next would overflow this
//              scheme.  Such a row gets a NaN as its LSE and raises a sticky per-device flag; the second launch of
//              the same kernel in SAFE mode, where every tile takes its exact row maximum first, leaves at once
//              while the flag has never been raised, and otherwise finds the marked items among its share and
//              recomputes exactly those.
//   warp 8     MMA issuer and tensor-memory owner.  Issue order per key tile j:
//                 PV_A(j), QK_A(j+1), PV_B(j), QK_B(j+1)
//              (P V in two halves of the keys, each as soon as its weights are there: a tile's softmax, P V and Q K^T are a chain, and
//              the first half's products come off it.  8192 + 4096 + 2048 + 1024 tokens 745 -> 721 us at the power limit, 613 -> 605 at full clocks)
//              (S = Q K^T: 8 x tcgen05.mma 128x128x16, both operands K-major in shared memory; O += P V: 8 x
//              tcgen05.mma with P read from tensor memory and V MN-major), so softmax_A(j) overlaps PV_B(j-1) and
//              QK_B(j), softmax_B(j) overlaps PV_A(j) and QK_A(j+1).
//   warps 9,10 TMA producers: both Q tiles once and K tiles, V tiles of paged keys (128 keys x 128 dims, two SWIZZLE_128B boxes
//              each) into two stages each, released by tcgen05.commit when the MMAs that read them retire.  One warp for
//              both let the next K tile wait for the last V tile's stage: a lone tile over paged keys took 1.7 us a key
//              tile and takes 1.3.  Ragged keys, two boxes a tile, are 0.6 % faster with one warp.
// Tensor memory (all 512 columns): S_A/P_A [0,128), S_B/P_B [128,256), O_A [256,384), O_B [384,512).
// Shared memory: Q_A, Q_B, 2 x K, 2 x V tiles of 32 KB = 192 KB.
// Under a causal mask tile A sees one key tile less than tile B; CTAs are dispatched heaviest-first.
// WINDOW: a query sees itself and the window - 1 keys before it.  A tile starts at the key tile where its first row begins
// to see; a row whose first visible key lies in a later tile takes its base from that tile.
// Keys have offsets and a row stride of their own, and the epilogue may gate a head's rows by a sigmoid.
// TENSOR: the Tensor surface's paged attention (see TensorPaging).  A row is a (token, head) pair of one key/value head's
// group, so that a sequence's few new tokens share one pass over its keys, and the value product takes the
// probabilities as two bf16 terms hi + lo, 16 - 17 bits of them: the general kernel has them in f32.  Log sums take them in f32.
// Every mbarrier wait is bounded; on a timeout the CTA records status 2, frees tensor memory and leaves.
#include <type_traits>

#include "common.cuh"
#include "tcgen05.cuh"

namespace singe {

namespace {

constexpr int kPrefillThreads = 352;
constexpr int kTile = 128;           // rows of one query tile, and keys per key tile
constexpr int kPair = 2 * kTile;     // query rows per CTA
constexpr int kChunk = 32;           // score columns taken out of tensor memory at a time
constexpr int kHalfTileBytes = kTile * 128;       // one TMA box: 128 rows x 128 bytes
constexpr int kTileBytes = 2 * kHalfTileBytes;    // 32 KB
constexpr int kPageTokens = 16;                   // paged form: tokens per cache page
constexpr int kPageBytes = kPageTokens * 128;     // one page box: 16 rows x 128 bytes
constexpr int kMaxRankTiles = 1024;               // heaviest-first dispatch: sequences up to 256 Ki tokens
constexpr float kRescaleThreshold = 8.0f;         // two-pass tiles: re-base when the max grew by 2^8 (log2 units)
constexpr float kRebaseLimit = 65536.0f;          // single-pass tiles: re-base a row when its sum passes 2^16
constexpr float kOverflowLimit = 1.8446744e19f;   // 2^64: beyond this the CTA is redone in SAFE mode
constexpr int kRedoCapacity = 2048;               // marked items one CTA lists; past that it redoes its whole share

// Raised (never lowered) by the first launch when a row leaves the single-pass range.  While it is zero the second
// launch has nothing to look for; once it is set every later call pays the scan of the LSE marks.
__device__ unsigned g_out_of_range_seen = 0;

struct PrefillParams {
    void *out;
    float *lse;
    const int32_t *lens_q;    // nullptr: the dense form, every sequence has uniform_q queries and uniform_kv keys,
    const int32_t *lens_kv;   //          sequence b starts at row b * uniform_q (queries) / b * uniform_kv (keys)
    const int32_t *offsets;
    int uniform_q;
    int uniform_kv;
    int lse_rows;   // 0: LSE is [total_q, heads] (packed forms); > 0: [batch, heads, lse_rows] (fmha_prefill_lse)
    int exact;      // 1: the exact-maximum launch walks every item (16-bit floats whose range the single-pass
                    // softmax would leave); 0: it only redoes what the first launch marked
    int batch;
    int heads;
    int kv_heads;
    int total_q;
    int total_kv;
    // paged form: keys and values live in a cache [pages, 16, kv_heads, 128] behind a block table [batch, table_stride]
    const uint32_t *block_table;
    int table_stride;
    int cache_pages;
    int causal;     // 0: none; 1: key index > query index hidden (sequence-local, the kernel surface's mask);
                    // 2: the queries are the sequence's last tokens (query i sits at position len_kv - len_q + i)
    float scale_log2;
    uint32_t *error;
    // windowed form
    int window;
    const int32_t *offsets_kv;
    const __nv_bfloat16 *gate;  // nullptr, or row t of head h is multiplied by sigmoid(gate[t * gate_stride + h])
    long long gate_stride;
};

// The Tensor surface's paging tensors (Tensor::paged_attention, singe/src/tensor/neural.rs:405-457), read as the caller
// gave them: query_offsets and page_offsets [sequences + 1], pages [table_len], last_page_lengths [sequences], 32- or
// 64-bit.  Every CTA checks all of them at its start and lists the sequences in shared memory; a sequence with a value
// out of range gets no work here, and the kernel that follows (left_rows_kernel) computes what can be computed of it.  It
// also does rows over that this one marks with a NaN as their LSE: rows that leave the single-pass range, and rows whose
// output is not finite (a hidden key's value may be anything, and zero times infinity is not zero).
// Bound by the tensor core and the special-function unit alike: 8 + 16 MMAs of 128 x 128 x 16 and 16384 exponentials a
// key tile.  One step of four 510-token chunks and 28 decoding sequences behind 0 - 3000 tokens of context, 32 query heads on 8:
// 150 us with the rows behind; 158 before the items were decoded ahead, 175 before one thread issued the MMAs and the weights came in halves, 238 with items in order of their pair
// index and lone tiles a key tile at a time, 40.2 ms by one warp per row and head.
// Against 64 bits, this step and twelve of other sizes: outputs 1.6585e-3 off by either kernel, which is their rounding to bf16
// (the squares of the two errors differ by 4e-6 squared: two terms, and long sums in the tensor core); log sums 5.6e-8, by the
// general kernel 6.3e-8.
// A pair's key tile has 3072 clk of MMA, and a tile's softmax and Q K^T are a chain; a lone tile's step took 3000 in this mix, whose cold
// cache all SMs read at once.
struct TensorPaging {
    const void *query_offsets;
    const void *page_offsets;
    const void *pages;
    const void *last_page_lengths;
    int index_width;   // 4 or 8
    int sequences;
    int tokens;
    int table_len;
    int pack;          // log2 of the query heads whose rows stand together; p.heads counts such packs
    uint32_t *status;
};
struct NoPaging {};

constexpr int kMaxTensorSequences = 1024;
constexpr int kTensorBarriers = 24;  // (one of them only keeps what follows aligned)
constexpr int kMaxOrdered = 1024;   // (sequence, pair) entries that are put in order of their cost

__device__ __forceinline__ long long paging_value(const void *list, int width, int at) {
    return width == 8 ? static_cast<const long long *>(list)[at] : static_cast<const int *>(list)[at];
}

// Per sequence: rows (tokens << pack), keys, first token, first place in the page list.
struct SequenceTable {
    int *rows, *keys, *first_token, *first_page;
};

// Fills the table; every thread of the CTA takes part.  Query offsets that run backwards would have two sequences own a
// token: then the whole call is left to the general kernel, which gives it to the first.
__device__ __forceinline__ void list_sequences(const TensorPaging &g, int cache_pages, const SequenceTable &table, int warp, int lane) {
    // A lane reads the offsets of one sequence, then the warp goes through its sequences' pages with several loads in
    // flight: one load after the other, the pages of 32 sequences took each CTA some 10 us.
    constexpr int kWarps = kPrefillThreads / 32, kFlight = 4;
    bool backwards = false;
    for (int base = warp; base < g.sequences; base += 32 * kWarps) {
        const int own = base + lane * kWarps;
        long long qf = 0, ql = 0, pf = 0, pl = 0, keys = 0;
        bool bad = false;
        if (own < g.sequences) {
            qf = paging_value(g.query_offsets, g.index_width, own);
            ql = paging_value(g.query_offsets, g.index_width, own + 1);
            pf = paging_value(g.page_offsets, g.index_width, own);
            pl = paging_value(g.page_offsets, g.index_width, own + 1);
            const long long last = paging_value(g.last_page_lengths, g.index_width, own);
            bad = !(0 <= qf && qf <= ql && ql <= g.tokens);
            backwards |= bad;
            bad |= !(0 <= pf && pf <= pl && pl <= g.table_len);
            if (!bad && pf != pl) {
                bad = last < 0 || last > kPageTokens;
                keys = (pl - pf - 1) * kPageTokens + last;
            }
        }
        for (int i = 0; i < 32 && base + i * kWarps < g.sequences; ++i) {
            const long long first = __shfl_sync(0xffffffffu, pf, i), end = __shfl_sync(0xffffffffu, pl, i);
            bool outside = false;
            if (__shfl_sync(0xffffffffu, bad ? 1 : 0, i) == 0) {
                for (long long at = first + lane; at < end; at += 32 * kFlight) {
#pragma unroll
                    for (int u = 0; u < kFlight; ++u) {
                        if (at + 32 * u < end) {
                            const long long page = paging_value(g.pages, g.index_width, static_cast<int>(at + 32 * u));
                            outside |= page < 0 || page >= cache_pages;
                        }
                    }
                }
            }
            outside = __any_sync(0xffffffffu, outside) != 0;
            if (lane == i) bad |= outside;
        }
        if (own < g.sequences) {
            table.rows[own] = bad ? 0 : static_cast<int>(ql - qf) << g.pack;
            table.keys[own] = bad ? 0 : static_cast<int>(keys);
            table.first_token[own] = bad ? 0 : static_cast<int>(qf);
            table.first_page[own] = bad ? 0 : static_cast<int>(pf);
            if (bad && blockIdx.x == 0) report_status(g.status, kStatusIndexOutOfBounds);
        }
    }
    if (__syncthreads_or(backwards ? 1 : 0) != 0) {
        for (int s = threadIdx.x; s < g.sequences; s += kPrefillThreads) table.rows[s] = 0;
        __syncthreads();
    }
}

// Lengths and first rows of sequence b.  DENSE is a template argument of the kernel: as run-time branches these four
// cost the packed form 2.5 % (every warp of a CTA decodes every work item).
template <bool DENSE>
__device__ __forceinline__ int seq_len_q(const PrefillParams &p, int b) { return DENSE ? p.uniform_q : p.lens_q[b]; }
template <bool DENSE>
__device__ __forceinline__ int seq_len_kv(const PrefillParams &p, int b) { return DENSE ? p.uniform_kv : p.lens_kv[b]; }
template <bool DENSE>
__device__ __forceinline__ int seq_offset_q(const PrefillParams &p, int b) { return DENSE ? b * p.uniform_q : p.offsets[b]; }
template <bool DENSE, bool WINDOW>
__device__ __forceinline__ int seq_offset_kv(const PrefillParams &p, int b) {
    return DENSE ? b * p.uniform_kv : (WINDOW ? p.offsets_kv[b] : p.offsets[b]);
}

__device__ __forceinline__ float exp2_approx(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

__device__ __forceinline__ float max3(float a, float b, float c) {
    float d;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}

// Which columns of a tile may be hidden: none, those from `limit` on (the diagonal tile and a sequence's last tile), or
// also those before `low` (where a sliding window begins).
constexpr int kMaskNone = 0, kMaskEnd = 1, kMaskBoth = 2;

template <int MASK>
__device__ __forceinline__ bool column_visible(int column, int low, int limit) {
    return MASK == kMaskBoth ? (column >= low && column < limit) : column < limit;
}

// Folds the 32 raw scores of one chunk into four running maxima (independent chains).  A mask other than none also
// handles a negative scale; `low` and `limit` count columns from the chunk's first.
template <int MASK>
__device__ __forceinline__ void chunk_max(const uint32_t (&sc)[kChunk], int low, int limit, float sign, float (&m)[4]) {
    if (MASK != kMaskNone) {
#pragma unroll
        for (int i = 0; i < kChunk; i += 4) {
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                if (column_visible<MASK>(i + u, low, limit)) m[u] = fmaxf(m[u], __uint_as_float(sc[i + u]) * sign);
            }
        }
    } else {
#pragma unroll
        for (int i = 0; i < kChunk; i += 8) {
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                m[u] = max3(m[u], __uint_as_float(sc[i + 2 * u]), __uint_as_float(sc[i + 2 * u + 1]));
            }
        }
    }
}

// P = exp2(s * scale + bias) for one chunk of 32 scores: the bf16 pairs go back to tensor memory (16 packed
// columns at `tmem_p`), the unrounded values are added to two running f32x2 sums.  Scores are handled as f32x2
// pairs.  (Evaluating part of the exponentials as a polynomial on the FMA pipe was measured slower at every ratio:
// with one softmax warp per scheduler the extra instructions cost more than the special-function unit saves.)
// SPLIT: 16 columns of leading terms, then 16 of what rounding them left out, over the chunk's own 32 score columns.
template <typename T, int MASK, bool SPLIT>
__device__ __forceinline__ void chunk_exp_store(const uint32_t (&sc)[kChunk], uint32_t tmem_p, float2 scale2,
                                                float2 bias2, int low, int limit, float2 (&sum)[2]) {
    uint32_t packed[SPLIT ? kChunk : kChunk / 2];
#pragma unroll
    for (int i = 0; i < kChunk; i += 2) {
        const float2 x = __ffma2_rn(make_float2(__uint_as_float(sc[i]), __uint_as_float(sc[i + 1])), scale2, bias2);
        float2 e;
        e.x = exp2_approx(x.x);
        e.y = exp2_approx(x.y);
        if (MASK != kMaskNone) {
            e.x = column_visible<MASK>(i, low, limit) ? e.x : 0.0f;
            e.y = column_visible<MASK>(i + 1, low, limit) ? e.y : 0.0f;
        }
        sum[(i >> 1) & 1] = __fadd2_rn(sum[(i >> 1) & 1], e);
        packed[i >> 1] = pack2<T>(e.x, e.y);
        if constexpr (SPLIT) {
            static_assert(std::is_same<T, __nv_bfloat16>::value, "a bf16 pair is two f32 upper halves");
            const float2 lead = make_float2(__uint_as_float(packed[i >> 1] << 16), __uint_as_float(packed[i >> 1] & 0xffff0000u));
            packed[(i >> 1) + kChunk / 2] = pack2<T>(e.x - lead.x, e.y - lead.y);
        }
    }
    if constexpr (SPLIT) {
        tmem_st_x32(tmem_p, packed);
    } else {
        tmem_st_x16(tmem_p, packed);
    }
}

// This warp's share of half a tile's weights is in tensor memory.
__device__ __forceinline__ void hand_over(uint32_t bar, int lane) {
    tmem_wait_st();
    tcgen05_fence_before();
    __syncwarp();
    if (lane == 0) mbar_arrive(bar);
}

// One row of one key tile: S (128 f32 columns at `tmem_s`) -> P (64 packed columns over the same place), chunk by
// chunk with the next chunk's load in flight.
template <typename T, int MASK, bool SPLIT>
__device__ __forceinline__ void tile_exp(uint32_t tmem_s, float2 scale2, float2 bias2, int low, int limit, float2 (&sum)[2],
                                         uint32_t bar_half, int lane) {
    uint32_t buf[2][kChunk];
    tmem_ld_x32(tmem_s, buf[0]);
#pragma unroll
    for (int c = 0; c < kTile / kChunk; ++c) {
        tmem_wait_ld_into(buf[c & 1]);
        if (c + 1 < kTile / kChunk) tmem_ld_x32(tmem_s + (c + 1) * kChunk, buf[(c + 1) & 1]);
        chunk_exp_store<T, MASK, SPLIT>(buf[c & 1], tmem_s + c * (SPLIT ? kChunk : kChunk / 2), scale2, bias2, low - c * kChunk,
                                        limit - c * kChunk, sum);
        if (c & 1) hand_over(bar_half + (c >> 1) * 8, lane);
    }
}

// Exact maximum of the visible raw scores (times `sign`) of one row of one key tile.
template <int MASK>
__device__ __forceinline__ float tile_max(uint32_t tmem_s, int low, int limit, float sign) {
    float m[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
    uint32_t buf[2][kChunk];
    tmem_ld_x32(tmem_s, buf[0]);
#pragma unroll
    for (int c = 0; c < kTile / kChunk; ++c) {
        tmem_wait_ld_into(buf[c & 1]);
        if (c + 1 < kTile / kChunk) tmem_ld_x32(tmem_s + (c + 1) * kChunk, buf[(c + 1) & 1]);
        chunk_max<MASK>(buf[c & 1], low - c * kChunk, limit - c * kChunk, sign, m);
    }
    return fmaxf(fmaxf(m[0], m[1]), fmaxf(m[2], m[3]));
}

// Multiplies this thread's row of O (HD f32 columns of tensor memory) by `factor`.
template <int HD>
__device__ __forceinline__ void scale_o_row(uint32_t tmem_o, float factor) {
#pragma unroll 1
    for (int c = 0; c < HD; c += 32) {
        uint32_t r[32];
        tmem_ld_x32(tmem_o + c, r);
        tmem_wait_ld_into(r);
#pragma unroll
        for (int i = 0; i < 32; ++i) r[i] = __float_as_uint(__uint_as_float(r[i]) * factor);
        tmem_st_x32(tmem_o + c, r);
    }
    tmem_wait_st();
}

// 32 bytes by one lane.  The lanes of a warp store to rows of their own, a line each, so what counts is how many stores there are.
__device__ __forceinline__ void store_sector(void *to, const uint32_t (&w)[8]) {
    asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(to), "r"(w[0]), "r"(w[1]), "r"(w[2]), "r"(w[3]),
                 "r"(w[4]), "r"(w[5]), "r"(w[6]), "r"(w[7])
                 : "memory");
}

// One unit of work: 256 query rows (tiles A and B) of one (sequence, head).
struct Item {
    int head;
    int kv_head;
    int seq;        // sequence index (row of the block table in the paged form)
    int offset;     // first packed query row of the sequence
    int offset_kv;  // first packed key row of the sequence (the same row except in the dense form)
    int q0;         // sequence-local index of the first query row
    int len_q;
    int len_kv;
    int shift;      // causal mask: query row i sees keys 0 .. max(i + shift, 0); 0 for the sequence-local mask,
                    // len_kv - len_q when the queries are the sequence's last tokens
    int first[2];   // first key tile tile A / tile B needs (0 unless a window hides the ones before); A's is the lower
    int tiles[2];   // one past the last key tile tile A / tile B needs (0: no real row, or no visible key)
    int key_tiles;  // max of the two
    int first_page; // TENSOR: place of the sequence's first page in the page list
    bool alternate; // TENSOR: a single query tile, whose key tiles go to tile A's and tile B's places in turn
    bool valid;     // false: the sequence's offsets leave the packed tensors
};

// The items of a CTA's first rounds are decoded by its warps side by side before the roles part (not where a CTA has one item only: held
// ahead it cost 0.5 - 1 us, 3 prompts of 13 - 53 tokens 12.4 -> 13.3 us, 2 of 100 - 300 16.3 -> 17.1): item by item, the softmax waited
// for its look-ups between two items, and for the stores of 32 rows' lines, 16 bytes a lane.  With stores of 32 bytes 8192 + 4096 +
// 2048 + 1024 tokens 726 -> 691 us at the power limit, eight prompts of 209 - 3355 268 -> 250, the tensor surface's mixed step 157 -> 150.
constexpr int kHeldItems = 64;

__device__ __forceinline__ int pairs_of(int len_q) { return (max(len_q, 0) + kPair - 1) / kPair; }

// Items are numbered heaviest first: rank = index / heads walks the query pairs of all sequences from the highest
// pair index down (under a causal mask a pair's work grows with its index), head = index % heads.  `counts[t]` is
// the number of sequences that have a pair t, `tmax` the largest pair count.  Every lane of the calling warp
// takes part and receives the same answer.
// TENSOR: rows are (token, head) pairs, `table` lists the sequences and `pack` is the log2 of a token's rows; `order`, unless
// it is nullptr, lists sequence and pair of every rank (see order_items).
template <bool DENSE, bool WINDOW, bool TENSOR>
__device__ __forceinline__ Item decode_item(const PrefillParams &p, const SequenceTable &table, int pack, const int *counts, int tmax,
                                            const unsigned *order, int index, int lane) {
    constexpr unsigned kFull = 0xffffffffu;
    Item item;
    int rank = index / p.heads;
    item.head = index - rank * p.heads;
    item.kv_head = item.head / (p.heads / p.kv_heads);
    int pair = -1;
    int seq = -1;
    if (TENSOR && order != nullptr) {
        const unsigned entry = order[rank];
        seq = static_cast<int>(entry % kMaxTensorSequences);
        pair = static_cast<int>(entry / kMaxTensorSequences);
        tmax = 0;
    }
    for (int first = 0; first < tmax && pair < 0; first += 32) {
        const int t = tmax - 1 - (first + lane);
        const int count = t >= 0 ? counts[t] : 0;
        int prefix = count;  // inclusive prefix sum over the lanes
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const int other = __shfl_up_sync(kFull, prefix, d);
            if (lane >= d) prefix += other;
        }
        const unsigned hit = __ballot_sync(kFull, rank < prefix);
        if (hit != 0) {
            const int where = __ffs(hit) - 1;
            pair = tmax - 1 - (first + where);
            rank -= __shfl_sync(kFull, prefix - count, where);
        } else {
            rank -= __shfl_sync(kFull, prefix, 31);
        }
    }
    for (int first = 0; first < p.batch && seq < 0 && pair >= 0; first += 32) {
        const int b = first + lane;
        const bool has = b < p.batch && pairs_of(TENSOR ? table.rows[b] : seq_len_q<DENSE>(p, b)) > pair;
        const unsigned mask = __ballot_sync(kFull, has);
        const int n = __popc(mask);
        if (rank < n) {
            seq = first + static_cast<int>(__fns(mask, 0, rank + 1));
        } else {
            rank -= n;
        }
    }
    item.valid = false;
    item.seq = seq < 0 ? 0 : seq;
    item.offset = 0;
    item.offset_kv = 0;
    item.q0 = max(pair, 0) * kPair;
    item.len_q = 0;
    item.len_kv = 0;
    item.shift = 0;
    item.first[0] = item.first[1] = 0;
    item.tiles[0] = item.tiles[1] = 0;
    item.key_tiles = 0;
    item.first_page = 0;
    item.alternate = false;
    if (seq < 0) return item;
    if (TENSOR) {
        item.len_q = table.rows[seq];
        item.len_kv = table.keys[seq];
        item.offset = table.first_token[seq];
        item.first_page = table.first_page[seq];
        item.valid = true;
        item.shift = item.len_kv - (item.len_q >> pack);
    } else {
        item.len_q = max(seq_len_q<DENSE>(p, seq), 0);
        item.len_kv = max(seq_len_kv<DENSE>(p, seq), 0);
        item.offset = seq_offset_q<DENSE>(p, seq);
        item.offset_kv = seq_offset_kv<DENSE, WINDOW>(p, seq);
        item.valid = item.offset >= 0 && item.offset_kv >= 0 && item.offset + item.len_q <= p.total_q &&
                     (p.block_table != nullptr ? item.len_kv <= p.table_stride * kPageTokens
                                               : item.offset_kv + item.len_kv <= p.total_kv);
        if (!item.valid) return item;
        item.shift = p.causal == 2 ? item.len_kv - item.len_q : 0;
    }
    if (WINDOW) {
#pragma unroll
        for (int x = 0; x < 2; ++x) {
            const int row = item.q0 + x * kTile;
            item.first[x] = max((TENSOR ? row >> pack : row) + item.shift - p.window + 1, 0) / kTile;
        }
    }
#pragma unroll
    for (int x = 0; x < 2; ++x) {
        const int first = item.q0 + x * kTile;
        const int real = min(max(item.len_q - first, 0), kTile);
        int visible = real > 0 ? item.len_kv : 0;
        if (p.causal && real > 0) {
            const int last = first + real - 1;
            visible = min(visible, max((TENSOR ? last >> pack : last) + item.shift, 0) + 1);
        }
        item.tiles[x] = (visible + kTile - 1) / kTile;
    }
    item.key_tiles = max(item.tiles[0], item.tiles[1]);
    item.alternate = TENSOR && item.tiles[1] == 0 && item.tiles[0] - item.first[0] > 1;
    return item;
}

// TENSOR: lists the (sequence, pair) entries of a call by the key tiles they take, the longest first.  A chunk's pairs and a
// decoding sequence's only one differ by what context lies behind them; dealt out by pair index alone, a CTA's share of
// four 512-token chunks and 28 decoding sequences behind 0 - 3000 tokens came to twice the mean.  Comparing every entry with every
// other pays up to the most there are (a 100-token chunk beside 100 sequences of up to 100 tokens 59.9 us, unordered 61.3;
// 400 of 300 207 and 220; 1000 of 30 415 and 451; 1000 of 1000 686 and 789).  Every CTA computes the same list; all its threads
// take part.  Returns the number of entries, or -1 with no list when there are more than
// kMaxOrdered.  `first`: kMaxTensorSequences ints, `costs` and `entries`: kMaxOrdered each.
template <bool WINDOW>
__device__ __forceinline__ int order_items(const PrefillParams &p, const SequenceTable &table, int pack, int *first, int *costs,
                                           unsigned *entries, unsigned *order, volatile int *total, int warp, int lane) {
    if (warp == 0) {
        int sum = 0;
        for (int b = 0; b < p.batch; b += 32) {
            const int own = b + lane < p.batch ? pairs_of(table.rows[b + lane]) : 0;
            int prefix = own;
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const int other = __shfl_up_sync(0xffffffffu, prefix, d);
                if (lane >= d) prefix += other;
            }
            if (b + lane < p.batch) first[b + lane] = sum + prefix - own;
            sum = min(sum + __shfl_sync(0xffffffffu, prefix, 31), 2 * kMaxOrdered);  // (pairs of one sequence fit 22 bits)
        }
        if (lane == 0) *total = sum;
    }
    __syncthreads();
    const int count = *total;
    if (count > kMaxOrdered) return -1;
    for (int b = warp; b < p.batch; b += kPrefillThreads / 32) {
        const int rows = table.rows[b], keys = table.keys[b];
        const int shift = keys - (rows >> pack);
        for (int t = lane; t < pairs_of(rows); t += 32) {
            const int last = min(rows, (t + 1) * kPair) - 1;
            int visible = keys;
            if (p.causal) visible = min(visible, max((last >> pack) + shift, 0) + 1);
            int tiles = (visible + kTile - 1) / kTile;
            if (WINDOW) tiles -= max(((t * kPair) >> pack) + shift - p.window + 1, 0) / kTile;
            const bool single = rows - t * kPair <= kTile;  // half as long: see `alternate`
            costs[first[b] + t] = single ? (tiles + 1) / 2 : tiles;
            entries[first[b] + t] = static_cast<unsigned>(b + t * kMaxTensorSequences);
        }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < count; i += kPrefillThreads) {
        const int own = costs[i];
        int place = 0;
        for (int j = 0; j < count; ++j) place += costs[j] > own || (costs[j] == own && j < i) ? 1 : 0;
        order[place] = entries[i];
    }
    __syncthreads();
    return count;
}

// SAFE = false: the first launch.  One persistent CTA per SM walks its share of the items (item round r of CTA c is
// index r * grid + c on even rounds and r * grid + grid - 1 - c on odd ones, which evens out the heaviest-first
// order); all pipelines run on across items, so the next item's loads and first MMAs overlap the current item's
// last tile and epilogue.  Softmax is single-pass after an item's first key tile.
// SAFE = true: the second launch, same grid and same shares: it leaves at once unless the flag above is raised, and
// otherwise recomputes it with the exact row maximum on every tile.
// PAGED: K and V tiles are gathered from 16-token cache pages through the block table (eight page boxes per
// 128-key tile and 64-wide half; the boxes land back to back, which is the layout one 128-row box would have).
// HD = 128 or 64: with 64 a tile is a single 128-byte-wide box (the second half of every 32 KB buffer stays unused).
// DENSE: uniform lengths, sequences back to back, LSE laid out [batch, heads, queries] (fmha_prefill_lse).
// LONE: no CTA has a second item, and none is held: see kHeldItems.
template <typename T, int HD, bool SAFE, bool PAGED, bool DENSE, bool WINDOW, bool TENSOR, bool LONE = false>
__global__ void __launch_bounds__(kPrefillThreads, 1)
    prefill_tcgen05_kernel(const __grid_constant__ CUtensorMap q_map, const __grid_constant__ CUtensorMap k_map,
                           const __grid_constant__ CUtensorMap v_map, const PrefillParams p,
                           const std::conditional_t<TENSOR, TensorPaging, NoPaging> paging) {
    extern __shared__ uint8_t smem_raw[];
    const uint32_t raw = smem_u32(smem_raw);
    const uint32_t base = (raw + 1023u) & ~1023u;
    const uint32_t q_smem = base;                        // [2 tiles]
    const uint32_t k_smem = base + 2 * kTileBytes;       // [2 stages]
    const uint32_t v_smem = base + 4 * kTileBytes;       // [2 stages]
    const uint32_t bars = base + 6 * kTileBytes;
    constexpr int kHalves = HD / 64;                       // 128-byte-wide boxes per tile
    constexpr int kLoadBytes = kHalves * kHalfTileBytes;   // bytes one tile load delivers
    const uint32_t bar_q_full = bars;         // [2 tiles]
    const uint32_t bar_q_empty = bars + 16;   // [2 tiles]
    const uint32_t bar_k_full = bars + 32;    // [2 stages]
    const uint32_t bar_k_empty = bars + 48;   // [2]
    const uint32_t bar_v_full = bars + 64;    // [2]
    const uint32_t bar_v_empty = bars + 80;   // [2]
    const uint32_t bar_s_full = bars + 96;    // [2 tiles]
    const uint32_t bar_o_full = bars + 112;   // [2 tiles]
    const uint32_t bar_p_full = bars + 128;   // [2 tiles][2 halves of the keys], one arrival per softmax warp of the tile
    const uint32_t bar_o_empty = bars + 160;  // [2 tiles], one arrival per softmax warp of the tile
    const uint32_t bar_share = bars + 176;    // TENSOR: tile B's half of an alternating item, one arrival per softmax warp
    constexpr int kBarriers = TENSOR ? kTensorBarriers : 22;
    const uint32_t words = bars + 8 * kBarriers;
    volatile uint32_t *holder_ptr = reinterpret_cast<volatile uint32_t *>(smem_raw + (words - raw));
    volatile int *shared_tmax = reinterpret_cast<volatile int *>(smem_raw + (words + 4 - raw));
    volatile int *shared_ranks = reinterpret_cast<volatile int *>(smem_raw + (words + 8 - raw));
    int *counts = reinterpret_cast<int *>(smem_raw + (words + 32 - raw));  // [kMaxRankTiles]
    volatile int *redo_list = reinterpret_cast<volatile int *>(counts + kMaxRankTiles);  // [kRedoCapacity], SAFE only

    const int tid = threadIdx.x;
    const int warp = tid >> 5;
    const int lane = tid & 31;
    SequenceTable table = {};
    int pack = 0;
    int ordered = -1;                  // TENSOR: entries in `order`, or -1: items go by `counts`
    unsigned *order = nullptr;
    Item *held = reinterpret_cast<Item *>(counts + kMaxRankTiles + kRedoCapacity);  // [kHeldItems]
    volatile float2 *share = nullptr;  // TENSOR: base and sum of tile B's rows of an alternating item
    if constexpr (TENSOR) {
        // (the redo list's place and what follows it)
        table.rows = counts + kMaxRankTiles;
        table.keys = table.rows + kMaxTensorSequences;
        table.first_token = table.keys + kMaxTensorSequences;
        table.first_page = table.first_token + kMaxTensorSequences;
        pack = paging.pack;
        int *costs = table.first_page + kMaxTensorSequences;
        unsigned *entries = reinterpret_cast<unsigned *>(costs + kMaxOrdered);
        order = entries + kMaxOrdered;
        share = reinterpret_cast<volatile float2 *>(order + kMaxOrdered);
        list_sequences(paging, p.cache_pages, table, warp, lane);
        __syncthreads();
        ordered = order_items<WINDOW>(p, table, pack, counts, costs, entries, order, shared_ranks, warp, lane);
        if (ordered < 0) order = nullptr;
        held = reinterpret_cast<Item *>(costs);  // (and the entries' place: both are done with)
        static_assert(kHeldItems * sizeof(Item) <= 2 * kMaxOrdered * sizeof(int), "the ordering's scratch holds the items");
        __syncthreads();  // `counts` may be used again below
    }
    if (SAFE && !p.exact && *reinterpret_cast<volatile unsigned *>(&g_out_of_range_seen) == 0u) {
        return;  // no first launch on this device has ever marked a row
    }

    // ---- the table behind the heaviest-first item order ----
    if (!TENSOR || ordered < 0) {
        int tmax = 0;
        for (int b = 0; b < p.batch; ++b) tmax = max(tmax, pairs_of(TENSOR ? table.rows[b] : seq_len_q<DENSE>(p, b)));
        tmax = min(tmax, kMaxRankTiles);
        for (int t = tid; t < tmax; t += kPrefillThreads) {
            int count = 0;
            for (int b = 0; b < p.batch; ++b) count += pairs_of(TENSOR ? table.rows[b] : seq_len_q<DENSE>(p, b)) > t ? 1 : 0;
            counts[t] = count;
        }
        __syncthreads();
        if (tid == 0) {
            int ranks = 0;
            for (int t = 0; t < tmax; ++t) ranks += counts[t];
            *shared_tmax = tmax;
            *shared_ranks = ranks;
        }
        __syncthreads();
    }
    const int tmax = TENSOR && ordered >= 0 ? 0 : *shared_tmax;
    auto decode = [&](int index) { return decode_item<DENSE, WINDOW, TENSOR>(p, table, pack, counts, tmax, order, index, lane); };
    const long long total_items = static_cast<long long>(TENSOR && ordered >= 0 ? ordered : *shared_ranks) * p.heads;
    // index of this CTA's share number `round`, or -1 past the end
    auto share_index = [&](int round) -> int {
        const long long first = static_cast<long long>(round) * gridDim.x;
        const long long index = first + ((round & 1) ? gridDim.x - 1 - blockIdx.x : blockIdx.x);
        return index < total_items ? static_cast<int>(index) : -1;
    };
    // where the LSE of (item, sequence-local query row) lives
    auto lse_at = [&](const Item &item, int row) -> float * {
        if (DENSE) {
            return p.lse + (static_cast<size_t>(item.seq) * p.heads + item.head) * p.lse_rows + row;
        }
        if (TENSOR) {
            return p.lse + (((static_cast<size_t>(item.offset) + (row >> pack)) * p.heads + item.head) << pack) + (row & ((1 << pack) - 1));
        }
        return p.lse + (static_cast<size_t>(item.offset) + row) * p.heads + item.head;
    };
    int listed = -1;  // SAFE: number of marked items in redo_list, or -1 = walk the whole share
    if (SAFE && !p.exact) {
        // The first launch leaves a NaN as the LSE of every row it could not finish in range: list the marked items.
        int found = 0;
        bool overflow = false;
        for (int round = 0;; ++round) {
            const int index = share_index(round);
            if (index < 0) break;
            const Item item = decode(index);
            const int row = item.q0 + tid;
            const bool marked = item.valid && item.key_tiles > 0 && tid < kPair && row < item.len_q &&
                                isnan(*lse_at(item, row));
            if (__syncthreads_or(marked ? 1 : 0) != 0) {
                if (found < kRedoCapacity) {
                    if (tid == 0) redo_list[found] = index;
                    ++found;
                } else {
                    overflow = true;
                }
            }
        }
        __syncthreads();
        if (found == 0) return;
        listed = overflow ? -1 : found;
    }
    // index of the item this CTA works on in `round`, or -1 when it is done
    auto item_index = [&](int round) -> int {
        if (SAFE && listed >= 0) return round < listed ? redo_list[round] : -1;
        return share_index(round);
    };

    for (int round = warp; !LONE && round < kHeldItems; round += kPrefillThreads / 32) {
        const int index = item_index(round);
        if (index < 0) break;
        const Item item = decode(index);
        if (lane == 0) held[round] = item;
    }
    auto item_at = [&](int round, int index) -> Item { return !LONE && round < kHeldItems ? held[round] : decode(index); };
    if (tid == 0) {
        for (int i = 0; i < kBarriers; ++i) {
            const bool by_warps = i >= 16;  // p_full, o_empty, share
            mbar_init(bars + 8 * i, by_warps ? 4 : 1);
        }
        mbar_init_fence();
    }
    if (warp == 8) {
        tmem_alloc(words, 512);
        tmem_relinquish();
    }
    tcgen05_fence_before();
    __syncthreads();
    tcgen05_fence_after();
    const uint32_t tmem_base = *holder_ptr;

    bool failed = false;

    if (warp >= 9) {
        // ---------------- TMA producers: warp 9 Q and K, warp 10 V (ragged keys come in whole boxes: warp 9 alone) ----------------
        const bool values = PAGED && warp == 10;
        const CUtensorMap *map = values ? &v_map : &k_map;
        const uint32_t tiles_smem = values ? v_smem : k_smem;
        const uint32_t bar_full = values ? bar_v_full : bar_k_full;
        const uint32_t bar_empty = values ? bar_v_empty : bar_k_empty;
        if (lane == 0) {
            if (!values) prefetch_tensor_map(&q_map);
            prefetch_tensor_map(map);
        }
        int g = 0;                // key tiles loaded so far, over all items: stage g & 1, use (g >> 1)
        int q_loads[2] = {0, 0};  // Q tiles loaded so far
        auto wait_lane0 = [&](uint32_t bar, uint32_t parity) -> bool {
            int ok = 1;
            if (lane == 0) ok = mbar_wait(bar, parity) ? 1 : 0;
            return __shfl_sync(0xffffffffu, ok, 0) != 0;
        };
        for (int round = 0; (PAGED || warp == 9) && !failed; ++round) {
            const int index = item_index(round);
            if (index < 0) break;
            const Item item = item_at(round, index);
            if (item.key_tiles == 0) continue;
#pragma unroll
            for (int x = 0; x < 2; ++x) {
                if (item.tiles[x] == 0 || failed || values) continue;
                // the tile's buffer is free when the previous item's last Q K^T of this tile has retired
                if (q_loads[x] > 0 && !wait_lane0(bar_q_empty + x * 8, (q_loads[x] - 1) & 1)) {
                    failed = true;
                    continue;
                }
                ++q_loads[x];
                if (elect_one()) {
                    mbar_expect_tx(bar_q_full + x * 8, kLoadBytes);
                    // TENSOR: a box holds the heads of a pack for 128 >> pack tokens, token by token
                    const int row0 = item.offset + ((item.q0 + x * kTile) >> pack);
                    const int head0 = item.head << pack;
                    tma_load_3d(q_smem + x * kTileBytes, &q_map, bar_q_full + x * 8, 0, head0, row0);
                    if (kHalves == 2) {
                        tma_load_3d(q_smem + x * kTileBytes + kHalfTileBytes, &q_map, bar_q_full + x * 8, 64,
                                    head0, row0);
                    }
                }
                __syncwarp();
            }
            // paged form: the page ids of a key tile, one per lane (by its low three bits), read a tile ahead; lanes 0-15 each
            // own one (page, half) box.  A page past the sequence's last one is replaced by the sequence's first page (finite
            // data that the mask hides), a page id outside the cache likewise, with status 1.
            auto page_of = [&](int j) -> int32_t {
                const int pages_of_sequence = (item.len_kv + kPageTokens - 1) / kPageTokens;
                const int wanted = j * (kTile / kPageTokens) + (lane & 7);
                const int place = wanted < pages_of_sequence ? wanted : 0;
                if constexpr (TENSOR) {
                    return static_cast<int32_t>(paging_value(paging.pages, paging.index_width, item.first_page + place));
                } else {
                    const uint32_t *row = p.block_table + static_cast<size_t>(item.seq) * p.table_stride;
                    uint32_t id = row[place];
                    if (id >= static_cast<uint32_t>(p.cache_pages)) {
                        report_status(p.error, kStatusIndexOutOfBounds);
                        id = 0u;
                    }
                    return static_cast<int32_t>(id);
                }
            };
            int32_t page = PAGED ? page_of(item.first[0]) : 0;
            for (int j = item.first[0]; j < item.key_tiles && !failed; ++j, ++g) {
                const int stage = g & 1;
                const int32_t coming = PAGED && j + 1 < item.key_tiles ? page_of(j + 1) : 0;
                if (g >= 2 && !wait_lane0(bar_empty + stage * 8, ((g >> 1) - 1) & 1)) {
                    failed = true;
                    break;
                }
                const uint32_t tile = tiles_smem + stage * kTileBytes;
                if (PAGED) {
                    if (lane == 0) mbar_expect_tx(bar_full + stage * 8, kLoadBytes);
                    __syncwarp();
                    if (lane < 8 * kHalves) {
                        const int half = lane >> 3;
                        tma_load_4d(tile + half * kHalfTileBytes + (lane & 7) * kPageBytes, map, bar_full + stage * 8, half * 64,
                                    item.kv_head, 0, page);
                    }
                    page = coming;
                } else {
                    const int row0 = item.offset_kv + j * kTile;
                    auto load = [&](uint32_t target, const CUtensorMap *from, uint32_t bar) {
                        if (elect_one()) {
                            mbar_expect_tx(bar, kLoadBytes);
                            tma_load_3d(target, from, bar, 0, item.kv_head, row0);
                            if (kHalves == 2) tma_load_3d(target + kHalfTileBytes, from, bar, 64, item.kv_head, row0);
                        }
                        __syncwarp();
                    };
                    load(tile, &k_map, bar_k_full + stage * 8);
                    if (g >= 2 && !wait_lane0(bar_v_empty + stage * 8, ((g >> 1) - 1) & 1)) {
                        failed = true;
                        break;
                    }
                    load(v_smem + stage * kTileBytes, &v_map, bar_v_full + stage * 8);
                }
            }
        }
    } else if (warp == 8) {
        // ---------------- MMA issuer ----------------
        constexpr bool kIsBf16 = std::is_same<T, __nv_bfloat16>::value;
        constexpr uint32_t kIdescQK = make_instr_desc(kTile, kTile, kIsBf16, 0, 0);      // A, B K-major
        constexpr uint32_t kIdescPV = make_instr_desc(kTile, HD, kIsBf16, 0, 1);   // B (V) MN-major
        // The loops over key tiles run in one elected thread, as those of the linear layers do: with every lane waiting, a vote
        // behind each wait and the issue under a lane test, the 24 MMAs of a tile with two-term weights came late: the step of four chunks
        // and 28 decoding sequences above 157 -> 131 us (kernel), 60 - 480 token prompts of 64 sequences 15.2 -> 13.0.  Long prompts are where
        // they were, 616 and 613: there softmax is the longer part of the chain.
        const uint64_t q_desc = make_smem_desc(q_smem, 16, 1024), k_desc = make_smem_desc(k_smem, 16, 1024);
        const uint64_t v_desc = make_smem_desc(v_smem, kHalfTileBytes, 1024);   // (a descriptor's address counts in 16 bytes)
        int p_uses[2] = {0, 0};    // P tiles consumed so far
        // S_x = Q_query K(stage)^T; `last` releases the Q tile
        auto issue_qk = [&](int x, int stage, bool last, int query) {
            const uint64_t a = q_desc + query * (kTileBytes >> 4), b = k_desc + stage * (kTileBytes >> 4);
#pragma unroll
            for (int ks = 0; ks < HD / 16; ++ks) {
                const uint32_t within = ((ks >> 2) * kHalfTileBytes + (ks & 3) * 32) >> 4;
                umma_ss(tmem_base + x * kTile, a + within, b + within, kIdescQK, ks > 0 ? 1u : 0u);
            }
            tcgen05_commit(bar_s_full + x * 8);
            if (last) tcgen05_commit(bar_q_empty + query * 8);
        };
        // O_x (+)= P_x V(stage): 16 keys per step, P advances 8 packed columns, V two 8-row groups (2 x 1024 bytes);
        // the second 64 dims of V are the next box, 16 KB further (leading byte offset).
        // The weights come in halves, so that the first half's products run beside the softmax of the second.
        auto issue_pv = [&](int x, int stage, bool accumulate, bool last) -> bool {
            const uint64_t v = v_desc + stage * (kTileBytes >> 4);
            const uint32_t parity = p_uses[x] & 1;
            ++p_uses[x];
            if (!mbar_wait(bar_p_full + x * 16, parity)) return false;
            tcgen05_fence_after();
#pragma unroll
            for (int ks = 0; ks < kTile / 16; ++ks) {
                if (ks == kTile / 32) {
                    if (!mbar_wait(bar_p_full + x * 16 + 8, parity)) return false;
                    tcgen05_fence_after();
                }
                // TENSOR: a chunk of 32 keys holds 16 columns of leading terms and 16 of the rest
                const uint32_t at = TENSOR ? (ks >> 1) * kChunk + (ks & 1) * 8 : ks * 8;
                umma_ts(tmem_base + 2 * kTile + x * HD, tmem_base + x * kTile + at, v + ks * (2048 >> 4), kIdescPV,
                        (accumulate || ks > 0) ? 1u : 0u);
                if (TENSOR) {
                    umma_ts(tmem_base + 2 * kTile + x * HD, tmem_base + x * kTile + at + kChunk / 2, v + ks * (2048 >> 4), kIdescPV, 1u);
                }
            }
            if (last) tcgen05_commit(bar_o_full + x * 8);
            return true;
        };
        int g = 0;                 // key tiles consumed so far, over all items
        int q_uses[2] = {0, 0};    // Q tiles consumed so far
        int o_done[2] = {0, 0};    // outputs handed to the epilogue so far
        int round = 0;
        // the next item with work, or key_tiles == 0 when there is none
        auto next_item = [&]() -> Item {
            Item item;
            item.key_tiles = 0;
            for (;;) {
                const int index = item_index(round);
                if (index < 0) {
                    item.key_tiles = 0;
                    return item;
                }
                item = item_at(round, index);
                ++round;
                if (item.key_tiles > 0) return item;
            }
        };
        // first Q K^T of both tiles of `item` on key stage `stage` (already waited for)
        auto first_qk = [&](const Item &item, int x, int stage) -> bool {
            if (item.tiles[x] == 0 || (WINDOW && item.first[x] != item.first[0])) return true;  // (tile B's may come later)
            if (!mbar_wait(bar_q_full + x * 8, q_uses[x] & 1)) return false;
            ++q_uses[x];
            tcgen05_fence_after();
            issue_qk(x, stage, item.tiles[x] == item.first[x] + 1, x);
            return true;
        };
        // Everything of one item, and the first Q K^T of the following one; one thread.
        bool begun = false;
        auto run_item = [&](const Item &item, const Item &following) {
            if (!begun) {
                if (!mbar_wait(bar_k_full, 0)) failed = true;
                if (!failed && (!first_qk(item, 0, 0) || !first_qk(item, 1, 0))) failed = true;
                if (!failed) tcgen05_commit(bar_k_empty);
            }
            if constexpr (TENSOR) {
                // A single query tile: key tile j's scores stand in tile A's or tile B's place by turns, so that Q K^T of the
                // next one runs beside this one's softmax, and each place has its own O.
                for (int j = item.first[0]; item.alternate && j < item.key_tiles && !failed; ++j, ++g) {
                    const int stage = g & 1;
                    const int next = (g + 1) & 1;
                    const int x = (j - item.first[0]) & 1;
                    const bool more = j + 1 < item.key_tiles;
                    auto next_keys = [&]() -> bool {
                        if (!mbar_wait(bar_k_full + next * 8, ((g + 1) >> 1) & 1)) return false;
                        tcgen05_fence_after();
                        return true;
                    };
                    auto release_keys = [&]() {
                        tcgen05_commit(bar_k_empty + next * 8);
                    };
                    if (more) {
                        if (!next_keys()) {
                            failed = true;
                            break;
                        }
                        issue_qk(x ^ 1, next, j + 2 == item.key_tiles, 0);
                        release_keys();
                    }
                    if (!mbar_wait(bar_v_full + stage * 8, (g >> 1) & 1) ||
                        (j < item.first[0] + 2 && o_done[x] > 0 && !mbar_wait(bar_o_empty + x * 8, (o_done[x] - 1) & 1))) {
                        failed = true;
                        break;
                    }
                    const bool last = j + 2 >= item.key_tiles;
                    if (!issue_pv(x, stage, j >= item.first[0] + 2, last)) {
                        failed = true;
                        break;
                    }
                    if (last) ++o_done[x];
                    tcgen05_commit(bar_v_empty + stage * 8);
                    if (!more && following.key_tiles > 0) {
                        if (!next_keys() || !first_qk(following, 0, next) || !first_qk(following, 1, next)) {
                            failed = true;
                            break;
                        }
                        release_keys();
                    }
                }
            }
            for (int j = item.first[0]; !item.alternate && j < item.key_tiles && !failed; ++j, ++g) {
                const int stage = g & 1;
                const int next = (g + 1) & 1;
                const bool more = j + 1 < item.key_tiles;          // this item has another key tile
                const bool onward = more || following.key_tiles > 0;  // some Q K^T follows on key tile g + 1
                if (!mbar_wait(bar_v_full + stage * 8, (g >> 1) & 1)) {
                    failed = true;
                    break;
                }
#pragma unroll
                for (int x = 0; x < 2; ++x) {
                    if (failed) continue;
                    if (j < item.tiles[x] && (!WINDOW || j >= item.first[x])) {
                        // the previous item's epilogue must have taken O out of tensor memory
                        if (j == item.first[x] && o_done[x] > 0 && !mbar_wait(bar_o_empty + x * 8, (o_done[x] - 1) & 1)) {
                            failed = true;
                            continue;
                        }
                        const bool last = j == item.tiles[x] - 1;
                        if (!issue_pv(x, stage, j > item.first[x], last)) {
                            failed = true;
                            continue;
                        }
                        if (last) ++o_done[x];
                    }
                    if (x == 1) {
                        tcgen05_commit(bar_v_empty + stage * 8);
                    }
                    if (onward) {
                        if (x == 0) {
                            if (!mbar_wait(bar_k_full + next * 8, ((g + 1) >> 1) & 1)) {
                                failed = true;
                                continue;
                            }
                            tcgen05_fence_after();
                        }
                        if (more) {
                            if (WINDOW && item.tiles[x] > 0 && item.first[x] != item.first[0] && j + 1 == item.first[x]) {
                                if (!mbar_wait(bar_q_full + x * 8, q_uses[x] & 1)) {
                                    failed = true;
                                    continue;
                                }
                                ++q_uses[x];
                                tcgen05_fence_after();
                            }
                            if (j + 1 < item.tiles[x] && (!WINDOW || j + 1 >= item.first[x])) {
                                issue_qk(x, next, j + 2 == item.tiles[x], x);
                            }
                        } else if (!first_qk(following, x, next)) {
                            failed = true;
                            continue;
                        }
                        if (x == 1) {
                            tcgen05_commit(bar_k_empty + next * 8);
                        }
                    }
                }
            }
        };
        Item item = next_item();
        while (item.key_tiles > 0 && !failed) {
            const Item following = next_item();   // (the whole warp takes part)
            const bool issues = elect_one();
            if (issues) run_item(item, following);
            __syncwarp();
            // the elected lane's counts and verdict
            begun = true;
            const int leader = __ffs(__ballot_sync(0xffffffffu, issues)) - 1;
            auto share = [&](int value) { return __shfl_sync(0xffffffffu, value, leader); };
            g = share(g);
#pragma unroll
            for (int x = 0; x < 2; ++x) {
                q_uses[x] = share(q_uses[x]);
                p_uses[x] = share(p_uses[x]);
                o_done[x] = share(o_done[x]);
            }
            failed = share(failed ? 1 : 0) != 0;
            item = following;
        }
    } else {
        // ---------------- softmax / correction / epilogue: warps 0-3 tile A, warps 4-7 tile B ----------------
        const int x = warp >> 2;
        const int quarter = warp & 3;                  // tensor-memory lanes 32*quarter .. +31
        const int local_row = quarter * 32 + lane;
        const uint32_t lane_base = static_cast<uint32_t>(quarter * 32) << 16;
        const uint32_t tmem_s = tmem_base + x * kTile + lane_base;
        const uint32_t tmem_o = tmem_base + 2 * kTile + x * HD + lane_base;
        const float2 scale2 = make_float2(p.scale_log2, p.scale_log2);
        const float sign = p.scale_log2 < 0.0f ? -1.0f : 1.0f;
        int s_uses = 0;   // score tiles consumed so far, over all items
        int o_uses = 0;   // outputs taken so far
        int shares = 0, others_done = 0;  // TENSOR, tile A: alternating items so far, outputs of tile B so far
        for (int round = 0; !failed; ++round) {
            const int index = item_index(round);
            if (index < 0) break;
            const Item item = item_at(round, index);
            if (!item.valid) {
                if (warp == 0 && lane == 0) report_status(p.error, kStatusIndexOutOfBounds);
                continue;
            }
            // sequence-local query index
            const int row = item.q0 + (TENSOR && item.alternate ? 0 : x * kTile) + local_row;
            const bool real = row < item.len_q;
            const int turn = row >> pack;                       // sequence-local token of the row
            const size_t token = static_cast<size_t>(item.offset) + (real ? turn : 0);
            T *dst = static_cast<T *>(p.out) + (((token * p.heads + item.head) << pack) + (real ? row & ((1 << pack) - 1) : 0)) * HD;
            float *lse_row = lse_at(item, real ? row : 0);
            const bool alternate = TENSOR && item.alternate;  // both places hold tile A's rows, of every other key tile
            const int my_tiles = x == 0 || alternate ? item.tiles[0] : item.tiles[1];
            const int my_first = alternate ? item.first[0] + x : x == 0 ? item.first[0] : item.first[1];
            const int my_step = alternate ? 2 : 1;
            if (my_tiles == 0) {
                // No key is visible to this tile's rows: zeros and LSE -1e20.
                if (real) {
#pragma unroll
                    for (int i = 0; i < HD / 8; ++i) reinterpret_cast<uint4 *>(dst)[i] = make_uint4(0u, 0u, 0u, 0u);
                    *lse_row = TENSOR ? -INFINITY : -1.0e20f;
                }
                continue;
            }
            float base_log2 = -INFINITY;  // what P, O and the row sum are relative to (log2 units); finite after tile 0
            float row_sum = 0.0f;
            bool in_range = true;
            bool unseen = WINDOW && real;  // no key seen yet: O and the sum are zero, so the base is free
            bool seen = false;             // TENSOR: some key was visible
            for (int j = my_first; j < my_tiles && !failed; j += my_step, ++s_uses) {
                if (!__all_sync(0xffffffffu, mbar_wait(bar_s_full + x * 8, s_uses & 1) ? 1 : 0)) {
                    failed = true;
                    break;
                }
                tcgen05_fence_after();  // S(j) is ready, and with it every earlier MMA of this tile: O holds P V up to j-1
                // number of keys of this key tile the row may see
                int limit = item.len_kv - j * kTile;
                if (p.causal) limit = min(limit, max(turn + item.shift, 0) + 1 - j * kTile);
                limit = real ? limit : 0;
                const int low = WINDOW ? turn + item.shift - p.window + 1 - j * kTile : 0;  // first column the row sees
                const bool partial = __any_sync(0xffffffffu, limit < kTile);
                const bool lower = WINDOW && __any_sync(0xffffffffu, low > 0);
                if (TENSOR) seen = seen || max(low, 0) < min(limit, kTile);

                if (SAFE || j == my_first || (WINDOW && __any_sync(0xffffffffu, unseen))) {
                    float wanted;
                    if (WINDOW && lower) {
                        wanted = tile_max<kMaskBoth>(tmem_s, low, limit, sign);
                    } else if (partial || sign < 0.0f) {
                        wanted = tile_max<kMaskEnd>(tmem_s, low, limit, sign);
                    } else {
                        wanted = tile_max<kMaskNone>(tmem_s, low, limit, sign);
                    }
                    wanted = fmaxf(base_log2, wanted * fabsf(p.scale_log2));
                    wanted = wanted == -INFINITY ? 0.0f : wanted;  // nothing visible yet: any base will do
                    const bool free_base = WINDOW && unseen;
                    if (WINDOW && unseen && max(low, 0) < min(limit, kTile)) unseen = false;
                    // Re-base O only when some row's max grew past the threshold; then every row of the warp does.
                    const bool grow = !free_base && wanted > base_log2 + kRescaleThreshold;
                    if (__any_sync(0xffffffffu, grow)) {
                        if (j > my_first) {
                            const float factor = free_base ? 1.0f : exp2_approx(base_log2 - wanted);
                            row_sum *= factor;
                            scale_o_row<HD>(tmem_o, factor);
                        }
                        base_log2 = wanted;
                    }
                    if (free_base) base_log2 = unseen ? -INFINITY : wanted;
                } else if (__any_sync(0xffffffffu, row_sum > kRebaseLimit)) {
                    // Single-pass tiles: pull the row back by the exponent of its sum, an exact power of two.
                    const int exponent = row_sum > kRebaseLimit ? ((__float_as_int(row_sum) >> 23) & 0xff) - 127 : 0;
                    const float factor = __int_as_float((127 - exponent) << 23);
                    row_sum *= factor;
                    base_log2 += static_cast<float>(exponent);
                    scale_o_row<HD>(tmem_o, factor);
                }
                const float bias = WINDOW && unseen ? 0.0f : -base_log2;
                const float2 bias2 = make_float2(bias, bias);
                float2 sum[2] = {make_float2(row_sum, 0.0f), make_float2(0.0f, 0.0f)};
                if (WINDOW && lower) {
                    tile_exp<T, kMaskBoth, TENSOR>(tmem_s, scale2, bias2, low, limit, sum, bar_p_full + x * 16, lane);
                } else if (partial) {
                    tile_exp<T, kMaskEnd, TENSOR>(tmem_s, scale2, bias2, low, limit, sum, bar_p_full + x * 16, lane);
                } else {
                    tile_exp<T, kMaskNone, TENSOR>(tmem_s, scale2, bias2, low, limit, sum, bar_p_full + x * 16, lane);
                }
                row_sum = (sum[0].x + sum[0].y) + (sum[1].x + sum[1].y);
                in_range = in_range && row_sum < kOverflowLimit;  // false for inf and NaN too
            }
            if (failed) break;
            // ---- epilogue: O / sum -> bf16, LSE ----
            if (!__all_sync(0xffffffffu, mbar_wait(bar_o_full + x * 8, o_uses & 1) ? 1 : 0)) {
                failed = true;
                break;
            }
            ++o_uses;
            tcgen05_fence_after();
            // TENSOR, an alternating item: tile B's warps hand base and sum of their rows to tile A's, which fold the two
            // outputs (both lie in tensor-memory lanes they may read) and store.  A place whose keys were visible but left no
            // weight, or that left the range, passes a NaN.
            float mine = 1.0f, others = 0.0f;  // weights of the two outputs
            if constexpr (TENSOR) {
                if (alternate) {
                    if (row_sum == 0.0f) base_log2 = -INFINITY;
                    if (!in_range || (seen && row_sum == 0.0f)) row_sum = __int_as_float(0x7fc00000);
                    if (x == 1) {
                        share[local_row].x = base_log2;
                        share[local_row].y = row_sum;
                        __syncwarp();
                        if (lane == 0) mbar_arrive(bar_share);
                        continue;
                    }
                    // tile B's output: complete before its warps arrived, the second wait orders this thread's reads
                    const bool there = mbar_wait(bar_share, shares & 1) && mbar_wait(bar_o_full + 8, others_done & 1);
                    if (!__all_sync(0xffffffffu, there ? 1 : 0)) {
                        failed = true;
                        break;
                    }
                    ++shares;
                    ++others_done;
                    tcgen05_fence_after();
                    const float base_b = share[local_row].x, sum_b = share[local_row].y;
                    const float base = fmaxf(base_log2, base_b);
                    mine = base_log2 == -INFINITY ? 0.0f : exp2_approx(base_log2 - base);
                    others = base_b == -INFINITY ? 0.0f : exp2_approx(base_b - base);
                    row_sum = row_sum * mine + sum_b * others;   // (no weight: 0 * 0, or a NaN that stays one)
                    in_range = in_range && row_sum < kOverflowLimit;
                    base_log2 = base;
                } else if (x == 0 && item.tiles[1] > 0) {
                    ++others_done;
                }
            }
            const bool empty = row_sum == 0.0f;
            float inverse = empty ? 0.0f : 1.0f / row_sum;
            if (WINDOW && p.gate != nullptr) {
                inverse /= 1.0f + __expf(-__bfloat162float(p.gate[token * p.gate_stride + item.head]));
            }
            float probes[4] = {0.0f, 0.0f, 0.0f, 0.0f};   // TENSOR: a NaN once an output is not finite
            const bool sectors = (reinterpret_cast<uintptr_t>(p.out) & 31u) == 0;  // whole sectors a lane
#pragma unroll 1
            for (int c = 0; c < HD; c += 32) {
                uint32_t r[32];
                tmem_ld_x32(tmem_o + c, r);
                if constexpr (TENSOR) {
                    if (alternate) {
                        uint32_t b[32];
                        tmem_ld_x32(tmem_o + HD + c, b);
                        tmem_wait_ld_into(r);
                        tmem_wait_ld_into(b);
#pragma unroll
                        for (int i = 0; i < 32; ++i) {
                            r[i] = __float_as_uint(__uint_as_float(r[i]) * mine + __uint_as_float(b[i]) * others);
                        }
                    }
                }
                if (!alternate) tmem_wait_ld_into(r);
                if (TENSOR) {
#pragma unroll
                    for (int i = 0; i < 32; ++i) probes[i % 4] = fmaf(__uint_as_float(r[i]) * inverse, 0.0f, probes[i % 4]);
                }
                if (c + 32 == HD) {
                    // O is out of tensor memory: the next item's first P V may overwrite it
                    tcgen05_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(bar_o_empty + x * 8);
                    if (lane == 0 && alternate) mbar_arrive(bar_o_empty + 8);
                }
                if (real) {
#pragma unroll
                    for (int i = 0; i < 32; i += 16) {
                        uint32_t words[8];
#pragma unroll
                        for (int n = 0; n < 8; ++n) {
                            words[n] = empty ? 0u : pack2<T>(__uint_as_float(r[i + 2 * n]) * inverse, __uint_as_float(r[i + 2 * n + 1]) * inverse);
                        }
                        if (sectors) {
                            store_sector(dst + c + i, words);
                        } else {
                            reinterpret_cast<uint4 *>(dst + c + i)[0] = make_uint4(words[0], words[1], words[2], words[3]);
                            reinterpret_cast<uint4 *>(dst + c + i)[1] = make_uint4(words[4], words[5], words[6], words[7]);
                        }
                    }
                }
            }
            if (real) {
                float value = empty ? -1.0e20f : (base_log2 + log2f(row_sum)) * 0.6931471805599453f;
                if constexpr (TENSOR) {
                    value = base_log2 + log2f(row_sum);
                    if (!in_range || empty || isnan((probes[0] + probes[1]) + (probes[2] + probes[3]))) value = __int_as_float(0x7fc00000);  // has the row done again: see left_rows_kernel
                } else if (!SAFE && !in_range) {
                    value = __int_as_float(0x7fc00000);  // has the second launch redo the item
                    atomicExch(&g_out_of_range_seen, 1u);
                }
                *lse_row = value;
            }
        }
    }
    if (failed && lane == 0) {
        report_status(p.error, kStatusWaitTimeout);
    }
    if (failed) linger_after_timeout();
    tcgen05_fence_before();
    __syncthreads();
    if (warp == 8) {
        tcgen05_fence_after();
        tmem_dealloc(tmem_base, 512);
    }
}

constexpr int kPrefillSmem = 6 * kTileBytes + 8 * 22 + 32 + kMaxRankTiles * 4 + kRedoCapacity * 4 + 1024;
constexpr int kPrefillBytes = kPrefillSmem + kHeldItems * static_cast<int>(sizeof(Item));
static_assert(kPrefillBytes <= 227 * 1024, "shared memory of one CTA");

}  // namespace

bool prefill_fast_path(size_t heads, size_t kv_heads, size_t head_dim, size_t total_query_tokens, const void *query,
                       const void *key, const void *value, const void *out) {
    // The heaviest-first item table holds kMaxRankTiles query pairs per sequence.
    if (total_query_tokens / kPair + 1 > kMaxRankTiles) return false;
    const uintptr_t all = reinterpret_cast<uintptr_t>(query) | reinterpret_cast<uintptr_t>(key) |
                          reinterpret_cast<uintptr_t>(value) | reinterpret_cast<uintptr_t>(out);
    return (head_dim == 128 || head_dim == 64) && heads % kv_heads == 0 && heads <= 65535 && (all & 15u) == 0;
}

namespace {

template <typename T, int HD, bool PAGED, bool DENSE, bool WINDOW, bool LONE>
int launch_passes(cudaStream_t stream, const CUtensorMap &q_map, const CUtensorMap &k_map, const CUtensorMap &v_map,
                  const PrefillParams &params, unsigned persistent) {
    constexpr bool kTwo = std::is_same<T, __nv_bfloat16>::value;
    const auto exact = prefill_tcgen05_kernel<T, HD, true, PAGED, DENSE, WINDOW, false, LONE && !kTwo>;
    SINGE_CUDA_TRY(cudaFuncSetAttribute(exact, cudaFuncAttributeMaxDynamicSharedMemorySize, kPrefillBytes));
    if (kTwo) {
        const auto first = prefill_tcgen05_kernel<__nv_bfloat16, HD, false, PAGED, DENSE, WINDOW, false, LONE>;
        SINGE_CUDA_TRY(cudaFuncSetAttribute(first, cudaFuncAttributeMaxDynamicSharedMemorySize, kPrefillBytes));
        first<<<persistent, kPrefillThreads, kPrefillBytes, stream>>>(q_map, k_map, v_map, params, NoPaging{});
        SINGE_TRY(launch_status());
    }
    // bf16: the redo pass over the same shares, a no-op while the device's out-of-range flag has never been raised.
    // f16 (params.exact): the only pass.  P must stay below 65504 there, so every tile takes its exact row maximum.
    exact<<<persistent, kPrefillThreads, kPrefillBytes, stream>>>(q_map, k_map, v_map, params, NoPaging{});
    return launch_status();
}

// One CTA for each of at most `items` items, or one for each of the `sms` SMs.
template <typename T, int HD, bool PAGED, bool DENSE = false, bool WINDOW = false>
int launch_prefill(cudaStream_t stream, const CUtensorMap &q_map, const CUtensorMap &k_map, const CUtensorMap &v_map,
                   const PrefillParams &params, size_t items, size_t sms) {
    if (items <= sms) {
        return launch_passes<T, HD, PAGED, DENSE, WINDOW, true>(stream, q_map, k_map, v_map, params, static_cast<unsigned>(items));
    }
    return launch_passes<T, HD, PAGED, DENSE, WINDOW, false>(stream, q_map, k_map, v_map, params, static_cast<unsigned>(sms));
}

template <int HD, bool WINDOW>
int launch_tensor(cudaStream_t stream, const CUtensorMap &q_map, const CUtensorMap &k_map, const CUtensorMap &v_map,
                  const PrefillParams &params, const TensorPaging &paging, unsigned persistent) {
    static int raised[kMaxDevices] = {0};
    constexpr int kBytes = kPrefillSmem + (4 * kMaxTensorSequences - kRedoCapacity + 3 * kMaxOrdered) * 4 +
                           (kTensorBarriers - 22) * 8 + kTile * 8;
    static_assert(kBytes <= 227 * 1024, "shared memory of one CTA");
    const auto kernel = prefill_tcgen05_kernel<__nv_bfloat16, HD, false, true, false, WINDOW, true>;
    SINGE_CUDA_TRY(ensure_dynamic_shared(kernel, kBytes, raised));
    kernel<<<persistent, kPrefillThreads, kBytes, stream>>>(q_map, k_map, v_map, params, paging);
    return launch_status();
}

// log2 of the query heads of a key/value head whose rows stand together: all of a group that divides a tile, else one.
int pack_of(size_t heads, size_t kv_heads) {
    const size_t group = heads / kv_heads;
    for (int pack = 0; pack <= 4; ++pack) {
        if (group == (size_t{1} << pack)) return pack;
    }
    return 0;
}

}  // namespace

// Packed queries over packed keys/values (block_table == nullptr: key/value are [total_kv_tokens, kv_heads, 128]) or
// over a paged cache (key/value are [cache_pages, 16, kv_heads, 128], rows of block_table [batch, table_stride] list
// each sequence's pages).  lens_q == nullptr selects the dense form: `uniform_q` queries and `uniform_kv` keys per
// sequence, back to back, and an LSE laid out [batch, heads, uniform_q].  is_f16: IEEE half instead of bf16.
int prefill_tcgen05(cudaStream_t stream, bool is_f16, void *out, float *lse, const void *query, const void *key,
                    const void *value, const int32_t *lens_q, const int32_t *lens_kv, const int32_t *offsets,
                    size_t batch, size_t total_query_tokens, size_t total_kv_tokens, size_t heads, size_t kv_heads,
                    size_t head_dim, int causal, float scale, const uint32_t *block_table, size_t table_stride,
                    size_t cache_pages, size_t uniform_q, size_t uniform_kv) {
    if (head_dim != 128 && head_dim != 64) return SINGE_ERR_UNSUPPORTED_WIDTH;
    const uint64_t kHeadDim = head_dim;
    int device = 0, sms = 0;
    SINGE_CUDA_TRY(cudaGetDevice(&device));
    SINGE_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device));
    const bool paged = block_table != nullptr;
    const CUtensorMapDataType type = is_f16 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16;
    CUtensorMap q_map, k_map, v_map;
    const uint32_t box[3] = {64, 1, kTile};
    {
        const uint64_t dims[3] = {kHeadDim, heads, total_query_tokens};
        const uint64_t strides[2] = {kHeadDim * 2, kHeadDim * 2 * heads};
        SINGE_TRY(encode_tensor_map(&q_map, type, 3, query, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_128B,
                                    CU_TENSOR_MAP_L2_PROMOTION_L2_256B));
    }
    if (paged) {
        const uint64_t dims[4] = {kHeadDim, kv_heads, kPageTokens, cache_pages};
        const uint64_t strides[3] = {kHeadDim * 2, kHeadDim * 2 * kv_heads, kHeadDim * 2 * kv_heads * kPageTokens};
        const uint32_t page_box[4] = {64, 1, kPageTokens, 1};
        SINGE_TRY(encode_tensor_map(&k_map, type, 4, key, dims, strides, page_box, CU_TENSOR_MAP_SWIZZLE_128B,
                                    CU_TENSOR_MAP_L2_PROMOTION_L2_256B));
        SINGE_TRY(encode_tensor_map(&v_map, type, 4, value, dims, strides, page_box, CU_TENSOR_MAP_SWIZZLE_128B,
                                    CU_TENSOR_MAP_L2_PROMOTION_L2_256B));
    } else {
        const uint64_t dims[3] = {kHeadDim, kv_heads, total_kv_tokens};
        const uint64_t strides[2] = {kHeadDim * 2, kHeadDim * 2 * kv_heads};
        SINGE_TRY(encode_tensor_map(&k_map, type, 3, key, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_128B,
                                    CU_TENSOR_MAP_L2_PROMOTION_L2_256B));
        SINGE_TRY(encode_tensor_map(&v_map, type, 3, value, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_128B,
                                    CU_TENSOR_MAP_L2_PROMOTION_L2_256B));
    }
    PrefillParams params = {};
    params.out = out;
    params.lse = lse;
    params.lens_q = lens_q;
    params.lens_kv = lens_kv;
    params.offsets = offsets;
    params.uniform_q = static_cast<int>(uniform_q);
    params.uniform_kv = static_cast<int>(uniform_kv);
    params.lse_rows = lens_q == nullptr ? static_cast<int>(uniform_q) : 0;
    params.exact = is_f16 ? 1 : 0;
    params.batch = static_cast<int>(batch);
    params.heads = static_cast<int>(heads);
    params.kv_heads = static_cast<int>(kv_heads);
    params.total_q = static_cast<int>(total_query_tokens);
    params.total_kv = static_cast<int>(total_kv_tokens);
    params.block_table = block_table;
    params.table_stride = static_cast<int>(table_stride);
    params.cache_pages = static_cast<int>(cache_pages);
    params.causal = causal == 2 ? 2 : (causal ? 1 : 0);
    params.scale_log2 = scale * 1.4426950408889634f;
    params.error = device_error_word();
    // Upper bound on the items: every sequence can add one partial 256-row pair.
    const size_t items = (total_query_tokens / kPair + batch) * heads;
    if (items > 0x7fffffffull) return SINGE_ERR_LENGTH_EXCEEDS_I32;
    if (items == 0) return SINGE_OK;
    if (lens_q == nullptr) {
        // the dense form: ragged keys only
        if (paged) return SINGE_ERR_UNSUPPORTED_CONFIGURATION;
        if (head_dim == 64) {
            return is_f16 ? launch_prefill<__half, 64, false, true>(stream, q_map, k_map, v_map, params, items, sms)
                          : launch_prefill<__nv_bfloat16, 64, false, true>(stream, q_map, k_map, v_map, params, items, sms);
        }
        return is_f16 ? launch_prefill<__half, 128, false, true>(stream, q_map, k_map, v_map, params, items, sms)
                      : launch_prefill<__nv_bfloat16, 128, false, true>(stream, q_map, k_map, v_map, params, items, sms);
    }
    if (head_dim == 64) {
        if (is_f16) {
            return paged ? launch_prefill<__half, 64, true>(stream, q_map, k_map, v_map, params, items, sms)
                         : launch_prefill<__half, 64, false>(stream, q_map, k_map, v_map, params, items, sms);
        }
        return paged ? launch_prefill<__nv_bfloat16, 64, true>(stream, q_map, k_map, v_map, params, items, sms)
                     : launch_prefill<__nv_bfloat16, 64, false>(stream, q_map, k_map, v_map, params, items, sms);
    }
    if (is_f16) {
        return paged ? launch_prefill<__half, 128, true>(stream, q_map, k_map, v_map, params, items, sms)
                     : launch_prefill<__half, 128, false>(stream, q_map, k_map, v_map, params, items, sms);
    }
    return paged ? launch_prefill<__nv_bfloat16, 128, true>(stream, q_map, k_map, v_map, params, items, sms)
                 : launch_prefill<__nv_bfloat16, 128, false>(stream, q_map, k_map, v_map, params, items, sms);
}

// The windowed form: keys and values are rows of kv_row_stride elements (heads side by side) with offsets of their own;
// the queries are their sequences' last tokens.
int prefill_tcgen05_windowed(cudaStream_t stream, void *out, float *lse, const void *query, const void *key,
                             const void *value, size_t kv_row_stride, const int32_t *lens_q, const int32_t *lens_kv,
                             const int32_t *offsets_q, const int32_t *offsets_kv, const void *gate, size_t gate_stride,
                             size_t batch, size_t total_query_tokens, size_t total_kv_tokens, size_t heads,
                             size_t kv_heads, size_t head_dim, size_t window, float scale) {
    const uint64_t kHeadDim = head_dim;
    const CUtensorMapDataType type = CU_TENSOR_MAP_DATA_TYPE_BFLOAT16;
    CUtensorMap q_map, k_map, v_map;
    const uint32_t box[3] = {64, 1, kTile};
    const uint64_t q_dims[3] = {kHeadDim, heads, total_query_tokens};
    const uint64_t q_strides[2] = {kHeadDim * 2, kHeadDim * 2 * heads};
    const uint64_t kv_dims[3] = {kHeadDim, kv_heads, total_kv_tokens};
    const uint64_t kv_strides[2] = {kHeadDim * 2, static_cast<uint64_t>(kv_row_stride) * 2};
    SINGE_TRY(encode_tensor_map(&q_map, type, 3, query, q_dims, q_strides, box, CU_TENSOR_MAP_SWIZZLE_128B,
                                CU_TENSOR_MAP_L2_PROMOTION_L2_256B));
    SINGE_TRY(encode_tensor_map(&k_map, type, 3, key, kv_dims, kv_strides, box, CU_TENSOR_MAP_SWIZZLE_128B,
                                CU_TENSOR_MAP_L2_PROMOTION_L2_256B));
    SINGE_TRY(encode_tensor_map(&v_map, type, 3, value, kv_dims, kv_strides, box, CU_TENSOR_MAP_SWIZZLE_128B,
                                CU_TENSOR_MAP_L2_PROMOTION_L2_256B));
    PrefillParams params = {};
    params.out = out;
    params.lse = lse;
    params.lens_q = lens_q;
    params.lens_kv = lens_kv;
    params.offsets = offsets_q;
    params.offsets_kv = offsets_kv;
    params.batch = static_cast<int>(batch);
    params.heads = static_cast<int>(heads);
    params.kv_heads = static_cast<int>(kv_heads);
    params.total_q = static_cast<int>(total_query_tokens);
    params.total_kv = static_cast<int>(total_kv_tokens);
    params.causal = 2;
    params.scale_log2 = scale * 1.4426950408889634f;
    params.error = device_error_word();
    params.window = static_cast<int>(window);
    params.gate = static_cast<const __nv_bfloat16 *>(gate);
    params.gate_stride = static_cast<long long>(gate_stride);
    const size_t items = (total_query_tokens / kPair + batch) * heads;
    if (items > 0x7fffffffull) return SINGE_ERR_LENGTH_EXCEEDS_I32;
    const size_t sms = static_cast<size_t>(device_sm_count());
    if (head_dim == 64) {
        return launch_prefill<__nv_bfloat16, 64, false, false, true>(stream, q_map, k_map, v_map, params, items, sms);
    }
    return launch_prefill<__nv_bfloat16, 128, false, false, true>(stream, q_map, k_map, v_map, params, items, sms);
}

// Whether tensor_prefill serves a call of the Tensor surface's paged attention (bf16, no score cap).
bool tensor_prefill_takes(size_t tokens, size_t heads, size_t kv_heads, size_t head_dim, size_t page_size, size_t cache_pages,
                          size_t sequences, size_t table_len, int causal, size_t window, const void *query, const void *key_cache,
                          const void *value_cache, const void *out) {
    const size_t rows = tokens << pack_of(heads, kv_heads);
    return page_size == kPageTokens && cache_pages > 0 && sequences <= kMaxTensorSequences &&
           table_len <= 0x7fffffff / kPageTokens - kTile &&
           (window == 0 || (causal && window <= 0x3fffffff)) && rows <= 0x7fffffff / 2 &&
           prefill_fast_path(heads, kv_heads, head_dim, rows, query, key_cache, value_cache, out);
}

// Tensor::paged_attention over 16-token pages; left_rows_kernel has to follow on the stream.
int tensor_prefill(cudaStream_t stream, void *out, float *lse, const void *query, const void *key_cache, const void *value_cache,
                   const void *query_offsets, const void *page_offsets, const void *pages, const void *last_page_lengths,
                   int index_width, size_t tokens, size_t heads, size_t kv_heads, size_t head_dim, size_t cache_pages,
                   size_t sequences, size_t table_len, float scale, int causal, size_t window, uint32_t *status) {
    const int pack = pack_of(heads, kv_heads);
    const uint64_t width = head_dim;
    const CUtensorMapDataType type = CU_TENSOR_MAP_DATA_TYPE_BFLOAT16;
    CUtensorMap q_map, k_map, v_map;
    const uint64_t q_dims[3] = {width, heads, tokens};
    const uint64_t q_strides[2] = {width * 2, width * 2 * heads};
    const uint32_t q_box[3] = {64, 1u << pack, static_cast<uint32_t>(kTile >> pack)};
    SINGE_TRY(encode_tensor_map(&q_map, type, 3, query, q_dims, q_strides, q_box, CU_TENSOR_MAP_SWIZZLE_128B,
                                CU_TENSOR_MAP_L2_PROMOTION_L2_256B));
    const uint64_t dims[4] = {width, kv_heads, kPageTokens, cache_pages};
    const uint64_t strides[3] = {width * 2, width * 2 * kv_heads, width * 2 * kv_heads * kPageTokens};
    const uint32_t box[4] = {64, 1, kPageTokens, 1};
    SINGE_TRY(encode_tensor_map(&k_map, type, 4, key_cache, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_128B,
                                CU_TENSOR_MAP_L2_PROMOTION_L2_256B));
    SINGE_TRY(encode_tensor_map(&v_map, type, 4, value_cache, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_128B,
                                CU_TENSOR_MAP_L2_PROMOTION_L2_256B));
    PrefillParams params = {};
    params.out = out;
    params.lse = lse;
    params.batch = static_cast<int>(sequences);
    params.heads = static_cast<int>(heads >> pack);
    params.kv_heads = static_cast<int>(kv_heads);
    params.total_q = static_cast<int>(tokens);
    params.cache_pages = static_cast<int>(cache_pages);
    params.causal = causal ? 1 : 0;
    params.scale_log2 = scale * 1.4426950408889634f;
    params.error = device_error_word();
    params.window = static_cast<int>(window);
    TensorPaging paging = {query_offsets, page_offsets, pages, last_page_lengths, index_width, static_cast<int>(sequences),
                           static_cast<int>(tokens), static_cast<int>(table_len), pack, status};
    const size_t items = ((tokens << pack) / kPair + sequences) * (heads >> pack);
    if (items > 0x7fffffffull) return SINGE_ERR_LENGTH_EXCEEDS_I32;
    const size_t sms = static_cast<size_t>(device_sm_count());
    const unsigned persistent = static_cast<unsigned>(items < sms ? items : sms);
    if (head_dim == 64) {
        return window > 0 ? launch_tensor<64, true>(stream, q_map, k_map, v_map, params, paging, persistent)
                          : launch_tensor<64, false>(stream, q_map, k_map, v_map, params, paging, persistent);
    }
    return window > 0 ? launch_tensor<128, true>(stream, q_map, k_map, v_map, params, paging, persistent)
                      : launch_tensor<128, false>(stream, q_map, k_map, v_map, params, paging, persistent);
}

int prefill_tcgen05_bf16(cudaStream_t stream, void *out, float *lse, const void *query, const void *key,
                         const void *value, const int32_t *lens_q, const int32_t *lens_kv, const int32_t *offsets,
                         size_t batch, size_t total_query_tokens, size_t total_kv_tokens, size_t heads,
                         size_t kv_heads, size_t head_dim, int causal, float scale, const uint32_t *block_table,
                         size_t table_stride, size_t cache_pages) {
    return prefill_tcgen05(stream, false, out, lse, query, key, value, lens_q, lens_kv, offsets, batch,
                           total_query_tokens, total_kv_tokens, heads, kv_heads, head_dim, causal, scale, block_table,
                           table_stride, cache_pages, 0, 0);
}

}  // namespace singe

extern "C" int singe_windowed_prefill_attention_bf16(
    singe_stream_t stream, void *out, float *lse, const void *query, const void *key, const void *value,
    size_t kv_row_stride, const int32_t *lens_q, const int32_t *lens_kv, const int32_t *offsets_q,
    const int32_t *offsets_kv, const void *gate, size_t gate_row_stride, size_t batch, size_t total_query_tokens,
    size_t total_kv_tokens, size_t heads, size_t kv_heads, size_t head_dim, size_t window, float scale) {
    using namespace singe;
    if (batch == 0 || total_query_tokens == 0 || total_kv_tokens == 0 || heads == 0 || kv_heads == 0 || heads % kv_heads != 0 ||
        window == 0 || kv_row_stride < kv_heads * head_dim || (gate != nullptr && gate_row_stride < heads) || !(scale == scale)) {
        return SINGE_ERR_INVALID_LENGTH;
    }
    if (!fits_i32(batch) || !fits_i32(total_query_tokens) || !fits_i32(total_kv_tokens) || !fits_i32(heads) ||
        !fits_i32(window)) {
        return SINGE_ERR_LENGTH_EXCEEDS_I32;
    }
    if (out == nullptr || lse == nullptr || query == nullptr || key == nullptr || value == nullptr || lens_q == nullptr ||
        lens_kv == nullptr || offsets_q == nullptr || offsets_kv == nullptr) {
        return SINGE_ERR_NULL_POINTER;
    }
    if (kv_row_stride % 8 != 0 || !prefill_fast_path(heads, kv_heads, head_dim, total_query_tokens, query, key, value, out)) {
        return SINGE_ERR_UNSUPPORTED_CONFIGURATION;
    }
    return prefill_tcgen05_windowed(static_cast<cudaStream_t>(stream), out, lse, query, key, value, kv_row_stride, lens_q,
                                    lens_kv, offsets_q, offsets_kv, gate, gate_row_stride, batch, total_query_tokens,
                                    total_kv_tokens, heads, kv_heads, head_dim, window, scale);
}
