// Paged-KV flash-decode whose CTAs share the cached keys of all sequences evenly: the pages of a call, counted over its
// sequences one after the other, are cut into as many equal runs as there are SMs, and a CTA reads whole pages, all KV
// heads of them.  Same meaning, softmax and tensor-core tiles as paged_decode.cu
// (paged_kv_decode_attention, singe-kernel/src/cpu/attention.rs:1172-1246); for calls whose (sequence, KV head, split)
// grid would take more than one wave there.
//
// Bound by HBM (4 * kv_heads * head_dim bytes per cached token).  What the split grid loses, and this one does not:
//   * a page's row of one head is 256 bytes at a stride of 2 KB, and the heads' CTAs read theirs at different times; here one
//     box brings the 16 tokens of all heads, 16 KB that lie together (probe without arithmetic, 4000 random pages
//     of 64 KB: 5.85 TB/s by heads, 6.30 by whole pages; 8192 pages: 6.15 and 6.6);
//   * pieces of equal size leave SMs idle in the last wave (2049 keys x 64 sequences: 4.6 waves of 512 keys) and ragged
//     lengths make it worse; here every SM gets the same number of pages to within one.
// Measured, bf16 and f16 (us, by the split grid and here, with the fold): 32 sequences of 128 - 4096 keys, 8 heads of 128 57.1 and
// 52.5; 64 x 1024 59.5 and 49.3; 4 x 4096 24.7 and 18.0; 32 x 4096 of 64 61.3 and 49.6.  A Llama-shaped decode step of 64 x 2048
// keys over six layers 1462 and 1384.  Against 64 bits the error is 0.84 of the split grid's (2.0e-3 -> 1.7e-3, the rounding of the
// output): the weights of cached keys enter the value product as two terms, in rows of the 16-row tile that carry no query head.  The
// one key that a fused step adds keeps the single rounded weight it has there.
// Structure: one persistent CTA per SM.  Warp 8 (producer) brings K and V of a step -- eight (page, head) tiles, so one page of
// eight heads or two of four -- into a ring of 32 KB slots (K and V have slots of their own, so that K's is free while V is
// read); warp w < 8 owns head w % kv_heads and, with four heads, every other page; one tile a step, ldmatrix from the
// swizzled slot, m16n8k16, online softmax in f32 as there.  A run of pages crosses sequences: at each sequence's end in it a
// warp writes its rows, the result if the run holds the whole sequence, else a normalised partial and its log sum that
// even_combine_kernel folds.  A (CTA, sequence) segment is the only one with its CTA + sequence, which is its scratch slot, and
// a sequence's segments stand in adjacent slots.
// Every wait on an mbarrier is bounded; on a timeout the CTA records status 2 and leaves.
#include "paged_decode.cuh"

namespace singe {

namespace {

constexpr int kEvenWarps = 8;
constexpr int kEvenThreads = (kEvenWarps + 1) * 32;
constexpr int kEvenRing = 192 * 1024;       // bytes of the ring
constexpr int kEvenMaxBatch = 2048;         // sequences of one call (their running page counts stand in shared memory)
constexpr int kEvenMaxCtas = 256;
constexpr int kEvenLeastPages = 2;          // pages a CTA takes at least: a segment of one page is mostly set-up and fold
constexpr int kEvenPlain = 0, kEvenFused = 1, kEvenChunked = 2;

// What a CTA finds at the head of the scratch's last slot: per sequence, how many segments it has and the slot of the first.
struct EvenRow {
    int segments, slot;
};

template <int HD>
constexpr int even_slot_bytes() {
    return kEvenWarps * (HD / 64) * kHalfBytes;
}

template <int HD>
constexpr int even_slots() {
    return kEvenRing / even_slot_bytes<HD>();
}

template <int HD, int KVH>
constexpr int even_merge_bytes() {
    return KVH == kEvenWarps ? 0 : KVH * 8 * (HD + 2) * 4;
}

// (what a call of few sequences leaves of an SM's shared memory is for the CTAs of kernels beside it)
template <int HD, int KVH>
constexpr int even_smem_bytes(int batch) {
    return kEvenRing + even_merge_bytes<HD, KVH>() + 16 * even_slots<HD>() + 16 * KVH + 40 + (2 * batch + 1) * 4 + 1024;
}

// What a sequence (chunked form: a query) reads.
struct EvenSequence {
    int first_page;
    int keys;      // cached keys it sees, from the first page's first slot on
    int hidden;    // of these, how many at the front are hidden (chunked form)
    int real;      // pages that hold them
    int counted;   // pages it counts as: one at least, so that every sequence has a segment
};

// The length of sequence b, 0 where it has nothing to read.
template <int FORM>
__device__ __forceinline__ int even_length(const DecodeParams &p, const ChunkedDecode &chunked, int b) {
    const int len = p.lens[b];
    const int bound = p.table_stride * kPageTokens;
    if (FORM == kEvenChunked) {
        const int sequence = chunked.sequence_of[b];
        if (sequence < 0 || sequence >= chunked.sequences || len > bound) {
            if (blockIdx.x == 0) report_status(p.status, kStatusIndexOutOfBounds);
            return 0;
        }
    }
    return len < 0 ? 0 : (len > bound ? bound : len);
}

template <int FORM>
__device__ __forceinline__ EvenSequence even_sequence(const ChunkedDecode &chunked, int len) {
    EvenSequence s = {0, len, 0, 0, 1};
    if (FORM == kEvenChunked && len > 0) {
        const int start = (len - 1) / chunked.size * chunked.size;
        s.first_page = start / kPageTokens;
        s.hidden = start - s.first_page * kPageTokens;
        s.keys = len - s.first_page * kPageTokens;
    }
    if (FORM == kEvenFused) s.keys = max(len - 1, 0);   // the step's own key is not in the cache yet
    s.real = (s.keys + kPageTokens - 1) / kPageTokens;
    s.counted = max(s.real, 1);
    return s;
}

// What rounding a pair of values to `lead` left out, rounded itself.
template <typename T>
__device__ __forceinline__ uint32_t pack_rest(uint32_t lead, float low, float high) {
    T rounded[2];
    *reinterpret_cast<uint16_t *>(&rounded[0]) = static_cast<uint16_t>(lead & 0xffffu);
    *reinterpret_cast<uint16_t *>(&rounded[1]) = static_cast<uint16_t>(lead >> 16);
    return pack2<T>(low - to_float<T>(rounded[0]), high - to_float<T>(rounded[1]));
}

template <typename T, int HD, int KVH, int FORM>
__global__ void __launch_bounds__(kEvenThreads, 1)
    paged_decode_even_kernel(const __grid_constant__ CUtensorMap k_map, const __grid_constant__ CUtensorMap v_map,
                             const DecodeParams p, const StepExtras x, const ChunkedDecode chunked, EvenRow *rows) {
    constexpr int NHALF = HD / 64;
    constexpr int KSTEPS = HD / 16;
    constexpr int NTILES = HD / 8;
    constexpr int SLOT = even_slot_bytes<HD>();
    constexpr int SLOTS = even_slots<HD>();
    constexpr int STEP_PAGES = kEvenWarps / KVH;     // pages of one step
    constexpr int BOX = KVH * kHalfBytes;            // 16 tokens x 128 bytes of every head
    static_assert(SLOTS % 2 == 0, "K and V take turns");
    extern __shared__ uint8_t smem_raw[];
    const uint32_t raw = smem_u32(smem_raw);
    const uint32_t base = (raw + 1023u) & ~1023u;
    uint8_t *aligned = smem_raw + (base - raw);
    float *merge = reinterpret_cast<float *>(aligned + kEvenRing);   // [KVH][8 rows][HD + 2]
    const uint32_t bar_full = base + kEvenRing + even_merge_bytes<HD, KVH>();
    const uint32_t bar_empty = bar_full + 8 * SLOTS;
    const uint32_t bar_merge = bar_empty + 8 * SLOTS;   // [KVH][written, read]
    int *warp_pages = reinterpret_cast<int *>(aligned + kEvenRing + even_merge_bytes<HD, KVH>() + 16 * SLOTS + 16 * KVH);   // [warps]
    int *before = warp_pages + 10;            // [batch + 1]: pages before sequence b
    int *lengths = before + p.batch + 1;      // [batch]
    const int tid = threadIdx.x;
    const int warp = tid >> 5;
    const int lane = tid & 31;
    // Fused step: lengths, table and cached rows may be read ahead of the kernels before (see StepExtras), the new row is this
    // kernel's own.
    const bool stable = FORM == kEvenFused && x.stable_paging != 0;

    if (tid == 0) {
        for (int i = 0; i < SLOTS; ++i) {
            mbar_init(bar_full + 8 * i, 1);
            mbar_init(bar_empty + 8 * i, kEvenWarps);
        }
        for (int i = 0; i < 2 * KVH; ++i) mbar_init(bar_merge + 8 * i, 1);
        mbar_init_fence();
    }
    if (warp == kEvenWarps && lane == 0) {
        prefetch_tensor_map(&k_map);
        prefetch_tensor_map(&v_map);
    }
    if (FORM != kEvenChunked && warp == 0) warm_l2(x.warm, blockIdx.x, gridDim.x, lane);
    {
        // The table is read behind the lengths: till then every CTA has some of its lines on their way to L2 (1 % of a call).
        const size_t words = static_cast<size_t>(FORM == kEvenChunked ? chunked.sequences : p.batch) * p.table_stride;
        const size_t word = (static_cast<size_t>(tid) * gridDim.x + blockIdx.x) * 32;
        if (word < words) asm volatile("prefetch.global.L2 [%0];" ::"l"(p.table + word));
    }
    if (!stable) grid_dependency_wait();

    // ---- pages before each sequence ----
    int total = 0;
    for (int first = 0; first < p.batch; first += kEvenThreads) {
        const int b = first + tid;
        const int length = b < p.batch ? even_length<FORM>(p, chunked, b) : 0;
        const int own = b < p.batch ? even_sequence<FORM>(chunked, length).counted : 0;
        int sum = own;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const int other = __shfl_up_sync(0xffffffffu, sum, d);
            if (lane >= d) sum += other;
        }
        if (lane == 31) warp_pages[warp] = sum;
        __syncthreads();
        int ahead = total;
#pragma unroll
        for (int w = 0; w <= kEvenWarps; ++w) {
            const int pages = warp_pages[w];
            if (w < warp) ahead += pages;
            total += pages;
        }
        if (b < p.batch) {
            before[b] = ahead + sum - own;
            lengths[b] = length;
        }
        __syncthreads();
    }
    if (tid == 0) before[p.batch] = total;
    __syncthreads();

    const int wanted = (total + kEvenLeastPages - 1) / kEvenLeastPages;
    const int ctas = min(static_cast<int>(gridDim.x), wanted);
    const int cta = blockIdx.x;
    if (cta >= ctas) return;
    const int lo = static_cast<int>(static_cast<long long>(total) * cta / ctas);
    const int hi = static_cast<int>(static_cast<long long>(total) * (cta + 1) / ctas);
    int first_sequence = 0;
    {
        int right = p.batch;   // before[first_sequence] <= lo < before[right]
        while (right - first_sequence > 1) {
            const int middle = (first_sequence + right) >> 1;
            if (before[middle] <= lo) first_sequence = middle;
            else right = middle;
        }
    }

    bool failed = false;
    if (warp == kEvenWarps) {
        // ---------------- producer ----------------
        int n = 0;   // steps sent for
        for (int b = first_sequence; before[b] < hi && !failed; ++b) {
            const EvenSequence s = even_sequence<FORM>(chunked, lengths[b]);
            const int from = max(lo - before[b], 0);
            const int to = min(min(hi - before[b], s.counted), s.real);
            const uint32_t *pages =
                p.table + static_cast<size_t>(FORM == kEvenChunked && s.real > 0 ? chunked.sequence_of[b] : b) * p.table_stride + s.first_page;
            for (int chunk = from; chunk < to && !failed; chunk += 32) {
                uint32_t page = chunk + lane < to ? pages[chunk + lane] : 0u;
                if (page >= static_cast<uint32_t>(p.physical_blocks)) {
                    report_status(p.status, kStatusIndexOutOfBounds);
                    page = 0u;
                }
                const int count = min(32, to - chunk);
                for (int j = 0; j < count && !failed; j += STEP_PAGES, ++n) {
                    const int held = min(STEP_PAGES, count - j);
#pragma unroll
                    for (int which = 0; which < 2; ++which) {
                        const int item = 2 * n + which;
                        const int slot = item % SLOTS;
                        const int use = item / SLOTS;
                        if (use > 0) {
                            int ok = 1;
                            if (lane == 0) ok = mbar_wait(bar_empty + 8 * slot, (use - 1) & 1) ? 1 : 0;
                            if (__shfl_sync(0xffffffffu, ok, 0) == 0) {
                                failed = true;
                                break;
                            }
                        }
                        const uint32_t full = bar_full + 8 * slot;
                        if (lane == 0) mbar_expect_tx(full, static_cast<uint32_t>(held * NHALF * BOX));
                        const int mine = lane / NHALF;   // page of the step, and half of the head, this lane sends for
                        const uint32_t id = __shfl_sync(0xffffffffu, page, (j + mine) & 31);
                        __syncwarp();
                        if (mine < held) {
                            tma_load_4d(base + slot * SLOT + lane * BOX, which == 0 ? &k_map : &v_map, full, (lane % NHALF) * 64, 0, 0,
                                        static_cast<int32_t>(id));
                        }
                    }
                }
            }
        }
        if (failed && lane == 0) report_status(p.status, kStatusWaitTimeout);
    } else {
        // ---------------- consumers ----------------
        const int head = warp % KVH;
        const int turn = warp / KVH;     // page of a step this warp takes
        const int row = lane >> 2;       // query head within the group (rows >= group are zero padding)
        const int quad = lane & 3;
        const int mat = lane >> 3;
        const int k_tok = ((mat >> 1) << 3) + (lane & 7);
        const int k_sel = mat & 1;
        const int v_tok = ((mat & 1) << 3) + (lane & 7);
        const int v_sel = mat >> 1;
        const uint32_t tile = base + turn * NHALF * BOX + head * kHalfBytes;
        if (stable) grid_dependency_wait();
        // Ahead of every wait that may run out: the fold reads the entry of each sequence, whatever has become of its rows.
        if (warp == 0) {
            for (int b = first_sequence + (before[first_sequence] < lo ? 1 : 0) + lane; b < p.batch && before[b] < hi; b += 32) {
                const int last = static_cast<int>((static_cast<long long>(before[b + 1]) * ctas - 1) / total);
                rows[b] = {last - cta + 1, cta + b};
            }
        }
        int n = 0;        // steps taken
        int merges = 0;   // merges of the head's two warps so far
        uint32_t qa[KSTEPS][2];
        auto load_query = [&](int b) {
            const uint32_t *q32 =
                FORM == kEvenFused
                    ? reinterpret_cast<const uint32_t *>(static_cast<const T *>(x.qkv) + static_cast<size_t>(b) * x.qkv_stride +
                                                         static_cast<size_t>(head * p.group + row) * HD)
                    : reinterpret_cast<const uint32_t *>(static_cast<const T *>(p.query) +
                                                         (static_cast<size_t>(b) * p.heads + head * p.group + row) * HD);
#pragma unroll
            for (int ks = 0; ks < KSTEPS; ++ks) {
                qa[ks][0] = row < p.group ? q32[ks * 8 + quad] : 0u;
                qa[ks][1] = row < p.group ? q32[ks * 8 + 4 + quad] : 0u;
            }
        };
        load_query(first_sequence);
        for (int b = first_sequence; before[b] < hi && !failed; ++b) {
            const int len = lengths[b];
            const EvenSequence s = even_sequence<FORM>(chunked, len);
            const int from = max(lo - before[b], 0);
            const int counted_to = min(hi - before[b], s.counted);
            const int to = min(counted_to, s.real);
            const bool whole = from == 0 && counted_to == s.counted;
            const int slot_of_row = cta + b;
            if (FORM == kEvenFused) rotate_query_fragments<T, HD>(qa, p, x, b, row, quad);
            float o[NTILES][4];
#pragma unroll
            for (int nt = 0; nt < NTILES; ++nt) o[nt][0] = o[nt][1] = o[nt][2] = o[nt][3] = 0.0f;
            float run_max = -INFINITY;
            float run_sum = 0.0f;

            for (int at = from; at < to; at += STEP_PAGES, ++n) {
                const int slot_k = (2 * n) % SLOTS;
                const uint32_t parity = ((2 * n) / SLOTS) & 1;
                const bool mine = STEP_PAGES == 1 || at + turn < to;
                if (!__all_sync(0xffffffffu, mbar_wait(bar_full + 8 * slot_k, parity) ? 1 : 0)) {
                    failed = true;
                    break;
                }
                float s0[4] = {0.0f, 0.0f, 0.0f, 0.0f};
                float s1[4] = {0.0f, 0.0f, 0.0f, 0.0f};
                if (mine) {
                    const uint32_t keys = tile + slot_k * SLOT;
#pragma unroll
                    for (int ks = 0; ks < KSTEPS; ++ks) {
                        const int c = ((ks & 3) << 1) + k_sel;
                        uint32_t r0, r1, r2, r3;
                        ldmatrix_x4(keys + (ks >> 2) * BOX + k_tok * 128 + ((c ^ (k_tok & 7)) << 4), r0, r1, r2, r3);
                        mma_m16n8k16<T>(s0, qa[ks][0], 0u, qa[ks][1], 0u, r0, r1);
                        mma_m16n8k16<T>(s1, qa[ks][0], 0u, qa[ks][1], 0u, r2, r3);
                    }
                }
                __syncwarp();
                if (lane == 0) mbar_arrive(bar_empty + 8 * slot_k);
                // The weights are taken as two terms of T: rows 8-15 of the products, where no query head stands, carry what
                // rounding the leading term left out.
                uint32_t pa0 = 0u, pa1 = 0u, pa2 = 0u, pa3 = 0u;
                if (mine) {
                    // row `row` of this lane: keys t0, t0+1 (tile 0) and t0+8, t0+9 (tile 1)
                    const int t0 = (at + turn) * kPageTokens + quad * 2;
                    auto seen = [&](int t) { return t < s.keys && (FORM != kEvenChunked || t >= s.hidden); };
                    float x00 = seen(t0) ? s0[0] * p.scale_log2 : -INFINITY;
                    float x01 = seen(t0 + 1) ? s0[1] * p.scale_log2 : -INFINITY;
                    float x10 = seen(t0 + 8) ? s1[0] * p.scale_log2 : -INFINITY;
                    float x11 = seen(t0 + 9) ? s1[1] * p.scale_log2 : -INFINITY;
                    float tile_max = fmaxf(fmaxf(x00, x01), fmaxf(x10, x11));
                    tile_max = fmaxf(tile_max, __shfl_xor_sync(0xffffffffu, tile_max, 1));
                    tile_max = fmaxf(tile_max, __shfl_xor_sync(0xffffffffu, tile_max, 2));
                    const float next_max = fmaxf(run_max, tile_max);
                    const float correction = fast_exp2(run_max - next_max);
                    run_max = next_max;
                    x00 = fast_exp2(x00 - next_max);
                    x01 = fast_exp2(x01 - next_max);
                    x10 = fast_exp2(x10 - next_max);
                    x11 = fast_exp2(x11 - next_max);
                    run_sum = run_sum * correction + (x00 + x01) + (x10 + x11);
#pragma unroll
                    for (int nt = 0; nt < NTILES; ++nt) {
#pragma unroll
                        for (int i = 0; i < 4; ++i) o[nt][i] *= correction;
                    }
                    pa0 = pack2<T>(x00, x01);
                    pa1 = pack_rest<T>(pa0, x00, x01);
                    pa2 = pack2<T>(x10, x11);
                    pa3 = pack_rest<T>(pa2, x10, x11);
                }
                const int slot_v = slot_k + 1;
                if (!__all_sync(0xffffffffu, mbar_wait(bar_full + 8 * slot_v, parity) ? 1 : 0)) {
                    failed = true;
                    break;
                }
                if (mine) {
                    const uint32_t values = tile + slot_v * SLOT;
#pragma unroll
                    for (int j = 0; j < NTILES / 2; ++j) {
                        const int cg = 2 * j + v_sel;
                        uint32_t r0, r1, r2, r3;
                        ldmatrix_x4_trans(values + (cg >> 3) * BOX + v_tok * 128 + (((cg & 7) ^ (v_tok & 7)) << 4), r0, r1, r2, r3);
                        mma_m16n8k16<T>(o[2 * j], pa0, pa1, pa2, pa3, r0, r1);
                        mma_m16n8k16<T>(o[2 * j + 1], pa0, pa1, pa2, pa3, r2, r3);
                    }
                }
                __syncwarp();
                if (lane == 0) mbar_arrive(bar_empty + 8 * slot_v);
            }
            if (failed) break;
            // A leading product that is not finite stands alone: zero or less of an infinite value has been left out of it.
#pragma unroll
            for (int nt = 0; nt < NTILES; ++nt) {
                if (fabsf(o[nt][0]) < INFINITY) o[nt][0] += o[nt][2];
                if (fabsf(o[nt][1]) < INFINITY) o[nt][1] += o[nt][3];
            }
            if (FORM == kEvenFused && counted_to == s.counted && turn == 0 && len > 0) {
                add_new_key<T, HD>(p, x, qa, o, run_max, run_sum, b, head, row, quad, lane);
            }
            if (before[b + 1] < hi) load_query(b + 1);   // on its way while this sequence's rows are written
            run_sum += __shfl_xor_sync(0xffffffffu, run_sum, 1);
            run_sum += __shfl_xor_sync(0xffffffffu, run_sum, 2);
            if (KVH < kEvenWarps) {
                // the other pages' warp hands its state over
                float *state = merge + (head * 8 + row) * (HD + 2);
                const uint32_t written = bar_merge + 16 * head;
                if (turn == 1) {
                    if (merges > 0 && !__all_sync(0xffffffffu, mbar_wait(written + 8, (merges - 1) & 1) ? 1 : 0)) {
                        failed = true;
                        break;
                    }
                    ++merges;
#pragma unroll
                    for (int nt = 0; nt < NTILES; ++nt) {
                        *reinterpret_cast<float2 *>(state + nt * 8 + quad * 2) = make_float2(o[nt][0], o[nt][1]);
                    }
                    if (quad == 0) *reinterpret_cast<float2 *>(state + HD) = make_float2(run_max, run_sum);
                    __syncwarp();
                    if (lane == 0) mbar_arrive(written);
                    continue;
                }
                if (!__all_sync(0xffffffffu, mbar_wait(written, merges & 1) ? 1 : 0)) {
                    failed = true;
                    break;
                }
                ++merges;
                const float2 other = *reinterpret_cast<const float2 *>(state + HD);
                const float top = fmaxf(run_max, other.x);
                const float here = run_max == -INFINITY ? 0.0f : fast_exp2(run_max - top);
                const float there = other.x == -INFINITY ? 0.0f : fast_exp2(other.x - top);
                run_sum = run_sum * here + other.y * there;
                run_max = top;
#pragma unroll
                for (int nt = 0; nt < NTILES; ++nt) {
                    const float2 theirs = *reinterpret_cast<const float2 *>(state + nt * 8 + quad * 2);
                    o[nt][0] = o[nt][0] * here + theirs.x * there;
                    o[nt][1] = o[nt][1] * here + theirs.y * there;
                }
                __syncwarp();
                if (lane == 0) mbar_arrive(written + 8);
            }
            const float inverse = 1.0f / run_sum;
            if (row < p.group) {
                const int query_head = head * p.group + row;
                if (whole) {
                    // (no key at all: zeros, as the reference writes)
                    const bool none = len == 0;
                    uint32_t *out = reinterpret_cast<uint32_t *>(static_cast<T *>(p.out) +
                                                                 (static_cast<size_t>(b) * p.heads + query_head) * HD);
#pragma unroll
                    for (int nt = 0; nt < NTILES; ++nt) {
                        out[nt * 4 + quad] = none ? 0u : pack2<T>(o[nt][0] * inverse, o[nt][1] * inverse);
                    }
                } else {
                    const size_t place = static_cast<size_t>(slot_of_row) * p.heads + query_head;
                    float2 *partial = reinterpret_cast<float2 *>(p.attn_partial + place * HD);
#pragma unroll
                    for (int nt = 0; nt < NTILES; ++nt) {
                        partial[nt * 4 + quad] = make_float2(o[nt][0] * inverse, o[nt][1] * inverse);
                    }
                    // natural-log LSE of the scaled scores: (max2 + log2(sum)) * ln 2
                    if (quad == 0) p.lse_partial[place] = (run_max + log2f(run_sum)) * 0.6931471805599453f;
                }
            }
        }
        if (failed && lane == 0) report_status(p.status, kStatusWaitTimeout);
    }
    // Only now may the next kernel's CTAs come: released at the top, 1 - 2 % slower (the fold's fit beside this kernel's).
    grid_launch_dependents();
    // A warp that gave up keeps the CTA alive until copies that were issued into its shared memory have landed.
    if (failed) linger_after_timeout();
}

// Folds the segments of every sequence that has more than one, with the arithmetic of decode_combine_kernel.  `TEAM` warps share a
// row, each every TEAM-th segment: few sequences have many segments, and a warp waits once for each batch of them.  A warp's
// lanes hold the weights of all segments, and its first segments' values are on their way before the weights are known (us a
// call, four of them early by eight warps and twelve: 2 x 7168 keys of 64 16.8 and 14.1, ragged 3 x 2901 of 128 11.5 and 10.3).
// Warps for a row, eight, four, two and one: 8 x 1088 of 128 12.6, 13.2, 14.0, 14.0; 15 x 580 14.6, 14.2, 14.3, 14.6; 28 x 310
// 17.3, 14.7, 14.7, 14.2; 48 x 298 24.3, 20.0, 18.9, 17.8.
constexpr int kFoldWarps = 8;

}  // namespace

// Whether a sequence's segments lie in a scratch of `slots` slots, whose last one is the list.
__host__ __device__ bool even_row_inside(int segments, int slot, int slots) {
    return segments > 0 && segments <= kEvenMaxCtas && slot >= 0 && segments < slots && slot < slots - segments;
}

namespace {

template <typename T, int HD, int TEAM>
__global__ void __launch_bounds__(32 * kFoldWarps)
    even_combine_kernel(T *out, const float *attn_partial, const float *lse_partial, const EvenRow *rows, int heads, int slots) {
    grid_launch_dependents();
    grid_dependency_wait();
    constexpr int kColumns = HD / 32;   // columns of a lane
    constexpr int kRounds = kEvenMaxCtas / 32;
    constexpr int kEarly = TEAM == 8 ? 12 : 8;
    struct __align__(kColumns * 4) Columns { float v[kColumns]; };
    __shared__ Columns parts[TEAM > 1 ? kFoldWarps : 1][32];
    const int b = blockIdx.y;
    const int warp = threadIdx.x >> 5;
    const int member = warp % TEAM;
    const int head = blockIdx.x * (kFoldWarps / TEAM) + warp / TEAM;
    const int lane = threadIdx.x & 31;
    const EvenRow row = rows[b];
    const int segments = row.segments;
    if (segments <= 1) return;   // written by the decode kernel
    // (an entry that calls which share a caller's scratch have written over each other ends here)
    if (!even_row_inside(segments, row.slot, slots)) return;
    const bool real = head < heads;
    const size_t first = static_cast<size_t>(row.slot) * heads + (real ? head : 0);
    const float *partial = attn_partial + first * HD + lane * kColumns;
    const size_t step = static_cast<size_t>(heads) * HD;
    Columns early[kEarly];
#pragma unroll
    for (int i = 0; i < kEarly; ++i) {
        const int s = member + i * TEAM;
        early[i] = {};
        if (s < segments) early[i] = *reinterpret_cast<const Columns *>(partial + s * step);
    }
    const float *lse = lse_partial + first;
    float weight[kRounds];
    float top = -INFINITY;
#pragma unroll
    for (int i = 0; i < kRounds; ++i) {
        weight[i] = i * 32 + lane < segments ? lse[static_cast<size_t>(i * 32 + lane) * heads] : -INFINITY;
        top = fmaxf(top, weight[i]);
    }
    top = warp_max(top);
    float sum = 0.0f;
#pragma unroll
    for (int i = 0; i < kRounds; ++i) {
        weight[i] = i * 32 + lane < segments ? expf(weight[i] - top) : 0.0f;
        sum += weight[i];
    }
    sum = warp_sum(sum);
    Columns value = {};
#pragma unroll
    for (int i = 0; i < kEarly; ++i) {
        const float w = __shfl_sync(0xffffffffu, weight[i * TEAM / 32], (member + i * TEAM) % 32);
#pragma unroll
        for (int c = 0; c < kColumns; ++c) {
            if (member + i * TEAM < segments) value.v[c] = fmaf(w, early[i].v[c], value.v[c]);
        }
    }
#pragma unroll
    for (int i = kEarly * TEAM / 32; i < kRounds; ++i) {
        const int end = min(segments - i * 32, 32);
#pragma unroll 4
        for (int s = member + max(kEarly * TEAM - i * 32, 0); s < end; s += TEAM) {
            const Columns part = *reinterpret_cast<const Columns *>(partial + static_cast<size_t>(i * 32 + s) * step);
            const float w = __shfl_sync(0xffffffffu, weight[i], s);
#pragma unroll
            for (int c = 0; c < kColumns; ++c) value.v[c] = fmaf(w, part.v[c], value.v[c]);
        }
    }
    if (TEAM > 1) {
        parts[warp][lane] = value;
        __syncthreads();
        if (member > 0) return;
#pragma unroll
        for (int m = 1; m < TEAM; ++m) {
#pragma unroll
            for (int c = 0; c < kColumns; ++c) value.v[c] += parts[warp + m][lane].v[c];
        }
    }
    if (!real) return;
    uint32_t *to = reinterpret_cast<uint32_t *>(out + (static_cast<size_t>(b) * heads + head) * HD + lane * kColumns);
#pragma unroll
    for (int c = 0; c < kColumns; c += 2) to[c / 2] = pack2<T>(value.v[c] / sum, value.v[c + 1] / sum);
}

template <typename T, int HD, int KVH, int FORM>
int launch_even(cudaStream_t stream, const DecodeParams &params, const StepExtras &extras, const ChunkedDecode &chunked,
                const void *key_cache, const void *value_cache, int slots) {
    static int configured[kMaxDevices] = {0};
    constexpr int most = even_smem_bytes<HD, KVH>(kEvenMaxBatch);
    static_assert(most <= 227 * 1024, "shared memory of one CTA");
    SINGE_CUDA_TRY(ensure_dynamic_shared(paged_decode_even_kernel<T, HD, KVH, FORM>, most, configured));
    const int smem = even_smem_bytes<HD, KVH>(params.batch);
    // tokens before heads: a box lands as one 16-row tile per head
    const uint64_t dims[4] = {static_cast<uint64_t>(HD), kPageTokens, static_cast<uint64_t>(KVH),
                              static_cast<uint64_t>(params.physical_blocks)};
    const uint64_t strides[3] = {static_cast<uint64_t>(HD) * sizeof(T) * KVH, static_cast<uint64_t>(HD) * sizeof(T),
                                 static_cast<uint64_t>(HD) * sizeof(T) * KVH * kPageTokens};
    const uint32_t box[4] = {64, kPageTokens, KVH, 1};
    CUtensorMap k_map, v_map;
    SINGE_TRY(encode_tensor_map(&k_map, TensorMapType<T>::value, 4, key_cache, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_128B,
                                CU_TENSOR_MAP_L2_PROMOTION_L2_256B));
    SINGE_TRY(encode_tensor_map(&v_map, TensorMapType<T>::value, 4, value_cache, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_128B,
                                CU_TENSOR_MAP_L2_PROMOTION_L2_256B));
    const int ctas = min(device_sm_count(), slots - params.batch);
    // the scratch's last slot (no segment has it: CTA + sequence stays below) lists the sequences' segments
    EvenRow *rows = reinterpret_cast<EvenRow *>(params.attn_partial + static_cast<size_t>(slots - 1) * params.heads * HD);
    SINGE_CUDA_TRY(launch_dependent(paged_decode_even_kernel<T, HD, KVH, FORM>, dim3(static_cast<unsigned>(ctas)),
                                    dim3(kEvenThreads), smem, stream, kLaunchDecode, 1, k_map, v_map, params, extras, chunked, rows));
    SINGE_TRY(launch_status());
    auto fold = [&](auto kernel, int team) {
        const int rows_per_cta = kFoldWarps / team;
        return launch_dependent(kernel, dim3(static_cast<unsigned>((params.heads + rows_per_cta - 1) / rows_per_cta),
                                             static_cast<unsigned>(params.batch)),
                                dim3(32 * kFoldWarps), 0, stream, kLaunchCombine, 1, static_cast<T *>(params.out),
                                params.attn_partial, params.lse_partial, rows, params.heads, slots);
    };
    SINGE_CUDA_TRY(params.batch < 12   ? fold(even_combine_kernel<T, HD, 8>, 8)
                   : params.batch < 20 ? fold(even_combine_kernel<T, HD, 4>, 4)
                                       : fold(even_combine_kernel<T, HD, 1>, 1));
    return launch_status();
}

template <typename T, int FORM>
int launch_even_shape(cudaStream_t stream, const DecodeParams &params, const StepExtras &extras, const ChunkedDecode &chunked,
                      const void *key_cache, const void *value_cache, size_t head_dim, int slots) {
    if (params.kv_heads == 8) {
        return head_dim == 128 ? launch_even<T, 128, 8, FORM>(stream, params, extras, chunked, key_cache, value_cache, slots)
                               : launch_even<T, 64, 8, FORM>(stream, params, extras, chunked, key_cache, value_cache, slots);
    }
    return head_dim == 128 ? launch_even<T, 128, 4, FORM>(stream, params, extras, chunked, key_cache, value_cache, slots)
                           : launch_even<T, 64, 4, FORM>(stream, params, extras, chunked, key_cache, value_cache, slots);
}

}  // namespace

// How many slots of [heads, head_dim] f32 partials and [heads] log sums the even form wants for a call of the tiled kernel
// (paged_decode_fast_path) with at most `bound` keys a sequence; 0: the split grid serves it.
// Lengths are device data, so the rule knows only what they may grow to.  Below 32 MB of keys and values setting up (a scan of
// the lengths, then the block table, then the first pages) and folding cost as much as the even shares gain, 24 MB for heads of
// 128 whose sequences the split grid has to split as well (us, calls one after the other, split grid and here; "to" is the shortest of a
// ragged batch): 4 x 1536 of 128 11.0 and 10.1, 384 to 1536 10.5 and 9.7; 20 x 307 14.2 and 10.5; 4 x 2901 19.2 and 13.5; 8 x
// 640, 20 MB, 10.0 and 10.4; 48 x 128, not split, 7.4 and 10.9; heads of 64, 14 x 877 12.6 and 10.6, but 219 to 877 8.9 and 9.6; at 32
// MB 8 x 2176 16.4 and 13.1, 544 to 2176 10.5 and 10.3.  (Ragged batches of more rows may lose, see paged_decode_even_pays.)  Sequences of one split each need no fold there: they stay while they fill the grid
// (three CTAs an SM) one and a half times, 96 x 256 24.1 against 25.1 here; 64 x 256, 1.15 times, 27.1 against 18.9.
size_t paged_decode_even_slots(size_t batch, size_t heads, size_t kv_heads, size_t head_dim, size_t bound) {
    const size_t sms = static_cast<size_t>(device_sm_count());
    const size_t stride = (bound + kPageTokens - 1) / kPageTokens;
    if ((kv_heads != 8 && kv_heads != 4) || batch > kEvenMaxBatch || sms > kEvenMaxCtas || 2 * batch > heads * head_dim ||
        stride > (size_t{1} << 30) / batch || stride >= (size_t{1} << 27)) {   // (positions stay below 2^31)
        return 0;
    }
    const bool split = bound > 128 && batch * kv_heads <= 3 * sms;
    const size_t least = size_t{head_dim == 128 && split ? 24u : 32u} << 20;
    if (batch * stride * kPageTokens * kv_heads * head_dim * 4 < least) return 0;
    if (bound <= 512 && 2 * batch * kv_heads > 9 * sms) return 0;
    return sms + batch;
}

// The same as a number of splits of a [batch, heads, splits, head_dim] scratch.
size_t paged_decode_even_splits(size_t batch, size_t heads, size_t kv_heads, size_t head_dim, size_t key_len_bound) {
    return (paged_decode_even_slots(batch, heads, kv_heads, head_dim, key_len_bound) + batch - 1) / batch;
}

// Whether a drop-in call takes the even form.  Its caller knows nothing of the lengths but the bound, so the line lies where ragged
// batches (lengths spread from 1/4 or 1/32 of the bound up to it) lose as a whole, measured on 750 shapes whose keys and values
// come from HBM (us, split grid and here, lengths from a quarter of the bound, then all at it):
//   * heads of 64 on 49 - 175 rows below 96 MB of keys and values at the bound, where ragged lengths leave the split grid a single
//     wave: 20 x 1024 11.5 and 12.7, 17.2 and 14.6; 24 x 2128 on 4 12.8 and 14.2, 20.2 and 16.6;
//   * 4 heads of 128 on more than 16 rows below 32 MB and on more than 32 below 40: 20 x 640 12.2 and 12.7, 13.9 and 13.5;
//   * what the split grid need not split of 8 heads of 128 below 40 MB: 64 x 128 11.9 and 12.3, 14.3 and 13.8;
//   * four rows an SM or more up to 512 keys, where a row of the split grid is one piece and needs no fold (8 heads of 128 up to 256):
//     81 x 320 of 64 1.1 - 1.2 times and 0.99, 166 x 400 of 128 on 4 1.04 - 1.07 and 1.06, 81 x 400 on 8 0.96 and 0.98.
// Of the calls it takes none with lengths from half of the bound on is slower, of 1221 from a quarter on 37 by 2 - 9 %, of 1130 from
// 1/32 on 114, 15 of them by more than 10 %; on all but 3 of 432 shapes, by 2 % at most, all three together gain.  Lengths far below the
// bound may lose: all at a sixteenth of it, heads of 64, 32 x 140 7.8 and 9.5, 64 x 280 17.2 and 14.7.
bool paged_decode_even_pays(size_t batch, size_t kv_heads, size_t head_dim, size_t bound) {
    const size_t rows = batch * kv_heads, stride = (bound + kPageTokens - 1) / kPageTokens, sms = static_cast<size_t>(device_sm_count());
    const bool wide = kv_heads * head_dim == 1024;   // 8 heads of 128
    if (rows >= 4 * sms && bound <= (wide ? 256 : 512)) return false;
    size_t least = 32;
    if (wide) {
        least = bound > 128 && rows <= 3 * sms ? 24 : 40;
    } else if (head_dim == 64) {
        if (rows > 48 && rows < 176) least = 96;
    } else {
        least = rows <= 16 ? 24 : rows <= 32 ? 32 : 40;
    }
    return batch * stride * kPageTokens * kv_heads * head_dim * 4 >= least << 20;
}

// The decode kernels' call in the even form; params.out, scratch of `slots` slots, extras.qkv (fused) as there.
int paged_decode_even(cudaStream_t stream, int element, const DecodeParams &params, const StepExtras &extras, const void *key_cache,
                      const void *value_cache, size_t head_dim, size_t slots) {
    const int places = static_cast<int>(slots);
    if (extras.qkv != nullptr) {
        return launch_even_shape<__nv_bfloat16, kEvenFused>(stream, params, extras, {}, key_cache, value_cache, head_dim, places);
    }
    return element == 0
               ? launch_even_shape<__nv_bfloat16, kEvenPlain>(stream, params, extras, {}, key_cache, value_cache, head_dim, places)
               : launch_even_shape<__half, kEvenPlain>(stream, params, extras, {}, key_cache, value_cache, head_dim, places);
}

int paged_decode_even_chunked(cudaStream_t stream, const DecodeParams &params, const ChunkedDecode &chunked, const void *key_cache,
                              const void *value_cache, size_t head_dim, size_t slots) {
    return launch_even_shape<__nv_bfloat16, kEvenChunked>(stream, params, {}, chunked, key_cache, value_cache, head_dim,
                                                          static_cast<int>(slots));
}

}  // namespace singe
