// Dense f32 attention in tiles: what Tensor::attend and fmha_prefill_lse compute for f32
// (singe/src/backend/cpu/normalization/attention.rs:191-276, singe-kernel/src/cuda/attention/fmha.rs:48-140), in true
// 32-bit arithmetic on the FMA pipe.
//
// Bound: issue slots and shared-memory reads, behind the FMA pipe (128 a clock and SM); up to 33 TFLOP/s.  One warp per query
// row, the general kernel's way (1.2 - 2.2 TFLOP/s), reads every key and value from L1 once per row and folds each score over
// the warp; here a CTA takes BM rows of one head, stages 64 keys at a time in shared memory, and a thread owns R rows x 4 keys
// of the scores and R rows x D/16 columns of the output in registers, so a value read from shared memory feeds R or 4 FMAs.
// The error of a sum grows with the length of its chains, and one warp per row has short ones (D / 32 products a lane, then a
// tree).  So eight dimensions are summed as packed pairs, four such blocks are added, and groups of 32 dimensions pairwise; the
// scale is applied by the FMA that takes a score's distance from the row's base.  Against 64 bits, 128 heads of 128 columns
// over 16, 40 and 100 causal keys, in units of the general kernel's error: 1.00, 0.99, 0.95 (64 columns 0.99, 0.98, 0.94); four
// chains of a quarter of the dimensions each, scaled afterwards: 1.19, 1.17, 1.11.  They took 4 % less time, but 8 % more in the
// form of four teams, where their registers spilled.  The value products take pairs of columns at a time (sums and order as one by
// one; together with what last tiles leave out, see below: 8 heads x 512 causal keys of 64, four teams, 24.4 us -> 23.6; of 128, two teams,
// 44.3 -> 42.0, 8 x 100 14.1 -> 12.0); reading every weight twice from shared memory instead cost 3 - 9 % more.
// Thread (ty, tx) owns rows ty, ty + BM/R, ... and keys tx, tx + 16, ...: a row's scores lie in 16 neighbouring lanes, and rows
// one apart keep the 16-byte reads of a warp on different banks (rows are padded by 16 bytes).
// Teams of threads walk alternate key tiles, each in buffers of its own, and are folded at the end through shared memory: the
// chain of key tiles is what a call of few CTAs waits for.
// In a last tile the scores stop at a half (32 keys) that holds the last visible key; the value products stop at the next multiple of
// four keys behind it with one team or two, while four teams walk the whole tile (no register is left for the end).
// 8 heads x 512 causal keys of 64: 417 us -> 23.6; x 900: 1011 -> 39.8; x 1500 of 128: 3367 -> 170.
// Keys a row does not see take no part at all, whatever their bits are: in tiles that hold hidden keys the value
// products are predicated, not multiplied by zero.
#include "common.cuh"
#include "attention_f32.cuh"

namespace singe {

namespace {

constexpr int kKeys = 64;      // keys of a tile
constexpr int kMostTeams = 4;
// Positions are ints: a walk may compute places up to a step of every team and a tile past the last key, and start where the
// window of the last row does.
constexpr int kMostPositions = 0x7fffffff - (kMostTeams + 1) * kKeys;

__device__ __forceinline__ void copy_16(float *dst, const float *src, bool real) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(dst)), "l"(src), "r"(real ? 16 : 0) : "memory");
}
__device__ __forceinline__ void copy_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int PENDING>
__device__ __forceinline__ void copy_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(PENDING) : "memory"); }

// Every thread of every CTA of the cluster takes part; what they wrote to shared memory before it is visible to all behind it.
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

template <int D, int R, int BM, int G>
struct Layout {
    static constexpr int kTeam = 16 * BM / R;          // threads that share a key tile
    static constexpr int kThreads = kTeam * G;
    static constexpr int kRows = BM / R;               // distance between a thread's rows
    static constexpr int kPitch = D + 4;               // floats between rows of Q and K
    static constexpr int kWeightPitch = kKeys + 4;
    static constexpr int kTeamFloats = kKeys * kPitch + kKeys * D + BM * kWeightPitch;
    static constexpr int kFloats = BM * kPitch + G * kTeamFloats;
    static_assert(G <= kMostTeams && BM <= kKeys, "see kMostPositions");
    static_assert(G == 1 || kTeam * (R * D / 16 + 2 * R) <= kTeamFloats, "the fold reuses a team's buffers");
};

// C > 1: a cluster of C CTAs shares a row tile, each with every C-th step of G key tiles; the others park their rows and the
// first folds them out of their shared memory.
template <int D, int R, int BM, int G, int C>
__global__ void __launch_bounds__(16 * BM / R * G) dense_attention_f32_kernel(const DenseF32 p, const int row_tiles) {
    using L = Layout<D, R, BM, G>;
    constexpr int kColumns = D / 64;   // float4 groups of output columns a thread owns
    constexpr int kBlock = 8, kGroup = 32;   // dimensions that are summed in a row, and apart from the others
    grid_launch_dependents();
    extern __shared__ __align__(16) float shared[];
    const int team = threadIdx.x / L::kTeam;
    const int t = threadIdx.x % L::kTeam;
    const int tx = t & 15, ty = t >> 4;
    float *q_tile = shared;
    float *k_tile = shared + BM * L::kPitch + team * L::kTeamFloats;
    float *v_tile = k_tile + kKeys * L::kPitch;
    float *weights = v_tile + kKeys * D;
    auto team_sync = [&]() {
        if (G == 1) {
            __syncthreads();
        } else {
            asm volatile("bar.sync %0, %1;" ::"r"(team + 1), "n"(L::kTeam) : "memory");
        }
    };

    // the heaviest row tiles (the last ones, under a causal mask) are dispatched first
    const int rank = static_cast<int>(blockIdx.x) % C, block = static_cast<int>(blockIdx.x) / C;
    const int pairs = gridDim.x / C / row_tiles;
    const int first_row = (row_tiles - 1 - block / pairs) * BM;
    const int pair = block % pairs;
    const int head = pair % p.heads;
    const long long batch = pair / p.heads;
    const int kv_head = head / (p.heads / p.kv_heads);
    const float *query = p.query + batch * p.q_batch + head * p.q_head;
    const float *keys = p.key + batch * p.k_batch + kv_head * p.k_head;
    const float *values = p.value + batch * p.k_batch + kv_head * p.k_head;
    auto begin_of = [&](int row) { return p.window > 0 && row + 1 > p.window ? static_cast<int>(row + 1 - p.window) : 0; };
    auto end_of = [&](int row) { return p.causal && row + 1 < p.key_len ? row + 1 : p.key_len; };
    const int last_row = min(first_row + BM, p.query_len) - 1;
    const int first_key = begin_of(first_row) / kKeys * kKeys;
    const int end_key = end_of(last_row);

    auto load_keys = [&](float *tile, const float *from, int pitch, int key0) {
        for (int i = t; i < kKeys * (D / 4); i += L::kTeam) {
            const int key = i / (D / 4), at = i % (D / 4) * 4;
            const bool real = key0 + key < p.key_len && at < p.head_dim;
            copy_16(tile + key * pitch + at, real ? from + (key0 + key) * p.k_row + at : from, real);
        }
        copy_commit();
    };

    grid_dependency_wait();
    int key0 = first_key + (rank * G + team) * kKeys;
    if (key0 < end_key) {
        load_keys(k_tile, keys, L::kPitch, key0);
        load_keys(v_tile, values, D, key0);
    }
    for (int i = threadIdx.x; i < BM * (D / 4); i += L::kThreads) {
        const int row = i / (D / 4), at = i % (D / 4) * 4;
        float4 word = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (first_row + row < p.query_len && at < p.head_dim) {
            word = *reinterpret_cast<const float4 *>(query + (first_row + row) * p.q_row + at);
        }
        *reinterpret_cast<float4 *>(q_tile + row * L::kPitch + at) = word;
    }
    __syncthreads();

    float top[R], sum[R];
    float4 out[R][kColumns];
    int begin[R], end[R];
    // a sink is one key of weight exp(sink - sink) = 1 and value zero; one thread of a row counts it
    const float sink = p.sinks != nullptr && team == 0 && rank == 0 ? p.sinks[head] : -INFINITY;
#pragma unroll
    for (int i = 0; i < R; ++i) {
        const int row = first_row + ty + i * L::kRows;
        begin[i] = row < p.query_len ? begin_of(row) : 0;
        end[i] = row < p.query_len ? end_of(row) : 0;
        top[i] = sink;
        sum[i] = sink != -INFINITY && tx == 0 ? 1.0f : 0.0f;
#pragma unroll
        for (int c = 0; c < kColumns; ++c) out[i][c] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    }

    // A score is s * unit, rounded only together with the base it is weighed against.
    const float unit = p.softcap > 0.0f || p.scale == 0.0f ? 1.0f : p.scale;
    const float hidden = unit < 0.0f ? INFINITY : -INFINITY;
    for (; key0 < end_key; key0 += C * G * kKeys) {
        copy_wait<1>();   // the keys; the values may still be on their way
        team_sync();
        // Even and odd dimensions are summed apart, as packed pairs, kBlock dimensions in a row; then the blocks of a group,
        // then the groups, two and two.
        float s[R][4], two[R][4];
#pragma unroll
        for (int i = 0; i < R; ++i) {
#pragma unroll
            for (int j = 0; j < 4; ++j) s[i][j] = 0.0f;
        }
        auto score = [&](auto columns) {   // how many of a thread's keys; the others lie behind the last visible one
            constexpr int kOf = decltype(columns)::value;
#pragma unroll 1
            for (int group = 0; group < D; group += kGroup) {
                // (in narrow heads, where threads have 128 registers, a pair is folded at the end of its block)
                std::conditional_t<D == 64, float, float2> total[R][4];
#pragma unroll
                for (int first = 0; first < kGroup; first += kBlock) {
                    float2 part[R][4];
#pragma unroll
                    for (int i = 0; i < R; ++i) {
#pragma unroll
                        for (int j = 0; j < kOf; ++j) part[i][j] = make_float2(0.0f, 0.0f);
                    }
#pragma unroll
                    for (int d = 0; d < kBlock; d += 4) {
                        const int at = group + first + d;
                        float4 a[R], b[4];
#pragma unroll
                        for (int i = 0; i < R; ++i) a[i] = *reinterpret_cast<const float4 *>(q_tile + (ty + i * L::kRows) * L::kPitch + at);
#pragma unroll
                        for (int j = 0; j < kOf; ++j) b[j] = *reinterpret_cast<const float4 *>(k_tile + (tx + 16 * j) * L::kPitch + at);
#pragma unroll
                        for (int i = 0; i < R; ++i) {
#pragma unroll
                            for (int j = 0; j < kOf; ++j) part[i][j] = __ffma2_rn(make_float2(a[i].x, a[i].y), make_float2(b[j].x, b[j].y), part[i][j]);
                        }
#pragma unroll
                        for (int i = 0; i < R; ++i) {
#pragma unroll
                            for (int j = 0; j < kOf; ++j) part[i][j] = __ffma2_rn(make_float2(a[i].z, a[i].w), make_float2(b[j].z, b[j].w), part[i][j]);
                        }
                    }
#pragma unroll
                    for (int i = 0; i < R; ++i) {
#pragma unroll
                        for (int j = 0; j < kOf; ++j) {
                            if constexpr (D == 64) {
                                const float sum_of_block = part[i][j].x + part[i][j].y;
                                total[i][j] = first == 0 ? sum_of_block : total[i][j] + sum_of_block;
                            } else {
                                total[i][j] = first == 0 ? part[i][j] : __fadd2_rn(total[i][j], part[i][j]);
                            }
                        }
                    }
                }
#pragma unroll
                for (int i = 0; i < R; ++i) {
#pragma unroll
                    for (int j = 0; j < kOf; ++j) {
                        if constexpr (D == 64) {
                            s[i][j] += total[i][j];
                        } else {
                            const float sum_of_group = total[i][j].x + total[i][j].y;
                            if (group % (2 * kGroup) == 0) {
                                two[i][j] = sum_of_group;
                            } else {
                                s[i][j] += two[i][j] + sum_of_group;
                            }
                        }
                    }
                }
            }
        };
        if (end_key - key0 > kKeys / 2) {
            score(std::integral_constant<int, 4>{});
        } else {
            score(std::integral_constant<int, 2>{});
        }
        team_sync();   // every thread has read the keys
        const bool more = key0 + C * G * kKeys < end_key;
        if (more) {
            load_keys(k_tile, keys, L::kPitch, key0 + C * G * kKeys);
        } else {
            copy_commit();
        }
        // whether every row of the tile sees every key of it
        const bool whole = begin_of(last_row) <= key0 && end_of(first_row) >= key0 + kKeys;
#pragma unroll
        for (int i = 0; i < R; ++i) {
            if (p.softcap > 0.0f) {
#pragma unroll
                for (int j = 0; j < 4; ++j) s[i][j] = p.softcap * tanhf(s[i][j] * p.scale / p.softcap);
            } else if (p.scale == 0.0f) {
#pragma unroll
                for (int j = 0; j < 4; ++j) s[i][j] *= 0.0f;
            }
            if (!whole) {
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const int key = key0 + tx + 16 * j;
                    if (key < begin[i] || key >= end[i]) s[i][j] = hidden;
                }
            }
            float most = fmaxf(fmaxf(s[i][0] * unit, s[i][1] * unit), fmaxf(s[i][2] * unit, s[i][3] * unit));
#pragma unroll
            for (int offset = 8; offset > 0; offset >>= 1) most = fmaxf(most, __shfl_xor_sync(0xffffffffu, most, offset));
            most = fmaxf(most, top[i]);
            const float base = most == -INFINITY ? 0.0f : most;
            const float factor = expf(top[i] - base);
            top[i] = most;
            sum[i] *= factor;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float weight = expf(fmaf(s[i][j], unit, -base));
                sum[i] += weight;
                weights[(ty + i * L::kRows) * L::kWeightPitch + tx + 16 * j] = weight;
            }
#pragma unroll
            for (int c = 0; c < kColumns; ++c) {
                out[i][c].x *= factor;
                out[i][c].y *= factor;
                out[i][c].z *= factor;
                out[i][c].w *= factor;
            }
        }
        copy_wait<1>();   // the values; the next keys may still be on their way
        team_sync();
        auto weigh = [&](auto whole_tile) {
            const int last = decltype(whole_tile)::value || G == 4 ? kKeys : min(kKeys, end_key - key0);   // (four teams have no register for it)
#pragma unroll 4
            for (int k = 0; k < last; k += 4) {
                float4 w[R];
#pragma unroll
                for (int i = 0; i < R; ++i) w[i] = *reinterpret_cast<const float4 *>(weights + (ty + i * L::kRows) * L::kWeightPitch + k);
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    float4 v[kColumns];
#pragma unroll
                    for (int c = 0; c < kColumns; ++c) v[c] = *reinterpret_cast<const float4 *>(v_tile + (k + u) * D + c * 64 + tx * 4);
#pragma unroll
                    for (int i = 0; i < R; ++i) {
                        if (!decltype(whole_tile)::value && (key0 + k + u < begin[i] || key0 + k + u >= end[i])) continue;
                        const float weight = u == 0 ? w[i].x : u == 1 ? w[i].y : u == 2 ? w[i].z : w[i].w;
#pragma unroll
                        for (int c = 0; c < kColumns; ++c) {
                            const float2 both = make_float2(weight, weight);
                            const float2 low = __ffma2_rn(both, make_float2(v[c].x, v[c].y), make_float2(out[i][c].x, out[i][c].y));
                            const float2 high = __ffma2_rn(both, make_float2(v[c].z, v[c].w), make_float2(out[i][c].z, out[i][c].w));
                            out[i][c] = make_float4(low.x, low.y, high.x, high.y);
                        }
                    }
                }
            }
        };
        if (whole) {
            weigh(std::true_type{});
        } else {
            weigh(std::false_type{});
        }
        team_sync();   // every thread has read the values
        if (more) {
            load_keys(v_tile, values, D, key0 + C * G * kKeys);
        } else {
            copy_commit();
        }
    }
    copy_wait<0>();
#pragma unroll
    for (int i = 0; i < R; ++i) {
#pragma unroll
        for (int offset = 8; offset > 0; offset >>= 1) sum[i] += __shfl_xor_sync(0xffffffffu, sum[i], offset);
    }
    // Rows are folded pairwise: one side parks its rows where the other reads them, one float of every thread, then the next.
    constexpr int kEach = 2 + 4 * kColumns;
    auto park = [&](float *parked) {
#pragma unroll
        for (int i = 0; i < R; ++i) {
            float *at = parked + i * kEach * L::kTeam;
            at[0] = top[i];
            at[L::kTeam] = sum[i];
#pragma unroll
            for (int c = 0; c < kColumns; ++c) {
                at[(2 + 4 * c) * L::kTeam] = out[i][c].x;
                at[(3 + 4 * c) * L::kTeam] = out[i][c].y;
                at[(4 + 4 * c) * L::kTeam] = out[i][c].z;
                at[(5 + 4 * c) * L::kTeam] = out[i][c].w;
            }
        }
    };
    auto fold = [&](auto read) {   // read(n): the n-th float this thread's counterpart parked
#pragma unroll
        for (int i = 0; i < R; ++i) {
            const float other = read(i * kEach);
            const float most = fmaxf(top[i], other);
            const float base = most == -INFINITY ? 0.0f : most;
            const float mine = expf(top[i] - base), theirs = expf(other - base);
            top[i] = most;
            sum[i] = sum[i] * mine + read(i * kEach + 1) * theirs;
#pragma unroll
            for (int c = 0; c < kColumns; ++c) {
                out[i][c].x = out[i][c].x * mine + read(i * kEach + 2 + 4 * c) * theirs;
                out[i][c].y = out[i][c].y * mine + read(i * kEach + 3 + 4 * c) * theirs;
                out[i][c].z = out[i][c].z * mine + read(i * kEach + 4 + 4 * c) * theirs;
                out[i][c].w = out[i][c].w * mine + read(i * kEach + 5 + 4 * c) * theirs;
            }
        }
    };
    // the upper half of the teams parks in the lower half's buffers, which nobody reads any more
#pragma unroll
    for (int half = G / 2; half > 0; half /= 2) {
        __syncthreads();
        float *parked = shared + BM * L::kPitch + (team % half) * L::kTeamFloats + t;
        if (team >= half && team < 2 * half) park(parked);
        __syncthreads();
        if (team < half) fold([&](int n) { return parked[n * L::kTeam]; });
    }
    if constexpr (C > 1) {
        __syncthreads();   // (with one team, all have read their tiles)
        float *parked = shared + BM * L::kPitch + t;
        if (team == 0 && rank > 0) park(parked);
        cluster_sync();
        if (team == 0 && rank == 0) {
#pragma unroll
            for (int r = 1; r < C; ++r) {
                uint32_t theirs;
                asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(theirs) : "r"(smem_u32(parked)), "r"(r));
                fold([&](int n) {
                    float value;
                    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(value) : "r"(theirs + n * L::kTeam * 4));
                    return value;
                });
            }
        }
        cluster_sync();    // nobody leaves before its rows have been read
        if (rank > 0) return;
    }
    if (team > 0) return;
#pragma unroll
    for (int i = 0; i < R; ++i) {
        const int row = first_row + ty + i * L::kRows;
        if (row >= p.query_len) continue;
        const bool unseen = end[i] <= begin[i];   // no key: nothing is weighed, and the log sum is that of the sink, whatever it is
        const float inverse = 1.0f / sum[i];
        float *to = p.out + batch * p.q_batch + head * p.q_head + row * p.q_row;
#pragma unroll
        for (int c = 0; c < kColumns; ++c) {
            if (c * 64 + tx * 4 < p.head_dim) {
                *reinterpret_cast<float4 *>(to + c * 64 + tx * 4) =
                    unseen ? make_float4(0.0f, 0.0f, 0.0f, 0.0f)
                           : make_float4(out[i][c].x * inverse, out[i][c].y * inverse, out[i][c].z * inverse, out[i][c].w * inverse);
            }
        }
        if (p.lse != nullptr && tx == 0) {
            p.lse[(batch * p.heads + head) * p.query_len + row] = unseen ? sink : top[i] + logf(sum[i]);
        }
    }
}

template <int D, int R, int BM, int G, int C = 1>
int launch(cudaStream_t stream, const DenseF32 &p, size_t pairs) {
    using L = Layout<D, R, BM, G>;
    static int raised[kMaxDevices] = {0};
    constexpr int kBytes = L::kFloats * 4;
    SINGE_CUDA_TRY(ensure_dynamic_shared(dense_attention_f32_kernel<D, R, BM, G, C>, kBytes, raised));
    const int row_tiles = (p.query_len + BM - 1) / BM;
    SINGE_CUDA_TRY(launch_dependent(dense_attention_f32_kernel<D, R, BM, G, C>, dim3(static_cast<unsigned>(pairs * row_tiles * C)),
                                    dim3(L::kThreads), kBytes, stream, kLaunchGlue, C, p, row_tiles));
    return launch_status();
}

}  // namespace

bool dense_attention_f32_takes(const DenseF32 &p, size_t batch) {
    const uintptr_t all = reinterpret_cast<uintptr_t>(p.query) | reinterpret_cast<uintptr_t>(p.key) |
                          reinterpret_cast<uintptr_t>(p.value) | reinterpret_cast<uintptr_t>(p.out);
    const size_t blocks = batch * static_cast<size_t>(p.heads) * ((static_cast<size_t>(p.query_len) + 31) / 32);
    return p.head_dim % 4 == 0 && p.head_dim <= 128 && p.query_len >= kDenseF32LeastRows && (all & 15u) == 0 &&
           blocks <= 0x7fffffffull && p.query_len <= kMostPositions && p.key_len <= kMostPositions;
}

int dense_attention_f32(cudaStream_t stream, const DenseF32 &p, size_t batch) {
    const size_t pairs = batch * static_cast<size_t>(p.heads);
    const size_t sms = static_cast<size_t>(device_sm_count());
    const size_t blocks = pairs * ((static_cast<size_t>(p.query_len) + 31) / 32);
    // A grid that leaves half of the SMs idle gives each row tile a cluster of two CTAs with two teams each, once there are more
    // keys than two teams' first tiles (us without and with: 4 causal heads of 64, 200 keys 12.3 and 10.2, 512 23.4 and 16.0; of
    // 128, 512 41.5 and 24.9; 128 keys 9.0 and 10.2).  Under a causal mask the short walks make room: up to four fifths of the SMs
    // where walks are long (8 heads x 400 20.5 and 19.5, 4 x 900 39.4 and 29.6, of 128 72.0 and 46.1; not 8 x 512, 128 tiles, 23.6
    // and 24.7, nor 12 x 256 13.9 and 17.4).
    long long longest = p.key_len;
    if (p.window > 0 && longest > p.window) longest = p.window;
    if (longest > 2 * kKeys && (2 * blocks <= sms || (p.causal && longest >= 6 * kKeys && 5 * blocks <= 4 * sms))) {
        return p.head_dim <= 64 ? launch<64, 4, 32, 2, 2>(stream, p, pairs) : launch<128, 4, 32, 2, 2>(stream, p, pairs);
    }
    if (p.head_dim <= 64) {
        // Four teams need more than two key tiles to share.  A grid that does not cover the SMs leaves each CTA alone on its SM,
        // and the longest walk decides (us with four teams and with two: 8 heads x 512 causal keys 23.6 and 25.7, x 900 39.8 and
        // 44.1; x 128 whole 9.6 and 8.9).  Else the mean walk does: from three tiles on (200 heads x 200 whole keys
        // 124 and 128, 64 x 400 causal 77.9 and 78.5, 24 x 1500 causal 256 and 281; 64 x 256 causal 39.1 and 38.1, 200 x 130 causal
        // 59.9 and 55.0).  64 rows and no teams never win by more than 3 % and lose up to half.
        long long walk = p.key_len;
        if (blocks > sms && p.causal) walk = (min(p.query_len, p.key_len) + 1) / 2;
        if (p.window > 0 && walk > p.window) walk = p.window;
        return walk > (blocks > sms ? 3 : 2) * kKeys ? launch<64, 4, 32, 4>(stream, p, pairs) : launch<64, 4, 32, 2>(stream, p, pairs);
    }
    // Two teams' tiles of 128 columns fill an SM's shared memory, so a CTA has an SM to itself and whole walks come in waves.  64
    // rows without teams read each key half as often and take 16/9 of a wave's time: they win where their waves are few enough
    // (us with two teams and with 64 rows, whole: 12 heads x 500, 2 waves and 1, 82.5 and 74.7; x 900, 3 and 2, 215 and 260; 24 x
    // 600, 4 and 2, 193 and 176; x 900, 5 and 3, 360 and 389; x 1500, 8 and 4, 902 and 847).  Causal walks fill each other's
    // gaps: 64 rows gain from three and a half waves on (12 x 700 59 and 100, 12 x 1200 166 and 170, 12 x 1500 234 and 227, 24 x
    // 700 117 and 105, 48 x 700 236 and 212).
    auto waves = [&](size_t ctas) { return (ctas + sms - 1) / sms; };
    const size_t tall = pairs * ((static_cast<size_t>(p.query_len) + 63) / 64);
    const bool teams = p.causal ? 2 * blocks < 7 * sms : 9 * waves(blocks) <= 16 * waves(tall);
    return teams ? launch<128, 4, 32, 2>(stream, p, pairs) : launch<128, 4, 64, 1>(stream, p, pairs);
}

}  // namespace singe
