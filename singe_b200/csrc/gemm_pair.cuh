// Prompt-sized linear layers on pairs of SMs: out[M, N] = lhs[M, K] . rhs^T with tcgen05.mma of cta_group::2.
//
// Bound: the tensor core, under the board's power limit.  The two CTAs of a cluster (two neighbouring SMs) share tiles of
// 256 x BN.  Each keeps its own 128 rows of A and HALF of the columns of B in shared memory, and one MMA of
// 256 x BN x 16, issued by the leader (cluster rank 0), reads both halves.  Against a tile of 256 x 256 in one CTA, whose
// bytes from L2 per flop are the same:
//   * an accumulator is 128 lanes x BN columns in each CTA, so two of them fit the 512 columns of tensor memory and a
//     tile's epilogue runs while the next tile's MMAs do;
//   * 74 pairs walk tiles that take half as long, so the last, partly filled wave costs half as much;
//   * an MMA reads B once for both SMs instead of once each: less shared-memory traffic per flop, hence less power and a
//     higher clock under the limit.
// Results leave through shared memory and TMA stores (whole 32-byte sectors, tails clipped by the tensor map); an output
// that TMA cannot address (odd strides) is written directly.
//
// The loops of the loading and the issuing warp run in one elected thread each.  Measured by the SM clock: with the warp in
// step, a vote after each wait and the issue under `lane == 0`, a 64-wide K slice took 650 clk whatever the tile's width
// (433 to issue, the rest to wait); in an elected thread 540 at 256 columns (512 of them MMA), 360 at 64.
// (M, N, K) = (4096, 14336, 4096): one CTA's tiles of 256 x 256 390 - 440 us, now 334 - 345 = 1410 - 1440 TFLOP/s under the
// power limit; (1024, 4096, 4096) 55 and 27; (256, 4096, 4096) 51 and 17.
//
// Barriers.  `full` and `acc_empty` live in the leader, which alone waits for them: loads of both CTAs complete their bytes
// on the leader's `full`, epilogue warps of both CTAs arrive at its `acc_empty`.  `empty` and `acc_full` exist in both:
// tcgen05.commit arrives at them in both CTAs at once.  The peer's loads may complete bytes before the leader has
// announced them: the phase cannot end before the leader's own arrival.  Every wait is bounded.
#pragma once

// Part of gemm_tcgen05.cu: uses its GemmParams, tile order and epilogue functions.
namespace singe {
namespace {

constexpr int kPairRows = 256;
constexpr int kPairStaging = 4 * 2 * 4096;  // per epilogue warp two buffers of 32 rows x up to 128 bytes

__device__ __forceinline__ void pair_tmem_alloc(uint32_t smem_holder, uint32_t columns) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_holder), "r"(columns)
                 : "memory");
}

__device__ __forceinline__ void pair_tmem_relinquish() {
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}

__device__ __forceinline__ void pair_tmem_dealloc(uint32_t address, uint32_t columns) {
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(address), "r"(columns) : "memory");
}

__device__ __forceinline__ void pair_umma(uint32_t tmem_d, uint64_t a_desc, uint64_t b_desc, uint32_t idesc,
                                          uint32_t accumulate) {
    asm volatile(
        "{\n"
        ".reg .pred p;\n"
        "setp.ne.b32 p, %4, 0;\n"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n"
        "}\n" ::"r"(tmem_d),
        "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
        : "memory");
}

// Arrives at the barrier of this offset in both CTAs when the thread's MMAs so far have completed.
__device__ __forceinline__ void pair_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
                 ::"r"(bar), "h"(static_cast<uint16_t>(3))
                 : "memory");
}

// A tile into this CTA's shared memory that completes its bytes on `bar`, a shared::cluster address in either CTA.
__device__ __forceinline__ void pair_load_2d(uint32_t dst, const CUtensorMap *map, uint32_t bar, int32_t c0, int32_t c1) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes.cta_group::2 "
        "[%0], [%1, {%3, %4}], [%2];"
        ::"r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(bar), "r"(c0), "r"(c1)
        : "memory");
}

__device__ __forceinline__ uint32_t leader_address(uint32_t own) {
    uint32_t address;
    asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(address) : "r"(own));
    return address;
}

__device__ __forceinline__ void pair_arrive(uint32_t cluster_bar) {
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_bar) : "memory");
}

__device__ __forceinline__ bool pair_wait(uint32_t bar, uint32_t parity) {
    long long start = 0;
    for (;;) {
        uint32_t done;
        asm volatile(
            "{\n"
            ".reg .pred p;\n"
            "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n"
            "selp.u32 %0, 1, 0, p;\n"
            "}\n"
            : "=r"(done)
            : "r"(bar), "r"(parity)
            : "memory");
        if (done) return true;
        if (start == 0) start = clock64();
        if (clock64() - start > kWaitLimitCycles) return false;
    }
}

// This CTA's half of a 64-wide K slice of B: BN / 2 rows of [N, K] weights, or BN / 128 boxes of 64 columns of a [K, N]
// operand (see load_b_slice).
template <int BN, bool KN>
__device__ __forceinline__ void pair_load_b(uint32_t dst, const CUtensorMap *map, uint32_t bar, int k0, int n0) {
    if (!KN) {
        pair_load_2d(dst, map, bar, k0, n0);
    } else {
#pragma unroll
        for (int h = 0; h < BN / 128; ++h) pair_load_2d(dst + h * 8192, map, bar, n0 + h * 64, k0);
    }
}

// 32 accumulators of a row, as 32-bit words, to what the row stores: 32 floats, 32 bf16 or 16 gated bf16.
__device__ __forceinline__ int pair_pack(const GemmParams &p, uint32_t (&r)[32]) {
    if (p.squared_relu) {
#pragma unroll
        for (int j = 0; j < 32; ++j) r[j] = __float_as_uint(squared_relu_f32(__uint_as_float(r[j])));
    }
    if (p.gated) {
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            r[j] = pack2<__nv_bfloat16>(gated_value(__uint_as_float(r[4 * j]), __uint_as_float(r[4 * j + 1])),
                                        gated_value(__uint_as_float(r[4 * j + 2]), __uint_as_float(r[4 * j + 3])));
        }
        return 2;
    }
    if (!p.out_f32) {
#pragma unroll
        for (int j = 0; j < 16; ++j) {
            r[j] = pack2<__nv_bfloat16>(__uint_as_float(r[2 * j]), __uint_as_float(r[2 * j + 1]));
        }
        return 4;
    }
    return 8;
}

template <int BN, bool KN>
__global__ void __launch_bounds__(kGemmThreads, 1)
    gemm_pair_kernel(const __grid_constant__ CUtensorMap a_map, const __grid_constant__ CUtensorMap b_map,
                     const __grid_constant__ CUtensorMap out_map, const GemmParams p) {
    constexpr uint32_t kTmemColumns = 512;
    constexpr uint32_t kAccumulator = 256;  // columns between the two accumulators
    constexpr uint32_t kIdesc = make_instr_desc(kPairRows, BN, true, 0, KN ? 1 : 0);
    constexpr int kABytes = kBlockM * 128;
    constexpr int kBBytes = BN / 2 * 128;
    constexpr int kStageBytes = kABytes + kBBytes;
    static_assert(BN % 32 == 0 && BN <= 256 && kBBytes % 1024 == 0, "tiles of whole swizzle atoms");

    grid_launch_dependents();
    extern __shared__ uint8_t smem_raw[];
    const uint32_t raw = smem_u32(smem_raw);
    const uint32_t base = (raw + 1023u) & ~1023u;
    const uint32_t staging = base + p.stages * kStageBytes;
    const uint32_t bars = staging + kPairStaging;
    const uint32_t bar_full = bars;
    const uint32_t bar_empty = bars + kMaxStages * 8;
    const uint32_t bar_acc_full = bars + 2 * kMaxStages * 8;
    const uint32_t bar_acc_empty = bar_acc_full + 16;
    const uint32_t tmem_holder = bar_acc_empty + 16;
    volatile uint32_t *tmem_holder_ptr = reinterpret_cast<volatile uint32_t *>(smem_raw + (tmem_holder - raw));

    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    const int rank = static_cast<int>(cluster_rank());
    const int pair = blockIdx.x >> 1;
    const int pairs = gridDim.x >> 1;
    const int total_tiles = p.tiles_m * p.tiles_n;

    if (threadIdx.x == 0) {
        for (int s = 0; s < p.stages; ++s) {
            mbar_init(bar_full + s * 8, 1);
            mbar_init(bar_empty + s * 8, 1);
        }
        for (int a = 0; a < 2; ++a) {
            mbar_init(bar_acc_full + a * 8, 1);
            mbar_init(bar_acc_empty + a * 8, 8);
        }
        mbar_init_fence();
    }
    if (warp == 1) {
        pair_tmem_alloc(tmem_holder, kTmemColumns);
        pair_tmem_relinquish();
    }
    tcgen05_fence_before();
    __syncthreads();
    cluster_barrier();  // both CTAs' barriers and accumulators exist
    tcgen05_fence_after();
    const uint32_t tmem_base = *tmem_holder_ptr;

    bool failed = false;

    if (warp == 0) {
        // ---------------- TMA producer (one thread): this CTA's rows of A and half of B ----------------
        if (elect_one()) {
            prefetch_tensor_map(&a_map);
            prefetch_tensor_map(&b_map);
            // stable weights: the B halves of the first tile's first stages are requested before the wait (see
            // gemm_bf16_kernel)
            int preloaded = 0;
            if (p.stable_rhs) {
                int tm, tn;
                tile_coordinates(pair, p.tiles_m, p.tiles_n, tm, tn);
                preloaded = min(p.stages, p.k_blocks);
                for (int kb = 0; kb < preloaded; ++kb) {
                    const uint32_t full = bar_full + kb * 8;
                    if (rank == 0) mbar_expect_tx(full, 2 * kStageBytes);
                    pair_load_b<BN, KN>(base + kb * kStageBytes + kABytes, &b_map, leader_address(full), kb * kBlockK,
                                        tn * BN + rank * (BN / 2));
                }
            }
            grid_dependency_wait();  // the A operand comes from the kernel before
            int s = 0;
            uint32_t phase = 0;
            for (int tile = pair; tile < total_tiles && !failed; tile += pairs) {
                int tm, tn;
                tile_coordinates(tile, p.tiles_m, p.tiles_n, tm, tn);
                const int row0 = tm * kPairRows + rank * kBlockM;
                const int column0 = tn * BN + rank * (BN / 2);
                for (int kb = 0; kb < p.k_blocks; ++kb) {
                    const bool early = preloaded > 0;
                    if (!early && !mbar_wait(bar_empty + s * 8, phase ^ 1)) {
                        failed = true;
                        break;
                    }
                    const uint32_t stage = base + s * kStageBytes;
                    const uint32_t full = leader_address(bar_full + s * 8);
                    if (!early && rank == 0) mbar_expect_tx(bar_full + s * 8, 2 * kStageBytes);
                    pair_load_2d(stage, &a_map, full, kb * kBlockK, row0);
                    if (!early) pair_load_b<BN, KN>(stage + kABytes, &b_map, full, kb * kBlockK, column0);
                    if (early) --preloaded;
                    if (++s == p.stages) {
                        s = 0;
                        phase ^= 1;
                    }
                }
            }
            // the commits of the last MMAs arrive here too: neither CTA ends with one of them on its way
            for (int i = 0; i < p.stages && !failed; ++i) {
                if (!mbar_wait(bar_empty + s * 8, phase ^ 1)) failed = true;
                if (++s == p.stages) {
                    s = 0;
                    phase ^= 1;
                }
            }
        }
        __syncwarp();
    } else if (warp == 1) {
        // ---------------- MMA issuer: one thread of the leader, for both CTAs ----------------
        if (rank == 0 && elect_one()) {
            int s = 0;
            uint32_t phase = 0;
            int local = 0;
            for (int tile = pair; tile < total_tiles && !failed; tile += pairs, ++local) {
                const int acc = local & 1;
                if (!pair_wait(bar_acc_empty + acc * 8, ((local >> 1) & 1) ^ 1)) {
                    failed = true;
                    break;
                }
                tcgen05_fence_after();
                const uint32_t tmem_d = tmem_base + acc * kAccumulator;
                for (int kb = 0; kb < p.k_blocks; ++kb) {
                    if (!pair_wait(bar_full + s * 8, phase)) {
                        failed = true;
                        break;
                    }
                    tcgen05_fence_after();
                    const uint32_t stage = base + s * kStageBytes;
                    const uint64_t a_desc = make_smem_desc(stage, 16, 1024);
                    const uint64_t b_desc = make_smem_desc(stage + kABytes, BWalk<KN>::kLeadingBytes, 1024);
#pragma unroll
                    for (int ks = 0; ks < kBlockK / 16; ++ks) {
                        pair_umma(tmem_d, a_desc + 2 * ks, b_desc + BWalk<KN>::kStep * ks, kIdesc, (kb > 0 || ks > 0) ? 1u : 0u);
                    }
                    pair_commit(bar_empty + s * 8);
                    if (kb == p.k_blocks - 1) pair_commit(bar_acc_full + acc * 8);
                    if (++s == p.stages) {
                        s = 0;
                        phase ^= 1;
                    }
                }
            }
        }
        __syncwarp();
    } else {
        // ---------------- epilogue: this CTA's 128 rows ----------------
        if (warp == 2) warm_l2(p.warm, blockIdx.x, gridDim.x, lane);
        grid_dependency_wait();  // nothing is stored while an earlier kernel may still read the output buffer
        const int quarter = warp & 3;  // tensor-memory lanes 32*quarter .. +31
        const uint32_t buffers = staging + quarter * 8192;
        const int halve = p.gated ? 1 : 0;
        int local = 0;
        uint32_t chunk = 0;
        for (int tile = pair; tile < total_tiles && !failed; tile += pairs, ++local) {
            int tm, tn;
            tile_coordinates(tile, p.tiles_m, p.tiles_n, tm, tn);
            const int acc = local & 1;
            if (!__all_sync(0xffffffffu, pair_wait(bar_acc_full + acc * 8, (local >> 1) & 1) ? 1 : 0)) {
                failed = true;
                break;
            }
            tcgen05_fence_after();
            const int row0 = tm * kPairRows + rank * kBlockM + quarter * 32;
            const uint32_t taddr = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + acc * kAccumulator;
#pragma unroll 1
            for (int c = 0; c < BN; c += 32) {
                const int column = tn * BN + c;
                if (row0 >= p.m || column >= p.n) break;  // the same for the whole warp
                uint32_t r[32];
                tmem_ld_x32(taddr + c, r);
                tmem_wait_ld();
                if (p.vector_store) {
                    const int pieces = pair_pack(p, r);  // 16-byte pieces of a row
                    const uint32_t buffer = buffers + (chunk++ & 1u) * 4096;
                    if (elect_one()) tma_store_wait_read<1>();  // the store that used this buffer has read it
                    __syncwarp();
#pragma unroll
                    for (int j = 0; j < 8; ++j) {
                        if (j < pieces) {
                            // the tensor map's swizzle: 16-byte pieces move within a row of `pieces` by address bits 7 and up
                            const uint32_t linear = lane * pieces * 16 + j * 16;
                            const uint32_t at = buffer + (linear ^ (((linear >> 7) & (pieces - 1)) << 4));
                            asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};"
                                         ::"r"(at), "r"(r[4 * j]), "r"(r[4 * j + 1]), "r"(r[4 * j + 2]), "r"(r[4 * j + 3])
                                         : "memory");
                        }
                    }
                    fence_proxy_async_shared();
                    __syncwarp();
                    if (elect_one()) {
                        tma_store_2d(&out_map, buffer, column >> halve, row0);
                        tma_store_commit();
                    }
                } else if (row0 + lane < p.m) {
                    const long long start = static_cast<long long>(row0 + lane) * p.ldo + (column >> halve);
                    const int count = min(32, p.n - column) >> halve;
                    if (p.out_f32) {
                        if (p.squared_relu) {
#pragma unroll
                            for (int j = 0; j < 32; ++j) r[j] = __float_as_uint(squared_relu_f32(__uint_as_float(r[j])));
                        }
                        float *dst = static_cast<float *>(p.out) + start;
#pragma unroll
                        for (int j = 0; j < 32; ++j) {
                            if (j < count) dst[j] = __uint_as_float(r[j]);
                        }
                    } else {
                        pair_pack(p, r);
                        unsigned short *dst = static_cast<unsigned short *>(p.out) + start;
#pragma unroll
                        for (int j = 0; j < 32; ++j) {
                            if (j < count) dst[j] = static_cast<unsigned short>(r[j / 2] >> (16 * (j & 1)));
                        }
                    }
                }
            }
            tcgen05_fence_before();
            __syncwarp();
            if (lane == 0) pair_arrive(leader_address(bar_acc_empty + acc * 8));
        }
        __syncwarp();
        if (elect_one()) tma_store_wait<0>();
    }
    if (failed) report_status(p.error, kStatusWaitTimeout);
    if (failed) linger_after_timeout();
    tcgen05_fence_before();
    __syncwarp();
    cluster_barrier();  // the peer's last MMA has read this CTA's shared memory, its last arrivals have landed
    if (warp == 1) {
        tcgen05_fence_after();
        pair_tmem_dealloc(tmem_base, kTmemColumns);
    }
}

}  // namespace
}  // namespace singe
