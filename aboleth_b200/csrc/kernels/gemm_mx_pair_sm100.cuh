// Block-scaled e4m3 GEMM main loop on CTA pairs: tcgen05.mma.cta_group::2.kind::mxf8f6f4.block_scale.
//
// The arithmetic and the packed scale factors are those of gemm_mx_sm100.cuh, the division of labour that of
// gemm_pair_sm100.cuh: two CTAs compute a 256 x 256 tile, each loads 128 rows of A and 128 rows of B per K block
// of 128 (32 KiB in 512 cycles of MMAs, what an SM takes in; a 128 x 256 tile of one CTA loads 48 KiB, a
// 256 x 192 one 56 KiB in 768).  A's scale factors are needed only where its rows are; B's in both CTAs, since
// each multiplies its rows with all 256 columns.  `tcgen05.cp.cta_group::2` copies in each CTA from its own
// shared memory.  The atoms travel as tiled copies ([atoms][128 words]), whose bytes may complete on the leader's
// barrier; untiled bulk copies may not.
//
// Tensor memory: two accumulators of 256 columns and 12 columns of scale factors are 12 more than there are.  So
// the accumulators share 32 columns: slot 0 is [0, 256), slot 1 [224, 480), the scales [480, 492).  The epilogue
// reads a finished tile's shared columns first and then lets the next tile start, in the other slot, while it reads
// the rest: of the epilogue only that first eighth is ever waited for.  (A slot's own previous tile is out by
// then: the same warps drained it before.)  The one-CTA loop has no second accumulator; its SwiGLU epilogue took
// about 6 of the 19 us of a 128 x 256 tile.
//
// MoE layer, 4096 tokens x 4096 x 14336, 8 experts, top-2, e4m3: gate and up product 1000 -> 751 us, down
// product 437 -> 388 us (2.5 PFLOP/s), the layer 1869 -> 1491 us.
#pragma once

#include "gemm_mx_sm100.cuh"
#include "gemm_pair_sm100.cuh"

namespace ab::gemm::mxpair {

using pair::cluster_rank;
using pair::cluster_sync;
using pair::map_to_cta;
using pair::pair_tma_load_2d;
using pair::pair_umma_commit;
using pair::pair_wait;
using pair::raise_abort;
using pair::remote_arrive;

struct Geometry {
    static constexpr int kTileRows = 2 * BM;
    static constexpr int kStages = 5;
    static constexpr unsigned kBytesA = BM * mx::kBlockK;            // per CTA and stage
    static constexpr unsigned kBytesB = (BN / 2) * mx::kBlockK;
    static constexpr unsigned kOffSfa = kBytesA + kBytesB;           // one atom
    static constexpr unsigned kOffSfb = kOffSfa + mx::kAtomBytes;    // two atoms
    static constexpr unsigned kStageTx = kOffSfb + 2 * mx::kAtomBytes;
    static constexpr unsigned kStageStride = (kStageTx + 1023) / 1024 * 1024;
    static constexpr unsigned kSmemBytes = kStages * kStageStride + kEpilogueStageBytes + 1024;
    static constexpr unsigned kSlot1 = BN - 32, kSfaCol = kSlot1 + BN, kSfbCol = kSfaCol + 4;
};

__device__ __forceinline__ void pair_sf_copy(std::uint32_t tmem_addr, std::uint64_t desc) {
    asm volatile("tcgen05.cp.cta_group::2.32x128b.warpx4 [%0], %1;" ::"r"(tmem_addr), "l"(desc) : "memory");
}

__device__ __forceinline__ void pair_umma_mx(std::uint32_t d_tmem, std::uint64_t a_desc, std::uint64_t b_desc,
                                             std::uint32_t idesc, std::uint32_t sfa_tmem, std::uint32_t sfb_tmem,
                                             std::uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::mxf8f6f4.block_scale [%0], %1, %2, %3, [%5], [%6], p;\n\t}"
        ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate), "r"(sfa_tmem), "r"(sfb_tmem)
        : "memory");
}

// Tensor maps of the packed scale factors: [atoms][128 words].
struct Maps {
    const CUtensorMap *a, *b, *sfa, *sfb;
};

// Policy concept: the one of gemm_mainloop_pair (the same tile for both CTAs, 256 rows), plus
//   k_blocks_a    - K blocks per row of A's atoms        granules - 64-column granules per K block of B's
template <typename Policy>
__device__ __forceinline__ void gemm_mx_mainloop_pair(Policy &policy, const Maps &maps, int k_blocks_a, int granules,
                                                      unsigned long long *status) {
    using G = Geometry;
    extern __shared__ std::uint8_t smem_raw[];
    __shared__ pair::PairState st;
    std::uint8_t *tiles = reinterpret_cast<std::uint8_t *>(
        (reinterpret_cast<std::uintptr_t>(smem_raw) + 1023) & ~static_cast<std::uintptr_t>(1023));
    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    const unsigned rank = cluster_rank();  // 0: leader
    const bool leader = rank == 0;

    if (threadIdx.x == 0) {
        for (int s = 0; s < G::kStages; ++s) {
            mbar_init(&st.full[s], 1);   // the leader's arrival carries the byte count of BOTH CTAs' loads
            mbar_init(&st.empty[s], 1);  // one multicast commit
        }
        for (int b = 0; b < 2; ++b)
            mbar_init(&st.tmem_full[b], 1);
        mbar_init(&st.tmem_empty[0], 2 * kEpilogueWarps);  // the shared columns of a tile are read
        st.abort = 0;
        mbar_fence_init();
        prefetch_tensormap(maps.a);
        prefetch_tensormap(maps.b);
        prefetch_tensormap(maps.sfa);
        prefetch_tensormap(maps.sfb);
    }
    if (warp == 1)
        pair::pair_tmem_alloc(&st.tmem_base, kTmemCols);
    tc_fence_before();
    __syncthreads();
    cluster_sync();  // both CTAs' barriers exist before anything is signalled across
    tc_fence_after();
    const std::uint32_t tmem_base = st.tmem_base;

    if (warp == 0) {
        // ---------------- producer (both CTAs): operand tiles and scale-factor atoms ----------------
        const bool elected = elect_one();
        int stage = 0;
        unsigned phase = 0;
        Tile t;
        for (int it = 0; !warp_aborted(st.abort) && policy.next(it, t); ++it) {
            if (!__all_sync(0xffffffffu, !elected || policy.ready(t))) {
                raise_abort(st, rank);
                set_status(status, aboleth::Status::Timeout, 0x3000 + t.tag);
                break;
            }
            const int a_row = t.a_row + static_cast<int>(rank) * BM;
            int b_row = t.b_row + static_cast<int>(rank) * (BN / 2), next_granule = BN / 2 / 64;
            if constexpr (Policy::kSwiGlu) {
                b_row = rank == 0 ? t.b_row : t.b_row2;
                next_granule = (t.b_row2 - t.b_row) / 64;
            }
            int sfa = a_row / BM * k_blocks_a, sfb = t.b_row / 64;
            for (int kb = 0; kb < t.k_blocks; ++kb) {
                if (!warp_wait(&st.empty[stage], phase ^ 1, &st.abort)) {
                    raise_abort(st, rank);
                    set_status(status, aboleth::Status::Timeout, 0x3100 + stage);
                    break;
                }
                std::uint8_t *s = tiles + stage * G::kStageStride;
                const std::uint32_t full_in_leader = map_to_cta(smem_u32(&st.full[stage]), 0);
                if (elected) {
                    if (leader)
                        mbar_expect_tx(&st.full[stage], 2 * G::kStageTx);
                    pair_tma_load_2d(s, maps.a, kb * mx::kBlockK, a_row, full_in_leader);
                    pair_tma_load_2d(s + G::kBytesA, maps.b, kb * mx::kBlockK, b_row, full_in_leader);
                    pair_tma_load_2d(s + G::kOffSfa, maps.sfa, 0, sfa, full_in_leader);
                    pair_tma_load_2d(s + G::kOffSfb, maps.sfb, 0, sfb, full_in_leader);
                    pair_tma_load_2d(s + G::kOffSfb + mx::kAtomBytes, maps.sfb, 0, sfb + next_granule, full_in_leader);
                }
                __syncwarp();
                ++sfa;
                sfb += granules;
                if (++stage == G::kStages) {
                    stage = 0;
                    phase ^= 1;
                }
            }
        }
    } else if (warp == 1) {
        // ---------------- MMA issuer (leader only) ----------------
        if (leader) {
            const bool elected = elect_one();
            int stage = 0;
            unsigned phase = 0;
            Tile t;
            for (int it = 0; !warp_aborted(st.abort) && policy.next(it, t); ++it) {
                const int slot = it & 1;
                const std::uint32_t d = tmem_base + slot * G::kSlot1;
                // Both CTAs' epilogues have read the columns that this tile shares with the one before.
                if (it > 0 && !__all_sync(0xffffffffu, pair_wait(&st.tmem_empty[0], (it - 1) & 1, &st.abort))) {
                    raise_abort(st, rank);
                    set_status(status, aboleth::Status::Timeout, 0x3200 + slot);
                    break;
                }
                tc_fence_after();
                for (int kb = 0; kb < t.k_blocks; ++kb) {
                    if (!warp_wait(&st.full[stage], phase, &st.abort)) {
                        raise_abort(st, rank);
                        set_status(status, aboleth::Status::Timeout, 0x3300 + stage);
                        break;
                    }
                    tc_fence_after();
                    const std::uint32_t s = smem_u32(tiles + stage * G::kStageStride);
                    const std::uint64_t da = smem_desc_sw128(s), db = smem_desc_sw128(s + G::kBytesA);
                    if (elected) {
                        pair_sf_copy(tmem_base + G::kSfaCol, mx::sf_desc(s + G::kOffSfa));
                        pair_sf_copy(tmem_base + G::kSfbCol, mx::sf_desc(s + G::kOffSfb));
                        pair_sf_copy(tmem_base + G::kSfbCol + 4, mx::sf_desc(s + G::kOffSfb + mx::kAtomBytes));
#pragma unroll
                        for (unsigned k = 0; k < 4; ++k)  // 32 e4m3 = 32 bytes of K each
                            pair_umma_mx(d, da + 2 * k, db + 2 * k, mx::idesc_mx(2 * BM, BN, k),
                                         tmem_base + G::kSfaCol, tmem_base + G::kSfbCol,
                                         (kb | static_cast<int>(k)) != 0);
                        pair_umma_commit(&st.empty[stage]);  // frees the stage in both CTAs
                    }
                    __syncwarp();
                    if (++stage == G::kStages) {
                        stage = 0;
                        phase ^= 1;
                    }
                }
                if (elected)
                    pair_umma_commit(&st.tmem_full[slot]);  // accumulator complete, both CTAs
                __syncwarp();
            }
        }
    } else {
        // ---------------- epilogue (warps 2..5, both CTAs) ----------------
        const int quarter = warp & 3;
        const int epi_thread = (warp - 2) * 32 + lane;
        constexpr int kEpiThreads = kEpilogueWarps * 32;
        uint4 *epi_stage = reinterpret_cast<uint4 *>(tiles + G::kStages * G::kStageStride +
                                                     (warp - 2) * kEpilogueWarpStageBytes);
        // As in gemm_mainloop: one sample of the abort flag decides for all four warps.
        auto epilogue_aborted = [&]() -> bool {
            if (epi_thread == 0)
                st.epi_abort = st.abort;
            asm volatile("bar.sync 1, 128;" ::: "memory");
            const int sample = st.epi_abort;
            asm volatile("bar.sync 1, 128;" ::: "memory");
            return sample != 0;
        };
        // Called by every warp once it has read its part of a tile's shared columns.
        auto release = [&]() {
            tc_fence_before();
            __syncwarp();
            if (lane == 0)
                remote_arrive(map_to_cta(smem_u32(&st.tmem_empty[0]), 0));
        };
        Tile t;
        bool aborted = false;
        for (int it = 0; policy.next(it, t); ++it) {
            if ((aborted = epilogue_aborted()))
                break;
            const int slot = it & 1;
            if (!warp_wait(&st.tmem_full[slot], (it >> 1) & 1, &st.abort)) {
                raise_abort(st, rank);
                set_status(status, aboleth::Status::Timeout, 0x3400 + slot);
            } else {
                tc_fence_after();
                const std::uint32_t taddr = tmem_base + (static_cast<std::uint32_t>(quarter * 32) << 16) +
                                            slot * G::kSlot1;
                const int row_base = static_cast<int>(rank) * BM + quarter * 32;
                // Slot 0 shares its last 32 columns, slot 1 its first.
                if constexpr (Policy::kSwiGlu) {
                    if (slot == 0)
                        mx::drain_swiglu_quant32<true>(policy, t, taddr, row_base, epi_stage, lane, status, release);
                    else
                        mx::drain_swiglu_quant32<false>(policy, t, taddr, row_base, epi_stage, lane, status, release);
                } else {
                    drain_rows32(policy, t, taddr, row_base, epi_stage, lane, slot == 0, release);
                }
            }
            asm volatile("bar.sync 1, 128;" ::: "memory");
            if (warp == 2 && lane == 0)
                policy.tile_done(t);
        }
        if (!aborted && !epilogue_aborted())
            policy.finish(epi_thread, kEpiThreads, status);
    }

    // ---------------- teardown ----------------
    __syncwarp();
    if (warp_aborted(st.abort)) {
        const std::uint64_t t0 = aboleth::detail::globaltimer_ns();
        while (aboleth::detail::globaltimer_ns() - t0 < 2000000ull)
            __nanosleep(1000);
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync();  // the peer no longer reads this CTA's shared memory or signals its barriers
    tc_fence_after();
    if (warp == 1)
        pair::pair_tmem_dealloc(tmem_base, kTmemCols);
}

}  // namespace ab::gemm::mxpair
