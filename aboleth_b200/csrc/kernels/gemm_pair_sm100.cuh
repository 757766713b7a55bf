// The CTA-pair form of the tcgen05 GEMM main loop (tcgen05 `cta_group::2`).
//
// Two CTAs of one cluster (the two SMs of a TPC) compute one 256 x 256 tile together:
//
//   * CTA r of the pair loads rows [r*128, r*128+128) of the A tile and rows
//     [r*128, r*128+128) of the B tile (half of N) into ITS OWN shared memory - 32 KiB per
//     128-byte K step, where a CTA with a 128 x 256 tile of its own would load 48.  An SM takes in
//     about 64 bytes a cycle, so a step's loads and its four MMAs (512 cycles) are in balance.
//   * Only the pair's leader (cluster rank 0) issues tcgen05.mma.cta_group::2 with
//     M = 256, N = 256: the instruction reads A and B from both CTAs' shared memory and
//     accumulates rows r*128.. of the tile in CTA r's tensor memory, 256 fp32 columns.
//   * Each CTA therefore needs 256 of its 512 TMEM columns per tile: the accumulator is
//     double buffered, and the epilogue of tile i overlaps the main loop of tile i+1.
//
// A 512 x 256 tile (two accumulators sharing a B tile, a third less traffic, the epilogue exposed) was the
// faster shape while issuing a K step took longer than its MMAs.  Both at full rate, back to back, inputs of two
// sets in turn: 8192 x 3584 x 8192 383 us (512 x 256: 423), 8192^3 831 (840), 8192 x 28672 x 8192 2913 (3031);
// e4m3 197 (234), 431 (465), 1481 (1633).  Half the tile also wastes half as much of a last wave.
//
// Barriers.  `full[s]` lives in the leader: both CTAs' TMA loads complete their bytes on
// it (the peer's loads name the leader's barrier through its shared::cluster address); the
// leader's producer makes the one arrival and announces the bytes of both.  `empty[s]`,
// `tmem_full[b]` exist in both CTAs and are signalled by one tcgen05.commit that is multicast
// to the pair.  `tmem_empty[b]` lives in the leader and counts the epilogue warps of both CTAs.
// No TMA load is multicast.
//
// Every wait is bounded as in the single-CTA loop; the two CTAs meet at a cluster barrier
// before the tensor memory is freed, so neither leaves while its peer can still touch it.
#pragma once

#include "gemm_sm100.cuh"

// Statements that exist only in a build with cycle counters (-DAB_GEMM_TRACE).
#ifdef AB_GEMM_TRACE
#define AB_TRACE(...) __VA_ARGS__
#else
#define AB_TRACE(...)
#endif

namespace ab::gemm::pair {

// NT = columns of the tile, 256 or 224 (a multiple of 32, the accumulators stay 256 columns apart).
template <int NT>
struct PairGeometry {
    static constexpr int kRowsPerCta = BM;
    static constexpr int kTileRows = 2 * kRowsPerCta;
    static constexpr int kStages = 6;
    static constexpr unsigned kBytesA = kRowsPerCta * BK * 2;    // per CTA and stage
    static constexpr unsigned kBytesB = (NT / 2) * BK * 2;
    static constexpr unsigned kStageBytes = kBytesA + kBytesB;
    static constexpr unsigned kSmemBytes = kStages * kStageBytes + kEpilogueStageBytes + 1024;
};
constexpr int kPairMaxStages = 6;

struct PairState {
    std::uint64_t full[kPairMaxStages];    // used in the leader only
    std::uint64_t empty[kPairMaxStages];
    std::uint64_t tmem_full[2];
    std::uint64_t tmem_empty[2];        // used in the leader only
    std::uint32_t tmem_base;
    volatile int abort;
    volatile int epi_abort;  // epilogue warps: shared sample of `abort`
};

// Raise `abort` in this CTA and in its pair CTA: either of them giving up must end both, because
// each one's barriers are completed by the other.
__device__ __forceinline__ void raise_abort(PairState &st, unsigned rank);

__device__ __forceinline__ unsigned cluster_rank() {
    unsigned r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}

// shared::cluster address of `local` (a shared::cta address of this CTA) in CTA `rank`.
__device__ __forceinline__ std::uint32_t map_to_cta(std::uint32_t local, unsigned rank) {
    std::uint32_t remote;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(local), "r"(rank));
    return remote;
}

__device__ __forceinline__ void raise_abort(PairState &st, unsigned rank) {
    st.abort = 1;
    const std::uint32_t remote = map_to_cta(smem_u32(const_cast<int *>(&st.abort)), rank ^ 1u);
    asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(remote), "r"(1) : "memory");
}

__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

__device__ __forceinline__ void pair_tmem_alloc(std::uint32_t *holder, unsigned cols) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32(holder)),
                 "r"(cols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}

__device__ __forceinline__ void pair_tmem_dealloc(std::uint32_t base, unsigned cols) {
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(base), "r"(cols)
                 : "memory");
}

template <typename Op>
__device__ __forceinline__ void pair_umma(std::uint32_t d_tmem, std::uint64_t a_desc, std::uint64_t b_desc,
                                          std::uint32_t idesc, std::uint32_t accumulate) {
    if constexpr (Op::kBK == 64) {
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "setp.ne.b32 p, %4, 0;\n\t"
            "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
            ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
            : "memory");
    } else {
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "setp.ne.b32 p, %4, 0;\n\t"
            "tcgen05.mma.cta_group::2.kind::f8f6f4 [%0], %1, %2, %3, p;\n\t}"
            ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
            : "memory");
    }
}

// One arrival on the barrier at this shared-memory offset in BOTH CTAs of the pair once
// every tcgen05 operation issued so far by this thread is done.
__device__ __forceinline__ void pair_umma_commit(std::uint64_t *bar) {
    const std::uint16_t mask = 3;
    asm volatile(
        "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::
            "r"(smem_u32(bar)),
        "h"(mask)
        : "memory");
}

// Tiled load into this CTA's shared memory whose bytes complete on a barrier that may
// belong to the peer CTA (shared::cluster address).  Not multicast.
__device__ __forceinline__ void pair_tma_load_2d(void *smem_dst, const CUtensorMap *map, int x, int y,
                                                 std::uint32_t bar_cluster_addr) {
    asm volatile(
        "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes "
        "[%0], [%1, {%3, %4}], [%2];" ::"r"(smem_u32(smem_dst)),
        "l"(map), "r"(bar_cluster_addr), "r"(x), "r"(y)
        : "memory");
}

__device__ __forceinline__ void remote_arrive(std::uint32_t bar_cluster_addr) {
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar_cluster_addr)
                 : "memory");
}

// A wait that also acquires, at cluster scope, what the peer CTA released.  Used once per tile
// (the accumulator hand-back); the per-K-step waits use the CTA-scope form.
__device__ __forceinline__ bool pair_try_wait(std::uint64_t *bar, unsigned parity) {
    unsigned ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}

__device__ __forceinline__ bool pair_wait(std::uint64_t *bar, unsigned parity, const volatile int *abort) {
    for (int i = 0; i < 4096; ++i)
        if (pair_try_wait(bar, parity))
            return true;
    const std::uint64_t start = aboleth::detail::globaltimer_ns();
    while (!pair_try_wait(bar, parity)) {
        if (aboleth::detail::globaltimer_ns() - start > 4000000000ull || *abort != 0)
            return false;
    }
    return true;
}

// Policy concept: the one of gemm_mainloop, with tiles of 256 rows, one A operand and no background work or drained
// hook.
// `policy.next` must hand the SAME tile to both CTAs of a pair (index tiles by blockIdx.x / 2
// out of gridDim.x / 2).  Rows passed to `store16` are rows of the tile.  map_a and map_b boxes
// are 128 and NT / 2 rows x 128 bytes; `Op` selects bf16 or e4m3 operands.
template <typename Op, int NT, typename Policy>
__device__ __forceinline__ void gemm_mainloop_pair(Policy &policy, const CUtensorMap *map_a,
                                                   const CUtensorMap *map_b, unsigned long long *status) {
    using G = PairGeometry<NT>;
    constexpr int kStagesG = G::kStages;
    extern __shared__ std::uint8_t smem_raw[];
    __shared__ PairState st;
    std::uint8_t *tiles = reinterpret_cast<std::uint8_t *>(
        (reinterpret_cast<std::uintptr_t>(smem_raw) + 1023) & ~static_cast<std::uintptr_t>(1023));
    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    const unsigned rank = cluster_rank();  // 0: leader
    const bool leader = rank == 0;

    if (threadIdx.x == 0) {
        for (int s = 0; s < kStagesG; ++s) {
            mbar_init(&st.full[s], 1);   // the leader's arrival carries the byte count of BOTH CTAs' loads
            mbar_init(&st.empty[s], 1);  // one multicast commit
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(&st.tmem_full[b], 1);
            mbar_init(&st.tmem_empty[b], 2 * kEpilogueWarps);
        }
        st.abort = 0;
        mbar_fence_init();
        prefetch_tensormap(map_a);
        prefetch_tensormap(map_b);
    }
    if (warp == 1)
        pair_tmem_alloc(&st.tmem_base, kTmemCols);
    tc_fence_before();
    __syncthreads();
    cluster_sync();  // both CTAs' barriers exist before anything is signalled across
    tc_fence_after();
    const std::uint32_t tmem_base = st.tmem_base;

    // Accumulator slot (TMEM half) and barrier parity of tile `it`.
    auto slot_of = [](int it) { return it & 1; };
    auto use_of = [](int it) -> unsigned { return (it >> 1) & 1; };

    if (warp == 0) {
        // ---------------- TMA producer (both CTAs) ----------------
        const bool elected = elect_one();
        int stage = 0;
        unsigned phase = 0;
        Tile t;
        AB_TRACE(long long t_wait = 0, t_begin = clock64();)
        for (int it = 0; !warp_aborted(st.abort) && policy.next(it, t); ++it) {
            if (!__all_sync(0xffffffffu, !elected || policy.ready(t))) {
                raise_abort(st, rank);
                set_status(status, aboleth::Status::Timeout, 0x3000 + t.tag);
                break;
            }
            const int a_row = t.a_row + static_cast<int>(rank) * G::kRowsPerCta;
            int b_row = t.b_row + static_cast<int>(rank) * (NT / 2);
            if constexpr (Policy::kSwiGlu)  // the leader brings the gate half, the peer the up half
                b_row = leader ? t.b_row : t.b_row2;
            for (int kb = 0; kb < t.k_blocks; ++kb) {
                AB_TRACE(const long long w0 = clock64();)
                const bool got = warp_wait(&st.empty[stage], phase ^ 1, &st.abort);
                AB_TRACE(t_wait += clock64() - w0;)
                if (!got) {
                    raise_abort(st, rank);
                    set_status(status, aboleth::Status::Timeout, 0x3100 + stage);
                    break;
                }
                std::uint8_t *sa = tiles + stage * G::kStageBytes;
                const std::uint32_t full_in_leader = map_to_cta(smem_u32(&st.full[stage]), 0);
                if (elected) {
                    // The peer does not arrive: its loads only complete bytes on the leader's barrier.
                    // (A cluster-scope release arrive per K step cost ~1400 cycles and starved the pipe.)
                    if (leader)
                        mbar_expect_tx(&st.full[stage], 2 * G::kStageBytes);
                    pair_tma_load_2d(sa, map_a, kb * Op::kBK, a_row, full_in_leader);
                    pair_tma_load_2d(sa + G::kBytesA, map_b, kb * Op::kBK, b_row, full_in_leader);
                }
                __syncwarp();
                if (++stage == kStagesG) {
                    stage = 0;
                    phase ^= 1;
                }
            }
        }
        AB_TRACE(if (blockIdx.x < 2 && status != nullptr) {
            status[2 + 2 * blockIdx.x] = t_wait;                 // producer: cycles waiting for a free stage
            status[3 + 2 * blockIdx.x] = clock64() - t_begin;    // producer: cycles in its loop
        })
    } else if (warp == 1) {
        // ---------------- MMA issuer (leader only) ----------------
        if (leader) {
            constexpr std::uint32_t idesc = Op::idesc(2 * BM, NT);
            const bool elected = elect_one();
            int stage = 0;
            unsigned phase = 0;
            Tile t;
            AB_TRACE(long long t_full = 0, t_acc = 0, t_begin = clock64();)
            for (int it = 0; !warp_aborted(st.abort) && policy.next(it, t); ++it) {
                const unsigned use = use_of(it);
                const int slot = slot_of(it);
                for (int kb = 0; kb < t.k_blocks; ++kb) {
                    AB_TRACE(const long long f0 = clock64();)
                    const bool filled = warp_wait(&st.full[stage], phase, &st.abort);
                    AB_TRACE(t_full += clock64() - f0;)
                    if (!filled) {
                        raise_abort(st, rank);
                        set_status(status, aboleth::Status::Timeout, 0x3300 + stage);
                        break;
                    }
                    tc_fence_after();
                    const std::uint32_t sa = smem_u32(tiles + stage * G::kStageBytes);
                    const std::uint64_t da = smem_desc_sw128(sa), db = smem_desc_sw128(sa + G::kBytesA);
                    if (kb == 0) {
                        // Both CTAs' epilogues must have drained this accumulator.
                        AB_TRACE(const long long a0 = clock64();)
                        const bool free_acc =
                            __all_sync(0xffffffffu, pair_wait(&st.tmem_empty[slot], use ^ 1, &st.abort));
                        AB_TRACE(t_acc += clock64() - a0;)
                        if (!free_acc) {
                            raise_abort(st, rank);
                            set_status(status, aboleth::Status::Timeout, 0x3200 + slot);
                            break;
                        }
                        tc_fence_after();
                    }
                    if (elected) {
#pragma unroll
                        for (int k = 0; k < 4; ++k)  // four MMAs per stage, 32 bytes of K each
                            pair_umma<Op>(tmem_base + slot * BN, da + 2 * k, db + 2 * k, idesc, (kb | k) != 0);
                        pair_umma_commit(&st.empty[stage]);  // frees the stage in both CTAs
                    }
                    __syncwarp();
                    if (++stage == kStagesG) {
                        stage = 0;
                        phase ^= 1;
                    }
                }
                if (elected)
                    pair_umma_commit(&st.tmem_full[slot]);  // accumulator complete, both CTAs
                __syncwarp();
            }
            AB_TRACE(if (blockIdx.x == 0 && status != nullptr) {
                status[6] = t_full;                  // MMA issuer: cycles waiting for operands
                status[7] = t_acc;                   // MMA issuer: cycles waiting for a free accumulator
                status[8] = clock64() - t_begin;     // MMA issuer: cycles in its loop
            })
        }
    } else {
        // ---------------- epilogue (warps 2..5, both CTAs) ----------------
        const int quarter = warp & 3;
        const int epi_thread = (warp - 2) * 32 + lane;
        constexpr int kEpiThreads = kEpilogueWarps * 32;
        uint4 *epi_stage = reinterpret_cast<uint4 *>(tiles + kStagesG * G::kStageBytes +
                                                     (warp - 2) * kEpilogueWarpStageBytes);
        // `abort` is raised asynchronously by the producer or the MMA lane.  The four epilogue warps
        // meet at named barrier 1, so they must all take the same way out: one thread samples the
        // flag and the sample is what all 128 threads branch on.
        auto epilogue_aborted = [&]() -> bool {
            if (epi_thread == 0)
                st.epi_abort = st.abort;
            asm volatile("bar.sync 1, 128;" ::: "memory");
            const int sample = st.epi_abort;
            asm volatile("bar.sync 1, 128;" ::: "memory");
            return sample != 0;
        };
        Tile t;
        bool aborted = false;
        for (int it = 0; policy.next(it, t); ++it) {
            if ((aborted = epilogue_aborted()))
                break;
            const unsigned use = use_of(it);
            const int slot = slot_of(it);
            if (!warp_wait(&st.tmem_full[slot], use, &st.abort)) {
                raise_abort(st, rank);
                set_status(status, aboleth::Status::Timeout, 0x3400 + slot);
            } else {
                tc_fence_after();
                const std::uint32_t taddr = tmem_base + (static_cast<std::uint32_t>(quarter * 32) << 16) + slot * BN;
                const int row_base = static_cast<int>(rank) * G::kRowsPerCta + quarter * 32;
                if constexpr (Policy::kSwiGlu)
                    drain_swiglu32(policy, t, taddr, row_base, epi_stage, lane);
                else
                    drain_rows32(policy, t, taddr, row_base, epi_stage, lane);
                tc_fence_before();
                __syncwarp();
                if (lane == 0)
                    remote_arrive(map_to_cta(smem_u32(&st.tmem_empty[slot]), 0));
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
        pair_tmem_dealloc(tmem_base, kTmemCols);
}

}  // namespace ab::gemm::pair
