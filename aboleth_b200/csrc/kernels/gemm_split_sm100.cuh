// Small-tile tcgen05 GEMM with the K dimension split over a thread-block cluster.
//
//   C[M, N] = A[M, K] * B[N, K]^T,  computed tile by tile as C^T: the MMA's 128 rows are rows of B (weights),
//   its NT columns rows of A (tokens).
//
// Why: the persistent pair loop gives 256 x 256 of C to two SMs.  With few tokens, or a small C, most SMs get
// no tile and the ones that work walk the whole K alone: 32 x 3584 x 8192 takes 43 us on 28 SMs, against the
// 9 us its 59 MB of weights take at copy bandwidth.  Here one CTA owns 128 x NT of C^T and 1 / S of K; the S
// CTAs of a cluster add their fp32 partial tiles through distributed shared memory, in cluster-rank order (the
// result does not depend on timing), and each stores 1 / S of the tile.  No workspace, no second launch.
//
// Weights on the MMA's M side make a token tile as narrow as 32 columns: a decode batch pads to 32 rows and
// not to 128.  It also leaves C's contiguous dimension on the TMEM lanes, so the fp32 tile is staged in
// shared memory as [token][weight row] without bank conflicts and leaves as 256-byte rows.
//
// One tile per CTA, three to five stages of 128-byte K steps; up to 128 columns leave room for two CTAs per SM,
// so that one's prologue and reduction run under the other's loads.  Roles and bounded waits as in
// gemm_sm100.cuh, but no look at the abort flag in them: with one tile the roles' limits run out together (and the
// look took 0.2 us of 18 at 32 x 3584 x 8192).
#pragma once

#include <type_traits>

#include "gemm_mx_sm100.cuh"

namespace ab::gemm::split {

struct OpMx {
    static constexpr int kBK = 128;
};

constexpr int kMaxSplit = 8;
constexpr int kMaxStages = 5;

template <typename Op, int NT>
struct SplitGeometry {
    static constexpr bool kMx = std::is_same<Op, OpMx>::value;
    static constexpr int kBK = Op::kBK;
    static constexpr unsigned kBytesX = BM * 128;   // 128 bytes of K per row and stage
    static constexpr unsigned kBytesY = NT * 128;
    static constexpr int kAtomsY = (NT + 127) / 128;
    static constexpr unsigned kOffSf = kBytesX + kBytesY;
    static constexpr unsigned kStageTx = kOffSf + (kMx ? (1 + kAtomsY) * mx::kAtomBytes : 0);
    static constexpr unsigned kStageStride = (kStageTx + 1023) / 1024 * 1024;
    // Two CTAs per SM up to 128 columns (about 100 KiB each), one with 256.
    static constexpr int kStages = NT >= 256 ? 4 : (NT == 128 ? 3 : (NT == 64 ? 4 : 5));
    static constexpr unsigned kPipeBytes = kStages * kStageStride;
    static constexpr unsigned kTileBytes = BM * NT * 4;  // fp32 partial tile, over the pipeline's stages
    static constexpr unsigned kSmemBytes = (kPipeBytes > kTileBytes ? kPipeBytes : kTileBytes) + 1024;
    static constexpr unsigned kColsUsed = NT + (kMx ? 4 + 4 * kAtomsY : 0);
    static constexpr unsigned kCols = kColsUsed <= 32 ? 32 : kColsUsed <= 64 ? 64 : kColsUsed <= 128 ? 128
                                      : kColsUsed <= 256 ? 256 : 512;
    static constexpr unsigned kSfxCol = NT, kSfyCol = NT + 4;
};

struct SplitParams {
    __nv_bfloat16 *c;
    int m, n, k_blocks, ldc;
    int tiles_y;             // token tiles; they are the fastest index, so a weight panel is shared at once
    int split;               // CTAs per cluster
    float alpha;
    const std::uint8_t *sf_x, *sf_y;  // packed scales of the weights / of the tokens (block-scaled only)
    int granules;            // of the weights' packed scales
    unsigned long long *status;
};

struct SplitState {
    std::uint64_t full[kMaxStages];
    std::uint64_t empty[kMaxStages];
    std::uint64_t done;
    std::uint32_t tmem_base;
    volatile int abort;
};

__device__ __forceinline__ unsigned cluster_rank() {
    unsigned r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}

__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// Four floats of CTA `rank`'s shared memory, at the address `local` has in this CTA.
__device__ __forceinline__ float4 ld_cluster(std::uint32_t local, unsigned rank) {
    std::uint32_t remote;
    float4 v;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(local), "r"(rank));
    asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];"
                 : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(remote) : "memory");
    return v;
}

template <typename Op>
__device__ __forceinline__ void umma(std::uint32_t d, std::uint64_t a, std::uint64_t b, std::uint32_t idesc,
                                     std::uint32_t accumulate) {
    if constexpr (Op::kBK == 64) {
        umma_bf16(d, a, b, idesc, accumulate);
    } else {
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "setp.ne.b32 p, %4, 0;\n\t"
            "tcgen05.mma.cta_group::1.kind::f8f6f4 [%0], %1, %2, %3, p;\n\t}"
            ::"r"(d), "l"(a), "l"(b), "r"(idesc), "r"(accumulate)
            : "memory");
    }
}

template <typename Op, int NT>
__global__ void __launch_bounds__(kThreads, NT >= 256 ? 1 : 2)
gemm_split_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_y,
                  const SplitParams p) {
    using G = SplitGeometry<Op, NT>;
    extern __shared__ std::uint8_t smem_raw[];
    __shared__ SplitState st;
    // Every CTA of a cluster has the same layout, so this address names the same bytes in each of them.
    std::uint8_t *tiles = reinterpret_cast<std::uint8_t *>(
        (reinterpret_cast<std::uintptr_t>(smem_raw) + 1023) & ~static_cast<std::uintptr_t>(1023));
    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    const unsigned rank = p.split > 1 ? cluster_rank() : 0;
    const int tile = blockIdx.x / p.split;
    const int x0 = tile / p.tiles_y * BM, y0 = (tile % p.tiles_y) * NT;
    const int kb0 = static_cast<int>(static_cast<long long>(p.k_blocks) * rank / p.split);
    const int kb1 = static_cast<int>(static_cast<long long>(p.k_blocks) * (rank + 1) / p.split);

    if (threadIdx.x == 0) {
        for (int s = 0; s < G::kStages; ++s) {
            mbar_init(&st.full[s], 1);
            mbar_init(&st.empty[s], 1);
        }
        mbar_init(&st.done, 1);
        st.abort = 0;
        mbar_fence_init();
        prefetch_tensormap(&map_x);
        prefetch_tensormap(&map_y);
    }
    if (warp == 1)
        tmem_alloc(&st.tmem_base, G::kCols);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const std::uint32_t tmem = st.tmem_base;

    // Whole-warp loops, one elected lane around the instructions (see elect_one).
    if (warp == 0) {
        const bool elected = elect_one();
        int stage = 0;
        unsigned phase = 0;
        for (int kb = kb0; kb < kb1; ++kb) {
            if (!warp_wait(&st.empty[stage], phase ^ 1)) {
                st.abort = 1;
                set_status(p.status, aboleth::Status::Timeout, 0x3700 + stage);
                break;
            }
            std::uint8_t *s = tiles + stage * G::kStageStride;
            if (elected) {
                mbar_expect_tx(&st.full[stage], G::kStageTx);
                tma_load_2d(s, &map_x, kb * G::kBK, x0, &st.full[stage]);
                tma_load_2d(s + G::kBytesX, &map_y, kb * G::kBK, y0, &st.full[stage]);
                if constexpr (G::kMx) {
                    bulk_load(s + G::kOffSf,
                              p.sf_x + (static_cast<std::size_t>(kb) * p.granules + x0 / 64) * mx::kAtomBytes,
                              mx::kAtomBytes, &st.full[stage]);
#pragma unroll
                    for (int h = 0; h < G::kAtomsY; ++h)
                        bulk_load(s + G::kOffSf + (1 + h) * mx::kAtomBytes,
                                  p.sf_y + (static_cast<std::size_t>(y0 / BM + h) * p.k_blocks + kb) * mx::kAtomBytes,
                                  mx::kAtomBytes, &st.full[stage]);
                }
            }
            __syncwarp();
            if (++stage == G::kStages) {
                stage = 0;
                phase ^= 1;
            }
        }
    } else if (warp == 1) {
        const bool elected = elect_one();
        int stage = 0;
        unsigned phase = 0;
        for (int kb = kb0; kb < kb1; ++kb) {
            if (!warp_wait(&st.full[stage], phase)) {
                st.abort = 1;
                set_status(p.status, aboleth::Status::Timeout, 0x3720 + stage);
                break;
            }
            tc_fence_after();
            const std::uint32_t s = smem_u32(tiles + stage * G::kStageStride);
            const std::uint64_t dx = smem_desc_sw128(s), dy = smem_desc_sw128(s + G::kBytesX);
            if (elected) {
                if constexpr (G::kMx) {
                    mx::sf_copy(tmem + G::kSfxCol, mx::sf_desc(s + G::kOffSf));
#pragma unroll
                    for (int h = 0; h < G::kAtomsY; ++h)
                        mx::sf_copy(tmem + G::kSfyCol + 4 * h, mx::sf_desc(s + G::kOffSf + (1 + h) * mx::kAtomBytes));
                }
#pragma unroll
                for (unsigned k = 0; k < 4; ++k) {  // four MMAs per stage, 32 bytes of K each
                    const bool more = kb != kb0 || k != 0;
                    if constexpr (G::kMx)
                        mx::umma_mx(tmem, dx + 2 * k, dy + 2 * k, mx::idesc_mx(BM, NT, k), tmem + G::kSfxCol,
                                    tmem + G::kSfyCol, more);
                    else
                        umma<Op>(tmem, dx + 2 * k, dy + 2 * k, Op::idesc(BM, NT), more);
                }
                umma_commit(&st.empty[stage]);
            }
            __syncwarp();
            if (++stage == G::kStages) {
                stage = 0;
                phase ^= 1;
            }
        }
        if (elected)
            umma_commit(&st.done);
        __syncwarp();
    } else {
        // TMEM lane = weight row, column = token: the partial tile goes to shared memory as [token][weight row],
        // over the stages, which every MMA has read by now.
        if (!warp_wait(&st.done, 0)) {
            st.abort = 1;
            set_status(p.status, aboleth::Status::Timeout, 0x3740);
        } else {
            tc_fence_after();
            const int quarter = warp & 3;
            float *out = reinterpret_cast<float *>(tiles) + quarter * 32 + lane;
            const int live = min(NT, p.m - y0);
#pragma unroll 1
            for (int c = 0; c < NT && c < live; c += 32) {
                float v[32];
                tmem_ld32(tmem + (static_cast<std::uint32_t>(quarter * 32) << 16) + c, v);
#pragma unroll
                for (int i = 0; i < 32; ++i)
                    out[(c + i) * BM] = v[i];
            }
            tc_fence_before();
        }
    }
    __syncwarp();
    if (warp_aborted(st.abort)) {
        // Let copies that are still in flight land before the shared memory is handed on.
        const std::uint64_t t0 = aboleth::detail::globaltimer_ns();
        while (aboleth::detail::globaltimer_ns() - t0 < 2000000ull)
            __nanosleep(1000);
    }
    __syncthreads();
    if (p.split > 1)
        cluster_sync();
    // Each CTA sums and stores its share of the tokens, eight weight rows (16 bytes of C) per thread.
    const int tokens = min(NT, p.m - y0);
    const int t_begin = tokens * static_cast<int>(rank) / p.split;
    const int t_end = tokens * (static_cast<int>(rank) + 1) / p.split;
    const std::uint32_t base = smem_u32(tiles);
    for (int i = t_begin * 16 + threadIdx.x; i < t_end * 16; i += kThreads) {
        const int y = i >> 4, x = (i & 15) * 8;
        if (x0 + x >= p.n)
            continue;
        const std::uint32_t at = (y * BM + x) * 4;
        float v[8] = {};
        for (int r = 0; r < p.split; ++r) {
            const float4 a = p.split > 1 ? ld_cluster(base + at, r) : *reinterpret_cast<const float4 *>(tiles + at);
            const float4 b = p.split > 1 ? ld_cluster(base + at + 16, r)
                                         : *reinterpret_cast<const float4 *>(tiles + at + 16);
            v[0] += a.x, v[1] += a.y, v[2] += a.z, v[3] += a.w;
            v[4] += b.x, v[5] += b.y, v[6] += b.z, v[7] += b.w;
        }
#pragma unroll
        for (int j = 0; j < 8; ++j)
            v[j] *= p.alpha;
        *reinterpret_cast<uint4 *>(p.c + static_cast<std::size_t>(y0 + y) * p.ldc + x0 + x) = pack8_bf16(v);
    }
    tc_fence_before();
    __syncthreads();
    if (p.split > 1)
        cluster_sync();  // no CTA leaves while another still reads its partial tile
    tc_fence_after();
    if (warp == 1)
        tmem_dealloc(tmem, G::kCols);
}

}  // namespace ab::gemm::split
