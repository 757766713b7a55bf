// Plain and grouped (per-expert) bf16 GEMM on tcgen05 / TMEM / TMA.
//
//   plain  : C[M, N] = A[M, K] * B[N, K]^T
//   grouped: for each expert e with rows [offsets[e], offsets[e] + counts[e]) of A:
//            C[rows, :] = A[rows, :] * W[e][N, K]^T
//
// The grouped form is the expert stage between EP dispatch and combine: A is
// the expert-contiguous activation matrix the permute kernel builds, counts and
// offsets stay on the device (no host round trip), and a CTA finds its tiles by
// walking the expert list.  The reference has no GEMM; the baseline for these
// kernels is cuBLAS through torch.matmul.
#include <algorithm>
#include <atomic>
#include <cstdlib>

#include "gemm_mx_pair_sm100.cuh"
#include "gemm_mx_sm100.cuh"
#include "gemm_pair_sm100.cuh"
#include "gemm_split_sm100.cuh"

namespace {

using namespace ab::gemm;

template <int NT>
struct PlainPolicy {
    static constexpr bool kBackground = false, kDrainedHook = false, kScaled = true, kSwiGlu = false, kNarrowA = false;
    __nv_bfloat16 *c;
    int m, n, k, ldc;
    int tiles_n, tiles_total;
    int group_n;  // tile columns per raster group: their B panels stay resident in L2
    int bk;       // elements of K per stage (64 for bf16, 128 for e4m3)
    float alpha;  // factor applied to the accumulator before rounding

    // Tiles are visited group by group: all row tiles of `group_n` tile columns
    // before the next group, column fastest inside a group.  B panels of one group
    // (group_n * 256 * K * 2 bytes) fit the L2, A streams once per group.
    __device__ __forceinline__ bool next(int it, Tile &t) const {
        constexpr int rows = pair::PairGeometry<NT>::kTileRows;
        const int idx = blockIdx.x / 2 + it * (gridDim.x / 2);  // two CTAs share a tile
        if (idx >= tiles_total)
            return false;
        const int tiles_m = tiles_total / tiles_n;
        const int per_group = group_n * tiles_m;
        const int group = idx / per_group;
        const int width = min(group_n, tiles_n - group * group_n);
        const int local = idx - group * per_group;
        const int tm = local / width, tn = group * group_n + (local - tm * width);
        t.a_row = tm * rows;
        t.b_row = tn * NT;
        t.k_blocks = (k + bk - 1) / bk;
        t.c_row = tm * rows;
        t.c_col = tn * NT;
        t.rows_valid = min(rows, m - tm * rows);
        t.cols_valid = min(NT, n - tn * NT);
        t.tag = 0;
        t.a_sel = 0;
        return true;
    }
    __device__ __forceinline__ bool ready(const Tile &) const { return true; }
    __device__ __forceinline__ void store16(const Tile &t, int row, int col, const uint4 &v) const {
        *reinterpret_cast<uint4 *>(c + static_cast<std::size_t>(t.c_row + row) * ldc + t.c_col + col) = v;
    }
    __device__ __forceinline__ void tile_done(const Tile &) const {}
    __device__ __forceinline__ void finish(int, int, unsigned long long *) const {}
};

// SWIGLU: an expert's weights are [2 * n, k], gate rows first; a tile multiplies 128 gate rows and the 128 up
// rows of the same output columns, and `n` counts output columns.
// CTAS: 1, or 2 for the pair loop (a worker is a CTA pair and a tile has 256 rows).
template <int CTAS, bool SWIGLU>
struct GroupedPolicy {
    static constexpr int kRows = BM * CTAS, kCols = SWIGLU ? BN / 2 : BN;
    static constexpr bool kBackground = false, kDrainedHook = false, kScaled = false;
    static constexpr bool kSwiGlu = SWIGLU, kNarrowA = CTAS == 1;
    __nv_bfloat16 *c;
    const int *counts, *offsets;
    int experts, n, k, ldc, tiles_n;
    int group_n;  // tile columns per raster group (their weight panels stay in L2)
    // cursor (per thread): expert `e` starts at linear tile `base`
    int e, base;

    // Inside one expert the tiles are visited like the plain GEMM's: all row tiles of
    // `group_n` tile columns before the next group, column fastest, so an expert's weight
    // panels are read from DRAM once however many row tiles it has.
    __device__ __forceinline__ bool next(int it, Tile &t) {
        const int idx = blockIdx.x / CTAS + it * (gridDim.x / CTAS);
        int tiles_m = 0;
        while (e < experts) {
            tiles_m = (counts[e] + kRows - 1) / kRows;
            const int tiles_e = tiles_m * tiles_n;
            if (idx < base + tiles_e)
                break;
            base += tiles_e;
            ++e;
        }
        if (e >= experts)
            return false;
        const int local = idx - base;
        const int per_group = group_n * tiles_m;
        const int group = local / per_group;
        const int width = min(group_n, tiles_n - group * group_n);
        const int in_group = local - group * per_group;
        const int tm = in_group / width, tn = group * group_n + (in_group - tm * width);
        const int row0 = offsets[e] + tm * kRows;
        t.a_row = row0;
        t.b_row = e * (SWIGLU ? 2 * n : n) + tn * kCols;
        t.b_row2 = t.b_row + n;
        t.k_blocks = (k + BK - 1) / BK;
        t.c_row = row0;
        t.c_col = tn * kCols;
        t.rows_valid = min(kRows, counts[e] - tm * kRows);
        t.cols_valid = min(kCols, n - tn * kCols);
        t.tag = e;
        t.a_sel = 0;
        return true;
    }
    __device__ __forceinline__ bool ready(const Tile &) const { return true; }
    __device__ __forceinline__ void store16(const Tile &t, int row, int col, const uint4 &v) const {
        *reinterpret_cast<uint4 *>(c + static_cast<std::size_t>(t.c_row + row) * ldc + t.c_col + col) = v;
    }
    __device__ __forceinline__ void tile_done(const Tile &) const {}
    __device__ __forceinline__ void finish(int, int, unsigned long long *) const {}
};

template <typename Policy>
__global__ void __launch_bounds__(kThreads, 1)
gemm_tcgen05_kernel(const __grid_constant__ CUtensorMap map_a,
                    const __grid_constant__ CUtensorMap map_b, Policy params,
                    unsigned long long *status) {
    Policy policy = params;
    gemm_mainloop<1>(policy, &map_a, &map_b, status);
}

template <typename Op, int NT, typename Policy>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kThreads, 1)
gemm_pair_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
                 Policy params, unsigned long long *status) {
    Policy policy = params;
    pair::gemm_mainloop_pair<Op, NT>(policy, &map_a, &map_b, status);
}

int sm_count() {
    static int sms = 0;
    if (sms == 0) {
        int device = 0;
        cudaGetDevice(&device);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
    }
    return sms;
}

// How many 2-CTA clusters of `kernel` the device can hold at the same time.
template <typename Kernel>
int resident_pairs(Kernel kernel, unsigned smem_bytes) {
    cudaLaunchConfig_t config{};
    config.gridDim = dim3(2 * sm_count());
    config.blockDim = dim3(kThreads);
    config.dynamicSmemBytes = smem_bytes;
    cudaLaunchAttribute attribute{};
    attribute.id = cudaLaunchAttributeClusterDimension;
    attribute.val.clusterDim.x = 2;
    attribute.val.clusterDim.y = 1;
    attribute.val.clusterDim.z = 1;
    config.attrs = &attribute;
    config.numAttrs = 1;
    int clusters = 0;
    if (cudaOccupancyMaxActiveClusters(&clusters, kernel, &config) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    return clusters;
}

template <typename Kernel>
bool configure(Kernel kernel, unsigned smem_bytes) {
    return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_bytes) ==
           cudaSuccess;
}

template <int CTAS, bool SWIGLU>
int launch_grouped(const void *a, const void *w, void *c, const int *counts, const int *offsets,
                   int experts, int total_rows, int n, int k, unsigned long long *status,
                   cudaStream_t stream) {
    using Policy = GroupedPolicy<CTAS, SWIGLU>;
    CUtensorMap map_a, map_b;
    const std::uint64_t w_rows = static_cast<std::uint64_t>(experts) * n * (SWIGLU ? 2 : 1);
    if (!make_map_bf16(&map_a, a, total_rows, k, k, Policy::kNarrowA ? kNarrowRows : BM) ||
        !make_map_bf16(&map_b, w, w_rows, k, k, SWIGLU || CTAS == 2 ? BN / 2 : BN))
        return -2;
    const int tiles_n = (n + Policy::kCols - 1) / Policy::kCols;
    const long long column_bytes = static_cast<long long>(BN) * k * 2;
    const int group_n = static_cast<int>(std::max(1LL, std::min<long long>(tiles_n, (48LL << 20) / column_bytes)));
    Policy p{static_cast<__nv_bfloat16 *>(c), counts, offsets, experts, n, k, n, tiles_n, group_n, 0, 0};
    // The tile count depends on counts the host never reads: a persistent grid that fills the device.
    if constexpr (CTAS == 2) {
        using G = pair::PairGeometry<BN>;
        auto kernel = gemm_pair_kernel<OpBf16, BN, Policy>;
        if (!configure(kernel, G::kSmemBytes))  // per device context: set on every call
            return -3;
        static const int resident = resident_pairs(kernel, G::kSmemBytes);
        if (resident < 1)
            return -3;
        kernel<<<2 * resident, kThreads, G::kSmemBytes, stream>>>(map_a, map_b, p, status);
    } else {
        auto kernel = gemm_tcgen05_kernel<Policy>;
        if (!configure(kernel, Geometry<1>::kSmemBytes))
            return -3;
        kernel<<<sm_count(), kThreads, Geometry<1>::kSmemBytes, stream>>>(map_a, map_b, p, status);
    }
    return ab::launch_result("grouped_gemm_bf16");
}

// Block-scaled e4m3 GEMM: the plain policy's raster order over 128 x 256 tiles of one CTA (gemm_mx_sm100.cuh)
// or 256 x 256 tiles of a pair.
template <int CTAS>
struct MxPolicy {
    static constexpr bool kBackground = false, kDrainedHook = false, kScaled = false, kSwiGlu = false, kNarrowA = false;
    __nv_bfloat16 *c;
    int m, n, k, ldc;
    int tiles_n, tiles_total, group_n;

    __device__ __forceinline__ bool next(int it, Tile &t) const {
        constexpr int rows = BM * CTAS, cols = BN;
        const int idx = blockIdx.x / CTAS + it * (gridDim.x / CTAS);
        if (idx >= tiles_total)
            return false;
        const int tiles_m = tiles_total / tiles_n;
        const int per_group = group_n * tiles_m;
        const int group = idx / per_group;
        const int width = min(group_n, tiles_n - group * group_n);
        const int local = idx - group * per_group;
        const int tm = local / width, tn = group * group_n + (local - tm * width);
        t.a_row = tm * rows;
        t.b_row = tn * cols;
        t.k_blocks = k / mx::kBlockK;
        t.c_row = tm * rows;
        t.c_col = tn * cols;
        t.rows_valid = min(rows, m - tm * rows);
        t.cols_valid = min(cols, n - tn * cols);
        t.tag = 0;
        t.a_sel = 0;
        return true;
    }
    __device__ __forceinline__ bool ready(const Tile &) const { return true; }
    __device__ __forceinline__ void store16(const Tile &t, int row, int col, const uint4 &v) const {
        *reinterpret_cast<uint4 *>(c + static_cast<std::size_t>(t.c_row + row) * ldc + t.c_col + col) = v;
    }
    __device__ __forceinline__ void tile_done(const Tile &) const {}
    __device__ __forceinline__ void finish(int, int, unsigned long long *) const {}
};

// Grouped block-scaled GEMM: GroupedPolicy's tile order with the block-scaled loop's tile shape.  An
// expert's rows must start on a multiple of 128 (a scale-factor atom covers 128 rows); a start that does
// not is reported as Malformed and ends the CTA's work.
// SWIGLU: an expert's weights are [2 * n, k], gate rows first, and a tile's 128 output columns leave as e4m3
// (row stride `ldc` bytes) with their scales in `packed`, the atoms of an A operand of n columns.
template <int CTAS, bool SWIGLU>
struct GroupedMxPolicy {
    static constexpr int kRows = BM * CTAS, kCols = SWIGLU ? BN / 2 : BN;
    static constexpr bool kBackground = false, kDrainedHook = false, kScaled = false;
    static constexpr bool kSwiGlu = SWIGLU, kNarrowA = CTAS == 1;
    std::uint8_t *c;
    std::uint32_t *packed;
    const int *counts, *offsets;
    unsigned long long *status;
    int experts, n, k;
    long long ldc;   // bytes
    int tiles_n;
    int group_n;
    float amax_floor;
    int e, base;   // cursor (per thread): expert `e` starts at linear tile `base`

    __device__ __forceinline__ bool next(int it, Tile &t) {
        const int idx = blockIdx.x / CTAS + it * (gridDim.x / CTAS);
        int tiles_m = 0;
        while (e < experts) {
            tiles_m = (counts[e] + kRows - 1) / kRows;
            const int tiles_e = tiles_m * tiles_n;
            if (idx < base + tiles_e)
                break;
            base += tiles_e;
            ++e;
        }
        if (e >= experts)
            return false;
        if (offsets[e] & (BM - 1)) {
            ab::set_status(status, aboleth::Status::Malformed, 0x3600 + e);
            return false;
        }
        const int local = idx - base;
        const int per_group = group_n * tiles_m;
        const int group = local / per_group;
        const int width = min(group_n, tiles_n - group * group_n);
        const int in_group = local - group * per_group;
        const int tm = in_group / width, tn = group * group_n + (in_group - tm * width);
        const int row0 = offsets[e] + tm * kRows;
        t.a_row = row0;
        t.b_row = e * (SWIGLU ? 2 * n : n) + tn * kCols;
        t.b_row2 = t.b_row + n;
        t.k_blocks = k / mx::kBlockK;
        t.c_row = row0;
        t.c_col = tn * kCols;
        t.rows_valid = min(kRows, counts[e] - tm * kRows);
        t.cols_valid = min(kCols, n - tn * kCols);
        t.tag = e;
        t.a_sel = 0;
        return true;
    }
    __device__ __forceinline__ bool ready(const Tile &) const { return true; }
    // `col` counts output elements: bf16, or e4m3 with SWIGLU.
    __device__ __forceinline__ void store16(const Tile &t, int row, int col, const uint4 &v) const {
        *reinterpret_cast<uint4 *>(c + (t.c_row + row) * ldc + (t.c_col + col) * (SWIGLU ? 1 : 2)) = v;
    }
    __device__ __forceinline__ void store_scale(const Tile &t, int row, std::uint32_t word) const {
        const int r = t.c_row + row;
        const std::size_t atom = static_cast<std::size_t>(r / BM) * (n / 128) + t.c_col / 128;
        packed[atom * 128 + (r % 32) * 4 + (r % BM) / 32] = word;
    }
    __device__ __forceinline__ void tile_done(const Tile &) const {}
    __device__ __forceinline__ void finish(int, int, unsigned long long *) const {}
};

template <typename Policy>
__global__ void __launch_bounds__(kThreads, 1)
gemm_mx_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
                  Policy params, mx::ScaleFactors sf, unsigned long long *status) {
    Policy policy = params;
    mx::gemm_mx_mainloop<1>(policy, &map_a, &map_b, sf, status);
}

template <typename Policy>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kThreads, 1)
gemm_mx_pair_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
                    const __grid_constant__ CUtensorMap map_sfa, const __grid_constant__ CUtensorMap map_sfb,
                    Policy params, int k_blocks, int granules, unsigned long long *status) {
    Policy policy = params;
    mxpair::gemm_mx_mainloop_pair(policy, mxpair::Maps{&map_a, &map_b, &map_sfa, &map_sfb}, k_blocks, granules,
                                  status);
}

// The exponent byte (ue8m0) of a positive power-of-two fp32; anything else is reported.
__device__ __forceinline__ unsigned ue8m0_of(float scale, unsigned long long *status, unsigned detail) {
    const unsigned bits = __float_as_uint(scale);
    if ((bits & 0x807fffffu) != 0 || (bits >> 23) == 0 || (bits >> 23) == 255)
        ab::set_status(status, aboleth::Status::Malformed, detail);
    return (bits >> 23) & 0xffu;
}

// Activation scales fp32 [rows, k_blocks] (one per row and 128 K) -> atoms [row block][K block] of 512
// bytes: byte (r % 32) * 16 + (r / 32) * 4 + s for row r of the block, the same value for s = 0..3.
__global__ void pack_scales_a_kernel(const float *scales, long long ld, std::uint32_t *out, int rows,
                                     int k_blocks, unsigned long long *status) {
    const long long row_blocks = mx::mx_row_blocks(rows);
    const long long total = row_blocks * k_blocks * 128;
    for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < total;
         i += static_cast<long long>(gridDim.x) * blockDim.x) {
        const int r = static_cast<int>(i % 128);
        const long long atom = i / 128;           // row_block * k_blocks + kb
        const int kb = static_cast<int>(atom % k_blocks);
        const int row = static_cast<int>(atom / k_blocks) * 128 + r;
        const unsigned e = row < rows ? ue8m0_of(scales[row * ld + kb], status, 0x3500) : 127u;
        out[atom * 128 + (r % 32) * 4 + r / 32] = e * 0x01010101u;
    }
}

// Weight scales fp32 [n_blocks, k_blocks] (one per 128 x 128 block) -> atoms [K block][granule]: atom g
// holds the scales of columns [64 g, 64 g + 128), so that a tile whose first column is any multiple of 64
// (256- and 192-column tiles both) finds its two atoms at g and g + 2.  `granules` per K block.
__global__ void pack_scales_b_kernel(const float *scales, long long ld, std::uint32_t *out, int n_blocks,
                                     int granules, int k_blocks, unsigned long long *status) {
    const long long total = static_cast<long long>(k_blocks) * granules * 128;
    for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < total;
         i += static_cast<long long>(gridDim.x) * blockDim.x) {
        const long long atom = i / 128;           // kb * granules + g
        const int w = static_cast<int>(i % 128);  // word of the atom: row (w / 4) + 32 * (w % 4)
        const int g = static_cast<int>(atom % granules);
        const int kb = static_cast<int>(atom / granules);
        const int nb = (64 * g + (w >> 2) + 32 * (w & 3)) >> 7;
        const unsigned e = nb < n_blocks ? ue8m0_of(scales[nb * ld + kb], status, 0x3501) : 127u;
        out[i] = e * 0x01010101u;
    }
}

using mx::mx_granules;
using mx::mx_row_blocks;

// Operand kinds of the dense products.
enum Kind { kKindBf16 = 0, kKindE4m3 = 1, kKindMx = 2 };

struct DenseArgs {
    const void *a, *b;
    void *c;
    const void *sfa, *sfb;
    int m, n, k, lda, ldb, ldc;
    float alpha;
    unsigned long long *status;
};

template <typename Op, int NT>
int launch_split(const DenseArgs &d, int split, cudaStream_t stream) {
    using G = split::SplitGeometry<Op, NT>;
    auto kernel = split::gemm_split_kernel<Op, NT>;
    CUtensorMap map_x, map_y;
    const bool mapped = G::kBK == 64
        ? make_map_bf16(&map_x, d.b, d.n, d.k, d.ldb, BM) && make_map_bf16(&map_y, d.a, d.m, d.k, d.lda, NT)
        : make_map_e4m3(&map_x, d.b, d.n, d.k, d.ldb, BM) && make_map_e4m3(&map_y, d.a, d.m, d.k, d.lda, NT);
    if (!mapped)
        return -2;
    if (!configure(kernel, G::kSmemBytes))
        return -3;
    split::SplitParams p{};
    p.c = static_cast<__nv_bfloat16 *>(d.c);
    p.m = d.m, p.n = d.n, p.ldc = d.ldc;
    p.k_blocks = (d.k + G::kBK - 1) / G::kBK;
    p.tiles_y = (d.m + NT - 1) / NT;
    p.split = std::max(1, std::min(std::min(split, split::kMaxSplit), p.k_blocks));
    p.alpha = d.alpha;
    p.sf_x = static_cast<const std::uint8_t *>(d.sfb);
    p.sf_y = static_cast<const std::uint8_t *>(d.sfa);
    p.granules = mx_granules(d.n);
    p.status = d.status;
    cudaLaunchConfig_t config{};
    config.gridDim = dim3(static_cast<unsigned>(p.tiles_y) * ((d.n + BM - 1) / BM) * p.split);
    config.blockDim = dim3(kThreads);
    config.dynamicSmemBytes = G::kSmemBytes;
    config.stream = stream;
    cudaLaunchAttribute attribute{};
    attribute.id = cudaLaunchAttributeClusterDimension;
    attribute.val.clusterDim.x = p.split;
    attribute.val.clusterDim.y = 1;
    attribute.val.clusterDim.z = 1;
    config.attrs = &attribute;
    config.numAttrs = 1;
    const cudaError_t e = cudaLaunchKernelEx(&config, kernel, map_x, map_y, p);
    if (e != cudaSuccess) {
        cudaGetLastError();
        fprintf(stderr, "aboleth_b200: gemm (split K) launch failed: %s\n", cudaGetErrorString(e));
        return static_cast<int>(e);
    }
    return 0;
}

// How many CTAs of the split kernel, in clusters of `split`, the device holds at once (a cluster stays inside one
// GPC, so not every size fills every SM).  Asked once.
template <typename Op, int NT>
int split_slots_of(int split) {
    using G = split::SplitGeometry<Op, NT>;
    static std::atomic<int> known[split::kMaxSplit + 1];
    int slots = known[split].load(std::memory_order_relaxed);
    if (slots == 0) {
        auto kernel = split::gemm_split_kernel<Op, NT>;
        cudaLaunchConfig_t config{};
        config.gridDim = dim3(4u * sm_count() / split * split);
        config.blockDim = dim3(kThreads);
        config.dynamicSmemBytes = G::kSmemBytes;
        cudaLaunchAttribute attribute{};
        attribute.id = cudaLaunchAttributeClusterDimension;
        attribute.val.clusterDim.x = split;
        attribute.val.clusterDim.y = attribute.val.clusterDim.z = 1;
        config.attrs = &attribute;
        config.numAttrs = 1;
        int clusters = 0;
        if (!configure(kernel, G::kSmemBytes) ||
            cudaOccupancyMaxActiveClusters(&clusters, kernel, &config) != cudaSuccess || clusters < 1) {
            cudaGetLastError();
            return sm_count();
        }
        slots = clusters * split;
        known[split].store(slots, std::memory_order_relaxed);
    }
    return slots;
}

template <typename Op>
int split_slots(int nt, int split) {
    switch (nt) {
    case 32: return split_slots_of<Op, 32>(split);
    case 64: return split_slots_of<Op, 64>(split);
    case 128: return split_slots_of<Op, 128>(split);
    default: return split_slots_of<Op, 256>(split);
    }
}

// The persistent pair loop over 256 x NT tiles.
template <typename Op, int NT>
int launch_pair(const DenseArgs &d, cudaStream_t stream) {
    using G = pair::PairGeometry<NT>;
    auto kernel = gemm_pair_kernel<Op, NT, PlainPolicy<NT>>;
    CUtensorMap map_a, map_b;
    // Each CTA of a pair loads 128 rows of A and NT / 2 rows of B per K step.
    const bool mapped = Op::kBK == 64
        ? make_map_bf16(&map_a, d.a, d.m, d.k, d.lda, BM) && make_map_bf16(&map_b, d.b, d.n, d.k, d.ldb, NT / 2)
        : make_map_e4m3(&map_a, d.a, d.m, d.k, d.lda, BM) && make_map_e4m3(&map_b, d.b, d.n, d.k, d.ldb, NT / 2);
    if (!mapped)
        return -2;
    if (!configure(kernel, G::kSmemBytes))  // per device context: set on every call
        return -3;
    // A persistent kernel must not launch more clusters than can be resident at once: the
    // surplus would start only after a resident one has finished all of its tiles.
    static const int resident = resident_pairs(kernel, G::kSmemBytes);
    if (resident < 1)
        return -3;
    const int tiles_n = (d.n + NT - 1) / NT;
    const int tiles = (d.m + G::kTileRows - 1) / G::kTileRows * tiles_n;
    // About 48 MiB of B per raster group.
    const long long column_bytes = static_cast<long long>(NT) * d.k * (Op::kBK == 64 ? 2 : 1);
    const int group_n = static_cast<int>(std::max(1LL, std::min<long long>(tiles_n, (48LL << 20) / column_bytes)));
    const PlainPolicy<NT> p{static_cast<__nv_bfloat16 *>(d.c), d.m, d.n, d.k, d.ldc, tiles_n, tiles, group_n, Op::kBK,
                        d.alpha};
    kernel<<<2 * std::min(tiles, resident), kThreads, G::kSmemBytes, stream>>>(map_a, map_b, p, d.status);
    return ab::launch_result(Op::kBK == 64 ? "gemm_bf16 (CTA pairs)" : "gemm_e4m3 (CTA pairs)");
}

template <typename Op>
int launch_split_nt(const DenseArgs &d, int nt, int split, cudaStream_t stream) {
    switch (nt) {
    case 32: return launch_split<Op, 32>(d, split, stream);
    case 64: return launch_split<Op, 64>(d, split, stream);
    case 128: return launch_split<Op, 128>(d, split, stream);
    case 256: return launch_split<Op, 256>(d, split, stream);
    default: return -1;
    }
}

}  // namespace

// The dense products with an explicit token tile (32, 64, 128 or 256; the block-scaled kind takes 32 and 64 only
// for as many tokens) and K split (1 to 8), for tests and tuning; `kind`: 0 bf16, 1 e4m3, 2 block-scaled.
AB_EXPORT int ab_gemm_split(int kind, const void *a, const void *b, void *c, const void *sfa, const void *sfb, int m,
                            int n, int k, int lda, int ldb, int ldc, float alpha, int nt, int split,
                            unsigned long long *status, cudaStream_t stream) {
    const int unit = kind == kKindBf16 ? 8 : 16;
    if (kind < kKindBf16 || kind > kKindMx || m < 1 || n < 1 || k < 1 || k % unit || lda % unit || ldb % unit ||
        ldc % 8 || split < 1 || split > split::kMaxSplit ||
        ((reinterpret_cast<std::uintptr_t>(a) | reinterpret_cast<std::uintptr_t>(b) |
          reinterpret_cast<std::uintptr_t>(c)) & 15))
        return -1;
    const DenseArgs d{a, b, c, sfa, sfb, m, n, k, lda, ldb, ldc, alpha, status};
    if (kind == kKindBf16)
        return launch_split_nt<OpBf16>(d, nt, split, stream);
    if (kind == kKindE4m3)
        return launch_split_nt<OpE4m3>(d, nt, split, stream);
    if (k % 128 || sfa == nullptr || sfb == nullptr || (nt < 128 && m > nt))
        return -1;
    return launch_split_nt<split::OpMx>(d, nt, split, stream);
}

namespace {

// Which kernel computes a dense product.  Times in us, fitted to B200 measurements of 47 shapes (1 to 8192
// rows, 256 to 8192 columns, K 256 to 8192) with every token tile and split, inputs of three sets in turn; the
// rule's choice is 3 % slower than the best one on average.
//   split kernel: launch, tile prologue and reduction, plus 128-byte K steps that take `lone` on an SM of
//     their own and `packed` beside a second CTA; at least what the slowest of the memory system needs
//     (6.3 GB/ms from memory, 19.8 GB/ms from L2 to the SMs).
//   pair loop: 4.6 + waves of resident pairs x (0.297 per K step + 0.45); 0.268 with 224 columns a tile, which wins
//     where it needs no more waves (8192 x 3584 x 8192: 7 waves either way, 339 us against 449; 8192^3: 16 waves
//     against 14, 860 and 842).
//   block-scaled: persistent 128 x 256 tiles of one CTA, 4.2 + waves x (0.30 per K step + 1), or of a pair,
//     5.4 + waves x (0.315 + 1), and 12.3 GB/ms of tile traffic (50 and 68 KB per tile and step).
// Back to back, launches included.  bf16: 32 x 3584 x 8192 split 17.3 us (pair loop 39.4); 1000 x 3584 x 8192 pair loop
// 51 (256 columns 61, split 67).  Block-scaled: 32 x 3584 x 8192 split 12.3 us (one CTA 28.7); 1000 x 8192 x 3584 pair
// loop 32.8 (one CTA 34.8); 8192^3 pair loop 452 (one CTA 499); 500 x 8192 x 512 one CTA 9.2 (pair 10.1).
struct DenseChoice {
    int nt, split;   // nt <= 0: a persistent loop, of `split` CTAs per tile (-1: with 224 columns a tile)
};

// What an environment variable asks for, or -1.
int asked(const char *name) {
    const char *v = std::getenv(name);
    return v == nullptr || *v == 0 ? -1 : std::atoi(v);
}

// ABOLETH_GEMM_PAIR: 0 = no CTA pairs (the split kernel), 1 = CTA pairs with 256 x 256 tiles, 2 = with 256 x 224
// tiles, for bf16 and per-tensor e4m3.
// ABOLETH_GEMM_MX_TILE: 1 = 128 x 256 tiles of one CTA, 2 = 256 x 256 tiles of a pair, for block-scaled e4m3.
template <typename Op>
DenseChoice choose_dense(int m, int n, int k_blocks, int kind) {
    const int forced = asked(kind == kKindMx ? "ABOLETH_GEMM_MX_TILE" : "ABOLETH_GEMM_PAIR");
    struct Row { int nt; double lone, packed; };
    static const Row kDense[4] = {{32, .213, .278}, {64, .251, .365}, {128, .278, .482}, {256, .336, .336}};
    static const Row kScaled[4] = {{32, .263, .586}, {64, .473, .473}, {128, .324, .564}, {256, .306, .306}};
    const Row *rows = kind == kKindMx ? kScaled : kDense;
    const double k_bytes = 128.0 * k_blocks;
    const double memory = ((static_cast<double>(m) + n) * k_bytes + 2.0 * m * n) / 6.3e6;
    const int sms = sm_count();
    DenseChoice best{0, 2};
    const long long pair_tiles = static_cast<long long>((m + 255) / 256) * ((n + 255) / 256);
    const double pair_waves = static_cast<double>((pair_tiles + sms / 2 - 1) / (sms / 2));
    double best_us = 4.6 + pair_waves * (0.297 * k_blocks + 0.45);
    if (kind != kKindMx) {
        const long long narrow = static_cast<long long>((m + 255) / 256) * ((n + 223) / 224);
        const double us = 4.6 + static_cast<double>((narrow + sms / 2 - 1) / (sms / 2)) * (0.268 * k_blocks + 0.45);
        if (us < best_us) {
            best_us = us;
            best = DenseChoice{-1, 2};
        }
    }
    if (kind == kKindMx) {
        best_us = std::max(5.4 + pair_waves * (0.315 * k_blocks + 1.0), 5.0 + pair_tiles * k_blocks * 68e3 / 12.3e6);
        const long long tiles = static_cast<long long>((m + 127) / 128) * ((n + 255) / 256);
        const double waves = static_cast<double>((tiles + sms - 1) / sms);
        const double one = std::max(4.2 + waves * (0.30 * k_blocks + 1.0), 4.2 + tiles * k_blocks * 50e3 / 12.3e6);
        if (one < best_us) {
            best_us = one;
            best = DenseChoice{0, 1};
        }
        if (forced > 0)
            return DenseChoice{0, forced == 1 ? 1 : 2};
    } else if (forced > 0) {
        return DenseChoice{forced == 1 ? 0 : -1, 2};
    } else if (forced == 0) {
        best_us = 1e30;
    }
    for (int i = 0; i < 4; ++i) {
        const int nt = rows[i].nt;
        if (nt > 32 && nt >= 2 * m)
            break;  // a tile that is mostly padding
        if (kind == kKindMx && nt < 128 && m > nt)
            continue;  // a scale atom covers 128 tokens
        const long long tiles = static_cast<long long>((m + nt - 1) / nt) * ((n + BM - 1) / BM);
        for (int split : {1, 2, 3, 4, 8}) {
            const long long ctas = tiles * split;
            if (split > k_blocks)
                break;
            const int slots = split_slots<Op>(nt, split);
            if ((split > 1 && ctas > slots) || (split == 8 && ctas > sms - 20))
                break;  // cutting K of a grid that already fills the device only adds reductions
            const long long full = ctas / slots, rest = ctas - full * slots;
            const double steps = (k_blocks + split - 1) / split, each = 2.1 + 2.8 * nt / 128;
            double us = 0.6 + (split > 1 ? 1.0 + 1.9 * nt / 128 * (split - 1) / split : 0.0) +
                        full * (steps * rows[i].packed + each);
            if (rest > 0)
                us += steps * (rest <= sms ? rows[i].lone : rows[i].packed) + each;
            us = std::max(us, 4.2 + std::max(memory, tiles * (128.0 + nt) * k_bytes / 19.8e6));
            if (us < best_us) {
                best_us = us;
                best = DenseChoice{nt, split};
            }
        }
    }
    return best;
}

}  // namespace

// Which kernel a dense product of this size takes: choice[0] > 0 - the split kernel with that token tile and K in
// choice[1] parts; 0 or -1 - a persistent loop over tiles of choice[1] CTAs, 256 or 224 columns wide.
AB_EXPORT int ab_gemm_choice(int kind, int m, int n, int k, int *choice) {
    if (kind < kKindBf16 || kind > kKindMx || m < 1 || n < 1 || k < 1 || choice == nullptr)
        return -1;
    const int k_blocks = kind == kKindBf16 ? (k + 63) / 64 : (k + 127) / 128;
    const DenseChoice c = kind == kKindBf16 ? choose_dense<OpBf16>(m, n, k_blocks, kind)
                          : kind == kKindE4m3 ? choose_dense<OpE4m3>(m, n, k_blocks, kind)
                                              : choose_dense<split::OpMx>(m, n, k_blocks, kind);
    choice[0] = c.nt;
    choice[1] = c.split;
    return 0;
}

namespace {

template <typename Op>
int launch_dense(const DenseArgs &d, int kind, cudaStream_t stream) {
    const DenseChoice choice = choose_dense<Op>(d.m, d.n, (d.k + Op::kBK - 1) / Op::kBK, kind);
    if (choice.nt > 0)
        return launch_split_nt<Op>(d, choice.nt, choice.split, stream);
    return choice.nt == 0 ? launch_pair<Op, BN>(d, stream) : launch_pair<Op, 224>(d, stream);
}

}  // namespace

// C[M,N] = A[M,K] * B[N,K]^T, all bf16 row-major, lda/ldb/ldc in elements.
// K and the leading dimensions must be multiples of 8 (16-byte TMA strides).
AB_EXPORT int ab_gemm_bf16(const void *a, const void *b, void *c, int m, int n, int k, int lda,
                           int ldb, int ldc, unsigned long long *status, cudaStream_t stream) {
    if (m < 1 || n < 1 || k < 1 || k % 8 || lda % 8 || ldb % 8 || ldc % 8 ||
        (reinterpret_cast<std::uintptr_t>(a) | reinterpret_cast<std::uintptr_t>(b) |
         reinterpret_cast<std::uintptr_t>(c)) & 15)
        return -1;
    return launch_dense<OpBf16>(DenseArgs{a, b, c, nullptr, nullptr, m, n, k, lda, ldb, ldc, 1.0f, status}, kKindBf16,
                                stream);
}

// C[M,N] (bf16) = alpha * A[M,K] * B[N,K]^T with A and B in e4m3 (one byte per element), row-major,
// lda/ldb in elements (= bytes), ldc in bf16 elements.  K, lda and ldb must be multiples of 16.
// `alpha` carries the product of the two per-tensor scales.  kind::f8f6f4.
AB_EXPORT int ab_gemm_e4m3(const void *a, const void *b, void *c, int m, int n, int k, int lda, int ldb,
                           int ldc, float alpha, unsigned long long *status, cudaStream_t stream) {
    if (m < 1 || n < 1 || k < 1 || k % 16 || lda % 16 || ldb % 16 || ldc % 8 ||
        (reinterpret_cast<std::uintptr_t>(a) | reinterpret_cast<std::uintptr_t>(b) |
         reinterpret_cast<std::uintptr_t>(c)) & 15)
        return -1;
    return launch_dense<OpE4m3>(DenseArgs{a, b, c, nullptr, nullptr, m, n, k, lda, ldb, ldc, alpha, status}, kKindE4m3,
                                stream);
}

namespace {

// 256-row pair tiles or 128-row tiles of single CTAs.  A pair takes 512 cycles per K step of its tile, a CTA 768
// (it loads 48 KiB, at 64 bytes a cycle), so two CTAs are ahead where one 128-row tile holds an expert's rows and the pair
// where it takes two of them; ragged ends put the line between.  Three 128-row tiles beat two pairs' (257 to 384 rows):
// 8 experts x 320 rows x 4096 x 4096 bf16 102 us against 109, with SwiGLU 113 and 131, block-scaled 69 and 76; 450 rows
// 142 against 126, 148 and 128, 84 and 79.
bool pair_tiles(int total_rows, int experts) {
    const int rows = total_rows / experts;
    return rows >= 192 && (rows <= 256 || rows > 384);
}

bool grouped_ok(const void *a, const void *w, const void *c, int experts, int total_rows, int n, int k) {
    return experts >= 1 && total_rows >= 1 && n >= 1 && k >= 1 && k % 8 == 0 && n % 8 == 0 &&
           ((reinterpret_cast<std::uintptr_t>(a) | reinterpret_cast<std::uintptr_t>(w) |
             reinterpret_cast<std::uintptr_t>(c)) & 15) == 0;
}

}  // namespace

// Whether the grouped products of this size run on CTA pairs.
AB_EXPORT int ab_grouped_pairs(int total_rows, int experts) {
    return total_rows < 1 || experts < 1 ? -1 : pair_tiles(total_rows, experts);
}

// Grouped GEMM over `experts` problems that share N and K.  a: [total_rows, K],
// w: [experts, N, K], c: [total_rows, N]; counts/offsets: device int32 [experts].
AB_EXPORT int ab_grouped_gemm_bf16(const void *a, const void *w, void *c, const int *counts,
                                   const int *offsets, int experts, int total_rows, int n, int k,
                                   unsigned long long *status, cudaStream_t stream) {
    if (!grouped_ok(a, w, c, experts, total_rows, n, k))
        return -1;
    const auto launch = pair_tiles(total_rows, experts) ? launch_grouped<2, false> : launch_grouped<1, false>;
    return launch(a, w, c, counts, offsets, experts, total_rows, n, k, status, stream);
}

// The same over w [experts, 2 N, K], an expert's N gate rows before its N up rows:
// c = silu(a gate^T) * (a up^T), the product taken in fp32 on the accumulators and rounded once.
AB_EXPORT int ab_grouped_gemm_swiglu_bf16(const void *a, const void *w, void *c, const int *counts,
                                          const int *offsets, int experts, int total_rows, int n, int k,
                                          unsigned long long *status, cudaStream_t stream) {
    if (!grouped_ok(a, w, c, experts, total_rows, n, k))
        return -1;
    const auto launch = pair_tiles(total_rows, experts) ? launch_grouped<2, true> : launch_grouped<1, true>;
    return launch(a, w, c, counts, offsets, experts, total_rows, n, k, status, stream);
}

// The persistent pair loop over `policy`'s tiles, at most `tiles` pairs.
template <typename Policy>
int launch_mx_pair(const void *a, const void *sfa, const void *b, const void *sfb, long long a_rows, long long b_rows,
                   int k, int lda, int ldb, const Policy &policy, long long tiles, unsigned long long *status,
                   cudaStream_t stream) {
    using G = mxpair::Geometry;
    auto kernel = gemm_mx_pair_kernel<Policy>;
    const int k_blocks = k / 128, granules = mx_granules(static_cast<int>(b_rows));
    CUtensorMap map_a, map_b, map_sfa, map_sfb;
    if (!make_map_e4m3(&map_a, a, a_rows, k, lda, BM) || !make_map_e4m3(&map_b, b, b_rows, k, ldb, BN / 2) ||
        !make_map_atoms(&map_sfa, sfa, mx_row_blocks(static_cast<int>(a_rows)) * k_blocks) ||
        !make_map_atoms(&map_sfb, sfb, static_cast<std::uint64_t>(k_blocks) * granules))
        return -2;
    if (!configure(kernel, G::kSmemBytes))
        return -3;
    static const int resident = resident_pairs(kernel, G::kSmemBytes);
    if (resident < 1)
        return -3;
    const int pairs = static_cast<int>(std::min<long long>(tiles, resident));
    kernel<<<2 * pairs, kThreads, G::kSmemBytes, stream>>>(map_a, map_b, map_sfa, map_sfb, policy, k_blocks, granules,
                                                           status);
    return ab::launch_result("gemm_e4m3_mx (CTA pairs)");
}

template <int CTAS, bool SWIGLU>
int launch_grouped_mx(const void *a, const void *sfa, const void *w, const void *sfb, void *c, void *packed,
                      float amax_floor, const int *counts, const int *offsets, int experts, int total_rows, int n,
                      int k, unsigned long long *status, cudaStream_t stream) {
    using Policy = GroupedMxPolicy<CTAS, SWIGLU>;
    const long long w_rows = static_cast<long long>(experts) * n * (SWIGLU ? 2 : 1);
    Policy p{static_cast<std::uint8_t *>(c), static_cast<std::uint32_t *>(packed), counts, offsets, status, experts,
             n, k, static_cast<long long>(n) * (SWIGLU ? 1 : 2), (n + Policy::kCols - 1) / Policy::kCols, 1,
             amax_floor, 0, 0};
    const long long column_bytes = static_cast<long long>(BN) * k;
    p.group_n = static_cast<int>(std::max(1LL, std::min<long long>(p.tiles_n, (48LL << 20) / column_bytes)));
    // The tile count depends on counts the host never reads: a persistent grid that fills the device.
    if constexpr (CTAS == 2) {
        return launch_mx_pair(a, sfa, w, sfb, total_rows, w_rows, k, k, k, p, 1 << 20, status, stream);
    } else {
        using G = mx::MxGeometry<1>;
        auto kernel = gemm_mx_kernel<Policy>;
        CUtensorMap map_a, map_b;
        if (!make_map_e4m3(&map_a, a, total_rows, k, k, kNarrowRows) ||
            !make_map_e4m3(&map_b, w, w_rows, k, k, Policy::kCols))
            return -2;
        if (!configure(kernel, G::kSmemBytes))
            return -3;
        const mx::ScaleFactors sf{static_cast<const std::uint8_t *>(sfa), static_cast<const std::uint8_t *>(sfb),
                                  k / 128, mx_granules(static_cast<int>(w_rows))};
        kernel<<<sm_count(), kThreads, G::kSmemBytes, stream>>>(map_a, map_b, p, sf, status);
        return ab::launch_result("grouped_gemm_e4m3_mx");
    }
}

namespace {

bool grouped_mx_ok(const void *a, const void *sfa, const void *w, const void *sfb, const void *c, int experts,
                   int total_rows, int n, int k) {
    return experts >= 1 && total_rows >= 1 && n >= 64 && n % 64 == 0 && k >= 128 && k % 128 == 0 &&
           sfa != nullptr && sfb != nullptr &&
           ((reinterpret_cast<std::uintptr_t>(a) | reinterpret_cast<std::uintptr_t>(w) |
             reinterpret_cast<std::uintptr_t>(c) | reinterpret_cast<std::uintptr_t>(sfa) |
             reinterpret_cast<std::uintptr_t>(sfb)) & 15) == 0;
}

}  // namespace

// Grouped block-scaled GEMM: a [total_rows, K] e4m3 in expert-contiguous order with every expert's first
// row on a multiple of 128, w [experts, N, K] e4m3, N a multiple of 64; `sfa` = ab_mx_pack_scales of the
// [total_rows, K/128] activation scales, `sfb` = of the [experts * N / 128, K/128] weight scales (the
// weights seen as one [experts * N, K] matrix).  c [total_rows, N] bf16.
AB_EXPORT int ab_grouped_gemm_e4m3_mx(const void *a, const void *sfa, const void *w, const void *sfb, void *c,
                                      const int *counts, const int *offsets, int experts, int total_rows,
                                      int n, int k, unsigned long long *status, cudaStream_t stream) {
    if (!grouped_mx_ok(a, sfa, w, sfb, c, experts, total_rows, n, k))
        return -1;
    const auto launch = pair_tiles(total_rows, experts) ? launch_grouped_mx<2, false> : launch_grouped_mx<1, false>;
    return launch(a, sfa, w, sfb, c, nullptr, 0.f, counts, offsets, experts, total_rows, n, k, status, stream);
}

// The gate and up products of a SwiGLU layer, quantised for the product that follows: w [experts, 2 N, K], an
// expert's N gate rows before its N up rows, N a multiple of 128; q [total_rows, N] e4m3 = silu(a gate^T) *
// (a up^T) over a power-of-two scale per row and 128 columns (maximum, at least amax_floor, / 448, rounded
// up), `packed` = the scale atoms of q as the next block-scaled product's A operand (ab_mx_scale_bytes(
// total_rows, ., N, 0) bytes).  Rows outside the experts, and their scales, are not written.
AB_EXPORT int ab_grouped_gemm_swiglu_e4m3_mx(const void *a, const void *sfa, const void *w, const void *sfb, void *q,
                                             void *packed, float amax_floor, const int *counts, const int *offsets,
                                             int experts, int total_rows, int n, int k, unsigned long long *status,
                                             cudaStream_t stream) {
    if (!grouped_mx_ok(a, sfa, w, sfb, q, experts, total_rows, n, k) || n % 128 || packed == nullptr ||
        (reinterpret_cast<std::uintptr_t>(packed) & 15))
        return -1;
    const auto launch = pair_tiles(total_rows, experts) ? launch_grouped_mx<2, true> : launch_grouped_mx<1, true>;
    return launch(a, sfa, w, sfb, q, packed, amax_floor, counts, offsets, experts, total_rows, n, k, status, stream);
}

// Bytes of the packed scale factors of a block-scaled GEMM: A atoms for `m` rows, B atoms for `n` columns.
AB_EXPORT long long ab_mx_scale_bytes(int m, int n, int k, int which) {
    const long long k_blocks = (k + 127) / 128;
    if (which == 0)
        return mx_row_blocks(m) * k_blocks * 512;
    return k_blocks * mx_granules(n) * 512;
}

// fp32 power-of-two scales -> ue8m0 atoms in the order the tensor core reads them.  which = 0: activation
// scales [rows, K/128] (one per row and K block); which = 1: weight scales [ceil(rows/128), K/128].  A scale
// that is not a positive power of two is reported as Malformed in `status` (the product would be wrong).
AB_EXPORT int ab_mx_pack_scales(const float *scales, long long ld, void *out, int rows, int k, int which,
                                unsigned long long *status, cudaStream_t stream) {
    if (scales == nullptr || out == nullptr || rows < 1 || k < 128 || k % 128)
        return -1;
    const int k_blocks = k / 128;
    if (which == 0) {
        pack_scales_a_kernel<<<148, 256, 0, stream>>>(scales, ld, static_cast<std::uint32_t *>(out), rows,
                                                      k_blocks, status);
    } else {
        pack_scales_b_kernel<<<148, 256, 0, stream>>>(scales, ld, static_cast<std::uint32_t *>(out),
                                                      (rows + 127) / 128, mx_granules(rows), k_blocks, status);
    }
    return ab::launch_result("mx_pack_scales");
}

namespace {

// The persistent block-scaled loops: 128 x 256 tiles of one CTA, or 256 x 256 tiles of a pair.
template <int CTAS>
int launch_mx(const DenseArgs &d, cudaStream_t stream) {
    MxPolicy<CTAS> p{};
    p.c = static_cast<__nv_bfloat16 *>(d.c);
    p.m = d.m, p.n = d.n, p.k = d.k, p.ldc = d.ldc;
    p.tiles_n = (d.n + BN - 1) / BN;
    p.tiles_total = (d.m + BM * CTAS - 1) / (BM * CTAS) * p.tiles_n;
    const long long column_bytes = static_cast<long long>(BN) * d.k;
    p.group_n = static_cast<int>(std::max(1LL, std::min<long long>(p.tiles_n, (48LL << 20) / column_bytes)));
    if constexpr (CTAS == 2) {
        return launch_mx_pair(d.a, d.sfa, d.b, d.sfb, d.m, d.n, d.k, d.lda, d.ldb, p, p.tiles_total, d.status, stream);
    } else {
        using G = mx::MxGeometry<1>;
        auto kernel = gemm_mx_kernel<MxPolicy<1>>;
        CUtensorMap map_a, map_b;
        if (!make_map_e4m3(&map_a, d.a, d.m, d.k, d.lda, BM) || !make_map_e4m3(&map_b, d.b, d.n, d.k, d.ldb, BN))
            return -2;
        if (!configure(kernel, G::kSmemBytes))
            return -3;
        const mx::ScaleFactors sf{static_cast<const std::uint8_t *>(d.sfa), static_cast<const std::uint8_t *>(d.sfb),
                                  d.k / 128, mx_granules(d.n)};
        kernel<<<std::min(p.tiles_total, sm_count()), kThreads, G::kSmemBytes, stream>>>(map_a, map_b, p, sf, d.status);
        return ab::launch_result("gemm_e4m3_mx");
    }
}

}  // namespace

// C[M,N] (bf16) = (A * sa) (B * sb)^T for e4m3 A [M,K] and B [N,K] (row-major, lda / ldb in bytes) whose
// scales were packed by ab_mx_pack_scales: tcgen05.mma.kind::mxf8f6f4.block_scale, no expansion pass.
// K must be a multiple of 128.
AB_EXPORT int ab_gemm_e4m3_mx(const void *a, const void *b, void *c, const void *sfa, const void *sfb, int m,
                              int n, int k, int lda, int ldb, int ldc, unsigned long long *status,
                              cudaStream_t stream) {
    if (m < 1 || n < 1 || k < 128 || k % 128 || lda % 16 || ldb % 16 || ldc % 8 || sfa == nullptr ||
        sfb == nullptr ||
        (reinterpret_cast<std::uintptr_t>(a) | reinterpret_cast<std::uintptr_t>(b) |
         reinterpret_cast<std::uintptr_t>(c) | reinterpret_cast<std::uintptr_t>(sfa) |
         reinterpret_cast<std::uintptr_t>(sfb)) & 15)
        return -1;
    const DenseArgs d{a, b, c, sfa, sfb, m, n, k, lda, ldb, ldc, 1.0f, status};
    const DenseChoice choice = choose_dense<split::OpMx>(m, n, k / 128, kKindMx);
    if (choice.nt > 0)
        return launch_split_nt<split::OpMx>(d, choice.nt, choice.split, stream);
    return choice.split == 2 ? launch_mx<2>(d, stream) : launch_mx<1>(d, stream);
}
