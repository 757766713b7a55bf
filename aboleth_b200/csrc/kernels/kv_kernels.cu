// KV-cache page push: a producer rank stores runs of pages into a consumer rank's
// slot storage over NVLink and publishes per-(slot, consumer, source) readiness.
//
// Grid (batches, workers).  The workers of one batch split its bytes; every worker
// ends with a CTA barrier and one atomic arrival.  Batches that publish the SAME
// readiness cell (several layers and runs of one readiness group) form a group with
// one arrival counter whose target is the group's worker total: only the worker that
// arrives last IN THE GROUP performs the system fence and release-stores the epoch,
// so the cell never shows the epoch while a sibling batch is still copying - "the
// last copy worker of a consumer performs the system fence and publishes the epoch"
// (reference docs/KV_CACHE.md:46-48; kernels
// python/aboleth/frontends/triton/kv_cache.py:133-292 count per batch and then per
// consumer, and copy 8-byte words; these count once per group and copy 16-byte
// vectors, four in flight per thread).
#include "common.cuh"

namespace {

struct KvBatch {
    std::uint64_t src;     // local address of the run (contiguous pages)
    std::uint64_t dst;     // peer address of the destination slot storage
    std::uint64_t bytes;   // run length (pages * page_bytes)
    std::uint64_t ready;   // peer address of the int64 readiness cell
};

// One worker CTA: copy its slice of batch `batch`, arrive, publish if last of the group.
//   group_of == nullptr : every batch is its own group (counter `batch`, target `workers`);
//   otherwise           : counter group_of[batch], target group_target[group_of[batch]].
__device__ __forceinline__ void push_worker(const KvBatch *batches, unsigned *arrivals,
                                            const int *group_of, const unsigned *group_target,
                                            int batch, int worker, std::uint64_t epoch, int workers,
                                            unsigned long long *status) {
    const KvBatch b = batches[batch];
    // 16-byte aligned worker slices.
    const std::uint64_t per = ((b.bytes + workers - 1) / workers + 15) & ~15ull;
    const std::uint64_t begin = ab::min64(per * worker, b.bytes);
    const std::uint64_t end = ab::min64(begin + per, b.bytes);
    // A run that is not 16-byte aligned is reported and still copied (8-byte or byte path).
    if (((b.src | b.dst) & 15) != 0 && threadIdx.x == 0 && worker == 0)
        ab::set_status(status, aboleth::Status::Malformed, 0x7000 + batch);
    aboleth::detail::copy_strided(reinterpret_cast<std::uint8_t *>(b.dst + begin),
                                  reinterpret_cast<const std::uint8_t *>(b.src + begin), end - begin,
                                  threadIdx.x, blockDim.x);
    __syncthreads();
    if (threadIdx.x == 0) {
        const int counter = group_of != nullptr ? group_of[batch] : batch;
        const unsigned target = group_of != nullptr ? group_target[counter] : static_cast<unsigned>(workers);
        __threadfence();
        const unsigned old = atomicAdd(arrivals + counter, 1u);
        if (old == target - 1) {
            arrivals[counter] = 0;  // self-cleaning for the next transfer
            aboleth::detail::fence_acq_rel_sys();
            aboleth::detail::st_release_sys(reinterpret_cast<std::uint64_t *>(b.ready), epoch);
        }
    }
}

__global__ void __launch_bounds__(512) kv_push_kernel(const KvBatch *batches, unsigned *arrivals,
                                                      const int *group_of, const unsigned *group_target,
                                                      std::uint64_t epoch, int workers,
                                                      unsigned long long *status) {
    push_worker(batches, arrivals, group_of, group_target, blockIdx.x, blockIdx.y, epoch, workers, status);
}

// Self-check form: the same push plus ONE consumer CTA in the same launch (block row `count`),
// which waits (bounded) for `cell` to show `epoch` and then, at once, sums the 8-byte words of
// every batch's destination into observed[0].  A cell that is published before the data has
// landed shows up as a sum that differs from the sources'.  One launch, every CTA resident:
// nothing here waits on another launch.
__global__ void __launch_bounds__(512) kv_push_observed_kernel(
    const KvBatch *batches, unsigned *arrivals, const int *group_of, const unsigned *group_target,
    int count, std::uint64_t epoch, int workers, const std::uint64_t *cell,
    unsigned long long *observed, std::uint64_t timeout_ns, unsigned long long *status) {
    if (static_cast<int>(blockIdx.x) < count) {
        push_worker(batches, arrivals, group_of, group_target, blockIdx.x, blockIdx.y, epoch, workers, status);
        return;
    }
    if (blockIdx.y != 0)
        return;
    __shared__ int s_ok;
    __shared__ unsigned long long s_sum;
    if (threadIdx.x == 0) {
        const aboleth::Status s = aboleth::wait_signal_status(cell, epoch, timeout_ns);
        ab::set_status(status, s, 0x7300);
        s_ok = s == aboleth::Status::Ok;
        s_sum = 0;
    }
    __syncthreads();
    if (!s_ok)
        return;
    unsigned long long sum = 0;
    for (int i = 0; i < count; ++i) {
        const KvBatch b = batches[i];
        const std::uint64_t *words = reinterpret_cast<const std::uint64_t *>(b.dst);
        for (std::uint64_t w = threadIdx.x; w < b.bytes / 8; w += blockDim.x)
            sum += aboleth::detail::ld_relaxed_sys(words + w);
    }
    atomicAdd(&s_sum, sum);
    __syncthreads();
    if (threadIdx.x == 0)
        observed[0] = s_sum;
}

// Consumer side: wait (bounded) until every listed readiness cell reached `epoch`.
__global__ void kv_wait_kernel(const std::uint64_t *cells, int count, std::uint64_t epoch,
                               std::uint64_t timeout_ns, unsigned long long *status) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < count; i += gridDim.x * blockDim.x) {
        const aboleth::Status s = aboleth::wait_signal_status(cells + i, epoch, timeout_ns);
        ab::set_status(status, s, 0x7100 + i);
    }
}

// ---- one transfer, described by its page runs -----------------------------------------
//
// A transfer moves the same page runs of every layer.  Its description - the runs, two strides, the readiness
// cells - fits the kernel's arguments, so nothing is built or uploaded per (run, layer) batch.  The grid is
// resident and takes the readiness groups one after the other; every CTA copies an equal share of a group's bytes,
// whatever runs they lie in, and arrives once per group.  So the first layers are published after their share of
// the time and not near the end, and there is one fence per CTA and group instead of one per 16 KiB: 32 layers x
// 64 pages of 64 KiB in 8 runs took 99 us as 8192 CTAs, 66 us so (2 x 134 MB at copy bandwidth: 43).
constexpr int kMaxRuns = 256;

struct KvRun {
    int src, dst;   // first page in the producer's pool and in the consumer's slot
    int first;      // pages before this run
};

struct KvPages {
    const std::uint8_t *pool;
    std::uint64_t slots, cells;          // of the consumer: layer 0 of the slot, readiness cell of group 0
    std::uint64_t pool_layer, slot_layer, cell_stride, page_bytes, epoch;
    unsigned *arrivals;                  // [groups], zero between launches
    unsigned long long *status;
    int layers, per_group, runs, pages;
    int misaligned;                      // the first (layer, run) that is not 16-byte aligned, or -1
    KvRun run[kMaxRuns];
};

// Bytes [begin, end) of one run of one layer, both multiples of 16 or the run's end.
__device__ __forceinline__ void copy_piece(std::uint8_t *dst, const std::uint8_t *src, std::uint64_t bytes) {
    constexpr int kDepth = 8;
    const std::uint64_t mix = reinterpret_cast<std::uint64_t>(dst) | reinterpret_cast<std::uint64_t>(src);
    if ((mix & 15) != 0) {
        aboleth::detail::copy_strided(dst, src, bytes, threadIdx.x, blockDim.x);
        return;
    }
    const std::uint64_t vecs = bytes >> 4;
    for (std::uint64_t base = threadIdx.x; base < vecs; base += static_cast<std::uint64_t>(kDepth) * blockDim.x) {
        uint4 v[kDepth];
#pragma unroll
        for (int u = 0; u < kDepth; ++u)
            if (base + static_cast<std::uint64_t>(u) * blockDim.x < vecs)
                v[u] = aboleth::detail::ld_stream16(src + ((base + static_cast<std::uint64_t>(u) * blockDim.x) << 4));
#pragma unroll
        for (int u = 0; u < kDepth; ++u)
            if (base + static_cast<std::uint64_t>(u) * blockDim.x < vecs)
                aboleth::detail::st_stream16(dst + ((base + static_cast<std::uint64_t>(u) * blockDim.x) << 4), v[u]);
    }
    for (std::uint64_t b = (vecs << 4) + threadIdx.x; b < bytes; b += blockDim.x)
        dst[b] = src[b];
}

__global__ void __launch_bounds__(512, 2) kv_push_pages_kernel(const __grid_constant__ KvPages p) {
    const std::uint64_t layer_bytes = static_cast<std::uint64_t>(p.pages) * p.page_bytes;
    // Such a run is reported and still copied (8-byte or byte path).
    if (p.misaligned >= 0 && blockIdx.x == 0 && threadIdx.x == 0)
        ab::set_status(p.status, aboleth::Status::Malformed, 0x7000 + p.misaligned);
    for (int group = 0, layer0 = 0; layer0 < p.layers; ++group, layer0 += p.per_group) {
        const int count = min(p.per_group, p.layers - layer0);
        const std::uint64_t total = layer_bytes * count;
        const std::uint64_t share = total / gridDim.x, rest = total % gridDim.x;
        std::uint64_t at = share * blockIdx.x + rest * blockIdx.x / gridDim.x;
        const std::uint64_t end = share * (blockIdx.x + 1) + rest * (blockIdx.x + 1) / gridDim.x;
        while (at < end) {
            // The run that byte `at` of the group lies in, and this CTA's bytes of it.  Cuts fall on 16-byte
            // boundaries of the run: the CTA before stops where this one starts.
            const int layer = static_cast<int>(at / layer_bytes);
            const std::uint64_t in_layer = at - layer * layer_bytes;
            const int page = static_cast<int>(in_layer / p.page_bytes);
            int lo = 0, hi = p.runs - 1;
            while (lo < hi) {
                const int mid = (lo + hi + 1) / 2;
                if (p.run[mid].first <= page)
                    lo = mid;
                else
                    hi = mid - 1;
            }
            const KvRun run = p.run[lo];
            const int next = lo + 1 < p.runs ? p.run[lo + 1].first : p.pages;
            const std::uint64_t run_at = layer * layer_bytes + run.first * p.page_bytes;
            const std::uint64_t run_bytes = static_cast<std::uint64_t>(next - run.first) * p.page_bytes;
            const std::uint64_t begin = (at - run_at) & ~15ull;
            const bool whole = end >= run_at + run_bytes;
            const std::uint64_t stop = whole ? run_bytes : (end - run_at) & ~15ull;
            if (stop > begin)
                copy_piece(reinterpret_cast<std::uint8_t *>(p.slots + (layer0 + layer) * p.slot_layer +
                                                            run.dst * static_cast<long long>(p.page_bytes) + begin),
                           p.pool + (layer0 + layer) * p.pool_layer + run.src * p.page_bytes + begin, stop - begin);
            at = whole ? run_at + run_bytes : end;
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            __threadfence();
            if (atomicAdd(p.arrivals + group, 1u) == gridDim.x - 1) {
                p.arrivals[group] = 0;  // self-cleaning for the next transfer
                aboleth::detail::fence_acq_rel_sys();
                aboleth::detail::st_release_sys(reinterpret_cast<std::uint64_t *>(p.cells + group * p.cell_stride),
                                                p.epoch);
            }
        }
    }
}

}  // namespace

// One transfer: page i of `src` (of the producer's pool: `layers` layers, `pool_layer` bytes apart) goes to page
// dst[i] of the consumer's slot (`slots`: its layer 0, layers `slot_layer` bytes apart); group g of `per_group`
// layers is published in the cell at cells + g * cell_stride.  `src` and `dst` are host arrays, read before the
// call returns.  arrivals: device u32 [groups], zeroed.  Every page of `src` lies inside the pool, where a negative one
// counts from its end, and every page of `dst` inside the slot.  A run is consecutive pages on both sides, so none
// continues from the pool's last page to page 0.  runs: how many were found; -3 when they are more than one launch
// carries (256), -4 when a page of `src`, -5 when a page of `dst` is outside; nothing was launched then.
AB_EXPORT int ab_kv_push_pages(const long long *src, const long long *dst, int pages, const void *pool, int layers,
                               int blocks, std::uint64_t pool_layer, std::uint64_t page_bytes, std::uint64_t slots,
                               std::uint64_t slot_layer, std::uint64_t cells, std::uint64_t cell_stride, int per_group,
                               std::uint64_t epoch, unsigned *arrivals, unsigned long long *status, int workers,
                               int threads, int *runs, cudaStream_t stream) {
    if (src == nullptr || dst == nullptr || pages < 1 || pool == nullptr || layers < 1 || per_group < 1 ||
        page_bytes < 1 || arrivals == nullptr || runs == nullptr || workers < 1 || threads < 32 || threads > 512 ||
        threads % 32 != 0)
        return -1;
    KvPages p;
    int n = 0;
    const long long slot_pages = static_cast<long long>(slot_layer / page_bytes);
    long long last_from = -1;
    for (int i = 0; i < pages; ++i) {
        const long long from = src[i] < 0 ? src[i] + blocks : src[i];
        if (from < 0 || from >= blocks)
            return -4;
        if (dst[i] < 0 || dst[i] >= slot_pages)
            return -5;
        const bool extends = i > 0 && from == last_from + 1 && dst[i] == dst[i - 1] + 1;
        last_from = from;
        if (extends)
            continue;
        if (n == kMaxRuns)
            return -3;
        p.run[n++] = KvRun{static_cast<int>(from), static_cast<int>(dst[i]), i};
    }
    *runs = n;
    p.pool = static_cast<const std::uint8_t *>(pool);
    p.slots = slots, p.cells = cells;
    p.pool_layer = pool_layer, p.slot_layer = slot_layer, p.cell_stride = cell_stride;
    p.page_bytes = page_bytes, p.epoch = epoch;
    p.arrivals = arrivals, p.status = status;
    p.layers = layers, p.per_group = per_group, p.runs = n, p.pages = pages;
    p.misaligned = -1;
    if (((reinterpret_cast<std::uint64_t>(pool) | slots | pool_layer | slot_layer | page_bytes) & 15) != 0)
        for (int i = 0; i < layers * n && p.misaligned < 0; ++i) {
            const std::uint64_t layer = i / n, from = p.run[i % n].src, to = p.run[i % n].dst;
            const std::uint64_t a = reinterpret_cast<std::uint64_t>(pool) + layer * pool_layer + from * page_bytes;
            if (((a | (slots + layer * slot_layer + to * page_bytes)) & 15) != 0)
                p.misaligned = i;
        }
    // Two CTAs per SM, a CTA's share of a full group at least one round of its threads' loads, and no more CTAs
    // than the profile's workers per batch allow.
    const std::uint64_t group_bytes = page_bytes * pages * ab::min64(layers, per_group);
    const std::uint64_t round = static_cast<std::uint64_t>(threads) * 16 * 2;
    std::uint64_t grid = (group_bytes + round - 1) / round;
    grid = ab::min64(grid, 296);
    grid = ab::min64(grid, static_cast<std::uint64_t>(n) * layers * workers);
    kv_push_pages_kernel<<<static_cast<unsigned>(grid < 1 ? 1 : grid), threads, 0, stream>>>(p);
    return ab::launch_result("kv_push_pages");
}

// batches: device array of `count` {src, dst, bytes, ready} records; arrivals: device u32, zeroed,
// one per batch (group_of == nullptr) or one per group.  group_of: device int [count], the group of
// each batch; group_target: device u32, arrivals that complete each group (its batches x workers).
// Batches that name the same readiness cell MUST share a group.
AB_EXPORT int ab_kv_push(const void *batches, unsigned *arrivals, const int *group_of,
                         const unsigned *group_target, int count, std::uint64_t epoch, int workers,
                         int threads, unsigned long long *status, cudaStream_t stream) {
    if (batches == nullptr || arrivals == nullptr || count < 1 || workers < 1 || workers > 65535 ||
        threads < 32 || threads > 512 || threads % 32 != 0 ||
        (group_of == nullptr) != (group_target == nullptr))
        return -1;
    kv_push_kernel<<<dim3(count, workers), threads, 0, stream>>>(
        static_cast<const KvBatch *>(batches), arrivals, group_of, group_target, epoch, workers, status);
    return ab::launch_result("kv_push");
}

// The push with a consumer CTA in the same launch (see kv_push_observed_kernel).
AB_EXPORT int ab_kv_push_observed(const void *batches, unsigned *arrivals, const int *group_of,
                                  const unsigned *group_target, int count, std::uint64_t epoch,
                                  int workers, int threads, const std::uint64_t *cell,
                                  unsigned long long *observed, std::uint64_t timeout_ns,
                                  unsigned long long *status, cudaStream_t stream) {
    if (batches == nullptr || arrivals == nullptr || cell == nullptr || observed == nullptr ||
        count < 1 || workers < 1 || workers > 64 || (count + 1) * workers > 148 || threads < 32 ||
        threads > 512 || threads % 32 != 0 || (group_of == nullptr) != (group_target == nullptr))
        return -1;  // the whole grid must be resident: at most one CTA per SM is asked for
    kv_push_observed_kernel<<<dim3(count + 1, workers), threads, 0, stream>>>(
        static_cast<const KvBatch *>(batches), arrivals, group_of, group_target, count, epoch, workers,
        cell, observed, timeout_ns, status);
    return ab::launch_result("kv_push_observed");
}

AB_EXPORT int ab_kv_wait(const std::uint64_t *cells, int count, std::uint64_t epoch,
                         std::uint64_t timeout_ns, unsigned long long *status, cudaStream_t stream) {
    if (count < 1)
        return -1;
    kv_wait_kernel<<<(count + 127) / 128, 128, 0, stream>>>(cells, count, epoch, timeout_ns, status);
    return ab::launch_result("kv_wait");
}

// Copy-engine path for few, large runs: one asynchronous copy per run (addresses may be peer
// mappings; unified addressing picks the direction).
AB_EXPORT int ab_memcpy_async(void *dst, const void *src, std::uint64_t bytes, cudaStream_t stream) {
    const cudaError_t e = cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDefault, stream);
    if (e != cudaSuccess) {
        fprintf(stderr, "aboleth_b200: asynchronous copy failed: %s\n", cudaGetErrorString(e));
        return static_cast<int>(e);
    }
    return 0;
}
