// k_dedup.cu -- duplicate removal of the read-end fingerprints when they fit
// one chunk of the reference's sort (2n <= M).
//
// The reference sorts all (fingerprint, rid) pairs stably and keeps the first
// pair of every equal-key run (cq_sort_by_key + cq_unique_by_key,
// overlap.cu:212-225, cqutils.cuh:180-202,272-306): with the rids in
// increasing order before the stable sort, the survivor of a run is its
// smallest rid.  Only that survivor set matters here (the list is rebuilt in
// id order afterwards), so no sort is needed:
//
//   hist     per-CTA shared-memory histogram of the key buckets (the top
//            bits of fp1 scaled to nb buckets), added into global counts
//   scan     bucket starts and cursors (one CTA); the counts zeroed for the
//            next call
//   scatter  each (key, rid) to its bucket: a CTA ranks a tile of keys per
//            bucket in shared memory and reserves each bucket's run with one
//            atomic (up to 2048 buckets), or one atomic per run of equal
//            buckets within a warp (more buckets, cursors rarely shared)
//   mark     one CTA per bucket: a shared-memory hash set of the bucket's
//            distinct keys holding the smallest rid of each (atomicMin),
//            then alive[rid] = (rid is its key's smallest)
//
// For the jobs of a batch each step is one launch over all of them (256 sets,
// 26.4M read-ends: 0.15, 0.005, 0.28 and 0.64 ms).
//
// About 45 bytes move per read-end (a sort moves over 200).  A bucket whose
// distinct keys do not fit the hash set raises kErrDedupFull; the engine then
// falls back to the sort.
#include <atomic>

#include "sort_block.cuh"

namespace emp {
namespace {

constexpr int kDT = 256;                // threads per CTA
constexpr uint32_t kDedupSlots = 8192;  // hash slots of the mark kernel (power of two)
constexpr uint32_t kDedupFull = 7680;   // distinct keys of one bucket at most
constexpr uint64_t kDedupEmpty = ~0ull; // never a key: fp1, fp2 < 2^29

__device__ __forceinline__ uint32_t dedup_bucket(uint64_t key, uint32_t nb) {
    return (uint32_t)(((key >> 32) * (uint64_t)nb) >> 29);  // fp1 < 2^29
}

EMP_DEV void dedup_hist_block(const DedupArgs &a, uint32_t bid) {
    const uint64_t *const __restrict__ keys = a.keys;
    const uint64_t n = a.n;
    const uint32_t nb = a.nb;
    uint32_t *const __restrict__ counts = a.counts;
    if (bid == 0 && a.zero)
        for (uint32_t i = threadIdx.x; i < a.zero_n; i += kDT) a.zero[i] = 0;
    extern __shared__ uint32_t s_hist[];  // nb
    for (uint32_t i = threadIdx.x; i < nb; i += kDT) s_hist[i] = 0;
    __syncthreads();
    for (uint64_t e = (uint64_t)bid * kDT + threadIdx.x; e < n; e += (uint64_t)a.hist_blocks * kDT)
        atomicAdd(&s_hist[dedup_bucket(__ldg(keys + e), nb)], 1u);
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < nb; i += kDT)
        if (s_hist[i]) atomicAdd(counts + i, s_hist[i]);
}
__global__ void __launch_bounds__(kDT) dedup_hist_kernel(const DedupArgs a) { dedup_hist_block(a, blockIdx.x); }
__global__ void __launch_bounds__(kDT) dedup_hist_many_kernel(const DedupArgs *a, const uint2 *blk) {
    const uint2 b = blk[blockIdx.x];
    dedup_hist_block(a[b.x], b.y);
}

// start[b] = cursor[b] = the exclusive scan of the counts (one CTA), which
// are zeroed for the next call.
constexpr int kScanT = 1024;
EMP_DEV void dedup_scan_block(const DedupArgs &a) {
    uint32_t *const __restrict__ counts = a.counts, *const __restrict__ start = a.start;
    uint32_t *const __restrict__ cursor = a.cursor;
    const uint32_t nb = a.nb;
    __shared__ uint32_t s_warp[32];
    uint32_t run = 0;
    for (uint32_t b0 = 0; b0 < nb; b0 += 4 * kScanT) {
        uint32_t c[4], sum = 0;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const uint32_t b = b0 + 4 * threadIdx.x + q;
            c[q] = b < nb ? counts[b] : 0u;
            if (b < nb) counts[b] = 0;
            sum += c[q];
        }
        uint32_t tot;
        uint32_t x = run + block_exclusive_scan<kScanT, uint32_t>(sum, s_warp, &tot);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const uint32_t b = b0 + 4 * threadIdx.x + q;
            if (b < nb) start[b] = cursor[b] = x;
            x += c[q];
        }
        run += tot;
    }
}
__global__ void __launch_bounds__(kScanT) dedup_scan_kernel(const DedupArgs a) { dedup_scan_block(a); }
__global__ void __launch_bounds__(kScanT) dedup_scan_many_kernel(const DedupArgs *a) { dedup_scan_block(a[blockIdx.x]); }

__global__ void __launch_bounds__(kDT) dedup_scatter_kernel(const uint64_t *__restrict__ keys, uint64_t n,
                                                            uint32_t nb, uint32_t *__restrict__ cursor,
                                                            uint64_t *__restrict__ pk, uint32_t *__restrict__ pr) {
    const uint64_t stride = (uint64_t)gridDim.x * kDT;
    for (uint64_t e0 = (uint64_t)blockIdx.x * kDT; e0 < n; e0 += stride) {  // uniform per warp
        const uint64_t e = e0 + threadIdx.x;
        const bool act = e < n;
        const uint64_t k = act ? __ldg(keys + e) : 0;
        const uint32_t b = act ? dedup_bucket(k, nb) : 0u;
        const uint32_t m = __ballot_sync(0xffffffffu, act);
        if (!act) continue;
        const uint32_t peers = __match_any_sync(m, b);
        const uint32_t lane = threadIdx.x & 31, leader = __ffs(peers) - 1;
        uint32_t pos = 0;
        if (lane == leader) pos = atomicAdd(cursor + b, (uint32_t)__popc(peers));
        pos = __shfl_sync(peers, pos, leader) + __popc(peers & lanemask_lt_u32());
        pk[pos] = k;
        pr[pos] = (uint32_t)e;
    }
}

// The same for few buckets (nb <= kTiledBuckets), where the bucket cursors
// would be hot: a CTA ranks a tile of kScatterTile keys per bucket in shared
// memory and reserves each bucket's run with one atomic.
constexpr uint32_t kTiledBuckets = kDedupTiled;
constexpr int kScatterPer = 16;
constexpr uint32_t kScatterTile = kDT * kScatterPer;

EMP_DEV void dedup_scatter_tiled_block(const DedupArgs &a, uint32_t bid) {
    const uint64_t *const __restrict__ keys = a.keys;
    const uint64_t n = a.n;
    const uint32_t nb = a.nb;
    uint32_t *const __restrict__ cursor = a.cursor, *const __restrict__ pr = a.pr;
    uint64_t *const __restrict__ pk = a.pk;
    __shared__ uint32_t s_cnt[kTiledBuckets];
    for (uint64_t t0 = (uint64_t)bid * kScatterTile; t0 < n; t0 += (uint64_t)a.scatter_blocks * kScatterTile) {
        for (uint32_t b = threadIdx.x; b < nb; b += kDT) s_cnt[b] = 0;
        __syncthreads();
        uint64_t k[kScatterPer];
        uint32_t bk[kScatterPer], rk[kScatterPer];
#pragma unroll
        for (int q = 0; q < kScatterPer; ++q) {
            const uint64_t e = t0 + (uint64_t)q * kDT + threadIdx.x;
            k[q] = e < n ? __ldg(keys + e) : 0;
            bk[q] = e < n ? dedup_bucket(k[q], nb) : 0u;
            rk[q] = e < n ? atomicAdd(&s_cnt[bk[q]], 1u) : 0u;
        }
        __syncthreads();
        for (uint32_t b = threadIdx.x; b < nb; b += kDT) {
            const uint32_t c = s_cnt[b];
            s_cnt[b] = c ? atomicAdd(cursor + b, c) : 0u;  // the run's global start
        }
        __syncthreads();
#pragma unroll
        for (int q = 0; q < kScatterPer; ++q) {
            const uint64_t e = t0 + (uint64_t)q * kDT + threadIdx.x;
            if (e >= n) continue;
            const uint32_t pos = s_cnt[bk[q]] + rk[q];
            pk[pos] = k[q];
            pr[pos] = (uint32_t)e;
        }
        __syncthreads();
    }
}
__global__ void __launch_bounds__(kDT) dedup_scatter_tiled_kernel(const DedupArgs a) {
    dedup_scatter_tiled_block(a, blockIdx.x);
}
__global__ void __launch_bounds__(kDT) dedup_scatter_many_kernel(const DedupArgs *a, const uint2 *blk) {
    const uint2 b = blk[blockIdx.x];
    dedup_scatter_tiled_block(a[b.x], b.y);
}

__device__ __forceinline__ uint32_t dedup_slot(uint64_t key) {
    return (uint32_t)((key * 0x9E3779B97F4A7C15ull) >> 40) & (kDedupSlots - 1);
}

constexpr size_t kMarkSmem = kDedupSlots * (8 + 4);

EMP_DEV void dedup_mark_block(const DedupArgs &a, uint32_t bid) {
    const uint64_t *const __restrict__ pk = a.pk;
    const uint32_t *const __restrict__ pr = a.pr, *const __restrict__ start = a.start;
    const uint32_t nb = a.nb;
    const uint64_t n = a.n;
    uint8_t *const __restrict__ alive = a.alive;
    uint32_t *const err = a.err;
    extern __shared__ __align__(16) uint8_t smem[];
    uint64_t *s_key = reinterpret_cast<uint64_t *>(smem);
    uint32_t *s_min = reinterpret_cast<uint32_t *>(s_key + kDedupSlots);
    __shared__ uint32_t s_used;
    for (uint32_t b = bid; b < nb; b += a.mark_blocks) {
        for (uint32_t i = threadIdx.x; i < kDedupSlots; i += kDT) {
            s_key[i] = kDedupEmpty;
            s_min[i] = 0xffffffffu;
        }
        if (threadIdx.x == 0) s_used = 0;
        __syncthreads();
        const uint64_t lo = start[b], hi = b + 1 < nb ? start[b + 1] : n;
        bool full = false;
        for (uint64_t x = lo + threadIdx.x; x < hi; x += kDT) {  // smallest rid of every key
            const uint64_t k = pk[x];
            const uint32_t r = pr[x];
            uint32_t s = dedup_slot(k);
            for (uint32_t probes = 0; probes < kDedupSlots; ++probes) {
                const uint64_t old = atomicCAS(reinterpret_cast<unsigned long long *>(s_key + s),
                                               (unsigned long long)kDedupEmpty, (unsigned long long)k);
                if (old == kDedupEmpty && atomicAdd(&s_used, 1u) >= kDedupFull) full = true;
                if (old == kDedupEmpty || old == k) {
                    atomicMin(s_min + s, r);
                    break;
                }
                s = (s + 1) & (kDedupSlots - 1);
            }
        }
        if (__syncthreads_or(full)) {  // too many distinct keys: the engine sorts instead
            if (threadIdx.x == 0) atomicOr(err, kErrDedupFull);
            return;
        }
        for (uint64_t x = lo + threadIdx.x; x < hi; x += kDT) {  // survivors
            const uint64_t k = pk[x];
            const uint32_t r = pr[x];
            uint32_t s = dedup_slot(k);
            while (s_key[s] != k) s = (s + 1) & (kDedupSlots - 1);  // present: inserted above
            alive[r] = s_min[s] == r ? 1 : 0;
        }
        __syncthreads();
    }
}
__global__ void __launch_bounds__(kDT) dedup_mark_hash_kernel(const DedupArgs a) { dedup_mark_block(a, blockIdx.x); }
__global__ void __launch_bounds__(kDT) dedup_mark_many_kernel(const DedupArgs *a, const uint2 *blk) {
    const uint2 b = blk[blockIdx.x];
    dedup_mark_block(a[b.x], b.y);
}

}  // namespace

uint32_t dedup_buckets(uint64_t n) {
    if (n == 0 || n > kDedupMaxEnds) return 0;
    uint64_t nb = (n + kDedupMean - 1) / kDedupMean;
    return (uint32_t)(nb > kDedupMaxBuckets ? kDedupMaxBuckets : nb);
}

// Shared-memory attributes of the kernels, set once per device.
static bool dedup_setup(int &sms) {
    constexpr int kDevs = 64;
    static std::atomic<int> done[kDevs] = {};  // SM count, 0: not set up yet
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kDevs) {
        cudaGetLastError();
        return false;
    }
    sms = done[dev].load(std::memory_order_acquire);
    if (sms) return true;
    int n = 0;
    cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
    if (cudaFuncSetAttribute(dedup_hist_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)(kDedupMaxBuckets * 4)) != cudaSuccess ||
        cudaFuncSetAttribute(dedup_mark_many_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMarkSmem) !=
            cudaSuccess ||
        cudaFuncSetAttribute(dedup_mark_hash_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMarkSmem) !=
            cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    sms = n > 0 ? n : 148;
    done[dev].store(sms, std::memory_order_release);
    return true;
}

bool dedup_args(DedupArgs *a, const uint64_t *keys, uint64_t n, uint32_t nb, void *scratch, uint64_t *pk, uint32_t *pr,
                uint8_t *alive, uint32_t *err) {
    int sms = 0;
    if (!n || !nb || !dedup_setup(sms)) return false;
    uint32_t *counts = reinterpret_cast<uint32_t *>(scratch);
    uint32_t *start = counts + kDedupMaxBuckets, *cursor = start + kDedupMaxBuckets;
    const uint64_t per = (n + kDT - 1) / kDT, tiles = (n + kScatterTile - 1) / kScatterTile, most = (uint64_t)sms;
    *a = DedupArgs{keys, n, nb, 0u, 0u, 0u, counts, start, cursor, pk, pr, alive, err, nullptr, 0u};
    a->hist_blocks = (uint32_t)(per < most * 4 ? per : most * 4);
    a->scatter_blocks = (uint32_t)(nb <= kTiledBuckets ? (tiles < most * 8 ? tiles : most * 8)
                                                       : (per < most * 8 ? per : most * 8));
    a->mark_blocks = nb < most * 2 ? nb : (uint32_t)most * 2;
    return true;
}

bool launch_dedup_hash(const uint64_t *keys, uint64_t n, uint32_t nb, void *scratch, uint64_t *pk, uint32_t *pr,
                       uint8_t *alive, uint32_t *err, cudaStream_t s) {
    DedupArgs a;
    if (!dedup_args(&a, keys, n, nb, scratch, pk, pr, alive, err)) return false;
    count_launch(4);
    dedup_hist_kernel<<<a.hist_blocks, kDT, nb * 4, s>>>(a);
    dedup_scan_kernel<<<1, kScanT, 0, s>>>(a);
    if (nb <= kTiledBuckets) dedup_scatter_tiled_kernel<<<a.scatter_blocks, kDT, 0, s>>>(a);
    else dedup_scatter_kernel<<<a.scatter_blocks, kDT, 0, s>>>(keys, n, nb, a.cursor, pk, pr);
    dedup_mark_hash_kernel<<<a.mark_blocks, kDT, kMarkSmem, s>>>(a);
    return true;
}

void launch_dedup_many(const DedupArgs *a, uint32_t jobs, uint32_t nb_max, ManyBlocks hist, ManyBlocks scatter,
                       ManyBlocks mark, cudaStream_t s) {
    if (!jobs) return;
    count_launch(4);
    dedup_hist_many_kernel<<<hist.n, kDT, nb_max * 4, s>>>(a, hist.blk);
    dedup_scan_many_kernel<<<jobs, kScanT, 0, s>>>(a);
    dedup_scatter_many_kernel<<<scatter.n, kDT, 0, s>>>(a, scatter.blk);
    dedup_mark_many_kernel<<<mark.n, kDT, kMarkSmem, s>>>(a, mark.blk);
}

}  // namespace emp
