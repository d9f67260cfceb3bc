// k_sort.cu -- stable sort of (u64 fingerprint, u32 value) pairs by the sort
// key  fp1:29 | fp2:29 | table:1  (common.cuh).
//
// Replaces the reference's thrust::sort_by_key calls on fingerprints
// (cqutils.cuh:163,195,213; in-core case of cq_sort_by_key 180-202), which
// are stable (CUB radix sort), so equal keys keep their input order.
//
//   groups   The pairs are first split by the key's top bits, stably, into
//            groups that fit shared memory: one radix pass of 8 bits up to
//            256 groups, two (16 bits) above (onesweep, below).  One CTA then
//            sorts each group there: 4096 finer key ranges, each pair ranked
//            among the few of its range by (key, position).  Fingerprints are
//            residues of a hash, so groups are even: 2900 pairs on average at
//            most, 21 sigma below the 4096 that fit.  Up to 4096 pairs are one
//            group, one launch.
//   radix    When a group is larger (keys that are no fingerprints, one key
//            thousands of times), or a key has bits above the 59: an LSD
//            radix sort of all 8 digits.  What the group passes did before
//            keeps equal keys in order, so it starts from there.
//   onesweep one kernel per 8-bit digit (Adinets & Merrill, "Onesweep", 2022).
//            A CTA turns the digit histogram into bucket bases, then
//            repeatedly takes the next tile (atomic ticket, so every
//            predecessor is already running) and runs onesweep_tile on it
//            (sort_block.cuh): stable warp match-any ranking, per-digit
//            decoupled look-back over epoch-tagged words with bounded waits,
//            reorder in shared memory, one contiguous run per digit.
//
// A full radix sort moves 24 bytes a pair in each of 8 passes; the groups move
// them in 2 passes and once in shared memory.  33.3M pairs: 3.28 -> 1.39 ms
// (histogram 0.04, two onesweep passes 0.41 each, groups 0.48; HBM alone would
// take 0.41); 1M pairs 250 -> 82 us on the device; up to 4096 pairs one launch
// of 11 us instead of eleven.  A onesweep pass is bound by its look-back (each
// tile reads the words of the tiles in flight before it: 2 CTAs of 512
// threads, 3 of 512, and windows of 16 words took 406, 497 and 528 us against
// 410 now), a group by the latency of shared memory.
#include <atomic>

#include "sort_block.cuh"

namespace emp {

namespace {

constexpr int kGT = 512;              // threads of a group's CTA
constexpr uint32_t kFineLog = 12;     // finer ranges of a group
constexpr uint32_t kFine = 1u << kFineLog;
constexpr uint32_t kFineMax = 32;     // pairs of one range ranked by comparing all of them
constexpr int kKeyBits = 59;
static_assert(kSmallSort == kSortTile && kSmallSort <= 65535, "u16 positions");

// key bits that pick a pair's group: the fewest that give kGroupMean pairs on average
int group_bits(uint64_t n) {
    int b = 0;
    while ((n >> b) > kGroupMean) ++b;
    return n <= kSmallSort ? 0 : b;
}
constexpr int kMaxGroupBits = 2 * kSortBits;
size_t lookback_bytes(uint64_t n) { return (size_t)sort_tiles(n < 1 ? 1 : n) * kSortRadix * sizeof(uint64_t); }
// Group bounds lie behind the look-back words of n pairs, where a later and
// larger sort has look-back words: they carry an epoch that no sort reaches.
uint64_t *group_bounds(SortScratch *sc, uint64_t n) {
    return reinterpret_cast<uint64_t *>(reinterpret_cast<uint8_t *>(sc + 1) + lookback_bytes(n));
}
constexpr uint64_t kBoundTag = 0xfffffull << 44;
static_assert((2 * kSortsPerClear + 2) * kSortPasses < 0xfffff, "no sort reaches the bounds' epoch");

}  // namespace

size_t sort_scratch_bytes(uint64_t n) {
    // group bounds: at most n / (kGroupMean / 2) groups
    return sizeof(SortScratch) + lookback_bytes(n) + (size_t)(n / (kGroupMean / 2) + 4) * sizeof(uint64_t);
}
int sort_moves(uint64_t n) {
    const int bits = group_bits(n);
    return bits == 0 ? 1 : bits <= kSortBits ? 2 : bits <= kMaxGroupBits ? 3 : kSortPasses;
}
uint32_t *sort_flags(void *scratch) { return &reinterpret_cast<SortScratch *>(scratch)->radix; }

namespace {

// A new sort on this scratch: a new epoch, tickets and histogram zero.
__global__ void __launch_bounds__(256) sort_prepare_kernel(SortScratch *sc, bool radix) {
    if (radix && !sc->radix) return;
    for (int i = threadIdx.x; i < kSortPasses * kSortRadix; i += blockDim.x) (&sc->hist[0][0])[i] = 0;
    if (threadIdx.x < kSortPasses) sc->tile_ctr[threadIdx.x] = 0;
    if (threadIdx.x == 0) {
        sc->epoch = (sc->epoch + 1) & 0x1ffffu;
        if (!radix) sc->radix = sc->err = 0;
    }
}

// Histograms of the top digit, and of the one below when kDigits = 2.
template <int kDigits>
__global__ void __launch_bounds__(512) group_hist_kernel(const uint64_t *__restrict__ keys, uint64_t n,
                                                         SortScratch *sc) {
    __shared__ uint32_t s_hist[kDigits][kSortRadix];
    for (int i = threadIdx.x; i < kDigits * kSortRadix; i += blockDim.x) (&s_hist[0][0])[i] = 0;
    __syncthreads();
    bool high = false;
    auto count = [&](uint64_t key) {
        const uint64_t sk = sort_key(key, 0);
        high |= (sk >> kKeyBits) != 0;
#pragma unroll
        for (int d = 0; d < kDigits; ++d)
            atomicAdd(&s_hist[d][(sk >> (kKeyBits - (kDigits - d) * kSortBits)) & (kSortRadix - 1)], 1u);
    };
    const uint64_t t = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x, step = (uint64_t)gridDim.x * blockDim.x;
    uint64_t i = t;
    for (; i + 3 * step < n; i += 4 * step) {  // four loads in flight
        uint64_t k[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) k[u] = __ldg(keys + i + u * step);
#pragma unroll
        for (int u = 0; u < 4; ++u) count(k[u]);
    }
    for (; i < n; i += step) count(__ldg(keys + i));
    if (__syncthreads_or(high) && threadIdx.x == 0) sc->radix = 1;
    for (int q = threadIdx.x; q < kDigits * kSortRadix; q += blockDim.x) {
        const uint32_t c = (&s_hist[0][0])[q];
        if (c) atomicAdd(&sc->hist[0][0] + q, c);
    }
}

// Histograms of all 8 digits.
__global__ void __launch_bounds__(256) sort_hist_kernel(const uint64_t *__restrict__ keys,
                                                        const uint32_t *__restrict__ vals, uint64_t n,
                                                        SortScratch *sc) {
    __shared__ uint32_t s_hist[kSortPasses][kSortRadix];
    if (!sc->radix) return;
    for (int i = threadIdx.x; i < kSortPasses * kSortRadix; i += blockDim.x) (&s_hist[0][0])[i] = 0;
    __syncthreads();
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t sk = sort_key(keys[i], vals[i]);
#pragma unroll
        for (int p = 0; p < kSortPasses; ++p) atomicAdd(&s_hist[p][(sk >> (p * kSortBits)) & (kSortRadix - 1)], 1u);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < kSortPasses * kSortRadix; i += blockDim.x) {
        const uint32_t c = (&s_hist[0][0])[i];
        if (c) atomicAdd(&sc->hist[0][0] + i, c);
    }
}

// One digit pass; when: the sort's radix flag that it runs under.
__global__ void __launch_bounds__(kBlkThreads, 3) onesweep_kernel(
    const uint64_t *__restrict__ kin, const uint32_t *__restrict__ vin, uint64_t *__restrict__ kout,
    uint32_t *__restrict__ vout, uint64_t n, int pass, int shift, uint32_t when, SortScratch *sc,
    uint32_t *__restrict__ err) {
    extern __shared__ __align__(16) uint8_t smem[];
    __shared__ uint32_t s_bucket[kSortRadix];
    __shared__ uint32_t s_scan[32];
    __shared__ uint32_t s_tile;
    if ((*(volatile uint32_t *)&sc->radix != 0) != (when != 0)) return;
    const int tid = threadIdx.x;
    const uint64_t ntiles = sort_tiles(n);
    const uint32_t epoch = ((*(volatile uint32_t *)&sc->epoch) * kSortPasses + pass) & 0xfffffu;
    uint64_t *lookback = reinterpret_cast<uint64_t *>(sc + 1);
    {  // bucket bases of this digit from the histogram
        uint32_t tot;
        const uint32_t c = tid < kSortRadix ? sc->hist[pass][tid] : 0u;
        const uint32_t ex = block_exclusive_scan<kBlkThreads, uint32_t>(c, s_scan, &tot);
        if (tid < kSortRadix) s_bucket[tid] = ex;
    }
    for (;;) {
        if (tid == 0) s_tile = atomicAdd(&sc->tile_ctr[pass], 1u);
        __syncthreads();
        const uint32_t tile = s_tile;
        __syncthreads();
        if (tile >= ntiles) break;
        onesweep_tile(kin, vin, kout, vout, n, tile, shift, s_bucket, lookback, epoch, err, smem);
    }
}

// bounds[g] = first pair of group g (sorted by group): one warp per group,
// 33-ary search.
__global__ void __launch_bounds__(256) group_bounds_kernel(const uint64_t *__restrict__ keys, uint64_t n, int bits,
                                                           const SortScratch *sc, uint64_t *__restrict__ bounds) {
    if (sc->radix) return;
    const uint32_t g = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (g > 1u << bits) return;
    uint64_t lo = 0, hi = n;  // the bound is in [lo, hi]
    while (hi > lo) {
        const uint64_t step = (hi - lo + 31) / 32, at = lo + lane * step;  // probes lo, lo + step, ..
        const bool below = at < hi && (sort_key(__ldg(keys + at), 0) >> (kKeyBits - bits)) < g;
        const uint32_t m = __popc(__ballot_sync(0xffffffffu, below));  // keys are in order: the first m are below
        const uint64_t l0 = lo;
        if (m == 0) break;
        lo = l0 + (m - 1) * step + 1;
        hi = min(hi, l0 + m * step);
    }
    if (lane == 0) bounds[g] = kBoundTag | lo;
}

// ---------------------------------------------------------------- groups
struct GroupSmem {
    uint64_t key[kSmallSort];
    uint32_t val[kSmallSort];
    uint32_t start[kFine + 1];  // counts, then starts of the finer ranges
    uint16_t tmp[kSmallSort];   // positions by finer range
    uint16_t ord[kSmallSort];   // positions in order
    uint32_t scan[32];
};

EMP_DEV bool pair_before(const GroupSmem &w, uint32_t a, uint64_t skb, uint32_t b) {
    const uint64_t ska = sort_key(w.key[a], w.val[a]);
    return ska < skb || (ska == skb && a < b);
}

// One CTA per group of 2^bits (by the top bits of the 59), from (kin, vin)
// to the same place of (kout, vout), which may be the same arrays.  bits = 0:
// all n <= kSmallSort pairs are one group, whatever their keys.
// Bound: the latency of shared memory across its phases (two CTAs of 512
// threads per SM: half of the warps; a variant with 57 KB that keeps the
// pairs in registers and permutes them in place was 4-20 % slower).
__global__ void __launch_bounds__(kGT, 2) group_sort_kernel(const uint64_t *kin, const uint32_t *vin, uint64_t *kout,
                                                            uint32_t *vout, uint64_t n, int bits,
                                                            const uint64_t *__restrict__ bounds, SortScratch *sc) {
    extern __shared__ __align__(16) uint8_t group_smem[];
    GroupSmem &w = *reinterpret_cast<GroupSmem *>(group_smem);
    const uint32_t tid = threadIdx.x, groups = 1u << bits;
    const int shift = kKeyBits - bits - (int)kFineLog;
    if (bits && *(volatile uint32_t *)&sc->radix == 1) return;  // not grouped: the pairs are still in (k0, v0)
    for (uint32_t g = blockIdx.x; g < groups; g += gridDim.x) {
        const uint64_t lo = bits ? bounds[g] & ~kBoundTag : 0, hi = bits ? bounds[g + 1] & ~kBoundTag : n;
        const uint32_t c = hi - lo > kSmallSort ? kSmallSort + 1 : (uint32_t)(hi - lo);
        if (c == 0) continue;
        if (c > kSmallSort) {  // too large: as it is, and the radix sort follows
            if (kin != kout)
                for (uint64_t i = lo + tid; i < hi; i += kGT) {
                    kout[i] = kin[i];
                    vout[i] = vin[i];
                }
            if (tid == 0) sc->radix = 2;
            continue;
        }
        constexpr int kPer = kSmallSort / kGT;
        uint32_t fr[kPer];  // finer range << 16 | arrival
#pragma unroll
        for (int q = 0; q < kPer; ++q) {
            const uint32_t i = q * kGT + tid;
            if (i >= c) continue;
            w.key[i] = __ldcg(kin + lo + i);
            w.val[i] = __ldcg(vin + lo + i);
        }
        for (uint32_t i = tid; i <= kFine; i += kGT) w.start[i] = 0;
        __syncthreads();
#pragma unroll
        for (int q = 0; q < kPer; ++q) {
            const uint32_t i = q * kGT + tid;
            if (i >= c) continue;
            const uint64_t f = sort_key(w.key[i], 0) >> shift;
            const uint32_t fi = bits ? (uint32_t)f & (kFine - 1) : (uint32_t)(f < kFine ? f : kFine - 1);
            fr[q] = (fi << 16) | atomicAdd(&w.start[fi], 1u);
        }
        __syncthreads();
        // range starts: kFine / kGT consecutive ranges a thread
        constexpr int kR = kFine / kGT;
        uint32_t cnt[kR], sum = 0, most = 0;
#pragma unroll
        for (int r = 0; r < kR; ++r) {
            cnt[r] = w.start[tid * kR + r];
            sum += cnt[r];
            most = max(most, cnt[r]);
        }
        uint32_t tot;
        uint32_t ex = block_exclusive_scan<kGT, uint32_t>(sum, w.scan, &tot);
#pragma unroll
        for (int r = 0; r < kR; ++r) {
            w.start[tid * kR + r] = ex;
            ex += cnt[r];
        }
        if (tid == 0) w.start[kFine] = tot;
        const bool crowded = __syncthreads_or(most > kFineMax) != 0;
        if (!crowded) {
#pragma unroll
            for (int q = 0; q < kPer; ++q)
                if (q * kGT + tid < c) w.tmp[w.start[fr[q] >> 16] + (fr[q] & 0xffffu)] = (uint16_t)(q * kGT + tid);
            __syncthreads();
#pragma unroll
            for (int q = 0; q < kPer; ++q) {  // the place among the few of its range
                const uint32_t i = q * kGT + tid;
                if (i >= c) continue;
                const uint32_t a = w.start[fr[q] >> 16], z = w.start[(fr[q] >> 16) + 1];
                uint32_t r = a;
                if (z - a > 1) {
                    const uint64_t sk = sort_key(w.key[i], w.val[i]);
                    for (uint32_t p = a; p < z; ++p) r += pair_before(w, w.tmp[p], sk, i);
                }
                w.ord[r] = (uint16_t)i;
            }
            __syncthreads();
        } else {  // one range holds many pairs (equal keys): bitonic sort of the positions by (key, position)
            uint32_t m = 32;
            while (m < c) m <<= 1;
            for (uint32_t i = tid; i < m; i += kGT) w.ord[i] = (uint16_t)i;  // positions c .. m - 1 sort last
            __syncthreads();
            for (uint32_t k = 2; k <= m; k <<= 1)
                for (uint32_t d = k >> 1; d; d >>= 1) {
                    for (uint32_t x = tid; x < m / 2; x += kGT) {
                        const uint32_t i = 2 * x - (x & (d - 1)), j = i + d;  // the pair (i, i + d)
                        const uint32_t a = w.ord[i], b = w.ord[j];
                        const bool up = (i & k) == 0;
                        const bool less = b >= c ? a < b : a < c && pair_before(w, a, sort_key(w.key[b], w.val[b]), b);
                        if (less != up) {
                            w.ord[i] = (uint16_t)b;
                            w.ord[j] = (uint16_t)a;
                        }
                    }
                    __syncthreads();
                }
        }
        for (uint32_t i = tid; i < c; i += kGT) {
            const uint32_t p = w.ord[i];
            kout[lo + i] = w.key[p];
            vout[lo + i] = w.val[p];
        }
        __syncthreads();
    }
}

// Persistent grids of a device (SMs x resident CTAs): onesweep, group sort.
// Found once per device (the first call sets the kernels' shared-memory
// attributes) and kept in a per-device atomic, so host threads driving
// different devices neither race nor see each other's grid.
struct SortGrid {
    unsigned sweep, group;
};
SortGrid sort_grid_find(int dev) {
    cudaFuncSetAttribute(onesweep_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kOnesweepSmem);
    cudaFuncSetAttribute(group_sort_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(GroupSmem));
    int sms = 148, occ = 0, og = 0;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, onesweep_kernel, kBlkThreads, kOnesweepSmem) !=
            cudaSuccess || occ < 1)
        occ = 1;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&og, group_sort_kernel, kGT, sizeof(GroupSmem)) != cudaSuccess ||
        og < 1)
        og = 1;
    cudaGetLastError();
    const unsigned m = (unsigned)(sms > 0 ? sms : 148);
    return SortGrid{m * (unsigned)occ, m * (unsigned)og};
}
SortGrid sort_setup() {
    constexpr int kDevs = 64;
    static std::atomic<uint64_t> grid[kDevs] = {};  // 0: not found yet
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kDevs) {
        cudaGetLastError();
        return sort_grid_find(dev < 0 ? 0 : dev);
    }
    uint64_t g = grid[dev].load(std::memory_order_acquire);
    if (g == 0) {
        const SortGrid f = sort_grid_find(dev);
        g = (uint64_t)f.sweep << 32 | f.group;
        grid[dev].store(g, std::memory_order_release);
    }
    return SortGrid{(unsigned)(g >> 32), (unsigned)g};
}
unsigned sweep_grid(uint64_t n, const SortGrid &sg) {
    const uint64_t tiles = sort_tiles(n);
    return (unsigned)(tiles < sg.sweep ? tiles : sg.sweep);
}

}  // namespace

void sort_groups(uint64_t *k0, uint32_t *v0, uint64_t *k1, uint32_t *v1, uint64_t n, void *scratch, uint32_t *err,
                 cudaStream_t s) {
    const SortGrid sg = sort_setup();
    SortScratch *sc = reinterpret_cast<SortScratch *>(scratch);
    const int bits = group_bits(n);
    if (n < 2) {
        cudaMemsetAsync(&sc->radix, 0, 2 * sizeof(uint32_t), s);
        return;
    }
    if (bits == 0) {
        count_launch();
        cudaMemsetAsync(&sc->radix, 0, 2 * sizeof(uint32_t), s);
        group_sort_kernel<<<1, kGT, sizeof(GroupSmem), s>>>(k0, v0, k0, v0, n, 0, nullptr, sc);
        return;
    }
    count_launch();
    sort_prepare_kernel<<<1, 256, 0, s>>>(sc, false);
    if (bits > kMaxGroupBits) {  // too many pairs for 2^16 groups
        cudaMemsetAsync(&sc->radix, 1, 1, s);
        return;
    }
    const uint64_t hb = (n + 2047) / 2048;
    const unsigned hblocks = (unsigned)(hb < 148 * 4 ? hb : 148 * 4);
    const unsigned grid = sweep_grid(n, sg);
    const uint32_t groups = 1u << bits;
    uint64_t *bounds = group_bounds(sc, n);
    uint64_t *ks = k1;
    uint32_t *vs = v1;
    if (bits <= kSortBits) {
        group_hist_kernel<1><<<hblocks, 512, 0, s>>>(k0, n, sc);
        onesweep_kernel<<<grid, kBlkThreads, kOnesweepSmem, s>>>(k0, v0, k1, v1, n, 0, kKeyBits - kSortBits, 0u, sc, err);
    } else {
        group_hist_kernel<2><<<hblocks, 512, 0, s>>>(k0, n, sc);
        onesweep_kernel<<<grid, kBlkThreads, kOnesweepSmem, s>>>(k0, v0, k1, v1, n, 0, kKeyBits - 2 * kSortBits, 0u, sc,
                                                                 err);
        onesweep_kernel<<<grid, kBlkThreads, kOnesweepSmem, s>>>(k1, v1, k0, v0, n, 1, kKeyBits - kSortBits, 0u, sc, err);
        ks = k0;
        vs = v0;
        count_launch();
    }
    count_launch(4);
    group_bounds_kernel<<<(groups + 1 + 7) / 8, 256, 0, s>>>(ks, n, bits, sc, bounds);
    group_sort_kernel<<<groups < sg.group ? groups : sg.group, kGT, sizeof(GroupSmem), s>>>(ks, vs, k0, v0, n, bits,
                                                                                           bounds, sc);
}

void sort_radix(uint64_t *k0, uint32_t *v0, uint64_t *k1, uint32_t *v1, uint64_t n, void *scratch, uint32_t *err,
                cudaStream_t s, cudaEvent_t *events) {
    const SortGrid sg = sort_setup();
    SortScratch *sc = reinterpret_cast<SortScratch *>(scratch);
    const uint64_t hb = (n + 255) / 256;
    const unsigned hblocks = (unsigned)(hb < 1 ? 1 : (hb < 148 * 4 ? hb : 148 * 4));
    const unsigned grid = sweep_grid(n < 1 ? 1 : n, sg);
    count_launch(2 + kSortPasses);
    sort_prepare_kernel<<<1, 256, 0, s>>>(sc, true);
    sort_hist_kernel<<<hblocks, 256, 0, s>>>(k0, v0, n, sc);
    uint64_t *kb[2] = {k0, k1};
    uint32_t *vb[2] = {v0, v1};
    for (int p = 0; p < kSortPasses; ++p) {
        if (events && p) cudaEventRecord(events[2 * p], s);
        onesweep_kernel<<<grid, kBlkThreads, kOnesweepSmem, s>>>(kb[p & 1], vb[p & 1], kb[(p & 1) ^ 1],
                                                                 vb[(p & 1) ^ 1], n, p, p * kSortBits, 1u, sc, err);
        if (events) cudaEventRecord(events[2 * p + 1], s);
    }
}

void sort_top_digit(const uint64_t *k0, const uint32_t *v0, uint64_t *k1, uint32_t *v1, uint64_t n, void *scratch,
                    uint32_t *err, cudaStream_t s) {
    static_assert(kTopDigitShift == kKeyBits - kSortBits + 2, "bit b >= 32 of a key is bit b - 2 of its sort key");
    if (!n) return;
    const SortGrid sg = sort_setup();
    SortScratch *sc = reinterpret_cast<SortScratch *>(scratch);
    const uint64_t hb = (n + 2047) / 2048;
    count_launch(3);
    sort_prepare_kernel<<<1, 256, 0, s>>>(sc, false);
    group_hist_kernel<1><<<(unsigned)(hb < 148 * 4 ? hb : 148 * 4), 512, 0, s>>>(k0, n, sc);
    onesweep_kernel<<<sweep_grid(n, sg), kBlkThreads, kOnesweepSmem, s>>>(k0, v0, k1, v1, n, 0, kKeyBits - kSortBits, 0u,
                                                                          sc, err);
}

void sort_pairs(uint64_t *k0, uint32_t *v0, uint64_t *k1, uint32_t *v1, uint64_t n, void *scratch, uint32_t *err,
                cudaStream_t s, cudaEvent_t *events) {
    if (events) cudaEventRecord(events[0], s);  // the first pass's events take in the groups
    sort_groups(k0, v0, k1, v1, n, scratch, err, s);
    if (n > kSmallSort) {
        sort_radix(k0, v0, k1, v1, n, scratch, err, s, events);
    } else if (events) {
        for (int p = 1; p < 2 * kSortPasses; ++p) cudaEventRecord(events[p], s);
    }
}

}  // namespace emp
