// sort_block.cuh -- block-level pieces of the stable LSD radix sort (k_sort.cu)
// and the shared helpers of the cooperative round kernel (k_bucket.cu).
// 256 threads per CTA (three CTAs per SM), 16 pairs per thread, 4096-pair
// tiles.
#pragma once

#include "kernels.h"

namespace emp {

constexpr int kBlkThreads = 256;
constexpr int kBlkWarps = kBlkThreads / 32;
constexpr int kBlkItems = kSortTile / kBlkThreads;  // 16

EMP_DEV uint32_t lanemask_lt_u32() {
    uint32_t m;
    asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
    return m;
}

EMP_DEV uint32_t digit_of(uint64_t k, uint32_t v, int shift) {
    return (uint32_t)(sort_key(k, v) >> shift) & (kSortRadix - 1);
}

// Stable rank of each thread's items within its warp (order: item j, lane);
// wh = this warp's 256 zeroed digit counters, left holding the warp's counts.
EMP_DEV void warp_rank(const uint64_t (&k)[kBlkItems], const uint32_t (&v)[kBlkItems], const bool (&ok)[kBlkItems],
                        int shift, uint32_t *wh, uint32_t (&rank)[kBlkItems]) {
    const uint32_t ltmask = lanemask_lt_u32();
#pragma unroll
    for (int j = 0; j < kBlkItems; ++j) {
        const uint32_t d = ok[j] ? digit_of(k[j], v[j], shift) : kSortRadix;
        const uint32_t peers = __match_any_sync(0xffffffffu, d);
        const uint32_t before = __popc(peers & ltmask);
        const uint32_t prior = d < kSortRadix ? wh[d] : 0u;
        __syncwarp();
        if (d < kSortRadix && before == 0) wh[d] = prior + __popc(peers);
        __syncwarp();
        rank[j] = prior + before;
    }
}

constexpr int kLook = 4;  // predecessors a look-back step reads at once

// Shared memory of onesweep_tile: one 4096-pair tile, warp counters, digit
// offsets, and scan room.  `bucket` (256 words, caller-owned) holds the
// global bucket bases of the pass's digit.
constexpr size_t kOnesweepSmem = kSortTile * (sizeof(uint64_t) + sizeof(uint32_t)) +
                                 (kBlkWarps + 2) * kSortRadix * sizeof(uint32_t) + 32 * sizeof(uint32_t);

// One tile of one stable digit pass: rank, publish per-digit counts, resolve
// the prefix of earlier tiles by decoupled look-back (epoch-tagged words,
// bounded waits), reorder in shared memory, write each digit's run.
EMP_DEV void onesweep_tile(const uint64_t *__restrict__ kin, const uint32_t *__restrict__ vin,
                           uint64_t *__restrict__ kout, uint32_t *__restrict__ vout, uint64_t n, uint32_t tile,
                           int shift, const uint32_t *bucket, uint64_t *lookback, uint32_t epoch, uint32_t *err,
                           uint8_t *smem) {
    uint64_t *s_keys = reinterpret_cast<uint64_t *>(smem);
    uint32_t *s_vals = reinterpret_cast<uint32_t *>(s_keys + kSortTile);
    uint32_t *s_whist = s_vals + kSortTile;
    uint32_t *s_texcl = s_whist + kBlkWarps * kSortRadix;
    uint32_t *s_glob = s_texcl + kSortRadix;
    uint32_t *s_scan = s_glob + kSortRadix;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint64_t base = (uint64_t)tile * kSortTile;
    for (int i = tid; i < kBlkWarps * kSortRadix; i += kBlkThreads) s_whist[i] = 0;
    __syncthreads();
    uint64_t k[kBlkItems];
    uint32_t v[kBlkItems], rank[kBlkItems];
    bool ok[kBlkItems];
#pragma unroll
    for (int j = 0; j < kBlkItems; ++j) {
        const uint64_t idx = base + warp * (kBlkItems * 32) + j * 32 + lane;
        ok[j] = idx < n;
        k[j] = ok[j] ? __ldcg(kin + idx) : 0;
        v[j] = ok[j] ? __ldcg(vin + idx) : 0;
    }
    warp_rank(k, v, ok, shift, s_whist + warp * kSortRadix, rank);
    __syncthreads();
    uint32_t cnt = 0;
    if (tid < kSortRadix) {
#pragma unroll
        for (int w = 0; w < kBlkWarps; ++w) {
            const uint32_t c = s_whist[w * kSortRadix + tid];
            s_whist[w * kSortRadix + tid] = cnt;
            cnt += c;
        }
        st_status(lookback + (uint64_t)tile * kSortRadix + tid, ep_word(epoch, tile == 0 ? kEpInc : kEpAgg, cnt));
    }
    uint32_t tot;
    const uint32_t dex = block_exclusive_scan<kBlkThreads, uint32_t>(tid < kSortRadix ? cnt : 0u, s_scan, &tot);
    if (tid < kSortRadix) {
        s_texcl[tid] = dex;
        uint64_t excl = 0;
        if (tile > 0) {
            int64_t t = (int64_t)tile - 1;
            bool done = false;
            while (t >= 0 && !done) {
                const int kk = t >= kLook - 1 ? kLook : (int)t + 1;
                uint64_t w[kLook];
#pragma unroll
                for (int i = 0; i < kLook; ++i)
                    if (i < kk) w[i] = ld_status(lookback + (uint64_t)(t - i) * kSortRadix + tid);
#pragma unroll
                for (int i = 0; i < kLook; ++i) {
                    if (i >= kk || done) break;
                    uint32_t f, spins = 0;
                    while ((f = ep_flag(w[i], epoch)) == 0) {
                        if (++spins > kSpinLimit) {
                            atomicOr(err, kErrSpin);
                            done = true;
                            break;
                        }
                        if (spins > 32) __nanosleep(32);
                        w[i] = ld_status(lookback + (uint64_t)(t - i) * kSortRadix + tid);
                    }
                    if (done) break;
                    excl += w[i] & kEpVal;
                    done = f == 2;
                }
                t -= kk;
            }
            st_status(lookback + (uint64_t)tile * kSortRadix + tid, ep_word(epoch, kEpInc, excl + cnt));
        }
        s_glob[tid] = bucket[tid] + (uint32_t)excl;
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < kBlkItems; ++j) {
        if (ok[j]) {
            const uint32_t d = digit_of(k[j], v[j], shift);
            const uint32_t pos = s_texcl[d] + s_whist[warp * kSortRadix + d] + rank[j];
            s_keys[pos] = k[j];
            s_vals[pos] = v[j];
        }
    }
    __syncthreads();
    const uint32_t valid = n - base < kSortTile ? (uint32_t)(n - base) : kSortTile;
    for (uint32_t i = tid; i < valid; i += kBlkThreads) {
        const uint64_t kk = s_keys[i];
        const uint32_t vv = s_vals[i];
        const uint32_t d = digit_of(kk, vv, shift);
        const uint64_t o = (uint64_t)s_glob[d] + (i - s_texcl[d]);
        kout[o] = kk;
        vout[o] = vv;
    }
    __syncthreads();
}

}  // namespace emp
