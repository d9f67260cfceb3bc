// k_sort_static.cu -- emp_sort_pairs_static: the stable onesweep sort of
// k_sort.cu with its whole working set in one statically sized device array,
// so a call allocates nothing (no cudaMalloc / cudaFree, no allocating
// library routine).
//
// The array holds, for at most kStaticMaxPairs pairs:
//   [alternate keys 8 B/pair][alternate values 4 B/pair]
//   [SortScratch header with the error word][look-back words, one per (4096-pair tile, digit)]
//   [group bounds]
// Each call clears the header and the look-back words of its
// own tiles before the sort reads them.  Every call on a device uses the
// same array: calls whose GPU work overlaps (other streams, other host
// threads) race on it and give wrong results.
#include <mutex>

#include "../../include/empanada.h"
#include "kernels.h"

namespace emp {
namespace {

constexpr uint64_t kStaticMaxPairs = EMP_SORT_STATIC_MAX_PAIRS;
constexpr size_t kAlign = 256;
constexpr size_t align_up(size_t x) { return (x + kAlign - 1) / kAlign * kAlign; }
constexpr size_t kOffK1 = 0;
constexpr size_t kOffV1 = align_up(kOffK1 + kStaticMaxPairs * sizeof(uint64_t));
constexpr size_t kOffScr = align_up(kOffV1 + kStaticMaxPairs * sizeof(uint32_t));
constexpr size_t kMaxTiles = (kStaticMaxPairs + kSortTile - 1) / kSortTile;
constexpr size_t kScrBytes = sizeof(SortScratch) + kMaxTiles * kSortRadix * sizeof(uint64_t) +
                             (kStaticMaxPairs / (kGroupMean / 2) + 4) * sizeof(uint64_t);
constexpr size_t kStaticBytes = align_up(kOffScr + kScrBytes);  // 12.6 MB at 2^20 pairs

static __device__ __align__(256) uint8_t g_sort_static[kStaticBytes];

constexpr int kMaxDevices = 64;
std::mutex g_mu;
uint8_t *g_ptr[kMaxDevices] = {};

// Device address of g_sort_static on the current device (looked up once).
emp_status static_scratch(uint8_t **out) {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) {
        cudaGetLastError();
        return EMP_E_CUDA;
    }
    if (dev < 0 || dev >= kMaxDevices) return EMP_E_UNSUPPORTED;
    std::lock_guard<std::mutex> lock(g_mu);
    if (!g_ptr[dev]) {
        uint8_t *p = nullptr;
        if (cudaGetSymbolAddress((void **)&p, g_sort_static) != cudaSuccess || !p) {
            cudaGetLastError();
            return EMP_E_CUDA;
        }
        g_ptr[dev] = p;
    }
    *out = g_ptr[dev];
    return EMP_OK;
}

}  // namespace
}  // namespace emp

extern "C" emp_status emp_sort_pairs_static(uint64_t *d_keys, uint32_t *d_vals, uint64_t n, void *stream) {
    using namespace emp;
    if (n > kStaticMaxPairs) return EMP_E_INVAL;
    if (n && (!d_keys || !d_vals)) return EMP_E_INVAL;  // the argument check of emp_sort_pairs
    if (n < 2) return EMP_OK;
    uint8_t *base = nullptr;
    const emp_status rc = static_scratch(&base);
    if (rc != EMP_OK) return rc;
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    uint8_t *scr = base + kOffScr;
    uint32_t *flags = sort_flags(scr);  // radix sort needed, error
    // header + look-back words of n's tiles
    if (cudaMemsetAsync(scr, 0, sort_scratch_bytes(n), s) != cudaSuccess) {
        cudaGetLastError();
        return EMP_E_CUDA;
    }
    uint64_t *k1 = reinterpret_cast<uint64_t *>(base + kOffK1);
    uint32_t *v1 = reinterpret_cast<uint32_t *>(base + kOffV1);
    uint32_t h[2] = {0, 0};
    sort_groups(d_keys, d_vals, k1, v1, n, scr, flags + 1, s);
    for (int radix = 0;; radix = 1) {
        if (cudaGetLastError() != cudaSuccess ||
            cudaMemcpyAsync(h, flags, sizeof h, cudaMemcpyDeviceToHost, s) != cudaSuccess ||
            cudaStreamSynchronize(s) != cudaSuccess) {
            cudaGetLastError();
            return EMP_E_CUDA;
        }
        if (!h[0] || radix) break;
        sort_radix(d_keys, d_vals, k1, v1, n, scr, flags + 1, s);  // uneven keys
    }
    const uint32_t herr = h[1];
    if (herr & kErrSpin) return EMP_E_TIMEOUT;
    return EMP_OK;
}
