// hostcopy.cu -- copies between pageable host memory and the device.
//
// The driver stages a pageable copy through one host thread (10 to 13 GB/s in,
// 4 GB/s out into fresh pages, whose faults that thread takes one by one,
// against 55 GB/s of PCIe).  Here several threads each move pieces through two
// page-locked pieces of their own, so that the host copies, the page faults
// and the transfers run beside one another: 31 MB of FASTQ in 2.5 -> 0.9 ms,
// 35 MB of unitigs out into fresh pages 8.9 -> 3.0 ms.
#include "hostcopy.h"

#include <atomic>
#include <cstring>
#include <thread>

namespace emp {

HostStage::~HostStage() {
    for (auto &e : ev_)
        if (e) cudaEventDestroy(e);
    if (pin_) cudaFreeHost(pin_);
    if (out_) cudaStreamDestroy(out_);
}

// the staging pieces and their events; false: not to be had (once and for all)
bool HostStage::ready() {
    if (pin_) return true;
    if (failed_) return false;
    void *p = nullptr;
    bool ok = true;
    for (auto &e : ev_) ok = ok && cudaEventCreateWithFlags(&e, cudaEventDisableTiming) == cudaSuccess;
    ok = ok && cudaHostAlloc(&p, 2 * kThreads * kPiece, cudaHostAllocDefault) == cudaSuccess;
    if (!ok) {
        cudaGetLastError();
        failed_ = true;
        return false;
    }
    pin_ = static_cast<uint8_t *>(p);
    return true;
}

cudaError_t HostStage::run(int device, bool in, uint8_t *dev, uint8_t *host, size_t n, cudaStream_t s) {
    const size_t pieces = (n + kPiece - 1) / kPiece;
    std::atomic<size_t> next{0};
    std::atomic<int> error{(int)cudaSuccess};
    auto work = [&](int t) {
        auto check = [&](cudaError_t e) {
            if (e != cudaSuccess) error.store((int)e, std::memory_order_relaxed);
            return e == cudaSuccess;
        };
        if (!check(cudaSetDevice(device))) return;
        struct {
            uint8_t *pin;
            cudaEvent_t ev;
            size_t at, len;
            bool busy;
        } p[2];
        for (int k = 0; k < 2; ++k) p[k] = {pin_ + (size_t)(2 * t + k) * kPiece, ev_[2 * t + k], 0, 0, false};
        auto land = [&](int k) {  // the piece's transfer is over, and its bytes are with the host
            if (!p[k].busy) return true;
            p[k].busy = false;
            if (!check(cudaEventSynchronize(p[k].ev))) return false;
            if (!in) std::memcpy(host + p[k].at, p[k].pin, p[k].len);
            return true;
        };
        for (int k = 0; error.load(std::memory_order_relaxed) == (int)cudaSuccess; k ^= 1) {
            const size_t i = next.fetch_add(1, std::memory_order_relaxed);
            if (i >= pieces) break;
            if (!land(k)) break;
            p[k].at = i * kPiece;
            p[k].len = n - p[k].at < kPiece ? n - p[k].at : kPiece;
            if (in) std::memcpy(p[k].pin, host + p[k].at, p[k].len);
            if (!check(in ? cudaMemcpyAsync(dev + p[k].at, p[k].pin, p[k].len, cudaMemcpyHostToDevice, s)
                          : cudaMemcpyAsync(p[k].pin, dev + p[k].at, p[k].len, cudaMemcpyDeviceToHost, s)) ||
                !check(cudaEventRecord(p[k].ev, s)))
                break;
            p[k].busy = true;
        }
        land(0);
        land(1);
    };
    std::thread helpers[kThreads];
    int started = 0;
    const int cores = (int)std::thread::hardware_concurrency();
    const int want = cores > 1 ? (cores < kThreads ? cores : kThreads) : 1;
    try {
        for (int t = 1; t < want && (size_t)t < pieces; ++t) {
            helpers[t] = std::thread(work, t);
            ++started;
        }
    } catch (...) {  // no more threads: with those there are (they are joined below)
    }
    work(0);
    for (int t = 1; t <= started; ++t) helpers[t].join();
    return (cudaError_t)error.load();
}

static bool pageable(const void *p) {
    cudaPointerAttributes a{};
    if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    return a.type == cudaMemoryTypeUnregistered;
}

cudaError_t HostStage::to_device(int device, void *dst, const void *src, size_t n, cudaStream_t s) {
    std::unique_lock<std::mutex> lock(mu_, std::defer_lock);
    if (n >= kLeast && pageable(src) && lock.try_lock() && ready())
        return run(device, true, static_cast<uint8_t *>(dst), static_cast<uint8_t *>(const_cast<void *>(src)), n, s);
    return cudaMemcpyAsync(dst, src, n, cudaMemcpyHostToDevice, s);
}

cudaError_t HostStage::to_host(int device, void *dst, const void *src, size_t n) {
    {
        std::lock_guard<std::mutex> g(out_mu_);
        if (!out_) {
            const cudaError_t e = cudaStreamCreateWithFlags(&out_, cudaStreamNonBlocking);
            if (e != cudaSuccess) return e;
        }
    }
    std::unique_lock<std::mutex> lock(mu_, std::defer_lock);
    if (n >= kLeast && pageable(dst) && lock.try_lock() && ready())
        return run(device, false, static_cast<uint8_t *>(const_cast<void *>(src)), static_cast<uint8_t *>(dst), n, out_);
    const cudaError_t e = cudaMemcpyAsync(dst, src, n, cudaMemcpyDeviceToHost, out_);
    return e == cudaSuccess ? cudaStreamSynchronize(out_) : e;
}

}  // namespace emp
