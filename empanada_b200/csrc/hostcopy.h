// hostcopy.h -- copies between pageable host memory and the device.
#pragma once

#include <cstddef>
#include <cstdint>
#include <mutex>

#include <cuda_runtime.h>

namespace emp {

// Page-locked staging pieces of a context, made when the first large pageable
// copy needs them (kThreads * 2 * kPiece = 12 MiB) and freed with it.  One
// copy uses them at a time; another one meanwhile takes the driver's own path.
class HostStage {
  public:
    ~HostStage();
    // n bytes to the device in the order of stream s; the host memory may be
    // written again once s has been waited for.
    cudaError_t to_device(int device, void *dst, const void *src, size_t n, cudaStream_t s);
    // n bytes that are ready on the device to the host, on a stream of their
    // own, so that they wait for no other job's work; returns when they are there.
    cudaError_t to_host(int device, void *dst, const void *src, size_t n);

  private:
    static constexpr int kThreads = 6;
    static constexpr size_t kPiece = 1 << 20;
    static constexpr size_t kLeast = 4 << 20;  // shorter copies: the driver's own path
    bool ready();
    cudaError_t run(int device, bool in, uint8_t *dev, uint8_t *host, size_t n, cudaStream_t s);
    std::mutex mu_;
    uint8_t *pin_ = nullptr;
    cudaEvent_t ev_[2 * kThreads] = {};
    cudaStream_t out_ = nullptr;
    std::mutex out_mu_;
    bool failed_ = false;
};

}  // namespace emp
