// readback.h -- large device-to-host copies into pageable memory.
//
// cudaMemcpy to pageable memory goes through one thread of the driver, which
// also takes the page faults of a fresh destination: 145 MB in 29-68 ms, as
// long as 90 or more linear-solver steps of the 800 x 800 grid it brings.  Here
// several threads take chunks in turn, each with two pinned buffers: one fills
// over PCIe while the other is copied out.  The same copy takes 11 ms (bound by
// the faults), 7.6 ms into memory already touched (cudaMemcpy 8-13).
#pragma once

#include <cuda_runtime.h>

#include <cstddef>
#include <mutex>

namespace clb {

class ReadBack {
public:
    ReadBack() = default;
    ReadBack(const ReadBack &) = delete;
    ReadBack &operator=(const ReadBack &) = delete;
    ~ReadBack();
    // cudaMemcpy(dst, src, bytes, cudaMemcpyDeviceToHost), with its order
    // towards other streams.  Copies below kMinBytes, into memory CUDA knows,
    // while another thread is in here, or without the buffers: that call itself.
    cudaError_t copy(void *dst, const void *src, size_t bytes);

private:
    // The buffers (4 MiB) are made by the first large copy and kept.  They take
    // 3.5 ms, less than a first copy of kMinBytes saves; with 1 MiB chunks
    // they took 12 ms and a fresh destination no less time.  Four threads
    // instead of eight: 18 ms.
    static constexpr size_t kMinBytes = (size_t)32 << 20, kChunk = (size_t)256 << 10;
    static constexpr int kMaxWorkers = 8;
    bool setup();
    void release();
    std::mutex busy_;
    int workers_ = 0;
    char *pinned_ = nullptr;   // [worker][2][kChunk]
    cudaStream_t stream_[kMaxWorkers] = {};
    cudaEvent_t arrived_[kMaxWorkers][2] = {};
};

}  // namespace clb
