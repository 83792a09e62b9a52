// readback.cpp -- see readback.h.
#include "readback.h"

#include <algorithm>
#include <atomic>
#include <cstring>
#include <thread>

namespace clb {

ReadBack::~ReadBack() { release(); }

void ReadBack::release()
{
    for (int w = 0; w < kMaxWorkers; w++) {
        if (stream_[w])
            cudaStreamDestroy(stream_[w]);
        stream_[w] = nullptr;
        for (cudaEvent_t &e : arrived_[w]) {
            if (e)
                cudaEventDestroy(e);
            e = nullptr;
        }
    }
    if (pinned_)
        cudaFreeHost(pinned_);
    pinned_ = nullptr;
    workers_ = 0;
}

bool ReadBack::setup()
{
    if (workers_ > 0)
        return true;
    const int workers = std::min<int>(kMaxWorkers, (int)std::thread::hardware_concurrency() / 2);
    if (workers < 2)
        return false;   // nothing to share the copies out to
    bool ok = cudaHostAlloc((void **)&pinned_, (size_t)workers * 2 * kChunk, cudaHostAllocPortable) == cudaSuccess;
    for (int w = 0; ok && w < workers; w++) {
        ok = cudaStreamCreateWithFlags(&stream_[w], cudaStreamNonBlocking) == cudaSuccess;
        for (cudaEvent_t &e : arrived_[w])
            ok = ok && cudaEventCreateWithFlags(&e, cudaEventDisableTiming) == cudaSuccess;
    }
    if (!ok) {
        cudaGetLastError();
        release();
        return false;
    }
    workers_ = workers;
    return true;
}

cudaError_t ReadBack::copy(void *dst, const void *src, size_t bytes)
{
    std::unique_lock<std::mutex> lock(busy_, std::defer_lock);
    bool shared = false;
    if (bytes >= kMinBytes) {
        cudaPointerAttributes at;
        if (cudaPointerGetAttributes(&at, dst) != cudaSuccess)
            cudaGetLastError();
        else
            shared = at.type == cudaMemoryTypeUnregistered && lock.try_lock() && setup();
    }
    if (!shared)
        return cudaMemcpy(dst, src, bytes, cudaMemcpyDeviceToHost);
    // the first chunk as before, on the legacy stream: it waits for all that
    // such a copy waits for
    const size_t head = kChunk;
    cudaError_t e = cudaMemcpy(dst, src, head, cudaMemcpyDeviceToHost);
    int device = 0;
    if (e == cudaSuccess)
        e = cudaGetDevice(&device);
    if (e != cudaSuccess)
        return e;
    const size_t chunks = (bytes - head + kChunk - 1) / kChunk;
    std::atomic<size_t> next{0};
    std::atomic<int> failed{(int)cudaSuccess};
    auto worker = [&](int w) {
        cudaError_t r = cudaSetDevice(device);
        size_t held[2] = {chunks, chunks};   // chunk in each buffer
        auto fetch = [&](int b) {
            held[b] = next.fetch_add(1);
            if (held[b] >= chunks || r != cudaSuccess)
                return;
            const size_t off = head + held[b] * kChunk;
            r = cudaMemcpyAsync(pinned_ + ((size_t)w * 2 + b) * kChunk, (const char *)src + off,
                                std::min(kChunk, bytes - off), cudaMemcpyDeviceToHost, stream_[w]);
            if (r == cudaSuccess)
                r = cudaEventRecord(arrived_[w][b], stream_[w]);
        };
        fetch(0);
        for (int b = 0; held[b] < chunks && r == cudaSuccess; b ^= 1) {
            fetch(b ^ 1);
            if (r == cudaSuccess)
                r = cudaEventSynchronize(arrived_[w][b]);
            if (r != cudaSuccess)
                break;
            const size_t off = head + held[b] * kChunk;
            std::memcpy((char *)dst + off, pinned_ + ((size_t)w * 2 + b) * kChunk, std::min(kChunk, bytes - off));
        }
        const cudaError_t end = cudaStreamSynchronize(stream_[w]);   // no copy outlives the call
        if (r == cudaSuccess)
            r = end;
        if (r != cudaSuccess)
            failed = (int)r;
    };
    std::thread others[kMaxWorkers];
    for (int w = 1; w < workers_; w++) {
        try {
            others[w] = std::thread(worker, w);
        } catch (...) {
            break;   // no more threads to be had: the others take its chunks
        }
    }
    worker(0);
    for (std::thread &t : others)
        if (t.joinable())
            t.join();
    return (cudaError_t)failed.load();
}

}  // namespace clb
