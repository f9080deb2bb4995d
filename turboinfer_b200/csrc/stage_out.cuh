// stage_out.cuh -- device results into ordinary host memory through a small pinned double buffer.
//
// A copy straight into pageable memory is staged by the driver one piece at a time (measured on a B200 host: 100 us for 512 KB of logits, half of
// a decode step of four requests; this way about 50).  Here the copy engine fills one pinned half while the host empties the other.  One buffer a library, made when
// it is initialised (a buffer a model made loading a small model 1.4 times as long); calls of several threads take it in turn.
#pragma once
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <cstring>
#include <mutex>

namespace tib {

struct StageOut {
    static constexpr size_t kHalf = (size_t)256 << 10;
    uint8_t* p = nullptr;   // two halves
    cudaEvent_t ev[2] = {nullptr, nullptr};
    std::mutex mu;
    StageOut() = default;
    StageOut(const StageOut&) = delete;
    StageOut& operator=(const StageOut&) = delete;
    ~StageOut() { close(); }
    void close() {
        std::lock_guard<std::mutex> lk(mu);
        if (p) cudaFreeHost(p);
        p = nullptr;
        for (auto& e : ev) {
            if (e) cudaEventDestroy(e);
            e = nullptr;
        }
    }
    cudaError_t open() {
        std::lock_guard<std::mutex> lk(mu);
        if (p) return cudaSuccess;
        for (auto& e : ev)
            if (!e)
                if (const cudaError_t r = cudaEventCreateWithFlags(&e, cudaEventDisableTiming)) return r;
        return cudaMallocHost(&p, 2 * kHalf);
    }
    // `bytes` at `src` (device), as the stream leaves them, to `dst`; returns when they are there.  Without the pinned buffer: the driver's own copy.
    cudaError_t copy(void* dst, const void* src, size_t bytes, cudaStream_t st) {
        std::lock_guard<std::mutex> lk(mu);
        if (!p) {
            const cudaError_t r = cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, st);
            return r ? r : cudaStreamSynchronize(st);
        }
        const size_t n = (bytes + kHalf - 1) / kHalf;
        auto size = [&](size_t i) { return std::min(kHalf, bytes - i * kHalf); };
        auto ask = [&](size_t i) {
            const cudaError_t r = cudaMemcpyAsync(p + (i & 1) * kHalf, static_cast<const uint8_t*>(src) + i * kHalf, size(i), cudaMemcpyDeviceToHost, st);
            return r ? r : cudaEventRecord(ev[i & 1], st);
        };
        for (size_t i = 0; i < n && i < 2; ++i)
            if (const cudaError_t r = ask(i)) return r;
        for (size_t i = 0; i < n; ++i) {
            if (const cudaError_t r = cudaEventSynchronize(ev[i & 1])) return r;
            memcpy(static_cast<uint8_t*>(dst) + i * kHalf, p + (i & 1) * kHalf, size(i));
            if (i + 2 < n)
                if (const cudaError_t r = ask(i + 2)) return r;
        }
        return cudaSuccess;
    }
};

}  // namespace tib
