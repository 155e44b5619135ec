// Copies between pageable host memory and the device, staged through pinned
// buffers.
//
// A cudaMemcpy of pageable memory goes through the driver's own staging on one
// host thread, which for arrays so large that the allocator maps fresh pages
// for each also faults those in one by one.  Here the copy is cut into chunks;
// several threads each move their chunks between the caller's memory and their
// own pinned buffers (and take the page faults in parallel), while the DMA of
// other chunks runs: a 256^3 FP32 field (67 MB) goes up in 3.5 ms (5.0) and
// comes down in 4.0 (14.1) on a B200 host of 16 cores.  From 192^3 (28 MB) down,
// where memory is reused without faults, the plain call is as fast or faster
// (1.5 ms up against 2.0; 128^3: 0.51 against 0.59).  Pinned, managed and
// device memory and captured streams take it too, and the per-thread default
// stream, which is another stream in every thread.  The caller's buffer is free
// for reuse (or complete) when the call returns, as with the plain call; the
// DMA keeps the stream's order.
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cstring>
#include <thread>
#include <vector>

namespace gbfk_host {

// While another thread captures a stream (in the global mode), a thread may
// neither allocate nor wait for its own work, or the capture is invalidated.
// Work that touches no captured stream is let off that in the scope of this.
struct Relaxed {
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
    Relaxed() { cudaThreadExchangeStreamCaptureMode(&mode); }
    ~Relaxed() { cudaThreadExchangeStreamCaptureMode(&mode); }
    Relaxed(const Relaxed &) = delete;
    Relaxed &operator=(const Relaxed &) = delete;
};

// The SMs that work on stream s of `device` may use: all of them, or its green
// context's (launches whose CTAs wait for one another must fit them).  0 when
// the device cannot be asked.
inline int stream_sms(int device, cudaStream_t s)
{
    int n = 0;
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, device) != cudaSuccess) return 0;
    if (!s || s == cudaStreamLegacy || s == cudaStreamPerThread) return n;
    auto entry = [](const char *name) -> void * {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPointByVersion(name, &p, 12040, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            return p;
        cudaGetLastError();
        return nullptr;
    };
    const auto of_stream = (CUresult(*)(CUstream, CUgreenCtx *))entry("cuStreamGetGreenCtx");
    const auto resource = (CUresult(*)(CUgreenCtx, CUdevResource *, CUdevResourceType))entry("cuGreenCtxGetDevResource");
    CUgreenCtx green = nullptr;
    CUdevResource r;
    if (of_stream && resource && of_stream((CUstream)s, &green) == CUDA_SUCCESS && green &&
        resource(green, &r, CU_DEV_RESOURCE_TYPE_SM) == CUDA_SUCCESS)
        n = std::min(n, (int)r.sm.smCount);
    return n;
}

class StagedCopy {
public:
    static constexpr size_t kChunk = (size_t)512 << 10;  // bytes of a pinned buffer
    static constexpr int kThreads = 8;                   // two buffers each: 8 MiB at most
    static constexpr size_t kSmall = (size_t)32 << 20;   // below: the plain call
    static constexpr size_t kPerThread = (size_t)2 << 20;

    StagedCopy() = default;
    StagedCopy(const StagedCopy &) = delete;
    StagedCopy &operator=(const StagedCopy &) = delete;

    // frees the buffers (the device current, no copy in flight)
    void release()
    {
        for (int i = 0; i < 2 * kThreads; i++) {
            if (event_[i]) cudaEventDestroy(event_[i]);
            event_[i] = nullptr;
        }
        if (buffers_) cudaFreeHost(buffers_);
        buffers_ = nullptr;
    }

    cudaError_t to_device(void *dev, const void *host, size_t bytes, int device, cudaStream_t s)
    {
        const int threads = plan(host, bytes, s);
        if (threads == 0) return cudaMemcpyAsync(dev, host, bytes, cudaMemcpyHostToDevice, s);
        return run(threads, device, [&](int t) -> cudaError_t {
            for (size_t k = t, turn = 0; k * kChunk < bytes; k += threads, turn++) {
                const int i = 2 * t + (int)(turn & 1);
                const size_t at = k * kChunk, len = std::min(kChunk, bytes - at);
                // the buffer's last DMA, of this call or of one before it
                cudaError_t e = cudaEventSynchronize(event_[i]);
                if (e != cudaSuccess) return e;
                std::memcpy(buffer(i), (const char *)host + at, len);
                e = cudaMemcpyAsync((char *)dev + at, buffer(i), len, cudaMemcpyHostToDevice, s);
                if (e == cudaSuccess) e = cudaEventRecord(event_[i], s);
                if (e != cudaSuccess) return e;
            }
            return cudaSuccess;
        });
    }

    // returns when `host` holds the data (the plain call: when the stream has
    // run so far, as its callers synchronise it)
    cudaError_t to_host(void *host, const void *dev, size_t bytes, int device, cudaStream_t s)
    {
        const int threads = plan(host, bytes, s);
        if (threads == 0) return cudaMemcpyAsync(host, dev, bytes, cudaMemcpyDeviceToHost, s);
        return run(threads, device, [&](int t) -> cudaError_t {
            const size_t chunks = (bytes + kChunk - 1) / kChunk;
            auto start = [&](size_t k, int i) {
                const size_t at = k * kChunk, len = std::min(kChunk, bytes - at);
                cudaError_t e = cudaMemcpyAsync(buffer(i), (const char *)dev + at, len, cudaMemcpyDeviceToHost, s);
                return e == cudaSuccess ? cudaEventRecord(event_[i], s) : e;
            };
            cudaError_t e = cudaSuccess;
            for (int j = 0; j < 2 && e == cudaSuccess; j++) {
                // a buffer may still feed an upload
                e = cudaEventSynchronize(event_[2 * t + j]);
                if (e == cudaSuccess && t + (size_t)j * threads < chunks) e = start(t + (size_t)j * threads, 2 * t + j);
            }
            size_t turn = 0;
            for (size_t k = t; k < chunks && e == cudaSuccess; k += threads, turn++) {
                const int i = 2 * t + (int)(turn & 1);
                e = cudaEventSynchronize(event_[i]);
                if (e != cudaSuccess) break;
                const size_t at = k * kChunk, len = std::min(kChunk, bytes - at);
                std::memcpy((char *)host + at, buffer(i), len);
                if (k + 2 * (size_t)threads < chunks) e = start(k + 2 * (size_t)threads, i);
            }
            return e;
        });
    }

private:
    char *buffers_ = nullptr;  // one pinned allocation (16 of them took 2 ms longer)
    cudaEvent_t event_[2 * kThreads] = {};

    char *buffer(int i) const { return buffers_ + i * kChunk; }

    // threads for a copy of pageable memory; 0: the plain call
    int plan(const void *host, size_t bytes, cudaStream_t s)
    {
        if (bytes < kSmall || s == cudaStreamPerThread) return 0;
        cudaStreamCaptureStatus st = cudaStreamCaptureStatusNone;
        if (cudaStreamIsCapturing(s, &st) != cudaSuccess || st != cudaStreamCaptureStatusNone) {
            cudaGetLastError();
            return 0;
        }
        cudaPointerAttributes a;
        if (cudaPointerGetAttributes(&a, host) != cudaSuccess) {
            cudaGetLastError();
            return 0;
        }
        if (a.type != cudaMemoryTypeUnregistered) return 0;
        Relaxed relaxed;
        const int cores = std::max(1, (int)std::thread::hardware_concurrency() / 2);
        const int threads = (int)std::min<size_t>({(size_t)kThreads, (size_t)cores, 1 + (bytes - 1) / kPerThread});
        if (!buffers_ && cudaHostAlloc((void **)&buffers_, 2 * kThreads * kChunk, cudaHostAllocDefault) != cudaSuccess) {
            buffers_ = nullptr;
            cudaGetLastError();
            return 0;
        }
        for (int i = 0; i < 2 * threads; i++) {
            if (!event_[i] && cudaEventCreateWithFlags(&event_[i], cudaEventDisableTiming) != cudaSuccess) {
                event_[i] = nullptr;
                cudaGetLastError();
                return 0;
            }
        }
        return threads;
    }

    // f(0) .. f(threads - 1), the first one here; the first error
    template <typename F>
    static cudaError_t run(int threads, int device, F &&f)
    {
        std::vector<std::thread> pool;
        std::vector<cudaError_t> err(threads, cudaSuccess);
        std::vector<char> mine(threads, 1);
        mine[0] = 1;
        for (int t = 1; t < threads; t++) {
            try {
                pool.emplace_back([&, t] {
                    Relaxed relaxed;
                    err[t] = cudaSetDevice(device);
                    if (err[t] == cudaSuccess) err[t] = f(t);
                });
                mine[t] = 0;
            } catch (...) {  // no thread to be had: its share is done here
                break;
            }
        }
        {
            Relaxed relaxed;
            for (int t = 0; t < threads; t++)
                if (mine[t]) err[t] = f(t);
        }
        for (auto &p : pool) p.join();
        for (cudaError_t e : err)
            if (e != cudaSuccess) return e;
        return cudaSuccess;
    }
};

}  // namespace gbfk_host
