// hostcopy.cuh -- large transfers between device memory and a caller's
// pageable host memory.
//
// A copy to or from pageable memory goes through the driver's own staging
// buffers on one host thread (about 17 GB/s on the measured box, a third of
// the link).  Here a few threads each own two page-locked chunks: a thread
// starts the transfer of its next chunk, then moves the bytes of the one
// before between its buffer and the caller's memory, so the link and the
// host copies overlap.  The threads live for one call; the buffers belong to
// the engine, are made on its first large transfer and are given back with
// it.  Where they cannot be made, transfers stay plain copies, and the share
// of a thread that cannot be started is done by the caller's.
#pragma once

#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>
#include <exception>
#include <thread>
#include <vector>

#include "error.cuh"

namespace mps {

class HostPipe {
public:
    static constexpr int kThreads = 6;
    static constexpr size_t kChunk = 1 << 20;       // bytes of a buffer
    static constexpr size_t kLarge = 4 << 20;       // below, one plain copy is as fast

    HostPipe() = default;
    HostPipe(const HostPipe &) = delete;
    HostPipe &operator=(const HostPipe &) = delete;
    ~HostPipe()
    {
        for (auto &e : ev_)
            if (e) cudaEventDestroy(e);
        if (buf_) cudaFreeHost(buf_);
    }

    // Whether a transfer of `bytes` with host memory `p` goes through the pipe.
    bool wanted(const void *p, size_t bytes)
    {
        if (bytes < kLarge) return false;
        cudaPointerAttributes a{};
        if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
            (void)cudaGetLastError();
            return ready();
        }
        return a.type == cudaMemoryTypeUnregistered && ready();
    }

    // `dev` (bytes) to host memory; returns when the bytes are there.
    void to_host(void *host, const void *dev, size_t bytes, cudaStream_t st)
    {
        chunks_to_host((bytes + kChunk - 1) / kChunk, st,
                       [&](size_t c, const void *&src, size_t &n) {
                           src = (const char *)dev + c * kChunk;
                           n = std::min(kChunk, bytes - c * kChunk);
                       },
                       [&](size_t c, const void *buf, size_t n) { std::memcpy((char *)host + c * kChunk, buf, n); });
    }

    // Host memory to `dev`; returns when the host memory has been read and
    // every copy is queued on `st`.
    void to_device(void *dev, const void *host, size_t bytes, cudaStream_t st)
    {
        chunks_to_device((bytes + kChunk - 1) / kChunk, st, [&](size_t c, void *buf, void *&dst) {
            size_t n = std::min(kChunk, bytes - c * kChunk);
            std::memcpy(buf, (const char *)host + c * kChunk, n);
            dst = (char *)dev + c * kChunk;
            return n;
        });
    }

    // Chunks 0..n-1 from the device: `where` names a chunk's source (at most
    // kChunk bytes), `take` moves it out of the buffer.
    template <class Where, class Take>
    void chunks_to_host(size_t n, cudaStream_t st, Where where, Take take)
    {
        run(n, [&](int t, size_t threads) {
            size_t prev = n, prev_bytes = 0;
            int b = 0;
            for (size_t c = t;; c += threads, b ^= 1) {
                size_t bytes = 0;
                if (c < n) {
                    const void *src = nullptr;
                    where(c, src, bytes);
                    ok(cudaMemcpyAsync(buffer(t, b), src, bytes, cudaMemcpyDeviceToHost, st));
                    ok(cudaEventRecord(event(t, b), st));
                }
                if (prev < n) {
                    ok(cudaEventSynchronize(event(t, b ^ 1)));
                    take(prev, (const void *)buffer(t, b ^ 1), prev_bytes);
                }
                if (c >= n) break;
                prev = c;
                prev_bytes = bytes;
            }
        });
    }

    // Chunks to the device: `fill` writes a chunk into the buffer, names its
    // destination and returns its bytes.
    template <class Fill>
    void chunks_to_device(size_t n, cudaStream_t st, Fill fill)
    {
        run(n, [&](int t, size_t threads) {
            int b = 0;
            size_t round = 0;
            for (size_t c = t; c < n; c += threads, b ^= 1, round++) {
                if (round >= 2) ok(cudaEventSynchronize(event(t, b)));   // the buffer's last copy
                void *dst = nullptr;
                size_t bytes = fill(c, buffer(t, b), dst);
                ok(cudaMemcpyAsync(dst, buffer(t, b), bytes, cudaMemcpyHostToDevice, st));
                ok(cudaEventRecord(event(t, b), st));
            }
            for (int q = 0; q < 2; q++)
                if (round > (size_t)q) ok(cudaEventSynchronize(event(t, q)));
        });
    }

private:
    char *buf_ = nullptr;
    cudaEvent_t ev_[2 * kThreads] = {};

    char *buffer(int t, int b) const { return buf_ + (size_t)(2 * t + b) * kChunk; }
    cudaEvent_t event(int t, int b) const { return ev_[2 * t + b]; }

    // Makes the events and the page-locked buffers on first use; false where
    // the system has none to give.
    bool ready()
    {
        if (buf_) return true;
        for (auto &e : ev_)
            if (!e && cudaEventCreateWithFlags(&e, cudaEventDisableTiming) != cudaSuccess) {
                e = nullptr;
                (void)cudaGetLastError();
                return false;
            }
        if (cudaMallocHost((void **)&buf_, 2 * kThreads * kChunk) != cudaSuccess) {
            buf_ = nullptr;
            (void)cudaGetLastError();
            return false;
        }
        return true;
    }

    static void ok(cudaError_t e)
    {
        if (e != cudaSuccess) throw CudaError(std::string("host transfer: ") + cudaGetErrorString(e), MPS_ERR_CUDA);
    }

    // body(t, threads) on each thread, the caller's being thread 0; the first
    // failure is thrown after all have ended and every copy is out of the
    // buffers.  Nothing is thrown past a running thread: what can fail between
    // the first one's start and the last one's end is caught on the spot.
    template <class Body>
    void run(size_t n, Body body)
    {
        if (n == 0) return;
        int dev = 0;
        MPS_CUDA(cudaGetDevice(&dev));
        size_t threads = std::min<size_t>(std::min<size_t>(kThreads, n), std::max(1u, std::thread::hardware_concurrency()));
        std::exception_ptr err[kThreads];
        std::vector<std::thread> pool;
        pool.reserve(threads);
        bool left[kThreads] = {};
        auto work = [&](int t) {
            try {
                if (t) ok(cudaSetDevice(dev));
                body(t, threads);
            } catch (...) {
                err[t] = std::current_exception();
            }
        };
        // a thread the system refuses to start does its share here instead
        for (size_t t = 1; t < threads; t++) {
            try {
                pool.emplace_back(work, (int)t);
            } catch (...) {
                left[t] = true;
            }
        }
        work(0);
        for (size_t t = 1; t < threads; t++)
            if (left[t]) work((int)t);
        for (auto &p : pool) p.join();
        for (size_t t = 0; t < threads; t++)
            if (err[t]) {
                for (auto &e : ev_) (void)cudaEventSynchronize(e);
                std::rethrow_exception(err[t]);
            }
    }
};

}  // namespace mps
