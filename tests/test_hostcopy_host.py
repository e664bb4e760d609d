"""The chunked host transfers (mps_b200/csrc/hostcopy.cuh) on the CPU, against
fakes of the CUDA runtime's calls.

Bytes arrive in both directions at sizes around whole numbers of chunks; where
page-locked memory or an event is refused the pipe is not used and no error is
left behind; where a thread or an allocation is refused, at any point of a
transfer, the bytes still arrive or the call throws, and the process goes on;
an error of a copy is thrown once no copy is left in the buffers.
"""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SOURCE = r'''
#include <pthread.h>

#include <atomic>
#include <cstdio>
#include <cstdlib>
#include <new>
#include <vector>

#include "hostcopy.cuh"

static std::atomic<int> copies_left{1 << 30}, last_error{0}, synced{0};
static int refuse_lock, refuse_event;
static thread_local int allocs_left = 1 << 30;
static std::atomic<int> threads_left{1 << 30};

void *operator new(std::size_t n)
{
    if (allocs_left-- <= 0) throw std::bad_alloc();
    return std::malloc(n);
}
void operator delete(void *p) noexcept { std::free(p); }
void operator delete(void *p, std::size_t) noexcept { std::free(p); }

extern "C" {
int __real_pthread_create(pthread_t *, const pthread_attr_t *, void *(*)(void *), void *);
int __wrap_pthread_create(pthread_t *t, const pthread_attr_t *a, void *(*f)(void *), void *x)
{
    return threads_left-- <= 0 ? 11 : __real_pthread_create(t, a, f, x);
}
static cudaError_t failed(int e) { last_error = e; return (cudaError_t)e; }
cudaError_t cudaMallocHost(void **p, size_t n)
{
    if (refuse_lock) return failed(cudaErrorMemoryAllocation);
    *p = std::malloc(n);
    return cudaSuccess;
}
cudaError_t cudaFreeHost(void *p) { std::free(p); return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned)
{
    if (refuse_event) return failed(cudaErrorMemoryAllocation);
    *e = (cudaEvent_t)std::malloc(1);
    return cudaSuccess;
}
cudaError_t cudaEventDestroy(cudaEvent_t e) { std::free(e); return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { synced++; return cudaSuccess; }
cudaError_t cudaGetDevice(int *d) { *d = 0; return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind, cudaStream_t)
{
    if (copies_left-- <= 0) return failed(cudaErrorInvalidValue);
    std::memcpy(d, s, n);
    return cudaSuccess;
}
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes *a, const void *)
{
    a->type = cudaMemoryTypeUnregistered;
    return cudaSuccess;
}
cudaError_t cudaGetLastError() { int e = last_error.exchange(0); return (cudaError_t)e; }
const char *cudaGetErrorString(cudaError_t) { return "refused"; }
}

static int bad;
static void expect(bool ok, const char *what, long k)
{
    if (!ok) { std::printf("wrong: %s (%ld)\n", what, k); bad++; }
}

// Both directions of `n` bytes; 0 arrived, 1 a call threw, 2 arrived wrong.
static int both(mps::HostPipe &pipe, size_t n, std::vector<char> &a, std::vector<char> &b, std::vector<char> &c)
{
    std::fill(b.begin(), b.end(), 0);
    std::fill(c.begin(), c.end(), 0);
    try {
        pipe.to_device(b.data(), a.data(), n, nullptr);
        pipe.to_host(c.data(), b.data(), n, nullptr);
    } catch (const std::exception &) {
        return 1;
    }
    for (size_t i = 0; i < n; i++)
        if (b[i] != a[i] || c[i] != a[i]) return 2;
    return 0;
}

int main()
{
    const size_t chunk = mps::HostPipe::kChunk, large = mps::HostPipe::kLarge;
    std::vector<char> a(large + 3 * chunk), b(a.size()), c(a.size());
    for (size_t i = 0; i < a.size(); i++) a[i] = (char)(i * 2654435761u >> 13);
    for (int refused = 0; refused < 2; refused++) {
        mps::HostPipe pipe;
        (refused ? refuse_lock : refuse_event) = 1;
        expect(!pipe.wanted(a.data(), large), "pipe without its buffers", refused);
        expect(cudaGetLastError() == cudaSuccess, "error left behind", refused);
        refuse_lock = refuse_event = 0;
        expect(pipe.wanted(a.data(), large) && !pipe.wanted(a.data(), large - 1), "pipe", refused);
        for (size_t n : {large, large + 1, large + chunk - 1, large + 3 * chunk})
            expect(both(pipe, n, a, b, c) == 0, "bytes", (long)n);
    }
    mps::HostPipe pipe;
    expect(pipe.wanted(a.data(), large), "pipe", 0);
    for (int k = 0; k < 12; k++) {
        threads_left = k;
        expect(both(pipe, large + 1, a, b, c) == 0, "bytes with threads refused", k);
        threads_left = 1 << 30;
    }
    for (int k = 0; k < 40; k++) {
        allocs_left = k;
        int r = both(pipe, large + 1, a, b, c);
        allocs_left = 1 << 30;
        expect(r != 2, "bytes with an allocation refused", k);
        expect(both(pipe, large + 1, a, b, c) == 0, "bytes after it", k);
    }
    for (int k = 0; k < 12; k++) {
        copies_left = k;
        synced = 0;
        bool full = both(pipe, large + 1, a, b, c) == 0;
        expect(full == (k >= 10), "a refused copy is thrown", k);
        expect(full || synced >= 2 * mps::HostPipe::kThreads, "copies out of the buffers", k);
        copies_left = 1 << 30;
    }
    return bad ? 1 : 0;
}
'''


def test_transfers_with_refusals(tmp_path):
    nvcc, cxx = shutil.which(os.environ.get("NVCC", "nvcc")), shutil.which(os.environ.get("MPS_CXX", "g++"))
    if not nvcc or not cxx:
        pytest.skip("no compiler")
    src = tmp_path / "pipe.cpp"
    src.write_text(SOURCE)
    exe = str(tmp_path / "pipe")
    inc = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(nvcc))), "include")
    r = subprocess.run([cxx, "-std=c++17", "-O1", "-I" + inc, "-I" + os.path.join(ROOT, "mps_b200", "csrc"),
                        "-Wl,--wrap=pthread_create", "-static-libstdc++", "-o", exe, str(src), "-pthread"],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, (r.stdout, r.stderr)
