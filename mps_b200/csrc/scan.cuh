// scan.cuh -- exclusive prefix sum over device arrays (any length).
//
// Template-only, so several translation units can include it.
#pragma once

#include <algorithm>

#include "device.cuh"

namespace mps {

// ---- exclusive scan (any length, recursive over block sums) -------------

// Elements of a thread: 16 where that makes the scan one tile and one launch
// (up to 8,192 elements), 4 above, where a thread's elements are one 16-byte
// piece of memory.  Measured, 16 against 4: 8,193 elements 18.5 / 12.4 us, 3 M
// 38.9 / 24.6, 200 M 1652 / 1031.
constexpr int SCAN_THREADS = 512;
constexpr int SCAN_SHORT = 16, SCAN_LONG = 4;
constexpr int SCAN_ONE = SCAN_THREADS * SCAN_SHORT;    // elements of a scan of one tile
constexpr int SCAN_TILE = SCAN_THREADS * SCAN_LONG;

// Two scans of the same kind in one launch (blockIdx.y names the scan): the
// short ones cost a launch each, whatever their length.  The kernels take it as
// a grid constant: indexed by blockIdx.y, a plain parameter is copied to every
// thread's stack, which made the addition pass 3.7 times slower (50 M elements,
// 516 against 141 us).
template <class T>
struct ScanPair {
    const T *in[2];
    T *out[2], *sums[2], *tot[2];
    const T *offs[2];
    int n[2], nb[2];
};

template <class T, int ITEMS>
__global__ void k_scan_tile(const __grid_constant__ ScanPair<T> p)
{
    constexpr int TILE = SCAN_THREADS * ITEMS;
    __shared__ T warp_tot[SCAN_THREADS / 32];
    int y = blockIdx.y;
    const T *in = p.in[y];
    T *out = p.out[y];
    int n = p.n[y];
    if (blockIdx.x * TILE >= max(n, 1)) return;   // the other scan is longer
    int base = blockIdx.x * TILE + threadIdx.x * ITEMS;
    T v[ITEMS];
    T run = 0;
#pragma unroll
    for (int k = 0; k < ITEMS; k++) {
        T x = (base + k < n) ? in[base + k] : T(0);
        v[k] = run;
        run += x;
    }
    // inclusive warp scan of the per-thread totals
    int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    T inc = run;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        T t = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += t;
    }
    if (lane == 31) warp_tot[w] = inc;
    __syncthreads();
    if (w == 0) {
        T t = (lane < SCAN_THREADS / 32) ? warp_tot[lane] : T(0);
        T ti = t;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            T q = __shfl_up_sync(0xffffffffu, ti, o);
            if (lane >= o) ti += q;
        }
        if (lane < SCAN_THREADS / 32) warp_tot[lane] = ti - t;   // exclusive
        if (lane == SCAN_THREADS / 32 - 1 && p.sums[y]) p.sums[y][blockIdx.x] = ti;
        if (lane == SCAN_THREADS / 32 - 1 && p.tot[y]) *p.tot[y] = ti;   // the only tile
    }
    __syncthreads();
    T off = warp_tot[w] + (inc - run);
#pragma unroll
    for (int k = 0; k < ITEMS; k++)
        if (base + k < n) out[base + k] = v[k] + off;
}

template <class T, int TILE>
__global__ void k_scan_add(const __grid_constant__ ScanPair<T> p)
{
    int y = blockIdx.y;
    if (!p.offs[y]) return;   // a scan of one tile
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < p.n[y]) p.out[y][i] += p.offs[y][i / TILE];
    if (i == 0) p.out[y][p.n[y]] = p.offs[y][p.nb[y]];
}

// out[0..n) = exclusive scan of in[0..n); out[n] = total.  `ws` needs
// scan_workspace(n) elements.
inline size_t scan_workspace(int n)
{
    size_t s = 0;
    int m = n;
    while (m > SCAN_TILE) {
        m = (m - 1) / SCAN_TILE + 1;
        s += 2 * (size_t)m + 1;
    }
    return s + 2;
}

template <class T>
void scan_exclusive2(const T *in, T *out, int n, const T *in2, T *out2, int n2, T *ws, cudaStream_t st);

template <class T, int ITEMS>
void scan_tiles(const T *in, T *out, int n, const T *in2, T *out2, int n2, T *ws, cudaStream_t st)
{
    constexpr int TILE = SCAN_THREADS * ITEMS;
    ScanPair<T> p{};
    int scans = in2 ? 2 : 1, tiles = 1, longest = 0;
    T *w[2] = {ws, ws + scan_workspace(n)};
    for (int y = 0; y < scans; y++) {
        p.in[y] = y ? in2 : in;
        p.out[y] = y ? out2 : out;
        p.n[y] = std::max(y ? n2 : n, 0);
        p.nb[y] = p.n[y] > 0 ? (p.n[y] - 1) / TILE + 1 : 1;
        tiles = std::max(tiles, p.nb[y]);
        if (p.nb[y] == 1) {
            p.tot[y] = p.out[y] + p.n[y];
        } else {
            p.sums[y] = w[y];
            p.offs[y] = w[y] + p.nb[y];   // nb + 1 entries via the recursion
            longest = std::max(longest, p.n[y]);
        }
    }
    launch(k_scan_tile<T, ITEMS>, dim3(tiles, scans), SCAN_THREADS, 0, st, p);
    if (!longest) return;
    for (int y = 0; y < scans; y++)
        if (p.offs[y])
            scan_exclusive2<T>(p.sums[y], const_cast<T *>(p.offs[y]), p.nb[y], nullptr, nullptr, 0,
                               w[y] + 2 * p.nb[y] + 1, st);
    launch(k_scan_add<T, TILE>, dim3((longest - 1) / 256 + 1, scans), 256, 0, st, p);
}

// The scans of a pair (in2 == nullptr: one scan); `ws` holds the workspace of
// both, one after the other.
template <class T>
void scan_exclusive2(const T *in, T *out, int n, const T *in2, T *out2, int n2, T *ws, cudaStream_t st)
{
    if (std::max(n, n2) <= SCAN_ONE) scan_tiles<T, SCAN_SHORT>(in, out, n, in2, out2, n2, ws, st);
    else scan_tiles<T, SCAN_LONG>(in, out, n, in2, out2, n2, ws, st);
}

template <class T>
void scan_exclusive(const T *in, T *out, int n, T *ws, cudaStream_t st)
{
    scan_exclusive2<T>(in, out, n, (const T *)nullptr, (T *)nullptr, 0, ws, st);
}

}  // namespace mps
