// scan.cuh -- exclusive prefix sum over device arrays (any length).
//
// Template-only, so several translation units can include it.
#pragma once

#include <algorithm>

#include "device.cuh"

namespace mps {

// ---- exclusive scan (any length, recursive over block sums) -------------

constexpr int SCAN_THREADS = 512;
constexpr int SCAN_ITEMS = 16;   // one tile, so one launch, up to 8,192 elements
constexpr int SCAN_TILE = SCAN_THREADS * SCAN_ITEMS;

// Two scans of the same kind in one launch (blockIdx.y names the scan): the
// short ones cost a launch each, whatever their length.
template <class T>
struct ScanPair {
    const T *in[2];
    T *out[2], *sums[2], *tot[2];
    const T *offs[2];
    int n[2], nb[2];
};

template <class T>
__global__ void k_scan_tile(ScanPair<T> p)
{
    __shared__ T warp_tot[SCAN_THREADS / 32];
    int y = blockIdx.y;
    const T *in = p.in[y];
    T *out = p.out[y];
    int n = p.n[y];
    if (blockIdx.x * SCAN_TILE >= max(n, 1)) return;   // the other scan is longer
    int base = blockIdx.x * SCAN_TILE + threadIdx.x * SCAN_ITEMS;
    T v[SCAN_ITEMS];
    T run = 0;
#pragma unroll
    for (int k = 0; k < SCAN_ITEMS; k++) {
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
    for (int k = 0; k < SCAN_ITEMS; k++)
        if (base + k < n) out[base + k] = v[k] + off;
}

template <class T>
__global__ void k_scan_add(ScanPair<T> p)
{
    int y = blockIdx.y;
    if (!p.offs[y]) return;   // a scan of one tile
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < p.n[y]) p.out[y][i] += p.offs[y][i / SCAN_TILE];
    if (i == 0) p.out[y][p.n[y]] = p.offs[y][p.nb[y]];
}

// out[0..n) = exclusive scan of in[0..n); out[n] = total.  `ws` needs
// scan_workspace(n) elements.
inline size_t scan_workspace(int n)
{
    size_t s = 0;
    int m = n;
    while (m > SCAN_TILE) {
        m = (m + SCAN_TILE - 1) / SCAN_TILE;
        s += 2 * (size_t)m + 1;
    }
    return s + 2;
}

// The scans of a pair (in2 == nullptr: one scan); `ws` holds the workspace of
// both, one after the other.
template <class T>
void scan_exclusive2(const T *in, T *out, int n, const T *in2, T *out2, int n2, T *ws, cudaStream_t st)
{
    ScanPair<T> p{};
    int scans = in2 ? 2 : 1, tiles = 1, longest = 0;
    bool multi = false;
    T *w[2] = {ws, ws + scan_workspace(n)};
    for (int y = 0; y < scans; y++) {
        p.in[y] = y ? in2 : in;
        p.out[y] = y ? out2 : out;
        p.n[y] = std::max(y ? n2 : n, 0);
        p.nb[y] = std::max(1, (p.n[y] + SCAN_TILE - 1) / SCAN_TILE);
        tiles = std::max(tiles, p.nb[y]);
        if (p.nb[y] == 1) {
            p.tot[y] = p.out[y] + p.n[y];
        } else {
            multi = true;
            p.sums[y] = w[y];
            p.offs[y] = w[y] + p.nb[y];   // nb + 1 entries via the recursion
            longest = std::max(longest, p.n[y]);
        }
    }
    launch(k_scan_tile<T>, dim3(tiles, scans), SCAN_THREADS, 0, st, p);
    if (!multi) return;
    for (int y = 0; y < scans; y++)
        if (p.offs[y])
            scan_exclusive2<T>(p.sums[y], const_cast<T *>(p.offs[y]), p.nb[y], nullptr, nullptr, 0,
                               w[y] + 2 * p.nb[y] + 1, st);
    launch(k_scan_add<T>, dim3((longest + 255) / 256, scans), 256, 0, st, p);
}

template <class T>
void scan_exclusive(const T *in, T *out, int n, T *ws, cudaStream_t st)
{
    scan_exclusive2<T>(in, out, n, (const T *)nullptr, (T *)nullptr, 0, ws, st);
}

}  // namespace mps
