// k_sort.cuh -- cell binning, counting sort and reorder (the neighbour search).
//
// Replaces the reference's cell linked list (neighbor_search.c:146-240).  The
// reference prepends particles to per-cell chains, so its neighbour lists
// visit a cell's particles in descending index order.  Here the particles
// are physically reordered every step by (cell, descending reference index):
// a histogram of cell counts, an exclusive scan, an atomic scatter into the
// cell's slot range, and a per-cell rank by index that makes the order within
// a cell deterministic.  Particles that are not binned (ghosts, outside the
// grid) go to a trailing bucket in their previous relative order.
#pragma once

#include "device.cuh"
#include "scan.cuh"

namespace mps {

// ---- binning --------------------------------------------------------------

template <int D>
__global__ void k_bin(State<D> s, Grid<D> g, int n, int *__restrict__ kcell,
                      int *__restrict__ count, int *__restrict__ excl)
{
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    int c = -1;
    if (s.type[i] != GHOST) {
        double p[D];
        load_vec<D>(p, s.pos, i);
        c = cell_of_pos<D>(g, p);
    }
    kcell[i] = c;
    excl[i] = (c < 0);
    if (c >= 0) atomicAdd(&count[c], 1);
}

__global__ void k_scatter(int n, int total, const int *__restrict__ kcell, const int *__restrict__ start,
                          int *__restrict__ cursor, const int *__restrict__ exoff,
                          int *__restrict__ tmp, int *__restrict__ perm)
{
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    int c = kcell[i];
    if (c >= 0) {
        int slot = start[c] + atomicAdd(&cursor[c], 1);
        tmp[slot] = i;
    } else {
        perm[start[total] + exoff[i]] = i;
    }
}

// Position within the cell = number of cell members with a larger
// reference index (descending order, as the reference's chains).
__global__ void k_rank(const int *__restrict__ nbinned, const int *__restrict__ tmp, const int *__restrict__ kcell,
                       const int *__restrict__ start, const int *__restrict__ id, int *__restrict__ perm)
{
    int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= *nbinned) return;
    int i = tmp[t];
    int c = kcell[i];
    int me = id[i];
    int b = start[c], e = start[c + 1];
    int r = 0;
    for (int u = b; u < e; u++) r += (id[tmp[u]] > me);
    perm[b + r] = i;
}

template <int D>
__global__ void k_gather(State<D> dst, State<D> src, const int *__restrict__ perm,
                         const int *__restrict__ kcell, int n, int *__restrict__ where, Grid<D> g,
                         float4 *__restrict__ kf)
{
    int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= n) return;
    int i = perm[q];
    float f[4] = {0.0f, 0.0f, 0.0f, 0.0f};   // the key in cell units, as k_key_cells
#pragma unroll
    for (int d = 0; d < D; d++) {
        double x = src.pos[d][i];
        f[d] = (float)((x - g.origin[d]) * g.cs_inv);
        dst.pos[d][q] = x;
        dst.key[d][q] = x;
        dst.vel[d][q] = src.vel[d][i];
        dst.acc[d][q] = src.acc[d][i];
    }
    dst.p[q] = src.p[i];
    dst.n[q] = src.n[i];
    dst.type[q] = src.type[i];
    dst.surf[q] = src.surf[i];
    dst.ncount[q] = src.ncount[i];
    int id = src.id[i];
    dst.id[q] = id;
    dst.cell[q] = kcell[i];
    where[id] = q;
    kf[q] = make_float4(f[0], f[1], f[2], f[3]);
}

// Reorder to reference order (engine index == reference index).
template <int D>
__global__ void k_unsort(State<D> dst, State<D> src, const int *__restrict__ where, int n)
{
    int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= n) return;
    int q = where[r];
#pragma unroll
    for (int d = 0; d < D; d++) {
        dst.pos[d][r] = src.pos[d][q];
        dst.key[d][r] = src.key[d][q];
        dst.vel[d][r] = src.vel[d][q];
        dst.acc[d][r] = src.acc[d][q];
    }
    dst.p[r] = src.p[q];
    dst.n[r] = src.n[q];
    dst.type[r] = src.type[q];
    dst.surf[r] = src.surf[q];
    dst.ncount[r] = src.ncount[q];
    dst.id[r] = r;
    dst.cell[r] = -1;
}

// ---- compact lists of the cell structure ---------------------------------------
//
// Every operator of a step visits the same neighbours: a seventh of the
// candidates in the 3^D cells.  Testing them in each operator costs a pass
// over all candidates in FP64 and, worse, runs the operator's body (square
// root and division) for every candidate that any lane of the warp accepts.
// The lists are built once per sort and the operators run over accepted
// neighbours only.
//
// The test is bit for bit that of CellSource.  Positions in cell units are
// first compared in FP32 (one 16-byte load per candidate and half the issue
// cost); only a candidate within `band` of the radius, where FP32 cannot
// decide, is tested in FP64.

// Sort keys in cell units, FP32.
template <int D>
__global__ void k_key_cells(State<D> s, Grid<D> g, int n, float4 *__restrict__ kf)
{
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    float f[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
    for (int d = 0; d < D; d++) f[d] = (float)((s.key[d][i] - g.origin[d]) * g.cs_inv);
    kf[i] = make_float4(f[0], f[1], f[2], f[3]);
}

// Lists of the current structure: idx[(slice * pitch + k) * 32 + lane], cnt
// the number of neighbours (those past `pitch` are counted, not stored).
template <int D>
__global__ void k_nbr_list(CellSource<D> src, int n, const float4 *__restrict__ kf, float band, int pitch,
                           int *__restrict__ idx, int *__restrict__ cnt)
{
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    int c = src.cell[i];
    int k = 0;
    if (c >= 0) {
        const Grid<D> &g = src.g;
        float4 me = kf[i];
        double ki[D];
#pragma unroll
        for (int d = 0; d < D; d++) ki[d] = src.key[d][i];
        int cc[D];
        int rem = c;
#pragma unroll
        for (int d = 0; d < D; d++) { cc[d] = rem % g.dims[d]; rem /= g.dims[d]; }
        int x0 = cc[0] > 0 ? cc[0] - 1 : 0;
        int x1 = cc[0] < g.dims[0] - 1 ? cc[0] + 1 : g.dims[0] - 1;
        int y0 = cc[1] > 0 ? cc[1] - 1 : 0;
        int y1 = cc[1] < g.dims[1] - 1 ? cc[1] + 1 : g.dims[1] - 1;
        int z0 = 0, z1 = 0;
        if (D == 3) {
            z0 = cc[D - 1] > 0 ? cc[D - 1] - 1 : 0;
            z1 = cc[D - 1] < g.dims[D - 1] - 1 ? cc[D - 1] + 1 : g.dims[D - 1] - 1;
        }
        int *out = idx + (size_t)(i >> 5) * 32 * pitch + (i & 31);
        for (int z = z0; z <= z1; z++) {
            for (int y = y0; y <= y1; y++) {
                int base = (D == 3) ? (z * g.dims[1] + y) * g.dims[0] : y * g.dims[0];
                int t0 = g.start[base + x0], t1 = g.start[base + x1 + 1];
#pragma unroll 4
                for (int t = t0; t < t1; t++) {
                    float4 o = __ldg(&kf[t]);
                    float dx = o.x - me.x, dy = o.y - me.y;
                    float d2 = fmaf(dx, dx, dy * dy);
                    if (D == 3) {
                        float dz = o.z - me.z;
                        d2 = fmaf(dz, dz, d2);
                    }
                    if (d2 < 1.0f + band) {
                        bool hit = t != i;
                        if (d2 >= 1.0f - band) {
                            double kt[D];
#pragma unroll
                            for (int d = 0; d < D; d++) kt[d] = src.key[d][t];
                            hit = hit && dist2<D>(ki, kt) < src.re2;
                        }
                        if (hit) {
                            if (k < pitch) out[(size_t)k * 32] = t;
                            k++;
                        }
                    }
                }
            }
        }
    }
    cnt[i] = k;
}

// The same lists with NBR_LANES lanes per particle, for systems too small to
// fill the device with a thread each: the lanes take consecutive candidates
// of a run and a ballot keeps the accepted ones in order.
constexpr int NBR_LANES = 8;

template <int D>
__global__ void k_nbr_list_lanes(CellSource<D> src, int n, const float4 *__restrict__ kf, float band, int pitch,
                                 int *__restrict__ idx, int *__restrict__ cnt)
{
    int i = (blockIdx.x * blockDim.x + threadIdx.x) / NBR_LANES;
    int lane = threadIdx.x & 31, l = lane % NBR_LANES;
    unsigned group = ((1u << NBR_LANES) - 1u) << (lane - l);
    if (i >= n) return;   // whole groups
    int c = src.cell[i];
    int k = 0;
    if (c >= 0) {
        const Grid<D> &g = src.g;
        float4 me = kf[i];
        double ki[D];
#pragma unroll
        for (int d = 0; d < D; d++) ki[d] = src.key[d][i];
        int cc[D];
        int rem = c;
#pragma unroll
        for (int d = 0; d < D; d++) { cc[d] = rem % g.dims[d]; rem /= g.dims[d]; }
        int x0 = cc[0] > 0 ? cc[0] - 1 : 0;
        int x1 = cc[0] < g.dims[0] - 1 ? cc[0] + 1 : g.dims[0] - 1;
        int y0 = cc[1] > 0 ? cc[1] - 1 : 0;
        int y1 = cc[1] < g.dims[1] - 1 ? cc[1] + 1 : g.dims[1] - 1;
        int z0 = 0, z1 = 0;
        if (D == 3) {
            z0 = cc[D - 1] > 0 ? cc[D - 1] - 1 : 0;
            z1 = cc[D - 1] < g.dims[D - 1] - 1 ? cc[D - 1] + 1 : g.dims[D - 1] - 1;
        }
        int *out = idx + (size_t)(i >> 5) * 32 * pitch + (i & 31);
        for (int z = z0; z <= z1; z++) {
            for (int y = y0; y <= y1; y++) {
                int base = (D == 3) ? (z * g.dims[1] + y) * g.dims[0] : y * g.dims[0];
                int t0 = g.start[base + x0], t1 = g.start[base + x1 + 1];
#pragma unroll 2
                for (int tb = t0; tb < t1; tb += NBR_LANES) {
                    int t = tb + l;
                    bool hit = false;
                    if (t < t1) {
                        float4 o = __ldg(&kf[t]);
                        float dx = o.x - me.x, dy = o.y - me.y;
                        float d2 = fmaf(dx, dx, dy * dy);
                        if (D == 3) {
                            float dz = o.z - me.z;
                            d2 = fmaf(dz, dz, d2);
                        }
                        hit = d2 < 1.0f + band && t != i;
                        if (hit && d2 >= 1.0f - band) {
                            double kt[D];
#pragma unroll
                            for (int d = 0; d < D; d++) kt[d] = src.key[d][t];
                            hit = dist2<D>(ki, kt) < src.re2;
                        }
                    }
                    unsigned m = __ballot_sync(group, hit) >> (lane - l);
                    int at = k + __popc(m & ((1u << l) - 1u));
                    if (hit && at < pitch) out[(size_t)at * 32] = t;
                    k += __popc(m);
                }
            }
        }
    }
    if (l == 0) cnt[i] = k;
}

// Neighbour list in the reference's layout (rows by reference index,
// entries as reference indices, reference order).  Row r starts at
// out_nb[r * pitch]; rows longer than max_nb raise the overflow flag.
template <int D>
__global__ void k_build_list(NbrSource<D> src, const int *__restrict__ id, int n, int max_nb, int pitch,
                             int *__restrict__ out_nb, int *__restrict__ out_cnt, unsigned *err)
{
    int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= n) return;
    int row = id[q];
    int cnt = 0;
    size_t base = (size_t)row * (size_t)pitch;
    src.for_each(q, [&](int t) {
        if (cnt < pitch && out_nb) out_nb[base + cnt] = id[t];
        cnt++;
    });
    if (cnt > max_nb) {
        atomicOr(err, ERR_NEIGHBOR_OVERFLOW);
        cnt = max_nb;
    }
    out_cnt[row] = cnt;
}

// Entries of an uploaded list outside the particles are reported.
__global__ void k_check_list(int used, int n, int *__restrict__ idx, unsigned *err)
{
    int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= used) return;
    int j = idx[k];
    if (j < 0 || j >= n) {
        atomicOr(err, ERR_LIST_MISMATCH);
        idx[k] = 0;
    }
}

// Rows of a pitched host list (already on the device) into CSR.
__global__ void k_compact_list(const int *__restrict__ rows, int pitch, const int *__restrict__ cnt,
                               const int *__restrict__ ptr, int n, int *__restrict__ idx, unsigned *err)
{
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    int c = cnt[i], o = ptr[i];
    const int *r = rows + (size_t)i * pitch;
    for (int k = 0; k < c; k++) {
        int j = r[k];
        if (j < 0 || j >= n) { atomicOr(err, ERR_LIST_MISMATCH); j = 0; }
        idx[o + k] = j;
    }
}

// The same compaction read straight from a caller's list in page-locked host
// memory (device-addressable under unified addressing): one warp per row, the
// lanes striding over the row's count, so only the used entries cross the
// host link, in 128-byte runs.
__global__ void k_gather_host_list(const int *__restrict__ rows, int pitch, const int *__restrict__ cnt,
                                   const int *__restrict__ ptr, int n, int *__restrict__ idx, unsigned *err)
{
    long long w = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    int lane = threadIdx.x & 31;
    if (w >= n) return;
    int c = min(cnt[w], pitch), o = ptr[w];
    const int *r = rows + (size_t)w * pitch;
    for (int k = lane; k < c; k += 32) {
        int j = r[k];
        if (j < 0 || j >= n) { atomicOr(err, ERR_LIST_MISMATCH); j = 0; }
        idx[o + k] = j;
    }
}

template <int D>
__global__ void k_cell_ref_order(const int *__restrict__ cell, const int *__restrict__ id, int n, int *out)
{
    int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q < n) out[id[q]] = cell[q];
}

// Compare a caller's list (CSR by reference index, reference indices) with
// the cell structure's list, entry by entry.
template <int D>
__global__ void k_compare_list(NbrSource<D> src, const int *__restrict__ id, int n,
                               const int *__restrict__ lptr, const int *__restrict__ lidx, unsigned *err)
{
    int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= n) return;
    int row = id[q];
    int k = lptr[row], e = lptr[row + 1];
    bool bad = false;
    src.for_each(q, [&](int t) {
        if (k >= e || lidx[k] != id[t]) bad = true;
        k++;
    });
    if (k != e) bad = true;
    if (bad) atomicOr(err, ERR_LIST_MISMATCH);
}

}  // namespace mps
