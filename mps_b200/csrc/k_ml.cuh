// k_ml.cuh -- multilevel preconditioner of the PPE solve: point Jacobi on the
// unknowns plus a coarse-grid correction through nested trilinear (2-D:
// bilinear) grids.
//
// The PPE is a graph Laplacian whose every row couples all unknowns within
// the interaction radius, so one Jacobi step removes error that varies inside
// a cell, and what an incomplete factorisation leaves slow is the smooth part,
// whose iteration count grows with the number of cells across the fluid.  A
// coarse grid with a node on every corner of the cell grid represents that
// part: interpolation P from the 2^D corners of a row's own cell to the row
// (the weights are the row's position in its cell), Galerkin operator
// A_1 = P^T A P, and further grids by doubling the spacing, A_{l+1} =
// I^T A_l I.  The preconditioner is the sum
//     z = D^-1 r + P V(P^T r),
// V a symmetric V-cycle over the grids (one l1-Jacobi step before and after
// each coarse correction, an explicit inverse on the coarsest grid), or, with
// `additive`, V(b) = s D_1^-1 b + I V_2(I^T b) (no product on the first grid).
// From the first grid of at most ML_DENSE nodes on, the V-cycle is one dense
// symmetric matrix, formed once per solve from the coarsest grid up: a chain
// of dependent steps, each a fraction of a microsecond of work, becomes one
// product.
// Both are symmetric and positive definite: D_l1 = diag(sum_j |a_ij|) >= A_l,
// so an l1-Jacobi step of relaxation below 2 always contracts (Baker, Falgout,
// Kolev, Yang 2011, "Multigrid smoothers for ultra-parallel computing"), and
// the sum with D^-1 is definite even where P has no reach.  CG iterations then
// do not depend on the resolution.
//
// Everything is FP64 in both precision forms, except the rows' positions in
// their cells, which are held in FP32: they define P, and the same numbers
// are used in P, P^T and A_1.
//
// Measured against the block-colour IC(0) (B200, the solve of a step): 3-D dam
// break of 2.85 M particles, mixed form, 619 -> 30 iterations, 747 -> 21.6 ms;
// 1.17 M particles in FP64, 507 -> 44, 333 -> 14.6 ms; 117 k particles, 173 ->
// 40, 31.1 -> 2.6 ms; 2,158 particles in 2-D, 92 -> 36, 6.3 -> 0.43 ms.  What
// remains of an iteration is the product with the matrix (HBM) at large sizes
// and the chain of dependent launches at small ones.  With a V-cycle of
// separate residual, restriction and interpolation steps the same solves took
// 28.6, 18.8, 5.0 and 1.8 ms; that V-cycle in one cluster of 8 CTAs, with C and
// C^T but the matrix on every grid, 26.3, 20.2, 5.5 and 1.2 ms (a step of a
// few index operations and dependent loads takes 2-7 us however few nodes it
// has), so the small grids became one dense product.
//
// No sum uses an atomic; every reduction runs in a fixed order, so results
// are the same bits on every run.
#pragma once

#include "device.cuh"
#include "k_ppe.cuh"

namespace mps {

constexpr int ML_MAXL = 26;       // grids at most: 2^30 cells, even in one direction, reach the coarsest size
constexpr int ML_BOX = 64;        // the grids end when their box holds at most this many nodes ...
// ... and a solve's at the first with at most this many nodes in use, whose
// inverse starts the dense V-cycle (128 took 175 us to invert, a pivot at a
// time; one more grid costs 30).
constexpr int ML_COARSEST = 64;
// Nodes up to which a grid's V-cycle is held as a dense matrix: 8 MB at most,
// read from L2 in about 3 us, against three dependent launches per grid for
// the steps it replaces.
constexpr int ML_DENSE = 1024;
// Relaxation of the l1-Jacobi steps (below 2 contracts); measured on the dam
// break at l0 = 0.01: 42 iterations at 1.0, 40 at 1.4 to 1.9.
constexpr double ML_OMEGA = 1.5;
// Weight of the additive first grid's D_1^-1 (D_1 the true diagonal).
constexpr double ML_ADD = 0.45;

constexpr int ML_PAD = 4;   // a C row reaches 3 beyond the node under its own, which may be 1 outside

template <int D>
struct MlDim {
    static constexpr int NC = 1 << D;                  // corners of a cell
    static constexpr int CELLS = D == 3 ? 27 : 9;      // a cell and its neighbours
    static constexpr int W4 = D == 3 ? 64 : 16;        // nodes of a cell and its neighbours (4 per axis)
    static constexpr int ST = D == 3 ? 125 : 25;       // stencil (5 per axis)
    static constexpr int STP = D == 3 ? 128 : 32;      // its stride in memory
    static constexpr int W7 = D == 3 ? 343 : 49;       // nodes within 3 of a node (7 per axis)
    static constexpr int W7P = D == 3 ? 352 : 64;      // their stride in memory
};

// One grid.  Vectors live on the whole box of nodes with a margin of ML_PAD
// nodes per side that stays zero, so a stencil never leaves its grid; the
// grids follow one another in one array.  at(x, y, z) = base + x + s1 y + s2 z.
struct MlGrid {
    int n[3];
    int s1, s2;
    int base;    // index of node (0, 0, 0)
    int first;   // start of the grid's box (margin included)
    int size;
};

__host__ __device__ __forceinline__ int ml_at(const MlGrid &g, int x, int y, int z)
{
    return g.base + x + g.s1 * y + g.s2 * z;
}

// Coordinates of a padded index of a grid.
template <int D>
__device__ __forceinline__ void ml_coords(const MlGrid &g, int idx, int *c)
{
    int rel = idx - g.first;
    if (D == 3) {
        c[2] = rel / g.s2 - ML_PAD;
        rel %= g.s2;
    } else {
        c[2] = 0;
    }
    c[1] = rel / g.s1 - ML_PAD;
    c[0] = rel % g.s1 - ML_PAD;
}

// Offset of stencil entry k (x fastest, -2..2 per axis).
template <int D>
__device__ __forceinline__ int ml_offset(const MlGrid &g, int k)
{
    int o = k % 5 - 2 + g.s1 * ((k / 5) % 5 - 2);
    if (D == 3) o += g.s2 * (k / 25 - 2);
    return o;
}

struct MlLevels {
    MlGrid g[ML_MAXL];
    int lo[ML_MAXL + 1];   // node numbers of the grids: grid l holds [lo[l], lo[l+1])
    int nl;
};

// ---- nodes -----------------------------------------------------------------------

// Corners of every active cell; `cnode` gets the cell's lowest corner.
template <int D>
__global__ void k_ml_flag1(int nact, const int *__restrict__ acells, Grid<D> cg, MlGrid g, int *__restrict__ flag,
                           int *__restrict__ cnode)
{
    int kk = blockIdx.x * blockDim.x + threadIdx.x;
    if (kk >= nact) return;
    int c[3] = {0, 0, 0};
    int rem = acells[kk];
#pragma unroll
    for (int d = 0; d < D; d++) { c[d] = rem % cg.dims[d]; rem /= cg.dims[d]; }
    int o = ml_at(g, c[0], c[1], c[2]);
    cnode[kk] = o;
#pragma unroll
    for (int k = 0; k < (1 << D); k++) flag[o + (k & 1) + g.s1 * ((k >> 1) & 1) + g.s2 * (k >> 2)] = 1;
}

// Parents of the flagged nodes of grid f on grid c.
template <int D>
__global__ void k_ml_flag_up(MlGrid f, MlGrid c, int *__restrict__ flag)
{
    int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= f.n[0] * f.n[1] * f.n[2]) return;
    int x = t % f.n[0], y = (t / f.n[0]) % f.n[1], z = t / (f.n[0] * f.n[1]);
    if (!flag[ml_at(f, x, y, z)]) return;
    for (int pz = z / 2; pz <= (D == 3 ? (z + 1) / 2 : 0); pz++)
        for (int py = y / 2; py <= (y + 1) / 2; py++)
            for (int px = x / 2; px <= (x + 1) / 2; px++) flag[ml_at(c, px, py, pz)] = 1;
}

// Node numbers: act[number] = index, amap[index] = number or -1.
__global__ void k_ml_compact(int total, const int *__restrict__ flag, const int *__restrict__ pos,
                             int *__restrict__ act, int *__restrict__ amap)
{
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= total) return;
    int f = flag[i];
    amap[i] = f ? pos[i] : -1;
    if (f) act[pos[i]] = i;
}

struct MlFirsts {
    int v[ML_MAXL + 1];
};

__global__ void k_ml_sizes(MlFirsts first, int nl, const int *__restrict__ pos, int *__restrict__ out)
{
    int l = threadIdx.x;
    if (l <= nl) out[l] = pos[first.v[l]];
}

// The active cells around every node of the first grid: cell k has the node
// as its corner k; -1 if it holds no unknown.
template <int D>
__global__ void k_ml_node_cells(int na, const int *__restrict__ act, MlGrid g, Grid<D> cg,
                                const int *__restrict__ cellact, int *__restrict__ ncell)
{
    int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= na) return;
    int c[3];
    ml_coords<D>(g, act[t], c);
#pragma unroll
    for (int k = 0; k < (1 << D); k++) {
        int lin = 0;
        bool in = true;
#pragma unroll
        for (int d = D - 1; d >= 0; d--) {
            int x = c[d] - ((k >> d) & 1);
            in = in && x >= 0 && x < cg.dims[d];
            lin = lin * cg.dims[d] + x;
        }
        ncell[(size_t)k * na + t] = in ? cellact[lin] : -1;
    }
}

// cellact[cell] = number of the active cell, -1 otherwise.
__global__ void k_ml_cellact(int total, const int *__restrict__ ccells, const int *__restrict__ ucol,
                             const int *__restrict__ apos, int *__restrict__ cellact)
{
    int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k < total) cellact[ccells[k]] = ucol[k] > 0 ? apos[k] : -1;
}

// ---- components without a source ------------------------------------------------------
//
// A connected set of unknowns whose right-hand side is zero and which no
// known pressure bounds (a dry wall region away from the fluid) has a
// singular block and the solution CG gives it from a zero start: zero, as
// long as nothing couples it to the rest.  Interpolation would (a coarse node
// may reach such a set and the fluid at once), so its rows are left out of P.
// The sets are found by union-find over the nonzero entries; every tree is
// rooted at its smallest row, so the result does not depend on the order.

__device__ __forceinline__ int uf_find(int *parent, int i)
{
    int p = __ldcg(&parent[i]);
    while (p != i) {
        int g = __ldcg(&parent[p]);
        if (g != p) parent[i] = g;   // halving; any ancestor is a valid parent
        i = p;
        p = g;
    }
    return i;
}

__global__ void k_uf_init(int n, const int *__restrict__ row_ptr, const int *__restrict__ diagpos,
                          const int *__restrict__ col, const double *__restrict__ A, int *__restrict__ parent,
                          int *__restrict__ keep)
{
    int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= n) return;
    int p = r;
    for (int q = row_ptr[r]; q < diagpos[r]; q++)
        if (A[q] != 0.0) {
            p = col[q];
            break;
        }
    parent[r] = p;
    keep[r] = 0;
}

// Joins the trees of rows i and j: the larger root goes under the smaller.
__device__ __forceinline__ void uf_join(int *parent, int i, int j)
{
    int a = uf_find(parent, i), b = uf_find(parent, j);
    while (a != b) {
        if (a < b) { int t = a; a = b; b = t; }
        int old = atomicCAS(&parent[a], a, b);
        if (old == a) break;
        a = uf_find(parent, old);
        b = uf_find(parent, b);
    }
}

// Most rows belong to one tree after a few of their entries (Sutton, Ben-Nun,
// Barak 2018, "Optimizing parallel graph connectivity computation via
// subgraph sampling"): three entries of every row first, then all entries of
// the rows that are not in the first row's tree.
__global__ void k_uf_sample(int n, const int *__restrict__ row_ptr, const int *__restrict__ diagpos,
                            const int *__restrict__ col, const double *__restrict__ A, int *parent)
{
    int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= n) return;
    int a = row_ptr[r], d = diagpos[r], e = row_ptr[r + 1];
    int q[3] = {(a + d) / 2, d - 1, e - 1};
#pragma unroll
    for (int k = 0; k < 3; k++)
        if (q[k] >= a && q[k] != d && A[q[k]] != 0.0) uf_join(parent, r, col[q[k]]);
}

__global__ void k_uf_flatten(int n, int *parent)
{
    int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r < n) parent[r] = uf_find(parent, r);
}

// Eight lanes per row.
__global__ void k_uf_hook(int n, const int *__restrict__ row_ptr, const int *__restrict__ col,
                          const double *__restrict__ A, int *parent)
{
    int r = (int)((blockIdx.x * (size_t)blockDim.x + threadIdx.x) >> 3);
    if (r >= n || uf_find(parent, r) == uf_find(parent, 0)) return;
    for (int q = row_ptr[r] + (threadIdx.x & 7); q < row_ptr[r + 1]; q += 8)
        if (A[q] != 0.0) uf_join(parent, r, col[q]);
}

__global__ void k_uf_keep(int n, const double *__restrict__ b, const unsigned char *__restrict__ bounded,
                          int *parent, int *__restrict__ keep)
{
    int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= n) return;
    if (b[r] != 0.0 || bounded[r]) keep[uf_find(parent, r)] = 1;
}

// ---- rows ------------------------------------------------------------------------------

// Position of every row in its cell (FP32, [axis][row]; a first coordinate of
// -1 marks a row left out of P) and the inverse diagonal, with the
// factorisation's rule for a pivot that is not positive
// (pressure_solver.c:200).
template <int D>
__global__ void k_ml_rows(State<D> s, Grid<D> cg, int n_eq, int stride, const int *__restrict__ part_of_row,
                          const int *__restrict__ diagpos, const double *__restrict__ A, int *parent,
                          const int *__restrict__ keep, float *__restrict__ frac, double *__restrict__ dinv)
{
    int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= n_eq) return;
    int i = part_of_row[r];
    int rem = s.cell[i];
    bool in = keep[uf_find(parent, r)] != 0;
#pragma unroll
    for (int d = 0; d < D; d++) {
        int c = rem % cg.dims[d];
        rem /= cg.dims[d];
        double t = (s.pos[d][i] - cg.origin[d]) * cg.cs_inv - (double)c;
        float f = (float)fmin(fmax(t, 0.0), 1.0);
        frac[(size_t)d * stride + r] = (d == 0 && !in) ? -1.0f : f;
    }
    double a = A[diagpos[r]];
    dinv[r] = a > 0.0 ? 1.0 / a : (a <= 0.0 ? 1.0e30 : a);   // NaN stays NaN
}

// Weights of a position in a cell on the cell's corners, all zero for a row
// left out of P.
template <int D>
__device__ __forceinline__ void ml_weights_of(const float *f32, double *w)
{
    double f[D];
#pragma unroll
    for (int d = 0; d < D; d++) f[d] = (double)f32[d];
    double on = f[0] < 0.0 ? 0.0 : 1.0;
    double x0 = on * (1.0 - f[0]), x1 = on * f[0];
    double y0 = 1.0 - f[1], y1 = f[1];
    w[0] = x0 * y0;
    w[1] = x1 * y0;
    w[2] = x0 * y1;
    w[3] = x1 * y1;
    if (D == 3) {
        double z1 = f[D - 1], z0 = 1.0 - z1;
#pragma unroll
        for (int k = 0; k < 4; k++) {
            w[(k + 4) & ((1 << D) - 1)] = w[k] * z1;
            w[k] = w[k] * z0;
        }
    }
}

template <int D>
__device__ __forceinline__ void ml_weights(const float *__restrict__ frac, int stride, int r, double *w)
{
    float f[D];
#pragma unroll
    for (int d = 0; d < D; d++) f[d] = __ldg(&frac[(size_t)d * stride + r]);
    ml_weights_of<D>(f, w);
}

// ---- Galerkin operators -------------------------------------------------------------------

// Part of one cell's rows in B = P^T (L + D / 2) P, with A = L + D + L^T, a
// warp per active cell and a lane per row (32 rows at a time): a lane walks
// its row's run in each neighbour cell in turn, sums the entries times the
// eight monomials of the column's position in its cell (half the arithmetic
// of eight weights), turns them into the sums on that cell's corners and adds
// those to its own row of nodes of the cell and its neighbours in shared
// memory.  The rows of nodes are then spread over the cell's own corners:
// out[cell][own corner][node].  Runs of one cell's rows are of similar length,
// so the lanes stay together; what bounds it is the latency of the entries,
// which are therefore read a batch ahead, across the ends of runs.
constexpr int ML_CW = 2;   // cells per block

template <int D>
__global__ void __launch_bounds__(32 * ML_CW)
k_ml_cellmat(int nact, const int *__restrict__ acells, const int2 *__restrict__ desc, Grid<D> cg,
             const int *__restrict__ row_ptr, const int *__restrict__ diagpos,
             const unsigned short *__restrict__ runs, const int *__restrict__ col, const double *__restrict__ A,
             const float *__restrict__ frac, int stride, double *__restrict__ out)
{
    using L = MlDim<D>;
    constexpr int NC = L::NC, LN = 33, U = 4;
    constexpr int NPL = (L::W4 + 31) / 32;   // nodes of a lane
    __shared__ double snode[ML_CW][L::W4 * LN];
    __shared__ double sw[ML_CW][32 * NC];
    int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    int kk = blockIdx.x * ML_CW + w;
    if (kk >= nact) return;   // whole warps; no block barrier below
    double *node = snode[w], *wt = sw[w];
    int2 dd = desc[kk];
    int par = cell_parity<D>(cg, acells[kk]);
    int qc = visit_rank<D>(par, L::CELLS / 2);   // the own cell: the last with lower entries
    double acc[NPL][NC];
#pragma unroll
    for (int j = 0; j < NPL; j++)
#pragma unroll
        for (int k = 0; k < NC; k++) acc[j][k] = 0.0;
    for (int i0 = 0; i0 < dd.y; i0 += 32) {
        int nr = min(32, dd.y - i0);
        bool in = lane < nr;
        int r = dd.x + i0 + (in ? lane : 0);
        int base = row_ptr[r], diag = diagpos[r];
        int last = in ? diag + 1 : base;
        int end = qc > 0 ? min(last, base + runs[(size_t)stride + r]) : last;
        int e = base;
        int cn[U];
        double an[U];
#pragma unroll
        for (int u = 0; u < U; u++) {
            cn[u] = e + u < last ? __ldg(&col[e + u]) : r;
            an[u] = e + u < last ? __ldg(&A[e + u]) : 0.0;
        }
#pragma unroll 8
        for (int nd = 0; nd < L::W4; nd++) node[nd * LN + lane] = 0.0;
        double own[NC];
        ml_weights<D>(frac, stride, r, own);
#pragma unroll
        for (int k = 0; k < NC; k++) wt[lane * NC + k] = own[k];
        for (int q = 0; q <= qc; q++) {
            int end1 = q + 1 < qc ? min(last, base + runs[(size_t)(q + 2) * stride + r]) : last;   // the next run's end
            double s[NC];
#pragma unroll
            for (int k = 0; k < NC; k++) s[k] = 0.0;
            bool any = false;
            while (__any_sync(0xffffffffu, e < end)) {
                any = true;
                double a[U];
                float f[U][D];
                int ne = min(e + U, end);
#pragma unroll
                for (int u = 0; u < U; u++) {
                    a[u] = e + u < end ? (e + u == diag ? 0.5 * an[u] : an[u]) : 0.0;
#pragma unroll
                    for (int d = 0; d < D; d++) f[u][d] = __ldg(&frac[(size_t)d * stride + cn[u]]);
                }
                if (ne != e) {   // a lane at the end of its run keeps what it has read ahead
#pragma unroll
                    for (int u = 0; u < U; u++) {
                        cn[u] = ne + u < last ? __ldg(&col[ne + u]) : r;
                        an[u] = ne + u < last ? __ldg(&A[ne + u]) : 0.0;
                    }
                }
                e = ne;
#pragma unroll
                for (int u = 0; u < U; u++) {
                    double x = (double)f[u][0], y = (double)f[u][1];
                    double v = f[u][0] < 0.0f ? 0.0 : a[u];
                    double vx = v * x;
                    s[0] += v;
                    s[1] += vx;
                    s[2] = fma(v, y, s[2]);
                    s[3] = fma(vx, y, s[3]);
                    if (D == 3) {
                        double z = (double)f[u][D - 1];
                        double vz = v * z, vxz = vx * z;
                        s[4 & (NC - 1)] += vz;
                        s[5 & (NC - 1)] += vxz;
                        s[6 & (NC - 1)] = fma(vz, y, s[6 & (NC - 1)]);
                        s[7 & (NC - 1)] = fma(vxz, y, s[7 & (NC - 1)]);
                    }
                }
            }
            end = end1;
            if (!any) continue;
            // monomials to corners: along each axis, (1 - f) and f
#pragma unroll
            for (int d = 0; d < D; d++)
#pragma unroll
                for (int k = 0; k < NC; k++)
                    if (!(k >> d & 1)) s[k] -= s[k | (1 << d)];
            int nb = visit_cell<D>(par, q);
            int n0 = nb % 3 + 4 * ((nb / 3) % 3) + (D == 3 ? 16 * (nb / 9) : 0);
#pragma unroll
            for (int k = 0; k < NC; k++) {
                int nd = n0 + (k & 1) + 4 * ((k >> 1) & 1) + 16 * (k >> 2);
                node[nd * LN + lane] += s[k];
            }
        }
        __syncwarp();
        for (int i = 0; i < nr; i++) {
            double wi[NC];
#pragma unroll
            for (int k = 0; k < NC; k++) wi[k] = wt[i * NC + k];
#pragma unroll
            for (int j = 0; j < NPL; j++) {
                int nd = lane + 32 * j;
                if (nd < L::W4) {
                    double v = node[nd * LN + i];
#pragma unroll
                    for (int k = 0; k < NC; k++) acc[j][k] = fma(wi[k], v, acc[j][k]);
                }
            }
        }
        __syncwarp();
    }
#pragma unroll
    for (int j = 0; j < NPL; j++) {
        int nd = lane + 32 * j;
        if (nd < L::W4)
#pragma unroll
            for (int k = 0; k < NC; k++) out[(size_t)kk * (NC * L::W4) + k * L::W4 + nd] = acc[j][k];
    }
}

// Row sums of |a| and the diagonal of one operator row held by a block, and
// the smoother's factor; `v` is this thread's entry (0 beyond the stencil).
template <int D>
__device__ __forceinline__ void ml_row_factor(double v, int k, double *sh, bool additive, double *dinv)
{
    using L = MlDim<D>;
    __shared__ double diag;
    if (k == L::ST / 2) diag = v;
    double a = fabs(v);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = a;
    __syncthreads();
    if (threadIdx.x == 0) {
        double s = 0.0;
        for (int w = 0; w < (int)(blockDim.x >> 5); w++) s += sh[w];
        double d = additive ? diag : s;
        double f = additive ? ML_ADD : ML_OMEGA;
        *dinv = d > 0.0 ? f / d : 0.0;
    }
}

// B's rows from the cells' parts: a block per node, a thread per stencil entry.
template <int D>
__global__ void __launch_bounds__(MlDim<D>::STP)
k_ml_b1(int na, const int *__restrict__ ncell, const double *__restrict__ cellmat, double *__restrict__ B)
{
    using L = MlDim<D>;
    int t = blockIdx.x, k = threadIdx.x;
    double s = 0.0;
    if (k < L::ST) {
        int o[3] = {k % 5 - 2, (k / 5) % 5 - 2, D == 3 ? k / 25 - 2 : 0};
#pragma unroll
        for (int j = 0; j < L::NC; j++) {
            int c = ncell[(size_t)j * na + t];
            if (c < 0) continue;
            // node of the cell's 4^D at offset o from its corner j
            int nd = 0;
            bool in = true;
#pragma unroll
            for (int d = D - 1; d >= 0; d--) {
                int x = o[d] + ((j >> d) & 1) + 1;
                in = in && x >= 0 && x < 4;
                nd = nd * 4 + x;
            }
            if (in) s += cellmat[(size_t)c * (L::NC * L::W4) + j * L::W4 + nd];
        }
    }
    B[(size_t)t * L::STP + k] = s;
}

// A_1 = B + B^T and its smoother factor: entry k of node t is also entry
// ST - 1 - k of the node at that offset.
template <int D>
__global__ void __launch_bounds__(MlDim<D>::STP)
k_ml_a1(MlGrid g, const int *__restrict__ act, const int *__restrict__ amap, const double *__restrict__ B,
        bool additive, double *__restrict__ Ac, double *__restrict__ dinv)
{
    using L = MlDim<D>;
    __shared__ double sh[4];
    int t = blockIdx.x, k = threadIdx.x;
    double s = 0.0;
    if (k < L::ST) {
        int o = amap[act[t] + ml_offset<D>(g, k)];
        s = B[(size_t)t * L::STP + k] + (o >= 0 ? B[(size_t)o * L::STP + L::ST - 1 - k] : 0.0);
    }
    Ac[(size_t)t * L::STP + k] = s;
    ml_row_factor<D>(s, k, sh, additive, &dinv[t]);
}

// A_{l+1} = I^T A_l I, a block per coarse node: the fine rows under the node
// combined on the 7^D fine nodes around it, T = I^T A_l, then gathered onto
// the coarse stencil.  With E = f D_l1^-1 the smoother, a pre-smoothed residual
// restricts as I^T (b - A E b) = C b, C = I^T - T E, and C^T is the
// post-smoothed interpolation (1 - E A) I: C is kept so that either direction
// of the V-cycle is one dependent step per grid.
template <int D>
__global__ void __launch_bounds__(MlDim<D>::STP)
k_ml_galerkin(MlGrid f, MlGrid c, int lof, int loc, const int *__restrict__ act, const int *__restrict__ amap,
              const double *__restrict__ Af, const double *__restrict__ dinvf, double *__restrict__ Ac,
              double *__restrict__ dinv, double *__restrict__ C)
{
    using L = MlDim<D>;
    __shared__ double T[L::W7];
    __shared__ double sh[4];
    __shared__ int frow[L::CELLS];
    int t = blockIdx.x, k = threadIdx.x;
    int cc[3];
    ml_coords<D>(c, act[loc + t], cc);
    int centre = ml_at(f, 2 * cc[0], 2 * cc[1], 2 * cc[2]);
    if (k < L::CELLS) {
        int x = k % 3 - 1, y = (k / 3) % 3 - 1, z = D == 3 ? k / 9 - 1 : 0;
        int a = amap[centre + x + f.s1 * y + f.s2 * z];   // -1 in the margins
        frow[k] = a < 0 ? -1 : a - lof;
    }
    __syncthreads();
    for (int w = k; w < L::W7; w += L::STP) {
        int p[3] = {w % 7 - 3, (w / 7) % 7 - 3, D == 3 ? w / 49 - 3 : 0};
        double s = 0.0, own = 0.0;
        for (int j = 0; j < L::CELLS; j++) {
            if (frow[j] < 0) continue;
            int i[3] = {j % 3 - 1, (j / 3) % 3 - 1, D == 3 ? j / 9 - 1 : 0};
            int e = 0;
            bool in = true, same = true;
            double wt = 1.0;
#pragma unroll
            for (int d = D - 1; d >= 0; d--) {
                int x = p[d] - i[d] + 2;
                in = in && x >= 0 && x < 5;
                same = same && x == 2;
                e = e * 5 + x;
                if (i[d]) wt *= 0.5;
            }
            if (same) own = wt;
            if (in) s = fma(wt, __ldg(&Af[(size_t)frow[j] * L::STP + e]), s);
        }
        T[w] = s;
        double v = 0.0;
        bool in = true;
#pragma unroll
        for (int d = 0; d < D; d++) {
            int x = 2 * cc[d] + p[d];
            in = in && x >= 0 && x < f.n[d];
        }
        if (in) {
            int a = amap[centre + p[0] + f.s1 * p[1] + f.s2 * p[2]];
            if (a >= 0) v = own - s * __ldg(&dinvf[a - lof]);
        }
        C[(size_t)t * L::W7P + w] = v;
    }
    __syncthreads();
    double s = 0.0;
    if (k < L::ST) {
        int o[3] = {k % 5 - 2, (k / 5) % 5 - 2, D == 3 ? k / 25 - 2 : 0};
        for (int j = 0; j < L::CELLS; j++) {
            int i[3] = {j % 3 - 1, (j / 3) % 3 - 1, D == 3 ? j / 9 - 1 : 0};
            int e = 0;
            bool in = true;
            double wt = 1.0;
#pragma unroll
            for (int d = D - 1; d >= 0; d--) {
                int x = 2 * o[d] + i[d] + 3;
                in = in && x >= 0 && x < 7;
                e = e * 7 + x;
                if (i[d]) wt *= 0.5;
            }
            if (in) s = fma(wt, T[e], s);
        }
    }
    Ac[(size_t)t * L::STP + k] = s;
    ml_row_factor<D>(s, k, sh, false, &dinv[t]);
}

// Inverse of the coarsest operator (n <= ML_COARSEST nodes), one CTA, the
// matrix in registers (4 entries a thread): Gauss-Jordan without pivoting on
// the symmetric matrix, one barrier per pivot.  A pivot that cancellation has
// emptied (below 1e-9 of its diagonal: a constant on a region no known
// pressure bounds, or a node no row reaches) is dropped, which keeps the
// inverse symmetric and semidefinite.
template <int D>
__global__ void __launch_bounds__(1024)
k_ml_inverse(MlGrid g, int lo, int n, const int *__restrict__ act, const int *__restrict__ amap,
             const double *__restrict__ A, double *__restrict__ inv)
{
    using L = MlDim<D>;
    constexpr int N = ML_COARSEST, T = N / 32;
    extern __shared__ double m[];   // N x N while loading and storing
    __shared__ double row[2][N], cl[2][N], dg[N], piv[2];
    int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    for (int w = threadIdx.x; w < N * N; w += blockDim.x) m[w] = 0.0;
    __syncthreads();
    for (int w = threadIdx.x; w < n * L::ST; w += blockDim.x) {
        int i = w / L::ST, k = w % L::ST;
        double v = A[(size_t)i * L::STP + k];
        if (v != 0.0) {
            int j = amap[act[lo + i] + ml_offset<D>(g, k)];
            if (j >= lo && j < lo + n) m[i * N + j - lo] = v;
        }
    }
    __syncthreads();
    double a[T][T];
#pragma unroll
    for (int p = 0; p < T; p++)
#pragma unroll
        for (int q = 0; q < T; q++) a[p][q] = m[(ty + 32 * p) * N + tx + 32 * q];
    if (threadIdx.x < N) dg[threadIdx.x] = m[threadIdx.x * N + threadIdx.x];
    __syncthreads();
    for (int k = 0; k < n; k++) {
        double *rk = row[k & 1], *ck = cl[k & 1];
        int kp = k >> 5, kt = k & 31;
        if (ty == kt) {
#pragma unroll
            for (int p = 0; p < T; p++)
                if (p == kp) {
#pragma unroll
                    for (int q = 0; q < T; q++) rk[tx + 32 * q] = a[p][q];
                }
        }
        if (tx == kt) {
#pragma unroll
            for (int q = 0; q < T; q++)
                if (q == kp) {
#pragma unroll
                    for (int p = 0; p < T; p++) ck[ty + 32 * p] = a[p][q];
                    if (ty == kt) {
                        double d = 0.0;
#pragma unroll
                        for (int p = 0; p < T; p++)
                            if (p == kp) d = a[p][q];
                        piv[k & 1] = d > 1.0e-9 * dg[k] ? 1.0 / d : 0.0;
                    }
                }
        }
        __syncthreads();
        double pv = piv[k & 1];
        double r[T];
#pragma unroll
        for (int q = 0; q < T; q++) r[q] = rk[tx + 32 * q];
#pragma unroll
        for (int p = 0; p < T; p++) {
            double f = ck[ty + 32 * p] * pv;
            bool prow = p == kp && ty == kt;
#pragma unroll
            for (int q = 0; q < T; q++) {
                bool pcol = q == kp && tx == kt;
                double v = fma(-f, r[q], a[p][q]);
                v = prow ? pv * r[q] : v;
                v = pcol ? (prow ? pv : -f) : v;
                a[p][q] = v;
            }
        }
    }
#pragma unroll
    for (int p = 0; p < T; p++)
#pragma unroll
        for (int q = 0; q < T; q++) m[(ty + 32 * p) * N + tx + 32 * q] = a[p][q];
    __syncthreads();
    for (int w = threadIdx.x; w < n * n; w += blockDim.x) {
        int i = w / n, j = w % n;
        inv[w] = 0.5 * (m[i * N + j] + m[j * N + i]);
    }
}

// Per node: the index of the fine node under it (grids beyond the first), and
// of the lowest coarse node whose C row reaches it (all but the last), with
// the parities of its coordinates.
template <int D>
__global__ void k_ml_tables(const __grid_constant__ MlLevels lv, const int *__restrict__ act, int *__restrict__ under,
                            int *__restrict__ above, unsigned char *__restrict__ parity)
{
    int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= lv.lo[lv.nl]) return;
    int l = 0;
    while (t >= lv.lo[l + 1]) l++;
    int c[3];
    ml_coords<D>(lv.g[l], act[t], c);
    if (l > 0) under[t] = ml_at(lv.g[l - 1], 2 * c[0], 2 * c[1], 2 * c[2]);
    if (l + 1 < lv.nl) {
        above[t] = ml_at(lv.g[l + 1], (c[0] >> 1) - 1, (c[1] >> 1) - 1, D == 3 ? (c[2] >> 1) - 1 : 0);
        parity[t] = (unsigned char)((c[0] & 1) | (c[1] & 1) << 1 | (D == 3 ? (c[2] & 1) << 2 : 0));
    }
}

// Candidate e (of 4^D) of a node's column of C: offset from above[node] and
// the entry within that coarse node's row, -1 if out of its reach.
template <int D>
__device__ __forceinline__ int ml_cand(const MlGrid &c, int par, int e, int &off)
{
    int e0 = e & 3, e1 = (e >> 2) & 3, e2 = D == 3 ? e >> 4 : 0;
    off = e0 + c.s1 * e1 + c.s2 * e2 * (D == 3);
    int x = 5 + (par & 1) - 2 * e0, y = 5 + ((par >> 1) & 1) - 2 * e1, z = D == 3 ? 5 + (par >> 2) - 2 * e2 : 0;
    if (x < 0 || y < 0 || z < 0) return -1;
    return x + 7 * y + (D == 3 ? 49 * z : 0);
}

// Dense V-cycle of grid l from that of grid l + 1 (M_c, symmetric):
// M = 2 E - E A E + C^T M_c C.  First MC = M_c C, a block per fine node.
template <int D>
__global__ void __launch_bounds__(128)
k_ml_dense_mc(MlGrid c, int lo, int nf, int loc, int nc, int na1, const int *__restrict__ amap,
              const int *__restrict__ above, const unsigned char *__restrict__ parity, const double *__restrict__ C,
              const double *__restrict__ Mc, double *__restrict__ MC)
{
    constexpr int NE = D == 3 ? 64 : 16;
    __shared__ int row[NE];
    __shared__ double val[NE];
    int i = blockIdx.x, t = threadIdx.x;
    if (t < NE) {
        int off, w = ml_cand<D>(c, parity[lo + i], t, off);
        int a = w >= 0 ? amap[above[lo + i] + off] : -1;
        row[t] = a >= 0 ? a - loc : 0;
        val[t] = a >= 0 ? C[(size_t)(a - na1) * MlDim<D>::W7P + w] : 0.0;
    }
    __syncthreads();
    for (int j = t; j < nc; j += 128) {
        double s = 0.0;
        for (int e = 0; e < NE; e++)
            if (val[e] != 0.0) s = fma(val[e], __ldg(&Mc[(size_t)row[e] * nc + j]), s);
        MC[(size_t)j * nf + i] = s;
    }
}

template <int D>
__global__ void __launch_bounds__(256)
k_ml_dense(MlGrid f, MlGrid c, int lo, int nf, int loc, int na1, const int *__restrict__ act,
           const int *__restrict__ amap, const int *__restrict__ above, const unsigned char *__restrict__ parity,
           const double *__restrict__ A, const double *__restrict__ dinv, const double *__restrict__ C,
           const double *__restrict__ MC, double *__restrict__ M)
{
    using L = MlDim<D>;
    constexpr int NE = D == 3 ? 64 : 16;
    __shared__ int row[NE];
    __shared__ double val[NE];
    int i = blockIdx.x, t = threadIdx.x;
    if (t < NE) {
        int off, w = ml_cand<D>(c, parity[lo + i], t, off);
        int a = w >= 0 ? amap[above[lo + i] + off] : -1;
        row[t] = a >= 0 ? a - loc : 0;
        val[t] = a >= 0 ? C[(size_t)(a - na1) * L::W7P + w] : 0.0;
    }
    __syncthreads();
    for (int j = t; j < nf; j += 256) {
        double s = 0.0;
        for (int e = 0; e < NE; e++)
            if (val[e] != 0.0) s = fma(val[e], __ldg(&MC[(size_t)row[e] * nf + j]), s);
        M[(size_t)i * nf + j] = s;
    }
    __syncthreads();
    if (t < L::ST) {
        int a = amap[act[lo + i] + ml_offset<D>(f, t)];
        if (a >= 0) {
            double ei = dinv[lo + i];
            double s = -ei * A[(size_t)(lo + i) * L::STP + t] * dinv[a];
            if (t == L::ST / 2) s += 2.0 * ei;
            M[(size_t)i * nf + a - lo] += s;
        }
    }
}

// ---- one application -------------------------------------------------------------------------

// Reduces NV = 8 or 4 values per lane over groups of W lanes; afterwards the
// group's lanes [v W / NV, (v + 1) W / NV) hold the sum of value v.
template <int NV, int W = 32>
__device__ __forceinline__ double ml_group_reduce(double *v, int lane)
{
#pragma unroll
    for (int o = W / 2, h = NV / 2; h >= 1; o >>= 1, h >>= 1) {
        bool up = lane & o;
#pragma unroll
        for (int i = 0; i < NV / 2; i++) {
            if (i < h) {
                double send = up ? v[i] : v[i + h], keep = up ? v[i + h] : v[i];
                v[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
            }
        }
    }
    double s = v[0];
#pragma unroll
    for (int o = W / NV / 2; o >= 1; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    return s;
}

// CG step and restriction, a warp per cell: x += alpha p, r -= alpha Ap and
// r.r as k_cg_axpy (skipped when RESTRICT_ONLY), and the cell's part of P^T r,
// csum[cell][corner].
template <int D, bool RESTRICT_ONLY>
__global__ void __launch_bounds__(CG_BLOCK)
k_ml_update(int nact, const int2 *__restrict__ desc, const float *__restrict__ frac, int stride, double *x,
            double *r, const double *p, const double *Ap, double *__restrict__ csum, double *partials,
            unsigned *ticket, CGScalars *sc)
{
    constexpr int NC = 1 << D;
    __shared__ double sh[CG_BLOCK / 32];
    pdl_trigger();
    pdl_wait();
    if (sc->done) return;
    double alpha = RESTRICT_ONLY ? 0.0 : sc->alpha;
    int lane = threadIdx.x & 31;
    double rr = 0.0;
    for (int kk = blockIdx.x * (CG_BLOCK / 32) + (threadIdx.x >> 5); kk < nact; kk += gridDim.x * (CG_BLOCK / 32)) {
        int2 dd = __ldg(&desc[kk]);
        double s[NC];
#pragma unroll
        for (int k = 0; k < NC; k++) s[k] = 0.0;
        for (int i = dd.x + lane; i < dd.x + dd.y; i += 32) {
            double ri;
            if (RESTRICT_ONLY) {
                ri = r[i];
            } else {
                x[i] += alpha * p[i];
                ri = r[i] - alpha * Ap[i];
                r[i] = ri;
                rr += ri * ri;
            }
            double w[NC];
            ml_weights<D>(frac, stride, i, w);
#pragma unroll
            for (int k = 0; k < NC; k++) s[k] = fma(w[k], ri, s[k]);
        }
        double v = ml_group_reduce<NC>(s, lane);
        constexpr int SH = D == 3 ? 2 : 3;
        if ((lane & ((1 << SH) - 1)) == 0) csum[(size_t)kk * NC + (lane >> SH)] = v;
    }
    if (RESTRICT_ONLY) return;
    double t = block_sum<CG_BLOCK>(rr, sh);
    if (threadIdx.x == 0) partials[blockIdx.x] = t;
    if (last_block(ticket, gridDim.x)) {
        double tot = final_sum(partials, gridDim.x, 1, 0, sh);
        if (threadIdx.x == 0) sc->rr = tot;
    }
}

// z = D^-1 r + P x_1, a warp per cell; with RZ also r.z and beta as k_cg_rz.
template <int D, bool RZ>
__global__ void __launch_bounds__(CG_BLOCK)
k_ml_prolong(int nact, const int2 *__restrict__ desc, const int *__restrict__ cnode, MlGrid g,
             const float *__restrict__ frac, int stride, const double *__restrict__ dinv, const double *r, double *z,
             const double *x1, double *partials, unsigned *ticket, CGScalars *sc)
{
    constexpr int NC = 1 << D;
    __shared__ double sh[CG_BLOCK / 32];
    pdl_trigger();
    pdl_wait();
    if (sc->done) return;
    int lane = threadIdx.x & 31;
    double rz = 0.0;
    for (int kk = blockIdx.x * (CG_BLOCK / 32) + (threadIdx.x >> 5); kk < nact; kk += gridDim.x * (CG_BLOCK / 32)) {
        int2 dd = __ldg(&desc[kk]);
        int o = __ldg(&cnode[kk]);
        double c = 0.0;
        if (lane < NC) c = x1[o + (lane & 1) + g.s1 * ((lane >> 1) & 1) + g.s2 * (lane >> 2)];
        double xc[NC];
#pragma unroll
        for (int k = 0; k < NC; k++) xc[k] = __shfl_sync(0xffffffffu, c, k);
        for (int i = dd.x + lane; i < dd.x + dd.y; i += 32) {
            double ri = r[i];
            double w[NC];
            ml_weights<D>(frac, stride, i, w);
            double zi = __ldg(&dinv[i]) * ri;
#pragma unroll
            for (int k = 0; k < NC; k++) zi = fma(w[k], xc[k], zi);
            z[i] = zi;
            if (RZ) rz += ri * zi;
        }
    }
    if (!RZ) return;
    double t = block_sum<CG_BLOCK>(rz, sh);
    if (threadIdx.x == 0) partials[blockIdx.x] = t;
    if (last_block(ticket, gridDim.x)) {
        double tot = final_sum(partials, gridDim.x, 1, 0, sh);
        if (threadIdx.x == 0) {
            sc->rz_new = tot;
            if (fabs(sc->rz) < 1.0e-60) { sc->done = 1; sc->breakdown = 1; }
            else { sc->beta = tot / sc->rz; sc->rz = tot; }
        }
    }
}

// ---- grid operations; each on nodes t0, t0 + step, ... of one grid ----

struct MlVecs {
    double *b, *x, *y;       // right-hand side, E b (or the dense grid's solution), result
    double *bd;              // right-hand side of the dense grid, by node
    const int *act, *amap, *under, *above;
    const unsigned char *parity;
    const double *A, *dinv;  // operators and smoother factors by node number
    const double *C;         // by node number beyond the first grid
    const int *ncell;
    const double *csum, *M;  // cells' parts of P^T r; the dense V-cycle
    int na1;                 // nodes of the first grid
    int ld;                  // the dense grid
};

// b_1 = P^T r from the cells' parts, x_1 = E b_1.
template <int D>
__global__ void __launch_bounds__(CG_BLOCK) k_ml_nodes1(MlVecs v, const CGScalars *sc)
{
    pdl_trigger();
    int t = blockIdx.x * blockDim.x + threadIdx.x;
    bool in = t < v.na1;
    int c[1 << D];
#pragma unroll
    for (int k = 0; k < (1 << D); k++) c[k] = in ? __ldg(&v.ncell[(size_t)k * v.na1 + t]) : -1;
    int o = in ? __ldg(&v.act[t]) : 0;
    double di = in ? __ldg(&v.dinv[t]) : 0.0;
    pdl_wait();
    if (!in || sc->done) return;
    double s = 0.0;
#pragma unroll
    for (int k = 0; k < (1 << D); k++)
        if (c[k] >= 0) s += v.csum[(size_t)c[k] * (1 << D) + k];
    if (v.ld == 0) {
        v.bd[t] = s;
    } else {
        v.b[o] = s;
        v.x[o] = di * s;
    }
}

// Down one grid: b_{l+1} = C b_l, x_{l+1} = E b_{l+1} (a warp per coarse node,
// the first blocks) and y_l = 2 x_l - E A x_l (eight lanes per node),
// independent of each other.  Operators are read before the wait.
template <int D>
__global__ void __launch_bounds__(CG_BLOCK)
k_ml_down(MlVecs v, MlGrid f, int l, int lo, int mid, int hi, const CGScalars *sc)
{
    using L = MlDim<D>;
    constexpr int NW = CG_BLOCK / 32;
    __shared__ int off5[L::ST], off7[L::W7];
    pdl_trigger();
    int lane = threadIdx.x & 31;
    int nc = hi - mid, nf = mid - lo;
    int cb = (nc + NW - 1) / NW;   // blocks of the coarse part
    if ((int)blockIdx.x < cb) {
        for (int e = threadIdx.x; e < L::W7; e += CG_BLOCK)
            off7[e] = e % 7 - 3 + f.s1 * ((e / 7) % 7 - 3) + (D == 3 ? f.s2 * (e / 49 - 3) : 0);
        int w = blockIdx.x * NW + (threadIdx.x >> 5);
        bool in = w < nc;
        constexpr int NE = (L::W7 + 31) / 32;
        double ca[NE];
        const double *C = v.C + (size_t)(mid + (in ? w : 0) - v.na1) * L::W7P;
#pragma unroll
        for (int j = 0; j < NE; j++) {
            int e = lane + 32 * j;
            ca[j] = in && e < L::W7 ? __ldg(&C[e]) : 0.0;
        }
        int o = in ? __ldg(&v.act[mid + w]) : 0, fo = in ? __ldg(&v.under[mid + w]) : f.base;
        double di = in ? __ldg(&v.dinv[mid + w]) : 0.0;
        __syncthreads();
        pdl_wait();
        if (sc->done) return;
        double s = 0.0;
#pragma unroll
        for (int j = 0; j < NE; j++) {
            int e = lane + 32 * j;
            s = fma(ca[j], v.b[fo + off7[e < L::W7 ? e : 0]], s);
        }
#pragma unroll
        for (int k = 16; k > 0; k >>= 1) s += __shfl_xor_sync(0xffffffffu, s, k);
        if (in && lane == 0) {
            if (v.ld == l + 1) {
                v.bd[w] = s;
            } else {
                v.b[o] = s;
                v.x[o] = di * s;
            }
        }
        return;
    }
    for (int e = threadIdx.x; e < L::ST; e += CG_BLOCK) off5[e] = ml_offset<D>(f, e);
    int t = (blockIdx.x - cb) * (CG_BLOCK / 8) + (threadIdx.x >> 3), k0 = threadIdx.x & 7;
    bool in = t < nf;
    constexpr int NE = L::STP / 8;
    double a[NE];
    const double *A = v.A + (size_t)(lo + (in ? t : 0)) * L::STP;
#pragma unroll
    for (int j = 0; j < NE; j++) a[j] = in ? __ldg(&A[k0 + 8 * j]) : 0.0;   // zero beyond the stencil
    int o = in ? __ldg(&v.act[lo + t]) : f.base;
    double di = in ? __ldg(&v.dinv[lo + t]) : 0.0;
    __syncthreads();
    pdl_wait();
    if (sc->done) return;
    double s = 0.0;
#pragma unroll
    for (int j = 0; j < NE; j++) {
        int k = k0 + 8 * j;
        s = fma(a[j], v.x[o + off5[k < L::ST ? k : 0]], s);
    }
    s += __shfl_xor_sync(0xffffffffu, s, 4);
    s += __shfl_xor_sync(0xffffffffu, s, 2);
    s += __shfl_xor_sync(0xffffffffu, s, 1);
    if (in && k0 == 0) v.y[o] = 2.0 * v.x[o] - di * s;
}

// Up one grid: y_l += C^T cx, eight lanes per node; cx is the coarser grid's
// result.
template <int D>
__global__ void __launch_bounds__(CG_BLOCK)
k_ml_up(MlVecs v, MlGrid c, int lo, int nf, const double *cx, const CGScalars *sc)
{
    using L = MlDim<D>;
    pdl_trigger();
    int t = blockIdx.x * (CG_BLOCK / 8) + (threadIdx.x >> 3), lane = threadIdx.x & 7;
    bool in = t < nf;
    int o = in ? __ldg(&v.act[lo + t]) : 0, q0 = in ? __ldg(&v.above[lo + t]) : c.base;
    int par = in ? __ldg(&v.parity[lo + t]) : 0;
    constexpr int NE = D == 3 ? 8 : 2;
    double ca[NE];
    int q[NE];
#pragma unroll
    for (int j = 0; j < NE; j++) {
        int off, w = ml_cand<D>(c, par, lane + 8 * j, off);
        q[j] = q0 + off;
        int a = in && w >= 0 ? __ldg(&v.amap[q[j]]) : -1;
        if (a < 0) q[j] = c.base;
        ca[j] = a >= 0 ? __ldg(&v.C[(size_t)(a - v.na1) * L::W7P + w]) : 0.0;
    }
    pdl_wait();
    if (sc->done) return;
    double s = 0.0;
#pragma unroll
    for (int j = 0; j < NE; j++) s = fma(ca[j], cx[q[j]], s);
    s += __shfl_xor_sync(0xffffffffu, s, 4);
    s += __shfl_xor_sync(0xffffffffu, s, 2);
    s += __shfl_xor_sync(0xffffffffu, s, 1);
    if (in && lane == 0) v.y[o] += s;
}

// The additive first grid: b_2 = I^T b_1, x_2 = E b_2, and y_1 = x_1 + I cx.
template <int D>
__global__ void __launch_bounds__(CG_BLOCK)
k_ml_add_down(MlVecs v, MlGrid f, int mid, int hi, const CGScalars *sc)
{
    pdl_trigger();
    int t = mid + blockIdx.x * blockDim.x + threadIdx.x;
    bool in = t < hi;
    int o = in ? __ldg(&v.act[t]) : 0, fo = in ? __ldg(&v.under[t]) : 0;
    double di = in ? __ldg(&v.dinv[t]) : 0.0;
    pdl_wait();
    if (!in || sc->done) return;
    double s = 0.0;
#pragma unroll
    for (int j = 0; j < MlDim<D>::CELLS; j++) {
        int dx = j % 3 - 1, dy = (j / 3) % 3 - 1, dz = D == 3 ? j / 9 - 1 : 0;
        double w = (dx ? 0.5 : 1.0) * (dy ? 0.5 : 1.0) * (dz ? 0.5 : 1.0);
        s = fma(w, v.b[fo + dx + f.s1 * dy + f.s2 * dz], s);
    }
    if (v.ld == 1) {
        v.bd[t - mid] = s;
    } else {
        v.b[o] = s;
        v.x[o] = di * s;
    }
}

template <int D>
__global__ void __launch_bounds__(CG_BLOCK) k_ml_add_up(MlVecs v, MlGrid c, const double *cx, const CGScalars *sc)
{
    pdl_trigger();
    int t = blockIdx.x * blockDim.x + threadIdx.x;
    bool in = t < v.na1;
    int o = in ? __ldg(&v.act[t]) : 0, q0 = in ? __ldg(&v.above[t]) : 0, par = in ? __ldg(&v.parity[t]) : 0;
    pdl_wait();
    if (!in || sc->done) return;
    double s = 0.0;
#pragma unroll
    for (int j = 0; j < (1 << D); j++) {
        // parents: node (i + bit) / 2, above[] being at i / 2 - 1
        int px = 1 + ((par & 1) & (j & 1)), py = 1 + (((par >> 1) & 1) & ((j >> 1) & 1));
        int pz = D == 3 ? 1 + ((par >> 2) & (j >> 2)) : 0;
        s += cx[q0 + px + c.s1 * py + c.s2 * pz];
    }
    v.y[o] = v.x[o] + s * (1.0 / (1 << D));
}

// The dense grid: x = M b, a warp per node; the matrix row is read before the
// wait.
__global__ void __launch_bounds__(CG_BLOCK) k_ml_matvec(MlVecs v, int lo, int n, const CGScalars *sc)
{
    pdl_trigger();
    int lane = threadIdx.x & 31;
    int t = blockIdx.x * (CG_BLOCK / 32) + (threadIdx.x >> 5);
    bool in = t < n;
    const double *M = v.M + (size_t)(in ? t : 0) * n;
    constexpr int U = 8;
    double m[U];
#pragma unroll
    for (int j = 0; j < U; j++) {
        int e = lane + 32 * j;
        m[j] = in && e < n ? __ldg(&M[e]) : 0.0;
    }
    int o = in ? __ldg(&v.act[lo + t]) : 0;
    pdl_wait();
    if (!in || sc->done) return;   // warp-uniform
    double s = 0.0;
    for (int e0 = 0; e0 < n; e0 += 32 * U) {
        if (e0) {
#pragma unroll
            for (int j = 0; j < U; j++) {
                int e = e0 + lane + 32 * j;
                m[j] = e < n ? __ldg(&M[e]) : 0.0;
            }
        }
#pragma unroll
        for (int j = 0; j < U; j++) {
            int e = e0 + lane + 32 * j;
            s = fma(m[j], e < n ? v.bd[e] : 0.0, s);
        }
    }
#pragma unroll
    for (int k = 16; k > 0; k >>= 1) s += __shfl_xor_sync(0xffffffffu, s, k);
    if (lane == 0) v.x[o] = s;
}

// ---- small systems: the whole loop in one cluster ------------------------------------
//
// At up to 8,192 unknowns an iteration of the launched kernels is six or seven
// launches of 3-9 us, nearly all of it launch and drain.  Here one cluster of
// ML_CL CTAs runs the loop to its end, four cluster barriers an iteration (the
// product, the update, the coarse correction, its interpolation).  A barrier costs about 1,700 cycles and a load from L2 about
// 700, so what counts is the number of dependent ones: the direction and the
// CTA's rows of the matrix (where they fit) sit in shared memory, loads go out
// in predicated batches, the dot products' parts are stored into every CTA's
// shared memory, and every CTA forms the direction, the first grid's
// right-hand side and the additive form's second whole.

constexpr int ML_CL = 16;
constexpr int ML_CL_THREADS = 1024;
constexpr size_t ML_CL_SMEM = 216 * 1024;        // dynamic shared memory at most

struct MlSmall {
    int n_eq, nact, na1, nd, additive, stride, resume, maxit;
    int cache;   // matrix entries a CTA can hold in shared memory
    double tol;
    const int2 *desc;
    const float *frac;
    const int *row_ptr, *col;
    const double *A, *dsum;
    const uint2 *ac;
    const double *dinv, *b, *zprev;
    const int *ncell, *cellnode, *fine, *parent;   // node numbers: corners of a cell, I^T's and I's entries
    const double *dinv1, *M;
    double *x, *r, *z, *p, *Ap, *csum, *xd;
    CGScalars *sc;
};

__device__ __forceinline__ void cluster_sync()
{
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

struct MlTotals {
    double part[3][ML_CL];
    double sh[ML_CL_THREADS / 32];
};

// This CTA's part of a dot product, into every CTA's table; the cluster
// barrier that follows makes it readable.
__device__ __forceinline__ void ml_cluster_part(double v, int slot, MlTotals &t)
{
    v = block_sum<ML_CL_THREADS>(v, t.sh);
    if (threadIdx.x < 32) {
        v = __shfl_sync(0xffffffffu, v, 0);
        if (threadIdx.x < ML_CL) {
            unsigned local = smem_u32(&t.part[slot][blockIdx.x]), remote;
            asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(local), "r"(threadIdx.x));
            asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(remote), "d"(v) : "memory");
        }
    }
}

// The sum of a slot's parts, the same bits in every thread of the cluster.
__device__ __forceinline__ double ml_cluster_total(int slot, const MlTotals &t)
{
    double s = 0.0;
    const volatile double *p = t.part[slot];
#pragma unroll
    for (int c = 0; c < ML_CL; c++) s += p[c];
    return s;
}

// TM = float: the packed FP32 matrix in difference form (k_cg_spmv).
//
// Rows are taken cell by cell, W lanes per cell (64: two warps, each with its
// own part of the cell's sums).  A lane's first row, the only one in most
// cells, lives in registers with its weights: an acquire at the cluster
// barrier empties L1, so anything read again comes from L2.
template <int D, class TM, int LPR, int W>
__global__ void __launch_bounds__(ML_CL_THREADS) k_ml_small(const __grid_constant__ MlSmall a)
{
    constexpr int NC = 1 << D, CELLS = MlDim<D>::CELLS;
    constexpr int NW = ML_CL * ML_CL_THREADS / 32;
    extern __shared__ __align__(16) double dyn[];
    __shared__ MlTotals tot;
    // shared: the direction, b_1, b_2, the CTA's matrix entries (values and columns, or words)
    double *ps = dyn, *b1 = ps + a.n_eq, *b2 = b1 + a.na1;
    double *mval = b2 + (a.additive ? a.nd : 0);
    uint2 *mac = reinterpret_cast<uint2 *>(mval);
    int *mcol = reinterpret_cast<int *>(mval + a.cache);
    constexpr int PARTS = W > 32 ? W / 32 : 1, WL = W < 32 ? W : 32;   // warps of a cell; lanes of one in a warp
    constexpr int CELLS_PASS = NW * 32 / W;
    int tid = threadIdx.x, lane = tid & 31;
    int warp = blockIdx.x * (ML_CL_THREADS / 32) + (tid >> 5);
    int wl = lane & (WL - 1), part = warp & (PARTS - 1);
    int hl = wl + 32 * part;
    int first = W < 32 ? warp * (32 / WL) + lane / WL : warp / PARTS;   // this lane's first cell

    // the CTA's rows of the product
    int rb = (int)((long long)a.n_eq * blockIdx.x / ML_CL), re = (int)((long long)a.n_eq * (blockIdx.x + 1) / ML_CL);
    int e0 = __ldg(&a.row_ptr[rb]), ne = __ldg(&a.row_ptr[re]) - e0;
    bool cached = ne <= a.cache;
    if (cached) {
        for (int e = tid; e < ne; e += ML_CL_THREADS) {
            if (sizeof(TM) == 8) {
                mval[e] = __ldg(&a.A[e0 + e]);
                mcol[e] = __ldg(&a.col[e0 + e]);
            } else {
                mac[e] = __ldg(&a.ac[e0 + e]);
            }
        }
    }

    // this lane's first row
    int rounds = (a.nact + CELLS_PASS - 1) / CELLS_PASS;
    int kk0 = first;
    int2 dd0 = kk0 < a.nact ? __ldg(&a.desc[kk0]) : make_int2(0, 0);
    int nd0 = kk0 < a.nact && wl < NC ? __ldg(&a.cellnode[(size_t)kk0 * NC + wl]) : 0;
    bool own = hl < dd0.y;
    int i0 = dd0.x + hl;
    float f0[D];
#pragma unroll
    for (int d = 0; d < D; d++) f0[d] = own ? __ldg(&a.frac[(size_t)d * a.stride + i0]) : -1.0f;
    double r0 = 0.0, x0 = 0.0;
    if (own) {
        r0 = a.resume ? a.r[i0] : a.b[i0];
        x0 = a.resume ? a.x[i0] : 0.0;
    }

    // x += alpha p, r -= alpha Ap where `step`; r.r and the cells' parts of P^T r
    auto update = [&](bool step, double alpha) {
        double rr = 0.0;
        for (int q = 0; q < rounds; q++) {
            int kk = first + q * CELLS_PASS;
            bool in = kk < a.nact;
            int2 dd = q == 0 ? dd0 : in ? __ldg(&a.desc[kk]) : make_int2(0, 0);
            double s[NC];
#pragma unroll
            for (int k = 0; k < NC; k++) s[k] = 0.0;
            for (int i = dd.x + hl; i < dd.x + dd.y; i += W) {
                double ri, w[NC];
                if (q == 0 && i == i0) {
                    if (step) {
                        x0 = fma(alpha, ps[i], x0);
                        r0 = fma(-alpha, __ldcg(&a.Ap[i]), r0);
                    }
                    ri = r0;
                    ml_weights_of<D>(f0, w);
                } else {
                    if (step) {
                        a.x[i] = fma(alpha, ps[i], a.x[i]);
                        ri = fma(-alpha, __ldcg(&a.Ap[i]), a.r[i]);
                        a.r[i] = ri;
                    } else if (a.resume) {
                        ri = a.r[i];
                    } else {
                        ri = a.b[i];
                        a.x[i] = 0.0;
                        a.r[i] = ri;
                    }
                    ml_weights<D>(a.frac, a.stride, i, w);
                }
                rr = fma(ri, ri, rr);
#pragma unroll
                for (int k = 0; k < NC; k++) s[k] = fma(w[k], ri, s[k]);
            }
            double v = ml_group_reduce<NC, WL>(s, lane);
            if (in && wl % (WL / NC) == 0) a.csum[((size_t)kk * PARTS + part) * NC + wl / (WL / NC)] = v;
        }
        ml_cluster_part(rr, 1, tot);
    };

    // z = D^-1 r + P M P^T r for the cluster's rows from the cells' parts, and r.z
    auto precondition = [&]() {
        for (int t = tid; t < a.na1; t += ML_CL_THREADS) {
            double s = 0.0;
#pragma unroll
            for (int k = 0; k < NC; k++) {
                int c = __ldg(&a.ncell[(size_t)k * a.na1 + t]);
#pragma unroll
                for (int u = 0; u < PARTS; u++)
                    s += c >= 0 ? __ldcg(&a.csum[((size_t)c * PARTS + u) * NC + k]) : 0.0;
            }
            b1[t] = s;
        }
        __syncthreads();
        const double *bd = b1;
        if (a.additive) {
            for (int t = tid; t < a.nd; t += ML_CL_THREADS) {
                double s = 0.0;
#pragma unroll
                for (int j = 0; j < CELLS; j++) {
                    int f = __ldg(&a.fine[(size_t)j * a.nd + t]);
                    double w = (j % 3 != 1 ? 0.5 : 1.0) * ((j / 3) % 3 != 1 ? 0.5 : 1.0) *
                               (D == 3 && j / 9 != 1 ? 0.5 : 1.0);
                    s = fma(w, f >= 0 ? b1[f] : 0.0, s);
                }
                b2[t] = s;
            }
            __syncthreads();
            bd = b2;
        }
        for (int t = warp; t < a.nd; t += NW) {
            const double *M = a.M + (size_t)t * a.nd;
            double s = 0.0;
            constexpr int U = 8;
            for (int j0 = lane; j0 < a.nd; j0 += 32 * U) {
                double m[U];
#pragma unroll
                for (int u = 0; u < U; u++) m[u] = j0 + 32 * u < a.nd ? __ldg(&M[j0 + 32 * u]) : 0.0;
#pragma unroll
                for (int u = 0; u < U; u++) s = fma(m[u], j0 + 32 * u < a.nd ? bd[j0 + 32 * u] : 0.0, s);
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
            if (lane == 0) a.xd[t] = s;
        }
        cluster_sync();
        double rz = 0.0;
        for (int q = 0; q < rounds; q++) {
            int kk = first + q * CELLS_PASS;
            bool in = kk < a.nact;
            int2 dd = q == 0 ? dd0 : in ? __ldg(&a.desc[kk]) : make_int2(0, 0);
            double c = 0.0;
            if (in && wl < NC) {
                int nd = q == 0 ? nd0 : __ldg(&a.cellnode[(size_t)kk * NC + wl]);
                if (a.additive) {
                    double s = 0.0;
#pragma unroll
                    for (int j = 0; j < NC; j++) s += __ldcg(&a.xd[__ldg(&a.parent[(size_t)nd * NC + j])]);
                    c = fma(__ldg(&a.dinv1[nd]), b1[nd], s * (1.0 / NC));
                } else {
                    c = __ldcg(&a.xd[nd]);
                }
            }
            double xc[NC];
#pragma unroll
            for (int k = 0; k < NC; k++) xc[k] = __shfl_sync(0xffffffffu, c, k, WL);
            for (int i = dd.x + hl; i < dd.x + dd.y; i += W) {
                double ri, w[NC];
                double zi = __ldg(&a.dinv[i]);
                if (q == 0 && i == i0) {
                    ri = r0;
                    ml_weights_of<D>(f0, w);
                } else {
                    ri = a.r[i];
                    ml_weights<D>(a.frac, a.stride, i, w);
                }
                zi *= ri;
#pragma unroll
                for (int k = 0; k < NC; k++) zi = fma(w[k], xc[k], zi);
                a.z[i] = zi;
                rz = fma(ri, zi, rz);
            }
        }
        ml_cluster_part(rz, 2, tot);
    };

    cluster_sync();   // every CTA runs before its shared memory is stored to
    int iter = a.resume ? a.sc->iter : 0;
    update(false, 0.0);
    cluster_sync();
    double rr = ml_cluster_total(1, tot);
    precondition();
    cluster_sync();
    double rz = ml_cluster_total(2, tot);
    for (int j = tid; j < a.n_eq; j += ML_CL_THREADS) {
        double z = __ldcg(&a.z[j]);
        ps[j] = a.resume ? a.p[j] + (z - a.zprev[j]) : z;
    }
    __syncthreads();
    bool breakdown = false;
    double pAp = 0.0, alpha = 0.0, beta = 0.0;
    for (;;) {
        // the loop head of k_cg_spmv; every thread holds the same scalars
        if (sqrt(rr) < a.tol || iter >= a.maxit) break;
        if (isnan(rr)) {
            breakdown = true;
            break;
        }
        double acc = 0.0;
        for (int t = tid; t < (((re - rb) * LPR + 31) & ~31); t += ML_CL_THREADS) {
            int r = rb + t / LPR;
            bool in = r < re;
            int q0 = in ? __ldg(&a.row_ptr[r]) - e0 : 0, q1 = in ? __ldg(&a.row_ptr[r + 1]) - e0 : 0;
            double pr = in ? ps[r] : 0.0;
            double s = 0.0;
            constexpr int U = 8;
            for (int q = q0 + (t & (LPR - 1)); q < q1; q += LPR * U) {
                double v[U];
                int c[U];
#pragma unroll
                for (int u = 0; u < U; u++) {
                    int e = q + u * LPR;
                    v[u] = 0.0;
                    c[u] = r;
                    if (e < q1) {
                        if (sizeof(TM) == 8) {
                            v[u] = cached ? mval[e] : __ldg(&a.A[e0 + e]);
                            c[u] = cached ? mcol[e] : __ldg(&a.col[e0 + e]);
                        } else {
                            uint2 w = cached ? mac[e] : __ldg(&a.ac[e0 + e]);
                            v[u] = (double)__uint_as_float(w.x);
                            c[u] = (int)w.y;
                        }
                    }
                }
#pragma unroll
                for (int u = 0; u < U; u++) s = fma(v[u], sizeof(TM) == 8 ? ps[c[u]] : ps[c[u]] - pr, s);
            }
#pragma unroll
            for (int o = LPR / 2; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
            if (in && (t & (LPR - 1)) == 0) {
                if (sizeof(TM) == 4) s = fma(__ldg(&a.dsum[r]), pr, s);
                a.Ap[r] = s;
                acc = fma(pr, s, acc);
            }
        }
        ml_cluster_part(acc, 0, tot);
        cluster_sync();
        pAp = ml_cluster_total(0, tot);
        if (fabs(pAp) < 1.0e-30) {
            breakdown = true;
            break;
        }
        alpha = rz / pAp;
        update(true, alpha);
        cluster_sync();
        rr = ml_cluster_total(1, tot);
        precondition();
        cluster_sync();
        double rz_new = ml_cluster_total(2, tot);
        if (fabs(rz) < 1.0e-60) {
            breakdown = true;
            break;
        }
        beta = rz_new / rz;
        rz = rz_new;
        for (int j = tid; j < a.n_eq; j += ML_CL_THREADS) ps[j] = fma(beta, ps[j], __ldcg(&a.z[j]));
        __syncthreads();
        iter++;
    }
    // what a resumed loop and the caller read
    if (own) {
        a.x[i0] = x0;
        a.r[i0] = r0;
    }
    for (int j = rb + tid; j < re; j += ML_CL_THREADS) a.p[j] = ps[j];
    if (blockIdx.x == 0 && tid == 0) {
        CGScalars *sc = a.sc;
        sc->rr = rr;
        sc->rz = rz;
        sc->pAp = pAp;
        sc->alpha = alpha;
        sc->beta = beta;
        sc->tol = a.tol;
        sc->maxit = a.maxit;
        sc->iter = iter;
        sc->done = 1;
        sc->breakdown = breakdown;
    }
}

// Node numbers the cluster loop needs: the corners of every active cell, and,
// with an additive first grid, the fine nodes under every coarse node ([entry]
// [node], -1 where there is none) and the 2^D parents of every fine node.
template <int D>
__global__ void k_ml_small_tables(int nact, int na1, int nd, bool additive, MlGrid f, MlGrid c,
                                  const int *__restrict__ cnode, const int *__restrict__ amap,
                                  const int *__restrict__ under, const int *__restrict__ above,
                                  const unsigned char *__restrict__ parity, int *__restrict__ cellnode,
                                  int *__restrict__ fine, int *__restrict__ parent)
{
    constexpr int NC = 1 << D, CELLS = MlDim<D>::CELLS;
    int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t < nact) {
#pragma unroll
        for (int k = 0; k < NC; k++)
            cellnode[(size_t)t * NC + k] = amap[cnode[t] + (k & 1) + f.s1 * ((k >> 1) & 1) + f.s2 * (k >> 2)];
    }
    if (!additive) return;
    if (t < nd) {
        int o = under[na1 + t];
#pragma unroll
        for (int j = 0; j < CELLS; j++)
            fine[(size_t)j * nd + t] =
                amap[o + j % 3 - 1 + f.s1 * ((j / 3) % 3 - 1) + (D == 3 ? f.s2 * (j / 9 - 1) : 0)];
    }
    if (t < na1) {
        int q0 = above[t], par = parity[t];
#pragma unroll
        for (int j = 0; j < NC; j++) {
            int px = 1 + ((par & 1) & (j & 1)), py = 1 + (((par >> 1) & 1) & ((j >> 1) & 1));
            int pz = D == 3 ? 1 + ((par >> 2) & (j >> 2)) : 0;
            parent[(size_t)t * NC + j] = amap[q0 + px + c.s1 * py + c.s2 * pz] - na1;
        }
    }
}

}  // namespace mps
