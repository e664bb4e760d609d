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
// `additive`, V(b) = s D_1^-1 b + I V_2(I^T b) (no matrix on the first grid).
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
// Measured against the block-colour IC(0) (a step, B200, one box): 3-D dam
// break of 2.85 M particles, mixed form, 619 -> 34 iterations, 887 -> 103 ms;
// 1.17 M particles in FP64, 507 -> 44, 387 -> 47 ms; 2,158 particles in 2-D,
// 94 -> 44, 7.1 -> 2.6 ms.  What remains of an iteration is the product with
// the matrix (HBM) at large sizes and the chain of dependent launches at
// small ones.
//
// No sum uses an atomic; every reduction runs in a fixed order, so results
// are the same bits on every run.
#pragma once

#include "device.cuh"
#include "k_ppe.cuh"

namespace mps {

constexpr int ML_MAXL = 26;       // grids at most: 2^30 cells, even in one direction, reach the coarsest size
constexpr int ML_COARSEST = 64;   // nodes (boundary box) of the coarsest grid at most
// Relaxation of the l1-Jacobi steps (below 2 contracts); measured on the dam
// break at l0 = 0.01: 42 iterations at 1.0, 40 at 1.4 to 1.9.
constexpr double ML_OMEGA = 1.5;
// Weight of the additive first grid's D_1^-1 (D_1 the true diagonal).
constexpr double ML_ADD = 0.45;

template <int D>
struct MlDim {
    static constexpr int NC = 1 << D;                  // corners of a cell
    static constexpr int CELLS = D == 3 ? 27 : 9;      // a cell and its neighbours
    static constexpr int W4 = D == 3 ? 64 : 16;        // nodes of a cell and its neighbours (4 per axis)
    static constexpr int ST = D == 3 ? 125 : 25;       // stencil (5 per axis)
    static constexpr int STP = D == 3 ? 128 : 32;      // its stride in memory
    static constexpr int W7 = D == 3 ? 343 : 49;       // nodes within 3 of a node (7 per axis)
};

// One grid.  Vectors live on the whole box of nodes with a margin of two
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
        c[2] = rel / g.s2 - 2;
        rel %= g.s2;
    } else {
        c[2] = 0;
    }
    c[1] = rel / g.s1 - 2;
    c[0] = rel % g.s1 - 2;
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

// Eight lanes per row take its lower entries.
__global__ void k_uf_hook(int n, const int *__restrict__ row_ptr, const int *__restrict__ diagpos,
                          const int *__restrict__ col, const double *__restrict__ A, int *parent)
{
    int r = (int)((blockIdx.x * (size_t)blockDim.x + threadIdx.x) >> 3);
    if (r >= n) return;
    int last = -1;
    for (int q = row_ptr[r] + (threadIdx.x & 7); q < diagpos[r]; q += 8) {
        int j = col[q];
        if (A[q] == 0.0) continue;
        int b = uf_find(parent, j);
        if (b == last) continue;
        int a = uf_find(parent, r);
        while (a != b) {
            if (a < b) { int t = a; a = b; b = t; }
            int old = atomicCAS(&parent[a], a, b);   // the larger root under the smaller
            if (old == a) break;
            a = uf_find(parent, old);
            b = uf_find(parent, b);
        }
        last = b;
    }
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

// Weights of a row on its cell's corners, all zero for a row left out of P.
template <int D>
__device__ __forceinline__ void ml_weights(const float *__restrict__ frac, int stride, int r, double *w)
{
    double f[D];
#pragma unroll
    for (int d = 0; d < D; d++) f[d] = (double)__ldg(&frac[(size_t)d * stride + r]);
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

// ---- Galerkin operators -------------------------------------------------------------------

// Part of one cell's rows in A_1 = P^T A P, a CTA per active cell, ML_RB rows
// at a time: a thread per (row, neighbour cell) sums the row's entries there
// weighted onto that cell's corners, the corner sums are added up on the 4^D
// nodes of the cell and its neighbours, and the rows of that product are
// spread over the cell's own corners: out[cell][own corner][node].
// (A thread per neighbour cell and corner, every entry read by 2^D threads,
// took 14.7 ms at 2.2 M rows.)
constexpr int ML_RB = 8;

template <int D>
__global__ void __launch_bounds__(D == 3 ? 256 : 128)
k_ml_cellmat(const int *__restrict__ acells, const int2 *__restrict__ desc, Grid<D> cg,
             const int *__restrict__ row_ptr, const unsigned short *__restrict__ runs, const int *__restrict__ col,
             const double *__restrict__ A, const float *__restrict__ frac, int stride, double *__restrict__ out)
{
    using L = MlDim<D>;
    constexpr int BLOCK = D == 3 ? 256 : 128;
    constexpr int ITEMS = (L::NC * L::W4 + BLOCK - 1) / BLOCK;
    __shared__ double sp[ML_RB][L::CELLS][L::NC];
    __shared__ double sn[ML_RB][L::W4];
    __shared__ double sw[ML_RB][L::NC];
    int kk = blockIdx.x, t = threadIdx.x;
    int2 dd = desc[kk];
    int par = cell_parity<D>(cg, acells[kk]);
    double acc[ITEMS];
#pragma unroll
    for (int j = 0; j < ITEMS; j++) acc[j] = 0.0;
    for (int i0 = 0; i0 < dd.y; i0 += ML_RB) {
        int nr = min(ML_RB, dd.y - i0);
        for (int w = t; w < nr * L::CELLS; w += BLOCK) {
            int i = w / L::CELLS, q = w % L::CELLS;
            int r = dd.x + i0 + i;
            int base = row_ptr[r];
            int e = base + runs[(size_t)q * stride + r];
            int end = q + 1 < L::CELLS ? base + runs[(size_t)(q + 1) * stride + r] : row_ptr[r + 1];
            double s[L::NC];
#pragma unroll
            for (int k = 0; k < L::NC; k++) s[k] = 0.0;
            for (; e < end; e++) {
                double a = __ldg(&A[e]);
                double wt[L::NC];
                ml_weights<D>(frac, stride, __ldg(&col[e]), wt);
#pragma unroll
                for (int k = 0; k < L::NC; k++) s[k] = fma(a, wt[k], s[k]);
            }
            int nb = visit_cell<D>(par, q);
#pragma unroll
            for (int k = 0; k < L::NC; k++) sp[i][nb][k] = s[k];
        }
        if (t < nr) {
            double w[L::NC];
            ml_weights<D>(frac, stride, dd.x + i0 + t, w);
#pragma unroll
            for (int j = 0; j < L::NC; j++) sw[t][j] = w[j];
        }
        __syncthreads();
        // the (cell, corner) pairs that name one node, in a fixed order
        for (int w = t; w < nr * L::W4; w += BLOCK) {
            int i = w / L::W4, nd = w % L::W4;
            int nx = nd % 4, ny = (nd / 4) % 4, nz = nd / 16;
            double s = 0.0;
#pragma unroll
            for (int kz = 0; kz < (D == 3 ? 2 : 1); kz++)
#pragma unroll
                for (int ky = 0; ky < 2; ky++)
#pragma unroll
                    for (int kx = 0; kx < 2; kx++) {
                        int qx = nx - kx, qy = ny - ky, qz = D == 3 ? nz - kz : 0;
                        if (qx < 0 || qx > 2 || qy < 0 || qy > 2 || qz < 0 || qz > 2) continue;
                        s += sp[i][qx + 3 * qy + 9 * qz][kx + 2 * ky + 4 * kz];
                    }
            sn[i][nd] = s;
        }
        __syncthreads();
#pragma unroll
        for (int j = 0; j < ITEMS; j++) {
            int w = t + j * BLOCK;
            if (w < L::NC * L::W4)
                for (int i = 0; i < nr; i++) acc[j] = fma(sw[i][w / L::W4], sn[i][w % L::W4], acc[j]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int j = 0; j < ITEMS; j++) {
        int w = t + j * BLOCK;
        if (w < L::NC * L::W4) out[(size_t)kk * (L::NC * L::W4) + w] = acc[j];
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

// A_1 rows from the cells' parts: a block per node, a thread per stencil entry.
template <int D>
__global__ void __launch_bounds__(MlDim<D>::STP)
k_ml_a1(int na, const int *__restrict__ ncell, const double *__restrict__ cellmat, bool additive,
        double *__restrict__ Ac, double *__restrict__ dinv)
{
    using L = MlDim<D>;
    __shared__ double sh[4];
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
    Ac[(size_t)t * L::STP + k] = s;
    ml_row_factor<D>(s, k, sh, additive, &dinv[t]);
}

// A_{l+1} = I^T A_l I, a block per coarse node: the fine rows under the node
// combined on the 7^D fine nodes around it, then gathered onto the coarse
// stencil.
template <int D>
__global__ void __launch_bounds__(MlDim<D>::STP)
k_ml_galerkin(MlGrid f, MlGrid c, int lof, int loc, const int *__restrict__ act, const int *__restrict__ amap,
              const double *__restrict__ Af, double *__restrict__ Ac, double *__restrict__ dinv)
{
    using L = MlDim<D>;
    __shared__ double T[L::W7];
    __shared__ double sh[4];
    __shared__ int frow[L::CELLS];
    int t = blockIdx.x, k = threadIdx.x;
    int cc[3];
    ml_coords<D>(c, act[loc + t], cc);
    if (k < L::CELLS) {
        int x = 2 * cc[0] + k % 3 - 1, y = 2 * cc[1] + (k / 3) % 3 - 1, z = D == 3 ? 2 * cc[2] + k / 9 - 1 : 0;
        bool in = x >= 0 && x < f.n[0] && y >= 0 && y < f.n[1] && z >= 0 && z < f.n[2];
        int a = in ? amap[ml_at(f, x, y, z)] : -1;
        frow[k] = a < 0 ? -1 : a - lof;
    }
    __syncthreads();
    for (int w = k; w < L::W7; w += L::STP) {
        int p[3] = {w % 7 - 3, (w / 7) % 7 - 3, D == 3 ? w / 49 - 3 : 0};
        double s = 0.0;
        for (int j = 0; j < L::CELLS; j++) {
            if (frow[j] < 0) continue;
            int i[3] = {j % 3 - 1, (j / 3) % 3 - 1, D == 3 ? j / 9 - 1 : 0};
            int e = 0;
            bool in = true;
            double wt = 1.0;
#pragma unroll
            for (int d = D - 1; d >= 0; d--) {
                int x = p[d] - i[d] + 2;
                in = in && x >= 0 && x < 5;
                e = e * 5 + x;
                if (i[d]) wt *= 0.5;
            }
            if (in) s = fma(wt, __ldg(&Af[(size_t)frow[j] * L::STP + e]), s);
        }
        T[w] = s;
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

// Inverse of the coarsest operator (n <= ML_COARSEST nodes), one CTA:
// Gauss-Jordan without pivoting on the symmetric matrix.  A pivot that
// cancellation has emptied (below 1e-9 of its diagonal: a constant on a region
// no known pressure bounds, or a node no row reaches) is dropped, which keeps
// the inverse symmetric and semidefinite.
template <int D>
__global__ void __launch_bounds__(1024)
k_ml_inverse(MlGrid g, int lo, int n, const int *__restrict__ act, const int *__restrict__ amap,
             const double *__restrict__ A, double *__restrict__ inv)
{
    using L = MlDim<D>;
    extern __shared__ double a[];   // n x n, then the diagonal
    double *dg = a + n * n;
    __shared__ double piv;
    for (int w = threadIdx.x; w < n * n; w += blockDim.x) a[w] = 0.0;
    __syncthreads();
    for (int w = threadIdx.x; w < n * L::ST; w += blockDim.x) {
        int i = w / L::ST, k = w % L::ST;
        int j = amap[act[lo + i] + ml_offset<D>(g, k)];
        double v = A[(size_t)i * L::STP + k];
        if (j >= lo && j < lo + n && v != 0.0) a[i * n + j - lo] = v;
    }
    __syncthreads();
    for (int i = threadIdx.x; i < n; i += blockDim.x) dg[i] = a[i * n + i];
    for (int k = 0; k < n; k++) {
        __syncthreads();
        if (threadIdx.x == 0) {
            double d = a[k * n + k];
            piv = d > 1.0e-9 * dg[k] ? 1.0 / d : 0.0;
        }
        __syncthreads();
        double p = piv;
        // off the pivot's row and column
        for (int w = threadIdx.x; w < n * n; w += blockDim.x) {
            int i = w / n, j = w % n;
            if (i != k && j != k && p != 0.0) a[w] -= a[i * n + k] * p * a[k * n + j];
        }
        __syncthreads();
        for (int i = threadIdx.x; i < n; i += blockDim.x) {
            if (i == k) continue;
            a[i * n + k] *= -p;
            a[k * n + i] *= p;
        }
        if (threadIdx.x == 0) a[k * n + k] = p;
    }
    __syncthreads();
    for (int w = threadIdx.x; w < n * n; w += blockDim.x) {
        int i = w / n, j = w % n;
        inv[w] = 0.5 * (a[i * n + j] + a[j * n + i]);
    }
}

// ---- one application -------------------------------------------------------------------------

// Reduces NV = 8 or 4 values per lane over the warp; afterwards lane
// (corner << (5 - log2 NV)) holds the sum of value `corner`.
template <int NV>
__device__ __forceinline__ double ml_warp_reduce(double *v, int lane)
{
    int n = NV;
#pragma unroll
    for (int o = 16, h = NV / 2; h >= 1; o >>= 1, h >>= 1) {
        bool up = lane & o;
#pragma unroll
        for (int i = 0; i < NV / 2; i++) {
            if (i < h) {
                double send = up ? v[i] : v[i + h], keep = up ? v[i + h] : v[i];
                v[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
            }
        }
        n = h;
    }
    double s = v[0];
    (void)n;
#pragma unroll
    for (int o = 16 / NV; o >= 1; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
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
        double v = ml_warp_reduce<NC>(s, lane);
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
    double *b, *x, *y;       // right-hand side, iterate, residual (or the iterate's other buffer)
    const int *act;
    const double *A, *dinv;  // operators and smoother factors by node number
    const int *ncell;
    const double *csum, *inv;
    int na1;                 // nodes of the first grid
};

// b_1 = P^T r from the cells' parts, x_1 = f b_1.
template <int D>
__device__ __forceinline__ void ml_nodes1(const MlVecs &v, int t0, int step)
{
    for (int t = t0; t < v.na1; t += step) {
        double s = 0.0;
#pragma unroll
        for (int k = 0; k < (1 << D); k++) {
            int c = __ldg(&v.ncell[(size_t)k * v.na1 + t]);
            if (c >= 0) s += __ldcg(&v.csum[(size_t)c * (1 << D) + k]);
        }
        int o = __ldg(&v.act[t]);
        v.b[o] = s;
        v.x[o] = __ldg(&v.dinv[t]) * s;
    }
}

// POST: y = x + f (b - A x), else y = b - A x; eight lanes per node.
template <int D, bool POST>
__device__ __forceinline__ void ml_residual(const MlVecs &v, const MlGrid &g, int lo, int hi, int t0, int step)
{
    using L = MlDim<D>;
    int lane = threadIdx.x & 7;
    int nrow = (hi - lo + 3) & ~3;   // whole warps
    for (int t = t0 >> 3; t < nrow; t += step >> 3) {
        bool in = lo + t < hi;
        int o = in ? __ldg(&v.act[lo + t]) : g.base;
        const double *a = v.A + (size_t)(in ? lo + t : lo) * L::STP;
        double s = 0.0;
        if (in) {
#pragma unroll
            for (int j = 0; j < L::STP / 8; j++) {
                int k = lane + 8 * j;
                if (k < L::ST) s = fma(__ldg(&a[k]), __ldcg(&v.x[o + ml_offset<D>(g, k)]), s);
            }
        }
        s += __shfl_xor_sync(0xffffffffu, s, 4);
        s += __shfl_xor_sync(0xffffffffu, s, 2);
        s += __shfl_xor_sync(0xffffffffu, s, 1);
        if (in && lane == 0) {
            double res = __ldcg(&v.b[o]) - s;
            v.y[o] = POST ? __ldcg(&v.x[o]) + __ldg(&v.dinv[lo + t]) * res : res;
        }
    }
}

// b_c = I^T src on the coarser grid c, x_c = f b_c.
template <int D>
__device__ __forceinline__ void ml_restrict(const MlVecs &v, const double *src, const MlGrid &f, const MlGrid &c,
                                            int lo, int hi, int t0, int step)
{
    for (int t = lo + t0; t < hi; t += step) {
        int o = __ldg(&v.act[t]);
        int cc[3];
        ml_coords<D>(c, o, cc);
        int fo = ml_at(f, 2 * cc[0], 2 * cc[1], 2 * cc[2]);
        double s = 0.0;
#pragma unroll
        for (int j = 0; j < MlDim<D>::CELLS; j++) {
            int dx = j % 3 - 1, dy = (j / 3) % 3 - 1, dz = D == 3 ? j / 9 - 1 : 0;
            double w = (dx ? 0.5 : 1.0) * (dy ? 0.5 : 1.0) * (dz ? 0.5 : 1.0);
            s = fma(w, __ldcg(&src[fo + dx + f.s1 * dy + f.s2 * dz]), s);
        }
        v.b[o] = s;
        v.x[o] = __ldg(&v.dinv[t]) * s;
    }
}

// x_f += I src, src on the coarser grid c.
template <int D>
__device__ __forceinline__ void ml_prolong(const MlVecs &v, const double *src, const MlGrid &f, const MlGrid &c,
                                           int lo, int hi, int t0, int step)
{
    for (int t = lo + t0; t < hi; t += step) {
        int o = __ldg(&v.act[t]);
        int fc[3];
        ml_coords<D>(f, o, fc);
        double s = 0.0;
#pragma unroll
        for (int j = 0; j < (1 << D); j++) {
            int q = ml_at(c, (fc[0] + (j & 1)) / 2, (fc[1] + ((j >> 1) & 1)) / 2, D == 3 ? (fc[2] + (j >> 2)) / 2 : 0);
            s += __ldcg(&src[q]);
        }
        v.x[o] = __ldcg(&v.x[o]) + s * (1.0 / (1 << D));
    }
}

template <int D>
__global__ void __launch_bounds__(CG_BLOCK) k_ml_nodes1(MlVecs v, const CGScalars *sc)
{
    pdl_trigger();
    pdl_wait();
    if (sc->done) return;
    ml_nodes1<D>(v, blockIdx.x * blockDim.x + threadIdx.x, gridDim.x * blockDim.x);
}

template <int D, bool POST>
__global__ void __launch_bounds__(CG_BLOCK) k_ml_residual(MlVecs v, MlGrid g, int lo, int hi, const CGScalars *sc)
{
    pdl_trigger();
    pdl_wait();
    if (sc->done) return;
    ml_residual<D, POST>(v, g, lo, hi, blockIdx.x * blockDim.x + threadIdx.x, gridDim.x * blockDim.x);
}

template <int D>
__global__ void __launch_bounds__(CG_BLOCK)
k_ml_restrict(MlVecs v, const double *src, MlGrid f, MlGrid c, int lo, int hi, const CGScalars *sc)
{
    pdl_trigger();
    pdl_wait();
    if (sc->done) return;
    ml_restrict<D>(v, src, f, c, lo, hi, blockIdx.x * blockDim.x + threadIdx.x, gridDim.x * blockDim.x);
}

template <int D>
__global__ void __launch_bounds__(CG_BLOCK)
k_ml_prolong_add(MlVecs v, const double *src, MlGrid f, MlGrid c, int lo, int hi, const CGScalars *sc)
{
    pdl_trigger();
    pdl_wait();
    if (sc->done) return;
    ml_prolong<D>(v, src, f, c, lo, hi, blockIdx.x * blockDim.x + threadIdx.x, gridDim.x * blockDim.x);
}

// The V-cycle from grid l0 down and back, in one cluster of ML_CL CTAs: the
// grids there are small, so what bounds a step is the time between dependent
// steps, and a cluster barrier costs a fraction of a kernel boundary.
// first_src: l0 == 0, the cells' parts; else the vector restricted to grid l0.
// The result is in y on grids with a smoothing step after the correction, in
// x on the coarsest and on an additive first grid.
constexpr int ML_CL = 8;
constexpr int ML_CL_THREADS = 512;

__device__ __forceinline__ void cluster_sync()
{
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

template <int D>
__global__ void __cluster_dims__(ML_CL, 1, 1) __launch_bounds__(ML_CL_THREADS)
k_ml_cycle(MlVecs v, const __grid_constant__ MlLevels lv, int l0, const double *src, bool additive,
           const CGScalars *sc)
{
    pdl_trigger();
    pdl_wait();
    if (sc->done) return;   // uniform over the cluster
    int t0 = blockIdx.x * ML_CL_THREADS + threadIdx.x;
    constexpr int step = ML_CL * ML_CL_THREADS;
    int nl = lv.nl;
    if (l0 == 0) ml_nodes1<D>(v, t0, step);
    else ml_restrict<D>(v, src, lv.g[l0 - 1], lv.g[l0], lv.lo[l0], lv.lo[l0 + 1], t0, step);
    cluster_sync();
    for (int l = l0; l + 1 < nl; l++) {
        bool add = additive && l == 0;
        if (!add) {
            ml_residual<D, false>(v, lv.g[l], lv.lo[l], lv.lo[l + 1], t0, step);
            cluster_sync();
        }
        ml_restrict<D>(v, add ? v.b : v.y, lv.g[l], lv.g[l + 1], lv.lo[l + 1], lv.lo[l + 2], t0, step);
        cluster_sync();
    }
    {
        // coarsest grid: x = inverse b, eight lanes per node
        int lo = lv.lo[nl - 1], n = lv.lo[nl] - lo;
        int lane = threadIdx.x & 7;
        int nrow = (n + 3) & ~3;
        for (int t = t0 >> 3; t < nrow; t += step >> 3) {
            double s = 0.0;
            if (t < n)
                for (int j = lane; j < n; j += 8)
                    s = fma(__ldg(&v.inv[t * n + j]), __ldcg(&v.b[__ldg(&v.act[lo + j])]), s);
            s += __shfl_xor_sync(0xffffffffu, s, 4);
            s += __shfl_xor_sync(0xffffffffu, s, 2);
            s += __shfl_xor_sync(0xffffffffu, s, 1);
            if (t < n && lane == 0) v.x[__ldg(&v.act[lo + t])] = s;
        }
        cluster_sync();
    }
    for (int l = nl - 2; l >= l0; l--) {
        const double *cx = l + 1 == nl - 1 ? v.x : v.y;
        ml_prolong<D>(v, cx, lv.g[l], lv.g[l + 1], lv.lo[l], lv.lo[l + 1], t0, step);
        if (additive && l == 0) continue;
        cluster_sync();
        ml_residual<D, true>(v, lv.g[l], lv.lo[l], lv.lo[l + 1], t0, step);
        cluster_sync();
    }
}

}  // namespace mps
