// dfea_mg.cu -- geometric multigrid on structured quadrilateral grids: the kernels of a V-cycle
// preconditioner for the PCG of the Newton-Krylov solve.
//
// Levels.  Level 0 is the finite-element mesh (Q4, or Q9 whose nodes form a grid refined twice); every
// coarser level l >= 1 is a Q4 grid of gx x gy cells with bilinear interpolation between levels, each
// level halving the cell count of the one above it in both directions (a last cell one line wide when
// the count is odd).  Coarse operators are Galerkin products built element by element: level 1 from
// the stored Gauss-point moduli of the fine mesh, K_C = sum_{e in C} sum_q (B_q P~)^T C_q (B_q P~), and
// level l + 1 from level l's 8 x 8 element matrices, K_C = sum P^T K_c P.  P~ zeroes fixed fine DOFs, so
// a coarse DOF whose whole support is fixed has a zero row and becomes an identity row; the coarse
// operator equals P~^T A P~ of A = M K M + (I - M) on the free DOFs.
//
// Everything here is deterministic: node-centric gathers in a fixed order, single-block reductions.
#include <cmath>
#include <cstdio>
#include <new>
#include <utility>

#include "dfea_cluster.cuh"
#include "dfea_common.cuh"
#include "dfea_mg.cuh"

namespace dfea {

int validate_mesh(const dfea_mesh_view* mv, bool need_grad32);

struct MgGrid {
    int gx, gy;
    const int32_t* line_x;
    const int32_t* line_y;
    const int32_t* cell_x;
    const int32_t* cell_y;
    double* K;
    uint8_t* fix;
    double* S;  // node stencils (k_mg_stencil), or NULL: products from the element matrices
};

static MgGrid mg_grid(const dfea_mg_grid& g, double* stencil = nullptr) {
    return MgGrid{g.gx, g.gy, g.line_x, g.line_y, g.cell_x, g.cell_y, g.K, g.fix, stencil};
}

// num / den for the integers of the grid maps: lines are 1 or 2 apart, so the quotient is exact without a division
__device__ __forceinline__ double frac(int num, int den) {
    return den == 1 ? (double)num : (den == 2 ? 0.5 * num : (double)num / (double)den);
}

static int validate_grid(const dfea_mg_grid* g, bool coarse, const char* what) {
    if (!g || g->gx < 1 || g->gy < 1) return set_error(DFEA_ERR_INVALID, "%s: bad grid", what);
    if ((int64_t)(g->gx + 1) * (g->gy + 1) >= (int64_t(1) << 30)) return set_error(DFEA_ERR_INVALID, "%s: grid too large", what);
    if (coarse && (!g->line_x || !g->line_y || !g->cell_x || !g->cell_y))
        return set_error(DFEA_ERR_INVALID, "%s: a coarse grid needs its line and cell maps", what);
    return DFEA_OK;
}

// weight of coarse line c (lines X) at finer line i, for i in [X[c-1], X[c+1]]
__device__ __forceinline__ double hat(const int32_t* X, int n_lines, int c, int i) {
    const int xc = X[c];
    if (i == xc) return 1.0;
    if (i < xc) {
        if (c == 0) return 0.0;
        const int xl = X[c - 1];
        return i <= xl ? 0.0 : frac(i - xl, xc - xl);
    }
    if (c == n_lines - 1) return 0.0;
    const int xr = X[c + 1];
    return i >= xr ? 0.0 : frac(xr - i, xr - xc);
}

// ------------------------------------------------------------------------------------------
// level 1 from the finite-element mesh: K_C = sum_e sum_q (B_q P~)^T C_q (B_q P~)
// ------------------------------------------------------------------------------------------
// MOD 0: FP64 physical moduli (16 per Gauss point) with the mesh gradients; 1: FP32 physical moduli; 2, 3: FP32 and
// FP64 reference-frame moduli (10 per Gauss point, DFEA_F32REF, DFEA_F64REF) with the reference gradients.
template <int NEN, int NQ, int MOD>
__global__ void __launch_bounds__(128)
k_mg_galerkin_fe(Mesh m, const void* __restrict__ moduli, RefGrad<NEN, NQ> rg, const int32_t* __restrict__ node_ij,
                 const int32_t* __restrict__ cell_slot, int span, int epc, int ncy, MgGrid cg) {
    const int n_cells = cg.gx * cg.gy;
    const int64_t S = m.stride;
    for (int C = blockIdx.x * blockDim.x + threadIdx.x; C < n_cells; C += gridDim.x * blockDim.x) {
        const int CX = C / cg.gy, CY = C % cg.gy;
        const int x0 = cg.line_x[CX], x1 = cg.line_x[CX + 1], y0 = cg.line_y[CY], y1 = cg.line_y[CY + 1];
        double K[64];
#pragma unroll
        for (int k = 0; k < 64; ++k) K[k] = 0.0;
#pragma unroll 1
        for (int fcx = x0 / span; fcx < x1 / span; ++fcx) {
#pragma unroll 1
            for (int fce = (y0 / span) * epc; fce < (y1 / span) * epc; ++fce) {
                // element fce % epc of the cell (fcx, fce / epc)
                const int64_t s = cell_slot[((int64_t)fcx * ncy + fce / epc) * epc + fce % epc];
                double P[NEN][4];
                int fix[NEN];
#pragma unroll
                for (int a = 0; a < NEN; ++a) {
                    const int c = m.conn[a * S + s];
                    const int n = c >> 2;
                    fix[a] = c & 3;
                    const double wx1 = frac(node_ij[2 * n] - x0, x1 - x0), wy1 = frac(node_ij[2 * n + 1] - y0, y1 - y0);
                    const double wx0 = 1.0 - wx1, wy0 = 1.0 - wy1;
                    P[a][0] = wx0 * wy0;
                    P[a][1] = wx1 * wy0;
                    P[a][2] = wx1 * wy1;
                    P[a][3] = wx0 * wy1;
                }
#pragma unroll 1
                for (int q = 0; q < NQ; ++q) {
                    double g[NEN][2], M[16];
                    if constexpr (MOD >= 2) {
                        double h[10];
                        if constexpr (MOD == 2) {
                            const float* Cf = static_cast<const float*>(moduli);
                            const int64_t base = (int64_t)q * 10 * S;
                            const float4 A = reinterpret_cast<const float4*>(Cf + base)[s];
                            const float4 B = reinterpret_cast<const float4*>(Cf + base + 4 * S)[s];
                            const float2 D = reinterpret_cast<const float2*>(Cf + base + 8 * S)[s];
                            h[0] = A.x; h[1] = A.y; h[2] = A.z; h[3] = A.w; h[4] = B.x;
                            h[5] = B.y; h[6] = B.z; h[7] = B.w; h[8] = D.x; h[9] = D.y;
                        } else {
                            const double2* Cd = static_cast<const double2*>(moduli) + (int64_t)(q * 5) * S + s;
#pragma unroll
                            for (int k = 0; k < 5; ++k) {
                                const double2 t = Cd[k * S];
                                h[2 * k] = t.x;
                                h[2 * k + 1] = t.y;
                            }
                        }
                        // packed upper triangle: (0,0..3) (1,1..3) (2,2..3) (3,3)
                        M[0] = h[0]; M[1] = h[1]; M[2] = h[2]; M[3] = h[3];
                        M[5] = h[4]; M[6] = h[5]; M[7] = h[6];
                        M[10] = h[7]; M[11] = h[8];
                        M[15] = h[9];
                        M[4] = M[1]; M[8] = M[2]; M[12] = M[3]; M[9] = M[6]; M[13] = M[7]; M[14] = M[11];
#pragma unroll
                        for (int a = 0; a < NEN; ++a) {
                            g[a][0] = rg.g[q][a][0];
                            g[a][1] = rg.g[q][a][1];
                        }
                    } else {
#pragma unroll
                        for (int r = 0; r < 4; ++r) {
                            if constexpr (MOD == 0) {
                                double row[4];
                                load_moduli_row(static_cast<const double*>(moduli), S, q, r, s, row);
#pragma unroll
                                for (int c = 0; c < 4; ++c) M[4 * r + c] = row[c];
                            } else {
                                float row[4];
                                load_moduli_row(static_cast<const float*>(moduli), S, q, r, s, row);
#pragma unroll
                                for (int c = 0; c < 4; ++c) M[4 * r + c] = row[c];
                            }
                        }
#pragma unroll
                        for (int a = 0; a < NEN; ++a) {
                            const double2 t = load_grad(m.grad, (int64_t)(q * NEN + a) * S + s);
                            g[a][0] = t.x;
                            g[a][1] = t.y;
                        }
                    }
                    // coarse gradients per component: G[i][b][J] = sum_a P~_(a,i),b dN_a,J
                    double G[2][4][2];
#pragma unroll
                    for (int i = 0; i < 2; ++i)
#pragma unroll
                        for (int b = 0; b < 4; ++b) {
                            double s0 = 0.0, s1 = 0.0;
#pragma unroll
                            for (int a = 0; a < NEN; ++a) {
                                const double w = (fix[a] >> i) & 1 ? 0.0 : P[a][b];
                                s0 += w * g[a][0];
                                s1 += w * g[a][1];
                            }
                            G[i][b][0] = s0;
                            G[i][b][1] = s1;
                        }
#pragma unroll
                    for (int c = 0; c < 4; ++c)
#pragma unroll
                        for (int k = 0; k < 2; ++k) {
                            double t[4];
#pragma unroll
                            for (int r = 0; r < 4; ++r) t[r] = M[4 * r + 2 * k] * G[k][c][0] + M[4 * r + 2 * k + 1] * G[k][c][1];
#pragma unroll
                            for (int b = 0; b < 4; ++b)
#pragma unroll
                                for (int i = 0; i < 2; ++i)
                                    K[(2 * b + i) * 8 + 2 * c + k] += G[i][b][0] * t[2 * i] + G[i][b][1] * t[2 * i + 1];
                        }
                }
            }
        }
#pragma unroll
        for (int k = 0; k < 64; ++k) cg.K[(int64_t)k * n_cells + C] = K[k];
    }
}

// ------------------------------------------------------------------------------------------
// level l + 1 from level l: K_C = sum_{fine cells c in C} P_c^T K_c P_c
// ------------------------------------------------------------------------------------------
// One thread per coarse cell and column of its matrix (cells fastest): a level of a few hundred cells fills more of
// the chip than with a thread per cell (26 us a level on the serving meshes, whatever its size), in the same order.
__global__ void __launch_bounds__(128) k_mg_galerkin(MgGrid fg, MgGrid cg) {
    const int n_cells = cg.gx * cg.gy, nf_cells = fg.gx * fg.gy;
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < 8 * n_cells; t += gridDim.x * blockDim.x) {
        const int col = t / n_cells, C = t - col * n_cells, kc = col & 1, bc = col >> 1;
        const int CX = C / cg.gy, CY = C % cg.gy;
        const int x0 = cg.line_x[CX], x1 = cg.line_x[CX + 1], y0 = cg.line_y[CY], y1 = cg.line_y[CY + 1];
        double K[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) K[k] = 0.0;
#pragma unroll 1
        for (int fx = x0; fx < x1; ++fx) {
#pragma unroll 1
            for (int fy = y0; fy < y1; ++fy) {
                const int fc = fx * fg.gy + fy;
                // P[a][b]: weight of coarse corner b at fine corner a (corners (0,0) (1,0) (1,1) (0,1))
                double P[4][4], Pc[4];
#pragma unroll
                for (int a = 0; a < 4; ++a) {
                    const int i = fx + ((a == 1 || a == 2) ? 1 : 0), j = fy + ((a >= 2) ? 1 : 0);
                    const double wx1 = frac(i - x0, x1 - x0), wy1 = frac(j - y0, y1 - y0);
                    const double wx0 = 1.0 - wx1, wy0 = 1.0 - wy1;
                    P[a][0] = wx0 * wy0;
                    P[a][1] = wx1 * wy0;
                    P[a][2] = wx1 * wy1;
                    P[a][3] = wx0 * wy1;
                    Pc[a] = bc == 0 ? P[a][0] : bc == 1 ? P[a][1] : bc == 2 ? P[a][2] : P[a][3];
                }
                // t = column of K_c P, then K += P^T t; P acts on both components alike
                double tc[8];
#pragma unroll
                for (int row = 0; row < 8; ++row) {
                    double acc = 0.0;
#pragma unroll
                    for (int a = 0; a < 4; ++a) acc += fg.K[(int64_t)(row * 8 + 2 * a + kc) * nf_cells + fc] * Pc[a];
                    tc[row] = acc;
                }
#pragma unroll
                for (int bb = 0; bb < 4; ++bb)
#pragma unroll
                    for (int i = 0; i < 2; ++i) {
                        double acc = 0.0;
#pragma unroll
                        for (int a = 0; a < 4; ++a) acc += P[a][bb] * tc[2 * a + i];
                        K[2 * bb + i] += acc;
                    }
            }
        }
#pragma unroll
        for (int r = 0; r < 8; ++r) cg.K[(int64_t)(r * 8 + col) * n_cells + C] = K[r];
    }
}

// ------------------------------------------------------------------------------------------
// node stencils: the rows of a coarse operator as the 2 x 2 blocks of a node with itself and its eight neighbours
// ------------------------------------------------------------------------------------------
// Block of node n = (I, J) with node (I + di, J + dj), both rows r and columns c as c4[2 r + c], summed over the cells
// that hold both nodes in cell order; the identity of a fixed DOF on the diagonal.
__device__ __forceinline__ void mg_stencil_block(const MgGrid& g, int I, int J, int di, int dj, double (&c4)[4]) {
    const int n_cells = g.gx * g.gy;
#pragma unroll
    for (int k = 0; k < 4; ++k) c4[k] = 0.0;
#pragma unroll
    for (int cx = -1; cx <= 0; ++cx)
#pragma unroll
        for (int cy = -1; cy <= 0; ++cy) {
            const int CX = I + cx, CY = J + cy;
            const int ai = -cx, aj = -cy, bi = di - cx, bj = dj - cy;  // corners of the two nodes in the cell
            if (bi < 0 || bi > 1 || bj < 0 || bj > 1 || CX < 0 || CY < 0 || CX >= g.gx || CY >= g.gy) continue;
            const int a = aj ? (ai ? 2 : 3) : ai, b = bj ? (bi ? 2 : 3) : bi;
            const int c = CX * g.gy + CY;
#pragma unroll
            for (int r = 0; r < 2; ++r)
#pragma unroll
                for (int q = 0; q < 2; ++q) c4[2 * r + q] += g.K[(int64_t)((2 * a + r) * 8 + 2 * b + q) * n_cells + c];
        }
    if (di == 0 && dj == 0) {
        const int f = g.fix[I * (g.gy + 1) + J];
        if (f & 1) c4[0] += 1.0;
        if (f & 2) c4[3] += 1.0;
    }
}

// S[(4 m + k) N + n], m = 3 (di + 1) + dj + 1: 36 numbers a node where the cells around it hold 64, and no identity or
// grid-edge cases left in the products.  diag: the operator's diagonal.  One thread per node and neighbour.
__global__ void __launch_bounds__(256) k_mg_stencil(MgGrid g, double* __restrict__ diag) {
    const int N = (g.gx + 1) * (g.gy + 1), ny = g.gy + 1;
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < 9 * N; t += gridDim.x * blockDim.x) {
        const int m = t / N, n = t - m * N;
        const int di = m / 3 - 1, dj = m % 3 - 1;
        double c4[4];
        mg_stencil_block(g, n / ny, n % ny, di, dj, c4);
#pragma unroll
        for (int k = 0; k < 4; ++k) g.S[(int64_t)(4 * m + k) * N + n] = c4[k];
        if (m == 4) reinterpret_cast<double2*>(diag)[n] = make_double2(c4[0], c4[3]);
    }
}

// The product's row at node n from its stencil: load(id) v at a neighbour, entry(4 m + k) of the stencil.  A neighbour
// past the grid's edge has a zero block: the node's own value stands in, so all nine loads are issued before the sums.
template <typename Load, typename Entry>
__device__ __forceinline__ double2 mg_stencil_row(const MgGrid& g, Load&& load, Entry&& entry, int n) {
    const int ny = g.gy + 1, I = n / ny, J = n - I * ny;
    double2 v[9];
#pragma unroll
    for (int m = 0; m < 9; ++m) {
        const int i = I + m / 3 - 1, j = J + m % 3 - 1;
        const bool in = i >= 0 && i <= g.gx && j >= 0 && j <= g.gy;
        v[m] = load(in ? n + (m / 3 - 1) * ny + m % 3 - 1 : n);
    }
    double2 y[3];  // a sum per grid line: three short chains
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        y[i] = make_double2(0.0, 0.0);
#pragma unroll
        for (int j = 0; j < 3; ++j) {
            const int m = 3 * i + j;
            y[i].x += entry(4 * m) * v[m].x + entry(4 * m + 1) * v[m].y;
            y[i].y += entry(4 * m + 2) * v[m].x + entry(4 * m + 3) * v[m].y;
        }
    }
    return make_double2(y[0].x + y[1].x + y[2].x, y[0].y + y[1].y + y[2].y);
}

// ------------------------------------------------------------------------------------------
// transfers; gnode maps a grid node of the finer level to its DOF node (level 0: the FE node id, -1 where
// the grid has no node), NULL for the lexicographic numbering of the coarse levels
// ------------------------------------------------------------------------------------------
__device__ __forceinline__ int fine_node(const int32_t* gnode, int fgy, int i, int j) {
    const int id = i * (fgy + 1) + j;
    return gnode ? gnode[id] : id;
}

// rc = P~^T r (masked at fixed fine DOFs); with fix_out, also the coarse fix bits (a coarse DOF is fixed
// when every fine DOF it interpolates to is fixed)
// coarse node n of the restriction r_c = P~^T r (and the coarse fixed-DOF bits); load(id): r at a fine node.  The
// kernels below and the cluster tail of the V-cycle share these per-node functions.
template <bool SUM, typename Load>
__device__ __forceinline__ double2 mg_restrict_sum(const MgGrid& fg, const MgGrid& cg, const int32_t* gnode,
                                                   const uint8_t* ffix, Load&& load, int n, int* fixed) {
    const int nx = cg.gx + 1, ny = cg.gy + 1;
    const int I = n / ny, J = n % ny;
    const int xc = cg.line_x[I], xl = I > 0 ? cg.line_x[I - 1] : xc, xr = I < cg.gx ? cg.line_x[I + 1] : xc;
    const int yc = cg.line_y[J], yl = J > 0 ? cg.line_y[J - 1] : yc, yr = J < cg.gy ? cg.line_y[J + 1] : yc;
    double ax = 0.0, ay = 0.0;
    int free_bits = 0;
    if (xc - xl <= 2 && xr - xc <= 2 && yc - yl <= 2 && yr - yc <= 2) {
        // lines one or two apart: the node itself and the fine lines halfway to its neighbours, all loads first
        int id[9], f[9];
        double2 t[9];
        double w[9];
#pragma unroll
        for (int m = 0; m < 9; ++m) {
            const int a = m / 3 - 1, b = m % 3 - 1;
            const bool in = (a == 0 || (a < 0 ? xc - xl == 2 : xr - xc == 2)) && (b == 0 || (b < 0 ? yc - yl == 2 : yr - yc == 2));
            w[m] = in ? (a == 0 ? 1.0 : 0.5) * (b == 0 ? 1.0 : 0.5) : 0.0;
            id[m] = fine_node(gnode, fg.gy, in ? xc + a : xc, in ? yc + b : yc);
        }
#pragma unroll
        for (int m = 0; m < 9; ++m) {
            const bool there = id[m] >= 0;
            f[m] = there ? ffix[id[m]] : 3;
            t[m] = SUM && there ? load(id[m]) : make_double2(0.0, 0.0);
        }
#pragma unroll
        for (int m = 0; m < 9; ++m) {
            if (w[m] == 0.0 || id[m] < 0) continue;
            if (SUM && !(f[m] & 1)) ax += w[m] * t[m].x;
            if (SUM && !(f[m] & 2)) ay += w[m] * t[m].y;
            free_bits |= (~f[m]) & 3;
        }
        if (fixed) *fixed = (~free_bits) & 3;
        return make_double2(ax, ay);
    }
    const int ilo = I > 0 ? xl + 1 : xc, ihi = I < cg.gx ? xr - 1 : xc;
    const int jlo = J > 0 ? yl + 1 : yc, jhi = J < cg.gy ? yr - 1 : yc;
    for (int i = ilo; i <= ihi; ++i) {
        const double wx = hat(cg.line_x, nx, I, i);
        for (int j = jlo; j <= jhi; ++j) {
            const int id = fine_node(gnode, fg.gy, i, j);
            if (id < 0) continue;
            const double w = wx * hat(cg.line_y, ny, J, j);
            const int f = ffix[id];
            if (SUM) {
                const double2 t = load(id);
                if (!(f & 1)) ax += w * t.x;
                if (!(f & 2)) ay += w * t.y;
            }
            if (w > 0.0) free_bits |= (~f) & 3;
        }
    }
    if (fixed) *fixed = (~free_bits) & 3;
    return make_double2(ax, ay);
}

__global__ void k_mg_restrict(MgGrid fg, MgGrid cg, const int32_t* __restrict__ gnode, const uint8_t* __restrict__ ffix,
                              const double* __restrict__ r, double* __restrict__ rc, uint8_t* __restrict__ fix_out) {
    const int n_nodes = (cg.gx + 1) * (cg.gy + 1);
    const double2* r2 = reinterpret_cast<const double2*>(r);
    const auto load = [&](int id) { return r2[id]; };
    for (int n = blockIdx.x * blockDim.x + threadIdx.x; n < n_nodes; n += gridDim.x * blockDim.x) {
        int fixed;
        const double2 t = r ? mg_restrict_sum<true>(fg, cg, gnode, ffix, load, n, &fixed)
                            : mg_restrict_sum<false>(fg, cg, gnode, ffix, load, n, &fixed);
        if (rc) reinterpret_cast<double2*>(rc)[n] = t;
        if (fix_out) fix_out[n] = (uint8_t)fixed;
    }
}

// x += P~ ec (x untouched at fixed fine DOFs) at fine grid node n; load(c): ec at a coarse node, x(id): the fine value
template <typename Load, typename X>
__device__ __forceinline__ void mg_prolong_node(const MgGrid& fg, const MgGrid& cg, const int32_t* gnode,
                                                const uint8_t* ffix, Load&& load, X&& x, int n) {
    const int fny = fg.gy + 1, cny = cg.gy + 1;
    const int i = n / fny, j = n % fny;
    const int id = gnode ? gnode[n] : n;
    if (id < 0) return;
    const int f = ffix[id];
    if ((f & 3) == 3) return;
    const int CX = cg.cell_x[i], CY = cg.cell_y[j];
    const int x0 = cg.line_x[CX], x1 = cg.line_x[CX + 1], y0 = cg.line_y[CY], y1 = cg.line_y[CY + 1];
    const double wx1 = frac(i - x0, x1 - x0), wy1 = frac(j - y0, y1 - y0);
    const double wx0 = 1.0 - wx1, wy0 = 1.0 - wy1;
    const double2 e00 = load(CX * cny + CY), e10 = load((CX + 1) * cny + CY);
    const double2 e11 = load((CX + 1) * cny + CY + 1), e01 = load(CX * cny + CY + 1);
    double2& t = x(id);
    if (!(f & 1)) t.x += wx0 * wy0 * e00.x + wx1 * wy0 * e10.x + wx1 * wy1 * e11.x + wx0 * wy1 * e01.x;
    if (!(f & 2)) t.y += wx0 * wy0 * e00.y + wx1 * wy0 * e10.y + wx1 * wy1 * e11.y + wx0 * wy1 * e01.y;
}

__global__ void k_mg_prolong_add(MgGrid fg, MgGrid cg, const int32_t* __restrict__ gnode, const uint8_t* __restrict__ ffix,
                                 const double* ec, double* x) {
    grid_dependency_wait();
    grid_dependents_launch();
    const int n_nodes = (fg.gx + 1) * (fg.gy + 1);
    for (int n = blockIdx.x * blockDim.x + threadIdx.x; n < n_nodes; n += gridDim.x * blockDim.x)
        mg_prolong_node(fg, cg, gnode, ffix, [&](int c) { return load_fresh(reinterpret_cast<const double2*>(ec) + c); },
                        [&](int id) -> double2& { return reinterpret_cast<double2*>(x)[id]; }, n);
}

// ------------------------------------------------------------------------------------------
// coarse-level operator: y = K v + (I - M) v (K has zero rows and columns at fixed DOFs); DIAG: diag(A)
// ------------------------------------------------------------------------------------------
// row of node n = I * ny + J (both DOFs): from the stencil, or from the element matrices of the cells around the node
template <bool DIAG, typename Load>
__device__ __forceinline__ double2 mg_node_row(const MgGrid& g, Load&& load, int n) {
    const int ny = g.gy + 1, n_cells = g.gx * g.gy;
    if (!DIAG && g.S != nullptr) {
        const int64_t N = (int64_t)(g.gx + 1) * ny;
        return mg_stencil_row(g, load, [&](int k) { return g.S[k * N + n]; }, n);
    }
    const int I = n / ny, J = n % ny;
    double y0 = 0.0, y1 = 0.0;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        // cells around the node and the node's corner in each: (I-1,J-1):2 (I,J-1):3 (I,J):0 (I-1,J):1
        const int CX = (k == 0 || k == 3) ? I - 1 : I, CY = (k <= 1) ? J - 1 : J;
        const int b = k == 0 ? 2 : k == 1 ? 3 : k == 2 ? 0 : 1;
        if (CX < 0 || CY < 0 || CX >= g.gx || CY >= g.gy) continue;
        const int c = CX * g.gy + CY;
        if (DIAG) {
            y0 += g.K[(int64_t)((2 * b) * 8 + 2 * b) * n_cells + c];
            y1 += g.K[(int64_t)((2 * b + 1) * 8 + 2 * b + 1) * n_cells + c];
        } else {
            const int cn[4] = {CX * ny + CY, (CX + 1) * ny + CY, (CX + 1) * ny + CY + 1, CX * ny + CY + 1};
#pragma unroll
            for (int a = 0; a < 4; ++a) {
                const double2 t = load(cn[a]);
                y0 += g.K[(int64_t)((2 * b) * 8 + 2 * a) * n_cells + c] * t.x +
                      g.K[(int64_t)((2 * b) * 8 + 2 * a + 1) * n_cells + c] * t.y;
                y1 += g.K[(int64_t)((2 * b + 1) * 8 + 2 * a) * n_cells + c] * t.x +
                      g.K[(int64_t)((2 * b + 1) * 8 + 2 * a + 1) * n_cells + c] * t.y;
            }
        }
    }
    const int f = g.fix[n];
    if (DIAG) {
        y0 = (f & 1) ? 1.0 : y0;
        y1 = (f & 2) ? 1.0 : y1;
    } else {
        const double2 t = load(n);
        if (f & 1) y0 += t.x;
        if (f & 2) y1 += t.y;
    }
    return make_double2(y0, y1);
}

template <bool DIAG>
__global__ void __launch_bounds__(256) k_mg_apply(MgGrid g, const double* __restrict__ v, double* __restrict__ y) {
    const int n_nodes = (g.gx + 1) * (g.gy + 1);
    const double2* v2 = reinterpret_cast<const double2*>(v);
    for (int n = blockIdx.x * blockDim.x + threadIdx.x; n < n_nodes; n += gridDim.x * blockDim.x)
        reinterpret_cast<double2*>(y)[n] = mg_node_row<DIAG>(g, [&](int i) { return v2[i]; }, n);
}

// ------------------------------------------------------------------------------------------
// Chebyshev smoothing steps (the Chebyshev iteration, e.g. Saad, Iterative Methods, Alg. 12.1, with the
// Jacobi diagonal as preconditioner)
// ------------------------------------------------------------------------------------------
// the coefficients are read from device memory, so a captured cycle follows them from one linearisation
// to the next
__global__ void k_mg_cheb_start(int64_t n, const double* __restrict__ r, const double* __restrict__ diag,
                                const double* __restrict__ scale, double* __restrict__ d) {
    const double s = *scale;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        d[i] = s * r[i] / diag[i];
}

__global__ void k_mg_cheb_step(int64_t n, double* __restrict__ x, double* __restrict__ r, double* __restrict__ d,
                               const double* __restrict__ q, const double* __restrict__ diag,
                               const double* __restrict__ c, int last) {
    const double c1 = last ? 0.0 : c[0], c2 = last ? 0.0 : c[1];
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const double di = d[i];
        x[i] += di;
        const double ri = r[i] - q[i];
        r[i] = ri;
        if (!last) d[i] = c1 * di + c2 * ri / diag[i];
    }
}

// Fused forms used inside a V-cycle.  A pre-smoothing starts from x = 0: its first step stores x = d and takes the
// residual before it from b.  A post-smoothing's residual has no reader, so its last step has no product: the pass
// before adds the new direction to x as well.  Launched with programmatic dependent launch, like the passes around them.

// start of the pre-smoothing on level 0 without node incidence: r = b, x = 0, d = s r / D
__global__ void k_mg_cheb_first(int64_t n, const double* __restrict__ b, const double* __restrict__ diag,
                                const double* __restrict__ scale, double* __restrict__ r, double* __restrict__ x,
                                double* __restrict__ d) {
    const double s = *scale;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const double bi = b[i];
        r[i] = bi;
        x[i] = 0.0;
        d[i] = s * bi / diag[i];
    }
}

// start of the post-smoothing there from the product q = A x in memory: r = b - q, d = s r / D
__global__ void k_mg_cheb_restart(int64_t n, const double* __restrict__ b, const double* __restrict__ q,
                                  const double* __restrict__ diag, const double* __restrict__ scale,
                                  double* __restrict__ r, double* __restrict__ d) {
    const double s = *scale;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const double ri = b[i] - q[i];
        r[i] = ri;
        d[i] = s * ri / diag[i];
    }
}

// the restriction onto a level, with its right-hand side the first direction d = s b / D
__global__ void __launch_bounds__(256) k_mg_restrict_first(MgGrid fg, MgGrid cg, const int32_t* __restrict__ gnode,
                                                           const uint8_t* __restrict__ ffix, const double* r,
                                                           const double* __restrict__ diag, const double* __restrict__ scale,
                                                           double* __restrict__ b, double* __restrict__ d) {
    grid_dependency_wait();
    grid_dependents_launch();
    const double s = *scale;
    const int n_nodes = (cg.gx + 1) * (cg.gy + 1);
    const double2* r2 = reinterpret_cast<const double2*>(r);
    for (int n = blockIdx.x * blockDim.x + threadIdx.x; n < n_nodes; n += gridDim.x * blockDim.x) {
        const double2 t = mg_restrict_sum<true>(fg, cg, gnode, ffix, [&](int id) { return load_fresh(r2 + id); }, n, nullptr);
        const double2 D = reinterpret_cast<const double2*>(diag)[n];
        reinterpret_cast<double2*>(b)[n] = t;
        reinterpret_cast<double2*>(d)[n] = make_double2(s * t.x / D.x, s * t.y / D.y);
    }
}

// start of the post-smoothing on a coarse level: r = b - A x, d = s r / D
__global__ void __launch_bounds__(256) k_mg_residual_restart(MgGrid g, const double* __restrict__ b,
                                                             const double* x, const double* __restrict__ diag,
                                                             const double* __restrict__ scale, double* __restrict__ r,
                                                             double* __restrict__ d) {
    grid_dependency_wait();
    grid_dependents_launch();
    const double s = *scale;
    const double2* x2 = reinterpret_cast<const double2*>(x);
    const int n_nodes = (g.gx + 1) * (g.gy + 1);
    for (int n = blockIdx.x * blockDim.x + threadIdx.x; n < n_nodes; n += gridDim.x * blockDim.x) {
        const double2 q = mg_node_row<false>(g, [&](int i) { return load_fresh(x2 + i); }, n);
        const double2 bn = reinterpret_cast<const double2*>(b)[n], dn = reinterpret_cast<const double2*>(diag)[n];
        const double r0 = bn.x - q.x, r1 = bn.y - q.y;
        reinterpret_cast<double2*>(r)[n] = make_double2(r0, r1);
        reinterpret_cast<double2*>(d)[n] = make_double2(s * r0 / dn.x, s * r1 / dn.y);
    }
}

// one Chebyshev step on a coarse level with its product computed at the node: q = A d_in, x += d_in, r = r_in - q,
// d_out = c1 d_in + c2 r / D (double-buffered: neighbouring nodes read d_in).  last: no next direction; add: the next
// direction goes into x at once and neither it nor r is stored; first: x = d_in.
__global__ void __launch_bounds__(256) k_mg_cheb_apply_step(MgGrid g, double* x, const double* r_in, double* r,
                                                            const double* d_in, double* __restrict__ d_out,
                                                            const double* __restrict__ diag, const double* __restrict__ c,
                                                            int first, int last, int add) {
    grid_dependency_wait();
    grid_dependents_launch();
    const double c1 = last ? 0.0 : c[0], c2 = last ? 0.0 : c[1];
    const double2* d2 = reinterpret_cast<const double2*>(d_in);
    double2* x2 = reinterpret_cast<double2*>(x);
    const int n_nodes = (g.gx + 1) * (g.gy + 1);
    for (int n = blockIdx.x * blockDim.x + threadIdx.x; n < n_nodes; n += gridDim.x * blockDim.x) {
        const double2 q = mg_node_row<false>(g, [&](int i) { return load_fresh(d2 + i); }, n), dn = load_fresh(d2 + n);
        double2 xn = first ? make_double2(0.0, 0.0) : x2[n];
        xn.x += dn.x;
        xn.y += dn.y;
        const double2 rn = load_fresh(reinterpret_cast<const double2*>(r_in) + n);
        const double r0 = rn.x - q.x, r1 = rn.y - q.y;
        if (!last) {
            const double2 Dn = reinterpret_cast<const double2*>(diag)[n];
            const double2 dd = make_double2(c1 * dn.x + c2 * r0 / Dn.x, c1 * dn.y + c2 * r1 / Dn.y);
            if (add) {
                xn.x += dd.x;
                xn.y += dd.y;
            } else {
                reinterpret_cast<double2*>(d_out)[n] = dd;
            }
        }
        x2[n] = xn;
        if (!add) reinterpret_cast<double2*>(r)[n] = make_double2(r0, r1);
    }
}

// ------------------------------------------------------------------------------------------
// Lanczos by Jacobi-preconditioned CG (the extreme eigenvalue of D^-1 A from the CG coefficients): the
// scalars stay on the device, s = [p.Ap, r.z, -, beta], hist = (alpha_k, beta_k) per step
// ------------------------------------------------------------------------------------------
// Dot products in two fixed-order passes: per-block partial sums (the block count depends on n only), then
// one block adds them in block order.
constexpr int kMgDotBlocks = 296;
constexpr int kMgDotThreads = 256;

__host__ __device__ static int mg_dot_blocks(int64_t n) {
    const int64_t b = (n + 4 * kMgDotThreads - 1) / (4 * kMgDotThreads);
    return (int)(b < 1 ? 1 : (b > kMgDotBlocks ? kMgDotBlocks : b));
}

// The library's own drivers take a dot product in ONE launch: every block stores its partial sum, and the last block to
// arrive (an integer ticket after the partials in dot_work, zeroed at every set-up and reset by that block) adds them.
__global__ void __launch_bounds__(kMgDotThreads) k_mg_dot_part(int64_t n, const double* __restrict__ x,
                                                                const double* __restrict__ y, double* __restrict__ part) {
    double a = 0.0;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        a += x[i] * y[i];
    a = block_sum<kMgDotThreads>(a);
    if (threadIdx.x == 0) part[blockIdx.x] = a;
}

// x.y in one launch (grid: mg_dot_blocks(n) blocks of kMgDotThreads)
template <int KIND>
__global__ void __launch_bounds__(kMgDotThreads) k_mg_dot1(int64_t n, const double* __restrict__ x,
                                                            const double* __restrict__ y, double* __restrict__ work,
                                                            double* __restrict__ out) {
    double a = 0.0;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        a += x[i] * y[i];
    dot_finish<kMgDotThreads, KIND>(a, work, out, nullptr, 0);
}
template <int KIND>
static int mg_dot1(int64_t n, const double* x, const double* y, double* out, double* work, cudaStream_t s) {
    k_mg_dot1<KIND><<<mg_dot_blocks(n), kMgDotThreads, 0, s>>>(n, x, y, work, out);
    note_launches(1);
    return launch_check("multigrid dot");
}

// k_mg_lanczos_step and the following r.z in one launch: r -= alpha q, z = r / D with alpha = s[1] / s[0], then the CG
// step's bookkeeping
__global__ void __launch_bounds__(kMgDotThreads) k_mg_lanczos_step_rz(int64_t n, const double* q,
                                                                       double* r, double* z,
                                                                       const double* __restrict__ diag,
                                                                       double* s, double* __restrict__ work,
                                                                       double* __restrict__ hist, int k) {
    grid_dependency_wait();
    grid_dependents_launch();
    const double alpha = s[1] / s[0];
    double a = 0.0;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const double ri = r[i] - alpha * load_fresh(q + i);
        r[i] = ri;
        const double zi = ri / diag[i];
        z[i] = zi;
        a += ri * zi;
    }
    dot_finish<kMgDotThreads, MG_DOT_LANCZOS>(a, work, s, hist, k);
}

// start of an estimate: r = sin(i + 1), z = r / D, p = z, s = [-, r.z, -, 0]
__global__ void __launch_bounds__(kMgDotThreads) k_mg_lanczos_start(int64_t n, double* __restrict__ r, double* __restrict__ z,
                                                                     double* __restrict__ p, const double* __restrict__ diag,
                                                                     double* __restrict__ s, double* __restrict__ work) {
    if (blockIdx.x == 0 && threadIdx.x == 0) s[3] = 0.0;
    double a = 0.0;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const double ri = sin((double)(i + 1)), zi = ri / diag[i];
        r[i] = ri;
        z[i] = zi;
        p[i] = zi;
        a += ri * zi;
    }
    dot_finish<kMgDotThreads, MG_DOT_PLAIN>(a, work, s + 1, nullptr, 0);
}

// a step's product on a coarse level: p_out = z + beta p_in, q = A p_out, s[0] = p.q (double-buffered: neighbouring
// nodes read p_in)
__global__ void __launch_bounds__(kMgDotThreads) k_mg_lanczos_apply(MgGrid g, const double* z,
                                                                     const double* p_in, double* __restrict__ p_out,
                                                                     double* __restrict__ q, double* s,
                                                                     double* __restrict__ work) {
    grid_dependency_wait();
    grid_dependents_launch();
    const double beta = s[3];
    const double2 *z2 = reinterpret_cast<const double2*>(z), *p2 = reinterpret_cast<const double2*>(p_in);
    const auto direction = [&](int i) {
        const double2 zn = load_fresh(z2 + i), pn = load_fresh(p2 + i);
        return make_double2(zn.x + beta * pn.x, zn.y + beta * pn.y);
    };
    double a = 0.0;
    const int n_nodes = (g.gx + 1) * (g.gy + 1);
    for (int n = blockIdx.x * blockDim.x + threadIdx.x; n < n_nodes; n += gridDim.x * blockDim.x) {
        const double2 qn = mg_node_row<false>(g, direction, n), pn = direction(n);
        reinterpret_cast<double2*>(p_out)[n] = pn;
        reinterpret_cast<double2*>(q)[n] = qn;
        a += pn.x * qn.x + pn.y * qn.y;
    }
    dot_finish<kMgDotThreads, MG_DOT_PLAIN>(a, work, s, nullptr, 0);
}

// LANCZOS: the sum is r.z of a CG step: alpha = s[1] / s[0], beta = sum / s[1] into hist, s[1] = sum, s[3] = beta
template <bool LANCZOS>
__global__ void __launch_bounds__(kMgDotThreads) k_mg_dot_final(int nb, const double* __restrict__ part,
                                                                 double* __restrict__ out, double* __restrict__ hist, int k) {
    double a = 0.0;
    for (int b = threadIdx.x; b < nb; b += blockDim.x) a += part[b];
    a = block_sum<kMgDotThreads>(a);
    if (threadIdx.x == 0) {
        if (LANCZOS) {
            const double alpha = out[1] / out[0], beta = a / out[1];
            hist[2 * k] = alpha;
            hist[2 * k + 1] = beta;
            out[1] = a;
            out[3] = beta;
        } else {
            *out = a;
        }
    }
}

__global__ void k_mg_lanczos_step(int64_t n, const double* __restrict__ q, double* __restrict__ r, double* __restrict__ z,
                                  const double* __restrict__ diag, const double* __restrict__ s) {
    const double alpha = s[1] / s[0];
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const double ri = r[i] - alpha * q[i];
        r[i] = ri;
        z[i] = ri / diag[i];
    }
}

__global__ void k_mg_lanczos_p(int64_t n, double* __restrict__ p, const double* __restrict__ z, const double* __restrict__ s) {
    const double beta = s[3];
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        p[i] = z[i] + beta * p[i];
}

// ------------------------------------------------------------------------------------------
// the small levels in distributed shared memory
// ------------------------------------------------------------------------------------------
// Levels of at most kMgTailNodes nodes are worked on by thread-block clusters: the nodes of a level are divided over the
// cluster's blocks in ranges, its vectors, its rows (node stencils) and its 1 / D lie in the owners' shared memory, and
// cluster barriers separate the phases.  What bounds a phase is latency: a gather through distributed shared memory, two
// chains of multiply-adds, a barrier: 1.7 us.  (A launch per phase costs 5 - 6 us; one block alone streams the rows
// through one SM; rows read from L2, divisions by D and neighbours loaded one after the other left a phase at 4 us.)
// The tail of a 128 x 128 Q9 cycle (levels of 4,225 nodes down to 25): 100 us in one block, plus 44 us of launches for
// the 4,225-node level, -> 54 us; the Lanczos estimates of these levels 247 -> 51 us, the clusters side by side.
constexpr int kMgTailNodes = 6000;
constexpr int kMgTailNodeBytes = 6 * 16 + 36 * 8;  // of a tail level: b, x, r, d, q, 1 / D and the node's rows
constexpr int kMgClusterThreads = 512;
constexpr int kMgClusterWarps = kMgClusterThreads / 32;

// a level's vector: entry n at place n % nb of block n / nb (n below 2^22: the quotient by a float reciprocal is exact)
struct ClusterVec {
    double2* mine;  // this block's range
    unsigned here;  // its shared address, the same in every block
    int nb;
    float inv_nb;
    __device__ __forceinline__ ClusterVec(unsigned char* smem, int offset, int nb_)
        : mine(reinterpret_cast<double2*>(smem + offset)), here((unsigned)__cvta_generic_to_shared(smem + offset)), nb(nb_),
          inv_nb(1.0f / (float)nb_) {}
    __device__ __forceinline__ double2 operator()(int n) const {
        const int who = (int)(((float)n + 0.5f) * inv_nb), at = n - who * nb;
        return cluster_load(cluster_address(here + at * 16, who));
    }
};

// the stencils of this block's nodes to shared memory, rows[entry][node]
__device__ __forceinline__ void load_rows(const MgGrid& g, double* rows, int nb, int first, int n_own, int n_nodes) {
    for (int t = threadIdx.x; t < 36 * n_own; t += kMgClusterThreads) {
        const int e = t / n_own, i = t - e * n_own;
        rows[e * nb + i] = __ldg(g.S + (int64_t)e * n_nodes + first + i);
    }
}

struct MgLanczosLevel {
    MgGrid grid;
    int n_nodes, nb;             // nodes, nodes per block
    const double* diag;
    double* s;                   // [p.Ap, r.z, -, beta]
    double* hist;                // (alpha_k, beta_k) per step
};

struct MgLanczosTail {
    int steps, size;             // blocks of a level's cluster
    MgLanczosLevel lv[DFEA_MG_MAX_LEVELS];
};

// Lanczos of the small smoothed levels, one cluster per level side by side: r = sin(i + 1), z = r / D, p = z, then the
// CG steps of the separate launches (their sums in the cluster's order)
__global__ void __launch_bounds__(kMgClusterThreads, 1) k_mg_tail_lanczos(const __grid_constant__ MgLanczosTail T) {
    constexpr int NT = kMgClusterThreads;
    extern __shared__ __align__(16) unsigned char mg_smem[];
    __shared__ double table[ClusterExchange<kMgClusterWarps>::kDoubles];
    const unsigned rank = cluster_rank();
    const MgLanczosLevel& L = T.lv[blockIdx.x / T.size];
    ClusterExchange<kMgClusterWarps> sums(table, rank, T.size);
    const ClusterVec p(mg_smem, 0, L.nb);
    double2* r = p.mine + L.nb;
    double2* z = p.mine + 2 * L.nb;
    double2* q = p.mine + 3 * L.nb;
    double* rows = reinterpret_cast<double*>(q + L.nb);
    const int first = rank * L.nb, n_own = min(L.nb, max(0, L.n_nodes - first));
    load_rows(L.grid, rows, L.nb, first, n_own, L.n_nodes);
    const double2* diag2 = reinterpret_cast<const double2*>(L.diag) + first;
    double rz = 0.0;
    for (int i = threadIdx.x; i < n_own; i += NT) {
        const double2 rn = make_double2(sin((double)(2 * (first + i) + 1)), sin((double)(2 * (first + i) + 2)));
        const double2 D = diag2[i], zn = make_double2(rn.x / D.x, rn.y / D.y);
        r[i] = rn;
        z[i] = zn;
        p.mine[i] = zn;
        rz += rn.x * zn.x + rn.y * zn.y;
    }
    cluster_barrier();  // every block has started
    rz = sums.one(rz);
    if (rank == 0 && threadIdx.x == 0) L.s[1] = rz;
    for (int k = 0; k < T.steps; ++k) {
        double a = 0.0;
        for (int i = threadIdx.x; i < n_own; i += NT) {
            const double2 qn = mg_stencil_row(L.grid, p, [&](int e) { return rows[e * L.nb + i]; }, first + i);
            q[i] = qn;
            a += p.mine[i].x * qn.x + p.mine[i].y * qn.y;
        }
        const double pq = sums.one(a);
        const double alpha = rz / pq;
        a = 0.0;
        for (int i = threadIdx.x; i < n_own; i += NT) {
            const double2 qn = q[i], D = diag2[i];
            double2 rn = r[i];
            rn.x -= alpha * qn.x;
            rn.y -= alpha * qn.y;
            const double2 zn = make_double2(rn.x / D.x, rn.y / D.y);
            r[i] = rn;
            z[i] = zn;
            a += rn.x * zn.x + rn.y * zn.y;
        }
        const double rz_new = sums.one(a);
        const double beta = rz_new / rz;
        if (rank == 0 && threadIdx.x == 0) {
            L.hist[2 * k] = alpha;
            L.hist[2 * k + 1] = beta;
            L.s[0] = pq;
            L.s[1] = rz_new;
            L.s[3] = beta;
        }
        rz = rz_new;
        for (int i = threadIdx.x; i < n_own; i += NT) {
            const double2 zn = z[i];
            double2 pn = p.mine[i];
            pn.x = zn.x + beta * pn.x;
            pn.y = zn.y + beta * pn.y;
            p.mine[i] = pn;
        }
        cluster_barrier();
    }
}

// ------------------------------------------------------------------------------------------
// coarsest level: dense A (assembled in cell order), inverted by Gauss-Jordan (A is SPD: no pivoting)
// ------------------------------------------------------------------------------------------
constexpr int kMgDenseMax = 256;     // DOFs
constexpr int kMgDenseShared = 112;  // up to this many DOFs the matrix is inverted in registers

// n <= kMgDenseShared: in-place Gauss-Jordan with the matrix in registers (a thread holds rows ti + 16 r, columns
// tj + 32 q), the pivot row and column of a step through shared memory, one barrier per step.  (The matrix in shared
// memory, assembled cell after cell, took 70 us for 50 DOFs and 115 us for 90.)
template <int R, int Q>
__global__ void __launch_bounds__(512) k_mg_dense_inverse_small(MgGrid g, double* __restrict__ Ainv_out) {
    __shared__ double row[2][32 * Q], col[2][16 * R];
    const int ny = g.gy + 1, n = 2 * (g.gx + 1) * ny;
    const int ti = threadIdx.x >> 5, tj = threadIdx.x & 31;
    double a[R][Q];
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
        for (int q = 0; q < Q; ++q) {
            const int i = ti + 16 * r, j = tj + 32 * q;
            a[r][q] = 0.0;
            if (i < n && j < n) {
                const int ni = i >> 1, nj = j >> 1, I = ni / ny, J = ni % ny, di = nj / ny - I, dj = nj % ny - J;
                if (di >= -1 && di <= 1 && dj >= -1 && dj <= 1) {
                    double c4[4];
                    mg_stencil_block(g, I, J, di, dj, c4);
                    a[r][q] = (i & 1) ? ((j & 1) ? c4[3] : c4[2]) : ((j & 1) ? c4[1] : c4[0]);
                }
            }
        }
#pragma unroll
    for (int kr = 0; kr < R; ++kr) {  // step k = 16 kr + kk: the pivot's register indices are constants
        for (int kk = 0; kk < 16 && 16 * kr + kk < n; ++kk) {
            const int k = 16 * kr + kk;
            double *rk = row[k & 1], *ck = col[k & 1];
            // publish pivot row and column and clear them: a_ij - c_i s_j then holds for every entry, with c_k = -1
            if (ti == kk) {
#pragma unroll
                for (int q = 0; q < Q; ++q) {
                    rk[tj + 32 * q] = a[kr][q];
                    if (tj + 32 * q != k) a[kr][q] = 0.0;
                }
            }
            if (tj == (k & 31)) {
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    ck[ti + 16 * r] = ti + 16 * r == k ? -1.0 : a[r][kr / 2];
                    a[r][kr / 2] = 0.0;
                }
            }
            __syncthreads();  // the next step writes the other buffers
            const double p = 1.0 / rk[k];
            double s[Q];
#pragma unroll
            for (int q = 0; q < Q; ++q) s[q] = tj + 32 * q == k ? p : rk[tj + 32 * q] * p;
#pragma unroll
            for (int r = 0; r < R; ++r) {
                const double c = ck[ti + 16 * r];
#pragma unroll
                for (int q = 0; q < Q; ++q) a[r][q] -= c * s[q];
            }
        }
    }
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
        for (int q = 0; q < Q; ++q) {
            const int i = ti + 16 * r, j = tj + 32 * q;
            if (i < n && j < n) Ainv_out[i * n + j] = a[r][q];
        }
}

// larger: A and Ainv in global memory
__global__ void __launch_bounds__(1024) k_mg_dense_inverse(MgGrid g, double* __restrict__ A, double* __restrict__ Ainv) {
    const int ny = g.gy + 1, nn = (g.gx + 1) * ny, n = 2 * nn, n_cells = g.gx * g.gy;
    __shared__ double fcol[kMgDenseMax];
    for (int k = threadIdx.x; k < n * n; k += blockDim.x) {
        A[k] = 0.0;
        Ainv[k] = (k / n == k % n) ? 1.0 : 0.0;
    }
    __syncthreads();
    for (int c = 0; c < n_cells; ++c) {
        const int CX = c / g.gy, CY = c % g.gy;
        if (threadIdx.x < 64) {
            const int row = threadIdx.x >> 3, col = threadIdx.x & 7;
            const int cn[4] = {CX * ny + CY, (CX + 1) * ny + CY, (CX + 1) * ny + CY + 1, CX * ny + CY + 1};
            const int R = 2 * cn[row >> 1] + (row & 1), Cc = 2 * cn[col >> 1] + (col & 1);
            A[R * n + Cc] += g.K[(int64_t)threadIdx.x * n_cells + c];
        }
        __syncthreads();
    }
    for (int d = threadIdx.x; d < n; d += blockDim.x)
        if ((g.fix[d >> 1] >> (d & 1)) & 1) A[d * n + d] += 1.0;
    __syncthreads();
    for (int k = 0; k < n; ++k) {
        const double p = 1.0 / A[k * n + k];
        __syncthreads();
        for (int j = threadIdx.x; j < n; j += blockDim.x) {
            A[k * n + j] *= p;
            Ainv[k * n + j] *= p;
        }
        __syncthreads();
        for (int r = threadIdx.x; r < n; r += blockDim.x) fcol[r] = A[r * n + k];
        __syncthreads();
        for (int t = threadIdx.x; t < n * n; t += blockDim.x) {
            const int r = t / n, j = t % n;
            if (r == k) continue;
            const double f = fcol[r];
            A[r * n + j] -= f * A[k * n + j];
            Ainv[r * n + j] -= f * Ainv[k * n + j];
        }
        __syncthreads();
    }
}

// x = Ainv b, one warp per row
// row r of x = Ainv b by one warp (lane-strided partial sums, then the warp's butterfly sum)
__device__ __forceinline__ void mg_dense_row(int n, const double* Ainv, const double* b, double* x, int r, int lane) {
    double s = 0.0;
    for (int j = lane; j < n; j += 32) s += Ainv[(int64_t)r * n + j] * b[j];
    s = warp_sum(s);
    if (lane == 0) x[r] = s;
}

__global__ void k_mg_dense_solve(int n, const double* __restrict__ Ainv, const double* __restrict__ b, double* __restrict__ x) {
    const int lane = threadIdx.x & 31;
    for (int r = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; r < n; r += (gridDim.x * blockDim.x) >> 5)
        mg_dense_row(n, Ainv, b, x, r, lane);
}

// ------------------------------------------------------------------------------------------
// the coarse tail of a V-cycle in one cluster: levels t .. L-1 are small enough that a launch per smoothing step costs
// more than the step, so one launch runs the restriction from level t - 1, the smoothing of every tail level, the
// coarsest solve and the prolongation back to level t - 1, with a cluster barrier between phases.  Each phase computes
// the per-node expressions of the kernel it replaces.
// ------------------------------------------------------------------------------------------
struct MgTailLevel {
    MgGrid grid;
    int n_nodes, nb;             // nodes, nodes per block
    int vec;                     // byte offset in shared memory: vectors b, x, r, d, q, 1 / D (nb pairs each), rows
    const double* diag;
    const double* coef;          // [scale, (c1, c2) per step]
};

struct MgTail {
    MgGrid fine;                 // level t - 1 (the transfers' fine side)
    const int32_t* gnode;
    const uint8_t* ffix;
    const double* r_fine;        // level t - 1's residual, restricted into level t's right-hand side
    double* x_fine;              // level t - 1's iterate, corrected by the prolongation of level t's
    const double* Ainv;
    int n_levels, degree;        // tail levels; the last is the coarsest
    MgTailLevel lv[DFEA_MG_MAX_LEVELS];
};

__global__ void __launch_bounds__(kMgClusterThreads, 1) k_mg_tail(const __grid_constant__ MgTail T) {
    constexpr int NT = kMgClusterThreads;
    extern __shared__ __align__(16) unsigned char mg_smem[];
    __shared__ double b_all[kMgDenseMax];
    const unsigned rank = cluster_rank();
    const int size = gridDim.x, last = T.n_levels - 1;  // the grid is the cluster
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    auto vec = [&](const MgTailLevel& L, int k) { return ClusterVec(mg_smem, L.vec + k * L.nb * 16, L.nb); };
    auto owned = [&](const MgTailLevel& L) { return min(L.nb, max(0, L.n_nodes - (int)rank * L.nb)); };
    enum { VB, VX, VR, VD, VQ, VI, VROWS };
    auto rows_of = [&](const MgTailLevel& L) { return reinterpret_cast<double*>(mg_smem + L.vec + VROWS * L.nb * 16); };

    // post: nobody reads the last residual, so the last step has no product and the pass before adds its direction too
    auto smooth = [&](const MgTailLevel& L, bool post) {
        const int first = rank * L.nb, n_own = owned(L);
        double2 *x = vec(L, VX).mine, *r = vec(L, VR).mine;
        const double2* inv = vec(L, VI).mine;
        const double* rows = rows_of(L);
        int in = VD, out = VQ;
        const int steps = post ? T.degree - 1 : T.degree;
        for (int k = 1; k <= steps; ++k) {
            const bool more = k < T.degree, add = post && k == steps;
            const double c1 = more ? L.coef[1 + 2 * (k - 1)] : 0.0, c2 = more ? L.coef[2 + 2 * (k - 1)] : 0.0;
            const ClusterVec d = vec(L, in);
            double2* d_out = vec(L, out).mine;
            for (int i = threadIdx.x; i < n_own; i += NT) {
                const double2 q = mg_stencil_row(L.grid, d, [&](int e) { return rows[e * L.nb + i]; }, first + i);
                const double2 dn = d.mine[i], I = inv[i];
                double2 xn = x[i];
                xn.x += dn.x;
                xn.y += dn.y;
                const double r0 = r[i].x - q.x, r1 = r[i].y - q.y;
                const double2 dd = make_double2(c1 * dn.x + c2 * r0 * I.x, c1 * dn.y + c2 * r1 * I.y);
                if (add) {
                    xn.x += dd.x;
                    xn.y += dd.y;
                } else {
                    r[i] = make_double2(r0, r1);
                    if (more) d_out[i] = dd;
                }
                x[i] = xn;
            }
            cluster_barrier();
            const int t = in;
            in = out;
            out = t;
        }
    };

    for (int l = 0; l < last; ++l) {
        const MgTailLevel& L = T.lv[l];
        const int first = rank * L.nb, n_own = owned(L);
        load_rows(L.grid, rows_of(L), L.nb, first, n_own, L.n_nodes);
        double2* inv = vec(L, VI).mine;
        for (int i = threadIdx.x; i < n_own; i += NT) {
            const double2 D = reinterpret_cast<const double2*>(L.diag)[first + i];
            inv[i] = make_double2(1.0 / D.x, 1.0 / D.y);
        }
    }
    // everything above was written by a set-up, which at least two launches of the cycle separate from this one; the
    // finer level's residual is the predecessor's
    grid_dependency_wait();
    grid_dependents_launch();
    cluster_barrier();  // every block has started, its rows are loaded
    for (int l = 0; l <= last; ++l) {
        const MgTailLevel& L = T.lv[l];
        const int first = rank * L.nb, n_own = owned(L);
        double2 *b = vec(L, VB).mine, *x = vec(L, VX).mine, *r = vec(L, VR).mine, *d = vec(L, VD).mine;
        const double2* inv = vec(L, VI).mine;
        const double s = l < last ? L.coef[0] : 0.0;
        for (int i = threadIdx.x; i < n_own; i += NT) {
            double2 bn;
            if (l == 0) {
                const double2* r2 = reinterpret_cast<const double2*>(T.r_fine);
                bn = mg_restrict_sum<true>(T.fine, L.grid, T.gnode, T.ffix, [&](int id) { return load_fresh(r2 + id); }, first + i, nullptr);
            } else {
                const MgTailLevel& F = T.lv[l - 1];
                bn = mg_restrict_sum<true>(F.grid, L.grid, nullptr, F.grid.fix, vec(F, VR), first + i, nullptr);
            }
            b[i] = bn;
            if (l < last) {
                r[i] = bn;
                x[i] = make_double2(0.0, 0.0);
                d[i] = make_double2(s * bn.x * inv[i].x, s * bn.y * inv[i].y);
            }
        }
        cluster_barrier();
        if (l < last) smooth(L, false);
    }
    {
        const MgTailLevel& C = T.lv[last];
        const ClusterVec b = vec(C, VB);
        for (int n = threadIdx.x; n < C.n_nodes; n += NT) {
            const double2 t = b(n);
            b_all[2 * n] = t.x;
            b_all[2 * n + 1] = t.y;
        }
        __syncthreads();
        const unsigned x_here = vec(C, VX).here;
        const int n = 2 * C.n_nodes;
        for (int row = rank * (NT / 32) + warp; row < n; row += size * (NT / 32)) {
            double s = 0.0;
            for (int j = lane; j < n; j += 32) s += T.Ainv[(int64_t)row * n + j] * b_all[j];
            s = warp_sum(s);
            if (lane == 0) cluster_store(cluster_address(x_here + (row / 2 % C.nb) * 16 + (row & 1) * 8, row / 2 / C.nb), s);
        }
        cluster_barrier();
    }
    for (int l = last; l >= 0; --l) {
        const MgTailLevel& L = T.lv[l];
        const ClusterVec ec = vec(L, VX);
        if (l == 0) {
            const int fine_nodes = (T.fine.gx + 1) * (T.fine.gy + 1);
            for (int n = rank * NT + threadIdx.x; n < fine_nodes; n += size * NT)
                mg_prolong_node(T.fine, L.grid, T.gnode, T.ffix, ec,
                                [&](int id) -> double2& { return reinterpret_cast<double2*>(T.x_fine)[id]; }, n);
            break;
        }
        const MgTailLevel& F = T.lv[l - 1];
        const int first = rank * F.nb, n_own = owned(F);
        const ClusterVec x = vec(F, VX);
        double2 *b = vec(F, VB).mine, *r = vec(F, VR).mine, *d = vec(F, VD).mine;
        for (int i = threadIdx.x; i < n_own; i += NT)
            mg_prolong_node(F.grid, L.grid, nullptr, F.grid.fix, ec, [&](int id) -> double2& { return x.mine[id - first]; }, first + i);
        cluster_barrier();
        const double s = F.coef[0];
        const double2* inv = vec(F, VI).mine;
        const double* rows = rows_of(F);
        for (int i = threadIdx.x; i < n_own; i += NT) {
            const double2 q = mg_stencil_row(F.grid, x, [&](int e) { return rows[e * F.nb + i]; }, first + i);
            const double r0 = b[i].x - q.x, r1 = b[i].y - q.y;
            r[i] = make_double2(r0, r1);
            d[i] = make_double2(s * r0 * inv[i].x, s * r1 * inv[i].y);
        }
        cluster_barrier();
        if (T.degree == 1) {  // the only direction
            for (int i = threadIdx.x; i < n_own; i += NT) {
                x.mine[i].x += d[i].x;
                x.mine[i].y += d[i].y;
            }
            cluster_barrier();
        } else {
            smooth(F, true);
        }
    }
    cluster_barrier();  // no block leaves while another may read its shared memory
}

// A launch of clusters of `size` blocks (a power of two of at most cluster_room's).
template <auto Kernel, typename... Args>
static int launch_clusters(int n_clusters, int size, size_t smem, bool pdl, cudaStream_t s, const Args&... args) {
    if (size > cluster_room<Kernel>(kMgClusterThreads).blocks)
        return set_error(DFEA_ERR_UNSUPPORTED, "multigrid: clusters of %d blocks find no place on this device", size);
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = size;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(n_clusters * size);
    cfg.blockDim = dim3(kMgClusterThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = pdl ? 2 : 1;
    return check_cuda(cudaLaunchKernelEx(&cfg, Kernel, args...), "cudaLaunchKernelEx");
}

// blocks for a largest level of n nodes: about 64 nodes a block, 16 blocks (or the fewer that are allowed) at the most
static int mg_cluster_size(int64_t n_nodes, int most) {
    int size = 1;
    while (2 * size <= most && (int64_t)size * 64 < n_nodes) size *= 2;
    return size;
}

}  // namespace dfea

using namespace dfea;

extern "C" int dfea_mg_galerkin_fe(const dfea_mesh_view* mesh, const void* moduli, int32_t moduli_dtype,
                                   const int32_t* node_ij, const int32_t* cell_slot, int32_t span,
                                   const dfea_mg_grid* fine, const dfea_mg_grid* coarse, void* stream) {
    int rc = validate_mesh(mesh, false);
    if (rc) return rc;
    if ((rc = validate_grid(fine, false, "dfea_mg_galerkin_fe")) || (rc = validate_grid(coarse, true, "dfea_mg_galerkin_fe")))
        return rc;
    if (!moduli || !node_ij || !cell_slot || !coarse->K) return set_error(DFEA_ERR_INVALID, "dfea_mg_galerkin_fe: NULL pointer");
    if (span != 1 && span != 2) return set_error(DFEA_ERR_INVALID, "dfea_mg_galerkin_fe: span must be 1 or 2");
    const int64_t n_cells = (int64_t)(fine->gx / span) * (fine->gy / span);
    const int epc = n_cells > 0 ? (int)(mesh->n_el / n_cells) : 0;   // elements per cell: 1, or 2 triangles
    if (fine->gx % span || fine->gy % span || (epc != 1 && epc != 2) || n_cells * epc != mesh->n_el)
        return set_error(DFEA_ERR_INVALID, "dfea_mg_galerkin_fe: the grid does not match the mesh's element count");
    const Mesh m = kernel_mesh(*mesh);
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const int n_ccells = coarse->gx * coarse->gy;
    const int grid = grid_for(n_ccells, 128, 8);
    const MgGrid cg = mg_grid(*coarse);
    const int ncy = fine->gy / span;
    rc = dispatch_element(mesh->nen, mesh->n_q, [&](auto nen_c, auto nq_c) -> int {
        constexpr int NEN = decltype(nen_c)::value, NQ = decltype(nq_c)::value;
        const RefGrad<NEN, NQ> rg = ref_grad_of<NEN, NQ>(*mesh);
        if (moduli_dtype == DFEA_F64)
            k_mg_galerkin_fe<NEN, NQ, 0><<<grid, 128, 0, s>>>(m, moduli, rg, node_ij, cell_slot, span, epc, ncy, cg);
        else if (moduli_dtype == DFEA_F32)
            k_mg_galerkin_fe<NEN, NQ, 1><<<grid, 128, 0, s>>>(m, moduli, rg, node_ij, cell_slot, span, epc, ncy, cg);
        else if (moduli_dtype == DFEA_F32REF)
            k_mg_galerkin_fe<NEN, NQ, 2><<<grid, 128, 0, s>>>(m, moduli, rg, node_ij, cell_slot, span, epc, ncy, cg);
        else if (moduli_dtype == DFEA_F64REF)
            k_mg_galerkin_fe<NEN, NQ, 3><<<grid, 128, 0, s>>>(m, moduli, rg, node_ij, cell_slot, span, epc, ncy, cg);
        else
            return set_error(DFEA_ERR_INVALID, "dfea_mg_galerkin_fe: bad moduli dtype");
        return DFEA_OK;
    });
    if (rc) return rc;
    note_launches(1);
    return launch_check("dfea_mg_galerkin_fe");
}

extern "C" int dfea_mg_galerkin(const dfea_mg_grid* fine, const dfea_mg_grid* coarse, void* stream) {
    int rc;
    if ((rc = validate_grid(fine, true, "dfea_mg_galerkin")) || (rc = validate_grid(coarse, true, "dfea_mg_galerkin")))
        return rc;
    if (!fine->K || !coarse->K) return set_error(DFEA_ERR_INVALID, "dfea_mg_galerkin: NULL element matrices");
    const int n_cells = coarse->gx * coarse->gy;
    k_mg_galerkin<<<grid_for(8 * (int64_t)n_cells, 128, 8), 128, 0, static_cast<cudaStream_t>(stream)>>>(mg_grid(*fine), mg_grid(*coarse));
    note_launches(1);
    return launch_check("dfea_mg_galerkin");
}

extern "C" int dfea_mg_restrict(const dfea_mg_grid* fine, const dfea_mg_grid* coarse, const int32_t* gnode,
                                const uint8_t* fine_fix, const double* r, double* rc_out, uint8_t* coarse_fix_out,
                                void* stream) {
    int rc;
    if ((rc = validate_grid(fine, false, "dfea_mg_restrict")) || (rc = validate_grid(coarse, true, "dfea_mg_restrict")))
        return rc;
    if (!fine_fix || (!rc_out && !coarse_fix_out) || (rc_out && !r))
        return set_error(DFEA_ERR_INVALID, "dfea_mg_restrict: NULL pointer");
    const int n = (coarse->gx + 1) * (coarse->gy + 1);
    k_mg_restrict<<<grid_for(n, kThreads, 8), kThreads, 0, static_cast<cudaStream_t>(stream)>>>(
        mg_grid(*fine), mg_grid(*coarse), gnode, fine_fix, r, rc_out, coarse_fix_out);
    note_launches(1);
    return launch_check("dfea_mg_restrict");
}

extern "C" int dfea_mg_prolong_add(const dfea_mg_grid* fine, const dfea_mg_grid* coarse, const int32_t* gnode,
                                   const uint8_t* fine_fix, const double* ec, double* x, void* stream) {
    int rc;
    if ((rc = validate_grid(fine, false, "dfea_mg_prolong_add")) || (rc = validate_grid(coarse, true, "dfea_mg_prolong_add")))
        return rc;
    if (!fine_fix || !ec || !x) return set_error(DFEA_ERR_INVALID, "dfea_mg_prolong_add: NULL pointer");
    const int n = (fine->gx + 1) * (fine->gy + 1);
    k_mg_prolong_add<<<grid_for(n, kThreads, 8), kThreads, 0, static_cast<cudaStream_t>(stream)>>>(
        mg_grid(*fine), mg_grid(*coarse), gnode, fine_fix, ec, x);
    note_launches(1);
    return launch_check("dfea_mg_prolong_add");
}

extern "C" int dfea_mg_apply(const dfea_mg_grid* grid, const double* v, double* y, void* stream) {
    int rc = validate_grid(grid, false, "dfea_mg_apply");
    if (rc) return rc;
    if (!grid->K || !grid->fix || !y || (v == nullptr)) return set_error(DFEA_ERR_INVALID, "dfea_mg_apply: NULL pointer");
    const int n = (grid->gx + 1) * (grid->gy + 1);
    k_mg_apply<false><<<grid_for(n, 256, 8), 256, 0, static_cast<cudaStream_t>(stream)>>>(mg_grid(*grid), v, y);
    note_launches(1);
    return launch_check("dfea_mg_apply");
}

extern "C" int dfea_mg_diag(const dfea_mg_grid* grid, double* diag, void* stream) {
    int rc = validate_grid(grid, false, "dfea_mg_diag");
    if (rc) return rc;
    if (!grid->K || !grid->fix || !diag) return set_error(DFEA_ERR_INVALID, "dfea_mg_diag: NULL pointer");
    const int n = (grid->gx + 1) * (grid->gy + 1);
    k_mg_apply<true><<<grid_for(n, 256, 8), 256, 0, static_cast<cudaStream_t>(stream)>>>(mg_grid(*grid), nullptr, diag);
    note_launches(1);
    return launch_check("dfea_mg_diag");
}

extern "C" int dfea_mg_cheb_start(int64_t n, const double* r, const double* diag, const double* scale, double* d,
                                  void* stream) {
    if (n < 0 || (n > 0 && (!r || !diag || !d || !scale))) return set_error(DFEA_ERR_INVALID, "dfea_mg_cheb_start: bad arguments");
    if (n == 0) return DFEA_OK;
    k_mg_cheb_start<<<grid_for(n, kThreads, 8), kThreads, 0, static_cast<cudaStream_t>(stream)>>>(n, r, diag, scale, d);
    note_launches(1);
    return launch_check("dfea_mg_cheb_start");
}

extern "C" int dfea_mg_cheb_step(int64_t n, double* x, double* r, double* d, const double* q, const double* diag,
                                 const double* c, int32_t last, void* stream) {
    if (n < 0 || (n > 0 && (!x || !r || !d || !q || !diag || (!last && !c))))
        return set_error(DFEA_ERR_INVALID, "dfea_mg_cheb_step: bad arguments");
    if (n == 0) return DFEA_OK;
    k_mg_cheb_step<<<grid_for(n, kThreads, 8), kThreads, 0, static_cast<cudaStream_t>(stream)>>>(n, x, r, d, q, diag, c,
                                                                                                    last);
    note_launches(1);
    return launch_check("dfea_mg_cheb_step");
}

extern "C" int64_t dfea_mg_dense_max(void) { return kMgDenseMax; }

extern "C" int dfea_mg_dense_inverse(const dfea_mg_grid* grid, double* work, double* Ainv, void* stream) {
    int rc = validate_grid(grid, false, "dfea_mg_dense_inverse");
    if (rc) return rc;
    const int n = 2 * (grid->gx + 1) * (grid->gy + 1);
    if (n > kMgDenseMax) return set_error(DFEA_ERR_INVALID, "dfea_mg_dense_inverse: %d DOFs exceed %d", n, kMgDenseMax);
    if (!grid->K || !grid->fix || !work || !Ainv) return set_error(DFEA_ERR_INVALID, "dfea_mg_dense_inverse: NULL pointer");
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (n <= 32)
        k_mg_dense_inverse_small<2, 1><<<1, 512, 0, st>>>(mg_grid(*grid), Ainv);
    else if (n <= 64)
        k_mg_dense_inverse_small<4, 2><<<1, 512, 0, st>>>(mg_grid(*grid), Ainv);
    else if (n <= 96)
        k_mg_dense_inverse_small<6, 3><<<1, 512, 0, st>>>(mg_grid(*grid), Ainv);
    else if (n <= kMgDenseShared)
        k_mg_dense_inverse_small<7, 4><<<1, 512, 0, st>>>(mg_grid(*grid), Ainv);
    else
        k_mg_dense_inverse<<<1, 1024, 0, st>>>(mg_grid(*grid), work, Ainv);
    note_launches(1);
    return launch_check("dfea_mg_dense_inverse");
}

extern "C" int dfea_mg_dense_solve(int32_t n, const double* Ainv, const double* b, double* x, void* stream) {
    if (n < 1 || n > kMgDenseMax || !Ainv || !b || !x) return set_error(DFEA_ERR_INVALID, "dfea_mg_dense_solve: bad arguments");
    k_mg_dense_solve<<<(n + 7) / 8, 256, 0, static_cast<cudaStream_t>(stream)>>>(n, Ainv, b, x);
    note_launches(1);
    return launch_check("dfea_mg_dense_solve");
}

extern "C" int64_t dfea_mg_dot_work(void) { return kMgDotWork; }

extern "C" int dfea_mg_dot(int64_t n, const double* x, const double* y, double* out, double* work, void* stream) {
    if (n < 0 || !x || !y || !out || !work) return set_error(DFEA_ERR_INVALID, "dfea_mg_dot: bad arguments");
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const int nb = mg_dot_blocks(n);
    k_mg_dot_part<<<nb, kMgDotThreads, 0, st>>>(n, x, y, work);
    k_mg_dot_final<false><<<1, kMgDotThreads, 0, st>>>(nb, work, out, nullptr, 0);
    note_launches(2);
    return launch_check("dfea_mg_dot");
}

extern "C" int dfea_mg_lanczos_step(int64_t n, double* p, const double* q, double* r, double* z, const double* diag,
                                    double* s, double* hist, int32_t k, double* work, void* stream) {
    if (n < 1 || !p || !q || !r || !z || !diag || !s || !hist || k < 0 || !work)
        return set_error(DFEA_ERR_INVALID, "dfea_mg_lanczos_step: bad arguments");
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const int nb = mg_dot_blocks(n);
    k_mg_dot_part<<<nb, kMgDotThreads, 0, st>>>(n, p, q, work);
    k_mg_dot_final<false><<<1, kMgDotThreads, 0, st>>>(nb, work, s, nullptr, 0);
    k_mg_lanczos_step<<<grid_for(n, kThreads, 8), kThreads, 0, st>>>(n, q, r, z, diag, s);
    k_mg_dot_part<<<nb, kMgDotThreads, 0, st>>>(n, r, z, work);
    k_mg_dot_final<true><<<1, kMgDotThreads, 0, st>>>(nb, work, s, hist, k);
    k_mg_lanczos_p<<<grid_for(n, kThreads, 8), kThreads, 0, st>>>(n, p, z, s);
    note_launches(6);
    return launch_check("dfea_mg_lanczos_step");
}

// ------------------------------------------------------------------------------------------
// the C++ driver: set-up, V-cycle, PCG
// ------------------------------------------------------------------------------------------
namespace dfea {

// Largest eigenvalue of the symmetric tridiagonal matrix (diagonal a, off-diagonal e) by bisection on the
// Sturm sequence count (number of eigenvalues below x), from the Gershgorin upper bound.
static double tridiag_max_eig(const double* a, const double* e, int m) {
    double lo = a[0], hi = a[0];
    for (int i = 0; i < m; ++i) {
        const double r = (i > 0 ? fabs(e[i - 1]) : 0.0) + (i + 1 < m ? fabs(e[i]) : 0.0);
        lo = fmin(lo, a[i] - r);
        hi = fmax(hi, a[i] + r);
    }
    auto below = [&](double x) {
        int c = 0;
        double d = 1.0;
        for (int i = 0; i < m; ++i) {
            d = a[i] - x - (i > 0 ? e[i - 1] * e[i - 1] / d : 0.0);
            if (d == 0.0) d = -1e-300;
            if (d < 0.0) ++c;
        }
        return c;
    };
    for (int it = 0; it < 200 && hi - lo > 1e-14 * fmax(1.0, fabs(hi)); ++it) {
        const double mid = 0.5 * (lo + hi);
        if (below(mid) >= m) hi = mid;   // every eigenvalue is below mid
        else lo = mid;
    }
    return hi;
}

// lambda_max of D^-1 A from Jacobi-CG coefficients (alpha_k, beta_k), over the prefix before a breakdown
static double ritz_max(const double* hist, int steps) {
    double a[64], e[64];
    int m = 0;
    for (; m < steps && m < 64; ++m) {
        const double al = hist[2 * m], be = hist[2 * m + 1];
        if (!(std::isfinite(al) && al > 0.0 && std::isfinite(be) && be >= 0.0)) break;
    }
    if (m == 0) return 2.5;
    for (int k = 0; k < m; ++k) {
        a[k] = 1.0 / hist[2 * k] + (k > 0 ? hist[2 * k - 1] / hist[2 * k - 2] : 0.0);
        if (k + 1 < m) e[k] = sqrt(hist[2 * k + 1]) / hist[2 * k];
    }
    return tridiag_max_eig(a, e, m);
}

// the stencils of level l >= 1 in mg->stencil (36 numbers a node, level after level), or NULL
static double* stencil_of(const dfea_mg* mg, int l) {
    if (!mg->stencil || l < 1) return nullptr;
    double* s = mg->stencil;
    for (int k = 1; k < l; ++k) s += 36 * (mg->level[k].n / 2);
    return s;
}
static MgGrid level_grid(const dfea_mg* mg, int l) { return mg_grid(mg->level[l].grid, stencil_of(mg, l)); }

static void transfer_args(const dfea_mesh_view* mesh, const dfea_mg* mg, int l, const int32_t** gnode,
                          const uint8_t** ffix) {
    *gnode = l == 0 ? mg->gnode : nullptr;
    *ffix = l == 0 ? mesh->node_fix : mg->level[l].grid.fix;
}

// level 0 in the gather form (the hierarchy was given element-product scratch and the mesh has node incidence)
static bool fe_gather(const dfea_mesh_view* mesh, const dfea_mg* mg) {
    return mg->fe_work && mesh->node_elem_ptr && mesh->node_elem;
}

static int mg_apply(const dfea_mesh_view* mesh, const dfea_mg* mg, const void* moduli, int32_t code, int l,
                    const double* v, double* y, cudaStream_t s) {
    if (l == 0)
        return fe_gather(mesh, mg)
                   ? dfea_tangent_apply_gather(mesh, moduli, code, v, y, DFEA_F64, mg->fe_work, s)
                   : dfea_tangent_apply(mesh, moduli, code, v, y, DFEA_F64, s);
    const int n_nodes = (int)(mg->level[l].n / 2);
    k_mg_apply<false><<<grid_for(n_nodes, 256, 8), 256, 0, s>>>(level_grid(mg, l), v, y);
    note_launches(1);
    return launch_check("multigrid product");
}

static LaunchOpts overlapping() {
    LaunchOpts o;
    o.pdl = true;
    return o;
}

// what the PCG asks of a cycle on level 0: its first direction is in place; r.z into the state (general form: after it)
struct CycleUse {
    bool started = false;
    MgPcgState* dot = nullptr;
};

// The Chebyshev steps of one smoothing pass at level l from the first direction in lv.d (coarse levels: d alternates
// between lv.d and lv.q).  Pre-smoothing (post = false): x starts at zero, the residual at b (level 0 without node
// incidence: set by k_mg_cheb_first), the residual after it in lv.r.  Post-smoothing: from x and lv.r, x only.
static int mg_cheb_steps(const dfea_mesh_view* mesh, const dfea_mg* mg, const void* moduli, int32_t code, int l, bool post,
                         const double* b, double* x, MgPcgState* dot, cudaStream_t s) {
    const dfea_mg_level& lv = mg->level[l];
    const double* row = mg->coef + (int64_t)l * 2 * DFEA_MG_MAX_DEGREE;
    double *d_in = lv.d, *d_out = lv.q;
    const int steps = post ? mg->degree - 1 : mg->degree;
    int rc = DFEA_OK;
    for (int k = 1; !rc && k <= steps; ++k) {
        const int first = !post && k == 1, last = k == mg->degree, add = post && k == steps;
        const double* c = last ? nullptr : row + 1 + 2 * (k - 1);
        if (l == 0 && fe_gather(mesh, mg)) {
            const MgNodePass pass = {lv.d, x, first ? b : lv.r, add ? nullptr : lv.r, last || add ? nullptr : lv.d,
                                     lv.diag, c, first, add};
            rc = mg_fe_smooth(mesh, moduli, code, mg->fe_work, MG_FE_STEP, pass, b, add ? dot : nullptr, mg->dot_work, s);
            continue;
        }
        if (l == 0) {
            if (!(rc = mg_apply(mesh, mg, moduli, code, 0, lv.d, lv.q, s)) &&
                !(rc = dfea_mg_cheb_step(lv.n, x, lv.r, lv.d, lv.q, lv.diag, c, last, s)) && add)
                rc = dfea_add_scaled(lv.n, x, 1.0, lv.d, x, s);
            continue;
        }
        const int n_nodes = (lv.grid.gx + 1) * (lv.grid.gy + 1);
        rc = launch_kernel(k_mg_cheb_apply_step, dim3(grid_for(n_nodes, 256, 8)), dim3(256), 0, s, overlapping(),
                           level_grid(mg, l), x, first ? b : (const double*)lv.r, lv.r, (const double*)d_in, d_out,
                           (const double*)lv.diag, c, first, last, add);
        note_launches(1);
        std::swap(d_in, d_out);
    }
    // degree 1: the first direction is the only one (the gather form's restart has added it)
    if (!rc && post && steps == 0 && !(l == 0 && fe_gather(mesh, mg))) rc = dfea_add_scaled(lv.n, x, 1.0, lv.d, x, s);
    return rc;
}

// First level (>= 1) of the cluster tail, n_levels: none.  A block holds its nodes of all the tail's levels.  Where both
// directions coarsen, the levels after the first add a third to it; on a thin strip one direction is soon a single cell,
// the levels only halve and double it (a 2,945 x 6 strip: 235 KB from its level of 5,892 nodes on), so the sum decides.
static int tail_level(const dfea_mg* mg, int blocks, int64_t bytes) {
    for (int l = 1; l < mg->n_levels; ++l) {
        if (mg->level[l].n / 2 > kMgTailNodes) continue;
        const int size = mg_cluster_size(mg->level[l].n / 2, blocks);
        int64_t need = 0;
        for (int k = l; k < mg->n_levels; ++k) need += (mg->level[k].n / 2 + size - 1) / size * kMgTailNodeBytes;
        if (need <= bytes) return l;
    }
    return mg->n_levels;
}
// blocks of the tail's clusters, 0: none (the Lanczos kernel needs less shared memory per node than the cycle's)
static int tail_blocks() {
    const int a = cluster_room<k_mg_tail>(kMgClusterThreads).blocks, b = cluster_room<k_mg_tail_lanczos>(kMgClusterThreads).blocks;
    return a < b ? a : b;
}
static int tail_start(const dfea_mg* mg) {
    if (!mg->stencil || tail_blocks() == 0) return mg->n_levels;
    return tail_level(mg, tail_blocks(), cluster_room<k_mg_tail>(kMgClusterThreads).bytes);
}

// restriction of level l's residual, the cycle of levels l + 1 .. L - 1 and the prolongation into x, in one launch
static int launch_tail(const dfea_mesh_view* mesh, const dfea_mg* mg, int l, double* x, cudaStream_t s) {
    MgTail T = {};
    const dfea_mg_level& lv = mg->level[l];
    T.fine = mg_grid(lv.grid);
    transfer_args(mesh, mg, l, &T.gnode, &T.ffix);
    T.r_fine = lv.r;
    T.x_fine = x;
    T.Ainv = mg->Ainv;
    T.n_levels = mg->n_levels - (l + 1);
    T.degree = mg->degree;
    const int size = mg_cluster_size(mg->level[l + 1].n / 2, tail_blocks());
    int at = 0;
    for (int k = 0; k < T.n_levels; ++k) {
        const dfea_mg_level& c = mg->level[l + 1 + k];
        const int n_nodes = (int)(c.n / 2), nb = (n_nodes + size - 1) / size;
        T.lv[k] = MgTailLevel{level_grid(mg, l + 1 + k), n_nodes, nb, at, c.diag, mg->coef + (int64_t)(l + 1 + k) * 2 * DFEA_MG_MAX_DEGREE};
        at += kMgTailNodeBytes * nb;
    }
    const int rc = launch_clusters<k_mg_tail>(1, size, at, true, s, T);
    if (rc) return rc;
    note_launches(1);
    return launch_check("dfea_mg_vcycle: coarse tail");
}

// x = one cycle on b from level l >= 1 or 0; on a level >= 1 the first direction is in place
static int mg_vcycle(const dfea_mesh_view* mesh, const dfea_mg* mg, const void* moduli, int32_t code, int l,
                     const double* b, double* x, const CycleUse& use, cudaStream_t s) {
    const dfea_mg_level& lv = mg->level[l];
    int rc;
    if (l == mg->n_levels - 1) return dfea_mg_dense_solve((int32_t)lv.n, mg->Ainv, b, x, s);
    const double* scale = mg->coef + (int64_t)l * 2 * DFEA_MG_MAX_DEGREE;
    const bool gather = l == 0 && fe_gather(mesh, mg);
    if (l == 0 && !gather) {
        k_mg_cheb_first<<<grid_for(lv.n, kThreads, 8), kThreads, 0, s>>>(lv.n, b, lv.diag, scale, lv.r, x, lv.d);
        note_launches(1);
        if ((rc = launch_check("dfea_mg_vcycle: smoothing start"))) return rc;
    } else if (l == 0 && !use.started && (rc = dfea_mg_cheb_start(lv.n, b, lv.diag, scale, lv.d, s))) {
        return rc;
    }
    if ((rc = mg_cheb_steps(mesh, mg, moduli, code, l, false, b, x, nullptr, s))) return rc;
    const dfea_mg_level& c = mg->level[l + 1];
    const int32_t* gn;
    const uint8_t* ffix;
    transfer_args(mesh, mg, l, &gn, &ffix);
    if (l + 1 == tail_start(mg)) {
        if ((rc = launch_tail(mesh, mg, l, x, s))) return rc;
    } else {
        const int c_nodes = (int)(c.n / 2), f_nodes = (lv.grid.gx + 1) * (lv.grid.gy + 1);
        const double* c_scale = scale + 2 * DFEA_MG_MAX_DEGREE;
        if (l + 1 == mg->n_levels - 1) {
            rc = dfea_mg_restrict(&lv.grid, &c.grid, gn, ffix, lv.r, c.b, nullptr, s);
        } else {
            rc = launch_kernel(k_mg_restrict_first, dim3(grid_for(c_nodes, 256, 8)), dim3(256), 0, s, overlapping(),
                               mg_grid(lv.grid), mg_grid(c.grid), gn, ffix, (const double*)lv.r, (const double*)c.diag, c_scale,
                               c.b, c.d);
            note_launches(1);
        }
        if (rc || (rc = mg_vcycle(mesh, mg, moduli, code, l + 1, c.b, c.x, CycleUse(), s)) ||
            (rc = launch_kernel(k_mg_prolong_add, dim3(grid_for(f_nodes, 256, 8)), dim3(256), 0, s, overlapping(),
                                mg_grid(lv.grid), mg_grid(c.grid), gn, ffix, (const double*)c.x, x)))
            return rc;
        note_launches(1);
    }
    if (gather) {
        const bool only = mg->degree == 1;
        const MgNodePass pass = {x, x, b, only ? nullptr : lv.r, only ? nullptr : lv.d, lv.diag, scale, 0, only};
        rc = mg_fe_smooth(mesh, moduli, code, mg->fe_work, MG_FE_RESTART, pass, b, only ? use.dot : nullptr, mg->dot_work, s);
    } else if (l == 0) {
        if ((rc = mg_apply(mesh, mg, moduli, code, 0, x, lv.q, s))) return rc;
        k_mg_cheb_restart<<<grid_for(lv.n, kThreads, 8), kThreads, 0, s>>>(lv.n, b, lv.q, lv.diag, scale, lv.r, lv.d);
        note_launches(1);
        rc = launch_check("dfea_mg_vcycle: residual");
    } else {
        const int n_nodes = (lv.grid.gx + 1) * (lv.grid.gy + 1);
        rc = launch_kernel(k_mg_residual_restart, dim3(grid_for(n_nodes, 256, 8)), dim3(256), 0, s, overlapping(),
                           level_grid(mg, l), b, (const double*)x, (const double*)lv.diag, scale, lv.r, lv.d);
        note_launches(1);
    }
    if (rc || (rc = mg_cheb_steps(mesh, mg, moduli, code, l, true, b, x, use.dot, s))) return rc;
    if (use.dot && !gather) return mg_dot1<MG_DOT_CYCLE>(lv.n, b, x, reinterpret_cast<double*>(use.dot), mg->dot_work, s);
    return launch_check("dfea_mg_vcycle");
}

static int validate_mg(const dfea_mesh_view* mesh, const dfea_mg* mg, const char* what) {
    int rc = validate_mesh(mesh, false);
    if (rc) return rc;
    if (!mg || mg->n_levels < 2 || mg->n_levels > DFEA_MG_MAX_LEVELS || mg->degree < 1 ||
        mg->degree > DFEA_MG_MAX_DEGREE || mg->lanczos_steps < 1 || mg->lanczos_steps > 64 || !(mg->ratio > 1.0))
        return set_error(DFEA_ERR_INVALID, "%s: bad hierarchy parameters", what);
    if (mg->level[0].n != 2 * mesh->n_nodes) return set_error(DFEA_ERR_INVALID, "%s: level 0 is not the mesh", what);
    for (int l = 0; l < mg->n_levels; ++l) {
        const dfea_mg_level& lv = mg->level[l];
        // level 0 holds the mesh's DOFs (a Q8 grid has no nodes at the cell centres), the others their grid's
        if ((l > 0 && lv.n != 2 * (int64_t)(lv.grid.gx + 1) * (lv.grid.gy + 1)) || !lv.diag || !lv.b || !lv.x || !lv.r ||
            !lv.d || !lv.q)
            return set_error(DFEA_ERR_INVALID, "%s: level %d buffers", what, l);
        if (l > 0 && (rc = validate_grid(&lv.grid, true, what))) return rc;
    }
    if (mg->level[mg->n_levels - 1].n > kMgDenseMax) return set_error(DFEA_ERR_INVALID, "%s: coarsest level too large", what);
    if (!mg->node_ij || !mg->gnode || !mg->cell_slot || !mg->Ainv || !mg->dense_work || !mg->coef || !mg->lscal ||
        !mg->lhist || !mg->dot_work || !mg->pcg || !mg->scal)
        return set_error(DFEA_ERR_INVALID, "%s: NULL buffer", what);
    return DFEA_OK;
}

// The passes over level 0 read and write nodal pairs.  A caller's vector that starts between two pairs stands in level 0's
// right-hand side, which nothing else uses.
static bool paired(const double* v) { return (reinterpret_cast<uintptr_t>(v) & 15u) == 0; }
static int copy_vector(double* to, const double* from, int64_t n, cudaStream_t s) {
    return check_cuda(cudaMemcpyAsync(to, from, n * sizeof(double), cudaMemcpyDeviceToDevice, s), "cudaMemcpyAsync");
}

static int read_scalars(double* host, const double* dev, int k, cudaStream_t s) {
    return read_to_host(host, dev, k * sizeof(double), s);
}

}  // namespace dfea

namespace dfea {

// ------------------------------------------------------------------------------------------
// the grid behind a structured mesh
// ------------------------------------------------------------------------------------------
// What a hierarchy needs to know of its mesh, from the device connectivity.  (Built on the host and compared with and
// copied to the device: 3.9 ms of a 384 x 384 Q4 hierarchy's construction, 1.4 ms of a 128 x 128 Q9 one's; here 0.1 ms.)
struct GridNumbering {
    int span, gx, gy, nen, k;  // k: 0 by columns, 1 by rows
    __device__ __forceinline__ GridNumbering(int nen_, int ncx, int ncy, int k_)
        : span(nen_ == 4 || nen_ == 3 ? 1 : 2), gx(span * ncx), gy(span * ncy), nen(nen_), k(k_) {}
    __device__ __forceinline__ int64_t operator()(int i, int j) const {
        if (k == 1) return i + (int64_t)j * (gx + 1);
        if (nen != 8) return (int64_t)i * (gy + 1) + j;
        // Q8: odd columns hold the nodes of even j only
        const int64_t pair = (gy + 1) + (gy / 2 + 1);
        return (i & 1) ? ((j & 1) ? -1 : (i / 2) * pair + gy + 1 + j / 2) : (i / 2) * pair + j;
    }
};

// positions (di, dj) of an element's nodes in its cell: quadrilaterals, the lower and the upper triangle
__device__ __forceinline__ void grid_corner(int nen, int half, int a, int& di, int& dj) {
    // corners counter-clockwise, mid-sides, centre, in half cells
    constexpr int qi[9] = {0, 2, 2, 0, 1, 2, 1, 0, 1}, qj[9] = {0, 0, 2, 2, 0, 1, 2, 1, 1};
    constexpr int t3[2][3] = {{0, 1, 3}, {1, 2, 3}}, t6[2][6] = {{0, 1, 3, 4, 8, 7}, {1, 2, 3, 5, 6, 8}};
    const int m = nen == 3 ? t3[half][a] : nen == 6 ? t6[half][a] : a;
    const int div = nen == 4 || nen == 3 ? 2 : 1;
    di = qi[m] / div;
    dj = qj[m] / div;
}

struct GridCandidates {
    int n, ncx[DFEA_GRID_CANDIDATES], ncy[DFEA_GRID_CANDIDATES];
};

__global__ void __launch_bounds__(256) k_grid_match(int64_t n_el, int nen, const int64_t* __restrict__ conn, GridCandidates c,
                                                    int32_t* __restrict__ mismatch) {
    const bool triangles = nen == 3 || nen == 6;
    const int numberings = nen == 4 || nen == 9 ? 2 : 1;
    for (int64_t base = blockIdx.x * (int64_t)blockDim.x; base < n_el; base += (int64_t)gridDim.x * blockDim.x) {
        const int64_t e = base + threadIdx.x;
        for (int i = 0; i < c.n; ++i) {
            const int64_t n_cells = (int64_t)c.ncx[i] * c.ncy[i];
            const int half = triangles && e >= n_cells ? 1 : 0;
            const int64_t cell = e - half * n_cells;
            for (int k = 0; k < numberings; ++k) {
                bool differs = false;
                if (e < n_el) {
                    const GridNumbering id(nen, c.ncx[i], c.ncy[i], k);
                    const int ci = (int)(cell / c.ncy[i]) * id.span, cj = (int)(cell % c.ncy[i]) * id.span;
                    for (int a = 0; a < nen; ++a) {
                        int di, dj;
                        grid_corner(nen, half, a, di, dj);
                        differs |= conn[e * nen + a] != id(ci + di, cj + dj);
                    }
                }
                if (__any_sync(0xffffffffu, differs) && (threadIdx.x & 31) == 0) mismatch[2 * i + k] = 1;
            }
        }
    }
    if (numberings == 1 && blockIdx.x == 0 && threadIdx.x < c.n) mismatch[2 * threadIdx.x + 1] = 1;
}

__global__ void __launch_bounds__(256) k_grid_nodes(int nen, int ncx, int ncy, int numbering, int32_t* __restrict__ gnode,
                                                    int2* __restrict__ node_ij) {
    const GridNumbering id(nen, ncx, ncy, numbering);
    const int64_t n = (int64_t)(id.gx + 1) * (id.gy + 1);
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < n; t += (int64_t)gridDim.x * blockDim.x) {
        const int i = (int)(t / (id.gy + 1)), j = (int)(t % (id.gy + 1));
        const int64_t node = id(i, j);
        gnode[t] = (int32_t)node;
        if (node >= 0) node_ij[node] = make_int2(i, j);
    }
}

struct GridLines {
    int n;
    int gx[DFEA_MG_MAX_LEVELS], gy[DFEA_MG_MAX_LEVELS];
    int32_t* at[DFEA_MG_MAX_LEVELS][4];  // line_x, line_y, cell_x, cell_y of level l >= 1
};

__global__ void __launch_bounds__(256) k_mg_maps(Mesh m, int n_cells, int epc, int32_t* __restrict__ cell_slot,
                                                 const __grid_constant__ GridLines g) {
    const int64_t first = blockIdx.x * (int64_t)blockDim.x + threadIdx.x, step = (int64_t)gridDim.x * blockDim.x;
    for (int64_t slot = first; slot < m.n_el; slot += step) {
        const int e = m.orig[slot], k = e / n_cells;
        cell_slot[(int64_t)(e - k * n_cells) * epc + k] = (int32_t)slot;
    }
    for (int l = 1; l < g.n; ++l)
#pragma unroll
        for (int d = 0; d < 2; ++d) {
            const int fine = d ? g.gy[l - 1] : g.gx[l - 1], coarse = d ? g.gy[l] : g.gx[l];
            for (int64_t i = first; i <= fine; i += step) {
                if (i <= coarse) g.at[l][d][i] = 2 * (int)i < fine ? 2 * (int)i : fine;
                g.at[l][2 + d][i] = (int)i / 2 < coarse - 1 ? (int)i / 2 : coarse - 1;
            }
        }
}

// ------------------------------------------------------------------------------------------
// graph-driven mode: the captured set-up and the device-side PCG loop
// ------------------------------------------------------------------------------------------
// the graphs of one hierarchy, each bound to the buffers it was captured with
struct MgGraphs {
    cudaStream_t capture = nullptr;
    cudaStream_t branch[2] = {};  // of a captured set-up, with the events that fork and join them
    cudaEvent_t fork[2] = {}, join[2] = {};
    // set-up: moduli, diag and the mesh arrays the level-0 product reads; with and without the Lanczos bounds
    const void* key_setup[6] = {};
    int32_t code_setup = -1;
    int calls_setup[2] = {0, 0};
    cudaGraphExec_t setup[2] = {nullptr, nullptr};
    long long kernels_setup[2] = {0, 0};
    // PCG: moduli, b, x and the mesh arrays
    const void* key_pcg[7] = {};
    int32_t code_pcg = -1;
    int calls_pcg = 0;
    cudaGraphExec_t loop = nullptr;
    long long kernels_body = 0;

    void drop_setup() {
        for (int i = 0; i < 2; ++i) {
            if (setup[i]) cudaGraphExecDestroy(setup[i]);
            setup[i] = nullptr;
            calls_setup[i] = 0;
        }
    }
    void drop_pcg() {
        if (loop) cudaGraphExecDestroy(loop);
        loop = nullptr;
    }
    ~MgGraphs() {
        drop_setup();
        drop_pcg();
        if (capture) cudaStreamDestroy(capture);
        for (int i = 0; i < 2; ++i) {
            if (branch[i]) cudaStreamDestroy(branch[i]);
            if (fork[i]) cudaEventDestroy(fork[i]);
            if (join[i]) cudaEventDestroy(join[i]);
        }
    }
    int make_branches() {
        int rc = DFEA_OK;
        for (int i = 0; !rc && i < 2; ++i) {
            if (!branch[i]) rc = check_cuda(cudaStreamCreateWithFlags(&branch[i], cudaStreamNonBlocking), "cudaStreamCreate");
            if (!rc && !fork[i]) rc = check_cuda(cudaEventCreateWithFlags(&fork[i], cudaEventDisableTiming), "cudaEventCreate");
            if (!rc && !join[i]) rc = check_cuda(cudaEventCreateWithFlags(&join[i], cudaEventDisableTiming), "cudaEventCreate");
        }
        return rc;
    }
};

static bool same_key(const void* const* a, const void* const* b, int n) {
    for (int i = 0; i < n; ++i)
        if (a[i] != b[i]) return false;
    return true;
}

// Lanczos of level l by launches (p in x, z in d), on reduction scratch w
static int level_lanczos(const dfea_mesh_view* mesh, const dfea_mg* mg, const void* moduli, int32_t code, int l, double* w,
                         cudaStream_t s) {
    const dfea_mg_level& lv = mg->level[l];
    const int64_t n = lv.n;
    double *sc = mg->lscal + 4 * l, *hist = mg->lhist + (int64_t)2 * mg->lanczos_steps * l;
    const int nb = mg_dot_blocks(n);
    int rc;
    k_mg_lanczos_start<<<nb, kMgDotThreads, 0, s>>>(n, lv.r, lv.d, lv.x, lv.diag, sc, w);
    note_launches(1);
    if ((rc = launch_check("dfea_mg_setup: Lanczos start"))) return rc;
    const bool fused = l == 0 && fe_gather(mesh, mg) && mg_fe_cg_supported(mesh, code);
    double *p = lv.x, *p_next = lv.b;
    for (int k = 0; k < mg->lanczos_steps; ++k) {
        if (fused) {
            MgCgStep a = {};
            a.z = lv.d, a.p = lv.x, a.r = lv.r, a.diag = lv.diag, a.scal = sc, a.hist = hist, a.k = k;
            if ((rc = mg_fe_cg_step(mesh, moduli, code, mg->fe_work, MG_CG_LANCZOS, a, w, s))) return rc;
            continue;
        }
        if (l == 0) {
            if ((rc = mg_apply(mesh, mg, moduli, code, 0, lv.x, lv.q, s)) ||
                (rc = mg_dot1<MG_DOT_PLAIN>(n, lv.x, lv.q, sc, w, s)))
                return rc;
        } else {
            rc = launch_kernel(k_mg_lanczos_apply, dim3(grid_for(n / 2, kMgDotThreads, 8)), dim3(kMgDotThreads), 0, s,
                               overlapping(), level_grid(mg, l), (const double*)lv.d, (const double*)p, p_next, lv.q, sc, w);
            if (rc) return rc;
            note_launches(1);
            std::swap(p, p_next);
        }
        rc = launch_kernel(k_mg_lanczos_step_rz, dim3(nb), dim3(kMgDotThreads), 0, s, overlapping(), n, (const double*)lv.q,
                           lv.r, lv.d, (const double*)lv.diag, sc, w, hist, k);
        if (rc) return rc;
        note_launches(1);
        if (l == 0) {
            k_mg_lanczos_p<<<grid_for(n, kThreads, 8), kThreads, 0, s>>>(n, lv.x, lv.d, sc);
            note_launches(1);
        }
    }
    return launch_check("dfea_mg_setup: Lanczos");
}

// Lanczos of the small levels t .. L-2, one cluster per level
static int tail_lanczos(const dfea_mg* mg, int t, cudaStream_t s) {
    const int L = mg->n_levels;
    MgLanczosTail T = {};
    T.steps = mg->lanczos_steps;
    T.size = mg_cluster_size(mg->level[t].n / 2, tail_blocks());
    int most = 0, rc;
    for (int k = 0; k < L - 1 - t; ++k) {
        const dfea_mg_level& lv = mg->level[t + k];
        const int n_nodes = (int)(lv.n / 2), nb = (n_nodes + T.size - 1) / T.size;
        T.lv[k] = MgLanczosLevel{level_grid(mg, t + k), n_nodes, nb, lv.diag, mg->lscal + 4 * (t + k),
                                 mg->lhist + (int64_t)2 * mg->lanczos_steps * (t + k)};
        most = nb > most ? nb : most;
    }
    if ((rc = launch_clusters<k_mg_tail_lanczos>(L - 1 - t, T.size, (size_t)(4 * 16 + 36 * 8) * most, false, s, T))) return rc;
    note_launches(1);
    return launch_check("dfea_mg_setup: Lanczos of the small levels");
}

// The device part of a set-up: coarse operators, coarsest inverse, Lanczos coefficients into mg->lhist.  The estimate of
// level 0 needs no coarse operator and those of the large coarse levels no coarsest inverse: chains of short launches
// that leave most of the GPU idle, so a captured set-up (g) runs them on branches beside the rest -- the same launches,
// the same results.  128 x 128 Q9: 450 us in line, 250 us in branches.
static int setup_device_part(const dfea_mesh_view* mesh, const dfea_mg* mg, const void* moduli, int32_t moduli_dtype,
                             const double* diag, cudaStream_t s, bool lanczos, MgGraphs* g) {
    int rc;
    const int L = mg->n_levels;
    const int t = tail_start(mg) < L - 1 ? tail_start(mg) : L - 1;
    double* scratch[2] = {mg->dot_work, mg->dot_work + kMgDotScratch};
    cudaStream_t on[2] = {s, s};
    const auto fork = [&](int i) -> int {
        if (!g) return DFEA_OK;
        on[i] = g->branch[i];
        const int e = check_cuda(cudaEventRecord(g->fork[i], s), "cudaEventRecord");
        return e ? e : check_cuda(cudaStreamWaitEvent(on[i], g->fork[i], 0), "cudaStreamWaitEvent");
    };
    const auto join = [&](int i) -> int {
        if (on[i] == s) return DFEA_OK;
        const int e = check_cuda(cudaEventRecord(g->join[i], on[i]), "cudaEventRecord");
        return e ? e : check_cuda(cudaStreamWaitEvent(s, g->join[i], 0), "cudaStreamWaitEvent");
    };
    for (double* w : scratch)
        if ((rc = check_cuda(cudaMemsetAsync(dot_ticket(w), 0, sizeof(unsigned), s), "cudaMemsetAsync"))) return rc;
    if ((rc = check_cuda(cudaMemcpyAsync(mg->level[0].diag, diag, mg->level[0].n * sizeof(double), cudaMemcpyDeviceToDevice, s),
                         "cudaMemcpyAsync")))
        return rc;
    if (lanczos && t > 0 && ((rc = fork(0)) || (rc = level_lanczos(mesh, mg, moduli, moduli_dtype, 0, scratch[0], on[0])))) return rc;
    for (int l = 1; l < L; ++l) {
        const int32_t* gn;
        const uint8_t* ffix;
        transfer_args(mesh, mg, l - 1, &gn, &ffix);
        if ((rc = dfea_mg_restrict(&mg->level[l - 1].grid, &mg->level[l].grid, gn, ffix, nullptr, nullptr,
                                   mg->level[l].grid.fix, s)))
            return rc;
        rc = l == 1 ? dfea_mg_galerkin_fe(mesh, moduli, moduli_dtype, mg->node_ij, mg->cell_slot, mg->span,
                                          &mg->level[0].grid, &mg->level[1].grid, s)
                    : dfea_mg_galerkin(&mg->level[l - 1].grid, &mg->level[l].grid, s);
        if (rc) return rc;
        if (mg->stencil) {
            k_mg_stencil<<<grid_for(9 * (mg->level[l].n / 2), 256, 8), 256, 0, s>>>(level_grid(mg, l), mg->level[l].diag);
            note_launches(1);
            rc = launch_check("dfea_mg_setup: stencils");
        } else {
            rc = dfea_mg_diag(&mg->level[l].grid, mg->level[l].diag, s);
        }
        if (rc) return rc;
    }
    if (lanczos && t > 1) {
        if ((rc = fork(1))) return rc;
        for (int l = 1; l < t; ++l)
            if ((rc = level_lanczos(mesh, mg, moduli, moduli_dtype, l, scratch[1], on[1]))) return rc;
    }
    if ((rc = dfea_mg_dense_inverse(&mg->level[L - 1].grid, mg->dense_work, mg->Ainv, s)) ||
        (lanczos && t < L - 1 && (rc = tail_lanczos(mg, t, s))))
        return rc;
    return (rc = join(0)) ? rc : join(1);
}

// Capture `body(stream)` into a new graph on the hierarchy's capture stream and instantiate it; the kernels
// the body notes while capturing are not launches yet (they are counted per replay instead).
template <typename F>
static int capture_exec(MgGraphs* g, F&& body, cudaGraphExec_t* out, long long* kernels) {
    int rc;
    if (!g->capture && (rc = check_cuda(cudaStreamCreateWithFlags(&g->capture, cudaStreamNonBlocking), "cudaStreamCreate")))
        return rc;
    const long long before = thread_launch_count();
    if ((rc = check_cuda(cudaStreamBeginCapture(g->capture, cudaStreamCaptureModeThreadLocal), "cudaStreamBeginCapture")))
        return rc;
    rc = body(g->capture);
    cudaGraph_t graph = nullptr;
    const int rc_end = check_cuda(cudaStreamEndCapture(g->capture, &graph), "cudaStreamEndCapture");
    *kernels = thread_launch_count() - before;
    note_launches(-*kernels);
    if (!rc && !rc_end) rc = check_cuda(cudaGraphInstantiate(out, graph, 0), "cudaGraphInstantiate");
    if (graph) cudaGraphDestroy(graph);
    return rc ? rc : rc_end;
}

__global__ void k_mgp_init(MgPcgState* st, double rtol, int max_iter) {
    st->rtol2 = rtol * rtol;
    st->max_iter = max_iter;
    st->k = 0;
    st->iters = 0;
    st->beta = 0.0;
    st->status = DFEA_PCG_RUNNING;
}

// start of a solve: x = 0, p = 0, r = b, the first cycle's first direction d = scale r / D, |b|^2, the tolerance and the
// ends that need no iteration; with `loop` the condition of the loop
__global__ void __launch_bounds__(kMgDotThreads) k_mgp_start(int64_t n, const double* __restrict__ b, double* __restrict__ x,
                                                             double* __restrict__ r, double* __restrict__ p,
                                                             double* __restrict__ d, const double* __restrict__ diag,
                                                             const double* __restrict__ scale, MgPcgState* st,
                                                             double* __restrict__ work, int loop, cudaGraphConditionalHandle cond) {
    const double s = *scale;
    double a = 0.0;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const double bi = b[i];
        x[i] = 0.0;
        p[i] = 0.0;
        r[i] = bi;
        d[i] = s * bi / diag[i];
        a += bi * bi;
    }
    const double vals[1] = {block_sum<kMgDotThreads>(a)};
    double tot[1];
    if (last_block_sum<kMgDotThreads, 1>(vals, RedSite{work, dot_ticket(work), nullptr}, tot) && threadIdx.x == 0) {
        st->nb2 = tot[0];
        st->tol2 = st->rtol2 * tot[0];
        if (tot[0] == 0.0) {
            st->status = DFEA_PCG_ZERO_RHS;
        } else if (st->max_iter <= 0) {
            st->status = DFEA_PCG_MAX_ITER;
            st->iters = st->max_iter;
        }
        if (loop) cudaGraphSetConditional(cond, st->status == DFEA_PCG_RUNNING ? 1u : 0u);
    }
}

// General form of an iteration (level 0 without reference-frame moduli or node incidence): p = z + beta p; ...
__global__ void k_mgp_direction(int64_t n, const MgPcgState* __restrict__ st, double* __restrict__ p,
                                const double* __restrict__ z) {
    const double beta = st->beta;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        p[i] = z[i] + beta * p[i];
}

// ... and after q = A p and p.q what k_mg_cg_node does at its nodes
__global__ void __launch_bounds__(kMgDotThreads) k_mgp_update(int64_t n, MgPcgState* st, double* __restrict__ x,
                                                              double* __restrict__ r, const double* __restrict__ p,
                                                              const double* __restrict__ q, const double* __restrict__ z,
                                                              double* __restrict__ work, int loop, cudaGraphConditionalHandle cond) {
    const double curv = st->curv, alpha = st->rz / curv;
    const bool curved = curv > 0.0, take_z = !curved && st->k == 0;
    double a = 0.0;
    if (curved || take_z)
        for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
            if (take_z) {
                x[i] = z[i];
                continue;
            }
            x[i] += alpha * p[i];
            const double ri = r[i] - alpha * q[i];
            r[i] = ri;
            a += ri * ri;
        }
    const double vals[1] = {block_sum<kMgDotThreads>(a)};
    double tot[1];
    if (last_block_sum<kMgDotThreads, 1>(vals, RedSite{work, dot_ticket(work), nullptr}, tot) && threadIdx.x == 0) {
        const bool on = pcg_iteration_end(st, curved, tot[0]);
        if (loop) cudaGraphSetConditional(cond, on ? 1u : 0u);
    }
}

// A solve: the state, the start, then iterations while the status says so.  An iteration begins with the cycle (z, r.z
// and beta), so no cycle runs that no step uses, and everything it decides it decides on the device.  A Newton solve on
// 128 x 128 Q9, 54 iterations in 14 solves: 24.6 ms with the cycle at the end of an iteration (one unused per solve) and a
// launch for each dot, update and smoothing start -> 18.8 ms.
static int pcg_start_part(const dfea_mg* mg, MgPcgState* st, const double* b, double* x, const cudaGraphConditionalHandle* cond,
                          cudaStream_t s) {
    const dfea_mg_level& lv = mg->level[0];
    const int64_t n = lv.n;
    double *r = mg->pcg, *p = mg->pcg + 2 * n;
    k_mgp_start<<<mg_dot_blocks(n), kMgDotThreads, 0, s>>>(n, b, x, r, p, lv.d, lv.diag, mg->coef, st, mg->dot_work,
                                                           cond ? 1 : 0, cond ? *cond : cudaGraphConditionalHandle{});
    note_launches(1);
    return launch_check("dfea_mg_pcg: start");
}

static int pcg_body_part(const dfea_mesh_view* mesh, const dfea_mg* mg, MgPcgState* st, const void* moduli, int32_t code,
                         double* x, const cudaGraphConditionalHandle* cond, cudaStream_t s) {
    const dfea_mg_level& lv = mg->level[0];
    const int64_t n = lv.n;
    double *r = mg->pcg, *z = mg->pcg + n, *p = mg->pcg + 2 * n, *q = mg->pcg + 3 * n;
    const bool fused = fe_gather(mesh, mg) && mg_fe_cg_supported(mesh, code);
    CycleUse use;
    use.started = fused;
    use.dot = st;
    int rc;
    if ((rc = mg_vcycle(mesh, mg, moduli, code, 0, r, z, use, s))) return rc;
    if (fused) {
        MgCgStep a = {};
        a.z = z, a.p = p, a.r = r, a.x = x, a.d = lv.d, a.diag = lv.diag, a.scale = mg->coef, a.st = st;
        a.loop = cond != nullptr;
        if (cond) a.cond = *cond;
        return mg_fe_cg_step(mesh, moduli, code, mg->fe_work, MG_CG_SOLVE, a, mg->dot_work, s);
    }
    k_mgp_direction<<<grid_for(n, kThreads, 8), kThreads, 0, s>>>(n, st, p, z);
    note_launches(1);
    if ((rc = launch_check("dfea_mg_pcg: direction")) || (rc = mg_apply(mesh, mg, moduli, code, 0, p, q, s)) ||
        (rc = mg_dot1<MG_DOT_PLAIN>(n, p, q, &st->curv, mg->dot_work, s)))
        return rc;
    k_mgp_update<<<mg_dot_blocks(n), kMgDotThreads, 0, s>>>(n, st, x, r, p, q, z, mg->dot_work, cond ? 1 : 0,
                                                            cond ? *cond : cudaGraphConditionalHandle{});
    note_launches(1);
    return launch_check("dfea_mg_pcg: update");
}

// the graph of a solve: the start, which sets the condition, then a while node around one iteration
static int build_loop_graph(MgGraphs* g, const dfea_mesh_view* mesh, const dfea_mg* mg, const void* moduli,
                            int32_t code, const double* b, double* x) {
    int rc;
    if (!g->capture && (rc = check_cuda(cudaStreamCreateWithFlags(&g->capture, cudaStreamNonBlocking), "cudaStreamCreate")))
        return rc;
    cudaGraph_t graph = nullptr;
    if ((rc = check_cuda(cudaGraphCreate(&graph, 0), "cudaGraphCreate"))) return rc;
    auto fail = [&](int code_) {
        cudaGraphDestroy(graph);
        return code_;
    };
    cudaGraphConditionalHandle cond;
    if ((rc = check_cuda(cudaGraphConditionalHandleCreate(&cond, graph, 0u, cudaGraphCondAssignDefault),
                         "cudaGraphConditionalHandleCreate")))
        return fail(rc);
    MgPcgState* st = reinterpret_cast<MgPcgState*>(mg->pcg_state);
    if ((rc = check_cuda(cudaStreamBeginCaptureToGraph(g->capture, graph, nullptr, nullptr, 0, cudaStreamCaptureModeThreadLocal),
                         "cudaStreamBeginCaptureToGraph")))
        return fail(rc);
    rc = pcg_start_part(mg, st, b, x, &cond, g->capture);
    note_launches(-1);
    cudaGraph_t cap = graph;
    int rc_end = check_cuda(cudaStreamEndCapture(g->capture, &cap), "cudaStreamEndCapture");
    if (rc || rc_end) return fail(rc ? rc : rc_end);
    cudaGraphNode_t first = nullptr;
    size_t n_nodes = 1;
    if ((rc = check_cuda(cudaGraphGetNodes(graph, &first, &n_nodes), "cudaGraphGetNodes"))) return fail(rc);
    if (n_nodes != 1) return fail(set_error(DFEA_ERR_CUDA, "dfea_mg_pcg: unexpected loop-graph prologue"));
    cudaGraphNodeParams cp = {cudaGraphNodeTypeConditional};
    cp.conditional.handle = cond;
    cp.conditional.type = cudaGraphCondTypeWhile;
    cp.conditional.size = 1;
    cudaGraphNode_t node;
    if ((rc = check_cuda(cudaGraphAddNode(&node, graph, &first, 1, &cp), "cudaGraphAddNode(while)"))) return fail(rc);
    cudaGraph_t body = cp.conditional.phGraph_out[0];
    const long long before = thread_launch_count();
    if ((rc = check_cuda(cudaStreamBeginCaptureToGraph(g->capture, body, nullptr, nullptr, 0, cudaStreamCaptureModeThreadLocal),
                         "cudaStreamBeginCaptureToGraph")))
        return fail(rc);
    rc = pcg_body_part(mesh, mg, st, moduli, code, x, &cond, g->capture);
    cudaGraph_t body_cap = body;
    rc_end = check_cuda(cudaStreamEndCapture(g->capture, &body_cap), "cudaStreamEndCapture");
    g->kernels_body = thread_launch_count() - before;
    note_launches(-g->kernels_body);
    if (rc || rc_end) return fail(rc ? rc : rc_end);
    rc = check_cuda(cudaGraphInstantiate(&g->loop, graph, 0), "cudaGraphInstantiate");
    cudaGraphDestroy(graph);
    return rc;
}

// a solve's end from its state
static int pcg_result(const MgPcgState& st, int32_t* iterations, int32_t* status) {
    if (st.status == DFEA_PCG_RUNNING) return set_error(DFEA_ERR_INVALID, "dfea_mg_pcg: the loop ended without a status");
    *status = st.status;
    *iterations = st.iters;
    return DFEA_OK;
}

// graph-driven PCG: the state, one graph launch, one status read
static int pcg_graph_solve(MgGraphs* g, const dfea_mg* mg, double rtol, int32_t max_iter, int32_t* iterations,
                           int32_t* status, cudaStream_t s) {
    MgPcgState* st = reinterpret_cast<MgPcgState*>(mg->pcg_state);
    k_mgp_init<<<1, 1, 0, s>>>(st, rtol, max_iter);
    int rc = launch_check("dfea_mg_pcg: init");
    if (rc || (rc = check_cuda(cudaGraphLaunch(g->loop, s), "cudaGraphLaunch"))) return rc;
    MgPcgState host;
    if ((rc = read_to_host(&host, st, sizeof(host), s))) return rc;
    const long long bodies = host.nb2 == 0.0 ? 0 : host.k + (host.status == DFEA_PCG_NEG_CURV ? 1 : 0);
    note_launches(2 + bodies * g->kernels_body);
    return pcg_result(host, iterations, status);
}

}  // namespace dfea

extern "C" int dfea_grid_match(int64_t n_el, int32_t nen, const int64_t* conn, int32_t n_cand, const int32_t* ncx,
                               const int32_t* ncy, int32_t* mismatch, void* stream) {
    const bool known = nen == 4 || nen == 9 || nen == 8 || nen == 3 || nen == 6;
    if (n_el < 1 || !known || !conn || n_cand < 1 || n_cand > DFEA_GRID_CANDIDATES || !ncx || !ncy || !mismatch)
        return set_error(DFEA_ERR_INVALID, "dfea_grid_match: bad arguments");
    GridCandidates c = {};
    c.n = n_cand;
    for (int i = 0; i < n_cand; ++i) {
        c.ncx[i] = ncx[i];
        c.ncy[i] = ncy[i];
        if (ncx[i] < 1 || ncy[i] < 1 || (int64_t)ncx[i] * ncy[i] * (nen == 3 || nen == 6 ? 2 : 1) != n_el)
            return set_error(DFEA_ERR_INVALID, "dfea_grid_match: candidate %d does not have the element count", i);
    }
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    int rc = check_cuda(cudaMemsetAsync(mismatch, 0, 2 * DFEA_GRID_CANDIDATES * sizeof(int32_t), s), "cudaMemsetAsync");
    if (rc) return rc;
    k_grid_match<<<grid_for(n_el, 256, 8), 256, 0, s>>>(n_el, nen, conn, c, mismatch);
    note_launches(1);
    return launch_check("dfea_grid_match");
}

extern "C" int dfea_grid_nodes(int32_t nen, int32_t ncx, int32_t ncy, int32_t numbering, int32_t* gnode, int32_t* node_ij,
                               void* stream) {
    const bool known = nen == 4 || nen == 9 || nen == 8 || nen == 3 || nen == 6;
    const int span = nen == 4 || nen == 3 ? 1 : 2;
    if (!known || ncx < 1 || ncy < 1 || numbering < 0 || numbering > (nen == 4 || nen == 9 ? 1 : 0) || !gnode || !node_ij ||
        (reinterpret_cast<uintptr_t>(node_ij) & 7))
        return set_error(DFEA_ERR_INVALID, "dfea_grid_nodes: bad arguments");
    const int64_t n = ((int64_t)span * ncx + 1) * ((int64_t)span * ncy + 1);
    if (n >= (int64_t(1) << 31)) return set_error(DFEA_ERR_INVALID, "dfea_grid_nodes: too many nodes");
    k_grid_nodes<<<grid_for(n, 256, 8), 256, 0, static_cast<cudaStream_t>(stream)>>>(nen, ncx, ncy, numbering, gnode,
                                                                                     reinterpret_cast<int2*>(node_ij));
    note_launches(1);
    return launch_check("dfea_grid_nodes");
}

extern "C" int dfea_mg_maps(const dfea_mesh_view* mesh, const dfea_mg* mg, void* stream) {
    int rc = validate_mesh(mesh, false);
    if (rc) return rc;
    if (!mg || mg->n_levels < 2 || mg->n_levels > DFEA_MG_MAX_LEVELS || !mg->cell_slot || mg->span < 1 || mg->span > 2)
        return set_error(DFEA_ERR_INVALID, "dfea_mg_maps: bad hierarchy parameters");
    GridLines g = {};
    g.n = mg->n_levels;
    for (int l = 0; l < g.n; ++l) {
        const dfea_mg_grid& lv = mg->level[l].grid;
        g.gx[l] = lv.gx;
        g.gy[l] = lv.gy;
        const int32_t* at[4] = {lv.line_x, lv.line_y, lv.cell_x, lv.cell_y};
        for (int k = 0; k < 4; ++k) {
            if (l > 0 && !at[k]) return set_error(DFEA_ERR_INVALID, "dfea_mg_maps: NULL map");
            g.at[l][k] = const_cast<int32_t*>(at[k]);
        }
        // a level's lines lie among twice as many finer ones
        if (lv.gx < 1 || lv.gy < 1 || (l > 0 && (lv.gx > g.gx[l - 1] || lv.gy > g.gy[l - 1])))
            return set_error(DFEA_ERR_INVALID, "dfea_mg_maps: level %d", l);
    }
    const int64_t n_cells = (int64_t)(g.gx[0] / mg->span) * (g.gy[0] / mg->span);
    const int64_t epc = n_cells > 0 ? mesh->n_el / n_cells : 0;
    if (epc < 1 || epc * n_cells != mesh->n_el) return set_error(DFEA_ERR_INVALID, "dfea_mg_maps: level 0 is not the mesh's grid");
    k_mg_maps<<<grid_for(mesh->n_el, 256, 8), 256, 0, static_cast<cudaStream_t>(stream)>>>(
        kernel_mesh(*mesh), (int)n_cells, (int)epc, const_cast<int32_t*>(mg->cell_slot), g);
    note_launches(1);
    return launch_check("dfea_mg_maps");
}

extern "C" int32_t dfea_mg_tail_level(const dfea_mg* mg, int32_t blocks, int64_t bytes) {
    if (!mg || mg->n_levels < 2 || mg->n_levels > DFEA_MG_MAX_LEVELS || blocks < 1 || bytes < 0) return -1;
    return tail_level(mg, blocks < kClusterMax ? blocks : kClusterMax, bytes);
}

extern "C" int dfea_mg_setup(const dfea_mesh_view* mesh, dfea_mg* mg, const void* moduli, int32_t moduli_dtype,
                             const double* diag, void* stream) {
    int rc = validate_mg(mesh, mg, "dfea_mg_setup");
    if (rc) return rc;
    if (!moduli || !diag) return set_error(DFEA_ERR_INVALID, "dfea_mg_setup: NULL pointer");
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const int L = mg->n_levels;
    // the smoother bounds: estimated now, or kept from an earlier set-up of this hierarchy
    const bool lanczos = mg->bounds_every <= 0 || mg->setups <= 0 || (mg->setups % mg->bounds_every) == 0;
    mg->setups = mg->setups < 0 ? 1 : mg->setups + 1;
    if (mg->pcg_state) {
        if (!mg->graphs) {
            MgGraphs* g = new (std::nothrow) MgGraphs;
            if (!g) return set_error(DFEA_ERR_INVALID, "dfea_mg_setup: out of host memory");
            mg->graphs = g;
        }
        MgGraphs* g = static_cast<MgGraphs*>(mg->graphs);
        const void* key[6] = {moduli, diag, mesh->conn, mesh->grad, mesh->grad32, mesh->jinv};
        if (!same_key(key, g->key_setup, 6) || g->code_setup != moduli_dtype) {
            g->drop_setup();
            for (int i = 0; i < 6; ++i) g->key_setup[i] = key[i];
            g->code_setup = moduli_dtype;
        }
        const int v = lanczos ? 1 : 0;
        if (g->calls_setup[v]++ == 0) {
            rc = setup_device_part(mesh, mg, moduli, moduli_dtype, diag, s, lanczos, nullptr);   // direct, the first time
        } else {
            if (!g->setup[v] &&
                ((rc = g->make_branches()) ||
                 (rc = capture_exec(g, [&](cudaStream_t cs) { return setup_device_part(mesh, mg, moduli, moduli_dtype, diag, cs, lanczos, g); },
                                    &g->setup[v], &g->kernels_setup[v]))))
                return rc;
            rc = check_cuda(cudaGraphLaunch(g->setup[v], s), "cudaGraphLaunch");
            note_launches(g->kernels_setup[v]);
        }
    } else {
        rc = setup_device_part(mesh, mg, moduli, moduli_dtype, diag, s, lanczos, nullptr);
    }
    if (rc) return rc;
    if (!lanczos) return DFEA_OK;   // bounds, coefficients and lam[] of the last estimate stay in force
    const int nh = 2 * mg->lanczos_steps * (L - 1);
    double hist[2 * 64 * DFEA_MG_MAX_LEVELS];
    if ((rc = read_scalars(hist, mg->lhist, nh, s))) return rc;
    double coef[DFEA_MG_MAX_LEVELS * 2 * DFEA_MG_MAX_DEGREE] = {0.0};
    for (int l = 0; l < L - 1; ++l) {
        const double lam = ritz_max(hist + 2 * mg->lanczos_steps * l, mg->lanczos_steps);
        mg->lam[l] = lam;
        const double hi = 1.1 * lam, lo = hi / mg->ratio;
        const double theta = 0.5 * (hi + lo), delta = 0.5 * (hi - lo), sigma = theta / delta;
        double rho = 1.0 / sigma;
        double* row = coef + l * 2 * DFEA_MG_MAX_DEGREE;
        row[0] = 1.0 / theta;
        for (int k = 1; k < mg->degree; ++k) {
            const double rho_new = 1.0 / (2.0 * sigma - rho);
            row[1 + 2 * (k - 1)] = rho_new * rho;
            row[2 + 2 * (k - 1)] = 2.0 * rho_new / delta;
            rho = rho_new;
        }
    }
    if ((rc = check_cuda(cudaMemcpyAsync(mg->coef, coef, sizeof(double) * 2 * DFEA_MG_MAX_DEGREE * (L - 1),
                                         cudaMemcpyHostToDevice, s), "cudaMemcpyAsync")))
        return rc;
    // the copy reads a stack array: it has completed when the stream has
    return check_cuda(cudaStreamSynchronize(s), "cudaStreamSynchronize");
}

extern "C" int dfea_mg_release(dfea_mg* mg) {
    if (mg && mg->graphs) {
        delete static_cast<MgGraphs*>(mg->graphs);
        mg->graphs = nullptr;
    }
    return DFEA_OK;
}

extern "C" double dfea_mg_lanczos_bound(const double* hist, int32_t steps) {
    if (!hist || steps < 1 || steps > 64) return -1.0;
    return ritz_max(hist, steps);
}

extern "C" int dfea_mg_vcycle(const dfea_mesh_view* mesh, const dfea_mg* mg, const void* moduli, int32_t moduli_dtype,
                              const double* r, double* z, void* stream) {
    int rc = validate_mg(mesh, mg, "dfea_mg_vcycle");
    if (rc) return rc;
    if (!moduli || !r || !z) return set_error(DFEA_ERR_INVALID, "dfea_mg_vcycle: NULL pointer");
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    if (!paired(r)) {
        if ((rc = copy_vector(mg->level[0].b, r, mg->level[0].n, s))) return rc;
        r = mg->level[0].b;
    }
    return mg_vcycle(mesh, mg, moduli, moduli_dtype, 0, r, z, CycleUse(), s);
}

static int mg_pcg(const dfea_mesh_view* mesh, const dfea_mg* mg, const void* moduli, int32_t moduli_dtype, const double* b,
                  double* x, double rtol, int32_t max_iter, int32_t* iterations, int32_t* status, cudaStream_t s) {
    int rc;
    if (mg->pcg_state && mg->graphs) {
        // graph-driven: the second solve with the same buffers captures the loop, later ones replay it
        MgGraphs* g = static_cast<MgGraphs*>(mg->graphs);
        const void* key[7] = {moduli, b, x, mesh->conn, mesh->grad, mesh->grad32, mesh->jinv};
        if (!same_key(key, g->key_pcg, 7) || g->code_pcg != moduli_dtype) {
            g->drop_pcg();
            for (int i = 0; i < 7; ++i) g->key_pcg[i] = key[i];
            g->code_pcg = moduli_dtype;
            g->calls_pcg = 0;
        }
        if (g->calls_pcg++ > 0) {
            if (!g->loop && (rc = build_loop_graph(g, mesh, mg, moduli, moduli_dtype, b, x))) {
                g->drop_pcg();
                return rc;
            }
            return pcg_graph_solve(g, mg, rtol, max_iter, iterations, status, s);
        }
    }
    // host-driven: the same launches, the status read after every iteration
    MgPcgState* st = host_driven_state(mg->dot_work);
    MgPcgState host;
    k_mgp_init<<<1, 1, 0, s>>>(st, rtol, max_iter);
    note_launches(1);
    if ((rc = launch_check("dfea_mg_pcg: init")) || (rc = pcg_start_part(mg, st, b, x, nullptr, s)) ||
        (rc = read_to_host(&host, st, sizeof(host), s)))
        return rc;
    while (host.status == DFEA_PCG_RUNNING)
        if ((rc = pcg_body_part(mesh, mg, st, moduli, moduli_dtype, x, nullptr, s)) ||
            (rc = read_to_host(&host, st, sizeof(host), s)))
            return rc;
    return pcg_result(host, iterations, status);
}

extern "C" int dfea_mg_pcg(const dfea_mesh_view* mesh, const dfea_mg* mg, const void* moduli, int32_t moduli_dtype,
                           const double* b, double* x, double rtol, int32_t max_iter, int32_t* iterations,
                           int32_t* status, void* stream) {
    int rc = validate_mg(mesh, mg, "dfea_mg_pcg");
    if (rc) return rc;
    if (!moduli || !b || !x || !iterations || !status || max_iter < 0)
        return set_error(DFEA_ERR_INVALID, "dfea_mg_pcg: bad arguments");
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    double* own = paired(x) ? x : mg->level[0].b;
    rc = mg_pcg(mesh, mg, moduli, moduli_dtype, b, own, rtol, max_iter, iterations, status, s);
    return rc || own == x ? rc : copy_vector(x, own, mg->level[0].n, s);
}
