// dfea_pcg.cu -- kernel (c): Jacobi-preconditioned CG resident on the device.
//
// The reference runs PCG in Python with three host synchronisations per iteration
// (newton_krylov.py:28-88).  Here one iteration is
//     colour passes of k_apply<DOT>   Ap = A p  and  p.Ap (energy form, per colour, fixed order)
//     k_pcg_update1                   alpha = rz / pAp;  x += alpha p;  r -= alpha Ap;
//                                     |r|^2 and r.z with z = r / diag   (z is never stored)
//     k_pcg_update2                   convergence test; beta; p = z + beta p; Ap := (1 - m) p
//                                     (the pivot term of the next product); sum of fixed p^2
//     k_pcg_cond                      sets the condition of the graph's while-loop node
// captured once in a CUDA graph whose conditional WHILE node repeats it on the device, so that a
// whole solve is one graph launch and one read-back.  Scalars (rz, |r|^2, status, k) live in a
// device state block; every reduction is a fixed-order two-level sum (no float atomics).
//
// Termination does not depend on the numerics: k_pcg_update2 stops at max_iter and k_pcg_cond keeps
// an independent execution counter that ends the loop after max_iter + 4 bodies in any case.
#include <cstring>
#include <mutex>
#include <new>
#include <type_traits>

#include "dfea_apply.cuh"
#include "dfea_cluster.cuh"
#include "dfea_common.cuh"

namespace dfea {

int validate_mesh(const dfea_mesh_view* mv, bool need_grad32);

struct PcgState {
    double rz;      // r.z of the current iterate
    double rr;      // |r|^2 after the last update   (result[0] of the update-1 site)
    double rz_new;  // r.z after the last update     (result[1] of the update-1 site)
    double norm_b;
    double rtol;
    double pfix;    // sum of p^2 over fixed DOFs (identity rows of A)
    double curv;    // last p.Ap
    double beta;    // fused form: beta of the last update (0 before the first iteration)
    double curv_c[DFEA_MAX_COLOURS];
    int32_t k;
    int32_t max_iter;
    int32_t done;
    int32_t iters;
    int32_t guard;
    int32_t spare_i[3];
    unsigned tickets[DFEA_MAX_COLOURS + 8];
};

// Work buffer: [r | p | Ap] vectors (2N each, 256-byte aligned), partials, state, and for the gather
// form the element results fe (nen * stride pairs) at the end.
struct PcgLayout {
    int64_t off_r, off_p, off_y, off_part, off_state, off_fe, total;
    PcgLayout(int64_t n_nodes, int vec_bytes, int n_colours, int64_t fe_pairs = 0) {
        auto up = [](int64_t x) { return (x + 255) / 256 * 256; };
        const int64_t vb = up(2 * n_nodes * vec_bytes);
        off_r = 0;
        off_p = vb;
        off_y = 2 * vb;
        off_part = 3 * vb;
        const int64_t n_sites = n_colours + 3;
        off_state = off_part + up(n_sites * 3 * (int64_t)kMaxBlocks * 8);
        off_fe = off_state + up(sizeof(PcgState));
        total = off_fe + up(fe_pairs * 2 * vec_bytes);
    }
};

// The preconditioner z = M^-1 r at node n.  BJ = false: point Jacobi, d = diag (2N);  BJ = true: nodal
// block-Jacobi, d = the inverse 2x2 blocks (Binv00, Binv01, Binv11, 0) per node (4N, double vectors only).
template <bool BJ, typename T>
__device__ __forceinline__ v2_t<T> precond(const T* __restrict__ d, int64_t n, v2_t<T> r) {
    if constexpr (BJ) {
        const double2* b2 = reinterpret_cast<const double2*>(d);
        const double2 a = b2[2 * n], b = b2[2 * n + 1];
        return make_v2<T>((T)(a.x * r.x + a.y * r.y), (T)(a.y * r.x + b.x * r.y));
    } else {
        const v2_t<T> dn = reinterpret_cast<const v2_t<T>*>(d)[n];
        return make_v2<T>(r.x / dn.x, r.y / dn.y);
    }
}

__global__ void k_pcg_reset(PcgState* st) {
    const int i = threadIdx.x;
    if (i < DFEA_MAX_COLOURS + 8) st->tickets[i] = 0u;
    if (i < DFEA_MAX_COLOURS) st->curv_c[i] = 0.0;
    if (i == 0) {
        st->done = DFEA_PCG_RUNNING;
        st->k = 0;
        st->iters = 0;
        st->guard = 0;
    }
}

// x = 0, r = b, z = b / d, p = z, Ap := (1 - m) p;  rz = r.z, |b|, pfix.
template <typename T, bool BJ>
__global__ void __launch_bounds__(kThreads)
k_pcg_setup(Mesh m, const T* __restrict__ b, const T* __restrict__ d, T* __restrict__ x, T* __restrict__ r,
            T* __restrict__ p, T* __restrict__ y, PcgState* st, RedSite site, double rtol, int max_iter) {
    using T2 = v2_t<T>;
    double rz = 0.0, bb = 0.0, pf = 0.0;
    for (int64_t n = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; n < m.n_nodes; n += (int64_t)gridDim.x * blockDim.x) {
        const int fix = m.node_fix[n];
        const T2 bn = reinterpret_cast<const T2*>(b)[n];
        const T2 zn = precond<BJ, T>(d, n, bn);
        const T zx = zn.x, zy = zn.y;
        reinterpret_cast<T2*>(x)[n] = make_v2<T>(T(0), T(0));
        reinterpret_cast<T2*>(r)[n] = bn;
        reinterpret_cast<T2*>(p)[n] = make_v2<T>(zx, zy);
        reinterpret_cast<T2*>(y)[n] = make_v2<T>((fix & 1) ? zx : T(0), (fix & 2) ? zy : T(0));
        rz += (double)bn.x * zx + (double)bn.y * zy;
        bb += (double)bn.x * bn.x + (double)bn.y * bn.y;
        if (fix & 1) pf += (double)zx * zx;
        if (fix & 2) pf += (double)zy * zy;
    }
    const double vals[3] = {block_sum<kThreads>(rz), block_sum<kThreads>(bb), block_sum<kThreads>(pf)};
    double tot[3];
    if (last_block_sum<kThreads, 3>(vals, site, tot) && threadIdx.x == 0) {
        st->rz = tot[0];
        st->norm_b = sqrt(tot[1]);
        st->pfix = tot[2];
        st->beta = 0.0;
        st->rtol = rtol;
        st->max_iter = max_iter;
        st->k = 0;
        st->iters = 0;
        st->guard = 0;
        st->done = (st->norm_b == 0.0) ? DFEA_PCG_ZERO_RHS : DFEA_PCG_RUNNING;
    }
}

// GATHER: Ap is not stored; each node sums its elements' results (fe, the element pass of the gather
// form) in the incidence order, and takes p on its fixed DOFs (the identity rows).
// The body of update 1 for block blk of nblk (one launch, or one solve's share of a batched launch).
template <typename T, bool GATHER, bool BJ>
__device__ __forceinline__ void pcg_update1_body(const Mesh& m, int n_colours, const T* p,
                                                 const T* y, const T* __restrict__ d, T* __restrict__ x,
                                                 T* __restrict__ r, PcgState* st, const RedSite& site,
                                                 const int32_t* __restrict__ inc_ptr, const int32_t* __restrict__ inc,
                                                 const T* fe, int64_t blk, int64_t nblk) {
    using T2 = v2_t<T>;
    if (st->done) return;
    double curv = st->pfix;
    for (int c = 0; c < n_colours; ++c) curv += st->curv_c[c];
    const int k = st->k;
    if (curv <= 0.0) {
        // not SPD along p: return z at k = 0 and x otherwise (newton_krylov.py:69-70)
        if (k == 0) {
            for (int64_t n = blk * (int64_t)blockDim.x + threadIdx.x; n < m.n_nodes; n += (int64_t)nblk * blockDim.x) {
                const T2 rn = reinterpret_cast<const T2*>(r)[n];
                reinterpret_cast<T2*>(x)[n] = precond<BJ, T>(d, n, rn);
            }
        }
        const double vals[1] = {0.0};
        double tot[1];
        if (last_block_sum_in<kThreads, 1>(vals, site, tot, blk, nblk) && threadIdx.x == 0) {
            st->curv = curv;
            st->iters = k;
            st->done = DFEA_PCG_NEG_CURV;
        }
        return;
    }
    const double alpha = st->rz / curv;
    const T a = (T)alpha;
    double rr = 0.0, rz = 0.0;
    for (int64_t n = blk * (int64_t)blockDim.x + threadIdx.x; n < m.n_nodes; n += (int64_t)nblk * blockDim.x) {
        const T2 pn = load_fresh(reinterpret_cast<const T2*>(p) + n);
        T2 yn;
        if constexpr (GATHER) {
            const int fix = m.node_fix[n];
            const T2 f = node_sum<T>(inc_ptr, inc, reinterpret_cast<const T2*>(fe), n);
            yn = make_v2<T>((fix & 1) ? pn.x : f.x, (fix & 2) ? pn.y : f.y);
        } else {
            yn = load_fresh(reinterpret_cast<const T2*>(y) + n);
        }
        T2 xn = reinterpret_cast<const T2*>(x)[n];
        T2 rn = reinterpret_cast<const T2*>(r)[n];
        xn.x += a * pn.x;
        xn.y += a * pn.y;
        rn.x -= a * yn.x;
        rn.y -= a * yn.y;
        reinterpret_cast<T2*>(x)[n] = xn;
        reinterpret_cast<T2*>(r)[n] = rn;
        rr += (double)rn.x * rn.x + (double)rn.y * rn.y;
        const T2 zn = precond<BJ, T>(d, n, rn);
        rz += (double)rn.x * zn.x + (double)rn.y * zn.y;
    }
    const double vals[2] = {block_sum<kThreads>(rr), block_sum<kThreads>(rz)};
    double tot[2];
    if (last_block_sum_in<kThreads, 2>(vals, site, tot, blk, nblk) && threadIdx.x == 0) {
        st->rr = tot[0];
        st->rz_new = tot[1];
        st->curv = curv;
    }
}

template <typename T, bool GATHER, bool BJ>
__global__ void __launch_bounds__(kThreads)
k_pcg_update1(Mesh m, int n_colours, const T* p, const T* y, const T* __restrict__ d,
              T* __restrict__ x, T* __restrict__ r, PcgState* st, RedSite site, const int32_t* __restrict__ inc_ptr,
              const int32_t* __restrict__ inc, const T* fe) {
    grid_dependency_wait();  // launched with PDL: everything below reads the predecessors' results
    grid_dependents_launch();
    pcg_update1_body<T, GATHER, BJ>(m, n_colours, p, y, d, x, r, st, site, inc_ptr, inc, fe, blockIdx.x, gridDim.x);
}

// PIVOT: write Ap := (1 - m) p, the identity rows the colour passes then add to (the colour form).
template <typename T, bool PIVOT, bool BJ>
__device__ __forceinline__ void pcg_update2_body(const Mesh& m, const T* r, const T* __restrict__ d,
                                                 T* __restrict__ p, T* __restrict__ y, PcgState* st,
                                                 const RedSite& site, int64_t blk, int64_t nblk) {
    using T2 = v2_t<T>;
    if (st->done) return;
    const int k = st->k;
    if (sqrt(st->rr) <= st->rtol * st->norm_b) {
        // converged: ||r|| <= rtol ||b||  (newton_krylov.py:77-79)
        const double vals[1] = {0.0};
        double tot[1];
        if (last_block_sum_in<kThreads, 1>(vals, site, tot, blk, nblk) && threadIdx.x == 0) {
            st->iters = k + 1;
            st->done = DFEA_PCG_CONVERGED;
        }
        return;
    }
    const double beta = st->rz_new / st->rz;
    const T bt = (T)beta;
    double pf = 0.0;
    for (int64_t n = blk * (int64_t)blockDim.x + threadIdx.x; n < m.n_nodes; n += (int64_t)nblk * blockDim.x) {
        const int fix = m.node_fix[n];
        const T2 rn = load_fresh(reinterpret_cast<const T2*>(r) + n);
        const T2 zn = precond<BJ, T>(d, n, rn);
        T2 pn = reinterpret_cast<const T2*>(p)[n];
        pn.x = zn.x + bt * pn.x;
        pn.y = zn.y + bt * pn.y;
        reinterpret_cast<T2*>(p)[n] = pn;
        if (PIVOT) reinterpret_cast<T2*>(y)[n] = make_v2<T>((fix & 1) ? pn.x : T(0), (fix & 2) ? pn.y : T(0));
        if (fix & 1) pf += (double)pn.x * pn.x;
        if (fix & 2) pf += (double)pn.y * pn.y;
    }
    const double vals[1] = {block_sum<kThreads>(pf)};
    double tot[1];
    if (last_block_sum_in<kThreads, 1>(vals, site, tot, blk, nblk) && threadIdx.x == 0) {
        st->rz = st->rz_new;
        st->pfix = tot[0];
        st->k = k + 1;
        if (k + 1 >= st->max_iter) {
            st->iters = st->max_iter;
            st->done = DFEA_PCG_MAX_ITER;
        }
    }
}

template <typename T, bool PIVOT, bool BJ>
__global__ void __launch_bounds__(kThreads)
k_pcg_update2(Mesh m, const T* r, const T* __restrict__ d, T* __restrict__ p, T* __restrict__ y,
              PcgState* st, RedSite site) {
    grid_dependency_wait();
    grid_dependents_launch();
    pcg_update2_body<T, PIVOT, BJ>(m, r, d, p, y, st, site, blockIdx.x, gridDim.x);
}

// ------------------------------------------------------------------------------------------------
// Fused gather form: 2 kernels per iteration.  The direction update p_k = M^-1 r_k + beta_{k-1} p_{k-1}
// moves out of the second vector kernel: the element pass computes p_k at the nodes it gathers, and the
// node pass computes it again (same expression, same bits) and stores it.  The node pass also sums the
// element results (Ap), updates x and r, reduces |r|^2 and r.z, and its last block does the scalar step
// (convergence test, beta, k).  The identity rows' part of p.Ap (fixed DOFs) is added by the element
// pass, counted once per node by the node's first incidence slot.
// ------------------------------------------------------------------------------------------------
template <bool BJ, typename T>
__device__ __forceinline__ v2_t<T> next_direction(const T* __restrict__ d, int64_t n, v2_t<T> r, v2_t<T> p, T beta) {
    const v2_t<T> z = precond<BJ, T>(d, n, r);
    return make_v2<T>(z.x + beta * p.x, z.y + beta * p.y);
}

template <typename T, bool BJ, int NEN>
__device__ __forceinline__ void fused_scatter(int64_t e, int64_t S, const int (&node)[NEN], const int (&fix)[NEN],
                                              const T (&fx)[NEN], const T (&fy)[NEN], v2_t<T>* __restrict__ fe2,
                                              const int32_t* __restrict__ inc_ptr, const int32_t* __restrict__ inc,
                                              const T* __restrict__ d, const v2_t<T>* r2,
                                              const v2_t<T>* p2, T beta, double& pfix) {
#pragma unroll
    for (int a = 0; a < NEN; ++a) fe2[(int64_t)a * S + e] = make_v2<T>(fx[a], fy[a]);
#pragma unroll
    for (int a = 0; a < NEN; ++a) {
        if (fix[a] && inc[inc_ptr[node[a]]] == (int32_t)((int64_t)a * S + e)) {
            const v2_t<T> pn = next_direction<BJ, T>(d, node[a], load_fresh(r2 + node[a]), load_fresh(p2 + node[a]), beta);
            if (fix[a] & 1) pfix += (double)pn.x * pn.x;
            if (fix[a] & 2) pfix += (double)pn.y * pn.y;
        }
    }
}

template <int NEN, int NQ, typename SD, typename T, bool BJ>
__global__ void __launch_bounds__(128)
k_pcg_elem_fused(Mesh m, const SD* __restrict__ C, const SD* __restrict__ G, const T* r,
                 const T* __restrict__ d, const T* p, T* __restrict__ fe, const int32_t* __restrict__ inc_ptr,
                 const int32_t* __restrict__ inc, PcgState* st, RedSite site) {
    using T2 = v2_t<T>;
    extern __shared__ __align__(16) unsigned char smem[];
    const T2* r2 = reinterpret_cast<const T2*>(r);
    const T2* p2 = reinterpret_cast<const T2*>(p);
    T2* fe2 = reinterpret_cast<T2*>(fe);
    double curv = 0.0, pfix = 0.0;
    T beta = T(0);
    const bool ran = apply_tiles<NEN, NQ, SD, T, true>(
        m, 0, m.n_el, C, G, smem, curv,
        [&]() -> bool {
            grid_dependency_wait();
            if (st->done) return false;
            beta = (T)st->beta;
            grid_dependents_launch();
            return true;
        },
        [&](int n) { return next_direction<BJ, T>(d, n, load_fresh(r2 + n), load_fresh(p2 + n), beta); },
        [&](int64_t e, const int (&node)[NEN], const int (&fix)[NEN], const T (&fx)[NEN], const T (&fy)[NEN]) {
            fused_scatter<T, BJ, NEN>(e, m.stride, node, fix, fx, fy, fe2, inc_ptr, inc, d, r2, p2, beta, pfix);
        });
    if (!ran) return;
    const double vals[1] = {block_sum<128>(curv + pfix)};
    double tot[1];
    if (last_block_sum<128, 1>(vals, site, tot) && threadIdx.x == 0) site.result[0] = tot[0];
}

template <int NEN, int NQ, typename SD, typename T, bool BJ>
__global__ void __launch_bounds__(FrameCfg<NEN, NQ>::NT, FrameCfg<NEN, NQ>::MINB)
k_pcg_elem_fused_ref(Mesh m, const SD* __restrict__ C, const RefGrad<NEN, NQ> rg, const T* r,
                     const T* __restrict__ d, const T* p, T* __restrict__ fe,
                     const int32_t* __restrict__ inc_ptr, const int32_t* __restrict__ inc, PcgState* st, RedSite site) {
    using T2 = v2_t<T>;
    constexpr int NT = FrameCfg<NEN, NQ>::NT;
    __shared__ FrameShared<NEN, NQ, T> sh;
    const T2* r2 = reinterpret_cast<const T2*>(r);
    const T2* p2 = reinterpret_cast<const T2*>(p);
    T2* fe2 = reinterpret_cast<T2*>(fe);
    double curv = 0.0, pfix = 0.0;
    T beta = T(0);
    const bool ran = frame_product<NEN, NQ, SD, T, true>(
        m, C, rg, sh, curv,
        [&]() -> bool {
            grid_dependency_wait();
            if (st->done) return false;
            beta = (T)st->beta;
            grid_dependents_launch();
            return true;
        },
        [&](int n) { return next_direction<BJ, T>(d, n, load_fresh(r2 + n), load_fresh(p2 + n), beta); },
        [&](int a, int64_t e, T2 f) {
            const int64_t slot = (int64_t)a * m.stride + e;
            fe2[slot] = f;
            const int c = __ldg(m.conn + slot);
            if ((c & 3) && inc[inc_ptr[c >> 2]] == (int32_t)slot) {  // a fixed DOF, counted by its first slot
                const T2 pn = next_direction<BJ, T>(d, c >> 2, load_fresh(r2 + (c >> 2)), load_fresh(p2 + (c >> 2)), beta);
                if (c & 1) pfix += (double)pn.x * pn.x;
                if (c & 2) pfix += (double)pn.y * pn.y;
            }
        },
        blockIdx.x, gridDim.x);
    if (!ran) return;
    const double vals[1] = {block_sum<NT>(curv + pfix)};
    double tot[1];
    if (last_block_sum<NT, 1>(vals, site, tot) && threadIdx.x == 0) site.result[0] = tot[0];
}

template <typename T, bool BJ>
__global__ void __launch_bounds__(kThreads)
k_pcg_node_fused(Mesh m, const int32_t* __restrict__ inc_ptr, const int32_t* __restrict__ inc, const T* fe,
                 const T* __restrict__ d, T* __restrict__ x, T* __restrict__ r, T* __restrict__ p, PcgState* st,
                 RedSite site) {
    using T2 = v2_t<T>;
    grid_dependency_wait();
    grid_dependents_launch();
    if (st->done) return;
    const double curv = st->curv_c[0];
    const int k = st->k;
    if (curv <= 0.0) {
        // not SPD along p: return z at k = 0 and x otherwise (newton_krylov.py:69-70)
        if (k == 0) {
            for (int64_t n = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; n < m.n_nodes; n += (int64_t)gridDim.x * blockDim.x)
                reinterpret_cast<T2*>(x)[n] = precond<BJ, T>(d, n, reinterpret_cast<const T2*>(r)[n]);
        }
        const double vals[1] = {0.0};
        double tot[1];
        if (last_block_sum<kThreads, 1>(vals, site, tot) && threadIdx.x == 0) {
            st->curv = curv;
            st->iters = k;
            st->done = DFEA_PCG_NEG_CURV;
        }
        return;
    }
    const T a = (T)(st->rz / curv);
    const T beta = (T)st->beta;
    const T2* fe2 = reinterpret_cast<const T2*>(fe);
    double rr = 0.0, rz = 0.0;
    for (int64_t n = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; n < m.n_nodes; n += (int64_t)gridDim.x * blockDim.x) {
        const int fix = m.node_fix[n];
        T2 rn = reinterpret_cast<const T2*>(r)[n];
        const T2 pn = next_direction<BJ, T>(d, n, rn, reinterpret_cast<const T2*>(p)[n], beta);
        reinterpret_cast<T2*>(p)[n] = pn;
        const T2 f = node_sum<T>(inc_ptr, inc, fe2, n);
        const T2 yn = make_v2<T>((fix & 1) ? pn.x : f.x, (fix & 2) ? pn.y : f.y);
        T2 xn = reinterpret_cast<const T2*>(x)[n];
        xn.x += a * pn.x;
        xn.y += a * pn.y;
        rn.x -= a * yn.x;
        rn.y -= a * yn.y;
        reinterpret_cast<T2*>(x)[n] = xn;
        reinterpret_cast<T2*>(r)[n] = rn;
        const T2 zn = precond<BJ, T>(d, n, rn);
        rr += (double)rn.x * rn.x + (double)rn.y * rn.y;
        rz += (double)rn.x * zn.x + (double)rn.y * zn.y;
    }
    const double vals[2] = {block_sum<kThreads>(rr), block_sum<kThreads>(rz)};
    double tot[2];
    if (last_block_sum<kThreads, 2>(vals, site, tot) && threadIdx.x == 0) {
        st->rr = tot[0];
        st->curv = curv;
        if (sqrt(tot[0]) <= st->rtol * st->norm_b) {  // newton_krylov.py:77-79
            st->iters = k + 1;
            st->done = DFEA_PCG_CONVERGED;
        } else {
            st->beta = tot[1] / st->rz;
            st->rz = tot[1];
            st->k = k + 1;
            if (k + 1 >= st->max_iter) {
                st->iters = st->max_iter;
                st->done = DFEA_PCG_MAX_ITER;
            }
        }
    }
}

// ------------------------------------------------------------------------------------------------
// Cluster form: a whole solve in one launch of one thread-block cluster (at most 16 blocks).
//
// Small meshes are bound by the latency of an iteration, not by bytes: the launch forms pay two launches, their tails
// and a dozen trips to L2 (14 - 17 us an iteration from 64 to 16k Q4 elements).  Here the nodes are divided over the
// cluster's blocks and every vector lives in the shared memory of the node's owner: the element pass gathers z and p
// from, and scatters its results to, distributed shared memory (each (element, node) slot has its own place in the
// owner's memory, summed there in incidence order), and the two reductions of an iteration ride on the cluster's
// hardware barriers -- each warp stores its sum into every block's table before the barrier, every warp adds the table
// in the same order after it, so all blocks take the same branch.  Only the moduli stream from L2.
// Microseconds an iteration, FP64, B200 (fused launch form -> this): 64 Q4 14.0 -> 3.0, 576 15.4 -> 3.7, 2,304
// 15.5 -> 5.1, 10,000 16.2 -> 7.9, 16,384 15.6 -> 10.1; 1,800 Q9 15.5 -> 7.7, 5,000 17.1 -> 10.9; 4,800 Tri6
// 16.8 -> 8.9; 20,000 Tri3 17.6 -> 7.9.  So wherever the vectors fit the cluster's shared memory it is the faster form,
// and it is taken there.  Past ~5k Q4 elements the element pass on 16 SMs (its FP64 chains) bounds it, below that the
// two exchanges.  (A grid-wide persistent form, exchanging through L2 with polled
// flags, took 7.7 us an iteration on one block and 13 - 18 us on many: its fences also empty L1.)
//
// There is no spin wait: the blocks of a cluster are scheduled together and meet at hardware barriers.  The number of
// iterations is bounded by max_iter.
// ------------------------------------------------------------------------------------------------
// Shared memory of a block (byte offsets; the same in every block).  Nodes are divided in ranges of nb.
struct ClusterLayout {
    int nb;                                         // nodes per block
    int x, r, p, z, d, fe, base, fix, el, table, total;  // d: 1 / diagonal, or the inverse 2 x 2 blocks (4 values)
    int slices;  // of 32 nodes; base[s] = first fe entry of slice s, node i's j-th entry at base[i / 32] + 32 j + i % 32
};


// Elements of a cluster's block: of every colour its share, in order -- so that with elements and nodes both numbered
// along the mesh a block's elements lie at its own nodes and most of its gathers stay in its own shared memory.
struct ClusterColours {
    int n;
    int begin[DFEA_MAX_COLOURS + 1];
    __host__ __device__ int lo(int c, int rank, int size) const {
        return begin[c] + (int)((int64_t)(begin[c + 1] - begin[c]) * rank / size);
    }
};

// The element pass of a block, two ways.  SPLIT: teams of NQ warps on tiles of 32 elements, a warp per Gauss point, sums
// through shared memory -- the shorter chain, while a block's elements are about one round of its teams.  Else one
// thread per element, its Gauss points independent chains and the reference gradients constants of the unrolled loop:
// no barriers, so more elements per block cost less.  Microseconds an iteration, FP64 (split / per element): 64 Q4
// 3.0 / 4.1, 576 3.7 / 5.6, 2,304 5.1 / 5.7, 10,000 9.1 / 7.9, 16,384 12.3 / 10.1; 576 Q9 6.1 / 7.9, 1,800 10.1 / 7.7.
template <int NEN, int NQ, bool SPLIT>
struct ClusterCfg {
    static constexpr int TEAMS = NQ == 9 ? 2 : (NQ == 6 ? 3 : 4);
    static constexpr int TEAM = 32 * NQ;
    static constexpr int NT = SPLIT ? TEAM * TEAMS : (NEN <= 4 ? 640 : (NEN == 6 ? 512 : 384));  // 96 - 168 registers
    static constexpr int W = NT / 32;
    static constexpr int TEAM_BYTES = SPLIT ? TEAMS * (int)sizeof(FrameShared<NEN, NQ, double>) : 0;
};

// SPLIT up to a round and a quarter of 16 blocks' teams
template <int NEN, int NQ>
bool cluster_split(int64_t n_el) {
    return NQ > 1 && n_el <= (int64_t)kClusterMax * ClusterCfg<NEN, NQ, true>::TEAMS * 32 * 5 / 4;
}

// Element results of a node lie 32 entries apart, those of neighbouring nodes side by side (slices of 32 nodes, each as
// deep as its busiest node): stored node by node, the element pass scattered with 8-way bank conflicts.
// One block per rank: base[rank][s] of its slices (entries), base[rank][slices] = their total.
__global__ void k_pcg_cluster_slices(int64_t n_nodes, int nb, int slices, const int32_t* __restrict__ inc_ptr,
                                     int32_t* __restrict__ base) {
    const int64_t first = (int64_t)blockIdx.x * nb;
    int32_t* mine = base + (int64_t)blockIdx.x * (slices + 1);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
    for (int s = warp; s < slices; s += warps) {
        const int i = s * 32 + lane;
        const int64_t n = first + i;
        int deg = (i < nb && n < n_nodes) ? inc_ptr[n + 1] - inc_ptr[n] : 0;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) deg = max(deg, __shfl_xor_sync(0xffffffffu, deg, o));
        if (lane == 0) mine[s] = 32 * deg;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        int32_t at = 0;
        for (int s = 0; s < slices; ++s) {
            const int32_t n = mine[s];
            mine[s] = at;
            at += n;
        }
        mine[slices] = at;
    }
}

// map[slot] = (rank << 18 | local << 2 | fix bits, rank << 18 | entry in the owner's fe) of every (a, e) slot
__global__ void __launch_bounds__(kThreads)
k_pcg_cluster_map(Mesh m, int nb, int slices, const int32_t* __restrict__ base, const int32_t* __restrict__ inc_ptr,
                  const int32_t* __restrict__ inc, int2* __restrict__ map) {
    for (int64_t n = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; n < m.n_nodes; n += (int64_t)gridDim.x * blockDim.x) {
        const int rank = (int)(n / nb), i = (int)(n - (int64_t)rank * nb), fix = m.node_fix[n];
        int at = base[(int64_t)rank * (slices + 1) + i / 32] + i % 32;
        for (int j = inc_ptr[n]; j < inc_ptr[n + 1]; ++j, at += 32)
            map[inc[j]] = make_int2(rank << 18 | i << 2 | fix, rank << 18 | at);
    }
}

template <int NEN, int NQ, typename SD, bool BJ, bool SPLIT>
__global__ void __launch_bounds__(ClusterCfg<NEN, NQ, SPLIT>::NT, 1)
k_pcg_cluster(Mesh m, const SD* __restrict__ C, const RefGrad<NEN, NQ> rg, const int2* __restrict__ map,
              const double* __restrict__ b, const double* __restrict__ diag, double* __restrict__ x_out,
              const int32_t* __restrict__ slice_base, PcgState* __restrict__ st, ClusterLayout L, ClusterColours colours,
              double rtol, int max_iter) {
    using Cfg = ClusterCfg<NEN, NQ, SPLIT>;
    constexpr int NT = Cfg::NT, W = Cfg::W;
    extern __shared__ __align__(16) unsigned char cluster_smem[];
    double2* xs = reinterpret_cast<double2*>(cluster_smem + L.x);
    double2* rs = reinterpret_cast<double2*>(cluster_smem + L.r);
    double2* ps = reinterpret_cast<double2*>(cluster_smem + L.p);
    double2* zs = reinterpret_cast<double2*>(cluster_smem + L.z);
    double* ds = reinterpret_cast<double*>(cluster_smem + L.d);
    double2* fes = reinterpret_cast<double2*>(cluster_smem + L.fe);
    int* base = reinterpret_cast<int*>(cluster_smem + L.base);
    unsigned char* fixs = cluster_smem + L.fix;
    int* els = reinterpret_cast<int*>(cluster_smem + L.el);
    double* table = reinterpret_cast<double*>(cluster_smem + L.table);  // [2][2][kClusterMax * W]
    const unsigned smem0 = (unsigned)__cvta_generic_to_shared(cluster_smem);
    const unsigned rank = cluster_rank();
    const int size = gridDim.x;  // the grid is the cluster
    const int lane32 = threadIdx.x & 31;
    ClusterExchange<W> sums(table, rank, size);

    const int64_t node0 = (int64_t)rank * L.nb;
    const int n_own = (int)(node0 >= m.n_nodes ? 0 : (m.n_nodes - node0 < L.nb ? m.n_nodes - node0 : L.nb));
    double rz = 0.0, bb = 0.0;
    for (int i = threadIdx.x; i < n_own; i += NT) {
        const int64_t n = node0 + i;
        const double2 bn = reinterpret_cast<const double2*>(b)[n];
        const double2 zn = precond<BJ, double>(diag, n, bn);
        if constexpr (BJ) {
            reinterpret_cast<double2*>(ds)[2 * i] = reinterpret_cast<const double2*>(diag)[2 * n];
            reinterpret_cast<double2*>(ds)[2 * i + 1] = reinterpret_cast<const double2*>(diag)[2 * n + 1];
        } else {
            const double2 dn = reinterpret_cast<const double2*>(diag)[n];
            reinterpret_cast<double2*>(ds)[i] = make_double2(1.0 / dn.x, 1.0 / dn.y);
        }
        xs[i] = make_double2(0.0, 0.0);
        rs[i] = bn;
        zs[i] = zn;
        ps[i] = make_double2(0.0, 0.0);
        fixs[i] = m.node_fix[n];
        rz += bn.x * zn.x + bn.y * zn.y;
        bb += bn.x * bn.x + bn.y * bn.y;
    }
    const int32_t* my_base = slice_base + (int64_t)rank * (L.slices + 1);
    for (int i = threadIdx.x; i <= L.slices; i += NT) base[i] = my_base[i];
    for (int i = threadIdx.x; i < my_base[L.slices]; i += NT) fes[i] = make_double2(0.0, 0.0);  // unused entries stay zero
    int n_els = 0;
    for (int c = 0; c < colours.n; ++c) {
        const int lo = colours.lo(c, rank, size), hi = colours.lo(c, rank + 1, size);
        for (int i = lo + threadIdx.x; i < hi; i += NT) els[n_els + i - lo] = i;
        n_els += hi - lo;
    }
    int status = DFEA_PCG_RUNNING, iters = 0;
    double rr = 0.0, curv = 0.0, beta = 0.0;
    cluster_barrier();  // every block has started: its shared memory may be written from here on
    sums.two(rz, bb, rz, bb);
    const double norm_b = sqrt(bb);
    if (norm_b == 0.0) status = DFEA_PCG_ZERO_RHS;

    // z and p at a node, from its owner
    auto fetch = [&](int word, double2& zn, double2& pn) {
        const unsigned who = (unsigned)word >> 18;
        const int at = (word & 0x3ffff) >> 2;
        if (who == rank) {
            zn = zs[at];
            pn = ps[at];
        } else {
            zn = cluster_load(cluster_address(smem0 + L.z + at * 16, who));
            pn = cluster_load(cluster_address(smem0 + L.p + at * 16, who));
        }
    };
    auto put = [&](int word, double2 f) {
        const unsigned who = (unsigned)word >> 18;
        const int at = word & 0x3ffff;
        if (who == rank) fes[at] = f;
        else cluster_store(cluster_address(smem0 + L.fe + at * 16, who), f);
    };
    // Slots and moduli of the first tile (or element) stay in flight around the end of the pass: they do not change from
    // iteration to iteration.
    constexpr bool KEEP = NEN <= 4;  // per element: the slots too, where registers allow
    constexpr int NS = SPLIT ? 1 : NEN;
    const int team = threadIdx.x / Cfg::TEAM, q = (threadIdx.x % Cfg::TEAM) / 32;       // SPLIT
    const int i_first = SPLIT ? team * 32 + lane32 : threadIdx.x;
    constexpr int step = SPLIT ? Cfg::TEAMS * 32 : NT;
    FrameModuli<SD> M;
    int2 s[NS], s_next = make_int2(-1, -1);
    auto element = [&](int i) -> int { return i < n_els ? els[i] : -1; };
    auto load_slot = [&](int a, int e) { return e >= 0 ? __ldg(map + (int64_t)a * m.stride + e) : make_int2(-1, -1); };
    auto load_first = [&]() {
        const int e = element(i_first);
        if constexpr (SPLIT) {
            s[0] = load_slot(q < NEN ? q : 0, q < NEN ? e : -1);
            s_next = load_slot(q < NEN ? q : 0, q < NEN ? element(i_first + step) : -1);
            if (e >= 0) M.template load<true>(C, m.stride, q, e);
            else M.clear();
        } else if (e >= 0) {
            if (KEEP) {
#pragma unroll
                for (int a = 0; a < NS; ++a) s[a] = load_slot(a, e);
            }
            M.template load<true>(C, m.stride, 0, e);
        }
    };
    load_first();

    for (int k = 0; status == DFEA_PCG_RUNNING; ++k) {
        double c = 0.0;
        if constexpr (SPLIT) {
            FrameShared<NEN, NQ, double>& sh = reinterpret_cast<FrameShared<NEN, NQ, double>*>(cluster_smem)[team];
            const RefRow<NEN, double> row(rg, q);
            auto team_sync = [&]() { asm volatile("bar.sync %0, %1;" ::"r"(team + 1), "n"(Cfg::TEAM) : "memory"); };
            // z and p of the next tile's nodes; combined when they go to shared memory, a tile later
            double2 zn = make_double2(0.0, 0.0), pn = zn;
            if (s[0].x >= 0) fetch(s[0].x, zn, pn);
            for (int tile = team * 32; tile < n_els; tile += step) {
                if (q < NEN)
                    sh.vs[q][lane32] = make_double2((s[0].x & 1) ? 0.0 : zn.x + beta * pn.x, (s[0].x & 2) ? 0.0 : zn.y + beta * pn.y);
                team_sync();
                const int to = s[0].y;
                const bool more = tile + step < n_els;
                if (more) {
                    s[0] = s_next;
                    zn = pn = make_double2(0.0, 0.0);
                    if (s[0].x >= 0) fetch(s[0].x, zn, pn);
                    s_next = load_slot(q < NEN ? q : 0, q < NEN ? element(tile + lane32 + 2 * step) : -1);
                }
                double G[4], P[4];
                frame_gradient<NEN, NQ, double>(row, lane32, sh.vs, G);
                M.apply(G, P);
                c += G[0] * P[0] + G[1] * P[1] + G[2] * P[2] + G[3] * P[3];
                if (more) {
                    const int e = element(tile + lane32 + step);
                    if (e >= 0) M.template load<true>(C, m.stride, q, e);
                    else M.clear();
                }
#pragma unroll
                for (int a = 0; a < NEN; ++a)
                    sh.red[q][a][lane32] = make_double2(P[0] * row.g[a][0] + P[1] * row.g[a][1], P[2] * row.g[a][0] + P[3] * row.g[a][1]);
                team_sync();
                if (q < NEN && to >= 0) {
                    double2 f = sh.red[0][q][lane32];
#pragma unroll
                    for (int g = 1; g < NQ; ++g) {
                        const double2 t = sh.red[g][q][lane32];
                        f.x += t.x;
                        f.y += t.y;
                    }
                    put(to, f);
                }
            }
        } else {
            for (int i = threadIdx.x; i < n_els; i += NT) {
                const int e = els[i];
                if (!KEEP || i >= NT) {
#pragma unroll
                    for (int a = 0; a < NS; ++a) s[a] = load_slot(a, e);
                }
                if (i >= NT) M.template load<true>(C, m.stride, 0, e);
                double2 v[NS], f[NS];
#pragma unroll
                for (int a = 0; a < NS; ++a) {
                    double2 zn, pn;
                    fetch(s[a].x, zn, pn);
                    v[a] = make_double2((s[a].x & 1) ? 0.0 : zn.x + beta * pn.x, (s[a].x & 2) ? 0.0 : zn.y + beta * pn.y);
                    f[a] = make_double2(0.0, 0.0);
                }
#pragma unroll(NQ > 4 ? 1 : NQ)
                for (int g = 0; g < NQ; ++g) {
                    const FrameModuli<SD> now = M;
                    if (g + 1 < NQ) M.template load<true>(C, m.stride, g + 1, e);
                    double G[4] = {0.0, 0.0, 0.0, 0.0}, P[4];
#pragma unroll
                    for (int a = 0; a < NS; ++a) {
                        G[0] += v[a].x * rg.g[g][a][0];
                        G[1] += v[a].x * rg.g[g][a][1];
                        G[2] += v[a].y * rg.g[g][a][0];
                        G[3] += v[a].y * rg.g[g][a][1];
                    }
                    now.apply(G, P);
                    c += G[0] * P[0] + G[1] * P[1] + G[2] * P[2] + G[3] * P[3];
#pragma unroll
                    for (int a = 0; a < NS; ++a) {
                        f[a].x += P[0] * rg.g[g][a][0] + P[1] * rg.g[g][a][1];
                        f[a].y += P[2] * rg.g[g][a][0] + P[3] * rg.g[g][a][1];
                    }
                }
#pragma unroll
                for (int a = 0; a < NS; ++a) put(s[a].y, f[a]);
            }
        }
        load_first();
        for (int i = threadIdx.x; i < n_own; i += NT) {  // the identity rows' part of p.Ap
            const int fix = fixs[i];
            if (fix) {
                const double px = zs[i].x + beta * ps[i].x, py = zs[i].y + beta * ps[i].y;
                if (fix & 1) c += px * px;
                if (fix & 2) c += py * py;
            }
        }
        curv = sums.one(c);
        if (curv <= 0.0) {
            // not SPD along p: return z at k = 0 and x otherwise (newton_krylov.py:69-70)
            if (k == 0)
                for (int i = threadIdx.x; i < n_own; i += NT) xs[i] = zs[i];
            iters = k;
            status = DFEA_PCG_NEG_CURV;
            break;
        }
        const double a = rz / curv;
        double s_rr = 0.0, s_rz = 0.0;
        for (int i = threadIdx.x; i < n_own; i += NT) {
            const int fix = fixs[i];
            const double2 zn = zs[i], po = ps[i];
            const double2 pn = make_double2(zn.x + beta * po.x, zn.y + beta * po.y);
            double2 f = make_double2(0.0, 0.0);
            const int j1 = base[(i >> 5) + 1];
#pragma unroll 4
            for (int j = base[i >> 5] + (i & 31); j < j1; j += 32) {
                const double2 t = fes[j];
                f.x += t.x;
                f.y += t.y;
            }
            const double2 yn = make_double2((fix & 1) ? pn.x : f.x, (fix & 2) ? pn.y : f.y);
            double2 xn = xs[i], rn = rs[i];
            xn.x += a * pn.x;
            xn.y += a * pn.y;
            rn.x -= a * yn.x;
            rn.y -= a * yn.y;
            double2 zw;
            if constexpr (BJ) {
                zw = precond<true, double>(ds, i, rn);
            } else {
                const double2 dn = reinterpret_cast<const double2*>(ds)[i];
                zw = make_double2(rn.x * dn.x, rn.y * dn.y);
            }
            xs[i] = xn;
            rs[i] = rn;
            ps[i] = pn;
            zs[i] = zw;
            s_rr += rn.x * rn.x + rn.y * rn.y;
            s_rz += rn.x * zw.x + rn.y * zw.y;
        }
        double rz_new;
        sums.two(s_rr, s_rz, rr, rz_new);
        beta = rz_new / rz;  // beside the square root: both chains are long
        if (sqrt(rr) <= rtol * norm_b) {  // newton_krylov.py:77-79
            iters = k + 1;
            status = DFEA_PCG_CONVERGED;
        } else {
            rz = rz_new;
            if (k + 1 >= max_iter) {
                iters = max_iter;
                status = DFEA_PCG_MAX_ITER;
            }
        }
    }
    for (int i = threadIdx.x; i < n_own; i += NT) reinterpret_cast<double2*>(x_out)[node0 + i] = xs[i];
    if (rank == 0 && threadIdx.x == 0) {
        st->rr = rr;
        st->rz = rz;
        st->norm_b = norm_b;
        st->curv = curv;
        st->iters = iters;
        st->k = iters;
        st->done = status;
    }
}

__global__ void k_pcg_cond(PcgState* st, cudaGraphConditionalHandle h) {
    if (threadIdx.x != 0) return;
    const int g = ++st->guard;
    if (st->done == DFEA_PCG_RUNNING && g >= st->max_iter + 4) {
        st->iters = st->max_iter;
        st->done = DFEA_PCG_MAX_ITER;
    }
    cudaGraphSetConditional(h, st->done == DFEA_PCG_RUNNING ? 1u : 0u);
}

}  // namespace dfea

using namespace dfea;

struct dfea_pcg {
    dfea_mesh_view mesh;
    const void* moduli;
    const void* diag;
    const void* b;
    void* x;
    int vec_dtype;
    char* work;
    PcgLayout layout{1, 8, 1};
    int use_graph;
    bool gather = false;             // product in the gather form (element pass + node sums in update 1)
    int grid_cap = 0;                // most blocks per launch (0: as many as the GPU holds)
    bool block = false;              // nodal block-Jacobi: diag holds the inverse 2x2 blocks (4N doubles)
    bool fused = false;              // fused gather form: 2 kernels per iteration
    bool clustered = false;          // the whole solve in one launch of a thread-block cluster
    int cluster_blocks = 0;
    ClusterLayout cluster{};
    // the cluster form's arrays, in room that the launch forms use for fe and the vectors
    int2* slot_map() const { return reinterpret_cast<int2*>(work + layout.off_fe); }
    int32_t* slice_base() const { return reinterpret_cast<int32_t*>(work + layout.off_r); }
    cudaStream_t capture_stream = nullptr;
    cudaGraph_t graph = nullptr;
    cudaGraphExec_t exec = nullptr;
    // [done, iters, bodies]: read after the stream has reached the copy, staged through the library's pool of
    // page-locked blocks (a page-locked allocation per handle cost a device-wide driver call per solve set up).
    int32_t status_buf[4] = {0, 0, 0, 0};
    int32_t* host_status = status_buf;

    PcgState* state() const { return reinterpret_cast<PcgState*>(work + layout.off_state); }
    RedSite site(int i, int k_slot_results) const {
        double* parts = reinterpret_cast<double*>(work + layout.off_part) + (int64_t)i * 3 * kMaxBlocks;
        PcgState* st = state();
        (void)k_slot_results;
        double* res = nullptr;
        if (i < mesh.n_colours) res = st->curv_c + i;          // colour curvature
        else if (i == mesh.n_colours) res = &st->rr;            // update 1: rr, rz_new
        return RedSite{parts, st->tickets + i, res};
    }
};

namespace {

// Kernels of one iteration without the loop condition: the non-empty colour passes and two updates
// (colour form), or the element pass and two updates (gather form).
int kernels_per_iteration(const dfea_pcg& h) {
    if (h.fused) return 2;
    if (h.gather) return 3;
    int nonempty = 0;
    for (int c = 0; c < h.mesh.n_colours; ++c) nonempty += h.mesh.colour_begin[c + 1] > h.mesh.colour_begin[c];
    return nonempty + 2;
}

// S: storage type of moduli and gradients, T: Krylov vector type; REF: DFEA_F32REF moduli (S = float),
// no gradients read.
template <typename S, typename T, bool REF = false, bool BJ = false>
int launch_iteration(const dfea_pcg& h, cudaStream_t s, cudaGraphConditionalHandle cond, bool with_cond) {
    const dfea_mesh_view& mv = h.mesh;
    const Mesh m = kernel_mesh(mv);
    const S* C = static_cast<const S*>(h.moduli);
    const S* G = std::is_same<S, float>::value ? reinterpret_cast<const S*>(mv.grad32) : reinterpret_cast<const S*>(mv.grad);
    T* r = reinterpret_cast<T*>(h.work + h.layout.off_r);
    T* p = reinterpret_cast<T*>(h.work + h.layout.off_p);
    T* y = reinterpret_cast<T*>(h.work + h.layout.off_y);
    const T* d = static_cast<const T*>(h.diag);
    T* x = static_cast<T*>(h.x);
    PcgState* st = h.state();
    // node passes with all the warps an SM holds; the colour form's two updates stream vectors, and keep the four blocks per
    // SM that its sums (and so its iterates, bit for bit) were always divided over
    const int gn = capped(grid_for(mv.n_nodes, kThreads, h.gather ? 8 : 4), h.grid_cap);
    LaunchOpts pdl;
    pdl.pdl = true;
    int rc;
    if (h.fused) {
        T* fe = reinterpret_cast<T*>(h.work + h.layout.off_fe);
        rc = dispatch_element(mv.nen, mv.n_q, [&](auto nen_c, auto nq_c) -> int {
            constexpr int NEN = decltype(nen_c)::value, NQ = decltype(nq_c)::value;
            if constexpr (REF) {
                const int grid = capped(frame_resident_grid<k_pcg_elem_fused_ref<NEN, NQ, S, T, BJ>, NEN, NQ>(mv.n_el),
                                        h.grid_cap);
                return launch_kernel(k_pcg_elem_fused_ref<NEN, NQ, S, T, BJ>, dim3(grid), dim3(FrameCfg<NEN, NQ>::NT), 0,
                                     s, pdl, m, C, ref_grad_of<NEN, NQ>(mv), (const T*)r,
                                     d, (const T*)p, fe, mv.node_elem_ptr, mv.node_elem, st, h.site(0, 1));
            } else {
                using Cfg = ApplyCfg<NEN, S>;
                const int grid = capped(resident_grid<k_pcg_elem_fused<NEN, NQ, S, T, BJ>, Cfg::SMEM, Cfg::NT>(mv.n_el),
                                        h.grid_cap);
                return launch_kernel(k_pcg_elem_fused<NEN, NQ, S, T, BJ>, dim3(grid), dim3(Cfg::NT), Cfg::SMEM, s, pdl,
                                     m, C, G, (const T*)r, d, (const T*)p, fe, mv.node_elem_ptr, mv.node_elem, st,
                                     h.site(0, 1));
            }
        });
        if (rc) return rc;
        if ((rc = launch_kernel(k_pcg_node_fused<T, BJ>, dim3(gn), dim3(kThreads), 0, s, pdl, m, mv.node_elem_ptr,
                                mv.node_elem, (const T*)fe, d, x, r, p, st, h.site(mv.n_colours, 2))))
            return rc;
    } else if (h.gather) {
        // element pass (curvature into site 0, read as colour 0), node sums fused into update 1
        T* fe = reinterpret_cast<T*>(h.work + h.layout.off_fe);
        rc = dispatch_element(mv.nen, mv.n_q, [&](auto nen_c, auto nq_c) -> int {
            constexpr int NEN = decltype(nen_c)::value, NQ = decltype(nq_c)::value;
            if constexpr (REF)
                return launch_apply_ref_elem<NEN, NQ, S, T, true>(mv, C, p, fe, h.site(0, 1),
                                                               &st->done, s, h.grid_cap);
            else
                return launch_apply_elem<NEN, NQ, S, T, true>(mv, C, G, p, fe, h.site(0, 1), &st->done, s, h.grid_cap);
        });
        if (rc) return rc;
        if ((rc = launch_kernel(k_pcg_update1<T, true, BJ>, dim3(gn), dim3(kThreads), 0, s, pdl, m, 1, p, (const T*)y, d, x,
                                r, st, h.site(mv.n_colours, 2), mv.node_elem_ptr, mv.node_elem, (const T*)fe)))
            return rc;
        if ((rc = launch_kernel(k_pcg_update2<T, false, BJ>, dim3(gn), dim3(kThreads), 0, s, pdl, m, (const T*)r, d, p, y,
                                st, h.site(mv.n_colours + 1, 1))))
            return rc;
    } else {
        RedSite sites[DFEA_MAX_COLOURS];
        for (int c = 0; c < mv.n_colours; ++c) sites[c] = h.site(c, 1);
        rc = dispatch_element(mv.nen, mv.n_q, [&](auto nen_c, auto nq_c) -> int {
            constexpr int NEN = decltype(nen_c)::value, NQ = decltype(nq_c)::value;
            if constexpr (REF && std::is_same<S, double>::value)
                return set_error(DFEA_ERR_UNSUPPORTED, "DFEA_F64REF moduli run in the gather forms");  // checked at create
            else if constexpr (REF)
                return launch_apply_ref_colours<NEN, NQ, T, true>(mv, reinterpret_cast<const float*>(C), p, y, sites,
                                                                  &st->done, s, h.grid_cap);
            else
                return launch_apply_colours<NEN, NQ, S, T, true>(mv, C, G, p, y, sites, &st->done, s, false,
                                                                 h.grid_cap);
        });
        if (rc) return rc;
        if ((rc = launch_kernel(k_pcg_update1<T, false, BJ>, dim3(gn), dim3(kThreads), 0, s, pdl, m, mv.n_colours, p,
                                (const T*)y, d, x, r, st, h.site(mv.n_colours, 2), (const int32_t*)nullptr,
                                (const int32_t*)nullptr, (const T*)nullptr)))
            return rc;
        if ((rc = launch_kernel(k_pcg_update2<T, true, BJ>, dim3(gn), dim3(kThreads), 0, s, pdl, m, (const T*)r, d, p, y,
                                st, h.site(mv.n_colours + 1, 1))))
            return rc;
    }
    if (with_cond) k_pcg_cond<<<1, 32, 0, s>>>(st, cond);
    else note_launches(kernels_per_iteration(h));  // graph-captured kernels are counted when the solve returns
    return launch_check("pcg iteration");
}

int launch_iteration_any(const dfea_pcg& h, cudaStream_t s, cudaGraphConditionalHandle cond, bool with_cond) {
    if (h.block) {  // block-Jacobi: double vectors only (checked at create)
        if (h.vec_dtype == DFEA_F64) return launch_iteration<double, double, false, true>(h, s, cond, with_cond);
        if (h.vec_dtype == DFEA_MIXED) return launch_iteration<float, double, false, true>(h, s, cond, with_cond);
        if (h.vec_dtype == DFEA_F64REF) return launch_iteration<double, double, true, true>(h, s, cond, with_cond);
        return launch_iteration<float, double, true, true>(h, s, cond, with_cond);
    }
    if (h.vec_dtype == DFEA_F64) return launch_iteration<double, double>(h, s, cond, with_cond);
    if (h.vec_dtype == DFEA_MIXED) return launch_iteration<float, double>(h, s, cond, with_cond);
    if (h.vec_dtype == DFEA_F32REF) return launch_iteration<float, double, true>(h, s, cond, with_cond);
    if (h.vec_dtype == DFEA_F64REF) return launch_iteration<double, double, true>(h, s, cond, with_cond);
    return launch_iteration<float, float>(h, s, cond, with_cond);
}

constexpr int kClusterSmem = 220 * 1024;  // dynamic shared memory a block may take (of 227 KB)

// The cluster of a mesh: blocks (a power of two, at most `most`) and shared memory, or 0 blocks where
// the mesh does not fit.  max_slots(blocks, nb, slices): the most fe entries of a block's node range.
template <int NEN, int NQ, bool SPLIT, typename MaxSlots>
int cluster_layout(const dfea_mesh_view& mv, bool block_jacobi, int most, ClusterLayout* out, MaxSlots&& max_slots) {
    using Cfg = ClusterCfg<NEN, NQ, SPLIT>;
    if (most < 1) return 0;
    int blocks = 1;
    while (2 * blocks <= most && (int64_t)blocks * Cfg::TEAMS * 32 < mv.n_el) blocks *= 2;
    const int64_t nb = (mv.n_nodes + blocks - 1) / blocks;
    if (nb >= (1 << 16) || 96 * nb > kClusterSmem) return 0;  // five vectors and an entry per node at the least
    const int slices = (int)((nb + 31) / 32);
    const int64_t slots = max_slots(blocks, nb, slices);
    if (slots >= (1 << 18)) return 0;
    int64_t at = (Cfg::TEAM_BYTES + 15) / 16 * 16;
    auto take = [&](int64_t bytes) {
        const int64_t o = at;
        at += (bytes + 15) / 16 * 16;
        return (int)(o < (int64_t(1) << 30) ? o : (int64_t(1) << 30));
    };
    ClusterLayout L;
    L.nb = (int)nb;
    L.x = take(16 * nb);
    L.r = take(16 * nb);
    L.p = take(16 * nb);
    L.z = take(16 * nb);
    L.d = take((block_jacobi ? 32 : 16) * nb);
    L.fe = take(16 * slots);
    L.base = take(4 * (slices + 1));
    L.slices = slices;
    L.fix = take(nb);
    L.el = take(4 * (mv.n_el / blocks + mv.n_colours + 1));
    L.table = take(2 * 2 * kClusterMax * Cfg::W * 8);
    if (at > kClusterSmem) return 0;
    L.total = (int)at;
    *out = L;
    return blocks;
}

template <typename SD, bool BJ>
int launch_cluster(const dfea_pcg& h, cudaStream_t s, double rtol, int max_iter) {
    const dfea_mesh_view& mv = h.mesh;
    const Mesh m = kernel_mesh(mv);
    PcgState* st = h.state();
    ClusterColours colours;
    colours.n = mv.n_colours;
    for (int c = 0; c <= mv.n_colours; ++c) colours.begin[c] = (int)mv.colour_begin[c];
    k_pcg_reset<<<1, 128, 0, s>>>(st);
    const int rc = dispatch_element(mv.nen, mv.n_q, [&](auto nen_c, auto nq_c) -> int {
        constexpr int NEN = decltype(nen_c)::value, NQ = decltype(nq_c)::value;
        const auto launch = [&](auto split_c) -> int {
            constexpr bool SPLIT = decltype(split_c)::value;
            constexpr auto kernel = k_pcg_cluster<NEN, NQ, SD, BJ, SPLIT>;
            cudaLaunchAttribute attr[1];
            attr[0].id = cudaLaunchAttributeClusterDimension;
            attr[0].val.clusterDim.x = h.cluster_blocks;
            attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
            cudaLaunchConfig_t cfg = {};
            cfg.gridDim = dim3(h.cluster_blocks);
            cfg.blockDim = dim3(ClusterCfg<NEN, NQ, SPLIT>::NT);
            cfg.dynamicSmemBytes = h.cluster.total;
            cfg.stream = s;
            cfg.attrs = attr;
            cfg.numAttrs = 1;
            return check_cuda(cudaLaunchKernelEx(&cfg, kernel, m, static_cast<const SD*>(h.moduli), ref_grad_of<NEN, NQ>(mv),
                                                 (const int2*)h.slot_map(), static_cast<const double*>(h.b),
                                                 static_cast<const double*>(h.diag), static_cast<double*>(h.x),
                                                 (const int32_t*)h.slice_base(), st, h.cluster, colours, rtol, max_iter),
                              "cudaLaunchKernelEx(cluster PCG)");
        };
        if constexpr (NQ > 1)
            if (cluster_split<NEN, NQ>(mv.n_el)) return launch(std::true_type{});
        return launch(std::false_type{});
    });
    if (rc) return rc;
    note_launches(2);
    return launch_check("cluster PCG");
}

int launch_cluster_any(const dfea_pcg& h, cudaStream_t s, double rtol, int max_iter) {
    if (h.vec_dtype == DFEA_F64REF)
        return h.block ? launch_cluster<double, true>(h, s, rtol, max_iter) : launch_cluster<double, false>(h, s, rtol, max_iter);
    return h.block ? launch_cluster<float, true>(h, s, rtol, max_iter) : launch_cluster<float, false>(h, s, rtol, max_iter);
}

// Lay the cluster out (exact entry counts of the node ranges, read once) and write the slot map of the handle.
template <typename SD, bool BJ>
int prepare_cluster(dfea_pcg* h) {
    const dfea_mesh_view& mv = h->mesh;
    cudaStream_t s = cudaStreamPerThread;
    int rc = DFEA_OK;
    h->cluster_blocks = dispatch_element(mv.nen, mv.n_q, [&](auto nen_c, auto nq_c) -> int {
        constexpr int NEN = decltype(nen_c)::value, NQ = decltype(nq_c)::value;
        const auto max_slots = [&](int blocks, int64_t nb, int slices) -> int64_t {
            k_pcg_cluster_slices<<<blocks, 256, 0, s>>>(mv.n_nodes, (int)nb, slices, mv.node_elem_ptr, h->slice_base());
            note_launches(1);
            int32_t total[kClusterMax];
            if ((rc = launch_check("cluster PCG slices")) ||
                (rc = check_cuda(cudaMemcpy2DAsync(total, sizeof(int32_t), h->slice_base() + slices,
                                                   (slices + 1) * sizeof(int32_t), sizeof(int32_t), blocks,
                                                   cudaMemcpyDeviceToHost, s), "cudaMemcpy2DAsync")) ||
                (rc = check_cuda(cudaStreamSynchronize(s), "cudaStreamSynchronize")))
                return 0;
            int64_t most = 0;
            for (int i = 0; i < blocks; ++i) most = total[i] > most ? total[i] : most;
            return most;
        };
        const auto layout = [&](auto split_c) -> int {
            constexpr bool SPLIT = decltype(split_c)::value;
            constexpr auto kernel = k_pcg_cluster<NEN, NQ, SD, BJ, SPLIT>;
            const ClusterRoom& room = cluster_room<kernel>(ClusterCfg<NEN, NQ, SPLIT>::NT);
            if (room.bytes < kClusterSmem) return 0;
            return cluster_layout<NEN, NQ, SPLIT>(mv, BJ, capped(room.blocks, h->grid_cap), &h->cluster, max_slots);
        };
        if constexpr (NQ > 1)
            if (cluster_split<NEN, NQ>(mv.n_el)) return layout(std::true_type{});
        return layout(std::false_type{});
    });
    if (rc) return rc;
    if (h->cluster_blocks == 0)
        return set_error(DFEA_ERR_UNSUPPORTED, "dfea_pcg_create: the mesh does not fit the shared memory of a cluster on this device");
    k_pcg_cluster_map<<<grid_for(mv.n_nodes, kThreads, 8), kThreads, 0, s>>>(
        kernel_mesh(mv), h->cluster.nb, h->cluster.slices, h->slice_base(), mv.node_elem_ptr, mv.node_elem, h->slot_map());
    note_launches(1);
    if ((rc = launch_check("cluster PCG map"))) return rc;
    return check_cuda(cudaStreamSynchronize(s), "cudaStreamSynchronize");
}

int prepare_cluster_any(dfea_pcg* h) {
    if (h->vec_dtype == DFEA_F64REF) return h->block ? prepare_cluster<double, true>(h) : prepare_cluster<double, false>(h);
    return h->block ? prepare_cluster<float, true>(h) : prepare_cluster<float, false>(h);
}

template <typename T, bool BJ = false>
int launch_setup(const dfea_pcg& h, cudaStream_t s, double rtol, int max_iter) {
    const dfea_mesh_view& mv = h.mesh;
    const Mesh m = kernel_mesh(mv);
    T* r = reinterpret_cast<T*>(h.work + h.layout.off_r);
    T* p = reinterpret_cast<T*>(h.work + h.layout.off_p);
    T* y = reinterpret_cast<T*>(h.work + h.layout.off_y);
    PcgState* st = h.state();
    k_pcg_reset<<<1, 128, 0, s>>>(st);
    k_pcg_setup<T, BJ><<<grid_for(mv.n_nodes, kThreads, 4), kThreads, 0, s>>>(
        m, static_cast<const T*>(h.b), static_cast<const T*>(h.diag), static_cast<T*>(h.x), r, p, y, st,
        h.site(mv.n_colours + 2, 3), rtol, max_iter);
    note_launches(2);
    return launch_check("pcg setup");
}

int build_graph(dfea_pcg* h) {
    int rc;
    if ((rc = check_cuda(cudaGraphCreate(&h->graph, 0), "cudaGraphCreate"))) return rc;
    cudaGraphConditionalHandle cond;
    if ((rc = check_cuda(cudaGraphConditionalHandleCreate(&cond, h->graph, 1u, cudaGraphCondAssignDefault),
                         "cudaGraphConditionalHandleCreate")))
        return rc;
    cudaGraphNodeParams cp = {cudaGraphNodeTypeConditional};  // aggregate init: the rest is zero
    cp.conditional.handle = cond;
    cp.conditional.type = cudaGraphCondTypeWhile;
    cp.conditional.size = 1;
    cudaGraphNode_t node;
    if ((rc = check_cuda(cudaGraphAddNode(&node, h->graph, nullptr, 0, &cp), "cudaGraphAddNode(while)"))) return rc;
    cudaGraph_t body = cp.conditional.phGraph_out[0];
    if ((rc = check_cuda(cudaStreamBeginCaptureToGraph(h->capture_stream, body, nullptr, nullptr, 0,
                                                       cudaStreamCaptureModeThreadLocal),
                         "cudaStreamBeginCaptureToGraph")))
        return rc;
    rc = launch_iteration_any(*h, h->capture_stream, cond, true);
    cudaGraph_t captured = body;
    const int rc_end = check_cuda(cudaStreamEndCapture(h->capture_stream, &captured), "cudaStreamEndCapture");
    if (rc) return rc;
    if (rc_end) return rc_end;
    return check_cuda(cudaGraphInstantiate(&h->exec, h->graph, 0), "cudaGraphInstantiate");
}

// Unrolled form: kUnrolled iterations captured back to back in a plain graph (no conditional node),
// replayed by the host until the status word reports an end.  Iterations after the end are no-ops.
constexpr int kUnrolled = 8;

int build_unrolled_graph(dfea_pcg* h) {
    int rc;
    if ((rc = check_cuda(cudaStreamBeginCapture(h->capture_stream, cudaStreamCaptureModeThreadLocal),
                         "cudaStreamBeginCapture")))
        return rc;
    for (int i = 0; i < kUnrolled && rc == DFEA_OK; ++i) rc = launch_iteration_any(*h, h->capture_stream, 0, false);
    cudaGraph_t g = nullptr;
    const int rc_end = check_cuda(cudaStreamEndCapture(h->capture_stream, &g), "cudaStreamEndCapture");
    h->graph = g;
    if (rc) return rc;
    if (rc_end) return rc_end;
    return check_cuda(cudaGraphInstantiate(&h->exec, h->graph, 0), "cudaGraphInstantiate");
}

void release(dfea_pcg* h) {
    if (h->exec) cudaGraphExecDestroy(h->exec);
    if (h->graph) cudaGraphDestroy(h->graph);
    if (h->capture_stream) cudaStreamDestroy(h->capture_stream);
    delete h;
}

}  // namespace

namespace {
// the layout of a handle: with room for the gather form's element results when the mesh has the
// node incidence that form needs
PcgLayout layout_for(const dfea_mesh_view& mv, int32_t vec_dtype) {
    const int64_t fe_pairs = (mv.node_elem_ptr && mv.node_elem) ? (int64_t)mv.nen * mv.stride : 0;
    return PcgLayout(mv.n_nodes, vec_dtype == DFEA_F32 ? 4 : 8, mv.n_colours, fe_pairs);
}
}  // namespace

extern "C" int64_t dfea_pcg_work_bytes(const dfea_mesh_view* mesh, int32_t vec_dtype) {
    if (!mesh || (vec_dtype != DFEA_F64 && vec_dtype != DFEA_F32 && vec_dtype != DFEA_MIXED && vec_dtype != DFEA_F32REF &&
                  vec_dtype != DFEA_F64REF))
        return -1;
    return layout_for(*mesh, vec_dtype).total;
}

extern "C" int dfea_pcg_create(const dfea_mesh_view* mesh, const void* moduli, const void* diag, const void* b,
                               void* x, int32_t vec_dtype, void* work, int32_t use_graph, dfea_pcg** out) {
    if (!out) return set_error(DFEA_ERR_INVALID, "dfea_pcg_create: out is NULL");
    *out = nullptr;
    int rc = validate_mesh(mesh, vec_dtype == DFEA_F32 || vec_dtype == DFEA_MIXED);
    if (rc) return rc;
    if (vec_dtype != DFEA_F64 && vec_dtype != DFEA_F32 && vec_dtype != DFEA_MIXED && vec_dtype != DFEA_F32REF &&
        vec_dtype != DFEA_F64REF)
        return set_error(DFEA_ERR_INVALID, "bad vector dtype");
    if (vec_dtype == DFEA_F64REF && !(use_graph & (DFEA_PCG_GATHER | DFEA_PCG_FUSED | DFEA_PCG_CLUSTER)))
        return set_error(DFEA_ERR_UNSUPPORTED, "dfea_pcg_create: DFEA_F64REF moduli need the gather or fused form");
    if (!moduli || !diag || !b || !x || !work) return set_error(DFEA_ERR_INVALID, "dfea_pcg_create: NULL pointer");
    auto al = [](const void* q) { return (reinterpret_cast<uintptr_t>(q) & 255u) == 0; };
    auto al16 = [](const void* q) { return (reinterpret_cast<uintptr_t>(q) & 15u) == 0; };
    if (!al(work)) return set_error(DFEA_ERR_INVALID, "dfea_pcg_create: work must be 256-byte aligned");
    if (!al16(moduli) || !al16(diag) || !al16(b) || !al16(x))
        return set_error(DFEA_ERR_INVALID, "dfea_pcg_create: moduli, diag, b and x must be 16-byte aligned");
    if (x == b) return set_error(DFEA_ERR_INVALID, "dfea_pcg_create: x must not alias b");

    dfea_pcg* h = new (std::nothrow) dfea_pcg;
    if (!h) return set_error(DFEA_ERR_INVALID, "dfea_pcg_create: out of host memory");
    h->mesh = *mesh;
    h->moduli = moduli;
    h->diag = diag;
    h->b = b;
    h->x = x;
    h->vec_dtype = vec_dtype;
    h->work = static_cast<char*>(work);
    h->layout = layout_for(*mesh, vec_dtype);
    h->gather = (use_graph & DFEA_PCG_GATHER) != 0;
    h->block = (use_graph & DFEA_PCG_BLOCK_JACOBI) != 0;
    h->fused = (use_graph & DFEA_PCG_FUSED) != 0;
    h->clustered = (use_graph & DFEA_PCG_CLUSTER) != 0;
    // beside a launch form, the cluster form is taken where the mesh fits it
    const bool cluster_optional = h->clustered && (use_graph & (DFEA_PCG_GATHER | DFEA_PCG_FUSED)) != 0;
    if (h->fused || h->clustered) h->gather = true;
    if (h->clustered && vec_dtype != DFEA_F64REF && vec_dtype != DFEA_F32REF) {
        delete h;
        return set_error(DFEA_ERR_UNSUPPORTED, "dfea_pcg_create: the cluster form takes reference-frame moduli");
    }
    h->grid_cap = (int)((uint32_t)use_graph >> 8);
    use_graph &= 0xff & ~(DFEA_PCG_GATHER | DFEA_PCG_BLOCK_JACOBI | DFEA_PCG_FUSED | DFEA_PCG_CLUSTER);
    if (h->block && vec_dtype == DFEA_F32) {
        delete h;
        return set_error(DFEA_ERR_UNSUPPORTED, "dfea_pcg_create: block-Jacobi needs f64 Krylov vectors");
    }
    h->use_graph = (use_graph == 2) ? 2 : (use_graph ? 1 : 0);
    if (h->gather && h->layout.off_fe == h->layout.total) {
        delete h;
        return set_error(DFEA_ERR_INVALID, "dfea_pcg_create: the gather form needs the mesh's node incidence");
    }
    if (h->clustered) {  // captures nothing, and every solve resets the state it uses
        rc = prepare_cluster_any(h);
        if (!rc) {
            *out = h;
            return DFEA_OK;
        }
        if (rc != DFEA_ERR_UNSUPPORTED || !cluster_optional) {
            release(h);
            return rc;
        }
        h->clustered = false;
    }
    // device queries and kernel attributes are set up before any stream capture
    (void)device_sm_count();
    dispatch_element(mesh->nen, mesh->n_q, [&](auto nen_c, auto nq_c) -> int {
        constexpr int NEN = decltype(nen_c)::value, NQ = decltype(nq_c)::value;
        if (vec_dtype == DFEA_F64) prepare_apply<NEN, NQ, double, double>();
        else if (vec_dtype == DFEA_MIXED) prepare_apply<NEN, NQ, float, double>();
        else if (vec_dtype == DFEA_F32REF) prepare_apply_ref<NEN, NQ, float, double>();
        else if (vec_dtype == DFEA_F64REF) prepare_apply_ref<NEN, NQ, double, double>();
        else prepare_apply<NEN, NQ, float, float>();
        if (h->fused) {  // the fused element pass of this handle's types
            if (vec_dtype == DFEA_F32REF) {
                if (h->block) (void)frame_resident_grid<k_pcg_elem_fused_ref<NEN, NQ, float, double, true>, NEN, NQ>(1);
                else (void)frame_resident_grid<k_pcg_elem_fused_ref<NEN, NQ, float, double, false>, NEN, NQ>(1);
            } else if (vec_dtype == DFEA_F64REF) {
                if (h->block) (void)frame_resident_grid<k_pcg_elem_fused_ref<NEN, NQ, double, double, true>, NEN, NQ>(1);
                else (void)frame_resident_grid<k_pcg_elem_fused_ref<NEN, NQ, double, double, false>, NEN, NQ>(1);
            } else if (vec_dtype == DFEA_F64) {
                using Cfg = ApplyCfg<NEN, double>;
                if (h->block) (void)resident_grid<k_pcg_elem_fused<NEN, NQ, double, double, true>, Cfg::SMEM, Cfg::NT>(1);
                else (void)resident_grid<k_pcg_elem_fused<NEN, NQ, double, double, false>, Cfg::SMEM, Cfg::NT>(1);
            } else if (vec_dtype == DFEA_MIXED) {
                using Cfg = ApplyCfg<NEN, float>;
                if (h->block) (void)resident_grid<k_pcg_elem_fused<NEN, NQ, float, double, true>, Cfg::SMEM, Cfg::NT>(1);
                else (void)resident_grid<k_pcg_elem_fused<NEN, NQ, float, double, false>, Cfg::SMEM, Cfg::NT>(1);
            } else {
                using Cfg = ApplyCfg<NEN, float>;
                (void)resident_grid<k_pcg_elem_fused<NEN, NQ, float, float, false>, Cfg::SMEM, Cfg::NT>(1);
            }
        }
        return DFEA_OK;
    });
    if ((rc = check_cuda(cudaStreamCreateWithFlags(&h->capture_stream, cudaStreamNonBlocking), "cudaStreamCreate"))) {
        release(h);
        return rc;
    }
    // zero the partial sums, tickets and state once (later solves reset what they use)
    if ((rc = check_cuda(cudaMemsetAsync(h->work + h->layout.off_part, 0, h->layout.total - h->layout.off_part,
                                         h->capture_stream), "cudaMemsetAsync")) ||
        (rc = check_cuda(cudaStreamSynchronize(h->capture_stream), "cudaStreamSynchronize"))) {
        release(h);
        return rc;
    }
    if (h->use_graph == 1 && (rc = build_graph(h))) {
        release(h);
        return rc;
    }
    if (h->use_graph == 2 && (rc = build_unrolled_graph(h))) {
        release(h);
        return rc;
    }
    *out = h;
    return DFEA_OK;
}

extern "C" int dfea_pcg_solve(dfea_pcg* h, double rtol, int32_t max_iter, int32_t* iters, int32_t* status,
                              void* stream) {
    if (!h) return set_error(DFEA_ERR_INVALID, "dfea_pcg_solve: NULL handle");
    if (max_iter < 1 || max_iter > 100000000) return set_error(DFEA_ERR_INVALID, "max_iter %d out of [1, 1e8]", max_iter);
    if (!(rtol >= 0.0)) return set_error(DFEA_ERR_INVALID, "rtol must be >= 0");
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    if (h->clustered) {
        int rcc = launch_cluster_any(*h, s, rtol, max_iter);
        if (rcc || (rcc = read_to_host(h->host_status, &h->state()->done, 2 * sizeof(int32_t), s))) return rcc;
        if (h->host_status[0] == DFEA_PCG_RUNNING)
            return set_error(DFEA_ERR_INVALID, "PCG ended without a status (internal error)");
        if (status) *status = h->host_status[0];
        if (iters) *iters = h->host_status[1];
        return DFEA_OK;
    }
    int rc = (h->vec_dtype == DFEA_F32) ? launch_setup<float>(*h, s, rtol, max_iter)
             : h->block                 ? launch_setup<double, true>(*h, s, rtol, max_iter)
                                        : launch_setup<double>(*h, s, rtol, max_iter);
    if (rc) return rc;
    PcgState* st = h->state();
    if (h->use_graph == 2) {
        int launched = 0;
        h->host_status[0] = DFEA_PCG_RUNNING;
        while (true) {
            if ((rc = check_cuda(cudaGraphLaunch(h->exec, s), "cudaGraphLaunch"))) return rc;
            launched += kUnrolled;
            if ((rc = read_to_host(h->host_status, &st->done, 2 * sizeof(int32_t), s))) return rc;
            if (h->host_status[0] != DFEA_PCG_RUNNING || launched > max_iter + kUnrolled) break;
        }
        note_launches((long long)launched * kernels_per_iteration(*h));
    } else if (h->use_graph) {
        if ((rc = check_cuda(cudaGraphLaunch(h->exec, s), "cudaGraphLaunch"))) return rc;
        if ((rc = read_to_host(h->host_status, &st->done, 3 * sizeof(int32_t), s))) return rc;
        // each executed body ran one iteration's kernels and the loop condition
        note_launches((long long)h->host_status[2] * (kernels_per_iteration(*h) + 1));
    } else {
        // the same kernels launched directly; the host reads the status every 16 iterations
        const int chunk = 16;
        int launched = 0;
        h->host_status[0] = DFEA_PCG_RUNNING;
        while (true) {
            for (int i = 0; i < chunk; ++i) {
                rc = launch_iteration_any(*h, s, 0, false);
                if (rc) return rc;
            }
            launched += chunk;
            if ((rc = read_to_host(h->host_status, &st->done, 2 * sizeof(int32_t), s))) return rc;
            if (h->host_status[0] != DFEA_PCG_RUNNING || launched > max_iter + chunk) break;
        }
    }
    if (h->host_status[0] == DFEA_PCG_RUNNING)
        return set_error(DFEA_ERR_INVALID, "PCG ended without a status (internal error)");
    if (status) *status = h->host_status[0];
    if (iters) *iters = h->host_status[1];
    return DFEA_OK;
}

extern "C" int dfea_pcg_clustered(const dfea_pcg* h) { return h && h->clustered ? 1 : 0; }

extern "C" int dfea_pcg_destroy(dfea_pcg* h) {
    if (h) release(h);
    return DFEA_OK;
}

// ------------------------------------------------------------------------------------------------
// Allocation-free PCG: the work area is a file-scope device array instead of a caller buffer.
// ------------------------------------------------------------------------------------------------
// Reserved in each GPU's memory when the library's module is loaded there; kept until exit.
static __device__ __align__(256) unsigned char g_noalloc_scratch[DFEA_NOALLOC_SCRATCH_BYTES];

namespace {

constexpr int kNoallocMaxColours = 16;
constexpr int kNoallocMaxDevices = 64;
std::mutex g_noalloc_mutex;
void* g_noalloc_address[kNoallocMaxDevices] = {};

// Device address of g_noalloc_scratch for the current device.  In host code the symbol itself is a
// host-side stand-in, so the address is looked up once per device, with that device current.
int noalloc_scratch(void** out) {
    int dev = 0;
    int rc = check_cuda(cudaGetDevice(&dev), "cudaGetDevice");
    if (rc) return rc;
    if (dev < 0 || dev >= kNoallocMaxDevices) return set_error(DFEA_ERR_INVALID, "device ordinal %d unsupported", dev);
    std::lock_guard<std::mutex> lock(g_noalloc_mutex);
    if (g_noalloc_address[dev] == nullptr) {
        void* p = nullptr;
        rc = check_cuda(cudaGetSymbolAddress(&p, g_noalloc_scratch), "cudaGetSymbolAddress(g_noalloc_scratch)");
        if (rc) return rc;
        g_noalloc_address[dev] = p;
    }
    *out = g_noalloc_address[dev];
    return DFEA_OK;
}

}  // namespace

extern "C" int dfea_pcg_solve_noalloc(const dfea_mesh_view* mesh, const void* moduli, const void* diag, const void* b,
                                      void* x, int32_t vec_dtype, double rtol, int32_t max_iter, int32_t* iters,
                                      int32_t* status, void* stream) {
    int rc = validate_mesh(mesh, vec_dtype != DFEA_F64);
    if (rc) return rc;
    if (vec_dtype != DFEA_F64 && vec_dtype != DFEA_F32 && vec_dtype != DFEA_MIXED)
        return set_error(DFEA_ERR_INVALID, "bad vector dtype");
    if (!moduli || !diag || !b || !x) return set_error(DFEA_ERR_INVALID, "dfea_pcg_solve_noalloc: NULL pointer");
    auto al16 = [](const void* q) { return (reinterpret_cast<uintptr_t>(q) & 15u) == 0; };
    if (!al16(moduli) || !al16(diag) || !al16(b) || !al16(x))
        return set_error(DFEA_ERR_INVALID, "dfea_pcg_solve_noalloc: moduli, diag, b and x must be 16-byte aligned");
    if (x == b) return set_error(DFEA_ERR_INVALID, "dfea_pcg_solve_noalloc: x must not alias b");
    if (mesh->n_nodes > DFEA_NOALLOC_MAX_NODES)
        return set_error(DFEA_ERR_INVALID, "dfea_pcg_solve_noalloc: %lld nodes exceed the fixed scratch limit of %d nodes",
                         (long long)mesh->n_nodes, DFEA_NOALLOC_MAX_NODES);
    if (mesh->n_colours > kNoallocMaxColours)
        return set_error(DFEA_ERR_INVALID, "dfea_pcg_solve_noalloc: %d colours exceed the limit of %d", mesh->n_colours,
                         kNoallocMaxColours);
    if (max_iter < 1 || max_iter > 100000000) return set_error(DFEA_ERR_INVALID, "max_iter %d out of [1, 1e8]", max_iter);
    if (!(rtol >= 0.0)) return set_error(DFEA_ERR_INVALID, "rtol must be >= 0");
    const PcgLayout layout(mesh->n_nodes, vec_dtype == DFEA_F32 ? 4 : 8, mesh->n_colours);
    if (layout.total > DFEA_NOALLOC_SCRATCH_BYTES)
        return set_error(DFEA_ERR_INVALID, "dfea_pcg_solve_noalloc: needs %lld scratch bytes, the fixed array has %d",
                         (long long)layout.total, DFEA_NOALLOC_SCRATCH_BYTES);
    void* scratch = nullptr;
    if ((rc = noalloc_scratch(&scratch))) return rc;

    // A handle on the stack bound to the fixed scratch: no graph, no stream, no pinned buffer.
    dfea_pcg h;
    int32_t host_status[4] = {DFEA_PCG_RUNNING, 0, 0, 0};
    h.mesh = *mesh;
    h.moduli = moduli;
    h.diag = diag;
    h.b = b;
    h.x = x;
    h.vec_dtype = vec_dtype;
    h.work = static_cast<char*>(scratch);
    h.layout = layout;
    h.use_graph = 0;
    h.host_status = host_status;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    (void)device_sm_count();
    // k_pcg_reset (first kernel of the setup) clears the tickets and state the previous call left behind
    rc = (vec_dtype == DFEA_F32) ? launch_setup<float>(h, s, rtol, max_iter) : launch_setup<double>(h, s, rtol, max_iter);
    if (rc) return rc;
    PcgState* st = h.state();
    const int chunk = 16;
    int launched = 0;
    while (true) {
        for (int i = 0; i < chunk; ++i) {
            rc = launch_iteration_any(h, s, 0, false);
            if (rc) return rc;
        }
        launched += chunk;
        if ((rc = check_cuda(cudaMemcpyAsync(host_status, &st->done, 2 * sizeof(int32_t), cudaMemcpyDeviceToHost, s),
                             "cudaMemcpyAsync")) ||
            (rc = check_cuda(cudaStreamSynchronize(s), "cudaStreamSynchronize")))
            return rc;
        if (host_status[0] != DFEA_PCG_RUNNING || launched > max_iter + chunk) break;
    }
    if (host_status[0] == DFEA_PCG_RUNNING) return set_error(DFEA_ERR_INVALID, "PCG ended without a status (internal error)");
    if (status) *status = host_status[0];
    if (iters) *iters = host_status[1];
    return DFEA_OK;
}

// ------------------------------------------------------------------------------------------------
// Batched PCG: the solves of several handles advance together, one set of launches per iteration for
// all of them (an element pass per element type, one launch of each vector update).  Every block works
// for one solve (a block map gives the solve and the block's number within it); each solve keeps its
// own state, partial sums and tickets.  A solve's blocks are as many, and split its work the same way,
// as when it runs alone with the same block cap, so its iterates are bitwise those of its own handle.
// Supported handles: gather form (not fused), Jacobi, DFEA_F32REF moduli on f64 vectors (the serving
// configuration).
// ------------------------------------------------------------------------------------------------
namespace dfea {

struct BatchSolve {
    Mesh m;
    const int32_t* inc_ptr;
    const int32_t* inc;
    const float* C;
    const double* d;
    double* x;
    double* r;
    double* p;
    double* fe;
    PcgState* st;
    RedSite site_elem, site_u1, site_u2;
    int elem_blocks;
    int node_blocks;
};

template <int NEN, int NQ>
__global__ void __launch_bounds__(FrameCfg<NEN, NQ>::NT, FrameCfg<NEN, NQ>::MINB)
k_batch_elem(const BatchSolve* __restrict__ solves, const int2* __restrict__ block_map, const RefGrad<NEN, NQ> rg) {
    constexpr int NT = FrameCfg<NEN, NQ>::NT;
    __shared__ FrameShared<NEN, NQ, double> sh;
    const int2 bm = block_map[blockIdx.x];
    const BatchSolve* S = solves + bm.x;
    const Mesh m = S->m;
    PcgState* st = S->st;
    const double2* p2 = reinterpret_cast<const double2*>(S->p);
    double2* fe2 = reinterpret_cast<double2*>(S->fe);
    const int64_t Sd = m.stride;
    double curv = 0.0;
    const bool ran = frame_product<NEN, NQ, float, double, true>(
        m, S->C, rg, sh, curv,
        [&]() -> bool {
            grid_dependency_wait();
            if (st->done) return false;
            grid_dependents_launch();
            return true;
        },
        [&](int n) { return load_fresh(p2 + n); },
        [&](int a, int64_t e, double2 f) { fe2[(int64_t)a * Sd + e] = f; }, bm.y, S->elem_blocks);
    if (!ran) return;
    const double vals[1] = {block_sum<NT>(curv)};
    double tot[1];
    if (last_block_sum_in<NT, 1>(vals, S->site_elem, tot, bm.y, S->elem_blocks) && threadIdx.x == 0)
        S->site_elem.result[0] = tot[0];
}

__global__ void __launch_bounds__(kThreads) k_batch_update1(const BatchSolve* __restrict__ solves,
                                                           const int2* __restrict__ block_map) {
    grid_dependency_wait();
    grid_dependents_launch();
    const int2 bm = block_map[blockIdx.x];
    const BatchSolve* S = solves + bm.x;
    pcg_update1_body<double, true, false>(S->m, 1, S->p, S->p, S->d, S->x, S->r, S->st, S->site_u1, S->inc_ptr, S->inc,
                                          S->fe, bm.y, S->node_blocks);
}

__global__ void __launch_bounds__(kThreads) k_batch_update2(const BatchSolve* __restrict__ solves,
                                                           const int2* __restrict__ block_map) {
    grid_dependency_wait();
    grid_dependents_launch();
    const int2 bm = block_map[blockIdx.x];
    const BatchSolve* S = solves + bm.x;
    pcg_update2_body<double, false, false>(S->m, S->r, S->d, S->p, S->p, S->st, S->site_u2, bm.y, S->node_blocks);
}

__global__ void k_batch_status(const BatchSolve* __restrict__ solves, int n, int32_t* __restrict__ out) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        out[2 * i] = solves[i].st->done;
        out[2 * i + 1] = solves[i].st->iters;
    }
}

}  // namespace dfea

struct dfea_batch {
    int capacity = 0;
    int max_blocks = 0;
    int n = 0;
    BatchSolve* d_solves = nullptr;
    BatchSolve* h_solves = nullptr;  // pinned
    int2* d_map = nullptr;
    int2* h_map = nullptr;           // pinned: element maps by type, then the node map
    int32_t* d_status = nullptr;
    int32_t* h_status = nullptr;     // pinned
    int map_entries = 0;
    struct TypeRange {
        int nen, nq, first, count;   // element-map entries [first, first + count)
        dfea_mesh_view view;         // a view of this type (for its reference gradients)
    } types[8];
    int n_types = 0;
    int node_first = 0, node_count = 0;
};

namespace {

void batch_release(dfea_batch* b) {
    if (b->d_solves) cudaFree(b->d_solves);
    if (b->d_map) cudaFree(b->d_map);
    if (b->d_status) cudaFree(b->d_status);
    if (b->h_solves) cudaFreeHost(b->h_solves);
    if (b->h_map) cudaFreeHost(b->h_map);
    if (b->h_status) cudaFreeHost(b->h_status);
    delete b;
}

}  // namespace

extern "C" int dfea_batch_create(int32_t capacity, int32_t max_blocks, dfea_batch** out) {
    if (!out) return set_error(DFEA_ERR_INVALID, "dfea_batch_create: out is NULL");
    *out = nullptr;
    if (capacity < 1 || capacity > 4096) return set_error(DFEA_ERR_INVALID, "dfea_batch_create: capacity out of [1, 4096]");
    if (max_blocks < 1 || max_blocks > kMaxBlocks)
        return set_error(DFEA_ERR_INVALID, "dfea_batch_create: max_blocks out of [1, %d]", kMaxBlocks);
    dfea_batch* b = new (std::nothrow) dfea_batch;
    if (!b) return set_error(DFEA_ERR_INVALID, "dfea_batch_create: out of host memory");
    b->capacity = capacity;
    b->max_blocks = max_blocks;
    b->map_entries = 2 * capacity * max_blocks;  // element blocks + node blocks, at most max_blocks each
    int rc;
    if ((rc = check_cuda(cudaMalloc(&b->d_solves, sizeof(BatchSolve) * capacity), "cudaMalloc")) ||
        (rc = check_cuda(cudaMalloc(&b->d_map, sizeof(int2) * b->map_entries), "cudaMalloc")) ||
        (rc = check_cuda(cudaMalloc(&b->d_status, sizeof(int32_t) * 2 * capacity), "cudaMalloc")) ||
        (rc = check_cuda(cudaHostAlloc(reinterpret_cast<void**>(&b->h_solves), sizeof(BatchSolve) * capacity,
                                       cudaHostAllocDefault), "cudaHostAlloc")) ||
        (rc = check_cuda(cudaHostAlloc(reinterpret_cast<void**>(&b->h_map), sizeof(int2) * b->map_entries,
                                       cudaHostAllocDefault), "cudaHostAlloc")) ||
        (rc = check_cuda(cudaHostAlloc(reinterpret_cast<void**>(&b->h_status), sizeof(int32_t) * 2 * capacity,
                                       cudaHostAllocDefault), "cudaHostAlloc"))) {
        batch_release(b);
        return rc;
    }
    *out = b;
    return DFEA_OK;
}

extern "C" int dfea_batch_destroy(dfea_batch* b) {
    if (b) batch_release(b);
    return DFEA_OK;
}

extern "C" int dfea_batch_start(dfea_batch* b, dfea_pcg* h, double rtol, int32_t max_iter, void* stream) {
    if (!b || !h) return set_error(DFEA_ERR_INVALID, "dfea_batch_start: NULL pointer");
    if (!h->gather || h->fused || h->clustered || h->block || h->vec_dtype != DFEA_F32REF)
        return set_error(DFEA_ERR_UNSUPPORTED,
                         "dfea_batch_start: batched solves need the gather form, Jacobi and DFEA_F32REF moduli");
    if (max_iter < 1 || max_iter > 100000000) return set_error(DFEA_ERR_INVALID, "max_iter %d out of [1, 1e8]", max_iter);
    if (!(rtol >= 0.0)) return set_error(DFEA_ERR_INVALID, "rtol must be >= 0");
    return launch_setup<double>(*h, static_cast<cudaStream_t>(stream), rtol, max_iter);
}

extern "C" int dfea_batch_set(dfea_batch* b, dfea_pcg* const* solves, int32_t n, void* stream) {
    if (!b || (n > 0 && !solves)) return set_error(DFEA_ERR_INVALID, "dfea_batch_set: NULL pointer");
    if (n < 0 || n > b->capacity) return set_error(DFEA_ERR_INVALID, "dfea_batch_set: %d solves, capacity %d", n, b->capacity);
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    // the previous table may still be read by launched kernels: wait for them before rewriting it
    int rc = check_cuda(cudaStreamSynchronize(s), "cudaStreamSynchronize");
    if (rc) return rc;
    b->n = n;
    b->n_types = 0;
    int entries = 0;
    for (int i = 0; i < n; ++i) {
        const dfea_pcg& h = *solves[i];
        if (!h.gather || h.fused || h.clustered || h.block || h.vec_dtype != DFEA_F32REF)
            return set_error(DFEA_ERR_UNSUPPORTED, "dfea_batch_set: solve %d is not in the batched configuration", i);
        const dfea_mesh_view& mv = h.mesh;
        BatchSolve& S = b->h_solves[i];
        S.m = kernel_mesh(mv);
        S.inc_ptr = mv.node_elem_ptr;
        S.inc = mv.node_elem;
        S.C = static_cast<const float*>(h.moduli);
        S.d = static_cast<const double*>(h.diag);
        S.x = static_cast<double*>(h.x);
        S.r = reinterpret_cast<double*>(h.work + h.layout.off_r);
        S.p = reinterpret_cast<double*>(h.work + h.layout.off_p);
        S.fe = reinterpret_cast<double*>(h.work + h.layout.off_fe);
        S.st = h.state();
        S.site_elem = h.site(0, 1);
        S.site_u1 = h.site(mv.n_colours, 2);
        S.site_u2 = h.site(mv.n_colours + 1, 1);
        const int cap = h.grid_cap > 0 ? h.grid_cap : b->max_blocks;
        rc = dispatch_element(mv.nen, mv.n_q, [&](auto nen_c, auto nq_c) -> int {
            constexpr int NEN = decltype(nen_c)::value, NQ = decltype(nq_c)::value;
            S.elem_blocks = capped(apply_ref_elem_grid<NEN, NQ, float, double, true>(mv.n_el), cap);
            (void)frame_resident_grid<k_batch_elem<NEN, NQ>, NEN, NQ>(1);
            return DFEA_OK;
        });
        if (rc) return rc;
        S.node_blocks = capped(grid_for(mv.n_nodes, kThreads, 4), cap);
        if (S.elem_blocks > b->max_blocks || S.node_blocks > b->max_blocks)
            return set_error(DFEA_ERR_INVALID, "dfea_batch_set: solve %d needs more blocks than the batch's cap", i);
    }
    // element maps grouped by element type, then the node map
    for (int i = 0; i < n; ++i) {
        const dfea_mesh_view& mv = solves[i]->mesh;
        int t = 0;
        while (t < b->n_types && !(b->types[t].nen == mv.nen && b->types[t].nq == mv.n_q)) ++t;
        if (t == b->n_types) {
            if (b->n_types == 8) return set_error(DFEA_ERR_UNSUPPORTED, "dfea_batch_set: too many element types");
            b->types[t] = {mv.nen, mv.n_q, 0, 0, mv};
            ++b->n_types;
        } else if (std::memcmp(b->types[t].view.ref_grad, mv.ref_grad, sizeof(double) * mv.nen * mv.n_q * 2) != 0) {
            // one launch per element type passes one table of reference gradients
            return set_error(DFEA_ERR_INVALID, "dfea_batch_set: solves of one element type differ in ref_grad");
        }
    }
    for (int t = 0; t < b->n_types; ++t) {
        b->types[t].first = entries;
        for (int i = 0; i < n; ++i) {
            const dfea_mesh_view& mv = solves[i]->mesh;
            if (mv.nen != b->types[t].nen || mv.n_q != b->types[t].nq) continue;
            for (int k = 0; k < b->h_solves[i].elem_blocks; ++k) b->h_map[entries++] = make_int2(i, k);
        }
        b->types[t].count = entries - b->types[t].first;
    }
    b->node_first = entries;
    for (int i = 0; i < n; ++i)
        for (int k = 0; k < b->h_solves[i].node_blocks; ++k) b->h_map[entries++] = make_int2(i, k);
    b->node_count = entries - b->node_first;
    if (n == 0) return DFEA_OK;
    if ((rc = check_cuda(cudaMemcpyAsync(b->d_solves, b->h_solves, sizeof(BatchSolve) * n, cudaMemcpyHostToDevice, s),
                         "cudaMemcpyAsync")) ||
        (rc = check_cuda(cudaMemcpyAsync(b->d_map, b->h_map, sizeof(int2) * entries, cudaMemcpyHostToDevice, s),
                         "cudaMemcpyAsync")))
        return rc;
    return DFEA_OK;
}

extern "C" int dfea_batch_iterate(dfea_batch* b, int32_t n_iterations, int32_t* status, int32_t* iters, void* stream) {
    if (!b) return set_error(DFEA_ERR_INVALID, "dfea_batch_iterate: NULL batch");
    if (n_iterations < 0 || n_iterations > 1000000) return set_error(DFEA_ERR_INVALID, "n_iterations out of range");
    if (b->n == 0) return DFEA_OK;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    LaunchOpts pdl;
    pdl.pdl = true;
    int rc = DFEA_OK;
    for (int it = 0; it < n_iterations && rc == DFEA_OK; ++it) {
        for (int t = 0; t < b->n_types && rc == DFEA_OK; ++t) {
            const auto& ty = b->types[t];
            rc = dispatch_element(ty.nen, ty.nq, [&](auto nen_c, auto nq_c) -> int {
                constexpr int NEN = decltype(nen_c)::value, NQ = decltype(nq_c)::value;
                return launch_kernel(k_batch_elem<NEN, NQ>, dim3(ty.count), dim3(FrameCfg<NEN, NQ>::NT), 0, s, pdl,
                                     (const BatchSolve*)b->d_solves, (const int2*)(b->d_map + ty.first),
                                     ref_grad_of<NEN, NQ>(ty.view));
            });
        }
        if (rc) break;
        if ((rc = launch_kernel(k_batch_update1, dim3(b->node_count), dim3(kThreads), 0, s, pdl,
                                (const BatchSolve*)b->d_solves, (const int2*)(b->d_map + b->node_first))))
            break;
        rc = launch_kernel(k_batch_update2, dim3(b->node_count), dim3(kThreads), 0, s, pdl, (const BatchSolve*)b->d_solves,
                           (const int2*)(b->d_map + b->node_first));
    }
    if (rc) return rc;
    note_launches((long long)n_iterations * (b->n_types + 2));
    k_batch_status<<<1, 128, 0, s>>>(b->d_solves, b->n, b->d_status);
    if ((rc = launch_check("k_batch_status")) ||
        (rc = check_cuda(cudaMemcpyAsync(b->h_status, b->d_status, sizeof(int32_t) * 2 * b->n, cudaMemcpyDeviceToHost, s),
                         "cudaMemcpyAsync")) ||
        (rc = check_cuda(cudaStreamSynchronize(s), "cudaStreamSynchronize")))
        return rc;
    for (int i = 0; i < b->n; ++i) {
        if (status) status[i] = b->h_status[2 * i];
        if (iters) iters[i] = b->h_status[2 * i + 1];
    }
    return DFEA_OK;
}
