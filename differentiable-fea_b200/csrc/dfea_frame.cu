// dfea_frame.cu -- linearisation, residual, sensitivity, post-processing and the tangent product on meshes whose
// dN/dX is Jinv^T dN/dxi at every Gauss point (dfea_frame.cuh); entry points in include/difffea_b200.h.
#include <type_traits>

#include "dfea_apply.cuh"
#include "dfea_common.cuh"
#include "dfea_frame.cuh"

namespace dfea {

int validate_mesh(const dfea_mesh_view* mv, bool need_grad32);
int validate_material(const dfea_material* mat);

// ------------------------------------------------------------------------------------------
// the frame: Jinv of every Gauss point, fitted to the packed gradients
// ------------------------------------------------------------------------------------------
// W[q] = (R^T R)^-1 R^T of the reference gradients R = dN/dxi (nen x 2), so that Jinv = W dN/dX reproduces a
// dN/dX of the form R Jinv to rounding -- also where the node coordinates have lost digits to their offset.
template <int NEN, int NQ>
struct RefPinv {
    double w[NQ][2][NEN];
};
template <int NEN, int NQ>
static RefPinv<NEN, NQ> ref_pinv_of(const dfea_mesh_view& v) {
    RefPinv<NEN, NQ> r;
    for (int q = 0; q < NQ; ++q) {
        const double* R = v.ref_grad + q * NEN * 2;
        double a = 0.0, b = 0.0, c = 0.0;
        for (int k = 0; k < NEN; ++k) {
            a += R[2 * k] * R[2 * k];
            b += R[2 * k] * R[2 * k + 1];
            c += R[2 * k + 1] * R[2 * k + 1];
        }
        const double det = a * c - b * b;
        for (int k = 0; k < NEN; ++k) {
            r.w[q][0][k] = (c * R[2 * k] - b * R[2 * k + 1]) / det;
            r.w[q][1][k] = (a * R[2 * k + 1] - b * R[2 * k]) / det;
        }
    }
    return r;
}

__device__ __forceinline__ void frame_max(double& m, double v) {  // a NaN wins
    if (v > m || v != v) m = (m != m) ? m : v;
}

// frame_out [q][2][S] pairs (zeros in the padding slots).  check[0], check[1]: the largest |Jn^T dN/dxi - dN/dX| and
// |dN/dX| of the mesh with Jn from the node coordinates; check[2]: the largest fit error of a Gauss point relative
// to its own largest |dN/dX|.  Maxima of non-negative values through atomic maxima of the bit patterns:
// order-independent.
template <int NEN, int NQ>
__global__ void __launch_bounds__(128)
k_frame(Mesh m, RefGrad<NEN, NQ> rg, RefPinv<NEN, NQ> pinv, const double* __restrict__ nodes,
        double* __restrict__ frame_out, double* __restrict__ check) {
    const int64_t S = m.stride;
    double2* out = reinterpret_cast<double2*>(frame_out);
    const double2* g2 = reinterpret_cast<const double2*>(m.grad);
    double dmax = 0.0, smax = 0.0, fmaxr = 0.0;
    const int64_t n = S * NQ;
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < n; t += (int64_t)gridDim.x * blockDim.x) {
        const int q = (int)(t / S);
        const int64_t e = t - q * S;
        if (e >= m.n_el) {
            out[(2 * q) * S + e] = make_double2(0.0, 0.0);
            out[(2 * q + 1) * S + e] = make_double2(0.0, 0.0);
            continue;
        }
        double ji[4] = {0.0, 0.0, 0.0, 0.0}, J[4] = {0.0, 0.0, 0.0, 0.0};
        double2 g[NEN];
        const int64_t n0 = m.conn[e] >> 2;
        const double x0 = nodes[2 * n0], y0 = nodes[2 * n0 + 1];
#pragma unroll
        for (int a = 0; a < NEN; ++a) {
            g[a] = __ldcs(g2 + (int64_t)(q * NEN + a) * S + e);
            ji[0] += pinv.w[q][0][a] * g[a].x;
            ji[1] += pinv.w[q][0][a] * g[a].y;
            ji[2] += pinv.w[q][1][a] * g[a].x;
            ji[3] += pinv.w[q][1][a] * g[a].y;
            const int64_t node = m.conn[a * S + e] >> 2;
            const double x = nodes[2 * node] - x0, y = nodes[2 * node + 1] - y0;
            J[0] += x * rg.g[q][a][0];
            J[1] += x * rg.g[q][a][1];
            J[2] += y * rg.g[q][a][0];
            J[3] += y * rg.g[q][a][1];
        }
        out[(2 * q) * S + e] = make_double2(ji[0], ji[1]);
        out[(2 * q + 1) * S + e] = make_double2(ji[2], ji[3]);
        const double det = J[0] * J[3] - J[1] * J[2];
        const double i00 = J[3] / det, i01 = -J[1] / det, i10 = -J[2] / det, i11 = J[0] / det;
        double fit = 0.0, scale = 0.0;
#pragma unroll
        for (int a = 0; a < NEN; ++a) {
            const double r0 = rg.g[q][a][0], r1 = rg.g[q][a][1];
            frame_max(dmax, fabs(r0 * i00 + r1 * i10 - g[a].x));
            frame_max(dmax, fabs(r0 * i01 + r1 * i11 - g[a].y));
            frame_max(fit, fabs(r0 * ji[0] + r1 * ji[2] - g[a].x));
            frame_max(fit, fabs(r0 * ji[1] + r1 * ji[3] - g[a].y));
            frame_max(scale, fabs(g[a].x));
            frame_max(scale, fabs(g[a].y));
        }
        frame_max(smax, scale);
        frame_max(fmaxr, fit / scale);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        frame_max(dmax, __shfl_down_sync(0xffffffffu, dmax, o));
        frame_max(smax, __shfl_down_sync(0xffffffffu, smax, o));
        frame_max(fmaxr, __shfl_down_sync(0xffffffffu, fmaxr, o));
    }
    if ((threadIdx.x & 31) == 0) {
        unsigned long long* c = reinterpret_cast<unsigned long long*>(check);
        atomicMax(c, (unsigned long long)__double_as_longlong(dmax));
        atomicMax(c + 1, (unsigned long long)__double_as_longlong(smax));
        atomicMax(c + 2, (unsigned long long)__double_as_longlong(fmaxr));
    }
}

// ------------------------------------------------------------------------------------------
// reference-frame moduli of a Gauss point, h = 00 01 02 03 11 12 13 22 23 33
// ------------------------------------------------------------------------------------------
// neo-Hookean in closed form: with p = F^-T pulled back (p_ia = F^-T_iJ Jinv_aJ) and M = Jinv Jinv^T,
// h_(ia),(kb) = w (mu d_ik M_ab + lambda p_ia p_kb + (mu - lambda lnJ) p_ka p_ib)
__device__ __forceinline__ void nh_frame_moduli(const NHPoint& pt, double mu, double lam, double w, const double (&ji)[4],
                                                double (&h)[10]) {
    const double wl = w * lam, wa = w * (mu - lam * pt.lnJ), wm = w * mu;
    double p[4];
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int a = 0; a < 2; ++a) p[2 * i + a] = pt.FiT[2 * i] * ji[2 * a] + pt.FiT[2 * i + 1] * ji[2 * a + 1];
    const double m00 = wm * (ji[0] * ji[0] + ji[1] * ji[1]), m01 = wm * (ji[0] * ji[2] + ji[1] * ji[3]),
                 m11 = wm * (ji[2] * ji[2] + ji[3] * ji[3]);
    const double s = wl + wa;  // i == k: both products are p_ia p_ib
    h[0] = m00 + s * p[0] * p[0];
    h[1] = m01 + s * p[0] * p[1];
    h[4] = m11 + s * p[1] * p[1];
    h[7] = m00 + s * p[2] * p[2];
    h[8] = m01 + s * p[2] * p[3];
    h[9] = m11 + s * p[3] * p[3];
    h[2] = s * p[0] * p[2];                       // (0,0),(1,0)
    h[3] = wl * p[0] * p[3] + wa * p[2] * p[1];   // (0,0),(1,1)
    h[5] = wl * p[1] * p[2] + wa * p[3] * p[0];   // (0,1),(1,0)
    h[6] = s * p[1] * p[3];                       // (0,1),(1,1)
}

// any symmetric moduli C (row-major 4 x 4): h = Jinv C Jinv^T
__device__ __forceinline__ void pull_back(const double (&c)[16], const double (&ji)[4], double (&h)[10]) {
    double f[16];
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int k = i; k < 2; ++k) {
            double t[2][2];
#pragma unroll
            for (int J = 0; J < 2; ++J)
#pragma unroll
                for (int b = 0; b < 2; ++b)
                    t[J][b] = c[(2 * i + J) * 4 + 2 * k] * ji[2 * b] + c[(2 * i + J) * 4 + 2 * k + 1] * ji[2 * b + 1];
#pragma unroll
            for (int a = 0; a < 2; ++a)
#pragma unroll
                for (int b = 0; b < 2; ++b) f[(2 * i + a) * 4 + 2 * k + b] = ji[2 * a] * t[0][b] + ji[2 * a + 1] * t[1][b];
        }
    h[0] = f[0];
    h[1] = f[1];
    h[2] = f[2];
    h[3] = f[3];
    h[4] = f[5];
    h[5] = f[6];
    h[6] = f[7];
    h[7] = f[10];
    h[8] = f[11];
    h[9] = f[15];
}

__device__ __forceinline__ void store_frame_moduli(double* C, int64_t S, int q, int64_t e, const double (&h)[10]) {
    double2* p = reinterpret_cast<double2*>(C) + (int64_t)(q * 5) * S + e;
#pragma unroll
    for (int k = 0; k < 5; ++k) __stcs(p + k * S, make_double2(h[2 * k], h[2 * k + 1]));
}
__device__ __forceinline__ void store_frame_moduli(float* C, int64_t S, int q, int64_t e, const double (&h)[10]) {
    float* base = C + (int64_t)q * 10 * S;
    __stcs(reinterpret_cast<float4*>(base) + e, make_float4((float)h[0], (float)h[1], (float)h[2], (float)h[3]));
    __stcs(reinterpret_cast<float4*>(base + 4 * S) + e, make_float4((float)h[4], (float)h[5], (float)h[6], (float)h[7]));
    __stcs(reinterpret_cast<float2*>(base + 8 * S) + e, make_float2((float)h[8], (float)h[9]));
}

// ------------------------------------------------------------------------------------------
// kernel (a) in the frame: moduli, element diagonals into fe (pairs) and the 2 x 2 coupling into fb
// ------------------------------------------------------------------------------------------
template <int NEN, int NQ, typename CT, bool GEN>
__global__ void __launch_bounds__(FrameCfg<NEN, NQ>::NT, GEN ? 1 : FrameCfg<NEN, NQ>::MINB)
k_frame_moduli(Mesh m, const double* __restrict__ frame, RefGrad<NEN, NQ> rg, const double* __restrict__ u,
               const double* __restrict__ theta, MatArg mat, CT* __restrict__ Cout, double* __restrict__ fe,
               double* __restrict__ fb) {
    constexpr int EB = FrameCfg<NEN, NQ>::EB;
    __shared__ FrameShared<NEN, NQ, double> sh;
    const int lane = threadIdx.x % EB, q = threadIdx.x / EB;
    const RefRow<NEN, double> row(rg, q);
    const int64_t S = m.stride, n_tiles = (m.n_el + EB - 1) / EB;
    const double2* u2 = reinterpret_cast<const double2*>(u);
    double2* fe2 = reinterpret_cast<double2*>(fe);
    const int64_t step = (int64_t)gridDim.x * EB;
    const auto load_u = [&](int n) { return __ldg(u2 + n); };
    ConnRow<NEN, NQ> conn;
    NodeRow<NEN, NQ, double> un;
    FramePoint next;
    int64_t e = (int64_t)blockIdx.x * EB + lane;
    conn.load(m, e, e < m.n_el, q);
    next.load(m, frame, theta, FramePoint::orig_of(m, e), e, e < m.n_el, q);
    un.template gather<false>(conn, load_u);
    int orig = FramePoint::orig_of(m, e + step);
    conn.load(m, e + step, e + step < m.n_el, q);
    for (int64_t tile = blockIdx.x; tile < n_tiles; tile += gridDim.x, e += step) {
        const bool live = e < m.n_el;
        un.store(sh.vs, q, lane);
        __syncthreads();
        const FramePoint pt_now = next;
        next.load(m, frame, theta, orig, e + step, e + step < m.n_el, q);
        un.template gather<false>(conn, load_u);
        orig = FramePoint::orig_of(m, e + 2 * step);
        conn.load(m, e + 2 * step, e + 2 * step < m.n_el, q);
        const double (&ji)[4] = pt_now.ji;
        const double w = pt_now.w, th = pt_now.th;
        double H[4], F[4], h[10], pe[DFEA_MAX_MAT_PARAMS];
        frame_gradient<NEN, NQ, double>(row, lane, sh.vs, H);
        frame_deformation(H, ji, F);
        frame_params(mat, th, pe);
        if constexpr (GEN) {
            double c[16];
            gen_moduli(mat.m.model, F, pe, w, c);
            pull_back(c, ji, h);
        } else {
            const NHPoint pt = nh_point(F);
            nh_frame_moduli(pt, pe[0], pe[1], w, ji, h);
        }
        if (Cout != nullptr && live) store_frame_moduli(Cout, S, q, e, h);
        if (fe != nullptr) {
            // e_k^T K_e e_k of the unit DOFs of node a, summed over the Gauss points
#pragma unroll
            for (int a = 0; a < NEN; ++a) {
                const double r0 = row.g[a][0], r1 = row.g[a][1];
                sh.red[q][a][lane] = make_double2(h[0] * r0 * r0 + 2.0 * h[1] * r0 * r1 + h[4] * r1 * r1,
                                                  h[7] * r0 * r0 + 2.0 * h[8] * r0 * r1 + h[9] * r1 * r1);
            }
            __syncthreads();
            frame_reduce<NEN, NQ, double>(e, live, q, lane, sh.red,
                                          [&](int a, int64_t el, double2 s) { fe2[(int64_t)a * S + el] = s; });
            if (fb != nullptr) {
                __syncthreads();
#pragma unroll
                for (int a = 0; a < NEN; ++a) {
                    const double r0 = row.g[a][0], r1 = row.g[a][1];
                    sh.red[q][a][lane] = make_double2(h[2] * r0 * r0 + (h[3] + h[5]) * r0 * r1 + h[6] * r1 * r1, 0.0);
                }
                __syncthreads();
                frame_reduce<NEN, NQ, double>(e, live, q, lane, sh.red,
                                              [&](int a, int64_t el, double2 s) { fb[(int64_t)a * S + el] = s.x; });
            }
        }
        __syncthreads();
    }
}

// node pass: diag = where(m > 0, max(sum, 1e-6), 1) and, with fb, the inverse 2 x 2 blocks of nodal block-Jacobi
// (B = M B_K M + (I - M) + 1e-12 I) as (Binv00, Binv01, Binv11, 0)
__global__ void __launch_bounds__(kThreads)
k_frame_node_diag(Mesh m, const int32_t* __restrict__ inc_ptr, const int32_t* __restrict__ inc,
                  const double* fe, const double* fb, double* __restrict__ diag,
                  double* __restrict__ blocks) {
    grid_dependency_wait();
    grid_dependents_launch();
    const double2* fe2 = reinterpret_cast<const double2*>(fe);
    for (int64_t n = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; n < m.n_nodes; n += (int64_t)gridDim.x * blockDim.x) {
        const int fix = m.node_fix[n];
        const double2 d = node_sum<double>(inc_ptr, inc, fe2, n);
        if (blocks != nullptr) {
            double c = 0.0;
            for (int j = inc_ptr[n]; j < inc_ptr[n + 1]; ++j) c += load_fresh(fb + inc[j]);
            const bool fx = fix & 1, fy = fix & 2;
            const double a00 = (fx ? 1.0 : d.x) + 1e-12, a11 = (fy ? 1.0 : d.y) + 1e-12;
            const double a01 = (fx || fy) ? 0.0 : c;
            const double det = a00 * a11 - a01 * a01;
            double2* b2 = reinterpret_cast<double2*>(blocks);
            b2[2 * n] = make_double2(a11 / det, -a01 / det);
            b2[2 * n + 1] = make_double2(a00 / det, 0.0);
        }
        reinterpret_cast<double2*>(diag)[n] = make_double2((fix & 1) ? 1.0 : fmax(d.x, 1e-6), (fix & 2) ? 1.0 : fmax(d.y, 1e-6));
    }
}

// ------------------------------------------------------------------------------------------
// residual: element pass (results into fe, energy partials per block), node pass (R, |R|^2, energy)
// ------------------------------------------------------------------------------------------
template <int NEN, int NQ, bool ENERGY, bool GEN>
__global__ void __launch_bounds__(FrameCfg<NEN, NQ>::NT, GEN ? 1 : FrameCfg<NEN, NQ>::MINB)
k_frame_residual(Mesh m, const double* __restrict__ frame, RefGrad<NEN, NQ> rg, const double* __restrict__ u,
                 const double* __restrict__ theta, MatArg mat, double* __restrict__ fe, double* __restrict__ part,
                 unsigned* __restrict__ ticket) {
    constexpr int EB = FrameCfg<NEN, NQ>::EB, NT = FrameCfg<NEN, NQ>::NT;
    __shared__ FrameShared<NEN, NQ, double> sh;
    const int lane = threadIdx.x % EB, q = threadIdx.x / EB;
    const RefRow<NEN, double> row(rg, q);
    const int64_t S = m.stride, n_tiles = (m.n_el + EB - 1) / EB;
    const double2* u2 = reinterpret_cast<const double2*>(u);
    double2* fe2 = reinterpret_cast<double2*>(fe);
    double energy = 0.0;
    if (blockIdx.x == 0 && threadIdx.x == 0 && ticket != nullptr) *ticket = 0u;  // of the node pass that follows
    const int64_t step = (int64_t)gridDim.x * EB;
    const auto load_u = [&](int n) { return __ldg(u2 + n); };
    ConnRow<NEN, NQ> conn;
    NodeRow<NEN, NQ, double> un;
    FramePoint next;
    int64_t e = (int64_t)blockIdx.x * EB + lane;
    conn.load(m, e, e < m.n_el, q);
    next.load(m, frame, theta, FramePoint::orig_of(m, e), e, e < m.n_el, q);
    un.template gather<false>(conn, load_u);
    int orig = FramePoint::orig_of(m, e + step);
    conn.load(m, e + step, e + step < m.n_el, q);
    for (int64_t tile = blockIdx.x; tile < n_tiles; tile += gridDim.x, e += step) {
        const bool live = e < m.n_el;
        un.store(sh.vs, q, lane);
        __syncthreads();
        const FramePoint pt_now = next;
        next.load(m, frame, theta, orig, e + step, e + step < m.n_el, q);
        un.template gather<false>(conn, load_u);
        orig = FramePoint::orig_of(m, e + 2 * step);
        conn.load(m, e + 2 * step, e + 2 * step < m.n_el, q);
        const double (&ji)[4] = pt_now.ji;
        const double w = pt_now.w, th = pt_now.th;
        double H[4], F[4], P[4], pe[DFEA_MAX_MAT_PARAMS];
        frame_gradient<NEN, NQ, double>(row, lane, sh.vs, H);
        frame_deformation(H, ji, F);
        frame_params(mat, th, pe);
        double psi;
        if constexpr (GEN) {
            psi = gen_stress(mat.m.model, F, pe, P);
        } else {
            const NHPoint pt = nh_point(F);
            nh_stress(F, pt, pe[0], pe[1], P);
            psi = ENERGY ? nh_energy(F, pt, pe[0], pe[1]) : 0.0;
        }
        if (ENERGY && live) energy += w * psi;
        // Phat_ib = w P_iJ Jinv_bJ
        const double p0 = w * (P[0] * ji[0] + P[1] * ji[1]), p1 = w * (P[0] * ji[2] + P[1] * ji[3]);
        const double p2 = w * (P[2] * ji[0] + P[3] * ji[1]), p3 = w * (P[2] * ji[2] + P[3] * ji[3]);
#pragma unroll
        for (int a = 0; a < NEN; ++a) {
            const double r0 = row.g[a][0], r1 = row.g[a][1];
            sh.red[q][a][lane] = make_double2(p0 * r0 + p1 * r1, p2 * r0 + p3 * r1);
        }
        __syncthreads();
        frame_reduce<NEN, NQ, double>(e, live, q, lane, sh.red,
                                      [&](int a, int64_t el, double2 s) { fe2[(int64_t)a * S + el] = s; });
        if (NQ == 1) __syncthreads();
    }
    if (ENERGY) {
        const double s = block_sum<NT>(energy);
        if (threadIdx.x == 0) part[blockIdx.x] = s;
    }
}

// The internal force summed over the fixed DOFs (support reactions), without storing it
__global__ void __launch_bounds__(kThreads)
k_frame_node_reactions(Mesh m, const int32_t* __restrict__ inc_ptr, const int32_t* __restrict__ inc,
                       const double* fe, const uint8_t* __restrict__ fixed, RedSite site, double* __restrict__ out) {
    grid_dependency_wait();
    grid_dependents_launch();
    const double2* fe2 = reinterpret_cast<const double2*>(fe);
    double rx = 0.0, ry = 0.0;
    for (int64_t n = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; n < m.n_nodes; n += (int64_t)gridDim.x * blockDim.x) {
        const bool fx = fixed[2 * n], fy = fixed[2 * n + 1];
        if (!fx && !fy) continue;
        const double2 s = node_sum<double>(inc_ptr, inc, fe2, n);
        if (fx) rx += s.x;
        if (fy) ry += s.y;
    }
    const double vals[2] = {block_sum<kThreads>(rx), block_sum<kThreads>(ry)};
    double tot[2];
    if (last_block_sum<kThreads, 2>(vals, site, tot) && threadIdx.x == 0) {
        out[0] = tot[0];
        out[1] = tot[1];
    }
}

// MASK: R = m (sum - lf f); else the unmasked sum.  NORM: |R|^2 into out_norm2 and the energy partials of the
// element pass (n_part of them) into out_energy by the last block.
template <bool MASK, bool NORM>
__global__ void __launch_bounds__(kThreads)
k_frame_node_residual(Mesh m, const int32_t* __restrict__ inc_ptr, const int32_t* __restrict__ inc,
                      const double* fe, const double* __restrict__ f, double lf, double* __restrict__ R,
                      RedSite site, double* __restrict__ out_norm2, const double* part, int n_part,
                      double* __restrict__ out_energy) {
    grid_dependency_wait();
    grid_dependents_launch();
    const double2* fe2 = reinterpret_cast<const double2*>(fe);
    const double2* f2 = reinterpret_cast<const double2*>(f);
    double rr = 0.0;
    for (int64_t n = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; n < m.n_nodes; n += (int64_t)gridDim.x * blockDim.x) {
        double2 s = node_sum<double>(inc_ptr, inc, fe2, n);
        if (MASK) {
            const int fix = m.node_fix[n];
            const double2 t = f ? f2[n] : make_double2(0.0, 0.0);
            s.x = (fix & 1) ? 0.0 : s.x - lf * t.x;
            s.y = (fix & 2) ? 0.0 : s.y - lf * t.y;
        }
        reinterpret_cast<double2*>(R)[n] = s;
        if (NORM) rr += s.x * s.x + s.y * s.y;
    }
    if (NORM) {
        const double vals[1] = {block_sum<kThreads>(rr)};
        double tot[1];
        if (last_block_sum<kThreads, 1>(vals, site, tot)) {
            if (threadIdx.x == 0 && out_norm2) *out_norm2 = tot[0];
            if (out_energy) {
                double E = 0.0;
                for (int i = threadIdx.x; i < n_part; i += kThreads) E += load_fresh(part + i);
                E = block_sum<kThreads>(E);
                if (threadIdx.x == 0) *out_energy = E;
            }
        }
    }
}

// ------------------------------------------------------------------------------------------
// kernel (d) in the frame: g_e = -lambda_e . f_e(u; slope)
// ------------------------------------------------------------------------------------------
template <int NEN, int NQ, bool GEN>
__global__ void __launch_bounds__(FrameCfg<NEN, NQ>::NT, GEN ? 1 : FrameCfg<NEN, NQ>::MINB)
k_frame_sensitivity(Mesh m, const double* __restrict__ frame, RefGrad<NEN, NQ> rg, const double* __restrict__ u,
                    const double* __restrict__ lam, MatArg mat, double* __restrict__ g) {
    constexpr int EB = FrameCfg<NEN, NQ>::EB;
    __shared__ double2 us[NEN][EB], ls[NEN][EB];
    __shared__ double red[NQ][EB];
    const int lane = threadIdx.x % EB, q = threadIdx.x / EB;
    const RefRow<NEN, double> row(rg, q);
    const int64_t S = m.stride, n_tiles = (m.n_el + EB - 1) / EB;
    const double2* u2 = reinterpret_cast<const double2*>(u);
    const double2* l2 = reinterpret_cast<const double2*>(lam);
    double pe[DFEA_MAX_MAT_PARAMS];
    // d p_e / d theta_e: the scalable parameters' nominal values, zero for the other prefactors
    if (mat.p != nullptr) {
        const int n = material_n_params(mat.m.model);
        const unsigned linear = material_linear_mask(mat.m.model);
#pragma unroll
        for (int k = 0; k < DFEA_MAX_MAT_PARAMS; ++k)
            pe[k] = k < n ? ((((linear >> k) & 1u) && !__ldg(mat.scalable + k)) ? 0.0 : __ldg(mat.p + k)) : 0.0;
    } else {
#pragma unroll
        for (int k = 0; k < DFEA_MAX_MAT_PARAMS; ++k) pe[k] = mat.m.p[k];
    }
    const int64_t step = (int64_t)gridDim.x * EB;
    const auto load_l = [&](int n) { return __ldg(l2 + n); };
    const auto load_u = [&](int n) { return __ldg(u2 + n); };
    ConnRow<NEN, NQ> conn;
    NodeRow<NEN, NQ, double> un, ln;
    FramePoint next;
    int64_t e = (int64_t)blockIdx.x * EB + lane;
    conn.load(m, e, e < m.n_el, q);
    next.load(m, frame, nullptr, 0, e, e < m.n_el, q);
    un.template gather<false>(conn, load_u);
    ln.template gather<true>(conn, load_l);
    conn.load(m, e + step, e + step < m.n_el, q);
    for (int64_t tile = blockIdx.x; tile < n_tiles; tile += gridDim.x, e += step) {
        const bool live = e < m.n_el;
        un.store(us, q, lane);
        ln.store(ls, q, lane);
        __syncthreads();
        const FramePoint pt_now = next;
        next.load(m, frame, nullptr, 0, e + step, e + step < m.n_el, q);
        un.template gather<false>(conn, load_u);
        ln.template gather<true>(conn, load_l);
        conn.load(m, e + 2 * step, e + 2 * step < m.n_el, q);
        const double (&ji)[4] = pt_now.ji;
        const double w = pt_now.w;
        double H[4], L[4], F[4], P[4];
        frame_gradient<NEN, NQ, double>(row, lane, us, H);
        frame_gradient<NEN, NQ, double>(row, lane, ls, L);
        frame_deformation(H, ji, F);
        if constexpr (GEN) {
            gen_stress(mat.m.model, F, pe, P);
        } else {
            const NHPoint pt = nh_point(F);
            nh_stress(F, pt, pe[0], pe[1], P);
        }
        // w P_iJ (L Jinv)_iJ
        red[q][lane] = w * (P[0] * (L[0] * ji[0] + L[1] * ji[2]) + P[1] * (L[0] * ji[1] + L[1] * ji[3]) +
                            P[2] * (L[2] * ji[0] + L[3] * ji[2]) + P[3] * (L[2] * ji[1] + L[3] * ji[3]));
        __syncthreads();
        if (q == 0 && live) {
            double s = red[0][lane];
#pragma unroll
            for (int k = 1; k < NQ; ++k) s += red[k][lane];
            g[__ldg(m.orig + e)] = -s;
        }
        __syncthreads();
    }
}

// ------------------------------------------------------------------------------------------
// post-processing in the frame: the seven element rows
// ------------------------------------------------------------------------------------------
template <int NEN, int NQ, bool GEN>
__global__ void __launch_bounds__(FrameCfg<NEN, NQ>::NT, GEN ? 1 : FrameCfg<NEN, NQ>::MINB)
k_frame_fields(Mesh m, const double* __restrict__ frame, RefGrad<NEN, NQ> rg, const double* __restrict__ u,
               const double* __restrict__ theta, MatArg mat, double* __restrict__ out, double* __restrict__ part) {
    constexpr int EB = FrameCfg<NEN, NQ>::EB, NT = FrameCfg<NEN, NQ>::NT;
    double energy = 0.0, min_J = INFINITY;  // of this block's elements: sum of psi area, smallest mean J (a NaN wins)
    __shared__ double2 us[NEN][EB];
    __shared__ double red[NQ][7][EB];
    const int lane = threadIdx.x % EB, q = threadIdx.x / EB;
    const RefRow<NEN, double> row(rg, q);
    const int64_t S = m.stride, n_el = m.n_el, n_tiles = (n_el + EB - 1) / EB;
    const double2* u2 = reinterpret_cast<const double2*>(u);
    const int64_t step = (int64_t)gridDim.x * EB;
    const auto load_u = [&](int n) { return __ldg(u2 + n); };
    ConnRow<NEN, NQ> conn;
    NodeRow<NEN, NQ, double> un;
    FramePoint next;
    int64_t e = (int64_t)blockIdx.x * EB + lane;
    conn.load(m, e, e < m.n_el, q);
    next.load(m, frame, theta, FramePoint::orig_of(m, e), e, e < m.n_el, q);
    un.template gather<false>(conn, load_u);
    int orig = FramePoint::orig_of(m, e + step);
    conn.load(m, e + step, e + step < m.n_el, q);
    for (int64_t tile = blockIdx.x; tile < n_tiles; tile += gridDim.x, e += step) {
        const bool live = e < m.n_el;
        un.store(us, q, lane);
        __syncthreads();
        const FramePoint pt_now = next;
        next.load(m, frame, theta, orig, e + step, e + step < m.n_el, q);
        un.template gather<false>(conn, load_u);
        orig = FramePoint::orig_of(m, e + 2 * step);
        conn.load(m, e + 2 * step, e + 2 * step < m.n_el, q);
        const double (&ji)[4] = pt_now.ji;
        const double w = pt_now.w, th = pt_now.th;
        double H[4], F[4], pe[DFEA_MAX_MAT_PARAMS];
        frame_gradient<NEN, NQ, double>(row, lane, us, H);
        frame_deformation(H, ji, F);
        frame_params(mat, th, pe);
        double J, sxx, syy, sxy, szz, psi;
        if constexpr (GEN) {
            double P[5];
            psi = gen_stress3(mat.m.model, F, pe, P);
            J = F[0] * F[3] - F[1] * F[2];
            const double iJ = 1.0 / J;
            sxx = (P[0] * F[0] + P[1] * F[1]) * iJ;
            syy = (P[2] * F[2] + P[3] * F[3]) * iJ;
            sxy = (P[0] * F[2] + P[1] * F[3]) * iJ;
            szz = P[4] * iJ;
        } else {
            const double mu = pe[0], lam = pe[1];
            const NHPoint pt = nh_point(F);
            const double iJ = 1.0 / pt.J, c = lam * pt.lnJ;
            const double b00 = F[0] * F[0] + F[1] * F[1], b11 = F[2] * F[2] + F[3] * F[3], b01 = F[0] * F[2] + F[1] * F[3];
            J = pt.J;
            sxx = (mu * (b00 - 1.0) + c) * iJ;
            syy = (mu * (b11 - 1.0) + c) * iJ;
            sxy = (mu * b01) * iJ;
            szz = c * iJ;
            psi = nh_energy(F, pt, mu, lam);
        }
        const double v[7] = {w, w * J, w * sxx, w * syy, w * sxy, w * szz, w * psi};
#pragma unroll
        for (int k = 0; k < 7; ++k) red[q][k][lane] = v[k];
        __syncthreads();
        if (q == 0 && live) {
            double acc[7];
#pragma unroll
            for (int k = 0; k < 7; ++k) {
                acc[k] = red[0][k][lane];
#pragma unroll
                for (int p = 1; p < NQ; ++p) acc[k] += red[p][k][lane];
            }
            const double area = acc[0];
            const double mJ = acc[1] / area, a = acc[2] / area, b = acc[3] / area, c = acc[4] / area, z = acc[5] / area,
                         mpsi = acc[6] / area;
            const double mises = sqrt(0.5 * ((a - b) * (a - b) + (b - z) * (b - z) + (z - a) * (z - a)) + 3.0 * c * c);
            const int64_t oe = __ldg(m.orig + e);
            out[0 * n_el + oe] = area;
            out[1 * n_el + oe] = mJ;
            out[2 * n_el + oe] = a;
            out[3 * n_el + oe] = b;
            out[4 * n_el + oe] = c;
            out[5 * n_el + oe] = mises;
            out[6 * n_el + oe] = mpsi;
            energy += mpsi * area;
            if (mJ < min_J || mJ != mJ) min_J = (min_J != min_J) ? min_J : mJ;
        }
        __syncthreads();
    }
    if (part != nullptr) {
        const double E = block_sum<NT>(energy);
        __shared__ double mins[NT / 32];
        auto take = [](double a, double b) { return (b < a || b != b) ? ((a != a) ? a : b) : a; };
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) min_J = take(min_J, __shfl_down_sync(0xffffffffu, min_J, o));
        if ((threadIdx.x & 31) == 0) mins[threadIdx.x >> 5] = min_J;
        __syncthreads();
        if (threadIdx.x == 0) {
            for (int w = 1; w < NT / 32; ++w) min_J = take(min_J, mins[w]);
            part[blockIdx.x] = E;
            part[kMaxBlocks + blockIdx.x] = min_J;
        }
    }
}

// nodal post-processing: the means of the six element rows over a node's elements (incidence order) and |u|, rows
// 0 .. 6 of out; block 0 adds the element pass's energy partials and takes its smallest J
__global__ void __launch_bounds__(kThreads)
k_frame_node_fields(Mesh m, const int32_t* __restrict__ inc_ptr, const int32_t* __restrict__ inc,
                    const double* elem, const double* __restrict__ u, double* __restrict__ out,
                    const double* part, int n_part, double* __restrict__ scal) {
    grid_dependency_wait();
    grid_dependents_launch();
    const int64_t S = m.stride, n_el = m.n_el, N = m.n_nodes;
    for (int64_t n = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; n < N; n += (int64_t)gridDim.x * blockDim.x) {
        double acc[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
        const int j0 = inc_ptr[n], j1 = inc_ptr[n + 1];
        for (int j = j0; j < j1; ++j) {
            const int64_t oe = m.orig[inc[j] % S];
#pragma unroll
            for (int k = 0; k < 6; ++k) acc[k] += load_fresh(elem + (k + 1) * n_el + oe);
        }
        const double cnt = (j1 > j0) ? (double)(j1 - j0) : 1.0;
#pragma unroll
        for (int k = 0; k < 6; ++k) out[k * N + n] = acc[k] / cnt;
        const double2 un = reinterpret_cast<const double2*>(u)[n];
        out[6 * N + n] = sqrt(un.x * un.x + un.y * un.y);
    }
    if (blockIdx.x == 0) {
        double E = 0.0, low = INFINITY;
        auto take = [](double a, double b) { return (b < a || b != b) ? ((a != a) ? a : b) : a; };
        for (int i = threadIdx.x; i < n_part; i += kThreads) {
            E += load_fresh(part + i);
            low = take(low, load_fresh(part + kMaxBlocks + i));
        }
        E = block_sum<kThreads>(E);
        __shared__ double lows[kThreads];
        lows[threadIdx.x] = low;
        __syncthreads();
        if (threadIdx.x == 0) {
            for (int i = 1; i < kThreads; ++i) low = take(low, lows[i]);
            scal[0] = E;
            scal[1] = low;
        }
    }
}

// ------------------------------------------------------------------------------------------
// physical moduli from the reference-frame ones: C = Jinv^-1 h Jinv^-T (16 FP64 entries per Gauss point)
// ------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(kThreads)
k_frame_push_forward(int64_t n_el, int64_t S, int nq, const double* __restrict__ frame, const double* __restrict__ H,
                     double* __restrict__ C) {
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < n_el * nq; t += (int64_t)gridDim.x * blockDim.x) {
        const int q = (int)(t / n_el);
        const int64_t e = t - q * n_el;
        double ji[4], c[16];
        load_jinv(frame, S, q, e, ji);
        const double det = ji[0] * ji[3] - ji[1] * ji[2];
        // J_Ja = (Jinv^-1): rows J, columns a
        const double J[4] = {ji[3] / det, -ji[1] / det, -ji[2] / det, ji[0] / det};
        const double2* p = reinterpret_cast<const double2*>(H) + (int64_t)(q * 5) * S + e;
        const double2 h0 = p[0], h1 = p[S], h2 = p[2 * S], h3 = p[3 * S], h4 = p[4 * S];
        const double f[16] = {h0.x, h0.y, h1.x, h1.y, h0.y, h2.x, h2.y, h3.x, h1.x, h2.y, h3.y, h4.x, h1.y, h3.x, h4.x, h4.y};
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
            for (int k = 0; k < 2; ++k) {
                double s[2][2];
#pragma unroll
                for (int a = 0; a < 2; ++a)
#pragma unroll
                    for (int L = 0; L < 2; ++L)
                        s[a][L] = f[(2 * i + a) * 4 + 2 * k] * J[2 * L] + f[(2 * i + a) * 4 + 2 * k + 1] * J[2 * L + 1];
#pragma unroll
                for (int Jj = 0; Jj < 2; ++Jj)
#pragma unroll
                    for (int L = 0; L < 2; ++L) c[(2 * i + Jj) * 4 + 2 * k + L] = J[2 * Jj] * s[0][L] + J[2 * Jj + 1] * s[1][L];
            }
        store_moduli(C, S, q, e, c);
    }
}

// scratch of the frame entry points: element results (pairs), couplings, energy and norm partials, ticket
struct FrameWork {
    double *fe, *fb, *part, *norm_part;
    unsigned* ticket;
    static int64_t up(int64_t x) { return (x + 255) / 256 * 256; }
    static int64_t bytes(const dfea_mesh_view& v) {
        return up((int64_t)v.nen * v.stride * 16) + up((int64_t)v.nen * v.stride * 8) + 3 * kMaxBlocks * 8 + 256;
    }
    FrameWork(const dfea_mesh_view& v, void* base) {
        char* p = static_cast<char*>(base);
        fe = reinterpret_cast<double*>(p);
        p += up((int64_t)v.nen * v.stride * 16);
        fb = reinterpret_cast<double*>(p);
        p += up((int64_t)v.nen * v.stride * 8);
        part = reinterpret_cast<double*>(p);
        norm_part = part + kMaxBlocks;
        ticket = reinterpret_cast<unsigned*>(norm_part + 2 * kMaxBlocks);
    }
};

template <int NEN, int NQ>
static int frame_grid(int64_t n_el) {
    const int64_t tiles = (n_el + FrameCfg<NEN, NQ>::EB - 1) / FrameCfg<NEN, NQ>::EB;
    return (int)(tiles < 1 ? 1 : (tiles > kMaxBlocks ? kMaxBlocks : tiles));
}

static int validate_frame(const dfea_mesh_view* mesh, const char* what) {
    int rc = validate_mesh(mesh, false);
    if (rc) return rc;
    if (!mesh->frame) return set_error(DFEA_ERR_INVALID, "%s: the mesh has no frame (dfea_mesh_frame)", what);
    return DFEA_OK;
}

static int validate_frame_material(const dfea_material* mat, const double* p, const uint8_t* scalable, MatArg* out,
                                   const char* what) {
    if (!mat) return set_error(DFEA_ERR_INVALID, "%s: material is NULL", what);
    if ((p == nullptr) != (scalable == nullptr))
        return set_error(DFEA_ERR_INVALID, "%s: give both device parameter arrays or none", what);
    if (p) {
        if (material_n_params(mat->model) == 0)
            return set_error(DFEA_ERR_UNSUPPORTED, "material model %d is not built", mat->model);
    } else {
        const int rc = validate_material(mat);
        if (rc) return rc;
    }
    *out = MatArg{*mat, p, scalable};
    return DFEA_OK;
}

static bool al16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

template <typename Fn>
static int dispatch_gen(int model, Fn&& fn) {
    if (model == DFEA_MAT_NEO_HOOKEAN) return fn(std::false_type{});
    return fn(std::true_type{});
}

}  // namespace dfea

using namespace dfea;

extern "C" int dfea_mesh_frame(const dfea_mesh_view* mesh, const double* nodes, double* frame_out, double* check,
                               void* stream) {
    int rc = validate_mesh(mesh, false);
    if (rc) return rc;
    if (!nodes || !frame_out || !check) return set_error(DFEA_ERR_INVALID, "dfea_mesh_frame: NULL pointer");
    if (!al16(frame_out)) return set_error(DFEA_ERR_INVALID, "dfea_mesh_frame: frame_out must be 16-byte aligned");
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    if ((rc = check_cuda(cudaMemsetAsync(check, 0, 3 * sizeof(double), s), "cudaMemsetAsync"))) return rc;
    rc = dispatch_element(mesh->nen, mesh->n_q, [&](auto nen_c, auto nq_c) -> int {
        constexpr int NEN = decltype(nen_c)::value, NQ = decltype(nq_c)::value;
        k_frame<NEN, NQ><<<grid_for(mesh->stride * NQ, 128, 8), 128, 0, s>>>(kernel_mesh(*mesh), ref_grad_of<NEN, NQ>(*mesh),
                                                                             ref_pinv_of<NEN, NQ>(*mesh), nodes, frame_out, check);
        return DFEA_OK;
    });
    if (rc) return rc;
    note_launches(1);
    return launch_check("dfea_mesh_frame");
}

extern "C" int64_t dfea_frame_work_bytes(const dfea_mesh_view* mesh) { return mesh ? FrameWork::bytes(*mesh) : -1; }

extern "C" int dfea_frame_moduli(const dfea_mesh_view* mesh, const double* u, const double* theta,
                                 const dfea_material* material, const double* mat_p, const uint8_t* mat_scalable,
                                 void* moduli, int32_t moduli_dtype, double* diag, double* blocks, void* work, void* stream) {
    int rc = validate_frame(mesh, "dfea_frame_moduli");
    MatArg mat;
    if (rc || (rc = validate_frame_material(material, mat_p, mat_scalable, &mat, "dfea_frame_moduli"))) return rc;
    if (!u || !theta || (!moduli && !diag)) return set_error(DFEA_ERR_INVALID, "dfea_frame_moduli: NULL pointer");
    if (blocks && !diag) return set_error(DFEA_ERR_INVALID, "dfea_frame_moduli: blocks need diag");
    if (moduli_dtype != DFEA_F64REF && moduli_dtype != DFEA_F32REF)
        return set_error(DFEA_ERR_INVALID, "dfea_frame_moduli: the moduli are DFEA_F64REF or DFEA_F32REF");
    if (diag && (!work || !mesh->node_elem_ptr || !mesh->node_elem))
        return set_error(DFEA_ERR_INVALID, "dfea_frame_moduli: the diagonal needs work and the node incidence");
    if (!al16(u) || !al16(moduli) || !al16(diag) || !al16(blocks) || !al16(work))
        return set_error(DFEA_ERR_INVALID, "dfea_frame_moduli: buffers must be 16-byte aligned");
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const Mesh m = kernel_mesh(*mesh);
    FrameWork w(*mesh, work);
    double *fe = diag ? w.fe : nullptr, *fb = blocks ? w.fb : nullptr;
    rc = dispatch_element(mesh->nen, mesh->n_q, [&](auto nen_c, auto nq_c) -> int {
        constexpr int NEN = decltype(nen_c)::value, NQ = decltype(nq_c)::value;
        return dispatch_gen(mat.m.model, [&](auto gen_c) -> int {
            constexpr bool GEN = decltype(gen_c)::value;
            const int grid = frame_grid<NEN, NQ>(mesh->n_el);
            const RefGrad<NEN, NQ> rg = ref_grad_of<NEN, NQ>(*mesh);
            if (moduli_dtype == DFEA_F64REF)
                k_frame_moduli<NEN, NQ, double, GEN><<<grid, FrameCfg<NEN, NQ>::NT, 0, s>>>(
                    m, mesh->frame, rg, u, theta, mat, static_cast<double*>(moduli), fe, fb);
            else
                k_frame_moduli<NEN, NQ, float, GEN><<<grid, FrameCfg<NEN, NQ>::NT, 0, s>>>(
                    m, mesh->frame, rg, u, theta, mat, static_cast<float*>(moduli), fe, fb);
            return DFEA_OK;
        });
    });
    if (rc) return rc;
    note_launches(1);
    if (diag) {
        LaunchOpts pdl;
        pdl.pdl = true;
        if ((rc = launch_kernel(k_frame_node_diag, dim3(grid_for(mesh->n_nodes, kThreads, 8)), dim3(kThreads), 0, s, pdl, m,
                                mesh->node_elem_ptr, mesh->node_elem, (const double*)fe, (const double*)fb, diag, blocks)))
            return rc;
        note_launches(1);
    }
    return launch_check("dfea_frame_moduli");
}

// the element pass of the residual and the node pass that follows it
static int frame_residual(const dfea_mesh_view* mesh, const double* u, const double* theta, const MatArg& mat,
                          const double* f, double lf, double* R, double* out_norm2, double* out_energy, void* work,
                          bool mask, cudaStream_t s, const uint8_t* fixed = nullptr, double* reactions = nullptr) {
    const Mesh m = kernel_mesh(*mesh);
    FrameWork w(*mesh, work);
    int n_part = 0;
    int rc = dispatch_element(mesh->nen, mesh->n_q, [&](auto nen_c, auto nq_c) -> int {
        constexpr int NEN = decltype(nen_c)::value, NQ = decltype(nq_c)::value;
        return dispatch_gen(mat.m.model, [&](auto gen_c) -> int {
            constexpr bool GEN = decltype(gen_c)::value;
            const int grid = n_part = frame_grid<NEN, NQ>(mesh->n_el);
            const RefGrad<NEN, NQ> rg = ref_grad_of<NEN, NQ>(*mesh);
            if (out_energy)
                k_frame_residual<NEN, NQ, true, GEN><<<grid, FrameCfg<NEN, NQ>::NT, 0, s>>>(m, mesh->frame, rg, u, theta,
                                                                                           mat, w.fe, w.part, w.ticket);
            else
                k_frame_residual<NEN, NQ, false, GEN><<<grid, FrameCfg<NEN, NQ>::NT, 0, s>>>(m, mesh->frame, rg, u, theta,
                                                                                            mat, w.fe, w.part, w.ticket);
            return DFEA_OK;
        });
    });
    if (rc) return rc;
    LaunchOpts pdl;
    pdl.pdl = true;
    const dim3 grid(grid_for(mesh->n_nodes, kThreads, 8));
    const RedSite site{w.norm_part, w.ticket, nullptr};
    if (reactions)
        rc = launch_kernel(k_frame_node_reactions, grid, dim3(kThreads), 0, s, pdl, m, mesh->node_elem_ptr, mesh->node_elem,
                           (const double*)w.fe, fixed, site, reactions);
    else if (!mask)
        rc = launch_kernel(k_frame_node_residual<false, false>, grid, dim3(kThreads), 0, s, pdl, m, mesh->node_elem_ptr,
                           mesh->node_elem, (const double*)w.fe, f, lf, R, site, out_norm2, (const double*)w.part, n_part, out_energy);
    else if (out_norm2 || out_energy)
        rc = launch_kernel(k_frame_node_residual<true, true>, grid, dim3(kThreads), 0, s, pdl, m, mesh->node_elem_ptr,
                           mesh->node_elem, (const double*)w.fe, f, lf, R, site, out_norm2, (const double*)w.part, n_part, out_energy);
    else
        rc = launch_kernel(k_frame_node_residual<true, false>, grid, dim3(kThreads), 0, s, pdl, m, mesh->node_elem_ptr,
                           mesh->node_elem, (const double*)w.fe, f, lf, R, site, out_norm2, (const double*)w.part, n_part, out_energy);
    if (rc) return rc;
    note_launches(2);
    return launch_check("frame residual");
}

extern "C" int dfea_frame_residual(const dfea_mesh_view* mesh, const double* u, const double* theta,
                                   const dfea_material* material, const double* mat_p, const uint8_t* mat_scalable,
                                   const double* f, double load_factor, double* R, double* out_norm2, double* out_energy,
                                   void* work, void* stream) {
    int rc = validate_frame(mesh, "dfea_frame_residual");
    MatArg mat;
    if (rc || (rc = validate_frame_material(material, mat_p, mat_scalable, &mat, "dfea_frame_residual"))) return rc;
    if (!u || !R || !work || !mesh->node_elem_ptr || !mesh->node_elem)
        return set_error(DFEA_ERR_INVALID, "dfea_frame_residual: NULL pointer or no node incidence");
    if (!al16(u) || !al16(R) || !al16(f) || !al16(work))
        return set_error(DFEA_ERR_INVALID, "dfea_frame_residual: vectors must be 16-byte aligned");
    return frame_residual(mesh, u, theta, mat, f, load_factor, R, out_norm2, out_energy, work, true,
                          static_cast<cudaStream_t>(stream));
}

extern "C" int dfea_frame_internal_force(const dfea_mesh_view* mesh, const double* u, const double* theta,
                                         const dfea_material* material, const double* mat_p, const uint8_t* mat_scalable,
                                         double* R_int, void* work, void* stream) {
    int rc = validate_frame(mesh, "dfea_frame_internal_force");
    MatArg mat;
    if (rc || (rc = validate_frame_material(material, mat_p, mat_scalable, &mat, "dfea_frame_internal_force"))) return rc;
    if (!u || !R_int || !work || !mesh->node_elem_ptr || !mesh->node_elem)
        return set_error(DFEA_ERR_INVALID, "dfea_frame_internal_force: NULL pointer or no node incidence");
    if (!al16(u) || !al16(R_int) || !al16(work)) return set_error(DFEA_ERR_INVALID, "dfea_frame_internal_force: alignment");
    return frame_residual(mesh, u, theta, mat, nullptr, 0.0, R_int, nullptr, nullptr, work, false,
                          static_cast<cudaStream_t>(stream));
}

extern "C" int dfea_frame_reactions(const dfea_mesh_view* mesh, const double* u, const double* theta,
                                    const dfea_material* material, const double* mat_p, const uint8_t* mat_scalable,
                                    const uint8_t* fixed, double* reactions, void* work, void* stream) {
    int rc = validate_frame(mesh, "dfea_frame_reactions");
    MatArg mat;
    if (rc || (rc = validate_frame_material(material, mat_p, mat_scalable, &mat, "dfea_frame_reactions"))) return rc;
    if (!u || !fixed || !reactions || !work || !mesh->node_elem_ptr || !mesh->node_elem)
        return set_error(DFEA_ERR_INVALID, "dfea_frame_reactions: NULL pointer or no node incidence");
    if (!al16(u) || !al16(work)) return set_error(DFEA_ERR_INVALID, "dfea_frame_reactions: alignment");
    return frame_residual(mesh, u, theta, mat, nullptr, 0.0, nullptr, nullptr, nullptr, work, false,
                          static_cast<cudaStream_t>(stream), fixed, reactions);
}

extern "C" int dfea_frame_sensitivity(const dfea_mesh_view* mesh, const double* u, const double* lam,
                                      const dfea_material* material, const double* mat_p, const uint8_t* mat_scalable,
                                      double* g, void* stream) {
    int rc = validate_frame(mesh, "dfea_frame_sensitivity");
    MatArg mat;
    if (rc || (rc = validate_frame_material(material, mat_p, mat_scalable, &mat, "dfea_frame_sensitivity"))) return rc;
    const unsigned linear = material_linear_mask(material->model);
    const int n_par = material_n_params(material->model);
    if (mat.p) {
        // parameters on the device: only models whose every parameter is a prefactor need no look at the flags
        if (linear != (1u << n_par) - 1u)
            return set_error(DFEA_ERR_UNSUPPORTED, "dfea_frame_sensitivity: model %d needs its parameters on the host", material->model);
    } else {
        if (material->scalable & ~linear)
            return set_error(DFEA_ERR_UNSUPPORTED, "dfea_frame_sensitivity: theta scales a parameter that enters the energy "
                                                   "nonlinearly (scalable 0x%x, linear 0x%x)", material->scalable, linear);
        for (int k = 0; k < DFEA_MAX_MAT_PARAMS; ++k)
            if (((linear >> k) & 1u) && !((material->scalable >> k) & 1u)) mat.m.p[k] = 0.0;
    }
    if (!u || !lam || !g) return set_error(DFEA_ERR_INVALID, "dfea_frame_sensitivity: NULL pointer");
    if (!al16(u) || !al16(lam)) return set_error(DFEA_ERR_INVALID, "u and lambda must be 16-byte aligned");
    if (mesh->n_el == 0) return DFEA_OK;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    rc = dispatch_element(mesh->nen, mesh->n_q, [&](auto nen_c, auto nq_c) -> int {
        constexpr int NEN = decltype(nen_c)::value, NQ = decltype(nq_c)::value;
        return dispatch_gen(mat.m.model, [&](auto gen_c) -> int {
            constexpr bool GEN = decltype(gen_c)::value;
            k_frame_sensitivity<NEN, NQ, GEN><<<frame_grid<NEN, NQ>(mesh->n_el), FrameCfg<NEN, NQ>::NT, 0, s>>>(
                kernel_mesh(*mesh), mesh->frame, ref_grad_of<NEN, NQ>(*mesh), u, lam, mat, g);
            return DFEA_OK;
        });
    });
    if (rc) return rc;
    note_launches(1);
    return launch_check("dfea_frame_sensitivity");
}

static int frame_fields(const dfea_mesh_view* mesh, const double* u, const double* theta, const MatArg& mat,
                        double* elem_out, double* part, int* n_part, cudaStream_t s) {
    const int rc = dispatch_element(mesh->nen, mesh->n_q, [&](auto nen_c, auto nq_c) -> int {
        constexpr int NEN = decltype(nen_c)::value, NQ = decltype(nq_c)::value;
        return dispatch_gen(mat.m.model, [&](auto gen_c) -> int {
            constexpr bool GEN = decltype(gen_c)::value;
            const int grid = *n_part = frame_grid<NEN, NQ>(mesh->n_el);
            k_frame_fields<NEN, NQ, GEN><<<grid, FrameCfg<NEN, NQ>::NT, 0, s>>>(
                kernel_mesh(*mesh), mesh->frame, ref_grad_of<NEN, NQ>(*mesh), u, theta, mat, elem_out, part);
            return DFEA_OK;
        });
    });
    if (rc) return rc;
    note_launches(1);
    return launch_check("frame fields");
}

extern "C" int dfea_frame_fields(const dfea_mesh_view* mesh, const double* u, const double* theta,
                                 const dfea_material* material, const double* mat_p, const uint8_t* mat_scalable,
                                 double* elem_out, void* stream) {
    int rc = validate_frame(mesh, "dfea_frame_fields"), n_part;
    MatArg mat;
    if (rc || (rc = validate_frame_material(material, mat_p, mat_scalable, &mat, "dfea_frame_fields"))) return rc;
    if (!u || !elem_out) return set_error(DFEA_ERR_INVALID, "dfea_frame_fields: NULL pointer");
    if (!al16(u)) return set_error(DFEA_ERR_INVALID, "dfea_frame_fields: u must be 16-byte aligned");
    return frame_fields(mesh, u, theta, mat, elem_out, nullptr, &n_part, static_cast<cudaStream_t>(stream));
}

extern "C" int dfea_frame_all_fields(const dfea_mesh_view* mesh, const double* u, const double* theta,
                                     const dfea_material* material, const double* mat_p, const uint8_t* mat_scalable,
                                     double* elem_out, double* node_out, double* scal_out, void* work, void* stream) {
    int rc = validate_frame(mesh, "dfea_frame_all_fields"), n_part = 0;
    MatArg mat;
    if (rc || (rc = validate_frame_material(material, mat_p, mat_scalable, &mat, "dfea_frame_all_fields"))) return rc;
    if (!u || !elem_out || !node_out || !scal_out || !work || !mesh->node_elem_ptr || !mesh->node_elem)
        return set_error(DFEA_ERR_INVALID, "dfea_frame_all_fields: NULL pointer or no node incidence");
    if (!al16(u) || !al16(work)) return set_error(DFEA_ERR_INVALID, "dfea_frame_all_fields: alignment");
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    FrameWork w(*mesh, work);
    if ((rc = frame_fields(mesh, u, theta, mat, elem_out, w.part, &n_part, s))) return rc;
    LaunchOpts pdl;
    pdl.pdl = true;
    if ((rc = launch_kernel(k_frame_node_fields, dim3(grid_for(mesh->n_nodes, kThreads, 8)), dim3(kThreads), 0, s, pdl,
                            kernel_mesh(*mesh), mesh->node_elem_ptr, mesh->node_elem, (const double*)elem_out, u, node_out,
                            (const double*)w.part, n_part, scal_out)))
        return rc;
    note_launches(1);
    return launch_check("dfea_frame_all_fields");
}

extern "C" int dfea_frame_push_forward(const dfea_mesh_view* mesh, const double* moduli_ref, double* moduli, void* stream) {
    int rc = validate_frame(mesh, "dfea_frame_push_forward");
    if (rc) return rc;
    if (!moduli_ref || !moduli || !al16(moduli_ref) || !al16(moduli))
        return set_error(DFEA_ERR_INVALID, "dfea_frame_push_forward: NULL or misaligned pointer");
    if (mesh->n_el == 0) return DFEA_OK;
    k_frame_push_forward<<<grid_for(mesh->n_el * mesh->n_q, kThreads, 8), kThreads, 0, static_cast<cudaStream_t>(stream)>>>(
        mesh->n_el, mesh->stride, mesh->n_q, mesh->frame, moduli_ref, moduli);
    note_launches(1);
    return launch_check("dfea_frame_push_forward");
}
