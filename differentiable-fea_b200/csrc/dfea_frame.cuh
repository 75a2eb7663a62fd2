// dfea_frame.cuh -- element kernels in the element's reference frame, one warp per Gauss point.
//
// With dN/dX = Jinv^T dN/dxi every per-element gradient array collapses to the 2 x 2 matrix Jinv of each
// Gauss point (32 B instead of 16 B per node) and the element type's reference gradients (a kernel parameter):
//     F = I + (sum_a u_a (x) dN_a/dxi) Jinv,   f_a = sum_q w (P Jinv^T) . dN_a/dxi,
//     Chat = Jinv C Jinv^T (10 symmetric entries),   (A v)_a = sum_q (Chat : sum_b v_b (x) dN_b/dxi) . dN_a/dxi.
//
// A block works on EB = 32 elements (128 for the one-point Tri3) with one warp per Gauss point, lanes over the
// elements.  The nodal values of the 32 elements go through shared memory once (warp a gathers local node a),
// each thread does one Gauss point, and the Gauss points are summed in order from shared memory.  Against one
// thread per element this multiplies the threads by n_q with a fraction of the registers: a mid-sized mesh
// fills the chip, and the FP64 chains of the point evaluation (log, division) overlap.
// Element results go to fe[a][e] and a node pass sums them in incidence order (no colours, no atomics).
//
// What bounds them: the large-mesh product and moduli, HBM (1M Q4 product: 436 MB in 75 us, 5.8 TB/s; moduli 600 MB in
// 116 us); the residual, the FP64 chain of log and division (1M Q4: 68 us); small meshes, the two memory latencies of a
// tile.  Measured (B200) against the kernels that read dN/dX colour by colour: product of 1M Q4 elements 172 -> 98 us,
// residual + moduli + product of 640k Q4 577 -> 220 us of kernel time, Jacobi-PCG at 16k Q4 42 -> 14 us an iteration.
#pragma once

#include "dfea_common.cuh"
#include "dfea_material.cuh"

namespace dfea {

// material of a launch: the host struct, or parameters (doubles) and scalable flags (bytes) read from device
// memory, so that a problem whose material lives on the device needs no copy to the host before the launch
struct MatArg {
    dfea_material m;
    const double* p;
    const uint8_t* scalable;
};

__device__ __forceinline__ void frame_params(const MatArg& mat, double th, double (&pe)[DFEA_MAX_MAT_PARAMS]) {
    if (mat.p != nullptr) {
        const int n = material_n_params(mat.m.model);
#pragma unroll
        for (int k = 0; k < DFEA_MAX_MAT_PARAMS; ++k)
            pe[k] = k < n ? (__ldg(mat.scalable + k) ? __ldg(mat.p + k) * th : __ldg(mat.p + k)) : 0.0;
    } else {
        element_params(mat.m, th, pe);
    }
}

template <int NEN, int NQ>
struct FrameCfg {
    static constexpr int EB = NQ == 1 ? 128 : 32;  // elements per block
    static constexpr int NT = EB * NQ;             // threads: warp(s) q at Gauss point q
    // resident blocks the closed-form kernels are compiled for: 18 - 24 warps per SM.  Left alone, the pipelined loads
    // of the 9-point elements take 130 - 140 registers, which leaves one block of 9 warps per SM.
    static constexpr int MINB = NT > 256 ? 2 : (NT > 128 ? 3 : 5);
};

// The block's connectivity of one tile, one local node per warp (three per thread with one Gauss point), requested
// two tiles ahead; the nodal pairs are gathered one tile ahead.  The chain connectivity -> pair -> shared memory is
// two memory latencies, longer than the arithmetic of a tile: unpipelined it left the product of a million Q4
// elements at 74 us.
template <int NEN, int NQ>
struct ConnRow {
    static constexpr int GA = (NEN + NQ - 1) / NQ;
    int c[GA];  // node << 2 | fix bits, -1: none
    __device__ __forceinline__ void load(const Mesh& m, int64_t e, bool live, int q) {
#pragma unroll
        for (int i = 0; i < GA; ++i) {
            const int a = i * NQ + q;
            c[i] = (a < NEN && live) ? __ldg(m.conn + (int64_t)a * m.stride + e) : -1;
        }
    }
};

template <int NEN, int NQ, typename T>
struct NodeRow {
    static constexpr int GA = ConnRow<NEN, NQ>::GA;
    v2_t<T> t[GA];
    // gather(node) -> pair; fixed components zeroed with MASK
    template <bool MASK, typename Gather>
    __device__ __forceinline__ void gather(const ConnRow<NEN, NQ>& row, Gather&& gather) {
#pragma unroll
        for (int i = 0; i < GA; ++i) {
            const int c = row.c[i];
            t[i] = make_v2<T>(T(0), T(0));
            if (c >= 0) {
                t[i] = gather(c >> 2);
                if (MASK && (c & 1)) t[i].x = T(0);
                if (MASK && (c & 2)) t[i].y = T(0);
            }
        }
    }
    __device__ __forceinline__ void store(v2_t<T> (*vs)[FrameCfg<NEN, NQ>::EB], int q, int lane) const {
#pragma unroll
        for (int i = 0; i < GA; ++i)
            if (i * NQ + q < NEN) vs[i * NQ + q][lane] = t[i];
    }
};

// The reference gradients of this warp's Gauss point, held in registers: indexed by the warp they would be loads
// from the constant bank at every use.
template <int NEN, typename T>
struct RefRow {
    T g[NEN][2];
    template <int NQ>
    __device__ __forceinline__ RefRow(const RefGrad<NEN, NQ>& rg, int q) {
#pragma unroll
        for (int a = 0; a < NEN; ++a) {
            g[a][0] = (T)rg.g[q][a][0];
            g[a][1] = (T)rg.g[q][a][1];
        }
    }
};

// G_ib = sum_a v_a,i dN_a/dxi_b at this warp's Gauss point
template <int NEN, int NQ, typename T>
__device__ __forceinline__ void frame_gradient(const RefRow<NEN, T>& r, int lane,
                                               const v2_t<T> (*vs)[FrameCfg<NEN, NQ>::EB], T (&G)[4]) {
    G[0] = G[1] = G[2] = G[3] = T(0);
#pragma unroll
    for (int a = 0; a < NEN; ++a) {
        const v2_t<T> t = vs[a][lane];
        const T r0 = r.g[a][0], r1 = r.g[a][1];
        G[0] += t.x * r0;
        G[1] += t.x * r1;
        G[2] += t.y * r0;
        G[3] += t.y * r1;
    }
}

// F = I + H Jinv, F[2i+J]; ji[2b+J] = Jinv_bJ
__device__ __forceinline__ void frame_deformation(const double (&H)[4], const double (&ji)[4], double (&F)[4]) {
    F[0] = 1.0 + H[0] * ji[0] + H[1] * ji[2];
    F[1] = H[0] * ji[1] + H[1] * ji[3];
    F[2] = H[2] * ji[0] + H[3] * ji[2];
    F[3] = 1.0 + H[2] * ji[1] + H[3] * ji[3];
}

// Geometry and stiffness scale of this warp's Gauss point on one tile, requested one tile ahead (the original
// element id, which theta is indexed by, two tiles ahead)
struct FramePoint {
    double ji[4], w, th;
    __device__ __forceinline__ void load(const Mesh& m, const double* frame, const double* theta, int orig, int64_t e,
                                         bool live, int q) {
        ji[0] = ji[3] = th = 1.0;
        ji[1] = ji[2] = w = 0.0;
        if (live) {
            const double2* j2 = reinterpret_cast<const double2*>(frame);
            const double2 r0 = __ldcs(j2 + (int64_t)(2 * q) * m.stride + e), r1 = __ldcs(j2 + (int64_t)(2 * q + 1) * m.stride + e);
            ji[0] = r0.x;
            ji[1] = r0.y;
            ji[2] = r1.x;
            ji[3] = r1.y;
            w = __ldcs(m.wdet + (int64_t)q * m.stride + e);
            if (theta) th = __ldg(theta + orig);
        }
    }
    static __device__ __forceinline__ int orig_of(const Mesh& m, int64_t e) { return e < m.n_el ? __ldg(m.orig + e) : 0; }
};

__device__ __forceinline__ void load_jinv(const double* frame, int64_t S, int q, int64_t e, double (&ji)[4]) {
    const double2* j2 = reinterpret_cast<const double2*>(frame);
    const double2 r0 = __ldcs(j2 + (int64_t)(2 * q) * S + e), r1 = __ldcs(j2 + (int64_t)(2 * q + 1) * S + e);
    ji[0] = r0.x;
    ji[1] = r0.y;
    ji[2] = r1.x;
    ji[3] = r1.y;
}

// Sum over the Gauss points of the block's element results, in order q = 0 .. NQ-1: red[q][a][lane] -> f(a, e, sum)
template <int NEN, int NQ, typename T, typename Out>
__device__ __forceinline__ void frame_reduce(int64_t e, bool live, int q, int lane,
                                             const v2_t<T> (*red)[NEN][FrameCfg<NEN, NQ>::EB], Out&& out) {
#pragma unroll
    for (int a0 = 0; a0 < NEN; a0 += NQ) {
        const int a = a0 + q;
        if (a < NEN && live) {
            v2_t<T> s = red[0][a][lane];
#pragma unroll
            for (int k = 1; k < NQ; ++k) {
                const v2_t<T> t = red[k][a][lane];
                s.x += t.x;
                s.y += t.y;
            }
            out(a, e, s);
        }
    }
}

// ------------------------------------------------------------------------------------------
// the product from stored reference-frame moduli
// ------------------------------------------------------------------------------------------
// 10 symmetric entries of Gauss point q: h = 00 01 02 03 11 12 13 22 23 33
//   f32 layout per q: float4 [S], float4 [S], float2 [S];   f64: 5 rows of double2 [S]
template <typename SD> struct FrameModuli;
template <> struct FrameModuli<double> {
    double2 h[5];
    template <bool CACHED>
    __device__ __forceinline__ void load(const double* C, int64_t S, int q, int64_t e) {
        const double2* p = reinterpret_cast<const double2*>(C) + (int64_t)(q * 5) * S + e;
#pragma unroll
        for (int k = 0; k < 5; ++k) h[k] = CACHED ? __ldg(p + k * S) : __ldcs(p + k * S);
    }
    __device__ __forceinline__ void clear() {
#pragma unroll
        for (int k = 0; k < 5; ++k) h[k] = make_double2(0.0, 0.0);
    }
    template <typename T>
    __device__ __forceinline__ void apply(const T (&G)[4], T (&P)[4]) const {
        const T c00 = h[0].x, c01 = h[0].y, c02 = h[1].x, c03 = h[1].y, c11 = h[2].x, c12 = h[2].y, c13 = h[3].x,
                c22 = h[3].y, c23 = h[4].x, c33 = h[4].y;
        P[0] = c00 * G[0] + c01 * G[1] + c02 * G[2] + c03 * G[3];
        P[1] = c01 * G[0] + c11 * G[1] + c12 * G[2] + c13 * G[3];
        P[2] = c02 * G[0] + c12 * G[1] + c22 * G[2] + c23 * G[3];
        P[3] = c03 * G[0] + c13 * G[1] + c23 * G[2] + c33 * G[3];
    }
};
template <> struct FrameModuli<float> {
    float4 a, b;
    float2 d;
    template <bool CACHED>
    __device__ __forceinline__ void load(const float* C, int64_t S, int q, int64_t e) {
        const float* base = C + (int64_t)q * 10 * S;
        const float4* pa = reinterpret_cast<const float4*>(base) + e;
        const float4* pb = reinterpret_cast<const float4*>(base + 4 * S) + e;
        const float2* pd = reinterpret_cast<const float2*>(base + 8 * S) + e;
        a = CACHED ? __ldg(pa) : __ldcs(pa);
        b = CACHED ? __ldg(pb) : __ldcs(pb);
        d = CACHED ? __ldg(pd) : __ldcs(pd);
    }
    __device__ __forceinline__ void clear() {
        a = b = make_float4(0.f, 0.f, 0.f, 0.f);
        d = make_float2(0.f, 0.f);
    }
    template <typename T>
    __device__ __forceinline__ void apply(const T (&G)[4], T (&P)[4]) const {
        const T c00 = a.x, c01 = a.y, c02 = a.z, c03 = a.w, c11 = b.x, c12 = b.y, c13 = b.z, c22 = b.w, c23 = d.x,
                c33 = d.y;
        P[0] = c00 * G[0] + c01 * G[1] + c02 * G[2] + c03 * G[3];
        P[1] = c01 * G[0] + c11 * G[1] + c12 * G[2] + c13 * G[3];
        P[2] = c02 * G[0] + c12 * G[1] + c22 * G[2] + c23 * G[3];
        P[3] = c03 * G[0] + c13 * G[1] + c23 * G[2] + c33 * G[3];
    }
};

template <int NEN, int NQ, typename T>
struct FrameShared {
    v2_t<T> vs[NEN][FrameCfg<NEN, NQ>::EB];
    v2_t<T> red[NQ][NEN][FrameCfg<NEN, NQ>::EB];
};

// All elements of the mesh by the blocks blk of nblk: gather(node) -> nodal pair (masked here), out(a, e, f)
// receives the element results; curv accumulates G . P per thread with DOT.  `start()` runs after the first
// tile's moduli were requested; returning false abandons the walk.
template <int NEN, int NQ, typename SD, typename T, bool DOT, typename Start, typename Gather, typename Out>
__device__ __forceinline__ bool frame_product(const Mesh& m, const SD* __restrict__ C, const RefGrad<NEN, NQ>& rg,
                                              FrameShared<NEN, NQ, T>& sh, double& curv, Start&& start, Gather&& gather,
                                              Out&& out, int64_t blk, int64_t nblk) {
    constexpr int EB = FrameCfg<NEN, NQ>::EB;
    const int lane = threadIdx.x % EB, q = threadIdx.x / EB;
    const int64_t n_tiles = (m.n_el + EB - 1) / EB;
    const RefRow<NEN, T> r(rg, q);
    FrameModuli<SD> M;
    ConnRow<NEN, NQ> conn;
    NodeRow<NEN, NQ, T> v;
    int64_t tile = blk;
    int64_t e = tile * EB + lane;
    bool live = tile < n_tiles && e < m.n_el;
    conn.load(m, e, live, q);
    if (live) M.template load<false>(C, m.stride, q, e);
    else M.clear();
    if (!start()) return false;
    v.template gather<true>(conn, gather);
    conn.load(m, e + nblk * EB, e + nblk * EB < m.n_el, q);
    while (tile < n_tiles) {
        v.store(sh.vs, q, lane);
        if (NQ > 1) __syncthreads();
        v.template gather<true>(conn, gather);  // of the next tile
        conn.load(m, e + 2 * nblk * EB, e + 2 * nblk * EB < m.n_el, q);
        T G[4], P[4];
        frame_gradient<NEN, NQ, T>(r, lane, sh.vs, G);
        M.apply(G, P);
        if (DOT) curv += (double)(G[0] * P[0] + G[1] * P[1] + G[2] * P[2] + G[3] * P[3]);
        // the next tile's moduli are requested before this tile's sums
        const int64_t e_now = e;
        const bool live_now = live;
        tile += nblk;
        e += nblk * EB;
        live = e < m.n_el;
        if (live) M.template load<false>(C, m.stride, q, e);
        else M.clear();
        if constexpr (NQ == 1) {
#pragma unroll
            for (int a = 0; a < NEN; ++a)
                if (live_now)
                    out(a, e_now, make_v2<T>(P[0] * r.g[a][0] + P[1] * r.g[a][1], P[2] * r.g[a][0] + P[3] * r.g[a][1]));
            // vs[.][lane] is private to the thread with one Gauss point: no barrier needed before the next gather
        } else {
#pragma unroll
            for (int a = 0; a < NEN; ++a) {
                const T r0 = r.g[a][0], r1 = r.g[a][1];
                sh.red[q][a][lane] = make_v2<T>(P[0] * r0 + P[1] * r1, P[2] * r0 + P[3] * r1);
            }
            __syncthreads();
            frame_reduce<NEN, NQ, T>(e_now, live_now, q, lane, sh.red, out);
        }
    }
    return true;
}

}  // namespace dfea
