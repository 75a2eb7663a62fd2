// dfea_mg.cuh -- what the multigrid (dfea_mg.cu) and its passes over the finite-element level (dfea_kernels.cu) share.
#pragma once

#include "dfea_common.cuh"

namespace dfea {

// State of a multigrid PCG solve on the device.
struct MgPcgState {
    double rz, curv, rr, beta, nb2, tol2, rtol2, spare;
    int32_t k, max_iter, status, iters, spare_i[4];
};
static_assert(sizeof(MgPcgState) <= 16 * sizeof(double), "pcg_state holds 16 doubles");

// dfea_mg.dot_work (doubles): two reduction scratches of block partials and a ticket (a set-up's branches reduce side by
// side), then the state of a host-driven solve; the tickets are zeroed at every set-up.
constexpr int kMgDotScratch = kMaxBlocks + 32;
constexpr int kMgDotWork = 2 * kMgDotScratch + 16;
__host__ __device__ inline unsigned* dot_ticket(double* work) { return reinterpret_cast<unsigned*>(work + kMaxBlocks); }
inline MgPcgState* host_driven_state(double* work) { return reinterpret_cast<MgPcgState*>(work + 2 * kMgDotScratch); }

// What a sum over the grid is for; stored by thread 0 of the block that holds the total.
enum {
    MG_DOT_PLAIN,    // *out
    MG_DOT_LANCZOS,  // r.z of a CG step of the Lanczos estimate: out = [p.Ap, r.z, -, beta], (alpha, beta) into hist[2k..]
    MG_DOT_CYCLE,    // r.z after a cycle of the PCG: out is its MgPcgState
};
template <int KIND>
__device__ __forceinline__ void dot_store(double a, double* out, double* hist, int k) {
    if (KIND == MG_DOT_LANCZOS) {
        const double alpha = out[1] / out[0], beta = a / out[1];
        hist[2 * k] = alpha;
        hist[2 * k + 1] = beta;
        out[1] = a;
        out[3] = beta;
    } else if (KIND == MG_DOT_CYCLE) {
        MgPcgState* st = reinterpret_cast<MgPcgState*>(out);
        st->beta = st->k == 0 ? 0.0 : a / st->rz;
        st->rz = a;
    } else {
        *out = a;
    }
}

// A thread's share of a sum handed to the last block of the grid (fixed order); every thread calls it.
template <int NT, int KIND>
__device__ __forceinline__ void dot_finish(double a, double* work, double* out, double* hist, int k) {
    const double vals[1] = {block_sum<NT>(a)};
    double tot[1];
    if (last_block_sum<NT, 1>(vals, RedSite{work, dot_ticket(work), nullptr}, tot) && threadIdx.x == 0)
        dot_store<KIND>(tot[0], out, hist, k);
}

// End of a PCG iteration from r.r: the status and the counters; true while the solve goes on.  (NaN: it goes on.)
__device__ __forceinline__ bool pcg_iteration_end(MgPcgState* st, bool curved, double rr) {
    if (!curved) {
        st->status = DFEA_PCG_NEG_CURV;
        st->iters = st->k;
        return false;
    }
    st->rr = rr;
    st->k += 1;
    st->iters = st->k;
    if (rr <= st->tol2) st->status = DFEA_PCG_CONVERGED;
    else if (st->k >= st->max_iter) st->status = DFEA_PCG_MAX_ITER;
    return st->status == DFEA_PCG_RUNNING;
}

// Smoothing on the finite-element level in the gather form, the update in the node pass of the product (v -> q = A v).
// The vectors may alias where a node touches its own entries only (all of them but v's neighbours).
enum { MG_FE_STEP = 0, MG_FE_RESTART = 1 };
struct MgNodePass {
    const double* v;     // MG_FE_STEP: the direction d; MG_FE_RESTART: the iterate x
    double* x;
    const double* r_in;  // the residual before (MG_FE_STEP), the right-hand side (MG_FE_RESTART)
    double* r_out;       // the residual after, or NULL: nobody reads it
    double* d;           // the next direction, or NULL: none follows, or it is added at once (add)
    const double* diag;
    const double* coef;  // (c1, c2) or the scale; not read without a next direction
    int first;           // MG_FE_STEP: x = d (the iterate was zero)
    int add;             // the next direction is the pass's last: added to x here, its product is not needed
};
// dot: after the pass x . rhs into the PCG state (rhs: the cycle's right-hand side); NULL: not taken
int mg_fe_smooth(const dfea_mesh_view* mesh, const void* moduli, int32_t moduli_dtype, void* fe_work, int mode,
                 const MgNodePass& pass, const double* rhs, MgPcgState* dot, double* dot_work, cudaStream_t s);

// A conjugate-gradient step on the finite-element level in two launches (reference-frame moduli, gather form): an
// element pass on the direction z + beta p with the curvature in energy form, and the node pass with every update.
//   MG_CG_SOLVE    an iteration of the PCG (st): p, x += alpha p, r -= alpha q, the next cycle's first direction
//                  d = scale r / D, r.r and the status; cond, if wanted, is the loop's condition
//   MG_CG_LANCZOS  a step of the estimate: p, r -= alpha q, z = r / D, r.z and the coefficients (scal = [p.Ap, r.z, -, beta])
enum { MG_CG_SOLVE = 0, MG_CG_LANCZOS = 1 };
struct MgCgStep {
    double *z, *p, *r, *x, *d;
    const double *diag, *scale;
    MgPcgState* st;
    double *scal, *hist;
    int k;
    bool loop;
    cudaGraphConditionalHandle cond;
};
bool mg_fe_cg_supported(const dfea_mesh_view* mesh, int32_t moduli_dtype);
int mg_fe_cg_step(const dfea_mesh_view* mesh, const void* moduli, int32_t moduli_dtype, void* fe_work, int kind,
                  const MgCgStep& step, double* dot_work, cudaStream_t s);

}  // namespace dfea
