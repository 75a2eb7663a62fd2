// dfea_cluster.cuh -- thread-block clusters with data in distributed shared memory: addresses in other blocks, the
// hardware barrier, and sums over the cluster that ride on it.
#pragma once

#include "dfea_common.cuh"

namespace dfea {

constexpr int kClusterMax = 16;  // blocks of a cluster (beyond 8: the kernel allows non-portable sizes)

__device__ __forceinline__ void cluster_barrier() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;\n" ::: "memory");
}
__device__ __forceinline__ unsigned cluster_rank() {
    unsigned r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
// address of the same shared-memory location in block `rank` of the cluster
__device__ __forceinline__ unsigned cluster_address(unsigned local, unsigned rank) {
    unsigned a;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(local), "r"(rank));
    return a;
}
// sum over the warp, the same bits in every lane
__device__ __forceinline__ double warp_all_sum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
__device__ __forceinline__ double2 cluster_load(unsigned addr) {
    double2 v;
    asm volatile("ld.shared::cluster.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "r"(addr) : "memory");
    return v;
}
__device__ __forceinline__ void cluster_store(unsigned addr, double2 v) {
    asm volatile("st.shared::cluster.v2.f64 [%0], {%1, %2};" ::"r"(addr), "d"(v.x), "d"(v.y) : "memory");
}
__device__ __forceinline__ void cluster_store(unsigned addr, double v) {
    asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(addr), "d"(v) : "memory");
}


// Sums over all threads of the cluster.  Every warp stores its sum into every block's table before the barrier and adds
// the whole table, in the same order, after it: all threads get the same bits, and one barrier both orders the pass
// and reduces.  Two tables alternate, so the next sums never meet a reader of the last.
template <int W>
struct ClusterExchange {
    double* table;  // [2][2][kClusterMax * W] in shared memory, at the same place in every block
    unsigned rank, turn;
    int size;
    static constexpr int kDoubles = 2 * 2 * kClusterMax * W;

    __device__ __forceinline__ ClusterExchange(double* t, unsigned r, int n) : table(t), rank(r), turn(0u), size(n) {}

    template <bool TWO>
    __device__ __forceinline__ void run(double v0, double v1, double& t0, double& t1) {
        const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
        v0 = warp_all_sum(v0);
        if (TWO) v1 = warp_all_sum(v1);
        double* tab = table + (turn & 1u) * 2 * kClusterMax * W;
        const unsigned here = (unsigned)__cvta_generic_to_shared(tab + rank * W + warp);
        if (lane < size) {
            const unsigned to = cluster_address(here, lane);
            cluster_store(to, v0);
            if (TWO) cluster_store(to + kClusterMax * W * 8, v1);
        }
        ++turn;
        __syncwarp();
        cluster_barrier();
        double a0 = 0.0, a1 = 0.0;
        for (int i = lane; i < size * W; i += 32) {
            a0 += tab[i];
            if (TWO) a1 += tab[kClusterMax * W + i];
        }
        t0 = warp_all_sum(a0);
        if (TWO) t1 = warp_all_sum(a1);
    }
    __device__ __forceinline__ double one(double v) {
        double t, unused;
        run<false>(v, 0.0, t, unused);
        return t;
    }
    __device__ __forceinline__ void two(double v0, double v1, double& t0, double& t1) { run<true>(v0, v1, t0, t1); }
};

}  // namespace dfea
