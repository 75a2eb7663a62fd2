// dfea_cluster.cuh -- thread-block clusters with data in distributed shared memory: addresses in other blocks, the
// hardware barrier, and sums over the cluster that ride on it.
#pragma once

#include <mutex>

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

// What clusters of a kernel can be on the current device: the dynamic shared memory a block may take, and the most blocks
// (a power of two) of a cluster that can be resident with that much each.  16 blocks and 225 KB on a whole B200; on a
// partition of one a large cluster may find no place, and its launch would fail.  Nothing: the kernel cannot be set up.
struct ClusterRoom {
    int blocks = 0, bytes = 0;
};
template <auto Kernel>
const ClusterRoom& cluster_room(int threads) {
    static std::once_flag once[64];
    static ClusterRoom room[64];
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) dev = 0;
    std::call_once(once[dev], [dev, threads] {
        int most = 0;
        cudaFuncAttributes fa;
        if (cudaDeviceGetAttribute(&most, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) == cudaSuccess &&
            cudaFuncGetAttributes(&fa, Kernel) == cudaSuccess &&
            cudaFuncSetAttribute(Kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, most - (int)fa.sharedSizeBytes) == cudaSuccess &&
            cudaFuncSetAttribute(Kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess) {
            cudaLaunchAttribute attr[1];
            attr[0].id = cudaLaunchAttributeClusterDimension;
            attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
            cudaLaunchConfig_t cfg = {};
            cfg.blockDim = dim3(threads);
            cfg.dynamicSmemBytes = most - fa.sharedSizeBytes;
            cfg.attrs = attr;
            cfg.numAttrs = 1;
            for (int size = kClusterMax; size >= 1 && room[dev].blocks == 0; size /= 2) {
                int clusters = 0;
                attr[0].val.clusterDim.x = size;
                cfg.gridDim = dim3(size);
                if (cudaOccupancyMaxActiveClusters(&clusters, Kernel, &cfg) == cudaSuccess && clusters > 0) room[dev].blocks = size;
            }
            room[dev].bytes = most - (int)fa.sharedSizeBytes;
        }
        (void)cudaGetLastError();  // a size that finds no place is no error of the caller's
    });
    return room[dev];
}

}  // namespace dfea
