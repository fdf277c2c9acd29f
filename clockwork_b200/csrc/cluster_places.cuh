// How many thread-block clusters the GPU holds at a time.
#pragma once
#include "common.cuh"
#include <atomic>

#define CLUSTER_PLACES_MAX 8

// A cluster lies within one group of SMs (GPC), so that the counts are well below SMs / size and differ from part to part: the
// driver is asked once per size (148 SMs, one CTA to an SM: 74, 45, 33, 26, 22, 15 and 15 clusters of 2 to 8; two: 148, 93, 71,
// 56, 45, 37 and 33).  It is asked about an empty kernel with the shared memory of one or two CTAs to an SM: of kernels that
// allocate tensor memory the occupancy calculator says one CTA to an SM whatever they hold.
static __global__ void __launch_bounds__(128) cluster_places_kernel() {}

static int clusters_at_once(int size, int per_sm, int sm_count) {
    static std::atomic<int> known[2][CLUSTER_PLACES_MAX + 1];
    if (size <= 1) return per_sm * sm_count;
    int n = known[per_sm - 1][size].load(std::memory_order_relaxed);
    if (n > 0) return n;
    const int most = 227 * 1024, smem = per_sm == 2 ? 113 * 1024 : most;
    cudaLaunchAttribute cluster;
    cluster.id = cudaLaunchAttributeClusterDimension;
    cluster.val.clusterDim.x = cluster.val.clusterDim.y = 1;
    cluster.val.clusterDim.z = size;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(1, 1, size);
    cfg.blockDim = dim3(128);
    cfg.dynamicSmemBytes = smem;
    cfg.attrs = &cluster;
    cfg.numAttrs = 1;
    if (cudaFuncSetAttribute(cluster_places_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, most) != cudaSuccess ||
        cudaOccupancyMaxActiveClusters(&n, cluster_places_kernel, &cfg) != cudaSuccess || n <= 0) {
        (void)cudaGetLastError();
        return per_sm * sm_count / size;  // (no answer: as if clusters could lie anywhere)
    }
    known[per_sm - 1][size].store(n, std::memory_order_relaxed);
    return n;
}
