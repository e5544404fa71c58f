#include "skinny_tc.cuh"

namespace b200p {
namespace {
constexpr int kMaxDevices = 64;
std::atomic<int> g_resident[kMaxDevices][kStcMaxCluster + 1];      // 0: not asked yet, n + 1: n clusters
__global__ void __launch_bounds__(kStcThreads, 1) stc_residency_kernel() {}
} // namespace

int stc_resident_clusters(int cluster) {
    int dev = -1;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) { cudaGetLastError(); return 0; }
    std::atomic<int>& kept = g_resident[dev][cluster];
    const int v = kept.load(std::memory_order_relaxed);
    if (v > 0) return v - 1;
    constexpr int kBytes = 200 * 1024;                              // more than half of an SM's shared memory: one CTA per SM
    int n = 0;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(unsigned(cluster)); cfg.blockDim = dim3(kStcThreads); cfg.dynamicSmemBytes = kBytes;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = unsigned(cluster); attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr; cfg.numAttrs = 1;
    if (cudaFuncSetAttribute(stc_residency_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kBytes) != cudaSuccess ||
        cudaOccupancyMaxActiveClusters(&n, stc_residency_kernel, &cfg) != cudaSuccess) {
        cudaGetLastError();
        return 0;                                                   // asked again by the next call
    }
    kept.store(n + 1, std::memory_order_relaxed);
    return n;
}

} // namespace b200p
