// The cluster size of a kernel that asks for more than the portable eight CTAs, by device.
#pragma once
#include <cuda_runtime_api.h>

#include <atomic>
#include <cstdint>

namespace sb {

// cudaFuncSetAttribute and the answer of the occupancy query hold for the current device only, and one process may drive
// several GPUs from several threads: one word a device, 0 until its answer is known.  Devices past the array ask every time.
struct ClusterFit {
    static constexpr int kDevices = 64;
    std::atomic<uint32_t> ctas[kDevices] = {};
};

// 16 where the current device can hold such a cluster of `config`, else the portable 8; 0: no current device.
inline uint32_t cluster_fit(const void *kernel, cudaLaunchConfig_t config, ClusterFit &known) {
    int device = 0;
    if (cudaGetDevice(&device) != cudaSuccess || device < 0) return 0u;
    const bool kept = device < ClusterFit::kDevices;
    if (kept)
        if (const uint32_t n = known.ctas[device].load(std::memory_order_acquire)) return n;
    constexpr uint32_t kWide = 16u, kPortable = 8u;
    cudaLaunchAttribute a{};
    a.id = cudaLaunchAttributeClusterDimension;
    a.val.clusterDim.x = kWide;
    a.val.clusterDim.y = a.val.clusterDim.z = 1;
    config.gridDim = dim3(kWide);
    config.attrs = &a;
    config.numAttrs = 1;
    int clusters = 0;
    const bool wide = cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess &&
                      cudaOccupancyMaxActiveClusters(&clusters, kernel, &config) == cudaSuccess && clusters >= 1;
    if (!wide) cudaGetLastError();  // a refusal is an answer
    if (kept) known.ctas[device].store(wide ? kWide : kPortable, std::memory_order_release);
    return wide ? kWide : kPortable;
}

}  // namespace sb
