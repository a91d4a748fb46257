// kernel_fit.cpp -- resident CTAs of a kernel, kept by device, kernel and shape.
#include "kernel_fit.h"

#include <map>
#include <mutex>
#include <tuple>

#include "gu_internal.h"

namespace gu {

int kernel_fit(int device, const void *kernel, int threads, size_t smem, size_t smem_most, int cluster)
{
    static std::mutex mu;
    static std::map<std::tuple<int, const void *, int, size_t, int>, int> known;
    std::lock_guard<std::mutex> lk(mu);
    const auto key = std::make_tuple(device, kernel, threads, smem, cluster);
    const auto it = known.find(key);
    if (it != known.end()) return it->second;
    GU_CUDA_CHECK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_most));
    int fit = 0;
    if (cluster > 1) {
        GU_CUDA_CHECK(cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
        cudaLaunchAttribute at[1];
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = (unsigned)cluster;
        at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3((unsigned)cluster);
        cfg.blockDim = dim3((unsigned)threads);
        cfg.dynamicSmemBytes = smem;
        cfg.attrs = at;
        cfg.numAttrs = 1;
        if (cudaOccupancyMaxActiveClusters(&fit, kernel, &cfg) != cudaSuccess) {
            (void)cudaGetLastError();
            fit = 0;
        }
    } else {
        GU_CUDA_CHECK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&fit, kernel, threads, smem));
    }
    if (known.size() > 4096) known.clear();
    known[key] = fit;
    return fit;
}

}  // namespace gu
