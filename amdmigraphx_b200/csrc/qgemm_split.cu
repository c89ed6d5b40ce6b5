// quant_dot with a shared K: how many clusters run at once.
#include "qgemm_kernel.cuh"
#include <mutex>

namespace mgx {

// Stands in for the kernels in the question how many clusters fit: what limits them is the block and its shared memory,
// the same for all, and to ask for one of them would load its code.
__global__ void __launch_bounds__(NTHREADS, 1) split_probe_kernel() {}

int qgemm_split_clusters(int split)
{
    static std::mutex m;
    static int cached[64][9] = {};
    int dev = 0;
    if(split < 2 or split > 8 or cudaGetDevice(&dev) != cudaSuccess or dev < 0 or dev >= 64)
        return 0;
    std::lock_guard<std::mutex> lock(m);
    int& n = cached[dev][split];
    if(n == 0)
    {
        using S     = qgemm_smem<64, false>;
        auto kernel = split_probe_kernel;
        cudaLaunchConfig_t cfg{};
        cfg.gridDim          = dim3(static_cast<unsigned>(device_sm_count() / split * split));
        cfg.blockDim         = dim3(NTHREADS);
        cfg.dynamicSmemBytes = S::total;
        cudaLaunchAttribute attr[1];
        attr[0].id               = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = static_cast<unsigned>(split);
        attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
        cfg.attrs    = attr;
        cfg.numAttrs = 1;
        if(ensure_smem_optin(reinterpret_cast<const void*>(kernel), S::total) != MGX_OK or
           cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) != cudaSuccess or n < 1)
        {
            (void)cudaGetLastError();
            n = device_sm_count() / (2 * split);
        }
    }
    return n;
}

} // namespace mgx
