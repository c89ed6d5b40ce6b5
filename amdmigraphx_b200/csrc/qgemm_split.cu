// quant_dot kernels: tiles of 128 x 64 whose K a cluster shares.
#include "qgemm_kernel.cuh"
#include <mutex>

namespace mgx {

int qgemm_split_launch(int split, const mgx_qgemm_desc& d, const qgemm_operands& o, const qout_args& qo, cudaStream_t stream)
{
    if(d.ab_type == MGX_I8)
        return dispatch_out<64, true, false, false, true>(d, o, qo, stream, split);
    if(d.ab_type == MGX_F16)
        return dispatch_out<64, false, true, false, true>(d, o, qo, stream, split);
    return dispatch_out<64, false, false, false, true>(d, o, qo, stream, split);
}

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

int qgemm_split_status(unsigned int* out) { return read_and_clear_status(out); }

} // namespace mgx
