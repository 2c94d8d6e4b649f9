// bg_cluster.cu -- launch of the cluster kernel (bg_cluster.cuh).
#include <map>
#include <mutex>
#include <set>
#include <utility>

#include "bg_cluster_host.h"

namespace {

cudaLaunchConfig_t config(cudaLaunchAttribute *at, int blocks, size_t smem, cudaStream_t s) {
    cudaLaunchConfig_t c = {};
    c.gridDim = dim3((unsigned)blocks);
    c.blockDim = dim3(bg::kClusterThreads + (blocks > 1 ? 32 : 0));   // and the arrivals' warp
    c.dynamicSmemBytes = smem;
    c.stream = s;
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = (unsigned)blocks;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    c.attrs = at;
    c.numAttrs = 1;
    return c;
}

}  // namespace

const void *bg_cluster_kernel(int precision, int nvar, int npt, bool diag, bool multi, int pat) {
    return precision == 64 ? bg_cluster_kernel_f64(nvar, npt, diag, multi, pat) : bg_cluster_kernel_f32(nvar, npt, diag, multi, pat);
}

bool bg_cluster_fits(const void *kernel, cudaKernel_t generated, int blocks, size_t smem) {
    int dev = 0, n = 0, most = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&most, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess)
        return false;
    auto set = [&](cudaFuncAttribute at, int v) {
        return generated ? cudaKernelSetAttributeForDevice(generated, at, v, dev) : cudaFuncSetAttribute(kernel, at, v);
    };
    // the limits belong to the kernel, not to this network: the largest there
    // is, so that no other network's call lowers them.  Built-in kernels are
    // set once; whether the device places a cluster of that many blocks with
    // that much shared memory is asked once per size (the query takes
    // milliseconds, and clusters of up to 8 blocks are always placed).
    static std::mutex mutex;
    static std::set<std::pair<int, const void *>> ready;
    static std::map<std::pair<int, int>, bool> placed;
    std::lock_guard<std::mutex> lock(mutex);
    if (generated || !ready.count({dev, kernel})) {
        if (set(cudaFuncAttributeMaxDynamicSharedMemorySize, most - kClusterStaticSmem) != cudaSuccess ||
            set(cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess) {
            cudaGetLastError();
            return false;
        }
        if (!generated) ready.insert({dev, kernel});
    }
    if ((int64_t)smem > most - kClusterStaticSmem) return false;
    if (blocks <= 8) return true;
    auto it = placed.find({dev, blocks});
    if (it == placed.end()) {
        cudaLaunchAttribute at[1];
        cudaLaunchConfig_t c = config(at, blocks, (size_t)(most - kClusterStaticSmem), nullptr);
        const bool ok = cudaOccupancyMaxActiveClusters(&n, generated ? (const void *)generated : kernel, &c) == cudaSuccess && n >= 1;
        cudaGetLastError();
        it = placed.emplace(std::make_pair(dev, blocks), ok).first;
    }
    return it->second;
}

cudaError_t bg_cluster_launch(const void *kernel, const void *args, int blocks, size_t smem, cudaStream_t s) {
    cudaLaunchAttribute at[1];
    cudaLaunchConfig_t c = config(at, blocks, smem, s);
    void *pa[] = {(void *)args};
    return cudaLaunchKernelExC(&c, kernel, pa);
}
