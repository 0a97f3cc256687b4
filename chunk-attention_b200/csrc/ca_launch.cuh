// One way to launch a kernel that may be a programmatic dependent of the kernel ahead of it on the stream, alone or in clusters.
#pragma once
#include <cuda_runtime.h>

#include <cstdlib>

namespace ca {

// CA_OPT_DEPENDENT_LAUNCH, as launches carry it
constexpr int DEPENDENT_MERGE = 1, DEPENDENT_ATTENTION = 2;

// dependent: the kernel is set up while the one ahead drains; it executes griddepcontrol.wait before it touches global memory.  Where the
// stream or the driver refuses that (or CA_DISABLE_PDL is set), an ordinary launch.  cluster: CTAs of a cluster, along x.
template <typename... P, typename... A>
cudaError_t launch_kernel(void (*kernel)(P...), dim3 grid, int threads, size_t smem, int cluster, bool dependent, cudaStream_t stream, const A&... args) {
    static const bool disabled = std::getenv("CA_DISABLE_PDL") != nullptr;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = cluster;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    const int n = cluster > 1 ? 1 : 0;
    attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[n].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = dependent && !disabled ? n + 1 : n;
    cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, args...);
    if (e != cudaSuccess && (int)cfg.numAttrs > n) {
        (void)cudaGetLastError();
        cfg.numAttrs = n;
        e = cudaLaunchKernelEx(&cfg, kernel, args...);
    }
    return e;
}

}  // namespace ca
