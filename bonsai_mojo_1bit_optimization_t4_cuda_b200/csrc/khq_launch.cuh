// khq_launch.cuh -- host-side launch helper shared by the entry points.
#pragma once
#include <cuda_runtime.h>

namespace khq {

// SMs of the current device (148 where the query fails).
static inline int sm_count() {
    static int n[64] = {};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 148;
    if (n[dev] == 0) {
        int v = 0;
        if (cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || v <= 0) v = 148;
        n[dev] = v;
    }
    return n[dev];
}

// cluster == 0: no cluster attribute.  All kernels launched through here call pdl_wait() and keep to the rules beside it, so they
// carry the programmatic-serialisation attribute: their launch latency and prologue overlap the end of the kernel before them.
template <typename Kernel, typename... Args>
static cudaError_t launch_pdl(Kernel kernel, unsigned grid, unsigned cluster, size_t smem_bytes,
                              cudaStream_t stream, unsigned threads, Args... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid, 1, 1);
    cfg.blockDim = dim3(threads, 1, 1);
    cfg.dynamicSmemBytes = smem_bytes;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = cluster;
    attr[1].val.clusterDim.y = 1;
    attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = cluster > 0 ? 2 : 1;
    return cudaLaunchKernelEx(&cfg, kernel, args...);
}

}  // namespace khq
