// Host-side launch with the programmatic-dependent-launch attribute: the kernel may start while its predecessor in the
// stream drains, and waits for it (grid_dependency_wait) before it touches anything the predecessor reads or writes.
#pragma once

#include <cuda_runtime.h>

namespace nerve {

// Multiprocessors of the current device, for grids and plans that go by waves of them.
inline int multiprocessors() {
    int device = 0, count = 0;
    if (cudaGetDevice(&device) != cudaSuccess || cudaDeviceGetAttribute(&count, cudaDevAttrMultiProcessorCount, device) != cudaSuccess || count < 1) return 1;
    return count;
}

template <typename... Parameters, typename... Arguments>
cudaError_t launch_dependent(void (*kernel)(Parameters...), dim3 grid, dim3 block, size_t smem, int cluster_z, cudaStream_t stream, Arguments... arguments) {
    cudaLaunchConfig_t config = {};
    config.gridDim = grid;
    config.blockDim = block;
    config.dynamicSmemBytes = smem;
    config.stream = stream;
    cudaLaunchAttribute attributes[2];
    attributes[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attributes[0].val.programmaticStreamSerializationAllowed = 1;
    attributes[1].id = cudaLaunchAttributeClusterDimension;
    attributes[1].val.clusterDim.x = 1;
    attributes[1].val.clusterDim.y = 1;
    attributes[1].val.clusterDim.z = static_cast<unsigned int>(cluster_z);
    config.attrs = attributes;
    config.numAttrs = cluster_z > 1 ? 2 : 1;
    return cudaLaunchKernelEx(&config, kernel, static_cast<Parameters>(arguments)...);
}

}  // namespace nerve
