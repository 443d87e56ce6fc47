// launch_early.cuh -- kernels that are set up while the one before them in the stream finishes
// (programmatic stream serialisation).
#pragma once
#include <cuda_runtime.h>

namespace nrrs {

template <class T>
struct ArgOf {
    using type = T;   // the kernel's parameter types decide, as with <<<>>>
};
// Launches k so; it calls wait_for_stream() before it touches memory that an earlier kernel may
// still use (2 to 3 us between the kernels of a step become about 1). `cluster` CTAs per cluster,
// 0 = none.
template <class... A>
cudaError_t launch_early(void (*k)(A...), dim3 grid, unsigned threads, size_t smem, unsigned cluster,
                         cudaStream_t s, const typename ArgOf<A>::type&... args) {
    cudaLaunchConfig_t c{};
    c.gridDim = grid;
    c.blockDim = dim3(threads);
    c.dynamicSmemBytes = smem;
    c.stream = s;
    cudaLaunchAttribute at[2]{};
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    at[1].id = cudaLaunchAttributeClusterDimension;
    at[1].val.clusterDim.x = cluster;
    at[1].val.clusterDim.y = at[1].val.clusterDim.z = 1;
    c.attrs = at;
    c.numAttrs = cluster ? 2 : 1;
    const cudaError_t e = cudaLaunchKernelEx(&c, k, A(args)...);
    if (e != cudaSuccess) cudaGetLastError();   // reported here, not by a later call
    return e;
}
// waits for the kernels before this one in its stream and has their writes visible
__device__ __forceinline__ void wait_for_stream() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
}
// lets the next kernel of the stream be set up while this one finishes
__device__ __forceinline__ void let_next_start() {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

}  // namespace nrrs
