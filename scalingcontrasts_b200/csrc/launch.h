// Launches that overlap the end of the kernel before them in the stream (programmatic dependent launch).
//
// A kernel launched this way may be placed on multiprocessors as soon as every block of the kernel before it has started and
// said so (`let_dependents_start`) or left; it sets up what needs no global memory (barriers, tensor memory, tensor-map
// prefetches) and then stands in `wait_for_kernels_before` until that kernel, and through it everything ahead in the
// stream, is complete and its writes are visible. So a kernel that is launched with `launch_dependent` calls the wait in every
// thread before its first access to global memory, reads and writes alike, and on every way out. What it reads may still be written
// when it starts, so none of it is read as constant for the kernel's lifetime: no __ldg, no `const __restrict__`. Kernels that do not say
// anything (another library's, the collectives that wait for other ranks) count when they are complete, copies and
// fills as ever.
//
// Measured (B200), forward and backward in turn: 128 rows, H=768, K=5 23.0 -> 20.0 us a pair, 1024 rows 31.2 -> 26.4, 2048 rows,
// H=2048, K=8 116 -> 106, 4096 rows, H=768, K=5 133.6 -> 131.7; at 16384 rows nothing, there the GPU is at its power limit.
#pragma once

#include <cuda_runtime.h>

#include <cstddef>

namespace sc {

__device__ __forceinline__ void let_dependents_start() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void wait_for_kernels_before() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// `overlap` false: an ordinary launch. `cluster`: CTAs of a cluster. Errors are left for cudaGetLastError, as with the launch syntax.
template <typename... parameters, typename... arguments>
void launch_dependent_clusters(bool overlap, uint32_t cluster, void (*kernel)(parameters...), dim3 grid, dim3 block, size_t shared_bytes,
                               cudaStream_t stream, arguments&&... values) {
    cudaLaunchAttribute attributes[2]{};
    attributes[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attributes[0].val.programmaticStreamSerializationAllowed = overlap ? 1 : 0;
    attributes[1].id = cudaLaunchAttributeClusterDimension;
    attributes[1].val.clusterDim.x = cluster, attributes[1].val.clusterDim.y = 1, attributes[1].val.clusterDim.z = 1;
    cudaLaunchConfig_t config{};
    config.gridDim = grid, config.blockDim = block, config.dynamicSmemBytes = shared_bytes, config.stream = stream;
    config.attrs = attributes, config.numAttrs = cluster > 1 ? 2 : 1;
    cudaLaunchKernelEx(&config, kernel, static_cast<parameters>(values)...);
}
template <typename... parameters, typename... arguments>
void launch_dependent(bool overlap, void (*kernel)(parameters...), dim3 grid, dim3 block, size_t shared_bytes, cudaStream_t stream,
                      arguments&&... values) {
    launch_dependent_clusters(overlap, 1, kernel, grid, block, shared_bytes, stream, static_cast<arguments&&>(values)...);
}

} // namespace sc
