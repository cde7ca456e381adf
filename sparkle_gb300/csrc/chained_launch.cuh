// chained_launch.cuh -- launches that overlap a kernel's start with the end of the kernel before it in its stream.
//
// A kernel started by launch_chained is launched as soon as every block of the kernel before it has called
// let_next_kernel_in (or has left). Its blocks take the places of those that leave and wait in
// after_previous_kernel, so what remains between two kernels is that wait, not a launch. Every such kernel calls
// after_previous_kernel before it touches memory that another kernel writes or reads, and before it takes what a
// block of the kernel before may still wait for (tensor memory). Then a kernel is complete only when all before it
// are, and any kernel, copy or event may follow.
#pragma once

#include <cuda_runtime.h>

namespace spk {

// From here on the kernel before is complete and its writes are visible.
__device__ __forceinline__ void after_previous_kernel() { cudaGridDependencySynchronize(); }

__device__ __forceinline__ void let_next_kernel_in() { cudaTriggerProgrammaticLaunchCompletion(); }

// With `early` false an ordinary launch, which starts when the kernel before is complete.
template <class... Params, class... Args>
cudaError_t launch_chained_if(bool early, void (*kernel)(Params...), dim3 grid, unsigned threads, size_t smem,
                              cudaStream_t stream, const Args &...args) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute chained{};
    chained.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    chained.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &chained;
    cfg.numAttrs = early ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kernel, Params(args)...);
}

template <class... Params, class... Args>
cudaError_t launch_chained(void (*kernel)(Params...), dim3 grid, unsigned threads, size_t smem, cudaStream_t stream,
                           const Args &...args) {
    return launch_chained_if(true, kernel, grid, threads, smem, stream, args...);
}

}  // namespace spk
