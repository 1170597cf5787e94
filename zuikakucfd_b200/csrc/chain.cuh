// Programmatic dependent launch for the kernels of a step.
//
// A step is a chain of dependent kernels of a few to a few hundred
// microseconds.  Launched plainly, each starts only when its predecessor has
// drained, been retired and its memory flushed; launched chained, its launch
// overlaps that end, and its CTAs wait (chain_wait) until all of the
// predecessor's memory is visible.  Every kernel of a chain calls chain_wait in
// every thread before it reads or writes anything another kernel writes or
// reads, so completion stays transitive along the chain.  A predecessor that is
// not a kernel orders a chained launch like a plain one.
//
// No kernel triggers its dependents before it ends (griddepcontrol.
// launch_dependents): a dependent's CTAs would then be placed around CTAs that
// still run, some SMs taking several and others none, and they stay there.
// Microseconds per step (graph replay, four-quadrant case), plainly launched /
// triggering at kernel start / as here:
//   WENO FP64 64^2                    16.8 /  18.9 /  15.8
//   WENO mixed 512^2                  55.6 /  49.5 /  50.2
//   DG P=1 mixed 128^2                17.6 /  24.7 /  16.2
//   DG P=2 mixed 128^2                26.0 /  38.2 /  24.8
//   DG P=3 FP64 96^2                  59.9 /  88.1 /  57.0
//   DG P=3 mixed, TVB, 128^2          47.5 /  66.4 /  45.4
//   DG P=2 mixed, TVB, 1024^2        714   / 703   / 701
//   DG P=3 mixed, indicator, 2048^2 5125   /5143   /5119
#pragma once

#include <cuda_runtime.h>

namespace zk {

__device__ __forceinline__ void chain_wait() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
}

template <typename... Params, typename... Args>
cudaError_t launch_chained(void (*kernel)(Params...), dim3 grid, unsigned threads, size_t smem, cudaStream_t s,
                           const Args&... args) {
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, Params(args)...);
    if (e != cudaSuccess) cudaGetLastError();  // reported here, not again by the next launch that asks for it
    return e;
}

}  // namespace zk
