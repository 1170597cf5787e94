// Programmatic dependent launch for the kernels of a step.
//
// A step is a chain of dependent kernels of a few to a few hundred
// microseconds.  Launched plainly, each starts only when its predecessor has
// drained and been retired; launched chained, its CTAs take their places while
// the predecessor's last CTAs still run, and wait there (chain_wait) until all
// of its memory is visible.  Every kernel of a chain calls chain_wait in every
// thread before it reads or writes anything another kernel writes or reads, so
// completion stays transitive along the chain.  A predecessor that is not a
// kernel, or that never signals, orders a chained launch like a plain one.
// Plain against chained, a pass of perf/cases.py: weno_fp64_64 47 -> 42 us,
// weno_mixed_173x301 55 -> 50, dg1_mixed_jet_512x1024 1,830 -> 1,765,
// weno_mixed_2048 697 -> 681, dg2_mixed_wave_1030 7,640 -> 7,445,
// dg3_mixed_2048 unchanged.
#pragma once

#include <cuda_runtime.h>

namespace zk {

__device__ __forceinline__ void chain_wait() {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
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
    return cudaLaunchKernelEx(&cfg, kernel, Params(args)...);
}

}  // namespace zk
