// Identity of the current CUDA context, for state cached per context: a device
// reset (cudaDeviceReset anywhere in the process) drops what the runtime held
// for the old one (symbol addresses, kernel attributes).
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>
#include <mutex>

namespace zk {

// Unique id of the calling thread's current CUDA context (driver entry
// points cuCtxGetCurrent / cuCtxGetId, looked up through the runtime so the
// library needs no link-time libcuda); false when there is none yet or the
// driver lacks them.
inline bool current_context_id(unsigned long long* id) {
    using GetCurrent = CUresult (*)(CUcontext*);
    using GetId = CUresult (*)(CUcontext, unsigned long long*);
    static GetCurrent get_current = nullptr;
    static GetId get_id = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuCtxGetCurrent", &p, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            get_current = reinterpret_cast<GetCurrent>(p);
        p = nullptr;
        if (cudaGetDriverEntryPoint("cuCtxGetId", &p, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            get_id = reinterpret_cast<GetId>(p);
    });
    if (!get_current || !get_id) return false;
    CUcontext ctx = nullptr;
    if (get_current(&ctx) != CUDA_SUCCESS || !ctx) return false;
    return get_id(ctx, id) == CUDA_SUCCESS;
}

}  // namespace zk
