// Identity of the current CUDA context, for state cached per context: a device
// reset (cudaDeviceReset anywhere in the process) drops what the runtime held
// for the old one (symbol addresses and contents, kernel attributes).
#pragma once

#include <atomic>
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

// What has been set up in each device's current context, once per kind of
// set-up (a static object).
class PerContext {
public:
    // Runs `set` unless it has run in the current device's context; any host
    // thread may call.  Without a context id (old driver) it runs every time.
    template <typename Set>
    cudaError_t once(Set set) {
        int dev = 0;
        cudaError_t e = cudaGetDevice(&dev);
        if (e != cudaSuccess) return e;
        unsigned long long id = 0;
        const bool slot = dev >= 0 && dev < 64;
        if (slot && current_context_id(&id) && done_[dev].load(std::memory_order_acquire) == id + 1) return cudaSuccess;
        e = set();
        // the runtime calls above made the context current if it was not
        if (e == cudaSuccess && slot && current_context_id(&id))
            done_[dev].store(id + 1, std::memory_order_release);
        return e;
    }

private:
    std::atomic<unsigned long long> done_[64] = {};  // context id + 1
};

}  // namespace zk
