// Copies between a caller's pageable host rows and pitched device rows.
#pragma once

#include <cuda_runtime.h>
#include <cstddef>

namespace zk {

// One context's (or batch's) staging buffers, page-locked, and the stream their
// copies run on, made at its first large copy and freed with it.  Used by one
// host thread at a time, as its owner is.
class HostStage {
public:
    HostStage() = default;
    HostStage(const HostStage&) = delete;
    HostStage& operator=(const HostStage&) = delete;
    ~HostStage() { release(); }
    void release();

    // `rows` rows of `width` bytes, dense on the host, `pitch` bytes apart on
    // the device.  Ordered after the work already on `s`; complete on return.
    cudaError_t to_device(void* dst, size_t pitch, const void* src, size_t width, size_t rows, cudaStream_t s);
    cudaError_t to_host(void* dst, const void* src, size_t pitch, size_t width, size_t rows, cudaStream_t s);

private:
    template <bool TO_DEVICE>
    cudaError_t copy(char* host, char* dev, size_t pitch, size_t width, size_t rows, cudaStream_t s);
    bool ready(const void* host, size_t bytes, size_t width, cudaStream_t s);
    bool allocate();
    char* base_ = nullptr;
    cudaStream_t stream_ = nullptr;
    cudaEvent_t before_ = nullptr;  // the work on the caller's stream
};

}  // namespace zk
