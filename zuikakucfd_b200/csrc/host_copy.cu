// Staged copies of pageable host memory.
//
// The runtime stages a pageable copy through one page-locked buffer on one
// host thread: to a fresh host array (numpy's, whose pages fault on the way)
// 2 GB/s.  Large copies are dealt to kWorkers host threads instead, each moving
// its share through two page-locked buffers of its own, so that one fills or
// empties while the other is in flight.  Milliseconds, plain and staged; "warm"
// is an array whose pages are there, and odd row lengths slow the plain copy:
//            read, fresh     read, warm     upload
//    32 MB   17.4 / 5.9      3.5 / 1.7      3.6 / 2.8
//    48 MB   23.0 / 8.7      2.4 / 2.5      3.7 / 3.4
//    96 MB   50   / 17       8.0 / 4.7     12   / 5.9
//   192 MB   92   / 34       9.0 / 9.0     17   / 8.9
//   400 MB  202   / 72      18.9 / 19      40   / 20
// The buffers are 1.5 MB in all: page-locking them takes 1 to 3 ms (nothing where
// other page-locked memory is about; 5 MB, five workers with 512 KB each, 4 to
// 5 ms), which the first staged copy pays, so that one starts at kFirstMin.
// Their release adds 0.6 ms to the context's.
//
// The workers' copies run on a stream of the staging's own, behind an event of
// the caller's: a stream handle may mean another stream in another thread
// (cudaStreamPerThread), so only the calling thread uses the caller's.
//
// Small copies, copies of memory the caller has page-locked (the runtime
// moves those directly) and copies on a stream being captured go to the
// runtime unchanged, as do all copies when page-locked memory runs out.
#include <atomic>
#include <cstring>
#include <exception>
#include <thread>

#include "host_copy.h"

namespace zk {
namespace {

constexpr int kWorkers = 3;
constexpr size_t kChunk = size_t(256) << 10;    // bytes of one staging buffer
constexpr size_t kStagedMin = size_t(32) << 20;  // smaller copies lose to the plain one where it is fast
constexpr size_t kFirstMin = size_t(64) << 20;   // as does one that makes the buffers

// Exempts this thread from the calls that another stream's capture forbids
// (page-locking memory, waiting for an event): none of them concerns it.
class CaptureExempt {
public:
    CaptureExempt() { cudaThreadExchangeStreamCaptureMode(&mode_); }
    ~CaptureExempt() { cudaThreadExchangeStreamCaptureMode(&mode_); }

private:
    cudaStreamCaptureMode mode_ = cudaStreamCaptureModeRelaxed;
};

// Rows [r0, r1) of the copy through the worker's two buffers.
template <bool TO_DEVICE>
cudaError_t move_rows(char* host, char* dev, size_t pitch, size_t width, size_t r0, size_t r1, char* stage,
                      cudaStream_t s) {
    const size_t per = kChunk / width;
    char* buf[2] = {stage, stage + kChunk};
    cudaEvent_t ev[2] = {nullptr, nullptr};
    cudaError_t e = cudaEventCreateWithFlags(&ev[0], cudaEventDisableTiming);
    if (e == cudaSuccess) e = cudaEventCreateWithFlags(&ev[1], cudaEventDisableTiming);
    size_t done = r0;  // to host: rows already unpacked
    int k = 0;
    for (size_t r = r0; r < r1 && e == cudaSuccess; r += per, ++k) {
        const size_t n = r + per < r1 ? per : r1 - r;
        const int i = k & 1;
        if (TO_DEVICE) {
            if (k >= 2) e = cudaEventSynchronize(ev[i]);
            if (e != cudaSuccess) break;
            std::memcpy(buf[i], host + r * width, n * width);
            e = cudaMemcpy2DAsync(dev + r * pitch, pitch, buf[i], width, width, n, cudaMemcpyHostToDevice, s);
            if (e == cudaSuccess) e = cudaEventRecord(ev[i], s);
        } else {
            if (k >= 2) {
                e = cudaEventSynchronize(ev[i]);
                if (e != cudaSuccess) break;
                std::memcpy(host + done * width, buf[i], per * width);
                done += per;
            }
            e = cudaMemcpy2DAsync(buf[i], width, dev + r * pitch, pitch, width, n, cudaMemcpyDeviceToHost, s);
            if (e == cudaSuccess) e = cudaEventRecord(ev[i], s);
        }
    }
    if (!TO_DEVICE)
        for (int j = k >= 2 ? k - 2 : 0; j < k && e == cudaSuccess; ++j) {
            const size_t n = done + per < r1 ? per : r1 - done;
            e = cudaEventSynchronize(ev[j & 1]);
            if (e == cudaSuccess) std::memcpy(host + done * width, buf[j & 1], n * width);
            done += n;
        }
    for (cudaEvent_t x : ev)
        if (x) cudaEventDestroy(x);
    return e;
}

}  // namespace

void HostStage::release() {
    const CaptureExempt exempt;
    if (stream_) cudaStreamDestroy(stream_);
    if (before_) cudaEventDestroy(before_);
    if (base_) cudaFreeHost(base_);
    stream_ = nullptr;
    before_ = nullptr;
    base_ = nullptr;
}

bool HostStage::allocate() {
    const CaptureExempt exempt;
    if (cudaStreamCreateWithFlags(&stream_, cudaStreamNonBlocking) == cudaSuccess &&
        cudaEventCreateWithFlags(&before_, cudaEventDisableTiming) == cudaSuccess &&
        cudaHostAlloc(reinterpret_cast<void**>(&base_), 2 * kWorkers * kChunk, cudaHostAllocPortable) == cudaSuccess)
        return true;
    release();
    cudaGetLastError();
    return false;
}

bool HostStage::ready(const void* host, size_t bytes, size_t width, cudaStream_t s) {
    if (width > kChunk || bytes < (base_ ? kStagedMin : kFirstMin)) return false;
    cudaPointerAttributes at;
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    if (cudaPointerGetAttributes(&at, host) != cudaSuccess || cudaStreamIsCapturing(s, &cs) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    if (at.type != cudaMemoryTypeUnregistered || cs != cudaStreamCaptureStatusNone) return false;
    return base_ || allocate();
}

template <bool TO_DEVICE>
cudaError_t HostStage::copy(char* host, char* dev, size_t pitch, size_t width, size_t rows, cudaStream_t s) {
    if (!ready(host, width * rows, width, s)) {
        const cudaError_t e =
            TO_DEVICE ? cudaMemcpy2DAsync(dev, pitch, host, width, width, rows, cudaMemcpyHostToDevice, s)
                      : cudaMemcpy2DAsync(host, width, dev, pitch, width, rows, cudaMemcpyDeviceToHost, s);
        return e != cudaSuccess ? e : cudaStreamSynchronize(s);
    }
    int device = 0;
    cudaError_t e = cudaGetDevice(&device);
    if (e == cudaSuccess) e = cudaEventRecord(before_, s);
    if (e == cudaSuccess) e = cudaStreamWaitEvent(stream_, before_);
    if (e != cudaSuccess) return e;
    std::atomic<int> err{cudaSuccess};
    const auto work = [&](int w) {
        const CaptureExempt exempt;
        cudaSetDevice(device);
        const cudaError_t r = move_rows<TO_DEVICE>(host, dev, pitch, width, rows * w / kWorkers,
                                                   rows * (w + 1) / kWorkers, base_ + 2 * w * kChunk, stream_);
        if (r != cudaSuccess) err = r;
    };
    std::thread threads[kWorkers];
    int started = 1;
    try {
        for (; started < kWorkers; ++started) threads[started] = std::thread(work, started);
    } catch (const std::exception&) {  // no more threads: this one takes the rest
    }
    work(0);
    for (int w = started; w < kWorkers; ++w) work(w);
    for (int w = 1; w < started; ++w) threads[w].join();
    const CaptureExempt exempt;
    e = cudaStreamSynchronize(stream_);  // uploads: every worker's last chunks
    return err != cudaSuccess ? static_cast<cudaError_t>(err.load()) : e;
}

cudaError_t HostStage::to_device(void* dst, size_t pitch, const void* src, size_t width, size_t rows, cudaStream_t s) {
    return copy<true>(static_cast<char*>(const_cast<void*>(src)), static_cast<char*>(dst), pitch, width, rows, s);
}
cudaError_t HostStage::to_host(void* dst, const void* src, size_t pitch, size_t width, size_t rows, cudaStream_t s) {
    return copy<false>(static_cast<char*>(dst), static_cast<char*>(const_cast<void*>(src)), pitch, width, rows, s);
}

}  // namespace zk
