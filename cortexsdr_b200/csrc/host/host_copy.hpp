// Copies between pageable host memory and the device, several host threads at a time.
#pragma once

#include <cuda_runtime.h>

#include <atomic>
#include <condition_variable>
#include <cstddef>
#include <mutex>
#include <thread>
#include <vector>

namespace csdr {

// The driver moves pageable memory through one staging buffer on the calling thread, page faults of
// a fresh destination included: 16 MB of hidden states took 0.9 ms, 64 MB of a weight 5 ms. Here up
// to eight threads each carry chunks through two page-locked slots of their own, so that faults and
// memory copies run side by side and the copy engine is kept fed. The threads and the slots (8 MB)
// belong to one context, are made on its first large copy and go with it.
class HostCopier {
public:
    HostCopier(int device, cudaStream_t stream) : device_(device), stream_(stream) {}
    ~HostCopier();
    HostCopier(const HostCopier&) = delete;
    HostCopier& operator=(const HostCopier&) = delete;
    // Behind earlier work on the stream. On return the source of an upload may be reused; a download
    // is complete. Throws Error.
    void upload(void* dst, const void* src, size_t bytes) { copy(dst, src, bytes, true); }
    // Below this many bytes a copy is the driver's (2 MB of logits took as long with the threads).
    static constexpr size_t kSmall = 4u << 20;
    void download(void* dst, const void* src, size_t bytes) { copy(dst, src, bytes, false); }

private:
    struct Worker {
        unsigned char* slot[2];
        cudaEvent_t event[2];
    };
    void copy(void* dst, const void* src, size_t bytes, bool up);
    bool start();
    void serve(size_t w);
    void work(size_t w);
    cudaError_t work_up(Worker& w);
    cudaError_t work_down(Worker& w);

    int device_;
    cudaStream_t stream_;
    std::mutex call_;                 // one copy at a time
    bool tried_ = false;
    unsigned char* pinned_ = nullptr;
    std::vector<Worker> workers_;     // [0] is the calling thread
    std::vector<std::thread> threads_;
    std::mutex mu_;
    std::condition_variable wake_, done_;
    unsigned generation_ = 0;
    size_t busy_ = 0;
    bool stop_ = false;
    // the job
    unsigned char* dst_ = nullptr;
    const unsigned char* src_ = nullptr;
    size_t bytes_ = 0, chunk_ = 0;
    bool up_ = false;
    std::atomic<size_t> next_{0};
    std::atomic<int> error_{0};
};

}  // namespace csdr
