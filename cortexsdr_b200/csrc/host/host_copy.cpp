#include "host_copy.hpp"

#include <algorithm>
#include <cstring>
#include <system_error>

#include "../internal.hpp"

namespace csdr {

namespace {
constexpr size_t kSlot = 512u << 10;      // bytes of a page-locked slot
constexpr size_t kMaxWorkers = 8;

// Memory the driver knows nothing of. What it knows (page-locked, managed, device) is its to copy or to refuse.
bool pageable(const void* p) {
    cudaPointerAttributes at{};
    if (cudaPointerGetAttributes(&at, p) != cudaSuccess) {
        (void)cudaGetLastError();
        return false;
    }
    return at.type == cudaMemoryTypeUnregistered;
}
}  // namespace

// Threads and slots on first use; false (and the driver's copies from then on) where the machine has
// too few threads or denies the memory.
bool HostCopier::start() {
    if (tried_) return !workers_.empty();
    tried_ = true;
    const size_t n = std::min<size_t>(kMaxWorkers, std::thread::hardware_concurrency() / 2u);
    if (n < 2u) return false;
    if (cudaHostAlloc(reinterpret_cast<void**>(&pinned_), n * 2u * kSlot, cudaHostAllocDefault) != cudaSuccess) {
        (void)cudaGetLastError();
        pinned_ = nullptr;
        return false;
    }
    for (size_t w = 0; w < n; ++w) {
        Worker k{{pinned_ + 2u * w * kSlot, pinned_ + (2u * w + 1u) * kSlot}, {nullptr, nullptr}};
        bool ok = cudaEventCreateWithFlags(&k.event[0], cudaEventDisableTiming) == cudaSuccess;
        ok = ok && cudaEventCreateWithFlags(&k.event[1], cudaEventDisableTiming) == cudaSuccess;
        if (!ok) {
            (void)cudaGetLastError();
            if (k.event[0]) cudaEventDestroy(k.event[0]);
            break;
        }
        workers_.push_back(k);
    }
    try {
        for (size_t w = 1; w < workers_.size(); ++w) threads_.emplace_back([this, w] { serve(w); });
    } catch (const std::system_error&) {
        // fewer helpers than planned: those that started share the work
    }
    return !workers_.empty();
}

HostCopier::~HostCopier() {
    {
        std::lock_guard<std::mutex> lk(mu_);
        stop_ = true;
    }
    wake_.notify_all();
    for (auto& t : threads_) t.join();
    for (auto& w : workers_)
        for (cudaEvent_t e : w.event) cudaEventDestroy(e);
    if (pinned_) cudaFreeHost(pinned_);
}

void HostCopier::serve(size_t w) {
    cudaSetDevice(device_);
    unsigned seen = 0;
    for (;;) {
        {
            std::unique_lock<std::mutex> lk(mu_);
            wake_.wait(lk, [&] { return stop_ || generation_ != seen; });
            if (stop_) return;
            seen = generation_;
        }
        work(w);
        {
            std::lock_guard<std::mutex> lk(mu_);
            if (--busy_ == 0) done_.notify_one();
        }
    }
}

void HostCopier::work(size_t w) {
    const cudaError_t e = up_ ? work_up(workers_[w]) : work_down(workers_[w]);
    if (e != cudaSuccess) {
        int none = 0;
        error_.compare_exchange_strong(none, static_cast<int>(e));
    }
}

cudaError_t HostCopier::work_up(Worker& w) {
    for (unsigned turn = 0; !error_.load(std::memory_order_relaxed); ++turn) {
        const size_t at = next_.fetch_add(chunk_);
        if (at >= bytes_) break;
        const size_t n = std::min(chunk_, bytes_ - at);
        const unsigned s = turn & 1u;
        cudaError_t e = cudaEventSynchronize(w.event[s]);      // the slot's previous chunk has left it
        if (e != cudaSuccess) return e;
        std::memcpy(w.slot[s], src_ + at, n);
        e = cudaMemcpyAsync(dst_ + at, w.slot[s], n, cudaMemcpyHostToDevice, stream_);
        if (e == cudaSuccess) e = cudaEventRecord(w.event[s], stream_);
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

cudaError_t HostCopier::work_down(Worker& w) {
    size_t at[2] = {0, 0}, n[2] = {0, 0};                      // what is on its way into each slot (0: nothing)
    cudaError_t first = cudaSuccess;
    auto fetch = [&](unsigned s) {
        n[s] = 0;
        if (first != cudaSuccess || error_.load(std::memory_order_relaxed)) return;
        const size_t a = next_.fetch_add(chunk_);
        if (a >= bytes_) return;
        const size_t len = std::min(chunk_, bytes_ - a);
        // an upload of this context may still be reading the slot: the copy is behind it on the stream
        first = cudaMemcpyAsync(w.slot[s], src_ + a, len, cudaMemcpyDeviceToHost, stream_);
        if (first == cudaSuccess) first = cudaEventRecord(w.event[s], stream_);
        if (first == cudaSuccess) {
            at[s] = a;
            n[s] = len;
        }
    };
    fetch(0);
    fetch(1);
    for (unsigned s = 0; n[0] || n[1]; s ^= 1u) {
        if (!n[s]) continue;
        const cudaError_t e = cudaEventSynchronize(w.event[s]);
        if (e != cudaSuccess) return e;
        std::memcpy(dst_ + at[s], w.slot[s], n[s]);
        fetch(s);
    }
    return first;
}

void HostCopier::copy(void* dst, const void* src, size_t bytes, bool up) {
    if (!bytes) return;
    std::lock_guard<std::mutex> call(call_);
    // cudaStreamPerThread names another stream in every helper: its copies stay with the calling thread
    if (bytes < kSmall || stream_ == cudaStreamPerThread || !pageable(up ? src : dst) || !start()) {
        CSDR_CUDA(cudaMemcpyAsync(dst, src, bytes, up ? cudaMemcpyHostToDevice : cudaMemcpyDeviceToHost, stream_));
        // a page-locked source is read behind the call's return: wait, as for a download
        CSDR_CUDA(cudaStreamSynchronize(stream_));
        return;
    }
    dst_ = static_cast<unsigned char*>(dst);
    src_ = static_cast<const unsigned char*>(src);
    bytes_ = bytes;
    chunk_ = std::min(kSlot, std::max<size_t>(64u << 10, bytes / (2u * workers_.size()) & ~static_cast<size_t>(4095)));
    up_ = up;
    next_.store(0);
    error_.store(0);
    {
        std::lock_guard<std::mutex> lk(mu_);
        busy_ = threads_.size();
        ++generation_;
    }
    wake_.notify_all();
    work(0);
    {
        std::unique_lock<std::mutex> lk(mu_);
        done_.wait(lk, [&] { return busy_ == 0; });
    }
    if (const int e = error_.load()) throw Error(CSDR_ERR_CUDA, std::string("host copy: ") + cudaGetErrorString(static_cast<cudaError_t>(e)));
}

}  // namespace csdr
