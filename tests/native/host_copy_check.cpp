// HostCopier against a stand-in for the CUDA runtime: streams are memcpys done at once, each noted
// with its stream and the thread that asked for it.
#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <set>
#include <thread>
#include <vector>

#include "../../cortexsdr_b200/csrc/internal.hpp"

namespace {
std::mutex mu;
std::set<std::thread::id> copied_from;
size_t copied = 0;
cudaMemoryType kind = cudaMemoryTypeUnregistered;      // of every host pointer
}  // namespace

extern "C" {
cudaError_t cudaMemcpyAsync(void* dst, const void* src, size_t n, cudaMemcpyKind, cudaStream_t) {
    std::memcpy(dst, src, n);
    std::lock_guard<std::mutex> lk(mu);
    copied_from.insert(std::this_thread::get_id());
    copied += n;
    return cudaSuccess;
}
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* at, const void*) {
    at->type = kind;
    return cudaSuccess;
}
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) {
    *p = std::malloc(n);
    return cudaSuccess;
}
cudaError_t cudaFreeHost(void* p) {
    std::free(p);
    return cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) {
    *e = reinterpret_cast<cudaEvent_t>(1);
    return cudaSuccess;
}
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetLastError(void) { return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t) { return ""; }
}

int main() {
    std::vector<unsigned char> src(csdr::HostCopier::kSmall * 4 + 12345), dst(src.size());
    for (size_t i = 0; i < src.size(); ++i) src[i] = static_cast<unsigned char>(i * 2654435761u >> 13);
    const cudaStream_t own = reinterpret_cast<cudaStream_t>(0x1000);
    for (cudaStream_t stream : {own, cudaStreamPerThread, cudaStreamLegacy})
        for (bool up : {true, false}) {
            csdr::HostCopier copier(0, stream);
            copied_from.clear();
            copied = 0;
            std::fill(dst.begin(), dst.end(), 0);
            if (up) copier.upload(dst.data(), src.data(), src.size());
            else copier.download(dst.data(), src.data(), src.size());
            if (dst != src || copied != src.size()) {
                std::printf("bytes differ\n");
                return 1;
            }
            if (stream == cudaStreamPerThread && (copied_from.size() != 1 || !copied_from.count(std::this_thread::get_id()))) {
                std::printf("the calling thread's stream was used from %zu threads\n", copied_from.size());
                return 1;
            }
        }
    // memory the driver knows is copied, or refused, by the driver
    for (cudaMemoryType known : {cudaMemoryTypeHost, cudaMemoryTypeDevice, cudaMemoryTypeManaged}) {
        kind = known;
        csdr::HostCopier copier(0, own);
        copied_from.clear();
        copier.download(dst.data(), src.data(), src.size());
        if (copied_from.size() != 1 || !copied_from.count(std::this_thread::get_id())) {
            std::printf("memory of type %d was copied from %zu threads\n", static_cast<int>(known), copied_from.size());
            return 1;
        }
    }
    std::printf("ok\n");
    return 0;
}
