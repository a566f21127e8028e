// HostCopy (csrc/cuda/hostcopy.h) on a stand-in for the CUDA runtime: streams are queues that run
// when they are waited for, pinned and device memory are address ranges. The first argument
// names the case; exit code 0 when it holds.
#include "hostcopy.h"

#include <dlfcn.h>
#include <pthread.h>

#include <cerrno>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <functional>
#include <mutex>

namespace {
struct Range {
    const char* p;
    size_t n;
    cudaMemoryType type;
};
std::mutex gMu;
std::vector<Range> gRanges;                       // everything else is pageable
std::vector<std::function<void()>> gQueue;        // the one stream
bool gNoPinned = false;                           // pinned memory cannot be had
int gDirect = 0;                                  // copies between two ranges neither of which is pinned or pageable
int gThreads = -1;                                // threads that can still be started (-1: any number)

cudaMemoryType typeOf(const void* p) {
    for (const Range& r : gRanges)
        if ((const char*)p >= r.p && (const char*)p < r.p + r.n) return r.type;
    return cudaMemoryTypeUnregistered;
}
void drain() {
    for (auto& f : gQueue) f();
    gQueue.clear();
}
}  // namespace

extern "C" {
int pthread_create(pthread_t* t, const pthread_attr_t* a, void* (*f)(void*), void* arg) {
    if (gThreads == 0) return EAGAIN;
    if (gThreads > 0) --gThreads;
    using Create = int (*)(pthread_t*, const pthread_attr_t*, void* (*)(void*), void*);
    return reinterpret_cast<Create>(dlsym(RTLD_NEXT, "pthread_create"))(t, a, f, arg);
}
cudaError_t cudaMemcpyAsync(void* dst, const void* src, size_t n, cudaMemcpyKind, cudaStream_t) {
    std::lock_guard<std::mutex> lk(gMu);
    const bool pageable = typeOf(dst) == cudaMemoryTypeUnregistered || typeOf(src) == cudaMemoryTypeUnregistered;
    if (typeOf(dst) == cudaMemoryTypeDevice && typeOf(src) == cudaMemoryTypeDevice) ++gDirect;
    auto copy = [=]() { std::memcpy(dst, src, n); };
    if (pageable) {   // staged before the call returns
        drain();
        copy();
    } else {
        gQueue.push_back(copy);
    }
    return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t) {
    std::lock_guard<std::mutex> lk(gMu);
    drain();
    return cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) {
    *e = (cudaEvent_t)std::malloc(1);
    return cudaSuccess;
}
cudaError_t cudaEventDestroy(cudaEvent_t e) {
    std::free(e);
    return cudaSuccess;
}
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaStreamSynchronize(nullptr); }
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) {
    if (gNoPinned) return cudaErrorMemoryAllocation;
    std::lock_guard<std::mutex> lk(gMu);
    *p = std::malloc(n);
    gRanges.push_back({(const char*)*p, n, cudaMemoryTypeHost});
    return cudaSuccess;
}
cudaError_t cudaFreeHost(void* p) {
    std::lock_guard<std::mutex> lk(gMu);
    for (size_t k = 0; k < gRanges.size(); ++k)
        if (gRanges[k].p == p) gRanges.erase(gRanges.begin() + (long)k--);
    std::free(p);
    return cudaSuccess;
}
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void* p) {
    std::lock_guard<std::mutex> lk(gMu);
    a->type = typeOf(p);
    return cudaSuccess;
}
cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t) { return "error"; }
cudaError_t cudaMalloc(void**, size_t) { return cudaErrorMemoryAllocation; }
cudaError_t cudaFree(void*) { return cudaSuccess; }
cudaError_t cudaMallocAsync(void**, size_t, cudaStream_t) { return cudaErrorMemoryAllocation; }
cudaError_t cudaFreeAsync(void*, cudaStream_t) { return cudaSuccess; }
}

namespace {
struct Memory {
    std::vector<unsigned char> bytes;
    Memory(size_t n, cudaMemoryType type, int seed) : bytes(n) {
        for (size_t k = 0; k < n; ++k) bytes[k] = (unsigned char)(k * 31 + (k >> 10) + seed);
        if (type != cudaMemoryTypeUnregistered) gRanges.push_back({(const char*)bytes.data(), n, type});
    }
    ~Memory() {
        for (size_t k = 0; k < gRanges.size(); ++k)
            if (gRanges[k].p == (const char*)bytes.data()) gRanges.erase(gRanges.begin() + (long)k--);
    }
};

// in and out of every size give the bytes, and the source may be reused when in() returns
bool roundTrip(cudaMemoryType hostType) {
    gnd::HostCopy c(0);
    for (size_t n : {size_t(1), size_t(4096), size_t(256) << 10, (size_t(256) << 10) + 1, (size_t(3) << 20) + 5,
                     (size_t(32) << 20) + 77}) {
        Memory src(n, hostType, 1), dev(n, cudaMemoryTypeDevice, 2), dst(n, hostType, 3);
        const std::vector<unsigned char> want = src.bytes;
        c.in(dev.bytes.data(), src.bytes.data(), n, nullptr);
        std::fill(src.bytes.begin(), src.bytes.end(), 0xEE);
        c.out(dst.bytes.data(), dev.bytes.data(), n, nullptr);
        if (dst.bytes != want) {
            std::printf("wrong bytes at size %zu\n", n);
            return false;
        }
    }
    return true;
}
}  // namespace

int main(int argc, char** argv) {
    const std::string what = argc > 1 ? argv[1] : "";
    if (what == "pageable") return roundTrip(cudaMemoryTypeUnregistered) ? 0 : 1;
    if (what == "pinned") return roundTrip(cudaMemoryTypeHost) ? 0 : 1;
    if (what == "no-pinned-memory") {
        gNoPinned = true;
        return roundTrip(cudaMemoryTypeUnregistered) ? 0 : 1;
    }
    if (what == "no-threads" || what == "one-thread") {
        gThreads = what == "one-thread" ? 1 : 0;
        return roundTrip(cudaMemoryTypeUnregistered) ? 0 : 1;
    }
    if (what == "device-pointers") {   // the runtime copies or refuses them; the host cannot read them
        return roundTrip(cudaMemoryTypeDevice) && gDirect == 2 * 6 ? 0 : 1;
    }
    return 2;
}
