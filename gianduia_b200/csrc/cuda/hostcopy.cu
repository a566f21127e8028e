// Staged host copies (hostcopy.h).
#include "hostcopy.h"

#include <algorithm>
#include <cstring>
#include <system_error>

namespace gnd {

HostCopy::~HostCopy() {
    {
        std::lock_guard<std::mutex> lk(m_);
        stop_.store(true);
    }
    wake_.notify_all();
    for (std::thread& t : threads_) t.join();
    if (pending_) cudaEventSynchronize(busy_);
    for (cudaEvent_t e : events_) cudaEventDestroy(e);
    if (busy_) cudaEventDestroy(busy_);
    if (stage_) cudaFreeHost(stage_);
}

bool HostCopy::pageable(const void* p) {
    cudaPointerAttributes a{};
    if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
        cudaGetLastError();
        return true;
    }
    return a.type == cudaMemoryTypeUnregistered;
}

// Room for `bytes` in the staging buffer, nothing still being read from it. False when no
// pinned memory can be had: the copy is then made plainly.
bool HostCopy::reserve(size_t bytes) {
    if (!busy_) GND_CUDA(cudaEventCreateWithFlags(&busy_, cudaEventDisableTiming));
    if (pending_) {
        GND_CUDA(cudaEventSynchronize(busy_));
        pending_ = false;
    }
    if (bytes <= stageBytes_) return true;
    if (stage_) GND_CUDA(cudaFreeHost(stage_));
    stage_ = nullptr;
    stageBytes_ = 0;
    size_t n = kChunk * 4;
    while (n < bytes) n *= 2;
    const cudaError_t e = cudaMallocHost(&stage_, n);
    if (e != cudaSuccess) {
        stage_ = nullptr;
        cudaGetLastError();
        if (e == cudaErrorMemoryAllocation) return false;
        GND_CUDA(e);
    }
    while (events_.size() < n / kChunk) {
        cudaEvent_t ev = nullptr;
        GND_CUDA(cudaEventCreateWithFlags(&ev, cudaEventDisableTiming));
        events_.push_back(ev);
    }
    stageBytes_ = n;
    return true;
}

void HostCopy::takeTasks() {
    for (int k; (k = take_.fetch_add(1)) < tasks_;) {
        (*task_)(k);
        done_.fetch_add(1);
    }
}

void HostCopy::worker() {
    cudaSetDevice(device_);
    uint64_t seen = 0;
    for (;;) {
        const auto t0 = std::chrono::steady_clock::now();
        while (round_.load() == seen && !stop_.load() && std::chrono::steady_clock::now() - t0 < kSpin) std::this_thread::yield();
        if (round_.load() == seen) {
            std::unique_lock<std::mutex> lk(m_);
            wake_.wait(lk, [&]() { return stop_.load() || round_.load() != seen; });
        }
        if (stop_.load()) return;
        {
            // entered under the mutex, so that run() does not hand out the next set (and
            // change task_ and tasks_) while a worker still looks at this one
            std::lock_guard<std::mutex> lk(m_);
            seen = round_.load();
            inside_.fetch_add(1);
        }
        takeTasks();
        inside_.fetch_sub(1);
    }
}

void HostCopy::run(int tasks, const std::function<void(int)>& f) {
    if (threads_.empty()) {
        const unsigned hw = std::thread::hardware_concurrency();
        const int n = std::min<int>(kWorkers, hw > 1 ? (int)hw - 1 : 0);
        try {
            for (int k = 0; k < n; ++k) threads_.emplace_back([this]() { worker(); });
        } catch (const std::system_error&) {
            // as many as there are: the calling thread takes the remaining tasks
        }
    }
    {
        std::lock_guard<std::mutex> lk(m_);
        while (inside_.load() != 0) std::this_thread::yield();   // late workers of the last set, about to leave
        task_ = &f;
        tasks_ = tasks;
        done_.store(0);
        take_.store(0);
        round_.fetch_add(1);
    }
    wake_.notify_all();
    takeTasks();
    while (done_.load() < tasks) std::this_thread::yield();
    // f goes out of scope: no worker may still hold it
    std::lock_guard<std::mutex> lk(m_);
    while (inside_.load() != 0) std::this_thread::yield();
    tasks_ = 0;
}

void HostCopy::parallel(size_t n, size_t piece, const std::function<void(size_t, size_t)>& f) {
    const size_t tasks = (n + piece - 1) / piece;
    if (tasks <= 1) {
        if (n) f(0, n);
        return;
    }
    run((int)tasks, [&](int k) { f((size_t)k * piece, std::min(n, ((size_t)k + 1) * piece)); });
}

void HostCopy::in(void* dst, const void* src, size_t bytes, cudaStream_t st) {
    const bool direct = !pageable(src);
    if (bytes <= kSmall || direct) {
        GND_CUDA(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, st));
        if (direct) GND_CUDA(cudaStreamSynchronize(st));   // the bus still reads it
        return;
    }
    for (size_t at = 0; at < bytes; at += kStage) {
        const size_t n = std::min(kStage, bytes - at);
        if (!reserve(n)) {
            GND_CUDA(cudaMemcpyAsync((char*)dst + at, (const char*)src + at, bytes - at, cudaMemcpyHostToDevice, st));
            return;
        }
        std::atomic<int> err{(int)cudaSuccess};
        run((int)((n + kChunk - 1) / kChunk), [&](int k) {
            const size_t o = (size_t)k * kChunk, m = std::min(kChunk, n - o);
            std::memcpy(stage_ + o, (const char*)src + at + o, m);
            const cudaError_t e = cudaMemcpyAsync((char*)dst + at + o, stage_ + o, m, cudaMemcpyHostToDevice, st);
            if (e != cudaSuccess) err = (int)e;
        });
        pending_ = true;
        GND_CUDA(cudaEventRecord(busy_, st));
        GND_CUDA((cudaError_t)err.load());
    }
}

void HostCopy::out(void* dst, const void* src, size_t bytes, cudaStream_t st) {
    if (bytes <= kSmall || !pageable(dst)) {
        GND_CUDA(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, st));
        GND_CUDA(cudaStreamSynchronize(st));
        return;
    }
    for (size_t at = 0; at < bytes; at += kStage) {
        const size_t n = std::min(kStage, bytes - at);
        if (!reserve(n)) {
            GND_CUDA(cudaMemcpyAsync((char*)dst + at, (const char*)src + at, bytes - at, cudaMemcpyDeviceToHost, st));
            GND_CUDA(cudaStreamSynchronize(st));
            return;
        }
        const int chunks = (int)((n + kChunk - 1) / kChunk);
        for (int k = 0; k < chunks; ++k) {
            const size_t o = (size_t)k * kChunk, m = std::min(kChunk, n - o);
            GND_CUDA(cudaMemcpyAsync(stage_ + o, (const char*)src + at + o, m, cudaMemcpyDeviceToHost, st));
            GND_CUDA(cudaEventRecord(events_[k], st));
        }
        std::atomic<int> err{(int)cudaSuccess};
        run(chunks, [&](int k) {
            const size_t o = (size_t)k * kChunk, m = std::min(kChunk, n - o);
            const cudaError_t e = cudaEventSynchronize(events_[k]);
            if (e != cudaSuccess) err = (int)e;
            else std::memcpy((char*)dst + at + o, stage_ + o, m);
        });
        GND_CUDA((cudaError_t)err.load());
    }
}

}  // namespace gnd
