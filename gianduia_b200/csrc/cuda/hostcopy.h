// Copies between device memory and a caller's pageable host memory through a pinned staging
// buffer, the host side shared by a few threads. A plain cudaMemcpy of pageable memory runs
// one thread's memcpy (and, into fresh memory, one thread's page faults) at about 20 GB/s in
// turn with the bus: a 12.6 MB image came back in 0.8 ms; four threads beside the bus take
// 0.3 ms.
#pragma once
#include <atomic>
#include <chrono>
#include <condition_variable>
#include <functional>
#include <mutex>
#include <thread>
#include <vector>

#include "runtime.h"

namespace gnd {

// One per context, used with the context's mutex held. The threads start with the first
// large copy and end with the context, as the staging memory (at most kStage bytes).
class HostCopy {
public:
    static constexpr size_t kStage = size_t(32) << 20, kChunk = size_t(1) << 20, kSmall = size_t(256) << 10;
    static constexpr int kWorkers = 3;
    explicit HostCopy(int device) : device_(device) {}
    ~HostCopy();
    HostCopy(const HostCopy&) = delete;
    HostCopy& operator=(const HostCopy&) = delete;
    // Queues the copy of src (host) to dst (device) on st; src may be reused on return.
    void in(void* dst, const void* src, size_t bytes, cudaStream_t st);
    // Copies src (device) to dst (host) after the work queued on st; dst is complete on return.
    void out(void* dst, const void* src, size_t bytes, cudaStream_t st);
    // f(begin, end) over pieces of [0, n), on the calling thread and the workers.
    void parallel(size_t n, size_t piece, const std::function<void(size_t, size_t)>& f);

private:
    bool reserve(size_t bytes);
    void run(int tasks, const std::function<void(int)>& f);   // f(0) .. f(tasks - 1), all done on return
    void worker();
    // Memory that only the host can read; the rest (pinned, managed, device) is the runtime's to copy.
    static bool pageable(const void* p);

    const int device_;
    char* stage_ = nullptr;
    size_t stageBytes_ = 0;
    std::vector<cudaEvent_t> events_;      // one per chunk of the staging buffer
    cudaEvent_t busy_ = nullptr;           // the last copy out of the staging buffer
    bool pending_ = false;
    std::vector<std::thread> threads_;
    // One set of tasks at a time: round_ counts them, take_ holds the next task's index.
    // A worker looks for the next set for kSpin before it sleeps: the copies of one call follow
    // each other closely, and waking a sleeping thread costs more than a megabyte's copy.
    static constexpr std::chrono::microseconds kSpin{100};
    std::mutex m_;
    std::condition_variable wake_;
    std::atomic<uint64_t> round_{0};
    std::atomic<int> take_{0}, done_{0}, inside_{0};
    std::atomic<bool> stop_{false};
    const std::function<void(int)>* task_ = nullptr;
    int tasks_ = 0;
    void takeTasks();
};

}  // namespace gnd
