// pt_stage.h — host threads and pinned chunks for queries whose rays or answers lie in pageable memory.
//
// A cudaMemcpyAsync to or from pageable memory is staged by the calling thread, and memory the caller
// has just allocated takes its page faults there, so the copies of a query (28 bytes up and 16 down per
// ray) ran one after another.  Here each worker thread takes the next part of the query and moves it
// through a pinned chunk of its own.  (Reading an image back this way was no faster: 1.4 ms against 1.06
// for the 7 MB of 960x600, the page faults of one fresh buffer contending for the same lock.)
#pragma once

#include <cuda_runtime.h>
#include <atomic>
#include <exception>
#include <mutex>
#include <thread>
#include <vector>
#include "pt_device.h"

namespace ptb {

constexpr size_t kStageChunk = size_t(1) << 21;   // 2 MiB
constexpr int kStageWorkers = 8;                  // at most this many threads per query
// One pinned chunk from a process-wide pool of at most kStagePool chunks; get() is null when the
// pool is exhausted or pinned memory cannot be had (the caller then copies without it).
class StageChunk {
public:
    StageChunk();
    ~StageChunk();
    StageChunk(const StageChunk &) = delete;
    StageChunk &operator=(const StageChunk &) = delete;
    unsigned char *get() const { return static_cast<unsigned char *>(ptr_); }
private:
    void *ptr_ = nullptr;
};

// A copy under way when an error leaves a worker's loop ends before its chunk goes back to the pool.
struct DrainOnError {
    cudaStream_t stream;
    int entered = std::uncaught_exceptions();
    ~DrainOnError() { if(std::uncaught_exceptions() > entered) cudaStreamSynchronize(stream); }
};

bool pageable(const void *p);                     // not pinned, managed or device memory
bool on_host(const void *p);                      // the host can read and write it: not device memory
// Threads worth starting for this many parts and bytes copied either way: one per 2 MiB (1.5M rays, 66 MB: 8
// threads 3.6 ms, 4 4.0, 2 5.5; 100,000 full records, 8.4 MB: 4 threads 1.15 ms, 8 1.37, 1 1.55).
int stage_workers(size_t parts, size_t bytes);

// Runs body(worker) on up to `workers` threads (the caller's among them) with `device` current and
// rethrows the first exception once all have ended.  The body takes its parts from a shared counter, so it
// makes no difference if fewer threads could be started.
template <class F> void run_workers(int workers, int device, F body) {
    std::exception_ptr failure;
    std::mutex mutex;
    auto guarded = [&](int k) {
        try {
            if(k) PT_CUDA(cudaSetDevice(device));
            body(k);
        } catch(...) {
            std::lock_guard<std::mutex> lock(mutex);
            if(!failure) failure = std::current_exception();
        }
    };
    std::vector<std::thread> threads;
    for(int k = 1; k < workers; k++) {
        try { threads.emplace_back(guarded, k); } catch(const std::exception &) { break; }
    }
    guarded(0);
    for(auto &t : threads) t.join();
    if(failure) std::rethrow_exception(failure);
}

} // namespace ptb
