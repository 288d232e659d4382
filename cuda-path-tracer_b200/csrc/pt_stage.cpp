// pt_stage.cpp — the pinned chunk pool (pt_stage.h).
#include <algorithm>
#include "pt_stage.h"

namespace ptb {
namespace {
constexpr int kStagePool = 2 * kStageWorkers;   // 32 MiB: two copies at full width at the same time
std::mutex g_mutex;
std::vector<void *> g_idle;                      // pinned chunks not in use
int g_chunks = 0;                                // chunks allocated
int g_users = 0;                                 // live handles (StageUser)
} // namespace

StageUser::StageUser() {
    std::lock_guard<std::mutex> lock(g_mutex);
    g_users++;
}
StageUser::~StageUser() {
    std::lock_guard<std::mutex> lock(g_mutex);
    if(--g_users) return;
    for(void *p : g_idle) { cudaFreeHost(p); g_chunks--; }   // no handle of this library is left
    g_idle.clear();
}

StageChunk::StageChunk() {
    std::lock_guard<std::mutex> lock(g_mutex);
    if(!g_idle.empty()) { ptr_ = g_idle.back(); g_idle.pop_back(); return; }
    if(g_chunks >= kStagePool) return;
    g_idle.reserve(size_t(kStagePool));
    if(cudaHostAlloc(&ptr_, kStageChunk, cudaHostAllocPortable) != cudaSuccess) { cudaGetLastError(); ptr_ = nullptr; return; }
    g_chunks++;
}
StageChunk::~StageChunk() {
    if(!ptr_) return;
    std::lock_guard<std::mutex> lock(g_mutex);
    if(g_users) g_idle.push_back(ptr_);          // reserved above: does not throw
    else { cudaFreeHost(ptr_); g_chunks--; }
}

namespace {
cudaMemoryType memory_type(const void *p) {
    cudaPointerAttributes a{};
    if(cudaPointerGetAttributes(&a, p) != cudaSuccess) { cudaGetLastError(); return cudaMemoryTypeDevice; }
    return a.type;
}
} // namespace
bool pageable(const void *p) { return memory_type(p) == cudaMemoryTypeUnregistered; }
bool on_host(const void *p) { return memory_type(p) != cudaMemoryTypeDevice; }

int stage_workers(size_t parts, size_t bytes) {
    const size_t cores = std::max(1u, std::thread::hardware_concurrency());
    return int(std::min({size_t(kStageWorkers), parts, std::max<size_t>(1, cores / 2), std::max<size_t>(1, bytes / kStageChunk)}));
}

} // namespace ptb
