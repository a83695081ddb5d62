// Workspace memory of the device-resident solvers.
//
// A solve needs O(l n) or O(m n) device scratch (Krylov vectors), a small
// pinned slot for the per-cycle read-back, a stream and a graph.  Taking the
// device scratch from cudaMalloc/cudaFree on every call costs milliseconds
// and synchronises the device (cudaFree); here it comes stream-ordered from
// a library-owned memory pool per device whose freed blocks stay reserved
// for the next solve (release threshold: unlimited).  The pool therefore
// holds the largest workspace used so far until hpb_solver_memory_release()
// or process exit.  Pinned slots are cached per host thread.
#include <mutex>
#include <new>
#include <vector>

#include "hpb_fused.cuh"

namespace hpb {
namespace fused {
namespace {

constexpr int kMaxDevices = 64;
// The analyses' pool holds on to freed memory while it has at most this much
// in all, in use or not (about 58 bytes a row and triangle: both triangles of
// nine million rows); what is beyond goes back to the device when a stream or
// the device is next synchronised.  (With 256 MB, callers that hold three
// matrices' analyses of a million rows paid 15 ms a set-up for memory going
// back and forth.)
constexpr uint64_t kAnalysisKeep = uint64_t(1) << 30;
std::mutex g_pool_mutex;
enum PoolKind { POOL_WORKSPACE = 0, POOL_ANALYSIS = 1 };
cudaMemPool_t g_pools[2][kMaxDevices] = {};

cudaMemPool_t pool_for(int device, PoolKind kind) {
    if (device < 0 || device >= kMaxDevices) return nullptr;
    std::lock_guard<std::mutex> lock(g_pool_mutex);
    if (g_pools[kind][device] == nullptr) {
        cudaMemPoolProps props{};
        props.allocType = cudaMemAllocationTypePinned;
        props.location.type = cudaMemLocationTypeDevice;
        props.location.id = device;
        cudaMemPool_t pool = nullptr;
        if (cudaMemPoolCreate(&pool, &props) != cudaSuccess) return nullptr;
        uint64_t keep = kind == POOL_WORKSPACE ? ~uint64_t(0) : kAnalysisKeep;
        cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep);
        g_pools[kind][device] = pool;
    }
    return g_pools[kind][device];
}

void* alloc_from(PoolKind kind, size_t bytes, cudaStream_t stream) {
    int device = 0;
    if (cudaGetDevice(&device) != cudaSuccess) return nullptr;
    cudaMemPool_t pool = pool_for(device, kind);
    if (!pool) return nullptr;
    void* p = nullptr;
    if (cudaMallocFromPoolAsync(&p, bytes ? bytes : 16, pool, stream) != cudaSuccess) {
        cudaGetLastError();
        return nullptr;
    }
    return p;
}

constexpr size_t kPinnedSlot = 4096;

struct PinnedCache {
    std::vector<void*> free_slots;
    ~PinnedCache() {
        for (void* p : free_slots) cudaFreeHost(p);  // may fail after CUDA shut down at exit: nothing to do then
    }
};
thread_local PinnedCache t_pinned;

}  // namespace

void* pool_alloc(size_t bytes, cudaStream_t stream) { return alloc_from(POOL_WORKSPACE, bytes, stream); }
void* analysis_alloc(size_t bytes, cudaStream_t stream) { return alloc_from(POOL_ANALYSIS, bytes, stream); }
void analysis_free(void* p, cudaStream_t stream) {
    if (p) cudaFreeAsync(p, stream);
}

void pool_free(void* p, cudaStream_t stream) {
    if (p) cudaFreeAsync(p, stream);
}

void* pinned_acquire(size_t bytes) {
    if (bytes > kPinnedSlot) return nullptr;
    if (!t_pinned.free_slots.empty()) {
        void* p = t_pinned.free_slots.back();
        t_pinned.free_slots.pop_back();
        return p;
    }
    void* p = nullptr;
    return cudaMallocHost(&p, kPinnedSlot) == cudaSuccess ? p : nullptr;
}

void pinned_release(void* p) {
    if (p) t_pinned.free_slots.push_back(p);
}

int SolverWorkspace::open(size_t pinned_bytes) {
    if (cudaStreamCreateWithFlags(&stream, cudaStreamNonBlocking) != cudaSuccess ||
        cudaEventCreateWithFlags(&ev, cudaEventDisableTiming) != cudaSuccess)
        return HPB_ERROR_CUDA;
    pinned = pinned_acquire(pinned_bytes);
    return pinned ? HPB_SUCCESS : HPB_ERROR_OUT_OF_MEMORY;
}

void* SolverWorkspace::alloc(size_t bytes) {
    void* p = pool_alloc(bytes, stream);
    if (p) dev.push_back(p);
    return p;
}

void SolverWorkspace::free_last() {
    pool_free(dev.back(), stream);
    dev.pop_back();
}

SolverWorkspace::~SolverWorkspace() {
    if (stream) cudaStreamSynchronize(stream);
    if (exec) cudaGraphExecDestroy(exec);
    if (graph) cudaGraphDestroy(graph);
    for (void* p : dev) pool_free(p, stream);
    if (stream) cudaStreamSynchronize(stream);
    pinned_release(pinned);
    if (ev) cudaEventDestroy(ev);
    if (stream) cudaStreamDestroy(stream);
}

}  // namespace fused
}  // namespace hpb

extern "C" int hpb_solver_memory_release(void) {
    std::lock_guard<std::mutex> lock(hpb::fused::g_pool_mutex);
    int status = HPB_SUCCESS;
    for (auto& kind : hpb::fused::g_pools)
        for (cudaMemPool_t pool : kind)
            if (pool && cudaMemPoolTrimTo(pool, 0) != cudaSuccess) status = HPB_ERROR_CUDA;
    return status;
}
