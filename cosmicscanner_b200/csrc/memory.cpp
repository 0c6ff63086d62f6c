// Device memory pool and the per-thread cuBLAS / cuSOLVER handles.
#include <cublas_v2.h>
#include <cuda_runtime.h>
#include <cusolverDn.h>

#include <atomic>
#include <cstdint>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <string>
#include <utility>
#include <vector>

#include "cs_internal.h"

namespace cs {

namespace {
constexpr int kMaxDevices = 64;
std::once_flag g_pool_once[kMaxDevices];

void prepare_pool(int dev) {
    std::call_once(g_pool_once[dev], [dev] {
        cudaMemPool_t pool;
        if (cudaDeviceGetDefaultMemPool(&pool, dev) != cudaSuccess) return;
        // keep freed blocks reserved for this process (released when the context ends)
        uint64_t keep = UINT64_MAX;
        cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep);
    });
}

// CS_B200_POISON_ALLOC=1 fills every new block with 0xFF bytes (NaN as FP64), so that a read of
// memory no kernel has written shows up in the results instead of depending on what the pool
// held before.
bool poison_allocations() {
    static const bool on = [] {
        const char* v = std::getenv("CS_B200_POISON_ALLOC");
        return v && v[0] == '1';
    }();
    return on;
}

// CS_B200_ALLOC_LIMIT=bytes:count refuses the process's first `count` blocks above a size as a full device
// would, for tests of what callers do then and when there is room again.
bool refuse_allocation(size_t bytes) {
    static size_t limit = SIZE_MAX;
    static std::atomic<long long> left{0};
    static const bool set = [] {
        const char* v = std::getenv("CS_B200_ALLOC_LIMIT");
        const char* c = v ? std::strchr(v, ':') : nullptr;
        if (!c) return false;
        limit = (size_t)std::strtoull(v, nullptr, 10);
        left = std::atoll(c + 1);
        return true;
    }();
    return set && bytes > limit && left.fetch_sub(1) > 0;
}

thread_local cublasHandle_t t_blas[kMaxDevices] = {};
thread_local cusolverDnHandle_t t_solver[kMaxDevices] = {};
// Handles given back by threads that ended (release_thread_handles), reused by new threads:
// creating and destroying them per request thread costs device-wide synchronisations.
std::mutex g_handle_mu;
std::vector<cublasHandle_t> g_free_blas[kMaxDevices];
std::vector<cusolverDnHandle_t> g_free_solver[kMaxDevices];

// Free page-locked blocks, by size (a power of two), at most kPinnedKeep bytes of them.
constexpr size_t kPinnedKeep = size_t(32) << 20;
std::mutex g_pinned_mu;
std::vector<std::pair<size_t, void*>> g_pinned;
size_t g_pinned_bytes = 0;

void trim_pinned() {
    std::lock_guard<std::mutex> lk(g_pinned_mu);
    for (auto& b : g_pinned) cudaFreeHost(b.second);
    g_pinned.clear();
    g_pinned_bytes = 0;
}

size_t pinned_size(size_t bytes) {
    size_t n = 4096;
    while (n < bytes) n *= 2;
    return n;
}

// Gives the pool's reserved free blocks back to the device (after the device has finished
// with them), when an allocation found no room: the pool keeps freed blocks reserved, which
// neither a block of another size nor the libraries' own allocations can use.
void trim_pool(int dev) {
    cudaMemPool_t pool;
    if (cudaDeviceSynchronize() == cudaSuccess && cudaDeviceGetDefaultMemPool(&pool, dev) == cudaSuccess)
        cudaMemPoolTrimTo(pool, 0);
    cudaGetLastError();
    trim_pinned();
}
}  // namespace

void* device_alloc(size_t bytes) {
    int dev = 0;
    CS_CUDA(cudaGetDevice(&dev));
    if (dev >= 0 && dev < kMaxDevices) prepare_pool(dev);
    void* p = nullptr;
    const bool refused = refuse_allocation(bytes);
    cudaError_t e = refused ? cudaErrorMemoryAllocation : cudaMallocAsync(&p, bytes, 0);
    if (e == cudaErrorMemoryAllocation && !refused) {
        // The pool keeps freed blocks reserved; when the device has no room left for a new
        // block, hand the reserved free blocks back and try once more.
        cudaGetLastError();
        trim_pool(dev);
        e = cudaMallocAsync(&p, bytes, 0);
    }
    if (e != cudaSuccess) {
        cudaGetLastError();
        const std::string msg = std::string("device allocation of ") + std::to_string(bytes) +
                                " bytes failed: " + cudaGetErrorString(e);
        if (e == cudaErrorMemoryAllocation) throw OutOfMemory(CS_ERR_CUDA, msg);
        fail(CS_ERR_CUDA, msg);
    }
    if (poison_allocations()) CS_CUDA(cudaMemsetAsync(p, 0xFF, bytes, 0));
    // usable from every stream once the allocation is ordered on the legacy stream
    CS_CUDA(cudaStreamSynchronize(0));
    return p;
}

size_t device_room() {
    size_t room = 0, total = 0;
    CS_CUDA(cudaMemGetInfo(&room, &total));
    int dev = 0;
    cudaMemPool_t pool;
    uint64_t reserved = 0, used = 0;
    if (cudaGetDevice(&dev) == cudaSuccess && cudaDeviceGetDefaultMemPool(&pool, dev) == cudaSuccess &&
        cudaMemPoolGetAttribute(pool, cudaMemPoolAttrReservedMemCurrent, &reserved) == cudaSuccess &&
        cudaMemPoolGetAttribute(pool, cudaMemPoolAttrUsedMemCurrent, &used) == cudaSuccess && reserved > used)
        room += reserved - used;
    cudaGetLastError();
    return room;
}

void* pinned_alloc(size_t bytes) {
    const size_t n = pinned_size(bytes);
    {
        std::lock_guard<std::mutex> lk(g_pinned_mu);
        for (size_t i = 0; i < g_pinned.size(); ++i)
            if (g_pinned[i].first == n) {
                void* p = g_pinned[i].second;
                g_pinned[i] = g_pinned.back();
                g_pinned.pop_back();
                g_pinned_bytes -= n;
                return p;
            }
    }
    void* p = nullptr;
    const cudaError_t e = cudaHostAlloc(&p, n, cudaHostAllocMapped | cudaHostAllocPortable);
    if (e != cudaSuccess) {
        cudaGetLastError();
        fail(CS_ERR_CUDA, std::string("page-locked allocation of ") + std::to_string(n) +
                              " bytes failed: " + cudaGetErrorString(e));
    }
    return p;
}

void pinned_free(void* p, size_t bytes) noexcept {
    if (!p) return;
    const size_t n = pinned_size(bytes);
    try {
        std::lock_guard<std::mutex> lk(g_pinned_mu);
        if (g_pinned_bytes + n <= kPinnedKeep) {
            g_pinned.emplace_back(n, p);
            g_pinned_bytes += n;
            return;
        }
    } catch (...) {
    }
    cudaFreeHost(p);
}

cublasHandle_t shared_blas() {
    int dev = 0;
    CS_CUDA(cudaGetDevice(&dev));
    if (dev < 0 || dev >= kMaxDevices) fail(CS_ERR_CUDA, "device ordinal out of range");
    if (!t_blas[dev]) {
        std::lock_guard<std::mutex> lk(g_handle_mu);
        if (!g_free_blas[dev].empty()) {
            t_blas[dev] = g_free_blas[dev].back();
            g_free_blas[dev].pop_back();
        }
    }
    if (!t_blas[dev] && cublasCreate(&t_blas[dev]) != CUBLAS_STATUS_SUCCESS) {
        t_blas[dev] = nullptr;
        trim_pool(dev);
        if (cublasCreate(&t_blas[dev]) != CUBLAS_STATUS_SUCCESS) {
            t_blas[dev] = nullptr;
            fail(CS_ERR_CUDA, "cublasCreate failed");
        }
    }
    return t_blas[dev];
}

cusolverDnHandle_t shared_solver() {
    int dev = 0;
    CS_CUDA(cudaGetDevice(&dev));
    if (dev < 0 || dev >= kMaxDevices) fail(CS_ERR_CUDA, "device ordinal out of range");
    if (!t_solver[dev]) {
        std::lock_guard<std::mutex> lk(g_handle_mu);
        if (!g_free_solver[dev].empty()) {
            t_solver[dev] = g_free_solver[dev].back();
            g_free_solver[dev].pop_back();
        }
    }
    if (!t_solver[dev] && cusolverDnCreate(&t_solver[dev]) != CUSOLVER_STATUS_SUCCESS) {
        t_solver[dev] = nullptr;
        trim_pool(dev);
        if (cusolverDnCreate(&t_solver[dev]) != CUSOLVER_STATUS_SUCCESS) {
            t_solver[dev] = nullptr;
            fail(CS_ERR_CUDA, "cusolverDnCreate failed");
        }
    }
    return t_solver[dev];
}

void release_thread_handles() noexcept {
    // back to the free lists, bound to the legacy stream (the thread's own stream is about to
    // be destroyed; every user sets its stream before use)
    std::lock_guard<std::mutex> lk(g_handle_mu);
    for (int d = 0; d < kMaxDevices; ++d) {
        if (t_blas[d]) {
            cublasSetStream(t_blas[d], 0);
            g_free_blas[d].push_back(t_blas[d]);
            t_blas[d] = nullptr;
        }
        if (t_solver[d]) {
            cusolverDnSetStream(t_solver[d], 0);
            g_free_solver[d].push_back(t_solver[d]);
            t_solver[d] = nullptr;
        }
    }
}

namespace {
thread_local cudaStream_t g_free_stream = nullptr;
}

void set_thread_free_stream(cudaStream_t s) { g_free_stream = s; }

namespace {
thread_local int t_free_scopes = 0;
}

FreeScope::FreeScope() {
    if (t_free_scopes++ == 0 && !g_free_stream) cudaDeviceSynchronize();
}
FreeScope::~FreeScope() { --t_free_scopes; }

void wait_before_free() noexcept {
    if (g_free_stream) cudaStreamSynchronize(g_free_stream);
    else if (!t_free_scopes) cudaDeviceSynchronize();
}

void device_free(void* p) noexcept {
    if (!p) return;
    if (g_free_stream) {
        // ordered after the work this thread queued on its stream (the pool reuses the block
        // only once the free has executed)
        cudaFreeAsync(p, g_free_stream);
        return;
    }
    if (!t_free_scopes) cudaDeviceSynchronize();
    cudaFreeAsync(p, 0);
}

}  // namespace cs
