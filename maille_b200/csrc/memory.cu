// memory.cu -- device memory of the library: one stream-ordered pool per device that keeps freed
// memory reserved for the library's next allocations.
//
// A solve handle owns several GB (matrices, factor, layouts, sort buffers of the analysis), and
// the one-shot entry point and GUI-style callers create and destroy one per solve. With plain
// cudaMalloc / cudaFree every such cycle maps and unmaps that memory again: on a B200 the first
// allocation of a handle's buffers took about 0.2 s and a handle's frees up to 0.5 s. The pool
// (cudaMemPoolCreate, release threshold at its maximum) hands the same memory back instead;
// maille_gpu_trim_memory returns what is unused to the device.
//
// Ordering: an allocation is made on the library's allocation stream and waited for before it is
// returned, so it is ready for any stream; a free first waits for the device to be idle (the same
// implicit synchronisation cudaFree performs), so no kernel still uses the memory when the pool
// may hand it out again.

#include <algorithm>
#include <atomic>
#include <cstdint>
#include <cstring>
#include <mutex>
#include <thread>
#include <vector>

#include <cuda_runtime.h>

#include "cuda_host.hpp"

namespace maille {
namespace {

struct DevicePool {
    cudaMemPool_t pool = nullptr;
    cudaStream_t stream = nullptr;
};

std::mutex g_pool_mutex;
std::vector<DevicePool> g_pools;

DevicePool& pool_of_current_device() {
    int dev = 0;
    CK(cudaGetDevice(&dev));
    std::lock_guard<std::mutex> lock(g_pool_mutex);
    if ((int)g_pools.size() <= dev) g_pools.resize(dev + 1);
    DevicePool& d = g_pools[dev];
    if (!d.pool) {
        cudaMemPoolProps props{};
        props.allocType = cudaMemAllocationTypePinned;
        props.location.type = cudaMemLocationTypeDevice;
        props.location.id = dev;
        CK(cudaMemPoolCreate(&d.pool, &props));
        uint64_t keep = UINT64_MAX;
        CK(cudaMemPoolSetAttribute(d.pool, cudaMemPoolAttrReleaseThreshold, &keep));
        CK(cudaStreamCreateWithFlags(&d.stream, cudaStreamNonBlocking));
    }
    return d;
}

}  // namespace

void* device_alloc(size_t bytes) {
    DevicePool& d = pool_of_current_device();
    void* p = nullptr;
    const cudaError_t e = cudaMallocFromPoolAsync(&p, bytes, d.pool, d.stream);
    if (e == cudaErrorMemoryAllocation) {
        cudaGetLastError();
        throw DeviceMemoryFull{{"cudaMallocFromPoolAsync of " + std::to_string(bytes) + " bytes: " + cudaGetErrorString(e)}};
    }
    CK(e);
    CK(cudaStreamSynchronize(d.stream));
    return p;
}

void device_free(void* p) {
    if (!p) return;
    DevicePool& d = pool_of_current_device();
    cudaDeviceSynchronize();
    cudaFreeAsync(p, d.stream);
    cudaStreamSynchronize(d.stream);
}

void device_free_all(const std::vector<void*>& ps) {
    bool any = false;
    for (void* p : ps) any = any || p != nullptr;
    if (!any) return;
    DevicePool& d = pool_of_current_device();
    for (void* p : ps)
        if (p) cudaFreeAsync(p, d.stream);
    cudaStreamSynchronize(d.stream);
}

namespace {

// Small pinned host slots (a handle's scalar read-back, a cancel flag). Each cudaFreeHost waits for
// every device, and a handle's destruction took tens of milliseconds in two of them; the slots are
// carved from mapped, portable chunks that stay allocated for the process, so a slot's device
// address is its host address on every device (unified addressing).
constexpr size_t kPinnedSlot = 256;
constexpr size_t kPinnedChunk = 64 * 1024;
std::mutex g_pinned_mutex;
std::vector<void*> g_pinned_free;

}  // namespace

void* pinned_slot_alloc(size_t bytes) {
    if (bytes > kPinnedSlot) throw CudaFailure{"pinned_slot_alloc: more than 256 bytes asked"};
    std::lock_guard<std::mutex> lock(g_pinned_mutex);
    if (g_pinned_free.empty()) {
        void* chunk = nullptr;
        CK(cudaHostAlloc(&chunk, kPinnedChunk, cudaHostAllocMapped | cudaHostAllocPortable));
        for (size_t off = kPinnedChunk; off >= kPinnedSlot; off -= kPinnedSlot)
            g_pinned_free.push_back(static_cast<char*>(chunk) + off - kPinnedSlot);
    }
    void* p = g_pinned_free.back();
    g_pinned_free.pop_back();
    std::memset(p, 0, kPinnedSlot);
    return p;
}

void pinned_slot_free(void* p) {
    if (!p) return;
    std::lock_guard<std::mutex> lock(g_pinned_mutex);
    g_pinned_free.push_back(p);
}

// ---- large copies between the device and pageable host memory ---------------------------------
//
// The driver copies pageable memory through one staging buffer on one thread (5.8 GB/s here, first
// touches of the caller's pages included): 27 of the 103 ms of a Tet10 40^3 solve were its results'
// way back. Here a few threads share a copy: each takes every n-th piece, moves it between the caller's
// memory and two pinned pieces of its own, and the DMA of one piece runs under the copy of the other.
// The pinned pieces stay allocated for the process (32 MB at most) until maille_gpu_trim_memory; a
// caller that finds them in use by another thread takes the driver's copy.
namespace {

constexpr size_t kPiece = size_t(2) << 20;
constexpr size_t kStagedFrom = size_t(2) * kPiece;  // smaller copies: the driver's
constexpr int kCopiers = 8;

std::mutex g_stage_mutex;
char* g_stage = nullptr;  // [kCopiers][2][kPiece]

bool page_locked(const void* p) {
    cudaPointerAttributes a{};
    if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    return a.type == cudaMemoryTypeHost || a.type == cudaMemoryTypeManaged;
}

// Copies `bytes` through the stage, up (host to device) or down; false when it did not (nothing copied).
bool staged_copy(char* dev, char* host, size_t bytes, bool up, cudaStream_t st) {
    if (bytes < kStagedFrom || page_locked(host)) return false;
    std::unique_lock<std::mutex> lock(g_stage_mutex, std::try_to_lock);
    if (!lock.owns_lock()) return false;
    if (!g_stage && cudaHostAlloc((void**)&g_stage, kCopiers * 2 * kPiece, cudaHostAllocPortable) != cudaSuccess) {
        cudaGetLastError();
        g_stage = nullptr;
        return false;
    }
    int device = 0;
    CK(cudaGetDevice(&device));
    const size_t pieces = (bytes + kPiece - 1) / kPiece;
    const int n = (int)std::min<size_t>({(size_t)kCopiers, pieces, std::max(1u, std::thread::hardware_concurrency())});
    std::atomic<int> error{(int)cudaSuccess};
    auto work = [&](int w) {
        auto ok = [&](cudaError_t e) {
            if (e != cudaSuccess) error.store((int)e);
            return e == cudaSuccess;
        };
        cudaEvent_t ev[2] = {};
        char* buf[2] = {g_stage + (size_t)(2 * w) * kPiece, g_stage + (size_t)(2 * w + 1) * kPiece};
        if (!ok(cudaSetDevice(device)) || !ok(cudaEventCreateWithFlags(&ev[0], cudaEventDisableTiming)) ||
            !ok(cudaEventCreateWithFlags(&ev[1], cudaEventDisableTiming)))
            return;
        auto size = [&](size_t p) { return std::min(kPiece, bytes - p * kPiece); };
        size_t last = pieces;  // down: the piece whose DMA is in flight
        int k = 0;
        for (size_t p = w; p < pieces; p += n, k ^= 1) {
            if (up) {
                if (!ok(cudaEventSynchronize(ev[k]))) break;  // the piece two before has left the buffer
                std::memcpy(buf[k], host + p * kPiece, size(p));
                if (!ok(cudaMemcpyAsync(dev + p * kPiece, buf[k], size(p), cudaMemcpyHostToDevice, st))) break;
                if (!ok(cudaEventRecord(ev[k], st))) break;
            } else {
                if (!ok(cudaMemcpyAsync(buf[k], dev + p * kPiece, size(p), cudaMemcpyDeviceToHost, st))) break;
                if (!ok(cudaEventRecord(ev[k], st))) break;
                if (last < pieces) {
                    if (!ok(cudaEventSynchronize(ev[k ^ 1]))) break;
                    std::memcpy(host + last * kPiece, buf[k ^ 1], size(last));
                }
                last = p;
            }
        }
        if (!up && last < pieces && ok(cudaEventSynchronize(ev[k ^ 1]))) std::memcpy(host + last * kPiece, buf[k ^ 1], size(last));
        for (auto& e : ev) {
            cudaEventSynchronize(e);  // the buffers are free again
            cudaEventDestroy(e);
        }
    };
    std::vector<std::thread> pool;
    for (int w = 1; w < n; ++w) {
        try {
            pool.emplace_back(work, w);
        } catch (...) {
            work(w);  // no thread to be had: its share on this one
        }
    }
    work(0);
    for (auto& t : pool) t.join();
    CK((cudaError_t)error.load());
    return true;
}

}  // namespace

void host_upload(void* dev, const void* host, size_t bytes, cudaStream_t st) {
    if (!bytes) return;
    if (!staged_copy(static_cast<char*>(dev), const_cast<char*>(static_cast<const char*>(host)), bytes, true, st))
        CK(cudaMemcpyAsync(dev, host, bytes, cudaMemcpyHostToDevice, st));
}

void host_download(void* host, const void* dev, size_t bytes, cudaStream_t st) {
    if (!bytes) return;
    if (!staged_copy(const_cast<char*>(static_cast<const char*>(dev)), static_cast<char*>(host), bytes, false, st))
        CK(cudaMemcpyAsync(host, dev, bytes, cudaMemcpyDeviceToHost, st));
}

int device_sms() {
    constexpr int kMaxDevices = 64;
    static std::atomic<int> cached[kMaxDevices];
    int dev = 0;
    CK(cudaGetDevice(&dev));
    if (dev < 0 || dev >= kMaxDevices) {
        int sms = 0;
        CK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
        return sms;
    }
    int sms = cached[dev].load(std::memory_order_relaxed);
    if (sms <= 0) {
        CK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
        cached[dev].store(sms, std::memory_order_relaxed);
    }
    return sms;
}

int32_t trim_device_memory(int device) {
    int prev = 0;
    if (cudaGetDevice(&prev) != cudaSuccess || cudaSetDevice(device) != cudaSuccess) return -1;
    int32_t status = 0;
    {
        std::lock_guard<std::mutex> lock(g_pool_mutex);
        if (device < (int)g_pools.size() && g_pools[device].pool) {
            cudaDeviceSynchronize();
            status = cudaMemPoolTrimTo(g_pools[device].pool, 0) == cudaSuccess ? 0 : -1;
        }
    }
    if (std::unique_lock<std::mutex> lock(g_stage_mutex, std::try_to_lock); lock.owns_lock() && g_stage) {
        cudaFreeHost(g_stage);
        g_stage = nullptr;
    }
    cudaSetDevice(prev);
    return status;
}

}  // namespace maille
