// cuda_host.hpp -- host-side CUDA helpers shared by the handle and batch drivers: error
// checking that throws to the C ABI boundary, device allocation and upload, a wall clock.
#pragma once

#include <chrono>
#include <cstdint>
#include <string>
#include <vector>

#include <cuda_runtime.h>
#include <nvtx3/nvToolsExt.h>

namespace maille {

// A named range on a profiler's host timeline (NVTX, header-only: without a tool attached the
// calls do nothing). One per entry point and per major phase.
struct NvtxRange {
    explicit NvtxRange(const char* name) { nvtxRangePushA(name); }
    ~NvtxRange() { nvtxRangePop(); }
    NvtxRange(const NvtxRange&) = delete;
    NvtxRange& operator=(const NvtxRange&) = delete;
};

struct CudaFailure {
    std::string what;
};
// device_alloc found no room. What holds a coarse correction (coarse.cuh) gives it up and tries again.
struct DeviceMemoryFull : CudaFailure {};

#define CK(call)                                                                             \
    do {                                                                                     \
        cudaError_t e_ = (call);                                                             \
        if (e_ != cudaSuccess)                                                               \
            throw ::maille::CudaFailure{std::string(#call) + ": " + cudaGetErrorString(e_)}; \
    } while (0)

inline double now_ms() {
    return std::chrono::duration<double, std::milli>(
               std::chrono::steady_clock::now().time_since_epoch())
        .count();
}

// Device memory from the library's per-device pool (memory.cu): an allocation is ready for any
// stream when it returns; a free waits for the device to be idle, like cudaFree.
void* device_alloc(size_t bytes);
void device_free(void* p);
// Frees every non-null pointer of `ps` on the pool's stream and waits for it; the caller has
// synchronised every stream that used them (a handle's destructor: its own stream).
void device_free_all(const std::vector<void*>& ps);
// Returns the pool's unused memory of `device` to the device (0, or -1 on a CUDA error).
int32_t trim_device_memory(int device);
// A zeroed pinned host slot of at most 256 bytes, mapped and portable (its device address equals
// its host address); slots are reused, never returned to the driver.
void* pinned_slot_alloc(size_t bytes);
void pinned_slot_free(void* p);
// Copies between the device and host memory, enqueued on st. A large copy from or to pageable memory is
// shared by several threads (memory.cu): an upload has read the host memory when it returns, a
// download has written it; smaller ones and page-locked memory are plain cudaMemcpyAsync.
void host_upload(void* dev, const void* host, size_t bytes, cudaStream_t st);
void host_download(void* host, const void* dev, size_t bytes, cudaStream_t st);
// Streaming multiprocessors of the current device (cudaDevAttrMultiProcessorCount, cached per
// device): grid caps are multiples of it.
int device_sms();

template <typename T>
T* dalloc(size_t n) {
    if (n == 0) n = 1;
    return static_cast<T*>(device_alloc(n * sizeof(T)));
}

template <typename T>
T* dupload(const T* src, size_t n, cudaStream_t st) {
    T* d = dalloc<T>(n);
    if (n && src) host_upload(d, src, n * sizeof(T), st);
    return d;
}

inline void dfree(void* p) { device_free(p); }

// A second stream beside a main one, for work that the main stream's next steps do not need: fork()
// makes it wait for everything enqueued on the main stream, join() makes the main stream wait for it.
// Its work may use the main stream's buffers between the two; the destructor waits for it.
struct SideStream {
    cudaStream_t st = nullptr;
    cudaEvent_t from = nullptr, to = nullptr;
    bool forked = false;
    cudaStream_t fork(cudaStream_t main) {
        if (!st) {
            CK(cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking));
            CK(cudaEventCreateWithFlags(&from, cudaEventDisableTiming));
            CK(cudaEventCreateWithFlags(&to, cudaEventDisableTiming));
        }
        CK(cudaEventRecord(from, main));
        CK(cudaStreamWaitEvent(st, from, 0));
        forked = true;
        return st;
    }
    void join(cudaStream_t main) {
        if (!forked) return;
        forked = false;
        CK(cudaEventRecord(to, st));
        CK(cudaStreamWaitEvent(main, to, 0));
    }
    void finish() {
        if (st) {
            cudaStreamSynchronize(st);
            cudaStreamDestroy(st);
        }
        if (from) cudaEventDestroy(from);
        if (to) cudaEventDestroy(to);
        st = nullptr;
        from = to = nullptr;
    }
    ~SideStream() { finish(); }
};

constexpr double kDefaultTol = 1e-12;      // iterative.rs:9
constexpr int32_t kDefaultMaxIter = 10000;  // iterative.rs:11
constexpr double kShifts[6] = {0.0, 1e-3, 1e-2, 1e-1, 1.0, 10.0};  // iterative.rs:14

void set_last_error(const std::string& message);

}  // namespace maille
