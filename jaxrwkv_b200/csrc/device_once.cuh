// Per-device, thread-safe one-time set-up.  The library is called from several host threads for
// different devices (a framework's executor threads), so nothing here is cached in a plain global:
// every cached fact is keyed by the device ordinal and guarded by std::call_once.
#pragma once
#include <cuda_runtime.h>

#include <functional>
#include <mutex>

namespace b200wkv {

constexpr int kMaxDevices = 64;

inline int current_device() {
    int dev = -1;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return -1;
    return dev;
}

// Number of SMs of the current device (148 on a B200; an SM-limited context reports its own count).
inline int sm_count_of_current_device() {
    static std::once_flag once[kMaxDevices];
    static int count[kMaxDevices];
    const int dev = current_device();
    if (dev < 0) return 148;
    std::call_once(once[dev], [dev]() {
        int n = 0;
        if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) n = 148;
        count[dev] = n;
    });
    return count[dev];
}

// Runs `setup` (returning a cudaError_t) once per device for one call site; later calls return the
// recorded result.  Use one DeviceOnce object (static storage) per thing that needs setting up.
struct DeviceOnce {
    std::once_flag once[kMaxDevices];
    cudaError_t result[kMaxDevices];
    bool ok(const std::function<cudaError_t()>& setup) {
        const int dev = current_device();
        if (dev < 0) return setup() == cudaSuccess;
        std::call_once(once[dev], [this, dev, &setup]() { result[dev] = setup(); });
        return result[dev] == cudaSuccess;
    }
};

// A chain of kernels with the gaps between them closed: each but the first is launched with programmatic stream serialization
// (launch_behind), so that its CTAs are set up while the one in front of it finishes, and starts with word_behind(), which
// waits until that one has completed and then reads the word that decides whether there is anything to do.  The read is
// volatile and everything else comes behind the caller's branch on it, so that no load can be moved in front of the wait.
// A kernel that others are launched behind lets them in with let_next_in().  Every CTA waits before it ends, so that a kernel's
// completion stands for that of all in front of it; what it does in front of the wait must not touch what they write or read, and what they
// have written is not read through a __restrict__ pointer, which would let the compiler move the read in front of the wait.
template <typename... P, typename... A>
cudaError_t launch_in_chain(bool first, void (*kernel)(P...), dim3 grid, unsigned block, size_t smem, cudaStream_t st, A... args) {
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cfg.attrs = attr;
    cfg.numAttrs = first ? 0 : 1;
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}
template <typename... P, typename... A>
cudaError_t launch_behind(void (*kernel)(P...), dim3 grid, unsigned block, size_t smem, cudaStream_t st, A... args) {
    return launch_in_chain(false, kernel, grid, block, smem, st, args...);
}
#ifdef __CUDACC__
__device__ __forceinline__ void wait_for_grid_in_front() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ int word_behind(const int* word) {
    wait_for_grid_in_front();
    return *static_cast<const volatile int*>(word);
}
__device__ __forceinline__ void let_next_in() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
#endif

}  // namespace b200wkv
