// host_util.h — host-side helpers shared by the C-ABI implementation files.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

#include "../../include/helio_cull.h"

// Formats `fmt` into the calling thread's helio_last_error() and returns `code`.
int32_t helio_fail(int32_t code, const char* fmt, ...);

#define HELIO_CK(call)                                                                                 \
    do {                                                                                               \
        cudaError_t e_ = (call);                                                                       \
        if (e_ != cudaSuccess) return helio_fail(HELIO_ERR_CUDA, "%s: %s", #call, cudaGetErrorString(e_)); \
    } while (0)

#define HELIO_ARG(cond, msg)                                            \
    do {                                                                \
        if (!(cond)) return helio_fail(HELIO_ERR_INVALID_ARG, "%s", msg); \
    } while (0)

namespace helio {

inline cudaStream_t as_stream(void* s) { return reinterpret_cast<cudaStream_t>(s); }

// Owned device allocation with grow-only semantics.
// Bytes to hold for `need` when `held` bytes are allocated: a buffer that must grow takes at
// least 1.5x what it held, so that a buffer which keeps growing (a server's batches of
// changing shapes) is reallocated a logarithmic number of times (cudaFree synchronises the
// whole device). A first allocation takes exactly `need`.
inline size_t grow_capacity(size_t need, size_t held) {
    if (need <= held) return held;
    if (held == 0) return need;
    const size_t g = held + held / 2;
    return need > g ? need : g;
}

struct DevBuf {
    void* ptr = nullptr;
    size_t bytes = 0;
    DevBuf() = default;
    DevBuf(const DevBuf&) = delete;
    DevBuf& operator=(const DevBuf&) = delete;
    ~DevBuf() { release(); }
    void release() {
        if (ptr) cudaFree(ptr);
        ptr = nullptr;
        bytes = 0;
    }
    cudaError_t ensure(size_t need) {
        if (need <= bytes && ptr) return cudaSuccess;
        if (need == 0) need = 16;
        const size_t cap = grow_capacity(need, ptr ? bytes : 0);
        release();
        cudaError_t e = cudaMalloc(&ptr, cap);
        if (e == cudaSuccess) bytes = cap;
        return e;
    }
    template <typename T>
    T* as() const {
        return reinterpret_cast<T*>(ptr);
    }
};

// Whether kernels read a caller's array of "device memory" themselves, with loads of `align` bytes.
// An array of another device is copied instead: a copy crosses devices, a kernel only with peer
// access; and so is one that is not device memory at all, which the copy turns into an error.
inline bool reads_directly(const cudaPointerAttributes& a, int device, const void* p, size_t align) {
    return p && (reinterpret_cast<uintptr_t>(p) & (align - 1)) == 0 && a.type == cudaMemoryTypeDevice && a.device == device;
}
// The same for an array that no copy brought in before: only what kernels cannot read is copied.
inline bool reads_mapped(const cudaPointerAttributes& a, int device, const void* p, size_t align) {
    return reads_directly(a, device, p, align) ||
           (p && (reinterpret_cast<uintptr_t>(p) & (align - 1)) == 0 &&
            (a.type == cudaMemoryTypeManaged || (a.type == cudaMemoryTypeHost && a.devicePointer == p)));
}
// One of the two for an array on the current device.
inline bool caller_array(bool (*rule)(const cudaPointerAttributes&, int, const void*, size_t), const void* p, size_t align) {
    cudaPointerAttributes a{};
    int device = -1;
    if (!p || cudaGetDevice(&device) != cudaSuccess || cudaPointerGetAttributes(&a, p) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    return rule(a, device, p, align);
}

// SMs of the current device (a cached attribute query), at least 1.
inline uint32_t device_sms() {
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    return sms > 0 ? (uint32_t)sms : 1u;
}

// Launches `kernel` with programmatic stream serialization: its CTAs are scheduled as those of the
// stream's previous kernel end, and wait in pdl_wait before their first global access, which
// hides a launch gap.
template <typename... P, typename... A>
inline cudaError_t launch_after(void (*kernel)(P...), uint32_t grid, uint32_t threads, size_t smem, cudaStream_t stream,
                                A&&... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, P(args)...);
}

inline uint32_t host_mip_levels(uint32_t w, uint32_t h) {
    uint32_t m = w > h ? w : h, bits = 0;
    while (m) {
        ++bits;
        m >>= 1;
    }
    return bits ? bits : 1u;
}

}  // namespace helio
