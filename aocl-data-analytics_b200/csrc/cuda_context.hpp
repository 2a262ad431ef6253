// The calling thread's CUDA context: what a thing that outlives one call compares
// before it uses addresses and events of an earlier one.
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>

namespace b200 {

template <typename F> F driver_entry(const char *name) {
    void *p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint(name, &p, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess)
        return nullptr;
    return reinterpret_cast<F>(p);
}

// Unique id of the calling thread's current context (0 when there is none); the
// context itself.
inline unsigned long long current_context_id(CUcontext *ctx = nullptr) {
    static const auto get_cur = driver_entry<CUresult (*)(CUcontext *)>("cuCtxGetCurrent");
    static const auto get_id =
        driver_entry<CUresult (*)(CUcontext, unsigned long long *)>("cuCtxGetId");
    CUcontext c = nullptr;
    unsigned long long id = 0;
    if (!get_cur || !get_id || get_cur(&c) != CUDA_SUCCESS || !c || get_id(c, &id) != CUDA_SUCCESS)
        return 0;
    if (ctx) *ctx = c;
    return id;
}

// The device's primary context (the runtime's) exists; nothing is created.
inline bool primary_context_active(int dev) {
    static const auto state =
        driver_entry<CUresult (*)(CUdevice, unsigned *, int *)>("cuDevicePrimaryCtxGetState");
    unsigned flags = 0;
    int active = 0;
    return state && state(dev, &flags, &active) == CUDA_SUCCESS && active;
}

// The calling thread's current context is the device's primary one.
inline bool in_primary_context(int dev) {
    static const auto retain =
        driver_entry<CUresult (*)(CUcontext *, CUdevice)>("cuDevicePrimaryCtxRetain");
    static const auto release =
        driver_entry<CUresult (*)(CUdevice)>("cuDevicePrimaryCtxRelease");
    CUcontext cur = nullptr, prim = nullptr;
    if (!retain || !release || !primary_context_active(dev) || current_context_id(&cur) == 0 ||
        retain(&prim, dev) != CUDA_SUCCESS)
        return false;
    release(dev);
    return cur == prim;
}

} // namespace b200
