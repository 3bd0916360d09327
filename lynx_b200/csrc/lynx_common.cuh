// Shared definitions for the lynx_b200 CUDA library (sm_100a).
#pragma once
#include <cuda_runtime.h>
#include <cstdint>
#include <cstdio>
#include <string>

#include "../../include/lynx_b200.h"

namespace lynxb {

// Largest finite-difference half-width (FD order / 2) the kernels are built for.
constexpr int kMaxRadius = 8;

// Per-thread error string, returned by lynx_last_error().
void set_error(const char* fmt, ...);

// Raises a kernel's dynamic shared-memory cap (cudaFuncAttributeMaxDynamicSharedMemorySize) to at
// least `bytes`.  The cap is one value per function and device for the whole process, and host
// threads solving different grids launch the same kernel with different sizes at once: a thread
// that lowered it would make another thread's larger launch fail.  So the cap only grows, under
// a lock.
cudaError_t raise_smem_cap(const void* func, size_t bytes);
template <typename K>
cudaError_t smem_cap(K* kern, size_t bytes) {
    return raise_smem_cap(reinterpret_cast<const void*>(kern), bytes);
}

// Programmatic dependent launch for the chains of short kernels of the filter: the next kernel's blocks
// may be set up while this one still runs, and wait in pdl_wait() for all of its results.  Every kernel
// launched this way calls pdl_wait() before it touches memory that an earlier kernel may read or write.
// A wait covers the grid before it only, so every grid must hold a block that waits: one whose blocks all
// leave early would let the next kernel start on results that are still being written.  Pointers to
// earlier results are not `const __restrict__`: that reads through the path for data that is constant while
// the kernel lives, and this kernel lives before its predecessor has written.
#ifdef __CUDACC__
__device__ __forceinline__ void pdl_wait() {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
}
template <typename... P, typename... A>
cudaError_t launch_pdl(void (*kern)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, A&&... args) {
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kern, static_cast<P>(args)...);
}
#endif

}  // namespace lynxb

#define LYNX_CUDA_TRY(...)                                                                      \
    do {                                                                                        \
        cudaError_t _e = (__VA_ARGS__);                                                         \
        if (_e != cudaSuccess) {                                                                \
            ::lynxb::set_error("%s failed: %s (%s:%d)", #__VA_ARGS__, cudaGetErrorString(_e), __FILE__, \
                               __LINE__);                                                       \
            return _e == cudaErrorMemoryAllocation ? LYNX_ERR_OOM : LYNX_ERR_CUDA;              \
        }                                                                                       \
    } while (0)

#define LYNX_TRY(...)                  \
    do {                               \
        int _s = (__VA_ARGS__);        \
        if (_s != LYNX_OK) return _s;  \
    } while (0)

#define LYNX_CHECK_ARG(cond, msg)                                   \
    do {                                                            \
        if (!(cond)) {                                              \
            ::lynxb::set_error("bad argument: %s", msg);            \
            return LYNX_ERR_BAD_ARG;                                \
        }                                                           \
    } while (0)
