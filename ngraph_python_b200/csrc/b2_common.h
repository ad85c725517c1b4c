// Shared host-side helpers of the b200ng library: error reporting and CUDA status checks.
#ifndef B2_COMMON_H
#define B2_COMMON_H

#include <cuda_runtime.h>

#include <cstdarg>
#include <cstdio>
#include <string>

#include "../../include/b200ng.h"

namespace b2 {

std::string& last_error_ref();

inline int fail(int code, const char* fmt, ...) {
    char buf[2048];
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(buf, sizeof(buf), fmt, ap);
    va_end(ap);
    last_error_ref() = buf;
    return code;
}

}  // namespace b2

#define B2_CUDA(call)                                                                     \
    do {                                                                                  \
        cudaError_t e__ = (call);                                                         \
        if (e__ != cudaSuccess)                                                           \
            return b2::fail(B2_ERR_CUDA, "%s failed: %s (%s:%d)", #call,                  \
                            cudaGetErrorString(e__), __FILE__, __LINE__);                 \
    } while (0)

#define B2_REQUIRE(cond, ...)                                   \
    do {                                                        \
        if (!(cond)) return b2::fail(B2_ERR_INVALID, __VA_ARGS__); \
    } while (0)

#ifdef __CUDACC__
// Programmatic dependent launch: a kernel launched with launch_after may be scheduled while the kernel
// before it in the stream drains (2 us less between two small kernels).  So every thread of it calls
// after_earlier_kernels() -- or issues the two instructions itself -- before it reads or writes
// global memory.
__device__ __forceinline__ void after_earlier_kernels() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
namespace b2 {
template <typename... P, typename... A>
cudaError_t launch_after(void (*kernel)(P...), dim3 grid, int block, size_t smem, cudaStream_t st, const A&... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid; cfg.blockDim = dim3(block); cfg.dynamicSmemBytes = smem; cfg.stream = st;
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &attr; cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, P(args)...);
}
}  // namespace b2
#endif
#endif  // B2_COMMON_H
