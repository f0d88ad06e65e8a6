// Host-side helpers shared by the C-ABI translation units: error recording, CUDA checks.
#pragma once

#include <cuda_runtime.h>

#include <cstdio>
#include <string>

#include "../../include/ldg_b200.h"

namespace ldg {

void set_error(const std::string& msg);
void clear_error();

// Checks a CUDA call; on failure records the message and returns LDG_ERR_CUDA from the caller. The runtime's own record
// of the failure is taken back, or the check of the next launch would report it.
#define LDG_CUDA(call)                                                                          \
    do {                                                                                        \
        cudaError_t e__ = (call);                                                               \
        if (e__ != cudaSuccess) {                                                               \
            (void)cudaGetLastError();                                                           \
            ::ldg::set_error(std::string(#call) + ": " + cudaGetErrorString(e__));              \
            return LDG_ERR_CUDA;                                                                \
        }                                                                                       \
    } while (0)

// Checks the last launch.
#define LDG_LAUNCHED(name)                                                                      \
    do {                                                                                        \
        cudaError_t e__ = cudaGetLastError();                                                   \
        if (e__ != cudaSuccess) {                                                               \
            ::ldg::set_error(std::string("launch of ") + (name) + ": " + cudaGetErrorString(e__)); \
            return LDG_ERR_CUDA;                                                                \
        }                                                                                       \
    } while (0)

#define LDG_REQUIRE(cond, code, msg)                                                            \
    do {                                                                                        \
        if (!(cond)) {                                                                          \
            ::ldg::set_error(msg);                                                              \
            return (code);                                                                      \
        }                                                                                       \
    } while (0)

// Makes a handle's device current for the scope of an entry point and restores the caller's
// device afterwards, so handles created on different GPUs can be used from one thread.
struct DeviceGuard {
    int prev = -1;
    explicit DeviceGuard(int dev) {
        int cur = -1;
        if (dev < 0 || cudaGetDevice(&cur) != cudaSuccess || cur == dev) return;
        if (cudaSetDevice(dev) == cudaSuccess) prev = cur;
    }
    ~DeviceGuard() {
        if (prev >= 0) cudaSetDevice(prev);
    }
    DeviceGuard(const DeviceGuard&) = delete;
    DeviceGuard& operator=(const DeviceGuard&) = delete;
};

// Launches a kernel with programmatic stream serialization (pdl_wait / pdl_trigger in ldg_common.cuh).
// A back-to-back step saves about 2 us of launch gap (64^3 box: 8.2 -> 6.2 us a step).
template <class... P, class... A>
inline cudaError_t launch_pdl(void (*k)(P...), dim3 grid, int threads, size_t smem, cudaStream_t st, A... args) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = dim3((unsigned)threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, k, static_cast<P>(args)...);
}

}  // namespace ldg
