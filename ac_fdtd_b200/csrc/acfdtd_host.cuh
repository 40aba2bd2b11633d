// acfdtd_host.cuh -- error reporting shared by the host code of every translation unit.

#ifndef ACFDTD_HOST_CUH
#define ACFDTD_HOST_CUH

#include <cuda_runtime.h>

#include "acfdtd_b200.h"

namespace acf {

// Keeps the message for acf_last_error() on this thread and returns `code`.
int fail(int code, const char *fmt, ...);

}  // namespace acf

#define ACF_CUDA(call)                                                                     \
    do {                                                                                   \
        cudaError_t err__ = (call);                                                        \
        if (err__ != cudaSuccess)                                                          \
            return acf::fail(ACF_ERR_CUDA, "%s failed: %s (%s:%d)", #call,                      \
                        cudaGetErrorString(err__), __FILE__, __LINE__);                    \
    } while (0)

#endif
