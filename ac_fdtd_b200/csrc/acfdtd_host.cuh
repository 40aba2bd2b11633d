// acfdtd_host.cuh -- error reporting shared by the host code of every translation unit.

#ifndef ACFDTD_HOST_CUH
#define ACFDTD_HOST_CUH

#include <cuda_runtime.h>

#include "acfdtd_b200.h"

namespace acf {

// Keeps the message for acf_last_error() on this thread and returns `code`.
int fail(int code, const char *fmt, ...);

// Launch a kernel that begins with step_begin(), so that its blocks may be resident, waiting there,
// when the kernel in front of it on the stream ends: the launch and the first instructions of a step
// overlap the tail of the one before, in a stream as in a captured graph. Measured: the chunk steps gain
// 2 % (203 x 187 x 211 in double precision 171 to 167 us per step, 8 uneven rooms 159 to 156); the lean
// single-precision step and its adjoint gain nothing or lose 3 %, and the two sweeps of small batches
// lose a third (28 to 41 us: a sweep's waiting blocks keep the other's from starting), so they are
// launched in turn.
template <typename... P, typename... A>
void launch_after(void (*kernel)(P...), dim3 grid, dim3 block, cudaStream_t st, const A &...args) {
    cudaLaunchConfig_t config = {};
    config.gridDim = grid;
    config.blockDim = block;
    config.stream = st;
    cudaLaunchAttribute early = {};
    early.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    early.val.programmaticStreamSerializationAllowed = 1;
    config.attrs = &early;
    config.numAttrs = 1;
    cudaLaunchKernelEx(&config, kernel, args...);   // an error is the caller's cudaGetLastError
}

}  // namespace acf

#define ACF_CUDA(call)                                                                     \
    do {                                                                                   \
        cudaError_t err__ = (call);                                                        \
        if (err__ != cudaSuccess)                                                          \
            return acf::fail(ACF_ERR_CUDA, "%s failed: %s (%s:%d)", #call,                      \
                        cudaGetErrorString(err__), __FILE__, __LINE__);                    \
    } while (0)

#endif
