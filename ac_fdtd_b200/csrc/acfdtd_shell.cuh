// acfdtd_shell.cuh -- wall gradients from the boundary sums of the adjoint (host interface).

#ifndef ACFDTD_SHELL_CUH
#define ACFDTD_SHELL_CUH

#include <cuda_runtime.h>

#include <cstdint>

namespace acf {

// From `grad` (dL/da per boundary cell of an n[0] x n[1] x n[2] room, each on the first face it
// touches): `cells`, scale times it at every cell of each face in turn, and `sums`, their sums per
// face and patch (patches x patches per face, over the face's two other axes in increasing order).
int shell_gradients(const double *grad, const int32_t n[3], double scale, int32_t patches, double *cells,
                    double *sums, cudaStream_t stream);

}  // namespace acf

#endif
