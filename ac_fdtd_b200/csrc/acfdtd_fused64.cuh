// acfdtd_fused64.cuh -- the fused step in double precision (host interface).

#ifndef ACFDTD_FUSED64_CUH
#define ACFDTD_FUSED64_CUH

#include "acfdtd_device.cuh"

namespace acf {

// One fused step of one room (or slab) from f.room's copy to the next, `f.planes` x planes and up
// to `block_threads` threads per block.
void launch_pack_sweep(const FusedParams<double> &f, bool layer, bool walls, int n_relax, int block_threads,
                       cudaStream_t stream);

}  // namespace acf

#endif
