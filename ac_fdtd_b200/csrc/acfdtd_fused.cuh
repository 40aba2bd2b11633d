// acfdtd_fused.cuh -- the fused step by 16-byte chunks (host interface).

#ifndef ACFDTD_FUSED_CUH
#define ACFDTD_FUSED_CUH

#include "acfdtd_device.cuh"

namespace acf {

// One fused step of one room (or slab) from f.room's copy to the next, `f.planes` x planes and up
// to `block_threads` threads per block. `early`: as launch_after does (not in a slab group, whose
// streams wait on one another's events between the launches).
void launch_pack_sweep(const FusedParams<double> &f, bool layer, bool walls, int n_relax, int block_threads,
                       bool early, cudaStream_t stream);

// The same step, also writing the forward history of the gradients.
template <typename T>
void launch_pack_rec(const FusedParams<T> &f, const History<T> &history, bool layer, bool walls, int n_relax,
                     int block_threads, cudaStream_t stream);

// One fused step of every room of a batch over tiles of at most kPackThreads packs (p.tiles' pairs are
// (row, 16-byte chunk) pairs), `ctas` CTAs; with p.history set, recorded.
constexpr int kPackThreads = 128;

// Its resident blocks per SM: see acfdtd_fused_batch.cu.
constexpr int pack_batch_blocks(int element_bytes, bool relaxation, bool recorded) {
    return !relaxation && !recorded ? 6 : element_bytes == 8 && relaxation ? 4 : 5;
}

template <typename T>
void launch_pack_batch(const FusedBatchParams<T> &p, bool layer, bool walls, int n_relax, int ctas,
                       cudaStream_t stream);

}  // namespace acf

#endif
