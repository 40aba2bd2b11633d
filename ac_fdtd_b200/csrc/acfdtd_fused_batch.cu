// acfdtd_fused_batch.cu -- the fused step of a batch of rooms, plain and recorded.
//
// Bound by HBM where the rooms together exceed L2, and by the tail and the ramp of a launch per step:
// 8 rooms of 60 to 200 cells a side (12.4M cells) move 692 MB in single precision with air in 155 us,
// 4.5 TB/s, with 20 of 64 warps resident. The step with four elements per thread in double precision
// and branches at the walls took (us per step, then now) 291 and 235 in double precision with walls,
// 409 and 380 with air; in single precision 157 and 136 with walls, 211 and 214 with air (other 8
// rooms of the same range); 64 rooms of 24 to 96 148 and 130, double precision 268 and 220;
// 4 rooms of 20 to 40 20 and 10, double precision 22 and 9. Resident
// blocks of 128: 6 without relaxation states, 5 with (4 in double precision); 6 spill the states
// (163 against 155 us, double precision 288 against 272), 4 in single precision cost with a layer.
//
// Recorded, it is the forward run of the wall gradients: three rooms of 96 to 160 with every term, two
// sweeps 126 us per step, this 105.

#include "acfdtd_fused.cuh"

#include "acfdtd_fused_kernel.cuh"
#include "acfdtd_host.cuh"

namespace acf {
namespace {

// A CTA copies the description of its tile's room into shared memory when the room changes (every
// thread takes part in the copy and both barriers, so they stay uniform); no CTA waits on another.
template <typename T, bool LAYER, bool WALLS, int NR, bool REC>
__global__ void __launch_bounds__(kPackThreads, pack_batch_blocks(sizeof(T), NR > 0, REC))
pack_batch(const FusedBatchParams<T> b) {
    step_next();
    constexpr int kWords = sizeof(FusedParams<T>) / sizeof(int), kHistoryWords = sizeof(History<T>) / sizeof(int);
    static_assert(sizeof(FusedParams<T>) % sizeof(int) == 0 && sizeof(History<T>) % sizeof(int) == 0, "whole words");
    __shared__ __align__(16) int raw[kWords + (REC ? kHistoryWords : 0)];
    const FusedParams<T> &f = *reinterpret_cast<const FusedParams<T> *>(raw);
    static_assert(kWords % 2 == 0, "the history is 8-byte aligned");
    const History<T> *history = REC ? reinterpret_cast<const History<T> *>(raw + kWords) : nullptr;
    int staged = -1;
    for (int t = blockIdx.x; t < b.n_tiles; t += gridDim.x) {
        const Tile tile = b.tiles[t];
        if (tile.room != staged) {
            __syncthreads();
            const int *from = reinterpret_cast<const int *>(b.rooms + tile.room);
            for (int w = threadIdx.x; w < kWords; w += blockDim.x) raw[w] = __ldg(from + w);
            if (REC) {
                const int *h = reinterpret_cast<const int *>(b.history + tile.room);
                for (int w = threadIdx.x; w < kHistoryWords; w += blockDim.x) raw[kWords + w] = __ldg(h + w);
            }
            __syncthreads();
            staged = tile.room;
        }
        step_wait();                             // tiles and descriptions are only written by the host
        const int64_t step = *b.step_base + b.local_step;
        if ((int)threadIdx.x < tile.count) {
            const int pack = tile.first + threadIdx.x, packs = (f.room.nz + Pack<T>::W - 1) / Pack<T>::W;
            pack_column<T, LAYER, WALLS, NR, REC>(f, tile.i_begin, tile.i_end, pack / packs, pack % packs, step,
                                                  history);
        }
    }
}

template <typename T, bool L, bool W, bool R>
void launch_relax(const FusedBatchParams<T> &p, int n_relax, dim3 grid, dim3 block, cudaStream_t st) {
    switch (n_relax) {
        case 0: launch_after(pack_batch<T, L, W, 0, R>, grid, block, st, p); break;
        case 1: launch_after(pack_batch<T, L, W, 1, R>, grid, block, st, p); break;
        case 2: launch_after(pack_batch<T, L, W, 2, R>, grid, block, st, p); break;
        case 3: launch_after(pack_batch<T, L, W, 3, R>, grid, block, st, p); break;
        default: launch_after(pack_batch<T, L, W, 4, R>, grid, block, st, p); break;
    }
}

template <typename T, bool R>
void launch_terms(const FusedBatchParams<T> &p, bool layer, bool walls, int n_relax, dim3 grid, dim3 block,
                  cudaStream_t st) {
    if (layer) {
        if (walls) launch_relax<T, true, true, R>(p, n_relax, grid, block, st);
        else launch_relax<T, true, false, R>(p, n_relax, grid, block, st);
    } else {
        if (walls) launch_relax<T, false, true, R>(p, n_relax, grid, block, st);
        else launch_relax<T, false, false, R>(p, n_relax, grid, block, st);
    }
}

}  // namespace

template <typename T>
void launch_pack_batch(const FusedBatchParams<T> &p, bool layer, bool walls, int n_relax, int ctas,
                       cudaStream_t st) {
    const dim3 grid(ctas), block(kPackThreads);
    if (p.history) launch_terms<T, true>(p, layer, walls, n_relax, grid, block, st);
    else launch_terms<T, false>(p, layer, walls, n_relax, grid, block, st);
}

template void launch_pack_batch<float>(const FusedBatchParams<float> &, bool, bool, int, int, cudaStream_t);
template void launch_pack_batch<double>(const FusedBatchParams<double> &, bool, bool, int, int, cudaStream_t);

}  // namespace acf
