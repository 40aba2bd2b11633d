// acfdtd_fused.cu -- the fused step in double precision, and the recorded fused step in either.
//
// Bound by HBM: (8 + 2R) elements per cell and step, 112 bytes with three relaxation states. The step
// with four z elements per thread held its loads in 128 registers, so an SM had 16 warps and the
// rest of the loads of a plane waited for them: 0.69 of the measured copy rate on 251 x 240 x 263
// with every term, no better than the two sweeps (397 against 404 us, which move 144 bytes). Here a
// thread takes two elements, one 16-byte access per field, so that twice the warps are resident with
// the same bytes in flight each; faces on walls are not asked for (the pressure outside is the
// cell's own, a difference of zero), and layer factors that are exactly 1 are skipped.
// Measured (us per step; TB/s of the 112 or 64 bytes per cell): 251 x 240 x 263 with every term 397 to
// 294 (6.04), walls only 214 to 161 (6.31); 320^3 with every term 589 (6.23, 0.96 of the copy);
// 160 x 161 x 163 128 to 87. Four planes per block: 8 cost 2 to 8 % more, 16 up to 30 %.

#include "acfdtd_fused.cuh"

#include <algorithm>

#include "acfdtd_fused_kernel.cuh"
#include "acfdtd_host.cuh"

namespace acf {
namespace {

template <bool LAYER, bool WALLS, int NR>
__global__ void __launch_bounds__(128, NR > 0 ? 6 : 8) pack_sweep(const __grid_constant__ FusedParams<double> f) {
    step_begin();
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = blockIdx.y * blockDim.y + threadIdx.y;
    if (c * Pack<double>::W >= f.room.nz || j >= f.room.ny) return;
    const bool any_point = (f.room.n_src | f.room.n_rec) != 0;
    const int64_t step = any_point ? (*f.step_base + f.local_step) : 0;
    const int i_begin = blockIdx.z * f.planes;
    pack_column<double, LAYER, WALLS, NR>(f, i_begin, min(f.room.nx, i_begin + f.planes), j, c, step);
}

template <typename T>
struct RecordParams {
    FusedParams<T> f;
    History<T> history;
};

template <typename T, bool LAYER, bool WALLS, int NR>
__global__ void __launch_bounds__(128, NR > 0 ? 5 : 7) pack_sweep_rec(const __grid_constant__ RecordParams<T> q) {
    step_begin();
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = blockIdx.y * blockDim.y + threadIdx.y;
    if (c * Pack<T>::W >= q.f.room.nz || j >= q.f.room.ny) return;
    const int64_t step = *q.f.step_base + q.f.local_step;
    const int i_begin = blockIdx.z * q.f.planes;
    pack_column<T, LAYER, WALLS, NR, true>(q.f, i_begin, min(q.f.room.nx, i_begin + q.f.planes), j, c, step,
                                           &q.history);
}

template <bool L, bool W, int NR>
void launch_one(const FusedParams<double> &f, dim3 grid, dim3 block, bool early, cudaStream_t st) {
    if (early) launch_after(pack_sweep<L, W, NR>, grid, block, st, f);
    else pack_sweep<L, W, NR><<<grid, block, 0, st>>>(f);
}
template <bool L, bool W, int NR, typename T>
void launch_one(const RecordParams<T> &q, dim3 grid, dim3 block, bool, cudaStream_t st) {
    launch_after(pack_sweep_rec<T, L, W, NR>, grid, block, st, q);
}

template <bool L, bool W, typename P>
void launch_relax(const P &p, int n_relax, dim3 grid, dim3 block, bool early, cudaStream_t st) {
    switch (n_relax) {
        case 0: launch_one<L, W, 0>(p, grid, block, early, st); break;
        case 1: launch_one<L, W, 1>(p, grid, block, early, st); break;
        case 2: launch_one<L, W, 2>(p, grid, block, early, st); break;
        case 3: launch_one<L, W, 3>(p, grid, block, early, st); break;
        default: launch_one<L, W, 4>(p, grid, block, early, st); break;
    }
}

template <typename T, typename P>
void launch_room(const Room<T> &room, int planes, const P &p, bool layer, bool walls, int n_relax,
                 int block_threads, bool early, cudaStream_t st) {
    const auto [grid, block] = chunk_shape(room, planes, std::min(block_threads, kPackThreads));
    if (layer) {
        if (walls) launch_relax<true, true>(p, n_relax, grid, block, early, st);
        else launch_relax<true, false>(p, n_relax, grid, block, early, st);
    } else {
        if (walls) launch_relax<false, true>(p, n_relax, grid, block, early, st);
        else launch_relax<false, false>(p, n_relax, grid, block, early, st);
    }
}

}  // namespace

void launch_pack_sweep(const FusedParams<double> &f, bool layer, bool walls, int n_relax, int block_threads,
                       bool early, cudaStream_t st) {
    launch_room(f.room, f.planes, f, layer, walls, n_relax, block_threads, early, st);
}

template <typename T>
void launch_pack_rec(const FusedParams<T> &f, const History<T> &history, bool layer, bool walls, int n_relax,
                     int block_threads, cudaStream_t st) {
    launch_room(f.room, f.planes, RecordParams<T>{f, history}, layer, walls, n_relax, block_threads, true, st);
}

template void launch_pack_rec<float>(const FusedParams<float> &, const History<float> &, bool, bool, int, int,
                                     cudaStream_t);
template void launch_pack_rec<double>(const FusedParams<double> &, const History<double> &, bool, bool, int, int,
                                      cudaStream_t);

}  // namespace acf
