// acfdtd_adjoint.cuh -- the adjoint step by 16-byte chunks: parameters and host interface.

#ifndef ACFDTD_ADJOINT_CUH
#define ACFDTD_ADJOINT_CUH

#include "acfdtd_device.cuh"

namespace acf {

template <typename T>
struct AdjointParams {
    Room<T> room;                  // coefficients, geometry, profiles, walls, points
    T *lp, *lvx, *lvy, *lvz, *lpsi, *ld;  // adjoint fields (room geometry)
    const double *grad_rec;        // n_rec rows of grad_stride, column = step - grad_step0
    double *grad_src;              // n_src rows of grad_stride
    int64_t grad_stride, grad_step0;
    History<T> hist;
    double *grad_shell;            // FP64 dL/da per boundary cell (shell index)
    double *air_partials;          // per block: G_r (R), m_r (R), delta_r (R), S
    const int64_t *step_base;      // the forward step reversed is *step_base + local_step
    int32_t local_step;
    int32_t planes;
    int32_t air;                   // accumulate air gradients (needs hist.fields)
    // Fused adjoint step only: mu^{n+1} and lambda_D^n go to these (the other copies); lvx..lvz
    // hold mu^{n+2} and ld holds lambda_D^{n+1}.
    T *out_vx, *out_vy, *out_vz, *out_d;
};

// The sums over a block of NA values per thread, sum(t) with t < NA, added to its partials in FP64. Blocks
// of rooms that are narrow in y and z are smaller than a warp, and smaller than NA.
template <int NA, int MAX_THREADS, typename F>
__device__ __forceinline__ void add_block_sums(double *air_partials, F sum) {
    __shared__ double part[NA][MAX_THREADS / 32];
    const int threads = blockDim.x * blockDim.y, tid = threadIdx.y * blockDim.x + threadIdx.x;
    const int lane = tid & 31, warp = tid >> 5, warps = (threads + 31) >> 5, lanes = min(32, threads - 32 * warp);
    const unsigned mask = lanes == 32 ? 0xffffffffu : (1u << lanes) - 1u;
#pragma unroll
    for (int t = 0; t < NA; t++) {
        double v = sum(t);
        for (int o = 16; o > 0; o >>= 1) {
            const double other = __shfl_down_sync(mask, v, o);
            if (lane + o < lanes) v += other;
        }
        if (lane == 0) part[t][warp] = v;
    }
    __syncthreads();
    const int64_t block = ((int64_t)blockIdx.z * gridDim.y + blockIdx.y) * gridDim.x + blockIdx.x;
    for (int t = tid; t < NA; t += threads) {
        double v = 0.0;
        for (int w = 0; w < warps; w++) v += part[t][w];
        air_partials[block * NA + t] += v;
    }
}

template <typename T>
struct BatchAdjointParams {
    const AdjointParams<T> *rooms;
    const Tile *tiles;
    int32_t n_tiles;
    int32_t local_step;
    const int64_t *step_base;
};

// The face sweep of forward step n + 1 and the cell sweep of step n in one launch, for one room; with
// `air` (and relaxation states) also the air sums, one set of partials per block.
template <typename T>
void launch_pack_adjoint(const AdjointParams<T> &a, bool layer, bool walls, int n_relax, bool air, int block_threads,
                         cudaStream_t stream);
// Its blocks: the sets of partials it adds to.
template <typename T>
int64_t pack_adjoint_blocks(const Room<T> &room, int planes, int block_threads);

// The same step for every room of a batch over its pack tiles (no air sums).
template <typename T>
void launch_pack_adjoint_batch(const BatchAdjointParams<T> &p, bool layer, bool walls, int n_relax, int ctas,
                               cudaStream_t stream);

}  // namespace acf

#endif
