// acfdtd_shell.cu -- wall gradients from the boundary sums of the adjoint: the map of every face and
// its sums per wall or patch.
//
// The adjoint leaves dL/da once per boundary cell, on the first face the cell touches; a wall's
// admittance acts on every cell of its face. Finding each cell's entry, gathering, scaling and summing
// on the host took 2.1 ms for 128^3 and 9 ms for three rooms of 96 to 160 with 4 x 4 patches per wall,
// a quarter of a gradient. Now (ms per gradient, before and after): 128^3 9.2 and 7.3, 101 x 86 x 92 with
// air 5.5 and 4.7, the three rooms 34.2 and 25.5. The maps are 0.8 MB at 128^3; the launches take
// microseconds, and what is left is the copy to the caller.

#include "acfdtd_shell.cuh"

#include "acfdtd_host.cuh"

namespace acf {
namespace {

struct Faces {
    int32_t n[3];
    int64_t off[7];                // start of each face's map; the last is the number of cells
};

__device__ __forceinline__ int64_t shell_slot(const Faces &s, int i, int j, int k) {
    if (i == 0) return s.off[0] + (int64_t)j * s.n[2] + k;
    if (i == s.n[0] - 1) return s.off[1] + (int64_t)j * s.n[2] + k;
    if (j == 0) return s.off[2] + (int64_t)i * s.n[2] + k;
    if (j == s.n[1] - 1) return s.off[3] + (int64_t)i * s.n[2] + k;
    if (k == 0) return s.off[4] + (int64_t)i * s.n[1] + j;
    return s.off[5] + (int64_t)i * s.n[1] + j;
}

__global__ void __launch_bounds__(256) shell_cells(const double *grad, const Faces s, double scale, double *cells) {
    const int64_t at = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (at >= s.off[6]) return;
    int f = 0;
    while (at >= s.off[f + 1]) f++;
    const int axis = f / 2, nc = axis == 2 ? s.n[1] : s.n[2];
    const int64_t local = at - s.off[f];
    const int b = (int)(local / nc), c = (int)(local % nc), side = f % 2 ? s.n[axis] - 1 : 0;
    const int i = axis == 0 ? side : b, j = axis == 1 ? side : axis == 0 ? b : c, k = axis == 2 ? side : c;
    cells[at] = scale * grad[shell_slot(s, i, j, k)];
}

// One block per face and patch. Patch q of P along n cells holds those with floor(cell P / n) = q.
constexpr int kSumThreads = 512;

__global__ void __launch_bounds__(kSumThreads) shell_sums(const double *cells, const Faces s, int patches, double *sums) {
    __shared__ double part[kSumThreads / 32];
    const int per_face = patches * patches, f = blockIdx.x / per_face, patch = blockIdx.x % per_face;
    const int axis = f / 2, nb = axis == 0 ? s.n[1] : s.n[0], nc = axis == 2 ? s.n[1] : s.n[2];
    const int64_t pb = patch / patches, pc = patch % patches, P = patches;
    const int64_t b0 = (pb * nb + P - 1) / P, b1 = ((pb + 1) * nb + P - 1) / P;
    const int64_t c0 = (pc * nc + P - 1) / P, c1 = ((pc + 1) * nc + P - 1) / P;
    const int64_t wide = c1 - c0, count = (b1 - b0) * wide;
    double v = 0.0;
    for (int64_t q = threadIdx.x; q < count; q += kSumThreads)
        v += cells[s.off[f] + (b0 + q / wide) * nc + c0 + q % wide];
    for (int d = 16; d > 0; d >>= 1) v += __shfl_down_sync(0xffffffffu, v, d);
    if (threadIdx.x % 32 == 0) part[threadIdx.x / 32] = v;
    __syncthreads();
    if (threadIdx.x == 0) {
        double sum = 0.0;
        for (int w = 0; w < kSumThreads / 32; w++) sum += part[w];
        sums[blockIdx.x] = sum;
    }
}

}  // namespace

int shell_gradients(const double *grad, const int32_t n[3], double scale, int32_t patches, double *cells,
                    double *sums, cudaStream_t st) {
    Faces s;
    for (int a = 0; a < 3; a++) s.n[a] = n[a];
    s.off[0] = 0;
    for (int f = 0; f < 6; f++)
        s.off[f + 1] = s.off[f] + (int64_t)(f < 2 ? n[1] : n[0]) * (f < 4 ? n[2] : n[1]);
    shell_cells<<<(unsigned)((s.off[6] + 255) / 256), 256, 0, st>>>(grad, s, scale, cells);
    shell_sums<<<(unsigned)(6 * patches * patches), kSumThreads, 0, st>>>(cells, s, patches, sums);
    ACF_CUDA(cudaGetLastError());
    return ACF_OK;
}

}  // namespace acf
