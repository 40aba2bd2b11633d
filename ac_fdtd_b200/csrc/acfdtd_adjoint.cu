// acfdtd_adjoint.cu -- the adjoint step by 16-byte chunks, for one room and for a batch.
//
// Bound by memory: (10 + 2R) elements per cell and step, and D and psi of every cell with the air sums;
// at sizes that stay in L2 by the latency of a plane's loads. The step it replaces took four elements
// per thread in double precision and, at every face, a branch for the room's edge. Backward runs of 120
// steps, before and after (ms): 128^3 in double precision 8.5 and 6.5; 101 x 86 x 92 with air in double
// precision 5.6 and 4.2; 101 x 86 x 93 in single precision 6.0 and 4.1; three rooms of 96 to 160 with every
// term 133 and 106 us per step. Single rooms of single precision with whole chunks keep the lean step
// (22 us at 128^3), whose factors stay in registers. Resident blocks of 128 threads: 4 with the air sums
// (3 cost 18 %: 5.0 and 4.8 ms) and in double precision with relaxation states, 5 otherwise.

#include "acfdtd_adjoint.cuh"

#include <algorithm>

#include "acfdtd_fused.cuh"
#include "acfdtd_host.cuh"
#include "acfdtd_pack.cuh"

namespace acf {
namespace {

// Sums over the cells of a thread: two lanes in single precision, one in double.
__device__ __forceinline__ float2 plus(float2 sum, const Pack<float> &x) { return add2(add2(sum, x.a), x.b); }
__device__ __forceinline__ double plus(double sum, const Pack<double> &x) { return (sum + x.a.x) + x.a.y; }
__device__ __forceinline__ double total(float2 sum) { return (double)sum.x + (double)sum.y; }
__device__ __forceinline__ double total(double sum) { return sum; }
template <typename T>
using Sum = decltype(finite_start(T(0)));

__device__ __forceinline__ Pack<float> pload_streaming(const float *x) {
    const float4 v = __ldcs(reinterpret_cast<const float4 *>(x));
    return {lo2(v), hi2(v)};
}
__device__ __forceinline__ Pack<double> pload_streaming(const double *x) {
    return {__ldcs(reinterpret_cast<const double2 *>(x))};
}

// One column of chunks over planes [i_begin, i_end): mu^{n+1} on the cell's six faces from mu^{n+2}
// (lvx..lvz) and lambda_D^{n+1} (ld) -- its three lower faces (stored, with the far boundary faces) and
// its three upper ones, as their owners compute them -- then lambda of the cells at step n. Elements
// past nz are zero in every adjoint field and stay so. AIR adds the air sums to `acc`.
template <typename T, bool LAYER, bool WALLS, int NR, bool AIR>
__device__ __forceinline__ void pack_adjoint_column(const AdjointParams<T> &a, int i_begin, int i_end, int j, int c,
                                                    int64_t step, Sum<T> *acc) {
    using P = Pack<T>;
    constexpr int W = P::W;
    const Room<T> &s = a.room;
    const int k0 = c * W, real = min(W, s.nz - k0);
    const bool tail = real < W;
    const int64_t column = (int64_t)j * s.pz + k0;
    const bool y_lo = j > 0, y_hi = j + 1 < s.ny, z_lo = k0 > 0, z_hi = k0 + W < s.nz;
    const bool top = k0 + W == s.nz;             // the far z face, not in any chunk of cells
    bool all_points = false;
    const uint32_t points = (s.n_src | s.n_rec) != 0 ? column_points(s, j, k0, all_points, W) : 0u;
    const bool any_mine = points != 0 || all_points;
    const bool wall_column = WALLS && (!y_lo || !y_hi || !z_lo || !z_hi);
    const P zero = pzero<T>();
    T fy_c = T(1), fy_l = T(1), fy_h = T(1);
    bool damp_y = false, damp_z = false;
    if (LAYER) {
        fy_c = __ldg(s.cell[1] + j);
        fy_l = __ldg(s.face[1] + j);
        fy_h = __ldg(s.face[1] + j + 1);
        damp_y = fy_c != T(1) || fy_l != T(1) || fy_h != T(1);
#pragma unroll
        for (int e = 0; e <= W; e++) {
            damp_z = damp_z || __ldg(s.face[2] + min(k0 + e, s.nz)) != T(1);
            if (e < W) damp_z = damp_z || __ldg(s.cell[2] + min(k0 + e, s.nz - 1)) != T(1);
        }
    }
    auto z_times = [&](const P &v, const T *profile, int last) {
        T x[W];
        unpack(v, x);
#pragma unroll
        for (int e = 0; e < W; e++) x[e] = x[e] * __ldg(profile + min(k0 + e, last));
        return repack(x);
    };
    auto z_cells = [&](const P &v) { return z_times(v, s.cell[2], s.nz - 1); };
    auto z_faces = [&](const P &v) { return z_times(v, s.face[2], s.nz); };

    P dc, xl;    // carried along x: lambda_D^{n+1} of this plane, mu^{n+1} on its lower x face
    {
        const int64_t base = (int64_t)i_begin * s.plane + column;
        dc = pload(a.ld + base);
        const P dm = i_begin > 0 ? pload(a.ld + base - s.plane) : zero;
        xl = padd(pload(a.lvx + base), psub(dm, dc));
        if (LAYER) {
            const T fx = __ldg(s.face[0] + i_begin);
            if (fx != T(1)) xl = pmul(xl, fx);
            if (damp_y) xl = pmul(xl, fy_c);
            if (damp_z) xl = z_cells(xl);
        }
    }
    const T *history = nullptr;
    if (AIR) history = a.hist.fields + (step - a.hist.fields_step0) % a.hist.fields_slots * (1 + NR) * s.field;

    for (int i = i_begin; i < i_end; i++) {
        const int64_t base = (int64_t)i * s.plane + column;
        const bool x_lo = i > 0, x_hi = i + 1 < s.nx;
        if (s.prefetch && i + 1 < i_end) {       // the next plane's own-row inputs into L2
            const int64_t next = base + s.plane;
            if (i + 2 < s.nx) prefetch_l2(a.ld + next + s.plane);
            prefetch_l2(a.lvx + next + s.plane);
            prefetch_l2(a.lvy + next);
            prefetch_l2(a.lvz + next);
            prefetch_l2(a.lp + next);
#pragma unroll
            for (int r = 0; r < NR; r++) prefetch_l2(a.lpsi + r * s.field + next);
            if (AIR) {
#pragma unroll
                for (int r = 0; r <= NR; r++) prefetch_l2(history + r * s.field + next);
            }
        }
        // ---- loads
        P hd = zero, hs[NR > 0 ? NR : 1];
        if (AIR) {                               // D^n and psi^n of the reversed step, read once
            hd = pload_streaming(history + base);
#pragma unroll
            for (int r = 0; r < NR; r++) hs[r] = pload_streaming(history + (1 + r) * s.field + base);
        }
        const P dx = x_hi ? pload(a.ld + base + s.plane) : zero;
        const P dy = y_lo ? pload(a.ld + base - s.pz) : zero, dyp = y_hi ? pload(a.ld + base + s.pz) : zero;
        const T d_below = z_lo ? a.ld[base - 1] : T(0), d_above = z_hi ? a.ld[base + W] : T(0);
        P xh = pload(a.lvx + base + s.plane), yl = pload(a.lvy + base), yh = pload(a.lvy + base + s.pz);
        P z = pload(a.lvz + base);
        T above = k0 + W <= s.nz ? a.lvz[base + W] : T(0);
        const P l = pload(a.lp + base);
        P ls[NR > 0 ? NR : 1];
#pragma unroll
        for (int r = 0; r < NR; r++) ls[r] = pload(a.lpsi + r * s.field + base);

        // ---- mu^{n+1} on the six faces: LV + (lambda_D[lower] - lambda_D[upper]), damped
        xh = padd(xh, psub(dc, dx));
        yl = padd(yl, psub(dy, dc));
        yh = padd(yh, psub(dc, dyp));
        z = padd(z, psub(below_of(dc, d_below), dc));
        above = above + (last_of(dc) - d_above);
        T fx = T(1);
        if (LAYER) {
            fx = __ldg(s.cell[0] + i);
            const T fx_h = __ldg(s.face[0] + i + 1);
            if (fx != T(1) || fx_h != T(1)) {
                xh = pmul(xh, fx_h);
                yl = pmul(yl, fx);
                yh = pmul(yh, fx);
                z = pmul(z, fx);
                above = above * fx;
            }
            if (damp_y) {
                xh = pmul(xh, fy_c);
                yl = pmul(yl, fy_l);
                yh = pmul(yh, fy_h);
                z = pmul(z, fy_c);
                above = above * fy_c;
            }
            if (damp_z) {
                xh = z_cells(xh);
                yl = z_cells(yl);
                yh = z_cells(yh);
                z = z_faces(z);
                above = above * __ldg(s.face[2] + min(k0 + W, s.nz));
            }
        }
        // ---- lambda(p^{n+1}) = L + c_v div(mu^{n+1}) over the interior faces
        P zi = tail ? keep_from(z, zero, real) : z;               // faces nz and on: boundary, padding
        const P zu = above_of(zi, z_hi ? above : T(0));
        if (!z_lo) zi = zero_first(zi);
        P d = psub(x_hi ? xh : zero, x_lo ? xl : zero);
        d = padd(d, psub(y_hi ? yh : zero, y_lo ? yl : zero));
        d = padd(d, psub(zu, zi));
        P h = psub(l, pmul(d, -s.cv));
        if (any_mine) {
            T lp[W];
            unpack(h, lp);
            uint32_t m = all_points ? 0u : receiver_bits(points, s.n_src);
            for (int r = all_points ? 0 : -1; all_points ? r < s.n_rec : m != 0; r++) {
                if (!all_points) {
                    r = __ffs(m) - 1;
                    m &= m - 1;
                }
                const int64_t at = s.rec_off[r] - base;
                if (at >= 0 && at < W && step >= s.rec_start[r]) {
                    const T g = (T)a.grad_rec[r * a.grad_stride + (step - a.grad_step0)];
#pragma unroll
                    for (int e = 0; e < W; e++)
                        if (e == at) lp[e] = lp[e] + g;
                }
            }
            m = all_points ? 0u : source_bits(points, s.n_src);
            for (int q = all_points ? 0 : -1; all_points ? q < s.n_src : m != 0; q++) {
                if (!all_points) {
                    q = __ffs(m) - 1;
                    m &= m - 1;
                }
                const int64_t at = s.src_off[q] - base;
                if (at >= 0 && at < W && step < s.src_len[q]) {
                    T v = lp[0];
#pragma unroll
                    for (int e = 1; e < W; e++)
                        if (e == at) v = lp[e];
                    a.grad_src[q * a.grad_stride + (step - a.grad_step0)] = (double)(s.cs * v);
                }
            }
            h = repack(lp);
        }
        // ---- the layer, wall and relaxation transposes
        if (LAYER) {
            if (fx != T(1)) h = pmul(h, fx);
            if (damp_y) h = pmul(h, fy_c);
            if (damp_z) h = z_cells(h);
        }
        P t = h, next = h;                       // lp_tilde; the new lambda(p)
        if (wall_column || (WALLS && (!x_lo || !x_hi))) {
            T lph[W], lpt[W], lpn[W];
            unpack(h, lph);
#pragma unroll
            for (int e = 0; e < W; e++) {
                lpt[e] = lpn[e] = lph[e];
                int64_t idx;
                const int f = e < real ? shell_face(s, i, j, k0 + e, idx) : -1;
                if (f < 0) continue;
                const T *entry = s.shell[f] + 2 * idx;
                const T u = __ldg(entry), q = __ldg(entry + 1);
                lpt[e] = u * lph[e];
                lpn[e] = lpt[e] - q * lph[e];
                if (a.grad_shell) {
                    const T *p = a.hist.shell + (step - a.hist.shell_step0) * 2 * a.hist.shell_total +
                                 a.hist.face_off[f] + idx;
                    const double uu = (double)u;
                    a.grad_shell[a.hist.face_off[f] + idx] +=
                        -(double)lph[e] * uu * uu * ((double)p[a.hist.shell_total] + (double)p[0]);
                }
            }
            t = repack(lpt);
            next = repack(lpn);
        }
        P ld = pmul(t, s.relax_scale - s.cp);
        if (AIR && tail) hd = keep_from(hd, zero, real);
#pragma unroll
        for (int r = 0; r < NR; r++) {
            const P in = psub(pmul(ls[r], T(1) - s.decay[r]), pmul(t, s.mean[r]));
            ld = psub(ld, pmul(in, -s.gain[r]));
            if (AIR) {
                P off = psub(hs[r], pmul(hd, s.gain[r]));
                if (tail) off = keep_from(off, zero, real);
                acc[r] = plus(acc[r], ptimes(hd, in));
                acc[NR + r] = plus(acc[NR + r], ptimes(t, off));
                acc[2 * NR + r] = plus(acc[2 * NR + r], ptimes(ls[r], off));
            }
            ls[r] = psub(pmul(ls[r], s.decay[r]), pmul(t, -s.mean[r]));
        }
        if (AIR) acc[3 * NR] = plus(acc[3 * NR], ptimes(hd, t));

        // ---- stores
        pstore(a.lp + base, next);
#pragma unroll
        for (int r = 0; r < NR; r++) pstore(a.lpsi + r * s.field + base, ls[r]);
        pstore(a.out_d + base, ld);
        pstore(a.out_vx + base, xl);
        pstore(a.out_vy + base, yl);
        pstore(a.out_vz + base, z);
        if (!x_hi) pstore(a.out_vx + base + s.plane, xh);
        if (!y_hi) pstore(a.out_vy + base + s.pz, yh);
        if (top) a.out_vz[base + W] = above;
        dc = dx;
        xl = xh;
    }
}

template <typename T, bool LAYER, bool WALLS, int NR, bool AIR>
__global__ void __launch_bounds__(kPackThreads, AIR || (sizeof(T) == 8 && NR > 0) ? 4 : 5)
pack_adjoint(const __grid_constant__ AdjointParams<T> a) {
    constexpr int W = Pack<T>::W, NA = 3 * NR + 1;
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = blockIdx.y * blockDim.y + threadIdx.y;
    step_begin();
    Sum<T> acc[AIR ? NA : 1];
    if (AIR) {
#pragma unroll
        for (int t = 0; t < NA; t++) acc[t] = finite_start(T(0));
    }
    if (c * W < a.room.nz && j < a.room.ny) {
        const int i_begin = blockIdx.z * a.planes;
        pack_adjoint_column<T, LAYER, WALLS, NR, AIR>(a, i_begin, min(a.room.nx, i_begin + a.planes), j, c,
                                                      *a.step_base + a.local_step, acc);
    }
    if (AIR)                                     // uniform per launch: every thread reaches the barrier
        add_block_sums<NA, kPackThreads>(a.air_partials, [&](int t) { return total(acc[t]); });
}

template <typename T, bool LAYER, bool WALLS, int NR>
__global__ void __launch_bounds__(kPackThreads, sizeof(T) == 8 && NR > 0 ? 4 : 5)
pack_adjoint_batch(const BatchAdjointParams<T> b) {
    constexpr int kWords = sizeof(AdjointParams<T>) / sizeof(int);
    static_assert(sizeof(AdjointParams<T>) % sizeof(int) == 0, "whole words");
    __shared__ __align__(16) int raw[kWords];
    const AdjointParams<T> &a = *reinterpret_cast<const AdjointParams<T> *>(raw);
    step_next();
    int staged = -1;
    for (int n = blockIdx.x; n < b.n_tiles; n += gridDim.x) {
        const Tile tile = b.tiles[n];
        if (tile.room != staged) {
            __syncthreads();
            const int *from = reinterpret_cast<const int *>(b.rooms + tile.room);
            for (int w = threadIdx.x; w < kWords; w += blockDim.x) raw[w] = __ldg(from + w);
            __syncthreads();
            staged = tile.room;
        }
        step_wait();                             // tiles and descriptions are only written by the host
        const int64_t step = *b.step_base + b.local_step;
        if ((int)threadIdx.x < tile.count) {
            const int pack = tile.first + threadIdx.x, packs = (a.room.nz + Pack<T>::W - 1) / Pack<T>::W;
            pack_adjoint_column<T, LAYER, WALLS, NR, false>(a, tile.i_begin, tile.i_end, pack / packs, pack % packs,
                                                            step, nullptr);
        }
    }
}

template <typename T>
ChunkShape room_shape(const Room<T> &room, int planes, int block_threads) {
    return chunk_shape(room, planes, std::min(block_threads, kPackThreads));
}

// Planes per block: fewer than `planes` while the blocks would leave SMs idle, since a small room's step is
// the chain of its planes' loads and wall terms (20 x 21 x 23 with air in single precision, 10 blocks of four planes:
// 18.9 us per step of the gradient's backward run with all its host work, 16.8 with the step of two elements per thread
// before it, 10.8 so).
template <typename T>
int room_planes(const Room<T> &room, int planes, int block_threads) {
    constexpr int kSms = 148;
    for (; planes > 1; planes = (planes + 1) / 2) {
        const ChunkShape q = room_shape(room, planes, block_threads);
        if ((int64_t)q.grid.x * q.grid.y * q.grid.z >= kSms) break;
    }
    return planes;
}

template <typename T, bool L, bool W, int NR>
void launch_one(const AdjointParams<T> &a, bool air, const ChunkShape &q, cudaStream_t st) {
    if constexpr (NR > 0) {
        if (air) {
            launch_after(pack_adjoint<T, L, W, NR, true>, q.grid, q.block, st, a);
            return;
        }
    }
    launch_after(pack_adjoint<T, L, W, NR, false>, q.grid, q.block, st, a);
}
template <typename T, bool L, bool W, int NR>
void launch_one(const BatchAdjointParams<T> &b, bool, const ChunkShape &q, cudaStream_t st) {
    launch_after(pack_adjoint_batch<T, L, W, NR>, q.grid, q.block, st, b);
}

template <typename T, bool L, bool W, typename P>
void launch_relax(const P &p, int n_relax, bool air, const ChunkShape &q, cudaStream_t st) {
    switch (n_relax) {
        case 0: launch_one<T, L, W, 0>(p, air, q, st); break;
        case 1: launch_one<T, L, W, 1>(p, air, q, st); break;
        case 2: launch_one<T, L, W, 2>(p, air, q, st); break;
        case 3: launch_one<T, L, W, 3>(p, air, q, st); break;
        default: launch_one<T, L, W, 4>(p, air, q, st); break;
    }
}

template <typename T, typename P>
void launch_terms(const P &p, bool layer, bool walls, int n_relax, bool air, const ChunkShape &q, cudaStream_t st) {
    if (layer) {
        if (walls) launch_relax<T, true, true>(p, n_relax, air, q, st);
        else launch_relax<T, true, false>(p, n_relax, air, q, st);
    } else {
        if (walls) launch_relax<T, false, true>(p, n_relax, air, q, st);
        else launch_relax<T, false, false>(p, n_relax, air, q, st);
    }
}

}  // namespace

template <typename T>
void launch_pack_adjoint(const AdjointParams<T> &a, bool layer, bool walls, int n_relax, bool air, int block_threads,
                         cudaStream_t st) {
    AdjointParams<T> q = a;
    q.planes = room_planes(a.room, a.planes, block_threads);
    launch_terms<T>(q, layer, walls, n_relax, air, room_shape(a.room, q.planes, block_threads), st);
}

template <typename T>
int64_t pack_adjoint_blocks(const Room<T> &room, int planes, int block_threads) {
    const ChunkShape q = room_shape(room, room_planes(room, planes, block_threads), block_threads);
    return (int64_t)q.grid.x * q.grid.y * q.grid.z;
}

template <typename T>
void launch_pack_adjoint_batch(const BatchAdjointParams<T> &p, bool layer, bool walls, int n_relax, int ctas,
                               cudaStream_t st) {
    launch_terms<T>(p, layer, walls, n_relax, false, ChunkShape{dim3(ctas), dim3(kPackThreads)}, st);
}

template void launch_pack_adjoint<float>(const AdjointParams<float> &, bool, bool, int, bool, int, cudaStream_t);
template void launch_pack_adjoint<double>(const AdjointParams<double> &, bool, bool, int, bool, int, cudaStream_t);
template int64_t pack_adjoint_blocks<float>(const Room<float> &, int, int);
template int64_t pack_adjoint_blocks<double>(const Room<double> &, int, int);
template void launch_pack_adjoint_batch<float>(const BatchAdjointParams<float> &, bool, bool, int, int, cudaStream_t);
template void launch_pack_adjoint_batch<double>(const BatchAdjointParams<double> &, bool, bool, int, int, cudaStream_t);

}  // namespace acf
