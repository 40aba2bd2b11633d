// acfdtd_resident_kernel.cuh -- many steps per launch with the room's state held on chip.
//
// A room whose state fits the SMs' registers and shared memory (70 MB on 148 SMs) need not be
// read and written every step, and below 10^6 cells a step costs its launches and their latency,
// not its bytes: in two launches per step 64^3 took 10.0 us (single precision) and 13.0 us (double),
// and 32^3 no less. Here one cooperative launch holds the room and takes every step; a step then
// costs one exchange between neighbour CTAs and its arithmetic. Measured per step, walls only, against the
// two sweeps: 32^3 1.3 us (from 10.1, single) and 1.3 us (from 12.6, double), 64^3 1.9 and 2.7 us, 80^3 2.8
// and 5.3 us (from 10.8 and 13.1), 96^3 5.2 us (from 11.6, single), 128^3 12.1 us (from 14.8, single);
// against the fused step 64^3 8.6 and 10.6, 80^3 8.2 and 10.8, 96^3 8.9 (single). Larger rooms are not always
// faster on chip: see resident_faster. What bounds it: up to 64^3 the exchange -- a store seen by another
// SM takes 500 cycles on the same die and 900 on the other, so about 1500 with the poll and the barrier of
// 2300 to 3300 a step; its warps wait at the barrier most -- and above it latency: 3 or 4 warps per scheduler, whose
// instructions wait for one another and for shared memory, issue in a third of the cycles.
//
// One CTA per SM owns a brick of the room, a thread K consecutive x planes of one (row, 16-byte
// chunk) column: velocities in the thread's registers, p in shared memory. Only p crosses bricks:
// the velocities of a brick's upper faces are carried along redundantly, updated by the same
// operations as by their owners, so nothing else is needed. Two forms share this: up to four
// planes per thread one barrier per step with p in two copies (resident_chunk_sweep), above that
// two barriers with one copy of p and with vy in shared memory (resident_sweep), which fits more.
// Every value is formed by the same operations in the same order as by the two sweeps.
//
// The exchange carries its own flag: each 32-bit word travels in a 64-bit word with the step's
// tag, stored and loaded whole, so the receiver polls the data itself and no fence, counter or
// second trip through L2 is needed. An inbox has two slots per word, used by even and odd steps:
// a brick sends step t + 2 only after it received step t + 1, which its neighbour sent after
// it had consumed step t. Tags never repeat between launches (they count on from `epoch`).
// The wait is bounded: a thread that waits longer than the limit raises kStatusWaitTimeout,
// stops waiting for the rest of the launch, and the kernel ends.

#ifndef ACFDTD_RESIDENT_KERNEL_CUH
#define ACFDTD_RESIDENT_KERNEL_CUH

#include <algorithm>

#include "acfdtd_pack.cuh"
#include "acfdtd_resident.cuh"

namespace acf {
namespace {

constexpr int kThreads = 512;      // most threads per CTA: 128 registers each
constexpr int kChunkPlanes = 4;    // up to so many planes per thread, the one-barrier form
constexpr int kRim = 4;            // most rim chunks one thread receives

// A chunk on its way to a neighbour: its 32-bit words, each with the tag in one 64-bit store or load.
constexpr int kWords = 4;

__device__ __forceinline__ uint64_t tagged(uint32_t word, uint32_t tag) {
    return (uint64_t)word | ((uint64_t)tag << 32);
}
__device__ __forceinline__ void send_two(uint64_t *to, uint32_t w0, uint32_t w1, uint32_t tag) {
    asm volatile("st.relaxed.gpu.global.v2.b64 [%0], {%1, %2};" ::"l"(to), "l"(tagged(w0, tag)), "l"(tagged(w1, tag))
                 : "memory");
}
__device__ __forceinline__ void send(uint64_t *to, const Pack<float> &v, uint32_t tag) {
    send_two(to, __float_as_uint(v.a.x), __float_as_uint(v.a.y), tag);
    send_two(to + 2, __float_as_uint(v.b.x), __float_as_uint(v.b.y), tag);
}
__device__ __forceinline__ void send(uint64_t *to, const Pack<double> &v, uint32_t tag) {
    const uint64_t x = (uint64_t)__double_as_longlong(v.a.x), y = (uint64_t)__double_as_longlong(v.a.y);
    send_two(to, (uint32_t)x, (uint32_t)(x >> 32), tag);
    send_two(to + 2, (uint32_t)y, (uint32_t)(y >> 32), tag);
}
template <int N>
__device__ __forceinline__ void load_tagged(const uint64_t *from, uint64_t (&w)[N]) {
#pragma unroll
    for (int n = 0; n < N; n += 2)
        asm volatile("ld.relaxed.gpu.global.v2.b64 {%0, %1}, [%2];"
                     : "=l"(w[n]), "=l"(w[n + 1])
                     : "l"(from + n)
                     : "memory");
}
// Whether every word carries the tag.
template <int N>
__device__ __forceinline__ bool all_tagged(const uint64_t (&w)[N], uint32_t tag) {
    uint32_t off = 0;
#pragma unroll
    for (int n = 0; n < N; n++) off |= (uint32_t)(w[n] >> 32) ^ tag;
    return off == 0;
}
// The words, their tags dropped, to shared memory.
template <int N>
__device__ __forceinline__ void put_words(void *to, const uint64_t (&w)[N]) {
#pragma unroll
    for (int n = 0; n < N; n += 4)
        reinterpret_cast<uint4 *>(to)[n / 4] =
            make_uint4((uint32_t)w[n], (uint32_t)w[n + 1], (uint32_t)w[n + 2], (uint32_t)w[n + 3]);
}

template <typename T>
struct ResidentParams {
    Room<T> room;
    int32_t tx, rows, chunks, bx, gx, gy;
    int32_t nr, psi_shared, walls, steps, stop_step;
    T neg_decay[ACF_MAX_RELAXATION], neg_mean[ACF_MAX_RELAXATION], neg_scale;
    uint64_t *mailbox;
    const int64_t *step_base;
    const uint32_t *epoch;
    uint64_t wait_limit_ns;
};

// The brick's part of p (with its rim), vy and the relaxation states in shared memory, in elements.
// A row is C chunks, so consecutive threads touch consecutive addresses.
template <int W>
struct BrickLayout {
    int row, p_plane, vy_plane, psi_plane, psi_field;
    int vy, psi, end;              // offsets; p is at 0

    __host__ __device__ BrickLayout(int bx, int rows, int C, int psi_shared) {
        row = C * W;
        p_plane = (rows + 2) * row;              // p: bx + 2 planes of rows + 2 rows
        vy_plane = (rows + 1) * row;             // vy: bx planes of rows + 1
        psi_plane = rows * row;
        psi_field = bx * psi_plane;
        vy = (bx + 2) * p_plane;
        psi = vy + bx * vy_plane;
        end = psi + psi_shared * psi_field;
    }
};

// A column's place and the layer's y and z factors.
template <typename T>
struct Column {
    static constexpr int W = Pack<T>::W;
    int j, k0, real;
    bool damp_y, damp_z, wall, tail;
    T y_cell, y_face, z_cell[W], z_face[W + 1];
};

template <typename T, int W>
__device__ __forceinline__ Pack<T> times(const Pack<T> &v, const T (&f)[W]) {
    T x[Pack<T>::W];
    unpack(v, x);
#pragma unroll
    for (int e = 0; e < Pack<T>::W; e++) x[e] = x[e] * f[e];
    return repack(x);
}

// Layer factors in x, y, z order; an axis whose factors here are all exactly 1 is skipped.
template <typename T>
__device__ __forceinline__ Pack<T> damped(const Column<T> &col, Pack<T> v, T fx, T fy) {
    if (fx != T(1)) v = pmul(v, fx);
    if (col.damp_y) v = pmul(v, fy);
    if (col.damp_z) v = times(v, col.z_cell);
    return v;
}

// The wall closed form of one chunk on plane i: `pe` before it, `pc` the pressure of step n.
template <typename T>
__device__ __forceinline__ Pack<T> walled(const Room<T> &s, const Column<T> &col, const Pack<T> &pe, const Pack<T> &pc,
                                          int i) {
    constexpr int W = Pack<T>::W;
    T pn[W], po[W];
    unpack(pe, pn);
    unpack(pc, po);
    const bool on_x = i == 0 || i + 1 == s.nx, on_y = col.j == 0 || col.j + 1 == s.ny;
    auto wall = [&](int e, const T *entry) {
        const T fu = __ldg(entry), fp = __ldg(entry + 1);
        if (fp != T(0) || fu != T(1)) pn[e] = pn[e] * fu - po[e] * fp;
    };
    // the first face in FACES order that the cell lies on
    if (on_x || on_y) {
        const T *entry = on_x ? s.shell[i == 0 ? 0 : 1] + 2 * ((int64_t)col.j * s.nz + col.k0)
                              : s.shell[col.j == 0 ? 2 : 3] + 2 * ((int64_t)i * s.nz + col.k0);
#pragma unroll
        for (int e = 0; e < W; e++)
            if (e < col.real) wall(e, entry + 2 * e);
    } else {
        const int64_t entry = 2 * ((int64_t)i * s.ny + col.j);
#pragma unroll
        for (int e = 0; e < W; e++) {
            if (col.k0 + e == 0) wall(e, s.shell[4] + entry);
            else if (col.k0 + e == s.nz - 1) wall(e, s.shell[5] + entry);
        }
    }
    return repack(pn);
}

// Two barriers per step, more than four planes per thread: vx and vz in registers, p with a one-cell
// rim, vy and what fits of the relaxation states in shared memory. Per step: barrier; the faces
// between cells of the brick, while the neighbours' p is on its way; the rim arrives; barrier;
// the faces on the rim, the cells, and the surface of the brick to the neighbours.
//
// LAYER: the room has an absorbing layer. NR: relaxation states, 4 standing for any number up to 4.
template <typename T, int K, int NR, bool LAYER>
__global__ void __launch_bounds__(kThreads, 1) resident_sweep(const __grid_constant__ ResidentParams<T> q) {
    using P = Pack<T>;
    constexpr int W = P::W;
    extern __shared__ __align__(16) unsigned char raw[];
    const Room<T> &s = q.room;
    const int C = q.chunks, rows = q.rows, bx = q.bx, gy = q.gy;
    const int cta = blockIdx.x, gxi = cta / gy, gyi = cta - gxi * gy;
    const int x0 = gxi * bx, y0 = gyi * rows;
    const int nbx = min(bx, s.nx - x0), nby = min(rows, s.ny - y0);   // planes and rows of this brick
    auto has_state = [&](int r) { return NR < 4 || r < q.nr; };
    const BrickLayout<W> lay(bx, rows, C, q.psi_shared);
    T *const sm = reinterpret_cast<T *>(raw);

    const int c = threadIdx.x % C, column = threadIdx.x / C;
    const int row = column % rows, tx = column / rows;
    const int first = tx * K, i0 = x0 + first;                                    // first plane of this thread
    const int kn = (tx < q.tx && row < nby) ? max(0, min(K, nbx - first)) : 0;    // and how many
    const bool last_row = row + 1 == nby;
    Column<T> col;
    col.j = y0 + row;
    col.k0 = c * W;
    col.real = min(W, s.nz - col.k0);
    col.tail = col.real < W;
    col.wall = q.walls && (col.j == 0 || col.j == s.ny - 1 || col.k0 == 0 || col.k0 + W >= s.nz);
    const int j = col.j, k0 = col.k0;
    const bool z_lo = k0 > 0, z_hi = k0 + W < s.nz;
    const int64_t in_plane = (int64_t)j * s.pz + k0;
    T *const my_p = sm + (first + 1) * lay.p_plane + (row + 1) * lay.row + k0;
    T *const my_vy = sm + lay.vy + first * lay.vy_plane + row * lay.row + k0;
    T *const my_psi = sm + lay.psi + first * lay.psi_plane + row * lay.row + k0;

    // ---- the state of the brick. A cell outside the room is held as a copy of the room's cell
    // next to it (the rim at a wall, the padding elements of a row), so that the face between
    // them sees no pressure difference and is left alone without being asked for.
    for (int n = threadIdx.x; n < (nbx + 2) * (nby + 2) * C; n += blockDim.x) {
        const int cc = n % C, rr = n / C % (nby + 2) - 1, ii = n / (C * (nby + 2)) - 1;
        const bool in_x = ii >= 0 && ii < nbx, in_y = rr >= 0 && rr < nby;
        if (!in_x && !in_y) continue;
        const int i = min(max(x0 + ii, 0), s.nx - 1), jj = min(max(y0 + rr, 0), s.ny - 1);
        P v = pload(s.p + (int64_t)i * s.plane + (int64_t)jj * s.pz + cc * W);
        if (cc * W + W > s.nz) v = mirrored(v, s.nz - cc * W);
        pstore(sm + (ii + 1) * lay.p_plane + (rr + 1) * lay.row + cc * W, v);
        if (in_x && rr >= 0)                     // vy: also the face above the last row
            pstore(sm + lay.vy + ii * lay.vy_plane + rr * lay.row + cc * W,
                   pload(s.vy + (int64_t)(x0 + ii) * s.plane + (int64_t)(y0 + rr) * s.pz + cc * W));
    }
    P vx[K + 1], vz[K];
    T vz_above[K];
#pragma unroll
    for (int e = 0; e < K; e++) {
        vx[e] = vx[e + 1] = vz[e] = pzero<T>();
        vz_above[e] = T(0);
    }
#pragma unroll
    for (int e = 0; e < K; e++) {
        if (e >= kn) continue;
        const int64_t at = (int64_t)(i0 + e) * s.plane + in_plane;
        vx[e] = pload(s.vx + at);
        if (e == kn - 1 || e == K - 1) vx[e + 1] = pload(s.vx + at + s.plane);
        vz[e] = pload(s.vz + at);
        vz_above[e] = k0 + W <= s.nz ? s.vz[at + W] : T(0);
        for (int r = 0; r < q.psi_shared; r++)
            pstore(my_psi + r * lay.psi_field + e * lay.psi_plane, pload(s.psi + r * s.field + at));
    }

    // ---- the rim: where each chunk of the inbox goes in shared memory (in chunks), -1 for none.
    // An inbox holds x-, x+ (rows * C chunks each), y-, y+ (bx * C each).
    const int nxh = rows * C, nyh = bx * C, total = 2 * (nxh + nyh);
    int *const place = reinterpret_cast<int *>(sm + lay.end);
    for (int n = threadIdx.x; n < total; n += blockDim.x) {
        int h = n, to = -1;
        if (h < nxh) {
            if (gxi > 0 && h / C < nby) to = C + h;
        } else if (h < 2 * nxh) {
            h -= nxh;
            if (gxi + 1 < q.gx && h / C < nby) to = (bx + 1) * (rows + 2) * C + C + h;
        } else if (h < 2 * nxh + nyh) {
            h -= 2 * nxh;
            if (gyi > 0 && h / C < nbx) to = (h / C + 1) * (rows + 2) * C + h % C;
        } else {
            h -= 2 * nxh + nyh;
            if (gyi + 1 < gy && h / C < nbx) to = ((h / C + 1) * (rows + 2) + rows + 1) * C + h % C;
        }
        place[n] = to;
    }
    // What this thread does for the brick's surface after each step: send a chunk to the neighbour's
    // inbox (entry of its first plane), or copy it to the rim where the room ends.
    const bool at_x0 = kn > 0 && first == 0, at_x1 = kn > 0 && first + kn == nbx;
    const bool at_y0 = kn > 0 && row == 0, at_y1 = kn > 0 && last_row;
    const bool from_x0 = at_x0 && gxi > 0, from_x1 = at_x1 && gxi + 1 < q.gx;     // faces on the rim
    const bool from_y0 = at_y0 && gyi > 0;
    const int rc = row * C + c;
    const int to_x0 = (cta - gy) * 2 * total + nxh + rc, to_x1 = (cta + gy) * 2 * total + rc;
    const int to_y0 = (cta - 1) * 2 * total + 2 * nxh + nyh + first * C + c;
    const int to_y1 = (cta + 1) * 2 * total + 2 * nxh + first * C + c;

    // ---- column constants
    const uint32_t epoch = *q.epoch;
    const T cv = s.cv;
    bool all_points = false;
    const uint32_t points = (kn > 0 && (s.n_src | s.n_rec) != 0) ? column_points(s, j, k0, all_points, W) : 0u;
    const bool any_mine = kn > 0 && (points != 0 || all_points);
    if (LAYER) {
        const int jj = min(j, s.ny - 1);
        col.y_cell = __ldg(s.cell[1] + jj);
        col.y_face = __ldg(s.face[1] + jj);
        col.damp_y = col.y_cell != T(1) || col.y_face != T(1) || __ldg(s.face[1] + jj + 1) != T(1);
        col.damp_z = false;
#pragma unroll
        for (int e = 0; e <= W; e++) {
            col.z_face[e] = __ldg(s.face[2] + min(k0 + e, s.nz));
            if (e < W) col.z_cell[e] = __ldg(s.cell[2] + min(k0 + e, s.nz - 1));
            col.damp_z = col.damp_z || col.z_face[e] != T(1) || (e < W && col.z_cell[e] != T(1));
        }
    }
    // A face's velocity moved by the pressures on its two sides.
    auto moved = [&](const P &v, const P &high, const P &low) { return psub(v, pmul(psub(high, low), cv)); };

    auto bad = finite_start(T(0));
    bool waiting = true;   // false once a wait of this thread ran out

    for (int t = 0; t < q.steps; t++) {
        __syncthreads();
        // ---- 1: the faces that need nothing from the neighbours, whose p is on its way. (A thread's
        // planes past the brick's last work on what lies there, unused.)
        if (kn > 0) {
            const T *p = my_p;
            T *vy = my_vy;
            P prev = pload(p - lay.p_plane);
#pragma unroll
            for (int e = 0; e < K; e++, p += lay.p_plane, vy += lay.vy_plane) {
                const P pc = pload(p);
                const T below = p[-1], above = p[W];
                const T fc = LAYER ? __ldg(s.cell[0] + min(i0 + e, s.nx - 1)) : T(1);
                if (e > 0 || !from_x0) {
                    vx[e] = moved(vx[e], pc, prev);
                    if (LAYER) vx[e] = damped(col, vx[e], __ldg(s.face[0] + min(i0 + e, s.nx)), col.y_cell);
                }
                prev = pc;
                if (!from_y0) {
                    P y = moved(pload(vy), pc, pload(p - lay.row));
                    if (LAYER) y = damped(col, y, fc, col.y_face);
                    pstore(vy, y);
                }
                vz[e] = moved(vz[e], pc, below_of(pc, z_lo ? below : first_of(pc)));
                vz_above[e] = vz_above[e] - cv * ((z_hi ? above : last_of(pc)) - last_of(pc));
                if (LAYER) {
                    if (fc != T(1)) {
                        vz[e] = pmul(vz[e], fc);
                        vz_above[e] = vz_above[e] * fc;
                    }
                    if (col.damp_y) {
                        vz[e] = pmul(vz[e], col.y_cell);
                        vz_above[e] = vz_above[e] * col.y_cell;
                    }
                    if (col.damp_z) {
                        vz[e] = times(vz[e], col.z_face);
                        vz_above[e] = vz_above[e] * col.z_face[W];
                    }
                }
            }
            if (!from_x1) {
                vx[K] = moved(vx[K], pload(p), prev);
                if (LAYER) vx[K] = damped(col, vx[K], __ldg(s.face[0] + min(i0 + K, s.nx)), col.y_cell);
            }
        }

        // ---- 2: the neighbours' p on the rim, every chunk of a thread in flight at once
        if (t > 0 && waiting) {
            const uint32_t tag = epoch + (uint32_t)t;
            const uint64_t *from = q.mailbox + ((int64_t)(cta * 2 + (t & 1)) * total + threadIdx.x) * kWords;
            int to[kRim];
            bool pending = false;
#pragma unroll
            for (int u = 0; u < kRim; u++) {
                to[u] = -1;
                if ((int)(threadIdx.x + u * blockDim.x) < total) to[u] = place[threadIdx.x + u * blockDim.x];
                pending = pending || to[u] >= 0;
            }
            uint64_t start = 0;
            for (int tries = 1; pending && waiting; tries++) {
                pending = false;
#pragma unroll
                for (int u0 = 0; u0 < kRim; u0 += 2) {
                    uint64_t w[2][kWords];
#pragma unroll
                    for (int u = u0; u < u0 + 2; u++)
                        if (to[u] >= 0) load_tagged(from + u * blockDim.x * kWords, w[u - u0]);
#pragma unroll
                    for (int u = u0; u < u0 + 2; u++) {
                        if (to[u] < 0) continue;
                        if (all_tagged(w[u - u0], tag)) {
                            put_words(sm + to[u] * W, w[u - u0]);
                            to[u] = -1;
                        } else {
                            pending = true;
                        }
                    }
                }
                if ((tries & 63) == 0) {
                    if (start == 0) start = global_ns();
                    else if (global_ns() - start > q.wait_limit_ns) waiting = false;
                }
            }
            if (!waiting && s.status != nullptr) atomicOr(s.status, kStatusWaitTimeout);
        }
        __syncthreads();

        // ---- 3: the faces on the rim
        if (from_x0) {
            vx[0] = moved(vx[0], pload(my_p), pload(my_p - lay.p_plane));
            if (LAYER) vx[0] = damped(col, vx[0], __ldg(s.face[0] + i0), col.y_cell);
        }
        if (from_x1) {
            vx[K] = moved(vx[K], pload(my_p + K * lay.p_plane), pload(my_p + (K - 1) * lay.p_plane));
            if (LAYER) vx[K] = damped(col, vx[K], __ldg(s.face[0] + i0 + K), col.y_cell);
        }
        if (from_y0 || at_y1) {
            const T *p = my_p;
            T *vy = my_vy;
#pragma unroll 1
            for (int e = 0; e < kn; e++, p += lay.p_plane, vy += lay.vy_plane) {
                const P pc = pload(p);
                const T fc = LAYER ? __ldg(s.cell[0] + i0 + e) : T(1);
                if (from_y0) {
                    P y = moved(pload(vy), pc, pload(p - lay.row));
                    if (LAYER) y = damped(col, y, fc, col.y_face);
                    pstore(vy, y);
                }
                if (at_y1) {                     // the face above the brick's last row
                    P y = moved(pload(vy + lay.row), pload(p + lay.row), pc);
                    if (LAYER) y = damped(col, y, fc, __ldg(s.face[1] + j + 1));
                    pstore(vy + lay.row, y);
                }
            }
        }

        // ---- 4: the cells
        {
            T *p = my_p, *psi = my_psi;
            const T *vy = my_vy;
#pragma unroll
            for (int e = 0; e < K; e++, p += lay.p_plane, vy += lay.vy_plane, psi += lay.psi_plane) {
                if (e >= kn) continue;
                const int i = i0 + e;
                const P pc = pload(p);
                const P yl = pload(vy), yh = pload(vy + lay.row);
                P S[NR > 0 ? NR : 1];
#pragma unroll
                for (int r = 0; r < NR; r++) {
                    if (!has_state(r)) continue;
                    if (r < q.psi_shared) S[r] = pload(psi + r * lay.psi_field);
                    else S[r] = pload(s.psi + r * s.field + (int64_t)i * s.plane + in_plane);
                }
                P d = psub(vx[e + 1], vx[e]);
                d = padd(d, psub(yh, yl));
                d = padd(d, psub(above_of(vz[e], vz_above[e]), vz[e]));

                P pe = pc;
#pragma unroll
                for (int r = 0; r < NR; r++) {
                    if (!has_state(r)) continue;
                    const P target = pmul(d, s.gain[r]);
                    const P offset = psub(S[r], target);
                    P next = psub(target, pmul(offset, q.neg_decay[r]));
                    pe = psub(pe, pmul(offset, q.neg_mean[r]));
                    if (r < q.psi_shared) {
                        pstore(psi + r * lay.psi_field, next);
                    } else {
                        if (col.tail) next = keep_from(next, S[r], col.real);
                        pstore(s.psi + r * s.field + (int64_t)i * s.plane + in_plane, next);
                    }
                }
                if (NR > 0) pe = psub(pe, pmul(d, q.neg_scale));
                pe = psub(pe, pmul(d, s.cp));
                if (col.wall || (q.walls && (i == 0 || i + 1 == s.nx))) pe = walled(s, col, pe, pc, i);
                if (LAYER) pe = damped(col, pe, __ldg(s.cell[0] + i), col.y_cell);
                if (col.tail) pe = mirrored(pe, col.real);
                bad = pfinite(bad, pe);
                pstore(p, pe);
            }
        }
        // ---- sources and receivers, in the few threads that have any
        if (any_mine) {
            T *p = my_p;
            const int64_t step = *q.step_base + t;
#pragma unroll 1
            for (int e = 0; e < kn; e++, p += lay.p_plane) {
                T pn[W];
                unpack(pload(p), pn);
                const int64_t base = (int64_t)(i0 + e) * s.plane + in_plane;
                add_sources<T, W>(s, points, all_points, base, k0, step, pn);
                record_receivers<T, W>(s, points, all_points, base, step, pn);
                P pe = repack(pn);
                if (col.tail) pe = mirrored(pe, col.real);
                bad = pfinite(bad, pe);
                pstore(p, pe);
            }
        }
        // ---- 5: the surface of the brick
        if (at_x0 || at_x1 || at_y0 || at_y1) {
            const bool open = t + 1 < q.steps && !(cta == 0 && q.stop_step >= 0 && t >= q.stop_step);
            const uint32_t tag = epoch + (uint32_t)t + 1u;
            uint64_t *const box = q.mailbox + ((t + 1) & 1) * total * kWords;
            if (at_x0) {
                const P v = pload(my_p);
                if (gxi == 0) pstore(my_p - lay.p_plane, v);
                else if (open) send(box + (int64_t)to_x0 * kWords, v, tag);
            }
            if (at_x1) {
                T *p = my_p + (kn - 1) * lay.p_plane;
                const P v = pload(p);
                if (gxi + 1 == q.gx) pstore(p + lay.p_plane, v);
                else if (open) send(box + (int64_t)to_x1 * kWords, v, tag);
            }
            if (at_y0 || at_y1) {
                T *p = my_p;
#pragma unroll 1
                for (int e = 0; e < kn; e++, p += lay.p_plane) {
                    const P v = pload(p);
                    if (at_y0) {
                        if (gyi == 0) pstore(p - lay.row, v);
                        else if (open) send(box + (int64_t)(to_y0 + e * C) * kWords, v, tag);
                    }
                    if (at_y1) {
                        if (gyi + 1 == gy) pstore(p + lay.row, v);
                        else if (open) send(box + (int64_t)(to_y1 + e * C) * kWords, v, tag);
                    }
                }
            }
        }
    }

    // ---- the state back to its fields: cells, lower faces, and the far boundary faces. No CTA
    // gets here before its neighbours read the p it overwrites: it has their step 1.
    {
        const T *p = my_p, *vy = my_vy;
#pragma unroll
        for (int e = 0; e < K; e++, p += lay.p_plane, vy += lay.vy_plane) {
            if (e >= kn) continue;
            const int i = i0 + e;
            const int64_t at = (int64_t)i * s.plane + in_plane;
            auto put = [&](T *to, const P &v, int lanes) {
                if (lanes >= W) {
                    pstore(to, v);
                } else {
                    T x[W];
                    unpack(v, x);
#pragma unroll
                    for (int e2 = 0; e2 < W; e2++)
                        if (e2 < lanes) to[e2] = x[e2];
                }
            };
            put(s.p + at, pload(p), col.real);
            put(s.vx + at, vx[e], col.real);
            if (i + 1 == s.nx) put(s.vx + at + s.plane, vx[e + 1], col.real);
            put(s.vy + at, pload(vy), col.real);
            if (j + 1 == s.ny) put(s.vy + at + s.pz, pload(vy + lay.row), col.real);
            put(s.vz + at, vz[e], col.real + 1);     // the top face k = nz of a padded chunk with it
            if (k0 + W == s.nz) s.vz[at + W] = vz_above[e];
            for (int r = 0; r < q.psi_shared; r++)
                put(s.psi + r * s.field + at, pload(my_psi + r * lay.psi_field + e * lay.psi_plane), col.real);
        }
    }
    report_nonfinite(s.status, is_bad(bad));
}

// The same with one barrier per step, for M <= 4 planes per thread: the velocities of all faces of a
// thread's chunks in its registers (the upper y faces, and the upper x face of its last plane,
// redundantly), p in two copies of shared memory, the relaxation states in registers for M <= 2.
// At these sizes a step is a chain of latencies (the exchange, the barrier, and the instructions
// a warp issues one after the other), so what counts is their number: no branch on where a chunk
// lies -- a neighbour outside the room is the chunk itself, a neighbour in another brick is in the
// rim, and both are only another address -- and no special pass for the brick's surface.
template <typename T, int M, int NR, bool LAYER>
__global__ void __launch_bounds__(kThreads, 1) resident_chunk_sweep(const __grid_constant__ ResidentParams<T> q) {
    using P = Pack<T>;
    constexpr int W = P::W;
    constexpr bool KEEP = M == 1;                // wall pairs and layer factors in registers
    constexpr bool PSI_REG = M <= 2;             // relaxation states in registers
    extern __shared__ __align__(16) unsigned char raw[];
    const Room<T> &s = q.room;
    const int C = q.chunks, rows = q.rows, bx = q.bx, gy = q.gy;
    const int cta = blockIdx.x, gxi = cta / gy, gyi = cta - gxi * gy;
    const int x0 = gxi * bx, y0 = gyi * rows;
    const int nbx = min(bx, s.nx - x0), nby = min(rows, s.ny - y0);   // planes and rows of this brick
    auto has_state = [&](int r) { return NR < 4 || r < q.nr; };

    const int c = threadIdx.x % C, column = threadIdx.x / C, row = column % rows, first = column / rows * M;
    const int kn = row < nby ? max(0, min(M, nbx - first)) : 0;       // planes of this thread
    const bool mine = kn > 0;
    const int i0 = min(x0 + first, s.nx - 1), k0 = c * W;
    Column<T> col;
    col.j = min(y0 + row, s.ny - 1);
    col.k0 = k0;
    col.real = min(W, s.nz - k0);
    col.tail = col.real < W;
    col.wall = q.walls && (col.j == 0 || col.j == s.ny - 1 || k0 == 0 || k0 + W >= s.nz);
    const int j = col.j, real = col.real;
    const bool tail = col.tail;
    const int64_t at0 = (int64_t)i0 * s.plane + (int64_t)j * s.pz + k0;

    // Shared memory: two copies of the brick's p, each followed by its rim as the inbox holds it --
    // x-, x+ (rows * C chunks each), y-, y+ (bx * C each) -- then the relaxation states.
    const int nxh = rows * C, nyh = bx * C, own = bx * nxh, total = 2 * (nxh + nyh);
    const int copy = (own + total) * W, me = (first * rows + row) * C + c, rc = row * C + c, xc = first * C + c;
    T *const sm = reinterpret_cast<T *>(raw);
    T *const my_psi = sm + 2 * copy + me * W;
    // the chunk below the first plane and above the last; the rows on either side of the first
    // plane's, with their distance from plane to plane
    const int x_lo = (i0 == 0 ? me : first > 0 ? me - nxh : own + rc) * W;
    const int x_hi = (i0 + kn == s.nx ? me + (kn - 1) * nxh : first + kn < bx ? me + kn * nxh : own + nxh + rc) * W;
    const bool rim_lo = row == 0 && j > 0, rim_hi = row + 1 == rows && j + 1 < s.ny;
    const int y_lo = (j == 0 ? me : row > 0 ? me - C : own + 2 * nxh + xc) * W, dy_lo = (rim_lo ? C : nxh) * W;
    const int y_hi = (j + 1 == s.ny ? me : row + 1 < rows ? me + C : own + 2 * nxh + nyh + xc) * W;
    const int dy_hi = (rim_hi ? C : nxh) * W;
    const int z_lo = k0 > 0 ? -1 : 0, z_hi = k0 + W < s.nz ? W : W - 1;

    // ---- the state of the thread's chunks, and p's first rim
    auto room_p = [&](int pi, int pj, int pc) {
        P v = pload(s.p + (int64_t)pi * s.plane + (int64_t)pj * s.pz + pc * W);
        return pc * W + W > s.nz ? mirrored(v, s.nz - pc * W) : v;
    };
    P xf[M + 1], yl[M], yh[M], zl[M], S[PSI_REG ? M : 1][NR > 0 ? NR : 1];
    T za[M];
#pragma unroll
    for (int m = 0; m < M; m++) {
        xf[m] = xf[m + 1] = yl[m] = yh[m] = zl[m] = pzero<T>();
        za[m] = T(0);
    }
#pragma unroll
    for (int m = 0; m < M; m++) {
        if (m >= kn) continue;
        const int64_t at = at0 + m * s.plane;
        if (m == 0) xf[0] = pload(s.vx + at);
        xf[m + 1] = pload(s.vx + at + s.plane);
        yl[m] = pload(s.vy + at);
        yh[m] = pload(s.vy + at + s.pz);
        zl[m] = pload(s.vz + at);
        if (k0 + W <= s.nz) za[m] = s.vz[at + W];
#pragma unroll
        for (int r = 0; r < NR; r++) {
            if (!has_state(r)) continue;
            const P v = pload(s.psi + r * s.field + at);
            if (PSI_REG) S[PSI_REG ? m : 0][r] = v;
            else pstore(my_psi + (r * own + m * nxh) * W, v);
        }
        pstore(sm + (me + m * nxh) * W, room_p(i0 + m, j, c));
    }
    uint32_t awaited = 0;                        // bit u: inbox entry threadIdx.x + u * blockDim.x
#pragma unroll
    for (int u = 0; u < kRim; u++) {
        const int h = threadIdx.x + u * blockDim.x;
        int pi = -1, pj = 0, px = 0;
        if (h < nxh) {
            if (gxi > 0 && h / C < nby) pi = x0 - 1, pj = y0 + h / C, px = h % C;
        } else if (h < 2 * nxh) {
            const int e = h - nxh;
            if (gxi + 1 < q.gx && e / C < nby) pi = x0 + bx, pj = y0 + e / C, px = e % C;
        } else if (h < 2 * nxh + nyh) {
            const int e = h - 2 * nxh;
            if (gyi > 0 && e / C < nbx) pi = x0 + e / C, pj = y0 - 1, px = e % C;
        } else if (h < total) {
            const int e = h - 2 * nxh - nyh;
            if (gyi + 1 < gy && e / C < nbx) pi = x0 + e / C, pj = y0 + rows, px = e % C;
        }
        if (pi < 0) continue;
        awaited |= 1u << u;
        pstore(sm + (own + h) * W, room_p(pi, pj, px));
    }
    // where the chunks on the brick's surface go: entries of the neighbours' inboxes
    const bool to_x0 = mine && first == 0 && gxi > 0, to_x1 = mine && first + kn == bx && gxi + 1 < q.gx;
    const bool to_y0 = mine && rim_lo, to_y1 = mine && rim_hi;
    const int e_x0 = (cta - gy) * 2 * total + nxh + rc, e_x1 = (cta + gy) * 2 * total + rc;
    const int e_y0 = (cta - 1) * 2 * total + 2 * nxh + nyh + xc, e_y1 = (cta + 1) * 2 * total + 2 * nxh + xc;

    // ---- constants of the column
    const uint32_t epoch = *q.epoch;
    const T cv = s.cv;
    bool all_points = false;
    const uint32_t points = (mine && (s.n_src | s.n_rec) != 0) ? column_points(s, j, k0, all_points, W) : 0u;
    const bool any_mine = mine && (points != 0 || all_points);
    T fu[W], fp[W];
    uint32_t walls = 0;                          // KEEP: the elements with an absorbing wall
    if (KEEP) {
#pragma unroll
        for (int e = 0; e < W; e++) {
            fu[e] = T(1);
            fp[e] = T(0);
            if (q.walls && mine && e < real && wall_pair(s, i0, j, k0 + e, fu[e], fp[e])) walls |= 1u << e;
        }
    }
    T y_high = T(1);
    if (LAYER) {
        col.y_cell = __ldg(s.cell[1] + j);
        col.y_face = __ldg(s.face[1] + j);
        y_high = __ldg(s.face[1] + j + 1);
        col.damp_y = col.y_cell != T(1) || col.y_face != T(1) || y_high != T(1);
        col.damp_z = false;
#pragma unroll
        for (int e = 0; e <= W; e++) {
            col.z_face[e] = __ldg(s.face[2] + min(k0 + e, s.nz));
            if (e < W) col.z_cell[e] = __ldg(s.cell[2] + min(k0 + e, s.nz - 1));
            col.damp_z = col.damp_z || col.z_face[e] != T(1) || (e < W && col.z_cell[e] != T(1));
        }
    }
    auto moved = [&](const P &v, const P &high, const P &low) { return psub(v, pmul(psub(high, low), cv)); };
    auto bad = finite_start(T(0));
    bool waiting = true;   // false once a wait of this thread ran out

    for (int t = 0; t < q.steps; t++) {
        const uint32_t tag = epoch + (uint32_t)t;
        T *const now = sm + (t & 1) * copy;
        // ---- the neighbours' p on the rim
        if (t > 0 && awaited != 0 && waiting) {
            const uint64_t *from = q.mailbox + ((int64_t)(cta * 2 + (t & 1)) * total + threadIdx.x) * kWords;
            uint32_t pending = awaited;
            uint64_t start = 0;
            for (int tries = 1; pending != 0 && waiting; tries++) {
#pragma unroll
                for (int u0 = 0; u0 < kRim; u0 += 2) {
                    uint64_t w[2][kWords];
#pragma unroll
                    for (int u = u0; u < u0 + 2; u++)
                        if (pending >> u & 1u) load_tagged(from + u * blockDim.x * kWords, w[u - u0]);
#pragma unroll
                    for (int u = u0; u < u0 + 2; u++) {
                        if (!(pending >> u & 1u) || !all_tagged(w[u - u0], tag)) continue;
                        put_words(now + (own + threadIdx.x + u * blockDim.x) * W, w[u - u0]);
                        pending &= ~(1u << u);
                    }
                }
                if ((tries & 63) == 0) {
                    if (start == 0) start = global_ns();
                    else if (global_ns() - start > q.wait_limit_ns) waiting = false;
                }
            }
            if (!waiting && s.status != nullptr) atomicOr(s.status, kStatusWaitTimeout);
        }
        __syncthreads();
        if (!mine) continue;
        const bool open = t + 1 < q.steps && !(cta == 0 && q.stop_step >= 0 && t >= q.stop_step);
        uint64_t *const box = q.mailbox + ((t + 1) & 1) * total * kWords;
        const T *p = now + me * W, *p_lo = now + y_lo, *p_hi = now + y_hi;
        T *next = sm + copy - (t & 1) * copy + me * W, *psi = my_psi;
        P pc = pload(p), below = pload(now + x_lo);
#pragma unroll
        for (int m = 0; m < M; m++, p += nxh * W, next += nxh * W, psi += nxh * W, p_lo += dy_lo, p_hi += dy_hi) {
            if (m >= kn) continue;
            // ---- the faces
            const int i = i0 + m;
            const P high = pload(m + 1 < M && m + 1 < kn ? p + nxh * W : now + x_hi);
            const P py_lo = pload(p_lo), py_hi = pload(p_hi);
            const T pz_lo = p[z_lo], pz_hi = p[z_hi];
            if (m == 0) xf[0] = moved(xf[0], pc, below);
            xf[m + 1] = moved(xf[m + 1], high, pc);
            yl[m] = moved(yl[m], pc, py_lo);
            yh[m] = moved(yh[m], py_hi, pc);
            zl[m] = moved(zl[m], pc, below_of(pc, pz_lo));
            za[m] = za[m] - cv * (pz_hi - last_of(pc));
            T fx = T(1);
            if (LAYER) {   // x, y, z order; an axis whose factors here are all exactly 1 is skipped
                fx = __ldg(s.cell[0] + i);
                const T fx_l = __ldg(s.face[0] + i), fx_h = __ldg(s.face[0] + i + 1);
                if (fx != T(1) || fx_l != T(1) || fx_h != T(1)) {
                    if (m == 0) xf[0] = pmul(xf[0], fx_l);
                    xf[m + 1] = pmul(xf[m + 1], fx_h);
                    yl[m] = pmul(yl[m], fx);
                    yh[m] = pmul(yh[m], fx);
                    zl[m] = pmul(zl[m], fx);
                    za[m] = za[m] * fx;
                }
                if (col.damp_y) {
                    if (m == 0) xf[0] = pmul(xf[0], col.y_cell);
                    xf[m + 1] = pmul(xf[m + 1], col.y_cell);
                    yl[m] = pmul(yl[m], col.y_face);
                    yh[m] = pmul(yh[m], y_high);
                    zl[m] = pmul(zl[m], col.y_cell);
                    za[m] = za[m] * col.y_cell;
                }
                if (col.damp_z) {
                    if (m == 0) xf[0] = times(xf[0], col.z_cell);
                    xf[m + 1] = times(xf[m + 1], col.z_cell);
                    yl[m] = times(yl[m], col.z_cell);
                    yh[m] = times(yh[m], col.z_cell);
                    zl[m] = times(zl[m], col.z_face);
                    za[m] = za[m] * col.z_face[W];
                }
            }
            // ---- the cells
            P d = psub(xf[m + 1], xf[m]);
            d = padd(d, psub(yh[m], yl[m]));
            d = padd(d, psub(above_of(zl[m], za[m]), zl[m]));
            P pe = pc;
#pragma unroll
            for (int r = 0; r < NR; r++) {
                if (!has_state(r)) continue;
                const P state = PSI_REG ? S[PSI_REG ? m : 0][r] : pload(psi + r * own * W);
                const P target = pmul(d, s.gain[r]);
                const P offset = psub(state, target);
                const P after = psub(target, pmul(offset, q.neg_decay[r]));
                pe = psub(pe, pmul(offset, q.neg_mean[r]));
                if (PSI_REG) S[PSI_REG ? m : 0][r] = after;
                else pstore(psi + r * own * W, after);
            }
            if (NR > 0) pe = psub(pe, pmul(d, q.neg_scale));
            pe = psub(pe, pmul(d, s.cp));
            if (KEEP) {
                if (walls != 0) {
                    T pn[W], po[W];
                    unpack(pe, pn);
                    unpack(pc, po);
#pragma unroll
                    for (int e = 0; e < W; e++)
                        if (walls >> e & 1u) pn[e] = pn[e] * fu[e] - po[e] * fp[e];
                    pe = repack(pn);
                }
            } else if (col.wall || (q.walls && (i == 0 || i + 1 == s.nx))) {
                pe = walled(s, col, pe, pc, i);
            }
            if (LAYER) pe = damped(col, pe, fx, col.y_cell);
            if (any_mine) {
                T pn[W];
                unpack(pe, pn);
                const int64_t step = *q.step_base + t, at = at0 + m * s.plane;
                add_sources<T, W>(s, points, all_points, at, k0, step, pn);
                record_receivers<T, W>(s, points, all_points, at, step, pn);
                pe = repack(pn);
            }
            if (tail) pe = mirrored(pe, real);
            pstore(next, pe);
            // ---- to the neighbours
            if ((to_y0 || to_y1) && open) {
                if (to_y0) send(box + (int64_t)(e_y0 + m * C) * kWords, pe, tag + 1u);
                if (to_y1) send(box + (int64_t)(e_y1 + m * C) * kWords, pe, tag + 1u);
            }
            if (m == 0 && to_x0 && open) send(box + (int64_t)e_x0 * kWords, pe, tag + 1u);
            if (m == M - 1 && to_x1 && open) send(box + (int64_t)e_x1 * kWords, pe, tag + 1u);
            bad = pfinite(bad, pe);
            pc = high;
        }
    }

    // ---- the state back to its fields: cells, lower faces, and the far boundary faces. No CTA
    // gets here before its neighbours read the p it overwrites: it has their step 1.
    const T *last = sm + (q.steps & 1) * copy + me * W;
#pragma unroll
    for (int m = 0; m < M; m++) {
        if (m >= kn) continue;
        const int64_t at = at0 + m * s.plane;
        auto put = [&](T *to, const P &v, int lanes) {
            if (lanes >= W) {
                pstore(to, v);
            } else {
                T x[W];
                unpack(v, x);
#pragma unroll
                for (int e = 0; e < W; e++)
                    if (e < lanes) to[e] = x[e];
            }
        };
        put(s.p + at, pload(last + m * nxh * W), real);
        put(s.vx + at, xf[m], real);
        if (i0 + m + 1 == s.nx) put(s.vx + at + s.plane, xf[m + 1], real);
        put(s.vy + at, yl[m], real);
        if (j + 1 == s.ny) put(s.vy + at + s.pz, yh[m], real);
        put(s.vz + at, zl[m], real + 1);         // the top face k = nz of a padded chunk with it
        if (k0 + W == s.nz) s.vz[at + W] = za[m];
#pragma unroll
        for (int r = 0; r < NR; r++)
            if (has_state(r))
                put(s.psi + r * s.field + at,
                    PSI_REG ? S[PSI_REG ? m : 0][r] : pload(my_psi + (r * own + m * nxh) * W), real);
    }
    report_nonfinite(s.status, is_bad(bad));
}

// The step counter and the launch's first tag: epoch[0] is this launch's, epoch[1] the next's.
__global__ void resident_begin(int64_t *step_base, int64_t first_step, uint32_t *epoch, uint32_t steps) {
    *step_base = first_step;
    epoch[0] = epoch[1] + 1u;
    epoch[1] = epoch[0] + steps;
}

template <typename T, int K>
const void *resident_kernel(int n_relax, bool layer) {
#define ACF_RESIDENT(KERNEL)                                                                            \
    (n_relax == 0   ? (layer ? (const void *)KERNEL<T, K, 0, true> : (const void *)KERNEL<T, K, 0, false>) \
     : n_relax == 3 ? (layer ? (const void *)KERNEL<T, K, 3, true> : (const void *)KERNEL<T, K, 3, false>) \
                    : (layer ? (const void *)KERNEL<T, K, 4, true> : (const void *)KERNEL<T, K, 4, false>))
    if constexpr (K <= kChunkPlanes) return ACF_RESIDENT(resident_chunk_sweep);
    else return ACF_RESIDENT(resident_sweep);
#undef ACF_RESIDENT
}

template <typename T>
const void *resident_kernel(int planes, int n_relax, bool layer) {
    switch (planes) {
        case 1: return resident_kernel<T, 1>(n_relax, layer);
        case 2: return resident_kernel<T, 2>(n_relax, layer);
        case 3: return resident_kernel<T, 3>(n_relax, layer);
        case 4: return resident_kernel<T, 4>(n_relax, layer);
        case 6: return resident_kernel<T, 6>(n_relax, layer);
        default: return resident_kernel<T, 8>(n_relax, layer);
    }
}

}  // namespace

// Among all bricks that fit, the one with the least work per step: warps x planes of arithmetic,
// plus the rim its threads receive. The weights are rough, and only rank the bricks of one room: three states held
// cost 10 to 20 % of a step (64^3 1.95 and 2.15 us, 96^3 5.2 and 5.9), one left in L2 more than all the held ones
// (112^3, two of three held, 8.7 and 13.9). The two-barrier form takes 1.0 to 1.4 times as long per chunk (96^3, 4
// planes of 384 threads, 5.2 and with air 5.9; 104^3, 6 of 352, 8.4 and 11.5); weighted twice, it is left to the rooms
// that the other does not fit. Whether the plan beats the step it replaces is resident_faster's question.
template <typename T>
ResidentPlan resident_plan(int nx, int ny, int nz, int n_relax, bool layer, int sms, size_t smem_limit) {
    constexpr int W = Pack<T>::W;
    ResidentPlan best;
    double least = 0.0;
    const int64_t chunks = ((int64_t)nz + W - 1) / W;
    if (chunks > kThreads) return best;
    const int C = (int)chunks;
    for (int K : {1, 2, 3, 4, 6, 8}) {
        for (int tx = 1; tx * C <= kThreads && (tx - 1) * K < nx; tx++) {
            const int bx = K * tx, gx = (nx + bx - 1) / bx;
            for (int rows = 1; rows * tx * C <= kThreads && rows <= ny; rows++) {
                const int gy = (ny + rows - 1) / rows;
                if ((int64_t)gx * gy > sms) continue;
                const int threads = (tx * rows * C + 31) / 32 * 32, rim = 2 * C * (rows + bx);
                if (rim > kRim * threads) continue;
                size_t smem;
                int held = n_relax;
                double psi_cost = 0.2;
                if (K <= kChunkPlanes) {         // every relaxation state on chip, or not this form
                    const size_t states = K <= 2 ? 0 : (size_t)n_relax * bx * rows * C;
                    smem = (2 * ((size_t)bx * rows * C + rim) + states) * W * sizeof(T);
                    if (smem > smem_limit) continue;
                } else {
                    const BrickLayout<W> none(bx, rows, C, 0);
                    const size_t fixed = (size_t)none.end * sizeof(T) + (size_t)rim * sizeof(int);
                    if (fixed > smem_limit) continue;
                    const size_t one_psi = (size_t)none.psi_field * sizeof(T);
                    held = (int)std::min<size_t>((size_t)n_relax, (smem_limit - fixed) / one_psi);
                    if (n_relax - held > 1) continue;
                    smem = fixed + held * one_psi;
                    psi_cost = 0.3;
                }
                // the two-barrier form costs about twice as much per chunk
                const double cost = (double)K * threads * (K <= kChunkPlanes ? 1.0 : 2.0) *
                                        (1.0 + psi_cost * held + 1.0 * (n_relax - held)) + 0.5 * rim;
                if (best.planes != 0 && cost >= least) continue;
                least = cost;
                best.planes = K;
                best.tx = tx;
                best.rows = rows;
                best.chunks = C;
                best.bx = bx;
                best.gx = gx;
                best.gy = gy;
                best.threads = threads;
                best.psi_shared = held;
                best.smem = smem;
                best.mailbox_bytes = (size_t)gx * gy * 2 * rim * kWords * sizeof(uint64_t);
            }
        }
    }
    if (best.planes > 0) {
        const void *kernel = resident_kernel<T>(best.planes, n_relax, layer);
        int per_sm = 0;
        if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_limit) != cudaSuccess ||
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, best.threads, best.smem) != cudaSuccess ||
            per_sm < 1) {
            cudaGetLastError();
            best.planes = 0;
        }
    }
    return best;
}

template <typename T>
cudaError_t resident_launch(const ResidentPlan &plan, const ResidentRun<T> &run, int64_t first_step,
                            cudaStream_t stream) {
    ResidentParams<T> q{};
    q.room = run.room;
    q.tx = plan.tx;
    q.rows = plan.rows;
    q.chunks = plan.chunks;
    q.bx = plan.bx;
    q.gx = plan.gx;
    q.gy = plan.gy;
    q.nr = run.n_relax;
    q.psi_shared = plan.psi_shared;
    q.walls = run.walls ? 1 : 0;
    q.steps = run.steps;
    q.stop_step = run.stop_step;
    for (int r = 0; r < ACF_MAX_RELAXATION; r++) {
        q.neg_decay[r] = -run.room.decay[r];
        q.neg_mean[r] = -run.room.mean[r];
    }
    q.neg_scale = -run.room.relax_scale;
    q.mailbox = (uint64_t *)run.mailbox;
    q.step_base = run.step_base;
    q.epoch = run.epoch;
    q.wait_limit_ns = run.wait_limit_ns;
    resident_begin<<<1, 1, 0, stream>>>(run.step_base, first_step, run.epoch, (uint32_t)run.steps);
    // Cooperative: every CTA is resident (they wait for their neighbours) or the launch fails.
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(plan.gx * plan.gy));
    cfg.blockDim = dim3((unsigned)plan.threads);
    cfg.dynamicSmemBytes = plan.smem;
    cfg.stream = stream;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    void *args[] = {&q};
    return cudaLaunchKernelExC(&cfg, resident_kernel<T>(plan.planes, run.n_relax, run.layer), args);
}

}  // namespace acf

#endif
