// acfdtd_device.cuh -- what the device code of every translation unit shares: vector access, the
// description of a room, walls, sources and receivers of a column, packed single precision.

#ifndef ACFDTD_DEVICE_CUH
#define ACFDTD_DEVICE_CUH

#include <cuda_runtime.h>

#include <cstdint>

#include "acfdtd_b200.h"

namespace acf {

constexpr int kVec = 4;            // elements per thread along z

// Limits of every wait inside a kernel: two seconds, or this many tries.
constexpr uint64_t kWaitLimitNs = 2000000000ull;
constexpr int kWaitLimitIterations = 1 << 21;

// ------------------------------------------------------------------------------------------
// Vector access: 4 consecutive elements, one 16-byte access for float, two for double.

template <typename T>
struct Vec4;

template <>
struct Vec4<float> {
    __device__ __forceinline__ static void load(const float *__restrict__ a, float v[4]) {
        const float4 t = *reinterpret_cast<const float4 *>(a);
        v[0] = t.x; v[1] = t.y; v[2] = t.z; v[3] = t.w;
    }
    __device__ __forceinline__ static void store(float *__restrict__ a, const float v[4]) {
        *reinterpret_cast<float4 *>(a) = make_float4(v[0], v[1], v[2], v[3]);
    }
    // Read-only path: only for arrays no thread writes during the kernel.
    __device__ __forceinline__ static void ldg(const float *__restrict__ a, float v[4]) {
        const float4 t = __ldg(reinterpret_cast<const float4 *>(a));
        v[0] = t.x; v[1] = t.y; v[2] = t.z; v[3] = t.w;
    }
    // Streaming (evict-first) load: data read once, such as the adjoint's history.
    __device__ __forceinline__ static void ldcs(const float *a, float v[4]) {
        const float4 t = __ldcs(reinterpret_cast<const float4 *>(a));
        v[0] = t.x; v[1] = t.y; v[2] = t.z; v[3] = t.w;
    }
};

template <>
struct Vec4<double> {
    __device__ __forceinline__ static void load(const double *__restrict__ a, double v[4]) {
        const double2 t0 = *reinterpret_cast<const double2 *>(a);
        const double2 t1 = *reinterpret_cast<const double2 *>(a + 2);
        v[0] = t0.x; v[1] = t0.y; v[2] = t1.x; v[3] = t1.y;
    }
    __device__ __forceinline__ static void store(double *__restrict__ a, const double v[4]) {
        *reinterpret_cast<double2 *>(a) = make_double2(v[0], v[1]);
        *reinterpret_cast<double2 *>(a + 2) = make_double2(v[2], v[3]);
    }
    __device__ __forceinline__ static void ldg(const double *__restrict__ a, double v[4]) {
        const double2 t0 = __ldg(reinterpret_cast<const double2 *>(a));
        const double2 t1 = __ldg(reinterpret_cast<const double2 *>(a + 2));
        v[0] = t0.x; v[1] = t0.y; v[2] = t1.x; v[3] = t1.y;
    }
    __device__ __forceinline__ static void ldcs(const double *a, double v[4]) {
        const double2 t0 = __ldcs(reinterpret_cast<const double2 *>(a));
        const double2 t1 = __ldcs(reinterpret_cast<const double2 *>(a + 2));
        v[0] = t0.x; v[1] = t0.y; v[2] = t1.x; v[3] = t1.y;
    }
};

// Streaming (evict-first) stores of 4 elements, for data written once and read once much later
// -- the adjoint's D/psi history -- so that it does not push the state out of L2.
__device__ __forceinline__ void store_streaming(float *a, const float v[4]) {
    __stcs(reinterpret_cast<float4 *>(a), make_float4(v[0], v[1], v[2], v[3]));
}
__device__ __forceinline__ void store_streaming(double *a, const double v[4]) {
    __stcs(reinterpret_cast<double2 *>(a), make_double2(v[0], v[1]));
    __stcs(reinterpret_cast<double2 *>(a + 2), make_double2(v[2], v[3]));
}

// The start of a kernel that launch_after may have launched before the kernel in front of it
// has finished (programmatic dependent launch). Every thread passes the wait before it reads anything
// a kernel writes, or writes: it ends when that kernel is complete and its writes are visible. The
// first instruction lets the next step's blocks be launched as soon as all of this kernel's have started,
// into the room that its last blocks leave.
__device__ __forceinline__ void step_next() { asm volatile("griddepcontrol.launch_dependents;"); }
__device__ __forceinline__ void step_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void step_begin() {
    step_next();
    step_wait();
}

// Ask L2 for the line holding `a` ahead of its load: the request holds no register and no
// shared memory, so a marching thread can have its next plane on the way from DRAM while it
// computes the current one. Only addresses the thread will load later are passed.
template <typename T>
__device__ __forceinline__ void prefetch_l2(const T *a) {
    asm volatile("prefetch.global.L2 [%0];" ::"l"(a));
}

// Bits of a handle's device status word.
constexpr int32_t kStatusWaitTimeout = 1;   // a staged sweep gave up waiting for its copies
constexpr int32_t kStatusNonFinite = 2;     // a sweep produced a NaN or infinite pressure

__device__ __forceinline__ unsigned lane_id() {
    unsigned lane;
    asm("mov.u32 %0, %%laneid;" : "=r"(lane));
    return lane;
}

// Non-finite detector: acc = fma(x, 0, acc) is acc + 0 for every finite x (one rounding, exact)
// and NaN once any x was NaN or infinite; NaN then stays. One fused instruction per value.
template <typename T>
__device__ __forceinline__ T finite_acc(T acc, T x) {
    if constexpr (sizeof(T) == 4) return __fmaf_rn(x, 0.0f, acc);
    else return __fma_rn(x, 0.0, acc);
}

// Raise kStatusNonFinite once per warp whose threads saw a non-finite value.
__device__ __forceinline__ void report_nonfinite(int32_t *status, bool bad) {
    const unsigned mask = __ballot_sync(__activemask(), bad);
    if (bad && status != nullptr && lane_id() == (unsigned)(__ffs(mask) - 1))
        atomicOr(status, kStatusNonFinite);
}

// ------------------------------------------------------------------------------------------
// What the sweeps read about one room. Plain data, identical on host and device.

template <typename T>
struct Room {
    int32_t nx, ny, nz, nchunks;
    int32_t prefetch;              // 1: marching threads ask L2 for their next plane ahead
    int32_t reserved;
    // A slab of a room cut along x: the single-room pressure sweep updates the planes
    // [own_lo, own_hi) only, and also stores p of planes own_lo and own_hi - 1 into the
    // neighbours' ghost planes (null: no neighbour on that side; a peer address when the
    // neighbour lives on another GPU). A whole room: [0, nx), no ghosts.
    int32_t own_lo, own_hi;
    T *ghost_lo, *ghost_hi;
    int64_t pz, plane, field;      // row pitch, plane pitch, elements per field
    T *p, *vx, *vy, *vz, *psi;     // psi: n_relax fields back to back
    T cv, cp, cs, relax_scale;
    T decay[ACF_MAX_RELAXATION], mean[ACF_MAX_RELAXATION], gain[ACF_MAX_RELAXATION];
    const T *cell[3];              // layer profiles at cell centres
    const T *face[3];              // layer profiles at faces
    const T *shell[6];             // wall pairs (1/(1+a), a/(1+a)) per face cell
    int32_t n_src;
    int32_t n_rec;
    const int64_t *src_off;        // padded offsets
    const int64_t *src_len;
    const T *src_sig;
    int64_t src_stride;
    const int64_t *rec_off;        // padded offsets
    const int64_t *rec_start;      // first absolute step recorded
    const int64_t *src_col;        // in-plane offsets (padded offset mod plane): j * pz + k
    const int64_t *rec_col;
    T *rec;
    int64_t rec_stride, rec_origin;
    // Status word of the handle (device memory): the sweeps that write p set kStatusNonFinite
    // in it when a pressure they produced is NaN or infinite. Null: not checked.
    int32_t *status;
};

// Forward history kept for the adjoint: per step, p^n and p-tilde^n -- pressure before the step
// and before the wall closed form -- on every boundary cell (two blocks of shell_total values,
// first every p^n, then every p-tilde^n), and, for a
// segment of steps, the divergence D^n and the relaxation states psi^n before their update.
// Boundary cells are indexed as in the wall shells: the first face of FACES order a cell lies
// on, then row-major over that face's two other axes; face f starts at face_off[f].
template <typename T>
struct History {
    T *shell;                      // steps x 2 x shell_total values, or null
    int64_t shell_total, shell_step0, shell_steps;
    int64_t face_off[6];
    T *fields;                     // slots x (1 + n_relax) fields (padded geometry), or null;
                                   // step n uses slot (n - fields_step0) mod fields_slots
    int64_t fields_step0;
    int32_t fields_slots;
    int32_t reserved;
};

// A fused step: the velocity and pressure updates of a step in one sweep, from the current copy of
// p and v into the next.
template <typename T>
struct FusedParams {
    Room<T> room;                  // p, vx, vy, vz: current state (read); psi updated in place
    T *np, *nvx, *nvy, *nvz;       // next state (written), same geometry
    const int64_t *step_base;
    int32_t local_step;
    int32_t planes;
};

// One unit of work of a batched sweep: up to blockDim.x consecutive (row, chunk) pairs of one
// room, over the x planes [i_begin, i_end).
struct Tile {
    int32_t room, first, count, i_begin, i_end, reserved;
};

// One fused step of every room: rooms points at the descriptions for the copy all rooms are at.
template <typename T>
struct FusedBatchParams {
    const FusedParams<T> *rooms;
    const Tile *tiles;
    int32_t n_tiles;
    int32_t local_step;
    const int64_t *step_base;
    const History<T> *history;     // recorded runs: one per room
};

// ------------------------------------------------------------------------------------------
// Walls, sources and receivers of one (row, chunk) column.

// First face (FACES order) that cell (i, j, k) lies on, and its index within that face's
// row-major (b, c) array; -1 for interior cells.
template <typename T>
__device__ __forceinline__ int shell_face(const Room<T> &s, int i, int j, int k, int64_t &idx) {
    if (i == 0) { idx = (int64_t)j * s.nz + k; return 0; }
    if (i == s.nx - 1) { idx = (int64_t)j * s.nz + k; return 1; }
    if (j == 0) { idx = (int64_t)i * s.nz + k; return 2; }
    if (j == s.ny - 1) { idx = (int64_t)i * s.nz + k; return 3; }
    if (k == 0) { idx = (int64_t)i * s.ny + j; return 4; }
    if (k == s.nz - 1) { idx = (int64_t)i * s.ny + j; return 5; }
    return -1;
}

template <typename T>
__device__ __forceinline__ bool wall_pair(const Room<T> &s, int i, int j, int k, T &fu, T &fp) {
    int64_t idx;
    const int f = shell_face(s, i, j, k, idx);
    if (f < 0) return false;
    const T *entry = s.shell[f] + 2 * idx;
    fu = __ldg(entry);
    fp = __ldg(entry + 1);
    return fp != T(0) || fu != T(1);
}

// The wall closed form for the cells of one column chunk at plane i: on an x-face plane or a
// y-face row (both uniform across a warp) every cell is tested; elsewhere only the chunk's
// k = 0 and k = nz - 1 cells can lie on a face -- a z face, the first in FACES order for them --
// so the thread reads just those pairs instead of searching four cells. `apply(e, fu, fp)` is
// called for each cell e (< real) with an absorbing pair.
template <typename T, typename Apply>
__device__ __forceinline__ void column_walls(const Room<T> &s, int i, int j, int k0, int real,
                                             Apply apply) {
    if (i == 0 || i == s.nx - 1 || j == 0 || j == s.ny - 1) {
#pragma unroll
        for (int e = 0; e < kVec; e++) {
            T fu, fp;
            if (e < real && wall_pair(s, i, j, k0 + e, fu, fp)) apply(e, fu, fp);
        }
        return;
    }
    const bool bottom = k0 == 0, top_chunk = k0 + kVec >= s.nz;
    if (!bottom && !top_chunk) return;
    const int64_t at = 2 * ((int64_t)i * s.ny + j);
    if (bottom) {
        const T fu = __ldg(s.shell[4] + at), fp = __ldg(s.shell[4] + at + 1);
        if (fp != T(0) || fu != T(1)) apply(0, fu, fp);
    }
    const int top = s.nz - 1 - k0;
    if (top_chunk && (top > 0 || k0 > 0)) {     // k = nz - 1 is not also k = 0
        const T fu = __ldg(s.shell[5] + at), fp = __ldg(s.shell[5] + at + 1);
        if (fp != T(0) || fu != T(1)) apply(top, fu, fp);
    }
}

// Sources (bit q) and receivers (bit n_src + r) that lie in one (row j, chunk at k0) column,
// found once per column so that the march visits them only at their own plane instead of
// scanning every point at every plane. Beyond 32 points `all` is set and every point is
// scanned, as before.
template <typename T>
__device__ __forceinline__ uint32_t column_points(const Room<T> &s, int j, int k0, bool &all,
                                                 int width = kVec) {
    const int total = s.n_src + s.n_rec;
    all = total > 32;
    uint32_t mask = 0;
    if (all) return 0;
    const int64_t first = (int64_t)j * s.pz + k0;
    for (int q = 0; q < total; q++) {
        const int64_t col = q < s.n_src ? s.src_col[q] : s.rec_col[q - s.n_src];
        if (col >= first && col < first + width) mask |= 1u << q;
    }
    return mask;
}

__device__ __forceinline__ uint32_t source_bits(uint32_t mask, int n_src) {
    return n_src >= 32 ? mask : mask & ((1u << n_src) - 1u);
}

__device__ __forceinline__ uint32_t receiver_bits(uint32_t mask, int n_src) {
    return n_src >= 32 ? 0u : mask >> n_src;
}

// Sources of the column's cell at `base`, after damping, in the order they were added
// (scheme.py:293,360-363).
template <typename T, int W = kVec>
__device__ __forceinline__ void add_sources(const Room<T> &s, uint32_t mask, bool all, int64_t base,
                                            int k0, int64_t step, T Pn[W]) {
    uint32_t m = all ? 0u : source_bits(mask, s.n_src);
    for (int q = all ? 0 : -1; all ? q < s.n_src : m != 0; q++) {
        if (!all) {
            q = __ffs(m) - 1;
            m &= m - 1;
        }
        const int64_t d = s.src_off[q] - base;
        if (d >= 0 && d < W && k0 + d < s.nz && step < s.src_len[q]) {
#pragma unroll
            for (int e = 0; e < W; e++)
                if (e == d) Pn[e] = Pn[e] + s.cs * s.src_sig[q * s.src_stride + step];
        }
    }
}

// Receivers of the column read the finished pressure (scheme.py:294-296).
template <typename T, int W = kVec>
__device__ __forceinline__ void record_receivers(const Room<T> &s, uint32_t mask, bool all,
                                                 int64_t base, int64_t step, const T Pn[W]) {
    uint32_t m = all ? 0u : receiver_bits(mask, s.n_src);
    for (int r = all ? 0 : -1; all ? r < s.n_rec : m != 0; r++) {
        if (!all) {
            r = __ffs(m) - 1;
            m &= m - 1;
        }
        const int64_t d = s.rec_off[r] - base;
        if (d >= 0 && d < W && step >= s.rec_start[r]) {
            T v = Pn[0];
#pragma unroll
            for (int e = 1; e < W; e++)
                if (e == d) v = Pn[e];
            s.rec[r * s.rec_stride + (step - s.rec_origin)] = v;
        }
    }
}

// Boundary history of one step for the wall gradients: p^n and p before the wall closed form,
// on every boundary cell, in two blocks of shell_total values per step (first p, then the other)
// indexed as the wall shells are -- each cell on the first face of FACES order it lies on, then
// row-major over that face's two other axes. A column on an x-face plane or a y-face row owns
// contiguous entries for its whole chunk; elsewhere only its k = 0 and k = nz - 1 cells are on a
// (z) face.
template <typename T, int W = kVec>
__device__ __forceinline__ void record_shell(const Room<T> &s, const History<T> &hist, int i, int j,
                                             int k0, int64_t step, const T (&P)[W], const T (&PT)[W]) {
    const int64_t slot = step - hist.shell_step0;
    if (slot < 0 || slot >= hist.shell_steps) return;
    T *hp = hist.shell + slot * 2 * hist.shell_total;
    T *ht = hp + hist.shell_total;
    if (i == 0 || i == s.nx - 1 || j == 0 || j == s.ny - 1) {
        const bool x_face = i == 0 || i == s.nx - 1;
        const int f = x_face ? (i == 0 ? 0 : 1) : (j == 0 ? 2 : 3);
        const int64_t at = hist.face_off[f] + (x_face ? (int64_t)j : (int64_t)i) * s.nz + k0;
#pragma unroll
        for (int e = 0; e < W; e++)
            if (k0 + e < s.nz) {
                hp[at + e] = P[e];
                ht[at + e] = PT[e];
            }
        return;
    }
    const int64_t at = (int64_t)i * s.ny + j;
    if (k0 == 0) {
        hp[hist.face_off[4] + at] = P[0];
        ht[hist.face_off[4] + at] = PT[0];
    }
    const int top = s.nz - 1 - k0;   // element of k = nz - 1, unless that cell is also k = 0
    if (s.nz > 1 && top >= 0 && top < W) {
#pragma unroll
        for (int e = 0; e < W; e++)
            if (e == top) {
                hp[hist.face_off[5] + at] = P[e];
                ht[hist.face_off[5] + at] = PT[e];
            }
    }
}

// ------------------------------------------------------------------------------------------
// Packed single precision (sm_100 f32x2), each lane rounded exactly as the scalar operation it
// replaces. a +- b is the fused a + (+-1) b: the product by +-1 is exact, so the one rounding is
// that of a +- b. The code generator was measured to fuse a packed multiply into a packed add
// that consumes it -- one rounding where the reference has two -- even with contraction
// disabled, and even through a + 1 * b; it was not measured to do so through a - b. So every
// "plus a product" below is written as "minus the product by the negated coefficient", which
// rounds identically (negation is exact and rounding is symmetric in sign), and add2 only ever
// adds values that are not products.
__device__ __forceinline__ float2 add2(float2 a, float2 b) {
    return __ffma2_rn(b, make_float2(1.0f, 1.0f), a);
}
__device__ __forceinline__ float2 sub2(float2 a, float2 b) {
    return __ffma2_rn(b, make_float2(-1.0f, -1.0f), a);
}
__device__ __forceinline__ float2 mul2(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ float2 dup2(float x) { return make_float2(x, x); }
__device__ __forceinline__ float2 damp2(float2 v, float2 fa, float2 fb, float2 fc) {
    return mul2(mul2(mul2(v, fa), fb), fc);
}

__device__ __forceinline__ float2 lo2(float4 v) { return make_float2(v.x, v.y); }
__device__ __forceinline__ float2 hi2(float4 v) { return make_float2(v.z, v.w); }

__device__ __forceinline__ uint64_t global_ns() {
    uint64_t t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

}  // namespace acf

#endif
