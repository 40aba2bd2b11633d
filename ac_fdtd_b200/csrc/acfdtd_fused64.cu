// acfdtd_fused64.cu -- the fused step in double precision.
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

#include "acfdtd_fused64.cuh"

#include <algorithm>

#include "acfdtd_pack.cuh"

namespace acf {
namespace {

template <typename T>
__device__ __forceinline__ Pack<T> pack_ldg(const T *a) {
    return {__ldg(reinterpret_cast<const double2 *>(a))};
}

template <bool LAYER, bool WALLS, int NR>
__device__ __forceinline__ void pack_column(const FusedParams<double> &f, int i_begin, int i_end, int j, int c,
                                            int64_t step) {
    using T = double;
    using P = Pack<T>;
    constexpr int W = P::W;
    const Room<T> &s = f.room;
    const int k0 = c * W, real = min(W, s.nz - k0);
    const bool tail = real < W;
    const T cv = s.cv;
    const int64_t column = (int64_t)j * s.pz + k0;
    // neighbours as offsets from the chunk, 0 where the room ends
    const int64_t y_lo = j > 0 ? -s.pz : 0, y_hi = j + 1 < s.ny ? s.pz : 0;
    const int z_lo = k0 > 0 ? -1 : 0, z_hi = k0 + W < s.nz ? W : W - 1;
    const bool top = k0 + W == s.nz;             // the far z face, not in any chunk of cells
    bool all_points = false;
    const uint32_t points = (s.n_src | s.n_rec) != 0 ? column_points(s, j, k0, all_points, W) : 0u;
    const bool any_mine = points != 0 || all_points;
    const bool wall_column = WALLS && (j == 0 || j + 1 == s.ny || k0 == 0 || k0 + W >= s.nz);

    T fy_c = 1.0, fy_l = 1.0, fy_h = 1.0;
    bool damp_y = false, damp_z = false;
    if (LAYER) {
        fy_c = __ldg(s.cell[1] + j);
        fy_l = __ldg(s.face[1] + j);
        fy_h = __ldg(s.face[1] + j + 1);
        damp_y = fy_c != 1.0 || fy_l != 1.0 || fy_h != 1.0;
#pragma unroll
        for (int e = 0; e <= W; e++) {
            damp_z = damp_z || __ldg(s.face[2] + min(k0 + e, s.nz)) != 1.0;
            if (e < W) damp_z = damp_z || __ldg(s.cell[2] + min(k0 + e, s.nz - 1)) != 1.0;
        }
    }
    // z factors at cells and at faces, read where used (they stay in L1)
    auto z_cells = [&](const P &v) {
        return P{make_double2(v.a.x * __ldg(s.cell[2] + k0), v.a.y * __ldg(s.cell[2] + min(k0 + 1, s.nz - 1)))};
    };
    auto z_faces = [&](const P &v) {
        return P{make_double2(v.a.x * __ldg(s.face[2] + k0), v.a.y * __ldg(s.face[2] + k0 + 1))};
    };
    auto moved = [&](const P &v, const P &high, const P &low) { return psub(v, pmul(psub(high, low), cv)); };

    // Carried from plane to plane: p(i) and the updated vx on face i.
    P pc, xl;
    {
        const int64_t base = (int64_t)i_begin * s.plane + column;
        pc = pack_ldg(s.p + base);
        const P below = pack_ldg(s.p + base - (i_begin > 0 ? s.plane : 0));
        xl = moved(pack_ldg(s.vx + base), pc, below);
        if (tail) pc = mirrored(pc, real);
        if (LAYER) {
            const T fx = __ldg(s.face[0] + i_begin);
            if (fx != 1.0) xl = pmul(xl, fx);
            if (damp_y) xl = pmul(xl, fy_c);
            if (damp_z) xl = z_cells(xl);
        }
    }
    T bad = finite_start(0.0);

    for (int i = i_begin; i < i_end; i++) {
        const int64_t base = (int64_t)i * s.plane + column;
        const bool inner = i + 1 < s.nx;
        if (s.prefetch && i + 1 < i_end) {       // the next plane's own-row inputs into L2
            const int64_t next = base + s.plane;
            if (i + 2 < s.nx) prefetch_l2(s.p + next + s.plane);
            prefetch_l2(s.vx + next + s.plane);
            prefetch_l2(s.vy + next);
            prefetch_l2(s.vz + next);
#pragma unroll
            for (int r = 0; r < NR; r++) prefetch_l2(s.psi + r * s.field + next);
        }
        // ---- loads, all before the first store
        P ph = pack_ldg(s.p + base + (inner ? s.plane : 0));
        const P py_l = pack_ldg(s.p + base + y_lo), py_h = pack_ldg(s.p + base + y_hi);
        P xh = pack_ldg(s.vx + base + s.plane), yl = pack_ldg(s.vy + base), yh = pack_ldg(s.vy + base + s.pz);
        P zl = pack_ldg(s.vz + base);
        const T pz_l = __ldg(s.p + base + z_lo), pz_h = __ldg(s.p + base + z_hi);
        T za = k0 + W <= s.nz ? __ldg(s.vz + base + W) : 0.0;
        P S[NR > 0 ? NR : 1];
#pragma unroll
        for (int r = 0; r < NR; r++) S[r] = pload(s.psi + r * s.field + base);

        // ---- the faces
        if (tail) ph = mirrored(ph, real);
        xh = moved(xh, ph, pc);
        yl = moved(yl, pc, py_l);
        yh = moved(yh, py_h, pc);
        zl = moved(zl, pc, below_of(pc, pz_l));
        za = za - cv * ((z_hi == W ? pz_h : pc.a.y) - pc.a.y);
        T fx = 1.0;
        if (LAYER) {   // x, y, z order; an axis whose factors here are all exactly 1 is skipped
            fx = __ldg(s.cell[0] + i);
            const T fx_h = __ldg(s.face[0] + i + 1);
            if (fx != 1.0 || fx_h != 1.0) {
                xh = pmul(xh, fx_h);
                yl = pmul(yl, fx);
                yh = pmul(yh, fx);
                zl = pmul(zl, fx);
                za = za * fx;
            }
            if (damp_y) {
                xh = pmul(xh, fy_c);
                yl = pmul(yl, fy_l);
                yh = pmul(yh, fy_h);
                zl = pmul(zl, fy_c);
                za = za * fy_c;
            }
            if (damp_z) {
                xh = z_cells(xh);
                yl = z_cells(yl);
                yh = z_cells(yh);
                zl = z_faces(zl);
                za = za * __ldg(s.face[2] + min(k0 + W, s.nz));
            }
        }
        // ---- the cells
        P d = psub(xh, xl);
        d = padd(d, psub(yh, yl));
        d = padd(d, psub(above_of(zl, za), zl));
        P pe = pc;
#pragma unroll
        for (int r = 0; r < NR; r++) {
            const P target = pmul(d, s.gain[r]);
            const P offset = psub(S[r], target);
            P next = padd(pmul(offset, s.decay[r]), target);
            pe = padd(pe, pmul(offset, s.mean[r]));
            if (tail) next = keep_from(next, S[r], real);
            S[r] = next;
        }
        if (NR > 0) pe = padd(pe, pmul(d, s.relax_scale));
        pe = psub(pe, pmul(d, s.cp));
        if (wall_column || (WALLS && (i == 0 || !inner))) {
            T pn[W], po[W];
            unpack(pe, pn);
            unpack(pc, po);
#pragma unroll
            for (int e = 0; e < W; e++) {
                T fu, fp;
                if (e < real && wall_pair(s, i, j, k0 + e, fu, fp)) pn[e] = pn[e] * fu - po[e] * fp;
            }
            pe = repack(pn);
        }
        if (LAYER) {
            if (fx != 1.0) pe = pmul(pe, fx);
            if (damp_y) pe = pmul(pe, fy_c);
            if (damp_z) pe = z_cells(pe);
        }
        T pn[W];
        unpack(pe, pn);
        if (any_mine) add_sources<T, W>(s, points, all_points, base, k0, step, pn);
        pe = repack(pn);
        if (tail) pe = mirrored(pe, real);
        bad = pfinite(bad, pe);

        // ---- stores: p, the three lower faces, the far boundary faces, psi in place. A slab's ghost
        // planes get their p from the neighbours' sweeps, its own boundary planes go there too.
        if (i >= s.own_lo && i < s.own_hi) pstore(f.np + base, pe);
        if (s.ghost_lo != nullptr && i == s.own_lo) pstore(s.ghost_lo + column, pe);
        if (s.ghost_hi != nullptr && i == s.own_hi - 1) pstore(s.ghost_hi + column, pe);
        pstore(f.nvx + base, xl);
        pstore(f.nvy + base, yl);
        pstore(f.nvz + base, zl);
        if (!inner) pstore(f.nvx + base + s.plane, xh);
        if (y_hi == 0) pstore(f.nvy + base + s.pz, yh);
        if (top) f.nvz[base + W] = za;
#pragma unroll
        for (int r = 0; r < NR; r++) pstore(s.psi + r * s.field + base, S[r]);
        if (any_mine) record_receivers<T, W>(s, points, all_points, base, step, pn);
        xl = xh;
        pc = ph;
    }
    report_nonfinite(s.status, is_bad(bad));
}

template <bool LAYER, bool WALLS, int NR>
__global__ void __launch_bounds__(128, NR > 0 ? 6 : 8) pack_sweep(const __grid_constant__ FusedParams<double> f) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = blockIdx.y * blockDim.y + threadIdx.y;
    if (c * Pack<double>::W >= f.room.nz || j >= f.room.ny) return;
    const bool any_point = (f.room.n_src | f.room.n_rec) != 0;
    const int64_t step = any_point ? (*f.step_base + f.local_step) : 0;
    const int i_begin = blockIdx.z * f.planes;
    pack_column<LAYER, WALLS, NR>(f, i_begin, min(f.room.nx, i_begin + f.planes), j, c, step);
}

template <bool LAYER, bool WALLS>
void launch_pack(const FusedParams<double> &f, int n_relax, dim3 grid, dim3 block, cudaStream_t st) {
    switch (n_relax) {
        case 0: pack_sweep<LAYER, WALLS, 0><<<grid, block, 0, st>>>(f); break;
        case 1: pack_sweep<LAYER, WALLS, 1><<<grid, block, 0, st>>>(f); break;
        case 2: pack_sweep<LAYER, WALLS, 2><<<grid, block, 0, st>>>(f); break;
        case 3: pack_sweep<LAYER, WALLS, 3><<<grid, block, 0, st>>>(f); break;
        default: pack_sweep<LAYER, WALLS, 4><<<grid, block, 0, st>>>(f); break;
    }
}

}  // namespace

void launch_pack_sweep(const FusedParams<double> &f, bool layer, bool walls, int n_relax, int block_threads,
                       cudaStream_t st) {
    const int chunks = (f.room.nz + Pack<double>::W - 1) / Pack<double>::W;
    int bx = 1;
    while (bx < chunks && bx < 32) bx <<= 1;
    const int by = std::max(1, std::min<int>(f.room.ny, std::min(block_threads, 128) / bx));
    const dim3 block(bx, by, 1);
    const dim3 grid((chunks + bx - 1) / bx, (f.room.ny + by - 1) / by, (f.room.nx + f.planes - 1) / f.planes);
    if (layer) {
        if (walls) launch_pack<true, true>(f, n_relax, grid, block, st);
        else launch_pack<true, false>(f, n_relax, grid, block, st);
    } else {
        if (walls) launch_pack<false, true>(f, n_relax, grid, block, st);
        else launch_pack<false, false>(f, n_relax, grid, block, st);
    }
}

}  // namespace acf
