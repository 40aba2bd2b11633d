// acfdtd_fused_kernel.cuh -- the fused step of one column of 16-byte chunks, in either precision.
//
// Faces on walls are not asked for (the pressure outside is the cell's own, a difference of zero:
// neighbour offsets are 0 where the room ends, so no load is conditional), layer factors that are
// exactly 1 are skipped, and a chunk that reaches past nz repeats its last real pressure.
//
// p, v and the relaxation states are read by plain loads: a step that was launched early is resident
// while the step before still writes them, and the read-only path (__ldg) is for data that nothing
// writes during the kernel. Layer profiles and wall pairs, written by the host alone, take that path.

#ifndef ACFDTD_FUSED_KERNEL_CUH
#define ACFDTD_FUSED_KERNEL_CUH

#include "acfdtd_pack.cuh"

namespace acf {
namespace {

// One column of chunks over planes [i_begin, i_end). REC: also write the forward history.
template <typename T, bool LAYER, bool WALLS, int NR, bool REC = false>
__device__ __forceinline__ void pack_column(const FusedParams<T> &f, int i_begin, int i_end, int j, int c,
                                            int64_t step, const History<T> *hist = nullptr) {
    using P = Pack<T>;
    constexpr int W = P::W;
    // With a layer in single precision the relaxation states are loaded after the faces: held through the damping of
    // the faces they do not fit the 96 registers of 20 warps per SM (136 bytes spilled, so 72; 8 rooms of 96 to 180
    // with air and a layer 331 us per step, so 295; at 128 registers and 16 warps 319).
    constexpr bool STATES_LATE = LAYER && sizeof(T) == 4 && !REC;
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
    const bool wall_column = (WALLS || REC) && (j == 0 || j + 1 == s.ny || k0 == 0 || k0 + W >= s.nz);

    T fy_c = T(1), fy_l = T(1), fy_h = T(1);
    bool damp_y = false, damp_z = false;
    if (LAYER) {
        fy_c = __ldg(s.cell[1] + j);
        fy_l = __ldg(s.face[1] + j);
        fy_h = __ldg(s.face[1] + j + 1);
        damp_y = fy_c != T(1) || fy_l != T(1) || fy_h != T(1);
#pragma unroll
        for (int e = 0; e <= W; e++) {
            const T face = __ldg(s.face[2] + min(k0 + e, s.nz));
            damp_z = damp_z || face != T(1);
            if (e < W) {
                const T cell = __ldg(s.cell[2] + min(k0 + e, s.nz - 1));
                damp_z = damp_z || cell != T(1);
            }
        }
    }
    // z factors at cells and at faces, read where used (they stay in L1)
    auto z_cells = [&](const P &v) {
        T x[W];
        unpack(v, x);
#pragma unroll
        for (int e = 0; e < W; e++) x[e] = x[e] * __ldg(s.cell[2] + min(k0 + e, s.nz - 1));
        return repack(x);
    };
    auto z_faces = [&](const P &v) {
        T x[W];
        unpack(v, x);
#pragma unroll
        for (int e = 0; e < W; e++) x[e] = x[e] * __ldg(s.face[2] + min(k0 + e, s.nz));
        return repack(x);
    };
    auto moved = [&](const P &v, const P &high, const P &low) { return psub(v, pmul(psub(high, low), cv)); };

    // Carried from plane to plane: p(i) and the updated vx on face i.
    P pc, xl;
    {
        const int64_t base = (int64_t)i_begin * s.plane + column;
        pc = pload(s.p + base);
        const P below = pload(s.p + base - (i_begin > 0 ? s.plane : 0));
        xl = moved(pload(s.vx + base), pc, below);
        if (tail) pc = mirrored(pc, real);
        if (LAYER) {
            const T fx = __ldg(s.face[0] + i_begin);
            if (fx != T(1)) xl = pmul(xl, fx);
            if (damp_y) xl = pmul(xl, fy_c);
            if (damp_z) xl = z_cells(xl);
        }
    }
    auto bad = finite_start(T(0));

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
        // ---- loads, before the first store
        P ph = pload(s.p + base + (inner ? s.plane : 0));
        const P py_l = pload(s.p + base + y_lo), py_h = pload(s.p + base + y_hi);
        P xh = pload(s.vx + base + s.plane), yl = pload(s.vy + base), yh = pload(s.vy + base + s.pz);
        P zl = pload(s.vz + base);
        const T pz_l = s.p[base + z_lo], pz_h = s.p[base + z_hi];
        T za = k0 + W <= s.nz ? s.vz[base + W] : T(0);
        P S[NR > 0 ? NR : 1];
        auto load_states = [&]() {
#pragma unroll
            for (int r = 0; r < NR; r++) S[r] = pload(s.psi + r * s.field + base);
        };
        if (!STATES_LATE) load_states();

        // ---- the faces
        if (tail) ph = mirrored(ph, real);
        xh = moved(xh, ph, pc);
        yl = moved(yl, pc, py_l);
        yh = moved(yh, py_h, pc);
        zl = moved(zl, pc, below_of(pc, pz_l));
        za = za - cv * ((z_hi == W ? pz_h : last_of(pc)) - last_of(pc));
        T fx = T(1);
        if (LAYER) {   // x, y, z order; an axis whose factors here are all exactly 1 is skipped
            fx = __ldg(s.cell[0] + i);
            const T fx_h = __ldg(s.face[0] + i + 1);
            if (fx != T(1) || fx_h != T(1)) {
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
        if (STATES_LATE) load_states();
        // ---- the cells
        P d = psub(xh, xl);
        d = padd(d, psub(yh, yl));
        d = padd(d, psub(above_of(zl, za), zl));
        if (REC && hist->fields) {               // D and psi of this step, for the air gradients
            const int64_t rel = step - hist->fields_step0;
            if (rel >= 0) {
                T *h = hist->fields + rel % hist->fields_slots * (1 + NR) * s.field + base;
                pstore_streaming(h, d);
#pragma unroll
                for (int r = 0; r < NR; r++) pstore_streaming(h + (1 + r) * s.field, S[r]);
            }
        }
        P pe = pc;
#pragma unroll
        for (int r = 0; r < NR; r++) {
            const P target = pmul(d, s.gain[r]);
            const P offset = psub(S[r], target);
            P next = psub(target, pmul(offset, -s.decay[r]));     // see padd
            pe = psub(pe, pmul(offset, -s.mean[r]));
            if (tail) next = keep_from(next, S[r], real);
            S[r] = next;
        }
        if (NR > 0) pe = psub(pe, pmul(d, -s.relax_scale));
        pe = psub(pe, pmul(d, s.cp));
        if (wall_column || ((WALLS || REC) && (i == 0 || !inner))) {
            T pn[W], po[W];
            unpack(pe, pn);
            unpack(pc, po);
            if (REC && hist->shell) record_shell<T, W>(s, *hist, i, j, k0, step, po, pn);
#pragma unroll
            for (int e = 0; e < W; e++) {
                T fu, fp;
                if (WALLS && e < real && wall_pair(s, i, j, k0 + e, fu, fp)) pn[e] = pn[e] * fu - po[e] * fp;
            }
            pe = repack(pn);
        }
        if (LAYER) {
            if (fx != T(1)) pe = pmul(pe, fx);
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

}  // namespace
}  // namespace acf

#endif
