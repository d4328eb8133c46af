// Face-flux kernel: reconstruction, viscous and convective flux of one face per thread.
#pragma once
#include "kernels.cuh"

namespace tg {

// arguments of a face-flux launch
struct FaceLaunch {
    Sizes s;
    const void *geom;  // Geometry<R>*
    const double *q;
    const void *rec;
    double gamma, mu, prandtl;
    void *G;
    int *err;  // device error word (bounded waits that give up set ERR_TIMEOUT)
    PressureRef pr_ref;  // FP32-flux form: reference pressure per instance
    int polls;           // limit of the staged kernel's first wait (MBAR_POLLS unless a test lowers it)
    Mask mask;
    const void *side;    // side records (k_gradient SIDES), or null: gradient records only
};

// ---- face fluxes (src/equations/derivative.c:18-227) ------------------------------------------
//
// Writes the flux record G[f] = (convective - viscous) flux * area; the cell gather adds it to the
// left cell and subtracts it from the right one, as teal's face loops do.

// Reconstructed face state of one side: q + (psi * grad) . offset per variable, streamed one
// variable at a time from the cell's gradient record so only the result stays live
// (derivative.c:158-164)
template <typename R, bool FOLD>
__device__ __forceinline__ void reconstruct(const Prim<R> &q, const R *__restrict__ rec, int c, V3<R> off,
                                            R (&out)[5])
{
    R qv[5] = {q.rho, q.u.x, q.u.y, q.u.z, q.p};
#pragma unroll
    for (int v = 0; v < 5; v++) {
        R gx, gy, gz, ps;
        grad_rec_load(rec, c, v, gx, gy, gz, ps);
        V3<R> gv = v3(gx, gy, gz);
        if (!FOLD) {
            gv = v3(gv.x * ps, gv.y * ps, gv.z * ps);
        }
        out[v] = at_face(qv[v], gv, off);
    }
}

// Two ways to reach the geometry of a face: straight from the SoA arrays (DirectGeo, one face per
// thread, loads issued by the thread) or from a tile staged in shared memory (FaceTile, bulk
// asynchronous copies). Both expose the same accessors; `i` is the face's element in the tile.

template <typename R>
struct DirectGeo {
    const Geometry<R> &g;
    int F, f;
    __device__ __forceinline__ int2 cells(int) const { return g.lr[f]; }
    __device__ __forceinline__ V3<R> normal(int) const { return load_v3(g.basis, F, f); }
    __device__ __forceinline__ Basis<R> basis(int) const { return load_basis(g.basis, F, f); }
    // the basis again later in the thread: re-read (L1) instead of kept live in registers
    __device__ __forceinline__ Basis<R> basis_again(int) const { return reload_basis(g.basis, F, f); }
    __device__ __forceinline__ V3<R> normal_again(int) const
    {
        return v3(reload(g.basis + f), reload(g.basis + F + f), reload(g.basis + 2 * F + f));
    }
    __device__ __forceinline__ V3<R> offl(int) const { return load_v3(g.offl, F, f); }
    __device__ __forceinline__ V3<R> offr(int) const { return load_v3(g.offr, F, f); }
    __device__ __forceinline__ R area(int) const { return __ldg(g.area + f); }
    __device__ __forceinline__ V3<R> corr(int) const { return load_v3(g.corr, F, f); }
    __device__ __forceinline__ R corr_norm(int) const { return __ldg(g.corr + 3 * F + f); }
};

// Geometry of one tile of FACE_BLOCK consecutive faces in shared memory, staged by bulk
// asynchronous copies (one per SoA row, all in flight at once, completing on one mbarrier) so the
// streamed face geometry costs the threads neither registers nor load instructions; rows: area,
// basis (9 in the exact form; the normal's 3 otherwise, see frame_of), offsets left / right
// (3 + 3, second order).
template <typename R, int ORDER>
struct FaceTile {
    static constexpr int PAD = 16 / int(sizeof(R));
    static constexpr int SROW = FACE_BLOCK + PAD;
    static constexpr int NBASIS = kExact ? 9 : 3;
    static constexpr int ROWS = 1 + NBASIS + (ORDER == 2 ? 6 : 0);
    static constexpr int R_AREA = 0, R_BASIS = 1, R_OFFL = 1 + NBASIS, R_OFFR = R_OFFL + 3;
    R geo[ROWS][SROW];
    int2 lr[FACE_BLOCK + 2];
    uint64_t bar;
    uint8_t shift[ROWS + 1];  // elements before the tile's first face in each staged row

    __device__ __forceinline__ const R *row_src(const Geometry<R> &g, int F, int r) const
    {
        if (r == R_AREA) return g.area;
        if (r < R_BASIS + NBASIS) return g.basis + (size_t)(r - R_BASIS) * F;
        if (ORDER == 2 && r < R_OFFL + 3) return g.offl + (size_t)(r - R_OFFL) * F;
        return g.offr + (size_t)(r - R_OFFR) * F;
    }

    // thread 0 issues the copies of faces [f0, f0 + n); every thread then waits (bounded).
    // Returns false after a wait that gave up (the error word then has the timeout bit); the
    // decision is the same in every thread of the block.
    // `polls` bounds the first wait (MBAR_POLLS normally; a smaller value lets a test make it give up);
    // the drain after a wait that gave up always uses the full MBAR_POLLS.
    __device__ __forceinline__ bool stage(const Geometry<R> &g, int F, int f0, int n, int *err, int polls)
    {
        if (threadIdx.x == 0) {
            mbar_init(&bar, 1);
            uint32_t total = stage_span(lr, g.lr + f0, n, &bar, false, &shift[ROWS]);
            for (int r = 0; r < ROWS; r++) {
                total += stage_span(geo[r], row_src(g, F, r) + f0, n, &bar, false, &shift[r]);
            }
            mbar_arrive_expect_tx(&bar, total);
            stage_span(lr, g.lr + f0, n, &bar, true, nullptr);
            for (int r = 0; r < ROWS; r++) {
                stage_span(geo[r], row_src(g, F, r) + f0, n, &bar, true, nullptr);
            }
        }
        __syncthreads();
        const bool ok = mbar_wait_bounded(&bar, 0, polls);
        if (__syncthreads_or(!ok)) {
            if (threadIdx.x == 0) {
                atomicOr(err, ERR_TIMEOUT);
            }
            mbar_wait_bounded(&bar, 0, MBAR_POLLS);  // let copies still in flight land before the block exits
            return false;
        }
        return true;
    }

    __device__ __forceinline__ R at(int r, int i) const { return geo[r][shift[r] + i]; }
    __device__ __forceinline__ V3<R> v3_at(int r, int i) const { return v3(at(r, i), at(r + 1, i), at(r + 2, i)); }
    __device__ __forceinline__ int2 cells(int i) const { return lr[shift[ROWS] + i]; }
    __device__ __forceinline__ V3<R> normal(int i) const { return v3_at(R_BASIS, i); }
    template <int NB = NBASIS>
    __device__ __forceinline__ Basis<R> basis(int i) const
    {
        static_assert(NB == 9, "the full basis is staged in the exact form only");
        Basis<R> b;
        b.x = v3_at(R_BASIS, i);
        b.y = v3_at(R_BASIS + 3, i);
        b.z = v3_at(R_BASIS + 6, i);
        return b;
    }
    template <int NB = NBASIS>
    __device__ __forceinline__ Basis<R> basis_again(int i) const { return basis<NB>(i); }
    __device__ __forceinline__ V3<R> normal_again(int i) const { return normal(i); }
    __device__ __forceinline__ V3<R> offl(int i) const { return v3_at(R_OFFL, i); }
    __device__ __forceinline__ V3<R> offr(int i) const { return v3_at(R_OFFR, i); }
    __device__ __forceinline__ R area(int i) const { return at(R_AREA, i); }
};

// The reconstructed states of a face's two sides while its viscous flux runs: in registers in FP64 (at 128 of
// them, 16 blocks an SM), in shared memory in the FP32-flux form (at 64 registers, 32 blocks an SM; a
// thread's own column, volatile so that the values do not stay in registers all the same)
template <typename R>
struct Sides {
    R v[10];
    __device__ __forceinline__ explicit Sides(R *) {}
    __device__ __forceinline__ void set(int k, R x) { v[k] = x; }
    __device__ __forceinline__ R get(int k) const { return v[k]; }
};
template <>
struct Sides<float> {
    volatile float *p;
    __device__ __forceinline__ explicit Sides(float *column) : p(column) {}
    __device__ __forceinline__ void set(int k, float x) { p[k * FACE_BLOCK] = x; }
    __device__ __forceinline__ float get(int k) const { return p[k * FACE_BLOCK]; }
};

// Viscous flux of face f (element i of its tile) and the reconstructed states pl, pr of its sides, from
// one pass over both cells' states and gradient records: the face average of the states and unlimited
// gradients, corrected along the centre-to-centre direction (derivative.c:71-89), in the face normal's frame.
template <typename R, bool FOLD, typename Geo>
__device__ __forceinline__ Cons<R> viscous_face(const Geo &geo, int i, bool boundary, int2 c, int N,
                                                const double *__restrict__ q, const R *__restrict__ rec, double pref,
                                                R gamma, R mu, R prandtl, Sides<R> &sides)
{
    R qm[5], gm[15];
    const V3<R> unit = geo.corr(i), offl = geo.offl(i), offr = geo.offr(i);
    const R cnorm = geo.corr_norm(i);
    const R inv_norm = R(1) / cnorm;
#pragma unroll
    for (int v = 0; v < 5; v++) {
        const double ql = __ldg(q + (size_t)v * N + c.x), qr = __ldg(q + (size_t)v * N + c.y);
        R ax, ay, az, ap;
        grad_rec_load(rec, c.x, v, ax, ay, az, ap);
        // FP32 fluxes reconstruct the pressure relative to the instance's reference (Local::dp); the
        // difference is taken in FP64, before the rounding to FP32
        const double p0 = (v == 4 && sizeof(R) == sizeof(float)) ? pref : 0.0;
        V3<R> ga = v3(ax, ay, az);
        sides.set(v, at_face(R(ql - p0), FOLD ? ga : v3(ax * ap, ay * ap, az * ap), offl));
        if (boundary) {  // the ghost state enters unreconstructed (derivative.c:203-211)
            sides.set(5 + v, R(qr - p0));
        }
        else {
            R bx, by, bz, bp;
            grad_rec_load(rec, c.y, v, bx, by, bz, bp);
            sides.set(5 + v, at_face(R(qr - p0), FOLD ? v3(bx, by, bz) : v3(bx * bp, by * bp, bz * bp), offr));
            ga = v3((ax + bx) / R(2), (ay + by) / R(2), (az + bz) / R(2));
        }
        qm[v] = (R(ql) + R(qr)) / R(2);
        const R dq = R(qr) - R(ql);
        const R adjust = dot(ga, unit) - (kExact ? (dq / cnorm) : (dq * inv_norm));
        ga = sub(ga, mul(adjust, unit));
        gm[3 * v] = ga.x;
        gm[3 * v + 1] = ga.y;
        gm[3 * v + 2] = ga.z;
    }
    Grad<R> gg;
    gg.rho = v3(gm[0], gm[1], gm[2]);
    gg.ux = v3(gm[3], gm[4], gm[5]);
    gg.uy = v3(gm[6], gm[7], gm[8]);
    gg.uz = v3(gm[9], gm[10], gm[11]);
    gg.p = v3(gm[12], gm[13], gm[14]);
    // the viscous flux needs only the normal row of the basis
    Basis<R> nb;
    nb.x = geo.normal_again(i);
    nb.y = nb.x;
    nb.z = nb.x;
    return viscous_central(prim_from(qm), gg, gamma, mu, prandtl, nb);
}

// Flux record of a face with a viscous flux. Its bound is the L1 data pipe and the latency of the gathers
// (66 % of peak LSU wavefronts, 25 % L1 hits with one pass for either flux), so both cells' states and
// gradient records are read once: the pass gives the viscous flux and the reconstructed states, then the
// convective flux follows. `column`: this thread's shared-memory column (FP32-flux form). Measured
// against two passes at 96 / 64 registers, TGV 128^3: FP64 0.467 -> 0.421 ms (0.464 at 96 registers with
// the states in shared memory, 0.438 at 80), FP32-flux 0.301 -> 0.267 ms (0.275-0.298 at fewer
// resident blocks). The exact form, whose viscous record is of its own, stores it before the convective flux:
// kept across it, its face kernel took 0.593 ms, so 0.580.
template <typename R, int FK, bool FOLD, typename Geo>
__device__ __forceinline__ void face_flux_ns(const Geo &geo, int i, int f, const Sizes &s,
                                             const double *__restrict__ q, const R *__restrict__ rec, R gamma, R ig,
                                             R mu, R prandtl, R *__restrict__ G, const PressureRefOf<R> &pr_ref,
                                             R *column)
{
    const bool boundary = (f >= s.F_in) && (f < s.F_bd);
    const int2 c = geo.cells(i);
    wait_for_previous();
    q = after_wait(q);
    rec = after_wait(rec);
    double pref = 0.0;
    if constexpr (sizeof(R) == sizeof(float)) {
        pref = after_wait(pr_ref).of(c.x);
    }
    Sides<R> sides(column);
    const Cons<R> fv = viscous_face<R, FOLD>(geo, i, boundary, c, s.N, q, rec, pref, gamma, mu, prandtl, sides);
    if constexpr (kExact) {
        const R area = geo.area(i);
        const R gv[5] = {fv.rho * area, fv.m.x * area, fv.m.y * area, fv.m.z * area, fv.e * area};
        flux_rec_store(G + flux_rec2_offset(s.F), s.F, f, gv);
    }
    R pl[5], pr[5];
#pragma unroll
    for (int v = 0; v < 5; v++) {
        pl[v] = sides.get(v);
        pr[v] = sides.get(5 + v);
    }
    Cons<R> fc{R(0), v3(R(0), R(0), R(0)), R(0)};
    if (FK != FK_NONE) {
        Basis<R> b;
        R factor = R(0);
        if constexpr (kExact) {
            b = geo.basis_again(i);
        }
        else {
            const V3<R> n = geo.normal_again(i);
            factor = frame_factor(n);
            b = frame_of(n, factor);
        }
        const Local<R> l = make_local(prim_from(pl), gamma, b, R(pref), ig);
        const Local<R> r = make_local(prim_from(pr), gamma, b, R(pref), ig);
        fc = convective_flux_local<FK>(l, r, gamma);
        if constexpr (kExact) {
            fc.m = to_global(geo.basis_again(i), fc.m);
        }
        else {
            fc.m = to_global(frame_of(geo.normal_again(i), factor), fc.m);
        }
    }
    const R area = geo.area(i);
    R gf[5] = {fc.rho * area, fc.m.x * area, fc.m.y * area, fc.m.z * area, fc.e * area};
    if constexpr (!kExact) {
        gf[0] -= fv.rho * area;
        gf[1] -= fv.m.x * area;
        gf[2] -= fv.m.y * area;
        gf[3] -= fv.m.z * area;
        gf[4] -= fv.e * area;
    }
    flux_rec_store(G, s.F, f, gf);
}

// The flux record of face f (element i of its tile) without a viscous flux.
// Records: G[f] = (convective - viscous) * area; in the exact translation units with a viscous
// flux, G[f] = convective * area and G[flux_rec2_offset(F) + f] = viscous * area instead, because teal adds all of a
// cell's viscous terms before its convective ones (derivative.c:279-292) and the cell gather must
// repeat that order.
template <typename R, int FK, int ORDER, bool FOLD, typename Geo>
__device__ __forceinline__ void face_flux(const Geo &geo, int i, int f, const Sizes &s, const double *__restrict__ q,
                                          const R *__restrict__ rec, R gamma, R *__restrict__ G,
                                          const PressureRefOf<R> &pr_ref)
{
    const int N = s.N;
    const bool boundary = (f >= s.F_in) && (f < s.F_bd);
    const int2 c = geo.cells(i);
    wait_for_previous();
    q = after_wait(q);
    rec = after_wait(rec);
    // FP32 fluxes work with the pressure relative to the instance's reference (Local::dp); the
    // difference is taken in FP64, before the rounding to FP32
    double pref = 0.0;
    if constexpr (sizeof(R) == sizeof(float)) {
        pref = after_wait(pr_ref).of(c.x);
    }

    // convective flux: the basis and the cell states are dead while the flux runs in the face frame
    // and are re-read afterwards
    Cons<R> fc{R(0), v3(R(0), R(0), R(0)), R(0)};
    if (FK != FK_NONE) {
        Local<R> l, r;
        {
            Prim<R> ql, qr;
            if constexpr (sizeof(R) == sizeof(float)) {
                ql = load_prim_rel<R>(q, N, c.x, pref);
                qr = load_prim_rel<R>(q, N, c.y, pref);
            }
            else {
                ql = load_prim<R>(q, N, c.x);
                qr = load_prim<R>(q, N, c.y);
            }
            // the stored basis in the exact form; the normal and tangents of its own otherwise
            Basis<R> b;
            if constexpr (kExact) {
                b = geo.basis(i);
            }
            else {
                b = frame_of(geo.normal(i));
            }
            if (ORDER == 1) {
                l = make_local(ql, gamma, b, R(pref));
                r = make_local(qr, gamma, b, R(pref));
            }
            else {
                R pl[5], pr[5];
                reconstruct<R, FOLD>(ql, rec, c.x, geo.offl(i), pl);
                if (boundary) {  // the ghost state enters unreconstructed (derivative.c:203-211)
                    pr[0] = qr.rho, pr[1] = qr.u.x, pr[2] = qr.u.y, pr[3] = qr.u.z, pr[4] = qr.p;
                }
                else {
                    reconstruct<R, FOLD>(qr, rec, c.y, geo.offr(i), pr);
                }
                l = make_local(prim_from(pl), gamma, b, R(pref));
                r = make_local(prim_from(pr), gamma, b, R(pref));
            }
        }
        fc = convective_flux_local<FK>(l, r, gamma);
        if constexpr (kExact) {
            fc.m = to_global(geo.basis_again(i), fc.m);
        }
        else {
            fc.m = to_global(frame_of(geo.normal_again(i)), fc.m);
        }
    }
    R area = geo.area(i);
    R gf[5] = {fc.rho * area, fc.m.x * area, fc.m.y * area, fc.m.z * area, fc.e * area};

    flux_rec_store(G, s.F, f, gf);
}

// Flux record of face f between two side records (k_gradient SIDES): the reconstructed states are read,
// not formed, so a face costs two records, its normal and its area, and no gather of states or gradients.
// l, r: the face's Geometry::sides. The states of inner cells are not read: the cells of k_cell_fluxes are
// updated in place while other blocks still form their fluxes. A periodic owner's side comes from its
// record alone; state rows that are read (boundary ghosts, a partition's halo) no cell update writes.
template <typename R, int FK>
__device__ __forceinline__ void side_flux(const Sizes &s, const Geometry<R> &g, int f, int l, int r, V3<R> n, R area,
                                          const double *__restrict__ q, const R *__restrict__ side,
                                          const R *__restrict__ rec, R gamma, R ig,
                                          const PressureRefOf<R> &pr_ref, R (&gf)[5])
{
    double pref = 0.0;
    R pl[5], pr[5];
    if constexpr (sizeof(R) == sizeof(float)) {
        pref = after_wait(pr_ref).of(side_cell(l >= 0 ? l : r));
    }
    auto row_state = [&](int row) {
        if constexpr (sizeof(R) == sizeof(float)) {
            return load_prim_rel<R>(q, s.N, row, pref);
        }
        else {
            return load_prim<R>(q, s.N, row);
        }
    };
    if (l >= 0) {
        side_load(side, s.SL, l, pl);
    }
    else {
        reconstruct<R, true>(row_state(~l), rec, ~l, load_v3(g.offl, s.F, f), pl);
    }
    if (r >= 0) {
        side_load(side, s.SL, r, pr);
    }
    else if (f >= s.F_in && f < s.F_bd) {  // the ghost state enters unreconstructed (derivative.c:203-211)
        const Prim<R> qr = row_state(~r);
        pr[0] = qr.rho, pr[1] = qr.u.x, pr[2] = qr.u.y, pr[3] = qr.u.z, pr[4] = qr.p;
    }
    else if (~r < s.C) {  // a periodic ghost's owner
        const V3<R> off = load_v3(g.offr, s.F, f);
#pragma unroll
        for (int v = 0; v < 5; v++) {
            R gx, gy, gz, qv;
            grad_rec_load(rec, ~r, v, gx, gy, gz, qv);
            pr[v] = at_face(qv, v3(gx, gy, gz), off);
        }
    }
    else {
        reconstruct<R, true>(row_state(~r), rec, ~r, load_v3(g.offr, s.F, f), pr);
    }
    const Basis<R> b = frame_of(n);
    Cons<R> fc{R(0), v3(R(0), R(0), R(0)), R(0)};
    if (FK != FK_NONE) {
        fc = convective_flux_local<FK>(make_local(prim_from(pl), gamma, b, R(pref), ig),
                                       make_local(prim_from(pr), gamma, b, R(pref), ig), gamma);
        fc.m = to_global(b, fc.m);
    }
    gf[0] = mul_rn(fc.rho, area);
    gf[1] = mul_rn(fc.m.x, area);
    gf[2] = mul_rn(fc.m.y, area);
    gf[3] = mul_rn(fc.m.z, area);
    gf[4] = mul_rn(fc.e, area);
}

template <typename R, int FK, bool M>
__global__ void __launch_bounds__(SIDE_BLOCK, side_minb<R>()) k_face_sides(Sizes s, Geometry<R> g,
                                                   const double *__restrict__ q, const R *__restrict__ side,
                                                   const R *__restrict__ rec, R gamma, R ig, R *__restrict__ G,
                                                   PressureRefOf<R> pr_ref, Mask mask)
{
    static_assert(sizeof(R) == 0 || !kExact, "the exact form has no side records");
    let_next_start();
    const int f = s.lo + blockIdx.x * SIDE_BLOCK + threadIdx.x;
    const int fc = min(f, s.hi - 1);
    const int2 e = __ldg(g.sides + fc);
    const V3<R> n = load_v3(g.basis, s.F, fc);
    const R area = __ldg(g.area + fc);
    wait_for_previous();
    q = after_wait(q);
    side = after_wait(side);
    rec = after_wait(rec);
    if (f >= s.hi || (M && mask.leaves_out(side_cell(e.x >= 0 ? e.x : e.y)))) {
        return;
    }
    R gf[5];
    side_flux<R, FK>(s, g, f, e.x, e.y, n, area, q, side, rec, gamma, ig, pr_ref, gf);
    flux_rec_store(G, s.F, f, gf);
}

// Face fluxes and cell update in one launch for small meshes: a block is a tile of 32 cells, warp j computes
// the fluxes of the cells' slots j (the left-to-right flux of the face, as k_face_sides: each inner face
// is computed by both of its cells, with the same bits), five warps sum them in slot order and one
// finishes the cells as k_cell does. It saves a launch and the round trip of the flux records, and pays
// with twice the flux arithmetic: worth it while a launch costs more than that arithmetic. Steps of periodic hllc
// boxes, two launches / one, us: 8 k cells 40.6 / 33.0, 16 k 46.6 / 39.5, 18.9 k 48.5 / 39.7, 20.5 k 51.4 / 47.8, 24.6 k
// 51.7 / 51.9, 49 k 67.7 / 72.3 (FP32 fluxes 39.0 / 28.9, 43.5 / 34.4, 43.5 / 34.8, 44.3 / 36.2, 47.6 / 43.3, 57.6 /
// 59.7); implicit steps of 37 k cells 2.06 / 2.17 ms. The line lies at one wave of 148 SMs x 128 cells
// (TG_FUSED_CELLS). The blocks update the state in place while others form their fluxes, so side_flux reads no
// inner cell's state.
template <typename R, int FK>
__global__ void __launch_bounds__(SIDE_TILE, 4) k_cell_fluxes(FaceLaunch a, Geometry<R> g, CellLaunch b)
{
    static_assert(sizeof(R) == 0 || !kExact, "the exact form has no side records");
    __shared__ R s_flux[5][SIDE_TILE];
    __shared__ int s_face[SIDE_TILE];
    __shared__ double s_sum[5][32];
    let_next_start();
    const Sizes &s = a.s;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int c = blockIdx.x * 32 + lane;
    const int cnt = c < s.C ? int(b.slot_cnt[c]) : 0;
    const bool in = warp < cnt;
    const int sf = in ? __ldg(b.slot_face + (size_t)warp * s.SL + c) : 0;
    const int f = sf >= 0 ? sf : ~sf;
    const int2 e = __ldg(g.sides + f);
    const V3<R> n = load_v3(g.basis, s.F, f);
    const R area = __ldg(g.area + f);
    PressureRefOf<R> pr_ref{};
    if constexpr (sizeof(R) == sizeof(float)) {
        pr_ref = a.pr_ref;
    }
    wait_for_previous();
    const double *q = after_wait(a.q);
    const R *side = after_wait(static_cast<const R *>(a.side));
    const R *rec = after_wait(static_cast<const R *>(a.rec));
    if (a.mask.on && !__any_sync(0xffffffffu, c < s.C && !a.mask.leaves_out(c))) {  // the same cells in every warp
        return;
    }
    R gf[5] = {R(0), R(0), R(0), R(0), R(0)};
    if (in) {
        side_flux<R, FK>(s, g, f, e.x, e.y, n, area, q, side, rec, R(a.gamma), R(1) / (R(a.gamma) - R(1)), pr_ref, gf);
    }
#pragma unroll
    for (int v = 0; v < 5; v++) {
        s_flux[v][threadIdx.x] = gf[v];
    }
    s_face[threadIdx.x] = sf;
    __syncthreads();
    if (warp < 5) {
        double acc = 0;
#pragma unroll
        for (int j = 0; j < MAX_SLOTS; j++) {
            if (j < cnt) {
                const double x = double(s_flux[warp][j * 32 + lane]);
                acc = s_face[j * 32 + lane] >= 0 ? acc + x : acc - x;
            }
        }
        s_sum[warp][lane] = acc;
    }
    __syncthreads();
    if (warp != 0 || c >= s.C || (b.mode == 0 && a.mask.leaves_out(c))) {
        return;
    }
    int act = 1;
    double step = 0.0;
    if (b.mode != 0) {
        const int inst = __ldg(b.seg.cell_inst + c);
        act = b.st.active[inst];
        step = b.st.step[inst];
    }
    const double ivol = 1.0 / __ldg(b.cd.volume + c);
    double r[5];
#pragma unroll
    for (int v = 0; v < 5; v++) {
        r[v] = -s_sum[v][lane] * ivol;
    }
    finish_cell(b.mode, b.ns, s.C, s.N, c, r, act, b.alpha, step, b.last, b.rows, b.prop, b.cd, b.U0, b.q, b.Rout, b.dtc);
}

// whether a residual leaves out face c: both cells lie in one instance, and a partition's faces may have
// a halo row on their left
__device__ __forceinline__ bool left_out(const Mask &mask, int2 c, int C)
{
    return mask.leaves_out(c.x < C ? c.x : c.y);
}

// One thread per face, geometry loaded by the threads. face_minb caps the registers so that
// several blocks stay resident per SM.
// X: this is the exact translation unit's instantiation (a distinct kernel name per arithmetic). M: some
// instances are left out (Mask; the test alone made the Navier-Stokes kernel 12 % slower, TGV 128^3
// 0.417 -> 0.467 ms, so launches without a mask have a kernel without it).
template <typename R, int FK, bool NS, int ORDER, bool FOLD, bool X, bool M>
__global__ void __launch_bounds__(FACE_BLOCK, face_minb<R>(NS)) k_face(Sizes s, Geometry<R> g, const double *__restrict__ q,
                                                   const R *__restrict__ rec, R gamma, R ig, R mu, R prandtl,
                                                   R *__restrict__ G, PressureRefOf<R> pr_ref, Mask mask)
{
    static_assert(X == kExact, "exact kernels live in the exact translation units only");
    let_next_start();
    const int f = s.lo + blockIdx.x * FACE_BLOCK + threadIdx.x;
    if (f >= s.hi) {
        wait_for_previous();
        return;
    }
    DirectGeo<R> geo{g, s.F, f};
    if (M) {
        wait_for_previous();
        if (left_out(mask, geo.cells(0), s.C)) {
            return;
        }
    }
    if constexpr (NS && ORDER == 2) {
        __shared__ R aside[sizeof(R) == sizeof(float) ? 10 * FACE_BLOCK : 1];
        face_flux_ns<R, FK, FOLD>(geo, 0, f, s, q, rec, gamma, ig, mu, prandtl, G, pr_ref,
                                  aside + (sizeof(R) == sizeof(float) ? threadIdx.x : 0));
    }
    else {
        face_flux<R, FK, ORDER, FOLD>(geo, 0, f, s, q, rec, gamma, G, pr_ref);
    }
}

// One tile of FACE_BLOCK faces per block, its geometry staged in shared memory by bulk copies
// before the threads (one face each) start (no viscous flux: its register budget leaves too few blocks
// resident to hide the copies). A wait that gives up sets ERR_TIMEOUT in the error
// word and ends the block.
template <typename R, int FK, int ORDER, bool FOLD, bool X>
__global__ void __launch_bounds__(FACE_BLOCK, face_minb<R>(false)) k_face_staged(Sizes s, Geometry<R> g,
                                                          const double *__restrict__ q,
                                                          const R *__restrict__ rec, R gamma,
                                                          R *__restrict__ G, int *err,
                                                          PressureRefOf<R> pr_ref, int polls, Mask mask)
{
    static_assert(X == kExact, "exact kernels live in the exact translation units only");
    __shared__ __align__(16) FaceTile<R, ORDER> t;
    let_next_start();
    const int f0 = s.lo + blockIdx.x * FACE_BLOCK;
    const int n = min(FACE_BLOCK, s.hi - f0);
    if (!t.stage(g, s.F, f0, n, err, polls)) {
        wait_for_previous();
        return;
    }
    wait_for_previous();
    if (threadIdx.x < n && !(mask.on && left_out(mask, t.cells(threadIdx.x), s.C))) {
        face_flux<R, FK, ORDER, FOLD>(t, threadIdx.x, f0 + threadIdx.x, s, q, rec, gamma, G,
                                          pr_ref);
    }
}

}  // namespace tg
