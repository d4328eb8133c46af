// Kernel launchers shared by the translation units. Face-flux kernels are instantiated per flux
// scheme in face_*.cu so the many template variants compile in parallel.
#pragma once

#include <cuda_runtime.h>

#include "face.cuh"

namespace tg {

// Launch of a kernel that waits for the one before it itself (wait_for_previous): it may start while that
// kernel drains. Steps of 513 k cells gain 0.7 % (ramp, 431 -> 428 us), of 111 k cells in 10 meshes 2 %,
// of 16 k cells 4 %, a residual of 2.4 k cells 14 %, implicit steps of six meshes 4 %.
template <typename... K, typename... A>
inline cudaError_t launch_next(void (*kernel)(K...), dim3 grid, dim3 block, cudaStream_t st, const A &...args)
{
    cudaLaunchAttribute attr = {};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.stream = st;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, K(args)...);
}

// The launchers below are local to each translation unit (unnamed namespace): the exact and the plain
// face translation units instantiate them with the same template arguments, and one shared
// definition would launch the other arithmetic's kernels.
namespace {

template <typename R, int FK, bool NS, int ORDER, bool FOLD>
inline void launch_face_v(bool staged, const FaceLaunch &a, const Geometry<R> &g, const R *rec, R *G, cudaStream_t st)
{
    constexpr bool X = kExact;
    if (a.s.hi <= a.s.lo) {
        return;
    }
    dim3 grid((a.s.hi - a.s.lo + FACE_BLOCK - 1) / FACE_BLOCK);
    const R gm = R(a.gamma), ig = R(1) / (gm - R(1)), mu = R(a.mu), pr = R(a.prandtl);
    PressureRefOf<R> pref{};
    if constexpr (sizeof(R) == sizeof(float)) {
        pref = a.pr_ref;
    }
    if constexpr (!NS) {
        if (staged) {
            launch_next(k_face_staged<R, FK, ORDER, FOLD, X>, grid, dim3(FACE_BLOCK), st, a.s, g, a.q, rec, gm, G,
                        a.err, pref, a.polls, a.mask);
            return;
        }
    }
    if (a.mask.on) {
        launch_next(k_face<R, FK, NS, ORDER, FOLD, X, true>, grid, dim3(FACE_BLOCK), st, a.s, g, a.q, rec, gm, ig, mu, pr, G,
                    pref, a.mask);
        return;
    }
    launch_next(k_face<R, FK, NS, ORDER, FOLD, X, false>, grid, dim3(FACE_BLOCK), st, a.s, g, a.q, rec, gm, ig, mu, pr, G, pref,
                a.mask);
}

// staged geometry (bulk copies into shared memory) or thread loads without a viscous flux (tuned.h)
template <int FK, typename R>
inline cudaError_t launch_face_r(bool ns, int order, bool fold, const FaceLaunch &a, cudaStream_t st)
{
    const Geometry<R> &g = *static_cast<const Geometry<R> *>(a.geom);
    const R *rec = static_cast<const R *>(a.rec);
    R *G = static_cast<R *>(a.G);
    if constexpr (!kExact) {
        if (a.side) {
            if (a.s.hi <= a.s.lo) {
                return cudaSuccess;
            }
            PressureRefOf<R> pref{};
            if constexpr (sizeof(R) == sizeof(float)) {
                pref = a.pr_ref;
            }
            const dim3 grid((a.s.hi - a.s.lo + SIDE_BLOCK - 1) / SIDE_BLOCK), block(SIDE_BLOCK);
            const R *side = static_cast<const R *>(a.side);
            if (a.mask.on) {
                return launch_next(k_face_sides<R, FK, true>, grid, block, st, a.s, g, a.q, side, rec, R(a.gamma), R(1) / (R(a.gamma) - R(1)), G, pref,
                                   a.mask);
            }
            return launch_next(k_face_sides<R, FK, false>, grid, block, st, a.s, g, a.q, side, rec, R(a.gamma), R(1) / (R(a.gamma) - R(1)), G, pref,
                               a.mask);
        }
    }
    const bool staged = !ns && TG_FACE_STAGED_EULER != 0;
    if (order == 1) {
        launch_face_v<R, FK, false, 1, true>(staged, a, g, rec, G, st);
    }
    else if (!ns) {
        if constexpr (kExact) {  // the other forms have side records
            launch_face_v<R, FK, false, 2, true>(staged, a, g, rec, G, st);
        }
        else {
            return cudaErrorInvalidValue;
        }
    }
    else if (fold) {
        launch_face_v<R, FK, true, 2, true>(staged, a, g, rec, G, st);
    }
    else {
        launch_face_v<R, FK, true, 2, false>(staged, a, g, rec, G, st);
    }
    return cudaGetLastError();
}

}  // namespace

// precision: 0 = FP64, 1 = FP32 flux path
template <int FK>
cudaError_t launch_face(int precision, bool ns, int order, bool fold, const FaceLaunch &a,
                        cudaStream_t st);

// face fluxes and cell updates in one launch (k_cell_fluxes); `a.side` must be set
template <int FK>
cudaError_t launch_cell_fluxes(int precision, const FaceLaunch &a, const CellLaunch &b, cudaStream_t st);

// FP64 with teal's exact arithmetic (face_*_exact.cu); with a viscous flux, `a.G` holds 2 x 5 F
// values (convective and viscous records)
template <int FK>
cudaError_t launch_face_exact(bool ns, int order, bool fold, const FaceLaunch &a, cudaStream_t st);

#define TG_INSTANTIATE_FACE(FK)                                                                 \
    template <>                                                                                 \
    cudaError_t launch_face<FK>(int precision, bool ns, int order, bool fold, const FaceLaunch &a, \
                                cudaStream_t st)                                                \
    {                                                                                           \
        if (precision == 0) {                                                                   \
            return launch_face_r<FK, double>(ns, order, fold, a, st);                           \
        }                                                                                       \
        return launch_face_r<FK, float>(ns, order, fold, a, st);                                \
    }                                                                                           \
    template <>                                                                                 \
    cudaError_t launch_cell_fluxes<FK>(int precision, const FaceLaunch &a, const CellLaunch &b, \
                                       cudaStream_t st)                                         \
    {                                                                                           \
        const dim3 grid((a.s.C + 31) / 32), block(SIDE_TILE);                                   \
        if (precision == 0) {                                                                   \
            return launch_next(k_cell_fluxes<double, FK>, grid, block, st, a,                   \
                               *static_cast<const Geometry<double> *>(a.geom), b);              \
        }                                                                                       \
        return launch_next(k_cell_fluxes<float, FK>, grid, block, st, a,                        \
                           *static_cast<const Geometry<float> *>(a.geom), b);                   \
    }

#define TG_INSTANTIATE_FACE_EXACT(FK)                                                              \
    static_assert(kExact, "face_*_exact.cu is compiled with TG_EXACT_TU=1");                       \
    template <>                                                                                 \
    cudaError_t launch_face_exact<FK>(bool ns, int order, bool fold, const FaceLaunch &a, cudaStream_t st) \
    {                                                                                           \
        return launch_face_r<FK, double>(ns, order, fold, a, st);                               \
    }

}  // namespace tg
