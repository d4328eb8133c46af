// Kernels of the implicit Euler step with a Jacobian-free Newton-GMRES solve
// (src/simulation/advance.c:119-195, src/simulation/gmres.c:12-149), for every instance of an
// arena at once. Vectors are the conserved state of the inner cells, [5][C] over the arena; each
// instance has its own scalars (norms, step, finite-difference scale, Hessenberg matrix, Givens
// rotations, right-hand side, coefficients) and its own Newton / Arnoldi progress, so instances
// converge independently: a finished instance is masked out of the vector updates. Dot products
// and norms are per-piece partial sums, then per-instance sums in piece order: deterministic, and
// the same bits for an instance alone or in a batch.
#pragma once

#include "kernels.cuh"

namespace tg {

// scalar slots of an instance's block in the device scalar array
enum GmresScalar {
    GS_NORM = 0,       // Newton residual norm
    GS_FD_SCALE = 1,   // finite-difference scale
    GS_STEP = 2,       // time step
    GS_KTOL = 3,       // Krylov tolerance * norm
    GS_TOL_NORM = 4,   // Newton tolerance * first norm
    GS_HEAD = 8        // H [(dim+1) x dim], cs [dim], sn [dim], rhs [dim+1], coef [dim], G [dim x dim]
};

// per-instance flags: Newton iterating, Arnoldi iterating, Krylov vectors used, Newton iterations
enum GmresFlag { GF_NEWTON = 0, GF_ARNOLDI = 1, GF_M = 2, GF_ITER = 3, GF_COUNT = 4 };

// device loop counters of the graph-driven solve: the Arnoldi column k, the Newton iterations of the
// current step, the instances that take part in the current Newton iteration and in the current
// Arnoldi column, and of these the ones that have finished it and the ones that go on
enum GmresControl {
    GC_K = 0,
    GC_N = 1,
    GC_IN_NEWTON = 2,
    GC_IN_ARNOLDI = 3,
    GC_DONE = 4,
    GC_GOING = 5,
    GC_COUNT = 6
};

// Newton iterations one implicit step may take on the device before it stops with ERR_LOOP_LIMIT
// (teal's own bound, 128 (cells + 1) per instance, advance.c:162, stays in force below it); the
// bound keeps every device loop of the step graph finite
constexpr int NEWTON_LOOP_LIMIT = 1000;

// threads of a block over one piece: one cell each in pieces of PIECE_CELLS, so that the vector being
// orthogonalised stays in registers
constexpr int KRYLOV_BLOCK = PIECE_CELLS;
// basis vectors per shared-memory accumulator tile, and loaded together
constexpr int KRYLOV_TILE = 64;
constexpr int KRYLOV_GROUP = 4;

struct GmresBatch {
    int dim;    // Krylov dimension
    int scn;    // doubles per instance block of `sc`
    int ninst;
    Segments seg;
    double *part;  // [2 dim + 1][pieces] partial sums
    double *sc;    // [ninst][scn]
    int *flag;     // [GF_COUNT][ninst]
    int *ctl;      // [GC_COUNT]

    __device__ __forceinline__ double *s(int i) const { return sc + (size_t)i * scn; }
    __device__ __forceinline__ double *H(int i, int r, int k) const { return s(i) + GS_HEAD + r * dim + k; }
    __device__ __forceinline__ double *cs(int i) const { return s(i) + GS_HEAD + (dim + 1) * dim; }
    __device__ __forceinline__ double *sn(int i) const { return cs(i) + dim; }
    __device__ __forceinline__ double *rhs(int i) const { return sn(i) + dim; }
    __device__ __forceinline__ double *coef(int i) const { return rhs(i) + dim + 1; }
    __device__ __forceinline__ double *G(int i, int r) const { return coef(i) + dim + r * dim; }
    __device__ __forceinline__ int &newton(int i) const { return flag[GF_NEWTON * ninst + i]; }
    __device__ __forceinline__ int &arnoldi(int i) const { return flag[GF_ARNOLDI * ninst + i]; }
    __device__ __forceinline__ int &m(int i) const { return flag[GF_M * ninst + i]; }
    __device__ __forceinline__ int &iter(int i) const { return flag[GF_ITER * ninst + i]; }
};

__host__ __device__ inline int gmres_scn(int dim)
{
    return GS_HEAD + (dim + 1) * dim + 4 * dim + 2 + dim * dim;
}

// One warp's sum of row v of the partial sums over the instance's pieces, in every lane
__device__ __forceinline__ double sum_pieces(const GmresBatch &gb, int inst, int v, int lane)
{
    const int beg = gb.seg.inst_piece_off[inst], end = gb.seg.inst_piece_off[inst + 1];
    return sum_partials(gb.part + (size_t)v * gb.seg.npieces + beg, end - beg, lane);
}

// An instance has finished the current Newton iteration or Arnoldi column and goes on or not. True in
// the thread that closes it for all instances (*going: the instances that go on). `in`: GC_IN_NEWTON or
// GC_IN_ARNOLDI. Called by one thread of the instance's last block.
__device__ __forceinline__ bool last_instance(const GmresBatch &gb, int in, bool goes_on, int *going)
{
    if (goes_on) {
        atomicAdd(gb.ctl + GC_GOING, 1);
    }
    __threadfence();
    if (atomicAdd(gb.ctl + GC_DONE, 1) != gb.ctl[in] - 1) {
        return false;
    }
    __threadfence();
    *going = atomicAdd(gb.ctl + GC_GOING, 0);
    gb.ctl[GC_GOING] = 0;
    gb.ctl[GC_DONE] = 0;
    gb.ctl[in] = *going;
    return true;
}

// start of a step, one block: Newton flag on for the active instances, steps copied; the Newton loop's
// condition off (the residual kernel turns it on when an instance iterates)
__global__ void __launch_bounds__(KRYLOV_BLOCK) k_newton_begin(GmresBatch gb, Steps st,
                                                               cudaGraphConditionalHandle h)
{
    __shared__ int n;
    if (threadIdx.x == 0) {
        n = 0;
    }
    __syncthreads();
    for (int i = threadIdx.x; i < gb.ninst; i += blockDim.x) {
        const int on = st.active[i] != 0;
        gb.newton(i) = on;
        gb.arnoldi(i) = 0;
        gb.m(i) = 0;
        gb.iter(i) = 0;
        if (on) {
            gb.s(i)[GS_STEP] = st.step[i];
            atomicAdd(&n, 1);
        }
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        gb.ctl[GC_N] = 0;
        gb.ctl[GC_IN_NEWTON] = n;
        gb.ctl[GC_DONE] = 0;
        gb.ctl[GC_GOING] = 0;
        cudaGraphSetConditional(h, 0u);
    }
}

// Newton residual of every iterating instance, its norms and the loop test.
//   first: r = -R step (advance.c:148-153), else r = U - U0 - R step (advance.c:176-181);
//   fd_scale = fd_rel max(1, |U|) / max(1, |r|) (advance.c:155-159, fd_rel = 1e-6 there), on the first
//   call of a step also the Newton target tol |r|;
//   loop test (advance.c:162-165): iterate while |r| > tol |r0| and within 128 (cells + 1) iterations;
//   a non-finite norm marks the instance failed;
//   an instance that iterates starts its GMRES cycle (gmres.c:68-83): rhs = (norm, 0, ...), Arnoldi on.
// 360 bytes a cell are read and written once; the rest is latency (a ticket and a sum over the pieces).
__global__ void __launch_bounds__(KRYLOV_BLOCK) k_newton_residual(int C, const double *__restrict__ U,
                                                                  const double *__restrict__ U0,
                                                                  const double *__restrict__ R, GmresBatch gb,
                                                                  Steps st, double fd_rel,
                                                                  double newton_tol, double krylov_tol, int first,
                                                                  double *__restrict__ r,
                                                                  cudaGraphConditionalHandle h)
{
    __shared__ double sh[KRYLOV_BLOCK / 32];
    let_next_start();
    wait_for_previous();
    U = after_wait(U);
    U0 = after_wait(U0);
    R = after_wait(R);
    const int beg = gb.seg.piece_beg[blockIdx.x], end = gb.seg.piece_beg[blockIdx.x + 1];
    const int inst = gb.seg.cell_inst[beg];
    if (!gb.newton(inst)) {
        return;
    }
    double *s = gb.s(inst);
    const double step = s[GS_STEP];
    double rr = 0, uu = 0;
    for (int c = beg + threadIdx.x; c < end; c += KRYLOV_BLOCK) {
#pragma unroll
        for (int v = 0; v < 5; v++) {
            const size_t k = (size_t)v * C + c;
            const double u = U[k];
            const double x = first ? -R[k] * step : (u - U0[k]) - (R[k] * step);
            r[k] = x;
            rr += x * x;
            uu += u * u;
        }
    }
    rr = block_sum<KRYLOV_BLOCK>(rr, sh);
    uu = block_sum<KRYLOV_BLOCK>(uu, sh);
    if (threadIdx.x == 0) {
        gb.part[blockIdx.x] = rr;
        gb.part[gb.seg.npieces + blockIdx.x] = uu;
    }
    if (!last_of_instance(gb.seg, inst) || threadIdx.x >= 32) {
        return;
    }
    const double norm = sqrt(sum_pieces(gb, inst, 0, threadIdx.x));
    const double cons = sqrt(sum_pieces(gb, inst, 1, threadIdx.x));
    if (threadIdx.x != 0) {
        return;
    }
    s[GS_NORM] = norm;
    s[GS_FD_SCALE] = fd_rel * fmax(1.0, cons) / fmax(1.0, norm);
    if (first) {
        s[GS_TOL_NORM] = newton_tol * norm;
    }
    bool on;
    if (!isfinite(norm)) {  // the instance stops (its residual follows as non-finite); the others go on
        atomicOr(st.error, ERR_NONFINITE);
        st.fail[inst] = 1;
        on = false;
    }
    else {
        const long max_iter = 128L * (gb.seg.inst_cell_off[inst + 1] - gb.seg.inst_cell_off[inst] + 1);
        on = norm > s[GS_TOL_NORM] && gb.iter(inst) < max_iter;
    }
    gb.newton(inst) = on;
    gb.arnoldi(inst) = on;  // |r| > tol |r0| >= 0
    gb.m(inst) = 0;
    if (on) {
        double *rhs = gb.rhs(inst);
        for (int k = 0; k <= gb.dim; k++) {
            rhs[k] = 0.0;
        }
        rhs[0] = norm;
        s[GS_KTOL] = krylov_tol * norm;
        gb.iter(inst) += 1;
    }
    int going;
    if (last_instance(gb, GC_IN_NEWTON, on, &going)) {
        const int n = first ? 0 : gb.ctl[GC_N] + 1;
        gb.ctl[GC_N] = n;
        if (going > 0 && n >= NEWTON_LOOP_LIMIT) {
            atomicOr(st.error, ERR_LOOP_LIMIT);
        }
        cudaGraphSetConditional(h, (going > 0 && n < NEWTON_LOOP_LIMIT) ? 1u : 0u);
    }
}

// U += delta, delta = sum of coef[j] V_j with j from m - 1 down to 0 (gmres.c:137-141), q = prim(U)
// (advance.c:168-173): the basis is read once, the increment is not stored
__global__ void k_newton_update(int C, int N, double *__restrict__ U, const double *__restrict__ V, GmresBatch gb,
                                double gamma, double *__restrict__ q)
{
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= C) {
        return;
    }
    const int i = gb.seg.cell_inst[c];
    if (!gb.newton(i)) {
        return;
    }
    const int m = gb.m(i);
    const double *coef = gb.coef(i);
    const size_t n = 5 * (size_t)C;
    double d[5] = {0, 0, 0, 0, 0};
#pragma unroll 2
    for (int j = m - 1; j >= 0; j--) {
        const double a = coef[j];
#pragma unroll
        for (int v = 0; v < 5; v++) {
            d[v] += a * V[(size_t)j * n + (size_t)v * C + c];
        }
    }
    Cons<double> u;
    u.rho = U[c] += d[0];
    u.m.x = U[C + c] += d[1];
    u.m.y = U[2 * (size_t)C + c] += d[2];
    u.m.z = U[3 * (size_t)C + c] += d[3];
    u.e = U[4 * (size_t)C + c] += d[4];
    store_prim(q, N, c, cons_to_prim(u, gamma));
}

// ---- device-driven loops ------------------------------------------------------------------------
//
// The implicit step runs from one CUDA graph whose Newton and Arnoldi loops are conditional WHILE
// nodes: the kernels below read the loop counters (GmresBatch::ctl) from device memory instead of
// taking them as launch arguments, and the last block of a body's last kernel sets the loop's
// condition, so no iteration waits for the host.

// start of an Arnoldi loop (one thread): column 0 of every instance that iterates
__global__ void k_arnoldi_enter(GmresBatch gb, cudaGraphConditionalHandle h)
{
    const int n = gb.ctl[GC_IN_NEWTON];
    gb.ctl[GC_K] = 0;
    gb.ctl[GC_IN_ARNOLDI] = n;
    cudaGraphSetConditional(h, n > 0 ? 1u : 0u);
}

// Krylov vector k, V_0 = -r / |r| or V_k = w / H[k][k-1] (gmres.c:75, :121-125), and the state it
// perturbs, q1 = prim(U + eps V_k) with eps = fd_scale / |V_k| (gmres.c:26-36): V_k has just been
// divided by its norm, so |V_k| is 1 to rounding and is not summed again (it scales a
// finite-difference step, whose own truncation error is some ten orders larger).
__global__ void k_krylov_vector(int C, int N, const double *__restrict__ U, const double *__restrict__ r,
                                const double *__restrict__ w, GmresBatch gb, double gamma, double *__restrict__ V,
                                double *__restrict__ q1)
{
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= C) {
        return;
    }
    const int i = gb.seg.cell_inst[c];
    const int k = gb.ctl[GC_K];
    if (!gb.arnoldi(i)) {
        return;
    }
    const double *x = (k == 0) ? r : w;
    const double norm = (k == 0) ? -gb.s(i)[GS_NORM] : *gb.H(i, k, k - 1);
    const double eps = gb.s(i)[GS_FD_SCALE];
    double *Vk = V + (size_t)k * 5 * (size_t)C;
    double u[5];
#pragma unroll
    for (int v = 0; v < 5; v++) {
        const size_t j = (size_t)v * C + c;
        const double y = x[j] / norm;
        Vk[j] = y;
        u[v] = U[j] + (eps * y);
    }
    store_prim(q1, N, c, cons_to_prim(Cons<double>{u[0], v3(u[1], u[2], u[3]), u[4]}, gamma));
}

// Sums of 8 values over the lanes of a warp in 9 exchanges (a butterfly that halves the values as it
// halves the lanes); lane l returns the sum of value l / 4.
__device__ __forceinline__ double warp_sum8(double (&a)[8], int lane)
{
#pragma unroll
    for (int o = 16, n = 4; o >= 4; o >>= 1, n >>= 1) {
        const bool hi = lane & o;
#pragma unroll
        for (int j = 0; j < 4; j++) {
            if (j < n) {
                const double send = hi ? a[j] : a[j + n], keep = hi ? a[j + n] : a[j];
                a[j] = keep + __shfl_xor_sync(0xffffffffu, send, o);
            }
        }
    }
    double t = a[0];
    t += __shfl_xor_sync(0xffffffffu, t, 2);
    t += __shfl_xor_sync(0xffffffffu, t, 1);
    return t;
}

// First pass of Arnoldi column k: w = V_k - step (R1 - R) / eps (gmres.c:41-46), t_i = V_i . w for
// i <= k and G_ki = V_i . V_k for i < k; the instance's last block then gets column k of H.
// Bound by the basis it reads (40 (k + 1) bytes a cell): w and V_k stay in registers, the loads of
// KRYLOV_GROUP basis vectors are in flight together and their 2 x KRYLOV_GROUP products are
// summed over the warp at once. Four blocks an SM (64 registers) hold all pieces of an instance at once:
// two implicit steps of 123 k cells 6.55 ms, 6.89 with three.
// GATHER: R1 is not read but summed here from the FP32 flux records (k_cell's sum): a launch and the round trip of
// R1 less per column; two implicit steps of six ramps 2.47 -> 2.39 ms. FP64 records (60 registers for a cell's
// six) gain nothing: 37 k cells 1.970 ms either way with spills at four blocks, 123 k cells 6.28 -> 6.89 at three.
template <bool GATHER>
__global__ void __launch_bounds__(KRYLOV_BLOCK, 4) k_arnoldi_dots(Sizes sz, const int *__restrict__ slot_face,
                                                                  const uint8_t *__restrict__ slot_cnt,
                                                                  const double *__restrict__ volume,
                                                                  const float *__restrict__ G, const double *__restrict__ V,
                                                                  const double *__restrict__ R1,
                                                                  const double *__restrict__ R, GmresBatch gb,
                                                                  double *__restrict__ w)
{
    constexpr int WARPS = KRYLOV_BLOCK / 32;
    __shared__ double acc[WARPS][2 * KRYLOV_TILE];
    let_next_start();
    wait_for_previous();
    G = after_wait(G);
    V = after_wait(V);
    R1 = after_wait(R1);
    R = after_wait(R);
    const int C = sz.C;
    const int beg = gb.seg.piece_beg[blockIdx.x], end = gb.seg.piece_beg[blockIdx.x + 1];
    const int inst = gb.seg.cell_inst[beg];
    if (!gb.arnoldi(inst)) {
        return;
    }
    const int k = gb.ctl[GC_K], dim = gb.dim;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const size_t n = 5 * (size_t)C;
    const double *s = gb.s(inst);
    const double eps = s[GS_FD_SCALE], step = s[GS_STEP];
    for (int i0 = 0; i0 <= k; i0 += KRYLOV_TILE) {
        const int ni = min(KRYLOV_TILE, k + 1 - i0);
        for (int i = lane; i < 2 * KRYLOV_TILE; i += 32) {
            acc[warp][i] = 0.0;
        }
        __syncwarp();
        // whole warps take part in every round: lanes past the end hold zeros
        for (int c0 = beg + 32 * warp; c0 < end; c0 += KRYLOV_BLOCK) {
            const int c = c0 + lane;
            const bool in = c < end;
            double x[5], vk[5], r1[5];
            if (GATHER && in && i0 == 0) {
                double acc[5];
                sum_fluxes(sz, slot_face, slot_cnt, G, c, acc);
                const double ivol = 1.0 / __ldg(volume + c);
#pragma unroll
                for (int v = 0; v < 5; v++) {
                    r1[v] = mul_rn(-acc[v], ivol);  // rounded as k_cell stores it
                }
            }
#pragma unroll
            for (int v = 0; v < 5; v++) {
                const size_t j = (size_t)v * C + c;
                x[v] = vk[v] = 0.0;
                if (in) {
                    vk[v] = V[(size_t)k * n + j];
                    if (i0 == 0) {
                        x[v] = vk[v] - ((step * ((GATHER ? r1[v] : R1[j]) - R[j])) / eps);
                        w[j] = x[v];
                    }
                    else {
                        x[v] = w[j];
                    }
                }
            }
            for (int i = 0; i < ni; i += KRYLOV_GROUP) {
                double a[2 * KRYLOV_GROUP];
#pragma unroll
                for (int g = 0; g < KRYLOV_GROUP; g++) {
                    double t = 0, u = 0;
                    if (in && i + g < ni) {
                        const double *Vi = V + (size_t)(i0 + i + g) * n + c;
#pragma unroll
                        for (int v = 0; v < 5; v++) {
                            const double y = Vi[(size_t)v * C];
                            t += y * x[v];
                            u += y * vk[v];
                        }
                    }
                    a[2 * g] = t;
                    a[2 * g + 1] = u;
                }
                const double t = warp_sum8(a, lane);
                if ((lane & 3) == 0) {
                    acc[warp][2 * i + (lane >> 2)] += t;
                }
                __syncwarp();
            }
        }
        __syncthreads();
        // part rows: t_i in row i, G_ki in row dim + i
        for (int i = threadIdx.x; i < 2 * ni; i += KRYLOV_BLOCK) {
            double t = 0;
#pragma unroll
            for (int q = 0; q < WARPS; q++) {
                t += acc[q][i];
            }
            const int row = i0 + (i >> 1);
            gb.part[(size_t)((i & 1) ? dim + row : row) * gb.seg.npieces + blockIdx.x] = t;
        }
        __syncthreads();
    }
    if (!last_of_instance(gb.seg, inst)) {
        return;
    }
    for (int i = warp; i < 2 * k + 1; i += WARPS) {
        const bool is_t = i <= k;
        const int row = is_t ? i : i - (k + 1);
        const double t = sum_pieces(gb, inst, is_t ? row : dim + row, lane);
        if (lane == 0) {
            *(is_t ? gb.H(inst, row, k) : gb.G(inst, k) + row) = t;
        }
    }
    __syncthreads();
    // h = (I + strictly lower G)^-1 t, column by column: h_j is final once all h_i, i < j, are subtracted
    for (int j = 0; j < k; j++) {
        const double hj = *(volatile double *)gb.H(inst, j, k);
        for (int i = j + 1 + threadIdx.x; i <= k; i += KRYLOV_BLOCK) {
            *gb.H(inst, i, k) -= gb.G(inst, i)[j] * hj;
        }
        __syncthreads();
    }
}

// Second pass of Arnoldi column k: w -= sum of H[i][k] V_i, |w|; the instance's last block then applies
// and extends the Givens rotations and the right-hand side (gmres.c:102-119); an instance that
// converged (or filled the basis) stops with m = k + 1 and its coefficients (gmres.c:128-136); the
// last instance sets the loop's condition. Bound by the basis it reads, as the first pass.
__global__ void __launch_bounds__(KRYLOV_BLOCK) k_arnoldi_update(int C, const double *__restrict__ V, GmresBatch gb,
                                                                 double *__restrict__ w,
                                                                 cudaGraphConditionalHandle h)
{
    __shared__ double sh[KRYLOV_BLOCK / 32];
    __shared__ int stop;
    let_next_start();
    wait_for_previous();
    V = after_wait(V);
    const int beg = gb.seg.piece_beg[blockIdx.x], end = gb.seg.piece_beg[blockIdx.x + 1];
    const int inst = gb.seg.cell_inst[beg];
    if (!gb.arnoldi(inst)) {
        return;
    }
    const int k = gb.ctl[GC_K], dim = gb.dim;
    const size_t n = 5 * (size_t)C;
    double t = 0;
    for (int c = beg + threadIdx.x; c < end; c += KRYLOV_BLOCK) {
        double x[5];
#pragma unroll
        for (int v = 0; v < 5; v++) {
            x[v] = w[(size_t)v * C + c];
        }
#pragma unroll 4
        for (int i = 0; i <= k; i++) {
            const double hi = *gb.H(inst, i, k);
            const double *Vi = V + (size_t)i * n + c;
#pragma unroll
            for (int v = 0; v < 5; v++) {
                x[v] -= hi * Vi[(size_t)v * C];
            }
        }
#pragma unroll
        for (int v = 0; v < 5; v++) {
            w[(size_t)v * C + c] = x[v];
            t += x[v] * x[v];
        }
    }
    t = block_sum<KRYLOV_BLOCK>(t, sh);
    if (threadIdx.x == 0) {
        gb.part[blockIdx.x] = t;
    }
    if (!last_of_instance(gb.seg, inst)) {
        return;
    }
    double *cs = gb.cs(inst), *sn = gb.sn(inst), *rhs = gb.rhs(inst), *coef = gb.coef(inst);
    if (threadIdx.x < 32) {
        const double norm = sqrt(sum_pieces(gb, inst, 0, threadIdx.x));
        if (threadIdx.x == 0) {
            *gb.H(inst, k + 1, k) = norm;
            double top = *gb.H(inst, 0, k);
#pragma unroll 4
            for (int r = 0; r < k; r++) {
                const double low = *gb.H(inst, r + 1, k);
                *gb.H(inst, r, k) = (cs[r] * top) + (sn[r] * low);
                top = (-sn[r] * top) + (cs[r] * low);
            }
            const double rot = sqrt((top * top) + (norm * norm));
            cs[k] = top / rot;
            sn[k] = norm / rot;
            *gb.H(inst, k, k) = rot;
            rhs[k + 1] = -sn[k] * rhs[k];
            rhs[k] = cs[k] * rhs[k];
            gb.m(inst) = k + 1;
            stop = fabs(rhs[k + 1]) < gb.s(inst)[GS_KTOL] || k + 1 >= dim;
        }
    }
    __syncthreads();
    if (stop) {
        // back substitution, column by column
        for (int i = threadIdx.x; i <= k; i += KRYLOV_BLOCK) {
            coef[i] = rhs[i];
        }
        __syncthreads();
        for (int j = k; j >= 0; j--) {
            if (threadIdx.x == 0) {
                coef[j] = coef[j] / *gb.H(inst, j, j);
            }
            __syncthreads();
            const double a = *(volatile double *)(coef + j);
            for (int i = threadIdx.x; i < j; i += KRYLOV_BLOCK) {
                coef[i] -= *gb.H(inst, i, j) * a;
            }
            __syncthreads();
        }
    }
    if (threadIdx.x == 0) {
        gb.arnoldi(inst) = !stop;
        int going;
        if (last_instance(gb, GC_IN_ARNOLDI, !stop, &going)) {
            gb.ctl[GC_K] = k + 1;
            cudaGraphSetConditional(h, (going > 0 && k + 1 < dim) ? 1u : 0u);
        }
    }
}

}  // namespace tg
