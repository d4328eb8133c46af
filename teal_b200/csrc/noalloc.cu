// Residual norm of a device-resident derivative that allocates no device memory.
//
// tg_residual goes through a context (tg_ctx), whose creation allocates the state, the geometry and
// the partial-sum scratch with cudaMalloc. Some callers cannot allocate while they solve: a serving
// process that committed its whole HBM budget to state arenas up front, or a host loop that must not
// stall the device (cudaMalloc and cudaFree can synchronise it). tg_residual_noalloc serves them: the
// derivative, the volumes and the result are the caller's device buffers, and the partial sums go to
// a fixed array compiled into this library (one copy per device).
//
// The reduction is the same as the context path's (k_step_end: per piece of piece_cells(num_cells) cells,
// one block sums volume * r^2 per variable; one warp per variable sums the pieces and takes
// sqrt(sum / sum_volume)), with the same loop order, so both give the same bits.
#include <cuda_runtime.h>

#include <cmath>
#include <cstdint>
#include <mutex>

#include "../../include/teal_b200.h"
#include "common.cuh"

using namespace tg;

int tg_record_error(int code, const char *msg);  // sets tg_last_error (context.cu)

namespace {

constexpr int NA_BLOCK = BLOCK;         // threads per piece, as k_step_end
constexpr int NA_FINISH_BLOCK = 5 * 32; // a warp per variable
constexpr int NA_MAX_DEVICES = 64;

}  // namespace

// partial sums, [5][pieces]: at most PIECE_COUNT pieces (24 KiB) per device. Every slot the finishing kernel
// reads is written by the partial kernel of the same call, so nothing has to start at zero.
static __device__ __align__(256) double g_noalloc_partials[5 * PIECE_COUNT];

// one block per piece of `per` cells: partials[k][p] = sum over the piece of volume * r_k^2
__global__ void __launch_bounds__(NA_BLOCK) k_noalloc_residual_pieces(int C, int per, const double *__restrict__ deriv,
                                                                      const double *__restrict__ volume,
                                                                      double *__restrict__ partials)
{
    const int beg = blockIdx.x * per;
    const int end = min(C, beg + per);
    double t[6] = {0, 0, 0, 0, 0, DBL_MAX};
    for (int c = beg + threadIdx.x; c < end; c += NA_BLOCK) {
        double v = volume[c];
#pragma unroll
        for (int k = 0; k < 5; k++) {
            double r = deriv[(size_t)c * 5 + k];
            t[k] += v * (r * r);
        }
    }
    const double x = block_reduce6(t);
    if (threadIdx.x < 5) {
        partials[threadIdx.x * gridDim.x + blockIdx.x] = x;
    }
}

// one block, a warp per variable: residual[k] = sqrt(sum over pieces / sum_volume)
__global__ void __launch_bounds__(NA_FINISH_BLOCK) k_noalloc_residual_finish(int npieces,
                                                                             const double *__restrict__ partials,
                                                                             double sum_volume,
                                                                             double *__restrict__ residual)
{
    const int k = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const double t = sum_partials(partials + (size_t)k * npieces, npieces, lane);
    if (lane == 0) {
        residual[k] = sqrt(t / sum_volume);
    }
}

// Address of this device's scratch array, looked up once per device (with that device current)
// and kept for the life of the process. A cudaDeviceReset after that first lookup unloads the module
// holding the array, and the kept address would then be stale: resetting a device on which
// tg_residual_noalloc has run is not supported. Returns null after recording the error.
static double *noalloc_scratch(int *status)
{
    static std::mutex lock;
    static double *addr[NA_MAX_DEVICES] = {};
    int dev = -1;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) {
        *status = tg_record_error(TG_ERR_NO_DEVICE, cudaGetErrorString(e));
        return nullptr;
    }
    if (dev < 0 || dev >= NA_MAX_DEVICES) {
        *status = tg_record_error(TG_ERR_INVALID, "tg_residual_noalloc: device ordinal out of range");
        return nullptr;
    }
    std::lock_guard<std::mutex> g(lock);
    if (!addr[dev]) {
        double *p = nullptr;
        e = cudaGetSymbolAddress((void **)&p, g_noalloc_partials);
        if (e != cudaSuccess || !p) {
            *status = tg_record_error(TG_ERR_CUDA, e != cudaSuccess ? cudaGetErrorString(e)
                                                                     : "tg_residual_noalloc: null scratch address");
            return nullptr;
        }
        addr[dev] = p;
    }
    return addr[dev];
}

// a buffer the kernels may read or write: managed memory, or device memory of device `dev` (the
// current one: memory of another GPU would be a peer access the kernels are not set up for), 8-byte
// aligned
static bool device_buffer(const void *p, int dev)
{
    if (!p || ((uintptr_t)p & 7u)) {
        return false;
    }
    cudaPointerAttributes a;
    if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    if (a.type == cudaMemoryTypeManaged) {
        return true;
    }
    return a.type == cudaMemoryTypeDevice && a.device == dev;
}

extern "C" int tg_residual_noalloc(const double *derivative, const double *volume, int num_cells, double sum_volume,
                                   double *residual, void *stream)
{
    if (num_cells < 0 || num_cells > TG_NOALLOC_MAX_CELLS) {
        return tg_record_error(TG_ERR_INVALID,
                               "tg_residual_noalloc: num_cells must be in [0, TG_NOALLOC_MAX_CELLS = 67108864]; "
                               "use tg_residual through a context for larger meshes");
    }
    if (!(sum_volume > 0.0) || !std::isfinite(sum_volume)) {
        return tg_record_error(TG_ERR_INVALID, "tg_residual_noalloc: sum_volume must be finite and positive");
    }
    int dev = -1;
    cudaError_t de = cudaGetDevice(&dev);
    if (de != cudaSuccess) {
        return tg_record_error(TG_ERR_NO_DEVICE, cudaGetErrorString(de));
    }
    if (!device_buffer(residual, dev) ||
        (num_cells > 0 && (!device_buffer(derivative, dev) || !device_buffer(volume, dev)))) {
        return tg_record_error(TG_ERR_INVALID,
                               "tg_residual_noalloc: derivative, volume and residual must be 8-byte aligned "
                               "memory of the current device (or managed memory)");
    }
    int status = TG_OK;
    double *partials = noalloc_scratch(&status);
    if (!partials) {
        return status;
    }
    cudaStream_t s = (cudaStream_t)stream;
    const int per = piece_cells(num_cells);
    const int npieces = (int)(((long)num_cells + per - 1) / per);
    if (npieces > 0) {
        k_noalloc_residual_pieces<<<npieces, NA_BLOCK, 0, s>>>(num_cells, per, derivative, volume, partials);
    }
    k_noalloc_residual_finish<<<1, NA_FINISH_BLOCK, 0, s>>>(npieces, partials, sum_volume, residual);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) {
        return tg_record_error(TG_ERR_CUDA, cudaGetErrorString(e));
    }
    return TG_OK;
}
