// lbm_io.cu -- FP64 host arrays on their way in: the conversion to the FP32
// device arrays, and the checks of the values, on the device.
//
// The caller's array is copied as it is (a pageable copy runs at 16 GB/s here)
// and narrowed by a kernel bound by memory: on the host one thread took 1 to 2
// ns per value, and helper threads wait for their turn while the caller's own
// thread pool spins.  614 400 cells: set_design 1.06 -> 0.4 ms.
#include "lbm_device.cuh"

namespace lbm {
namespace {

// out = in in FP32; with `unit` a value outside [0, 1] (or NaN) sets *bad.
__global__ void __launch_bounds__(BLOCK) k_narrow(const double* __restrict__ in, float* __restrict__ out, int64_t n,
                                                  int unit, int* bad) {
    bool off = false;
    for (int64_t i = (int64_t)blockIdx.x * BLOCK + threadIdx.x; i < n; i += (int64_t)gridDim.x * BLOCK) {
        const double v = in[i];
        off = off || !(v >= 0.0 && v <= 1.0);
        out[i] = (float)v;
    }
    if (unit && off) atomicOr(bad, 1);
}

// f[cell][q] -> planes g[q][cell] = f - w_q (plane stride n), k cells.  A block
// reads a contiguous run of values and writes coalesced planes through shared
// memory (Q is odd: no bank conflicts).  A non-finite value in a solid cell
// sets *solid_nonfinite.
struct Weights {
    double w[27];
};
template <int Q>
__global__ void __launch_bounds__(BLOCK) k_cells_to_planes(const double* __restrict__ f, float* __restrict__ g, int64_t n,
                                                           int64_t k, Weights W, const uint8_t* __restrict__ cls,
                                                           int* solid_nonfinite) {
    constexpr int CELLS = BLOCK;
    __shared__ float sh[CELLS * Q];
    bool bad = false;
    for (int64_t c0 = (int64_t)blockIdx.x * CELLS; c0 < k; c0 += (int64_t)gridDim.x * CELLS) {
        const int cells = (int)(k - c0 < CELLS ? k - c0 : CELLS);
        __syncthreads();
        for (int i = threadIdx.x; i < cells * Q; i += BLOCK) {
            const double v = f[c0 * Q + i];
            const int c = i / Q;
            sh[i] = (float)(v - W.w[i - c * Q]);
            if (!isfinite(v) && cls[c0 + c] == 0) bad = true;
        }
        __syncthreads();
        if ((int)threadIdx.x < cells)
#pragma unroll
            for (int q = 0; q < Q; ++q) g[(int64_t)q * n + c0 + threadIdx.x] = sh[threadIdx.x * Q + q];
    }
    if (bad) atomicOr(solid_nonfinite, 1);
}

int io_grid(int64_t n) { return blocks_for(n, 148 * 8); }

}  // namespace

cudaError_t launch_narrow(const double* in, float* out, int64_t n, int unit, int* bad, cudaStream_t s) {
    if (n <= 0) return cudaSuccess;
    k_narrow<<<io_grid(n), BLOCK, 0, s>>>(in, out, n, unit, bad);
    return cudaGetLastError();
}

cudaError_t launch_cells_to_planes(int Q, const double* f, float* g, int64_t n, int64_t k, const double* w,
                                   const uint8_t* cls, int* solid_nonfinite, cudaStream_t s) {
    if (k <= 0) return cudaSuccess;
    Weights W{};
    for (int q = 0; q < Q; ++q) W.w[q] = w[q];
    if (Q == 19) k_cells_to_planes<19><<<io_grid(k), BLOCK, 0, s>>>(f, g, n, k, W, cls, solid_nonfinite);
    else k_cells_to_planes<27><<<io_grid(k), BLOCK, 0, s>>>(f, g, n, k, W, cls, solid_nonfinite);
    return cudaGetLastError();
}

}  // namespace lbm
