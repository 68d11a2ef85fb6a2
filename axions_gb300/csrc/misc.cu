// Deterministic reduction of per-block diagnostic partials, the
// double <-> float conversions of the FP32 path, and lat_dtrig_eval (the FP64
// step's sine and cosine on given arguments, for checks).
#include <string>

#include "dtrig.cuh"
#include "lattice_handle.hpp"

namespace lat {

namespace {

// Sums of (energy, |G|) pairs: every block takes `per` of the n pairs (`step`
// pairs apart), every thread a fixed strided subset of them with Neumaier
// compensation, then a fixed tree combines the threads.  The result does not
// depend on timing, only on n.  A block's sum goes to out[2*b*out_step].
constexpr int FIN_THREADS = 256;
constexpr int FIN_PER = 4096;  // pairs per block

__global__ void __launch_bounds__(FIN_THREADS) finalize_kernel(const double* partials, int n, int step, int per,
                                                               double* out, int out_step)
{
    chain_wait();
    __shared__ double se[FIN_THREADS], sg[FIN_THREADS];
    const int end = min(n, ((int)blockIdx.x + 1) * per);
    double e = 0, ce = 0, g = 0, cg = 0;
    for (int b = (int)blockIdx.x * per + (int)threadIdx.x; b < end; b += FIN_THREADS) {
        const double2 v = *reinterpret_cast<const double2*>(partials + 2 * (size_t)b * step);
        double t = e + v.x;
        ce += (fabs(e) >= fabs(v.x)) ? (e - t) + v.x : (v.x - t) + e;
        e = t;
        t = g + v.y;
        cg += (fabs(g) >= fabs(v.y)) ? (g - t) + v.y : (v.y - t) + g;
        g = t;
    }
    se[threadIdx.x] = e + ce;
    sg[threadIdx.x] = g + cg;
    __syncthreads();  // also: every pair of the block has been read before one is overwritten below
    for (int w = FIN_THREADS / 2; w > 0; w >>= 1) {
        if ((int)threadIdx.x < w) {
            se[threadIdx.x] += se[threadIdx.x + w];
            sg[threadIdx.x] += sg[threadIdx.x + w];
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        out[2 * (size_t)blockIdx.x * out_step] = se[0];
        out[2 * (size_t)blockIdx.x * out_step + 1] = sg[0];
    }
}

__global__ void d2f_kernel(const double* __restrict__ in, float* __restrict__ out, int64_t n)
{
    for (int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; q < n; q += (int64_t)gridDim.x * blockDim.x)
        out[q] = (float)in[q];
}

__global__ void f2d_kernel(const float* __restrict__ in, double* __restrict__ out, int64_t n)
{
    for (int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; q < n; q += (int64_t)gridDim.x * blockDim.x)
        out[q] = (double)in[q];
}

// the FP64 step's dsin/dsincos and CUDA's sin/cos on the same arguments
__global__ void dtrig_kernel(const double* __restrict__ x, int64_t n, double* __restrict__ out)
{
    for (int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; q < n; q += (int64_t)gridDim.x * blockDim.x) {
        const double v = x[q];
        double s, c;
        dsincos(v, &s, &c);
        out[q] = dsin(v);
        out[n + q] = s;
        out[2 * n + q] = c;
        out[3 * n + q] = ::sin(v);
        out[4 * n + q] = ::cos(v);
    }
}

inline unsigned grid_for(int64_t n)
{
    int64_t b = (n + 255) / 256;
    if (b > 152 * 32) b = 152 * 32;
    return (unsigned)(b < 1 ? 1 : b);
}

}  // namespace

// One block up to FIN_PER pairs; above, blocks of FIN_PER pairs leave their sum
// in their first pair, until one block's worth is left.  A single block walked
// all of a large lattice's pairs before: 0.90 ms for the 221,184 of a 384^3
// step, as much as 1/20 of the step itself; 42 us at 128^3.
cudaError_t launch_finalize(double* partials, int nblocks, double* out, cudaStream_t st, int* launches)
{
    int n = nblocks, step = 1;
    *launches = 1;
    while (n > FIN_PER) {
        const int blocks = (n + FIN_PER - 1) / FIN_PER;
        const cudaError_t e = launch_chained(finalize_kernel, blocks, FIN_THREADS, 0, st, partials, n, step, FIN_PER, partials,
                                             step * FIN_PER);
        if (e != cudaSuccess) return e;
        ++*launches;
        n = blocks;
        step *= FIN_PER;
    }
    return launch_chained(finalize_kernel, 1, FIN_THREADS, 0, st, partials, n, step, FIN_PER, out, 1);
}

cudaError_t launch_d2f(const double* in, float* out, int64_t n, cudaStream_t st)
{
    d2f_kernel<<<grid_for(n), 256, 0, st>>>(in, out, n);
    return cudaGetLastError();
}

cudaError_t launch_f2d(const float* in, double* out, int64_t n, cudaStream_t st)
{
    f2d_kernel<<<grid_for(n), 256, 0, st>>>(in, out, n);
    return cudaGetLastError();
}

}  // namespace lat

using namespace lat;

extern "C" int lat_dtrig_eval(const double* x, int64_t n, double* out)
{
    if (!x || !out || n < 0 || n > ((int64_t)1 << 26)) {
        set_error("lat_dtrig_eval: null pointer or n outside [0, 2^26]");
        return LAT_ERR_INVALID;
    }
    if (n == 0) return LAT_OK;
    double* d = nullptr;
    cudaError_t e = cudaMalloc((void**)&d, sizeof(double) * 6 * (size_t)n);
    if (e == cudaSuccess) e = cudaMemcpy(d, x, sizeof(double) * (size_t)n, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) {
        dtrig_kernel<<<grid_for(n), 256>>>(d, n, d + n);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpy(out, d + n, sizeof(double) * 5 * (size_t)n, cudaMemcpyDeviceToHost);
    cudaFree(d);
    if (e != cudaSuccess) {
        set_error(std::string("lat_dtrig_eval: ") + cudaGetErrorString(e));
        return LAT_ERR_CUDA;
    }
    return LAT_OK;
}
