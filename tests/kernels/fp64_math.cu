// fp64_math.cu -- the FP64 passes' own 1/a, 1/sqrt(a), sqrt(a) and exp(x) beside CUDA's, for the
// tests: run(what, n, in, out), host arrays.
#include <cuda_runtime.h>

#include "psim_device.cuh"
#include "psim_exp.cuh"

namespace {

enum { RCP, RCP_CUDA, RSQRT, RSQRT_CUDA, EXP, EXP_CUDA, SQRT };

__global__ void eval(int what, int n, const double* in, double* out, const double2* e2) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double a = in[i];
    switch (what) {
    case RCP: out[i] = psim::rcp64(a); break;
    case RCP_CUDA: out[i] = 1.0 / a; break;
    case RSQRT: out[i] = psim::rsqrt64(a); break;
    case RSQRT_CUDA: out[i] = 1.0 / sqrt(a); break;
    case EXP: out[i] = psim::exp_table(a, e2); break;
    case EXP_CUDA: out[i] = exp(a); break;
    case SQRT: out[i] = psim::sqrt64(a, psim::rsqrt64(a)); break;
    }
}

}  // namespace

extern "C" int run(int what, int n, const double* in, double* out) {
    double *a = nullptr, *b = nullptr;
    double2 e2[psim::kExpTable], *t = nullptr;
    psim::exp_table_values(e2);
    cudaError_t e = cudaMalloc(&a, 8 * (size_t)n);
    if (e == cudaSuccess) e = cudaMalloc(&b, 8 * (size_t)n);
    if (e == cudaSuccess) e = cudaMalloc(&t, sizeof e2);
    if (e == cudaSuccess) e = cudaMemcpy(a, in, 8 * (size_t)n, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemcpy(t, e2, sizeof e2, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) {
        eval<<<(n + 255) / 256, 256>>>(what, n, a, b, t);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpy(out, b, 8 * (size_t)n, cudaMemcpyDeviceToHost);
    cudaFree(a);
    cudaFree(b);
    cudaFree(t);
    return (int)e;
}
