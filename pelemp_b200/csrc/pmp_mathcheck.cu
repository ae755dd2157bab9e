// pmp_mathcheck.cu -- pmp_debug_math: the FP64 kernels' branch-free functions
// (MathFast) beside the plain ones (MathPlain) on given arguments.
#include <cuda_runtime.h>

#include "../../include/pmp_spray.h"
#include "phys/math_fast64.cuh"

namespace {

template <class Math>
__device__ double eval(Math& M, int fn, double x, double y)
{
  double a = 0., b = 0.;
  switch (fn) {
    case 0:
      return M.exp(x);
    case 1:
      return M.log(x);
    case 2:
      return M.pow(x, y);
    case 3:
      return M.cbrt(x);
    case 4:
      M.log1p_pow07(x, a, b);
      return a;
    case 5:
      M.log1p_pow07(x, a, b);
      return b;
    case 6:
      return M.div(x, y);
    case 7:
      return M.inv(x);
    case 8:
      return M.div(x, M.divisor_near1(y));
    default:
      return M.divk(x, y, 1. / y);
  }
}

__global__ void __launch_bounds__(256) k_math(int fn, const double* x, const double* y, long long n, double* fast, double* plain, int* odd)
{
  pmp::stage_math_tables();
  __syncthreads();
  for (long long i = blockIdx.x * 256LL + threadIdx.x; i < n; i += gridDim.x * 256LL) {
    pmp::MathFast F;
    pmp::MathPlain P;
    fast[i] = eval(F, fn, x[i], y[i]);
    plain[i] = eval(P, fn, x[i], y[i]);
    odd[i] = F.odd ? 1 : 0;
  }
}

}  // namespace

extern "C" int pmp_debug_math(int fn, const double* x, const double* y, long long n, double* fast, double* plain, int* odd)
{
  if (fn < 0 || fn > 9 || !x || !y || n < 1 || !fast || !plain || !odd) {
    return PMP_ERR_INVALID;
  }
  double* d = nullptr;
  const size_t b = sizeof(double) * (size_t)n;
  if (cudaMalloc(&d, 4 * b + sizeof(int) * (size_t)n) != cudaSuccess) {
    return PMP_ERR_CUDA;
  }
  int* o = reinterpret_cast<int*>(d + 4 * n);
  bool ok = cudaMemcpy(d, x, b, cudaMemcpyHostToDevice) == cudaSuccess &&
            cudaMemcpy(d + n, y, b, cudaMemcpyHostToDevice) == cudaSuccess;
  k_math<<<1184, 256>>>(fn, d, d + n, n, d + 2 * n, d + 3 * n, o);
  ok = ok && cudaMemcpy(fast, d + 2 * n, b, cudaMemcpyDeviceToHost) == cudaSuccess &&
       cudaMemcpy(plain, d + 3 * n, b, cudaMemcpyDeviceToHost) == cudaSuccess &&
       cudaMemcpy(odd, o, sizeof(int) * (size_t)n, cudaMemcpyDeviceToHost) == cudaSuccess;
  cudaFree(d);
  return ok ? PMP_OK : PMP_ERR_CUDA;
}
