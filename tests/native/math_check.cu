// The scalar helpers of the step kernels (contracted variant) evaluated for arrays of arguments.
#include "../../woo_gb300/csrc/wdem_math.cuh"
using namespace wdem::contracted;
__global__ void k_eval(int what, const double* x, const double* y, double* out, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double a = x[i], b = y[i];
  double r = 0;
  switch (what) {
    case 0: r = recipFast(a); break;
    case 1: r = rsqrtFast(a); break;
    case 2: r = sqrtRefined(a); break;
    case 3: r = halfOf(a); break;
    case 4: r = twice(a); break;
    case 5: r = plusZero(a); break;
    case 6: r = flipSign(a); break;
    case 7: r = greaterBits(a, b) ? 1. : 0.; break;
    case 8: r = belowHi(a, 1e-8) ? 1. : 0.; break;
    case 9: r = pick(i & 1, a, b); break;
    case 10: r = 1.0 / a; break;
    case 11: r = rsqrt(a); break;
    case 12: r = sqrt(a); break;
  }
  out[i] = r;
}
extern "C" int math_eval(int what, const double* x, const double* y, double* out, int n) {
  double* d = nullptr;
  const size_t bytes = (size_t)n * sizeof(double);
  if (cudaMalloc((void**)&d, 3 * bytes) != cudaSuccess) return 1;
  cudaMemcpy(d, x, bytes, cudaMemcpyHostToDevice);
  cudaMemcpy(d + n, y, bytes, cudaMemcpyHostToDevice);
  k_eval<<<(n + 255) / 256, 256>>>(what, d, d + n, d + 2 * (size_t)n, n);
  cudaMemcpy(out, d + 2 * (size_t)n, bytes, cudaMemcpyDeviceToHost);
  cudaFree(d);
  return (int)cudaGetLastError();
}
