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
__global__ void k_quat(const double* c, double* out, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double* m = c + 9 * (size_t)i;
  const qd q = quatFromCols(mk(m[0], m[1], m[2]), mk(m[3], m[4], m[5]), mk(m[6], m[7], m[8]));
  out[4 * (size_t)i] = q.w; out[4 * (size_t)i + 1] = q.x; out[4 * (size_t)i + 2] = q.y; out[4 * (size_t)i + 3] = q.z;
}
// quaternions (4n) of n frames given by their columns (9n)
extern "C" int quat_eval(const double* c, double* out, int n) {
  double* d = nullptr;
  if (cudaMalloc((void**)&d, 13 * (size_t)n * sizeof(double)) != cudaSuccess) return 1;
  cudaMemcpy(d, c, 9 * (size_t)n * sizeof(double), cudaMemcpyHostToDevice);
  k_quat<<<(n + 255) / 256, 256>>>(d, d + 9 * (size_t)n, n);
  cudaMemcpy(out, d + 9 * (size_t)n, 4 * (size_t)n * sizeof(double), cudaMemcpyDeviceToHost);
  cudaFree(d);
  return (int)cudaGetLastError();
}
