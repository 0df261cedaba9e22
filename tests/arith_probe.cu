// The arithmetic of rp_arith.cuh on arrays, for tests/test_gpu_arithmetic.py.
#include <cuda_runtime.h>

#include "rp_arith.cuh"

using namespace rp;

__global__ void k_probe(int op, size_t n, const double* a, const double* b, double* out) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    double r = 0.0, s;
    switch (op) {
      case 0: r = sqrt_rn(a[i]); break;
      case 1: s = sqrt_rn(a[i], r); break;
      case 2: s = sqrt_rn(a[i], r); r = s; break;
      case 3: r = div_rn(a[i], b[i]); break;
      case 4: r = div_rn(vmk(a[i], 0.0, -a[i]), b[i]).x; break;
      case 5: r = div_rn(vmk(-0.0, a[i], a[i]), b[i]).z; break;
      case 6: r = __longlong_as_double((long long)__float_as_uint(d2f_exact(a[i]))); break;
      case 7: r = f2d_exact(__uint_as_float((uint32_t)__double_as_longlong(a[i]))); break;
      case 8: r = less_nn(a[i], b[i]) ? 1.0 : 0.0; break;
      case 9: r = not_positive(a[i]) ? 1.0 : 0.0; break;
      case 10: r = relu(a[i]); break;
      case 11: r = finite_bits(a[i]) ? 1.0 : 0.0; break;
      case 12: r = plus_zero(a[i]); break;
      case 13: r = div_near(a[i], b[i]); break;
    }
    out[i] = r;
  }
}

extern "C" int probe(int op, size_t n, const double* a, const double* b, double* out) {
  double *da = nullptr, *db = nullptr, *dr = nullptr;
  const size_t bytes = n * sizeof(double);
  cudaError_t e = cudaMalloc(&da, bytes);
  if (e == cudaSuccess) e = cudaMalloc(&db, bytes);
  if (e == cudaSuccess) e = cudaMalloc(&dr, bytes);
  if (e == cudaSuccess) e = cudaMemcpy(da, a, bytes, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemcpy(db, b, bytes, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) {
    k_probe<<<608, 256>>>(op, n, da, db, dr);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaMemcpy(out, dr, bytes, cudaMemcpyDeviceToHost);
  cudaFree(da);
  cudaFree(db);
  cudaFree(dr);
  return (int)e;
}
