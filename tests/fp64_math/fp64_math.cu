// The functions of gbmd_fp64.cuh and CUDA's own, element by element.
#include "gbmd_fp64.cuh"

__global__ void k_math(int n, const double* x, int nr, double* r, double* y, double* r0, double* inv, double* sq,
                       double* rec, int* m, double* p) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  r[i] = gbmd::root<true>(x[i], y[i]);
  double unused;
  r0[i] = gbmd::root<false>(x[i], unused);
  inv[i] = gbmd::inverse(x[i]);
  sq[i] = sqrt(x[i]);
  rec[i] = 1.0 / x[i];
  m[i] = gbmd::r_knot_d(x[i], nr, p[i]);
}

extern "C" int fp64_math(int n, const double* x, int nr, double* r, double* y, double* r0, double* inv, double* sq,
                         double* rec, int* m, double* p) {
  k_math<<<(n + 127) / 128, 128>>>(n, x, nr, r, y, r0, inv, sq, rec, m, p);
  const cudaError_t e = cudaDeviceSynchronize();
  return (int)e;
}
