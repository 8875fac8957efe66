// Runs the device forms of gp_crmath.cuh on argument arrays: 0 acos, 1 sin, 2 cos,
// 3 the start value of acos_cr's inverse sine.
#include "../gpluto_dev_b200/csrc/gp_crmath.cuh"

__global__ void probe(const double* x, double* out, int n, int which) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  double s, c;
  if (which == 0) {
    out[i] = gpcr::acos_cr(x[i]);
  } else if (which == 3) {
    out[i] = (double)asinf((float)x[i]);
  } else {
    gpcr::sincos_cr(x[i], &s, &c);
    out[i] = which == 1 ? s : c;
  }
}

extern "C" int crmath_probe(const double* x, double* out, int n, int which) {
  probe<<<(n + 255) / 256, 256>>>(x, out, n, which);
  if (cudaGetLastError() != cudaSuccess) return 1;
  return cudaDeviceSynchronize() != cudaSuccess;
}
