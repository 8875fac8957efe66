// Runs gp_exact.cuh on argument arrays beside the language's operators.
#include "../gpluto_dev_b200/csrc/gp_exact.cuh"

__global__ void probe(const double* a, const double* b, double* out, double* ref, int* bad,
                      int n, int op) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  gp::FastArith f;
  if (op == 0) {
    out[i] = f.div(a[i], b[i]);
    ref[i] = a[i] / b[i];
  } else if (op == 1) {
    out[i] = f.inv(b[i]);
    ref[i] = 1.0 / b[i];
  } else if (op == 2) {
    out[i] = f.root(a[i]);
    ref[i] = sqrt(a[i]);
  } else if (op == 3) {
    out[i] = f.quot_pos(a[i], b[i], f.inv_pos(b[i]));
    ref[i] = a[i] / b[i];
  } else if (op == 5) {
    out[i] = f.div_any(a[i], b[i]);
    ref[i] = a[i] / b[i];
  } else if (op == 6) {  // 1 - b y0 of the reciprocal's seed, 1 - a y0^2 of the root's
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(b[i]));
    out[i] = __fma_rn(-b[i], y, 1.0);
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(a[i]));
    ref[i] = __fma_rn(-a[i], __dmul_rn(y, y), 1.0);
  } else {
    out[i] = gp::fixed_quot(a[i], b[i], gp::fixed_inv(b[i]));
    ref[i] = a[i] / b[i];
  }
  bad[i] = f.bad;
}

extern "C" int exact_probe(const double* a, const double* b, double* out, double* ref, int* bad,
                           int n, int op) {
  probe<<<(n + 255) / 256, 256>>>(a, b, out, ref, bad, n, op);
  if (cudaGetLastError() != cudaSuccess) return 1;
  return cudaDeviceSynchronize() != cudaSuccess;
}
