// newton_rcp and Quotient<double> of dense_ops.cuh, element by element, for
// tests/test_gpu_reciprocals.py (device pointers; null on success).
#include "dense_ops.cuh"

using namespace hodlr;

__global__ void rcp_kernel(const double *x, int n, double *y, int *usual, double *division) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  y[i] = newton_rcp(x[i]);
  usual[i] = rcp_usual(x[i]);
  division[i] = 1.0 / x[i];
}

__global__ void quotient_kernel(const double *u, const double *x, int n, double *q, double *division) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  q[i] = Quotient<double>::by(u[i]).of(x[i]);
  division[i] = x[i] / u[i];
}

static const char *done() {
  cudaError_t e = cudaGetLastError();
  if (e == cudaSuccess) e = cudaDeviceSynchronize();
  return e == cudaSuccess ? nullptr : cudaGetErrorString(e);
}

extern "C" const char *reciprocals(const double *x, int n, double *y, int *usual, double *division) {
  rcp_kernel<<<(n + 255) / 256, 256>>>(x, n, y, usual, division);
  return done();
}

extern "C" const char *quotients(const double *u, const double *x, int n, double *q, double *division) {
  quotient_kernel<<<(n + 255) / 256, 256>>>(u, x, n, q, division);
  return done();
}
