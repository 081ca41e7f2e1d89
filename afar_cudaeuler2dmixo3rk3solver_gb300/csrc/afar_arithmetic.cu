// afar_debug_arithmetic: the FP64 arithmetic that the kernels do off the FP64 pipe (afar_policy.cuh), one
// function at a time over arrays, for tests against IEEE arithmetic and error bounds.
#include <cuda_runtime.h>

#include "afar_internal.h"
#include "afar_policy.cuh"

namespace {

using namespace afar;

__global__ void k_arithmetic(const int op, const int n, const double* a, const double* b, double* out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double x = a[i], y = b[i];
  double r = 0.0;
  switch (op) {
    case AFAR_ARITH_RCP: r = rcp64(x); break;
    case AFAR_ARITH_RSQRT: r = rsq64(x); break;
    case AFAR_ARITH_DIV: r = div64(x, y); break;
    case AFAR_ARITH_TO_FLOAT: r = to_float(x); break;
    case AFAR_ARITH_TO_DOUBLE: r = to_double((float)x); break;
    case AFAR_ARITH_HALF: r = half64(x); break;
    case AFAR_ARITH_BLEND_FIRST: r = blend64(true, false, x, y); break;
    case AFAR_ARITH_BLEND_SECOND: r = blend64(false, true, x, y); break;
    case AFAR_ARITH_MAX: r = dmax_(x, y); break;
    case AFAR_ARITH_MIN: r = dmin_(x, y); break;
    case AFAR_ARITH_TOP_FLOAT: r = top_float(x); break;
    case AFAR_ARITH_COMPARE:  // bits: x > 0, x <= 0, |x| < y, |x| >= y, NaN
      r = gt_zero(x) + 2 * le_zero(x) + 4 * abs_lt(x, y) + 8 * abs_ge(x, y) + 16 * dnan_(x);
      break;
  }
  out[i] = r;
}

struct Buffer {
  double* p = nullptr;
  ~Buffer() { cudaFree(p); }
};

}  // namespace

extern "C" afar_status afar_debug_arithmetic(int device, int op, int n, const double* a, const double* b, double* out) {
  if (op < AFAR_ARITH_RCP || op > AFAR_ARITH_COMPARE || n < 0 || !a || !b || !out) {
    set_error("afar_debug_arithmetic: unknown operation, negative size or null array");
    return AFAR_ERR_ARGUMENT;
  }
  if (n == 0) return AFAR_OK;
  Buffer d;
  cudaError_t e = cudaSetDevice(device);
  if (e == cudaSuccess) e = cudaMalloc(&d.p, 3 * sizeof(double) * (size_t)n);
  if (e == cudaSuccess) e = cudaMemcpy(d.p, a, sizeof(double) * (size_t)n, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemcpy(d.p + n, b, sizeof(double) * (size_t)n, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) {
    k_arithmetic<<<(n + 255) / 256, 256>>>(op, n, d.p, d.p + n, d.p + 2 * (size_t)n);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaMemcpy(out, d.p + 2 * (size_t)n, sizeof(double) * (size_t)n, cudaMemcpyDeviceToHost);
  if (e != cudaSuccess) {
    set_error("afar_debug_arithmetic failed: %s", cudaGetErrorString(e));
    return AFAR_ERR_CUDA;
  }
  return AFAR_OK;
}
