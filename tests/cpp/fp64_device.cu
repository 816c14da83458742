// The FP64 path's arithmetic on the device, on arrays: reciprocals, quotients
// and roots from the hardware's seeds, the limiter's switch from its table,
// the limiter in pairs of floats.  Compiled like the kernels that use it.
#include <cuda_runtime.h>

#include "limiter_pair.cuh"
#include "physics_fp64.cuh"
#include "step_body_fp64.cuh"

using namespace splash;
using namespace splash::f64;

namespace {
enum Op : int { kRecip = 0, kDivide = 1, kRoot = 2, kRatio = 3, kSwitch = 4, kLimiter = 5 };

// in: up to 3 planes of n; out: up to 3 planes of n
__global__ void apply(int op, int n, const double* in, double p0, double p1, double* out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const size_t N = n;
  const double a = in[i], b = in[N + i], c = in[2 * N + i];
  double r[3] = {0.0, 0.0, 0.0};
  if (op == kRecip) {
    r[0] = recip(a);
  } else if (op == kDivide) {
    r[0] = divide(a, b);
  } else if (op == kRoot) {
    r[0] = root_pair(a, r[1]);
  } else if (op == kRatio) {
    r[0] = slope_ratio(b, a);
  } else if (op == kSwitch) {
    r[0] = switch_pos(a);
  } else if (op == kLimiter) {  // dp, num, nu; eta_p, sbs: in pairs, in FP64, 1 where pairs serve
    r[2] = limiter_pair(a, b, a - b, pair_line(p0, p1, c), r[0]) ? 1.0 : 0.0;
    const double ts = (1 + c) / 3;
    r[1] = limiter_field(b / a, LimiterLine<double>{p0, p1 / c, ts, 1 - ts});
  }
  for (int k = 0; k < 3; ++k) out[k * N + i] = r[k];
}
}  // namespace

// 0, or the CUDA error
extern "C" int run(int op, int n, const double* in, double p0, double p1, double* out) {
  double *d_in = nullptr, *d_out = nullptr;
  const size_t bytes = 3 * (size_t)n * sizeof(double);
  cudaError_t e = cudaMalloc(&d_in, bytes);
  if (e == cudaSuccess) e = cudaMalloc(&d_out, bytes);
  if (e == cudaSuccess) e = cudaMemcpy(d_in, in, bytes, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) {
    apply<<<(n + 255) / 256, 256>>>(op, n, d_in, p0, p1, d_out);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaMemcpy(out, d_out, bytes, cudaMemcpyDeviceToHost);
  cudaFree(d_in);
  cudaFree(d_out);
  return (int)e;
}
