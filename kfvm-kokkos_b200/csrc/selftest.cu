// selftest.cu -- the device arithmetic of physics.cuh evaluated on the caller's arrays, so
// that its own error bounds and its special cases can be tested (no reference counterpart).
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "kernels.cuh"
#include "launch.h"

namespace kfvm {

__global__ void __launch_bounds__(256)
    math_probe_kernel(int fn, int64_t n, const double *__restrict__ in, double *__restrict__ out) {
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < n; t += (int64_t)gridDim.x * blockDim.x) {
    const double a = in[t], b = in[n + t], c = in[2 * n + t];
    out[t] = fn == KFVM_SELFTEST_SQRT ? sqrt_nr(a)
             : fn == KFVM_SELFTEST_ONE_MINUS_POW ? one_minus_pow(a, b, c)
                                                 : Eos<EQ_HYDRO>::weno_power64(a, b);
  }
}

// states and flux [v][n]
template <int EQ>
__global__ void __launch_bounds__(128)
    flux_probe_kernel(int rs, double gamma, double ch, int dir, int64_t n, const double *__restrict__ in,
                      double *__restrict__ out) {
  constexpr int NV = Eos<EQ>::NV;
  const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (t >= n) return;
  double uL[NV], uR[NV], F[NV];
#pragma unroll
  for (int v = 0; v < NV; v++) {
    uL[v] = in[v * n + t];
    uR[v] = in[(NV + v) * n + t];
  }
  const double s = Eos<EQ>::solve(rs, gamma, ch, dir, uL, uR, F);
#pragma unroll
  for (int v = 0; v < NV; v++) out[v * n + t] = F[v];
  out[NV * n + t] = s;
}

cudaError_t launch_math_probe(int fn, int64_t n, const double *in, double *out, cudaStream_t s) {
  math_probe_kernel<<<(unsigned)std::min<int64_t>((n + 255) / 256, 148 * 8), 256, 0, s>>>(fn, n, in, out);
  return cudaGetLastError();
}

cudaError_t launch_flux_probe(int eq, int rs, double gamma, double ch, int dir, int64_t n, const double *in,
                              double *out, cudaStream_t s) {
  const unsigned blocks = (unsigned)((n + 127) / 128);
  if (eq == EQ_HYDRO || eq == EQ_NS) flux_probe_kernel<EQ_HYDRO><<<blocks, 128, 0, s>>>(rs, gamma, ch, dir, n, in, out);
  else if (eq == EQ_GLM) flux_probe_kernel<EQ_GLM><<<blocks, 128, 0, s>>>(rs, gamma, ch, dir, n, in, out);
  else if (eq == EQ_SR) flux_probe_kernel<EQ_SR><<<blocks, 128, 0, s>>>(rs, gamma, ch, dir, n, in, out);
  else return cudaErrorInvalidValue;
  return cudaGetLastError();
}

}  // namespace kfvm
