// Scalar functions of the kernels, an element per thread.
#include "device_common.cuh"
#include "refine_tc.cu"

namespace {
__global__ void k_level_sum(int n, const long long* hs, const long long* ls, const int* e, double* out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) out[i] = gsk::level_sum(hs[i], ls[i], e[i]);
}
__global__ void k_f32_of(int n, const double* r, int h, float* out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) out[i] = gsk::f32_of(r[i], h);
}
// the floats with exponent field `ex` and every significand: number of differences from the rounded quotient
__global__ void k_rcp(int ex, int neg, unsigned long long* bad) {
  const unsigned m = blockIdx.x * blockDim.x + threadIdx.x;
  const float d = __uint_as_float(((unsigned)neg << 31) | ((unsigned)ex << 23) | (m & 0x7fffffu));
  if (__float_as_uint(gsk::rcp_markstein(d)) != __float_as_uint(__frcp_rn(d))) atomicAdd(bad, 1ull);
}
int done() {
  const cudaError_t e = cudaGetLastError();
  return (int)(e != cudaSuccess ? e : cudaDeviceSynchronize());
}
}  // namespace

#define EXPORT extern "C" __attribute__((visibility("default")))
EXPORT int level_sums(int n, const long long* hs, const long long* ls, const int* e, double* out) {
  k_level_sum<<<(n + 255) / 256, 256>>>(n, hs, ls, e, out);
  return done();
}
EXPORT int f32_ofs(int n, const double* r, int h, float* out) {
  k_f32_of<<<(n + 255) / 256, 256>>>(n, r, h, out);
  return done();
}
EXPORT int rcp_differences(int ex, int neg, unsigned long long* bad) {
  k_rcp<<<(1 << 23) / 256, 256>>>(ex, neg, bad);
  return done();
}
