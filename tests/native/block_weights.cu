// block_weights of the large mixed refinement, one thread per block pair.
#include "refine.cu"

namespace {
// Entries of block pair i: tp and tq (2 x 2, row-major, only the leading zp x zp / zq x zq), rhs[a + 2 b].
__global__ void k_weights(int count, const double* tp, const double* tq, const int* zp, const int* zq, const double* rhs,
                          double floor, double* w, int* fine) {
  __shared__ double Ta[2][gsk::kSt + 1], Tb[2][gsk::kSt + 1];
  const int i = blockIdx.x, a = threadIdx.x & 1, b = threadIdx.x >> 1;
  Ta[a][b] = tp[4 * i + 2 * a + b];
  Tb[a][b] = tq[4 * i + 2 * a + b];
  __syncthreads();
  if (a >= zp[i] || b >= zq[i]) return;
  double k[4];
  const bool ok = gsk::block_weights(Ta, Tb, 0, zp[i], 0, zq[i], a, b, floor, k);
  double s = 0.0;
  for (int e = 0; e < 4; ++e)
    if (k[e] != 0.0) s = fma(k[e], rhs[4 * i + e], s);
  w[4 * i + threadIdx.x] = s;
  if (!ok) atomicAnd(&fine[i], 0);
}
}  // namespace

extern "C" __attribute__((visibility("default"))) int weights(int count, const double* tp, const double* tq, const int* zp,
                                                              const int* zq, const double* rhs, double floor, double* w,
                                                              int* fine) {
  k_weights<<<count, 4>>>(count, tp, tq, zp, zq, rhs, floor, w, fine);
  cudaError_t e = cudaGetLastError();
  return (int)(e != cudaSuccess ? e : cudaDeviceSynchronize());
}
