// The priorities of the streams of the size bins, the largest bin first.
#include "gschur_api.cu"

extern "C" __attribute__((visibility("default"))) int bin_priorities(int* out, int* least, int* greatest) {
  cudaError_t e = cudaDeviceGetStreamPriorityRange(least, greatest);
  for (int i = 0; i < gsk::kNumBins && e == cudaSuccess; ++i) {
    cudaStream_t s;
    if ((e = bin_stream(&s, i)) != cudaSuccess) break;
    e = cudaStreamGetPriority(s, &out[i]);
    cudaStreamDestroy(s);
  }
  return (int)e;
}
