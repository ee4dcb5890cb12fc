// launch_he_tridiag for a chip of any number of SMs.
#include "gs_internal.h"

template <class S>
static int run(const S* A, int n, S* B, S* W, S* partial, int npart, void* ctl, S* tau, double* d, double* e, int num_sms) {
  cudaError_t r = gsk::launch_he_tridiag<S>(A, n, n, 0, B, W, partial, npart, (gsk::HeCtlBuf*)ctl, tau, d, e, num_sms, 0);
  if (r == cudaSuccess) r = cudaDeviceSynchronize();
  return (int)(r != cudaSuccess ? r : cudaGetLastError());
}

extern "C" __attribute__((visibility("default"))) int tridiag_r(const double* A, int n, double* B, double* W, double* partial,
                                                                int npart, void* ctl, double* tau, double* d, double* e,
                                                                int num_sms) {
  return run(A, n, B, W, partial, npart, ctl, tau, d, e, num_sms);
}
extern "C" __attribute__((visibility("default"))) int tridiag_c(const double2* A, int n, double2* B, double2* W,
                                                                double2* partial, int npart, void* ctl, double2* tau,
                                                                double* d, double* e, int num_sms) {
  return run(A, n, B, W, partial, npart, ctl, tau, d, e, num_sms);
}
