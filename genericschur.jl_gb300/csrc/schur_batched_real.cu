// Batched real Schur decomposition, one CTA per matrix (n <= 128), FP64 (and an FP32
// instance of the same code for Float32 batches and the FP32 stage of the mixed form).
//
// Per size bin two launches over the bin's queue of matrices (largest first):
//   k_hess_real64 / k_hess_real32, k_formq_real32   load + _scale! (util.jl:14-29), Householder Hessenberg reduction
//                 (hessenberg.jl:3-17; reflector as in householder.jl:12-54, lmul!/rmul!
//                 as householder.jl:140-172) and Q formation (hessenberg.jl:150-166);
//   k_schur_real  the real double-shift Francis iteration of gschur!(H::Hessenberg{<:Real}, Z)
//                 (GenericSchur.jl:513-699) with doubleShiftQR! (837-952) and _gs2x2!
//                 (716-803) on a packed copy of H in shared memory (column j keeps rows
//                 1..j+3: the Hessenberg part and the two rows of the 3x3 bulge); T,
//                 eigenvalues and status written back, undoing the scaling.
// They are separate kernels because they want different shapes: the reduction needs the full
// matrix (and Z) in shared memory and many threads, the iteration is a chain of short
// dependent steps per matrix that wants as many matrices per SM as fit.
#include <algorithm>
#include <type_traits>

#include "device_common.cuh"
#include "gs_internal.h"

namespace gsk {
namespace {

template <class T>
struct Refl {
  T t1, t2, t3, v2, v3;
};

// Packed QR layout: column j (1-based) holds rows 1..j+3.
__host__ __device__ __forceinline__ int rpk(int j) { return ((j - 1) * (j + 6)) >> 1; }

#define HH(i, j) H[rpk(j) + (i) - 1]

// ---------------------------------------------------------------------------------
// Hessenberg reduction and Q formation.
//
// 4*NC threads (NC >= n): the dot product of a column (or row) with the reflector keeps two
// accumulators, over alternate elements, and each has its own thread: thread (c, par) of the
// first 2*NC holds column c (left update) or row c (right update) of A, the last 2*NC hold the
// rows of Z, whose update only needs the reflector and runs beside the left update of A.
// Bound: FP64, the FP64 pipe (4n^3 FMAs: 4.1 of the 5 n^3 / 3 needed are full warps);
// FP32, the latency of the seven barrier-separated steps per column.  With the matrix read
// from the L2-resident output buffer, one column per thread (32 lines per warp load), this phase
// took 31M cycles of an FP32 matrix of order 128 (57% of its time) and 17M of an FP64 one.
template <class T>
struct HessCtl {
  T tau, t, beta;  // of the current column
  int mode;        // 0: zero column, 1: reflector ready, 2: underflow guard needed
};

// max |.| over nonnegative values by their bit patterns: NaN compares largest, as block_max
template <class T> __device__ __forceinline__ unsigned long long abs_bits(T v);
template <> __device__ __forceinline__ unsigned long long abs_bits<double>(double v) {
  return (unsigned long long)__double_as_longlong(fabs(v));
}
template <> __device__ __forceinline__ unsigned long long abs_bits<float>(float v) {
  return (unsigned long long)__float_as_uint(fabsf(v));
}
template <class T> __device__ __forceinline__ T bits_abs(unsigned long long b);
template <> __device__ __forceinline__ double bits_abs<double>(unsigned long long b) { return __longlong_as_double((long long)b); }
template <> __device__ __forceinline__ float bits_abs<float>(unsigned long long b) { return __uint_as_float((unsigned)b); }

template <class T>
struct HessShared {
  T red[32];
  unsigned long long gmax[4];
  T gssq[4];
  HessCtl<T> c;
};

// Entries outside the range where squaring is safe, or the underflow guard
// (householder.jl:25-42): rescale x, alpha and beta.  All NT threads; ends behind a barrier.
template <class T, int NT>
__device__ __noinline__ void hess_reflector_guarded(T* col, int m, HessShared<T>& sh, T& tau, T& t, T& beta) {
  const int tid = threadIdx.x;
  const T sfmin = T(2) * Prec<T>::fmin / Prec<T>::eps;
  T big = T(0);
  for (int w = 0; w < 4; ++w) { const T v = bits_abs<T>(sh.gmax[w]); big = (v > big || v != v) ? v : big; }
  const bool safe = (big < Prec<T>::safe_hi && big > Prec<T>::safe_lo);
  const T sc = safe ? T(1) : T(1) / big;
  T ls = T(0);
  for (int r = 1 + tid; r < m; r += NT) { const T v = col[r] * sc; ls = fma(v, v, ls); }
  const T ssq = block_sum<NT>(ls, sh.red);
  T xnorm = safe ? sqrt(ssq) : big * sqrt(ssq);
  T alpha = col[0];
  beta = -copysign(hypot(alpha, xnorm), alpha);
  int kount = 0;
  if (fabs(beta) < sfmin) {
    const T rsfmin = T(1) / sfmin;
    T bb = beta;
    do { ++kount; bb *= rsfmin; alpha *= rsfmin; } while (fabs(bb) < sfmin && kount < 20);
    __syncthreads();
    for (int r = 1 + tid; r < m; r += NT) {
      T v = col[r];
      for (int q = 0; q < kount; ++q) v *= rsfmin;
      col[r] = v;
    }
    __syncthreads();
    T lm2 = T(0);
    for (int r = 1 + tid; r < m; r += NT) lm2 = fmax(lm2, fabs(col[r]));
    const T big2 = block_max<NT>(lm2, sh.red);
    const T sc2 = (big2 > T(0)) ? T(1) / big2 : T(0);
    T ls2 = T(0);
    for (int r = 1 + tid; r < m; r += NT) { const T v = col[r] * sc2; ls2 = fma(v, v, ls2); }
    const T ssq2 = block_sum<NT>(ls2, sh.red);
    xnorm = big2 * sqrt(ssq2);
    beta = -copysign(hypot(alpha, xnorm), alpha);
  }
  tau = (beta - alpha) / beta;
  t = T(1) / (alpha - beta);
  for (int q = 0; q < kount; ++q) beta *= sfmin;
  __syncthreads();
}

// Scalars of the reflector from the warps' maxima and sums: the mode as in HessCtl.
template <class T>
__device__ __forceinline__ int hess_scalars(const HessShared<T>& sh, T alpha, T& tau, T& t, T& beta) {
  const T sfmin = T(2) * Prec<T>::fmin / Prec<T>::eps;
  unsigned long long mb = sh.gmax[0];
  for (int w = 1; w < 4; ++w) mb = sh.gmax[w] > mb ? sh.gmax[w] : mb;
  const T big = bits_abs<T>(mb);
  tau = t = beta = T(0);
  if (big == T(0)) return 0;
  if (!(big < Prec<T>::safe_hi && big > Prec<T>::safe_lo)) return 2;
  T ssq = sh.gssq[0];
  for (int w = 1; w < 4; ++w) ssq += sh.gssq[w];
  const T xnorm = sqrt(ssq);
  beta = -copysign(hypot(alpha, xnorm), alpha);
  if (fabs(beta) < sfmin) return 2;
  tau = (beta - alpha) / beta;
  t = T(1) / (alpha - beta);
  return 1;
}

// Reflector of col[0..m): tau, the scale t of the tail and beta (householder.jl:12-54); false when
// the tail is zero.  All 4*NC threads call it; it ends behind a barrier.
template <class T, int NT>
__device__ __forceinline__ bool hess_reflector(T* col, int m, HessShared<T>& sh, T& tau, T& t, T& beta) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  // norm of the tail: elements 1+32w..32+32w are warp w's, summed by a tree, the warps' sums in order
  if (warp < 4) {
    const T x = (1 + tid < m) ? col[1 + tid] : T(0);
    unsigned long long mb = abs_bits<T>(x);
    T q = fma(x, x, T(0));
    for (int o = 16; o > 0; o >>= 1) {
      const unsigned long long w = __shfl_xor_sync(0xffffffffu, mb, o);
      mb = w > mb ? w : mb;
      q += __shfl_xor_sync(0xffffffffu, q, o);
    }
    if (lane == 0) { sh.gmax[warp] = mb; sh.gssq[warp] = q; }
  }
  __syncthreads();
  if (warp == 0) {
    T tau_, t_, beta_;
    const int mode = hess_scalars(sh, col[0], tau_, t_, beta_);
    if (lane == 0) { sh.c.mode = mode; sh.c.tau = tau_; sh.c.t = t_; sh.c.beta = beta_; }
  }
  __syncthreads();
  const int mode = sh.c.mode;
  if (mode == 0) return false;
  tau = sh.c.tau; t = sh.c.t; beta = sh.c.beta;
  if (mode == 2) hess_reflector_guarded<T, NT>(col, m, sh, tau, t, beta);
  return true;
}

// _scale! factors (util.jl:14-29) on element-wise access; returns whether the matrix was scaled.
template <class T, class F>
__device__ __forceinline__ void hess_scale(double amax, F each) {
  const double smlnum = sqrt((double)Prec<T>::fmin) / (double)Prec<T>::eps;
  const double bignum = 1.0 / smlnum;
  double cscale = 0.0;
  if (amax > 0.0 && amax < smlnum) cscale = smlnum;
  else if (amax > bignum) cscale = bignum;
  if (cscale == 0.0) return;
  double mul[8];
  const int nf = safescale_factors(amax, cscale, mul);
  for (int f = 0; f < nf; ++f) each(mul[f]);
  __syncthreads();
}

// Where the reduction leaves max|a| for the iteration, which undoes the scaling: below the subdiagonal of
// A.  (Not with the eigenvalues: where the iteration gives up, those that it did not find keep what the
// caller had there.)  Orders 1 and 2 have no such place, but deflate at once.
template <class T, class W>
__device__ __forceinline__ T* amax_place(T* Ag, W* wr, int n) {
  return n > 2 ? Ag + (n - 1) : reinterpret_cast<T*>(wr);
}

template <class W, int NC>
__global__ void __launch_bounds__(4 * NC) k_hess_real64(RealBatchT<double, W> bt, const int* __restrict__ order,
                                                        const int* __restrict__ sched, int bin, int nmax, int cap) {
  typedef double T;
  constexpr int NT = 4 * NC;
  extern __shared__ __align__(16) double smem_raw[];
  __shared__ T part[4][NC];
  __shared__ HessShared<T> sh;
  const int tid = threadIdx.x;
  const int start = sched[3 * bin], end = sched[3 * bin + 1];
  const bool isz = tid >= 2 * NC;
  const int c = tid % NC, par = (tid / NC) & 1;
  for (int job = start + blockIdx.x; job < end; job += gridDim.x) {
    const int b = order[job];
    const int n = bt.ns[b];
    if (n <= 0 || n > nmax) continue;  // k_schur_real reports it
    T* __restrict__ Ag = bt.A + bt.offs[b];
    T* __restrict__ Zg = bt.wantz ? bt.Z + bt.offs[b] : nullptr;
    const int ld = n | 1;
    T* A = smem_raw;
    // Z in shared memory beside A where the launch left room for it
    const bool zs = Zg && 2 * n * ld <= cap;
    T* Z = zs ? A + n * ld : Zg;
    const int ldz = zs ? ld : n;
    __syncthreads();  // the previous matrix is out of shared memory
    double amax = 0.0;
    for (int idx = tid; idx < n * n; idx += NT) {
      const int i = idx % n, j = idx / n;
      const T a = Ag[idx];
      A[i + j * ld] = a;
      if (Zg) Z[i + j * ldz] = (i == j) ? T(1) : T(0);
      const double aa = fabs(a);
      amax = (aa > amax || aa != aa) ? aa : amax;
    }
    amax = block_max<NT>(amax, sh.red);
    __syncthreads();
    if (bt.scale)
      hess_scale<T>(amax, [&](double f) {
        for (int idx = tid; idx < n * n; idx += NT) A[idx % n + idx / n * ld] *= f;
      });
    for (int i = 1; i <= n - 2; ++i) {
      const int m = n - i;                     // reflector length: rows i+1..n
      T* col = A + i + (size_t)(i - 1) * ld;   // col[0] = alpha, col[1..m-1] = x
      T tau, t, beta;
      if (!hess_reflector<T, NT>(col, m, sh, tau, t, beta)) continue;
      if (1 + tid < m) col[1 + tid] *= t;
      __syncthreads();
      if (tid == 0) col[0] = beta;
      if (tau == T(0)) { __syncthreads(); continue; }
      // lmul!(H', A[i+1:n, i+1:n]), a column of A per pair of threads, and rmul!(Z, H), a row
      // of Z per pair: both are x[0], x[1..m-1] against 1, col[1..m-1]
      {
        T* x = nullptr;
        int st = 1;
        if (!isz) { if (c < m) x = A + i + (size_t)(i + c) * ld; }
        else if (Zg && c < n) { x = Z + c + (size_t)i * ldz; st = ldz; }
        T a = T(0);
        if (x) {
          if (par == 0) a = x[0];
#pragma unroll 4
          for (int r = 1 + par; r < m; r += 2) a = fma(col[r], x[r * st], a);
        }
        part[tid / NC][c] = a;
        __syncthreads();
        if (x) {
          const int g = isz ? 2 : 0;
          const T va = (part[g][c] + part[g + 1][c]) * tau;
          if (par == 0) x[0] -= va;
#pragma unroll 4
          for (int r = 1 + par; r < m; r += 2) x[r * st] = fma(-va, col[r], x[r * st]);
        }
      }
      __syncthreads();
      // rmul!(A[:, i+1:n], H): a row of A per pair of threads
      {
        T* x = (!isz && c < n) ? A + c + (size_t)i * ld : nullptr;
        T a = T(0);
        if (x) {
          if (par == 0) a = x[0];
#pragma unroll 4
          for (int q = 1 + par; q < m; q += 2) a = fma(x[q * ld], col[q], a);
          part[par][c] = a;
        }
        __syncthreads();
        if (x) {
          const T va = (part[0][c] + part[1][c]) * tau;
          if (par == 0) x[0] -= va;
#pragma unroll 4
          for (int q = 1 + par; q < m; q += 2) x[q * ld] = fma(-va, col[q], x[q * ld]);
        }
      }
      __syncthreads();
    }
    __syncthreads();
    for (int idx = tid; idx < n * n; idx += NT) {
      const int i = idx % n, j = idx / n;
      if (i <= j + 1) Ag[idx] = A[i + j * ld];
      if (zs) Zg[idx] = Z[i + j * ld];
    }
    if (tid == 0) *amax_place(Ag, bt.wr + bt.woffs[b], n) = amax;
  }
}

// FP32: bound by latency (a line's sum is a serial chain; about seven cycles per instruction and warp,
// four barriers per column), so many CTAs per SM matter: the reduction of A and the formation of Z
// are kernels of their own.  A pair of neighbouring lanes holds a column or row of A.  A line's entries
// stay in registers between its dot product and its update, in blocks of eight (A is padded by 16
// zero rows and columns so that a block needs no bounds), and the reflector is read four entries at a
// time.  The essential parts of the reflectors stay below the subdiagonal of A, for k_formq_real32, and
// their scalars and max|a|, whose place they take, in the (not yet formed) Z.
constexpr int kHessPad = 16;
// leading dimension = 18 mod 32: sixteen columns' pairs of neighbouring rows fall into 32 banks,
// and sixteen rows' pairs of neighbouring columns into 30
__host__ __device__ __forceinline__ int hess_ld32(int n) { return ((n + kHessPad + 13) & ~31) + 18; }

// dst[8 k + e], e = 0..7, for the blocks k < nb: f(k, u) with u the coefficients of block k
template <int NB, class F>
__device__ __forceinline__ void coef_blocks(const float* co, int k0, int k1, F f) {
#pragma unroll
  for (int k = 0; k < NB; ++k)
    if (k >= k0 && k < k1) {
      const float4 u0 = *(const float4*)(co + 8 * k), u1 = *(const float4*)(co + 8 * k + 4);
      const float u[8] = {u0.x, u0.y, u0.z, u0.w, u1.x, u1.y, u1.z, u1.w};
      f(k, u);
    }
}

// One line p[0], p[st], p[2 st], ... of A against 1, co: p -= tau (p . v) v.  x: registers.  All
// lanes of the warp call it, those without a line of their own (on = false) with another's.
template <int NB>
__device__ __forceinline__ void hess_line32(float* p, int st, int par, int nb, const float* co, float tau, bool on,
                                            float (&x)[8 * NB]) {
  const float x0 = p[0];
  float a = par == 0 ? x0 : 0.f;
  float* q = p + (1 + par) * st;
#pragma unroll
  for (int k = 0; k <= NB; ++k) {
    // the loads of block k are in flight during the sums of block k-1
    if (k < NB && k < nb) {
#pragma unroll
      for (int e = 0; e < 8; ++e) x[(8 * k + e) % (8 * NB)] = q[2 * (8 * k + e) * st];
    }
    if (k > 0 && k - 1 < nb) {
      const float4 u0 = *(const float4*)(co + 8 * (k - 1)), u1 = *(const float4*)(co + 8 * (k - 1) + 4);
      const float u[8] = {u0.x, u0.y, u0.z, u0.w, u1.x, u1.y, u1.z, u1.w};
#pragma unroll
      for (int e = 0; e < 8; ++e) a = fmaf(u[e], x[8 * (k > 0 ? k - 1 : 0) + e], a);
    }
  }
  const float va = (a + __shfl_xor_sync(0xffffffffu, a, 1)) * tau;
  if (!on) return;
  if (par == 0) p[0] = x0 - va;
  coef_blocks<NB>(co, 0, nb, [&](int k, const float* u) {
#pragma unroll
    for (int e = 0; e < 8; ++e) q[2 * (8 * k + e) * st] = fmaf(-va, u[e], x[8 * k + e]);
  });
}

template <class W, int NC>
__global__ void __launch_bounds__(NC == 32 ? 128 : 2 * NC, NC == 128 ? 2 : (NC == 64 ? 6 : 8))
    k_hess_real32(RealBatchT<float, W> bt, const int* __restrict__ order, const int* __restrict__ sched, int bin,
                  int nmax) {
  typedef float T;
  // at least the four warps of the norm
  constexpr int NT = 2 * NC < 128 ? 128 : 2 * NC, HC = NC / 2, NB = HC / 8;
  extern __shared__ __align__(16) double smem_raw[];
  __shared__ __align__(16) T ca[2][HC + 4];  // the reflector's odd and even entries, in different banks
  __shared__ HessShared<T> sh;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int start = sched[3 * bin], end = sched[3 * bin + 1];
  const int c = tid >> 1, par = tid & 1;
  const int cw = c & ~15;  // the warp's first line
  for (int job = start + blockIdx.x; job < end; job += gridDim.x) {
    const int b = order[job];
    const int n = bt.ns[b];
    if (n <= 0 || n > nmax) continue;  // k_schur_real reports it
    T* __restrict__ Ag = bt.A + bt.offs[b];
    T* __restrict__ taus = bt.wantz ? bt.Z + bt.offs[b] : nullptr;
    const int ld = hess_ld32(n);
    T* A = (T*)smem_raw;
    __syncthreads();  // the previous matrix is out of shared memory
    T amaxt = T(0);
    for (int j = warp; j < n + kHessPad; j += NT / 32)
      for (int i = lane; i < n + kHessPad; i += 32) {
        const T a = (i < n && j < n) ? Ag[i + j * n] : T(0);
        A[i + j * ld] = a;
        const T aa = fabsf(a);
        amaxt = (aa > amaxt || aa != aa) ? aa : amaxt;
      }
    const double amax = (double)block_max<NT>(amaxt, sh.red);
    __syncthreads();
    if (bt.scale)
      hess_scale<T>(amax, [&](double f) {
        for (int idx = tid; idx < n * n; idx += NT) {
          T& a = A[idx % n + idx / n * ld];
          a = (T)((double)a * f);
        }
      });
    T x[HC];
    for (int i = 1; i <= n - 2; ++i) {
      const int m = n - i;                     // reflector length: rows i+1..n
      T* col = A + i + (i - 1) * ld;           // col[0] = alpha, col[1..m-1] = x
      // the first four warps: norm of the tail, the scalars (each for itself), the reflector
      const T alpha = col[0];
      const T xt = (tid < 128 && 1 + tid < m) ? col[1 + tid] : T(0);
      if (warp < 4) {
        T q = fmaf(xt, xt, T(0));
        for (int o = 16; o > 0; o >>= 1) q += __shfl_xor_sync(0xffffffffu, q, o);
        const unsigned mb = __reduce_max_sync(0xffffffffu, __float_as_uint(fabsf(xt)));
        if (lane == 0) { sh.gmax[warp] = mb; sh.gssq[warp] = q; }
      }
      __syncthreads();
      if (warp < 4) {
        T tau, t, beta;
        const int mode = hess_scalars(sh, alpha, tau, t, beta);
        if (tid == 0) {
          sh.c.mode = mode;
          sh.c.tau = tau;
          if (taus) taus[i - 1] = tau;
          if (mode == 1) col[0] = beta;
        }
        if (mode == 1 && tid < NC) {
          const T v = xt * t;
          if (1 + tid < m) col[1 + tid] = v;
          ca[tid & 1][tid >> 1] = v;
        }
      }
      __syncthreads();
      const int mode = sh.c.mode;
      if (mode == 0) continue;
      T tau = sh.c.tau;
      if (mode == 2) {
        T t, beta;
        hess_reflector_guarded<T, NT>(col, m, sh, tau, t, beta);
        if (tid < NC) {
          const T v = (1 + tid < m) ? col[1 + tid] * t : T(0);
          if (1 + tid < m) col[1 + tid] = v;
          ca[tid & 1][tid >> 1] = v;
        }
        if (tid == 0) {
          col[0] = beta;
          if (taus) taus[i - 1] = tau;
        }
        __syncthreads();
      }
      if (tau == T(0)) continue;
      const int nb = (m / 2 + 7) / 8;  // of either parity: zeros beyond
      // lmul!(H', A[i+1:n, i+1:n]): a column of A per pair of lanes
      if (cw < m) hess_line32<NB>(A + i + (i + min(c, m - 1)) * ld, 1, par, nb, ca[par], tau, c < m, x);
      __syncthreads();
      // rmul!(A[:, i+1:n], H): a row of A per pair of lanes
      if (cw < n) hess_line32<NB>(A + min(c, n - 1) + i * ld, ld, par, nb, ca[par], tau, c < n, x);
      __syncthreads();
    }
    __syncthreads();
    for (int j = warp; j < n; j += NT / 32)
      for (int i = lane; i < n; i += 32) Ag[i + j * n] = A[i + j * ld];
    __syncthreads();
    if (tid == 0) {
      if (taus && n > 2) taus[n - 1] = (T)amax;
      else *amax_place(Ag, bt.wr + bt.woffs[b], n) = (T)amax;
    }
  }
}

// FP32 formation of Z (hessenberg.jl:150-166) from the reflectors that k_hess_real32 left in A and Z.
// Z stays in registers from the identity to the end: a pair of neighbouring lanes holds a row, one lane
// the even columns, the other the odd ones.  Two reflectors are staged in shared memory ahead, by
// absolute column: cd with 0, cu with 1 at column i.
template <class W, int NC>
__global__ void __launch_bounds__(2 * NC, NC == 128 ? 2 : (NC == 64 ? 6 : 16))
    k_formq_real32(RealBatchT<float, W> bt, const int* __restrict__ order, const int* __restrict__ sched, int bin,
                   int nmax) {
  typedef float T;
  constexpr int HC = NC / 2, NB = HC / 8;
  __shared__ __align__(16) T cd[2][2][HC + 4], cu[2][2][HC + 4];
  __shared__ T taus[NC];
  const int tid = threadIdx.x;
  const int start = sched[3 * bin], end = sched[3 * bin + 1];
  const int c = tid >> 1, par = tid & 1;
  for (int job = start + blockIdx.x; job < end; job += gridDim.x) {
    const int b = order[job];
    const int n = bt.ns[b];
    if (n <= 0 || n > nmax) continue;
    T* Ag = bt.A + bt.offs[b];
    T* Zg = bt.Z + bt.offs[b];
    if (tid < n && n > 2) taus[tid] = Zg[tid];
    const bool zrow = (c & ~15) < n;
    const int bz = ((n + 1) / 2 + 7) / 8;
    T z[HC];  // Z(c, par + 2 e)
#pragma unroll
    for (int e = 0; e < HC; ++e) z[e] = (2 * e + par == c) ? T(1) : T(0);
    T next = (tid < n && tid > 1 && n > 2) ? Ag[tid] : T(0);  // entry at absolute column tid of reflector 1
    for (int i = 1; i <= n - 2; ++i) {
      const int buf = i & 1;
      if (tid < NC) {
        const T v = tid > i ? next : T(0);
        cd[buf][tid & 1][tid >> 1] = v;
        cu[buf][tid & 1][tid >> 1] = tid == i ? T(1) : v;
        next = (tid < n && tid > i + 1) ? Ag[tid + i * n] : T(0);
      }
      __syncthreads();  // the buffer of step i - 1 is rewritten after the next one
      const T tau = taus[i - 1];
      if (tau == T(0) || !zrow) continue;
      const int b0 = i >> 4;         // of either parity
      const bool own = par == (i & 1);  // this lane holds column i
      T x0 = T(0);  // Z(c, i): cu - cd is 1 at column i, 0 elsewhere
#pragma unroll
      for (int k = 0; k < NB; ++k)
        if (k == b0) {
#pragma unroll
          for (int e = 0; e < 8; ++e) x0 = fmaf(cu[buf][par][8 * k + e] - cd[buf][par][8 * k + e], z[8 * k + e], x0);
        }
      x0 = __shfl_xor_sync(0xffffffffu, x0, 1);
      T a = own ? T(0) : x0;
      coef_blocks<NB>(cd[buf][par], b0, bz, [&](int k, const T* u) {
#pragma unroll
        for (int e = 0; e < 8; ++e) a = fmaf(u[e], z[8 * k + e], a);
      });
      const T va = (a + __shfl_xor_sync(0xffffffffu, a, 1)) * tau;
      coef_blocks<NB>(cu[buf][par], b0, bz, [&](int k, const T* u) {
#pragma unroll
        for (int e = 0; e < 8; ++e) z[8 * k + e] = fmaf(-va, u[e], z[8 * k + e]);
      });
    }
    if (c < n) {
#pragma unroll
      for (int e = 0; e < HC; ++e)
        if (2 * e + par < n) Zg[c + (2 * e + par) * n] = z[e];
    }
    if (tid == n - 1 && n > 2) *amax_place(Ag, bt.wr, n) = taus[tid];  // (this thread alone has read that place)
    __syncthreads();  // before the next matrix's reflectors
  }
}

// ---------------------------------------------------------------------------------
// Francis iteration.
//
// Warp specialisation: one warp (the chain warp) runs the serial part of the sweeps -- the
// deflation scan, the shifts, the start row, and the bulge chase inside a window of at most
// kWin rows around the diagonal -- and the other warps apply the reflectors it logged, a chunk of steps
// at a time and one phase later, to the columns right of the window, the rows above it and
// Z (the far work).  One CTA barrier per phase.  Every element sees the same operations in the
// same order as in the step-by-step iteration: for an element right of the window the
// left updates of a chunk come before its right updates of later chunks, and
//   - the columns that enter the next window get this chunk's left updates from the chain warp
//     itself at the start of the next phase (urgent columns), the rest from the far warps;
//   - row ka-1 (just above the window) stays with the chain warp, so that the diagonal and
//     both its neighbours are final when a sweep's last chunk is done, and the next sweep's scan,
//     shifts and start row overlap the far work of that chunk;
//   - the next sweep's first window must not reach the columns ka.. of that chunk above its
//     rows: its first chunk is shortened, or the chain warp skips a phase.
// The 2x2 blocks are standardised together at the end, a block per thread (GenericSchur.jl
// standardises each as it deflates; the block, its eigenvalues and Z see the same operations,
// entries above a block see its rotation after instead of before later sweeps' reflectors).  The
// windows of the FP32 large path (kInOrder), where such a rounding difference could change a later
// decision, have the far warps standardise and rotate before the next chunk.
//
// Why: with one CTA barrier per chase step (the near block and the next reflector on one
// warp, far updates on the others, the Z pass after each sweep), a step of an order-128 matrix took
// 1040 cycles in FP32 and 3880 in FP64 plus 400 / 1020 for its part of the Z pass.
template <class T>
struct Cmd {
  int type;  // 0 nothing, 1 chunk, 2 done
  int ka;    // first step
  int n3;    // steps with a 3-element reflector
  int last2; // then a 2-element one
  int jfar;  // first column of the far left updates
  int giv0, giv1;  // kInOrder: the pairs to standardise before the chunk
};

constexpr int kWin = 28;    // most steps of a chunk (kWin + 3 columns, kWin + 3 rows in a warp's lanes)
constexpr int kChunk = 16;  // steps of a chunk of a longer sweep
constexpr int kMinChunk = 4;
constexpr int kLogStep = 8; // log entries per step: t1, t2, t3, v2, v3 (16-byte aligned)
constexpr int kLogElems = 2 * kLogStep * (kWin + 1);

template <class T> __device__ __forceinline__ Refl<T> ld_refl(const T* l);
template <> __device__ __forceinline__ Refl<float> ld_refl<float>(const float* l) {
  const float4 a = *(const float4*)l;
  return {a.x, a.y, a.z, a.w, l[4]};
}
template <> __device__ __forceinline__ Refl<double> ld_refl<double>(const double* l) {
  const double2 a = *(const double2*)l, b = *(const double2*)(l + 2);
  return {a.x, a.y, b.x, b.y, l[4]};
}

// The phase barrier: the chain warp and the far warps meet it at different places of the code.
template <int NT> __device__ __forceinline__ void phase_barrier() { asm volatile("bar.sync 1, %0;" ::"n"(NT) : "memory"); }

template <int NT> __device__ __forceinline__ void far_barrier() { asm volatile("bar.sync 2, %0;" ::"n"(NT - 32) : "memory"); }

// One 3-element reflector on (z0, z1, z2): returns the finished first element.
template <class T>
__device__ __forceinline__ T slide3(const Refl<T>& r, T& z0, T& z1, T z2) {
  const T ss = fma(r.v3, z2, fma(r.v2, z1, z0));
  const T out = fma(-ss, r.t1, z0);
  z0 = fma(-ss, r.t2, z1);
  z1 = fma(-ss, r.t3, z2);
  return out;
}

// The logged reflectors of a chunk applied to one line (a column of H below row ka, a row of
// H or Z from column ka): element e+1 follows element e at distance inc, growing by d per step.
template <class T>
__device__ __forceinline__ void apply_line(T* p, int inc, int d, const T* lg, int n3, int last2) {
  T* p1 = p + inc;
  inc += d;
  T* p2 = p1 + inc;
  inc += d;
  T z0 = *p, z1 = *p1;
  int s = 0;
  for (; s + 4 <= n3; s += 4, lg += 4 * kLogStep) {
    T* q1 = p2 + inc;
    T* q2 = q1 + inc + d;
    T* q3 = q2 + inc + 2 * d;
    const T y0 = *p2, y1 = *q1, y2 = *q2, y3 = *q3;
    *p = slide3(ld_refl<T>(lg), z0, z1, y0);
    *p1 = slide3(ld_refl<T>(lg + kLogStep), z0, z1, y1);
    *p2 = slide3(ld_refl<T>(lg + 2 * kLogStep), z0, z1, y2);
    *q1 = slide3(ld_refl<T>(lg + 3 * kLogStep), z0, z1, y3);
    p = q2;
    p1 = q3;
    p2 = q3 + inc + 3 * d;
    inc += 4 * d;
  }
  for (; s < n3; ++s, lg += kLogStep) {
    const T y0 = *p2;
    *p = slide3(ld_refl<T>(lg), z0, z1, y0);
    p = p1;
    p1 = p2;
    p2 += inc;
    inc += d;
  }
  if (last2) {
    const Refl<T> r = ld_refl<T>(lg);
    const T ss = fma(r.v2, z1, z0);
    z0 = fma(-ss, r.t1, z0);
    z1 = fma(-ss, r.t2, z1);
  }
  *p = z0;
  *p1 = z1;
}

// Reflector (householder.jl:12-54, as reflector_fast) of (a, x1, x2), x2 = 0 for a 2-element one;
// a <- beta.  One test sends every case off the plain path to reflector_fast.
__device__ __forceinline__ Refl<float> chain_refl(float& a, float x1, float x2, int nr, int) {
  const float ss = fmaf(a, a, fmaf(x1, x1, x2 * x2));
  if (!(ss > 1.0e-30f && ss < 1.0e30f) || ((__float_as_uint(x1) | __float_as_uint(x2)) << 1) == 0) {
    const float t1 = reflector_fast(a, x1, x2, nr);
    return {t1, t1 * x1, t1 * x2, x1, x2};
  }
  float y;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(ss));
  const float s = ss * y;
  const float aa = fabsf(a);
  const float tau = fmaf(aa, y, 1.0f);
  const float t = copysignf(rcp_markstein(aa + s), a);
  x1 *= t;
  x2 *= t;
  a = -copysignf(s, a);
  return {tau, tau * x1, tau * x2, x1, x2};
}
// FP64: every FP64 instruction holds the sub-partition's pipe for 64 cycles whether 1 or 32 lanes are
// active, so a step of the chase costs its number of FP64 instructions: 5 for the left update (a column
// per lane), 5 for the right update (a row per lane) and 17 here: independent pairs (tau and s,
// v2 and v3, t2 and t3) are one instruction on two lanes each, the range tests are on the bits.
__device__ __forceinline__ Refl<double> chain_refl(double& a, double x1, double x2, int nr, int lane) {
  const double xs = fma(x1, x1, x2 * x2);
  const double ss = fma(a, a, xs);
  // xs != 0 and 1e-290 < ss < 1e290 (nonnegative values; NaN is above all)
  const long long sb = __double_as_longlong(ss);
  if (__double_as_longlong(xs) == 0 || sb <= __double_as_longlong(1.0e-290) || sb >= __double_as_longlong(1.0e290)) {
    const double t1 = reflector_fast(a, x1, x2, nr);
    return {t1, t1 * x1, t1 * x2, x1, x2};
  }
  const double y = rsqrt_nr(ss);
  const double aa = fabs(a);
  // even lanes tau = |a| y + 1, odd lanes s = ss y
  const double ts = fma((lane & 1) ? ss : aa, y, (lane & 1) ? 0.0 : 1.0);
  const double tau = __shfl_sync(0xffffffffu, ts, 0), s = __shfl_sync(0xffffffffu, ts, 1);
  const double t = copysign(rcp_nr(aa + s), a);
  // even lanes v2, t2; odd lanes v3, t3
  const double v = ((lane & 1) ? x2 : x1) * t;
  const double tv = tau * v;
  a = -copysign(s, a);
  return {tau, __shfl_sync(0xffffffffu, tv, 0), __shfl_sync(0xffffffffu, tv, 1), __shfl_sync(0xffffffffu, v, 0),
          __shfl_sync(0xffffffffu, v, 1)};
}

__device__ __forceinline__ void st_refl(float* l, const Refl<float>& r) {
  *(float4*)l = make_float4(r.t1, r.t2, r.t3, r.v2);
  l[4] = r.v3;
}
__device__ __forceinline__ void st_refl(double* l, const Refl<double>& r) {
  *(double2*)l = make_double2(r.t1, r.t2);
  *(double2*)(l + 2) = make_double2(r.t3, r.v2);
  l[4] = r.v3;
}

// Bounds by exponents, off the FP64 pipe and without quotients: for a normal x with exponent field e(x),
// 2^(e(x) - bias) <= |x| < 2^(e(x) - bias + 1) (0 and denormals have field 0).
template <class T> struct ExpF;
template <> struct ExpF<double> {
  static constexpr int digits = 52, lo = 923, hi = 1223;  // bias 1023: |x| in [2^-100, 2^201]
  static __device__ __forceinline__ int field(const double& x) { return (__double2hiint(x) >> 20) & 0x7ff; }
};
template <> struct ExpF<float> {
  static constexpr int digits = 23, lo = 97, hi = 157;     // bias 127: |x| in [2^-30, 2^31]
  static __device__ __forceinline__ int field(const float& x) { return (__float_as_int(x) >> 23) & 0xff; }
};

// Whether the deflation test at row k certainly fails: |H[k,k-1]| > eps (|H[k-1,k-1]| + |H[k,k]|), all
// of moderate size (so that it is not below the absolute threshold either).
template <class T>
__device__ __forceinline__ bool no_split(const T& hk, const T& hkk, const T& hkm1) {
  using E = ExpF<T>;
  const int e = E::field(hk), m = max(E::field(hkk), E::field(hkm1));
  return e > E::lo && m > 0 && e > m + 2 - E::digits;
}

// Whether the start-row test at row m certainly fails:
//   |h10| (|v1| + |v2|) > eps |v0| d,  with |v1| + |v2| >= |h21 h32| / c, |v0| <= (|h21 h12| +
//   |(h11 - r1r)(h11 - r2r)| + |r1i r2i|) / c for the same c > 0 and d the sum of three moduli;
// entries outside the moderate range go to the test itself.
template <class T>
__device__ __forceinline__ bool no_start(const T& h10, const T& h21, const T& h32, const T& h12, const T& h11,
                                         const T& h00, const T& h22, T r1r, T r1i, T r2r, T r2i) {
  using E = ExpF<T>;
  const int e10 = E::field(h10), e21 = E::field(h21), e32 = E::field(h32), e11 = E::field(h11);
  const int x = max(e11, E::field(r1r)), y = max(e11, E::field(r2r));
  const int e12 = E::field(h12), i1 = E::field(r1i), i2 = E::field(r2i);
  const int d = max(E::field(h00), max(e11, E::field(h22)));
  if (min(e10, min(e21, e32)) < E::lo || max(max(max(e21, e12), max(x, y)), max(max(i1, i2), d)) > E::hi) return false;
  const int t = max(e21 + e12, max(x + y + 2, i1 + i2));
  // lhs >= 2^(e10 + e21 + e32 - 3 bias); rhs < 2^-digits 2^(t - 2 bias + 2 + 2) 2^(d - bias + 1 + 2)
  return e10 + e21 + e32 > t + d + 7 - E::digits;
}

// The start vector's first entry and its reflector, with the sums and products fused as in the
// per-lane start code that they replace (FP64: a rounding here changes the iteration's path).
__device__ __forceinline__ float start_v0(float a, float b, float c, float d, float e, float f) { return a * b + c * d - e * f; }
__device__ __forceinline__ double start_v0(double a, double b, double c, double d, double e, double f) {
  return fma(-e, f, fma(a, b, c * d));
}
__device__ __forceinline__ Refl<float> start_refl(float a, float x1, float x2, int lane) { return chain_refl(a, x1, x2, 3, lane); }
__device__ __forceinline__ Refl<double> start_refl(double a, double x1, double x2, int lane) {
  const double xs = fma(x1, x1, x2 * x2);
  const double ss = fma(a, a, xs);
  const long long sb = __double_as_longlong(ss);
  if (__double_as_longlong(xs) == 0 || sb <= __double_as_longlong(1.0e-290) || sb >= __double_as_longlong(1.0e290)) {
    const double t1 = reflector_fast(a, x1, x2, 3);
    return {t1, t1 * x1, t1 * x2, x1, x2};
  }
  const double y = rsqrt_nr(ss);
  const double aa = fabs(a);
  const double tau = fma(aa, y, 1.0);
  const double t = copysign(rcp_nr(fma(ss, y, aa)), a);
  const double v = ((lane & 1) ? x2 : x1) * t;
  const double tv = tau * v;
  return {tau, __shfl_sync(0xffffffffu, tv, 0), __shfl_sync(0xffffffffu, tv, 1), __shfl_sync(0xffffffffu, v, 0),
          __shfl_sync(0xffffffffu, v, 1)};
}

// Chain warp: steps ka..ka+nst-1 inside the window (columns ..wl, rows ka-1..).  r: the reflector of
// step ka on entry, of step ka+nst on return.  The loop is written for few instructions and no
// branches: one warp runs it alone, so each costs about four cycles.  Lanes outside the window
// compute on clamped addresses and store nothing.
template <class T>
__device__ __forceinline__ void chase_chunk(T* H, int ka, int nst, int iend, int wl, Refl<T>& r, T* lg, int lane) {
  const unsigned all = 0xffffffffu;
  const int n3 = min(nst, iend - 1 - ka);     // steps with a 3-element reflector
  const int j = min(ka + lane, wl);           // left updates: a column per lane
  const bool colok = ka + lane <= wl;
  T* hc = H + rpk(j) + ka - 1;                // H(k, j)
  const int i = ka - 1 + lane;                // right updates: a row per lane
  const bool rowok = i >= 1 && i <= iend;
  const int ic = min(max(i, 1), iend) - 1;
  int c0 = rpk(ka);
  T* p0 = H + c0 + ic;                        // H(i, k), H(i, k+1), H(i, k+2)
  T* p1 = p0 + ka + 3;
  T* p2 = p1 + ka + 4;
  T* hb = H + c0 + ka;                        // H(k+1, k)
  T a0 = hc[0], a1 = hc[1], a2 = hc[2];
  for (int s = 0; s < n3; ++s) {
    const int k = ka + s;
    if (lane == 0) st_refl(lg, r);
    lg += kLogStep;
    {
      const T ss = fma(r.v3, a2, fma(r.v2, a1, a0));
      a0 = fma(-ss, r.t1, a0);
      a1 = fma(-ss, r.t2, a1);
      a2 = fma(-ss, r.t3, a2);
    }
    if (colok && j >= k) { hc[0] = a0; hc[1] = a1; hc[2] = a2; }
    __syncwarp();
    T b0 = *p0, b1 = *p1, b2 = *p2;
    {
      const T ss = fma(r.v3, b2, fma(r.v2, b1, b0));
      b0 = fma(-ss, r.t1, b0);
      b1 = fma(-ss, r.t2, b1);
      b2 = fma(-ss, r.t3, b2);
    }
    // column k, rows k+1..k+3: the next reflector
    T a = __shfl_sync(all, b0, s + 2);
    const T x1 = __shfl_sync(all, b0, s + 3);
    T x2 = __shfl_sync(all, b0, s + 4);
    if (rowok && i <= k + 3) { *p0 = b0; *p1 = b1; *p2 = b2; }
    __syncwarp();
    ++hc;
    a0 = hc[0]; a1 = hc[1]; a2 = hc[2];
    const int nr = min(3, iend - k);
    if (nr < 3) x2 = T(0);
    r = chain_refl(a, x1, x2, nr, lane);
    if (lane == 0) { hb[0] = a; hb[1] = T(0); hb[2] = T(0); }
    hb += k + 4;
    p0 = p1;
    p1 = p2;
    p2 += k + 5;
  }
  if (n3 < nst) {
    // 2-element reflector at k = iend-1
    const int k = iend - 1;
    if (lane == 0) st_refl(lg, r);
    if (colok && j >= k) {
      const T ss = fma(r.v2, a1, a0);
      hc[0] = fma(-ss, r.t1, a0);
      hc[1] = fma(-ss, r.t2, a1);
    }
    __syncwarp();
    if (rowok) {
      const T b0 = *p0, b1 = *p1;
      const T ss = fma(r.v2, b1, b0);
      *p0 = fma(-ss, r.t1, b0);
      *p1 = fma(-ss, r.t2, b1);
    }
  }
  __syncwarp();
}

// Rotation of a standardised block at (p, p+1): rmul!(HH[1:p-1, :], G') and Z, lmul!(G, HH[:, p+2:n]),
// thread t of nt.
template <class T>
__device__ __forceinline__ void rotate_cols(T* H, int n, int p, T cs, T sn, int t, int nt, T* Zg) {
  for (int i = 1 + t; i <= p - 1; i += nt) {
    const T a1 = HH(i, p), a2 = HH(i, p + 1);
    HH(i, p) = cs * a1 + sn * a2;
    HH(i, p + 1) = -sn * a1 + cs * a2;
  }
  if (Zg)
    for (int i = t; i < n; i += nt) {
      T* zp = Zg + i + (long long)(p - 1) * n;
      const T a1 = zp[0], a2 = zp[n];
      zp[0] = cs * a1 + sn * a2;
      zp[n] = -sn * a1 + cs * a2;
    }
}
template <class T>
__device__ __forceinline__ void rotate_rows(T* H, int n, int p, T cs, T sn, int t, int nt) {
  for (int j = p + 2 + t; j <= n; j += nt) {
    const T a1 = HH(p, j), a2 = HH(p + 1, j);
    HH(p, j) = cs * a1 + sn * a2;
    HH(p + 1, j) = -sn * a1 + cs * a2;
  }
}

// nmax: the largest order the launch sized shared memory for.  Orders come from device
// memory (GS_DEVICE calls are not checked on the host), so an order outside [0, nmax]
// gets ST_BADARG before anything is read or written.
template <class T, class W, int NT>
__device__ void solve_real(const RealBatchT<T, W>& bt, int b, int nmax, T* smem, int cw) {
  __shared__ Cmd<T> cmd[2];
  __shared__ int s_status, s_npair;
  __shared__ int pairs[kSmallMax / 2];
  __shared__ T gcs[kSmallMax / 2], gsn[kSmallMax / 2];
  __shared__ T blks[kSmallMax * 2];  // kInOrder: the standardised blocks
  constexpr bool kInOrder = sizeof(T) == 4 && sizeof(W) == 8;
  __shared__ int s_giv;
  __shared__ double s_amax;
  const int tid = threadIdx.x;
  const int lane = tid & 31, warp = tid >> 5;
  const int n = bt.ns[b];
  if (n <= 0 || n > nmax) {
    if (tid == 0) bt.status[b] = (n == 0) ? ST_OK : ST_BADARG;
    return;
  }
  T* __restrict__ Ag = bt.A + bt.offs[b];
  T* Zg = bt.wantz ? bt.Z + bt.offs[b] : nullptr;
  W* __restrict__ wr = bt.wr + bt.woffs[b];
  W* __restrict__ wi = bt.wi + bt.woffs[b];
  T* logs = smem;
  T* H = smem + kLogElems;  // packed H
  if (tid == 0) s_amax = (double)*amax_place(Ag, wr, n);
  for (int j = 1 + warp; j <= n; j += NT / 32)
    for (int i = 1 + lane; i <= j + 3; i += 32)
      HH(i, j) = (i <= min(j + 1, n)) ? Ag[(i - 1) + (long long)(j - 1) * n] : T(0);
  __syncthreads();

  const T eps = Prec<T>::eps;
  const T smallnum = Prec<T>::fmin * ((T)n / eps);
  if (warp == cw) {
    // ---- chain warp (all its variables are uniform over the lanes) ----
    const long long maxiter = bt.maxiter_abs > 0 ? bt.maxiter_abs : (long long)bt.maxiter_mult * n;
    long long iter = 0;
    int status = ST_OK, iend = n, istart = 1, iterqr = 0, npair = 0, ngiv = 0;
    int state = 0;             // 0: between sweeps, 1: first chunk of a sweep is next, 2: inside a sweep
    int kn = 0;                // next step
    int pka = 0, pn3 = 0, pwl = 0;  // previous chunk of this sweep
    int fka = 0;               // ka of the sweep's last chunk while the far warps apply it (0: none)
    Refl<T> r{};
    for (int ph = 0;; ++ph) {
      Cmd<T>& cm = cmd[ph & 1];
      T* lg = logs + (ph & 1) * (kLogElems / 2);
      bool done = false;
      while (state == 0) {
        if (iend < 1) { done = true; break; }
        if (++iter > maxiter) { status = ST_UNCONVERGED; done = true; break; }
        // deflation scan (GenericSchur.jl:563-600): largest k with a negligible H[k,k-1]
        int found = 0;
        for (int top = iend; top >= istart + 1; top -= 32) {
          const int k = top - lane;
          bool split = false;
          if (k >= istart + 1) {
            const T hk = HH(k, k - 1);
            const T hkk = HH(k, k), hkm1 = HH(k - 1, k - 1);
            if (no_split(hk, hkk, hkm1)) {
              split = false;
            } else if (fabs(hk) < smallnum) {
              split = true;
            } else {
              T t = fabs(hkm1) + fabs(hkk);
              if (t == T(0)) {
                if (k > 2) t += fabs(HH(k - 1, k - 2));
                if (k + 1 <= n) t += fabs(HH(k + 1, k));
              }
              const T ahkkm1 = fabs(hk);
              if (ahkkm1 <= t * eps) {
                const T ahkm1k = fabs(HH(k - 1, k));
                const T ab = fmax(ahkkm1, ahkm1k), ba = fmin(ahkkm1, ahkm1k);
                const T aa = fmax(fabs(hkk), fabs(hkm1 - hkk)), bb = fmin(fabs(hkk), fabs(hkm1 - hkk));
                const T s = aa + bb;
                if (ba * (ab / s) <= fmax(smallnum, eps * (bb * (aa / s)))) split = true;
              }
            }
          }
          const unsigned bal = __ballot_sync(0xffffffffu, split);
          if (bal) { found = top - (__ffs(bal) - 1); break; }
        }
        istart = found > 0 ? found : 1;
        if (istart > 1 && lane == 0) HH(istart, istart - 1) = T(0);
        __syncwarp();
        if (istart >= iend - 1) {
          if (lane == 0) {
            if (istart >= iend) {
              wr[iend - 1] = (W)HH(iend, iend);
              wi[iend - 1] = W(0);
            } else {
              pairs[npair] = iend - 1;
              if (iend > 2) HH(iend - 1, iend - 2) = T(0);
            }
          }
          if (istart < iend) ++npair;
          __syncwarp();
          iend = istart - 1;
          istart = 1;
          iterqr = 0;
          continue;
        }
        ++iterqr;
        // shifts (GenericSchur.jl:614-665); the four quotients are one division over four lanes
        T r1r, r1i, r2r, r2i;
        {
          T h11, h12, h21, h22;
          if (iterqr == 10) {
            const T s = fabs(HH(istart + 1, istart)) + fabs(HH(istart + 2, istart + 1));
            h11 = T(0.75) * s + HH(istart, istart); h12 = T(-0.4375) * s; h21 = s; h22 = h11;
          } else if (iterqr == 20) {
            const T s = fabs(HH(iend, iend - 1)) + fabs(HH(iend - 1, iend - 2));
            h11 = T(0.75) * s + HH(iend, iend); h12 = T(-0.4375) * s; h21 = s; h22 = h11;
          } else {
            h11 = HH(iend - 1, iend - 1); h21 = HH(iend, iend - 1);
            h12 = HH(iend - 1, iend); h22 = HH(iend, iend);
          }
          const T s = fabs(h11) + fabs(h12) + fabs(h21) + fabs(h22);
          if (s == T(0)) {
            r1r = r2r = r1i = r2i = T(0);
          } else {
            T hq = (lane & 2) ? ((lane & 1) ? h22 : h21) : ((lane & 1) ? h12 : h11);
            hq /= s;
            h11 = __shfl_sync(0xffffffffu, hq, 0); h12 = __shfl_sync(0xffffffffu, hq, 1);
            h21 = __shfl_sync(0xffffffffu, hq, 2); h22 = __shfl_sync(0xffffffffu, hq, 3);
            const T tr = (h11 + h22) / T(2);
            const T d = (h11 - tr) * (h22 - tr) - h12 * h21;
            const T rtd = sqrt(fabs(d));
            if (d >= T(0)) {
              r1r = tr * s; r2r = r1r; r1i = rtd * s; r2i = -r1i;
            } else {
              r1r = tr + rtd; r2r = tr - rtd;
              if (fabs(r1r - h22) <= fabs(r2r - h22)) { r1r *= s; r2r = r1r; }
              else { r2r *= s; r1r = r2r; }
              r1i = r2i = T(0);
            }
          }
        }
        // start row (GenericSchur.jl:850-872): largest m with two small subdiagonals, else
        // istart; the start vector comes with it
        int mx = istart;
        for (int top = iend - 2; top >= istart + 1; top -= 32) {
          const int m = top - lane;
          bool hit = false;
          if (m >= istart + 1 &&
              !no_start(HH(m, m - 1), HH(m + 1, m), HH(m + 2, m + 1), HH(m, m + 1), HH(m, m), HH(m - 1, m - 1),
                        HH(m + 1, m + 1), r1r, r1i, r2r, r2i)) {
            T h21s = HH(m + 1, m);
            T s = fabs(HH(m, m) - r2r) + fabs(r2i) + fabs(h21s);
            h21s /= s;
            T v0 = h21s * HH(m, m + 1) + (HH(m, m) - r1r) * ((HH(m, m) - r2r) / s) - r1i * (r2i / s);
            T v1 = h21s * (HH(m, m) + HH(m + 1, m + 1) - r1r - r2r);
            T v2 = h21s * HH(m + 2, m + 1);
            s = fabs(v0) + fabs(v1) + fabs(v2);
            v0 /= s; v1 /= s; v2 /= s;
            hit = fabs(HH(m, m - 1)) * (fabs(v1) + fabs(v2)) <=
                  eps * fabs(v0) * (fabs(HH(m - 1, m - 1)) + fabs(HH(m, m)) + fabs(HH(m + 1, m + 1)));
          }
          const unsigned bal = __ballot_sync(0xffffffffu, hit);
          if (bal) { mx = top - (__ffs(bal) - 1); break; }
        }
        // the start vector, its two triples of quotients one division each
        T v0, v1, v2;
        {
          const int q = lane % 3;
          const T h11 = HH(mx, mx);
          T h21s = HH(mx + 1, mx);
          T s = fabs(h11 - r2r) + fabs(r2i) + fabs(h21s);
          T w = (q == 0 ? h21s : (q == 1 ? h11 - r2r : r2i)) / s;
          h21s = __shfl_sync(0xffffffffu, w, 0);
          const T ds = __shfl_sync(0xffffffffu, w, 1), rs = __shfl_sync(0xffffffffu, w, 2);
          v0 = start_v0(h21s, HH(mx, mx + 1), h11 - r1r, ds, r1i, rs);
          v1 = h21s * (h11 + HH(mx + 1, mx + 1) - r1r - r2r);
          v2 = h21s * HH(mx + 2, mx + 1);
          s = fabs(v0) + fabs(v1) + fabs(v2);
          w = (q == 0 ? v0 : (q == 1 ? v1 : v2)) / s;
          v0 = __shfl_sync(0xffffffffu, w, 0);
          v1 = __shfl_sync(0xffffffffu, w, 1);
          v2 = __shfl_sync(0xffffffffu, w, 2);
        }
        // reflector of the first step from the start vector
        r = start_refl(v0, v1, v2, lane);  // 3 elements: mx <= iend - 2
        if (mx > istart && lane == 0) HH(mx, mx - 1) *= (T(1) - r.t1);
        __syncwarp();
        kn = mx;
        state = 1;
      }
      int type = done ? 2 : 0;
      if (!done) {
        // the next chunk: steps kn..kn+nst-1
        int nst = iend - kn;
        if (nst > kWin) nst = kChunk;
        if (state == 1 && fka > 0 && kn < fka && min(kn + nst + 2, iend) >= fka) {
          // the far warps are still in columns fka.. above row fka-1
          nst = min(nst, fka - kn - 3);
          if (nst < kMinChunk) nst = 0;
        }
        if (nst > 0) {
          const int kb = kn + nst - 1;
          const int wl = min(kb + 3, iend);
          if (state == 2) {
            // urgent columns: the previous chunk's left updates on the columns entering the window
            const T* pl = logs + ((ph & 1) ^ 1) * (kLogElems / 2);
            const int j = pwl + 1 + lane;
            if (j <= wl) apply_line(&HH(pka, j), 1, 0, pl, pn3, 0);
            __syncwarp();
          }
          chase_chunk(H, kn, nst, iend, wl, r, lg, lane);
          const bool last = kb == iend - 1;
          int jfar = wl + 1;
          if (!last) {
            int nn = iend - kb - 1;
            if (nn > kWin) nn = kChunk;
            jfar = min(kb + nn + 3, iend) + 1;  // beyond the next chunk's window
          }
          if (lane == 0) {
            cm.ka = kn;
            cm.n3 = last ? nst - 1 : nst;
            cm.last2 = last;
            cm.jfar = jfar;
            cm.giv0 = ngiv;
            cm.giv1 = npair;
          }
          ngiv = npair;
          type = 1;
          pka = kn; pn3 = nst; pwl = wl;
          kn = kb + 1;
          fka = last ? pka : 0;
          state = last ? 0 : 2;
        } else {
          fka = 0;  // this phase's barrier ends the far work
        }
      }
      if (lane == 0) cm.type = type;
      phase_barrier<NT>();
      if (done) break;
    }
    if (lane == 0) { s_status = status; s_giv = kInOrder ? ngiv : 0; s_npair = npair; }
  } else {
    // ---- far warps ----
    const int ft = tid - (warp > cw ? 32 : 0);
    for (int ph = 0;; ++ph) {
      if (ph > 0 && cmd[(ph - 1) & 1].type == 1) {
        const Cmd<T> cm = cmd[(ph - 1) & 1];
        const T* lg = logs + ((ph - 1) & 1) * (kLogElems / 2);
        const int ka = cm.ka;
        if constexpr (kInOrder) {
          for (int q = cm.giv0; q < cm.giv1; ++q) {
            const int p = pairs[q];
            double a = HH(p, p), bq = HH(p, p + 1), cc = HH(p + 1, p), d = HH(p + 1, p + 1), cs, sn, w1r, w1i, w2r, w2i;
            gs2x2(a, bq, cc, d, cs, sn, w1r, w1i, w2r, w2i);
            rotate_cols(H, n, p, (T)cs, (T)sn, ft, NT - 32, Zg);
            rotate_rows(H, n, p, (T)cs, (T)sn, ft, NT - 32);
            if (ft == 0) {
              wr[p] = (W)w2r; wi[p] = (W)w2i; wr[p - 1] = (W)w1r; wi[p - 1] = (W)w1i;
              blks[4 * q] = (T)a; blks[4 * q + 1] = (T)bq; blks[4 * q + 2] = (T)cc; blks[4 * q + 3] = (T)d;
            }
            far_barrier<NT>();
          }
        }
        const int nl = n - cm.jfar + 1, nr = max(ka - 2, 0), nz = Zg ? n : 0;
        for (int t = ft; t < nl + nr + nz; t += NT - 32) {
          T* p;
          int inc, d = 0;
          if (t < nl) {
            p = &HH(ka, cm.jfar + t);
            inc = 1;
          } else if (t < nl + nr) {
            p = &HH(t - nl + 1, ka);
            inc = ka + 3;
            d = 1;
          } else {
            p = Zg + (t - nl - nr) + (long long)(ka - 1) * n;
            inc = n;
          }
          apply_line(p, inc, d, lg, cm.n3, cm.last2);
        }
      }
      phase_barrier<NT>();
      if (cmd[ph & 1].type == 2) break;
    }
  }
  __syncthreads();
  const int status = s_status, npair = s_npair;

  // ---- standardise the (remaining) 2x2 blocks (GenericSchur.jl:667-690) ----
  const int g0 = s_giv;
  if constexpr (kInOrder)
    for (int q = tid; q < g0; q += NT) {
      const int p = pairs[q];
      HH(p, p) = blks[4 * q]; HH(p, p + 1) = blks[4 * q + 1];
      HH(p + 1, p) = blks[4 * q + 2]; HH(p + 1, p + 1) = blks[4 * q + 3];
    }
  for (int q = g0 + tid; q < npair; q += NT) {
    const int p = pairs[q];
    double a = HH(p, p), bq = HH(p, p + 1), cc = HH(p + 1, p), d = HH(p + 1, p + 1), cs, sn, w1r, w1i, w2r, w2i;
    gs2x2(a, bq, cc, d, cs, sn, w1r, w1i, w2r, w2i);
    wr[p] = (W)w2r; wi[p] = (W)w2i; wr[p - 1] = (W)w1r; wi[p - 1] = (W)w1i;
    gcs[q] = (T)cs; gsn[q] = (T)sn;
    HH(p, p) = (T)a; HH(p, p + 1) = (T)bq; HH(p + 1, p) = (T)cc; HH(p + 1, p + 1) = (T)d;
  }
  __syncthreads();
  for (int q = g0 + warp; q < npair; q += NT / 32) rotate_cols(H, n, pairs[q], gcs[q], gsn[q], lane, 32, Zg);
  __syncthreads();
  for (int q = g0 + warp; q < npair; q += NT / 32) rotate_rows(H, n, pairs[q], gcs[q], gsn[q], lane, 32);
  __syncthreads();

  // ---- write back ----
  // (undoing the scale that the reduction applied)
  double mul[8];
  int nf = 0;
  if (bt.scale) {
    const double smlnum = sqrt((double)Prec<T>::fmin) / (double)Prec<T>::eps, amax = s_amax;
    const double bignum = 1.0 / smlnum;
    if (amax > 0.0 && amax < smlnum) nf = safescale_factors(smlnum, amax, mul);
    else if (amax > bignum) nf = safescale_factors(bignum, amax, mul);
  }
  for (int idx = tid; idx < n * n; idx += NT) {
    const int i = idx % n, j = idx / n;
    double v = (i > j + 1) ? 0.0 : (double)HH(i + 1, j + 1);
    for (int f = 0; f < nf; ++f) v *= mul[f];
    Ag[idx] = (T)v;
  }
  if (nf)
    for (int i = tid; i < n; i += NT) {
      double a = wr[i], bq = wi[i];
      for (int f = 0; f < nf; ++f) { a *= mul[f]; bq *= mul[f]; }
      wr[i] = (W)a; wi[i] = (W)bq;
    }
  if (tid == 0) bt.status[b] = status;
  __syncthreads();
}
#undef HH

// 768 threads per SM: at most 80 registers, at which FP64 spills 72 bytes (for one matrix too, where the
// occupancy is of no use)
template <class T, class W, int NT>
__global__ void __launch_bounds__(NT, 768 / NT) k_schur_real(RealBatchT<T, W> bt, const int* __restrict__ order,
                                                   int* __restrict__ sched, int bin, int nmax, int num_sms, int once) {
  extern __shared__ __align__(16) double smem_raw[];
  T* smem = (T*)smem_raw;
  __shared__ int s_job;
  const int start = sched[3 * bin], end = sched[3 * bin + 1];
  // the chain warps of an SM's CTAs sit on different sub-partitions (warps are dealt to the
  // four in turn): NW = 4, 8 warps shift by CTA, 2, 6 by pairs of CTAs, odd NW shift by themselves
  constexpr int NW = NT / 32;
  const int slot = blockIdx.x / num_sms;
  const int cw = NW % 4 == 0 ? slot % 4 : (NW % 2 == 0 ? (slot >> 1) & 1 : 0);
  if (once) {  // a CTA per matrix
    const int job = start + blockIdx.x;
    if (job < end) solve_real<T, W, NT>(bt, order[job], nmax, smem, cw);
    return;
  }
  for (;;) {
    if (threadIdx.x == 0) s_job = start + atomicAdd(&sched[3 * bin + 2], 1);
    __syncthreads();
    const int job = s_job;
    __syncthreads();
    if (job >= end) break;
    solve_real<T, W, NT>(bt, order[job], nmax, smem, cw);
  }
}

// Dynamic shared memory of one CTA of the iteration for orders up to nmax: the reflector
// log and the packed H.
size_t bin_smem_elems(int nmax) { return kLogElems + (size_t)rpk(nmax + 1); }
// ... of the reduction: FP64 the matrix, and Z where both fit; FP32 the padded matrix.
size_t hess_smem_elems(int nmax, size_t tsize) {
  if (tsize == 4) return (size_t)(nmax + kHessPad) * hess_ld32(nmax);
  const size_t one = (size_t)nmax * (nmax | 1), most = kMostSmem / tsize;
  return 2 * one <= most ? 2 * one : (one > most ? one : most);
}

template <class T, class W, int NC>
cudaError_t launch_hess(const RealBatchT<T, W>& bt, const int* order, const int* sched, int bin, int nmax,
                        int num_sms, cudaStream_t s) {
  const size_t elems = hess_smem_elems(nmax, sizeof(T)), smem = sizeof(T) * elems;
  constexpr int NT = sizeof(T) == 8 ? 4 * NC : (2 * NC < 128 ? 128 : 2 * NC);
  const void* f;
  if constexpr (sizeof(T) == 8) f = (const void*)k_hess_real64<W, NC>;
  else f = (const void*)k_hess_real32<W, NC>;
  cudaError_t e = allow_smem(f, sizeof(T) * hess_smem_elems(NC, sizeof(T)));
  if (e != cudaSuccess) return e;
  const int ctas = bin_grid(bt.count, num_sms, kReduceCtas);
  if constexpr (sizeof(T) == 8) {
    k_hess_real64<W, NC><<<ctas, NT, smem, s>>>(bt, order, sched, bin, nmax, (int)elems);
  } else {
    k_hess_real32<W, NC><<<ctas, NT, smem, s>>>(bt, order, sched, bin, nmax);
    if (bt.wantz) {
      k_formq_real32<W, NC><<<ctas, 2 * NC, 0, s>>>(bt, order, sched, bin, nmax);
    }
  }
  return cudaGetLastError();
}

template <class T, class W, int NT>
cudaError_t launch_bin(const RealBatchT<T, W>& bt, const int* order, int* sched, int bin, int nmax, int ctas,
                       int num_sms, cudaStream_t s) {
  cudaError_t e = nmax <= 32 ? launch_hess<T, W, 32>(bt, order, sched, bin, nmax, num_sms, s)
                             : (nmax <= 64 ? launch_hess<T, W, 64>(bt, order, sched, bin, nmax, num_sms, s)
                                           : launch_hess<T, W, 128>(bt, order, sched, bin, nmax, num_sms, s));
  if (e != cudaSuccess) return e;
  const size_t smem = sizeof(T) * bin_smem_elems(nmax);
  e = allow_smem(k_schur_real<T, W, NT>, sizeof(T) * bin_smem_elems(kSmallMax));
  if (e != cudaSuccess) return e;
  // a CTA per matrix, or a ticket queue: of bin_grid's CTAs, or, with a cap on CTAs per SM, of as many as
  // may be resident
  int grid = bin_grid(bt.count, num_sms, sizeof(T) == 4 ? kIterCtas32 : kIterCtas64);
  const int once = ctas == 0 && grid == bt.count;
  if (ctas > 0) {
    int per_sm = 0;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_schur_real<T, W, NT>, NT, smem);
    if (e != cudaSuccess) return e;
    grid = std::min(bt.count, num_sms * std::min(std::max(per_sm, 1), ctas));
  }
  k_schur_real<T, W, NT><<<grid, NT, smem, s>>>(bt, order, sched, bin, nmax, num_sms, once);
  return cudaGetLastError();
}

// One bin with the requested shape: FP64 compiles every thread count of kTuneThreads, the FP32
// kernel with FP32 eigenvalues (Float32 batches and the FP32 stage of the mixed form) all but
// 160, the FP32 kernel with FP64 eigenvalues (the large path's small solves) the default ones.
template <class T, class W>
cudaError_t launch_shape(const RealBatchT<T, W>& bt, const int* order, int* sched, int bin, int nmax, int nt,
                         int ctas, int num_sms, cudaStream_t s) {
#define GS_SHAPE(NTV) \
  if (nt == NTV) return launch_bin<T, W, NTV>(bt, order, sched, bin, nmax, ctas, num_sms, s);
  if constexpr (sizeof(T) == 8) {
    GS_SHAPE(64) GS_SHAPE(96) GS_SHAPE(128) GS_SHAPE(160) GS_SHAPE(192) GS_SHAPE(256)
  } else if constexpr (std::is_same_v<W, float>) {
    GS_SHAPE(64) GS_SHAPE(96) GS_SHAPE(128) GS_SHAPE(192) GS_SHAPE(256)
  } else {
    GS_SHAPE(64) GS_SHAPE(128)
  }
#undef GS_SHAPE
  return cudaErrorInvalidValue;
}

template <class T, class W>
cudaError_t launch_all_bins(const RealBatchT<T, W>& bt, const int* order, int* sched, int num_sms,
                            cudaStream_t* streams, int nstreams, const BinTuning& t) {
  // largest bin first: it carries most of the work
  for (int i = 0; i < kNumBins; ++i) {
    const int bin = kNumBins - 1 - i;
    if (bt.empty >> bin & 1) continue;
    cudaError_t e = launch_shape(bt, order, sched, bin, t.bounds[bin], t.nt[bin], t.ctas[bin], num_sms,
                                 streams[i % nstreams]);
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

}  // namespace

// A tuning row's hsmem flag (the Hessenberg phase in shared memory) selects nothing here any
// more: the reduction always runs in shared memory.
size_t real_bin_smem_bytes(int nmax, int) {
  return sizeof(double) * (bin_smem_elems(nmax) > hess_smem_elems(nmax, 8) ? bin_smem_elems(nmax) : hess_smem_elems(nmax, 8));
}
size_t real32_bin_smem_bytes(int nmax, int) {
  return sizeof(float) * (bin_smem_elems(nmax) > hess_smem_elems(nmax, 4) ? bin_smem_elems(nmax) : hess_smem_elems(nmax, 4));
}

template <class T, class W>
cudaError_t launch_schur_batched_real(const RealBatchT<T, W>& bt, const int* order, int* sched, int num_sms,
                                      cudaStream_t* streams, int nstreams) {
  return launch_all_bins(bt, order, sched, num_sms, streams, nstreams, default_tuning_real());
}
template cudaError_t launch_schur_batched_real<double, double>(const RealBatchT<double, double>&, const int*, int*, int,
                                                               cudaStream_t*, int);
template cudaError_t launch_schur_batched_real<float, double>(const RealBatchT<float, double>&, const int*, int*, int,
                                                              cudaStream_t*, int);
template cudaError_t launch_schur_batched_real<float, float>(const RealBatchT<float, float>&, const int*, int*, int,
                                                             cudaStream_t*, int);

template <class T, class W>
cudaError_t launch_schur_real_bin(const RealBatchT<T, W>& bt, const int* order, int* sched, int bin,
                                  const BinTuning& t, int num_sms, cudaStream_t s) {
  return launch_shape(bt, order, sched, bin, t.bounds[bin], t.nt[bin], t.ctas[bin], num_sms, s);
}
template cudaError_t launch_schur_real_bin<double, double>(const RealBatchT<double, double>&, const int*, int*, int,
                                                           const BinTuning&, int, cudaStream_t);
template cudaError_t launch_schur_real_bin<float, float>(const RealBatchT<float, float>&, const int*, int*, int,
                                                         const BinTuning&, int, cudaStream_t);

template <class T, class W>
cudaError_t launch_schur_real_one(const RealBatchT<T, W>& bt, int m, const int* order, int* sched, cudaStream_t s) {
  const BinTuning t = default_tuning_real();
  const int bin = default_bin_of(m);
  return launch_shape(bt, order, sched, bin, t.bounds[bin], t.nt[bin], 1, 1, s);
}
template cudaError_t launch_schur_real_one<double, double>(const RealBatchT<double, double>&, int, const int*, int*,
                                                           cudaStream_t);
template cudaError_t launch_schur_real_one<float, double>(const RealBatchT<float, double>&, int, const int*, int*,
                                                          cudaStream_t);

cudaError_t launch_schur_batched_real_tuned(const RealBatchT<double, double>& bt, const int* order, int* sched,
                                            int num_sms, cudaStream_t* streams, int nstreams, const BinTuning& tun) {
  return launch_all_bins(bt, order, sched, num_sms, streams, nstreams, tun);
}

cudaError_t launch_schur_batched_real32_tuned(const RealBatchT<float, float>& bt, const int* order, int* sched,
                                              int num_sms, cudaStream_t* streams, int nstreams, const BinTuning& tun) {
  return launch_all_bins(bt, order, sched, num_sms, streams, nstreams, tun);
}

}  // namespace gsk
