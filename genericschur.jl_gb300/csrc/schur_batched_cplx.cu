// Batched complex Schur decomposition, one CTA per matrix (n <= 128), FP64.
//
// Per size bin two launches over the bin's queue of matrices (GenericSchur.jl:350-372 driver):
//   k_hess_cplx   load + _scale! (util.jl:14-29), complex Householder Hessenberg reduction
//                 (hessenberg.jl:3-17; reflector householder.jl:56-102, which also makes the
//                 last subdiagonal real) and Q formation (hessenberg.jl:150-166);
//   k_schur_cplx  single-shift complex QR of gschur!(H::Hessenberg{Complex}, Z)
//                 (GenericSchur.jl:194-335) with singleShiftQR! (374-504): Ahues-Tisseur
//                 deflation, Wilkinson / exceptional shifts, 2-element reflector chase, the
//                 phase fix-ups that keep the subdiagonal real, in the (L2-resident) output buffer
//                 with the window around the diagonal in shared memory; T = triu(H),
//                 w = diag(T), scaling undone.
#include <algorithm>

#include "device_common.cuh"
#include "gs_internal.h"

namespace gsk {
namespace {

#define HH(i, j) H[((i) - 1) + ((j) - 1) * n]

// ---------------------------------------------------------------------------------
// Hessenberg reduction and Q formation: 4*NC threads (NC >= n).  Thread (c, p) of the first 2*NC
// computes the real (p = 0) or imaginary part of the sums and updates of column c (left update) or
// row c (right update) of A, the last 2*NC those of the rows of Z, whose update runs beside
// the left update of A.  Each element's operations are those of one thread per line with complex
// arithmetic.  A is in shared memory where it fits (n <= 116), else in the output buffer.
// Bound: the FP64 pipe (16/3 n^3 + 8/3 n^3 + 8/3 n^3 FMAs); the loads are in batches ahead of the chain.
struct ZHessCtl {
  double2 tau, t;
  double beta;
  int mode;  // 0: nothing to do, 1: reflector ready, 2: rescaling needed
};

// Component p of acc + conj(b) c  /  acc + b c  /  acc - b c, each as zfmac / zfma / zfms.
__device__ __forceinline__ double fmac_p(double2 b, double2 c, double acc, int p) {
  return fma(b.x, p ? c.y : c.x, fma(p ? -b.y : b.y, p ? c.x : c.y, acc));
}
__device__ __forceinline__ double fma_p(double2 b, double2 c, double acc, int p) {
  return fma(b.x, p ? c.y : c.x, fma(p ? b.y : -b.y, p ? c.x : c.y, acc));
}
__device__ __forceinline__ double fms_p(double2 b, double2 c, double acc, int p) {
  return fma(-b.x, p ? c.y : c.x, fma(p ? -b.y : b.y, p ? c.x : c.y, acc));
}

template <int NC>
__global__ void __launch_bounds__(4 * NC) k_hess_cplx(CplxBatch bt, const int* __restrict__ order,
                                                      const int* __restrict__ sched, int bin, int nmax, int cap) {
  constexpr int NT = 4 * NC;
  extern __shared__ double2 smemz[];
  __shared__ double2 cs[NC];  // the reflector
  __shared__ double red[32], gssq[4];
  __shared__ unsigned long long gmax[4];
  __shared__ ZHessCtl hc;
  const double sfmin = kFmin / kEps;
  const int tid = threadIdx.x;
  const int start = sched[3 * bin], end = sched[3 * bin + 1];
  const bool isz = tid >= 2 * NC;
  const int c = (tid % (2 * NC)) >> 1, p = tid & 1;
  // hypot3(ar, ai, xnorm) (util.jl:562-570)
  auto hyp3 = [](double x, double y, double z) {
    const double w = fmax(fabs(x), fmax(fabs(y), fabs(z)));
    if (w == 0.0) return 0.0;
    const double rw = 1.0 / w;
    const double a = x * rw, b = y * rw, d = z * rw;
    return w * sqrt(fma(a, a, fma(b, b, d * d)));
  };
  for (int job = start + blockIdx.x; job < end; job += gridDim.x) {
    const int b = order[job];
    const int n = bt.ns[b];
    if (n <= 0 || n > nmax) continue;  // k_schur_cplx reports it
    double2* Ag = bt.A + bt.offs[b];
    double2* Zg = bt.wantz ? bt.Z + bt.offs[b] : nullptr;
    const bool as = n * (n | 1) <= cap;
    const int ld = as ? (n | 1) : n;
    double2* A = as ? smemz : Ag;
    __syncthreads();  // the previous matrix is out of shared memory
    double amax = 0.0;
    for (int idx = tid; idx < n * n; idx += NT) {
      const int i = idx % n, j = idx / n;
      const double2 a = Ag[idx];
      if (as) A[i + j * ld] = a;
      if (Zg) Zg[idx] = make_double2(i == j ? 1.0 : 0.0, 0.0);
      const double aa = hypot(a.x, a.y);
      amax = (aa > amax || aa != aa) ? aa : amax;
    }
    amax = block_max<NT>(amax, red);
    __syncthreads();
    if (bt.scale) {
      const double smlnum = sqrt(kSafemin) / kEps;
      const double bignum = 1.0 / smlnum;
      double cscale = 0.0;
      if (amax > 0.0 && amax < smlnum) cscale = smlnum;
      else if (amax > bignum) cscale = bignum;
      if (cscale != 0.0) {
        double mul[8];
        const int nf = safescale_factors(amax, cscale, mul);
        for (int f = 0; f < nf; ++f)
          for (int idx = tid; idx < n * n; idx += NT) {
            double2& a = A[idx % n + idx / n * ld];
            a = zscal(a, mul[f]);
          }
        __syncthreads();
      }
    }
    for (int i = 1; i <= n - 1; ++i) {
      const int m = n - i;
      double2* col = A + i + (i - 1) * ld;
      // largest component and sum of squares of the tail: elements 1+32w..32+32w are warp w's, summed
      // by a tree, the warps' sums in order
      const double2 xt = (tid < 128 && 1 + tid < m) ? col[1 + tid] : make_double2(0.0, 0.0);
      if (tid < 128) {
        unsigned long long mb = max((unsigned long long)__double_as_longlong(fabs(xt.x)),
                                    (unsigned long long)__double_as_longlong(fabs(xt.y)));
        double q = fma(xt.x, xt.x, fma(xt.y, xt.y, 0.0));
        for (int o = 16; o > 0; o >>= 1) {
          const unsigned long long w = __shfl_xor_sync(0xffffffffu, mb, o);
          mb = w > mb ? w : mb;
          q += __shfl_xor_sync(0xffffffffu, q, o);
        }
        if ((tid & 31) == 0) { gmax[tid >> 5] = mb; gssq[tid >> 5] = q; }
      }
      __syncthreads();
      const double2 alpha0 = col[0];
      if (tid < 32) {
        unsigned long long mb = gmax[0];
        double ssq = gssq[0];
        for (int w = 1; w < 4; ++w) { mb = gmax[w] > mb ? gmax[w] : mb; ssq += gssq[w]; }
        const double big = __longlong_as_double((long long)mb);
        ZHessCtl h;
        h.tau = h.t = make_double2(0.0, 0.0);
        h.beta = 0.0;
        h.mode = (big == 0.0 && alpha0.y == 0.0) ? 0 : ((big == 0.0 || (big < 1.0e150 && big > 1.0e-150)) ? 1 : 2);
        if (h.mode == 1) {
          const double ar = alpha0.x, ai = alpha0.y;
          h.beta = -copysign(hyp3(ar, ai, big != 0.0 ? sqrt(ssq) : 0.0), ar);
          if (fabs(h.beta) < sfmin) {
            h.mode = 2;
          } else {
            h.tau = make_double2((h.beta - ar) / h.beta, -ai / h.beta);
            h.t = zdiv(make_double2(1.0, 0.0), make_double2(ar - h.beta, ai));
          }
        }
        if (tid == 0) hc = h;
      }
      __syncthreads();
      if (hc.mode == 0) { __syncthreads(); continue; }
      double2 tau = hc.tau, t = hc.t;
      double beta = hc.beta;
      if (hc.mode == 2) {
        // entries outside the range where squaring is safe, or the underflow guard: rescale
        unsigned long long mb = gmax[0];
        for (int w = 1; w < 4; ++w) mb = gmax[w] > mb ? gmax[w] : mb;
        const double big = __longlong_as_double((long long)mb);
        const bool safe = (big < 1.0e150 && big > 1.0e-150);
        double xnorm = 0.0;
        if (big != 0.0) {
          const double sc = safe ? 1.0 : 1.0 / big;
          const double a = xt.x * sc, q = xt.y * sc;
          const double ssq = block_sum<NT>(fma(a, a, fma(q, q, 0.0)), red);
          xnorm = safe ? sqrt(ssq) : big * sqrt(ssq);
        }
        double ar = alpha0.x, ai = alpha0.y;
        beta = -copysign(hyp3(ar, ai, xnorm), ar);
        int kount = 0;
        if (fabs(beta) < sfmin) {
          const double rsfmin = 1.0 / sfmin;
          double bb = beta;
          do { ++kount; bb *= rsfmin; ar *= rsfmin; ai *= rsfmin; } while (fabs(bb) < sfmin && kount < 20);
          __syncthreads();
          double2 v = xt;
          for (int q = 0; q < kount; ++q) v = zscal(v, rsfmin);
          if (tid < 128 && 1 + tid < m) col[1 + tid] = v;
          const double big2 = block_max<NT>(fmax(fabs(v.x), fabs(v.y)), red);
          const double sc2 = big2 > 0.0 ? 1.0 / big2 : 0.0;
          const double a2 = v.x * sc2, q2 = v.y * sc2;
          const double ssq2 = block_sum<NT>(fma(a2, a2, fma(q2, q2, 0.0)), red);
          xnorm = big2 * sqrt(ssq2);
          beta = -copysign(hyp3(ar, ai, xnorm), ar);
        }
        tau = make_double2((beta - ar) / beta, -ai / beta);
        t = zdiv(make_double2(1.0, 0.0), make_double2(ar - beta, ai));
        for (int q = 0; q < kount; ++q) beta *= sfmin;
        __syncthreads();
      }
      if (tid < 128 && 1 + tid < m) {
        const double2 v = zmul(col[1 + tid], t);
        col[1 + tid] = v;
        cs[1 + tid] = v;
      }
      if (tid == 0) col[0] = make_double2(beta, 0.0);
      __syncthreads();
      // lmul!(H', A[i+1:n, i+1:n]) with conj(tau), and rmul!(Z, H): x = Z1 v + z1; z1 -= tau x;
      // Z1 -= tau x v^H
      {
        const bool on = isz ? (Zg && c < n) : c < m;
        double2* x = isz ? Zg + c + i * n : A + i + (i + c) * ld;
        const int st = isz ? n : 1;
        double a = 0.0;
        double2 x0 = make_double2(0.0, 0.0);
        if (on) {
          x0 = x[0];
          a = p ? x0.y : x0.x;
          if (isz) {
#pragma unroll 8
            for (int r = 1; r < m; ++r) a = fma_p(x[r * st], cs[r], a, p);
          } else {
#pragma unroll 8
            for (int r = 1; r < m; ++r) a = fmac_p(cs[r], x[r], a, p);
          }
        }
        // the pair's two parts
        const double o = __shfl_xor_sync(0xffffffffu, a, 1);
        const double2 sv = p ? make_double2(o, a) : make_double2(a, o);
        __syncwarp();  // both lanes of the pair have read their line
        if (on) {
          // va = conj(tau) s for A, s tau for Z
          const double2 va = isz ? zmul(sv, tau) : zmul(zconj(tau), sv);
          double* xp = (double*)x + p;
          xp[0] = (p ? x0.y : x0.x) - (p ? va.y : va.x);
          for (int r0 = 1; r0 < m; r0 += 4) {
            double v[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) v[e] = (r0 + e < m) ? xp[2 * (r0 + e) * st] : 0.0;
#pragma unroll
            for (int e = 0; e < 4; ++e)
              if (r0 + e < m) {
                const double2 q = cs[r0 + e];
                xp[2 * (r0 + e) * st] = fms_p(va, isz ? zconj(q) : q, v[e], p);
              }
          }
        }
      }
      __syncthreads();
      // rmul!(A[:, i+1:n], H): x = A1 v + a1; a1 -= tau x; A1 -= tau x v^H
      {
        const bool on = !isz && c < n;
        double2* x = A + c + i * ld;
        double a = 0.0;
        double2 x0 = make_double2(0.0, 0.0);
        if (on) {
          x0 = x[0];
          a = p ? x0.y : x0.x;
#pragma unroll 8
          for (int q = 1; q < m; ++q) a = fma_p(x[q * ld], cs[q], a, p);
        }
        const double o = __shfl_xor_sync(0xffffffffu, a, 1);
        const double2 sv = p ? make_double2(o, a) : make_double2(a, o);
        __syncwarp();
        if (on) {
          const double2 va = zmul(tau, sv);
          double* xp = (double*)x + p;
          xp[0] = (p ? x0.y : x0.x) - (p ? va.y : va.x);
          for (int r0 = 1; r0 < m; r0 += 4) {
            double v[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) v[e] = (r0 + e < m) ? xp[2 * (r0 + e) * ld] : 0.0;
#pragma unroll
            for (int e = 0; e < 4; ++e)
              if (r0 + e < m) xp[2 * (r0 + e) * ld] = fms_p(va, zconj(cs[r0 + e]), v[e], p);
          }
        }
      }
      __syncthreads();
    }
    __syncthreads();
    if (as)
      for (int idx = tid; idx < n * n; idx += NT) {
        const int i = idx % n, j = idx / n;
        if (i <= j + 1) Ag[idx] = A[i + j * ld];
      }
    if (tid == 0) bt.w[bt.woffs[b]] = make_double2(amax, 0.0);  // for the unscaling
  }
}

// ---------------------------------------------------------------------------------
// Single-shift QR, warp-specialised as the real iteration (schur_batched_real.cu): the chain warp runs the
// deflation scan, the shift, the start row and the chase inside a window around the diagonal, the far
// warps apply the logged reflectors one phase later to the columns right of the window, the rows
// above it and Z, a line per thread.  In the chain warp a pair of lanes holds a column or row, one
// lane its real and one its imaginary part: an FP64 instruction costs the same for 1 or 32 lanes, and
// a step takes 6 for the left update, 6 for the right and 23 for the reflector.
// A sweep that starts below istart is rare: its first step is a chunk of its own, after which the far
// warps also apply the phase that keeps H[k0+1, k0] real to every element (GenericSchur.jl:461-482).
// H stays in the output buffer; only the window of a chunk is in shared memory, so that several
// matrices of any order share an SM's FP64 pipe, which bounds the batch (a packed copy of one
// order-128 matrix filled the SM, whose pipe was then 53% busy: 1824 of them took 980 ms).
// Why: one CTA barrier per step with the near block's complex arithmetic on single lanes and the Z pass
// after each sweep took 98 ms for one matrix of order 128.
struct ZCmd {
  int type;     // 0 nothing, 1 chunk, 2 done
  int ka, nst;  // steps ka .. ka+nst-1
  int jfar;     // first column of the far left updates
  int iend;
  int fix;      // the phase fix-up after step ka
  int tail_on;  // the chunk ends the sweep with a tail phase
  double2 ph, tail;
};
struct ZR {
  double2 t1, v2;
  double t2;
};

constexpr int kZWin = 13;    // most steps of a chunk: kZWin + 3 rows in 16 lane pairs
constexpr int kZChunk = 12;  // steps of a chunk of a longer sweep
constexpr int kZMinChunk = 3;
constexpr int kZLog = 3;     // double2 per step: t1, v2, (t2, 0)
constexpr int kZLogElems = kZLog * (kZWin + 1);
constexpr int kZLd = 17;     // the window: 16 columns of 16 rows at this distance
constexpr int kZWinElems = 16 * kZLd;

template <int NT> __device__ __forceinline__ void zphase_barrier() { asm volatile("bar.sync 1, %0;" ::"n"(NT) : "memory"); }
template <int NT> __device__ __forceinline__ void zfar_barrier() { asm volatile("bar.sync 2, %0;" ::"n"(NT - 32) : "memory"); }

// One reflector on (z0, z1) of a line; left updates use conj(t1) and v2, right ones t1 and conj(v2):
// sy, vy are those with the sign of the imaginary part set.  Returns the finished first element.
__device__ __forceinline__ double2 zslide(const ZR& r, double ty, double vy, double2& z0, double2 z1) {
  const double2 ss = make_double2(fma(z1.x, r.t2, fma(r.t1.x, z0.x, -ty * z0.y)),
                                  fma(z1.y, r.t2, fma(r.t1.x, z0.y, ty * z0.x)));
  const double2 out = zsub(z0, ss);
  z0 = zfms(ss, make_double2(r.v2.x, vy), z1);
  return out;
}

__device__ __forceinline__ ZR ld_zr(const double2* l) { return {l[0], l[1], l[2].x}; }

// The logged reflectors on one line, whose elements are inc apart; returns the last element.
__device__ __forceinline__ double2* zapply_line(double2* p, int inc, const double2* lg, int nst, bool left) {
  double2 z0 = *p;
  int s = 0;
  for (; s + 4 <= nst; s += 4, lg += 4 * kZLog) {
    double2 y[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) y[e] = p[(e + 1) * inc];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const ZR r = ld_zr(lg + e * kZLog);
      p[e * inc] = zslide(r, left ? -r.t1.y : r.t1.y, left ? r.v2.y : -r.v2.y, z0, y[e]);
    }
    p += 4 * inc;
  }
  for (; s < nst; ++s, lg += kZLog) {
    const double2 y0 = p[inc];
    const ZR r = ld_zr(lg);
    *p = zslide(r, left ? -r.t1.y : r.t1.y, left ? r.v2.y : -r.v2.y, z0, y0);
    p += inc;
  }
  *p = z0;
  return p;
}

// 2-element complex reflector (zreflector2_fast) with its independent products on different lanes.
__device__ __forceinline__ ZR chain_zrefl(double2& a, double2 x1, int lane) {
  const unsigned all = 0xffffffffu;
  const double xs = fma(x1.x, x1.x, x1.y * x1.y);
  const double ss = fma(a.x, a.x, fma(a.y, a.y, xs));
  const long long sb = __double_as_longlong(ss);
  const bool triv = ((__double_as_longlong(x1.x) | __double_as_longlong(x1.y) | __double_as_longlong(a.y)) << 1) == 0;
  if (triv || sb <= __double_as_longlong(1.0e-290) || sb >= __double_as_longlong(1.0e290)) {
    const double2 t1 = zreflector2_fast(a, x1);
    return {t1, x1, zmul(t1, x1).x};
  }
  const double y = rsqrt_nr(ss);
  const double aa = fabs(a.x);
  const double sy = copysign(y, a.x);
  // tau = (|Re a| y + 1, Im a sy), s = ss y: lanes 0, 1, 2 (mod 4)
  const int q = lane & 3;
  const double m3 = fma(q == 0 ? aa : (q == 1 ? a.y : ss), q == 1 ? sy : y, q == 0 ? 1.0 : 0.0);
  const double2 tau = make_double2(__shfl_sync(all, m3, 0), __shfl_sync(all, m3, 1));
  const double s = __shfl_sync(all, m3, 2);
  const double dr = a.x + copysign(s, a.x);
  const double r = rcp_nr(fma(dr, dr, a.y * a.y));
  // t = (dr r, -Im a r)
  const double tp = ((lane & 1) ? -a.y : dr) * r;
  const double2 t = make_double2(__shfl_sync(all, tp, 0), __shfl_sync(all, tp, 1));
  // v2 = x1 t by parts
  const double vp = fma(x1.x, (lane & 1) ? t.y : t.x, ((lane & 1) ? x1.y : -x1.y) * ((lane & 1) ? t.x : t.y));
  const double2 v2 = make_double2(__shfl_sync(all, vp, 0), __shfl_sync(all, vp, 1));
  a = make_double2(-copysign(s, a.x), 0.0);
  return {tau, v2, fma(tau.x, v2.x, -tau.y * v2.y)};
}

// Exponent field of a double: 2^(e - 1023) <= |x| < 2^(e - 1022) for a normal x (0 and denormals: 0).
__device__ __forceinline__ int zfield(const double& x) { return (__double2hiint(x) >> 20) & 0x7ff; }
__device__ __forceinline__ int zfield(const double2& x) { return max(zfield(x.x), zfield(x.y)); }

// Whether the deflation test at row k certainly fails: |Re sd| > ulp (|hkk|_1 + |hk1|_1), all of moderate size.
__device__ __forceinline__ bool no_zsplit(const double2& sd, const double2& hkk, const double2& hk1) {
  const int e = zfield(sd.x), m = max(zfield(hkk), zfield(hk1));
  return e > 923 && m > 0 && e > m + 3 - 52;
}
// Whether the start-row test at row mm certainly fails: |h10| |h21| > ulp |h11 - shift|_1 (|h11|_1 + |h22|_1).
__device__ __forceinline__ bool no_zstart(const double& h10, const double& h21, const double2& h11, const double2& h22,
                                          double2 shift) {
  const int e10 = zfield(h10), e21 = zfield(h21), x = max(zfield(h11), zfield(shift)), d = max(zfield(h11), zfield(h22));
  if (min(e10, e21) < 923 || max(max(e10, e21), max(x, d)) > 1223) return false;
  // lhs >= 2^(e10 + e21 - 2 bias); rhs < 2^-52 2^(x - bias + 1 + 2) 2^(d - bias + 1 + 2)
  return e10 + e21 > x + d + 6 - 52;
}

// Chain warp: steps ka..ka+nst-1 inside the window (columns ..wl, rows ka-1..), which is loaded into W and
// stored back.  r: the reflector of step ka on entry, of step ka+nst on return (unless that is past the
// sweep, or fix: the phase fix-up comes before it).
__device__ __forceinline__ void zchase_chunk(double2* H, int n, double2* W, int ka, int nst, int iend, int wl, bool fix,
                                             ZR& r, double2* lg, int lane) {
  // rows ka-1.. of column ka+c at W[c * kZLd]
  const int wr = lane & 15, gr = ka - 1 + wr;  // row of the window, of H
  const bool rin = gr >= 1 && gr <= min(ka + nst + 1, iend);
  for (int c = lane >> 4; c <= wl - ka; c += 2)
    if (rin) async_load(&W[wr + c * kZLd], &HH(gr, ka + c));
  async_wait();
  __syncwarp();
  const unsigned all = 0xffffffffu;
  const int p = lane & 1, e = lane >> 1;
  const int j = min(ka + e, wl);
  const bool colok = ka + e <= wl;
  double2* hc = W + (j - ka) * kZLd + 1;  // H(k, j)
  const int i = ka - 1 + e;
  const bool rowok = i >= 1 && i <= iend;
  double2* p0 = W + e;                    // H(i, k), H(i, k+1)
  double2* p1 = p0 + kZLd;
  double2* hb = W + 2;                    // H(k+1, k)
  for (int s = 0; s < nst; ++s) {
    const int k = ka + s;
    if (lane == 0) { lg[0] = r.t1; lg[1] = r.v2; lg[2] = make_double2(r.t2, 0.0); }
    lg += kZLog;
    {
      const double2 h0 = hc[0], h1 = hc[1];
      const double h0p = p ? h0.y : h0.x, h1p = p ? h1.y : h1.x;
      const double ss = fma(h1p, r.t2, fma(r.t1.x, h0p, (p ? -r.t1.y : r.t1.y) * (p ? h0.x : h0.y)));
      const double so = __shfl_xor_sync(all, ss, 1);
      const double2 sv = p ? make_double2(so, ss) : make_double2(ss, so);
      const double o0 = h0p - ss, o1 = fms_p(sv, r.v2, h1p, p);
      __syncwarp();
      if (colok && j >= k) {
        ((double*)hc)[p] = o0;
        ((double*)(hc + 1))[p] = o1;
      }
    }
    __syncwarp();
    double x;
    {
      const double2 h0 = *p0, h1 = *p1;
      const double h0p = p ? h0.y : h0.x, h1p = p ? h1.y : h1.x;
      const double ss = fma(h1p, r.t2, fma(r.t1.x, h0p, (p ? r.t1.y : -r.t1.y) * (p ? h0.x : h0.y)));
      const double so = __shfl_xor_sync(all, ss, 1);
      const double2 sv = p ? make_double2(so, ss) : make_double2(ss, so);
      x = h0p - ss;
      const double o1 = fms_p(sv, zconj(r.v2), h1p, p);
      __syncwarp();
      if (rowok && i <= k + 2) {
        ((double*)p0)[p] = x;
        ((double*)p1)[p] = o1;
      }
    }
    // column k, rows k+1, k+2: the next reflector
    double2 a = make_double2(__shfl_sync(all, x, 2 * (s + 2)), __shfl_sync(all, x, 2 * (s + 2) + 1));
    const double2 x1 = make_double2(__shfl_sync(all, x, 2 * (s + 3) & 31), __shfl_sync(all, x, (2 * (s + 3) + 1) & 31));
    __syncwarp();
    if (k < iend - 1 && !fix) {
      r = chain_zrefl(a, x1, lane);
      if (lane == 0) { hb[0] = a; hb[1] = make_double2(0.0, 0.0); }
    }
    ++hc;
    hb += kZLd + 1;
    p0 = p1;
    p1 += kZLd;
  }
  __syncwarp();
  for (int c = lane >> 4; c <= wl - ka; c += 2)
    if (rin) HH(gr, ka + c) = W[wr + c * kZLd];
  __syncwarp();
}

// nmax: the largest order the launch sized its buffers for (the bin's maximum, or the
// single large matrix's order).  An order outside [0, nmax] read from device memory gets
// ST_BADARG before anything is read or written.
template <int NT>
__device__ void solve_cplx(const CplxBatch& bt, int b, int nmax, double2* smem, int cw) {
  __shared__ ZCmd cmd[2];
  __shared__ int s_status;
  const int tid = threadIdx.x;
  const int lane = tid & 31, warp = tid >> 5;
  const int n = bt.ns[b];
  if (n <= 0 || n > nmax) {
    if (tid == 0) bt.status[b] = (n == 0) ? ST_OK : ST_BADARG;
    return;
  }
  double2* Ag = bt.A + bt.offs[b];
  double2* Zg = bt.wantz ? bt.Z + bt.offs[b] : nullptr;
  double2* wg = bt.w + bt.woffs[b];
  double2* logs = smem;
  double2* W = smem + 2 * kZLogElems;
  double2* H = Ag;
  // the scale that k_hess_cplx applied
  const double amax = wg[0].x;
  const double smlnum = sqrt(kSafemin) / kEps;
  const double bignum = 1.0 / smlnum;
  bool scaled = false;
  double cscale = 1.0;
  if (bt.scale) {
    if (amax > 0.0 && amax < smlnum) { scaled = true; cscale = smlnum; }
    else if (amax > bignum) { scaled = true; cscale = bignum; }
  }
  for (int j = 1 + tid; j <= n - 2; j += NT) HH(j + 2, j) = make_double2(0.0, 0.0);  // the bulge's row
  __syncthreads();
  const double ulp = kEps;
  const double smallnum = kSafemin * ((double)n / ulp);
  if (warp == cw) {
    // ---- chain warp (all its variables are uniform over the lanes) ----
    const long long maxiter = bt.maxiter_abs > 0 ? bt.maxiter_abs : (long long)bt.maxiter_mult * n;
    const long long maxinner = bt.maxinner_abs > 0 ? bt.maxinner_abs : (long long)bt.maxinner_mult * n;
    long long it = 0, its = 0;
    int status = ST_OK, iend = n, istart = 1;
    int state = 0;              // 0: between sweeps, 1: first chunk of a sweep is next, 2: inside a sweep
    int kn = 0, k0 = 0;
    int pka = 0, pnst = 0, pwl = 0;
    int fka = 0;                // ka of the sweep's last chunk while the far warps apply it
    bool hold = false, fixed = false;  // skip a phase for a phase fix-up; it is done
    ZR r{};
    for (int ph = 0;; ++ph) {
      ZCmd& cm = cmd[ph & 1];
      double2* lg = logs + (ph & 1) * kZLogElems;
      bool done = false;
      while (state == 0 && !hold) {
        if (iend < 1) { done = true; break; }
        if (its > maxinner) { its = 0; istart = 1; }
        ++it;
        if (it > maxiter) { status = ST_UNCONVERGED; done = true; break; }
        // deflation scan (GenericSchur.jl:240-286): largest k in [istart, iend-1] that splits
        int found = 0;
        for (int top = iend - 1; top >= istart; top -= 32) {
          const int k = top - lane;
          bool split = false;
          if (k >= istart) {
            const double2 sd = HH(k + 1, k);
            const double2 hkk = HH(k, k), hk1 = HH(k + 1, k + 1);
            if (no_zsplit(sd, hkk, hk1)) {
              split = false;
            } else if (zabs1(sd) <= smallnum) {
              split = true;
            } else {
              double tst = zabs1(hkk) + zabs1(hk1);
              if (tst == 0.0) {
                if (k - 1 >= 1) tst += fabs(HH(k, k - 1).x);
                if (k + 2 <= n) tst += fabs(HH(k + 2, k + 1).x);
              }
              if (fabs(sd.x) <= ulp * tst) {
                const double2 up = HH(k, k + 1);
                const double ab = fmax(zabs1(sd), zabs1(up)), ba = fmin(zabs1(sd), zabs1(up));
                const double2 df = zsub(hkk, hk1);
                const double aa = fmax(zabs1(hk1), zabs1(df)), bb = fmin(zabs1(hk1), zabs1(df));
                const double s = aa + ab;
                if (ba * (ab / s) <= fmax(smallnum, ulp * (bb * (aa / s)))) split = true;
              }
            }
          }
          const unsigned bal = __ballot_sync(0xffffffffu, split);
          if (bal) { found = top - (__ffs(bal) - 1); break; }
        }
        if (found > 0) istart = found + 1;
        if (istart > 1 && lane == 0) HH(istart, istart - 1) = make_double2(0.0, 0.0);
        __syncwarp();
        if (istart >= iend) {
          iend -= 1;
          istart = 1;
          its = 0;
          continue;
        }
        // shift (GenericSchur.jl:302-325)
        double2 t;
        if (its % 30 == 10) {
          const double s = 0.75 * fabs(HH(istart + 1, istart).x);
          t = zadd(make_double2(s, 0.0), HH(istart, istart));
        } else if (its % 30 == 20) {
          const double s = 0.75 * fabs(HH(iend, iend - 1).x);
          t = zadd(make_double2(s, 0.0), HH(iend, iend));
        } else {
          t = HH(iend, iend);
          // the two square roots on two lanes
          const double2 rt = zsqrt((lane & 1) ? HH(iend, iend - 1) : HH(iend - 1, iend));
          const double2 ra = make_double2(__shfl_sync(0xffffffffu, rt.x, 0), __shfl_sync(0xffffffffu, rt.y, 0));
          const double2 rb = make_double2(__shfl_sync(0xffffffffu, rt.x, 1), __shfl_sync(0xffffffffu, rt.y, 1));
          const double2 u = zmul(ra, rb);
          double s = zabs1(u);
          if (s != 0.0) {
            const double2 x = zscal(zsub(HH(iend - 1, iend - 1), t), 0.5);
            const double sx = zabs1(x);
            s = fmax(s, zabs1(x));
            const double2 xs = zscal(x, 1.0 / s), us = zscal(u, 1.0 / s);
            double2 y = zscal(zsqrt(zadd(zmul(xs, xs), zmul(us, us))), s);
            if (sx > 0.0) {
              const double2 xn = zscal(x, 1.0 / sx);
              if (xn.x * y.x + xn.y * y.y < 0.0) y = zneg(y);
            }
            t = zsub(t, zmul(u, zdiv(u, zadd(x, y))));
          }
        }
        const double2 shift = t;
        // start row (GenericSchur.jl:390-407): largest mm with a negligible product
        k0 = istart;
        for (int top = iend - 1; top >= istart + 1; top -= 32) {
          const int mm = top - lane;
          bool hit = false;
          if (mm >= istart + 1 && !no_zstart(HH(mm, mm - 1).x, HH(mm + 1, mm).x, HH(mm, mm), HH(mm + 1, mm + 1), shift)) {
            const double2 h11 = HH(mm, mm), h22 = HH(mm + 1, mm + 1);
            double2 h11s = zsub(h11, shift);
            double h21 = HH(mm + 1, mm).x;
            const double s = zabs1(h11s) + fabs(h21);
            h11s = zscal(h11s, 1.0 / s);
            h21 /= s;
            const double h10 = HH(mm, mm - 1).x;
            hit = fabs(h10) * fabs(h21) <= ulp * (zabs1(h11s) * (zabs1(h11) + zabs1(h22)));
          }
          const unsigned bal = __ballot_sync(0xffffffffu, hit);
          if (bal) { k0 = top - (__ffs(bal) - 1); break; }
        }
        {
          const double2 h11s = zsub(HH(k0, k0), shift);
          const double h21 = HH(k0 + 1, k0).x;
          const double s = zabs1(h11s) + fabs(h21);
          double2 a = zdiv(h11s, make_double2(s, 0.0)), x1 = make_double2(h21 / s, 0.0);
          r = chain_zrefl(a, x1, lane);
        }
        __syncwarp();
        ++its;
        kn = k0;
        state = 1;
      }
      int type = done ? 2 : 0;
      if (hold) {
        hold = false;   // the far warps apply the phase fix-up in this phase
        fixed = state == 2;
      } else if (!done) {
        if (fixed) {
          // the second reflector of the sweep, from the phased column
          fixed = false;
          double2 a = HH(kn, kn - 1);
          const double2 x1 = HH(kn + 1, kn - 1);
          r = chain_zrefl(a, x1, lane);
          __syncwarp();
          if (lane == 0) { HH(kn, kn - 1) = a; HH(kn + 1, kn - 1) = make_double2(0.0, 0.0); }
          __syncwarp();
        }
        const bool first = state == 1;
        const bool fix = first && k0 > istart;
        // the next chunk: steps kn..kn+nst-1
        int nst = iend - kn;
        if (nst > kZWin) nst = kZChunk;
        if (fix) nst = 1;
        if (first && fka > 0 && kn < fka && min(kn + nst + 1, iend) >= fka) {
          // the far warps are still in columns fka.. above row fka-1
          nst = min(nst, fka - kn - 2);
          if (nst < kZMinChunk) nst = 0;
        }
        if (nst > 0) {
          const int kb = kn + nst - 1;
          const int wl = min(kb + 2, iend);
          if (state == 2 && pnst > 0) {
            // urgent columns: the previous chunk's left updates on the columns entering the window
            const double2* pl = logs + ((ph & 1) ^ 1) * kZLogElems;
            const int j = pwl + 1 + lane;
            if (j <= wl) zapply_line(&HH(pka, j), 1, pl, pnst, true);
            __syncwarp();
          }
          double2 pht = make_double2(1.0, 0.0);
          if (fix) {
            pht = zsub(pht, r.t1);
            pht = zscal(pht, 1.0 / hypot(pht.x, pht.y));
          }
          zchase_chunk(H, n, W, kn, nst, iend, wl, fix, r, lg, lane);
          if (fix) {
            if (lane == 0) {
              HH(kn + 1, kn) = zmul(HH(kn + 1, kn), zconj(pht));
              if (kn + 2 <= iend) HH(kn + 2, kn + 1) = zmul(HH(kn + 2, kn + 1), pht);
            }
            __syncwarp();
          }
          const bool last = kb == iend - 1;
          int jfar = wl + 1;
          if (!last && !fix) {
            int nn = iend - kb - 1;
            if (nn > kZWin) nn = kZChunk;
            jfar = min(kb + nn + 2, iend) + 1;  // beyond the next chunk's window
          }
          int tail_on = 0;
          double2 tail = make_double2(1.0, 0.0);
          if (last) {
            // tail: keep H[iend, iend-1] real (GenericSchur.jl:486-500)
            const double2 tt = HH(iend, iend - 1);
            __syncwarp();
            if (tt.y != 0.0) {
              const double rt = hypot(tt.x, tt.y);
              if (lane == 0) HH(iend, iend - 1) = make_double2(rt, 0.0);
              tail = zscal(tt, 1.0 / rt);
              tail_on = 1;
              const int rr = max(kn - 1, 1) + lane;
              if (rr <= iend - 1 && !fix) HH(rr, iend) = zmul(HH(rr, iend), tail);
            }
            __syncwarp();
          }
          if (lane == 0) {
            cm.ka = kn;
            cm.nst = nst;
            cm.jfar = jfar;
            cm.iend = iend;
            cm.fix = fix;
            cm.ph = pht;
            cm.tail_on = tail_on;
            cm.tail = tail;
          }
          type = 1;
          pka = kn; pnst = fix ? 0 : nst; pwl = wl;
          kn = kb + 1;
          fka = last && !fix ? pka : 0;
          state = last ? 0 : 2;
          hold = fix;
        } else {
          fka = 0;  // this phase's barrier ends the far work
        }
      }
      if (lane == 0) cm.type = type;
      zphase_barrier<NT>();
      if (done) break;
    }
    if (lane == 0) s_status = status;
  } else {
    // ---- far warps ----
    const int ft = tid - (warp > cw ? 32 : 0);
    for (int ph = 0;; ++ph) {
      if (ph > 0 && cmd[(ph - 1) & 1].type == 1) {
        const ZCmd& cm = cmd[(ph - 1) & 1];
        const double2* lg = logs + ((ph - 1) & 1) * kZLogElems;
        const int ka = cm.ka, nst = cm.nst, jfar = cm.jfar, tail_on = cm.tail_on;
        const double2 tail = cm.tail;
        const int nl = n - jfar + 1, nr = max(ka - 2, 0), nz = Zg ? n : 0;
        for (int t = ft; t < nl + nr + nz; t += NT - 32) {
          double2* p;
          int inc;
          const bool left = t < nl;
          if (left) {
            p = &HH(ka, jfar + t);
            inc = 1;
          } else if (t < nl + nr) {
            p = &HH(t - nl + 1, ka);
            inc = n;
          } else {
            p = Zg + (t - nl - nr) + (ka - 1) * n;
            inc = n;
          }
          p = zapply_line(p, inc, lg, nst, left);
          if (tail_on && !cm.fix) *p = zmul(*p, left ? zconj(tail) : tail);
        }
        if (cm.fix) {
          // the phase (GenericSchur.jl:461-482) on rows ka, ka+2..iend right of the diagonal and its
          // conjugate on columns ka, ka+2..iend above it, then the tail phase; the same on Z
          zfar_barrier<NT>();
          const int ie = cm.iend, fw = ft >> 5;
          const double2 ph1 = cm.ph, ph2 = zconj(cm.ph);
          for (int c = ka + fw; c <= n; c += NT / 32 - 1)
            for (int q = 1 + lane; q < c; q += 32) {
              double2 v = HH(q, c);
              if (c > ka && q >= ka && q <= ie && q != ka + 1) v = zmul(v, ph1);
              if (c <= ie && c != ka + 1) v = zmul(v, ph2);
              if (tail_on && q == ie) v = zmul(v, zconj(tail));
              if (tail_on && c == ie) v = zmul(v, tail);
              HH(q, c) = v;
            }
          if (Zg)
            for (int c = ka + fw; c <= ie; c += NT / 32 - 1)
              for (int q = lane; q < n; q += 32) {
                double2* z = Zg + q + (c - 1) * n;
                if (c != ka + 1) *z = zmul(*z, ph2);
                if (tail_on && c == ie) *z = zmul(*z, tail);
              }
        }
      }
      zphase_barrier<NT>();
      if (cmd[ph & 1].type == 2) break;
    }
  }
  __syncthreads();
  const int status = s_status;

  // ---- write back ----
  double mul[8];
  int nf = 0;
  if (scaled) nf = safescale_factors(cscale, amax, mul);
  for (int idx = tid; idx < n * n; idx += NT) {
    const int i = idx % n, j = idx / n;
    double2 v = (i > j) ? make_double2(0.0, 0.0) : Ag[idx];
    for (int f = 0; f < nf; ++f) v = zscal(v, mul[f]);
    Ag[idx] = v;
    if (i == j) wg[i] = v;
  }
  if (tid == 0) bt.status[b] = status;
  __syncthreads();
}
#undef HH

// All matrices of a batch of a few per SM in one launch, whatever their bin, after all reductions.  The time of such
// a batch is that of its largest matrices and of what shares an SM with them.  The bins' own launches left that
// to chance: a bin's CTAs went where the next one's reductions were done first, four of the largest to an
// SM (600 matrices of orders 8 to 128 114 to 117 ms, 101 to 135 with a persistent CTA per SM before).  Here
// the sorted order is dealt to the SMs in rounds of num_sms, every other round backwards, so that the
// largest shares its SM with the smallest; between two and four per SM the shared memory asked for keeps two
// at a time, the rest as they end: 600 99 to 101 ms, 500 96 to 101 (104 to 118; 98 to 103), 304 of 112 to
// 128 115 (150; 178).  With four at a time 600 take 111 to 114, 500 100 to 107.
__global__ void __launch_bounds__(128, 4) k_schur_cplx_all(CplxBatch bt, const int* __restrict__ order, int num_sms) {
  extern __shared__ double2 smemz[];
  const int round = blockIdx.x / num_sms, at = blockIdx.x % num_sms;
  const int job = round * num_sms + (round & 1 ? num_sms - 1 - at : at);
  if (job < bt.count) solve_cplx<128>(bt, order[job], kSmallMax, smemz, round & 3);
}

template <int NT>
__global__ void __launch_bounds__(NT, NT <= 128 ? 512 / NT : 2) k_schur_cplx(CplxBatch bt, const int* __restrict__ order,
                                                                int* __restrict__ sched, int bin, int nmax,
                                                                int num_sms, int once) {
  extern __shared__ double2 smemz[];
  __shared__ int s_job;
  const int start = sched[3 * bin], end = sched[3 * bin + 1];
  // the chain warps of an SM's CTAs on different sub-partitions (as in schur_batched_real.cu)
  constexpr int NW = NT / 32;
  const int slot = blockIdx.x / num_sms;
  const int cw = NW % 4 == 0 ? slot % 4 : (NW % 2 == 0 ? (slot >> 1) & 1 : 0);
  if (once) {  // a CTA per matrix
    const int job = start + blockIdx.x;
    if (job < end) solve_cplx<NT>(bt, order[job], nmax, smemz, cw);
    return;
  }
  for (;;) {
    if (threadIdx.x == 0) s_job = start + atomicAdd(&sched[3 * bin + 2], 1);
    __syncthreads();
    const int job = s_job;
    __syncthreads();
    if (job >= end) break;
    solve_cplx<NT>(bt, order[job], nmax, smemz, cw);
  }
}

// Dynamic shared memory of one CTA of the iteration and of the reduction for orders up to nmax.
size_t ciqr_smem_bytes() { return sizeof(double2) * (2 * kZLogElems + kZWinElems); }
size_t chess_smem_elems(int nmax) {
  const size_t one = (size_t)nmax * (nmax | 1), most = kMostSmem / sizeof(double2);
  return one <= most ? one : most;
}

template <int NC>
cudaError_t launch_hess_c(const CplxBatch& bt, const int* order, const int* sched, int bin, int nmax, int num_sms,
                          cudaStream_t s) {
  const size_t elems = chess_smem_elems(nmax), smem = sizeof(double2) * elems;
  cudaError_t e = allow_smem(k_hess_cplx<NC>, sizeof(double2) * chess_smem_elems(NC));
  if (e != cudaSuccess) return e;
  k_hess_cplx<NC><<<bin_grid(bt.count, num_sms, kReduceCtas), 4 * NC, smem, s>>>(bt, order, sched, bin, nmax, (int)elems);
  return cudaGetLastError();
}

template <int NT>
cudaError_t launch_bin_c(const CplxBatch& bt, const int* order, int* sched, int bin, int nmax, int ctas, int num_sms,
                         cudaStream_t s, bool iterate) {
  cudaError_t e = nmax <= 32 ? launch_hess_c<32>(bt, order, sched, bin, nmax, num_sms, s)
                             : (nmax <= 64 ? launch_hess_c<64>(bt, order, sched, bin, nmax, num_sms, s)
                                           : launch_hess_c<128>(bt, order, sched, bin, nmax, num_sms, s));
  if (e != cudaSuccess || !iterate) return e;
  const size_t smem = ciqr_smem_bytes();
  e = allow_smem(k_schur_cplx<NT>, smem);
  if (e != cudaSuccess) return e;
  // as launch_bin of schur_batched_real.cu
  int grid = bin_grid(bt.count, num_sms, kIterCtas64);
  const int once = ctas == 0 && grid == bt.count;
  if (ctas > 0) {
    int per_sm = 0;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_schur_cplx<NT>, NT, smem);
    if (e != cudaSuccess) return e;
    grid = std::min(bt.count, num_sms * std::min(std::max(per_sm, 1), ctas));
  }
  k_schur_cplx<NT><<<grid, NT, smem, s>>>(bt, order, sched, bin, nmax, num_sms, once);
  return cudaGetLastError();
}

// One bin with the requested thread count (kTuneThreads).
cudaError_t launch_shape_c(const CplxBatch& bt, const int* order, int* sched, int bin, int nmax, int nt, int ctas,
                           int num_sms, cudaStream_t s, bool iterate = true) {
#define GS_SHAPE(NTV) \
  if (nt == NTV) return launch_bin_c<NTV>(bt, order, sched, bin, nmax, ctas, num_sms, s, iterate);
  GS_SHAPE(64) GS_SHAPE(96) GS_SHAPE(128) GS_SHAPE(160) GS_SHAPE(192) GS_SHAPE(256)
#undef GS_SHAPE
  return cudaErrorInvalidValue;
}

}  // namespace

cudaError_t launch_schur_cplx_all(const CplxBatch& bt, const int* order, int num_sms, cudaStream_t s) {
  const int grid = (bt.count + num_sms - 1) / num_sms * num_sms;
  const size_t pair = 100 * 1024;
  const size_t smem = bt.count > 2 * num_sms && bt.count <= 4 * num_sms ? pair : ciqr_smem_bytes();
  cudaError_t e = allow_smem(k_schur_cplx_all, pair, smem);
  if (e != cudaSuccess) return e;
  k_schur_cplx_all<<<grid, 128, smem, s>>>(bt, order, num_sms);
  return cudaGetLastError();
}

cudaError_t launch_schur_batched_cplx_tuned(const CplxBatch& bt, const int* order, int* sched, int num_sms,
                                            cudaStream_t* streams, int nstreams, const BinTuning& t, bool iterate) {
  // largest bin first: it carries most of the work
  for (int i = 0; i < kNumBins; ++i) {
    const int bin = kNumBins - 1 - i;
    if (bt.empty >> bin & 1) continue;
    cudaError_t e = launch_shape_c(bt, order, sched, bin, t.bounds[bin], t.nt[bin], t.ctas[bin], num_sms,
                                   streams[i % nstreams], iterate);
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

cudaError_t launch_schur_batched_cplx(const CplxBatch& bt, const int* order, int* sched, int num_sms,
                                      cudaStream_t* streams, int nstreams) {
  return launch_schur_batched_cplx_tuned(bt, order, sched, num_sms, streams, nstreams, default_tuning_cplx());
}

// A tuning row's hsmem flag selects nothing any more (the reduction runs in shared memory where the
// matrix fits); a row that asks for it where a full matrix does not fit is refused as before.
size_t cplx_bin_smem_bytes(int nmax, int hsmem) {
  const size_t full = hsmem ? sizeof(double2) * ((size_t)nmax * (nmax | 1) + 4 * (size_t)nmax) + 32 * sizeof(double) + 64 : 0;
  return full > ciqr_smem_bytes() ? full : ciqr_smem_bytes();
}

cudaError_t launch_schur_cplx_bin(const CplxBatch& bt, const int* order, int* sched, int bin, const BinTuning& t,
                                  int num_sms, cudaStream_t s) {
  return launch_shape_c(bt, order, sched, bin, t.bounds[bin], t.nt[bin], t.ctas[bin], num_sms, s);
}

cudaError_t launch_schur_cplx_one(const CplxBatch& bt, int m, const int* order, int* sched, cudaStream_t s) {
  const BinTuning t = default_tuning_cplx();
  const int bin = default_bin_of(m);
  return launch_shape_c(bt, order, sched, bin, t.bounds[bin], t.nt[bin], 1, 1, s);
}

}  // namespace gsk
