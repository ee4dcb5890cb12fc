// FP64-accurate matrix products of the batched mixed-precision refinement on the BF16
// tensor cores (tcgen05), one CTA per matrix of order n <= 128.
//
// Every Newton step of the refinement (refine_batched.cu) needs three products whose
// small parts carry the signal and which therefore must be accurate to FP64 rounding:
//   P  = A_s Z                      (A_s = A 2^-e, the unit-scaled input),
//   At = Z^T P                      (its block-lower part is the Schur residual),
//   G  = Z^T Z                      (N = (I - G) / 2 is the orthogonality correction).
// On GB300 the FP64 pipe runs about 1.2 TFLOP/s while the BF16 tensor cores run about
// 2 PFLOP/s, so these products use the error-free splitting of Ozaki, Ogita, Oishi and
// Rump (Numer. Algorithms 59, 2012) in the tensor-core form of Mukunoki, Ozaki, Ogita and
// Imamura (ISC 2020), sized for n <= 128:
//   * row i of op(X) is scaled by 2^e_i with max_k |x_ik| < 2^e_i, column j of Y by 2^f_j;
//   * the scaled entries are cut into S = 8 slices of 7 bits (56 bits, exact up to the
//     last slice): x = 2^e sum_s q_s 2^{-7 s}, |q_s| <= 127, each slice a BF16 integer;
//   * a slice product summed over k <= 128 is at most 127^2 * 128 < 2^21, and the up to 8
//     slice products of one level s + t add up to less than 2^24, so the tensor core's
//     FP32 accumulation of a whole level is exact in any order;
//   * C_ij = 2^{e_i + f_j} sum_{s + t <= 9} 2^{-7 (s + t)} (level sums), the 8 exact level
//     sums converted to FP64 and added least significant first.  The truncation (2^-56
//     of the row maximum) and the dropped levels (s + t >= 10) stay below the rounding
//     error of an FP64 dot product of the same length.
//
// Kernel k_refine_tc: persistent CTAs of 512 threads (one per SM: the eight level
// accumulators fill the SM's 512 TMEM columns), each taking the matrices still being
// refined from a ticket counter, largest first.  Per product, per 64-column panel of Y:
// chunks of 32 contraction indices are split straight into shared memory
// in the tensor core's canonical K-major layout (no swizzle; 8 x 8 core matrices of 128
// contiguous bytes, K-adjacent core matrices 128 B apart, 8-row groups 512 B apart),
// double-buffered so that one chunk is split while the MMAs of the previous one run: a
// thread of warp 0 issues the 36 slice products per 16-wide K step (tcgen05.mma, M = 128,
// N = 64, K = 16) into the accumulator of their level, and the other fifteen warps split
// (with thread 0 also splitting and a CTA barrier per chunk, the issue of 72 MMAs, which
// read 6 KiB of shared memory each, came on top of the split: the products of 20000
// matrices of orders 8 to 128 36.2 -> 31.6 ms);
// after the panel's last chunk the
// sixteen warps (four per TMEM lane quarter, 16 columns each) drain the levels with
// tcgen05.ld.  Every wait is bounded: a timeout hands the matrix to the FP64 kernel
// (status kStFallback), records the error, waits for the CTA's MMAs, frees TMEM and ends
// the CTA.
#include <cstdint>

#include "refine_batched.cuh"
#include "tc_common.cuh"

namespace gsk {
namespace {

using namespace tc;

constexpr int kQBits = 7;                          // bits per slice
constexpr int kQSlices = 8;                        // slices per operand (56 bits)
constexpr int kQLevels = 8;                        // levels s + t = 0 .. 7 (0-based slices)
constexpr int kQM = 128;                           // MMA M (rows of op(X), zero-padded)
constexpr int kQN = 64;                            // MMA N: panel width of Y
constexpr int kQK = 32;                            // contraction indices per chunk
constexpr int kQThreads = 512;
constexpr int kQXSlice = kQM * kQK * 2;            // bytes of one X slice of a chunk (8 KiB)
constexpr int kQYSlice = kQN * kQK * 2;            // bytes of one Y slice of a chunk (4 KiB)
constexpr int kQStage = kQSlices * (kQXSlice + kQYSlice);  // 96 KiB
constexpr int kQD = 8;                             // columns that a warp drains at once (spills 368 bytes, 1020 with 16)
constexpr int kQSbo = (kQK / 8) * 128;             // bytes between 8-row groups
constexpr uint32_t kQIdesc = idesc_bf16(kQM, kQN);
constexpr int kQExpZero = kExpZeroRow;             // row / column of zeros
constexpr int kQExpBad = kExpBadRow;               // row / column with Inf or NaN
constexpr unsigned long long kQTimeout = 4000000000ull;  // ~2 s of SM clock
#ifndef GS_TC_WAIT_CYCLES  // limit of the pipeline's waits (a test builds with 0)
#define GS_TC_WAIT_CYCLES kQTimeout
#endif
constexpr unsigned long long kQWait = GS_TC_WAIT_CYCLES;

struct QCtl {
  uint64_t bar[2];     // MMA completion per stage (tcgen05.commit)
  uint64_t done;       // every MMA of the CTA complete (before TMEM is freed)
  uint32_t tslot;
  int ticket;
  int fail;
  unsigned passed;     // chunks whose stage the issuing warp has seen full
  int exA[kQM];        // row exponents of A (the rows of op(X) in A_s Z)
  int exZ[kQM];        // column exponents of Z (rows of Z^T, columns of Z)
  int exP[kQM];        // column exponents of P = A_s Z
};

constexpr size_t kQSmem = 2 * (size_t)kQStage + sizeof(QCtl) + 128;

// floor(|x| 2^(56 - e)) for |x| < 2^e (so below 2^56), from the IEEE bits; its 7-bit
// groups are the slices of |x| 2^-e.
__device__ __forceinline__ unsigned long long fixed56(double x, int e) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(x) & 0x7fffffffffffffffull;
  const int be = (int)(b >> 52);
  if (b == 0ull) return 0ull;
  const unsigned long long m = (b & 0xfffffffffffffull) | (be ? (1ull << 52) : 0ull);
  const int ex = be ? be - 1075 : -1074;  // |x| = m 2^ex
  const int sh = ex + 56 - e;             // <= 3
  if (sh >= 0) return m << sh;
  return sh <= -64 ? 0ull : (m >> (-sh));
}

// (hs 2^28 + ls) 2^e rounded to nearest even, |hs|, |ls| < 2^47: what
// ldexp(fma((double)hs, 2^28, (double)ls), e) gives, by integer operations.  The drain is
// every element of every product, and the FP64 pipe takes 19 cycles a warp for each of its
// conversions and operations: with those the products of 20000 matrices of orders 8 to 128
// took 50 ms, with integers 40.6 (and 36.2 with the levels read by float-to-int conversions
// and only the rows split that reach an output).
__device__ __forceinline__ double level_sum(long long hs, long long ls, int e) {
  long long t = hs + (ls >> 28);
  unsigned l = (unsigned)ls & 0xfffffffu;
  const bool neg = t < 0;
  if (neg) {
    t = -t - (l != 0u);
    l = (0u - l) & 0xfffffffu;
  }
  if (t == 0 && l == 0u) return 0.0;
  // the magnitude's leading 64 bits: m 2^sh, with what fell off in `rest`
  const int sh = max(0, 28 - __clzll(t));  // t has at most 47 bits
  unsigned long long m = ((unsigned long long)t << (28 - sh)) | (l >> sh);
  const bool rest = (l & ((1u << sh) - 1u)) != 0u;
  const int z = __clzll((long long)m);
  m <<= z;
  unsigned long long q = m >> 11;
  const unsigned low = ((unsigned)m & 2047u) | (rest ? 1u : 0u);
  q += (low > 1024u || (low == 1024u && (q & 1u))) ? 1u : 0u;
  const int be = 1023 + 63 + sh - z + e;  // biased exponent of 2^63 2^(sh - z + e)
  if (be < 1 || be > 2045) {
    const double r = ldexp(fma((double)hs, 0x1p28, (double)ls), e);
    return r;
  }
  const unsigned long long bits = ((unsigned long long)(unsigned)be << 52) + (q - (1ull << 52));
  return __longlong_as_double((long long)(bits | (neg ? 1ull << 63 : 0ull)));
}

// (float)(r 2^-h), h = 0 or 1, by integer operations where the result is normal.
__device__ __forceinline__ float f32_of(double r, int h) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(r);
  const int be = (int)((b >> 52) & 2047u) - h;
  if (be < 1023 - 126 || be > 1023 + 126) return (float)(h ? 0.5 * (0.0 + r) : r);
  const unsigned rem = (unsigned)b & 0x1fffffffu;
  unsigned f = ((unsigned)(be - 896) << 23) + (unsigned)((b & 0xfffffffffffffull) >> 29);
  f += (rem > 0x10000000u || (rem == 0x10000000u && (f & 1u))) ? 1u : 0u;
  return __uint_as_float(f | ((unsigned)(b >> 32) & 0x80000000u));
}

// Two 7-bit integers q0, q1 (< 128) as a packed BF16 pair (q0 low), exact: in FP32,
// (2^23 + q) - 2^23 = q, and the upper 16 bits of an FP32 integer below 2^8 are its BF16.
__device__ __forceinline__ unsigned bf16x2_q(unsigned q0, unsigned q1) {
  const float f0 = __uint_as_float(0x4B000000u | q0) - 8388608.f;
  const float f1 = __uint_as_float(0x4B000000u | q1) - 8388608.f;
  return __byte_perm(__float_as_uint(f0), __float_as_uint(f1), 0x7632);
}

// Eight values of one row (op(X) row i, or Y column j) at k0 .. k0 + 7 -> the 16-byte
// core-matrix row of each slice, at `dst` + s * slice_bytes.  The 56-bit fixed-point
// magnitudes are held as two 28-bit halves of four slices each; the sign is applied to
// every slice.
__device__ __forceinline__ void split8(const double (&v)[8], int e, unsigned char* dst, int slice_bytes) {
  unsigned hi[8], lo[8], sg[4];
  const bool live = e != kQExpZero && e != kQExpBad;
#pragma unroll
  for (int x = 0; x < 8; ++x) {
    const unsigned long long f = live ? fixed56(v[x], e) : 0ull;
    hi[x] = (unsigned)(f >> 28);
    lo[x] = (unsigned)f & 0xfffffffu;
  }
#pragma unroll
  for (int x = 0; x < 4; ++x) {
    const unsigned n0 = (unsigned)(((unsigned long long)__double_as_longlong(v[2 * x])) >> 63);
    const unsigned n1 = (unsigned)(((unsigned long long)__double_as_longlong(v[2 * x + 1])) >> 63);
    sg[x] = (n0 << 15) | (n1 << 31);
  }
#pragma unroll
  for (int s = 0; s < kQSlices; ++s) {
    const int sh = 21 - kQBits * (s & 3);
    unsigned w[4];
#pragma unroll
    for (int x = 0; x < 4; ++x) {
      const unsigned a0 = ((s < 4 ? hi[2 * x] : lo[2 * x]) >> sh) & 127u;
      const unsigned a1 = ((s < 4 ? hi[2 * x + 1] : lo[2 * x + 1]) >> sh) & 127u;
      w[x] = bf16x2_q(a0, a1) ^ sg[x];
    }
    *reinterpret_cast<uint4*>(dst + s * slice_bytes) = make_uint4(w[0], w[1], w[2], w[3]);
  }
}

__device__ __forceinline__ void zero8(unsigned char* dst, int slice_bytes) {
#pragma unroll
  for (int s = 0; s < kQSlices; ++s) *reinterpret_cast<uint4*>(dst + s * slice_bytes) = make_uint4(0u, 0u, 0u, 0u);
}

// A stage is full: the splitting warps arrive, the issuing warp waits.  A stage's second arrival
// follows a wait for the MMAs that its first one released, or, once a wait has timed out, the issuing
// warp's count, so arrivals never mix: the barrier counts threads, and with the arrivals of two chunks in
// one phase the issuing warp could wait for ever.
__device__ __forceinline__ void named_sync(int id, int count) {
  asm volatile("barrier.cta.sync %0, %1;" ::"r"(id), "r"(count) : "memory");
}
__device__ __forceinline__ void named_arrive(int id, int count) {
  asm volatile("barrier.cta.arrive %0, %1;" ::"r"(id), "r"(count) : "memory");
}

// One product C = op(X) Y of n x n column-major FP64 matrices with the exponents of the
// rows of op(X) in ex and of the columns of Y in fy.  XT = 0: op(X) = X, XT = 1:
// op(X) = X^T.  KIND 0: P = C 2^extra; KIND 1: Q = C, F = fp32(C); KIND 2:
// F = fp32((I - C) / 2).  Returns false after a timed-out wait (the CTA must stop).
template <int XT, int KIND>
__device__ bool tc_product(int n, const double* X, const double* Y, const int* ex, const int* fy, int extra,
                           double* Cd, float* Cf, unsigned char* smem, QCtl& ctl, uint32_t tmem,
                           unsigned& gchunk) {
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int nchunks = (n + kQK - 1) / kQK;
  const uint32_t s0 = smem_u32(smem);
  const auto vfail = [&]() { return *(volatile int*)&ctl.fail != 0; };
  // one thread: the MMAs of chunk c, in stage st, of the panel at column j0
  const auto issue = [&](int c, int st, int j0) {
    tc_fence_after();
    const uint32_t xa = s0 + st * kQStage;
    const uint32_t ya = KIND == 2 ? xa + (j0 >> 3) * kQSbo : xa + kQSlices * kQXSlice;
    constexpr int kBSlice = KIND == 2 ? kQXSlice : kQYSlice;
    const uint64_t adesc = smem_desc(xa, 128, kQSbo), bdesc = smem_desc(ya, 128, kQSbo);
    // the 36 slice pairs (s, t), s + t = L <= 7, into the accumulator of level L; the
    // level's first pair at the panel's first K step overwrites it (descriptor start
    // addresses are in units of 16 bytes)
#pragma unroll
    for (int L = 0; L < kQLevels; ++L) {
#pragma unroll
      for (int s = 0; s <= L; ++s) {
#pragma unroll
        for (int kk = 0; kk < kQK / 16; ++kk) {
          const uint32_t acc = (c > 0 || kk > 0 || s > 0) ? 1u : 0u;
          tc_mma(tmem + (uint32_t)(L * kQN), adesc + (uint64_t)((s * kQXSlice + kk * 256) >> 4),
                 bdesc + (uint64_t)(((L - s) * kBSlice + kk * 256) >> 4), kQIdesc, acc);
        }
      }
    }
    tc_commit(&ctl.bar[st]);
  };
  for (int j0 = 0; j0 < n; j0 += kQN) {
    for (int c = 0; c < nchunks; ++c, ++gchunk) {
      const int st = gchunk & 1;
      if (warp == 0) {
        // the issuing warp: every splitting warp has filled the stage
        named_sync(1 + st, kQThreads);
        if (lane == 0) {
          *(volatile unsigned*)&ctl.passed = gchunk + 1;
          if (!vfail()) issue(c, st, j0);
        }
        __syncwarp();
        continue;
      }
      // the MMAs that last read this stage must be complete before it is overwritten
      if (lane == 0 && gchunk >= 2) {
        if (!vfail() && !mbar_wait(&ctl.bar[st], ((gchunk >> 1) - 1) & 1u, kQWait)) *(volatile int*)&ctl.fail = 1;
        if (vfail()) {
          // (ends as soon as the slowest splitting warp's own wait does)
          const unsigned long long t0 = clock64();
          while (*(volatile unsigned*)&ctl.passed < gchunk - 1 && clock64() - t0 <= 4 * kQTimeout) __nanosleep(200);
        }
      }
      __syncwarp();
      unsigned char* xs = smem + st * kQStage;
      const int k0 = c * kQK;
      // items: (row of op(X) or column of Y) x 4 groups of 8 k, only those that reach a stored
      // output, dealt to all threads (by fixed rows, an order of 72 left every fourth warp,
      // and with it a scheduler, without work); contraction indices beyond n are zero in
      // both operands.  In Z^T Z the columns of Y are rows of op(X): split once.
      const int x0 = KIND == 2 ? j0 : 0, nx = n - x0;
      const int nrow = nx + (KIND == 2 ? 0 : min(kQN, n - j0));
      constexpr int kPer = ((kQM + (KIND == 2 ? 0 : kQN)) * (kQK / 8) + kQThreads - 33) / (kQThreads - 32);
      double v[kPer][8];
      int eit[kPer], sb[kPer];
      int dst[kPer];  // byte offset in the stage
#pragma unroll
      for (int u = 0; u < kPer; ++u) {
        const int it = tid - 32 + u * (kQThreads - 32);
        const int kg = it / nrow, r = it - kg * nrow;
        sb[u] = 0;
        if (kg >= kQK / 8) continue;
        const bool isx = r < nx;
        const int slot = isx ? x0 + r : r - nx;  // row of the stage's X or Y part
        const int row = isx ? slot : j0 + slot;  // row of op(X) or column of Y
        sb[u] = isx ? kQXSlice : kQYSlice;
        dst[u] = (isx ? 0 : kQSlices * kQXSlice) + (((slot >> 3) * (kQK / 8) + kg) * 64 + (slot & 7) * 8) * 2;
        const int kb = k0 + kg * 8;
        eit[u] = kb < n ? (isx ? ex[row] : fy[row]) : kQExpZero;
#pragma unroll
        for (int x = 0; x < 8; ++x) {
          const int k = kb + x;
          double val = 0.0;
          if (k < n) {
            if (isx) val = XT ? X[(size_t)row * n + k] : X[(size_t)k * n + row];
            else val = Y[(size_t)row * n + k];
          }
          v[u][x] = val;
        }
      }
#pragma unroll
      for (int u = 0; u < kPer; ++u) {
        if (sb[u] == 0) continue;
        if (eit[u] == kQExpZero) zero8(xs + dst[u], sb[u]);
        else split8(v[u], eit[u], xs + dst[u], sb[u]);
      }
      fence_proxy_async_smem();
      __syncwarp();
      named_arrive(1 + st, kQThreads);
    }
    // drain the panel: the last chunk's commit covers every MMA before it
    if (tid == 0 && !vfail()) {
      const unsigned last = gchunk - 1;
      if (!mbar_wait(&ctl.bar[last & 1], (last >> 1) & 1u, kQWait)) *(volatile int*)&ctl.fail = 1;
    }
    __syncthreads();
    if (ctl.fail) return false;
    tc_fence_after();
    {
      const int q = warp & 3, cq = warp >> 2;  // TMEM lane quarter, 16-column quarter of the panel
      const int i = q * 32 + lane;
      const int ei = i < n ? ex[i] : 0;
#pragma unroll 1
      for (int jl = cq * 16; jl < cq * 16 + 16; jl += kQD) {
        const int jb = j0 + jl;
        // G = Z^T Z is symmetric: only the lower triangle is formed (and mirrored)
        if (jb >= n || q * 32 >= n || (KIND == 2 && q * 32 + 32 <= jb)) break;  // warp-uniform
        // the eight exact level sums as integers: level L is at most (L + 1) 127^2 128, so two
        // levels make one 32-bit integer (128 v6 + v7 < 2^31) and four a 64-bit one
        long long hs[kQD], ls[kQD];
        const uint32_t tb = tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)jl;
#pragma unroll
        for (int h = 0; h < 2; ++h) {  // most significant levels first
          int p[kQD];
#pragma unroll
          for (int g = 0; g < 2; ++g) {
            uint32_t v0[kQD], v1[kQD];
            tc_ld8(tb + (4 * h + 2 * g) * kQN, v0);
            tc_ld8(tb + (4 * h + 2 * g + 1) * kQN, v1);
            tc_wait_ld();
#pragma unroll
            for (int x = 0; x < kQD; ++x) {
              const int w = __float2int_rn(__uint_as_float(v0[x])) * 128 + __float2int_rn(__uint_as_float(v1[x]));
              if (g == 0) p[x] = w;
              else (h == 0 ? hs : ls)[x] = (long long)p[x] * 16384 + w;
            }
          }
        }
        if (i < n) {
#pragma unroll
          for (int x = 0; x < kQD; ++x) {
            const int j = jb + x;
            if (j < n && (KIND != 2 || i >= j)) {
              const int fj = fy[j];
              double r;
              if (ei == kQExpBad || fj == kQExpBad) r = __longlong_as_double(0x7ff8000000000000ll);
              else if (ei == kQExpZero || fj == kQExpZero) r = 0.0;
              else {
                // sum_L lev_L 2^(-7 L) = hs 2^-21 + ls 2^-49, times 2^(e_i + f_j - 14)
                r = level_sum(hs[x], ls[x], ei + fj - 2 * kQBits - 49 + (KIND == 0 ? extra : 0));
              }
              const size_t o = (size_t)j * n + i;
              if (KIND == 0) Cd[o] = r;
              else if (KIND == 1) { Cd[o] = r; Cf[o] = f32_of(r, 0); }
              else {
                const float h2 = i == j ? (float)(0.5 * (1.0 - r)) : f32_of(-r, 1);
                Cf[o] = h2;
                Cf[(size_t)i * n + j] = h2;
              }
            }
          }
        }
      }
    }
    tc_fence_before();
    __syncthreads();
  }
  return true;
}

__global__ void __launch_bounds__(kQThreads, 1) k_refine_tc(RefineArgs a, int step) {
  extern __shared__ __align__(1024) unsigned char smem[];
  QCtl& ctl = *reinterpret_cast<QCtl*>(smem + 2 * kQStage);
  const int tid = threadIdx.x;
  if (tid == 0) {
    mbar_init(&ctl.bar[0], 1);
    mbar_init(&ctl.bar[1], 1);
    mbar_init(&ctl.done, 1);
    ctl.fail = 0;
    ctl.passed = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if ((tid >> 5) == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smem_u32(&ctl.tslot))
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = ctl.tslot;
  unsigned gchunk = 0;
  int* ticket = a.ticket + kRefineTicketsPerStep * step + kNumBins;
  // bins largest first: ticket t walks bin 3's range of the order array, then bin 2's, ...
  int total = 0;
  for (int bin = 0; bin < kNumBins; ++bin) total += a.sched[3 * bin + 1] - a.sched[3 * bin];
  for (;;) {
    __syncthreads();
    if (tid == 0) ctl.ticket = atomicAdd(ticket, 1);
    __syncthreads();
    int t = ctl.ticket;
    if (t >= total) break;
    int pos = -1;
    for (int bin = kNumBins - 1; bin >= 0; --bin) {
      const int len = a.sched[3 * bin + 1] - a.sched[3 * bin];
      if (t < len) { pos = a.sched[3 * bin] + t; break; }
      t -= len;
    }
    if (pos < 0) continue;
    const int b = a.order[pos];
    const int n = a.ns[b];
    if (n < 1 || n > kSmallMax || a.status[b] != kStRefining) continue;
    const long long off = a.offs[b];
    const double* A = a.A + off;
    double* P = a.P + off;
    double* Z = a.Z + off;
    {  // the exponents of A's rows (fixed) and Z's columns (from the previous step's update)
      const int* ga = a.exA + a.woffs[b];
      const int* gz = a.exZ + a.woffs[b];
      for (int i = tid; i < n; i += kQThreads) { ctl.exA[i] = ga[i]; ctl.exZ[i] = gz[i]; }
    }
    __syncthreads();
    bool ok = tc_product<0, 0>(n, A, Z, ctl.exA, ctl.exZ, -a.exps[b], P, nullptr, smem, ctl, tmem, gchunk);
    if (ok) {
      refine_col_exps<kQThreads>(n, P, ctl.exP);  // P was written by this CTA before the panel's closing barrier
      __syncthreads();
      ok = tc_product<1, 1>(n, Z, P, ctl.exZ, ctl.exP, 0, a.Q + off, a.T32 + off, smem, ctl, tmem, gchunk);
    }
    if (ok) ok = tc_product<1, 2>(n, Z, Z, ctl.exZ, ctl.exZ, 0, nullptr, a.NF + off, smem, ctl, tmem, gchunk);
    if (ok && tid == 0) a.status[b] = kStStepReady;
    if (!ok) {
      if (tid == 0) {
        a.status[b] = a.nofallback ? ST_UNCONVERGED : kStFallback;
        atomicExch(a.err, 1);
      }
      break;
    }
  }
  // every MMA issued must be complete before TMEM is freed
  if (tid == 0) {
    tc_commit(&ctl.done);
    if (!mbar_wait(&ctl.done, 0, kQTimeout)) atomicExch(a.err, 2);
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if ((tid >> 5) == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem) : "memory");
}

}  // namespace

cudaError_t launch_refine_tc(const RefineArgs& a, int step, int num_sms, cudaStream_t s) {
  cudaError_t e = cudaFuncSetAttribute(k_refine_tc, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kQSmem);
  if (e != cudaSuccess) return e;
  k_refine_tc<<<num_sms, kQThreads, kQSmem, s>>>(a, step);
  return cudaGetLastError();
}

}  // namespace gsk
