// Real standard-form quasi-triangular Schur pair -> complex triangular Schur pair
// (triangularize, triang.jl:9-43): batched, one CTA per matrix, and one matrix over the whole GPU.
//
// For each 2x2 block [a b; c a] (bc < 0) at rows/columns (j-1, j), j = n..2, the
// unitary rotation G = [cs, -i sn; -i sn, cs] with cs = sqrt|b|/r, sn = sqrt|c|/r,
// r = hypot(sqrt|c|, sqrt|b|) is applied as T <- G T G^H, Z <- Z G^H.  Work is done
// in the complex output buffers (L2-resident); rotations of different blocks act
// on disjoint coordinates and are applied one block after another.
//
// colmap[b][ki] receives the column of the reference's real-Schur eigenvalue order
// (GenericSchur.jl:678-679 puts a + i*rti first) that complex eigenvalue ki
// corresponds to, so eigenvectors computed from the complex pair can be returned
// in the order of S.values.
#include "device_common.cuh"
#include "gs_internal.h"

#include <algorithm>

namespace gsk {
namespace {

// One rotation after the other by one CTA, on a copy of T and Z in Tc and Zc (everything but the
// closing triu!).
template <int NT>
__device__ void tri_sequential(int n, const double* __restrict__ Tr, const double* __restrict__ Zr,
                               double2* __restrict__ Tc, double2* __restrict__ Zc) {
  const int tid = threadIdx.x;
  for (long long idx = tid; idx < (long long)n * n; idx += NT) {
    Tc[idx] = make_double2(Tr[idx], 0.0);
    if (Zc) Zc[idx] = make_double2(Zr ? Zr[idx] : ((idx % n) == (idx / n) ? 1.0 : 0.0), 0.0);
  }
  __syncthreads();
  for (int j = n; j >= 2; --j) {
    const double sub = Tr[(j - 1) + (long long)(j - 2) * n];  // Tr[j, j-1]
    if (sub == 0.0) continue;
    const double s = sqrt(fabs(sub));
    const double cc = sqrt(fabs(Tr[(j - 2) + (long long)(j - 1) * n]));  // sqrt|Tr[j-1, j]|
    const double r = hypot(s, cc);
    const double gc = cc / r;      // Givens c (real)
    const double gs = -(s / r);    // Givens s = i * gs (purely imaginary)
    const int p = j - 2, q = j - 1;  // 0-based rows/cols of the block
    // lmul!(G, T): rows p, q; new_p = c a1 + s a2; new_q = -conj(s) a1 + c a2, s = i gs
    for (int k = tid; k < n; k += NT) {
      const double2 a1 = Tc[p + (long long)k * n], a2 = Tc[q + (long long)k * n];
      Tc[p + (long long)k * n] = make_double2(gc * a1.x - gs * a2.y, gc * a1.y + gs * a2.x);
      Tc[q + (long long)k * n] = make_double2(gc * a2.x - gs * a1.y, gc * a2.y + gs * a1.x);
    }
    __syncthreads();
    // rmul!(T, G') and rmul!(Z, G'): columns p, q; new_p = a1 c + a2 conj(s); new_q = -a1 s + a2 c
    for (int k = tid; k < n; k += NT) {
      double2 a1 = Tc[k + (long long)p * n], a2 = Tc[k + (long long)q * n];
      Tc[k + (long long)p * n] = make_double2(gc * a1.x + gs * a2.y, gc * a1.y - gs * a2.x);
      Tc[k + (long long)q * n] = make_double2(gc * a2.x + gs * a1.y, gc * a2.y - gs * a1.x);
      if (Zc) {
        a1 = Zc[k + (long long)p * n];
        a2 = Zc[k + (long long)q * n];
        Zc[k + (long long)p * n] = make_double2(gc * a1.x + gs * a2.y, gc * a1.y - gs * a2.x);
        Zc[k + (long long)q * n] = make_double2(gc * a2.x + gs * a1.y, gc * a2.y - gs * a1.x);
      }
    }
    __syncthreads();
  }
}

template <int NT>
__global__ void __launch_bounds__(NT) k_triangularize(TriBatch tb) {
  const int tid = threadIdx.x;
  for (int b = blockIdx.x; b < tb.count; b += gridDim.x) {
    const int n = tb.ns ? tb.ns[b] : tb.n1;
    const long long off = tb.ns ? tb.offs[b] : 0, woff = tb.ns ? tb.woffs[b] : 0;
    const double* __restrict__ Tr = tb.Tr + off;
    double2* __restrict__ Tc = tb.Tc + off;
    tri_sequential<NT>(n, Tr, tb.Zr ? tb.Zr + off : nullptr, Tc, tb.Zc ? tb.Zc + off : nullptr);
    // triu!(T), values = diag(T), column map
    for (int idx = tid; idx < n * n; idx += NT) {
      const int i = idx % n, jj = idx / n;
      if (i > jj) Tc[idx] = make_double2(0.0, 0.0);
    }
    __syncthreads();
    for (int k = tid; k < n; k += NT) {
      const double2 d = Tc[k + (long long)k * n];
      if (tb.w) tb.w[woff + k] = d;
      if (tb.colmap) {
        int dst = k;
        const bool lower = (k + 1 < n) && Tr[(k + 1) + (long long)k * n] != 0.0;  // k is first of a pair
        const bool upper = (k > 0) && Tr[k + (long long)(k - 1) * n] != 0.0;      // k is second of a pair
        if (lower && d.y < 0.0) dst = k + 1;
        if (upper && Tc[(k - 1) + (long long)(k - 1) * n].y < 0.0) dst = k - 1;
        tb.colmap[woff + k] = dst;
      }
    }
    __syncthreads();
  }
}

// One large matrix, over the whole GPU.  The rotations of different blocks act on disjoint
// rows and columns, so an entry above the blocks' diagonal meets two of them, its column
// block's and then its row block's (descending order), and each 2x2 tile of blocks is one
// thread's.  k_tri_rot leaves (cs, -sn) of each block in the block's subdiagonal place, which
// k_tri_finish clears.  One CTA, two passes and two barriers per block, took 12.8 ms at
// n = 1024 with vectors; these launches take less than 0.4 ms together.
// In a T that is not quasi-triangular (two nonzero subdiagonal entries in a row) the rotations
// overlap: k_tri_rot then sets the flag, and k_tri_runs applies them one after the other.
__host__ __device__ __forceinline__ double* tri_flag(int n, double2* Tc) { return n > 2 ? &Tc[2].x : nullptr; }  // place (3, 1)

__global__ void k_tri_rot(int n, const double* __restrict__ Tr, double2* __restrict__ Tc) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x + 2;
  if (j > n) return;
  const double sub = Tr[(j - 1) + (long long)(j - 2) * n];  // Tr[j, j-1]
  double2 g = make_double2(0.0, 0.0);
  if (sub != 0.0) {
    const double s = sqrt(fabs(sub));
    const double cc = sqrt(fabs(Tr[(j - 2) + (long long)(j - 1) * n]));  // sqrt|Tr[j-1, j]|
    const double r = hypot(s, cc);
    g = make_double2(cc / r, -(s / r));
    if (j > 2 && Tr[(j - 2) + (long long)(j - 3) * n] != 0.0) *tri_flag(n, Tc) = 1.0;
  }
  Tc[(j - 1) + (long long)(j - 2) * n] = g;
}

// columns p, q under G^H: (a1, a2) -> (c a1 + conj(s) a2, -s a1 + c a2), s = i gs
__device__ __forceinline__ void tri_cols(double gc, double gs, double2& x1, double2& x2) {
  const double2 a1 = x1, a2 = x2;
  x1 = make_double2(gc * a1.x + gs * a2.y, gc * a1.y - gs * a2.x);
  x2 = make_double2(gc * a2.x + gs * a1.y, gc * a2.y - gs * a1.x);
}
// rows p, q under G
__device__ __forceinline__ void tri_rows(double gc, double gs, double2& x1, double2& x2) {
  const double2 a1 = x1, a2 = x2;
  x1 = make_double2(gc * a1.x - gs * a2.y, gc * a1.y + gs * a2.x);
  x2 = make_double2(gc * a2.x - gs * a1.y, gc * a2.y + gs * a1.x);
}

// blockIdx.x: a column j; threads: rows i.  The thread of a tile's first entry does the tile.
__global__ void __launch_bounds__(128) k_tri_apply(int n, const double* __restrict__ Tr, const double* __restrict__ Zr,
                                                   double2* Tc, double2* __restrict__ Zc) {
  const int i = blockIdx.y * blockDim.x + threadIdx.x, j = blockIdx.x;
  if (i >= n || (n > 2 && *tri_flag(n, Tc) != 0.0)) return;
  const auto sub = [&](int k) { return k >= 0 && k + 1 < n && Tr[(k + 1) + (long long)k * n] != 0.0; };
  const auto second = [&](int k) { return sub(k - 1); };
  if (second(j)) return;  // second column of a block
  const bool c2 = sub(j);
  const double2 gj = c2 ? Tc[(j + 1) + (long long)j * n] : make_double2(1.0, 0.0);
  if (Zc) {
    const auto zin = [&](int c) { return make_double2(Zr ? Zr[i + (long long)c * n] : (i == c ? 1.0 : 0.0), 0.0); };
    double2 z1 = zin(j);
    if (c2) {
      double2 z2 = zin(j + 1);
      tri_cols(gj.x, gj.y, z1, z2);
      Zc[i + (long long)(j + 1) * n] = z2;
    }
    Zc[i + (long long)j * n] = z1;
  }
  if (i > j || second(i)) return;  // below the diagonal blocks, or second row of a block
  const bool r2 = sub(i);
  const auto tin = [&](int a, int b) { return make_double2(Tr[a + (long long)b * n], 0.0); };
  const double2 zero = make_double2(0.0, 0.0);
  double2 x11 = tin(i, j), x21 = r2 ? tin(i + 1, j) : zero, x12 = c2 ? tin(i, j + 1) : zero,
          x22 = r2 && c2 ? tin(i + 1, j + 1) : zero;
  if (i == j) {
    if (r2) {  // the block itself: its rows, then its columns
      tri_rows(gj.x, gj.y, x11, x21);
      tri_rows(gj.x, gj.y, x12, x22);
      tri_cols(gj.x, gj.y, x11, x12);
      tri_cols(gj.x, gj.y, x21, x22);
    }
  } else {
    if (c2) {
      tri_cols(gj.x, gj.y, x11, x12);
      tri_cols(gj.x, gj.y, x21, x22);
    }
    if (r2) {
      const double2 gi = Tc[(i + 1) + (long long)i * n];
      tri_rows(gi.x, gi.y, x11, x21);
      tri_rows(gi.x, gi.y, x12, x22);
    }
  }
  Tc[i + (long long)j * n] = x11;
  if (r2 && i != j) Tc[(i + 1) + (long long)j * n] = x21;  // (the block's own holds its rotation)
  if (c2) Tc[i + (long long)(j + 1) * n] = x12;
  if (r2 && c2) Tc[(i + 1) + (long long)(j + 1) * n] = x22;
}

// One CTA; nothing to do for a quasi-triangular T.
__global__ void __launch_bounds__(256) k_tri_runs(int n, const double* Tr, const double* Zr, double2* Tc, double2* Zc) {
  const bool runs = *tri_flag(n, Tc) != 0.0;
  __syncthreads();  // the flag is in the way of the copy
  if (runs) tri_sequential<256>(n, Tr, Zr, Tc, Zc);
}

// triu!(T), values = diag(T), column map
__global__ void k_tri_finish(int n, const double* __restrict__ Tr, double2* __restrict__ Tc, double2* __restrict__ w,
                             int* __restrict__ colmap) {
  const size_t tot = (size_t)n * n;
  for (size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x; e < tot; e += (size_t)gridDim.x * blockDim.x) {
    const int i = (int)(e % n), j = (int)(e / n);
    if (i > j) Tc[e] = make_double2(0.0, 0.0);
    if (i != j) continue;
    const double2 d = Tc[e];
    if (w) w[j] = d;
    if (colmap) {
      int dst = j;
      const bool lower = (j + 1 < n) && Tr[(j + 1) + (long long)j * n] != 0.0;  // j is first of a pair
      const bool upper = (j > 0) && Tr[j + (long long)(j - 1) * n] != 0.0;      // j is second of a pair
      if (lower && d.y < 0.0) dst = j + 1;
      if (upper && Tc[(j - 1) + (long long)(j - 1) * n].y < 0.0) dst = j - 1;
      colmap[j] = dst;
    }
  }
}

}  // namespace

cudaError_t launch_triangularize_one(int n, const double* Tr, const double* Zr, double2* Tc, double2* Zc, double2* w,
                                     int* colmap, cudaStream_t s) {
  if (n < 1) return cudaSuccess;
  // One CTA up to order 16: there a launch costs more than the rotations one after the other (host
  // call, n = 3 40.7 us, with the launches below 48.4; 10 50.9, 57.6; 16 64.2, 67.1 with the one-CTA
  // kernel and its orders in device memory).
  if (n <= 16) {
    TriBatch tb{};
    tb.count = 1;
    tb.n1 = n;
    tb.Tr = Tr;
    tb.Zr = Zr;
    tb.Tc = Tc;
    tb.Zc = Zc;
    tb.w = w;
    tb.colmap = colmap;
    k_triangularize<128><<<1, 128, 0, s>>>(tb);
    return cudaGetLastError();
  }
  if (double* flag = tri_flag(n, Tc)) {
    cudaError_t e = cudaMemsetAsync(flag, 0, sizeof(double), s);
    if (e != cudaSuccess) return e;
  }
  k_tri_rot<<<(n + 127) / 128, 128, 0, s>>>(n, Tr, Tc);
  k_tri_apply<<<dim3(n, (n + 127) / 128), 128, 0, s>>>(n, Tr, Zr, Tc, Zc);
  if (n > 2) k_tri_runs<<<1, 256, 0, s>>>(n, Tr, Zr, Tc, Zc);
  k_tri_finish<<<(int)std::min<size_t>(((size_t)n * n + 255) / 256, 4096), 256, 0, s>>>(n, Tr, Tc, w, colmap);
  return cudaGetLastError();
}

cudaError_t launch_triangularize(const TriBatch& tb, int num_sms, cudaStream_t s) {
  int grid = tb.count < 4 * num_sms ? tb.count : 4 * num_sms;
  if (grid < 1) grid = 1;
  k_triangularize<128><<<grid, 128, 0, s>>>(tb);
  return cudaGetLastError();
}

}  // namespace gsk
