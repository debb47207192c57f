// Dense kernels of the whitening chain: tall-skinny Gram products (FP32
// partial sums, FP64 across row chunks), tall-skinny x small products, small
// FP64 GEMMs, upper Cholesky with the modified-Gram-Schmidt drop rule, upper
// triangular inverse, one-sided Jacobi eigen-solver, and the Philox Gaussian
// sketch panel.
//
// Why FP64 only on p x p data: GB300's FP64 rate is ~1/64 of its FP32 rate,
// so every n-sized product stays FP32 and only the p x p factors (p = 2k <= 512)
// are FP64.
#include "common.cuh"

#include <cooperative_groups.h>

#include <algorithm>
#include <type_traits>

namespace mmsb {

namespace {

// ---- tall-skinny Gram: S = alpha * A^T B --------------------------------------

constexpr int GT = 64;      // output tile edge
constexpr int GR = 32;      // rows per smem stage
constexpr int GCHUNK = 256; // rows accumulated in FP32 before the FP64 add

__global__ void __launch_bounds__(256) gram_partial_kernel(
    const float* __restrict__ A, int lda, int pa, const float* __restrict__ B, int ldb, int pb,
    int64_t n, int64_t rows_per_split, double* __restrict__ partials) {
  __shared__ __align__(16) float As[GR][GT + 4];
  __shared__ __align__(16) float Bs[GR][GT + 4];
  const int ta = blockIdx.x, tb = blockIdx.y, split = blockIdx.z;
  const int tid = threadIdx.x;
  const int tx = tid % 16, ty = tid / 16;  // 4x4 patch at (ty*4, tx*4)
  const int64_t r0 = split * rows_per_split;
  const int64_t r1 = min(n, r0 + rows_per_split);
  double accd[4][4];
  float acc[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      accd[i][j] = 0.0;
      acc[i][j] = 0.f;
    }
  // A split has up to 8 stages and often an SM to itself: the next stage's rows
  // are loaded while this one is summed, and patches past the columns are left
  // out, since the shared memory's bandwidth sets the time of a stage (5,000 rows
  // of 50 columns 23.4 -> 14.3 us, 1,000 rows of 10 columns 20 -> 11.9 us).
  const bool live = ta * GT + ty * 4 < pa && tb * GT + tx * 4 < pb;
  int since = 0;
  constexpr int PER = GR * GT / 256;
  float va[PER], vb[PER];
  auto load = [&](int64_t rb) {
#pragma unroll
    for (int u = 0; u < PER; ++u) {
      const int e = tid + 256 * u, rr = e / GT, cc = e % GT;
      const int64_t row = rb + rr;
      const int ca = ta * GT + cc, cb = tb * GT + cc;
      va[u] = (row < r1 && ca < pa) ? __ldg(A + row * lda + ca) : 0.f;
      vb[u] = (row < r1 && cb < pb) ? __ldg(B + row * ldb + cb) : 0.f;
    }
  };
  load(r0);
  for (int64_t rb = r0; rb < r1; rb += GR) {
#pragma unroll
    for (int u = 0; u < PER; ++u) {
      const int e = tid + 256 * u;
      As[e / GT][e % GT] = va[u];
      Bs[e / GT][e % GT] = vb[u];
    }
    __syncthreads();
    if (rb + GR < r1) load(rb + GR);
    if (live) {
#pragma unroll 8
      for (int rr = 0; rr < GR; ++rr) {
        float a[4], b[4];
        *reinterpret_cast<float4*>(a) = *reinterpret_cast<const float4*>(&As[rr][ty * 4]);
        *reinterpret_cast<float4*>(b) = *reinterpret_cast<const float4*>(&Bs[rr][tx * 4]);
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
      }
    }
    __syncthreads();
    since += GR;
    if (live && since >= GCHUNK) {
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          accd[i][j] += (double)acc[i][j];
          acc[i][j] = 0.f;
        }
      since = 0;
    }
  }
  // partials layout: [split][pb][pa] (column-major per split)
  double* out = partials + (int64_t)split * pa * pb;
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int ia = ta * GT + ty * 4 + i, jb = tb * GT + tx * 4 + j;
      if (ia < pa && jb < pb) out[(int64_t)jb * pa + ia] = accd[i][j] + (double)acc[i][j];
    }
}

// (the splits in order, 8 loads in flight: the FP64 sums stay one chain; mirror >
// 0: only tiles of that edge on and above the diagonal hold partials, p x p)
__global__ void gram_reduce_kernel(const double* __restrict__ partials, int nsplit, int64_t m,
                                   double alpha, double* __restrict__ S, int mirror, int p) {
  for (int64_t at = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; at < m;
       at += (int64_t)gridDim.x * blockDim.x) {
    int64_t e = at;
    if (mirror > 0) {
      const int i = (int)(at % p), j = (int)(at / p);
      if (i / mirror > j / mirror) e = (int64_t)i * p + j;
    }
    double s = 0.0;
    int t = 0;
    for (; t + 8 <= nsplit; t += 8) {
      double v[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) v[u] = __ldg(partials + (int64_t)(t + u) * m + e);
#pragma unroll
      for (int u = 0; u < 8; ++u) s += v[u];
    }
    for (; t < nsplit; ++t) s += __ldg(partials + (int64_t)t * m + e);
    S[at] = alpha * s;
  }
}

int gram_nsplit(int64_t n, int pa, int pb) {
  const int tiles = (int)(ceil_div(pa, GT) * ceil_div(pb, GT));
  int64_t want = ceil_div(2 * kNumSMs, tiles);
  want = std::min<int64_t>(want, ceil_div(n, GCHUNK));
  return (int)std::max<int64_t>(1, std::min<int64_t>(want, 256));
}

// ---- M (n x p, FP32 row-major) * F (p x q, FP64 column-major) ----------------

// (float)x in integer arithmetic (round to nearest even): a conversion costs
// the FP64 unit 64 cycles per warp and SM quarter, and F is converted again in
// every CTA (with that, and 16-byte loads of F, two concurrent products of n =
// 50,000, p = q = 200 went from 271 to 258 us; the shared memory's bandwidth sets
// the rest).  Results outside the normal FP32 range take the conversion.
__device__ __forceinline__ bool narrows(double x) {  // to a normal FP32 number (or past the largest)
  return (((unsigned)__double2hiint(x) >> 20) & 0x7ffu) - 897u <= 253u;
}

__device__ __forceinline__ float narrow_normal(double x) {
  const unsigned hi = (unsigned)__double2hiint(x), lo = (unsigned)__double2loint(x);
  const unsigned e = (hi >> 20) & 0x7ffu;
  const unsigned m = ((e - 896u) << 23) | ((hi & 0xfffffu) << 3) | (lo >> 29);
  const unsigned rem = lo & 0x1fffffffu;
  return __uint_as_float((hi & 0x80000000u) | (m + (rem + (m & 1u) > 0x10000000u ? 1u : 0u)));
}

__device__ __forceinline__ float narrow(double x) {
  if (!narrows(x)) return x == 0.0 ? __uint_as_float((unsigned)__double2hiint(x) & 0x80000000u) : (float)x;
  return narrow_normal(x);
}

// (double)x of a normal number the same way
__device__ __forceinline__ double widen_normal(float x) {
  const unsigned u = __float_as_uint(x);
  return __hiloint2double((int)((u & 0x80000000u) | (((u & 0x7fffffffu) >> 3) + (896u << 20))),
                          (int)(u << 29));
}

constexpr int PT_R = 64, PT_C = 64, PT_K = 32;

__global__ void __launch_bounds__(256) panel_small_kernel(
    const float* __restrict__ M, int ldm, int p, int64_t n, const double* __restrict__ F,
    int ldf, int q, float* __restrict__ Y, int ldy) {
  __shared__ float Ms[PT_R][PT_K + 1];
  __shared__ __align__(16) float Fs[PT_K][PT_C + 4];
  const int tid = threadIdx.x;
  const int tx = tid % 16, ty = tid / 16;
  const int64_t row0 = (int64_t)blockIdx.x * PT_R;
  const int col0 = blockIdx.y * PT_C;
  float acc[4][4] = {};
  for (int k0 = 0; k0 < p; k0 += PT_K) {
    for (int e = tid; e < PT_R * PT_K; e += 256) {
      const int rr = e / PT_K, kk = e % PT_K;
      const int64_t row = row0 + rr;
      Ms[rr][kk] = (row < n && k0 + kk < p) ? M[row * ldm + k0 + kk] : 0.f;
    }
    for (int e = tid; e < PT_K * PT_C; e += 256) {
      const int kk = e % PT_K, cc = e / PT_K;
      Fs[kk][cc] = (k0 + kk < p && col0 + cc < q) ? narrow(F[(int64_t)(col0 + cc) * ldf + k0 + kk])
                                                  : 0.f;
    }
    __syncthreads();
#pragma unroll 8
    for (int kk = 0; kk < PT_K; ++kk) {
      float a[4], b[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) a[i] = Ms[ty * 4 + i][kk];
      *reinterpret_cast<float4*>(b) = *reinterpret_cast<const float4*>(&Fs[kk][tx * 4]);
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int64_t row = row0 + ty * 4 + i;
    if (row >= n) continue;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int col = col0 + tx * 4 + j;
      if (col < ldy) Y[row * ldy + col] = col < q ? acc[i][j] : 0.f;
    }
  }
}

// ---- small FP64 GEMM ------------------------------------------------------------

// FP64 FMAs go at 2 per clock and SM (64 cycles per warp and SM quarter), so the
// time is the largest number of warps on one quarter, times k: 8 x 8 tiles, an
// entry per thread, spread the work in units of a warp.  (16 x 16 tiles of 8
// warps, with k rounded up to 32: the 56 products of a whitening took 32 us on
// average with 200 columns, 27 us here, 4.2 and 3.3 us with 10.)  A product of a matrix with its own transpose computes one
// triangle of tiles: (i, j) and (j, i) are the same sums, bit for bit.
constexpr int DG_T = 8, DG_K = 64;

__global__ void __launch_bounds__(DG_T * DG_T) dgemm_small_kernel(
    bool ta, bool tb, bool sym, int m, int n, int k, double alpha, const double* __restrict__ A,
    int lda, const double* __restrict__ B, int ldb, double beta, const double* __restrict__ C0,
    double* __restrict__ C, int ldc) {
  constexpr int T = DG_T, KC = DG_K, NT = T * T;
  if (sym && blockIdx.x > blockIdx.y) return;
  __shared__ double As[T][KC + 1];
  __shared__ double Bs[KC][T + 1];
  const int tid = threadIdx.x;
  const int tx = tid % T, ty = tid / T;
  const int i0 = blockIdx.x * T, j0 = blockIdx.y * T;
  double acc = 0.0;
  for (int k0 = 0; k0 < k; k0 += KC) {
#pragma unroll
    for (int u = 0; u < KC / T; ++u) {
      const int e = tid + NT * u;
      {  // As[ii][kk] = op(A)[i0+ii, k0+kk]; consecutive threads walk a column of A
        const int ii = ta ? e / KC : e % T, kk = ta ? e % KC : e / T;
        const int gi = i0 + ii, gk = k0 + kk;
        double v = 0.0;
        if (gi < m && gk < k) v = ta ? A[(int64_t)gi * lda + gk] : A[(int64_t)gk * lda + gi];
        As[ii][kk] = v;
      }
      {  // Bs[kk][jj] = op(B)[k0+kk, j0+jj]; consecutive threads walk a column of B
        const int kk = tb ? e / T : e % KC, jj = tb ? e % T : e / KC;
        const int gk = k0 + kk, gj = j0 + jj;
        double v = 0.0;
        if (gk < k && gj < n) v = tb ? B[(int64_t)gk * ldb + gj] : B[(int64_t)gj * ldb + gk];
        Bs[kk][jj] = v;
      }
    }
    __syncthreads();
    const int kn = k - k0 < KC ? k - k0 : KC;
#pragma unroll 4
    for (int kk = 0; kk < kn; ++kk) acc = fma(As[ty][kk], Bs[kk][tx], acc);
    __syncthreads();
  }
  const int gi = i0 + ty, gj = j0 + tx;
  if (gi < m && gj < n) {
    const int64_t at = (int64_t)gj * ldc + gi;
    const double v = alpha * acc + (beta == 0.0 ? 0.0 : beta * C0[at]);
    C[at] = v;
    if (sym && blockIdx.x != blockIdx.y) C[(int64_t)gi * ldc + gj] = v;
  }
}

// ---- upper Cholesky with drop rule (one CTA) ---------------------------------

__global__ void __launch_bounds__(1024) chol_upper_kernel(int p, const double* __restrict__ S,
                                                          int lds, double* __restrict__ R,
                                                          double drop2, unsigned* flags) {
  extern __shared__ double rowj[];  // row j of R (p values)
  const int tid = threadIdx.x, nt = blockDim.x, lane = tid & 31, warp = tid >> 5, nw = nt >> 5;
  for (int l = warp; l < p; l += nw)
    for (int i = lane; i < p; i += 32) R[(int64_t)l * p + i] = i <= l ? S[(int64_t)l * lds + i] : 0.0;
  __syncthreads();
  __shared__ double rjj;
  for (int j = 0; j < p; ++j) {
    if (tid == 0) {
      const double d = R[(int64_t)j * p + j];
      if (!(d > drop2)) {
        rjj = 0.0;
        if (!(d == d)) atomicOr(flags, kFlagNonFinite);
      } else {
        rjj = sqrt(d);
      }
      R[(int64_t)j * p + j] = rjj;
    }
    __syncthreads();
    const double r = rjj;
    // one FP64 division per pivot (the FP64 pipe is ~2 operations per clock
    // per SM here), then multiplications
    const double ri = r > 0.0 ? 1.0 / r : 0.0;
    for (int l = j + 1 + tid; l < p; l += nt) {
      double* x = &R[(int64_t)l * p + j];
      const double v = *x * ri;
      *x = v;
      rowj[l] = v;
    }
    __syncthreads();
    // trailing update R[i, l] -= R[j, i] R[j, l] for j < i <= l: a warp per
    // column l, its lanes along the contiguous rows i
    for (int l = j + 1 + warp; l < p; l += nw) {
      const double rl = rowj[l];
      double* col = R + (int64_t)l * p;
      for (int i = j + 1 + lane; i <= l; i += 32) col[i] = fma(-rowj[i], rl, col[i]);
    }
    __syncthreads();
  }
}

// ---- T = R^{-1} (upper), one warp per column ------------------------------------

// The same factorisation on a cluster of CL CTAs, blocked by KB columns, for
// p up to 512: column l of R lives in the shared memory of CTA l % CL.  Per
// block J = [jb, jb + KB):
//   1. every CTA gathers the (updated) diagonal block S_JJ through DSMEM and
//      factors it (the drop rule of chol_upper_kernel, pivot by pivot);
//   2. each CTA solves R_JJ^T X = S_J,l for its columns l past the block
//      (forward substitution, zero where a pivot was dropped): row block J;
//   3. after a cluster barrier every CTA gathers row block J and updates its
//      columns: S[i, l] -= sum_{c in J} R[c, i] R[c, l], jb + KB <= i <= l.
// Two cluster barriers per block (the second also orders every CTA's gather
// of S_JJ before the owners overwrite those columns with R_JJ); the FP64
// update (p^3 / 6 multiply-adds)
// runs on CL SMs.  The steps equal the unblocked ones up to the order of the
// FP64 sums.
template <int CL, int KB, typename T>
__global__ void __launch_bounds__(256, 1) chol_upper_cluster_kernel(int p, const double* __restrict__ S,
                                                                 int lds, double* __restrict__ R,
                                                                 double drop2, unsigned* flags) {
  namespace cg = cooperative_groups;
  cg::cluster_group cluster = cg::this_cluster();
  extern __shared__ __align__(16) unsigned char chraw[];
  T* chs = reinterpret_cast<T*>(chraw);
  const int rank = (int)cluster.block_rank();
  const int ncl = (p + CL - 1) / CL;            // local columns: l = lc CL + rank
  T* Rl = chs;                                   // Rl[lc p + i]
  T* BR = Rl + (size_t)ncl * p;                  // row block: BR[c p + i] = R[jb + c, i]
  __shared__ T DJ[KB * KB];                 // DJ[cc KB + c] = R[jb + c, jb + cc]
  __shared__ T DR[KB];                      // R[jb + c, jb + c] (0 where dropped; FP64 form)
  __shared__ T DI[KB];                      // and its reciprocal (0 where dropped)
  const int tid = threadIdx.x, nt = blockDim.x, lane = tid & 31, warp = tid >> 5, nw = nt >> 5;
  for (int e = tid; e < ncl * p; e += nt) {
    const int lc = e / p, i = e % p, l = lc * CL + rank;
    Rl[e] = (l < p && i <= l) ? (T)S[(int64_t)l * lds + i] : (T)0;
  }
  for (int jb = 0; jb < p; jb += KB) {
    const int bs = min(KB, p - jb);
    cluster.sync();  // the previous block's updates are complete everywhere
    for (int e = tid; e < KB * KB; e += nt) {
      const int c = e % KB, cc = e / KB;
      T v = 0;
      if (c <= cc && cc < bs) {
        const int l = jb + cc;
        v = cluster.map_shared_rank(Rl, l % CL)[(size_t)(l / CL) * p + jb + c];
      }
      DJ[e] = v;
    }
    __syncthreads();
    if constexpr (std::is_same<T, double>::value) {
      // FP64: 4 warps, 2 entries per thread.  Every thread forms the pivot's root
      // and reciprocal and scales the two entries of row c that it needs; row c
      // itself is scaled at the end, so a pivot takes one barrier.  The products
      // are those of the column-by-column form, bit for bit: the signs of the
      // eigenvectors behind this factor hang on its last bits (root-free, with the
      // rows scaled at the end, 28 of 70 graphs with k from 130 on came out in
      // another frame).  p = 200: 290 us (182 us root-free).
      if (tid < 128) {
        static_assert(KB == 16, "two entries per thread");
        for (int c = 0; c < bs; ++c) {
          const double d = DJ[c * KB + c];
          const double r = d > drop2 ? sqrt(d) : 0.0, ri = r > 0.0 ? 1.0 / r : 0.0;
          if (tid == 0) {
            if (!(d > drop2) && !(d == d)) atomicOr(flags, kFlagNonFinite);
            DR[c] = r;
            DI[c] = ri;
          }
          double v[2];
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const int e = tid + 128 * h, i = e % KB, l = e / KB;
            v[h] = DJ[e];
            if (i > c && i <= l && l < bs) v[h] = fma(-(DJ[i * KB + c] * ri), DJ[l * KB + c] * ri, v[h]);
          }
#pragma unroll
          for (int h = 0; h < 2; ++h) {  // (row c, read by others, is not written)
            const int e = tid + 128 * h, i = e % KB, l = e / KB;
            if (i > c && i <= l && l < bs) DJ[e] = v[h];
          }
          asm volatile("bar.sync 1, 128;" ::: "memory");
        }
        double v[2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int e = tid + 128 * h, i = e % KB, l = e / KB;
          v[h] = i < l && l < bs ? DJ[e] * DI[i] : i == l && l < bs ? DR[i] : 0.0;
        }
#pragma unroll
        for (int h = 0; h < 2; ++h) DJ[tid + 128 * h] = v[h];
      }
    } else if (warp == 0) {  // upper Cholesky of the diagonal block with the drop rule
      for (int c = 0; c < bs; ++c) {
        if (lane == 0) {
          const T d = DJ[c * KB + c];
          T r = 0;
          if (d > (T)drop2) {
            r = sqrt(d);
          } else if (!(d == d)) {
            atomicOr(flags, kFlagNonFinite);
          }
          DJ[c * KB + c] = r;
          DI[c] = r > (T)0 ? (T)1 / r : (T)0;  // one division per pivot
        }
        __syncwarp();
        const T ri = DI[c];
        for (int cc = c + 1 + lane; cc < bs; cc += 32) DJ[cc * KB + c] *= ri;
        __syncwarp();
        for (int e = lane; e < KB * KB; e += 32) {
          const int i = e % KB, cc = e / KB;
          if (i > c && i <= cc && cc < bs) DJ[cc * KB + i] = fma(-DJ[i * KB + c], DJ[cc * KB + c], DJ[cc * KB + i]);
        }
        __syncwarp();
      }
    }
    __syncthreads();
    // row block J of this CTA's columns past the block: the forward
    // substitution R_JJ^T x = S_J,l (a thread per column)
    const int i0 = jb + bs;
    if constexpr (std::is_same<T, double>::value) {
      // (FP64: 16 lanes per column, lane c its entry c: 16 steps of a product
      // and an update instead of a chain of 136)
      for (int l0 = 0; l0 < ncl; l0 += nt / KB) {
        const int lc = l0 + tid / KB, c = tid % KB, l = lc * CL + rank;
        const bool live = lc < ncl && l >= i0 && l < p;
        T* col = Rl + (size_t)(live ? lc : 0) * p + jb;
        T v = live && c < bs ? col[c] : (T)0;
        const unsigned half = (lane & 16) ? 0xffff0000u : 0x0000ffffu;
        if (__any_sync(0xffffffffu, live)) {
          for (int c2 = 0; c2 < bs; ++c2) {
            if (c == c2) v *= DI[c2];
            const T x = __shfl_sync(half, v, c2, KB);
            if (c > c2) v = fma(-DJ[c * KB + c2], x, v);
          }
        }
        if (live && c < bs) col[c] = v;
      }
    } else {
    for (int lc = tid; lc < ncl; lc += nt) {
      const int l = lc * CL + rank;
      if (l < i0 || l >= p) continue;
      T* col = Rl + (size_t)lc * p + jb;
      for (int c = 0; c < bs; ++c) {
        T x = col[c];
        for (int c2 = 0; c2 < c; ++c2) x = fma(-DJ[c * KB + c2], col[c2], x);
        col[c] = x * DI[c];
      }
    }
    }
    // every CTA has gathered S_JJ and row block J is complete everywhere;
    // only now may the owners overwrite the block's own columns with R_JJ
    cluster.sync();
    for (int lc = tid; lc < ncl; lc += nt) {
      const int l = lc * CL + rank;
      if (l < jb || l >= i0) continue;
      const int cc = l - jb;
      T* col = Rl + (size_t)lc * p + jb;
      for (int c = 0; c <= cc; ++c) col[c] = DJ[cc * KB + c];
    }
    if (i0 >= p) break;
    // (a thread per row i, its entries of the block loaded together)
    for (int i = i0 + (tid >> 1); i < p; i += nt >> 1) {
      const T* src = cluster.map_shared_rank(Rl, i % CL) + (size_t)(i / CL) * p + jb;
      T v[KB / 2];
#pragma unroll
      for (int u = 0; u < KB / 2; ++u) v[u] = 2 * u + (tid & 1) < bs ? src[2 * u + (tid & 1)] : (T)0;
#pragma unroll
      for (int u = 0; u < KB / 2; ++u)
        if (2 * u + (tid & 1) < bs) BR[(size_t)(2 * u + (tid & 1)) * p + i] = v[u];
    }
    __syncthreads();
    // trailing update of this CTA's columns: a warp per column, lanes on rows
    for (int lc = warp; lc < ncl; lc += nw) {
      const int l = lc * CL + rank;
      if (l < i0 || l >= p) continue;
      T* col = Rl + (size_t)lc * p;
      T rc[KB];
#pragma unroll
      for (int c = 0; c < KB; ++c) rc[c] = c < bs ? col[jb + c] : (T)0;
      for (int i = i0 + lane; i <= l; i += 32) {
        T x = col[i];
#pragma unroll
        for (int c = 0; c < KB; ++c) x = fma(-BR[(size_t)c * p + i], rc[c], x);
        col[i] = x;
      }
    }
    __syncthreads();
  }
  __syncthreads();  // the last block's copy of R_JJ is complete
  for (int e = tid; e < ncl * p; e += nt) {
    const int lc = e / p, i = e % p, l = lc * CL + rank;
    if (l < p) R[(int64_t)l * p + i] = i <= l ? (double)Rl[e] : 0.0;
  }
  cluster.sync();  // keep shared memory alive until every remote read is done
}

// Column j of T solves R t = e_j by back substitution in column (axpy) form:
// for l = j..0: t_l = b_l / R_ll (0 where R_ll == 0), then b_i -= t_l R_il for
// i < l.  Column l of R is contiguous, so each step is one coalesced axpy;
// lane i % 32 keeps b_i (and then t_i) in register slot i / 32 (p <= 32 SLOTS),
// and column l - 1 is loaded while step l runs: with the load inside the step
// its latency set the time (144 us at p = 200, 95 us here).
template <int SLOTS>
__global__ void __launch_bounds__(64) trinv_upper_kernel(int p, const double* __restrict__ R,
                                                         double* __restrict__ T) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int j = blockIdx.x * (blockDim.x >> 5) + w;
  if (j >= p) return;
  double b[SLOTS], rinv[SLOTS], next[SLOTS];
  auto load = [&](int l) {
#pragma unroll
    for (int q = 0; q < SLOTS; ++q)
      if (32 * q <= l) next[q] = lane + 32 * q < l ? __ldg(R + (int64_t)l * p + lane + 32 * q) : 0.0;
  };
#pragma unroll
  for (int q = 0; q < SLOTS; ++q) next[q] = 0.0;
  load(j);
  // 1 / R_ll of the rows this lane holds, all divisions issued together (the
  // FP64 pipe is ~2 operations per clock per SM): the back substitution's
  // dependent chain then has multiplications only
#pragma unroll
  for (int q = 0; q < SLOTS; ++q) {
    const int i = lane + 32 * q;
    b[q] = i == j ? 1.0 : 0.0;
    rinv[q] = 0.0;
    if (32 * q <= j) {
      const double rii = i <= j ? R[(int64_t)i * p + i] : 0.0;
      rinv[q] = rii != 0.0 ? 1.0 / rii : 0.0;
    }
  }
  for (int l = j; l >= 0; --l) {
    const int ql = l >> 5, ll = l & 31;
    double rc[SLOTS];
#pragma unroll
    for (int q = 0; q < SLOTS; ++q) rc[q] = next[q];
    if (l > 0) load(l - 1);
    double bl = 0.0, il = 0.0;
#pragma unroll
    for (int q = 0; q < SLOTS; ++q)
      if (q == ql) bl = b[q], il = rinv[q];
    bl = __shfl_sync(0xffffffffu, bl, ll);
    il = __shfl_sync(0xffffffffu, il, ll);
    const double tl = bl * il;
    // only slots holding rows i <= l take part: a warp-uniform branch per
    // slot, so the FP64 pipe (~2 DFMA per clock per SM) does no dead work
#pragma unroll
    for (int q = 0; q < SLOTS; ++q) {
      if (q > ql) break;
      if (q == ql && lane == ll) b[q] = tl;
      if (lane + 32 * q < l) b[q] = fma(-tl, rc[q], b[q]);
    }
  }
#pragma unroll
  for (int q = 0; q < SLOTS; ++q) {
    const int i = lane + 32 * q;
    if (i < p) T[(int64_t)j * p + i] = i <= j ? b[q] : 0.0;
  }
}

// ---- one-sided Jacobi: eigenpairs of Y Y^T -------------------------------------

// Eigenpairs from the converged columns of X (column-major, ld): eigenvalue
// = squared column norm, eigenvector = normalised column, sorted descending;
// exactly zero columns are completed to an orthonormal basis.  Called by one
// CTA (any block size that is a multiple of 32).
__device__ void jacobi_finish(int p, const float* X, int ld, double* __restrict__ evals,
                              double* __restrict__ evecs, unsigned* flags) {
  __shared__ int order[512];
  __shared__ float nrm2[512];
  const int tid = threadIdx.x, nt = blockDim.x;
  const int lane = tid & 31, warp = tid >> 5, nw = nt >> 5;
  // eigenvalue i = squared norm of column i
  for (int i = warp; i < p; i += nw) {
    float s = 0.f;
    for (int t = lane; t < p; t += 32) s = fmaf(X[(int64_t)i * ld + t], X[(int64_t)i * ld + t], s);
#pragma unroll
    for (int off = 16; off; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
    if (lane == 0) nrm2[i] = s;
  }
  __syncthreads();
  // descending order by rank (ties broken by index); NaN ranks below
  // everything, so the ranks always form a permutation, and is reported
  for (int i = tid; i < p; i += nt) {
    const float ki = isnan(nrm2[i]) ? -INFINITY : nrm2[i];
    if (!isfinite(nrm2[i])) atomicOr(flags, kFlagNonFinite);
    int rank = 0;
    for (int j = 0; j < p; ++j) {
      const float kj = isnan(nrm2[j]) ? -INFINITY : nrm2[j];
      rank += (kj > ki) || (kj == ki && j < i);
    }
    order[rank] = i;
  }
  __syncthreads();
  for (int r = warp; r < p; r += nw) {
    const int i = order[r];
    const float s = nrm2[i];
    const float inv = s > 0.f ? rsqrtf(s) : 0.f;
    if (lane == 0) evals[r] = (double)s;
    for (int t = lane; t < p; t += 32)
      evecs[(int64_t)r * p + t] = (double)(X[(int64_t)i * ld + t] * inv);
  }
  // Exactly zero columns (null directions of a rank-deficient factor, ranked
  // last) carry no direction: complete the basis so that the refinement
  // starts from an orthonormal matrix.  Column r becomes e_t minus its
  // projection on columns 0..r-1 (twice), for the t with the smallest
  // weight sum_c X_tc^2 (the unit vector farthest from their span).
  __shared__ double wsm[512], vsm[512];
  __shared__ int s_t;
  __syncthreads();  // evecs (global) complete
  for (int r = 0; r < p; ++r) {
    if (nrm2[order[r]] > 0.f) continue;  // uniform: every thread reads the same value
    for (int t = tid; t < p; t += nt) {
      double w = 0.0;
      for (int c = 0; c < r; ++c) {
        const double x = evecs[(int64_t)c * p + t];
        w = fma(x, x, w);
      }
      wsm[t] = w;
    }
    __syncthreads();
    if (tid == 0) {
      int best = 0;
      for (int t = 1; t < p; ++t)
        if (wsm[t] < wsm[best]) best = t;
      s_t = best;
    }
    __syncthreads();
    const int tb = s_t;
    for (int u = tid; u < p; u += nt) {
      double v = u == tb ? 1.0 : 0.0;
      for (int c = 0; c < r; ++c) v -= evecs[(int64_t)c * p + u] * evecs[(int64_t)c * p + tb];
      vsm[u] = v;
    }
    __syncthreads();
    for (int c = tid; c < r; c += nt) {  // second projection: wsm[c] = X_c . v
      double d = 0.0;
      for (int u = 0; u < p; ++u) d = fma(evecs[(int64_t)c * p + u], vsm[u], d);
      wsm[c] = d;
    }
    __syncthreads();
    for (int u = tid; u < p; u += nt) {
      double v = vsm[u];
      for (int c = 0; c < r; ++c) v -= wsm[c] * evecs[(int64_t)c * p + u];
      vsm[u] = v;
    }
    __syncthreads();
    if (tid == 0) {
      double nn = 0.0;
      for (int u = 0; u < p; ++u) nn = fma(vsm[u], vsm[u], nn);
      wsm[0] = nn > 0.0 ? 1.0 / sqrt(nn) : 0.0;
    }
    __syncthreads();
    for (int u = tid; u < p; u += nt) evecs[(int64_t)r * p + u] = vsm[u] * wsm[0];
    __syncthreads();
  }}

// p < 96: the columns in shared memory, 8 lanes per pair of a round, 8 v + lane
// (v < NV) being a lane's rows, held in registers between the sums and the
// rotation; only as many threads as there are pairs to rotate, since a round
// ends with a barrier.  What bounds it is the latency of a round: loads, three
// sums, the rotation's divisions and square roots, stores, barrier.  (1,024
// threads and loops over p read twice: 250 us at p = 50, 145 us here.)  Pairs, tests
// and formulas as in jacobi_kernel below.
__host__ __device__ constexpr int jacobi_small_ld(int NV) {  // == 8 mod 32: 4 neighbouring columns
  return 8 * NV <= 8 ? 8 : 8 * NV <= 40 ? 40 : 8 * NV <= 72 ? 72 : 104;
}

template <int NV>
__global__ void __launch_bounds__(384) jacobi_small_kernel(int p, const double* __restrict__ Y,
                                                           double* __restrict__ evals,
                                                           double* __restrict__ evecs,
                                                           unsigned* flags, int max_sweeps,
                                                           float tol) {
  extern __shared__ float smem[];
  constexpr int ld = jacobi_small_ld(NV);
  float* X = smem;
  const int tid = threadIdx.x, nt = blockDim.x;
  for (int e = tid; e < p * ld; e += nt) {
    const int j = e / ld, i = e % ld;
    X[e] = i < p ? (float)Y[j * p + i] : 0.f;
  }
  const int m = p + (p & 1), w = m - 1;
  const int s = tid >> 3, l8 = tid & 7;
  __syncthreads();
  for (int sweep = 0; sweep < max_sweeps; ++sweep) {
    int a = s == 0 ? 0 : 1 + (s - 1) % w, b = 1 + (m - 2 - s + 2 * w) % w;
    int rotated = 0;
    for (int r = 0; r < m - 1; ++r) {
      const int i = min(a, b), j = max(a, b);
      if (s != 0) a = a == w ? 1 : a + 1;
      b = b == w ? 1 : b + 1;
      const bool live = s < m / 2 && j < p;
      float* xi = X + (live ? i : 0) * ld + l8;
      float* xj = X + (live ? j : 0) * ld + l8;
      // (threads without a pair load nothing: their column 0 has an owner that
      // may be storing it)
      float x[NV] = {}, y[NV] = {};
      if (live) {
#pragma unroll
        for (int v = 0; v < NV; ++v) x[v] = xi[8 * v], y[v] = xj[8 * v];
      }
      float al = 0.f, be = 0.f, ga = 0.f;
#pragma unroll
      for (int v = 0; v < NV; ++v) {
        al = fmaf(x[v], x[v], al);
        be = fmaf(y[v], y[v], be);
        ga = fmaf(x[v], y[v], ga);
      }
#pragma unroll
      for (int off = 4; off; off >>= 1) {
        al += __shfl_xor_sync(0xffffffffu, al, off);
        be += __shfl_xor_sync(0xffffffffu, be, off);
        ga += __shfl_xor_sync(0xffffffffu, ga, off);
      }
      if (live && fabsf(ga) > tol * sqrtf(al * be) && ga != 0.f) {
        const float zeta = (be - al) / (2.f * ga);
        const float t = copysignf(1.f, zeta) / (fabsf(zeta) + sqrtf(1.f + zeta * zeta));
        const float c = rsqrtf(1.f + t * t), sn = c * t;
#pragma unroll
        for (int v = 0; v < NV; ++v) {
          xi[8 * v] = c * x[v] - sn * y[v];
          xj[8 * v] = sn * x[v] + c * y[v];
        }
        rotated = 1;
      }
      __syncthreads();
    }
    if (!__syncthreads_or(rotated)) break;
  }
  jacobi_finish(p, X, ld, evals, evecs, flags);
}

template <int NV>
cudaError_t launch_jacobi_small(int p, const double* Y, double* evals, double* evecs,
                                unsigned* flags, int max_sweeps, float tol, cudaStream_t s) {
  const int threads = (int)std::max<int64_t>(64, round_up(8 * ((p + 1) / 2), 32));
  static bool set = false;
  if (!set) {  // (static and dynamic together pass 48 KB from p = 87)
    MMSB_CUDA_TRY(cudaFuncSetAttribute(jacobi_small_kernel<NV>,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)sizeof(float) * 8 * NV * jacobi_small_ld(NV)));
    set = true;
  }
  jacobi_small_kernel<NV><<<1, threads, sizeof(float) * p * jacobi_small_ld(NV), s>>>(
      p, Y, evals, evecs, flags, max_sweeps, tol);
  ++g_launch_count;
  return cudaGetLastError();
}

// (the columns in global memory: where the cluster form below does not fit)
__global__ void __launch_bounds__(1024) jacobi_kernel(int p, const double* __restrict__ Y,
                                                      double* __restrict__ evals,
                                                      double* __restrict__ evecs,
                                                      float* __restrict__ gwork,
                                                      unsigned* flags, int max_sweeps, float tol) {
  float* X = gwork;  // column-major p x p
  const int tid = threadIdx.x, nt = blockDim.x;
  for (int64_t e = tid; e < (int64_t)p * p; e += nt) X[e] = (float)Y[e];
  const int m = p + (p & 1);  // players in the round-robin tournament
  __syncthreads();
  int sweep = 0;
  // a group of 8 lanes per column pair: up to nt / 8 pairs of a round at once
  const int grp = tid >> 3, l8 = tid & 7, ngrp = nt >> 3;
  // circle method: in round r, slot s pairs player a = 1 + (s - 1 + r) mod (m - 1)
  // (player 0 for s = 0) with b = 1 + (m - 2 - s + r) mod (m - 1); both
  // advance by one (wrapping inside 1 .. m - 1) from round to round.  A
  // thread serves slots s = grp, grp + ngrp (up to m / 2 <= 256 slots).
  const int w = m - 1;
  auto wrap_next = [w](int v) { return v == w ? 1 : v + 1; };
  for (; sweep < max_sweeps; ++sweep) {
    int pa[2], pb[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int s = grp + h * ngrp;
      pa[h] = s == 0 ? 0 : 1 + (s - 1) % w;
      pb[h] = 1 + (m - 2 - s + 2 * w) % w;
    }
    int rotated = 0;  // any rotation by this thread's groups in this sweep
    for (int r = 0; r < m - 1; ++r) {
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int s = grp + h * ngrp;
        if (h * ngrp >= m / 2) break;  // uniform across the block
        const int a = pa[h], b = pb[h];
        if (s != 0) pa[h] = wrap_next(a);
        pb[h] = wrap_next(b);
        const int i = min(a, b), j = max(a, b);
        const bool live = s < m / 2 && j < p;
        float* xi = X + (int64_t)(live ? i : 0) * p;
        float* xj = X + (int64_t)(live ? j : 0) * p;
        float al = 0.f, be = 0.f, ga = 0.f;
        if (live) {
#pragma unroll 4
          for (int t = l8; t < p; t += 8) {
            const float u = xi[t], v = xj[t];
            al = fmaf(u, u, al);
            be = fmaf(v, v, be);
            ga = fmaf(u, v, ga);
          }
        }
#pragma unroll
        for (int off = 4; off; off >>= 1) {
          al += __shfl_xor_sync(0xffffffffu, al, off);
          be += __shfl_xor_sync(0xffffffffu, be, off);
          ga += __shfl_xor_sync(0xffffffffu, ga, off);
        }
        if (live && fabsf(ga) > tol * sqrtf(al * be) && ga != 0.f) {
          const float zeta = (be - al) / (2.f * ga);
          const float t = copysignf(1.f, zeta) / (fabsf(zeta) + sqrtf(1.f + zeta * zeta));
          const float c = rsqrtf(1.f + t * t), sn = c * t;
#pragma unroll 4
          for (int u = l8; u < p; u += 8) {
            const float x = xi[u], y = xj[u];
            xi[u] = c * x - sn * y;
            xj[u] = sn * x + c * y;
          }
          rotated = 1;
        }
      }
      __syncthreads();
    }
    if (!__syncthreads_or(rotated)) break;
  }
  jacobi_finish(p, X, p, evals, evecs, flags);
}

// ---- one-sided Jacobi on a cluster (block round-robin) --------------------------
//
// The p columns form 16 blocks of b = ceil(p / 16) columns; CTA t of an
// 8-CTA cluster holds two blocks in shared memory.  A sweep is 15 block rounds
// of the circle method over the 16 blocks (every pair of blocks meets once);
// in a block round each CTA rotates every column of its first block against
// every column of its second (b rounds of b disjoint pairs), and in the first
// block round of a sweep also the pairs inside each of its blocks.  So each
// sweep visits every column pair once, as the cyclic method does, while all
// rotations run on columns in local shared memory.  Between block rounds
// each CTA pulls the two blocks of its next round from their holders through
// DSMEM into its other buffer set (one cluster barrier per block round).
// A pair group of 16 lanes rotates one pair; rotations use the same test and
// formulas as jacobi_kernel.
constexpr int kJcCtas = 8, kJcBlocks = 2 * kJcCtas;

__host__ __device__ inline int jc_ld(int p) { return p + ((16 - p % 32) + 32) % 32; }  // == 16 mod 32
__host__ __device__ inline int jc_b(int p) { return (p + kJcBlocks - 1) / kJcBlocks; }

// blocks of CTA t in block round r (circle method, player 0 fixed)
__device__ __forceinline__ void jc_players(int t, int r, int& a, int& b) {
  constexpr int w = kJcBlocks - 1;
  a = t == 0 ? 0 : 1 + ((t - 1 + r) % w);
  b = 1 + ((kJcBlocks - 2 - t + r) % w);
}

// LANES lanes rotate one pair: 32 (a warp, shorter dependent chains) while a
// block has at most 16 columns, else 16 so that 32 pairs fit a round
template <int LANES, int NV>
__global__ void __launch_bounds__(512) jacobi_cluster_kernel(int p, const double* __restrict__ Y,
                                                             double* __restrict__ evals,
                                                             double* __restrict__ evecs,
                                                             float* __restrict__ gwork,
                                                             unsigned* flags, int max_sweeps,
                                                             float tol) {
  namespace cg = cooperative_groups;
  cg::cluster_group cluster = cg::this_cluster();
  extern __shared__ __align__(16) float jsm[];
  const int ld = jc_ld(p), b = jc_b(p);
  const int t = (int)cluster.block_rank();
  // buffer set q holds slot 0 (first block) and slot 1 (second block)
  auto slot = [&](int q, int sl) { return jsm + (size_t)(2 * q + sl) * b * ld; };
  __shared__ int s_rot[2];
  const int tid = threadIdx.x, nt = blockDim.x;
  const int grp = tid / LANES, ln = tid % LANES, ngrp = nt / LANES;
  auto ncols = [&](int x) { return max(0, min(b, p - x * b)); };
  int cur = 0, pa, pb;
  jc_players(t, 0, pa, pb);
  for (int sl = 0; sl < 2; ++sl) {
    const int x = sl ? pb : pa, nc = ncols(x);
    float* dst = slot(0, sl);
    for (int e = tid; e < b * ld; e += nt) {
      const int c = e / ld, i = e % ld;
      dst[e] = (c < nc && i < p) ? (float)Y[(int64_t)(x * b + c) * p + i] : 0.f;
    }
  }
  if (tid == 0) s_rot[0] = s_rot[1] = 0;
  __syncthreads();
  // rotate column u against column v (both in local shared memory) if they
  // are not yet orthogonal to tol; uniform shuffles across the warp
  // (16-byte vectors: a column's ld is a multiple of 16 floats and its rows
  // past p hold zeros, which the rotations keep; the rotation parameters use
  // the fast division: the FP64 refinement that follows absorbs its ulps.
  // The sweep count is set by the issue rate of this loop: ~200 instructions
  // per rotation with scalar words)
  const int n4 = (p + 3) / 4;
  const float tol2 = tol * tol;
  auto rotate = [&](float* u, float* v, bool live, int& rotated) {
    float al = 0.f, be = 0.f, ga = 0.f;
    float4* u4 = reinterpret_cast<float4*>(u);
    float4* v4 = reinterpret_cast<float4*>(v);
    if (live) {
#pragma unroll 2
      for (int i = ln; i < n4; i += LANES) {
        const float4 x = u4[i], y = v4[i];
        al = fmaf(x.x, x.x, fmaf(x.y, x.y, fmaf(x.z, x.z, fmaf(x.w, x.w, al))));
        be = fmaf(y.x, y.x, fmaf(y.y, y.y, fmaf(y.z, y.z, fmaf(y.w, y.w, be))));
        ga = fmaf(x.x, y.x, fmaf(x.y, y.y, fmaf(x.z, y.z, fmaf(x.w, y.w, ga))));
      }
    }
#pragma unroll
    for (int off = LANES / 2; off; off >>= 1) {
      al += __shfl_xor_sync(0xffffffffu, al, off);
      be += __shfl_xor_sync(0xffffffffu, be, off);
      ga += __shfl_xor_sync(0xffffffffu, ga, off);
    }
    if (live && ga * ga > tol2 * (al * be) && ga != 0.f) {
      const float zeta = __fdividef(be - al, 2.f * ga);
      const float tt = __fdividef(copysignf(1.f, zeta), fabsf(zeta) + sqrtf(fmaf(zeta, zeta, 1.f)));
      const float c = rsqrtf(fmaf(tt, tt, 1.f)), sn = c * tt;
#pragma unroll 2
      for (int i = ln; i < n4; i += LANES) {
        const float4 x = u4[i], y = v4[i];
        u4[i] = make_float4(c * x.x - sn * y.x, c * x.y - sn * y.y, c * x.z - sn * y.z,
                            c * x.w - sn * y.w);
        v4[i] = make_float4(sn * x.x + c * y.x, sn * x.y + c * y.y, sn * x.z + c * y.z,
                            sn * x.w + c * y.w);
      }
      rotated = 1;
    }
  };
  const int bp = b + (b & 1);  // players of the round-robin inside one block
  bool go = true;
  for (int sweep = 0; sweep < max_sweeps && go; ++sweep) {
    int rotated = 0;
    for (int r = 0; r < kJcBlocks - 1; ++r) {
      float* A = slot(cur, 0);
      float* B = slot(cur, 1);
      const int na = ncols(pa), nb = ncols(pb);
      if (r == 0) {  // pairs inside each block: groups [0, bp/2) block A, [bp/2, bp) block B
        for (int rr = 0; rr < bp - 1; ++rr) {
          for (int g0 = 0; g0 < bp; g0 += ngrp) {
            const int g = g0 + grp, s = g % (bp / 2), side = g / (bp / 2);
            int x, y;
            {
              const int w = bp - 1;
              x = s == 0 ? 0 : 1 + ((s - 1 + rr) % w);
              y = 1 + ((bp - 2 - s + rr) % w);
            }
            const int n = side ? nb : na;
            const bool live = g < bp && x < n && y < n;
            float* base = side ? B : A;
            rotate(base + (size_t)(live ? x : 0) * ld, base + (size_t)(live ? y : 0) * ld, live,
                   rotated);
          }
          __syncthreads();
        }
      }
      // A[i] against B[(i + q) mod b], i = grp + g0.  A[i] stays in the group's
      // registers while it meets the columns of B (NV 16-byte words per lane);
      // sums and rotations are those of rotate(), in the same order: the signs
      // of the eigenvectors hang on every rounding of the early sweeps.  (p =
      // 200 and 101: 1.31 ms on average with both columns in shared memory, 1.03
      // ms here.)
      for (int g0 = 0; g0 < b; g0 += ngrp) {  // (once: ngrp >= b)
        const int i = g0 + grp;
        const bool mine = i < b && i < na;
        float4* u4 = reinterpret_cast<float4*>(A + (size_t)(mine ? i : 0) * ld);
        float4 ax[NV];
#pragma unroll
        for (int e = 0; e < NV; ++e)
          if (ln + LANES * e < n4) ax[e] = u4[ln + LANES * e];
        for (int q = 0; q < b; ++q) {
          int j = i + q;
          if (j >= b) j -= b;
          const bool live = mine && j < nb;
          float4* v4 = reinterpret_cast<float4*>(B + (size_t)(live ? j : 0) * ld);
          float4 bx[NV];
          float al = 0.f, be = 0.f, ga = 0.f;
          if (live) {
#pragma unroll
            for (int e = 0; e < NV; ++e)
              if (ln + LANES * e < n4) {
                bx[e] = v4[ln + LANES * e];
                const float4 x = ax[e], y = bx[e];
                al = fmaf(x.x, x.x, fmaf(x.y, x.y, fmaf(x.z, x.z, fmaf(x.w, x.w, al))));
                be = fmaf(y.x, y.x, fmaf(y.y, y.y, fmaf(y.z, y.z, fmaf(y.w, y.w, be))));
                ga = fmaf(x.x, y.x, fmaf(x.y, y.y, fmaf(x.z, y.z, fmaf(x.w, y.w, ga))));
              }
          }
#pragma unroll
          for (int off = LANES / 2; off; off >>= 1) {
            al += __shfl_xor_sync(0xffffffffu, al, off);
            be += __shfl_xor_sync(0xffffffffu, be, off);
            ga += __shfl_xor_sync(0xffffffffu, ga, off);
          }
          if (live && ga * ga > tol2 * (al * be) && ga != 0.f) {
            const float zeta = __fdividef(be - al, 2.f * ga);
            const float tt = __fdividef(copysignf(1.f, zeta), fabsf(zeta) + sqrtf(fmaf(zeta, zeta, 1.f)));
            const float c = rsqrtf(fmaf(tt, tt, 1.f)), sn = c * tt;
#pragma unroll
            for (int e = 0; e < NV; ++e)
              if (ln + LANES * e < n4) {
                const float4 x = ax[e], y = bx[e];
                ax[e] = make_float4(c * x.x - sn * y.x, c * x.y - sn * y.y, c * x.z - sn * y.z,
                                    c * x.w - sn * y.w);
                v4[ln + LANES * e] = make_float4(sn * x.x + c * y.x, sn * x.y + c * y.y,
                                                 sn * x.z + c * y.z, sn * x.w + c * y.w);
              }
            rotated = 1;
          }
          __syncthreads();
        }
        if (mine) {
#pragma unroll
          for (int e = 0; e < NV; ++e)
            if (ln + LANES * e < n4) u4[ln + LANES * e] = ax[e];
        }
      }
      // end of the sweep: the cluster-wide decision travels with this barrier
      const bool last = r == kJcBlocks - 2;
      if (last) {
        const int any = __syncthreads_or(rotated);
        if (tid == 0) s_rot[sweep & 1] = any;
      }
      __threadfence_block();
      cluster.sync();
      if (last) {
        int any = 0;
        for (int q = 0; q < kJcCtas; ++q) any |= *cluster.map_shared_rank(&s_rot[sweep & 1], q);
        if (!any || sweep + 1 >= max_sweeps) {
          go = false;
          break;  // every CTA decides alike; the blocks stay where they are
        }
      }
      // pull the blocks of the next round from their holders into the other set
      const int rn = (r + 1) % (kJcBlocks - 1);
      int na2, nb2;
      jc_players(t, rn, na2, nb2);
      for (int sl = 0; sl < 2; ++sl) {
        const int x = sl ? nb2 : na2;
        int src = -1, ssl = 0;
        for (int u = 0; u < kJcCtas; ++u) {
          int ua, ub;
          jc_players(u, r, ua, ub);
          if (ua == x) { src = u; ssl = 0; }
          if (ub == x) { src = u; ssl = 1; }
        }
        const float4* from = reinterpret_cast<const float4*>(cluster.map_shared_rank(slot(cur, ssl), src));
        float4* to = reinterpret_cast<float4*>(slot(cur ^ 1, sl));
        for (int e = tid; e < b * ld / 4; e += nt) to[e] = from[e];
      }
      cur ^= 1;
      pa = na2;
      pb = nb2;
      __syncthreads();
    }
  }
  // converged columns to the work array (column-major, ld p), then CTA 0
  // forms the eigenpairs
  for (int sl = 0; sl < 2; ++sl) {
    const int x = sl ? pb : pa, nc = ncols(x);
    const float* src = slot(cur, sl);
    for (int e = tid; e < nc * p; e += nt) {
      const int c = e / p, i = e % p;
      gwork[(int64_t)(x * b + c) * p + i] = src[(size_t)c * ld + i];
    }
  }
  __threadfence();
  cluster.sync();
  if (t == 0) jacobi_finish(p, gwork, p, evals, evecs, flags);
}

// ---- Gram-Schmidt of the columns of a small m x p FP64 matrix (one CTA) -------------
// orthogonalize_cols (CPU/Spectral.cpp:146-166) processes the columns left to
// right, removes the projections on the previous (orthonormal or zero)
// columns and normalises; a residual norm <= tol zeroes the column.  Here each
// column is projected twice with classical Gram-Schmidt (CGS2), which matches
// modified Gram-Schmidt to round-off and turns the inner loop into parallel
// dot products (m, p <= 512).

__global__ void __launch_bounds__(1024) cgs2_cols_kernel(int m, int p, const double* __restrict__ P,
                                                         int ldp, double* __restrict__ Q, int ldq,
                                                         double tol) {
  constexpr int kGroups = 8;  // thread groups splitting the projection sum
  extern __shared__ double sh[];
  double* v = sh;                // m
  double* d = sh + m;            // p
  double* part = sh + m + p;     // kGroups x m partial projections
  __shared__ double red[32];
  const int tid = threadIdx.x, nt = blockDim.x, lane = tid & 31, warp = tid >> 5, nw = nt >> 5;
  const int gsz = nt / kGroups, grp = tid / gsz, gt = tid % gsz;
  __shared__ int kept;
  __shared__ bool skip;
  if (tid == 0) kept = 0;
  for (int j = 0; j < p; ++j) {
    for (int r = tid; r < m; r += nt) v[r] = P[(int64_t)j * ldp + r];
    __syncthreads();
    if (kept == m) {
      // the kept columns span R^m: the residual of v is round-off, about
      // 1e-15 |v|, below tol whenever |v| < 1e10 tol, and the column is
      // dropped without the projections
      double nv = 0.0;
      for (int r = tid; r < m; r += nt) nv = fma(v[r], v[r], nv);
#pragma unroll
      for (int off = 16; off; off >>= 1) nv += __shfl_xor_sync(0xffffffffu, nv, off);
      if (lane == 0) red[warp] = nv;
      __syncthreads();
      if (tid == 0) {
        double tot = 0.0;
        for (int w = 0; w < nw; ++w) tot += red[w];
        skip = sqrt(tot) < 1e10 * tol;
      }
      __syncthreads();
      if (skip) {
        for (int r = tid; r < m; r += nt) Q[(int64_t)j * ldq + r] = 0.0;
        continue;  // (no shared state written below before the next barrier)
      }
    }
    for (int pass = 0; pass < 2; ++pass) {
      // d_i = Q_i . v for i < j: a warp per previous column, lanes along rows
      for (int i = warp; i < j; i += nw) {
        const double* qi = Q + (int64_t)i * ldq;
        double s = 0.0;
        for (int r = lane; r < m; r += 32) s = fma(qi[r], v[r], s);
#pragma unroll
        for (int off = 16; off; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
        if (lane == 0) d[i] = s;
      }
      __syncthreads();
      // v -= sum_i d_i Q_i: group g sums the columns i = g (mod kGroups)
      for (int r = gt; r < m; r += gsz) {
        double s = 0.0;
        for (int i = grp; i < j; i += kGroups) s = fma(d[i], Q[(int64_t)i * ldq + r], s);
        part[grp * m + r] = s;
      }
      __syncthreads();
      for (int r = tid; r < m; r += nt) {
        double s = 0.0;
#pragma unroll
        for (int g = 0; g < kGroups; ++g) s += part[g * m + r];
        v[r] -= s;
      }
      __syncthreads();
    }
    double nrm = 0.0;
    for (int r = tid; r < m; r += nt) nrm = fma(v[r], v[r], nrm);
#pragma unroll
    for (int off = 16; off; off >>= 1) nrm += __shfl_xor_sync(0xffffffffu, nrm, off);
    if (lane == 0) red[warp] = nrm;
    __syncthreads();
    double tot = 0.0;
    for (int w = 0; w < nw; ++w) tot += red[w];
    const double nn = sqrt(tot);
    const double sc = nn > tol ? 1.0 / nn : 0.0;
    for (int r = tid; r < m; r += nt) Q[(int64_t)j * ldq + r] = v[r] * sc;
    if (tid == 0 && nn > tol) ++kept;
    __syncthreads();
  }
}

// The same CGS2 with the rows spread over a cluster of CL CTAs, so that the
// FP64 work (about 4 m p^2 / 2 multiply-adds) runs on CL SMs instead of one.
// CTA r keeps rows [r R, r R + R) of every finished column of Q in shared
// memory; each projection pass forms partial dot products over its rows, the
// cluster sums them (every CTA reads all partials through DSMEM, adding in
// rank order, so all CTAs hold identical sums and take identical branches),
// and each CTA updates its own rows.  Three cluster barriers per column
// (pass 1 with |v|^2, pass 2, the final norm) are what bounds it; the partial
// buffers alternate so that a buffer is rewritten only after every CTA has read
// it.  m = 101, p = 200: 1.25 ms; m = 151, p = 300: 3.7 ms.  (Three sums per
// block of 8 columns took 0.68 and 2.65 ms, but in another order: the signs of
// W's columns hang on it.)
template <int CL>
__global__ void __launch_bounds__(256) cgs2_cols_cluster_kernel(int m, int p,
                                                                const double* __restrict__ P,
                                                                int ldp, double* __restrict__ Q,
                                                                int ldq, double tol) {
  namespace cg = cooperative_groups;
  cg::cluster_group cluster = cg::this_cluster();
  extern __shared__ double csh[];
  const int R = (m + CL - 1) / CL;                 // rows per CTA
  const int rank = (int)cluster.block_rank();
  const int r0 = rank * R, nr = max(0, min(R, m - r0));
  double* Qs = csh;                                 // Qs[i R + rr] = Q[r0 + rr, i]
  double* v = Qs + (size_t)R * p;                   // R
  double* part = v + R;                             // 2 x (p + 1) partial sums
  double* d = part + 2 * (p + 1);                   // p + 1 reduced sums
  const int tid = threadIdx.x, nt = blockDim.x, lane = tid & 31, warp = tid >> 5, nw = nt >> 5;
  int buf = 0, kept = 0;
  // partial sums of Q_i . v (i < cnt) and, with_norm, |v|^2 in slot cnt;
  // then the cluster-wide sums into d[0 .. cnt]
  auto reduce = [&](int cnt, bool with_norm) {
    double* pb = part + buf * (p + 1);
    for (int i = tid; i < cnt; i += nt) {
      double s = 0.0;
      for (int rr = 0; rr < nr; ++rr) s = fma(Qs[(size_t)i * R + rr], v[rr], s);
      pb[i] = s;
    }
    if (with_norm && warp == 0) {
      double s = 0.0;
      for (int rr = lane; rr < nr; rr += 32) s = fma(v[rr], v[rr], s);
#pragma unroll
      for (int off = 16; off; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
      if (lane == 0) pb[cnt] = s;
    }
    cluster.sync();
    const int tot = cnt + (with_norm ? 1 : 0);
    for (int i = tid; i < tot; i += nt) {
      double s = 0.0;
      for (int q = 0; q < CL; ++q) s += cluster.map_shared_rank(pb, q)[i];
      d[i] = s;
    }
    buf ^= 1;
    __syncthreads();
  };
  // v -= sum_{i < cnt} d_i Q_i over this CTA's rows (a warp per row)
  auto subtract = [&](int cnt) {
    for (int rr = warp; rr < nr; rr += nw) {
      double s = 0.0;
      for (int i = lane; i < cnt; i += 32) s = fma(d[i], Qs[(size_t)i * R + rr], s);
#pragma unroll
      for (int off = 16; off; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
      if (lane == 0) v[rr] -= s;
    }
    __syncthreads();
  };
  for (int j = 0; j < p; ++j) {
    for (int rr = tid; rr < nr; rr += nt) v[rr] = P[(int64_t)j * ldp + r0 + rr];
    __syncthreads();
    reduce(j, true);  // pass 1 dots and |v|^2
    // the kept columns span R^m: the residual of v is round-off, about
    // 1e-15 |v|, below tol whenever |v| < 1e10 tol, and the column is dropped
    if (kept == m && sqrt(d[j]) < 1e10 * tol) {
      for (int rr = tid; rr < nr; rr += nt) {
        Qs[(size_t)j * R + rr] = 0.0;
        Q[(int64_t)j * ldq + r0 + rr] = 0.0;
      }
      __syncthreads();
      continue;
    }
    subtract(j);
    reduce(j, false);  // pass 2
    subtract(j);
    reduce(0, true);   // |v|^2 after both passes
    const double nn = sqrt(d[0]);
    const double sc = nn > tol ? 1.0 / nn : 0.0;
    for (int rr = tid; rr < nr; rr += nt) {
      const double qv = v[rr] * sc;
      Qs[(size_t)j * R + rr] = qv;
      Q[(int64_t)j * ldq + r0 + rr] = qv;
    }
    if (nn > tol) ++kept;
    __syncthreads();
  }
  cluster.sync();  // keep shared memory alive until every remote read is done
}

template <int CL>
static cudaError_t launch_cgs2_cluster(int m, int p, const double* P, int ldp, double* Q, int ldq,
                                       double tol, size_t sm, cudaStream_t s) {
  static bool set = false;
  if (!set) {
    MMSB_CUDA_TRY(cudaFuncSetAttribute(cgs2_cols_cluster_kernel<CL>,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024));
    if (CL > 8)
      MMSB_CUDA_TRY(cudaFuncSetAttribute(cgs2_cols_cluster_kernel<CL>,
                                         cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    set = true;
  }
  cudaLaunchConfig_t lc = {};
  lc.gridDim = dim3(CL);
  lc.blockDim = dim3(256);
  lc.dynamicSmemBytes = sm;
  lc.stream = s;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = CL;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = 1;
  lc.attrs = at;
  lc.numAttrs = 1;
  return cudaLaunchKernelEx(&lc, cgs2_cols_cluster_kernel<CL>, m, p, P, ldp, Q, ldq, tol);
}

// ---- Ogita-Aishima refinement of all eigenpairs (FP64) ------------------------------
// Given A (n x n), X (approximate eigenvectors), R = I - X^T X and S = X^T A X,
// computes E with X' = X + X E (Ogita & Aishima 2018, Algorithm 1); eigenvalue
// estimates are written to lam.  One CTA (n <= 512).

// Statistics: lam_i = S_ii / (X^T X)_ii and the three maxima behind the
// cluster threshold delta = 2 (||S - diag(lam)|| + ||A|| ||I - X^T X||):
// spectral norms bounded by the maximum column abs-sum (symmetric matrices),
// ||A|| ~ max |lam_i| (Frobenius norms would over-cluster by ~sqrt(n)).  A
// warp per column, lanes along its contiguous rows, eight columns per CTA;
// the maxima (non-negative, so their IEEE bit patterns order like the
// values) are combined with atomicMax into mx[0..2], zeroed beforehand.
__global__ void __launch_bounds__(256) oa_stats_kernel(int n, const double* __restrict__ XtX,
                                                       const double* __restrict__ S,
                                                       double* __restrict__ lam,
                                                       unsigned long long* __restrict__ mx) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int j = blockIdx.x * (blockDim.x >> 5) + warp;
  if (j >= n) return;
  const double xx = XtX[(int64_t)j * n + j];  // = 1 - R_jj
  const double lj = xx > 0.0 ? S[(int64_t)j * n + j] / xx : 0.0;
  double cs = 0.0, cr = 0.0;
  for (int i = lane; i < n; i += 32) {
    const int64_t e = (int64_t)j * n + i;
    cs += fabs(S[e] - (i == j ? lj : 0.0));
    cr += fabs((i == j ? 1.0 : 0.0) - XtX[e]);
  }
#pragma unroll
  for (int off = 16; off; off >>= 1) {
    cs += __shfl_xor_sync(0xffffffffu, cs, off);
    cr += __shfl_xor_sync(0xffffffffu, cr, off);
  }
  if (lane == 0) {
    lam[j] = lj;
    atomicMax(mx + 0, (unsigned long long)__double_as_longlong(cs));
    atomicMax(mx + 1, (unsigned long long)__double_as_longlong(fabs(lj)));
    atomicMax(mx + 2, (unsigned long long)__double_as_longlong(cr));
  }
}

// The correction E (Ogita & Aishima 2018, Algorithm 1): E_ii = R_ii / 2,
// E_ij = (S_ij + lam_j R_ij) / (lam_j - lam_i) where |lam_j - lam_i| > delta,
// else R_ij / 2, with R = I - X^T X.  One CTA row per column j (blockIdx.y),
// spreading the n^2 FP64 divisions over the GPU.
__global__ void __launch_bounds__(256) oa_correction_kernel(int n, const double* __restrict__ XtX,
                                                            const double* __restrict__ S,
                                                            double* __restrict__ E,
                                                            const double* __restrict__ lam,
                                                            const unsigned long long* __restrict__ mx,
                                                            double* __restrict__ delta_state) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x, j = blockIdx.y;
  const double dl = 2.0 * (__longlong_as_double((long long)mx[0]) +
                           __longlong_as_double((long long)mx[1]) * __longlong_as_double((long long)mx[2]));
  if (i == 0 && j == 0) delta_state[0] = dl;  // reported for diagnostics
  if (i >= n) return;
  const int64_t e = (int64_t)j * n + i;
  const double r = (i == j ? 1.0 : 0.0) - XtX[e];
  double v = 0.5 * r;
  if (i != j) {
    const double gap = lam[j] - lam[i];
    if (fabs(gap) > dl) v = (S[e] + lam[j] * r) / gap;
  }
  E[e] = v;
}

// Columns of X reordered by descending lam (ties by index; NaN ranks last so
// the ranks always form a permutation, and is reported through the flag word).
// A warp per column: its rank, then the copy.  (One CTA for all took 51 us at n =
// 200, most of it FP64 comparisons at 2 per clock: the keys compare as integers
// whose order is that of the values.)
__device__ __forceinline__ long long order_key(double v) {
  if (isnan(v)) v = -INFINITY;
  if (v == 0.0) v = 0.0;  // -0 ties with +0
  const long long b = __double_as_longlong(v);
  return b < 0 ? (long long)0x8000000000000000ull - b : b;
}

__global__ void __launch_bounds__(256) sort_eigen_kernel(int n, const double* __restrict__ lam,
                                                         const double* __restrict__ X,
                                                         double* __restrict__ evals,
                                                         double* __restrict__ evecs,
                                                         unsigned* flags) {
  const int lane = threadIdx.x & 31, i = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (i >= n) return;
  const double li = lam[i];
  const long long ki = order_key(li);
  int rank = 0;
  for (int j = lane; j < n; j += 32) {
    const long long kj = order_key(lam[j]);
    rank += (kj > ki) || (kj == ki && j < i);
  }
  rank = __reduce_add_sync(0xffffffffu, rank);
  if (lane == 0) {
    evals[rank] = li;
    if (!isfinite(li) && flags) atomicOr(flags, kFlagNonFinite);
  }
  for (int r = lane; r < n; r += 32) evecs[(int64_t)rank * n + r] = X[(int64_t)i * n + r];
}

// All refinement steps and the sort in one kernel, for small n: as kernels of
// their own (four products, the two above and a memset per step, each over n / 8
// tiles) they are 3 to 6 us of latency each, about 90 us at n = 10 and 130 us at n = 50,
// 20 and 45 us here.  The columns are split over a cluster (one CTA up to n =
// 16, else 16: the FP64 units of more SMs); each CTA holds A and all of X and
// sends its new columns, eigenvalues and column sums to the others.  An entry per
// thread; every sum is the same chain as in the kernels above.
constexpr int kOaMax = 64;

template <int CL>
__global__ void __launch_bounds__(256) oa_refine_kernel(int n, int steps, const double* __restrict__ A,
                                                        const double* __restrict__ X0,
                                                        double* __restrict__ evals,
                                                        double* __restrict__ evecs,
                                                        double* __restrict__ delta_state,
                                                        unsigned* flags) {
  namespace cg = cooperative_groups;
  extern __shared__ double sm[];
  const int ld = n | 1, nc = (n + CL - 1) / CL;  // odd stride: rows and columns free of conflicts
  const int rank = CL > 1 ? (int)cg::this_cluster().block_rank() : 0;
  const int j0 = rank * nc, own = max(0, min(nc, n - j0));
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  double *As = sm, *Xs = As + n * ld, *Xn = Xs + n * ld, *AX = Xn + n * ld, *G = AX + nc * ld,
         *S = G + nc * ld, *lam = S + nc * ld, *mx = lam + n;  // mx: 3 column sums of n each
  auto sync_all = [&]() {
    if (CL > 1) cg::this_cluster().sync();
    else __syncthreads();
  };
  auto put = [&](double* p, int q, double v) {  // p in CTA q's shared memory
    if (CL > 1) *cg::this_cluster().map_shared_rank(p, q) = v;
    else *p = v;
  };
  for (int e = tid; e < n * n; e += 256) {
    const int i = e % n, j = e / n;
    As[j * ld + i] = A[e];
    Xs[j * ld + i] = X0[e];
  }
  sync_all();  // (and every CTA of the cluster has started)
  const int i = tid % n, jc = tid / n, j = j0 + jc;
  const bool live = jc < own;
  const int o = jc * ld + i;
  for (int step = 0; step < steps; ++step) {
    if (live) {
      double ax = 0.0, g = 0.0;
#pragma unroll 2
      for (int kk = 0; kk < n; ++kk) {
        const double x = Xs[j * ld + kk];
        ax = fma(As[kk * ld + i], x, ax);
        g = fma(Xs[i * ld + kk], x, g);
      }
      AX[o] = ax;
      G[o] = g;
    }
    __syncthreads();
    if (live) {
      double v = 0.0;
#pragma unroll 2
      for (int kk = 0; kk < n; ++kk) v = fma(Xs[i * ld + kk], AX[jc * ld + kk], v);
      S[o] = v;
    }
    __syncthreads();
    for (int c = warp; c < own; c += 8) {
      const int jj = j0 + c;
      const double xx = G[c * ld + jj];  // = 1 - R_jj
      const double lj = xx > 0.0 ? S[c * ld + jj] / xx : 0.0;
      double cs = 0.0, cr = 0.0;
      for (int r = lane; r < n; r += 32) {
        cs += fabs(S[c * ld + r] - (r == jj ? lj : 0.0));
        cr += fabs((r == jj ? 1.0 : 0.0) - G[c * ld + r]);
      }
#pragma unroll
      for (int off = 16; off; off >>= 1) {
        cs += __shfl_xor_sync(0xffffffffu, cs, off);
        cr += __shfl_xor_sync(0xffffffffu, cr, off);
      }
      if (lane < CL) {
        put(lam + jj, lane, lj);
        put(mx + jj, lane, cs);
        put(mx + n + jj, lane, fabs(lj));
        put(mx + 2 * n + jj, lane, cr);
      }
    }
    sync_all();
    unsigned long long m[3];  // (bit patterns order like the values, NaN above all)
#pragma unroll
    for (int q = 0; q < 3; ++q) {
      m[q] = 0ull;
      for (int r = lane; r < n; r += 32)
        m[q] = max(m[q], (unsigned long long)__double_as_longlong(mx[q * n + r]));
#pragma unroll
      for (int off = 16; off; off >>= 1) m[q] = max(m[q], __shfl_xor_sync(0xffffffffu, m[q], off));
    }
    const double dl = 2.0 * (__longlong_as_double((long long)m[0]) +
                             __longlong_as_double((long long)m[1]) * __longlong_as_double((long long)m[2]));
    if (rank == 0 && tid == 0) delta_state[0] = dl;  // reported for diagnostics
    if (live) {
      const double r = (i == j ? 1.0 : 0.0) - G[o];
      double v = 0.5 * r;
      if (i != j) {
        const double gap = lam[j] - lam[i];
        if (fabs(gap) > dl) v = (S[o] + lam[j] * r) / gap;
      }
      AX[o] = v;  // E
    }
    __syncthreads();
    if (live) {
      double v = 0.0;
#pragma unroll 2
      for (int kk = 0; kk < n; ++kk) v = fma(Xs[kk * ld + i], AX[jc * ld + kk], v);
      v += Xs[j * ld + i];
      for (int q = 0; q < CL; ++q) put(Xn + j * ld + i, q, v);
    }
    sync_all();
    double* t = Xs;
    Xs = Xn;
    Xn = t;
  }
  for (int c = warp; c < own; c += 8) {  // as sort_eigen_kernel
    const int jj = j0 + c;
    const double lj = lam[jj];
    const long long kj = order_key(lj);
    int at = 0;
    for (int r = lane; r < n; r += 32) {
      const long long kr = order_key(lam[r]);
      at += (kr > kj) || (kr == kj && r < jj);
    }
    at = __reduce_add_sync(0xffffffffu, at);
    if (lane == 0) {
      evals[at] = lj;
      if (!isfinite(lj) && flags) atomicOr(flags, kFlagNonFinite);
    }
    for (int r = lane; r < n; r += 32) evecs[(int64_t)at * n + r] = Xs[jj * ld + r];
  }
}

size_t oa_refine_smem(int n, int CL) {
  const int ld = n | 1, nc = (n + CL - 1) / CL;
  return sizeof(double) * ((size_t)3 * n * ld + 3 * nc * ld + 4 * n);
}

template <int CL>
cudaError_t oa_refine_config(int n, cudaStream_t s, cudaLaunchConfig_t* lc,
                             cudaLaunchAttribute* at) {
  static bool set = false;
  if (!set) {
    MMSB_CUDA_TRY(cudaFuncSetAttribute(oa_refine_kernel<CL>,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)oa_refine_smem(CL > 1 ? kOaMax : 16, CL)));
    if (CL > 8)
      MMSB_CUDA_TRY(cudaFuncSetAttribute(oa_refine_kernel<CL>,
                                         cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    set = true;
  }
  *lc = cudaLaunchConfig_t{};
  lc->gridDim = dim3(CL);
  lc->blockDim = dim3(256);
  lc->dynamicSmemBytes = oa_refine_smem(n, CL);
  lc->stream = s;
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = CL;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = 1;
  lc->attrs = at;
  lc->numAttrs = CL > 1 ? 1 : 0;
  return cudaSuccess;
}

// P (rows x q, row-major panel ld) gets column `col` = v (FP64 vector, length rows)
__global__ void panel_set_col_kernel(float* __restrict__ P, int ld, int64_t rows, int col,
                                     const double* __restrict__ v) {
  for (int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; r < rows;
       r += (int64_t)gridDim.x * blockDim.x)
    P[r * ld + col] = (float)v[r];
}

// dst (rows x ld_d) first q columns = src (rows x ld_s) first q columns, rest zero
__global__ void panel_copy_kernel(const float* __restrict__ src, int lds, int64_t rows, int q,
                                  float* __restrict__ dst, int ldd) {
  const int64_t total = rows * ldd;
  for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < total;
       e += (int64_t)gridDim.x * blockDim.x) {
    const int64_t r = e / ldd;
    const int c = (int)(e % ldd);
    dst[e] = c < q ? src[r * lds + c] : 0.f;
  }
}

// ---- Philox-4x32-10 Gaussian panel (Salmon et al., SC'11) -----------------------

__device__ __forceinline__ void philox_round(uint32_t c[4], uint32_t k[2]) {
  const uint32_t M0 = 0xD2511F53u, M1 = 0xCD9E8D57u;
  const uint32_t hi0 = __umulhi(M0, c[0]), lo0 = M0 * c[0];
  const uint32_t hi1 = __umulhi(M1, c[2]), lo1 = M1 * c[2];
  const uint32_t n0 = hi1 ^ c[1] ^ k[0], n1 = lo1, n2 = hi0 ^ c[3] ^ k[1], n3 = lo0;
  c[0] = n0;
  c[1] = n1;
  c[2] = n2;
  c[3] = n3;
  k[0] += 0x9E3779B9u;
  k[1] += 0xBB67AE85u;
}

__global__ void gaussian_panel_kernel(float* __restrict__ P, int64_t n, int q, int ld,
                                      uint64_t seed, uint64_t stream) {
  const int64_t total = n * q;
  for (int64_t g = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; g * 4 < total;
       g += (int64_t)gridDim.x * blockDim.x) {
    uint32_t c[4] = {(uint32_t)g, (uint32_t)(g >> 32), (uint32_t)stream, (uint32_t)(stream >> 32)};
    uint32_t k[2] = {(uint32_t)seed, (uint32_t)(seed >> 32)};
#pragma unroll
    for (int r = 0; r < 10; ++r) philox_round(c, k);
    float z[4];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      // Box-Muller on two uniforms in (0, 1]
      const float u1 = ((float)(c[2 * h] >> 8) + 1.f) * (1.f / 16777216.f);
      const float u2 = ((float)(c[2 * h + 1] >> 8) + 0.5f) * (1.f / 16777216.f);
      const float rad = sqrtf(-2.f * logf(u1));
      float sn, cs;
      sincospif(2.f * u2, &sn, &cs);
      z[2 * h] = rad * cs;
      z[2 * h + 1] = rad * sn;
    }
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int64_t idx = g * 4 + e;
      if (idx < total) P[(idx / q) * ld + (idx % q)] = z[e];
    }
  }
}

__global__ void colmajor_to_panel_kernel(const double* __restrict__ A, int64_t rows, int cols,
                                         int64_t lda, float* __restrict__ P, int ldp) {
  const int64_t total = rows * ldp;
  for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < total;
       e += (int64_t)gridDim.x * blockDim.x) {
    const int64_t r = e / ldp;
    const int c = (int)(e % ldp);
    P[e] = c < cols ? (float)A[(int64_t)c * lda + r] : 0.f;
  }
}

__global__ void panel_to_colmajor_kernel(const float* __restrict__ P, int ldp, int64_t rows,
                                         int cols, double* __restrict__ A, int64_t lda) {
  const int64_t total = rows * cols;
  for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < total;
       e += (int64_t)gridDim.x * blockDim.x) {
    const int64_t r = e % rows;
    const int c = (int)(e / rows);
    A[(int64_t)c * lda + r] = (double)P[r * ldp + c];
  }
}

// out = P with column j < q scaled by d[j] (row-major, ld a multiple of 4, also
// in place).  A warp per row, 16 bytes per lane.  Bound by the FP64 unit: one
// FP64 product per entry, rounded to FP32 (the products stand in front of the
// eigensolvers, whose vectors' signs hang on every rounding), with the
// conversions on both sides in integer arithmetic where all four entries allow it
// (a branch: as a select the conversions ran all the same).  50,000 x 100: 18.5 us
// (31 us as a select; 35 us with conversions and the copy before it).
__global__ void __launch_bounds__(256) scale_cols_kernel(const float4* P, int ld4, int64_t n, int q,
                                                         const double* __restrict__ d,
                                                         float4* out) {
  const int lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  for (int c0 = 0; c0 < ld4; c0 += 32) {
    const int c4 = c0 + lane;
    if (c4 >= ld4) continue;
    double f[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) f[u] = 4 * c4 + u < q ? d[4 * c4 + u] : 1.0;
    for (int64_t r = (int64_t)blockIdx.x * nw + (threadIdx.x >> 5); r < n; r += (int64_t)gridDim.x * nw) {
      const float4 v = P[r * ld4 + c4];
      const float x[4] = {v.x, v.y, v.z, v.w};
      float y[4];
      bool plain = true;
#pragma unroll
      for (int u = 0; u < 4; ++u) plain = plain && ((__float_as_uint(x[u]) >> 23) & 0xffu) - 1u <= 253u;
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const double t = widen_normal(x[u]) * f[u];
        plain = plain && narrows(t);
        y[u] = narrow_normal(t);
      }
      if (!plain) {
#pragma unroll
        for (int u = 0; u < 4; ++u) y[u] = (float)((double)x[u] * f[u]);
      }
      out[r * ld4 + c4] = make_float4(y[0], y[1], y[2], y[3]);
    }
  }
}

template <typename T>
__global__ void fill_kernel(T* __restrict__ p, int64_t n, T v) {
  for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < n;
       e += (int64_t)gridDim.x * blockDim.x)
    p[e] = v;
}

__global__ void axpy_kernel(int64_t n, double a, const double* __restrict__ x,
                            double* __restrict__ y) {
  for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < n;
       e += (int64_t)gridDim.x * blockDim.x)
    y[e] += a * x[e];
}

unsigned grid_for(int64_t n, int T = 256) {
  return (unsigned)std::max<int64_t>(1, std::min<int64_t>(8 * kNumSMs, ceil_div(n, T)));
}

}  // namespace

size_t gram_tsk_partials(int64_t n, int pa, int pb) {
  const int ns = gram_use_tc(n, pa, pb) ? gram_tc_nsplit(n, pa, pb) : gram_nsplit(n, pa, pb);
  return (size_t)ns * pa * pb;
}

cudaError_t gram_tsk(const float* A, int lda, int pa, const float* B, int ldb, int pb, int64_t n,
                     double alpha, double* S, double* partials, int64_t partials_cap,
                     cudaStream_t s, unsigned* flags, long long wait_limit) {
  if (gram_use_tc(n, pa, pb)) {
    // tcgen05 (kind::tf32, 3xTF32) partials over row splits, then the FP64 sum
    const int nsplit = gram_tc_nsplit(n, pa, pb);
    const bool sym = A == B && lda == ldb && pa == pb;  // tiles of 128 x 128
    if ((int64_t)nsplit * pa * pb > partials_cap) return cudaErrorInvalidValue;
    MMSB_CUDA_TRY(gram_tc_partial(A, lda, pa, B, ldb, pb, n, partials, nsplit, flags, s,
                                  wait_limit, sym));
    gram_reduce_kernel<<<grid_for((int64_t)pa * pb), 256, 0, s>>>(
        partials, nsplit, (int64_t)pa * pb, alpha, S, sym ? 128 : 0, pa);
    ++g_launch_count;
    return cudaGetLastError();
  }
  const int nsplit = gram_nsplit(n, pa, pb);
  if ((int64_t)nsplit * pa * pb > partials_cap) return cudaErrorInvalidValue;
  const int64_t rows_per_split = round_up(ceil_div(n, nsplit), GR);
  dim3 grid((unsigned)ceil_div(pa, GT), (unsigned)ceil_div(pb, GT), (unsigned)nsplit);
  gram_partial_kernel<<<grid, 256, 0, s>>>(A, lda, pa, B, ldb, pb, n, rows_per_split, partials);
  ++g_launch_count;
  gram_reduce_kernel<<<grid_for((int64_t)pa * pb), 256, 0, s>>>(
      partials, nsplit, (int64_t)pa * pb, alpha, S, 0, pa);
  ++g_launch_count;
  return cudaGetLastError();
}

cudaError_t panel_times_small(const float* M, int ldm, int p, int64_t n, const double* F, int ldf,
                              int q, float* Y, int ldy, cudaStream_t s) {
  if (n == 0) return cudaSuccess;
  dim3 grid((unsigned)ceil_div(n, PT_R), (unsigned)ceil_div(ldy, PT_C));
  panel_small_kernel<<<grid, 256, 0, s>>>(M, ldm, p, n, F, ldf, q, Y, ldy);
  ++g_launch_count;
  return cudaGetLastError();
}

cudaError_t dgemm_small(bool ta, bool tb, int m, int n, int k, double alpha, const double* A,
                        int lda, const double* B, int ldb, double beta, const double* C0, double* C,
                        int ldc, cudaStream_t s) {
  if (m == 0 || n == 0) return cudaSuccess;
  const bool sym = A == B && lda == ldb && ta != tb && m == n && beta == 0.0;
  dim3 grid((unsigned)ceil_div(m, DG_T), (unsigned)ceil_div(n, DG_T));
  dgemm_small_kernel<<<grid, DG_T * DG_T, 0, s>>>(ta, tb, sym, m, n, k, alpha, A, lda, B, ldb, beta,
                                                  C0, C, ldc);
  ++g_launch_count;
  return cudaGetLastError();
}

template <int CL, int KB, typename T>
static cudaError_t launch_chol_cluster(int p, const double* S, int lds, double* R, double drop2,
                                       unsigned* flags, size_t sm, cudaStream_t s) {
  static bool set = false;
  if (!set) {
    MMSB_CUDA_TRY(cudaFuncSetAttribute(chol_upper_cluster_kernel<CL, KB, T>,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024));
    if (CL > 8)
      MMSB_CUDA_TRY(cudaFuncSetAttribute(chol_upper_cluster_kernel<CL, KB, T>,
                                         cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    set = true;
  }
  cudaLaunchConfig_t lc = {};
  lc.gridDim = dim3(CL);
  lc.blockDim = dim3(256);
  lc.dynamicSmemBytes = sm;
  lc.stream = s;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = CL;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = 1;
  lc.attrs = at;
  lc.numAttrs = 1;
  return cudaLaunchKernelEx(&lc, chol_upper_cluster_kernel<CL, KB, T>, p, S, lds, R, drop2, flags);
}

template <typename T>
static cudaError_t chol_upper_drop_t(int p, const double* S, int lds, double* R, double drop2,
                                     unsigned* flags, cudaStream_t s) {
  if (p > 4096) return cudaErrorInvalidValue;
  // p > 64: a 16-CTA cluster (8 where 16 cannot be co-scheduled) while the
  // columns and one row block fit shared memory, else one CTA a column at a time
  // (p = 50: 78 us, the blocked form on one CTA 82 us)
  constexpr int KB = 16;
  static int wide = -1;
  for (int cl : {16, 8}) {
    if (p <= 64) break;
    if (cl == 16 && wide == 0) continue;
    const size_t sm = sizeof(T) * ((size_t)((p + cl - 1) / cl) + KB) * p;
    if (sm > 200 * 1024) break;
    cudaError_t e = cl == 16 ? launch_chol_cluster<16, KB, T>(p, S, lds, R, drop2, flags, sm, s)
                             : launch_chol_cluster<8, KB, T>(p, S, lds, R, drop2, flags, sm, s);
    if (e == cudaSuccess) {
      if (cl == 16) wide = 1;
      ++g_launch_count;
      return e;
    }
    if (cl == 16 && wide == 1) return e;
    cudaGetLastError();
    if (cl == 16) wide = 0;
  }
  chol_upper_kernel<<<1, 1024, sizeof(double) * p, s>>>(p, S, lds, R, drop2, flags);
  ++g_launch_count;
  return cudaGetLastError();
}

cudaError_t chol_upper_drop(int p, const double* S, int lds, double* R, double drop2,
                            unsigned* flags, cudaStream_t s) {
  return chol_upper_drop_t<double>(p, S, lds, R, drop2, flags, s);
}

cudaError_t chol_upper_drop_f32(int p, const double* S, int lds, double* R, unsigned* flags,
                                cudaStream_t s) {
  return chol_upper_drop_t<float>(p, S, lds, R, 0.0, flags, s);
}

cudaError_t trinv_upper(int p, const double* R, double* T, cudaStream_t s) {
  if (p > 512) return cudaErrorInvalidValue;
  // two columns per CTA: the FP64 work spreads over ~p / 2 SMs
  const unsigned grid = (unsigned)ceil_div(p, 2);
  if (p <= 64) trinv_upper_kernel<2><<<grid, 64, 0, s>>>(p, R, T);
  else if (p <= 128) trinv_upper_kernel<4><<<grid, 64, 0, s>>>(p, R, T);
  else if (p <= 256) trinv_upper_kernel<8><<<grid, 64, 0, s>>>(p, R, T);
  else trinv_upper_kernel<16><<<grid, 64, 0, s>>>(p, R, T);
  ++g_launch_count;
  return cudaGetLastError();
}

cudaError_t eig_from_factor(int p, const double* Y, double* evals, double* evecs, float* work,
                            unsigned* flags, cudaStream_t s) {
  if (p > 512) return cudaErrorInvalidValue;
  // the FP64 refinement converges quadratically only from a converged FP32
  // start (6 sweeps left 1e-3 off-diagonal mass at n = 200; 9-10 suffice)
  const int max_sweeps = 15;
  const float tol = 8.f * sqrtf((float)p) * 6e-8f;
  if (p < 96)
    return p <= 16   ? launch_jacobi_small<2>(p, Y, evals, evecs, flags, max_sweeps, tol, s)
           : p <= 32 ? launch_jacobi_small<4>(p, Y, evals, evecs, flags, max_sweeps, tol, s)
           : p <= 56 ? launch_jacobi_small<7>(p, Y, evals, evecs, flags, max_sweeps, tol, s)
           : p <= 72 ? launch_jacobi_small<9>(p, Y, evals, evecs, flags, max_sweeps, tol, s)
                     : launch_jacobi_small<12>(p, Y, evals, evecs, flags, max_sweeps, tol, s);
  // the 8-CTA cluster version while four blocks fit shared memory
  {
    const size_t smc = sizeof(float) * 4 * (size_t)jc_b(p) * jc_ld(p);
    if (smc <= 200 * 1024) {
      // 32 lanes per pair up to p = 256, else 16; NV: words of a column per lane
      const int form = jc_b(p) <= 16 ? 0 : p <= 320 ? 1 : 2;
      auto kernel = form == 0   ? jacobi_cluster_kernel<32, 2>
                    : form == 1 ? jacobi_cluster_kernel<16, 5>
                                : jacobi_cluster_kernel<16, 8>;
      static bool set[3] = {false, false, false};
      if (!set[form]) {
        MMSB_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                           200 * 1024));
        set[form] = true;
      }
      cudaLaunchConfig_t lc = {};
      lc.gridDim = dim3(kJcCtas);
      lc.blockDim = dim3(512);
      lc.dynamicSmemBytes = smc;
      lc.stream = s;
      cudaLaunchAttribute at[1];
      at[0].id = cudaLaunchAttributeClusterDimension;
      at[0].val.clusterDim.x = kJcCtas;
      at[0].val.clusterDim.y = 1;
      at[0].val.clusterDim.z = 1;
      lc.attrs = at;
      lc.numAttrs = 1;
      ++g_launch_count;
      return cudaLaunchKernelEx(&lc, kernel, p, Y, evals, evecs, work, flags, max_sweeps, tol);
    }
  }
  jacobi_kernel<<<1, 1024, 0, s>>>(p, Y, evals, evecs, work, flags, max_sweeps, tol);
  ++g_launch_count;
  return cudaGetLastError();
}

cudaError_t gaussian_panel(float* P, int64_t n, int q, int ld, uint64_t seed, uint64_t stream,
                           cudaStream_t s) {
  if (q < ld) MMSB_CUDA_TRY(cudaMemsetAsync(P, 0, sizeof(float) * n * ld, s));
  gaussian_panel_kernel<<<grid_for(ceil_div(n * q, 4)), 256, 0, s>>>(P, n, q, ld, seed, stream);
  ++g_launch_count;
  return cudaGetLastError();
}

cudaError_t colmajor64_to_panel(const double* A, int64_t rows, int cols, int64_t lda, float* P,
                                int ldp, cudaStream_t s) {
  colmajor_to_panel_kernel<<<grid_for(rows * ldp), 256, 0, s>>>(A, rows, cols, lda, P, ldp);
  ++g_launch_count;
  return cudaGetLastError();
}

cudaError_t panel_to_colmajor64(const float* P, int ldp, int64_t rows, int cols, double* A,
                                int64_t lda, cudaStream_t s) {
  panel_to_colmajor_kernel<<<grid_for(rows * cols), 256, 0, s>>>(P, ldp, rows, cols, A, lda);
  ++g_launch_count;
  return cudaGetLastError();
}

cudaError_t panel_scale_cols(const float* P, int ldp, int64_t n, int q, const double* d,
                             float* out, cudaStream_t s) {
  if (n == 0) return cudaSuccess;
  if (ldp % 4 != 0) return cudaErrorInvalidValue;
  const unsigned grid = (unsigned)std::min<int64_t>(8 * kNumSMs, ceil_div(n, 8));
  scale_cols_kernel<<<grid, 256, 0, s>>>(reinterpret_cast<const float4*>(P), ldp / 4, n, q, d,
                                         reinterpret_cast<float4*>(out));
  ++g_launch_count;
  return cudaGetLastError();
}

cudaError_t fill_f32(float* p, int64_t n, float v, cudaStream_t s) {
  fill_kernel<float><<<grid_for(n), 256, 0, s>>>(p, n, v);
  ++g_launch_count;
  return cudaGetLastError();
}

cudaError_t fill_f64(double* p, int64_t n, double v, cudaStream_t s) {
  fill_kernel<double><<<grid_for(n), 256, 0, s>>>(p, n, v);
  ++g_launch_count;
  return cudaGetLastError();
}

cudaError_t axpy_f64(int64_t n, double a, const double* x, double* y, cudaStream_t s) {
  axpy_kernel<<<grid_for(n), 256, 0, s>>>(n, a, x, y);
  ++g_launch_count;
  return cudaGetLastError();
}

cudaError_t mgs_cols(int m, int p, const double* P, int ldp, double* Q, int ldq, double tol,
                     cudaStream_t s) {
  if (m > 4096 || p > 4096) return cudaErrorInvalidValue;
  // a 16-CTA cluster (8 where the device cannot co-schedule 16), else one CTA
  static int wide = -1;
  for (int cl : {16, 8}) {
    if (cl == 16 && wide == 0) continue;
    const int rows = (m + cl - 1) / cl;
    const size_t smc = sizeof(double) * ((size_t)rows * p + rows + 3 * ((size_t)p + 1));
    if (smc > 200 * 1024) break;
    cudaError_t e = cl == 16 ? launch_cgs2_cluster<16>(m, p, P, ldp, Q, ldq, tol, smc, s)
                             : launch_cgs2_cluster<8>(m, p, P, ldp, Q, ldq, tol, smc, s);
    if (e == cudaSuccess) {
      if (cl == 16) wide = 1;
      ++g_launch_count;
      return e;
    }
    if (cl == 16 && wide == 1) return e;
    cudaGetLastError();
    if (cl == 16) wide = 0;
  }
  const size_t sm = sizeof(double) * ((size_t)9 * m + p);
  if (sm > 48 * 1024) return cudaErrorInvalidValue;
  cgs2_cols_kernel<<<1, 1024, sm, s>>>(m, p, P, ldp, Q, ldq, tol);
  ++g_launch_count;
  return cudaGetLastError();
}

cudaError_t oa_correction(int n, const double* A, const double* XtX, const double* S, double* E,
                          double* lam, double* delta_state, cudaStream_t s) {
  (void)A;  // ||A|| enters through max |lam_i|
  if (n > 512) return cudaErrorInvalidValue;
  // delta_state[1..3] hold the three maxima (as bit patterns) between the kernels
  unsigned long long* mx = reinterpret_cast<unsigned long long*>(delta_state + 1);
  MMSB_CUDA_TRY(cudaMemsetAsync(mx, 0, 3 * sizeof(unsigned long long), s));
  oa_stats_kernel<<<(unsigned)ceil_div(n, 8), 256, 0, s>>>(n, XtX, S, lam, mx);
  oa_correction_kernel<<<dim3((unsigned)ceil_div(n, 256), (unsigned)n), 256, 0, s>>>(n, XtX, S, E,
                                                                                    lam, mx, delta_state);
  g_launch_count += 2;
  return cudaGetLastError();
}

bool oa_refine_fits(int n) {
  if (n <= 16) return true;
  if (n > kOaMax) return false;
  static const bool wide = []() {  // 16 CTAs are a non-portable cluster size
    cudaLaunchConfig_t lc;
    cudaLaunchAttribute at[1];
    int clusters = 0;
    const bool ok = oa_refine_config<16>(kOaMax, nullptr, &lc, at) == cudaSuccess &&
                    cudaOccupancyMaxActiveClusters(&clusters, oa_refine_kernel<16>, &lc) == cudaSuccess;
    if (!ok) cudaGetLastError();
    return ok && clusters > 0;
  }();
  return wide;
}

cudaError_t oa_refine(int n, int steps, const double* A, const double* X, double* evals,
                      double* evecs, double* delta_state, unsigned* flags, cudaStream_t s) {
  if (n < 1 || n > kOaMax) return cudaErrorInvalidValue;
  cudaLaunchConfig_t lc;
  cudaLaunchAttribute at[1];
  if (n <= 16) {
    MMSB_CUDA_TRY(oa_refine_config<1>(n, s, &lc, at));
    MMSB_CUDA_TRY(cudaLaunchKernelEx(&lc, oa_refine_kernel<1>, n, steps, A, X, evals, evecs,
                                     delta_state, flags));
  } else {
    MMSB_CUDA_TRY(oa_refine_config<16>(n, s, &lc, at));
    MMSB_CUDA_TRY(cudaLaunchKernelEx(&lc, oa_refine_kernel<16>, n, steps, A, X, evals, evecs,
                                     delta_state, flags));
  }
  ++g_launch_count;
  return cudaGetLastError();
}

cudaError_t sort_eigen(int n, const double* lam, const double* X, double* evals, double* evecs,
                       unsigned* flags, cudaStream_t s) {
  sort_eigen_kernel<<<(unsigned)ceil_div(n, 8), 256, 0, s>>>(n, lam, X, evals, evecs, flags);
  ++g_launch_count;
  return cudaGetLastError();
}

cudaError_t panel_set_col(float* P, int ld, int64_t rows, int col, const double* v,
                          cudaStream_t s) {
  panel_set_col_kernel<<<grid_for(rows), 256, 0, s>>>(P, ld, rows, col, v);
  ++g_launch_count;
  return cudaGetLastError();
}

cudaError_t panel_copy(const float* src, int lds, int64_t rows, int q, float* dst, int ldd,
                       cudaStream_t s) {
  panel_copy_kernel<<<grid_for(rows * ldd), 256, 0, s>>>(src, lds, rows, q, dst, ldd);
  ++g_launch_count;
  return cudaGetLastError();
}

}  // namespace mmsb
