// The k x k step for KP = 32 (k <= 32), by columns: an earlier form of the step
// of k_stpm.cu, kept for its roundings.  Up to k of about ten a solve of a
// graph is determined by its input, but its first steps (minibatches of some
// tens of nodes, condition numbers up to 1e5) and the sign rule behind the
// memberships enlarge round-off: in the form by rows, with the sums in another
// order, 1 to 4 of 100 graphs of 2,200 nodes with k from 4 to 8 and 25 with k =
// 12 got another lambda, though its error is smaller.  Users keep results.
// (From k = 32 on 99 of 100 change with any rounding: there the faster form
// runs.)  Measured: 100 steps of 100 nodes at k = 10 2.09 ms, contraction
// included, 1.64 ms by rows.  Bound by latency: a chain of small products, of
// broadcasts of a CTA's columns to the cluster, and of the factor's pivots.
//
// Layout: a cluster of 4 CTAs; every CTA holds whole k x k matrices
// (column-major, leading dimension KP + 4) and owns NB = KP / CL columns.  The
// products X^T Y[:, blk] (Gram) and X B_blk (times) run as warp-level m16n8k8
// TF32 MMAs with the 3xTF32 split (a = a_hi + a_lo; hi hi + hi lo + lo hi
// accumulated in FP32, relative error ~1e-6 per product; the first-order
// correction M F, |F| <= ~1e-5, as one TF32 product), a warp per 16 x 8 output
// tile and half of the sum.  A CTA's new column block is staged in shared memory
// and sent to every CTA by bulk asynchronous copies that complete on the
// receiver's per-block mbarrier; a CTA proceeds once all CL blocks have
// arrived.  A staging tile used for broadcast n is rewritten at broadcast n + 2
// only, after every receiver has waited for broadcast n + 1 (sent by each rank
// after it received all of broadcast n).
//
// Hardware barriers of the CTA: 0 = __syncthreads, 1 = the four panel warps of
// inverse_columns (128 threads), 2 = the block-row release of chol_blocked (warp
// 0 arrives, the other warps sync; whole CTA).  The three are never in use at
// the same time.
//
// Included by k_stpm.cu inside its namespace (its barrier and copy helpers).
#pragma once

namespace step32 {

constexpr int KP = 32;
constexpr int XLD = step_xld(KP);  // == 4 mod 8: the Gram's fragment loads are free of conflicts
constexpr int NBK = KP / 8;        // 8-column blocks of the Cholesky factor

constexpr int CL = 4, NB = KP / CL;  // CTAs of the cluster, columns of each
constexpr int MT = KP / 16, TILES = MT * (NB / 8);
// two matrices; B block, 2 staging tiles, G block; the tiles' second halves; mean
// terms, mu1..3, d-sums, |phi_i|^2, scratch; inverse diagonal blocks and
// corners; original diagonal, 1 / R_jj
constexpr size_t kSmem = sizeof(float) * ((size_t)2 * KP * XLD + 4 * NB * XLD + TILES * 128 + 6 * KP +
                                          4 * NB + 136 + 64 * NBK + 64 * (KP / 16) + 2 * KP);
static_assert(kSmem <= 47 * 1024, "no opt-in for shared memory");

__device__ __forceinline__ uint32_t tf32_round(float x) {
  uint32_t r;
  asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(r) : "f"(x));
  return r;
}

__device__ __forceinline__ void mma_tf32(float (&d)[4], const uint32_t (&a)[4],
                                         const uint32_t (&b)[2]) {
  asm volatile(
      "mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, "
      "{%8,%9}, {%0,%1,%2,%3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}

// One warp: acc = sum over k in [kb, ke) of A(m, k) B(k, n) for the 16 x 8
// tile at pa = &A(0, 0) of the tile, pb = &B(0, 0) of the tile, with
// A(m, k) = pa[m AM + k AK] and B(k, n) = pb[k BK + n BN].  Fragments of
// m16n8k8 (g = lane / 4, t = lane % 4): a = A(g|g+8, t|t+4), b = B(t|t+4, g),
// acc = C(g|g+8, 2t|2t+1).  SPLIT = false: one TF32 product (for a small
// correction term whose relative error may be ~1e-3).
template <int AM, int AK, int BK, int BN, bool SPLIT = true>
__device__ __forceinline__ void warp_tile_3xtf32(const float* __restrict__ pa,
                                                 const float* __restrict__ pb, int kb, int ke,
                                                 float (&acc)[4]) {
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  float c0[4] = {0.f, 0.f, 0.f, 0.f}, c1[4] = {0.f, 0.f, 0.f, 0.f}, c2[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 2
  for (int k0 = kb; k0 < ke; k0 += 8) {
    const float av[4] = {pa[g * AM + (k0 + t) * AK], pa[(g + 8) * AM + (k0 + t) * AK],
                         pa[g * AM + (k0 + t + 4) * AK], pa[(g + 8) * AM + (k0 + t + 4) * AK]};
    const float bv[2] = {pb[(k0 + t) * BK + g * BN], pb[(k0 + t + 4) * BK + g * BN]};
    uint32_t ah[4], al[4], bh[2], bl[2];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      ah[q] = tf32_round(av[q]);
      al[q] = __float_as_uint(av[q] - __uint_as_float(ah[q]));  // the MMA reads its top 19 bits
    }
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      bh[q] = tf32_round(bv[q]);
      bl[q] = __float_as_uint(bv[q] - __uint_as_float(bh[q]));
    }
    mma_tf32(c0, ah, bh);
    if (SPLIT) {
      mma_tf32(c1, ah, bl);
      mma_tf32(c2, al, bh);
    }
  }
#pragma unroll
  for (int q = 0; q < 4; ++q) acc[q] = SPLIT ? c0[q] + (c1[q] + c2[q]) : c0[q];
}

// Tile products of the step.  Warp w < 2 TILES owns tile w % TILES and
// half w / TILES of the K range; the halves meet in `part`.
// kProdGram:  C_blk = X^T Y[:, c0 .. c0+NB)   (A(m=i, k=r) = X[i XLD + r], B = Y block)
// kProdTimes: C_blk = X B_blk                 (A(m=r, k=i) = X[i XLD + r])
// epi(acc, m0, n0) receives each finished 16 x 8 tile.
enum Prod : int { kProdGram = 0, kProdTimes = 1 };

template <int PROD, bool SPLIT = true, typename Epi>
__device__ __forceinline__ void tiles(const float* __restrict__ X, const float* __restrict__ Bm,
                                      float* part, Epi&& epi) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  auto product = [&](int tile, int kb, int ke, float (&acc)[4]) {
    const int m0 = (tile % MT) * 16, n0 = (tile / MT) * 8;
    if (PROD == kProdGram)
      warp_tile_3xtf32<XLD, 1, 1, XLD, SPLIT>(X + m0 * XLD, Bm + n0 * XLD, kb, ke, acc);
    else
      warp_tile_3xtf32<1, XLD, 1, XLD, SPLIT>(X + m0, Bm + n0 * XLD, kb, ke, acc);
  };
  const int tile = warp % TILES, ks = warp / TILES;
  const bool active = warp < TILES * 2;
  float acc[4] = {0.f, 0.f, 0.f, 0.f};
  if (active) {
    product(tile, ks * (KP / 2), ks * (KP / 2) + KP / 2, acc);
    if (ks == 1) {
#pragma unroll
      for (int q = 0; q < 4; ++q) part[tile * 128 + q * 32 + lane] = acc[q];
    }
  }
  __syncthreads();
  if (!active || ks != 0) return;
#pragma unroll
  for (int q = 0; q < 4; ++q) acc[q] += part[tile * 128 + q * 32 + lane];
  epi(acc, (tile % MT) * 16, (tile / MT) * 8);
}

// ---- Cholesky factor and its inverse on one CTA ----------------------------------
//
// A (KP x KP symmetric, column-major, leading dimension XLD, upper triangle
// read) = R^T R with R upper triangular, blocked by 8 columns (right-looking,
// one block of look-ahead).  Per block J: every thread forms one column of
// the block row R_J = R_JJ^-T A_J by forward substitution; then warp 0,
// which formed the block row's first 8 columns itself, goes straight on to
// update the next 8 x 8 diagonal block, and one thread factors it in
// registers (no shuffles on the pivot chain), while the other warps wait at
// a named barrier for the whole block row and update the rest of the
// trailing upper triangle with 3xTF32 tensor-core tiles (a rank-8 update is
// one k-step); one CTA barrier closes the block.  R overwrites A's upper
// triangle, 1 / R_jj goes to rd; the inverses T_JJ = R_JJ^-1 of the diagonal
// blocks (tinv, 8 x 8 column-major each) are formed afterwards, one block per
// thread, off the pivot chain.  Rows and columns >= k must hold the identity
// (the caller sets their diagonal to 1; X's padding columns are zero).

// One thread: the (already updated) 8 x 8 diagonal block at (j0, j0).  A
// pivot that is not above kPivotFloor * dg (breakdown, or NaN) is raised to
// it and counted as ratio 0.  Returns the smallest ratio R_jj^2 / dg[j] over
// the live columns j0 + j < k.
__device__ __forceinline__ float factor_diag8(float* A, int j0, int k, float* rd, const float* dg) {
  float a[8][8];
#pragma unroll
  for (int l = 0; l < 8; ++l)
#pragma unroll
    for (int i = 0; i <= l; ++i) a[i][l] = A[(j0 + i) + (j0 + l) * XLD];
  float rmin = 1.f;
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    float d = a[j][j];
    const float d0 = dg[j0 + j];
    float ratio = __fdividef(d, d0);
    if (!(d > kPivotFloor * d0)) {
      d = kPivotFloor * d0;
      ratio = 0.f;
    }
    if (j0 + j < k) rmin = fminf(rmin, ratio);
    const float ri = rsqrtf(d);
    rd[j0 + j] = ri;
    a[j][j] = d * ri;
#pragma unroll
    for (int l = j + 1; l < 8; ++l) a[j][l] *= ri;
#pragma unroll
    for (int i = j + 1; i < 8; ++i)
#pragma unroll
      for (int l = i; l < 8; ++l) a[i][l] = fmaf(-a[j][i], a[j][l], a[i][l]);
  }
#pragma unroll
  for (int l = 0; l < 8; ++l)
#pragma unroll
    for (int i = 0; i <= l; ++i) A[(j0 + i) + (j0 + l) * XLD] = a[i][l];
  return rmin;
}

// One thread: T = R_JJ^-1 (upper, 8 x 8 column-major into tb) of the
// diagonal block at (j0, j0), column by column: T(j, j) = 1 / R_jj,
// T(m, j) = -(sum_{m <= i < j} T(m, i) R(i, j)) / R(j, j).
__device__ __forceinline__ void invert_diag8(const float* A, int j0, const float* rd, float* tb) {
  float r[8][8], t[8][8];
#pragma unroll
  for (int l = 0; l < 8; ++l)
#pragma unroll
    for (int i = 0; i < l; ++i) r[i][l] = A[(j0 + i) + (j0 + l) * XLD];
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const float rv = rd[j0 + j];
    t[j][j] = rv;
#pragma unroll
    for (int m = 0; m < j; ++m) {
      float s = 0.f;
#pragma unroll
      for (int i = m; i < j; ++i) s = fmaf(t[m][i], r[i][j], s);
      t[m][j] = -s * rv;
    }
  }
#pragma unroll
  for (int l = 0; l < 8; ++l)
#pragma unroll
    for (int i = 0; i < 8; ++i) tb[i + 8 * l] = i <= l ? t[i][l] : 0.f;
}

// Whole CTA.  Returns the smallest pivot ratio (the same value in every
// thread: every CTA of a cluster factors the same matrix the same way).
// (No __restrict__ on these shared-memory pointers: other threads write what
// a thread reads after each barrier, and the ratio decides the control flow
// of the whole CTA, so no load may be moved across a barrier.  With
// __restrict__ the compiler did move the read of the ratio above the
// barrier: warps left the pass loop apart and the kernel hung.)
inline __device__ float chol_blocked(float* A, int k, float* tinv, float* rd, float* dg,
                              volatile float* s_ratio, float shift = 0.f) {
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t4 = lane & 3;
  const int nw = blockDim.x >> 5;
  for (int i = tid; i < KP; i += blockDim.x) {
    float d = A[i + i * XLD] + shift;
    if (i >= k) d = 1.f;
    A[i + i * XLD] = d;
    dg[i] = fmaxf(d, 1e-30f);
  }
  __syncthreads();
  float rmin = 1.f;
  if (tid == 0) rmin = factor_diag8(A, 0, k, rd, dg);
  __syncthreads();
  for (int J = 0; J + 1 < NBK; ++J) {
    const int j0 = 8 * J, rest = KP - j0 - 8;
    // block row: R(j0 + a, c) = (A(j0 + a, c) - sum_{b < a} R(j0 + b, j0 + a)
    // R(j0 + b, c)) / R(j0 + a, j0 + a), c >= j0 + 8 (a thread per column)
    for (int e = tid; e < rest; e += blockDim.x) {
      const int c = j0 + 8 + e;
      float x[8];
#pragma unroll
      for (int b = 0; b < 8; ++b) x[b] = A[(j0 + b) + c * XLD];
#pragma unroll
      for (int aa = 0; aa < 8; ++aa) {
        float s = x[aa];
#pragma unroll
        for (int b = 0; b < aa; ++b) s = fmaf(-A[(j0 + b) + (j0 + aa) * XLD], x[b], s);
        x[aa] = s * rd[j0 + aa];
      }
#pragma unroll
      for (int b = 0; b < 8; ++b) A[(j0 + b) + c * XLD] = x[b];
    }
    // trailing update of the upper triangle, A(c, c') -= sum_b R(j0+b, c)
    // R(j0+b, c') for j0 + 8 <= c <= c'
    const int n0 = j0 + 8;
    if (warp == 0) {
      // the next diagonal block needs only the block row's columns n0 ..
      // n0+7, which lanes 0-7 of this warp formed: the other warps are
      // released through barrier 2 (arrive: release), and this warp goes on
      // with the diagonal block and its factorisation at once
      asm volatile("bar.arrive 2, %0;" ::"r"(nw * 32) : "memory");
      __syncwarp();
      float sv[2];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int e = lane + 32 * h, i = e & 7, l = e >> 3;
        sv[h] = A[(n0 + i) + (n0 + l) * XLD];
#pragma unroll
        for (int b = 0; b < 8; ++b)
          sv[h] = fmaf(-A[(j0 + b) + (n0 + i) * XLD], A[(j0 + b) + (n0 + l) * XLD], sv[h]);
      }
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int e = lane + 32 * h, i = e & 7, l = e >> 3;
        if (i <= l) A[(n0 + i) + (n0 + l) * XLD] = sv[h];
      }
      __syncwarp();
      if (lane == 0) rmin = fminf(rmin, factor_diag8(A, n0, k, rd, dg));
    } else {
      asm volatile("bar.sync 2, %0;" ::"r"(nw * 32) : "memory");  // every block-row column
    }
    if (warp != 0 && rest > 8) {
      // columns c' >= n0 + 8 in 8-wide tiles, rows c in [n0, c'] in 16-row
      // tiles from mb; a last tile that would pass KP is computed at KP - 16
      // (rows below mb not written), so no read leaves the matrix
      const int mt = (rest + 15) / 16, ntl = (rest - 8) / 8;
      for (int tl = warp - 1; tl < mt * ntl; tl += nw - 1) {
        const int mb = n0 + 16 * (tl % mt), nc0 = n0 + 8 + 8 * (tl / mt);
        if (mb > nc0 + 7) continue;  // entirely below the diagonal
        const int m0 = min(mb, KP - 16);
        float acc[4];
        warp_tile_3xtf32<XLD, 1, 1, XLD>(A + j0 + m0 * XLD, A + j0 + nc0 * XLD, 0, 8, acc);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const int r = m0 + g + ((q & 2) ? 8 : 0), c = nc0 + 2 * t4 + (q & 1);
          if (r >= mb && r <= c) A[r + c * XLD] -= acc[q];
        }
      }
    }
    __syncthreads();
  }
  // the inverses of the diagonal blocks, one block per thread
  for (int J = tid; J < NBK; J += blockDim.x) invert_diag8(A, 8 * J, rd, tinv + 64 * J);
  if (tid == 0) *s_ratio = rmin;
  __syncthreads();
  return *s_ratio;
}

// Columns c0 .. c0+NB of W = R^-1 (whole 8-column blocks) into
// Wb (column jb at Wb + jb * XLD, rows past the diagonal block zero), by
// block back substitution per 8-column block K: W_KK = T_KK, then upwards in
// levels of 16 rows aligned to 16 (one 8-row level first when K is odd):
// W_Q = -T_Q S_Q with S_Q = sum over the rows P below Q of R_QP W_PK, where
// for a 16-row superblock Q = (a, b) of 8-row blocks T_Q = [T_a X; 0 T_b],
// X = -T_a R_ab T_b (x16, 8 x 8 column-major per superblock, formed here
// first).  One barrier per level: warps 0-3 add the last term of S_Q and
// apply -T_Q (a named barrier between the two), while the other warps add
// R_rP W_PK of the last level into the partial sums of the rows above
// (held in Wb until their level).  The levels of the last column block are
// about KP / 16 instead of KP / 8, which is what the cluster waits for.
// Blocks that lie wholly in the padding (8K >= k: R is the identity there)
// get unit columns.  tmp: 128 floats.  Whole CTA of at least 5 warps; ends
// with a barrier.
inline __device__ void inverse_columns(const float* R, const float* tinv, float* x16, int c0, int k,
                                       float* Wb, float* tmp) {
  const int tid = threadIdx.x, nt = blockDim.x;
  for (int e = tid; e < NB * XLD; e += nt) Wb[e] = 0.f;
  // X(a, b) = -sum_i T_2m(a, i) sum_j R(16m + i, 16m + 8 + j) T_2m+1(j, b)
  // (the T blocks hold explicit zeros below their diagonals; the R reads of
  // a warp are broadcasts)
  for (int e = tid; e < (KP / 16) * 64; e += nt) {
    const int m = e >> 6, aa = e & 7, b = (e >> 3) & 7, r0 = 16 * m;
    const float* ta = tinv + 64 * (2 * m);
    const float* tb = ta + 64;
    float tv[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) tv[j] = tb[j + 8 * b];
    float x = 0.f;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      float y = 0.f;
#pragma unroll
      for (int j = 0; j < 8; ++j) y = fmaf(R[(r0 + i) + (r0 + 8 + j) * XLD], tv[j], y);
      x = fmaf(ta[aa + 8 * i], y, x);
    }
    x16[e] = -x;
  }
#pragma unroll 1
  for (int sb = 0; sb < NB / 8; ++sb) {
    const int K = c0 / 8 + sb;
    float* W = Wb + 8 * sb * XLD;
    __syncthreads();  // zero fill, X and the previous column block done
    if (8 * K >= k) {
      if (tid < 8) W[8 * K + tid + tid * XLD] = 1.f;
      continue;
    }
    for (int e = tid; e < 64; e += nt) {
      const int aa = e & 7, jb = e >> 3;
      W[8 * K + aa + jb * XLD] = tinv[64 * K + e];  // W_KK = T_KK (column-major)
    }
    __syncthreads();
    int lo = 8 * K, h = 8;  // rows [lo, lo + h) were the last level
    while (lo > 0) {
      const int hn = (lo & 15) ? 8 : 16, nlo = lo - hn;
      if (tid < 128) {
        // S_Q (row i, column jb) = partial sum + R(nlo + i, lo ..) W(lo .., jb)
        const int i = tid & 15, jb = tid >> 4;
        if (i < hn) {
          float sv = W[nlo + i + jb * XLD];
#pragma unroll
          for (int b = 0; b < 8; ++b) sv = fmaf(R[(nlo + i) + (lo + b) * XLD], W[lo + b + jb * XLD], sv);
          if (h == 16) {
#pragma unroll
            for (int b = 8; b < 16; ++b) sv = fmaf(R[(nlo + i) + (lo + b) * XLD], W[lo + b + jb * XLD], sv);
          }
          tmp[i + 16 * jb] = sv;
        }
        asm volatile("bar.sync 1, 128;" ::: "memory");
        if (i < hn) {
          const float* s = tmp + 16 * jb;
          float w = 0.f;
          // T rows from the diagonal on (zeros below it are stored)
          const int ii = i & 7;
          const float* t = tinv + 64 * (nlo / 8 + (i >> 3));
          const float* sv = s + (i & 8);
#pragma unroll
          for (int b = 0; b < 8; ++b) w = fmaf(t[ii + 8 * b], sv[b], w);
          if (hn == 16 && i < 8) {
            const float* x = x16 + 64 * (nlo / 16) + i;
#pragma unroll
            for (int j = 0; j < 8; ++j) w = fmaf(x[8 * j], s[8 + j], w);
          }
          W[nlo + i + jb * XLD] = -w;
        }
      } else {
        // rows above the level accumulate R(r, lo ..) W(lo .., jb)
        for (int e = tid - 128; e < nlo * 8; e += nt - 128) {
          const int r = e % nlo, jb = e / nlo;
          float sv = W[r + jb * XLD];
#pragma unroll
          for (int b = 0; b < 8; ++b) sv = fmaf(R[r + (lo + b) * XLD], W[lo + b + jb * XLD], sv);
          if (h == 16) {
#pragma unroll
            for (int b = 8; b < 16; ++b) sv = fmaf(R[r + (lo + b) * XLD], W[lo + b + jb * XLD], sv);
          }
          W[r + jb * XLD] = sv;
        }
      }
      __syncthreads();
      h = hn;
      lo = nlo;
    }
  }
  __syncthreads();
}


__device__ __forceinline__ void body(const StpmUpdateArgs& a) {
  cg::cluster_group cluster = cg::this_cluster();
  const int rank = (int)cluster.block_rank();
  extern __shared__ __align__(16) float sm[];
  float* Xa = sm;
  float* Xb = Xa + KP * XLD;
  float* Ab = Xb + KP * XLD;                      // B block of the products, column jb at Ab + jb * XLD
  float* Ot = Ab + NB * XLD;                      // two staging tiles of the broadcasts
  float* Gb = Ot + 2 * NB * XLD;                  // G block (online step)
  float* part = Gb + NB * XLD;                    // K-split partial tiles
  float* mv = part + TILES * 128;                    // m1, m2, m3 of this block
  float* dcol = mv + 3 * KP;                      // 3 * NB d-sums
  float* nn = dcol + 3 * NB;                      // |phi_i|^2 of this block
  float* mus = nn + NB;                           // mu1, mu2, mu3 (KP each)
  float* tmp = mus + 3 * KP;                      // 128 (inverse columns)
  float* tinv = tmp + 128 + 8;                    // 8 x 8 inverse diagonal blocks
  float* x16 = tinv + 64 * NBK;                // corners of the 16 x 16 inverse blocks
  float* dg = x16 + 64 * (KP / 16);               // original diagonal
  float* rd = dg + KP;                            // 1 / R_jj
  __shared__ float s_ratio;
  __shared__ float s_emax[16];
  __shared__ __align__(8) uint64_t s_blk[2][16];  // block q of Xa / Xb arrived
  __shared__ __align__(8) uint64_t s_csync[2];    // bounded cluster barrier, in turn
  const int k = a.k;
  const int c0 = rank * NB;
  const int tid = threadIdx.x, lane = tid & 31, g = lane >> 2, t4 = lane & 3;
  const long long wl = tc::wait_limit_or_default(a.wait_limit);
  {
    // Phi: loads issued in batches of 8 per thread so that their latencies overlap
    constexpr int N = KP * XLD, B = 8;
    for (int e0 = tid; e0 < N; e0 += 512 * B) {
      float v[B];
#pragma unroll
      for (int u = 0; u < B; ++u) {
        const int e = e0 + 512 * u, r = e % XLD, c = e / XLD;
        v[u] = (e < N && r < k && c < k) ? __ldg(a.phi + (int64_t)c * k + r) : 0.f;
      }
#pragma unroll
      for (int u = 0; u < B; ++u)
        if (e0 + 512 * u < N) {
          Xa[e0 + 512 * u] = v[u];
          Xb[e0 + 512 * u] = 0.f;
        }
    }
  }
  for (int e = tid; e < 2 * NB * XLD; e += blockDim.x) Ot[e] = 0.f;
  if (tid < 2 * CL) mbar_init(&s_blk[tid / CL][tid % CL], 1);
  else if (tid < 2 * CL + 2) mbar_init(&s_csync[tid - 2 * CL], CL);
  if (tid < 2 * CL + 2) asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  __syncthreads();
  if (a.step_mode == kStepOnline) {
    // mu1..3 for the G block below, and the mean terms phi_i . mu and
    // |phi_i|^2 of this block's columns (a warp per dot product, lanes along
    // the k entries): Phi and mu only, so before the wait
    for (int e = tid; e < 3 * KP; e += blockDim.x) {
      const int which = e / KP, j = e % KP;
      const float* mu = which == 0 ? a.mu1 : which == 1 ? a.mu2 : a.mu3;
      mus[e] = (mu && j < k) ? __ldg(mu + j) : 0.f;
    }
    for (int e = tid / 32; e < 4 * NB; e += blockDim.x / 32) {
      const int which = e / NB, jb = e % NB, i = c0 + jb;
      const float* col = Xa + i * XLD;
      const float* mu = which == 0 ? a.mu1 : which == 1 ? a.mu2 : which == 2 ? a.mu3 : col;
      float sv = 0.f;
      if (i < k && mu)
        for (int j = lane; j < k; j += 32) sv = fmaf(col[j], mu[j], sv);
#pragma unroll
      for (int off = 16; off; off >>= 1) sv += __shfl_xor_sync(0xffffffffu, sv, off);
      if (lane == 0) {
        if (which < 3) mv[which * KP + jb] = sv; else nn[jb] = sv;
      }
    }
  }
  cluster.sync();  // Phi read and barriers initialised everywhere before any copy
  // launched with programmatic serialization after the contraction, the
  // prologue above overlapped its tail (Phi is final: the contraction lets
  // this kernel start only after its own wait on the previous step); from
  // here on its partials are read, so wait for it to complete, and let the
  // next contraction be scheduled (it waits for this kernel in turn)
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  uint32_t parity = 0u;  // bit b: phase parity awaited on the barriers of buffer b
  uint32_t csync_n = 0u;
  int nbcast = 0;
  bool timed_out = false;
  constexpr uint32_t kBlockBytes = sizeof(float) * NB * XLD;
  auto buf_of = [&](const float* b) { return b == Xa ? 0 : 1; };
  // staging tile of the next broadcast (or of the final block)
  auto stage_next = [&]() -> float* {
    float* p = Ot + (nbcast & 1) * NB * XLD;
    ++nbcast;
    return p;
  };
  // bounded cluster barrier: every thread of every CTA has passed the
  // __syncthreads before its rank's arrival (remote mbarrier arrives with
  // release semantics, waited for with acquire); false after a timeout
  auto csync_arrive = [&]() {
    __syncthreads();
    if (tid < CL) {
      uint32_t remote;
      asm volatile("mapa.shared::cluster.u32 %0, %1, %2;"
                   : "=r"(remote)
                   : "r"(smem_addr(&s_csync[csync_n & 1])), "r"(tid));
      asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(remote) : "memory");
    }
  };
  auto csync_wait = [&]() -> bool {
    bool ok = true;
    if (tid == 0) ok = mbar_wait_cluster_bounded(&s_csync[csync_n & 1], (csync_n >> 1) & 1u, wl);
    ++csync_n;
    return !__syncthreads_or(!ok);
  };
  auto csync = [&]() -> bool {
    csync_arrive();
    return csync_wait();
  };
  // the staged block Otc (this CTA's columns) into `dst` of every rank,
  // own copy included; sync_first: a cluster barrier first, because some
  // rank may still be reading its `dst`
  auto broadcast = [&](float* Otc, float* dst, bool sync_first) {
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // staging -> async proxy
    if (sync_first) {
      if (!csync()) timed_out = true;
    } else {
      __syncthreads();
    }
    float* own = dst + c0 * XLD;
    for (int e = tid; e < NB * XLD; e += blockDim.x) own[e] = Otc[e];
    const int bi = buf_of(dst), w = tid >> 5;
    // one issuing thread per warp (copies issued by lanes of one warp
    // serialise); rank q sends to q+1, q+2, ... first, so every rank receives
    // its blocks spread over the exchange
    if (lane == 0 && w < CL - 1)
      bulk_copy_to_rank(own, Otc, kBlockBytes, &s_blk[bi][rank], (uint32_t)((rank + 1 + w) % CL));
    if (tid < CL && tid != rank) mbar_arrive_expect_tx(&s_blk[bi][tid], kBlockBytes);
  };
  // every block of `buf` has arrived (false after a timeout of any wait)
  auto wait_buf = [&](const float* buf) -> bool {
    const int bi = buf_of(buf);
    bool ok = true;
    if (tid < CL && tid != rank) ok = mbar_wait_bounded(&s_blk[bi][tid], (parity >> bi) & 1u, wl);
    parity ^= 1u << bi;
    return !__syncthreads_or(!ok);
  };
  // Gram block C = P^T P[:, c0 .. c0+NB) into the staging tile, zero outside
  // k x k; a non-finite entry raises kFlagNonFinite
  auto gram_stage = [&](const float* P, float* Otc) {
    bool bad = false;
    tiles<kProdGram>(P, P + c0 * XLD, part, [&](const float (&acc)[4], int m0, int n0) {
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int i = m0 + g + ((q & 2) ? 8 : 0), jb = n0 + 2 * t4 + (q & 1), col = c0 + jb;
        const float v = acc[q];
        if (!isfinite(v)) bad = true;
        Otc[jb * XLD + i] = (i < k && col < k) ? v : 0.f;
      }
    });
    if (bad) atomicOr(a.flags, kFlagNonFinite);
  };

  float* M = Xa;               // the matrix to orthonormalise (full in every CTA)
  float* F = Xb;               // the other buffer
  if (a.step_mode == kStepOnline) {
    // G block (columns c0 .. c0+NB) from the per-CTA partials.  The first 8
    // partials of this thread's (up to) two G entries are loaded together
    // with the d-sum partials, so that one round trip covers them all.
    constexpr int kPre = 2, kPreParts = 8;
    float gpre[kPre][kPreParts];
#pragma unroll
    for (int h = 0; h < kPre; ++h) {
      const int e = tid + h * (int)blockDim.x, jb = e / KP, j = e % KP, i = c0 + jb;
      const bool live = e < NB * KP && i < k && j < k;
#pragma unroll
      for (int u = 0; u < kPreParts; ++u)
        gpre[h][u] = (live && u < a.nparts)
                         ? __ldg(a.gpart + (int64_t)u * a.part_stride + (int64_t)i * k + j)
                         : 0.f;
    }
    // per-column sums of the d partials (3 x NB)
    for (int e = tid / 32; e < 3 * NB; e += blockDim.x / 32) {
      const int which = e / NB, jb = e % NB, i = c0 + jb;
      float sd = 0.f;
      if (i < k && (which == 0 || a.mode == kModeAdjoint))
        for (int pp = tid % 32; pp < a.nparts; pp += 32)
          sd += a.gpart[(int64_t)pp * a.part_stride + (int64_t)k * k + which * k + i];
#pragma unroll
      for (int off = 16; off; off >>= 1) sd += __shfl_xor_sync(0xffffffffu, sd, off);
      if ((tid & 31) == 0) dcol[e] = sd;
    }
    __syncthreads();
    for (int e = tid; e < NB * KP; e += blockDim.x) {
      const int jb = e / KP, j = e % KP, i = c0 + jb;
      float gval = 0.f;
      if (i < k && j < k) {
        const float* gp = a.gpart + (int64_t)i * k + j;
        float s0 = 0.f, s1 = 0.f, s2 = 0.f, s3 = 0.f;
        int pp = 0;
        const int h = (e - tid) / (int)blockDim.x;  // 0 or 1 for the preloaded entries
        if (h < kPre) {
#pragma unroll
          for (int h2 = 0; h2 < kPre; ++h2)
            if (h2 == h) {
              s0 += gpre[h2][0] + gpre[h2][4];
              s1 += gpre[h2][1] + gpre[h2][5];
              s2 += gpre[h2][2] + gpre[h2][6];
              s3 += gpre[h2][3] + gpre[h2][7];
            }
          pp = kPreParts;
        }
        for (; pp + 8 <= a.nparts; pp += 8) {
          float v[8];
#pragma unroll
          for (int u = 0; u < 8; ++u) v[u] = __ldg(gp + (int64_t)(pp + u) * a.part_stride);
          s0 += v[0] + v[4];
          s1 += v[1] + v[5];
          s2 += v[2] + v[6];
          s3 += v[3] + v[7];
        }
        for (; pp < a.nparts; ++pp) s0 += __ldg(gp + (int64_t)pp * a.part_stride);
        float gv = ((s0 + s1) + (s2 + s3)) * a.scale;
        const float m1 = mv[jb], m2 = mv[KP + jb], m3 = mv[2 * KP + jb];
        const float c1 = a.c1, c2 = a.c2;
        if (a.mode == kModePlain) {
          gv += mus[2 * KP + j] * (c1 * m1 * m2 + c2 * dcol[jb]);
        } else {
          const float ic = a.inv_count;
          gv += mus[j] * (c2 * dcol[jb] * ic + c1 * m2 * m3) +
                mus[KP + j] * (c2 * dcol[NB + jb] * ic + c1 * m1 * m3) +
                mus[2 * KP + j] * (c2 * dcol[2 * NB + jb] * ic + c1 * m1 * m2);
        }
        gval = gv;
      }
      Gb[jb * XLD + j] = gval;
    }
    // X = Phi - beta (3 theta Phi (Phi^T Phi)^.2 - gscale G)   (Util.cpp:259-272)
    float* Otc;
    const float alpha = -a.beta * a.theta3, gamma = a.beta * a.gscale;
    if (a.phi_general) {
      // the literal product (first step of a run: Phi0 need not be orthonormal)
      tiles<kProdGram>(M, M + c0 * XLD, part, [&](const float (&acc)[4], int m0, int n0) {
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const int i = m0 + g + ((q & 2) ? 8 : 0), jb = n0 + 2 * t4 + (q & 1);
          Ab[jb * XLD + i] = acc[q] * acc[q];
        }
      });
      __syncthreads();
      Otc = stage_next();
      tiles<kProdTimes>(M, Ab, part, [&](const float (&acc)[4], int m0, int n0) {
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const int r = m0 + g + ((q & 2) ? 8 : 0), jb = n0 + 2 * t4 + (q & 1), col = c0 + jb;
          const float v = alpha * acc[q] + M[col * XLD + r] + gamma * Gb[jb * XLD + r];
          Otc[jb * XLD + r] = (r < k && col < k) ? v : 0.f;
        }
      });
    } else {
      // Phi is the previous step's Q: Phi^T Phi = I to ~1e-7, so
      // (Phi^T Phi)^.2 = diag(|phi_i|^4) + O(1e-14) and Phi times it is
      // phi_i |phi_i|^4, column by column
      __syncthreads();
      Otc = stage_next();
      for (int e = tid; e < NB * XLD; e += blockDim.x) {
        const int r = e % XLD, jb = e / XLD, col = c0 + jb;
        const float n2 = nn[jb] * nn[jb];
        Otc[e] = (r < k && col < k) ? M[col * XLD + r] * (1.f + alpha * n2) + gamma * Gb[e] : 0.f;
      }
    }
    broadcast(Otc, F, false);
    if (!wait_buf(F)) timed_out = true;
    float* t = M;
    M = F;
    F = t;
  }
  // Cholesky QR passes on M: A = M^T M gathered into F, R = chol(A) and the
  // columns of R^-1 this CTA needs (computed by every CTA from the same A),
  // M R^-1 gathered into F, which becomes M.
  int passes = 0, shifts = 0, plain_left = a.max_passes;
  float shift = 0.f;
  bool resync = false;  // a rank may still be factoring the last Gram in F
  __shared__ float s_shift;
  while (!timed_out) {
    float* Otc = stage_next();
    gram_stage(M, Otc);
    broadcast(Otc, F, resync);
    resync = false;
    if (!wait_buf(F)) {
      timed_out = true;
      break;
    }
    const float ratio = chol_blocked(F, k, tinv, rd, dg, &s_ratio, shift);
    if (__syncthreads_or(ratio < kShiftBelow) && shifts < kMaxShifts) {
      // near breakdown: the Gram again, factored with a diagonal shift
      if (tid == 0) {
        float tr = 0.f;
        for (int i = 0; i < k; ++i) tr += dg[i];
        s_shift = shift > 0.f ? 100.f * shift : kShiftScale * tr;
      }
      __syncthreads();
      shift = s_shift;
      ++shifts;
      resync = true;
      continue;
    }
    inverse_columns(F, tinv, x16, c0, k, Ab, tmp);
    ++passes;
    Otc = stage_next();
    tiles<kProdTimes>(M, Ab, part, [&](const float (&acc)[4], int m0, int n0) {
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int r = m0 + g + ((q & 2) ? 8 : 0), jb = n0 + 2 * t4 + (q & 1), col = c0 + jb;
        Otc[jb * XLD + r] = (r < k && col < k) ? acc[q] : 0.f;
      }
    });
    // every rank has finished its Cholesky in F before any block of M R^-1 is
    // written there
    broadcast(Otc, F, true);
    if (!wait_buf(F)) {
      timed_out = true;
      break;
    }
    float* t = M;
    M = F;
    F = t;
    if (shift > 0.f) {
      // Q1 of a shifted factor is well conditioned, not orthonormal: plain
      // passes follow
      shift = 0.f;
      plain_left = a.max_passes;
      continue;
    }
    --plain_left;
    // the decision is taken by the whole CTA together (a barrier OR), so
    // every warp leaves or repeats the loop
    const bool again = __syncthreads_or(ratio < kQrExactBelow) != 0;
    if (!again || plain_left <= 0) {
      if (again && rank == 0 && tid == 0) atomicOr(a.flags, kFlagNoConvergence);
      break;
    }
  }
  // every copy of the last exchange has landed in this CTA, and each rank
  // sent its blocks only after the barrier that opened that exchange, so
  // every rank's phase of that barrier is complete: this CTA's arrival at
  // the closing barrier (no remote access follows) goes out now, its wait
  // comes at the end
  const bool early_arrive = !timed_out;
  if (early_arrive) csync_arrive();
  // first-order second pass: E = M^T M - I, F = strict upper part of E plus
  // half its diagonal (this CTA's columns, in Ab), Phi = M (I - F)
  float emax = 0.f;
  if (!timed_out) {
    tiles<kProdGram>(M, M + c0 * XLD, part, [&](const float (&acc)[4], int m0, int n0) {
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int i = m0 + g + ((q & 2) ? 8 : 0), jb = n0 + 2 * t4 + (q & 1), col = c0 + jb;
        const bool live = i < k && col < k;
        const float e = live ? acc[q] - (i == col ? 1.f : 0.f) : 0.f;
        emax = fmaxf(emax, fabsf(e));
        Ab[jb * XLD + i] = i < col ? e : i == col ? 0.5f * e : 0.f;
      }
    });
#pragma unroll
    for (int off = 16; off; off >>= 1) emax = fmaxf(emax, __shfl_xor_sync(0xffffffffu, emax, off));
    if (lane == 0) s_emax[tid >> 5] = emax;
    __syncthreads();
    float* Otc = stage_next();
    // |F| is at most ~1e-5 here (an exact pass left M orthonormal to u times
    // at most 1 / the pivot ratio bound), so a single TF32 product keeps
    // M F to ~1e-9, below the FP32 resolution of Phi's entries
    tiles<kProdTimes, false>(M, Ab, part, [&](const float (&acc)[4], int m0, int n0) {
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int r = m0 + g + ((q & 2) ? 8 : 0), jb = n0 + 2 * t4 + (q & 1), col = c0 + jb;
        Otc[jb * XLD + r] = (r < k && col < k) ? M[col * XLD + r] - acc[q] : 0.f;
      }
    });
    __syncthreads();
    if (tid == 0) {
      float m = 0.f;
      for (int w = 0; w < (int)(blockDim.x >> 5); ++w) m = fmaxf(m, s_emax[w]);
      if (a.orth_err) atomicMax(reinterpret_cast<int*>(a.orth_err), __float_as_int(m));
    }
    for (int e = tid; e < KP * NB; e += blockDim.x) {
      const int r = e % KP, jb = e / KP, col = c0 + jb;
      if (r < k && col < k) a.phi[(int64_t)col * k + r] = Otc[jb * XLD + r];
    }
    if (a.phi_img) {
      // the next contraction's operand image of this CTA's columns i (rows
      // of its A operand, K = j): TF32 hi / lo in the core-matrix layout,
      // then Phi^T mu1, Phi^T mu2 of the columns
      using CT = ContractTc<KP>;
      unsigned char* img = static_cast<unsigned char*>(a.phi_img);
      for (int e = tid; e < NB * (KP / 4); e += blockDim.x) {
        const int jb = e / (KP / 4), jq = e % (KP / 4), i = c0 + jb;
        float v[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) v[u] = Otc[jb * XLD + 4 * jq + u];  // zero past k
        uint4 h;
        float4 l;
        tc::split4(v, h, l);
        const uint32_t off = tc::kmajor_off(i, 4 * jq, CT::SBOJ);
        *reinterpret_cast<uint4*>(img + CT::PH + off) = h;
        *reinterpret_cast<float4*>(img + CT::PL + off) = l;
      }
      float* mimg = reinterpret_cast<float*>(img + 2 * CT::PSZ);
      for (int e = tid >> 5; e < 2 * NB; e += blockDim.x >> 5) {
        const int which = e / NB, jb = e % NB, i = c0 + jb;
        const float* mu = which == 0 ? a.mu1 : a.mu2;
        float sv = 0.f;
        if (mu && i < k)
          for (int j = lane; j < k; j += 32) sv = fmaf(Otc[jb * XLD + j], mu[j], sv);
#pragma unroll
        for (int off = 16; off; off >>= 1) sv += __shfl_xor_sync(0xffffffffu, sv, off);
        if (lane == 0) mimg[which * KP + i] = sv;
      }
    }
    if (a.trace_out) {  // ||Phi_new - snapshot||_F^2 over this CTA's columns, fixed order
      double d2 = 0.0;
      for (int e = tid; e < KP * NB; e += blockDim.x) {
        const int r = e % KP, jb = e / KP, col = c0 + jb;
        if (r < k && col < k) {
          const float v = Otc[jb * XLD + r];
          const double d = (double)v - (double)a.trace_snap[(int64_t)col * k + r];
          d2 = fma(d, d, d2);
          a.trace_snap[(int64_t)col * k + r] = v;
        }
      }
#pragma unroll
      for (int off = 16; off; off >>= 1) d2 += __shfl_xor_sync(0xffffffffu, d2, off);
      __shared__ double tpart[16];
      if (lane == 0) tpart[tid >> 5] = d2;
      __syncthreads();
      if (tid == 0) {
        double t = 0.0;
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t += tpart[w];
        a.trace_out[rank] = t;
      }
    }
  }
  if (timed_out) {
    if (tid == 0) atomicOr(a.flags, kFlagTimeout);
  }
  if (rank == 0 && tid == 0 && a.orth_passes) atomicAdd(a.orth_passes, passes);
  // keep shared memory alive until remote writers are done (bounded: after a
  // timeout the ranks may stand at different barriers)
  if (!(early_arrive ? csync_wait() : csync())) {
    if (tid == 0) atomicOr(a.flags, kFlagTimeout);
    __nanosleep(100000);  // let copies a stalled exchange left in flight land
  }
}

}  // namespace step32
