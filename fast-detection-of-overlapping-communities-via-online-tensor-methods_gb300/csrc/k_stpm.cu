// Tensor power method kernels (FP32 form and BF16 form).
//
// The reference's STPM (GPU/stpm.c:497-790) issues ~2k+10 tiny library calls
// per sample; tensorDecom_alpha0 (CPU/Util.cpp:131-184) runs k sparse
// mat-vecs per column per iteration.  Both reduce to one contraction shape,
// computed here per tile of T nodes:
//
//   Z1 = Y1 Phi, Z2 = Y2 Phi                      (T x k, Phi resident in smem)
//   C  = c0 Z1.Z2 + c2 (Z1 diag(m2) + diag(m1) Z2) (alpha0 correction terms)
//   G += Yout^T C ,  d += colsum(Z1.Z2)            (k x k partial per CTA)
//
// with m1 = Phi^T mu1, m2 = Phi^T mu2.  The online update (Diff_Loss,
// Util.cpp:257-304) uses (Y1,Y2,Yout) = (y_A,y_B,y_C); the batch power
// iteration (tensor_form_main/shift1/shift0, Util.cpp:187-206) uses
// (y_B,y_C,y_A).  The adjoint mode computes all three partial derivatives of
// the cubic form (three Z's, three coefficient matrices, one stacked
// contraction) and the loss.
//
// The contraction (stpm_contract_kernel) runs on tcgen05 in the plain FP32 form
// and the BF16 adjoint form up to KP = 112, on mma.sync in the other BF16 forms
// and the FP32 adjoint steps of KP = 32, else as FFMA; partials of 8-CTA
// clusters are summed through distributed shared memory and reduced
// deterministically by stpm_reduce or by the step kernel.  The k x k update
// (orthogonality term, step, Cholesky QR) runs on one cluster that splits the
// rows of the iterate and exchanges Gram blocks by bulk copies (at KP = 32 its
// columns, k_step32.cuh).
#include "common.cuh"

#include <cstdlib>
#include "k_stpm.cuh"
#include "tc_util.cuh"

#include <cooperative_groups.h>
#include <cuda_bf16.h>

#include <type_traits>

namespace cg = cooperative_groups;

namespace mmsb {

namespace {

constexpr int kPartialCluster = 8;  // CTAs whose partials are summed through DSMEM

__device__ __forceinline__ int64_t ceil_div_dev(int64_t a, int64_t b) { return (a + b - 1) / b; }

// Sum of v over the first 32 nw threads of the CTA, in a fixed order; red
// holds 8 doubles.  Every thread gets the sum.  (FP64 runs at 2 operations
// per clock and SM: warps without a value stay out.)
__device__ __forceinline__ double cta_sum(double v, int nw, double* red) {
  const int warp = threadIdx.x >> 5;
  if (warp < nw) {
#pragma unroll
    for (int off = 16; off; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
  }
  __syncthreads();  // red may still be read from the previous sum
  if ((threadIdx.x & 31) == 0 && warp < nw) red[warp] = v;
  __syncthreads();
  double s = red[0];
#pragma unroll 1
  for (int w = 1; w < nw; ++w) s += red[w];
  return s;
}

// G = sum_parts gpart + mu-terms; d-vectors folded in.  One CTA per column i,
// a thread per entry: bound by two dependent L2 round trips (Phi and mu before
// the wait, the partials after it), so the column's mean terms are warp
// reductions and a thread's partials are loaded 8 at a time.  A power
// iteration's normalisation runs here too (a.lambda): the column is complete
// in its CTA, and a kernel of its own took 214 us per iteration at k = 33 (a
// thread per column walking the matrix).  The two scalars over all columns
// (the loss, the iterate's change) are summed in a fixed order by the CTA that
// finishes last.
__global__ void __launch_bounds__(256) stpm_reduce_kernel(StpmReduceArgs a) {
  const int k = a.k, i = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int64_t kk = (int64_t)k * k;
  __shared__ double m[3], ds[3], red[8], inv_norm;
  __shared__ bool last;
  if (tid < 3) m[tid] = 0.0;
  __syncthreads();
  if (warp < 3) {
    const float* mu = warp == 0 ? a.mu1 : warp == 1 ? a.mu2 : a.mu3;
    double s = 0.0;
    if (mu)
#pragma unroll 1
      for (int j = lane; j < k; j += 32) s += (double)a.phi[(int64_t)i * k + j] * (double)mu[j];
#pragma unroll
    for (int off = 16; off; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
    if (lane == 0) m[warp] = s;
  }
  // the contraction may let this kernel start early (it writes only gpart,
  // and starts only when Phi is final); everything below reads gpart
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  double gsum = 0.0;
  if (a.mode != kModeLoss && tid < k) {
    const float* gp = a.gpart + (int64_t)i * k + tid;
    int p = 0;
#pragma unroll 1
    for (; p + 8 <= a.nparts; p += 8) {
      float v[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) v[u] = __ldcg(gp + (int64_t)(p + u) * a.part_stride);
#pragma unroll
      for (int u = 0; u < 8; ++u) gsum += (double)v[u];
    }
#pragma unroll 1
    for (; p < a.nparts; ++p) gsum += (double)__ldcg(gp + (int64_t)p * a.part_stride);
  }
  if (warp >= 5) {  // the d-sums of the column
    const int q = warp - 5;
    double s = 0.0;
#pragma unroll 1
    for (int p = lane; p < a.nparts; p += 32)
      s += (double)__ldcg(a.gpart + (int64_t)p * a.part_stride + kk + q * k + i);
#pragma unroll
    for (int off = 16; off; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
    if (lane == 0) ds[q] = s;
  }
  __syncthreads();
  float g = 0.f;
  if (tid < k) {
    double s = gsum * a.scale;
    if (a.mode == kModePlain) {
      // mu_out * (c1 m1 m2 + c2 sum Z1 Z2)
      s += (double)a.mu_out[tid] * (a.c1 * m[0] * m[1] + a.c2 * ds[0]);
    } else if (a.mode == kModeAdjoint) {
      const double dm1 = a.c2 * ds[0] * a.inv_count + a.c1 * m[1] * m[2];
      const double dm2 = a.c2 * ds[1] * a.inv_count + a.c1 * m[0] * m[2];
      const double dm3 = a.c2 * ds[2] * a.inv_count + a.c1 * m[0] * m[1];
      s += (double)a.mu1[tid] * dm1 + (double)a.mu2[tid] * dm2 + (double)a.mu3[tid] * dm3;
    }
    g = (float)s;
    a.G[(int64_t)i * k + tid] = g;
  }
  double term = 0.0;
  if (a.lambda) {
    // Phi_new = G (already includes the shift terms), lambda = ||col||^3,
    // column normalisation, the column's share of ||Phi_new - Phi_old||^2
    const int nw = (k + 31) / 32;
    const double s = cta_sum((double)g * (double)g, nw, red);
    if (tid == 0) {
      const double nrm = sqrt(s);
      inv_norm = 1.0 / nrm;  // one division per column
      a.lambda[i] = s * nrm;
    }
    __syncthreads();
    double e = 0.0;
    if (tid < k) {
      float* x = a.phi_out + (int64_t)i * k + tid;
      const double v = (double)g * inv_norm, d = v - (double)*x;
      e = d * d;
      *x = (float)v;
    }
    term = cta_sum(e, nw, red);
  } else if (a.mode == kModeLoss) {
    term = a.c1 * m[0] * m[1] * m[2];
  } else {
    return;  // no scalar over the columns
  }
  if (tid == 0) {
    a.parts[i] = term;
    __threadfence();
    last = atomicAdd(a.done, 1u) + 1u == gridDim.x;
  }
  __syncthreads();
  if (!last) return;
  if (tid == 0) *a.done = 0u;
  double v = tid < k ? __ldcg(a.parts + tid) : 0.0;
  if (a.mode == kModeLoss) {
    // one loss slot per contraction column block
    double t = 0.0;
#pragma unroll 1
    for (int e = tid; e < 4 * a.nparts; e += 256)
      t += (double)__ldcg(a.gpart + (int64_t)(e >> 2) * a.part_stride + kk + 3 * k + (e & 3));
    v += t * a.inv_count;
  }
  v = cta_sum(v, 8, red);
  if (tid == 0) {
    if (a.mode == kModeLoss) {
      a.loss_out[0] = v;  // sum_i That(phi_i, phi_i, phi_i)
    } else {
      v = sqrt(v);
      a.err_out[0] = v;
      if (a.trace_out) a.trace_out[0] = v;
    }
  }
}

// ---- k x k step on one thread-block cluster -------------------------------------
//
// The update of one minibatch step (Diff_Loss, CPU/Util.cpp:257-284, as the
// GPU tree applies it at GPU/stpm.c:649-691, then its re-orthonormalisation
// by culaDeviceDgeqrfp + culaDeviceDorgqr, GPU/stpm.c:783-784):
//
//   X   = Phi - beta (3 theta Phi (Phi^T Phi)^.2 - gscale G)
//   Phi = Q  of  X = Q R  with R upper triangular, diag(R) > 0
//
// Q is computed by Cholesky QR: A = X^T X = R1^T R1 (Cholesky), Q1 = X R1^-1,
// then E = Q1^T Q1 - I and Q = Q1 (I - F) with F upper triangular,
// F + F^T = E (F = strict upper part of E plus half its diagonal), which is
// the second Cholesky QR pass to first order in E.  Every factor applied to X
// from the right is upper triangular with a positive diagonal, so Q is the
// Q of the QR factorisation with diag(R) > 0 (it is unique), the factor the
// reference forms.  When a pivot of the Cholesky shows that X's columns are
// far from independent (R_jj^2 / A_jj below kQrExactBelow; the loss of
// orthogonality of one pass grows like eps / that ratio), further exact
// Cholesky QR passes run on Q1 before the first-order step.  When a pivot
// has lost (nearly) all its digits (ratio below kShiftBelow: the FP32 Gram
// squares cond(X), which reaches 1e4 - 2e5 in the first sweep of the
// benchmarked workloads, beyond 1 / sqrt(eps)), the Gram is formed again
// and factored with a diagonal shift s = kShiftScale trace(A) (shifted
// Cholesky QR, Fukaya et al., SIAM J. Sci. Comput. 42 (2020)): A + s I is
// safely positive definite, Q1 = X R_s^-1 has cond ~ sqrt(s) / sigma_min, and
// the plain passes that follow orthonormalise it.  Every CTA of the cluster
// computes the same Cholesky from the same data, so the pass count needs no
// vote.
//
// Split: the step is a chain of small dependent products, so what bounds it
// is the number of exchanges and the Cholesky's pivots, not arithmetic.  CTA
// q of the cluster owns RB = KP / CL ROWS of X.  A Gram is then the sum of
// the CTAs' X_q^T X_q (a rank-RB product each): CTA q sends column block s of
// its partial to CTA s, which adds the CL partials in rank order and sends
// the finished block to everybody -- two one-way exchanges per Gram, no
// cluster barrier.  Q1 = X R1^-1 needs no exchange at all: the rows of X ride
// along as RB extra columns of the factorisation (R1^-T [A | X_q^T] leaves
// (X_q R1^-1)^T), so neither R1^-1 nor Q1 is ever gathered, and the
// first-order product is on the own rows as well.  (Owning columns instead
// took an exchange of X, of A and of Q1 per pass, the triangular inverse and
// three k^3 products: a minibatch step, contraction included, took 54 us at
// k = 100 and 330 us at k = 200; 45 and 295 us here, 250 us with the contraction
// in FFMA.)  KP = 32 has a form of its own (k_step32.cuh).
//
// All products are FP32 FMAs (a thread per column, 8 rows at a time, the row
// operand broadcast from shared memory): mma.sync TF32 in 3xTF32 form gives
// ~50 multiply-adds per clock and SM here, FFMA up to 128, without the split.
//
// Exchanges are bulk asynchronous copies (cp.async.bulk shared::cta ->
// shared::cluster) completing on the receiver's mbarrier of the source rank.
// Buffers are reused without further synchronisation: a rank sends its
// partials of Gram n + 1 only after it has all blocks of Gram n, and a block
// of Gram n is sent only after its owner has consumed every partial of it.
//
// Hardware barriers of the step kernel's CTA: 0 = __syncthreads (whole CTA);
// in chol_solve 1 = a diagonal block is factored (diagonal warp -> panel), 2 =
// a block row is published and the previous trailing update complete (whole
// CTA), 3 = the next block row is up to date (panel -> diagonal warp).

// pivot ratio R_jj^2 / A_jj below which one more exact Cholesky QR pass runs
// (one pass leaves Q1^T Q1 - I of about eps / ratio times a small constant, and
// the first-order pass squares it), the floor a pivot below FP32 round-off of
// A_jj is raised to (a column numerically dependent on the ones before it:
// the floor keeps R^-1 bounded, the next pass orthonormalises); the largest
// number of plain exact passes per step is StpmUpdateArgs::max_passes
constexpr float kQrExactBelow = 1e-2f;
constexpr float kPivotFloor = 1e-7f;
// shifted restarts: below this pivot ratio the factorisation is redone with
// the shift kShiftScale trace(A) (times 100 for each further restart, at
// most kMaxShifts)
constexpr float kShiftBelow = 1e-5f;
// a first-order pass leaves about k |E|^2: it is repeated while an entry of E
// is above this (the pivot ratios do not bound cond(X): with a few hundred
// nodes per minibatch at k = 160 an exact pass left 0.1), at most 4 times; from
// |E| = 1 / k on it need not contract, and exact passes run instead
constexpr float kFirstOrderBelow = 1e-4f;
constexpr float kShiftScale = 1e-5f;
constexpr int kMaxShifts = 3;

// column stride of the k x k matrices and row blocks: KP + 4 floats, so that
// columns stay 16-byte aligned and the 16-byte accesses of 8 consecutive
// columns fall into different banks
__host__ __device__ constexpr int step_xld(int KP) { return KP + 4; }

// CTAs of the step cluster: KP / 8 to 128, KP / 16 above (at most 16).  A step of
// 4,000 nodes at k = 45, contraction included: 35.8 us with one CTA, 29.4 us
// with KP / 16, 27.8 us with KP / 8; 5,000 nodes at k = 64: 43.6, 33.2, 31.3 us.
__host__ __device__ constexpr int step_ctas(int KP) {
  return KP <= 128 ? KP / 8 : KP / 16;
}

template <int KP, int CL>
struct StepSmem {
  static constexpr int RB = KP / CL, XLD = step_xld(KP), NT = 512;
  // above KP = 128 the partials of all ranks do not fit beside the matrix:
  // each owner then reads them from the ranks' matrix buffers between two
  // cluster barriers
  static constexpr bool PULL = KP > 128;
  static constexpr int PW = (KP + RB + 63) / 64, BW = NT / 32 - PW - 1;  // panel, bulk warps
  static constexpr size_t recv = !PULL ? (size_t)KP * XLD : 0;
  static constexpr size_t rows = (size_t)RB * XLD;
  // matrix, partials, X rows | Q1 rows | block to send, m1..3 and |phi_i|^2,
  // mu1..3, d-sums, original diagonal, diagonal block
  static constexpr size_t floats = (size_t)KP * XLD + recv + 3 * rows + 11 * KP + 128;
  static_assert(KP % CL == 0 && RB % 8 == 0 && BW >= 4, "row blocks of whole 8-row blocks");
  static_assert(KP <= 256 && CL > 1, "16-byte words per column");
  static_assert(floats * sizeof(float) <= 227 * 1024 - 1024, "step kernel shared memory");
};

__device__ __forceinline__ uint32_t smem_addr(const void* p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(bar)), "r"(count)
               : "memory");
}

__device__ __forceinline__ void mbar_arrive_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(bar)),
               "r"(bytes)
               : "memory");
}

// global -> this CTA's shared memory, completing on `bar` (16-byte aligned
// addresses, bytes a multiple of 16)
__device__ __forceinline__ void bulk_copy_g2s(void* dst, const void* src, uint32_t bytes,
                                              uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
          smem_addr(dst)),
      "l"(src), "r"(bytes), "r"(smem_addr(bar))
      : "memory");
}

// waits for the phase with the given parity to complete; false after `limit`
// clock64 cycles (then the caller reports kFlagTimeout instead of hanging)
__device__ __forceinline__ bool mbar_wait_bounded(uint64_t* bar, uint32_t parity,
                                                  long long limit) {
  const long long start = clock64();
  while (true) {
    uint32_t ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
        " selp.u32 %0, 1, 0, p;\n}"
        : "=r"(ok)
        : "r"(smem_addr(bar)), "r"(parity)
        : "memory");
    if (ok) return true;
    if (clock64() - start > limit) return false;
  }
}

__device__ __forceinline__ bool mbar_wait_cluster_bounded(uint64_t* bar, uint32_t parity,
                                                          long long limit) {
  const long long start = clock64();
  while (true) {
    uint32_t ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n"
        " selp.u32 %0, 1, 0, p;\n}"
        : "=r"(ok)
        : "r"(smem_addr(bar)), "r"(parity)
        : "memory");
    if (ok) return true;
    if (clock64() - start > limit) return false;
  }
}

// bulk copy of `bytes` (multiple of 16, 16-byte aligned) from this CTA's
// shared memory to the same offset as dst_local in cluster rank `rank`,
// completing on that rank's copy of the mbarrier at bar_local
__device__ __forceinline__ void bulk_copy_to_rank(const void* dst_local, const void* src,
                                                  uint32_t bytes, uint64_t* bar_local,
                                                  uint32_t rank) {
  uint32_t dst, bar;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(dst) : "r"(smem_addr(dst_local)), "r"(rank));
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(bar) : "r"(smem_addr(bar_local)), "r"(rank));
  asm volatile(
      "cp.async.bulk.shared::cluster.shared::cta.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
      "r"(smem_addr(src)), "r"(bytes), "r"(bar)
      : "memory");
}

__device__ __forceinline__ void load8(const float* p, float (&v)[8]) {
  const float4 a = *reinterpret_cast<const float4*>(p), b = *reinterpret_cast<const float4*>(p + 4);
  v[0] = a.x, v[1] = a.y, v[2] = a.z, v[3] = a.w, v[4] = b.x, v[5] = b.y, v[6] = b.z, v[7] = b.w;
}

__device__ __forceinline__ void store8(float* p, const float (&v)[8]) {
  *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
  *reinterpret_cast<float4*>(p + 4) = make_float4(v[4], v[5], v[6], v[7]);
}

// y_hi -= sum_b R(j0 + b, i0 + i) x_hb, i < 8: rows i0 .. i0+7 of H columns of
// the trailing matrix (x_h: a column's entries of block row j0; Rj = &R(j0, i0)).
// Every lane of a warp reads the same 16-byte words of R, which costs the
// shared memory as much as different ones would: H columns share each.
template <int XLD, int H>
__device__ __forceinline__ void rank8(const float* Rj, const float (&x)[H][8], float (&y)[H][8]) {
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    float r[8];
    load8(Rj + i * XLD, r);
#pragma unroll
    for (int h = 0; h < H; ++h)
#pragma unroll
      for (int b = 0; b < 8; ++b) y[h][i] = fmaf(-r[b], x[h][b], y[h][i]);
  }
}

__device__ __forceinline__ float rsqrt_ftz(float x) {
  float r;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

// ---- Cholesky factorisation and forward substitution on one CTA -------------------
//
// Whole CTA.  A (symmetric, column-major, ld XLD, upper triangle read, rows
// and columns < 8 nb, nb = ceil(k / 8)) = R^T R, and Y (RB columns, ld XLD, the
// first `rows` of them not zero) becomes
// R^-T Y: right-looking over 8-row blocks of the KP + RB columns.  The chain
// that sets the time is that of the diagonal blocks, so one warp does nothing
// else: it factors block J in registers (every lane the same), forward-
// substitutes the 8 columns of block J + 1 and updates that diagonal block.
// Panel warps (two columns per thread) take the factor for the other columns
// of block row J and bring block row J + 1 up to date before the diagonal warp
// asks for it; the bulk warps apply the block to the rows below.  The
// entries of R stay in A above the diagonal blocks; the diagonal blocks are
// not kept.  Rows and columns >= k hold the identity.  Returns the smallest
// pivot ratio (the same in every thread: every CTA of a cluster factors the
// same matrix the same way); a pivot that is not above kPivotFloor times its
// original diagonal (breakdown, or NaN) is raised to that and counts as 0.
// Measured per call at k = 100 (13 blocks): 21k cycles, 1.5k per block (factor
// 0.65k, the rest round trips through shared memory and barriers), against
// 30.7k for a single-thread diagonal factor plus about 5k for the triangular
// inverse and product.
// (No __restrict__ on these shared-memory pointers: other threads write what
// a thread reads after each barrier, and the ratio decides the control flow
// of the whole CTA, so no load may be moved across a barrier.)
template <int KP, int CL>
__device__ float chol_solve(float* A, float* Y, int k, int rows, float* dg, float* dgi,
                            float* dblk, float* rblk, volatile float* s_ratio, float shift) {
  using S = StepSmem<KP, CL>;
  constexpr int XLD = S::XLD, PW = S::PW, BW = S::BW;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int nb = (k + 7) / 8, kk = 8 * nb;
#pragma unroll 1
  for (int i = tid; i < kk; i += S::NT) {
    float d = A[i + i * XLD] + shift;
    if (i >= k) d = 1.f;
    A[i + i * XLD] = d;
    d = fmaxf(d, 1e-30f);
    dg[i] = d;
    dgi[i] = __fdividef(1.f, d);
  }
  __syncthreads();
  if (warp == 0) {
    // the chain of diagonal blocks: factor block J (in every lane's
    // registers), forward-substitute the next 8 columns (lane l: column n0 +
    // l), update the next diagonal block
    float rmin = 1.f;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int e = lane + 32 * h;
      dblk[e] = A[(e & 7) + (e >> 3) * XLD];
    }
#pragma unroll 1
    for (int J = 0; J < nb; ++J) {
      const int j0 = 8 * J, n0 = j0 + 8;
      __syncwarp();
      float d[8][8], d0[8], di[8], ri[8];
      load8(dg + j0, d0);
      load8(dgi + j0, di);
#pragma unroll
      for (int l = 0; l < 8; ++l) {
        float t[8];
        load8(dblk + 8 * l, t);
#pragma unroll
        for (int i = 0; i <= l; ++i) d[i][l] = t[i];
      }
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const float p = d[j][j], least = kPivotFloor * d0[j];
        if (j0 + j < k) rmin = fminf(rmin, p > least ? p * di[j] : 0.f);
        // (fmaxf: a NaN pivot is raised too)
        ri[j] = rsqrt_ftz(fmaxf(p, least));
#pragma unroll
        for (int l = j + 1; l < 8; ++l) d[j][l] *= ri[j];
#pragma unroll
        for (int i = j + 1; i < 8; ++i)
#pragma unroll
          for (int l = i; l < 8; ++l) d[i][l] = fmaf(-d[j][i], d[j][l], d[i][l]);
      }
      // column a: R(b, a) for b < a, then 1 / R(a, a) (every lane stores the same)
#pragma unroll
      for (int l = 0; l < 8; ++l) {
        float t[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) t[i] = i < l ? d[i][l] : ri[l];
        *reinterpret_cast<float4*>(rblk + 8 * l) = make_float4(t[0], t[1], t[2], t[3]);
        if (l >= 4) *reinterpret_cast<float4*>(rblk + 8 * l + 4) = make_float4(t[4], t[5], t[6], t[7]);
      }
      __syncwarp();
      asm volatile("bar.arrive 1, %0;" ::"n"(32 * (PW + 1)) : "memory");
      if (J + 1 < nb) {
        // the panel has brought block row J of these columns up to date
        if (J > 0) asm volatile("bar.sync 3, %0;" ::"n"(32 * (PW + 1)) : "memory");
        if (lane < 8) {
          float* col = A + j0 + (n0 + lane) * XLD;
          float y[8];
          load8(col, y);
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            y[i] *= ri[i];
#pragma unroll
            for (int l = i + 1; l < 8; ++l) y[l] = fmaf(-d[i][l], y[i], y[l]);
          }
          store8(col, y);
        }
      }
      asm volatile("bar.sync 2, %0;" ::"n"(S::NT) : "memory");
      if (J + 1 < nb) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int e = lane + 32 * h, i = e & 7, l = e >> 3;
          float xi[8], xl[8];
          load8(A + j0 + (n0 + i) * XLD, xi);
          load8(A + j0 + (n0 + l) * XLD, xl);
          float v = A[(n0 + i) + (n0 + l) * XLD];
#pragma unroll
          for (int b = 0; b < 8; ++b) v = fmaf(-xi[b], xl[b], v);
          dblk[e] = v;
        }
      }
    }
    if (lane == 0) *s_ratio = rmin;
  } else if (warp <= PW) {
    // the panel, two columns per thread (of A, and past KP the rows of the
    // block as columns): forward substitution of the columns past the diagonal
    // warp's, then their next 8 entries
    constexpr int H = 2;
    float* col[H];
    int cs[H];  // the column; a large number for a row of the block, -1: none
    float y[H][8];
#pragma unroll
    for (int h = 0; h < H; ++h) {
      const int c = tid - 32 + 32 * PW * h;
      const bool aug = c >= KP && c < KP + rows;
      cs[h] = c < kk ? c : aug ? 1 << 30 : -1;
      col[h] = c < kk ? A + c * XLD : Y + (aug ? c - KP : 0) * XLD;
      load8(col[h], y[h]);
    }
#pragma unroll 1
    for (int J = 0; J < nb; ++J) {
      const int j0 = 8 * J, n0 = j0 + 8;
      asm volatile("bar.sync 1, %0;" ::"n"(32 * (PW + 1)) : "memory");  // R_JJ published
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        float r[8];  // R(0 .. i-1, i), 1 / R(i, i)
        load8(rblk + 8 * i, r);
#pragma unroll
        for (int h = 0; h < H; ++h) {
#pragma unroll
          for (int l = 0; l < i; ++l) y[h][i] = fmaf(-r[l], y[h][l], y[h][i]);
          y[h][i] *= r[i];
        }
      }
#pragma unroll
      for (int h = 0; h < H; ++h)
        if (cs[h] >= n0 + 8) store8(col[h] + j0, y[h]);
      // block row J is complete, and the bulk warps are done with J - 1
      asm volatile("bar.sync 2, %0;" ::"n"(S::NT) : "memory");
      if (J + 1 < nb) {
        float x[H][8];
#pragma unroll
        for (int h = 0; h < H; ++h) {
#pragma unroll
          for (int b = 0; b < 8; ++b) x[h][b] = y[h][b];
          load8(col[h] + n0, y[h]);
        }
        rank8<XLD, H>(A + j0 + n0 * XLD, x, y);
        if (J + 2 < nb) {
#pragma unroll
          for (int h = 0; h < H; ++h)
            if (cs[h] >= n0 + 8 && cs[h] < n0 + 16) store8(col[h] + n0, y[h]);
          asm volatile("bar.arrive 3, %0;" ::"n"(32 * (PW + 1)) : "memory");
        }
      }
    }
  } else {
    // rows >= j0 + 16 (the panel threads update the 8 before): a warp per 8
    // rows, the columns from the row block's diagonal on and then those of Y,
    // 32 at a time; the row operand stays in registers (every lane the same
    // words: a broadcast load costs the shared memory as much as any other).
    // (mma.sync TF32 in 3xTF32 form took 3.2k cycles for the first block at k
    // = 100.)
#pragma unroll 1
    for (int J = 0; J < nb; ++J) {
      const int j0 = 8 * J;
      asm volatile("bar.sync 2, %0;" ::"n"(S::NT) : "memory");
#pragma unroll 1
      for (int i0 = j0 + 16 + 8 * (warp - PW - 1); i0 < kk; i0 += 8 * BW) {
        const int nc = kk - i0 + rows;
        float r[8][8];
#pragma unroll
        for (int i = 0; i < 8; ++i) load8(A + j0 + (i0 + i) * XLD, r[i]);
#pragma unroll 1
        for (int u = lane; u < nc; u += 32) {
          float* col = u < kk - i0 ? A + (i0 + u) * XLD : Y + (u - (kk - i0)) * XLD;
          float x[8], y[8];
          load8(col + j0, x);
          load8(col + i0, y);
#pragma unroll
          for (int i = 0; i < 8; ++i)
#pragma unroll
            for (int b = 0; b < 8; ++b) y[i] = fmaf(-r[i][b], x[b], y[i]);
          store8(col + i0, y);
        }
      }
    }
  }
  __syncthreads();
  return *s_ratio;
}

template <int KP>
struct ContractTc;  // the tensor-core contraction's shared-memory layout (below)

template <int KP, int CL>
__device__ __forceinline__ void step_body(const StpmUpdateArgs& a) {
  using S = StepSmem<KP, CL>;
  constexpr int RB = S::RB, XLD = S::XLD, NT = S::NT;
  // one warp of the 512 threads issues the copy to each rank
  static_assert(CL <= 16, "cluster size");
  const int rank = (int)cg::this_cluster().block_rank();
  extern __shared__ __align__(16) float sm[];
  float* A = sm;                       // Phi, then Grams and factors, columns at A + c XLD
  float* Rv = A + KP * XLD;            // column block of the Gram partials of every rank
  float* Xr = Rv + S::recv;            // own rows of X / Q1: row r at Xr + r XLD
  float* Yr = Xr + S::rows;
  float* St = Yr + S::rows;            // finished column block to send
  float* mv = St + S::rows;            // m1 | m2 | m3 | |phi_i|^2 (KP each)
  float* mus = mv + 4 * KP;            // mu1 | mu2 | mu3
  float* dcol = mus + 3 * KP;          // d-sums (3 KP), later 1 / dg
  float* dg = dcol + 3 * KP;           // original diagonal of the Gram
  float* dblk = dg + KP;               // 8 x 8 diagonal block and its factor
  __shared__ float s_ratio, s_shift;
  __shared__ float s_emax[16];
  __shared__ __align__(8) uint64_t s_part[16], s_blk[16];  // partial / block of rank q arrived
  __shared__ __align__(8) uint64_t s_csync[2];             // bounded cluster barrier, in turn
  const int k = a.k, nb = (k + 7) / 8, kk = 8 * nb;
  const int r0 = rank * RB, rows = max(0, min(RB, k - r0));  // own rows that are not padding
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const long long wl = tc::wait_limit_or_default(a.wait_limit);
  {
    // Phi: loads issued in batches of 8 per thread so that their latencies overlap
    constexpr int N = KP * XLD, B = 8;
#pragma unroll 1
    for (int e0 = tid; e0 < N; e0 += NT * B) {
      float v[B];
#pragma unroll
      for (int u = 0; u < B; ++u) {
        const int e = e0 + NT * u, r = e % XLD, c = e / XLD;
        v[u] = (e < N && r < k && c < k) ? __ldg(a.phi + (int64_t)c * k + r) : 0.f;
      }
#pragma unroll
      for (int u = 0; u < B; ++u)
        if (e0 + NT * u < N) A[e0 + NT * u] = v[u];
    }
  }
  const bool online = a.step_mode == kStepOnline;
  if (online)
#pragma unroll 1
    for (int e = tid; e < 3 * KP; e += NT) {
      const int which = e / KP, j = e % KP;
      const float* mu = which == 0 ? a.mu1 : which == 1 ? a.mu2 : a.mu3;
      mus[e] = (mu && j < k) ? __ldg(mu + j) : 0.f;
    }
  if (tid < CL) mbar_init(&s_part[tid], 1);
  else if (tid < 2 * CL) mbar_init(&s_blk[tid - CL], 1);
  else if (tid < 2 * CL + 2) mbar_init(&s_csync[tid - 2 * CL], CL);
  if (tid < 2 * CL + 2) asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  __syncthreads();
  if (online) {
    // mean terms phi_i . mu and |phi_i|^2 of all columns: Phi and mu only, so
    // before the wait.  8 columns x 4 quarters of the rows per warp.
    static_assert(KP % 16 == 0, "quarters of whole 16-byte words");
#pragma unroll 1
    for (int i0 = 8 * warp; i0 < KP; i0 += NT / 4) {
      const int i = i0 + (lane & 7), h = lane >> 3;
      float s[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 1
      for (int j = h * (KP / 4); j < (h + 1) * (KP / 4); j += 4) {
        const float4 x = *reinterpret_cast<const float4*>(A + i * XLD + j);
#pragma unroll
        for (int q = 0; q < 3; ++q) {
          const float4 m = *reinterpret_cast<const float4*>(mus + q * KP + j);
          s[q] = fmaf(x.x, m.x, fmaf(x.y, m.y, fmaf(x.z, m.z, fmaf(x.w, m.w, s[q]))));
        }
        s[3] = fmaf(x.x, x.x, fmaf(x.y, x.y, fmaf(x.z, x.z, fmaf(x.w, x.w, s[3]))));
      }
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        s[q] += __shfl_xor_sync(0xffffffffu, s[q], 8);
        s[q] += __shfl_xor_sync(0xffffffffu, s[q], 16);
        if (h == 0) mv[q * KP + i] = s[q];
      }
    }
  }
  cg::this_cluster().sync();  // barriers initialised everywhere before any copy
  // launched with programmatic serialization after the contraction, the
  // prologue above overlapped its tail (Phi is final: the contraction lets
  // this kernel start only after its own wait on the previous step); from
  // here on its partials are read, so wait for it to complete, and let the
  // next contraction be scheduled (it waits for this kernel in turn)
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  uint32_t par_part = 0u, par_blk = 0u, csync_n = 0u;
  bool timed_out = false;
  // bounded cluster barrier: every thread of every CTA has passed the
  // __syncthreads before its rank's arrival (remote mbarrier arrives with
  // release semantics, waited for with acquire); false after a timeout.  Two
  // mbarriers in turn: a rank past barrier n may arrive for n + 1 where phase
  // n still misses an arrival.
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
  constexpr uint32_t kBlockBytes = sizeof(float) * RB * XLD;

  // X^T X of the CTA's rows X into A (upper triangle, 8-row blocks), summed
  // over the cluster; first_order: F of E = X^T X - I instead.  Leaves the
  // whole matrix in every CTA; false after a timeout.  (One call site: the
  // step runs through its code once, and instruction fetch from L2 was its
  // largest cost while the kernel had 88 KB of it.)
  float emax = 0.f;
  auto gram = [&](const float* X, bool first_order) -> bool {
    __syncthreads();  // X complete, A free
    // a warp per 8 rows, 4 columns per lane (the row operand is a broadcast:
    // every load of it serves 4 columns)
#pragma unroll 1
    for (int i0 = 8 * warp; i0 < kk; i0 += 8 * (NT / 32)) {
#pragma unroll 1
      for (int c0 = i0; c0 < kk; c0 += 128) {
        float acc[4][8];
#pragma unroll
        for (int h = 0; h < 4; ++h)
#pragma unroll
          for (int i = 0; i < 8; ++i) acc[h][i] = 0.f;
#pragma unroll 1
        for (int rb = 0; rb < rows; rb += 8) {
          // 8 rows apart from the sum so far: less round-off than one long chain
          float part[4][8];
#pragma unroll
          for (int h = 0; h < 4; ++h)
#pragma unroll
            for (int i = 0; i < 8; ++i) part[h][i] = 0.f;
#pragma unroll 2
          for (int r = rb; r < rb + 8; ++r) {
            float w[8];
            load8(X + r * XLD + i0, w);
#pragma unroll
            for (int h = 0; h < 4; ++h) {
              const int c = c0 + 32 * h + lane;
              const float x = c < kk ? X[r * XLD + c] : 0.f;
#pragma unroll
              for (int i = 0; i < 8; ++i) part[h][i] = fmaf(w[i], x, part[h][i]);
            }
          }
#pragma unroll
          for (int h = 0; h < 4; ++h)
#pragma unroll
            for (int i = 0; i < 8; ++i) acc[h][i] += part[h][i];
        }
#pragma unroll
        for (int h = 0; h < 4; ++h) {
          const int c = c0 + 32 * h + lane;
          if (c < kk) store8(A + c * XLD + i0, acc[h]);
        }
      }
    }
    bool bad = false;
    auto finish = [&](float4 v, int c, int i4) {
      float w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int i = 4 * i4 + u;
        if (i <= c && !isfinite(w[u])) bad = true;  // (nothing below the diagonal is read)
        if (first_order) {
          const float e = i <= c && c < k ? w[u] - (i == c ? 1.f : 0.f) : 0.f;
          emax = fmaxf(emax, fabsf(e));
          w[u] = i < c ? e : 0.5f * e;
        }
      }
      return make_float4(w[0], w[1], w[2], w[3]);
    };
    const int cols = max(0, min(RB, kk - r0)), n4 = kk / 4;
    bool ok = true;
    if (!S::PULL) {
      // column block s of the partial to rank s, rank q's next neighbours
      // first (copies issued by lanes of one warp serialise)
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncthreads();
      if (lane == 0 && warp < CL - 1) {
        const int to = (rank + 1 + warp) % CL;
        bulk_copy_to_rank(Rv + rank * RB * XLD, A + to * RB * XLD, kBlockBytes, &s_part[rank],
                          (uint32_t)to);
      }
      if (tid < CL && tid != rank) {
        mbar_arrive_expect_tx(&s_part[tid], kBlockBytes);
        ok = mbar_wait_bounded(&s_part[tid], par_part, wl);
      }
      par_part ^= 1u;
      if (__syncthreads_or(!ok)) return false;
    } else {
      csync_arrive();
      if (!csync_wait()) return false;
    }
    // own block: the ranks' partials added in rank order
#pragma unroll 1
    for (int e = tid; e < cols * 64; e += NT) {
      const int c = e >> 6, i4 = e & 63;  // (n4 <= 52)
      if (i4 >= n4) continue;
      float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
      for (int q = 0; q < CL; ++q) {
        const float* src;
        if (S::PULL)
          src = cg::this_cluster().map_shared_rank(A, q) + (r0 + c) * XLD;
        else
          src = q == rank ? A + (r0 + c) * XLD : Rv + (q * RB + c) * XLD;
        const float4 t = reinterpret_cast<const float4*>(src)[i4];
        v.x += t.x, v.y += t.y, v.z += t.z, v.w += t.w;
      }
      reinterpret_cast<float4*>(St + c * XLD)[i4] = finish(v, r0 + c, i4);
    }
    if (bad) atomicOr(a.flags, kFlagNonFinite);
    if (S::PULL) {
      csync_arrive();  // every rank has read the partials: blocks may land on them
      if (!csync_wait()) return false;
    }
    // (a flag in the padding of the block's first column: see left_over)
    const bool large = __syncthreads_or(first_order && emax > kFirstOrderBelow) != 0;
    const bool wide = large && __syncthreads_or(emax * (float)k > 1.f) != 0;
    const float flag = wide ? 2.f : large ? 1.f : 0.f;
    if (tid == 0) St[KP] = flag;
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncthreads();
    if (lane == 0 && warp < CL - 1)
      bulk_copy_to_rank(A + r0 * XLD, St, kBlockBytes, &s_blk[rank],
                        (uint32_t)((rank + 1 + warp) % CL));
#pragma unroll 1
    for (int e = tid; e < cols * 64; e += NT)
      if ((e & 63) < n4)
        reinterpret_cast<float4*>(A + (r0 + (e >> 6)) * XLD)[e & 63] =
            reinterpret_cast<const float4*>(St + (e >> 6) * XLD)[e & 63];
    if (tid == 0) A[r0 * XLD + KP] = flag;
    if (tid < CL && tid != rank) {
      mbar_arrive_expect_tx(&s_blk[tid], kBlockBytes);
      ok = mbar_wait_bounded(&s_blk[tid], par_blk, wl);
    }
    par_blk ^= 1u;
    return !__syncthreads_or(!ok);
  };

  // 1 where any rank's block of E had an entry above kFirstOrderBelow, 2 where
  // one was above 1 / k (the same in every CTA: the blocks carry it in their
  // padding)
  auto left_over = [&]() -> float {
    float f = 0.f;
    for (int q = 0; q < CL; ++q) f = fmaxf(f, A[q * RB * XLD + KP]);
    return f;
  };

  float* M = Xr;  // own rows of the matrix to orthonormalise
  float* F = Yr;
  if (online) {
    // own rows of G from the contraction's partials, 4 rows of one column per
    // item (a 16-byte load per partial where the rows allow it), and the
    // d-sums of all columns (3 KP, zero past k).  The first 8 partials of a
    // thread's first item and of its d-sum are loaded together: one L2 round
    // trip (~1.7k cycles for lines another SM has just written) covers them.
    const bool vec = ((k | (int)a.part_stride) & 3) == 0 && ((uintptr_t)a.gpart & 15) == 0;
    constexpr int PRE = 8, ITEMS = KP * (RB / 4);
    static_assert(3 * KP <= 2 * NT, "two d-sums per thread");
    auto load4 = [&](const float* p, int j) {  // rows j .. j+3 of one partial
      if (vec) return __ldg(reinterpret_cast<const float4*>(p));
      float4 v = make_float4(__ldg(p), 0.f, 0.f, 0.f);
      if (j + 1 < k) v.y = __ldg(p + 1);
      if (j + 2 < k) v.z = __ldg(p + 2);
      if (j + 3 < k) v.w = __ldg(p + 3);
      return v;
    };
#pragma unroll 1
    for (int e = tid; e < max(ITEMS, 3 * KP); e += NT) {
      const int i = e / (RB / 4), rr = 4 * (e % (RB / 4)), j = r0 + rr;
      const bool live = e < ITEMS && i < k && j < k;
      const float* gp = a.gpart + (int64_t)i * k + j;
      const int which = e / KP, di = e % KP;
      const bool dlive = which < 3 && di < k && (which == 0 || a.mode == kModeAdjoint);
      const float* dp = a.gpart + (int64_t)k * k + which * k + di;
      float4 g = make_float4(0.f, 0.f, 0.f, 0.f);
      float d = 0.f;
#pragma unroll 1
      for (int p0 = 0; p0 < a.nparts; p0 += PRE) {
        float4 v[PRE];
        float w[PRE];
#pragma unroll
        for (int u = 0; u < PRE; ++u) {
          const bool has = p0 + u < a.nparts;
          v[u] = has && live ? load4(gp + (int64_t)(p0 + u) * a.part_stride, j)
                             : make_float4(0.f, 0.f, 0.f, 0.f);
          w[u] = has && dlive ? __ldg(dp + (int64_t)(p0 + u) * a.part_stride) : 0.f;
        }
        // (8 partials as a tree: the sum's round-off grows with its depth)
#pragma unroll
        for (int h = PRE / 2; h; h >>= 1)
#pragma unroll
          for (int u = 0; u < h; ++u) {
            v[u].x += v[u + h].x, v[u].y += v[u + h].y;
            v[u].z += v[u + h].z, v[u].w += v[u + h].w;
            w[u] += w[u + h];
          }
        g.x += v[0].x, g.y += v[0].y, g.z += v[0].z, g.w += v[0].w;
        d += w[0];
      }
      if (e < ITEMS) {
        Xr[rr * XLD + i] = g.x;
        Xr[(rr + 1) * XLD + i] = g.y;
        Xr[(rr + 2) * XLD + i] = g.z;
        Xr[(rr + 3) * XLD + i] = g.w;
      }
      if (which < 3) dcol[e] = d;
    }
    // X = Phi - beta (3 theta Phi (Phi^T Phi)^.2 - gscale G)   (Util.cpp:259-272)
    const float alpha = -a.beta * a.theta3, gamma = a.beta * a.gscale;
    if (a.phi_general) {
      // the literal product (first step of a run: Phi0 need not be
      // orthonormal), 16 columns of (Phi^T Phi)^.2 at a time (in Yr | St); every
      // CTA forms all of them, once per run.  Xr then holds both terms.
      float* S2 = Yr;
      static_assert(2 * RB * XLD >= 16 * XLD, "16 columns in Q1's rows and the staged block");
      constexpr int PER = (16 * RB + NT - 1) / NT;  // products per thread and 16 columns
#pragma unroll 1
      for (int i0 = 0; i0 < KP; i0 += 16) {
        __syncthreads();
#pragma unroll 1
        for (int e = tid; e < KP * 16; e += NT) {
          const int l = e % KP, i = i0 + e / KP;
          float s = 0.f;
#pragma unroll 1
          for (int j = 0; j < KP; j += 4) {
            const float4 x = *reinterpret_cast<const float4*>(A + l * XLD + j);
            const float4 y = *reinterpret_cast<const float4*>(A + i * XLD + j);
            s = fmaf(x.x, y.x, fmaf(x.y, y.y, fmaf(x.z, y.z, fmaf(x.w, y.w, s))));
          }
          S2[(i - i0) * XLD + l] = s * s;
        }
        __syncthreads();
#pragma unroll
        for (int t = 0; t < PER; ++t) {
          const int e = tid + NT * t, r = e % RB, ii = e / RB, i = i0 + ii;
          if (e < 16 * RB) {
            float s = 0.f;
#pragma unroll 1
            for (int l = 0; l < k; ++l) s = fmaf(A[l * XLD + r0 + r], S2[ii * XLD + l], s);
            Xr[r * XLD + i] = fmaf(alpha, s, gamma * (Xr[r * XLD + i] * a.scale));
          }
        }
      }
    }
    __syncthreads();
#pragma unroll 1
    for (int e = tid; e < RB * XLD; e += NT) {
      const int r = e / XLD, i = e % XLD, j = r0 + r;
      float x = 0.f;
      if (i < k && j < k) {
        const float m1 = mv[i], m2 = mv[KP + i], m3 = mv[2 * KP + i];
        const float c1 = a.c1, c2 = a.c2;
        // (explicit fmaf here: the single and the batched kernel must round alike)
        float gm;  // the mean terms of the gradient
        if (a.mode == kModePlain) {
          gm = mus[2 * KP + j] * fmaf(c1 * m1, m2, c2 * dcol[i]);
        } else {
          const float c2n = c2 * a.inv_count;
          gm = fmaf(mus[j], fmaf(c1 * m2, m3, c2n * dcol[i]),
                    fmaf(mus[KP + j], fmaf(c1 * m1, m3, c2n * dcol[KP + i]),
                         mus[2 * KP + j] * fmaf(c1 * m1, m2, c2n * dcol[2 * KP + i])));
        }
        const float phi = A[i * XLD + j], g = Xr[e];
        if (a.phi_general) {
          x = phi + fmaf(gamma, gm, g);
        } else {
          // Phi is the previous step's Q: Phi^T Phi = I to ~1e-7, so
          // (Phi^T Phi)^.2 = diag(|phi_i|^4) + O(1e-14) and Phi times it is
          // phi_i |phi_i|^4, column by column
          const float n2 = mv[3 * KP + i] * mv[3 * KP + i];
          x = fmaf(phi, fmaf(alpha, n2, 1.f), gamma * fmaf(g, a.scale, gm));
        }
      }
      Xr[e] = x;
    }
  } else {
#pragma unroll 1
    for (int e = tid; e < RB * XLD; e += NT) {
      const int r = e / XLD, i = e % XLD;
      Xr[e] = i < KP ? A[i * XLD + r0 + r] : 0.f;
    }
  }
  // Cholesky QR passes: A = M^T M, M <- M R^-1
  int passes = 0, shifts = 0, plain_left = a.max_passes;
  float shift = 0.f;
  bool first_order = false;  // the second pass: E = M^T M - I, Phi = M (I - F)
  int orders = 0, wide_left = a.max_passes;
  float emax_all = 0.f;
  while (true) {
    if (!gram(M, first_order)) {
      timed_out = true;
      break;
    }
    if (first_order) {
      const float left = left_over();
      if (left > 1.f && wide_left > 0) {
        --wide_left;
        emax_all = fmaxf(emax_all, emax);
        emax = 0.f;
        first_order = false;
        continue;
      }
      const bool more = left > 0.f && orders < 4;
      if (left > 0.f && !more && rank == 0 && tid == 0) atomicOr(a.flags, kFlagNoConvergence);
      ++orders;
      // no copy to this CTA is outstanding after the last pass; its own may
      // still be read by others, so it stays until every rank has arrived here
      if (!more) csync_arrive();
      // own rows of M - M F: RT rows of one column per item, F's column in
      // 16-byte words down to the diagonal
      constexpr int RT = RB >= 32 ? 4 : 2;
#pragma unroll 1
      for (int e = tid; e < KP * (RB / RT); e += NT) {
        const int c = e % KP, r = RT * (e / KP);
        float s[RT];
#pragma unroll
        for (int u = 0; u < RT; ++u) s[u] = 0.f;
        if (c < k && r < rows)
#pragma unroll 2
          for (int i = 0; i <= c; i += 4) {
            const float4 f = *reinterpret_cast<const float4*>(A + c * XLD + i);
#pragma unroll
            for (int u = 0; u < RT; ++u) {
              const float4 m = *reinterpret_cast<const float4*>(M + (r + u) * XLD + i);
              s[u] = fmaf(m.x, f.x, fmaf(m.y, f.y, fmaf(m.z, f.z, fmaf(m.w, f.w, s[u]))));
            }
          }
#pragma unroll
        for (int u = 0; u < RT; ++u) {
          const int j = r0 + r + u;
          const float v = c < k && j < k ? M[(r + u) * XLD + c] - s[u] : 0.f;
          F[(r + u) * XLD + c] = v;
        }
      }
      if (!more) break;
      emax_all = fmaxf(emax_all, emax);
      emax = 0.f;
      float* t = M;
      M = F;
      F = t;
      continue;
    }
#pragma unroll 1
    for (int e = tid; e < RB * XLD; e += NT) F[e] = M[e];
    const float ratio = chol_solve<KP, CL>(A, F, k, rows, dg, dcol, dblk, dblk + 64, &s_ratio, shift);
    if (__syncthreads_or(ratio < kShiftBelow) && shifts < kMaxShifts) {
      // near breakdown: the Gram again, factored with a diagonal shift
      if (tid == 0) {
        float tr = 0.f;
#pragma unroll 1
        for (int i = 0; i < k; ++i) tr += dg[i];
        s_shift = shift > 0.f ? 100.f * shift : kShiftScale * tr;
      }
      __syncthreads();
      shift = s_shift;
      ++shifts;
      continue;
    }
    ++passes;
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
      first_order = true;
    }
  }
  if (!timed_out) {
    emax = fmaxf(emax, emax_all);
#pragma unroll
    for (int off = 16; off; off >>= 1) emax = fmaxf(emax, __shfl_xor_sync(0xffffffffu, emax, off));
    if (lane == 0) s_emax[warp] = emax;
    __syncthreads();
#pragma unroll 1
    for (int e = tid; e < KP * RB; e += NT) {
      const int r = e % RB, c = e / RB;
      if (c < k && r0 + r < k) a.phi[(int64_t)c * k + r0 + r] = F[r * XLD + c];
    }
    if (tid == 0) {
      float m = 0.f;
#pragma unroll 1
      for (int w = 0; w < NT / 32; ++w) m = fmaxf(m, s_emax[w]);
      if (a.orth_err) atomicMax(reinterpret_cast<int*>(a.orth_err), __float_as_int(m));
    }
    if constexpr (KP <= 112) {
      if (a.phi_img) {
        // the next contraction's operand image (rows i of its A operand, K =
        // j): TF32 hi / lo of the own 16-byte words along j, in the core-matrix
        // layout
        using CT = ContractTc<KP>;
        unsigned char* img = static_cast<unsigned char*>(a.phi_img);
#pragma unroll 1
        for (int e = tid; e < KP * (RB / 4); e += NT) {
          const int i = e % KP, r = 4 * (e / KP);
          float v[4];
#pragma unroll
          for (int u = 0; u < 4; ++u) v[u] = F[(r + u) * XLD + i];  // zero past k
          uint4 h;
          float4 l;
          tc::split4(v, h, l);
          const uint32_t off = tc::kmajor_off(i, r0 + r, CT::SBOJ);
          *reinterpret_cast<uint4*>(img + CT::PH + off) = h;
          *reinterpret_cast<float4*>(img + CT::PL + off) = l;
        }
      }
    }
    if (a.trace_out) {  // ||Phi_new - snapshot||_F^2 over this CTA's rows, fixed order
      double d2 = 0.0;
#pragma unroll 1
      for (int e = tid; e < KP * RB; e += NT) {
        const int r = e % RB, c = e / RB, j = r0 + r;
        if (j < k && c < k) {
          const float v = F[r * XLD + c];
          const double d = (double)v - (double)a.trace_snap[(int64_t)c * k + j];
          d2 = fma(d, d, d2);
          a.trace_snap[(int64_t)c * k + j] = v;
        }
      }
#pragma unroll
      for (int off = 16; off; off >>= 1) d2 += __shfl_xor_sync(0xffffffffu, d2, off);
      __shared__ double tpart[16];
      if (lane == 0) tpart[warp] = d2;
      __syncthreads();
      if (tid == 0) {
        double t = 0.0;
#pragma unroll 1
        for (int w = 0; w < NT / 32; ++w) t += tpart[w];
        a.trace_out[rank] = t;
      }
    }
  }
  if (timed_out && tid == 0) atomicOr(a.flags, kFlagTimeout);
  if (rank == 0 && tid == 0 && a.orth_passes) atomicAdd(a.orth_passes, passes);
  // keep shared memory alive until remote readers and writers are done
  // (bounded: after a timeout the ranks may stand at different barriers)
  if (timed_out) csync_arrive();
  if (!csync_wait()) {
    if (tid == 0) atomicOr(a.flags, kFlagTimeout);
    __nanosleep(100000);  // let copies a stalled exchange left in flight land
  }
}

// ---- partial contractions --------------------------------------------------------
//
// Per tile of TM nodes, with Phi resident in shared memory:
//   Z_q^T = Phi^T Y_q^T           (k x TM)
//   C = c0 Z1.Z2 + c2 (Z1 m2 + m1 Z2)
//   G += Yout^T C                 (k x k, accumulated over the CTA's tiles)
//   d_i += sum_x Z1 Z2            (per column i)
// in one of four forms: contract_tc (tcgen05, 3xTF32: the plain FP32 form up to
// KP = 112), contract_tc_bf (tcgen05, BF16: the adjoint form up to KP = 112),
// contract_ffma (the other FP32 forms) and the mma.sync body of contract_body
// (the other BF16 forms, m16n8k16; m16n8k8 in 3xTF32 form for the FP32 adjoint
// steps of KP = 32).  The BF16 forms read y rounded to BF16, Phi as a BF16 pair
// (hi + lo: Z = hi^T y + lo^T y, two MMAs) and the coefficients C rounded to
// BF16, and accumulate in FP32.
//
// Tensor-core form of the plain FP32 contraction (tcgen05.mma kind::tf32,
// 3xTF32: D += Ahi Bhi + Ahi Blo + Alo Bhi), for KP in [32, 112].  Per tile
// of TM = 32 nodes:
//   [Z1 Z2] = Phi^T [y1 y2]      A = Phi  (M = i, K = j), B = y1 | y2 (N = 2 TM, K = j)
//   C   = c0 Z1 Z2 + c2 (Z1 m2 + m1 Z2)   (TMEM -> registers -> shared)
//   G  += y3^T C                 A = y3   (M = j, K = x), B = C   (N = i, K = x)
// Z1, Z2 and G live in tensor memory (columns [0, TM), [TM, 2 TM),
// [2 TM, 2 TM + KP)); G accumulates over the CTA's tiles.  Every accumulation
// truncates (about 0.3 of an ulp each), so the products are spread:
// the small ones (hi lo, lo hi) of Z come first, its large ones go to two or
// three accumulators, and the small products of G have one of their own.  The
// first steps of a run, where the iterate is near singular, multiply that error
// by 10 to 50: after 4 of them Phi was 3.6e-5 off at k = 100 (median of 8 runs)
// with one chain of each and 1.5e-5 here, 0.9e-5 and 0.6e-5 at k = 33.  (KP = 32
// keeps one chain of each, see CHAIN.)  Operands are
// staged hi / lo in shared memory, K-major without swizzle; y3 is staged
// transposed (node index along K).  An M = 128 operand of KP < 128 rows
// reads its rows past KP from the buffer after it: their products land in
// TMEM lanes that are never read.
template <int KP>
struct ContractTc {
  static constexpr int TM = 32;
  static constexpr uint32_t SBOJ = (KP / 4) * 128u;  // 8-row groups of a K = j operand
  static constexpr uint32_t SBOX = (TM / 4) * 128u;  // 8-row groups of a K = x operand
  static constexpr uint32_t PSZ = 4u * KP * KP, TSZ = 4u * TM * KP;
  static constexpr uint32_t PH = 0, PL = PSZ;                                   // Phi, KP rows i
  // y1 hi | y2 hi | y1 lo | y2 lo (TM rows x each): y1 and y2 stack into one
  // operand of N = 2 TM rows, so one MMA makes Z1 and Z2 side by side
  static constexpr uint32_t Y1H = 2 * PSZ, Y2H = Y1H + TSZ, Y1L = Y2H + TSZ, Y2L = Y1L + TSZ;
  static constexpr uint32_t Y3H = Y2L + TSZ, Y3L = Y3H + TSZ;                   // KP rows j
  static constexpr uint32_t CH = Y3L + TSZ, CLO = CH + TSZ;                     // KP rows i
  static constexpr uint32_t END = CLO + TSZ;
  static constexpr uint32_t READ_END =  // furthest byte read by an M = 128 operand
      (Y3L + 16 * SBOX > PL + 16 * SBOJ) ? Y3L + 16 * SBOX : PL + 16 * SBOJ;
  static constexpr uint32_t STAGE = 4u * (KP * KP + 3 * KP + 1);  // partial for the cluster sum
  static constexpr uint32_t REGION0 = END > READ_END ? END : READ_END;
  static constexpr uint32_t REGION = ((REGION0 > STAGE ? REGION0 : STAGE) + 127) / 128 * 128;
  // alignment slack, m1 | m2, d-sums of the 4 node groups
  static constexpr size_t smem = 1024 + REGION + sizeof(float) * (2 * KP + 4 * KP);
  // KP = 32: one accumulator for Z1 | Z2 and one for G, each a single chain, and
  // Phi^T mu from the step kernel, behind the image: results up to k = 32 keep
  // their roundings (k_step32.cuh)
  static constexpr bool CHAIN = KP == 32;
  // further accumulators of Z1 | Z2: two, or one where two CTAs share an SM
  static constexpr int NZX = CHAIN ? 0 : KP <= 64 ? 1 : 2;
  static constexpr uint32_t ZX = 2 * TM + 2 * KP;
  static constexpr uint32_t TMEM_COLS = KP <= 64 ? 256 : 512;
  static_assert(ZX + NZX * 2 * TM <= TMEM_COLS, "tensor memory columns");
  static_assert(KP <= 64 || smem > 114 * 1024, "512 tensor memory columns: one CTA per SM");
  static_assert(KP % 16 == 0 && KP >= 32 && KP <= 112, "tensor-core contraction: KP in [32, 112]");
  static_assert(smem <= 227 * 1024, "tensor-core contraction shared memory");
};

#include "k_step32.cuh"

template <int KP, int CL>
__global__ void __launch_bounds__(512, 1) stpm_step_kernel(StpmUpdateArgs a) {
  if constexpr (KP == 32) step32::body(a);
  else step_body<KP, CL>(a);
}

// one cluster per graph: blockIdx.y selects the graph's arguments; graphs
// with no update in this round (active == 0) leave at once
template <int KP, int CL>
__global__ void __launch_bounds__(512, 1) stpm_step_batched(const StpmUpdateArgs* __restrict__ args) {
  const StpmUpdateArgs a = args[blockIdx.y];
  if (!a.active) return;
  if constexpr (KP == 32) step32::body(a);
  else step_body<KP, CL>(a);
}

// BF16 tensor-core form of the adjoint contraction (tcgen05.mma kind::f16,
// BF16 operands, FP32 accumulation), for KP in [32, 112]: per tile of TM = 64
// nodes
//   [Z1 Z2 Z3] = Phi^T [y1 y2 y3]  A = Phi as a BF16 hi / lo pair (M = i, K = j),
//                                  B = y1 | y2 | y3 (N = 3 TM, K = j)
//   C_1..3 (alpha0 terms of the Z pairs, BF16)       TMEM -> registers -> shared
//   G += sum_c y_c^T C_c           A = y_c staged transposed (M = j, K = x),
//                                  B = C_c (N = i, K = x)
// Z in TMEM columns [0, 3 TM), G in [3 TM, 3 TM + KP).  16-bit operands: a
// core matrix is 8 rows x 8 elements, one MMA consumes K = 16.
template <int KP>
struct ContractTcBf {
  static constexpr int TM = 64;
  static constexpr uint32_t SBOJ = (KP / 8) * 128u;  // 8-row groups of a K = j operand
  static constexpr uint32_t SBOX = (TM / 8) * 128u;  // 8-row groups of a K = x operand
  static constexpr uint32_t PSZ = 2u * KP * KP, TSZ = 2u * TM * KP;
  static constexpr uint32_t PH = 0, PL = PSZ;   // Phi hi / lo, KP rows i
  static constexpr uint32_t YB = 2 * PSZ;       // y1 | y2 | y3, TM rows x each
  static constexpr uint32_t YT = YB + 3 * TSZ;  // y_c transposed, KP rows j each
  static constexpr uint32_t CB = YT + 3 * TSZ;  // C_c, KP rows i each
  static constexpr uint32_t END = CB + 3 * TSZ;
  static constexpr uint32_t READ_END =  // furthest byte an M = 128 operand reads (Phi lo, y3^T)
      (YT + 2 * TSZ + 16 * SBOX > PL + 16 * SBOJ) ? YT + 2 * TSZ + 16 * SBOX : PL + 16 * SBOJ;
  static constexpr uint32_t STAGE = 4u * (KP * KP + 3 * KP + 1);
  static constexpr uint32_t REGION0 = END > READ_END ? END : READ_END;
  static constexpr uint32_t REGION = ((REGION0 > STAGE ? REGION0 : STAGE) + 127) / 128 * 128;
  // alignment slack, m1 | m2 | m3, d-sums (3 pairs x 4 node groups)
  static constexpr size_t smem = 1024 + REGION + sizeof(float) * (3 * KP + 12 * KP);
  static constexpr uint32_t TMEM_COLS = 512;
  static_assert(KP % 16 == 0 && KP >= 32 && KP <= 112, "BF16 tensor-core contraction: KP in [32, 112]");
  static_assert(3 * TM + KP <= 512, "tensor memory columns");
  static_assert(smem <= 227 * 1024, "BF16 tensor-core contraction shared memory");
};

template <int KP, bool TC, bool TCBF>
constexpr size_t contract_smem(size_t cuda_core_form) {
  if constexpr (TC)
    return ContractTc<KP>::smem;
  else if constexpr (TCBF)
    return ContractTcBf<KP>::smem;
  else
    return cuda_core_form;
}

template <int KP, int MODE, bool BF>
struct Contract {
  static constexpr bool TC = MODE == kModePlain && !BF && KP <= 112;
  static constexpr bool TCBF = MODE == kModeAdjoint && BF && KP <= 112;
  // FP32 on mma.sync in 3xTF32 form: the adjoint steps of KP = 32, whose results
  // keep their roundings (k_step32.cuh); the other FP32 forms off tcgen05 are FFMA
  static constexpr bool MMA32 = MODE == kModeAdjoint && !BF && KP == 32;
  static constexpr bool FFMA = !BF && !TC && !MMA32;
  using T = typename std::conditional<BF, __nv_bfloat16, float>::type;
  // two CTAs per SM up to KP = 64 (64 registers a thread: without the bound the
  // compiler takes 82 at KP = 48, and an iteration of the power method at k = 33,
  // 10,000 nodes, took 28.8 us against 23.1 us)
  static constexpr int CTAS = TC && KP <= 64 ? 2 : 1;
  static constexpr int TM = BF ? 64 : 32;  // nodes per tile
  static constexpr int NZ = MODE == kModePlain ? 2 : 3;
  static constexpr int NC = MODE == kModePlain ? 1 : MODE == kModeAdjoint ? 3 : 0;
  // columns i of Phi handled by one CTA: all of them up to KP = 128, above
  // that halves in FP32 and blocks of 64 in BF16 (blockIdx.y), so that Phi's
  // block, the G accumulators and the staged partial fit one SM; Z, C, G and
  // the d-sums are separable by column
  static constexpr int IB = KP <= 128 ? KP : BF ? 64 : KP / 2;
  static constexpr int NBC = (KP + IB - 1) / IB;  // column blocks (<= 4: one loss slot each)
  static constexpr int PAD = BF ? 8 : 4;   // row strides == 4 words mod 8: conflict-free fragments
  static constexpr int PLD = KP + PAD, LDY = KP + PAD, LDC = TM + PAD;
  static constexpr int MTI = IB / 16, NTX = TM / 8;        // Z^T tiles: i (16) x nodes (8)
  static constexpr int MTJ = KP / 16, NTI = IB / 8;        // G tiles: j (16) x i (8)
  static constexpr int NW = 16, NT = 32 * NW;               // warps, threads per CTA
  static constexpr int GT = MTJ * NTI, GPW = (GT + NW - 1) / NW;  // G tiles, per warp
  static constexpr int KSTEP = BF ? 16 : 8;
  // the BF16 form keeps Phi as a pair of BF16 arrays (hi + lo): rounding Phi
  // itself to BF16 would bias every product Phi^T y of a step the same way
  static constexpr int NPHI = BF ? 2 : 1;
  static constexpr size_t tile_bytes =
      sizeof(T) * ((size_t)NPHI * IB * PLD + (size_t)3 * TM * LDY + (size_t)NC * IB * LDC);
  // FP32 form on the CUDA cores (contract_ffma): thread tiles of the Z products
  // (4 columns i x XT nodes) and of the G products (8 j x GI columns i)
  static constexpr int XT = KP >= 96 ? 4 : 2;
  static constexpr int ZTH = (IB / 4) * (TM / XT);
  static constexpr int GI = (KP / 8) * (IB / 4) <= NT ? 4 : 8;
  static constexpr int GTH = (KP / 8) * (IB / GI);
  // the nodes of a tile go to GPARTS thread groups where one leaves most idle
  // (an adjoint step of 16,384 nodes at k = 20: 36.7 us with one, 29.7 us)
  static constexpr int GPARTS = NC == 0 ? 1 : 8 * GTH <= NT ? 8 : 4 * GTH <= NT ? 4 : 2 * GTH <= NT ? 2 : 1;
  static_assert(BF || (ZTH <= NT && GTH <= NT && IB % 8 == 0), "thread tiles");
  // the staged partial; the FP32 form's d-sums of the node groups and the other
  // thread groups' G follow it
  static constexpr size_t DPART = ((size_t)KP * IB + 3 * IB + 4 + 3) / 4 * 4;
  static constexpr size_t stage_bytes =
      sizeof(float) *
      (DPART + (FFMA ? (size_t)(TM / 2) * 3 * IB + (size_t)(GPARTS - 1) * KP * IB : 0));
  static constexpr size_t region = ((tile_bytes > stage_bytes ? tile_bytes : stage_bytes) + 15) / 16 * 16;
  // m1..3, loss partials, and the warps' d-sums (MMA) or mu1..3 (FFMA)
  static constexpr size_t smem_mma =
      region + sizeof(float) * (3 * IB + NW + (FFMA ? 3 * KP : NW * 3 * IB));
  static_assert(TC || TCBF || smem_mma <= 227 * 1024 - 1024, "contraction shared memory");
  static constexpr size_t smem = contract_smem<KP, TC, TCBF>(smem_mma);
  static_assert(NBC <= 4, "one loss slot per column block");
};

template <typename T>
__device__ __forceinline__ T to_elem(float v);
template <>
__device__ __forceinline__ float to_elem<float>(float v) { return v; }
template <>
__device__ __forceinline__ __nv_bfloat16 to_elem<__nv_bfloat16>(float v) { return __float2bfloat16_rn(v); }

__device__ __forceinline__ float to_f32(float v) { return v; }
__device__ __forceinline__ float to_f32(__nv_bfloat16 v) { return __bfloat162float(v); }

__device__ __forceinline__ uint32_t ld_b32(const void* p) { return *reinterpret_cast<const uint32_t*>(p); }

__device__ __forceinline__ void mma_bf16(float (&d)[4], const uint32_t (&a)[4], const uint32_t (&b)[2]) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, "
      "{%8,%9}, {%0,%1,%2,%3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}

__device__ __forceinline__ void ldsm_x4_trans(uint32_t (&r)[4], const void* p) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(smem_addr(p)));
}

// v = hi + lo with hi rounded to TF32; lo is passed as full FP32 bits: a TF32
// MMA reads only the top 19 bits of an operand, so lo enters truncated to
// TF32 (|error| <= 2^-10 |lo| <= 2^-21 |v|) without a second conversion
__device__ __forceinline__ void split_tf32(float v, uint32_t& hi, uint32_t& lo) {
  hi = step32::tf32_round(v);
  lo = __float_as_uint(v - __uint_as_float(hi));
}

// The cluster's CTAs staged their partials (column block cb: G block, 3
// d-sums, loss) at the same shared-memory offset `stage`; CTA r sums a 1/CLP
// slice over the cluster through DSMEM and writes it out.  Column block cb
// writes loss slot cb of the 4 spare floats of the partial row (block 0 also
// clears the unused slots).
template <int KP, int IB, int NBC, int MODE>
__device__ __forceinline__ void partial_cluster_sum(const StpmPartialArgs& a, float* stage, int cb,
                                                    int i0) {
  cg::cluster_group cluster = cg::this_cluster();
  const int crank = (int)cluster.block_rank(), tid = threadIdx.x, NT = blockDim.x, k = a.k;
  constexpr int CLP = kPartialCluster;
  constexpr int STAGE = KP * IB + 3 * IB + 1;
  // 16-byte slices: the staging areas have room past STAGE (the tile region
  // they overlay is larger), and KP, IB are multiples of 4, so the 4 entries
  // of a vector share their row i of G
  constexpr int STAGE4 = (STAGE + 3) / 4;
  static_assert(KP % 4 == 0 && IB % 4 == 0, "16-byte slices");
  cluster.sync();
  float* gp = a.gpart + (int64_t)(blockIdx.x / CLP) * a.part_stride;
  const int slice4 = (STAGE4 + CLP - 1) / CLP;
  auto put = [&](int e, float v) {
    if (e < KP * IB) {
      const int i = i0 + e / KP, j = e % KP;
      if (i < k && j < k && MODE != kModeLoss) gp[(int64_t)i * k + j] = v;
    } else if (e < KP * IB + 3 * IB) {
      const int q = (e - KP * IB) / IB, i = i0 + (e - KP * IB) % IB;
      if (i < k) gp[(int64_t)k * k + q * k + i] = v;
    } else if (e < STAGE) {
      gp[(int64_t)k * k + 3 * k + cb] = v;
    }
  };
  for (int e4 = crank * slice4 + tid; e4 < min(STAGE4, (crank + 1) * slice4); e4 += NT) {
    float4 r[CLP];
#pragma unroll
    for (int q = 0; q < CLP; ++q) r[q] = reinterpret_cast<const float4*>(cluster.map_shared_rank(stage, q))[e4];
    float4 v = r[0];
#pragma unroll
    for (int q = 1; q < CLP; ++q) {
      v.x += r[q].x;
      v.y += r[q].y;
      v.z += r[q].z;
      v.w += r[q].w;
    }
    put(4 * e4, v.x);
    put(4 * e4 + 1, v.y);
    put(4 * e4 + 2, v.z);
    put(4 * e4 + 3, v.w);
  }
  if (cb == 0 && crank == 0 && tid < 4 && tid >= NBC) gp[(int64_t)k * k + 3 * k + tid] = 0.f;
  cluster.sync();  // keep shared memory alive until every remote read is done
}

// The tensor-core contraction of one CTA (plain mode, FP32): stages this
// CTA's partial -- G column-major (stage[i KP + j]), the d-sums d1 (then
// d2 = d3 = 0) and a zero loss -- at `stage`, as the CUDA-core form does.
template <int KP>
__device__ __forceinline__ void contract_tc(const StpmPartialArgs& a, int nblocks,
                                            unsigned char* smraw, float* stage) {
  using C = ContractTc<KP>;
  constexpr int TM = C::TM, NT = 512, NQ = KP / 4;
  __shared__ __align__(8) uint64_t bars[3];  // Z products done | G products done | Phi image
  __shared__ uint32_t tmem_slot;
  unsigned char* base = smraw + ((1024 - (tc::sm_addr(smraw) & 1023)) & 1023);
  float* mv = reinterpret_cast<float*>(base + C::REGION);  // m1 | m2
  float* dsum = mv + 2 * KP;                               // d1 per node group (4 x KP)
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int k = a.k;
  if (warp == 0) tc::tmem_alloc(&tmem_slot, C::TMEM_COLS);
  if (tid == 0) {
    tc::mbar_init(&bars[0], 1);
    tc::mbar_init(&bars[1], 1);
    tc::mbar_init(&bars[2], 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  // Staging tasks are laid out so that the 8 lanes of a quarter-warp write
  // one whole core matrix (8 consecutive rows x 16 bytes, 128 contiguous
  // bytes: no bank conflicts), and the global loads of a warp still cover
  // whole 32-byte sectors.  y1, y2 (row x, 16-byte chunks along j): lane l
  // takes row 8 g + (l & 7) and chunk 4 h + (l >> 3) of warp-task (g, h); y3
  // (transposed: row j, 4 nodes along K): lane = j, four scalar loads.
  // A tile's loads go to registers one tile ahead.
  constexpr int T12 = 2 * TM * NQ, S12 = (T12 + NT - 1) / NT;
  constexpr int T3 = KP * (TM / 4), S3 = (T3 + NT - 1) / NT;
  static_assert(NQ % 4 == 0 && TM % 8 == 0, "warp-task shape");
  uint4 p12[S12];
  float p3[S3][4];
  auto task12 = [&](int e, int& q, int& x, int& jq) {
    const int l = e & 31, w = e >> 5;
    x = 8 * (w % (TM / 8)) + (l & 7);
    jq = 4 * ((w / (TM / 8)) % (NQ / 4)) + (l >> 3);
    q = w / ((TM / 8) * (NQ / 4));
  };
  auto tile_nodes = [&](int64_t tile, int64_t& x0) {
    x0 = a.begin + tile * TM;
    const int64_t left = a.begin + a.count - x0;
    return left < TM ? (int)left : TM;
  };
  auto load_tile = [&](int64_t tile) {
    int64_t x0;
    const int nv = tile_nodes(tile, x0);
#pragma unroll
    for (int s = 0; s < S12; ++s) {
      const int e = tid + NT * s;
      p12[s] = make_uint4(0u, 0u, 0u, 0u);
      if (e < T12) {
        int q, x, jq;
        task12(e, q, x, jq);
        const float* Y = q == 0 ? a.y1 : a.y2;
        if (x < nv && 4 * jq < a.ldy)
          p12[s] = __ldg(reinterpret_cast<const uint4*>(Y + (x0 + x) * a.ldy + 4 * jq));
      }
    }
#pragma unroll
    for (int s = 0; s < S3; ++s) {
      const int e = tid + NT * s, j = e % KP, xq = e / KP;
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int x = 4 * xq + u;
        p3[s][u] = (e < T3 && x < nv && j < a.ldy) ? __ldg(a.y3 + (x0 + x) * a.ldy + j) : 0.f;
      }
    }
  };
  auto store_tile = [&]() {
#pragma unroll
    for (int s = 0; s < S12; ++s) {
      const int e = tid + NT * s;
      if (e < T12) {
        int q, x, jq;
        task12(e, q, x, jq);
        const float v[4] = {__uint_as_float(p12[s].x), __uint_as_float(p12[s].y),
                            __uint_as_float(p12[s].z), __uint_as_float(p12[s].w)};
        uint4 h;
        float4 l;
        tc::split4(v, h, l);
        const uint32_t off = tc::kmajor_off(x, 4 * jq, C::SBOJ);
        *reinterpret_cast<uint4*>(base + (q == 0 ? C::Y1H : C::Y2H) + off) = h;
        *reinterpret_cast<float4*>(base + (q == 0 ? C::Y1L : C::Y2L) + off) = l;
      }
    }
#pragma unroll
    for (int s = 0; s < S3; ++s) {
      const int e = tid + NT * s, j = e % KP, xq = e / KP;
      if (e < T3) {
        uint4 h;
        float4 l;
        tc::split4(p3[s], h, l);
        const uint32_t off = tc::kmajor_off(j, 4 * xq, C::SBOX);
        *reinterpret_cast<uint4*>(base + C::Y3H + off) = h;
        *reinterpret_cast<float4*>(base + C::Y3L + off) = l;
      }
    }
  };
  const int64_t ntiles = ceil_div_dev(a.count, TM);
  float* mus = mv;  // mu_1 | mu_2 staged in mv
  // Launched as a programmatic dependent of the step that writes Phi: all
  // that does not read Phi -- TMEM, barriers, mu and the whole first node
  // tile -- is done before the wait and overlaps that kernel's tail.
  const bool first_staged = (int64_t)blockIdx.x < ntiles;
  if (first_staged) load_tile(blockIdx.x);
  for (int e = tid; e < 2 * KP; e += NT) {
    const float* mu = e < KP ? a.mu1 : a.mu2;
    const int j = e % KP;
    mus[e] = (mu && j < k) ? mu[j] : 0.f;
  }
  for (int e = tid; e < 4 * KP; e += NT) dsum[e] = 0.f;
  if (first_staged) store_tile();
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  // Phi hi / lo (operand row i = column i of Phi, contiguous in j), all of
  // a thread's loads issued together; the partial dot products of its
  // chunks with mu_1, mu_2 go to part[] (in the C area, free until the first
  // epilogue) and are summed per column in a fixed order: m_q = Phi^T mu_q
  constexpr int PT = (KP * NQ + NT - 1) / NT;
  auto task_phi = [&](int e, int& i, int& jq) {  // 8 rows i x 4 chunks per warp
    const int l = e & 31, w = e >> 5;
    i = 8 * (w % (KP / 8)) + (l & 7);
    jq = 4 * (w / (KP / 8)) + (l >> 3);
  };
  float* part = reinterpret_cast<float*>(base + C::CH);  // [q][i][jq]
  static_assert(2 * KP * NQ * 4 <= 2 * C::TSZ, "partials fit the C area");
  bool img_timed_out = false;
  // part -> m_q (mv and mus share storage)
  auto finish_means = [&]() {
    __syncthreads();
    float m = 0.f;
    if (tid < 2 * KP) {
      const float* pp = part + (tid / KP) * KP * NQ + (tid % KP) * NQ;
#pragma unroll 4
      for (int jq = 0; jq < NQ; ++jq) m += pp[jq];
    }
    __syncthreads();  // every read of mus done
    if (tid < 2 * KP) mv[tid] = m;
    __syncthreads();
  };
  bool need_means = !C::CHAIN && a.phi_img != nullptr;
  if (a.phi_img) {
    // the previous step kernel wrote Phi's operand image: bulk copies of the
    // hi | lo image (in 4 pieces); Phi^T mu_q is formed behind the first
    // tile's Z products
    __syncthreads();  // every thread past its first-tile stores (the barrier init is ordered)
    if (tid == 0) {
      constexpr uint32_t bytes = 2 * C::PSZ, piece = bytes / 4;
      static_assert(bytes % 64 == 0, "16-byte pieces");
      mbar_arrive_expect_tx(&bars[2], bytes);
#pragma unroll
      for (int q = 0; q < 4; ++q)
        bulk_copy_g2s(base + C::PH + q * piece, static_cast<const unsigned char*>(a.phi_img) + q * piece,
                      piece, &bars[2]);
    }
    if constexpr (C::CHAIN) {
      const float* mimg =
          reinterpret_cast<const float*>(static_cast<const unsigned char*>(a.phi_img) + 2 * C::PSZ);
      float m = 0.f;
      if (tid < 2 * KP) m = mimg[tid];
      __syncthreads();  // every read of mus done (mv and mus share storage)
      if (tid < 2 * KP) mv[tid] = m;
    }
    if (!tc::mbar_wait(&bars[2], 0u, tc::wait_limit_or_default(a.wait_limit))) img_timed_out = true;
  } else {
    float v[PT][4];
#pragma unroll
    for (int t = 0; t < PT; ++t) {
      int i, jq;
      task_phi(tid + NT * t, i, jq);
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int j = 4 * jq + u;
        v[t][u] = (tid + NT * t < KP * NQ && i < k && j < k) ? __ldg(a.phi + (int64_t)i * k + j) : 0.f;
      }
    }
    __syncthreads();  // mus staged
#pragma unroll
    for (int t = 0; t < PT; ++t) {
      const int e = tid + NT * t;
      int i, jq;
      task_phi(e, i, jq);
      if (e < KP * NQ) {
        uint4 h;
        float4 l;
        tc::split4(v[t], h, l);
        const uint32_t off = tc::kmajor_off(i, 4 * jq, C::SBOJ);
        *reinterpret_cast<uint4*>(base + C::PH + off) = h;
        *reinterpret_cast<float4*>(base + C::PL + off) = l;
        float p1 = 0.f, p2 = 0.f;
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          p1 = fmaf(v[t][u], mus[4 * jq + u], p1);
          p2 = fmaf(v[t][u], mus[KP + 4 * jq + u], p2);
        }
        part[i * NQ + jq] = p1;
        part[KP * NQ + i * NQ + jq] = p2;
      }
    }
    finish_means();
  }

  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tmem = tmem_slot, sbase = tc::sm_addr(base);
  const float cc0 = a.c0, cc2 = a.c2;
  uint32_t ph_z = 0u, ph_g = 0u;
  bool g_pending = false, timed_out = img_timed_out, any = false;
  int64_t tile = blockIdx.x;
  for (; tile < ntiles; tile += nblocks) {
    // the G products of the previous tile read y3 and C
    if (g_pending) {
      if (!tc::mbar_wait(&bars[1], ph_g, tc::wait_limit_or_default(a.wait_limit))) timed_out = true;
      ph_g ^= 1u;
      g_pending = false;
    }
    if (__syncthreads_or(timed_out)) {
      timed_out = true;
      break;
    }
    if (tile != (int64_t)blockIdx.x) store_tile();  // the first tile was staged before the wait
    int64_t x0;
    const int nv = tile_nodes(tile, x0);
    if (tile + nblocks < ntiles) load_tile(tile + nblocks);  // in flight during the MMAs
    tc::fence_async_smem();
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    if (tid == 0) {
      // K-step ks starts 256 B further: + 16 in the descriptor's address field
      constexpr uint32_t iz = tc::tf32_idesc(128, 2 * TM);
      const uint64_t dph = tc::smem_desc(sbase + C::PH, 128, C::SBOJ);
      const uint64_t dpl = tc::smem_desc(sbase + C::PL, 128, C::SBOJ);
      const uint64_t dyh = tc::smem_desc(sbase + C::Y1H, 128, C::SBOJ);
      const uint64_t dyl = tc::smem_desc(sbase + C::Y1L, 128, C::SBOJ);
      // the small products, then the first share of the large ones; the other
      // shares in accumulators of their own (added in the epilogue)
#pragma unroll
      for (int ks = 0; ks < KP / 8; ++ks) {
        const uint64_t ko = 16u * ks;
        if (C::CHAIN) tc::mma_tf32(tmem, dph + ko, dyh + ko, iz, ks > 0 ? 1u : 0u);
        tc::mma_tf32(tmem, dph + ko, dyl + ko, iz, C::CHAIN || ks > 0 ? 1u : 0u);
        tc::mma_tf32(tmem, dpl + ko, dyh + ko, iz, 1u);
      }
      constexpr int SHARE = (KP / 8 + C::NZX) / (C::NZX + 1);
#pragma unroll
      for (int ks = 0; ks < (C::CHAIN ? 0 : KP / 8); ++ks) {
        const int part = ks / SHARE;
        tc::mma_tf32(tmem + (part > 0 ? C::ZX + 2 * TM * (part - 1) : 0), dph + 16u * ks,
                     dyh + 16u * ks, iz, part > 0 && ks % SHARE == 0 ? 0u : 1u);
      }
      tc::commit(&bars[0]);
    }
    if (need_means) {  // from the image in shared memory (hi + lo = Phi), behind the MMAs
      need_means = false;
#pragma unroll
      for (int t = 0; t < PT; ++t) {
        const int e = tid + NT * t;
        int i, jq;
        task_phi(e, i, jq);
        if (e < KP * NQ) {
          const uint32_t off = tc::kmajor_off(i, 4 * jq, C::SBOJ);
          const float4 h = *reinterpret_cast<const float4*>(base + C::PH + off);
          const float4 l = *reinterpret_cast<const float4*>(base + C::PL + off);
          const float v[4] = {h.x + l.x, h.y + l.y, h.z + l.z, h.w + l.w};
          float p1 = 0.f, p2 = 0.f;
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            p1 = fmaf(v[u], mus[4 * jq + u], p1);
            p2 = fmaf(v[u], mus[KP + 4 * jq + u], p2);
          }
          part[i * NQ + jq] = p1;
          part[KP * NQ + i * NQ + jq] = p2;
        }
      }
      finish_means();
    }
    if (!tc::mbar_wait(&bars[0], ph_z, tc::wait_limit_or_default(a.wait_limit))) timed_out = true;
    ph_z ^= 1u;
    tc::fence_after_sync();
    {
      // warp w: TMEM lanes (rows i) 32 (w % 4) .., nodes 8 (w / 4) .. + 7
      const int sub = warp & 3, xg = warp >> 2, i = 32 * sub + lane;
      const uint32_t lb = tmem + ((uint32_t)(32 * sub) << 16) + (uint32_t)(8 * xg);
      float z1[8], z2[8];
      tc::tmem_ld8(lb, z1);
      tc::tmem_ld8(lb + TM, z2);
#pragma unroll
      for (int part = 0; part < C::NZX; ++part) {
        float x1[8], x2[8];
        tc::tmem_ld8(lb + C::ZX + 2 * TM * part, x1);
        tc::tmem_ld8(lb + C::ZX + 2 * TM * part + TM, x2);
#pragma unroll
        for (int u = 0; u < 8; ++u) z1[u] += x1[u], z2[u] += x2[u];
      }
      if (i < KP) {
        const float m1 = mv[i], m2 = mv[KP + i];
        float cv[8], d = 0.f;
#pragma unroll
        for (int u = 0; u < 8; ++u) {
          const bool valid = 8 * xg + u < nv && i < k;
          cv[u] = valid ? cc0 * z1[u] * z2[u] + cc2 * (z1[u] * m2 + m1 * z2[u]) : 0.f;
          if (valid) d = fmaf(z1[u], z2[u], d);
        }
#pragma unroll
        for (int h2 = 0; h2 < 2; ++h2) {
          const float v[4] = {cv[4 * h2], cv[4 * h2 + 1], cv[4 * h2 + 2], cv[4 * h2 + 3]};
          uint4 h;
          float4 l;
          tc::split4(v, h, l);
          const uint32_t off = tc::kmajor_off(i, 8 * xg + 4 * h2, C::SBOX);
          *reinterpret_cast<uint4*>(base + C::CH + off) = h;
          *reinterpret_cast<float4*>(base + C::CLO + off) = l;
        }
        dsum[xg * KP + i] += d;
      }
    }
    tc::fence_async_smem();
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    if (tid == 0) {
      constexpr uint32_t ig = tc::tf32_idesc(128, KP);
      const uint32_t d = tmem + (uint32_t)(2 * TM);
      const uint64_t dah = tc::smem_desc(sbase + C::Y3H, 128, C::SBOX);
      const uint64_t dal = tc::smem_desc(sbase + C::Y3L, 128, C::SBOX);
      const uint64_t dbh = tc::smem_desc(sbase + C::CH, 128, C::SBOX);
      const uint64_t dbl = tc::smem_desc(sbase + C::CLO, 128, C::SBOX);
#pragma unroll
      for (int ks = 0; ks < TM / 8; ++ks) {
        const uint64_t ko = 16u * ks;
        const uint32_t acc = (any || ks > 0) ? 1u : 0u, dl = C::CHAIN ? d : d + KP;
        tc::mma_tf32(d, dah + ko, dbh + ko, ig, acc);
        tc::mma_tf32(dl, dah + ko, dbl + ko, ig, C::CHAIN ? 1u : acc);
        tc::mma_tf32(dl, dal + ko, dbh + ko, ig, 1u);
      }
      tc::commit(&bars[1]);
    }
    g_pending = true;
    any = true;
  }
  if (g_pending) {
    if (!tc::mbar_wait(&bars[1], ph_g, tc::wait_limit_or_default(a.wait_limit))) timed_out = true;
    ph_g ^= 1u;
  }
  tc::fence_after_sync();
  const bool ok = !__syncthreads_or(timed_out);
  // the tiles are dead: stage the partial over them (stage <= base)
  {
    const int sub = warp & 3, cg4 = warp >> 2, j = 32 * sub + lane;
    for (int c4 = 0; c4 < NQ; c4 += 4) {
      const int ic = cg4 * NQ + c4;
      float v[4] = {0.f, 0.f, 0.f, 0.f};
      if (ok && any) {
        const uint32_t at = tmem + ((uint32_t)(32 * sub) << 16) + (uint32_t)(2 * TM + ic);
        tc::tmem_ld4(at, v);
        if (!C::CHAIN) {
          float lo[4];
          tc::tmem_ld4(at + KP, lo);
#pragma unroll
          for (int u = 0; u < 4; ++u) v[u] += lo[u];
        }
      }
      if (j < KP)
#pragma unroll
        for (int u = 0; u < 4; ++u) stage[(ic + u) * KP + j] = v[u];
    }
  }
  for (int e = tid; e < 3 * KP + 1; e += NT)
    stage[KP * KP + e] = e < KP ? ((dsum[e] + dsum[KP + e]) + (dsum[2 * KP + e] + dsum[3 * KP + e])) : 0.f;
  if (!ok && tid == 0 && a.flags) atomicOr(a.flags, kFlagTimeout);
  tc::fence_before_sync();
  __syncthreads();
  if (warp == 0) tc::tmem_dealloc(tmem, C::TMEM_COLS);
}

// The BF16 tensor-core adjoint contraction of one CTA: stages this CTA's
// partial (G column-major at stage[i KP + j], the three d-sums, a zero loss)
// at `stage`, as the CUDA-core form does.
template <int KP>
__device__ __forceinline__ void contract_tc_bf(const StpmPartialArgs& a, int nblocks,
                                               unsigned char* smraw, float* stage) {
  using C = ContractTcBf<KP>;
  constexpr int TM = C::TM, NT = 512, NJ = KP / 8;  // 16-byte chunks (8 elements) along j
  __shared__ __align__(8) uint64_t bars[2];  // Z products done | G products done
  __shared__ uint32_t tmem_slot;
  unsigned char* base = smraw + ((1024 - (tc::sm_addr(smraw) & 1023)) & 1023);
  float* mv = reinterpret_cast<float*>(base + C::REGION);  // m1 | m2 | m3
  float* dsum = mv + 3 * KP;                               // [pair][node group][i]
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int k = a.k;
  if (warp == 0) tc::tmem_alloc(&tmem_slot, C::TMEM_COLS);
  if (tid == 0) {
    tc::mbar_init(&bars[0], 1);
    tc::mbar_init(&bars[1], 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  // Node tiles, one tile ahead in registers.  Row form (B of the Z product):
  // task (q, x, chunk) = one 16-byte load of y_q's row x; the 8 lanes of a
  // quarter-warp take 8 consecutive rows, so they write one whole core matrix.
  // Transposed form (A of the G product): task (c, j, node chunk) = 8 scalar
  // loads of column j (lanes along j: coalesced) packed into one 16-byte row.
  constexpr int TR = 3 * TM * NJ, SR = (TR + NT - 1) / NT;
  constexpr int TT = 3 * KP * (TM / 8), ST = (TT + NT - 1) / NT;
  uint4 pr[SR], pt[ST];
  auto yh = [&](int q) {
    return static_cast<const unsigned short*>(q == 0 ? a.yh1 : q == 1 ? a.yh2 : a.yh3);
  };
  auto task_row = [&](int e, int& q, int& x, int& jc) {
    const int grp = e >> 3, rest = grp / (TM / 8);
    x = 8 * (grp % (TM / 8)) + (e & 7);
    jc = rest % NJ;
    q = rest / NJ;
  };
  auto tile_nodes = [&](int64_t tile, int64_t& x0) {
    x0 = a.begin + tile * TM;
    const int64_t left = a.begin + a.count - x0;
    return left < TM ? (int)left : TM;
  };
  auto load_tile = [&](int64_t tile) {
    int64_t x0;
    const int nv = tile_nodes(tile, x0);
#pragma unroll
    for (int s = 0; s < SR; ++s) {
      const int e = tid + NT * s;
      pr[s] = make_uint4(0u, 0u, 0u, 0u);
      if (e < TR) {
        int q, x, jc;
        task_row(e, q, x, jc);
        if (x < nv && 8 * jc < a.ldyh)
          pr[s] = __ldg(reinterpret_cast<const uint4*>(yh(q) + (x0 + x) * a.ldyh + 8 * jc));
      }
    }
#pragma unroll
    for (int s = 0; s < ST; ++s) {
      const int e = tid + NT * s, j = e % KP, rest = e / KP, xc = rest % (TM / 8), c = rest / (TM / 8);
      uint32_t w[4] = {0u, 0u, 0u, 0u};
      if (e < TT && j < a.ldyh) {
        const unsigned short* Yc = yh(c);
#pragma unroll
        for (int u = 0; u < 8; ++u) {
          const int x = 8 * xc + u;
          const uint32_t v = x < nv ? (uint32_t)__ldg(Yc + (x0 + x) * a.ldyh + j) : 0u;
          w[u >> 1] |= v << (16 * (u & 1));
        }
      }
      pt[s] = make_uint4(w[0], w[1], w[2], w[3]);
    }
  };
  auto store_tile = [&]() {
#pragma unroll
    for (int s = 0; s < SR; ++s) {
      const int e = tid + NT * s;
      if (e < TR) {
        int q, x, jc;
        task_row(e, q, x, jc);
        *reinterpret_cast<uint4*>(base + C::YB + q * C::TSZ + tc::kmajor16_off(x, 8 * jc, C::SBOJ)) = pr[s];
      }
    }
#pragma unroll
    for (int s = 0; s < ST; ++s) {
      const int e = tid + NT * s, j = e % KP, rest = e / KP, xc = rest % (TM / 8), c = rest / (TM / 8);
      if (e < TT)
        *reinterpret_cast<uint4*>(base + C::YT + c * C::TSZ + tc::kmajor16_off(j, 8 * xc, C::SBOX)) = pt[s];
    }
  };
  const int64_t ntiles = ceil_div_dev(a.count, TM);
  float* mus = mv;  // mu_1 | mu_2 | mu_3 staged in mv
  // everything that does not read Phi happens before the dependency wait
  const bool first_staged = (int64_t)blockIdx.x < ntiles;
  if (first_staged) load_tile(blockIdx.x);
  for (int e = tid; e < 3 * KP; e += NT) {
    const float* mu = e < KP ? a.mu1 : e < 2 * KP ? a.mu2 : a.mu3;
    const int j = e % KP;
    mus[e] = (mu && j < k) ? mu[j] : 0.f;
  }
  for (int e = tid; e < 12 * KP; e += NT) dsum[e] = 0.f;
  if (first_staged) store_tile();
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  // Phi as a BF16 pair (hi = bf16(Phi), lo = bf16(Phi - hi)); the partial dot
  // products of each chunk with mu_1..3 (FP32 Phi) go to part[] in the C
  // area and are summed per column in a fixed order: m_q = Phi^T mu_q
  constexpr int PT = (KP * NJ + NT - 1) / NT;
  float* part = reinterpret_cast<float*>(base + C::CB);  // [q][i][jc]
  static_assert(3 * KP * NJ * 4 <= 3 * C::TSZ, "partials fit the C area");
  {
    float v[PT][8];
#pragma unroll
    for (int t = 0; t < PT; ++t) {
      const int e = tid + NT * t, grp = e >> 3, i = 8 * (grp % (KP / 8)) + (e & 7), jc = grp / (KP / 8);
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        const int j = 8 * jc + u;
        v[t][u] = (e < KP * NJ && i < k && j < k) ? __ldg(a.phi + (int64_t)i * k + j) : 0.f;
      }
    }
    __syncthreads();  // mus staged
#pragma unroll
    for (int t = 0; t < PT; ++t) {
      const int e = tid + NT * t, grp = e >> 3, i = 8 * (grp % (KP / 8)) + (e & 7), jc = grp / (KP / 8);
      if (e < KP * NJ) {
        uint32_t h[4] = {0u, 0u, 0u, 0u}, l[4] = {0u, 0u, 0u, 0u};
        float p1 = 0.f, p2 = 0.f, p3 = 0.f;
#pragma unroll
        for (int u = 0; u < 8; ++u) {
          const __nv_bfloat16 hb = __float2bfloat16_rn(v[t][u]);
          const __nv_bfloat16 lb = __float2bfloat16_rn(v[t][u] - __bfloat162float(hb));
          h[u >> 1] |= (uint32_t)__bfloat16_as_ushort(hb) << (16 * (u & 1));
          l[u >> 1] |= (uint32_t)__bfloat16_as_ushort(lb) << (16 * (u & 1));
          p1 = fmaf(v[t][u], mus[8 * jc + u], p1);
          p2 = fmaf(v[t][u], mus[KP + 8 * jc + u], p2);
          p3 = fmaf(v[t][u], mus[2 * KP + 8 * jc + u], p3);
        }
        const uint32_t off = tc::kmajor16_off(i, 8 * jc, C::SBOJ);
        *reinterpret_cast<uint4*>(base + C::PH + off) = make_uint4(h[0], h[1], h[2], h[3]);
        *reinterpret_cast<uint4*>(base + C::PL + off) = make_uint4(l[0], l[1], l[2], l[3]);
        part[i * NJ + jc] = p1;
        part[KP * NJ + i * NJ + jc] = p2;
        part[2 * KP * NJ + i * NJ + jc] = p3;
      }
    }
    __syncthreads();
    float m = 0.f;
    if (tid < 3 * KP) {
      const float* pp = part + (tid / KP) * KP * NJ + (tid % KP) * NJ;
#pragma unroll 2
      for (int jc = 0; jc < NJ; ++jc) m += pp[jc];
    }
    __syncthreads();  // every read of mus done
    if (tid < 3 * KP) mv[tid] = m;
  }
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tmem = tmem_slot, sbase = tc::sm_addr(base);
  const float cc0 = a.c0, cc2 = a.c2;
  uint32_t ph_z = 0u, ph_g = 0u;
  bool g_pending = false, timed_out = false, any = false;
  for (int64_t tile = blockIdx.x; tile < ntiles; tile += nblocks) {
    if (g_pending) {  // the G products of the previous tile read y^T and C
      if (!tc::mbar_wait(&bars[1], ph_g, tc::wait_limit_or_default(a.wait_limit))) timed_out = true;
      ph_g ^= 1u;
      g_pending = false;
    }
    if (__syncthreads_or(timed_out)) {
      timed_out = true;
      break;
    }
    if (tile != (int64_t)blockIdx.x) store_tile();
    int64_t x0;
    const int nv = tile_nodes(tile, x0);
    if (tile + nblocks < ntiles) load_tile(tile + nblocks);
    tc::fence_async_smem();
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    if (tid == 0) {
      constexpr uint32_t iz = tc::bf16_idesc(128, 3 * TM);
      const uint64_t dph = tc::smem_desc(sbase + C::PH, 128, C::SBOJ);
      const uint64_t dpl = tc::smem_desc(sbase + C::PL, 128, C::SBOJ);
      const uint64_t dy = tc::smem_desc(sbase + C::YB, 128, C::SBOJ);
#pragma unroll
      for (int ks = 0; ks < KP / 16; ++ks) {
        const uint64_t ko = 16u * ks;  // 256 bytes: two core matrices along K
        tc::mma_bf16(tmem, dph + ko, dy + ko, iz, ks > 0 ? 1u : 0u);
        tc::mma_bf16(tmem, dpl + ko, dy + ko, iz, 1u);
      }
      tc::commit(&bars[0]);
    }
    if (!tc::mbar_wait(&bars[0], ph_z, tc::wait_limit_or_default(a.wait_limit))) timed_out = true;
    ph_z ^= 1u;
    tc::fence_after_sync();
    {
      // warp w: TMEM lanes (rows i) 32 (w % 4) .., nodes 16 (w / 4) .. + 15
      const int sub = warp & 3, xg = warp >> 2, i = 32 * sub + lane;
      const uint32_t lb = tmem + ((uint32_t)(32 * sub) << 16) + (uint32_t)(16 * xg);
      const float m1 = i < KP ? mv[i] : 0.f, m2 = i < KP ? mv[KP + i] : 0.f,
                  m3 = i < KP ? mv[2 * KP + i] : 0.f;
      float d0 = 0.f, d1 = 0.f, d2 = 0.f;
#pragma unroll
      for (int h2 = 0; h2 < 2; ++h2) {  // 8 nodes at a time (warp-wide TMEM loads)
        float z1[8], z2[8], z3[8];
        tc::tmem_ld8(lb + 8 * h2, z1);
        tc::tmem_ld8(lb + TM + 8 * h2, z2);
        tc::tmem_ld8(lb + 2 * TM + 8 * h2, z3);
        if (i < KP) {
          uint32_t w0[4] = {0u, 0u, 0u, 0u}, w1[4] = {0u, 0u, 0u, 0u}, w2[4] = {0u, 0u, 0u, 0u};
#pragma unroll
          for (int u = 0; u < 8; ++u) {
            const bool valid = 16 * xg + 8 * h2 + u < nv && i < k;
            const float a1 = z1[u], a2 = z2[u], a3 = z3[u];
            const float v0 = valid ? cc0 * a2 * a3 + cc2 * (a2 * m3 + m2 * a3) : 0.f;
            const float v1 = valid ? cc0 * a1 * a3 + cc2 * (a1 * m3 + m1 * a3) : 0.f;
            const float v2 = valid ? cc0 * a1 * a2 + cc2 * (a1 * m2 + m1 * a2) : 0.f;
            if (valid) {
              d0 = fmaf(a2, a3, d0);
              d1 = fmaf(a1, a3, d1);
              d2 = fmaf(a1, a2, d2);
            }
            const int sh = 16 * (u & 1);
            w0[u >> 1] |= (uint32_t)__bfloat16_as_ushort(__float2bfloat16_rn(v0)) << sh;
            w1[u >> 1] |= (uint32_t)__bfloat16_as_ushort(__float2bfloat16_rn(v1)) << sh;
            w2[u >> 1] |= (uint32_t)__bfloat16_as_ushort(__float2bfloat16_rn(v2)) << sh;
          }
          const uint32_t off = tc::kmajor16_off(i, 16 * xg + 8 * h2, C::SBOX);
          *reinterpret_cast<uint4*>(base + C::CB + off) = make_uint4(w0[0], w0[1], w0[2], w0[3]);
          *reinterpret_cast<uint4*>(base + C::CB + C::TSZ + off) = make_uint4(w1[0], w1[1], w1[2], w1[3]);
          *reinterpret_cast<uint4*>(base + C::CB + 2 * C::TSZ + off) = make_uint4(w2[0], w2[1], w2[2], w2[3]);
        }
      }
      if (i < KP) {
        dsum[(0 * 4 + xg) * KP + i] += d0;
        dsum[(1 * 4 + xg) * KP + i] += d1;
        dsum[(2 * 4 + xg) * KP + i] += d2;
      }
    }
    tc::fence_async_smem();
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    if (tid == 0) {
      constexpr uint32_t ig = tc::bf16_idesc(128, KP);
      const uint32_t d = tmem + (uint32_t)(3 * TM);
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        const uint64_t da = tc::smem_desc(sbase + C::YT + c * C::TSZ, 128, C::SBOX);
        const uint64_t db = tc::smem_desc(sbase + C::CB + c * C::TSZ, 128, C::SBOX);
#pragma unroll
        for (int ks = 0; ks < TM / 16; ++ks)
          tc::mma_bf16(d, da + 16u * ks, db + 16u * ks, ig, (any || c > 0 || ks > 0) ? 1u : 0u);
      }
      tc::commit(&bars[1]);
    }
    g_pending = true;
    any = true;
  }
  if (g_pending) {
    if (!tc::mbar_wait(&bars[1], ph_g, tc::wait_limit_or_default(a.wait_limit))) timed_out = true;
    ph_g ^= 1u;
  }
  tc::fence_after_sync();
  const bool ok = !__syncthreads_or(timed_out);
  {
    const int sub = warp & 3, cg4 = warp >> 2, j = 32 * sub + lane;
    constexpr int NQ = KP / 4;
    for (int c4 = 0; c4 < NQ; c4 += 4) {
      const int ic = cg4 * NQ + c4;
      float v[4] = {0.f, 0.f, 0.f, 0.f};
      if (ok && any)
        tc::tmem_ld4(tmem + ((uint32_t)(32 * sub) << 16) + (uint32_t)(3 * TM + ic), v);
      if (j < KP)
#pragma unroll
        for (int u = 0; u < 4; ++u) stage[(ic + u) * KP + j] = v[u];
    }
  }
  for (int e = tid; e < 3 * KP + 1; e += NT) {
    float v = 0.f;
    if (e < 3 * KP) {
      const float* ds = dsum + (e / KP) * 4 * KP + e % KP;
      v = (ds[0] + ds[KP]) + (ds[2 * KP] + ds[3 * KP]);
    }
    stage[KP * KP + e] = v;
  }
  if (!ok && tid == 0 && a.flags) atomicOr(a.flags, kFlagTimeout);
  tc::fence_before_sync();
  __syncthreads();
  if (warp == 0) tc::tmem_dealloc(tmem, C::TMEM_COLS);
}

// FP32 contraction on the CUDA cores, for the forms that do not fit the
// tensor-core one (plain above KP = 112, adjoint and loss).  Register-tiled
// FFMA from shared memory, K (= j, then nodes) in 16-byte words: 4 i x XT nodes
// x NZ per thread for Z (4 + XT NZ words per 16 XT NZ products), 8 j x GI i for
// G, accumulated in registers over the CTA's tiles.  It is bound by the shared
// memory's bandwidth.  The mma.sync form in 3xTF32 that it replaces issues one
// m16n8k8 per 22 cycles and SM: the adjoint form of 8,192 nodes at k = 100 took
// 94 us (69 us here), a minibatch step of 8,192 nodes at k = 200 295 us (250 us).
// And the FFMA sums round to nearest, where the tensor cores' accumulators
// truncate: the loss's gradient was 1.9e-6 off, 0.07e-6 here.
template <int KP, int MODE>
__device__ __forceinline__ void contract_ffma(const StpmPartialArgs& a, int nblocks,
                                              unsigned char* smraw) {
  using Cfg = Contract<KP, MODE, false>;
  constexpr int TM = Cfg::TM, NZ = Cfg::NZ, NC = Cfg::NC, PLD = Cfg::PLD, LDY = Cfg::LDY,
                LDC = Cfg::LDC, IB = Cfg::IB, NT = Cfg::NT, XT = Cfg::XT, GI = Cfg::GI;
  // programmatic serialization: wait for the previous kernel (the step that
  // wrote Phi), then let the next one be scheduled early
  const int cb = (Cfg::NBC > 1) ? (int)blockIdx.y : 0, i0 = cb * IB;
  float* Phis = reinterpret_cast<float*>(smraw);  // Phis[ii PLD + j] = Phi_j,i0+ii
  float* Ys = Phis + IB * PLD;                    // 3 node-major tiles: Ys[q TM LDY + x LDY + j]
  float* CT = Ys + 3 * TM * LDY;                  // CT[c IB LDC + ii LDC + x]
  float* mv = reinterpret_cast<float*>(smraw + Cfg::region);  // m1 | m2 | m3 (IB each)
  float* tred = mv + 3 * IB;
  float* mus = tred + Cfg::NW;  // mu1..3 (3 KP), then d-sums
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, k = a.k;
#pragma unroll 1
  for (int e = tid; e < 3 * KP; e += NT) {
    const int which = e / KP, j = e % KP;
    const float* mu = which == 0 ? a.mu1 : which == 1 ? a.mu2 : a.mu3;
    mus[e] = (mu && j < k) ? mu[j] : 0.f;
  }
  const int64_t ntiles = ceil_div_dev(a.count, TM);
  auto load_tile = [&](int64_t tile) {  // 16-byte words; columns past the stored row are zero
    const int64_t x0 = a.begin + tile * TM;
    const int64_t left = a.begin + a.count - x0;
    const int nvalid = left < TM ? (int)left : TM;
    constexpr int NCH = KP / 4, N = 3 * TM * NCH, B = 4;
#pragma unroll 1
    for (int e0 = tid; e0 < N; e0 += NT * B) {
      float4 v[B];
#pragma unroll
      for (int u = 0; u < B; ++u) {
        const int e = e0 + NT * u, q = e / (TM * NCH), rem = e % (TM * NCH), xx = rem / NCH,
                  c = rem % NCH;
        v[u] = make_float4(0.f, 0.f, 0.f, 0.f);
        const float* Y = q == 0 ? a.y1 : q == 1 ? a.y2 : a.y3;
        if (e < N && xx < nvalid && 4 * c < a.ldy)
          v[u] = __ldg(reinterpret_cast<const float4*>(Y + (x0 + xx) * a.ldy + 4 * c));
      }
#pragma unroll
      for (int u = 0; u < B; ++u) {
        const int e = e0 + NT * u, q = e / (TM * NCH), rem = e % (TM * NCH), xx = rem / NCH,
                  c = rem % NCH;
        if (e < N) *reinterpret_cast<float4*>(Ys + q * TM * LDY + xx * LDY + 4 * c) = v[u];
      }
    }
    return nvalid;
  };
  int nvalid = 0;
  if ((int64_t)blockIdx.x < ntiles) nvalid = load_tile(blockIdx.x);  // (y only: before the wait)
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  // Phi: loads issued in batches of 8 per thread so that their latencies overlap
  {
    constexpr int N = IB * PLD, B = 8;
#pragma unroll 1
    for (int e0 = tid; e0 < N; e0 += NT * B) {
      float v[B];
#pragma unroll
      for (int u = 0; u < B; ++u) {
        const int e = e0 + NT * u, i = i0 + e / PLD, j = e % PLD;
        v[u] = (e < N && i < k && j < k) ? __ldg(a.phi + (int64_t)i * k + j) : 0.f;
      }
#pragma unroll
      for (int u = 0; u < B; ++u)
        if (e0 + NT * u < N) Phis[e0 + NT * u] = v[u];
    }
  }
  __syncthreads();
  // m_q = Phi^T mu_q: a column i per 4 lanes
#pragma unroll 1
  for (int e = tid >> 2; e < 3 * IB; e += NT / 4) {
    const float* mu = mus + (e / IB) * KP;
    const float* ph = Phis + (e % IB) * PLD;
    float s = 0.f;
#pragma unroll 4
    for (int j = tid & 3; j < KP; j += 4) s = fmaf(ph[j], mu[j], s);
    s += __shfl_xor_sync(0xffffffffu, s, 1);
    s += __shfl_xor_sync(0xffffffffu, s, 2);
    if ((tid & 3) == 0) mv[e] = s;
  }
  // this thread's Z tile: columns zi + (IB / 4) u, nodes zx .. zx + XT - 1
  const int zi = tid % (IB / 4), zx = (tid / (IB / 4)) * XT;
  const bool zlive = tid < Cfg::ZTH;
  // and G tile: rows 8 gj .. + 7, columns gi + (IB / GI) u
  const int gpart = tid / Cfg::GTH, gt = tid % Cfg::GTH, gj = gt / (IB / GI), gi = gt % (IB / GI);
  const bool glive = gpart < Cfg::GPARTS;
  float gacc[8][GI];
#pragma unroll
  for (int j = 0; j < 8; ++j)
#pragma unroll
    for (int u = 0; u < GI; ++u) gacc[j][u] = 0.f;
  float dl[MODE == kModePlain ? 1 : 3][4] = {};
  float tsum = 0.f;
  const float cc0 = a.c0, cc2 = a.c2;
#pragma unroll 1
  for (int64_t tile = blockIdx.x; tile < ntiles; tile += nblocks) {
    if (tile != (int64_t)blockIdx.x) nvalid = load_tile(tile);
    __syncthreads();
    // ---- Z, C and the d-sums
    if (zlive) {
      float z[NZ][4][XT];
#pragma unroll
      for (int q = 0; q < NZ; ++q)
#pragma unroll
        for (int u = 0; u < 4; ++u)
#pragma unroll
          for (int x = 0; x < XT; ++x) z[q][u][x] = 0.f;
#pragma unroll 2
      for (int j = 0; j < KP; j += 4) {
        float4 p[4];
#pragma unroll
        for (int u = 0; u < 4; ++u)
          p[u] = *reinterpret_cast<const float4*>(Phis + (zi + (IB / 4) * u) * PLD + j);
#pragma unroll
        for (int q = 0; q < NZ; ++q)
#pragma unroll
          for (int x = 0; x < XT; ++x) {
            const float4 y = *reinterpret_cast<const float4*>(Ys + (q * TM + zx + x) * LDY + j);
#pragma unroll
            for (int u = 0; u < 4; ++u)
              z[q][u][x] = fmaf(p[u].x, y.x, fmaf(p[u].y, y.y, fmaf(p[u].z, y.z, fmaf(p[u].w, y.w, z[q][u][x]))));
          }
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int i = zi + (IB / 4) * u;
        const float m1 = mv[i], m2 = mv[IB + i], m3 = mv[2 * IB + i];
#pragma unroll
        for (int x = 0; x < XT; ++x) {
          const bool valid = zx + x < nvalid && i0 + i < k;
          const float z1 = z[0][u][x], z2 = z[1][u][x];
          if (MODE == kModePlain) {
            CT[i * LDC + zx + x] = valid ? cc0 * z1 * z2 + cc2 * (z1 * m2 + m1 * z2) : 0.f;
            if (valid) dl[0][u] = fmaf(z1, z2, dl[0][u]);
          } else {
            const float z3 = z[NZ - 1][u][x];
            if (MODE == kModeAdjoint) {
              CT[i * LDC + zx + x] = valid ? cc0 * z2 * z3 + cc2 * (z2 * m3 + m2 * z3) : 0.f;
              CT[(IB + i) * LDC + zx + x] = valid ? cc0 * z1 * z3 + cc2 * (z1 * m3 + m1 * z3) : 0.f;
              CT[(2 * IB + i) * LDC + zx + x] = valid ? cc0 * z1 * z2 + cc2 * (z1 * m2 + m1 * z2) : 0.f;
            }
            if (valid) {
              dl[0][u] = fmaf(z2, z3, dl[0][u]);
              dl[MODE == kModePlain ? 0 : 1][u] = fmaf(z1, z3, dl[MODE == kModePlain ? 0 : 1][u]);
              dl[MODE == kModePlain ? 0 : 2][u] = fmaf(z1, z2, dl[MODE == kModePlain ? 0 : 2][u]);
              if (MODE == kModeLoss)
                tsum += cc0 * z1 * z2 * z3 + cc2 * (z1 * z2 * m3 + z1 * m2 * z3 + m1 * z2 * z3);
            }
          }
        }
      }
    }
    __syncthreads();
    // ---- G (8 j x GI i per thread) += Yout^T C over this tile's nodes
    if (NC > 0 && glive) {
#pragma unroll
      for (int c = 0; c < NC; ++c) {
        const float* Yo = Ys + (MODE == kModePlain ? 2 : c) * TM * LDY + 8 * gj;
        const float* Cc = CT + c * IB * LDC;
#pragma unroll 2
        for (int x = 4 * gpart; x < TM; x += 4 * Cfg::GPARTS) {
          float4 cv[GI];
#pragma unroll
          for (int u = 0; u < GI; ++u)
            cv[u] = *reinterpret_cast<const float4*>(Cc + (gi + (IB / GI) * u) * LDC + x);
#pragma unroll
          for (int h = 0; h < 4; ++h) {
            float y[8];
            load8(Yo + (x + h) * LDY, y);
#pragma unroll
            for (int u = 0; u < GI; ++u) {
              const float cx = h == 0 ? cv[u].x : h == 1 ? cv[u].y : h == 2 ? cv[u].z : cv[u].w;
#pragma unroll
              for (int j = 0; j < 8; ++j) gacc[j][u] = fmaf(y[j], cx, gacc[j][u]);
            }
          }
        }
      }
    }
    __syncthreads();
  }
  if (MODE == kModeLoss) {
#pragma unroll
    for (int off = 16; off; off >>= 1) tsum += __shfl_xor_sync(0xffffffffu, tsum, off);
    if (lane == 0) tred[warp] = tsum;
  }
  // stage this CTA's partial over the dead tiles for the cluster sum
  // (partial_cluster_sum): G column-major, 3 d-sums, loss
  float* stage = reinterpret_cast<float*>(smraw);
  float* dpart = stage + Cfg::DPART;  // d-sums of the TM / XT node groups
  float* gmore = dpart + (TM / 2) * 3 * IB;  // G of the thread groups past the first
  constexpr int ND = MODE == kModePlain ? 1 : 3;
  if (NC > 0 && glive) {
#pragma unroll
    for (int u = 0; u < GI; ++u) {
      float v[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) v[j] = gacc[j][u];
      store8((gpart ? gmore + (gpart - 1) * KP * IB : stage) + (gi + (IB / GI) * u) * KP + 8 * gj, v);
    }
  }
  if (zlive) {
#pragma unroll
    for (int d = 0; d < ND; ++d)
#pragma unroll
      for (int u = 0; u < 4; ++u)
        dpart[((tid / (IB / 4)) * ND + d) * IB + zi + (IB / 4) * u] = dl[d][u];
  }
  __syncthreads();
#pragma unroll 1
  for (int e = tid; e < 3 * IB; e += NT) {
    float v = 0.f;
    if (e < ND * IB)
      for (int x = 0; x < TM / XT; ++x) v += dpart[x * ND * IB + e];
    stage[KP * IB + e] = v;
  }
  if (Cfg::GPARTS > 1) {
#pragma unroll 1
    for (int e = 4 * tid; e < KP * IB; e += 4 * NT) {
      float4 v = *reinterpret_cast<const float4*>(stage + e);
#pragma unroll
      for (int q = 0; q < Cfg::GPARTS - 1; ++q) {
        const float4 w = *reinterpret_cast<const float4*>(gmore + q * KP * IB + e);
        v.x += w.x;
        v.y += w.y;
        v.z += w.z;
        v.w += w.w;
      }
      *reinterpret_cast<float4*>(stage + e) = v;
    }
  }
  if (tid == 0) {
    float t = 0.f;
    if (MODE == kModeLoss)
      for (int w = 0; w < Cfg::NW; ++w) t += tred[w];
    stage[KP * IB + 3 * IB] = t;
  }
  partial_cluster_sum<KP, IB, Cfg::NBC, MODE>(a, stage, cb, i0);
}

template <int KP, int MODE, bool BF>
__device__ __forceinline__ void contract_body(const StpmPartialArgs& a, int nblocks) {
  using Cfg = Contract<KP, MODE, BF>;
  using T = typename Cfg::T;
  constexpr int TM = Cfg::TM, NZ = Cfg::NZ, NC = Cfg::NC, PLD = Cfg::PLD, LDY = Cfg::LDY,
                LDC = Cfg::LDC;
  constexpr int IB = Cfg::IB;
  static_assert(KP % 16 == 0 && KP <= 256, "KP");
  extern __shared__ __align__(16) unsigned char smraw[];
  if constexpr (Cfg::TC) {  // waits for the previous kernel itself, after its own prologue
    static_assert(Cfg::NT == 512 && Cfg::NBC == 1, "tensor-core contraction launch shape");
    float* stage = reinterpret_cast<float*>(smraw);
    contract_tc<KP>(a, nblocks, smraw, stage);
    partial_cluster_sum<KP, IB, Cfg::NBC, MODE>(a, stage, 0, 0);
    return;
  } else if constexpr (Cfg::TCBF) {  // likewise
    static_assert(Cfg::NT == 512 && Cfg::NBC == 1, "tensor-core contraction launch shape");
    float* stage = reinterpret_cast<float*>(smraw);
    contract_tc_bf<KP>(a, nblocks, smraw, stage);
    partial_cluster_sum<KP, IB, Cfg::NBC, MODE>(a, stage, 0, 0);
    return;
  } else if constexpr (Cfg::FFMA) {
    contract_ffma<KP, MODE>(a, nblocks, smraw);
    return;
  }
  if constexpr (BF || Cfg::MMA32) {
  // programmatic serialization: wait for the previous kernel (the step that
  // wrote Phi), then let the next one be scheduled early
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  // this CTA's columns of Phi: i0 + ii, ii < IB (i local below)
  const int cb = (Cfg::NBC > 1) ? (int)blockIdx.y : 0, i0 = cb * IB;
  T* Phis = reinterpret_cast<T*>(smraw);  // Phis[ii PLD + j] = Phi_j,i0+ii (column i0+ii of Phi)
  T* Ys = Phis + IB * PLD;                // 3 node-major tiles: Ys[q TM LDY + x LDY + j]
  T* CT = Ys + 3 * TM * LDY;              // NC coefficient tiles, i-major: CT[c IB LDC + ii LDC + x]
  T* PhiLo = CT + NC * IB * LDC;          // BF16 form: Phi - hi(Phi), same layout as Phis
  float* mv = reinterpret_cast<float*>(smraw + Cfg::region);  // m1 | m2 | m3 (IB each)
  constexpr int NW = Cfg::NW, NT = Cfg::NT;
  float* tred = mv + 3 * IB;                                  // NW loss partials
  float* dw = tred + NW;  // per-warp d-sums (3 IB each), summed in a fixed order at the end
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t4 = lane & 3;
  const int k = a.k;

  // Phi: loads issued in batches of 8 per thread so that their latencies overlap
  {
    constexpr int N = IB * PLD, B = 8;
    for (int e0 = tid; e0 < N; e0 += NT * B) {
      float v[B];
#pragma unroll
      for (int u = 0; u < B; ++u) {
        const int e = e0 + NT * u, i = i0 + e / PLD, j = e % PLD;
        v[u] = (e < N && i < k && j < k) ? __ldg(a.phi + (int64_t)i * k + j) : 0.f;
      }
#pragma unroll
      for (int u = 0; u < B; ++u)
        if (e0 + NT * u < N) {
          const T hi = to_elem<T>(v[u]);
          Phis[e0 + NT * u] = hi;
          if (BF) PhiLo[e0 + NT * u] = to_elem<T>(v[u] - to_f32(hi));
        }
    }
  }
  // m_P = Phi^T mu_P with Phi as staged (mu_1..3 staged in dw, which is
  // free until the d-sums start)
  for (int e = tid; e < 3 * KP; e += NT) {
    const int which = e / KP, j = e % KP;
    const float* mu = which == 0 ? a.mu1 : which == 1 ? a.mu2 : a.mu3;
    dw[e] = (mu && j < k) ? mu[j] : 0.f;
  }
  __syncthreads();
  for (int e = tid; e < 3 * IB; e += NT) {
    const float* mu = dw + (e / IB) * KP;
    const T* ph = Phis + (e % IB) * PLD;
    const T* pl = PhiLo + (e % IB) * PLD;
    float s0 = 0.f, s1 = 0.f;
#pragma unroll 4
    for (int j = 0; j < KP; j += 2) {
      float p0 = to_f32(ph[j]), p1 = to_f32(ph[j + 1]);
      if (BF) {
        p0 += to_f32(pl[j]);
        p1 += to_f32(pl[j + 1]);
      }
      s0 = fmaf(p0, mu[j], s0);
      s1 = fmaf(p1, mu[j + 1], s1);
    }
    mv[e] = s0 + s1;
  }
  __syncthreads();
  for (int e = tid; e < NW * 3 * IB; e += NT) dw[e] = 0.f;
  if (tid < NW) tred[tid] = 0.f;
  __syncthreads();

  float gacc[Cfg::GPW][4];
#pragma unroll
  for (int u = 0; u < Cfg::GPW; ++u)
#pragma unroll
    for (int q = 0; q < 4; ++q) gacc[u][q] = 0.f;
  float tsum = 0.f;
  const float cc0 = a.c0, cc2 = a.c2;

  const int64_t ntiles = ceil_div_dev(a.count, TM);
  for (int64_t tile = blockIdx.x; tile < ntiles; tile += nblocks) {
    const int64_t x0 = a.begin + tile * TM;
    const int64_t left = a.begin + a.count - x0;
    const int nvalid = left < TM ? (int)left : TM;
    // node tiles, 16-byte chunks; columns past the stored row are zero
    constexpr int CH = 16 / (int)sizeof(T), NCH = KP / CH;
    {
      constexpr int N = 3 * TM * NCH, B = 4;
      for (int e0 = tid; e0 < N; e0 += NT * B) {
        uint4 v[B];
#pragma unroll
        for (int u = 0; u < B; ++u) {
          const int e = e0 + NT * u;
          const int q = e / (TM * NCH), rem = e % (TM * NCH), xx = rem / NCH, c = rem % NCH;
          v[u] = make_uint4(0u, 0u, 0u, 0u);
          if (e < N) {
            const T* Y = BF ? static_cast<const T*>(q == 0 ? a.yh1 : q == 1 ? a.yh2 : a.yh3)
                            : reinterpret_cast<const T*>(q == 0 ? a.y1 : q == 1 ? a.y2 : a.y3);
            const int64_t ld = BF ? a.ldyh : a.ldy;
            if (xx < nvalid && c * CH < ld)
              v[u] = __ldg(reinterpret_cast<const uint4*>(Y + (x0 + xx) * ld + c * CH));
          }
        }
#pragma unroll
        for (int u = 0; u < B; ++u) {
          const int e = e0 + NT * u;
          if (e >= N) break;
          const int q = e / (TM * NCH), rem = e % (TM * NCH), xx = rem / NCH, c = rem % NCH;
          *reinterpret_cast<uint4*>(Ys + q * TM * LDY + xx * LDY + c * CH) = v[u];
        }
      }
    }
    __syncthreads();

    // ---- Z^T tiles (16 i x 8 x), C and the d-sums
    for (int p = warp; p < Cfg::MTI * Cfg::NTX; p += NW) {
      const int m0 = (p % Cfg::MTI) * 16, n0 = (p / Cfg::MTI) * 8;
      float z[NZ][4];
#pragma unroll
      for (int q = 0; q < NZ; ++q)
#pragma unroll
        for (int r = 0; r < 4; ++r) z[q][r] = 0.f;
      if constexpr (BF) {
#pragma unroll 2
        for (int k0 = 0; k0 < KP; k0 += 16) {
          const T* pa = Phis + m0 * PLD + k0 + 2 * t4;
          const T* pl = PhiLo + m0 * PLD + k0 + 2 * t4;
          const uint32_t af[4] = {ld_b32(pa + g * PLD), ld_b32(pa + (g + 8) * PLD),
                                  ld_b32(pa + g * PLD + 8), ld_b32(pa + (g + 8) * PLD + 8)};
          const uint32_t afl[4] = {ld_b32(pl + g * PLD), ld_b32(pl + (g + 8) * PLD),
                                   ld_b32(pl + g * PLD + 8), ld_b32(pl + (g + 8) * PLD + 8)};
#pragma unroll
          for (int q = 0; q < NZ; ++q) {
            const T* pb = Ys + q * TM * LDY + (n0 + g) * LDY + k0 + 2 * t4;
            const uint32_t bf[2] = {ld_b32(pb), ld_b32(pb + 8)};
            mma_bf16(z[q], af, bf);
            mma_bf16(z[q], afl, bf);
          }
        }
      } else {
        float zc[NZ][4];
#pragma unroll
        for (int q = 0; q < NZ; ++q)
#pragma unroll
          for (int r = 0; r < 4; ++r) zc[q][r] = 0.f;
#pragma unroll 2
        for (int k0 = 0; k0 < KP; k0 += 8) {
          const float* pa = Phis + m0 * PLD + k0 + t4;
          uint32_t ah[4], al[4];
          split_tf32(pa[g * PLD], ah[0], al[0]);
          split_tf32(pa[(g + 8) * PLD], ah[1], al[1]);
          split_tf32(pa[g * PLD + 4], ah[2], al[2]);
          split_tf32(pa[(g + 8) * PLD + 4], ah[3], al[3]);
#pragma unroll
          for (int q = 0; q < NZ; ++q) {
            const float* pb = Ys + q * TM * LDY + (n0 + g) * LDY + k0 + t4;
            uint32_t bh[2], bl[2];
            split_tf32(pb[0], bh[0], bl[0]);
            split_tf32(pb[4], bh[1], bl[1]);
            step32::mma_tf32(z[q], ah, bh);
            step32::mma_tf32(zc[q], ah, bl);
            step32::mma_tf32(zc[q], al, bh);
          }
        }
#pragma unroll
        for (int q = 0; q < NZ; ++q)
#pragma unroll
          for (int r = 0; r < 4; ++r) z[q][r] += zc[q][r];
      }
      // epilogue: fragment r holds (i = m0 + g + 8 (r >> 1), x = n0 + 2 t4 + (r & 1))
      float dl[3][2] = {{0.f, 0.f}, {0.f, 0.f}, {0.f, 0.f}};
      float cv[3][4];
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        const int i = m0 + g + 8 * (r >> 1), x = n0 + 2 * t4 + (r & 1);
        const bool valid = x < nvalid && i0 + i < k;
        const float m1 = mv[i], m2 = mv[IB + i];
        const float z1 = z[0][r], z2 = z[1][r];
        if (MODE == kModePlain) {
          cv[0][r] = valid ? cc0 * z1 * z2 + cc2 * (z1 * m2 + m1 * z2) : 0.f;
          if (valid) dl[0][r >> 1] = fmaf(z1, z2, dl[0][r >> 1]);
        } else {
          const float m3 = mv[2 * IB + i], z3 = z[NZ - 1][r];
          if (MODE == kModeAdjoint) {
            cv[0][r] = valid ? cc0 * z2 * z3 + cc2 * (z2 * m3 + m2 * z3) : 0.f;
            cv[1][r] = valid ? cc0 * z1 * z3 + cc2 * (z1 * m3 + m1 * z3) : 0.f;
            cv[2][r] = valid ? cc0 * z1 * z2 + cc2 * (z1 * m2 + m1 * z2) : 0.f;
          }
          if (valid) {
            dl[0][r >> 1] = fmaf(z2, z3, dl[0][r >> 1]);
            dl[1][r >> 1] = fmaf(z1, z3, dl[1][r >> 1]);
            dl[2][r >> 1] = fmaf(z1, z2, dl[2][r >> 1]);
            if (MODE == kModeLoss)
              tsum += cc0 * z1 * z2 * z3 + cc2 * (z1 * z2 * m3 + z1 * m2 * z3 + m1 * z2 * z3);
          }
        }
      }
#pragma unroll
      for (int c = 0; c < NC; ++c)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          T* dst = CT + c * IB * LDC + (m0 + g + 8 * h) * LDC + n0 + 2 * t4;
          if constexpr (BF)
            *reinterpret_cast<__nv_bfloat162*>(dst) = __floats2bfloat162_rn(cv[c][2 * h], cv[c][2 * h + 1]);
          else
            *reinterpret_cast<float2*>(dst) = make_float2(cv[c][2 * h], cv[c][2 * h + 1]);
        }
#pragma unroll
      for (int qd = 0; qd < 3; ++qd) {
        if (MODE == kModePlain && qd > 0) continue;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          float v = dl[qd][h];
          v += __shfl_xor_sync(0xffffffffu, v, 1);
          v += __shfl_xor_sync(0xffffffffu, v, 2);
          if (t4 == 0) dw[warp * 3 * IB + qd * IB + m0 + g + 8 * h] += v;
        }
      }
    }
    __syncthreads();

    // ---- G (16 j x 8 i tiles) += Yout^T C over this tile's nodes
    if (NC > 0) {
#pragma unroll
      for (int k0 = 0; k0 < TM; k0 += Cfg::KSTEP) {
#pragma unroll
        for (int u = 0; u < Cfg::GPW; ++u) {
          const int tt = warp + NW * u;
          if (tt >= Cfg::GT) continue;
          const int m0 = (tt % Cfg::MTJ) * 16, n0 = (tt / Cfg::MTJ) * 8;
#pragma unroll
          for (int c = 0; c < NC; ++c) {
            const T* Yo = Ys + (MODE == kModePlain ? 2 : c) * TM * LDY;
            const T* Cc = CT + c * IB * LDC;
            if constexpr (BF) {
              uint32_t af[4];
              const int q = lane >> 3, rr = lane & 7;
              ldsm_x4_trans(af, Yo + (k0 + (q >> 1) * 8 + rr) * LDY + m0 + (q & 1) * 8);
              const T* pb = Cc + (n0 + g) * LDC + k0 + 2 * t4;
              const uint32_t bf[2] = {ld_b32(pb), ld_b32(pb + 8)};
              mma_bf16(gacc[u], af, bf);
            } else {
              const float* pa = Yo + (k0 + t4) * LDY + m0 + g;
              uint32_t ah[4], al[4];
              split_tf32(pa[0], ah[0], al[0]);
              split_tf32(pa[8], ah[1], al[1]);
              split_tf32(pa[4 * LDY], ah[2], al[2]);
              split_tf32(pa[4 * LDY + 8], ah[3], al[3]);
              const float* pb = Cc + (n0 + g) * LDC + k0 + t4;
              uint32_t bh[2], bl[2];
              split_tf32(pb[0], bh[0], bl[0]);
              split_tf32(pb[4], bh[1], bl[1]);
              step32::mma_tf32(gacc[u], ah, bh);
              step32::mma_tf32(gacc[u], ah, bl);
              step32::mma_tf32(gacc[u], al, bh);
            }
          }
        }
      }
    }
    __syncthreads();
  }
  if (MODE == kModeLoss) {
#pragma unroll
    for (int off = 16; off; off >>= 1) tsum += __shfl_xor_sync(0xffffffffu, tsum, off);
    if (lane == 0) tred[warp] = tsum;
  }
  // cluster reduction: every CTA stages its partial (this column block of
  // the k x k column-major contraction, its 3 d-sums, loss) in shared memory;
  // CTA r of the cluster sums a 1/CLP slice over the cluster's CTAs through
  // DSMEM and writes it out.  Column block cb writes loss slot cb of the 4
  // spare floats of the partial row (block 0 also clears the unused slots).
  float* stage = reinterpret_cast<float*>(smraw);  // tiles are dead from here on
  if (NC > 0) {
#pragma unroll
    for (int u = 0; u < Cfg::GPW; ++u) {
      const int tt = warp + NW * u;
      if (tt >= Cfg::GT) continue;
      const int m0 = (tt % Cfg::MTJ) * 16, n0 = (tt / Cfg::MTJ) * 8;
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        const int j = m0 + g + 8 * (r >> 1), i = n0 + 2 * t4 + (r & 1);
        stage[i * KP + j] = gacc[u][r];
      }
    }
  }
  __syncthreads();
  for (int e = tid; e < 3 * IB; e += NT) {
    float v = 0.f;
#pragma unroll
    for (int w = 0; w < NW; ++w) v += dw[w * 3 * IB + e];
    stage[KP * IB + e] = v;
  }
  if (tid == 0) {
    float t = 0.f;
    if (MODE == kModeLoss)
      for (int w = 0; w < NW; ++w) t += tred[w];
    stage[KP * IB + 3 * IB] = t;
  }
  partial_cluster_sum<KP, IB, Cfg::NBC, MODE>(a, stage, cb, i0);
  }
}

template <int KP, int MODE, bool BF>
__global__ void __launch_bounds__(Contract<KP, MODE, BF>::NT, Contract<KP, MODE, BF>::CTAS) stpm_contract_kernel(StpmPartialArgs a) {
  contract_body<KP, MODE, BF>(a, gridDim.x);
}

// blockIdx.y selects the graph; its first a.nblocks CTAs (a multiple of the
// cluster size) work, the rest and graphs without nodes this round leave
template <int KP, int MODE, bool BF>
__global__ void __launch_bounds__(Contract<KP, MODE, BF>::NT, Contract<KP, MODE, BF>::CTAS) stpm_contract_batched(const StpmPartialArgs* __restrict__ args) {
  const StpmPartialArgs a = args[blockIdx.y];
  if ((int)blockIdx.x >= a.nblocks || a.count <= 0) return;
  contract_body<KP, MODE, BF>(a, a.nblocks);
}

// lambda_i = phi_i . G_i (tensor value); sign fix so lambda_i > 0
__global__ void tensor_value_kernel(int k, float* __restrict__ phi, const float* __restrict__ G,
                                    double* __restrict__ lambda, double* __restrict__ phi64) {
  const int lane = threadIdx.x & 31;
  const int i = blockIdx.x * (blockDim.x / 32) + threadIdx.x / 32;
  if (i >= k) return;
  double s = 0.0;
  for (int j = lane; j < k; j += 32)
    s += (phi64 ? phi64[(int64_t)i * k + j] : (double)phi[(int64_t)i * k + j]) * G[(int64_t)i * k + j];
#pragma unroll
  for (int off = 16; off; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
  const bool flip = s < 0.0;
  if (lane == 0) lambda[i] = flip ? -s : s;
  if (flip)
    for (int j = lane; j < k; j += 32) {
      phi[(int64_t)i * k + j] = -phi[(int64_t)i * k + j];
      if (phi64) phi64[(int64_t)i * k + j] = -phi64[(int64_t)i * k + j];
    }
}

// launch configuration of the contraction; attr holds 2 attributes
template <int KP, int MODE, bool BF>
cudaError_t partial_config(int grid, cudaStream_t s, cudaLaunchConfig_t* cfg,
                           cudaLaunchAttribute* attr) {
  const size_t smem = Contract<KP, MODE, BF>::smem;
  static bool set = false;
  if (!set) {
    MMSB_CUDA_TRY(cudaFuncSetAttribute(stpm_contract_kernel<KP, MODE, BF>,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    set = true;
  }
  *cfg = cudaLaunchConfig_t{};
  cfg->gridDim = dim3((unsigned)grid, (unsigned)Contract<KP, MODE, BF>::NBC, 1);
  cfg->blockDim = dim3(Contract<KP, MODE, BF>::NT, 1, 1);
  cfg->dynamicSmemBytes = smem;
  cfg->stream = s;
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = kPartialCluster;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;  // see contract_body
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg->attrs = attr;
  cfg->numAttrs = 2;
  return cudaSuccess;
}

template <int KP, int MODE, bool BF>
cudaError_t launch_partial_t(const StpmPartialArgs& a, int grid, cudaStream_t s) {
  cudaLaunchConfig_t cfg;
  cudaLaunchAttribute attr[2];
  MMSB_CUDA_TRY((partial_config<KP, MODE, BF>(grid, s, &cfg, attr)));
  MMSB_CUDA_TRY(cudaLaunchKernelEx(&cfg, stpm_contract_kernel<KP, MODE, BF>, a));
  ++g_launch_count;
  return cudaGetLastError();
}

// CTAs (per column block, a multiple of the cluster size) that run at the
// same time: clusters of 8 pack into the GPCs, so this is less than one per SM
// (120 of 152 for the forms that fill an SM)
template <int KP, int MODE, bool BF>
int partial_resident_t() {
  static const int ctas = []() {
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute attr[2];
    int n = 0;
    cudaError_t e = partial_config<KP, MODE, BF>(kPartialCluster, nullptr, &cfg, attr);
    cfg.numAttrs = 1;
    if (e == cudaSuccess)
      e = cudaOccupancyMaxActiveClusters(&n, stpm_contract_kernel<KP, MODE, BF>, &cfg);
    if (e != cudaSuccess) cudaGetLastError();
    n = e == cudaSuccess ? n / Contract<KP, MODE, BF>::NBC : 0;
    return kPartialCluster * std::max(1, n);
  }();
  return ctas;
}

template <int MODE, bool BF>
int partial_resident_m(int KP) {
  switch (KP) {
    case 32: return partial_resident_t<32, MODE, BF>();
    case 48: return partial_resident_t<48, MODE, BF>();
    case 64: return partial_resident_t<64, MODE, BF>();
    case 80: return partial_resident_t<80, MODE, BF>();
    case 96: return partial_resident_t<96, MODE, BF>();
    case 112: return partial_resident_t<112, MODE, BF>();
    case 128: return partial_resident_t<128, MODE, BF>();
    case 160: return partial_resident_t<160, MODE, BF>();
    default: return partial_resident_t<208, MODE, BF>();
  }
}

template <bool BF>
int partial_resident_p(int mode, int KP) {
  return mode == kModePlain     ? partial_resident_m<kModePlain, BF>(KP)
         : mode == kModeAdjoint ? partial_resident_m<kModeAdjoint, BF>(KP)
                                : partial_resident_m<kModeLoss, BF>(KP);
}

template <int MODE, bool BF>
cudaError_t launch_partial_m(int KP, const StpmPartialArgs& a, int grid, cudaStream_t s) {
  switch (KP) {
    case 32: return launch_partial_t<32, MODE, BF>(a, grid, s);
    case 48: return launch_partial_t<48, MODE, BF>(a, grid, s);
    case 64: return launch_partial_t<64, MODE, BF>(a, grid, s);
    case 80: return launch_partial_t<80, MODE, BF>(a, grid, s);
    case 96: return launch_partial_t<96, MODE, BF>(a, grid, s);
    case 112: return launch_partial_t<112, MODE, BF>(a, grid, s);
    case 128: return launch_partial_t<128, MODE, BF>(a, grid, s);
    case 160: return launch_partial_t<160, MODE, BF>(a, grid, s);
    case 208: return launch_partial_t<208, MODE, BF>(a, grid, s);
    default: return cudaErrorInvalidValue;
  }
}

template <bool BF>
cudaError_t launch_partial_p(int mode, int KP, const StpmPartialArgs& a, int grid, cudaStream_t s) {
  switch (mode) {
    case kModePlain: return launch_partial_m<kModePlain, BF>(KP, a, grid, s);
    case kModeAdjoint: return launch_partial_m<kModeAdjoint, BF>(KP, a, grid, s);
    case kModeLoss: return launch_partial_m<kModeLoss, BF>(KP, a, grid, s);
    default: return cudaErrorInvalidValue;
  }
}

template <int KP, int MODE, bool BF>
cudaError_t launch_partial_batched_t(const StpmPartialArgs* args, int graphs, int grid,
                                     cudaStream_t s) {
  const size_t smem = Contract<KP, MODE, BF>::smem;
  static bool set = false;
  if (!set) {
    MMSB_CUDA_TRY(cudaFuncSetAttribute(stpm_contract_batched<KP, MODE, BF>,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    set = true;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)grid, (unsigned)graphs, 1);
  cfg.blockDim = dim3(Contract<KP, MODE, BF>::NT, 1, 1);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = kPartialCluster;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  MMSB_CUDA_TRY(cudaLaunchKernelEx(&cfg, stpm_contract_batched<KP, MODE, BF>, args));
  ++g_launch_count;
  return cudaGetLastError();
}

template <int MODE, bool BF>
cudaError_t launch_partial_batched_m(int KP, const StpmPartialArgs* args, int graphs, int grid,
                                     cudaStream_t s) {
  switch (KP) {
    case 32: return launch_partial_batched_t<32, MODE, BF>(args, graphs, grid, s);
    case 48: return launch_partial_batched_t<48, MODE, BF>(args, graphs, grid, s);
    case 64: return launch_partial_batched_t<64, MODE, BF>(args, graphs, grid, s);
    case 80: return launch_partial_batched_t<80, MODE, BF>(args, graphs, grid, s);
    case 96: return launch_partial_batched_t<96, MODE, BF>(args, graphs, grid, s);
    case 112: return launch_partial_batched_t<112, MODE, BF>(args, graphs, grid, s);
    case 128: return launch_partial_batched_t<128, MODE, BF>(args, graphs, grid, s);
    default: return cudaErrorInvalidValue;
  }
}

template <int KP, int CL>
constexpr size_t step_smem() {
  if constexpr (KP == 32)
    return step32::kSmem;
  else
    return sizeof(float) * StepSmem<KP, CL>::floats;
}

template <int KP, int CL>
cudaError_t launch_step_t(const StpmUpdateArgs& a, cudaStream_t s) {
  const size_t smem = step_smem<KP, CL>();
  static bool set = false;
  if (!set) {
    MMSB_CUDA_TRY(cudaFuncSetAttribute(stpm_step_kernel<KP, CL>,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    if (CL > 8)
      MMSB_CUDA_TRY(cudaFuncSetAttribute(stpm_step_kernel<KP, CL>,
                                         cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    set = true;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(CL, 1, 1);
  cfg.blockDim = dim3(512, 1, 1);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = CL;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;  // see step_body
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  MMSB_CUDA_TRY(cudaLaunchKernelEx(&cfg, stpm_step_kernel<KP, CL>, a));
  ++g_launch_count;
  return cudaGetLastError();
}

// step_ctas(KP) CTAs (up to 16, a non-portable cluster size) where the device
// can co-schedule them, else KP / 16 of 16 rows
template <int KP>
cudaError_t launch_step_k(const StpmUpdateArgs& a, cudaStream_t s) {
  if constexpr (KP <= 64 || KP > 128) {
    return launch_step_t<KP, step_ctas(KP)>(a, s);
  } else {
    static int wide = -1;
    if (wide != 0) {
      cudaError_t e = launch_step_t<KP, step_ctas(KP)>(a, s);
      if (e == cudaSuccess) {
        wide = 1;
        return e;
      }
      if (wide == 1) return e;
      cudaGetLastError();
      wide = 0;
    }
    return launch_step_t<KP, KP / 16>(a, s);
  }
}

template <int KP, int CL>
cudaError_t launch_step_batched_t(const StpmUpdateArgs* args, int graphs, cudaStream_t s) {
  const size_t smem = step_smem<KP, CL>();
  static bool set = false;
  if (!set) {
    MMSB_CUDA_TRY(cudaFuncSetAttribute(stpm_step_batched<KP, CL>,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    if (CL > 8)
      MMSB_CUDA_TRY(cudaFuncSetAttribute(stpm_step_batched<KP, CL>,
                                         cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    set = true;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(CL, (unsigned)graphs, 1);
  cfg.blockDim = dim3(512, 1, 1);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = CL;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  MMSB_CUDA_TRY(cudaLaunchKernelEx(&cfg, stpm_step_batched<KP, CL>, args));
  ++g_launch_count;
  return cudaGetLastError();
}

template <int KP>
cudaError_t launch_step_batched_k(const StpmUpdateArgs* args, int graphs, cudaStream_t s) {
  if constexpr (KP <= 64) {
    return launch_step_batched_t<KP, step_ctas(KP)>(args, graphs, s);
  } else {
    static int wide = -1;
    if (wide != 0) {
      cudaError_t e = launch_step_batched_t<KP, step_ctas(KP)>(args, graphs, s);
      if (e == cudaSuccess) {
        wide = 1;
        return e;
      }
      if (wide == 1) return e;
      cudaGetLastError();
      wide = 0;
    }
    return launch_step_batched_t<KP, KP / 16>(args, graphs, s);
  }
}

}  // namespace

int stpm_partial_cluster() { return kPartialCluster; }

// padded k of the STPM kernels: multiples of 16 from 32 to 128, then 160 and
// 208 (k <= 208); -1 beyond
int stpm_kp(int k) {
  const int r = (int)round_up(k, 16);
  if (r <= 32) return 32;
  if (r <= 128) return r;
  if (r <= 160) return 160;
  if (r <= 208) return 208;
  return -1;
}

int stpm_partial_grid(int mode, int k, int64_t count, bool bf16) {
  // at least 64 nodes per CTA (two FP32 tiles, one BF16 tile): measured on
  // 4,096-node minibatches at k = 100, 64 CTAs beat 128 (44 vs 53 us in FP32;
  // staging Phi and the cluster reduction are per-CTA costs)
  // MMSB_CONTRACT_NODES overrides the 64 nodes per CTA (a tuning override)
  static const int64_t per_cta = []() {
    const char* e = std::getenv("MMSB_CONTRACT_NODES");
    const long v = e ? std::strtol(e, nullptr, 10) : 0;
    return v >= 16 ? (int64_t)v : (int64_t)64;
  }();
  // MMSB_CONTRACT_CTAS caps the contraction CTAs of single-graph runs (a
  // tuning override; default 2 per SM)
  static const int64_t cap = []() {
    const char* e = std::getenv("MMSB_CONTRACT_CTAS");
    const long v = e ? std::strtol(e, nullptr, 10) : 0;
    return v > 0 ? (int64_t)v : (int64_t)2 * kNumSMs;
  }();
  int64_t g = std::max<int64_t>(1, std::min<int64_t>(ceil_div(count, per_cta), cap));
  // one wave: a second one repeats the per-CTA costs for a few CTAs (8,192
  // nodes, k = 100: 128 CTAs where 120 fit took 55 / 95 us in the loss and
  // adjoint forms, 39 / 69 us with 88).  As few CTAs as keep the largest share
  // of tiles per CTA.  Not the iterations of KP = 32, whose results keep their
  // roundings (k_step32.cuh): the split is the order of their sums.
  const int KP = stpm_kp(k);
  const bool keep = mode != kModeLoss && KP <= 32;
  const int64_t resident = KP < 0 || keep ? 0
                           : bf16               ? partial_resident_p<true>(mode, KP)
                                                : partial_resident_p<false>(mode, KP);
  if (resident > 0 && g > resident) {
    const int64_t tiles = ceil_div(count, bf16 ? 64 : 32);
    g = ceil_div(tiles, ceil_div(tiles, resident));
  }
  return (int)round_up(g, kPartialCluster);
}

cudaError_t stpm_partial(int mode, const StpmPartialArgs& a, int grid, bool bf16, cudaStream_t s) {
  const int KP = stpm_kp(a.k);
  if (KP < 0) return cudaErrorInvalidValue;
  if (bf16 && (!a.yh1 || !a.yh2 || !a.yh3 || a.ldyh % 8 != 0)) return cudaErrorInvalidValue;
  if (!bf16 && a.ldy % 4 != 0) return cudaErrorInvalidValue;
  return bf16 ? launch_partial_p<true>(mode, KP, a, grid, s)
              : launch_partial_p<false>(mode, KP, a, grid, s);
}

// The power iteration of k = 33, 10,000 nodes (151 iterations): 261 us per
// iteration with a thread per column summing the mean terms and normalising,
// 22 us here; the reduction behind the lambda pass (38 partials) 49 us -> 8 us
// at k = 100 and 245 us -> 115 us at k = 200, nearly all of that the wait for
// the contraction it overlaps.
cudaError_t stpm_reduce(const StpmReduceArgs& a, cudaStream_t s) {
  if (a.k > 256 || (!a.done && (a.lambda || a.mode == kModeLoss))) return cudaErrorInvalidValue;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)a.k, 1, 1);
  cfg.blockDim = dim3(256, 1, 1);
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;  // follows the contraction
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  MMSB_CUDA_TRY(cudaLaunchKernelEx(&cfg, stpm_reduce_kernel, a));
  ++g_launch_count;
  return cudaGetLastError();
}

cudaError_t stpm_update(const StpmUpdateArgs& a, cudaStream_t s) {
  switch (stpm_step_kp(a.k)) {
    case 32: return launch_step_k<32>(a, s);
    case 48: return launch_step_k<48>(a, s);
    case 64: return launch_step_k<64>(a, s);
    case 80: return launch_step_k<80>(a, s);
    case 96: return launch_step_k<96>(a, s);
    case 112: return launch_step_k<112>(a, s);
    case 128: return launch_step_k<128>(a, s);
    case 160: return launch_step_k<160>(a, s);
    case 208: return launch_step_k<208>(a, s);
    default: return cudaErrorInvalidValue;
  }
}

int stpm_step_kp(int k) { return stpm_kp(k); }

size_t stpm_phi_image_bytes(int k) {
  const int kp = stpm_kp(k);
  if (kp < 32 || kp > 112) return 0;
  // hi | lo (ContractTc<KP>::PSZ each); at KP = 32 then m1 | m2
  return (size_t)8 * kp * kp + (kp == 32 ? (size_t)8 * kp : 0);
}

cudaError_t stpm_partial_batched(int mode, int KP, const StpmPartialArgs* args, int graphs,
                                 int grid, bool bf16, cudaStream_t s) {
  if (KP > 128 || grid % kPartialCluster != 0 || graphs < 1 || graphs > 65535)
    return cudaErrorInvalidValue;
  switch (mode) {
    case kModePlain:
      return bf16 ? launch_partial_batched_m<kModePlain, true>(KP, args, graphs, grid, s)
                  : launch_partial_batched_m<kModePlain, false>(KP, args, graphs, grid, s);
    case kModeAdjoint:
      return bf16 ? launch_partial_batched_m<kModeAdjoint, true>(KP, args, graphs, grid, s)
                  : launch_partial_batched_m<kModeAdjoint, false>(KP, args, graphs, grid, s);
    default: return cudaErrorInvalidValue;
  }
}

cudaError_t stpm_update_batched(int KP, const StpmUpdateArgs* args, int graphs, cudaStream_t s) {
  if (graphs < 1 || graphs > 65535) return cudaErrorInvalidValue;
  switch (KP) {
    case 32: return launch_step_batched_k<32>(args, graphs, s);
    case 48: return launch_step_batched_k<48>(args, graphs, s);
    case 64: return launch_step_batched_k<64>(args, graphs, s);
    case 80: return launch_step_batched_k<80>(args, graphs, s);
    case 96: return launch_step_batched_k<96>(args, graphs, s);
    case 112: return launch_step_batched_k<112>(args, graphs, s);
    case 128: return launch_step_batched_k<128>(args, graphs, s);
    default: return cudaErrorInvalidValue;
  }
}

cudaError_t stpm_tensor_values(int k, float* phi, const float* G, double* lambda, cudaStream_t s,
                               double* phi64) {
  tensor_value_kernel<<<(unsigned)ceil_div(k, 8), 256, 0, s>>>(k, phi, G, lambda, phi64);
  ++g_launch_count;
  return cudaGetLastError();
}

}  // namespace mmsb
