/* k_small.cu -- small dense FP64 linear algebra on the device (ell x ell,
 * column-major), replacing the reference's LAPACK calls:
 *
 *   potrf   DPOTRF("L") of the Gram matrix with the single diagonal jitter
 *           retry of glr_common_impl.h:386-398 (1e-12 tr/ell) or of
 *           glr_scalapack_impl.h:129-139 (1e-12 max(dmax, 1)).  One CTA,
 *           32-column panels staged in shared memory, right-looking.
 *   trtri   L^{-1} by column (one warp per column), optionally stored
 *           transposed so that X L^{-T} is a plain GEMM (the DTRSM of
 *           glr_common_impl.h:402).
 *   syev    DSYEVD("V","U") of the projected T (glr_common_impl.h:496-514):
 *           cyclic two-sided block Jacobi in round-robin parallel order,
 *           relative-accuracy rotation threshold, at most 40 sweeps.
 *   select  ordering by |lambda| descending, the cut max(trunc_abs,
 *           trunc_rel max|lambda|), treatment FLIP/RELU/NONE and the report
 *           fields (glr_common_impl.h:517-559; glr_scalapack_impl.h:375-425),
 *           plus the gathered eigenvector columns C_kept.
 */

#include <algorithm>
#include <cmath>
#include <vector>

#include "lgh_device.cuh"
#include "lgh_internal.h"

namespace lgh
{

/* ---------------------------------------------------------------- potrf -- */

/* One CTA, panels of NB columns.  The panel's NB x NB diagonal block is
 * factored by one warp with a row per lane in registers, the rows below it
 * by a thread each with theirs in registers; the arithmetic and its order
 * are those of a column at a time.  A column at a time over the whole panel
 * cost three barriers of 1024 threads for each, 0.8 us a column (n = 60: 47
 * us, now 41; 220: 328 and 237; 800: 6.2 and 5.2 ms); what is left is the
 * chain of a square root and a division per column.  The trailing update is m8n8k4 products of the panel, a warp per
 * 8 x 8 tile.  16 columns: the rows fit the registers of 512 threads. */
constexpr int NB = 16;

__global__ void __launch_bounds__ (512)
k_potrf (int n, double *G, const double *G0, int jitter_mode, int *info)
{
  extern __shared__ double P[];     /* (n - k0) x (NB + 1) panel */
  __shared__ int fail;
  __shared__ double jit;
  const int tid = threadIdx.x, nt = blockDim.x;
  constexpr int ps = NB + 1;
  if (tid == 0) { info[0] = 0; info[1] = 0; }
  for (int attempt = 0; attempt < 2; attempt++) {
    if (attempt == 1) {
      /* re-form G (the factorization destroyed it) and jitter the diagonal */
      if (G0 == nullptr) break;
      for (int e = tid; e < n * n; e += nt) G[e] = G0[e];
      __syncthreads ();
      if (tid == 0) {
        double v = 0.;
        if (jitter_mode == 0) {
          for (int i = 0; i < n; i++) v += G[i + (size_t) i * n];
          v = 1e-12 * v / n;
        } else {
          for (int i = 0; i < n; i++) v = fmax (v, G[i + (size_t) i * n]);
          v = 1e-12 * fmax (v, 1.0);
        }
        jit = v;
        info[1] = 1;
      }
      __syncthreads ();
      for (int i = tid; i < n; i += nt) G[i + (size_t) i * n] += jit;
      __syncthreads ();
    }
    if (tid == 0) fail = 0;
    __syncthreads ();
    for (int k0 = 0; k0 < n && !fail; k0 += NB) {
      const int kb = min (NB, n - k0);
      const int m = n - k0;
      for (int e = tid; e < m * kb; e += nt) {
        const int r = e % m, kk = e / m;
        P[r * ps + kk] = G[(k0 + r) + (size_t) (k0 + kk) * n];
      }
      __syncthreads ();
      if (tid < 32) {
        /* lane r: row r of the diagonal block; columns kb .. NB - 1 of a
         * last panel are never reached */
        double a[NB];
#pragma unroll
        for (int j = 0; j < NB; j++) a[j] = (tid < kb && j < kb) ? P[tid * ps + j] : 0.;
        bool ok = true;
#pragma unroll
        for (int k = 0; k < NB; k++) {
          if (k < kb && ok) {
            const double d = __shfl_sync (0xffffffffu, a[k], k);
            ok = d > 0. && isfinite (d);
            if (ok) {
              const double dk = sqrt (d);
              if (tid == k) a[k] = dk;
              if (tid > k) a[k] /= dk;
#pragma unroll
              for (int j = k + 1; j < NB; j++) {
                const double l = __shfl_sync (0xffffffffu, a[k], j);
                if (tid >= j) a[j] -= a[k] * l;
              }
            }
          }
        }
        if (tid < kb)
#pragma unroll
          for (int j = 0; j < NB; j++)
            if (j <= tid) P[tid * ps + j] = a[j];
        if (tid == 0 && !ok) fail = 1;
      }
      __syncthreads ();
      if (fail) break;
      if (kb == NB) {               /* a shorter panel is the last one */
        for (int r = NB + tid; r < m; r += nt) {
          double x[NB];
#pragma unroll
          for (int j = 0; j < NB; j++) x[j] = P[r * ps + j];
#pragma unroll
          for (int k = 0; k < NB; k++) {
            x[k] /= P[k * ps + k];
#pragma unroll
            for (int j = k + 1; j < NB; j++) x[j] -= x[k] * P[j * ps + k];
          }
#pragma unroll
          for (int j = 0; j < NB; j++) P[r * ps + j] = x[j];
        }
      }
      __syncthreads ();
      for (int e = tid; e < m * kb; e += nt) {
        const int r = e % m, kk = e / m;
        if (r >= kk) G[(k0 + r) + (size_t) (k0 + kk) * n] = P[r * ps + kk];
      }
      /* trailing update G(i, j) -= P(i, :) P(j, :)^T, i >= j >= k0 + kb */
      const int mt = m - kb, nt8 = (mt + 7) / 8;
      const int lane = tid & 31, kl = lane & 3, ml = lane >> 2;
      for (int t = tid >> 5; t < nt8 * nt8; t += nt / 32) {
        const int ti = t % nt8, tj = t / nt8;
        if (ti < tj) continue;
        const int ri = ti * 8 + ml, rj = tj * 8 + ml;
        double c0 = 0., c1 = 0.;
#pragma unroll
        for (int k = 0; k < NB; k += 4) {
          const double a = ri < mt ? P[(kb + ri) * ps + k + kl] : 0.;
          const double b = rj < mt ? P[(kb + rj) * ps + k + kl] : 0.;
          asm volatile ("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 "
                        "{%0, %1}, {%2}, {%3}, {%0, %1};"
                        : "+d"(c0), "+d"(c1) : "d"(a), "d"(b));
        }
        const int cj = tj * 8 + kl * 2;
        double *g = G + (k0 + kb + ri) + (size_t) (k0 + kb + cj) * n;
        if (ri < mt && cj <= ri) g[0] -= c0;
        if (ri < mt && cj + 1 <= ri) g[n] -= c1;
      }
      __syncthreads ();
    }
    __syncthreads ();
    if (!fail) break;
  }
  __syncthreads ();
  if (tid == 0 && fail) info[0] = 1;
  /* clear the strict upper triangle */
  for (int e = tid; e < n * n; e += nt) {
    const int i = e % n, j = e / n;
    if (i < j) G[e] = 0.;
  }
}

int
launch_potrf (int n, double *G, double *G0, int jitter_mode, int *info,
              cudaStream_t s)
{
  if (n <= 0) return 0;
  const int smem = n * (NB + 1) * (int) sizeof (double);
  LGH_CHECK (smem <= 220 * 1024, LGH_ERR_SUP, "potrf: n=%d too large", n);
  if (G0) LGH_CUDA (cudaMemcpyAsync (G0, G, (size_t) n * n * sizeof (double),
                                     cudaMemcpyDeviceToDevice, s));
  LGH_TRY (allow_smem ((const void *) k_potrf, smem));
  k_potrf<<<1, 512, smem, s>>> (n, G, G0, jitter_mode, info);
  LGH_LAUNCH_CHECK ();
  return 0;
}

/* ---------------------------------------------------------------- trtri -- */

__global__ void __launch_bounds__ (256)
k_trtri_lower (int n, const double *__restrict__ L, double *__restrict__ out,
               int transpose)
{
  extern __shared__ double xs[];    /* 8 warps x n */
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int j = blockIdx.x * 8 + warp;
  if (j >= n) return;
  double *x = xs + (size_t) warp * n;
  for (int i = lane; i < n; i += 32) x[i] = (i == j) ? 1. : 0.;
  __syncwarp ();
  for (int k = j; k < n; k++) {
    const double xk = x[k] / L[k + (size_t) k * n];
    __syncwarp ();
    if (lane == 0) x[k] = xk;
    for (int i = k + 1 + lane; i < n; i += 32) x[i] -= L[i + (size_t) k * n] * xk;
    __syncwarp ();
  }
  for (int i = lane; i < n; i += 32) {
    const double v = (i >= j) ? x[i] : 0.;
    if (transpose) out[j + (size_t) i * n] = v;
    else out[i + (size_t) j * n] = v;
  }
}

/* the same with the column in registers, row i in lane i % 32: up to 32 T
 * rows.  Through shared memory a step cost two warp barriers and a round
 * trip, 0.5 us a row; here it is a shuffle, the division and a multiply-add
 * (n = 60: 29.3 us and 16.0; 220: 206 and 62; 500: 851 and 153). */
template <int T>
__global__ void __launch_bounds__ (128)
k_trtri_regs (int n, const double *__restrict__ L, double *__restrict__ out,
              int transpose)
{
  const int lane = threadIdx.x & 31;
  const int j = blockIdx.x * 4 + (threadIdx.x >> 5);
  if (j >= n) return;
  double x[T];
#pragma unroll
  for (int t = 0; t < T; t++) x[t] = 32 * t + lane == j ? 1. : 0.;
#pragma unroll
  for (int t = 0; t < T; t++) {
    const int kend = min (32, n - 32 * t);
    for (int kk = max (0, j - 32 * t); kk < kend; kk++) {
      const int k = 32 * t + kk;
      const double *c = L + (size_t) k * n;
      double l[T];
#pragma unroll
      for (int q = t; q < T; q++) {
        const int i = 32 * q + lane;
        l[q] = i > k && i < n ? __ldg (c + i) : 0.;
      }
      const double xk = __shfl_sync (0xffffffffu, x[t], kk) / __ldg (c + k);
      if (lane == kk) x[t] = xk;
#pragma unroll
      for (int q = t; q < T; q++)
        if (q > t || lane > kk) x[q] -= l[q] * xk;
    }
  }
#pragma unroll
  for (int t = 0; t < T; t++) {
    const int i = 32 * t + lane;
    if (i >= n) break;
    const double v = i >= j ? x[t] : 0.;
    if (transpose) out[j + (size_t) i * n] = v;
    else out[i + (size_t) j * n] = v;
  }
}

int
launch_trtri_lower (int n, const double *L, double *Linv, int transpose,
                    cudaStream_t s)
{
  if (n <= 0) return 0;
  /* columns of up to 512 rows in registers */
  if (n <= 512) {
    auto k = n <= 64 ? k_trtri_regs<2> : n <= 128 ? k_trtri_regs<4>
             : n <= 256 ? k_trtri_regs<8> : k_trtri_regs<16>;
    k<<<(n + 3) / 4, 128, 0, s>>> (n, L, Linv, transpose);
    LGH_LAUNCH_CHECK ();
    return 0;
  }
  const int smem = 8 * n * (int) sizeof (double);
  LGH_TRY (allow_smem ((const void *) k_trtri_lower, smem));
  k_trtri_lower<<<(n + 7) / 8, 256, smem, s>>> (n, L, Linv, transpose);
  LGH_LAUNCH_CHECK ();
  return 0;
}

/* ------------------------------------------------------------- jacobi -- */

/* Block Jacobi: the matrix in blocks of JB rows, paired round-robin.  A
 * round rotates the index pairs of every block pair in shared memory
 * (k_jacobi_pairs, one CTA per pair, the accumulated rotations W kept) and
 * applies the W's to the rest of A and to V as small tensor-core products
 * (k_jacobi_apply, one CTA per tile).  A sweep is nblk - 1 rounds of two
 * launches, 13 at n = 220, where the scalar ordering needs n - 1 rounds,
 * each with a barrier over the whole grid and an update of every entry.
 * Blocks of 16: the steps inside a pair are the longest chain of a round,
 * and a 32 x 32 submatrix is also one tile of the products.
 *
 * Every index pair is rotated once a sweep, as in the scalar ordering: the
 * pairs across the two blocks in each round, those inside a block in the
 * sweep's last round.  (All pairs of the submatrix in every round: twice the
 * rotations and their rounding for the same number of sweeps, 4.1 ms against
 * 3.0 for a random matrix of n = 220, 0.67 and 0.63 at 60; the scalar
 * ordering took 11.3 and 2.1.)  The products are of W - I, added to the tile, so that the late
 * sweeps' small rotations round a tile once, and the eigenvalues are the
 * Rayleigh quotients of the result.  Residual, loss of orthogonality and
 * eigenvalue error (Frobenius, over the norm) at n = 220, of the scalar
 * ordering / all pairs in every round and the diagonal / now: a spectrum
 * that decays to 1e-12 5.1e-15 9.8e-13 2.0e-15 / 7.2e-15 1.3e-12 4.9e-15 /
 * 2.7e-15 1.0e-13 1.3e-16; a third of full rank 4.4e-15 8.1e-13 1.4e-15 /
 * 5.9e-15 9.4e-13 3.6e-15 / 2.5e-15 9.8e-14 1.7e-16. */
constexpr int JB = 16, JT = 2 * JB, JS = JT + 4;   /* block, tile, row stride */

/* index at position `pos` in round r of the round-robin over np entries */
__host__ __device__ __forceinline__ int
rr_index (int pos, int r, int np)
{
  return pos == 0 ? 0 : 1 + ((pos - 1 + r) % (np - 1));
}

/* the matrix index of row i of block pair k in round r (n or more: padding) */
__device__ __forceinline__ int
jacobi_row (int i, int k, int r, int nblk)
{
  const int b = rr_index (i < JB ? k : nblk - 1 - k, r, nblk);
  return b * JB + (i & (JB - 1));
}

/* a power of two that takes x (normal or infinite) to [1, 2), or to [2, 4)
 * from the last binade up, whose inverse is no normal number */
__device__ __forceinline__ double
exponent_scale (double x)
{
  const int e = (__double2hiint (x) >> 20) & 0x7ff;
  return __hiloint2double (max (2046 - e, 1) << 20, 0);
}

/* the rotation that annihilates apq: tan t = s / c with |t| <= 1, from the
 * double angle, d = aqq - app, b = 2 apq: cos 2a = |d| / r, c^2 = (1 + cos
 * 2a) / 2, t = b / (2 r c^2), r^2 = d^2 + b^2.  Reciprocal square roots
 * where t from the quotient d / b takes two divisions and a square root one
 * after the other; d and b are scaled by a power of two first, so nothing
 * overflows.  c and s are then those of t as it is rounded: from the double
 * angle itself c^2 + s^2 is off by a few roundings more, which the columns
 * of V collect (1e-12 at n = 220, now 1e-13).  False (no rotation) below
 * the relative threshold 1e-15 sqrt |app aqq|. */
__device__ __forceinline__ bool
jacobi_rotation (double app, double aqq, double apq, double &c, double &s,
                 double &t)
{
  c = 1.;
  s = t = 0.;
  if (!(fabs (apq) > 1e-300)) return false;
  const double f = exponent_scale (apq), x = apq * f;
  if (!(x * x > 1e-30 * ((fabs (app) * f) * (fabs (aqq) * f)))) return false;
  double d = aqq - app, b = 2. * apq;
  const double g = exponent_scale (fmax (fabs (d), fabs (b)));
  d *= g;
  b *= g;
  const double ri = rsqrt (fma (d, d, b * b));
  const double c2 = fma (0.5 * fabs (d), ri, 0.5);
  const double ci = rsqrt (c2);
  t = (d < 0. ? -0.5 : 0.5) * b * ri * ci * ci;
  c = rsqrt (fma (t, t, 1.));
  s = t * c;
  return true;
}

/* the 2 JB x 2 JB submatrix of each pair: up to `sweeps` passes over its
 * index pairs, all of them where inner is set, else those across the blocks
 * (stopping at a pass without a rotation); the rotated submatrix goes back
 * to A, the rotations to W (row-major), whether there were any to rot[pair],
 * and any_rot / done (sweeps run) record the round */
__global__ void __launch_bounds__ (256)
k_jacobi_pairs (int n, int nblk, int r, int sweeps, int inner, double *A,
                double *Wg, int *rot, int *any_rot, int *done)
{
  __shared__ double S[JT][JS], W[JT][JS];
  __shared__ double cs[JB], sn[JB], tt[JB];
  __shared__ int pp[JB], qq[JB];
  __shared__ int rotated, ever;
  const int tid = threadIdx.x, k = blockIdx.x;
  for (int e = tid; e < JT * JT; e += 256) {
    const int i = e % JT, j = e / JT;
    const int gi = jacobi_row (i, k, r, nblk), gj = jacobi_row (j, k, r, nblk);
    S[i][j] = (gi < n && gj < n) ? A[gi + (size_t) gj * n] : 0.;
    W[i][j] = i == j ? 1. : 0.;
  }
  if (tid == 0) ever = 0;
  int sw = 0;
  for (; sw < sweeps; sw++) {
    if (tid == 0) rotated = 0;
    __syncthreads ();
    for (int q = 0; q < (inner ? JT - 1 : JB); q++) {
      if (tid < JB) {
        const int a = inner ? rr_index (tid, q, JT) : tid;
        const int b = inner ? rr_index (JT - 1 - tid, q, JT)
                            : JB + ((tid + q) & (JB - 1));
        const int pi = a < b ? a : b, qi = a < b ? b : a;
        double c, s, t;
        if (jacobi_rotation (S[pi][pi], S[qi][qi], S[pi][qi], c, s, t)) rotated = 1;
        cs[tid] = c;
        sn[tid] = s;
        tt[tid] = t;
        pp[tid] = pi;
        qq[tid] = qi;
      }
      __syncthreads ();
      {
        /* one 2 x 2 block of S per thread, a half-warp along one row pair */
        const int a = tid / JB, b = tid & (JB - 1);
        const int pa = pp[a], qa = qq[a], pb = pp[b], qb = qq[b];
        const double ca = cs[a], sa = sn[a], cb = cs[b], sb = sn[b];
        if (a == b) {
          if (sa != 0.) {
            const double apq = S[pa][qa], t = tt[a];
            S[pa][pa] -= t * apq;
            S[qa][qa] += t * apq;
            S[pa][qa] = 0.;
            S[qa][pa] = 0.;
          }
        } else if (sa != 0. || sb != 0.) {
          const double x00 = S[pa][pb], x01 = S[pa][qb];
          const double x10 = S[qa][pb], x11 = S[qa][qb];
          const double y00 = cb * x00 - sb * x01, y01 = sb * x00 + cb * x01;
          const double y10 = cb * x10 - sb * x11, y11 = sb * x10 + cb * x11;
          S[pa][pb] = ca * y00 - sa * y10;
          S[pa][qb] = ca * y01 - sa * y11;
          S[qa][pb] = sa * y00 + ca * y10;
          S[qa][qb] = sa * y01 + ca * y11;
        }
        /* two rows of W's columns pb, qb */
        if (sb != 0.) {
#pragma unroll
          for (int h = 0; h < 2; h++) {
            const int i = a + h * JB;
            const double w0 = W[i][pb], w1 = W[i][qb];
            W[i][pb] = cb * w0 - sb * w1;
            W[i][qb] = sb * w0 + cb * w1;
          }
        }
      }
      __syncthreads ();
    }
    if (!rotated) break;
    if (tid == 0) ever = 1;
    __syncthreads ();
  }
  __syncthreads ();
  if (tid == 0) {
    rot[k] = ever;
    if (ever) *any_rot = 1;
    if (k == 0) *done = sw + 1 < sweeps ? sw + 1 : sweeps;
  }
  if (!ever) return;
  for (int e = tid; e < JT * JT; e += 256) {
    const int i = e % JT, j = e / JT;
    const int gi = jacobi_row (i, k, r, nblk), gj = jacobi_row (j, k, r, nblk);
    if (gi < n && gj < n) A[gi + (size_t) gj * n] = S[i][j];
    Wg[(size_t) k * JT * JT + e] = W[e / JT][e % JT];
  }
}

/* D = op (P) Q for 32 x 32 shared tiles, 8 warps: warp w makes row fragment
 * w / 2 and column fragments 2 (w % 2) + {0, 1}; TP: P is transposed */
template <bool TP>
__device__ __forceinline__ void
jacobi_mma (const double (*Pm)[JS], const double (*Qm)[JS], double (&acc)[2][2])
{
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int i0 = (warp >> 1) * 8, j0 = (warp & 1) * 16;
#pragma unroll
  for (int t = 0; t < 2; t++) acc[t][0] = acc[t][1] = 0.;
#pragma unroll
  for (int kk = 0; kk < JT; kk += 4) {
    const int k = kk + (lane & 3), x = lane >> 2;
    const double a = TP ? Pm[k][i0 + x] : Pm[i0 + x][k];
#pragma unroll
    for (int t = 0; t < 2; t++) {
      const double b = Qm[k][j0 + t * 8 + x];
      asm volatile ("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 "
                    "{%0, %1}, {%2}, {%3}, {%0, %1};"
                    : "+d"(acc[t][0]), "+d"(acc[t][1])
                    : "d"(a), "d"(b));
    }
  }
}

/* blockIdx.y < npair: tile (x, y) of A, x < y: W_x^T A W_y, with its mirror;
 * above: 32 rows of V times W_x.  WP and WQ hold W - I. */
__global__ void __launch_bounds__ (256)
k_jacobi_apply (int n, int nblk, int r, double *A, double *V,
                const double *__restrict__ Wg, const int *__restrict__ rot)
{
  __shared__ double T[JT][JS], WP[JT][JS], WQ[JT][JS];
  const int npair = nblk / 2, tid = threadIdx.x;
  const int lane = tid & 31, warp = tid >> 5;
  const int fi = (warp >> 1) * 8 + (lane >> 2), fj = (warp & 1) * 16 + (lane & 3) * 2;
  const bool isv = (int) blockIdx.y >= npair;
  const int kq = isv ? blockIdx.x : blockIdx.y, kp = isv ? 0 : blockIdx.x;
  const int v0 = isv ? ((int) blockIdx.y - npair) * JT : 0;
  double acc[2][2];
  if (isv) {
    if (!rot[kq]) return;
  } else if (kp >= kq || (!rot[kp] && !rot[kq])) {
    return;
  }
  for (int e = tid; e < JT * JT; e += 256) {
    const int i = e % JT, j = e / JT;
    const int gj = jacobi_row (j, kq, r, nblk);
    const int gi = isv ? v0 + i : jacobi_row (i, kp, r, nblk);
    const double *src = isv ? V : A;
    T[i][j] = (gi < n && gj < n) ? src[gi + (size_t) gj * n] : 0.;
    const int wi = e / JT, wj = e % JT;
    const double one = wi == wj ? 1. : 0.;
    WQ[wi][wj] = rot[kq] ? Wg[(size_t) kq * JT * JT + e] - one : 0.;
    if (!isv) WP[wi][wj] = rot[kp] ? Wg[(size_t) kp * JT * JT + e] - one : 0.;
  }
  __syncthreads ();
  /* a thread's entries of T are its own to replace */
  auto add_tile = [&] () {
#pragma unroll
    for (int t = 0; t < 2; t++)
#pragma unroll
      for (int c = 0; c < 2; c++) acc[t][c] += T[fi][fj + t * 8 + c];
  };
  jacobi_mma<false> (T, WQ, acc);
  add_tile ();
  if (!isv) {
    __syncthreads ();
#pragma unroll
    for (int t = 0; t < 2; t++)
#pragma unroll
      for (int c = 0; c < 2; c++) T[fi][fj + t * 8 + c] = acc[t][c];
    __syncthreads ();
    jacobi_mma<true> (WP, T, acc);
    add_tile ();
  }
  __syncthreads ();
#pragma unroll
  for (int t = 0; t < 2; t++)
#pragma unroll
    for (int c = 0; c < 2; c++) T[fi][fj + t * 8 + c] = acc[t][c];
  __syncthreads ();
  for (int e = tid; e < JT * JT; e += 256) {
    const int i = e % JT, j = e / JT;
    const int gj = jacobi_row (j, kq, r, nblk);
    const int gi = isv ? v0 + i : jacobi_row (i, kp, r, nblk);
    if (gi < n && gj < n) (isv ? V : A)[gi + (size_t) gj * n] = T[i][j];
    if (!isv) {
      /* the mirror tile, again along its columns */
      const int mi = jacobi_row (i, kq, r, nblk), mj = jacobi_row (j, kp, r, nblk);
      if (mi < n && mj < n) A[mi + (size_t) mj * n] = T[j][i];
    }
  }
}

__global__ void
k_jacobi_start (int n, double *V, int *flags, int nflags)
{
  const int64_t nn = (int64_t) n * n;
  for (int64_t e = (int64_t) blockIdx.x * blockDim.x + threadIdx.x; e < nn;
       e += (int64_t) gridDim.x * blockDim.x)
    V[e] = ((e % n) == (e / n)) ? 1. : 0.;
  if (blockIdx.x == 0)
    for (int e = threadIdx.x; e < nflags; e += blockDim.x) flags[e] = 0;
}

/* w_j = v_j^T A v_j / v_j^T v_j: JR eigenvectors per CTA, a warp per row of
 * the symmetric A (its contiguous column) */
constexpr int JR = 2;

__global__ void __launch_bounds__ (256)
k_jacobi_rayleigh (int n, const double *__restrict__ A,
                   const double *__restrict__ V, double *w)
{
  extern __shared__ double sv[];               /* [JR][n] */
  __shared__ double red[8][JR][2];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int j0 = blockIdx.x * JR;
  for (int e = tid; e < JR * n; e += 256)
    sv[e] = j0 + e / n < n ? V[(size_t) j0 * n + e] : 0.;
  __syncthreads ();
  double num[JR], den[JR];
#pragma unroll
  for (int q = 0; q < JR; q++) num[q] = den[q] = 0.;
  for (int i = warp; i < n; i += 8) {
    double y[JR];
#pragma unroll
    for (int q = 0; q < JR; q++) y[q] = 0.;
    for (int k = lane; k < n; k += 32) {
      const double a = A[k + (size_t) i * n];
#pragma unroll
      for (int q = 0; q < JR; q++) y[q] = fma (a, sv[q * n + k], y[q]);
    }
#pragma unroll
    for (int q = 0; q < JR; q++) {
      const double v = sv[q * n + i];
      num[q] = fma (v, warp_sum (y[q]), num[q]);
      den[q] = fma (v, v, den[q]);
    }
  }
  if (lane == 0)
#pragma unroll
    for (int q = 0; q < JR; q++) {
      red[warp][q][0] = num[q];
      red[warp][q][1] = den[q];
    }
  __syncthreads ();
  if (tid < JR && j0 + tid < n) {
    double a = 0., b = 0.;
    for (int k = 0; k < 8; k++) {
      a += red[k][tid][0];
      b += red[k][tid][1];
    }
    w[j0 + tid] = a / b;
  }
}

int
launch_syev_jacobi (int n, double *A, double *V, double *w, int *sweeps,
                    cudaStream_t s)
{
  if (n <= 0) return 0;
  LGH_CHECK (n <= 2048, LGH_ERR_SUP, "syev: n=%d > 2048", n);
  constexpr int MAXS = 40;
  const int npair = (n + JT - 1) / JT, nblk = 2 * npair;
  DBuf<double> Wg, A0;
  DBuf<int> flags;     /* rot[npair], any_rot[MAXS], done */
  LGH_TRY (Wg.alloc ((size_t) npair * JT * JT));
  LGH_TRY (A0.alloc ((size_t) n * n));
  LGH_CUDA (cudaMemcpyAsync (A0.p, A, (size_t) n * n * sizeof (double),
                             cudaMemcpyDeviceToDevice, s));
  LGH_TRY (flags.alloc (npair + MAXS + 1));
  int *rot = flags.p, *any = rot + npair, *done = any + MAXS;
  k_jacobi_start<<<std::max (1, std::min (num_sms () * 4, (n * n + 255) / 256)),
                   256, 0, s>>> (n, V, flags.p, npair + MAXS + 1);
  LGH_LAUNCH_CHECK ();
  int ran = 0;
  const dim3 tiles ((unsigned) npair, (unsigned) (npair + npair));
  if (npair == 1) {
    /* the whole matrix in one CTA, to convergence */
    k_jacobi_pairs<<<1, 256, 0, s>>> (n, nblk, 0, MAXS, 1, A, Wg.p, rot, any, done);
    LGH_LAUNCH_CHECK ();
    k_jacobi_apply<<<tiles, 256, 0, s>>> (n, nblk, 0, A, V, Wg.p, rot);
    LGH_LAUNCH_CHECK ();
    LGH_CUDA (cudaMemcpyAsync (&ran, done, sizeof (int), cudaMemcpyDeviceToHost, s));
    LGH_CUDA (cudaStreamSynchronize (s));
  } else {
    for (; ran < MAXS; ) {
      for (int r = 0; r < nblk - 1; r++) {
        k_jacobi_pairs<<<npair, 256, 0, s>>> (n, nblk, r, 1, r == nblk - 2, A, Wg.p,
                                              rot, any + ran, done);
        k_jacobi_apply<<<tiles, 256, 0, s>>> (n, nblk, r, A, V, Wg.p, rot);
      }
      LGH_LAUNCH_CHECK ();
      ran++;
      /* four sweeps before the first look at convergence */
      if (ran < 4) continue;
      int more = 0;
      LGH_CUDA (cudaMemcpyAsync (&more, any + ran - 1, sizeof (int),
                                 cudaMemcpyDeviceToHost, s));
      LGH_CUDA (cudaStreamSynchronize (s));
      if (!more) break;
    }
  }
  k_jacobi_rayleigh<<<(n + JR - 1) / JR, 256, JR * n * (int) sizeof (double), s>>> (
      n, A0.p, V, w);
  LGH_LAUNCH_CHECK ();
  if (sweeps) *sweeps = std::max (ran, 1);
  return 0;
}

/* ------------------------------------------------------------- select -- */

__global__ void __launch_bounds__ (1024)
k_select (int n, const double *__restrict__ w, const double *__restrict__ V,
          double trunc_abs, double trunc_rel, int treat, int *order,
          double *sel, double *lam, double *C)
{
  __shared__ double absmax, cut;
  __shared__ int kept;
  const int tid = threadIdx.x, nt = blockDim.x;
  /* rank: |w| descending, ties by larger raw value, then by index */
  for (int i = tid; i < n; i += nt) {
    const double ai = fabs (w[i]);
    int rank = 0;
    for (int j = 0; j < n; j++) {
      const double aj = fabs (w[j]);
      if (aj > ai || (aj == ai && (w[j] > w[i] || (w[j] == w[i] && j < i))))
        rank++;
    }
    order[rank] = i;
  }
  __syncthreads ();
  if (tid == 0) {
    absmax = fabs (w[order[0]]);
    double c = 0.;
    if (trunc_abs > 0.) c = fmax (c, trunc_abs);
    if (trunc_rel > 0.) c = fmax (c, trunc_rel * absmax);
    cut = c;
    int k = 0;
    while (k < n && fabs (w[order[k]]) > c) k++;
    kept = k;
    double mn = w[0], mx = w[0];
    int nneg = 0;
    for (int i = 0; i < n; i++) {
      mn = fmin (mn, w[i]);
      mx = fmax (mx, w[i]);
      if (w[i] < 0.) nneg++;
    }
    sel[0] = k;
    sel[1] = absmax;
    sel[2] = (k < n) ? fabs (w[order[k]]) : 0.;
    sel[3] = mn;
    sel[4] = mx;
    sel[5] = nneg;
  }
  __syncthreads ();
  for (int j = tid; j < kept; j += nt) {
    const double l = w[order[j]];
    lam[j] = (treat == 0) ? fabs (l) : (treat == 1 ? fmax (l, 0.) : l);
  }
  for (int64_t e = tid; e < (int64_t) n * kept; e += nt) {
    const int i = (int) (e % n), j = (int) (e / n);
    C[e] = V[i + (size_t) order[j] * n];
  }
}

int
launch_select (int n, const double *w, const double *V, double trunc_abs,
               double trunc_rel, int treat, int *order, double *sel,
               double *lam, double *C, cudaStream_t s)
{
  k_select<<<1, 1024, 0, s>>> (n, w, V, trunc_abs, trunc_rel, treat, order,
                               sel, lam, C);
  LGH_LAUNCH_CHECK ();
  return 0;
}

/* extreme eigenvalues of the CG-Lanczos tridiagonal T(k,k) = 1/a_k +
 * b_{k-1}/a_{k-1}, T(k,k+1) = sqrt(b_k)/a_k, through the device Jacobi */
int
device_tridiag_extremes (int m, const double *alpha, const double *beta,
                         double *emin, double *emax)
{
  cudaStream_t s = stream ();
  std::vector<double> T ((size_t) m * m, 0.);
  for (int k = 0; k < m; k++) {
    double d = 1. / alpha[k];
    if (k > 0) d += beta[k - 1] / alpha[k - 1];
    T[k + (size_t) k * m] = d;
    if (k + 1 < m) {
      const double e = sqrt (fabs (beta[k])) / alpha[k];
      T[k + (size_t) (k + 1) * m] = e;
      T[k + 1 + (size_t) k * m] = e;
    }
  }
  DBuf<double> A, V, w;
  LGH_TRY (A.alloc ((size_t) m * m));
  LGH_TRY (V.alloc ((size_t) m * m));
  LGH_TRY (w.alloc (m));
  LGH_CUDA (cudaMemcpyAsync (A.p, T.data (), T.size () * sizeof (double),
                             cudaMemcpyHostToDevice, s));
  LGH_TRY (launch_syev_jacobi (m, A.p, V.p, w.p, nullptr, s));
  std::vector<double> wh (m);
  LGH_CUDA (cudaMemcpyAsync (wh.data (), w.p, m * sizeof (double),
                             cudaMemcpyDeviceToHost, s));
  LGH_CUDA (cudaStreamSynchronize (s));
  *emin = *std::min_element (wh.begin (), wh.end ());
  *emax = *std::max_element (wh.begin (), wh.end ());
  return 0;
}

} /* namespace lgh */
