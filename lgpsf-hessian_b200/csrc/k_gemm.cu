/* k_gemm.cu -- tall-skinny dense products on row-major blocks, FP64
 * accumulation (the plain form's DGEMMs):
 *
 *   gemm_tn  C = A^T B over n rows: the Gram X^T X (glr_common_impl.h:
 *            340-366), the projection Q^T Y (:469-489), U^T X (:825-855),
 *            BCGS2 coefficients (glr_scalapack_impl.h:178).  64 x 64 output
 *            tiles, split over n into slices whose partial tiles are summed
 *            in a fixed order (deterministic), optional symmetrisation
 *            T = (C + C^T)/2 in the same pass (glr_common_impl.h:490-494).
 *   gemm_nn  Y = alpha X M + beta Y0 with a small column-major M: the
 *            triangular update X L^{-T} of CholQR2 (:402), U = Q C_kept
 *            (:567), Y += U W (:876).  64 x 64 tiles, k in steps of 16.
 *
 *   dense_apply  Y = A^{-1} B on the multigrid's dense coarse level.
 *
 * The tall products run on the FP64 tensor cores (mma.sync m8n8k4): a CTA of
 * 4 (or 8) warps owns a 64 (128) x 64 output tile, each warp a 32 x 32 part
 * of 4 x 4 fragments.  Operands come into shared memory 16 k-values at a
 * time with cp.async in a ring of three stages, in their own layout: a block
 * whose columns are the output's rows (A^T B) stays k-major, one whose
 * columns are summed over (X M) stays row-major; the row strides (68 and 20
 * doubles, 72 and 20 floats) put the 16 values of a fragment load's
 * half-warp in distinct banks either way.  Float blocks (mixed path) are
 * widened to FP64 as the fragments are read; every product accumulates in
 * FP64.  Fragments past the operands' edges are not multiplied (220 columns
 * are 27.5 fragments, not the 32 of four whole tiles), and the Gram X^T X
 * forms the tiles on and above its diagonal alone.  At 262144 x 220 x 220
 * the scalar register staging this replaces took 1.42 ms a product (17.9
 * TFLOP/s, the load pipe 76-88 % busy with 8-byte accesses); now 1.00 for
 * X M (25 TFLOP/s of the FP64 tensor pipe's 33) and 0.83 on average over a
 * build's A^T B and X^T X. */

#include <algorithm>
#include <type_traits>

#include "lgh_batch.h"
#include "lgh_device.cuh"
#include "lgh_internal.h"

namespace lgh
{

constexpr int GB = 64, GK = 16, GSTAGES = 3;

/* CB bytes from global to shared memory, the last CB - bytes zero */
template <int CB>
__device__ __forceinline__ void
cp_async (void *smem, const void *src, int bytes)
{
  const unsigned d = (unsigned) __cvta_generic_to_shared (smem);
  if constexpr (CB == 16)
    asm volatile ("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d),
                  "l"(src), "r"(bytes) : "memory");
  else if constexpr (CB == 8)
    asm volatile ("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(d),
                  "l"(src), "r"(bytes) : "memory");
  else
    asm volatile ("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(d),
                  "l"(src), "r"(bytes) : "memory");
}

/* one operand's stage: BX values of x by GK of k.  KM: element (x, k) at
 * k * ld + x in memory and [k][x] in shared memory; else x * ld + k and
 * [x][k]. */
template <typename T, bool KM, int BX>
struct GOp
{
  static constexpr int S = KM ? (sizeof (T) == 8 ? BX + 4 : BX + 8) : GK + 4;
  static constexpr int ROWS = KM ? GK : BX;
  static constexpr int ELEMS = ROWS * S;

  template <int CB, int NT>
  static __device__ __forceinline__ void
  load (T *sm, const T *g, int64_t ld, int64_t x0, int64_t k0, int64_t xmax,
        int64_t kmax, int tid)
  {
    constexpr int E = CB / (int) sizeof (T);
    constexpr int CPR = (KM ? BX : GK) / E;       /* copies per row */
    constexpr int RPP = NT / CPR > 0 ? NT / CPR : 1;
    static_assert (NT % CPR == 0 && ROWS % RPP == 0, "copy split");
    const int c = (tid % CPR) * E, r0 = tid / CPR;
    if constexpr (KM) {
      const int64_t left = xmax - x0 - c;         /* columns from here on */
      /* whole fragments past the edge are never read */
      if (left <= -8) return;
      const int eb = (int) (left >= E ? E : (left > 0 ? left : 0)) * (int) sizeof (T);
#pragma unroll
      for (int r = r0; r < ROWS; r += RPP) {
        const int64_t k = k0 + r;
        const int bytes = k < kmax ? eb : 0;
        cp_async<CB> (sm + r * S + c, bytes ? g + k * ld + x0 + c : g, bytes);
      }
    } else {
      const int64_t left = kmax - k0 - c;
      const int eb = (int) (left >= E ? E : (left > 0 ? left : 0)) * (int) sizeof (T);
#pragma unroll
      for (int r = r0; r < ROWS; r += RPP) {
        const int64_t x = x0 + r;
        if (x >= xmax + 8) break;
        const int bytes = x < xmax ? eb : 0;
        cp_async<CB> (sm + r * S + c, bytes ? g + x * ld + k0 + c : g, bytes);
      }
    }
  }

  static __device__ __forceinline__ double
  frag (const T *sm, int x, int k)
  {
    return (double) sm[KM ? k * S + x : x * S + k];
  }
};

/* acc += the product over k in [k0, k1) of the CTA's tile: BM x 64 output
 * values, BM / 16 warps.  ma, nb: fragments of this warp that hold output
 * (warp-uniform).  m8n8k4 f64 fragments: A (8 x 4, row) holds A[lane / 4]
 * [lane % 4], B (4 x 8, col) holds B[lane % 4][lane / 4], C holds
 * C[lane / 4][2 (lane % 4) + {0, 1}]. */
template <typename TA, bool AKM, int CA, typename TB, bool BKM, int CBB, int BM>
__device__ __forceinline__ void
gemm_tile (const TA *A, int64_t lda, int64_t i0, int64_t imax, const TB *B,
           int64_t ldb, int64_t j0, int64_t jmax, int64_t k0, int64_t k1, int ma,
           int nb, unsigned char *smem, double (&acc)[4][4][2])
{
  using OA = GOp<TA, AKM, BM>;
  using OB = GOp<TB, BKM, GB>;
  constexpr int NT = BM * 2;
  constexpr int ABYTES = OA::ELEMS * (int) sizeof (TA);
  constexpr int SBYTES = ABYTES + OB::ELEMS * (int) sizeof (TB);
  static_assert (ABYTES % 16 == 0 && SBYTES % 16 == 0, "stage alignment");
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int wm = warp >> 1, wn = warp & 1;
  auto stage = [&] (int st) { return smem + st * SBYTES; };
  auto fetch = [&] (int st, int64_t k) {
    unsigned char *p = stage (st);
    OA::template load<CA, NT> ((TA *) p, A, lda, i0, k, imax, k1, tid);
    OB::template load<CBB, NT> ((TB *) (p + ABYTES), B, ldb, j0, k, jmax, k1, tid);
  };
  const int64_t nk = (k1 - k0 + GK - 1) / GK;
#pragma unroll
  for (int q = 0; q < GSTAGES - 1; q++) {
    if (q < nk) fetch (q, k0 + q * GK);
    asm volatile ("cp.async.commit_group;" ::: "memory");
  }
  int st = 0;
  for (int64_t q = 0; q < nk; q++) {
    asm volatile ("cp.async.wait_group %0;" ::"n"(GSTAGES - 2) : "memory");
    __syncthreads ();
    const int sn = st + GSTAGES - 1 >= GSTAGES ? st - 1 : st + GSTAGES - 1;
    if (q + GSTAGES - 1 < nk) fetch (sn, k0 + (q + GSTAGES - 1) * GK);
    asm volatile ("cp.async.commit_group;" ::: "memory");
    const TA *As = (const TA *) stage (st);
    const TB *Bs = (const TB *) (stage (st) + ABYTES);
    if (ma > 0 && nb > 0) {
#pragma unroll
      for (int kk = 0; kk < GK; kk += 4) {
        double a[4], b[4];
#pragma unroll
        for (int t = 0; t < 4; t++) {
          a[t] = t < ma ? OA::frag (As, wm * 32 + t * 8 + (lane >> 2), kk + (lane & 3)) : 0.;
          b[t] = t < nb ? OB::frag (Bs, wn * 32 + t * 8 + (lane >> 2), kk + (lane & 3)) : 0.;
        }
#pragma unroll
        for (int ti = 0; ti < 4; ti++)
          if (ti < ma)
#pragma unroll
            for (int tj = 0; tj < 4; tj++)
              if (tj < nb)
                asm volatile ("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 "
                              "{%0, %1}, {%2}, {%3}, {%0, %1};"
                              : "+d"(acc[ti][tj][0]), "+d"(acc[ti][tj][1])
                              : "d"(a[ti]), "d"(b[tj]));
      }
    }
    st = st + 1 == GSTAGES ? 0 : st + 1;
  }
  asm volatile ("cp.async.wait_group 0;" ::: "memory");
}

template <typename TA, bool AKM, typename TB, bool BKM, int BM>
constexpr int
gemm_smem ()
{
  return GSTAGES * (GOp<TA, AKM, BM>::ELEMS * (int) sizeof (TA)
                    + GOp<TB, BKM, GB>::ELEMS * (int) sizeof (TB));
}

/* fragments of a warp's 32 values from x that lie below xmax */
__device__ __forceinline__ int
gemm_frags (int64_t x, int64_t xmax)
{
  return xmax <= x ? 0 : (int) (xmax - x >= 32 ? 4 : (xmax - x + 7) / 8);
}

__device__ __forceinline__ void
gemm_zero (double (&acc)[4][4][2])
{
#pragma unroll
  for (int a = 0; a < 4; a++)
#pragma unroll
    for (int b = 0; b < 4; b++) acc[a][b][0] = acc[a][b][1] = 0.;
}

/* the C element of acc[ti][tj][c] inside the CTA tile */
__device__ __forceinline__ int
dmma_row (int wm, int ti, int lane)
{
  return wm * 32 + ti * 8 + (lane >> 2);
}

__device__ __forceinline__ int
dmma_col (int wn, int tj, int c, int lane)
{
  return wn * 32 + tj * 8 + (lane & 3) * 2 + c;
}

/* bytes per copy that an operand's base and leading dimension allow */
template <typename T>
static int
copy_bytes (const T *p, int64_t ld)
{
  const uintptr_t a = (uintptr_t) p;
  const size_t l = (size_t) ld * sizeof (T);
  if (a % 16 == 0 && l % 16 == 0) return 16;
  if (sizeof (T) == 8 || (a % 8 == 0 && l % 8 == 0)) return 8;
  return 4;
}

/* partial C = A^T B over rows [kb0, kb1) of row-major A (n x m1), B
 * (n x m2), into work[z] (column-major m1 x m2).  sym (A = B): blockIdx.x
 * counts the tiles on and above the diagonal, column by column. */
template <typename T, int CA, int CB>
__global__ void __launch_bounds__ (128, 4)
k_gemm_tn_part (int64_t n, int m1, int m2, const T *__restrict__ A, int lda,
                const T *__restrict__ B, int ldb, double *__restrict__ work,
                int64_t kchunk, int sym)
{
  extern __shared__ __align__ (16) unsigned char smem[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int wm = warp >> 1, wn = warp & 1;
  int ti0, tj0;
  if (sym) {
    tj0 = 0;
    int t = blockIdx.x;
    while (t > tj0) t -= ++tj0;
    ti0 = t;
  } else {
    const int tm = (m1 + GB - 1) / GB;
    tj0 = blockIdx.x / tm;
    ti0 = blockIdx.x - tj0 * tm;
  }
  const int i0 = ti0 * GB, j0 = tj0 * GB;
  const int64_t kb0 = (int64_t) blockIdx.z * kchunk;
  const int64_t kb1 = kb0 + kchunk < n ? kb0 + kchunk : n;
  double acc[4][4][2];
  gemm_zero (acc);
  int ma = gemm_frags (i0 + wm * 32, m1), nb = gemm_frags (j0 + wn * 32, m2);
  if (sym && i0 + wm * 32 > j0 + wn * 32) ma = 0;   /* below the diagonal */
  if (kb0 < kb1)
    gemm_tile<T, true, CA, T, true, CB, GB> (A, lda, i0, m1, B, ldb, j0, m2,
                                             kb0, kb1, ma, nb, smem, acc);
  double *wz = work + (size_t) blockIdx.z * m1 * m2;
#pragma unroll
  for (int ti = 0; ti < 4; ti++)
#pragma unroll
    for (int tj = 0; tj < 4; tj++)
#pragma unroll
      for (int c = 0; c < 2; c++) {
        const int i = i0 + dmma_row (wm, ti, lane), j = j0 + dmma_col (wn, tj, c, lane);
        if (i < m1 && j < m2 && (!sym || i <= j)) wz[i + (size_t) j * m1] = acc[ti][tj][c];
      }
}

/* acc += one stage of k_gemm_tn_tile (gemm_tile keeps its own copy of this
 * loop: calling it there cost 13 to 40 % through its registers) */
template <typename O>
__device__ __forceinline__ void
gemm_stage (const double *As, const double *Bs, int wm, int wn, int lane, int ma,
            int nb, double (&acc)[4][4][2])
{
  if (ma == 0 || nb == 0) return;
#pragma unroll
  for (int kk = 0; kk < GK; kk += 4) {
    double a[4], b[4];
#pragma unroll
    for (int t = 0; t < 4; t++) {
      a[t] = t < ma ? O::frag (As, wm * 32 + t * 8 + (lane >> 2), kk + (lane & 3)) : 0.;
      b[t] = t < nb ? O::frag (Bs, wn * 32 + t * 8 + (lane >> 2), kk + (lane & 3)) : 0.;
    }
#pragma unroll
    for (int ti = 0; ti < 4; ti++)
      if (ti < ma)
#pragma unroll
        for (int tj = 0; tj < 4; tj++)
          if (tj < nb)
            asm volatile ("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 "
                          "{%0, %1}, {%2}, {%3}, {%0, %1};"
                          : "+d"(acc[ti][tj][0]), "+d"(acc[ti][tj][1])
                          : "d"(a[ti]), "d"(b[tj]));
  }
}

/* k_gemm_tn_part for one output tile of FP64 operands, staged through
 * registers: the next stage is read while the current one is multiplied, in
 * 8-byte loads at any alignment.  SAME: B is A, loaded once.  The whole
 * lgh_gram_noalloc with an even / odd ldx, us with the ring of copies (8-byte
 * ones where ldx is odd) and here: 262144 x 33 130 / 148 and 128 / 129, x 64
 * 143 / 176 and 143 / 143, 20000 x 48 40 / 46 and 39 / 39.  For A^T B the
 * ring is kept where its copies are 16 bytes. */
template <bool SAME>
__global__ void __launch_bounds__ (128)
k_gemm_tn_tile (int64_t n, int m1, int m2, const double *__restrict__ A, int lda,
                const double *__restrict__ B, int ldb, double *__restrict__ work,
                int64_t kchunk)
{
  using O = GOp<double, true, GB>;
  __shared__ double As[O::ELEMS], Bs[SAME ? 1 : O::ELEMS];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int wm = warp >> 1, wn = warp & 1;
  const int64_t kb0 = (int64_t) blockIdx.x * kchunk;
  const int64_t kb1 = kb0 + kchunk < n ? kb0 + kchunk : n;
  const int ma = SAME && wm > wn ? 0 : gemm_frags (wm * 32, m1);
  const int nb = gemm_frags (wn * 32, m2);
  double acc[4][4][2];
  gemm_zero (acc);
  /* k row tid / 8; columns tid % 8, tid % 8 + 8, ... */
  const int lk = tid >> 3, lc = tid & 7;
  double ra[8], rb[SAME ? 1 : 8];
  auto fetch = [&] (int64_t k0) {
    const int64_t k = k0 + lk;
#pragma unroll
    for (int e = 0; e < 8; e++) {
      const int c = lc + e * 8;
      ra[e] = k < kb1 && c < m1 ? A[k * lda + c] : 0.;
      if constexpr (!SAME) rb[e] = k < kb1 && c < m2 ? B[k * ldb + c] : 0.;
    }
  };
  fetch (kb0);
  for (int64_t k0 = kb0; k0 < kb1; k0 += GK) {
#pragma unroll
    for (int e = 0; e < 8; e++) {
      As[lk * O::S + lc + e * 8] = ra[e];
      if constexpr (!SAME) Bs[lk * O::S + lc + e * 8] = rb[e];
    }
    __syncthreads ();
    fetch (k0 + GK);
    gemm_stage<O> (As, SAME ? As : Bs, wm, wn, lane, ma, nb, acc);
    __syncthreads ();
  }
  double *wz = work + (size_t) blockIdx.x * m1 * m2;
#pragma unroll
  for (int ti = 0; ti < 4; ti++)
#pragma unroll
    for (int tj = 0; tj < 4; tj++)
#pragma unroll
      for (int c = 0; c < 2; c++) {
        const int i = dmma_row (wm, ti, lane), j = dmma_col (wn, tj, c, lane);
        if (i < m1 && j < m2 && (!SAME || i <= j)) wz[i + (size_t) j * m1] = acc[ti][tj][c];
      }
}

/* C = the sum of the slices in slice order; upper: the slices hold the
 * entries on and above the diagonal of a symmetric product */
__global__ void
k_gemm_tn_reduce (int m1, int m2, int nsplit, const double *__restrict__ work,
                  double *C, int ldc, int sym, int upper)
{
  const int64_t total = (int64_t) m1 * m2;
  auto sum = [&] (int64_t e) {
    double s[4] = { 0., 0., 0., 0. };
    for (int z = 0; z < nsplit; z += 4)
#pragma unroll
      for (int q = 0; q < 4; q++)
        if (z + q < nsplit) s[q] += work[(size_t) (z + q) * total + e];
    return (s[0] + s[1]) + (s[2] + s[3]);
  };
  for (int64_t e = (int64_t) blockIdx.x * blockDim.x + threadIdx.x; e < total;
       e += (int64_t) gridDim.x * blockDim.x) {
    const int i = (int) (e % m1), j = (int) (e / m1);
    if (upper && i > j) continue;
    double s = sum (e);
    if (sym && !upper) s = 0.5 * (s + sum ((int64_t) j + (int64_t) i * m1));
    C[i + (size_t) j * ldc] = s;
    if (upper) C[j + (size_t) i * ldc] = s;
  }
}

/* the same sum with one warp per entry, for products of few entries in many
 * slices (the 200 coefficients of one vector: one CTA of serial sums took
 * 16 us) */
__global__ void __launch_bounds__ (256)
k_gemm_tn_reduce_warp (int64_t total, int m1, int nsplit,
                       const double *__restrict__ work, double *C, int ldc)
{
  const int lane = threadIdx.x & 31;
  for (int64_t e = (int64_t) blockIdx.x * 8 + (threadIdx.x >> 5); e < total;
       e += (int64_t) gridDim.x * 8) {
    double s = 0.;
    for (int z = lane; z < nsplit; z += 32) s += work[(size_t) z * total + e];
    s = warp_sum (s);
    if (lane == 0) C[e % m1 + (size_t) (e / m1) * ldc] = s;
  }
}

/* the sum of k_gemm_tn_reduce_warp, in its order, with one thread per
 * entry: the same bits for products of many entries, whose slices a warp
 * per entry would read a sector at a time.  For the request loop, whose
 * columns must not depend on how many of them are harvested together. */
__global__ void __launch_bounds__ (128)
k_gemm_tn_reduce_same (int64_t total, int m1, int nsplit,
                       const double *__restrict__ work, double *C, int ldc)
{
  for (int64_t e = (int64_t) blockIdx.x * 128 + threadIdx.x; e < total;
       e += (int64_t) gridDim.x * 128) {
    double s[32];
#pragma unroll
    for (int q = 0; q < 32; q++) s[q] = 0.;
    for (int z = 0; z < nsplit; z += 32)
#pragma unroll
      for (int q = 0; q < 32; q++)
        if (z + q < nsplit) s[q] += work[(size_t) (z + q) * total + e];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
      for (int q = 0; q < o; q++) s[q] += s[q + o];
    C[e % m1 + (size_t) (e / m1) * ldc] = s[0];
  }
}

/* slices of 256 rows, or of 64 up to 64 of them: few rows are bound by the
 * stages of a slice (the whole Gram product at 1000 x 130 35 us in 4 slices,
 * 22 in 16; 5000 x 65 36 in 20, 30 in 64) */
static int64_t
tn_max_splits (int64_t n)
{
  return std::max ((n + 255) / 256, std::min<int64_t> ((n + 63) / 64, 64));
}

static int
tn_splits (int64_t n, int m1, int m2)
{
  /* one wave of 4 resident 4-warp CTAs per SM over all tiles and slices
   * (gemm_tn_work_max follows this rule) */
  const int tiles = ((m1 + GB - 1) / GB) * ((m2 + GB - 1) / GB);
  int want = 4 * num_sms () / tiles;
  const int64_t maxs = tn_max_splits (n);
  if (want > maxs) want = (int) maxs;
  if (want < 1) want = 1;
  if (want > 256) want = 256;
  return want;
}

size_t
gemm_tn_work_elems (int64_t n, int m1, int m2)
{
  /* one column: two CTAs of k_gemv_t per SM (one: 134 us at 512^2 x 220,
   * two: 83) */
  const int ns = tn_splits (n, m1, m2);
  return (size_t) (m2 == 1 ? std::max (ns, 2 * num_sms ()) : ns) * m1 * m2;
}

/* a workspace bound for every shape m1 <= m1max, m2 <= m2max: with t tiles
 * the split count is at most ceil(4 S / t), so splits x tiles <= 4 S + t,
 * and each tile holds at most GB x GB partial sums */
size_t
gemm_tn_work_max (int m1max, int m2max)
{
  const size_t tmax = (size_t) ((m1max + GB - 1) / GB) * ((m2max + GB - 1) / GB);
  return (4 * (size_t) num_sms () + tmax) * GB * GB;
}

/* the tiled form takes as many slices as one column does at every width
 * (launch_gemm_tn with tiles set): this many partial sums */
size_t
gemm_tn_work_tiles (int64_t n, int m1, int m2max)
{
  return (size_t) tn_splits (n, m1, 1) * m1 * m2max;
}

/* C from nsplit slices of partial sums in work; tiles: each entry's sum in
 * an order that does not depend on m2 */
static int
gemm_tn_sum (int m1, int m2, int nsplit, const double *work, double *C, int ldc,
             int sym, int upper, cudaStream_t s, int tiles = 0)
{
  const int64_t total = (int64_t) m1 * m2;
  if (!sym && !upper && nsplit >= 16 && total <= 8192) {
    k_gemm_tn_reduce_warp<<<(int) ((total + 7) / 8), 256, 0, s>>> (
        total, m1, nsplit, work, C, ldc);
  } else if (!sym && !upper && nsplit >= 16 && tiles) {
    const int rg = (int) std::min<int64_t> ((total + 127) / 128, num_sms () * 8);
    k_gemm_tn_reduce_same<<<rg, 128, 0, s>>> (total, m1, nsplit, work, C, ldc);
  } else {
    const int rg = (int) std::min<int64_t> ((total + 255) / 256, num_sms () * 8);
    k_gemm_tn_reduce<<<rg, 256, 0, s>>> (m1, m2, nsplit, work, C, ldc, sym, upper);
  }
  LGH_LAUNCH_CHECK ();
  return 0;
}

/* work[z] = the part of A^T x in this CTA's rows (A n x m1 row-major, x a
 * strided vector): two packs of a row per thread, 512 / L rows of a CTA at
 * once, four rows of a thread in flight.  HBM streams A once; the 64-column
 * output tiles of k_gemm_tn_part read it at 2 TB/s for one column. */
constexpr int GV_THREADS = 512;

template <typename T>
__global__ void __launch_bounds__ (GV_THREADS)
k_gemv_t (int64_t n, int m1, const T *__restrict__ A, int lda,
          const T *__restrict__ x, int ldx, double *__restrict__ work, int L,
          int rpc)
{
  constexpr int W = Pack<T>::W, CH = 2, U = 4;
  extern __shared__ double red[];          /* [rpc][nvec * W] */
  const int nvec = (m1 + W - 1) / W;
  const int rl = threadIdx.x / L, lane = threadIdx.x - rl * L;
  const int64_t stride = (int64_t) gridDim.x * rpc;
  double acc[CH][W];
#pragma unroll
  for (int h = 0; h < CH; h++)
#pragma unroll
    for (int e = 0; e < W; e++) acc[h][e] = 0.;
  if (rl < rpc)
    for (int64_t i = (int64_t) blockIdx.x * rpc + rl; i < n; i += U * stride) {
      Pack<T> a[U][CH];
      double xv[U];
#pragma unroll
      for (int u = 0; u < U; u++) {
        const int64_t r = i + u * stride;
        xv[u] = r < n ? (double) x[r * ldx] : 0.;
#pragma unroll
        for (int h = 0; h < CH; h++) {
          const int vi = lane + h * L;
          a[u][h] = (r < n && vi < nvec) ? ldp (A + r * lda + vi * W) : pzero<T> ();
        }
      }
#pragma unroll
      for (int u = 0; u < U; u++)
#pragma unroll
        for (int h = 0; h < CH; h++)
#pragma unroll
          for (int e = 0; e < W; e++)
            acc[h][e] = fma ((double) a[u][h].v[e], xv[u], acc[h][e]);
    }
  const int mw = nvec * W;
  if (rl < rpc)
#pragma unroll
    for (int h = 0; h < CH; h++) {
      const int vi = lane + h * L;
      if (vi < nvec)
#pragma unroll
        for (int e = 0; e < W; e++) red[rl * mw + vi * W + e] = acc[h][e];
    }
  __syncthreads ();
  for (int c = threadIdx.x; c < m1; c += GV_THREADS) {
    double sum = 0.;
    for (int r = 0; r < rpc; r++) sum += red[r * mw + c];
    work[(size_t) blockIdx.x * m1 + c] = sum;
  }
}

/* y = alpha X m + beta y0 for one column: a warp per row, two rows in
 * flight, m in shared memory */
template <typename T>
__global__ void __launch_bounds__ (256)
k_gemv_n (int64_t n, int k, double alpha, const T *__restrict__ X, int ldx,
          const double *__restrict__ M, double beta, const T *Y0, int ldy0,
          T *Y, int ldy)
{
  constexpr int W = Pack<T>::W;
  extern __shared__ __align__ (16) unsigned char smem[];
  double *m = reinterpret_cast<double *> (smem);
  for (int e = threadIdx.x; e < k; e += 256) m[e] = M[e];
  __syncthreads ();
  const int lane = threadIdx.x & 31, nfull = k / W;
  const int64_t nw = (int64_t) gridDim.x * 8;
  for (int64_t i = (int64_t) blockIdx.x * 8 + (threadIdx.x >> 5); i < n; i += 2 * nw) {
    const int64_t i1 = i + nw;
    const bool two = i1 < n;
    const T *x0 = X + i * ldx, *x1 = X + (two ? i1 : i) * ldx;
    double s0 = 0., s1 = 0.;
#pragma unroll 4
    for (int v = lane; v < nfull; v += 32) {
      const Pack<T> a = ldp (x0 + v * W), b = ldp (x1 + v * W);
#pragma unroll
      for (int e = 0; e < W; e++) {
        const double mv = m[v * W + e];
        s0 = fma ((double) a.v[e], mv, s0);
        s1 = fma ((double) b.v[e], mv, s1);
      }
    }
    const int t = nfull * W + lane;
    if (t < k) {
      s0 = fma ((double) x0[t], m[t], s0);
      s1 = fma ((double) x1[t], m[t], s1);
    }
    s0 = alpha * warp_sum (s0);
    s1 = alpha * warp_sum (s1);
    if (lane == 0) {
      if (beta != 0.) s0 += beta * (double) Y0[i * ldy0];
      Y[i * ldy] = (T) s0;
      if (two) {
        if (beta != 0.) s1 += beta * (double) Y0[i1 * ldy0];
        Y[i1 * ldy] = (T) s1;
      }
    }
  }
}

/* nsplit slices (their partial tiles in work), then the sum */
template <typename T>
static int
gemm_tn_run (int64_t n, int m1, int m2, const T *A, int lda, const T *B, int ldb,
             double *C, int ldc, int sym, double *work, int nsplit, bool upper,
             cudaStream_t s, int tiles = 0)
{
  int64_t kchunk = (n + nsplit - 1) / nsplit;
  kchunk = (kchunk + GK - 1) / GK * GK;
  const int tm = (m1 + GB - 1) / GB, tn = (m2 + GB - 1) / GB;
  dim3 grid ((unsigned) (upper ? tm * (tm + 1) / 2 : tm * tn), 1, (unsigned) nsplit);
  constexpr int smem = gemm_smem<T, true, T, true, GB> ();
  auto run = [&] (auto ca, auto cb) -> int {
    auto k = k_gemm_tn_part<T, decltype (ca)::value, decltype (cb)::value>;
    LGH_TRY (allow_smem ((const void *) k, smem));
    k<<<grid, 128, smem, s>>> (n, m1, m2, A, lda, B, ldb, work, kchunk, upper);
    LGH_LAUNCH_CHECK ();
    return 0;
  };
  using C16 = std::integral_constant<int, 16>;
  using CS = std::integral_constant<int, sizeof (T)>;
  const bool a16 = copy_bytes (A, lda) == 16, b16 = copy_bytes (B, ldb) == 16;
  if constexpr (sizeof (T) == 8) {
    if ((upper || !(a16 && b16)) && m1 <= GB && m2 <= GB) {
      auto k = upper ? k_gemm_tn_tile<true> : k_gemm_tn_tile<false>;
      k<<<nsplit, 128, 0, s>>> (n, m1, m2, A, lda, B, ldb, work, kchunk);
      LGH_LAUNCH_CHECK ();
      return gemm_tn_sum (m1, m2, nsplit, work, C, ldc, sym, upper, s, tiles);
    }
  }
  if (a16 && b16) LGH_TRY (run (C16 (), C16 ()));
  else if (a16) LGH_TRY (run (C16 (), CS ()));
  else if (b16) LGH_TRY (run (CS (), C16 ()));
  else LGH_TRY (run (CS (), CS ()));
  return gemm_tn_sum (m1, m2, nsplit, work, C, ldc, sym, upper, s, tiles);
}

template <typename T>
int
launch_gemm_tn (int64_t n, int m1, int m2, const T *A, int lda, const T *B,
                int ldb, double *C, int ldc, int sym, double *work,
                size_t work_elems, cudaStream_t s, int tiles)
{
  if (m1 == 0 || m2 == 0) return 0;
  LGH_CHECK (!sym || m1 == m2, LGH_ERR_ARG_SIZ, "gemm_tn: sym needs square");
  int ns = tn_splits (n, m1, tiles ? 1 : m2);
  LGH_CHECK ((size_t) ns * m1 * m2 <= work_elems, LGH_ERR_ARG_SIZ,
             "gemm_tn: workspace too small");
  constexpr int W = Pack<T>::W;
  if (!tiles && m2 == 1 && m1 > 1 && copy_bytes (A, lda) == 16 && (m1 + W - 1) / W <= 2 * GV_THREADS) {
    const int nvec = (m1 + W - 1) / W, L = (nvec + 1) / 2, rpc = GV_THREADS / L;
    const int64_t tiles = (n + rpc - 1) / rpc;
    const int nb = (int) std::max<int64_t> (1, std::min<int64_t> (
        std::min<int64_t> (2 * num_sms (), (tiles + 3) / 4),
        (int64_t) (work_elems / (size_t) m1)));
    const int smem = rpc * nvec * W * (int) sizeof (double);
    k_gemv_t<T><<<nb, GV_THREADS, smem, s>>> (n, m1, A, lda, B, ldb, work, L, rpc);
    LGH_LAUNCH_CHECK ();
    return gemm_tn_sum (m1, 1, nb, work, C, ldc, 0, 0, s);
  }
  /* X^T X: its upper tiles alone, over as many more slices as fit */
  const bool upper = !tiles && (const void *) A == (const void *) B && lda == ldb
                     && m1 == m2;
  if (upper) {
    const int tm = (m1 + GB - 1) / GB;
    const int64_t want = std::max (1, 4 * num_sms () / (tm * (tm + 1) / 2));
    ns = (int) std::min<int64_t> (std::min<int64_t> (want, 256),
                                  std::min<int64_t> (tn_max_splits (n),
                                                     (int64_t) (work_elems / ((size_t) m1 * m2))));
    ns = std::max (ns, 1);
  }
  return gemm_tn_run<T> (n, m1, m2, A, lda, B, ldb, C, ldc, sym, work, ns, upper, s,
                         tiles);
}

/* the same product with an explicit split count and caller-provided
 * partial-sum storage of nsplit * m1 * m2 doubles */
int
launch_gemm_tn_fixed (int64_t n, int m1, int m2, const double *A, int lda,
                      const double *B, int ldb, double *C, int ldc,
                      double *work, int nsplit, cudaStream_t s)
{
  if (m1 == 0 || m2 == 0) return 0;
  if (nsplit < 1) nsplit = 1;
  return gemm_tn_run<double> (n, m1, m2, A, lda, B, ldb, C, ldc, 0, work, nsplit,
                              A == B && lda == ldb && m1 == m2, s);
}

int
gemm_tn_splits (int64_t n, int m1, int m2)
{
  return tn_splits (n, m1, m2);
}

template int launch_gemm_tn<double> (int64_t, int, int, const double *, int,
                                     const double *, int, double *, int, int,
                                     double *, size_t, cudaStream_t, int);
template int launch_gemm_tn<float> (int64_t, int, int, const float *, int,
                                    const float *, int, double *, int, int,
                                    double *, size_t, cudaStream_t, int);

/* Y = alpha X M + beta Y0: X row-major n x k, M column-major k x m2.
 * Column tiles run fastest, so the CTAs resident at once share a band of X
 * rows in L2 (rows fastest read X from HBM once per column tile). */
template <typename T, int CA, int CB>
__global__ void __launch_bounds__ (128, 3)
k_gemm_nn (int64_t n, int k, int m2, double alpha, const T *__restrict__ X,
           int ldx, const double *__restrict__ M, int ldm, double beta,
           const T *Y0, int ldy0, T *Y, int ldy, int tn)
{
  extern __shared__ __align__ (16) unsigned char smem[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int wm = warp >> 1, wn = warp & 1;
  const int64_t rt = blockIdx.x / tn;
  const int64_t i0 = rt * GB;
  const int j0 = (int) (blockIdx.x - rt * tn) * GB;
  double acc[4][4][2];
  gemm_zero (acc);
  gemm_tile<T, false, CA, double, false, CB, GB> (
      X, ldx, i0, n, M, ldm, j0, m2, 0, k, gemm_frags (i0 + wm * 32, n),
      gemm_frags (j0 + wn * 32, m2), smem, acc);
#pragma unroll
  for (int ti = 0; ti < 4; ti++)
#pragma unroll
    for (int tj = 0; tj < 4; tj++)
#pragma unroll
      for (int c = 0; c < 2; c++) {
        const int64_t i = i0 + dmma_row (wm, ti, lane);
        const int j = j0 + dmma_col (wn, tj, c, lane);
        if (i < n && j < m2) {
          double v = alpha * acc[ti][tj][c];
          if (beta != 0.) v += beta * (double) Y0[i * ldy0 + j];
          Y[i * ldy + j] = (T) v;
        }
      }
}

/* The Woodbury combination of many shifts in one launch (the batched
 * solve / sample of the shift-independent form x_c = f(c) y0 + W D_c U^T r,
 * glr_common_impl.h:910-929 applied per shift):
 *   out[:, J] = fc[si] Y0[:, j] + W S[:, J],  J = si m + j,
 * W n x kept row-major (the shift-independent W = Z^{-1} M^{1/2} U), S kept
 * x (nshift m) column-major (k_shift_scale: g[:, si] .* (U^T r)[:, j] with
 * g[k, si] = f(lam_k + c_si) - f(c_si)), Y0 n x m row-major, out
 * column-major with leading dimension *ldo at *out (the output pointer is
 * read from device memory so that a captured graph serves every call).
 * One GEMM on the FP64 tensor cores, whose epilogue adds f(c) y0 and writes
 * the caller's column-major result.  Column tiles run fastest, so the CTAs
 * resident at once share a band of W rows in L2. */
template <int BM, int CA, int CB>
__global__ void __launch_bounds__ (BM * 2, BM == 128 ? 2 : 3)
k_shift_combine (int64_t n, int kept, int m, int ncol,
                 const double *__restrict__ W, int ldw,
                 const double *__restrict__ S, const double *__restrict__ fc,
                 const double *__restrict__ Y0, int ldy0,
                 double *const *__restrict__ out, const int64_t *__restrict__ ldo)
{
  extern __shared__ __align__ (16) unsigned char smem[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int wm = warp >> 1, wn = warp & 1;
  const int64_t i0 = (int64_t) blockIdx.y * BM;
  const int j0 = blockIdx.x * GB;
  double acc[4][4][2];
  gemm_zero (acc);
  gemm_tile<double, false, CA, double, false, CB, BM> (
      W, ldw, i0, n, S, kept, j0, ncol, 0, kept, gemm_frags (i0 + wm * 32, n),
      gemm_frags (j0 + wn * 32, ncol), smem, acc);
  double *const o = *out;
  const int64_t ld = *ldo;
#pragma unroll
  for (int tj = 0; tj < 4; tj++)
#pragma unroll
    for (int c = 0; c < 2; c++) {
      const int J = j0 + dmma_col (wn, tj, c, lane);
      if (J >= ncol) continue;
      const int si = J / m, j = J - si * m;
      const double f = fc[si];
#pragma unroll
      for (int ti = 0; ti < 4; ti++) {
        const int64_t i = i0 + dmma_row (wm, ti, lane);
        if (i < n)
          o[i + (int64_t) J * ld] = acc[ti][tj][c] + f * Y0[i * ldy0 + j];
      }
    }
}

/* S[k + J kept] = g[k, si] C[k, j], J = si m + j */
__global__ void
k_shift_scale (int kept, int m, int64_t ncol, const double *__restrict__ C,
               const double *__restrict__ g, double *__restrict__ S)
{
  const int64_t total = (int64_t) kept * ncol;
  for (int64_t e = (int64_t) blockIdx.x * blockDim.x + threadIdx.x; e < total;
       e += (int64_t) gridDim.x * blockDim.x) {
    const int64_t J = e / kept;
    const int k = (int) (e - J * kept);
    const int64_t si = J / m;
    S[e] = g[k + si * kept] * C[k + (J - si * m) * kept];
  }
}

/* 128-row tiles (8 warps) or 64-row tiles (4 warps), as the autotuner picks
 * (262144 rows x 200 kept, 16 shifts x 96 columns: 8.5 ms with the scalar
 * staging, 18.9 TFLOP/s) */
int
launch_shift_combine_variant (int variant, int64_t n, int kept, int m,
                              int nshift, const double *W, int ldw,
                              const double *C, const double *g, double *S,
                              const double *fc, const double *Y0, int ldy0,
                              double *const *out, const int64_t *ldo,
                              cudaStream_t s)
{
  if (n == 0 || m == 0 || nshift == 0) return 0;
  const int BM = variant == 1 ? 128 : 64;
  const int64_t ncol = (int64_t) nshift * m;
  const int64_t rt = (n + BM - 1) / BM;
  LGH_CHECK (ncol < INT32_MAX && rt < 65536, LGH_ERR_ARG_OUTOFRANGE,
             "shift combine: %lld rows x %lld columns exceed the grid",
             (long long) n, (long long) ncol);
  if (kept > 0) {
    const int sg = (int) std::min<int64_t> (((int64_t) kept * ncol + 255) / 256,
                                            num_sms () * 8);
    k_shift_scale<<<sg, 256, 0, s>>> (kept, m, ncol, C, g, S);
    LGH_LAUNCH_CHECK ();
  }
  dim3 grid ((unsigned) ((ncol + GB - 1) / GB), (unsigned) rt);
  auto run = [&] (auto bm, auto cb) -> int {
    constexpr int BM_ = decltype (bm)::value;
    constexpr int smem = gemm_smem<double, false, double, false, BM_> ();
    /* W's rows are padded to 4 values at a 256-byte base */
    auto k = k_shift_combine<BM_, 16, decltype (cb)::value>;
    LGH_TRY (allow_smem ((const void *) k, smem));
    k<<<grid, BM_ * 2, smem, s>>> (n, kept, m, (int) ncol, W, ldw, S, fc, Y0,
                                   ldy0, out, ldo);
    LGH_LAUNCH_CHECK ();
    return 0;
  };
  LGH_CHECK (kept == 0 || copy_bytes (W, ldw) == 16, LGH_ERR_ARG_WRONG,
             "shift combine: W must be 16-byte aligned");
  using std::integral_constant;
  const bool b16 = copy_bytes (S, kept) == 16;
  if (variant == 1)
    return b16 ? run (integral_constant<int, 128> (), integral_constant<int, 16> ())
               : run (integral_constant<int, 128> (), integral_constant<int, 8> ());
  return b16 ? run (integral_constant<int, 64> (), integral_constant<int, 16> ())
             : run (integral_constant<int, 64> (), integral_constant<int, 8> ());
}

/* Y = A^{-1} B on the dense coarse level: A^{-1} n0 x n0 column-major (and
 * symmetric), B and Y n0 x ld row-major; columns w .. ld - 1 of Y are set to
 * zero.  n0 is 33 to 1500 and w as small as one, so the product is bound by
 * latency, not by the FP64 tensor pipe: a CTA takes a small tile (8 MT rows
 * x 8 NT columns) and its NW warps split the n0 terms, each reading its
 * fragments straight from L2 (for a fixed k, 8 consecutive rows of A^{-1}
 * and 8 consecutive columns of B: whole 32-byte sectors) with the loads of
 * several k steps in flight; the warps' partial tiles are added in warp
 * order through shared memory.  A 64 x 64 tile with one serial pass over n0
 * left 9 to 36 CTAs on the chip: 45 us at n0 = 559 x 220 columns and 46 us
 * at 704 x 1, now 10.6 and 4.3 (back to back launches alone take 4). */
template <typename T, int MT, int NT, int NW, int U>
__global__ void __launch_bounds__ (NW * 32, NT > 1 ? 2 : 1)
k_dense_apply (int n0, const double *__restrict__ Ainv, const T *__restrict__ B,
               T *__restrict__ Y, int w, int ld)
{
  pdl_wait ();
  constexpr int TM = 8 * MT, TN = 8 * NT;
  extern __shared__ double red[];              /* [NW][TM * TN] */
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int i0 = blockIdx.x * TM, c0 = blockIdx.y * TN;
  /* this warp's k range, in steps of 4 */
  const int steps = (n0 + 3) / 4;
  const int s0 = (int) ((int64_t) steps * warp / NW);
  const int s1 = (int) ((int64_t) steps * (warp + 1) / NW);
  const int kl = lane & 3, ml = lane >> 2;
  double acc[MT][NT][2];
#pragma unroll
  for (int a = 0; a < MT; a++)
#pragma unroll
    for (int b = 0; b < NT; b++) acc[a][b][0] = acc[a][b][1] = 0.;
#pragma unroll U
  for (int s = s0; s < s1; s++) {
    const int k = 4 * s + kl;
    double a[MT], b[NT];
#pragma unroll
    for (int t = 0; t < MT; t++) {
      const int i = i0 + t * 8 + ml;
      a[t] = (k < n0 && i < n0) ? __ldg (Ainv + i + (size_t) k * n0) : 0.;
    }
#pragma unroll
    for (int t = 0; t < NT; t++) {
      const int c = c0 + t * 8 + ml;
      b[t] = (k < n0 && c < w) ? (double) B[(size_t) k * ld + c] : 0.;
    }
#pragma unroll
    for (int ti = 0; ti < MT; ti++)
#pragma unroll
      for (int tj = 0; tj < NT; tj++)
        asm volatile ("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 "
                      "{%0, %1}, {%2}, {%3}, {%0, %1};"
                      : "+d"(acc[ti][tj][0]), "+d"(acc[ti][tj][1])
                      : "d"(a[ti]), "d"(b[tj]));
  }
#pragma unroll
  for (int ti = 0; ti < MT; ti++)
#pragma unroll
    for (int tj = 0; tj < NT; tj++)
#pragma unroll
      for (int c = 0; c < 2; c++)
        red[warp * (TM * TN) + (ti * 8 + ml) * TN + tj * 8 + kl * 2 + c]
            = acc[ti][tj][c];
  __syncthreads ();
  for (int e = threadIdx.x; e < TM * TN; e += NW * 32) {
    double v = 0.;
#pragma unroll
    for (int q = 0; q < NW; q++) v += red[q * (TM * TN) + e];
    const int gi = i0 + e / TN, gc = c0 + e % TN;
    if (gi < n0 && gc < ld) Y[(size_t) gi * ld + gc] = gc < w ? (T) v : T (0);
  }
}

template <typename T, int MT, int NT, int NW, int U>
static int
dense_apply_tile (int n0, const double *Ainv, const T *B, T *Y, int w, int ld,
                  cudaStream_t s)
{
  const int smem = NW * 64 * MT * NT * (int) sizeof (double);
  static_assert (NW * 64 * MT * NT * 8 <= 48 * 1024, "default shared limit");
  dim3 grid ((unsigned) ((n0 + 8 * MT - 1) / (8 * MT)),
             (unsigned) ((ld + 8 * NT - 1) / (8 * NT)));
  LGH_CUDA (launch_pdl (0, k_dense_apply<T, MT, NT, NW, U>, grid, NW * 32, smem, s, n0,
                        Ainv, B, Y, w, ld));
  LGH_LAUNCH_CHECK ();
  return 0;
}

template <typename T>
int
launch_dense_apply (int n0, const double *Ainv, const T *B, T *Y, int w, int ld,
                    cudaStream_t s)
{
  /* one tile of columns: 8 rows over 16 warps while that is one wave
   * (n0 = 704: 4.3 us, 6.3 with 16 rows; 1500: 8.1 and 6.3).  Up to 64
   * columns 16 x 16 over 16 warps (32 KB of partials), wider 32 x 16 over 8:
   * us in FP64 of the two, and of 32 x 32 over 4 warps, at 704 x 33 columns
   * 6.3, 8.3, 14.5; 1500 x 60 16.5, 18.6, 24.7; 559 x 132 11.4, 10.4, 12.5;
   * 559 x 220 12.5, 10.6, 12.8; FP32 at 1500 x 90 20.6, 18.6, 35.0 */
  if (ld <= 8 && n0 <= 8 * num_sms ())
    return dense_apply_tile<T, 1, 1, 16, 8> (n0, Ainv, B, Y, w, ld, s);
  if (ld <= 8) return dense_apply_tile<T, 2, 1, 16, 4> (n0, Ainv, B, Y, w, ld, s);
  if (ld <= 64) return dense_apply_tile<T, 2, 2, 16, 2> (n0, Ainv, B, Y, w, ld, s);
  return dense_apply_tile<T, 4, 2, 8, 4> (n0, Ainv, B, Y, w, ld, s);
}

template int launch_dense_apply<double> (int, const double *, const double *,
                                         double *, int, int, cudaStream_t);
template int launch_dense_apply<float> (int, const double *, const float *,
                                        float *, int, int, cudaStream_t);

template <typename T>
int
launch_gemm_nn (int64_t n, int k, int m2, double alpha, const T *X, int ldx,
                const double *M, int ldm, double beta, const T *Y0, int ldy0,
                T *Y, int ldy, cudaStream_t s, int tiles_only)
{
  if (n == 0 || m2 == 0) return 0;
  if (!tiles_only && m2 == 1 && k > 0 && k <= 2048 && copy_bytes (X, ldx) == 16) {
    const int want = (int) std::min<int64_t> ((n + 15) / 16, 1 << 20);
    const int smem = k * (int) sizeof (double);
    auto f = k_gemv_n<T>;
    f<<<fit_grid (f, std::max (want, 1), 256, smem), 256, smem, s>>> (
        n, k, alpha, X, ldx, M, beta, Y0, ldy0, Y, ldy);
    LGH_LAUNCH_CHECK ();
    return 0;
  }
  const int tn = (m2 + GB - 1) / GB;
  const int64_t tiles = (n + GB - 1) / GB * tn;
  LGH_CHECK (tiles < INT32_MAX, LGH_ERR_ARG_OUTOFRANGE, "gemm_nn: too many tiles");
  constexpr int smem = gemm_smem<T, false, double, false, GB> ();
  auto run = [&] (auto ca, auto cb) -> int {
    auto f = k_gemm_nn<T, decltype (ca)::value, decltype (cb)::value>;
    LGH_TRY (allow_smem ((const void *) f, smem));
    f<<<(unsigned) tiles, 128, smem, s>>> (n, k, m2, alpha, X, ldx, M, ldm, beta,
                                           Y0, ldy0, Y, ldy, tn);
    LGH_LAUNCH_CHECK ();
    return 0;
  };
  using C16 = std::integral_constant<int, 16>;
  using CT = std::integral_constant<int, sizeof (T)>;
  using C8 = std::integral_constant<int, 8>;
  const bool a16 = copy_bytes (X, ldx) == 16, b16 = copy_bytes (M, ldm) == 16;
  if (a16) return b16 ? run (C16 (), C16 ()) : run (C16 (), C8 ());
  return b16 ? run (CT (), C16 ()) : run (CT (), C8 ());
}

template int launch_gemm_nn<double> (int64_t, int, int, double,
                                     const double *, int, const double *, int,
                                     double, const double *, int, double *,
                                     int, cudaStream_t, int);
template int launch_gemm_nn<float> (int64_t, int, int, double, const float *,
                                    int, const double *, int, double,
                                    const float *, int, float *, int,
                                    cudaStream_t, int);

} /* namespace lgh */
