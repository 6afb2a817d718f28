/* k_strip.cu -- the B product Y = B X in strip form.
 *
 * The reference multiplies B into a block one column at a time (MatMult per
 * column, glr_common_impl.h:325-332).  Row by row on the device (k_spmm.cu)
 * every nonzero (i, j) gathers the whole row X[j, :], so a 220-wide FP64
 * block pulls nnz x 1760 bytes through L1/L2 per product: 84 GB at the
 * 512^2 configuration, for 1.5 GB of algorithmic traffic.  Consecutive rows
 * of a local operator (a kernel matrix on a grid or a well-ordered mesh)
 * share most of their columns, so the strip form groups R consecutive rows
 * and stores, per strip, the union of their column indices with an R-value
 * column of the strip's entries at each (zero where a row has none).  The
 * product then loads each gathered X row once per strip and applies it to
 * the R rows from registers: the gather traffic falls by about the factor
 * (R * nnz per row) / (union per strip), 5x at R = 8 on the 2D kernel
 * matrix, for some padded FMAs.
 *
 * Layout (device):
 *   sptr[s] .. sptr[s+1]   the union entries of strip s (int64)
 *   scol[k]                the column of entry k (int32)
 *   sval[k * R + r]        row r0 + r's value at scol[k] (FP64; sval32 FP32)
 * Building: one group of R lanes per strip merges the R rows' column lists
 * (warp min-reduction over the lanes' current columns; the lanes whose
 * current column is the minimum emit their value and advance).  Each
 * nonzero is emitted exactly once, so the form is exact for any CSR (rows
 * need not be sorted; unsorted rows only lengthen the unions).  Two passes:
 * union lengths, a scan, then the fill.  The strip height R (2, 4 or 8) is
 * chosen per operator from the union lengths by a cost model of the
 * product: padded FMA slots against gathered bytes.
 */

#include <algorithm>
#include <type_traits>

#include "lgh_device.cuh"
#include "lgh_flat.cuh"
#include "lgh_internal.h"
#include "lgh_strip.h"

namespace lgh
{

namespace
{

/* union length (count pass, sval == nullptr) or the fill of each strip of
 * R rows; lanes grouped by R inside a warp, one strip per group */
template <int R>
__global__ void __launch_bounds__ (256)
k_strip_merge (int64_t n, int64_t nstrips, const int64_t *__restrict__ rowptr,
               const int32_t *__restrict__ colidx,
               const double *__restrict__ vals, int64_t *__restrict__ counts,
               const int64_t *__restrict__ sptr, int32_t *__restrict__ scol,
               double *__restrict__ sval, float *__restrict__ sval32,
               unsigned long long *__restrict__ total)
{
  const int lane = threadIdx.x & 31;
  const int sub = lane & (R - 1);
  const unsigned gmask = (R == 32) ? 0xffffffffu
                         : (((1u << R) - 1u) << (lane & ~(R - 1)));
  const int64_t groups_per_cta = blockDim.x / R;
  const int64_t gstride = (int64_t) gridDim.x * groups_per_cta;
  for (int64_t s0 = (int64_t) blockIdx.x * groups_per_cta; s0 < nstrips;
       s0 += gstride) {
    /* every group of the warp runs the loop trip of its own strip; the
     * merge's reductions involve only the group's lanes */
    const int64_t s = s0 + (threadIdx.x / R);
    const bool live = s < nstrips;
    const int64_t row = s * R + sub;
    int64_t k = 0, kend = 0;
    if (live && row < n) {
      k = rowptr[row];
      kend = rowptr[row + 1];
    }
    int64_t pos = (live && sptr) ? sptr[s] : 0;
    int64_t len = 0;
    for (;;) {
      const int cur = (k < kend) ? colidx[k] : INT32_MAX;
      const int m = (int) __reduce_min_sync (gmask, (unsigned) cur);
      if (m == INT32_MAX) break;
      const bool mine = (cur == m);
      if (sval) {
        const double v = mine ? vals[k] : 0.;
        sval[pos * R + sub] = v;
        sval32[pos * R + sub] = (float) v;
        if (sub == 0) scol[pos] = m;
        pos++;
      }
      if (mine) k++;
      len++;
    }
    if (live && !sval && sub == 0) {
      counts[s] = len;
      atomicAdd (total, (unsigned long long) len);
    }
  }
}

/* exclusive scan of counts (one CTA; each thread a contiguous chunk) */
__global__ void __launch_bounds__ (1024)
k_scan_counts (int64_t m, const int64_t *__restrict__ counts,
               int64_t *__restrict__ ptr)
{
  __shared__ int64_t part[1024];
  const int t = threadIdx.x;
  const int64_t chunk = (m + blockDim.x - 1) / blockDim.x;
  const int64_t a = (t * chunk < m) ? t * chunk : m;
  const int64_t b = (a + chunk < m) ? a + chunk : m;
  int64_t s = 0;
  for (int64_t i = a; i < b; i++) s += counts[i];
  part[t] = s;
  __syncthreads ();
  if (t == 0) {
    int64_t run = 0;
    for (int i = 0; i < (int) blockDim.x; i++) {
      const int64_t x = part[i];
      part[i] = run;
      run += x;
    }
    ptr[m] = run;
  }
  __syncthreads ();
  int64_t run = part[t];
  for (int64_t i = a; i < b; i++) {
    ptr[i] = run;
    run += counts[i];
  }
}

/* FP64 blocks, strips of 8 rows: an 8-row strip times 8 columns of X is the
 * m8n8k4 product of the tensor cores, four union entries at a time.  The A
 * fragment is the entries' values as they lie (4 entries x 8 rows, 256
 * contiguous bytes), the B fragment the gathered X rows (8 columns of each,
 * whole sectors), so nothing is staged.  A warp takes one strip and NT x 8
 * columns, U steps of loads in flight; the warps of a CTA are neighbouring
 * column slices of the same strips.  The vector form of this (a warp per
 * strip and 128 columns, values staged in shared memory, 16 FMAs per
 * gathered pack) was bound by FP64 issue and the load pipe: 2.49 ms at
 * 512^2 x 220 columns, now 1.42 (1.0 at the FP64 rate with the strips'
 * zeros).  w: columns, a multiple of 2. */
template <int NT, int U, int MINB>
__global__ void __launch_bounds__ (256, MINB)
k_strip_mma (int64_t n, int64_t items, int ncs, const int64_t *__restrict__ sptr,
             const int32_t *__restrict__ scol, const double *__restrict__ sval,
             const double *__restrict__ X, int ldx, double *__restrict__ Y,
             int ldy, int w)
{
  const int lane = threadIdx.x & 31;
  const int64_t item = (int64_t) blockIdx.x * 8 + (threadIdx.x >> 5);
  if (item >= items) return;
  const int64_t s = item / ncs;
  const int c0 = (int) (item - s * ncs) * NT * 8;
  const int kl = lane & 3, x = lane >> 2;
  const int64_t k0 = sptr[s];
  const int cnt = (int) (sptr[s + 1] - k0);
  const int32_t *sc = scol + k0;
  const double *sv = sval + k0 * 8;
  double acc[NT][2];
#pragma unroll
  for (int t = 0; t < NT; t++) acc[t][0] = acc[t][1] = 0.;
  for (int k = 0; k < cnt; k += 4 * U) {
    double a[U], b[U][NT];
#pragma unroll
    for (int u = 0; u < U; u++) {
      const int kk = k + 4 * u + kl;
      const bool in = kk < cnt;
      const int c = in ? __ldg (sc + kk) : 0;
      a[u] = in ? __ldg (sv + (size_t) kk * 8 + x) : 0.;
      const double *xr = X + (int64_t) c * ldx + c0 + x;
#pragma unroll
      for (int t = 0; t < NT; t++)
        b[u][t] = (in && c0 + t * 8 + x < w) ? __ldg (xr + t * 8) : 0.;
    }
#pragma unroll
    for (int u = 0; u < U; u++)
#pragma unroll
      for (int t = 0; t < NT; t++)
        asm volatile ("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 "
                      "{%0, %1}, {%2}, {%3}, {%0, %1};"
                      : "+d"(acc[t][0]), "+d"(acc[t][1])
                      : "d"(a[u]), "d"(b[u][t]));
  }
  const int64_t i = s * 8 + x;
  if (i >= n) return;
#pragma unroll
  for (int t = 0; t < NT; t++) {
    const int c = c0 + t * 8 + kl * 2;
    double *y = Y + i * ldy + c;
    if (c < w) {              /* w is even */
      Pack<double> o;
      o.v[0] = acc[t][0];
      o.v[1] = acc[t][1];
      stp (y, o);
    }
  }
}

/* two FP32 fused multiply-adds in one instruction, each rounded as fmaf */
__device__ __forceinline__ void
fma_f32x2 (unsigned long long &d, unsigned long long a, unsigned long long b)
{
  asm ("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b));
}

/* the product of U entries from the k-th (see k_strip_f32) */
template <int CH, int U>
__device__ __forceinline__ void
strip_step_f32 (int k, const int32_t *__restrict__ sc,
                const ulonglong2 *__restrict__ sv,
                const float *__restrict__ X, int ldx, int lane, int L,
                int nvec, unsigned long long (&acc)[4][CH][4])
{
  ulonglong2 v[U][2];
  Pack<float> x[U][CH];
#pragma unroll
  for (int u = 0; u < U; u++) {
    const float *xr = X + (int64_t) __ldg (sc + k + u) * ldx;
#pragma unroll
    for (int q = 0; q < 2; q++) v[u][q] = __ldg (sv + (size_t) (k + u) * 2 + q);
#pragma unroll
    for (int h = 0; h < CH; h++) {
      const int vi = lane + h * L;
      if (h < CH - 1 || vi < nvec) x[u][h] = ldp (xr + vi * 4);
    }
  }
#pragma unroll
  for (int u = 0; u < U; u++)
#pragma unroll
    for (int h = 0; h < CH; h++)
      if (h < CH - 1 || lane + h * L < nvec)
#pragma unroll
        for (int e = 0; e < 4; e++) {
          const unsigned b = __float_as_uint (x[u][h].v[e]);
          const unsigned long long bb = ((unsigned long long) b << 32) | b;
          fma_f32x2 (acc[0][h][e], v[u][0].x, bb);
          fma_f32x2 (acc[1][h][e], v[u][0].y, bb);
          fma_f32x2 (acc[2][h][e], v[u][1].x, bb);
          fma_f32x2 (acc[3][h][e], v[u][1].y, bb);
        }
}

/* FP32 blocks, strips of 8 rows, in the flat mapping of lgh_flat.cuh over
 * strips: a thread holds CH packs of all 8 rows, as 4 pairs of rows (the
 * values lie in pairs; an X element is repeated once for four FMAs of two),
 * U entries in flight.  The accumulators take 32 CH registers, so at 2
 * packs two CTAs are resident and two entries in flight hide the gathers;
 * one entry at 4 CTAs of single packs was bound by issue.  256^2 (118 union
 * entries per strip), us at 131 / 220 columns: a warp per 64 packs 140 /
 * 155, one pack 113 / 199, two packs with one entry 112 / 191, with two 88 /
 * 146 (96 / 165 without the paired FMAs); 389 x 511 of 286 entries at 131
 * columns 866 and 608. */
template <int CH, int U>
__global__ void __launch_bounds__ (FLAT_THREADS, 2)
k_strip_f32 (int64_t n, int64_t nstrips, const int64_t *__restrict__ sptr,
             const int32_t *__restrict__ scol, const float *__restrict__ sval,
             const float *__restrict__ X, int ldx, float *__restrict__ Y,
             int ldy, int nvec, int L, int rpc)
{
  const int rl = threadIdx.x / L, lane = threadIdx.x - rl * L;
  const int64_t s = (int64_t) blockIdx.x * rpc + rl;
  if (rl >= rpc || s >= nstrips) return;
  const int64_t k0 = sptr[s];
  const int cnt = (int) (sptr[s + 1] - k0);
  const int32_t *sc = scol + k0;
  const ulonglong2 *sv = reinterpret_cast<const ulonglong2 *> (sval + k0 * 8);
  unsigned long long acc[4][CH][4];
#pragma unroll
  for (int r = 0; r < 4; r++)
#pragma unroll
    for (int h = 0; h < CH; h++)
#pragma unroll
      for (int e = 0; e < 4; e++) acc[r][h][e] = 0;
  int k = 0;
  for (; k + U <= cnt; k += U)
    strip_step_f32<CH, U> (k, sc, sv, X, ldx, lane, L, nvec, acc);
  for (; k < cnt; k++)
    strip_step_f32<CH, 1> (k, sc, sv, X, ldx, lane, L, nvec, acc);
  const int64_t r0 = s * 8;
#pragma unroll
  for (int r = 0; r < 8; r++) {
    if (r0 + r >= n) break;
#pragma unroll
    for (int h = 0; h < CH; h++) {
      const int vi = lane + h * L;
      if (h < CH - 1 || vi < nvec) {
        Pack<float> o;
#pragma unroll
        for (int e = 0; e < 4; e++)
          o.v[e] = __uint_as_float ((unsigned) (acc[r / 2][h][e] >> (r & 1) * 32));
        stp (Y + (r0 + r) * ldy + vi * 4, o);
      }
    }
  }
}

/* the product of the k-th entry (see k_strip_flat).  The packs load together
 * where a thread has 4 of them or 4 rows to multiply each by; two packs of
 * two rows are faster one after the other (131 columns: FP64 173 us and 187,
 * FP32 85 and 94) */
template <int R, int CH, typename T>
__device__ __forceinline__ void
strip_step (int k, const int32_t *__restrict__ sc, const T *__restrict__ sv,
            const T *__restrict__ X, int ldx, int lane, int L, int nvec,
            T (&acc)[R][CH][Pack<T>::W])
{
  constexpr int W = Pack<T>::W;
  constexpr bool TOGETHER = R == 4 || CH == 4;
  const T *xr = X + (int64_t) __ldg (sc + k) * ldx;
  T v[R];
  Pack<T> x[CH];
  if constexpr (R >= W) {
#pragma unroll
    for (int r = 0; r < R; r += W) {
      const Pack<T> p = ldp_nc (sv + (size_t) k * R + r);
#pragma unroll
      for (int e = 0; e < W; e++) v[r + e] = p.v[e];
    }
  } else {
#pragma unroll
    for (int r = 0; r < R; r++) v[r] = __ldg (sv + (size_t) k * R + r);
  }
  if constexpr (TOGETHER) {
#pragma unroll
    for (int h = 0; h < CH; h++) {
      const int vi = lane + h * L;
      if (h < CH - 1 || vi < nvec) x[h] = ldp (xr + vi * W);
    }
  }
#pragma unroll
  for (int h = 0; h < CH; h++) {
    const int vi = lane + h * L;
    if (h < CH - 1 || vi < nvec) {
      if constexpr (!TOGETHER) x[h] = ldp (xr + vi * W);
#pragma unroll
      for (int r = 0; r < R; r++)
#pragma unroll
        for (int e = 0; e < W; e++)
          acc[r][h][e] = fma (v[r], x[h].v[e], acc[r][h][e]);
    }
  }
}

/* strips of 2 or 4 rows (operators whose rows share few columns): the flat
 * mapping over strips, a thread holding CH packs of all R rows.  256^2 rows
 * of 56 entries, us at 60 / 131 / 220 / 400 columns, with a warp per strip
 * and 128 (R = 4) or 256 packs, and here: FP64 R = 2 340 / 369 / 394 / 438
 * and 94 / 158 / 231 / 409, R = 4 206 / 226 / 246 / 466 and 82 / 157 / 239 /
 * 402; FP32 R = 2 356 / 365 / 369 / 400 and 47 / 84 / 123 / 207, R = 4 210 /
 * 216 / 220 / 241 and 45 / 82 / 127 / 204.  A diagonal operator of as many
 * rows, FP64 at 131 / 400: 48 / 77 and 27 / 81 (64 at the copy rate).  CTAs
 * per SM: FP64 takes 128 registers at 4 packs of 4 rows, 80 otherwise. */
template <typename T, int R, int CH>
__global__ void __launch_bounds__ (FLAT_THREADS, sizeof (T) == 4 ? 4 : (R * CH > 8 ? 2 : 3))
k_strip_flat (int64_t n, int64_t nstrips, const int64_t *__restrict__ sptr,
              const int32_t *__restrict__ scol, const T *__restrict__ sval,
              const T *__restrict__ X, int ldx, T *__restrict__ Y, int ldy,
              int nvec, int L, int rpc)
{
  constexpr int W = Pack<T>::W;
  const int rl = threadIdx.x / L, lane = threadIdx.x - rl * L;
  if (rl >= rpc) return;
  for (int64_t s = (int64_t) blockIdx.x * rpc + rl; s < nstrips;
       s += (int64_t) gridDim.x * rpc) {
    const int64_t k0 = sptr[s];
    const int cnt = (int) (sptr[s + 1] - k0);
    const int32_t *sc = scol + k0;
    const T *sv = sval + k0 * R;
    T acc[R][CH][W];
#pragma unroll
    for (int r = 0; r < R; r++) flat_zero<T, CH, W> (acc[r]);
    for (int k = 0; k < cnt; k++)
      strip_step<R, CH, T> (k, sc, sv, X, ldx, lane, L, nvec, acc);
    const int64_t r0 = s * R;
#pragma unroll
    for (int r = 0; r < R; r++) {
      if (r0 + r >= n) break;
#pragma unroll
      for (int h = 0; h < CH; h++) {
        const int vi = lane + h * L;
        if (h < CH - 1 || vi < nvec) {
          Pack<T> o;
#pragma unroll
          for (int e = 0; e < W; e++) o.v[e] = acc[r][h][e];
          stp (Y + (r0 + r) * ldy + vi * W, o);
        }
      }
    }
  }
}

} /* namespace */

int
launch_scan_counts (int64_t m, const int64_t *counts, int64_t *ptr,
                    cudaStream_t s)
{
  k_scan_counts<<<1, 1024, 0, s>>> (m, counts, ptr);
  LGH_LAUNCH_CHECK ();
  return 0;
}

namespace
{

template <int R>
int
merge_pass (const Csr &A, int64_t nstrips, int64_t *counts,
            unsigned long long *total, const StripForm *S, cudaStream_t s)
{
  const int grid = (int) std::min<int64_t> ((nstrips * R + 255) / 256,
                                            (int64_t) num_sms () * 16);
  if (S)
    k_strip_merge<R><<<std::max (grid, 1), 256, 0, s>>> (
        A.n, nstrips, A.rowptr, A.colidx, A.vals, nullptr, S->sptr, S->scol,
        S->sval, S->sval32, nullptr);
  else
    k_strip_merge<R><<<std::max (grid, 1), 256, 0, s>>> (
        A.n, nstrips, A.rowptr, A.colidx, A.vals, counts, nullptr, nullptr,
        nullptr, nullptr, total);
  LGH_LAUNCH_CHECK ();
  return 0;
}

int
merge_any (int R, const Csr &A, int64_t nstrips, int64_t *counts,
           unsigned long long *total, const StripForm *S, cudaStream_t s)
{
  if (R == 2) return merge_pass<2> (A, nstrips, counts, total, S, s);
  if (R == 4) return merge_pass<4> (A, nstrips, counts, total, S, s);
  return merge_pass<8> (A, nstrips, counts, total, S, s);
}

/* modelled cost of one product per block column at strip height R: each
 * union entry costs R FMA slots and one gathered X element; a gathered
 * element costs about as much as kGather FMA slots (on-chip bandwidth
 * against the FP64 FMA rate) */
constexpr double kGather = 12.0;

double
strip_cost (double unions, int R)
{
  return unions * std::max ((double) R, kGather);
}

} /* namespace */

void
strip_free (StripForm &S)
{
  dfree (S.sptr);
  dfree (S.scol);
  dfree (S.sval);
  dfree (S.sval32);
  S = StripForm ();
}

int
strip_build (const Csr &A, int force_R, StripForm &S)
{
  cudaStream_t s = stream ();
  strip_free (S);
  const int64_t n = A.n;
  if (n == 0 || A.nnz == 0) return 0;
  const int cand[3] = { 2, 4, 8 };
  DBuf<unsigned long long> tot;
  LGH_TRY (tot.alloc (4));
  LGH_CUDA (cudaMemsetAsync (tot.p, 0, 4 * sizeof (unsigned long long), s));
  DBuf<int64_t> cnt[3];
  for (int c = 0; c < 3; c++)
    LGH_TRY (cnt[c].alloc ((size_t) (n + cand[c] - 1) / cand[c] + 1));
  int R = force_R;
  if (R <= 0) {
    for (int c = 0; c < 3; c++)
      LGH_TRY (merge_any (cand[c], A, (n + cand[c] - 1) / cand[c], cnt[c].p,
                          tot.p + c, nullptr, s));
    unsigned long long th[3];
    LGH_CUDA (cudaMemcpyAsync (th, tot.p, sizeof (th), cudaMemcpyDeviceToHost, s));
    LGH_CUDA (cudaStreamSynchronize (s));
    double best = 0.;
    for (int c = 0; c < 3; c++) {
      const double cost = strip_cost ((double) th[c], cand[c]);
      if (R <= 0 || cost < best) { best = cost; R = cand[c]; }
    }
  }
  S.R = R;
  S.n = n;
  S.nstrips = (n + R - 1) / R;
  S.nnz = A.nnz;
  const int ci = R == 2 ? 0 : (R == 4 ? 1 : 2);
  int64_t *counts = cnt[ci].p;
  if (force_R > 0)   /* only the forced height was not counted above */
    LGH_TRY (merge_any (R, A, S.nstrips, counts, tot.p + ci, nullptr, s));
  unsigned long long nent = 0;
  LGH_CUDA (cudaMemcpyAsync (&nent, tot.p + ci, sizeof (nent),
                             cudaMemcpyDeviceToHost, s));
  LGH_CUDA (cudaStreamSynchronize (s));
  S.nent = (int64_t) nent;
  LGH_TRY (dalloc ((void **) &S.sptr, (size_t) (S.nstrips + 1) * sizeof (int64_t)));
  LGH_TRY (dalloc ((void **) &S.scol, (size_t) S.nent * sizeof (int32_t) + 16));
  LGH_TRY (dalloc ((void **) &S.sval, (size_t) S.nent * R * sizeof (double) + 16));
  LGH_TRY (dalloc ((void **) &S.sval32, (size_t) S.nent * R * sizeof (float) + 16));
  LGH_TRY (launch_scan_counts (S.nstrips, counts, S.sptr, s));
  LGH_TRY (merge_any (R, A, S.nstrips, nullptr, nullptr, &S, s));
  LGH_CUDA (cudaStreamSynchronize (s));
  return 0;
}

template <int NT, int U, int MINB>
static int
strip_mma (const StripForm &S, const double *X, int ldx, double *Y, int ldy,
           int w, cudaStream_t s)
{
  const int ncs = (w + NT * 8 - 1) / (NT * 8);
  const int64_t items = S.nstrips * ncs, ctas = (items + 7) / 8;
  LGH_CHECK (ctas < (int64_t) INT32_MAX, LGH_ERR_ARG_OUTOFRANGE,
             "strip product: grid too large");
  k_strip_mma<NT, U, MINB><<<(unsigned) ctas, 256, 0, s>>> (
      S.n, items, ncs, S.sptr, S.scol, S.sval, X, ldx, Y, ldy, w);
  LGH_LAUNCH_CHECK ();
  return 0;
}

/* strips of 2 and 4 rows: two packs per thread where there are that many,
 * in FP64 four above 32 packs (R = 2) or 24 (R = 4); fewer where some SM
 * would not get two CTAs.  56 entries a row, two packs and four: R = 2 at 60
 * columns 94 and 99 us, 131 175 and 158; R = 4 at 20 54 and 65, 60 91 and
 * 80; FP32 keeps two (R = 4 at 60 46 and 51, 400 203 and 239) */
template <typename T, int R>
static int
strip_flat (const StripForm &S, const T *sval, const T *X, int ldx, T *Y,
            int ldy, int nvec, cudaStream_t s)
{
  constexpr int W = Pack<T>::W;
  for (int p0 = 0; p0 < nvec; p0 += FLAT_THREADS) {
    const int nv = std::min (nvec - p0, FLAT_THREADS);
    int ch = nv <= 2 ? 1 : (sizeof (T) == 4 || nv <= (R == 2 ? 32 : 24) ? 2 : 4);
    FlatShape f = flat_shape_ch (nv, ch);
    while (ch > 1 && (S.nstrips + f.rpc - 1) / f.rpc < 2 * num_sms ()) {
      ch /= 2;
      f = flat_shape_ch (nv, ch);
    }
    auto run = [&] (auto chc) {
      k_strip_flat<T, R, decltype (chc)::value>
          <<<flat_grid (f, S.nstrips), FLAT_THREADS, 0, s>>> (
              S.n, S.nstrips, S.sptr, S.scol, sval, X + p0 * W, ldx, Y + p0 * W,
              ldy, nv, f.L, f.rpc);
    };
    if (ch == 1) run (std::integral_constant<int, 1> ());
    else if (ch == 2) run (std::integral_constant<int, 2> ());
    else if constexpr (sizeof (T) == 8) run (std::integral_constant<int, 4> ());
    LGH_LAUNCH_CHECK ();
  }
  return 0;
}

/* FP32, 8 rows: two packs per thread, one where there are no more than two
 * (256^2 x 5 columns: 75 us and 32) or some SM would not get its two CTAs
 * (64^2 x 60: 68 us and 42; 256^2 x 131, 547 CTAs: 88 us and 116) */
static int
strip_f32 (const StripForm &S, const float *X, int ldx, float *Y, int ldy,
           int nvec, cudaStream_t s)
{
  for (int p0 = 0; p0 < nvec; p0 += FLAT_THREADS) {
    const int nv = std::min (nvec - p0, FLAT_THREADS);
    FlatShape f = flat_shape_ch (nv, 2);
    int64_t ctas = (S.nstrips + f.rpc - 1) / f.rpc;
    if (nv <= 2 || ctas < 2 * num_sms ()) {
      f = flat_shape_ch (nv, 1);
      ctas = (S.nstrips + f.rpc - 1) / f.rpc;
    }
    LGH_CHECK (ctas < (int64_t) INT32_MAX, LGH_ERR_ARG_OUTOFRANGE,
               "strip product: grid too large");
    auto kern = f.ch == 2 ? k_strip_f32<2, 2> : k_strip_f32<1, 4>;
    kern<<<(unsigned) ctas, FLAT_THREADS, 0, s>>> (
        S.n, S.nstrips, S.sptr, S.scol, S.sval32, X + p0 * 4, ldx,
        Y + p0 * 4, ldy, nv, f.L, f.rpc);
    LGH_LAUNCH_CHECK ();
  }
  return 0;
}

template <typename T>
int
launch_strip_spmm (const StripForm &S, const T *X, int ldx, T *Y, int ldy,
                   int w, cudaStream_t s)
{
  constexpr int W = Pack<T>::W;
  LGH_CHECK (ldx % W == 0 && ldy % W == 0 && (uintptr_t) X % 16 == 0
             && (uintptr_t) Y % 16 == 0, LGH_ERR_ARG_WRONG,
             "strip product: blocks must be 16-byte aligned row-major");
  if (S.nstrips == 0 || w == 0) return 0;
  const int nvec = (w + W - 1) / W;
  /* FP32 blocks take the FP32 copy of the values (the mixed form) */
  const T *sv;
  if constexpr (sizeof (T) == 4) sv = S.sval32;
  else sv = S.sval;
  if (S.R == 2) return strip_flat<T, 2> (S, sv, X, ldx, Y, ldy, nvec, s);
  if (S.R == 4) return strip_flat<T, 4> (S, sv, X, ldx, Y, ldy, nvec, s);
  if constexpr (sizeof (T) == 4) {
    return strip_f32 (S, X, ldx, Y, ldy, nvec, s);
  } else {
    /* 112 columns per warp (the strip's columns and values read twice at
     * 220 columns) against 32: 1.42 ms and 1.68 at 512^2 x 220, so the wide
     * tile unless it pads a fifth more columns or leaves an SM with fewer
     * than 16 warps (64^2 x 60 columns: 36 us and 17.5).  Whole packs are
     * computed and stored, as everywhere. */
    const int wp = nvec * W, n14 = (wp + 111) / 112, n4 = (wp + 31) / 32;
    if (n14 * 112 * 5 > n4 * 32 * 6
        || S.nstrips * n14 < (int64_t) num_sms () * 16)
      return strip_mma<4, 2, 4> (S, X, ldx, Y, ldy, wp, s);
    return strip_mma<14, 2, 2> (S, X, ldx, Y, ldy, wp, s);
  }
}

template int launch_strip_spmm<double> (const StripForm &, const double *, int,
                                        double *, int, int, cudaStream_t);
template int launch_strip_spmm<float> (const StripForm &, const float *, int,
                                       float *, int, int, cudaStream_t);

} /* namespace lgh */
