/* k_pcg.cu -- the passes of blocked PCG around an explicit preconditioner
 * z = V(r) (the reference's per-column CG + PCGAMG, zsolve_impl.h:674-683,
 * 808-818), every column of the block with its own scalars and mask.
 *
 * One iteration is four passes over the block besides the V-cycle, 12 block
 * transfers: direction with the deferred x update (z, p, x in; p, x out: the
 * direction is formed in place), product with (p, q) (p gathered in, q
 * out), residual (r, q in; r out), dots (r, z in).  Column sums: a thread
 * keeps the sums of its packs over all its rows in registers, the CTA adds
 * its rows in shared memory, and the per-CTA partials are summed in a fixed
 * order, one warp per column.  Up to 32 columns the last CTA to finish does
 * that; wider blocks leave it to a small launch of one warp per column,
 * since one CTA takes 40 us over the 592 partials of 220 columns and the
 * launch 4 us (the whole product pass: 347 us with the last-CTA sum).  A
 * column's scalars load while its partials do, and the partials all at
 * once.
 *
 * The preconditioner's output may be FP32 (a mixed solve's float V-cycle):
 * the passes that read z widen it as they load it, which gives the values a
 * separate widening pass would have stored, and the residual pass stores
 * r's FP32 copy beside r.  Separate passes took 98 and 49 us of an
 * iteration's 1900 at 64^3 x 90 columns. */

#include <type_traits>

#include "lgh_flat.cuh"
#include "lgh_pcg.h"

namespace lgh
{

namespace
{

/* z packs: 16 bytes of T's width in elements, loaded from TZ */
template <typename T, typename TZ>
__device__ __forceinline__ Pack<T>
ldz (const TZ *p)
{
  if constexpr (std::is_same<T, TZ>::value) {
    return ldp (p);
  } else {
    static_assert (sizeof (T) == 8 && sizeof (TZ) == 4, "widening only");
    const float2 f = *reinterpret_cast<const float2 *> (p);
    Pack<T> r;
    r.v[0] = (T) f.x;
    r.v[1] = (T) f.y;
    return r;
  }
}

template <typename T>
__device__ __forceinline__ void
st32 (float *p, const Pack<T> &r)
{
  if constexpr (sizeof (T) == 8)
    *reinterpret_cast<float2 *> (p) = make_float2 ((float) r.v[0], (float) r.v[1]);
  else
    stp (p, r);
}

/* a thread's pack sums (NS of them) -> this CTA's column sums ->
 * part[q][c * grid + block].  red: NS rpc ld doubles and, behind them, 256
 * more. */
template <typename T, int CH, int NS>
__device__ __forceinline__ void
flat_colsum (const double (&acc)[NS][CH][Pack<T>::W], int rl, int lane, int L,
             int rpc, int nvec, int ld, double *red, double *partA,
             double *partB)
{
  constexpr int W = Pack<T>::W;
  const int cols = NS * ld;
  if (rl < rpc) {
#pragma unroll
    for (int q = 0; q < NS; q++)
#pragma unroll
      for (int h = 0; h < CH; h++) {
        const int vi = lane + h * L;
        if (h < CH - 1 || vi < nvec)
#pragma unroll
          for (int e = 0; e < W; e++)
            red[rl * cols + q * ld + vi * W + e] = acc[q][h][e];
      }
  }
  __syncthreads ();
  auto put = [&] (int c, double v) {
    double *part = NS == 1 || c < ld ? partA + (size_t) c * gridDim.x
                                     : partB + (size_t) (c - ld) * gridDim.x;
    part[blockIdx.x] = v;
  };
  /* narrow blocks hold many rows per CTA: nseg threads share a column */
  int nseg = 1;
  while (nseg < 16 && 2 * nseg * cols <= FLAT_THREADS) nseg *= 2;
  if (nseg == 1) {
    for (int c = threadIdx.x; c < cols; c += FLAT_THREADS) {
      double s = 0.;
#pragma unroll 4
      for (int r = 0; r < rpc; r++) s += red[r * cols + c];
      put (c, s);
    }
    return;
  }
  double *red2 = red + rpc * cols;
  const int seg = threadIdx.x / cols, c = threadIdx.x - seg * cols;
  if (seg < nseg) {
    double s = 0.;
#pragma unroll 4
    for (int r = seg; r < rpc; r += nseg) s += red[r * cols + c];
    red2[seg * cols + c] = s;
  }
  __syncthreads ();
  if (threadIdx.x < cols) {
    double s = 0.;
    for (int q = 0; q < nseg; q++) s += red2[q * cols + threadIdx.x];
    put (threadIdx.x, s);
  }
}

/* the sum of one column's nb partials by one warp, in a fixed order; the
 * loads of 512 partials go out together */
__device__ __forceinline__ double
part_sum (const double *part, int nb, int lane)
{
  double s = 0.;
  for (int b = lane; b < nb; b += 512) {
    double v[16];
#pragma unroll
    for (int q = 0; q < 16; q++)
      v[q] = b + 32 * q < nb ? __ldcg (part + b + 32 * q) : 0.;
#pragma unroll
    for (int d = 8; d > 0; d /= 2)
#pragma unroll
      for (int q = 0; q < d; q++) v[q] += v[q + d];
    s += v[0];
  }
  return warp_sum (s);
}

struct PcgCols
{
  double *scal;
  int *ival;
  int cap, w;
  double rtol;
  int first, iter;
  double *hist;
  const int *fresh;
  volatile int *host;   /* polled by the host: seq << 16 | active columns */
  int seq;

  /* a column's scalars, loaded before its partials are summed */
  struct Old
  {
    int act, fresh;
    double rz, n0;
  };
  __device__ Old load (int c, bool dots) const
  {
    Old o{ ival[I_ACTIVE * cap + c], 0, scal[S_RZ * cap + c], 0. };
    if (dots) {
      o.n0 = scal[S_NORM0 * cap + c];
      o.fresh = fresh != nullptr ? fresh[c] : 0;
    }
    return o;
  }

  /* alpha from (p, q) */
  __device__ int prod (int c, double pq, const Old &o) const
  {
    double al = 0.;
    if (o.act) {
      if (pq != 0. && isfinite (pq)) al = o.rz / pq;
      else ival[I_ACTIVE * cap + c] = 0;
    }
    scal[S_ALPHA * cap + c] = al;
    return 0;
  }

  /* the start of a column, or beta and the convergence test; returns
   * whether the column is active */
  __device__ int dots (int c, double srz, double szz, const Old &o) const
  {
    double *rz = scal + S_RZ * cap, *be = scal + S_BETA * cap;
    double *al = scal + S_ALPHA * cap, *n0 = scal + S_NORM0 * cap;
    int *act = ival + I_ACTIVE * cap, *its = ival + I_ITS * cap;
    if (first || o.fresh) {
      const int on = (c < w && szz > 0.) ? 1 : 0;
      rz[c] = srz;
      n0[c] = sqrt (szz);
      act[c] = on;
      al[c] = 0.;
      be[c] = 0.;
      its[c] = 0;
      return on;
    }
    if (!o.act) { be[c] = 0.; return 0; }
    const double b = (o.rz != 0.) ? srz / o.rz : 0.;
    if (hist != nullptr && c == 0 && iter < 10000) {
      hist[2 * iter] = al[0];
      hist[2 * iter + 1] = b;
    }
    rz[c] = srz;
    /* a converged column keeps its alpha: its x update may still be
     * pending (launch_pcg_dir or launch_pcg_out applies it), and the next
     * product zeroes alpha for inactive columns */
    if (sqrt (szz) <= rtol * o.n0 || srz == 0.) {
      act[c] = 0;
      be[c] = 0.;
      its[c] = iter + 1;
      return 0;
    }
    be[c] = b;
    return 1;
  }

  /* the count of active columns, to the device's slot and the host's */
  __device__ void report (int cnt) const
  {
    ival[I_NSLOT * cap] = cnt;
    if (host) *host = (int) (((unsigned) seq << 16) | (unsigned) cnt);
  }
};

/* columns up to which the last CTA sums the partials */
constexpr int PCG_TAIL_COLS = 32;

/* columns c0, c0 + cstep, ... of one warp; returns its active ones (lane 0) */
template <bool DOTS>
__device__ __forceinline__ int
pcg_columns (const double *partA, const double *partB, int nb, int c0, int cstep,
             int ld, const PcgCols &pc)
{
  const int lane = threadIdx.x & 31;
  int on = 0;
  for (int c = c0; c < ld; c += cstep) {
    const PcgCols::Old o = pc.load (c, DOTS);
    const double a = part_sum (partA + (size_t) c * nb, nb, lane);
    const double b = DOTS ? part_sum (partB + (size_t) c * nb, nb, lane) : 0.;
    if (lane == 0) on += DOTS ? pc.dots (c, a, b, o) : pc.prod (c, a, o);
  }
  return on;
}

/* the sum of the warps' lane 0 values, in thread 0 */
__device__ __forceinline__ int
warps_total (int v)
{
  __shared__ int sh[FLAT_THREADS / 32];
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = v;
  __syncthreads ();
  int t = 0;
  if (threadIdx.x == 0)
#pragma unroll
    for (int q = 0; q < FLAT_THREADS / 32; q++) t += sh[q];
  return t;
}

template <bool DOTS>
__device__ __forceinline__ void
pcg_tail (const double *partA, const double *partB, int ld, unsigned *counter,
          const PcgCols &pc)
{
  if (!last_block_ticket (counter)) return;
  const int on = pcg_columns<DOTS> (partA, partB, gridDim.x, threadIdx.x >> 5,
                                    FLAT_THREADS / 32, ld, pc);
  if (DOTS) {
    const int cnt = warps_total (on);
    if (threadIdx.x == 0) pc.report (cnt);
  }
  if (threadIdx.x == 0) *counter = 0u;
}

/* the partials of a wide block: one warp per column over all CTAs.  The
 * active columns are counted in the ticket itself (tickets above bit 16,
 * columns below), so the last CTA reads nothing back. */
template <bool DOTS>
__global__ void __launch_bounds__ (FLAT_THREADS)
k_pcg_columns (const double *partA, const double *partB, int nb, int ld,
               unsigned *counter, PcgCols pc)
{
  pdl_wait ();
  const int on = pcg_columns<DOTS> (
      partA, partB, nb,
      (int) (blockIdx.x * (FLAT_THREADS / 32) + (threadIdx.x >> 5)),
      (int) (gridDim.x * (FLAT_THREADS / 32)), ld, pc);
  if (!DOTS) return;
  const int cnt = warps_total (on);
  if (threadIdx.x == 0) {
    const unsigned t = atomicAdd (counter, (1u << 16) + (unsigned) cnt);
    if (t >> 16 == gridDim.x - 1) {
      *counter = 0u;
      pc.report ((int) (t & 0xffffu) + cnt);
    }
  }
}

/* ---- the passes ----------------------------------------------------------- */

template <typename T>
__global__ void __launch_bounds__ (256)
k_pcg_start (int64_t n, int w, int ld, const T *__restrict__ B, int ldb,
             const double *__restrict__ rs, T *__restrict__ R,
             float *__restrict__ R32, int vec)
{
  pdl_wait ();
  constexpr int W = Pack<T>::W;
  const int nvec = ld / W;
  const int64_t total = n * nvec;
  for (int64_t e = (int64_t) blockIdx.x * blockDim.x + threadIdx.x; e < total;
       e += (int64_t) gridDim.x * blockDim.x) {
    const int64_t i = e / nvec;
    const int c = (int) (e - i * nvec) * W;
    const double sc = rs ? rs[i] : 1.0;
    Pack<T> r;
    if (vec && c + W <= w) {
      r = ldp (B + i * ldb + c);
    } else {
      /* a single vector (ldb = 1), an unaligned view or the pad columns */
#pragma unroll
      for (int k = 0; k < W; k++) r.v[k] = c + k < w ? B[i * ldb + c + k] : T (0);
    }
#pragma unroll
    for (int k = 0; k < W; k++) r.v[k] = (T) (sc * (double) r.v[k]);
    stp (R + i * ld + c, r);
    if (R32) st32<T> (R32 + i * ld + c, r);
  }
}

template <typename T, typename TZ, int CH, bool TAIL>
__global__ void __launch_bounds__ (FLAT_THREADS, CH == 4 ? 3 : (CH == 2 ? 5 : 6))
k_pcg_dots (int64_t n, int ld, int nvec, int L, int rpc, const T *__restrict__ R,
            const TZ *__restrict__ Zb, double *partA, double *partB,
            unsigned *counter, PcgCols pc)
{
  pdl_wait ();
  constexpr int W = Pack<T>::W;
  extern __shared__ double red[];
  const int rl = threadIdx.x / L, lane = threadIdx.x - rl * L;
  double acc[2][CH][W];   /* (r, z), (z, z) */
  flat_zero<double, CH, W> (acc[0]);
  flat_zero<double, CH, W> (acc[1]);
  if (rl < rpc)
#pragma unroll (CH == 1 ? 4 : 1)
    for (int64_t i = (int64_t) blockIdx.x * rpc + rl; i < n;
         i += (int64_t) gridDim.x * rpc) {
#pragma unroll
      for (int h = 0; h < CH; h++) {
        const int vi = lane + h * L;
        if (h < CH - 1 || vi < nvec) {
          const Pack<T> r = ldp (R + i * ld + vi * W);
          const Pack<T> z = ldz<T, TZ> (Zb + i * ld + vi * W);
#pragma unroll
          for (int e = 0; e < W; e++) {
            acc[0][h][e] += (double) r.v[e] * (double) z.v[e];
            acc[1][h][e] += (double) z.v[e] * (double) z.v[e];
          }
        }
      }
    }
  flat_colsum<T, CH, 2> (acc, rl, lane, L, rpc, nvec, ld, red, partA, partB);
  if (TAIL) pcg_tail<true> (partA, partB, ld, counter, pc);
}

template <typename T, typename TZ, int FLAGS>
__global__ void __launch_bounds__ (256)
k_pcg_dir (int64_t n, int ld, const TZ *__restrict__ Zb, T *__restrict__ P,
           T *__restrict__ X, const double *__restrict__ beta,
           const double *__restrict__ alpha)
{
  pdl_wait ();
  constexpr int W = Pack<T>::W;
  const int nvec = ld / W;
  const int64_t total = n * nvec;
  for (int64_t e = (int64_t) blockIdx.x * blockDim.x + threadIdx.x; e < total;
       e += (int64_t) gridDim.x * blockDim.x) {
    const int64_t i = e / nvec;
    const int vi = (int) (e - i * nvec);
    const int64_t o = i * ld + vi * W;
    Pack<T> z = ldz<T, TZ> (Zb + o);
    if constexpr (!(FLAGS & PCG_P_FIRST)) {
      const Pack<T> p = ldp (P + o);
      Pack<T> x = (FLAGS & PCG_X_ADD) ? ldp (X + o) : pzero<T> ();
#pragma unroll
      for (int k = 0; k < W; k++)
        x.v[k] = fma ((T) alpha[vi * W + k], p.v[k], x.v[k]);
      stp (X + o, x);
#pragma unroll
      for (int k = 0; k < W; k++)
        z.v[k] = fma ((T) beta[vi * W + k], p.v[k], z.v[k]);
    }
    stp (P + o, z);
  }
}

/* 4 packs: 16 gather and 16 sum registers in 80 (3 CTAs per SM; 512^2 x 220
 * columns 250 us, 304 at 4 CTAs with spills, 299 with 2 packs).  I: entry
 * offsets in 32 bits, or 64 for an operator of 2^31 entries or more. */
template <typename T, typename I, int CH, bool TAIL>
__global__ void __launch_bounds__ (FLAT_THREADS, CH == 4 ? 3 : (CH == 2 ? 4 : 6))
k_pcg_prod (int64_t n, const int64_t *__restrict__ rowptr,
            const int32_t *__restrict__ colidx, const T *__restrict__ vals,
            const T *__restrict__ P, T *__restrict__ Q, int ld, int nvec, int L,
            int rpc, double *partA, unsigned *counter, PcgCols pc)
{
  pdl_wait ();
  constexpr int W = Pack<T>::W;
  extern __shared__ double red[];
  const int rl = threadIdx.x / L, lane = threadIdx.x - rl * L;
  const int64_t stride = (int64_t) gridDim.x * rpc;
  double apq[1][CH][W];
  flat_zero<double, CH, W> (apq[0]);
  int64_t i = (int64_t) blockIdx.x * rpc + rl;
  if (rl < rpc && i < n) {
    I k0 = (I) rowptr[i], k1 = (I) rowptr[i + 1];
    for (; i < n; i += stride) {
      I k0n = 0, k1n = 0;
      if (i + stride < n) {
        k0n = (I) rowptr[i + stride];
        k1n = (I) rowptr[i + stride + 1];
      }
      T acc[CH][W];
      flat_zero<T, CH, W> (acc);
      flat_gather<T, CH> (colidx, vals, k0, k1, 1, P, ld, lane, L, nvec, acc);
#pragma unroll
      for (int h = 0; h < CH; h++) {
        const int vi = lane + h * L;
        if (h < CH - 1 || vi < nvec) {
          const int64_t o = i * ld + vi * W;
          const Pack<T> p = ldp (P + o);
          Pack<T> q;
#pragma unroll
          for (int e = 0; e < W; e++) {
            q.v[e] = acc[h][e];
            apq[0][h][e] += (double) p.v[e] * (double) q.v[e];
          }
          stp (Q + o, q);
        }
      }
      k0 = k0n;
      k1 = k1n;
    }
  }
  flat_colsum<T, CH, 1> (apq, rl, lane, L, rpc, nvec, ld, red, partA, nullptr);
  if (TAIL) pcg_tail<false> (partA, nullptr, ld, counter, pc);
}

template <typename T>
__global__ void __launch_bounds__ (256)
k_pcg_resid (int64_t n, int ld, T *__restrict__ R, const T *__restrict__ Qv,
             float *__restrict__ R32, const double *__restrict__ alpha)
{
  pdl_wait ();
  constexpr int W = Pack<T>::W;
  const int nvec = ld / W;
  const int64_t total = n * nvec;
  for (int64_t e = (int64_t) blockIdx.x * blockDim.x + threadIdx.x; e < total;
       e += (int64_t) gridDim.x * blockDim.x) {
    const int64_t i = e / nvec;
    const int vi = (int) (e - i * nvec);
    const int64_t o = i * ld + vi * W;
    Pack<T> r = ldp (R + o);
    const Pack<T> q = ldp (Qv + o);
#pragma unroll
    for (int k = 0; k < W; k++)
      r.v[k] = fma (-(T) alpha[vi * W + k], q.v[k], r.v[k]);
    stp (R + o, r);
    if (R32) st32<T> (R32 + o, r);
  }
}

template <typename T>
__global__ void __launch_bounds__ (256)
k_pcg_out (int64_t n, int w, int ld, const T *__restrict__ X,
           const T *__restrict__ P, int have_x, const double *__restrict__ rs,
           T *__restrict__ Y, int ldy, const double *__restrict__ alpha, int vec)
{
  pdl_wait ();
  constexpr int W = Pack<T>::W;
  const int nvec = (w + W - 1) / W;
  const int64_t total = n * nvec;
  for (int64_t e = (int64_t) blockIdx.x * blockDim.x + threadIdx.x; e < total;
       e += (int64_t) gridDim.x * blockDim.x) {
    const int64_t i = e / nvec;
    const int c = (int) (e - i * nvec) * W;
    const double sc = rs ? rs[i] : 1.0;
    Pack<T> x = have_x ? ldp (X + i * ld + c) : pzero<T> ();
    if (P != nullptr) {
      const Pack<T> p = ldp (P + i * ld + c);
#pragma unroll
      for (int k = 0; k < W; k++) x.v[k] = fma ((T) alpha[c + k], p.v[k], x.v[k]);
    }
#pragma unroll
    for (int k = 0; k < W; k++) x.v[k] = (T) (sc * (double) x.v[k]);
    if (vec && c + W <= w) {
      stp (Y + i * ldy + c, x);
    } else {
#pragma unroll
      for (int k = 0; k < W; k++)
        if (c + k < w) Y[i * ldy + c + k] = x.v[k];
    }
  }
}

/* One step of the fixed-count iteration around an explicit preconditioner:
 * x += b z, r -= b Z z (first: x = b z); r is updated in place, row by row,
 * from the gathered z: 5 block transfers (7 with an x, d and r written
 * beside the old ones: 37 us at 257 x 255 x 48 columns).  The product is of
 * b z as it is rounded, which r has to follow: with b times the product of
 * z the error of FP32 solves was 3 to 10 % larger.  With z = V(r) and
 * the Chebyshev recurrence's step lengths b this is the short form of
 * zsolve_block, without the recurrence's direction term; with the direction
 * in z's place and b = 1 it is a Chebyshev step. */
template <typename T, typename I, int CH, bool FIRST>
__global__ void __launch_bounds__ (FLAT_THREADS, FlatOcc<CH>::v)
k_pcg_cheb (int64_t n, const int64_t *__restrict__ rowptr,
            const int32_t *__restrict__ colidx, const T *__restrict__ vals,
            const T *__restrict__ Zb, T *__restrict__ R, T *__restrict__ X,
            int ld, int nvec, int L, int rpc, T b)
{
  pdl_wait ();
  constexpr int W = Pack<T>::W;
  const int rl = threadIdx.x / L, lane = threadIdx.x - rl * L;
  const int64_t stride = (int64_t) gridDim.x * rpc;
  int64_t i = (int64_t) blockIdx.x * rpc + rl;
  if (rl >= rpc || i >= n) return;
  I k0 = (I) rowptr[i], k1 = (I) rowptr[i + 1];
  for (; i < n; i += stride) {
    I k0n = 0, k1n = 0;
    if (i + stride < n) {
      k0n = (I) rowptr[i + stride];
      k1n = (I) rowptr[i + stride + 1];
    }
    T acc[CH][W];
    flat_zero<T, CH, W> (acc);
    flat_gather<T, CH, true> (colidx, vals, k0, k1, 1, Zb, ld, lane, L, nvec, acc, b);
#pragma unroll
    for (int h = 0; h < CH; h++) {
      const int vi = lane + h * L;
      if (h < CH - 1 || vi < nvec) {
        const int64_t o = i * ld + vi * W;
        const Pack<T> z = ldp (Zb + o);
        Pack<T> r = ldp (R + o), x = FIRST ? pzero<T> () : ldp (X + o);
#pragma unroll
        for (int e = 0; e < W; e++) {
          x.v[e] = fma (b, z.v[e], x.v[e]);
          r.v[e] -= acc[h][e];
        }
        stp (X + o, x);
        stp (R + o, r);
      }
    }
    k0 = k0n;
    k1 = k1n;
  }
}

/* the Chebyshev direction, in place: p = a p + b z (first: p = b z) */
template <typename T>
__global__ void __launch_bounds__ (256)
k_pcg_cheb_dir (int64_t n, int ld, const T *__restrict__ Zb, T *__restrict__ P,
                T a, T b, int first)
{
  pdl_wait ();
  constexpr int W = Pack<T>::W;
  const int64_t total = n * (ld / W);
  for (int64_t e = (int64_t) blockIdx.x * blockDim.x + threadIdx.x; e < total;
       e += (int64_t) gridDim.x * blockDim.x) {
    const Pack<T> z = ldp (Zb + e * W);
    Pack<T> p = first ? pzero<T> () : ldp (P + e * W);
#pragma unroll
    for (int k = 0; k < W; k++) p.v[k] = fma (b, z.v[k], a * p.v[k]);
    stp (P + e * W, p);
  }
}

/* the last step with the row scaling, Y = S (x + b z) over the w columns:
 * its residual is not needed, so there is no product.  only: it is also
 * the first (x = 0). */
template <typename T>
__global__ void __launch_bounds__ (256)
k_pcg_cheb_out (int64_t n, int w, int ld, const T *__restrict__ Zb,
                const T *__restrict__ X, T b, int only,
                const double *__restrict__ rs, T *__restrict__ Y, int ldy,
                int vec)
{
  pdl_wait ();
  constexpr int W = Pack<T>::W;
  const int nvec = (w + W - 1) / W;
  const int64_t total = n * nvec;
  for (int64_t e = (int64_t) blockIdx.x * blockDim.x + threadIdx.x; e < total;
       e += (int64_t) gridDim.x * blockDim.x) {
    const int64_t i = e / nvec;
    const int c = (int) (e - i * nvec) * W;
    const double sc = rs ? rs[i] : 1.0;
    const Pack<T> z = ldp (Zb + i * ld + c);
    Pack<T> x = only ? pzero<T> () : ldp (X + i * ld + c);
#pragma unroll
    for (int k = 0; k < W; k++)
      x.v[k] = (T) (sc * (double) fma (b, z.v[k], x.v[k]));
    if (vec && c + W <= w) {
      stp (Y + i * ldy + c, x);
    } else {
#pragma unroll
      for (int k = 0; k < W; k++)
        if (c + k < w) Y[i * ldy + c + k] = x.v[k];
    }
  }
}

/* CTAs of a streaming pass of `total` packs */
int
stream_grid (int64_t total)
{
  return (int) std::max<int64_t> (1, std::min<int64_t> (
      (int64_t) num_sms () * 8, (total + 255) / 256));
}

/* two packs per thread at most: the sums, not the loads, set the registers */
FlatShape
sum_shape (int nvec, int64_t n)
{
  FlatShape f = flat_shape (nvec, n);
  if (f.ch == 4 && (nvec + 1) / 2 <= FLAT_THREADS) f = flat_shape_ch (nvec, 2);
  return f;
}

int
sum_smem (const FlatShape &f, int cols)
{
  return (f.rpc * cols + FLAT_THREADS) * (int) sizeof (double);
}

/* two packs per thread at most: the column sums fit the 48 KB of shared
 * memory that need no opt-in (a Z-solve's tile is 512 columns) */
int
pcg_width (int ld, int W)
{
  return ld > 0 && ld % W == 0 && ld / W <= 2 * FLAT_THREADS
             ? 0
             : set_error (LGH_ERR_SUP, "PCG pass: block width %d unsupported", ld);
}

} /* namespace */

template <typename T>
int
launch_pcg_start (int64_t n, int w, int ld, const T *B, int ldb,
                  const double *rs, T *R, float *R32, cudaStream_t s)
{
  const int64_t bytes = n * ld * (int64_t) sizeof (T);
  constexpr int W = Pack<T>::W;
  const int vec = ldb % W == 0 && (uintptr_t) B % 16 == 0;
  LGH_CUDA (launch_pdl (bytes, k_pcg_start<T>, stream_grid (n * (ld / W)), 256, 0, s,
      n, w, ld, B, ldb, rs, R, R32, vec));
  LGH_LAUNCH_CHECK ();
  return 0;
}

template <typename T, typename TZ>
int
launch_pcg_dots (int64_t n, int w, int ld, const T *R, const TZ *Zb, int first,
                 double rtol, int iter, double *hist, const int *fresh,
                 ZWork &ws, cudaStream_t s, int report)
{
  const int64_t bytes = n * ld * (int64_t) sizeof (T);
  constexpr int W = Pack<T>::W;
  LGH_TRY (pcg_width (ld, W));
  const int nvec = ld / W;
  const FlatShape f = sum_shape (nvec, n);
  const int smem = sum_smem (f, 2 * ld);
  /* one pack per thread and the last CTA's sum: two CTAs per SM, four rows
   * in flight each, leave it few partials */
  const int want = std::min (flat_grid (f, n), f.ch == 1 && ld <= PCG_TAIL_COLS
                                                   ? 2 * num_sms () : ws.nblocks);
  if (report) ws.nact.seq = (ws.nact.seq + 1) & 0x7fff;
  const PcgCols pc{ ws.scal.p, ws.ival.p, ws.cap, w, rtol, first, iter, hist,
                    fresh, report ? ws.nact.p : nullptr, ws.nact.seq };
  int nb = 0;
  LGH_FLAT_DISPATCH (f.ch, {
    if (ld <= PCG_TAIL_COLS) {
      auto k = k_pcg_dots<T, TZ, CH_, true>;
      LGH_CUDA (launch_pdl (bytes, k, fit_grid (k, want, FLAT_THREADS, smem),
          FLAT_THREADS, smem, s, n, ld, nvec, f.L, f.rpc, R, Zb, ws.partA.p,
          ws.partB.p, ws.counters.p + 1, pc));
    } else {
      auto k = k_pcg_dots<T, TZ, CH_, false>;
      nb = fit_grid (k, want, FLAT_THREADS, smem);
      LGH_CUDA (launch_pdl (bytes, k, nb, FLAT_THREADS, smem, s, n, ld, nvec, f.L,
          f.rpc, R, Zb, ws.partA.p, ws.partB.p, ws.counters.p + 1, pc));
    }
  });
  LGH_LAUNCH_CHECK ();
  if (nb > 0) {
    LGH_CUDA (launch_pdl (0, k_pcg_columns<true>, (ld + 7) / 8, FLAT_THREADS, 0,
        s, ws.partA.p, ws.partB.p, nb, ld, ws.counters.p + 1, pc));
    LGH_LAUNCH_CHECK ();
  }
  return 0;
}

template <typename T, typename TZ>
int
launch_pcg_dir (int64_t n, int ld, const TZ *Zb, T *P, T *X, int flags,
                ZWork &ws, cudaStream_t s)
{
  const int64_t bytes = n * ld * (int64_t) sizeof (T);
  constexpr int W = Pack<T>::W;
  const int grid = stream_grid (n * (ld / W));
  const double *be = ws.scal.p + S_BETA * ws.cap, *al = ws.scal.p + S_ALPHA * ws.cap;
  switch (flags) {
  case PCG_P_FIRST:
    LGH_CUDA (launch_pdl (bytes, k_pcg_dir<T, TZ, PCG_P_FIRST>, grid, 256, 0, s, n,
        ld, Zb, P, X, be, al));
    break;
  case PCG_X_FIRST:
    LGH_CUDA (launch_pdl (bytes, k_pcg_dir<T, TZ, PCG_X_FIRST>, grid, 256, 0, s, n,
        ld, Zb, P, X, be, al));
    break;
  case PCG_X_ADD:
    LGH_CUDA (launch_pdl (bytes, k_pcg_dir<T, TZ, PCG_X_ADD>, grid, 256, 0, s, n, ld,
        Zb, P, X, be, al));
    break;
  default:
    return set_error (LGH_ERR_ARG_WRONG, "PCG direction: flags %d", flags);
  }
  LGH_LAUNCH_CHECK ();
  return 0;
}

template <typename T>
int
launch_pcg_prod (const Csr &Z, const T *P, T *Q, int ld, ZWork &ws,
                 cudaStream_t s)
{
  const int64_t bytes = Z.n * ld * (int64_t) sizeof (T);
  constexpr int W = Pack<T>::W;
  LGH_TRY (pcg_width (ld, W));
  const T *vals;
  if constexpr (std::is_same<T, double>::value) vals = Z.vals;
  else vals = Z.vals32;
  const int nvec = ld / W;
  const FlatShape f = flat_shape (nvec, Z.n);
  const int smem = sum_smem (f, ld);
  const int want = std::min (flat_grid (f, Z.n), ws.nblocks);
  const PcgCols pc{ ws.scal.p, ws.ival.p, ws.cap, 0, 0., 0, 0, nullptr, nullptr,
                    nullptr, 0 };
  int nb = 0;
  auto run = [&] (auto idx, auto ch, auto tail) -> int {
    auto k = k_pcg_prod<T, decltype (idx), decltype (ch)::value,
                        decltype (tail)::value>;
    const int g = fit_grid (k, want, FLAT_THREADS, smem);
    if (!decltype (tail)::value) nb = g;
    LGH_CUDA (launch_pdl (bytes, k, g, FLAT_THREADS, smem, s, Z.n, Z.rowptr,
        Z.colidx, vals, P, Q, ld, nvec, f.L, f.rpc, ws.partA.p, ws.counters.p,
        pc));
    LGH_LAUNCH_CHECK ();
    return 0;
  };
  const bool tail = ld <= PCG_TAIL_COLS, big = Z.nnz >= FLAT_NNZ_MAX;
  LGH_FLAT_DISPATCH (f.ch, {
    using C = std::integral_constant<int, CH_>;
    if (big) {
      if (tail) LGH_TRY (run (int64_t (), C (), std::true_type ()));
      else LGH_TRY (run (int64_t (), C (), std::false_type ()));
    } else {
      if (tail) LGH_TRY (run (int (), C (), std::true_type ()));
      else LGH_TRY (run (int (), C (), std::false_type ()));
    }
  });
  if (nb > 0) {
    LGH_CUDA (launch_pdl (0, k_pcg_columns<false>, (ld + 7) / 8, FLAT_THREADS, 0,
        s, ws.partA.p, nullptr, nb, ld, ws.counters.p, pc));
    LGH_LAUNCH_CHECK ();
  }
  return 0;
}

template <typename T>
int
launch_pcg_resid (int64_t n, int ld, T *R, const T *Q, float *R32, ZWork &ws,
                  cudaStream_t s)
{
  const int64_t bytes = n * ld * (int64_t) sizeof (T);
  const int grid = stream_grid (n * (ld / Pack<T>::W));
  const double *al = ws.scal.p + S_ALPHA * ws.cap;
  LGH_CUDA (launch_pdl (bytes, k_pcg_resid<T>, grid, 256, 0, s, n, ld, R, Q, R32,
      al));
  LGH_LAUNCH_CHECK ();
  return 0;
}

template <typename T>
int
launch_pcg_out (int64_t n, int w, int ld, const T *X, const T *P, int have_x,
                const double *rs, T *Y, int ldy, ZWork &ws, cudaStream_t s)
{
  const int64_t bytes = n * ld * (int64_t) sizeof (T);
  constexpr int W = Pack<T>::W;
  const int vec = ldy % W == 0 && (uintptr_t) Y % 16 == 0;
  LGH_CUDA (launch_pdl (bytes, k_pcg_out<T>, stream_grid (n * ((w + W - 1) / W)),
      256, 0, s, n, w, ld, X, P, have_x, rs, Y, ldy,
      ws.scal.p + S_ALPHA * ws.cap, vec));
  LGH_LAUNCH_CHECK ();
  return 0;
}

template <typename T>
int
launch_pcg_cheb (const Csr &Z, const T *Zb, T *R, T *X, int ld, double b,
                 int first, cudaStream_t s)
{
  constexpr int W = Pack<T>::W;
  LGH_TRY (pcg_width (ld, W));
  const int64_t bytes = Z.n * ld * (int64_t) sizeof (T);
  const T *vals;
  if constexpr (std::is_same<T, double>::value) vals = Z.vals;
  else vals = Z.vals32;
  const int nvec = ld / W;
  const FlatShape f = flat_shape (nvec, Z.n);
  auto run = [&] (auto idx, auto ch, auto fst) -> int {
    auto k = k_pcg_cheb<T, decltype (idx), decltype (ch)::value,
                        decltype (fst)::value>;
    LGH_CUDA (launch_pdl (bytes, k,
        fit_grid (k, flat_grid (f, Z.n), FLAT_THREADS, 0), FLAT_THREADS, 0, s,
        Z.n, Z.rowptr, Z.colidx, vals, Zb, R, X, ld, nvec, f.L, f.rpc, (T) b));
    LGH_LAUNCH_CHECK ();
    return 0;
  };
  const bool big = Z.nnz >= FLAT_NNZ_MAX;
  LGH_FLAT_DISPATCH (f.ch, {
    using C = std::integral_constant<int, CH_>;
    if (big) {
      if (first) LGH_TRY (run (int64_t (), C (), std::true_type ()));
      else LGH_TRY (run (int64_t (), C (), std::false_type ()));
    } else {
      if (first) LGH_TRY (run (int (), C (), std::true_type ()));
      else LGH_TRY (run (int (), C (), std::false_type ()));
    }
  });
  return 0;
}

template <typename T>
int
launch_pcg_cheb_dir (int64_t n, int ld, const T *Zb, T *P, double a, double b,
                     int first, cudaStream_t s)
{
  const int64_t bytes = n * ld * (int64_t) sizeof (T);
  LGH_CUDA (launch_pdl (bytes, k_pcg_cheb_dir<T>, stream_grid (n * (ld / Pack<T>::W)),
      256, 0, s, n, ld, Zb, P, (T) a, (T) b, first));
  LGH_LAUNCH_CHECK ();
  return 0;
}

template <typename T>
int
launch_pcg_cheb_out (int64_t n, int w, int ld, const T *Zb, const T *X, double b,
                     int only, const double *rs, T *Y, int ldy, cudaStream_t s)
{
  constexpr int W = Pack<T>::W;
  const int64_t bytes = n * ld * (int64_t) sizeof (T);
  const int vec = ldy % W == 0 && (uintptr_t) Y % 16 == 0;
  LGH_CUDA (launch_pdl (bytes, k_pcg_cheb_out<T>,
      stream_grid (n * ((w + W - 1) / W)), 256, 0, s, n, w, ld, Zb, X, (T) b,
      only, rs, Y, ldy, vec));
  LGH_LAUNCH_CHECK ();
  return 0;
}

/* the active columns of the last reported dots: the host spins on the flag
 * that its kernel writes, a few us after the write; a copy of the count and
 * a synchronisation left the device idle for 31 us a look.  Now and then it
 * asks the stream, so that a failed launch ends the wait. */
int
pcg_wait_count (ZWork &ws, cudaStream_t s, int *count)
{
  if (!ws.nact.p) {
    LGH_CUDA (cudaMemcpyAsync (count, ws.ival.p + I_NSLOT * ws.cap, sizeof (int),
                               cudaMemcpyDeviceToHost, s));
    LGH_CUDA (cudaStreamSynchronize (s));
    return 0;
  }
  auto seen = [&] () {
    const unsigned v = (unsigned) *ws.nact.p;
    if ((int) (v >> 16) != ws.nact.seq) return false;
    *count = (int) (v & 0xffffu);
    return true;
  };
  for (long spin = 1;; spin++) {
    if (seen ()) return 0;
    if (spin % 4096 == 0) {
      const cudaError_t e = cudaStreamQuery (s);
      if (e == cudaSuccess) {
        if (seen ()) return 0;
        return set_error (LGH_ERR_GPU, "zsolve: the column count did not arrive");
      }
      if (e != cudaErrorNotReady)
        return set_error (LGH_ERR_GPU, "zsolve: %s", cudaGetErrorString (e));
      cudaGetLastError ();
    }
  }
}

#define LGH_PCG_INST(T)                                                      \
  template int launch_pcg_start<T> (int64_t, int, int, const T *, int,       \
                                    const double *, T *, float *,            \
                                    cudaStream_t);                           \
  template int launch_pcg_prod<T> (const Csr &, const T *, T *, int,         \
                                   ZWork &, cudaStream_t);                   \
  template int launch_pcg_resid<T> (int64_t, int, T *, const T *, float *,   \
                                    ZWork &, cudaStream_t);                  \
  template int launch_pcg_out<T> (int64_t, int, int, const T *, const T *,   \
                                  int, const double *, T *, int, ZWork &,    \
                                  cudaStream_t);
#define LGH_PCG_INST_C(T)                                                    \
  template int launch_pcg_cheb<T> (const Csr &, const T *, T *, T *, int,    \
                                   double, int, cudaStream_t);               \
  template int launch_pcg_cheb_dir<T> (int64_t, int, const T *, T *, double, \
                                       double, int, cudaStream_t);           \
  template int launch_pcg_cheb_out<T> (int64_t, int, int, const T *,         \
                                       const T *, double, int,               \
                                       const double *, T *, int,             \
                                       cudaStream_t);
LGH_PCG_INST_C (double)
LGH_PCG_INST_C (float)
#undef LGH_PCG_INST_C
#define LGH_PCG_INST_Z(T, TZ)                                                \
  template int launch_pcg_dots<T, TZ> (int64_t, int, int, const T *,         \
                                       const TZ *, int, double, int,         \
                                       double *, const int *, ZWork &,       \
                                       cudaStream_t, int);                        \
  template int launch_pcg_dir<T, TZ> (int64_t, int, const TZ *, T *, T *,    \
                                      int, ZWork &, cudaStream_t);
LGH_PCG_INST (double)
LGH_PCG_INST (float)
LGH_PCG_INST_Z (double, double)
LGH_PCG_INST_Z (double, float)
LGH_PCG_INST_Z (float, float)
#undef LGH_PCG_INST
#undef LGH_PCG_INST_Z

} /* namespace lgh */
