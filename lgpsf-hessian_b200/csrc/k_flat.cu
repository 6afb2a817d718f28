/* k_flat.cu -- the V-cycle's passes over one smoothed level, in the flat
 * row mapping (lgh_flat.cuh).
 *
 * With S the two-step Chebyshev-Jacobi smoother (from zero: S r =
 * D^{-1} ((g + b2) r - b2 F1 r), F1 = b1 A D^{-1}, g = b1 (1 + a2)), the
 * level's V-cycle on a right-hand side r0 is
 *   r1 = r0 - F1 r0                     the first step's residual
 *   r2 = r1 - a2 (r0 - r1) - (b2 / b1) F1 r1    the second step's residual
 *   xc = V_coarse (P^T r2)
 *   z  = S r0 + S r2 + (I - S A) P xc
 *      = D^{-1} (g (r0 + r2) + b2 (r1 + r2 - F1 r2)) + Q xc,
 * the same operator as pre-smoothing, coarse correction, residual refresh
 * and post-smoothing done one after the other.  Q = (I - S A) P is formed
 * once at set-up, so neither the iterate before the correction nor the
 * residual after it is ever stored, and each pass gathers one fine block:
 * in the second step A d2 = a2 A d1 + b2 A D^{-1} r1, and A d1 = r0 - r1
 * is at hand, so r1 alone is gathered where d2 = a2 d1 + b2 D^{-1} r1 was.
 * Block passes: 2 + 3 + 4 (and the coarse blocks), against 2 + 4 + 2 + 3
 * with the stored iterate.  All four are bound by L1 wavefronts at the
 * residency their registers allow (lgh_flat.cuh); I is the type of entry
 * offsets, 64 bits only for operators of 2^31 entries; each kernel gives its
 * time at 512^2 x 220 columns FP64 on the finest level, its floor at the
 * measured HBM rate and what the passes it replaces took. */

#include <type_traits>

#include "lgh_flat.cuh"
#include "lgh_internal.h"

namespace lgh
{

/* Y = B - A X (first step: X = B = r0): 180 us, floor 141; a row per power
 * of two of lanes with shuffled entries 247 */
template <typename T, typename I, int CH>
__global__ void __launch_bounds__ (FLAT_THREADS, FlatOcc<CH>::v)
k_flat_resid (int64_t n, const int64_t *__restrict__ rowptr,
              const int32_t *__restrict__ colidx, const T *__restrict__ vals,
              const T *__restrict__ X, const T *__restrict__ B,
              T *__restrict__ Y, int ld, int nvec, int L, int rpc)
{
  pdl_wait ();
  constexpr int W = Pack<T>::W;
  const int rl = threadIdx.x / L, lane = threadIdx.x - rl * L;
  const int64_t stride = (int64_t) gridDim.x * rpc;
  int64_t i = (int64_t) blockIdx.x * rpc + rl;
  if (rl >= rpc || i >= n) return;
  I k0 = (I) rowptr[i], k1 = (I) rowptr[i + 1];
  for (; i < n; i += stride) {
    /* the next row's bounds load during this row's gathers */
    I k0n = 0, k1n = 0;
    if (i + stride < n) {
      k0n = (I) rowptr[i + stride];
      k1n = (I) rowptr[i + stride + 1];
    }
    T acc[CH][W];
    flat_zero<T, CH, W> (acc);
    flat_gather<T, CH> (colidx, vals, k0, k1, 1, X, ld, lane, L, nvec, acc);
#pragma unroll
    for (int h = 0; h < CH; h++) {
      const int vi = lane + h * L;
      if (h < CH - 1 || vi < nvec) {
        const int64_t o = i * ld + vi * W;
        Pack<T> b = ldp (B + o);
#pragma unroll
        for (int e = 0; e < W; e++) b.v[e] -= acc[h][e];
        stp (Y + o, b);
      }
    }
    k0 = k0n;
    k1 = k1n;
  }
}

/* r2 = r1 - a2 (r0 - r1) - s2 F1 r1 (s2 = b2 / b1): reads r1 (gathered)
 * and r0, writes r2.  280 us, floor 211; with d and x re-formed from two
 * gathered blocks 580 */
template <typename T, typename I, int CH>
__global__ void __launch_bounds__ (FLAT_THREADS, FlatOcc<CH>::v)
k_flat_second (int64_t n, const int64_t *__restrict__ rowptr,
               const int32_t *__restrict__ colidx, const T *__restrict__ vals,
               const T *__restrict__ R0, const T *__restrict__ R1,
               T *__restrict__ R2, int ld, int nvec, int L, int rpc, T a2,
               T s2)
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
    flat_gather<T, CH> (colidx, vals, k0, k1, 1, R1, ld, lane, L, nvec, acc);
#pragma unroll
    for (int h = 0; h < CH; h++) {
      const int vi = lane + h * L;
      if (h < CH - 1 || vi < nvec) {
        const int64_t o = i * ld + vi * W;
        const Pack<T> r0 = ldp (R0 + o);
        Pack<T> r = ldp (R1 + o);
#pragma unroll
        for (int e = 0; e < W; e++) {
          const T t = fma (-a2, r0.v[e] - r.v[e], r.v[e]);
          r.v[e] = fma (-s2, acc[h][e], t);
        }
        stp (R2 + o, r);
      }
    }
    k0 = k0n;
    k1 = k1n;
  }
}

/* z = dinv (g (r0 + r2) + b2 (r1 + r2 - F1 r2)) + Q xc: reads r0, r1, r2
 * (gathered) and the coarse block (gathered), writes z.  487 us in a job
 * (470 alone), floor 297; the post residual and the two post-smoothing steps
 * took 787 */
template <typename T, typename I, int CH>
__global__ void __launch_bounds__ (FLAT_THREADS, CH == 2 ? 5 : (CH == 3 ? 4 : FlatOcc<CH>::v))
k_flat_finish (int64_t n, const int64_t *__restrict__ frp,
               const int32_t *__restrict__ fci, const T *__restrict__ fv,
               const int64_t *__restrict__ qrp,
               const int32_t *__restrict__ qci, const T *__restrict__ qv,
               const T *__restrict__ dinv, const T *__restrict__ R0,
               const T *__restrict__ R1, const T *__restrict__ R2,
               const T *__restrict__ Xc, T *__restrict__ Z, int ld, int nvec,
               int L, int rpc, T g, T b2)
{
  pdl_wait ();
  constexpr int W = Pack<T>::W;
  const int rl = threadIdx.x / L, lane = threadIdx.x - rl * L;
  const int64_t stride = (int64_t) gridDim.x * rpc;
  int64_t i = (int64_t) blockIdx.x * rpc + rl;
  if (rl >= rpc || i >= n) return;
  I k0 = (I) frp[i], k1 = (I) frp[i + 1];
  I q0 = (I) qrp[i], q1 = (I) qrp[i + 1];
  for (; i < n; i += stride) {
    I k0n = 0, k1n = 0, q0n = 0, q1n = 0;
    if (i + stride < n) {
      k0n = (I) frp[i + stride];
      k1n = (I) frp[i + stride + 1];
      q0n = (I) qrp[i + stride];
      q1n = (I) qrp[i + stride + 1];
    }
    T acc[CH][W];
    flat_zero<T, CH, W> (acc);
    flat_gather<T, CH> (fci, fv, k0, k1, 1, R2, ld, lane, L, nvec, acc);
    const T di = dinv[i];
#pragma unroll
    for (int h = 0; h < CH; h++) {
      const int vi = lane + h * L;
      if (h < CH - 1 || vi < nvec) {
        const int64_t o = i * ld + vi * W;
        const Pack<T> r0 = ldp (R0 + o), r1 = ldp (R1 + o), r2 = ldp (R2 + o);
#pragma unroll
        for (int e = 0; e < W; e++) {
          const T u = b2 * ((r1.v[e] + r2.v[e]) - acc[h][e]);
          acc[h][e] = di * fma (g, r0.v[e] + r2.v[e], u);
        }
      }
    }
    flat_gather<T, CH> (qci, qv, q0, q1, 1, Xc, ld, lane, L, nvec, acc);
#pragma unroll
    for (int h = 0; h < CH; h++) {
      const int vi = lane + h * L;
      if (h < CH - 1 || vi < nvec) {
        Pack<T> z;
#pragma unroll
        for (int e = 0; e < W; e++) z.v[e] = acc[h][e];
        stp (Z + i * ld + vi * W, z);
      }
    }
    k0 = k0n;
    k1 = k1n;
    q0 = q0n;
    q1 = q1n;
  }
}

/* Y = A X for the restriction P^T: its rows hold 15 (2D) to 230 (3D)
 * entries and there are few of them on the lower levels, so a row's
 * entries are dealt out to S neighbouring thread groups of the CTA, whose
 * sums are added in group order through shared memory.  128 us for the
 * finest level's, 154 with a warp group per row */
template <typename T, typename I, int CH, bool SPLIT>
__global__ void __launch_bounds__ (FLAT_THREADS, FlatOcc<CH>::v)
k_flat_mult (int64_t n, const int64_t *__restrict__ rowptr,
             const int32_t *__restrict__ colidx, const T *__restrict__ vals,
             const T *__restrict__ X, T *__restrict__ Y, int ld, int nvec,
             int L, int rows, int S)
{
  pdl_wait ();
  constexpr int W = Pack<T>::W;
  extern __shared__ __align__ (16) unsigned char smem[];
  T *part = reinterpret_cast<T *> (smem);   /* [rows * S][nvec * W] */
  const int grp = threadIdx.x / L, lane = threadIdx.x - grp * L;
  const int rl = SPLIT ? grp / S : grp, sp = SPLIT ? grp - rl * S : 0;
  for (int64_t i0 = (int64_t) blockIdx.x * rows; i0 < n;
       i0 += (int64_t) gridDim.x * rows) {
    const int64_t i = i0 + rl;
    const bool on = rl < rows && i < n;
    T acc[CH][W];
    flat_zero<T, CH, W> (acc);
    if (on) {
      flat_gather<T, CH> (colidx, vals, (I) rowptr[i] + sp, (I) rowptr[i + 1],
                          SPLIT ? S : 1, X, ld, lane, L, nvec, acc);
    }
    if constexpr (SPLIT) {
      if (on && sp > 0) {
#pragma unroll
        for (int h = 0; h < CH; h++) {
          const int vi = lane + h * L;
          if (h < CH - 1 || vi < nvec) {
            Pack<T> p;
#pragma unroll
            for (int e = 0; e < W; e++) p.v[e] = acc[h][e];
            stp (part + ((int64_t) grp * nvec + vi) * W, p);
          }
        }
      }
      __syncthreads ();
      if (on && sp == 0) {
        for (int q = 1; q < S; q++)
#pragma unroll
          for (int h = 0; h < CH; h++) {
            const int vi = lane + h * L;
            if (h < CH - 1 || vi < nvec) {
              const Pack<T> p = ldp (part + ((int64_t) (grp + q) * nvec + vi) * W);
#pragma unroll
              for (int e = 0; e < W; e++) acc[h][e] += p.v[e];
            }
          }
      }
    }
    if (on && sp == 0) {
#pragma unroll
      for (int h = 0; h < CH; h++) {
        const int vi = lane + h * L;
        if (h < CH - 1 || vi < nvec) {
          Pack<T> p;
#pragma unroll
          for (int e = 0; e < W; e++) p.v[e] = acc[h][e];
          stp (Y + i * ld + vi * W, p);
        }
      }
    }
    if constexpr (SPLIT) __syncthreads ();
  }
}

/* ---- host side ------------------------------------------------------------ */

template <typename T>
static const T *
fvals (const Csr &A)
{
  if constexpr (std::is_same<T, double>::value) return A.vals;
  else return A.vals32;
}

/* Column slices: a gathered row is read again by the rows up to the
 * operator's bandwidth away, so the band of 2 bandwidth rows has to stay in
 * L2 (126 MB, shared with the streams); a band wider than the smoothers'
 * budget (smoother_l2_budget) is swept in slices of whole packs.  f (first
 * pack, packs) runs one slice. */
template <typename F>
static int
flat_slices (int64_t n, int64_t bandwidth, int ld, int nvec, size_t elem, F f)
{
  const double band = (double) std::min (2 * bandwidth, n) * ld * elem;
  /* a single vector's band is a few KB: no look at the override */
  const double budget = band > 16384. ? smoother_l2_budget () : 0.;
  int ns = (nvec + FLAT_MAXPACKS - 1) / FLAT_MAXPACKS;
  if (budget > 0. && band > budget)
    ns = std::max (ns, (int) std::min ((double) nvec, band / budget + 1.));
  for (int s = 0; s < ns; s++) {
    const int v0 = (int) ((int64_t) nvec * s / ns);
    const int v1 = (int) ((int64_t) nvec * (s + 1) / ns);
    if (v1 > v0) LGH_TRY (f (v0, v1 - v0));
  }
  return 0;
}

template <typename T>
static int
flat_check (const Csr &A, const void *a, const void *b, const void *c, int ld)
{
  if (fvals<T> (A) == nullptr || ld <= 0 || ld % Pack<T>::W
      || (uintptr_t) a % 16 || (uintptr_t) b % 16 || (uintptr_t) c % 16)
    return set_error (LGH_ERR_ARG_WRONG, "V-cycle pass: needs an operator's "
                      "values and 16-byte aligned row-major blocks");
  return 0;
}

template <typename T>
int
launch_vc_first (const Csr &F1, const T *R0, T *R1, int ld, cudaStream_t s,
                 int wide)
{
  constexpr int W = Pack<T>::W;
  const bool big = wide || F1.nnz >= FLAT_NNZ_MAX;
  const int64_t bytes = F1.n * ld * (int64_t) sizeof (T);
  LGH_TRY (flat_check<T> (F1, R0, R1, nullptr, ld));
  return flat_slices (F1.n, F1.bandwidth, ld, ld / W, sizeof (T), [&] (int v0, int nv) {
    const FlatShape f = flat_shape (nv, F1.n);
    LGH_FLAT_DISPATCH (f.ch, {
      auto run = [&] (auto idx) -> int {
        auto k = k_flat_resid<T, decltype (idx), CH_>;
        LGH_CUDA (launch_pdl (bytes, k,
            fit_grid (k, flat_grid (f, F1.n), FLAT_THREADS, 0), FLAT_THREADS, 0,
            s, F1.n, F1.rowptr, F1.colidx, fvals<T> (F1), R0 + v0 * W,
            R0 + v0 * W, R1 + v0 * W, ld, nv, f.L, f.rpc));
        return 0;
      };
      LGH_TRY (big ? run (int64_t ()) : run (int ()));
    });
    LGH_LAUNCH_CHECK ();
    return 0;
  });
}

template <typename T>
int
launch_vc_second (const Csr &F1, const T *R0, const T *R1, T *R2, int ld,
                  double a2, double s2, cudaStream_t s, int wide)
{
  constexpr int W = Pack<T>::W;
  const bool big = wide || F1.nnz >= FLAT_NNZ_MAX;
  const int64_t bytes = F1.n * ld * (int64_t) sizeof (T);
  LGH_TRY (flat_check<T> (F1, R0, R1, R2, ld));
  return flat_slices (F1.n, F1.bandwidth, ld, ld / W, sizeof (T), [&] (int v0, int nv) {
    const FlatShape f = flat_shape (nv, F1.n);
    LGH_FLAT_DISPATCH (f.ch, {
      auto run = [&] (auto idx) -> int {
        auto k = k_flat_second<T, decltype (idx), CH_>;
        LGH_CUDA (launch_pdl (bytes, k,
            fit_grid (k, flat_grid (f, F1.n), FLAT_THREADS, 0), FLAT_THREADS, 0,
            s, F1.n, F1.rowptr, F1.colidx, fvals<T> (F1), R0 + v0 * W,
            R1 + v0 * W, R2 + v0 * W, ld, nv, f.L, f.rpc, (T) a2, (T) s2));
        return 0;
      };
      LGH_TRY (big ? run (int64_t ()) : run (int ()));
    });
    LGH_LAUNCH_CHECK ();
    return 0;
  });
}

template <typename T>
int
launch_vc_finish (const Csr &F1, const Csr &Q, const T *dinv, const T *R0,
                  const T *R1, const T *R2, const T *Xc, T *Z, int ld, double g,
                  double b2, cudaStream_t s, int wide)
{
  constexpr int W = Pack<T>::W;
  const bool big = wide || F1.nnz >= FLAT_NNZ_MAX || Q.nnz >= FLAT_NNZ_MAX;
  const int64_t bytes = F1.n * ld * (int64_t) sizeof (T);
  LGH_TRY (flat_check<T> (F1, R0, R1, R2, ld));
  LGH_TRY (flat_check<T> (Q, Xc, Z, nullptr, ld));
  LGH_CHECK (dinv && Q.n == F1.n, LGH_ERR_ARG_WRONG, "V-cycle finish: operators");
  return flat_slices (F1.n, F1.bandwidth, ld, ld / W, sizeof (T), [&] (int v0, int nv) {
    /* three packs per thread where that wastes under 5 % of them and the
     * rows are long (3D: 25 entries with Q's; 46 packs FP64 305 us against
     * 375 with four and 340 with two, 110 packs 802, 1036, 824), or divides
     * a 2D block of up to 64 packs (48: 210, 218, 230); 110 packs in 2D
     * keep four (alone 470, three 522) */
    FlatShape f = flat_shape (nv, F1.n);
    const int L3 = (nv + 2) / 3;
    const bool lng = F1.nnz + Q.nnz > 16 * F1.n;
    if (f.ch > 1 && nv > 16 && L3 <= FLAT_THREADS && 20 * (3 * L3 - nv) <= 3 * L3
        && (lng || (nv % 3 == 0 && nv <= 64)))
      f = flat_shape_ch (nv, 3);
    LGH_FLAT_DISPATCH (f.ch, {
      auto run = [&] (auto idx) -> int {
        auto k = k_flat_finish<T, decltype (idx), CH_>;
        LGH_CUDA (launch_pdl (bytes, k,
            fit_grid (k, flat_grid (f, F1.n), FLAT_THREADS, 0), FLAT_THREADS, 0,
            s, F1.n, F1.rowptr, F1.colidx, fvals<T> (F1), Q.rowptr, Q.colidx,
            fvals<T> (Q), dinv, R0 + v0 * W, R1 + v0 * W, R2 + v0 * W,
            Xc + v0 * W, Z + v0 * W, ld, nv, f.L, f.rpc, (T) g, (T) b2));
        return 0;
      };
      LGH_TRY (big ? run (int64_t ()) : run (int ()));
    });
    LGH_LAUNCH_CHECK ();
    return 0;
  });
}

template <typename T>
int
launch_flat_mult (const Csr &A, const T *X, T *Y, int ld, cudaStream_t s,
                  int wide)
{
  constexpr int W = Pack<T>::W;
  const bool big = wide || A.nnz >= FLAT_NNZ_MAX;
  const int64_t bytes = A.ncols * ld * (int64_t) sizeof (T);
  LGH_TRY (flat_check<T> (A, X, Y, nullptr, ld));
  /* one launch holds at most FLAT_MAXPACKS packs of a row */
  return flat_slices (0, 0, ld, ld / W, sizeof (T), [&] (int v0, int nv) {
    const FlatShape f = flat_shape (nv, A.n);
    /* split the rows until the grid covers the SMs six times, while a part
     * keeps at least four entries */
    const int64_t avg = A.n > 0 ? A.nnz / A.n : 0;
    int S = 1;
    while (2 * S <= f.rpc && avg >= 8 * S
           && (A.n + f.rpc / S - 1) / (f.rpc / S) < 6 * num_sms ())
      S *= 2;
    const int rows = f.rpc / S;
    const int64_t tiles = (A.n + rows - 1) / rows;
    const int want = (int) std::max<int64_t> (1, std::min<int64_t> (tiles, 1 << 20));
    const int smem = S > 1 ? rows * S * nv * 16 : 0;
    LGH_FLAT_DISPATCH (f.ch, {
      auto run = [&] (auto idx, auto split) -> int {
        constexpr bool SPLIT = decltype (split)::value;
        auto k = k_flat_mult<T, decltype (idx), CH_, SPLIT>;
        LGH_CUDA (launch_pdl (bytes, k, fit_grid (k, want, FLAT_THREADS, smem),
            FLAT_THREADS, smem, s, A.n, A.rowptr, A.colidx, fvals<T> (A),
            X + v0 * W, Y + v0 * W, ld, nv, f.L, rows, S));
        return 0;
      };
      if (S > 1)
        LGH_TRY (big ? run (int64_t (), std::true_type ())
                     : run (int (), std::true_type ()));
      else
        LGH_TRY (big ? run (int64_t (), std::false_type ())
                     : run (int (), std::false_type ()));
    });
    LGH_LAUNCH_CHECK ();
    return 0;
  });
}

#define LGH_FLAT_INST(T)                                                     \
  template int launch_vc_first<T> (const Csr &, const T *, T *, int,         \
                                   cudaStream_t, int);                       \
  template int launch_vc_second<T> (const Csr &, const T *, const T *, T *,  \
                                    int, double, double, cudaStream_t, int); \
  template int launch_vc_finish<T> (const Csr &, const Csr &, const T *,     \
                                    const T *, const T *, const T *,         \
                                    const T *, T *, int, double, double,     \
                                    cudaStream_t, int);                      \
  template int launch_flat_mult<T> (const Csr &, const T *, T *, int,        \
                                    cudaStream_t, int);
LGH_FLAT_INST (double)
LGH_FLAT_INST (float)
#undef LGH_FLAT_INST

} /* namespace lgh */
