/* k_spmm.cu -- CSR times row-major block: Y = A X.
 *
 * Replaces the reference's per-column MatMult loop (glr_common_impl.h:
 * 325-332, and MatMatMult in the Chebyshev core, zsolve_impl.h:123-136).
 * A group of G lanes (a power of two <= 32) owns one row; lane l covers the
 * 16-byte vector columns l, l+G, ..., so every nonzero (i, j) gathers the
 * contiguous row segment X[j, :] with coalesced vector loads, reused from
 * L1/L2 by the neighbouring rows of the same CTA.  The group's lanes fetch
 * G (col, val) pairs at once and broadcast them with shuffles.  Each CTA
 * owns a contiguous row range.  HBM bound; algorithmic bytes
 * nnz (s_v + 4) + 8 (N + 1) + 2 N w s_x.
 */

#include <algorithm>
#include <type_traits>

#include "lgh_device.cuh"
#include "lgh_internal.h"

namespace lgh
{

/* MODE 0: Y = A X;  1: Y += A X;  2: Y = B - A X */
template <typename T, typename TV, int CH, int MODE>
__global__ void __launch_bounds__ (256)
k_spmm (int64_t n, const int64_t *__restrict__ rowptr,
        const int32_t *__restrict__ colidx, const TV *__restrict__ vals,
        const T *__restrict__ X, int ldx, T *__restrict__ Y, int ldy,
        int nvec, int glog, const T *__restrict__ Bm, int ldb)
{
  constexpr int W = Pack<T>::W;
  const int G = 1 << glog;
  const int lane = threadIdx.x & (G - 1);
  const int group = threadIdx.x >> glog;
  const int ngroups = blockDim.x >> glog;
  const unsigned gmask = (G == 32) ? 0xffffffffu
                         : (((1u << G) - 1u) << ((threadIdx.x & 31) & ~(G - 1)));
  /* row tiles of ngroups rows interleaved over the CTAs (L2 locality of
   * the gathered neighbour rows); the next row's bounds and first G
   * (column, value) pairs are loaded during the current row's gathers */
  const int64_t stride = (int64_t) gridDim.x * ngroups;
  int64_t i = (int64_t) blockIdx.x * ngroups + group;
  int64_t k0 = 0, k1 = 0;
  int mc = 0;
  T mv = T (0);
  if (i < n) {
    k0 = rowptr[i];
    k1 = rowptr[i + 1];
    if (lane < k1 - k0) {
      mc = colidx[k0 + lane];
      mv = (T) vals[k0 + lane];
    }
  }
  for (; i < n; i += stride) {
    const int64_t inx = i + stride;
    int64_t k0n = 0, k1n = 0;
    if (inx < n) {
      k0n = rowptr[inx];
      k1n = rowptr[inx + 1];
    }
    T acc[CH][W];
#pragma unroll
    for (int h = 0; h < CH; h++)
#pragma unroll
      for (int e = 0; e < W; e++) acc[h][e] = T (0);
    for (int64_t kb = k0; kb < k1; kb += G) {
      const int cnt = (int) ((k1 - kb) < G ? (k1 - kb) : G);
      if (kb != k0) {
        mc = 0;
        mv = T (0);
        if (lane < cnt) {
          mc = colidx[kb + lane];
          mv = (T) vals[kb + lane];
        }
      }
      for (int t = 0; t < cnt; t++) {
        const int c = __shfl_sync (gmask, mc, t, G);
        const T v = __shfl_sync (gmask, mv, t, G);
        const T *xr = X + (int64_t) c * ldx;
#pragma unroll
        for (int h = 0; h < CH; h++) {
          const int vi = lane + h * G;
          if (vi < nvec) {
            Pack<T> x = ldp_nc (xr + vi * W);
#pragma unroll
            for (int e = 0; e < W; e++) acc[h][e] = fma (v, x.v[e], acc[h][e]);
          }
        }
      }
    }
    T *yr = Y + i * ldy;
#pragma unroll
    for (int h = 0; h < CH; h++) {
      const int vi = lane + h * G;
      if (vi < nvec) {
        Pack<T> o;
        if (MODE == 1) {
          Pack<T> y = ldp (yr + vi * W);
#pragma unroll
          for (int e = 0; e < W; e++) o.v[e] = y.v[e] + acc[h][e];
        } else if (MODE == 2) {
          Pack<T> b = ldp (Bm + i * ldb + vi * W);
#pragma unroll
          for (int e = 0; e < W; e++) o.v[e] = b.v[e] - acc[h][e];
        } else {
#pragma unroll
          for (int e = 0; e < W; e++) o.v[e] = acc[h][e];
        }
        stp (yr + vi * W, o);
      }
    }
    k0 = k0n;
    k1 = k1n;
    mc = 0;
    mv = T (0);
    if (inx < n && lane < k1n - k0n) {
      mc = colidx[k0n + lane];
      mv = (T) vals[k0n + lane];
    }
  }
}

/* what becomes of a row's product: / div_i (nullable), then stored, or
 * (add) scaled and added to Y */
template <typename T>
struct SpvEp
{
  const T *div;
  T scale;
  int add;
};

/* Scalar form for single vectors and unaligned views (ld not a multiple
 * of the 16-byte vector, or an offset base): G lanes split a row's
 * nonzeros (CSR-vector), reduce with shuffles; columns in a loop.  A lane
 * issues U entries' column and value loads, then U gathers of x (which L2
 * holds): HBM streams the operator.  G and U: see spmv_dispatch. */
template <typename T, typename TV, int G, int U>
__global__ void __launch_bounds__ (256)
k_spmm_scalar (int64_t n, const int64_t *__restrict__ rowptr,
               const int32_t *__restrict__ colidx, const TV *__restrict__ vals,
               const T *__restrict__ X, int ldx, T *__restrict__ Y, int ldy,
               int w, SpvEp<T> ep)
{
  pdl_wait ();
  const int lane = threadIdx.x & (G - 1);
  const unsigned gmask = G == 32 ? 0xffffffffu
                         : ((1u << (G & 31)) - 1u) << ((threadIdx.x & 31) & ~(G - 1));
  const int64_t row0 = ((int64_t) blockIdx.x * blockDim.x + threadIdx.x) / G;
  const int64_t rstride = ((int64_t) gridDim.x * blockDim.x) / G;
  int64_t k0n = 0, k1n = 0;
  if (row0 < n) {
    k0n = rowptr[row0];
    k1n = rowptr[row0 + 1];
  }
  for (int64_t i = row0; i < n; i += rstride) {
    const int64_t k0 = k0n, k1 = k1n;
    if (i + rstride < n) {   /* the next row's bounds, behind this one's loads */
      k0n = rowptr[i + rstride];
      k1n = rowptr[i + rstride + 1];
    }
    for (int c = 0; c < w; c++) {
      T acc = T (0);
      for (int64_t k = k0 + lane; k < k1; k += G * U) {
        int32_t j[U];
        T v[U], x[U];
#pragma unroll
        for (int u = 0; u < U; u++) {
          const bool in = k + u * G < k1;
          j[u] = in ? __ldcs (colidx + k + u * G) : 0;
          v[u] = in ? (T) __ldcs (vals + k + u * G) : T (0);
        }
#pragma unroll
        for (int u = 0; u < U; u++)
          x[u] = k + u * G < k1 ? X[(int64_t) j[u] * ldx + c] : T (0);
#pragma unroll
        for (int u = 0; u < U; u++) acc = fma (v[u], x[u], acc);
      }
#pragma unroll
      for (int o = G / 2; o > 0; o >>= 1)
        acc += __shfl_xor_sync (gmask, acc, o, G);
      if (lane == 0) {
        if (ep.div) acc /= ep.div[i];
        Y[i * ldy + c] = ep.add ? fma (ep.scale, acc, Y[i * ldy + c]) : acc;
      }
    }
  }
}

/* lanes per row and vector chunks per lane for a width of nvec vectors */
void
row_group_shape (int nvec, int &glog, int &ch, int kmax)
{
  int g = 1;
  glog = 0;
  while (g < nvec && g < 32) { g <<= 1; glog++; }
  ch = (nvec + g - 1) / g;
  /* a narrow block (one pack per lane) of an operator whose rows fit half
   * the lanes: half the lanes with two packs each keep twice the loads in
   * flight per thread (the smoother, the PCG kernels and the residual at
   * 64 columns measured 8-23% faster; the restriction, whose coarse rows
   * are long, and the prolongation keep kmax = 0) */
  if (kmax > 0 && ch == 1 && g >= 16 && g / 2 >= kmax) {
    g >>= 1;
    glog--;
    ch = (nvec + g - 1) / g;
  }
}

int
row_grid (int64_t n, int glog)
{
  const int rows_per_cta_iter = 256 >> glog;
  int64_t want = (n + rows_per_cta_iter - 1) / rows_per_cta_iter;
  int64_t cap = (int64_t) num_sms () * 8;
  if (want > cap) want = cap;
  return (int) (want > 0 ? want : 1);
}

template <typename T, typename TV>
static int
spmv_dispatch (const Csr &A, const TV *vals, const T *X, int ldx, T *Y, int ldy,
               int w, SpvEp<T> ep, cudaStream_t s)
{
  auto run = [&] (auto gl, auto un) -> int {
    constexpr int G = decltype (gl)::value, U = decltype (un)::value;
    auto k = k_spmm_scalar<T, TV, G, U>;
    const int want = (int) std::max<int64_t> (1, std::min<int64_t> (
        (A.n * G + 255) / 256, 1 << 20));
    /* H v is three products of 6, 104 and 6 us at 512^2: the next one's
     * CTAs are in place when the last of the previous one leave */
    LGH_CUDA (launch_pdl (A.n * (int64_t) sizeof (T), k,
                          fit_grid (k, want, 256, 0), 256, 0, s, A.n, A.rowptr,
                          A.colidx, vals, X, ldx, Y, ldy, w, ep));
    LGH_LAUNCH_CHECK ();
    return 0;
  };
  using std::integral_constant;
#define LGH_SPV(G, U) return run (integral_constant<int, G> (), integral_constant<int, U> ())
  if (w > 1) {
    /* columns of an unaligned view: the entries are read again for each */
    const int64_t avg = A.n > 0 ? A.nnz / A.n : 0;
    if (avg > 128) LGH_SPV (32, 8);
    if (avg > 32) LGH_SPV (32, 4);
    if (avg >= 8) LGH_SPV (8, 4);
    LGH_SPV (4, 2);
  }
  /* One vector: the fewest lanes whose G U entries cover the mean row in
   * one round of loads, as idle slots cost issue and a second round costs a
   * round trip.  262144 rows, us with this rule / with 4 x 2 below 8
   * entries, 8 x 4 to 32, 32 x 4 to 128, 32 x 8 above: 3 entries 10 / 16, 5
   * 11 / 16, 7 12 / 16, 9 14 / 25, 19 20 / 31, 27 25 / 37, 40 33 / 76, 57 45
   * / 82, 81 59 / 96, 100 76 / 102, 150 102 / 125, 183 111 / 131 (floor 90),
   * 220 and 256 the same; 300 141 / 160, 400 145 / 145.  Rows of 8 times
   * what a round covers take the next shape; 8 x 6 goes to 16 rounds, as the
   * shapes after it cost the short rows more (a row of 400 / 600 entries in
   * 4096 of 5: 42 / 51 us, 8 x 8 45 / 55, 16 x 6 51 / 55, one entry a lane
   * and round 65 / 82). */
  auto fits = [&] (int cover, int rounds = 8) {
    return A.nnz <= cover * A.n && A.max_row_nnz <= rounds * cover;
  };
  if (fits (5)) LGH_SPV (1, 5);
  if (fits (10)) LGH_SPV (1, 8);
  if (fits (28)) LGH_SPV (4, 7);
  if (fits (48, 16)) LGH_SPV (8, 6);
  if (fits (64)) LGH_SPV (8, 8);
  if (fits (96)) LGH_SPV (16, 6);
  if (fits (128)) LGH_SPV (16, 8);
  if (!fits (192) && fits (256)) LGH_SPV (32, 8);
  LGH_SPV (32, 6);
#undef LGH_SPV
}

/* y = (A x) ./ div, or y += scale A x (div null) of single FP64 vectors */
int
launch_spmv_div (const Csr &A, const double *x, const double *div, double *y,
                 cudaStream_t s)
{
  return spmv_dispatch<double, double> (A, A.vals, x, 1, y, 1, 1,
                                        SpvEp<double>{ div, 0., 0 }, s);
}

int
launch_spmv_add (const Csr &A, const double *x, double scale, double *y,
                 cudaStream_t s)
{
  return spmv_dispatch<double, double> (A, A.vals, x, 1, y, 1, 1,
                                        SpvEp<double>{ nullptr, scale, 1 }, s);
}

template <typename T, typename TV>
static int
spmm_dispatch (const Csr &A, const TV *vals, const T *X, int ldx, T *Y,
               int ldy, int w, cudaStream_t s, int mode = 0,
               const T *Bm = nullptr, int ldb = 0)
{
  constexpr int W = Pack<T>::W;
  const int MAXCH = 10;
  const bool vec_ok = (ldx % W == 0) && (ldy % W == 0)
                      && ((uintptr_t) X % 16 == 0) && ((uintptr_t) Y % 16 == 0)
                      && (mode < 2 || (ldb % W == 0 && (uintptr_t) Bm % 16 == 0));
  if (!vec_ok) {
    if (mode != 0)
      return set_error (LGH_ERR_ARG_WRONG, "spmm: accumulate/residual forms "
                        "need 16-byte aligned row-major blocks");
    return spmv_dispatch<T, TV> (A, vals, X, ldx, Y, ldy, w,
                                 SpvEp<T>{ nullptr, T (0), 0 }, s);
  }
  /* column chunks of at most 32 lanes * MAXCH vectors */
  for (int c0 = 0; c0 < w; c0 += 32 * MAXCH * W) {
    const int wc = (w - c0) < 32 * MAXCH * W ? (w - c0) : 32 * MAXCH * W;
    const int nvec = (wc + W - 1) / W;
    int glog, ch;
    row_group_shape (nvec, glog, ch, mode >= 2 ? A.max_row_nnz : 0);
    const int grid = row_grid (A.n, glog);
    const T *Xc = X + c0;
    T *Yc = Y + c0;
    const T *Bc = Bm ? Bm + c0 : nullptr;
#define LGH_SPMM_MODE(C, M)                                                  \
  k_spmm<T, TV, C, M><<<fit_grid (k_spmm<T, TV, C, M>, grid, 256, 0), 256,   \
                        0, s>>> (A.n, A.rowptr, A.colidx, vals, Xc, ldx, Yc, \
                                 ldy, nvec, glog, Bc, ldb)
#define LGH_SPMM_CASE(C)                                                     \
  case C:                                                                    \
    if (mode == 0) LGH_SPMM_MODE (C, 0);                                     \
    else if (mode == 1) LGH_SPMM_MODE (C, 1);                                \
    else LGH_SPMM_MODE (C, 2);                                               \
    break;
    switch (ch) {
      LGH_SPMM_CASE (1) LGH_SPMM_CASE (2) LGH_SPMM_CASE (3)
      LGH_SPMM_CASE (4) LGH_SPMM_CASE (5) LGH_SPMM_CASE (6)
      LGH_SPMM_CASE (7) LGH_SPMM_CASE (8) LGH_SPMM_CASE (9)
      LGH_SPMM_CASE (10)
    default:
      return set_error (LGH_ERR_SUP, "spmm: unsupported chunking %d", ch);
    }
#undef LGH_SPMM_CASE
#undef LGH_SPMM_MODE
    LGH_LAUNCH_CHECK ();
  }
  return 0;
}

template <>
int
launch_spmm<double> (const Csr &A, const double *X, int ldx, double *Y,
                     int ldy, int w, cudaStream_t s)
{
  return spmm_dispatch<double, double> (A, A.vals, X, ldx, Y, ldy, w, s);
}

template <>
int
launch_spmm<float> (const Csr &A, const float *X, int ldx, float *Y, int ldy,
                    int w, cudaStream_t s)
{
  return spmm_dispatch<float, float> (A, A.vals32, X, ldx, Y, ldy, w, s);
}

/* Y += A X (mode 1) or Y = B - A X (mode 2) on aligned row-major blocks */
template <>
int
launch_spmm_mode<double> (const Csr &A, const double *X, int ldx, double *Y,
                          int ldy, int w, int mode, const double *Bm, int ldb,
                          cudaStream_t s)
{
  return spmm_dispatch<double, double> (A, A.vals, X, ldx, Y, ldy, w, s, mode,
                                        Bm, ldb);
}

template <>
int
launch_spmm_mode<float> (const Csr &A, const float *X, int ldx, float *Y,
                         int ldy, int w, int mode, const float *Bm, int ldb,
                         cudaStream_t s)
{
  return spmm_dispatch<float, float> (A, A.vals32, X, ldx, Y, ldy, w, s, mode,
                                      Bm, ldb);
}

} /* namespace lgh */
