/* lgh_flat.cuh -- the flat row mapping of the gather kernels.
 *
 * A row of nvec 16-byte packs is covered by L = ceil (nvec / CH) threads of
 * CH packs each (thread l: packs l, l + L, ...), and a CTA of 256 threads
 * holds 256 / L rows, whatever L is: rows straddle warps, so no lanes are
 * lost to rounding L up to a power of two (18 packs: 9 threads x 2, 28 rows
 * per CTA, against 16 threads x 2 with 14 of 32 packs idle).  Every thread
 * reads its row's (column, value) entries itself: the threads of a row read
 * the same address (one broadcast from L1), which costs the load pipe less
 * than the three shuffles per entry of a lane-distributed row and leaves
 * the entry loop free of lane masks.  The loop takes one entry at a time:
 * the kernels are bound by L1 wavefronts and by how many warps are
 * resident, so registers spent on more entries in flight cost more than
 * they hide (first smoothing step, 512^2 x 220 columns FP64: 180 us with
 * one entry in flight at 4 CTAs per SM, 206 with two, 275 with five).  One
 * pack per thread is the other regime, narrow blocks or few rows on a chip
 * that is not full: there five entries go out at once (one solve of one
 * column at 512^2: 3.18 ms with one, 2.92 with four at 6 CTAs per SM, 2.83
 * at 5, 2.76 with five at 5, 2.93 with eight at 4; 64^2 x 1: 0.53, 0.48,
 * 0.47, 0.46, 0.47).
 * Packs per thread: 4 above 32 packs, 2 down to 3, 1 below (4 columns
 * FP64); fewer where the grid would not reach two CTAs per SM.  At 64
 * columns FP64, 2 packs 59 us, 4 packs 62, 1 pack 72; at 4 columns, 1 pack
 * 8.6 us, 2 packs 10.6. */

#ifndef LGH_FLAT_CUH
#define LGH_FLAT_CUH

#include <algorithm>

#include "lgh_device.cuh"
#include "lgh_internal.h"

namespace lgh
{

constexpr int FLAT_THREADS = 256;
constexpr int FLAT_BATCH = 5;           /* entries in flight at one pack */
constexpr int FLAT_MAXPACKS = FLAT_THREADS * 4;   /* packs of one launch */

/* threads per row, packs per thread, rows per CTA */
struct FlatShape
{
  int L, ch, rpc;
};

inline FlatShape
flat_shape_ch (int nvec, int ch)
{
  FlatShape f;
  f.ch = ch;
  f.L = (nvec + ch - 1) / ch;
  f.rpc = FLAT_THREADS / f.L;
  return f;
}

inline FlatShape
flat_shape (int nvec, int64_t n)
{
  int ch = nvec > 32 ? 4 : (nvec > 2 ? 2 : 1);
  FlatShape f = flat_shape_ch (nvec, ch);
  while (ch > 1 && (nvec + ch / 2 - 1) / (ch / 2) <= FLAT_THREADS
         && (n + f.rpc - 1) / f.rpc < 2 * num_sms ()) {
    ch /= 2;
    f = flat_shape_ch (nvec, ch);
  }
  return f;
}

/* CTAs that cover n rows once */
inline int
flat_grid (const FlatShape &f, int64_t n)
{
  const int64_t g = (n + f.rpc - 1) / f.rpc;
  return (int) std::max<int64_t> (1, std::min<int64_t> (g, 1 << 20));
}

/* CTAs per SM each shape is built for: 4 packs fit 64 registers, 2 packs
 * 42 (without spills in the single-gather kernels), 1 pack with its batch
 * 48 */
template <int CH>
struct FlatOcc
{
  static constexpr int v = CH == 4 ? 4 : (CH == 3 ? 5 : (CH == 2 ? 6 : 5));
};

/* one row's product: acc += sum_k v_k X[c_k, :] over its entries k0, k0 +
 * step, ... below k1; I: int for operators of fewer than 2^31 entries (the
 * wider offsets cost the registers that spill).  SC: each value of X is
 * first multiplied by sc, and rounded */
template <typename T, int CH, bool SC = false, typename I>
__device__ __forceinline__ void
flat_gather (const int32_t *__restrict__ ci, const T *__restrict__ va, I k0,
             I k1, int step, const T *__restrict__ X, int ld, int lane,
             int L, int nvec, T (&acc)[CH][Pack<T>::W], T sc = T (1))
{
  constexpr int W = Pack<T>::W;
  if constexpr (CH == 1) {
    /* bound by latency: a batch of entries' loads go out together.  Past
     * the row's end an entry of the row is loaded again and not used, so
     * the sum is the one of the loop below */
    for (I k = k0; k < k1; k += FLAT_BATCH * step) {
      int c[FLAT_BATCH];
      T v[FLAT_BATCH];
      Pack<T> x[FLAT_BATCH];
#pragma unroll
      for (int u = 0; u < FLAT_BATCH; u++) {
        const I ku = k + u * step < k1 ? k + u * step : k;
        c[u] = __ldg (ci + ku);
        v[u] = __ldg (va + ku);
      }
#pragma unroll
      for (int u = 0; u < FLAT_BATCH; u++)
        x[u] = ldp (X + (int64_t) c[u] * ld + lane * W);
#pragma unroll
      for (int u = 0; u < FLAT_BATCH; u++)
        if (k + u * step < k1)
#pragma unroll
          for (int e = 0; e < W; e++)
            acc[0][e] = fma (v[u], SC ? sc * x[u].v[e] : x[u].v[e], acc[0][e]);
    }
    return;
  }
  for (I k = k0; k < k1; k += step) {
    const int c = __ldg (ci + k);
    const T v = __ldg (va + k);
    const T *xr = X + (int64_t) c * ld;
#pragma unroll
    for (int h = 0; h < CH; h++) {
      const int vi = lane + h * L;
      if (h < CH - 1 || vi < nvec) {
        const Pack<T> x = ldp (xr + vi * W);
#pragma unroll
        for (int e = 0; e < W; e++)
          acc[h][e] = fma (v, SC ? sc * x.v[e] : x.v[e], acc[h][e]);
      }
    }
  }
}

template <typename T, int CH, int W>
__device__ __forceinline__ void
flat_zero (T (&acc)[CH][W])
{
#pragma unroll
  for (int h = 0; h < CH; h++)
#pragma unroll
    for (int e = 0; e < W; e++) acc[h][e] = T (0);
}

#define LGH_FLAT_DISPATCH(CHV, ...)                                          \
  switch (CHV) {                                                             \
  case 1: { constexpr int CH_ = 1; __VA_ARGS__; } break;                     \
  case 2: { constexpr int CH_ = 2; __VA_ARGS__; } break;                     \
  case 3: { constexpr int CH_ = 3; __VA_ARGS__; } break;                     \
  default: { constexpr int CH_ = 4; __VA_ARGS__; } break;                    \
  }

} /* namespace lgh */

#endif /* LGH_FLAT_CUH */
