/* lgh_pcg.h -- the passes of the blocked PCG around an explicit
 * preconditioner (k_pcg.cu), and the slots of its per-column scalars. */

#ifndef LGH_PCG_H
#define LGH_PCG_H

#include "lgh_internal.h"

namespace lgh
{

/* per-column scalar slots in ZWork::scal (each `cap` long) */
enum { S_RZ = 0, S_ALPHA, S_BETA, S_NORM0, S_NSLOT };
/* int slots in ZWork::ival; the active-column count follows them */
enum { I_ACTIVE = 0, I_ITS, I_NSLOT };

/* R = S B (pads zero; rs nullable), and its FP32 copy where R32 is given */
template <typename T>
int launch_pcg_start (int64_t n, int w, int ld, const T *B, int ldb,
                      const double *rs, T *R, float *R32, cudaStream_t s);

/* (r, z), (z, z) per column and what follows from them: the first call of a
 * solve (first, or a column marked in fresh) sets rz, norm0 and the mask,
 * later ones beta and the convergence test on ||z|| */
template <typename T, typename TZ>
int launch_pcg_dots (int64_t n, int w, int ld, const T *R, const TZ *Zb,
                     int first, double rtol, int iter, double *hist,
                     const int *fresh, ZWork &ws, cudaStream_t s,
                     int report = 0);
/* report: the count of active columns also goes to the host, where this
 * waits for it */
int pcg_wait_count (ZWork &ws, cudaStream_t s, int *count);

/* the direction, in place: p = z (PCG_P_FIRST), p = z + beta p; with it the
 * previous iteration's deferred x = alpha p_old (PCG_X_FIRST) or x += alpha
 * p_old (PCG_X_ADD): x is read by nothing inside an iteration */
enum { PCG_P_FIRST = 1, PCG_X_FIRST = 2, PCG_X_ADD = 4 };
template <typename T, typename TZ>
int launch_pcg_dir (int64_t n, int ld, const TZ *Zb, T *P, T *X, int flags,
                    ZWork &ws, cudaStream_t s);

/* q = Z p, (p, q) per column and alpha = rz / (p, q) */
template <typename T>
int launch_pcg_prod (const Csr &Z, const T *P, T *Q, int ld, ZWork &ws,
                     cudaStream_t s);

/* r -= alpha q, and the FP32 copy of r where R32 is given */
template <typename T>
int launch_pcg_resid (int64_t n, int ld, T *R, const T *Q, float *R32,
                      ZWork &ws, cudaStream_t s);

/* Y = S (x + alpha p) over the w columns (have_x 0: x is zero; P null: no
 * alpha p): the last iteration's deferred update with the solution's row
 * scaling */
template <typename T>
int launch_pcg_out (int64_t n, int w, int ld, const T *X, const T *P,
                    int have_x, const double *rs, T *Y, int ldy, ZWork &ws,
                    cudaStream_t s);

/* the fixed-count iteration around z = V(r): a step x += b z, r -= b Z z
 * (first: x = b z), the last step's x with the row scaling, and the
 * Chebyshev direction p = a p + b z (first: p = b z) that may stand for z,
 * with b = 1 */
template <typename T>
int launch_pcg_cheb (const Csr &Z, const T *Zb, T *R, T *X, int ld, double b,
                     int first, cudaStream_t s);
template <typename T>
int launch_pcg_cheb_dir (int64_t n, int ld, const T *Zb, T *P, double a,
                         double b, int first, cudaStream_t s);
template <typename T>
int launch_pcg_cheb_out (int64_t n, int w, int ld, const T *Zb, const T *X,
                         double b, int only, const double *rs, T *Y, int ldy,
                         cudaStream_t s);

} /* namespace lgh */

#endif /* LGH_PCG_H */
