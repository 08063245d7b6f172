// pcg_common.cuh -- the SELL-32 addressing of a 3x3 block (kernels_sparse.cu and kernels_pcg.cu), and the block-Jacobi
// product and scalar epilogues of kernels_sparse.cu's PCG kernels (the resident solves have their own, step_scalars).
#pragma once
#include "kernels.cuh"

namespace ssim_gb {

__device__ __forceinline__ size_t sell_base(int q) { return (size_t)9 * (size_t)(q & ~31) + (size_t)(q & 31); }

// the scalar epilogues of standard PCG (two-launch and persistent)
__device__ __forceinline__ void pcg_after_pq(DevScalars* sc, double pq) {
  sc->pq = pq;
  sc->alpha = sc->rz / pq;
  if (!(pq > 0.0)) {  // breakdown: not SPD along p (or non-finite)
    sc->done = 1;
    sc->status = 1;
  }
}

__device__ __forceinline__ void pcg_after_rz(DevScalars* sc, double rz, double rr, int max_iters) {
  sc->rz_old = sc->rz;
  sc->rz = rz;
  sc->beta = rz / sc->rz_old;
  sc->rr = rr;
  sc->iters += 1;
  if (!isfinite(rr)) {
    sc->done = 1;
    sc->status = 2;
  } else if (rr <= sc->tol2 || sc->iters >= max_iters || rz == 0.0) {
    sc->done = 1;
  }
}

// Chronopoulos-Gear and pipelined PCG: scalar epilogue after the dots (one thread): stop tests on the residual of the current x, then the
// step lengths.  iters counts the x updates; rr is |r|^2 of the current x.
__device__ __forceinline__ void cgcg_after(DevScalars* sc, double g, double d, double rr, int max_iters) {
  sc->rr = rr;
  if (!isfinite(rr)) {
    sc->done = 1;
    sc->status = 2;
    return;
  }
  if (rr <= sc->tol2 || g == 0.0 || sc->iters >= max_iters) {
    sc->done = 1;
    return;
  }
  // beta = g / g_old and den = d - beta g / alpha_old from the reciprocals kept by the previous step, so
  // only two independent divisions remain on this serial path (FP64 divisions are slow on GB300)
  double beta = 0.0, den = d;
  if (sc->iters > 0) {
    beta = g * sc->inv_rz;
    den = d - beta * g * sc->inv_alpha;
  }
  if (!(den > 0.0)) {  // breakdown: not SPD along p (or non-finite)
    sc->done = 1;
    sc->status = 1;
    return;
  }
  const double inv_den = 1.0 / den, inv_g = 1.0 / g;
  sc->rz_old = sc->rz;
  sc->rz = g;
  sc->pq = den;
  sc->beta = beta;
  sc->alpha = g * inv_den;
  sc->inv_rz = inv_g;
  sc->inv_alpha = den * inv_g;
  sc->iters += 1;
}

template <typename S>
__device__ __forceinline__ V4<S> block_jacobi(const V4<S>* __restrict__ dinv, int u, S a0, S a1, S a2) {
  const V4<S> d0 = dinv[3 * u], d1 = dinv[3 * u + 1], d2 = dinv[3 * u + 2];
  return mk4<S>(d0.x * a0 + d0.y * a1 + d0.z * a2, d1.x * a0 + d1.y * a1 + d1.z * a2,
                d2.x * a0 + d2.y * a1 + d2.z * a2);
}

}  // namespace ssim_gb
