// pip_mixed_cell.cuh -- FP64 per-cell parts of the FP32-mixed form (primitives, floors,
// collisional and ionisation/recombination source), shared by the 1D/2D mixed stage
// kernels and the batched ensemble so that both compute identical cell updates.
#pragma once

#include "pip_fp64_forms.cuh"
#include "pip_ghosts.cuh"
#include "pip_kernels.cuh"
#include "pip_physics.cuh"

namespace pip {
namespace mixed {

// FP64 primitives of a conserved cell (cq2pv's, without the rewrite): the velocity of the
// unfloored density, the floored density and pressure.
template <int NVM>
__device__ __forceinline__ Prim<double> prim_mhd(const double (&u)[NVM], const KParams &p) {
  double inv;
  Prim<double> q = pip::prim_mhd<NVM>(u, p.gm, inv);
  q.pr = max_(q.pr, p.pr_lim);
  q.de = max_(q.de, p.ro_lim);
  return q;
}
__device__ __forceinline__ Prim<double> prim_hd(const double (&u)[5], const KParams &p) {
  double inv;
  Prim<double> q = pip::prim_hd(u, p.gm, inv);
  q.pr = max_(q.pr, p.pr_lim);
  q.de = max_(q.de, p.ro_lim);
  return q;
}

// Density/pressure floors of cq2pv (Scheme_rot.f90:171-178), applied only when they fire;
// an FP32 estimate skips the FP64 test far from the floors.
template <int NVM>
__device__ __forceinline__ void floors_mhd(double (&u)[NVM], const KParams &p) {
  {
    const float d = (float)u[0];
    const float pf = (float)(p.gm - 1.0) *
                     ((float)u[4] - 0.5f * ((float)u[1] * (float)u[1] + (float)u[2] * (float)u[2] +
                                            (float)u[3] * (float)u[3]) / d -
                      0.5f * ((float)u[5] * (float)u[5] + (float)u[6] * (float)u[6] +
                              (float)u[7] * (float)u[7]));
    if (d > 2.0f * (float)p.ro_lim && pf > 2.0f * (float)p.pr_lim + 1e-3f * (float)u[4]) return;
  }
  const double de = u[0];
  const double k = 0.5 * (u[1] * u[1] + u[2] * u[2] + u[3] * u[3]) / de;
  const double b = 0.5 * (u[5] * u[5] + u[6] * u[6] + u[7] * u[7]);
  const double pr = (p.gm - 1.0) * (u[4] - k - b);
  if (pr <= p.pr_lim || de <= p.ro_lim) cq2pv_mhd<double, NVM>(u, p.gm, p.ro_lim, p.pr_lim);
}
__device__ __forceinline__ void floors_hd(double (&u)[5], const KParams &p) {
  {
    const float d = (float)u[0];
    const float pf = (float)(p.gm - 1.0) *
                     ((float)u[4] - 0.5f * ((float)u[1] * (float)u[1] + (float)u[2] * (float)u[2] +
                                            (float)u[3] * (float)u[3]) / d);
    if (d > 2.0f * (float)p.ro_lim && pf > 2.0f * (float)p.pr_lim + 1e-3f * (float)u[4]) return;
  }
  const double de = u[0];
  const double pr = (p.gm - 1.0) * (u[4] - 0.5 * (u[1] * u[1] + u[2] * u[2] + u[3] * u[3]) / de);
  if (pr <= p.pr_lim || de <= p.ro_lim) cq2pv_hd<double>(u, p.gm, p.ro_lim, p.pr_lim);
}

template <int NVM>
__device__ __forceinline__ void ir_rates(const double (&u)[NVM], const KParams &p, double &gr,
                                         double &gi) {
  const double gm = p.gm, inv = rcp_(u[0]);
  double pr = (gm - 1.0) * (u[4] - 0.5 * ((u[1] * u[1] + u[2] * u[2] + u[3] * u[3]) * inv +
                                          u[5] * u[5] + u[6] * u[6] + u[7] * u[7]));
  pr = max_(pr, p.pr_lim);
  const double te = 0.5 * gm * (pr * inv);
  const double rs = rsqrt_nr(te);
  gr = p.ir_rec * rs;
  gi = p.ir_ion * rs * exp(-p.ir_chi * rcp_(te));
}

// FP64 collisional dS (PIP_rot.f90:1333-1368) from FP64 primitives and the densities as they
// are (um[0], uh[0]: the momentum exchange takes them unfloored).  Where no density floor
// acts this is collision_prim, with two exponentials and five reciprocals instead of four and
// about ten divisions: the exponential form was most of an ensemble's cell update (three
// calls a step beside two pairs of FP32 solvers).
template <int NVM>
__device__ __forceinline__ void collision_ds(const double (&um)[NVM], const double (&uh)[5],
                                             const Prim<double> &qm, const Prim<double> &qh,
                                             const KParams &p, double dt_coll, double (&ds)[5]) {
  collision_prim(qm, qh, p, p.ac, dt_coll, ds);
  if (um[0] != qm.de || uh[0] != qh.de) {
    const double s = um[0] + uh[0];
    double c = p.ac * um[0] * uh[0];
    if (p.imp) c = um[0] * uh[0] * (1.0 - exp(-p.ac * (dt_coll * s))) / (dt_coll * s);
    ds[1] = c * (qh.vx - qm.vx);
    ds[2] = c * (qh.vy - qm.vy);
    ds[3] = c * (qh.vz - qm.vz);
  }
}

__device__ __forceinline__ void ir_ds(const Prim<double> &qm, const Prim<double> &qh, double gr,
                                      double gi, const KParams &p, double (&ds)[5]) {
  ds[0] = gr * qm.de - gi * qh.de;
  ds[1] = gr * qm.de * qm.vx - gi * qh.de * qh.vx;
  ds[2] = gr * qm.de * qm.vy - gi * qh.de * qh.vy;
  ds[3] = gr * qm.de * qm.vz - gi * qh.de * qh.vz;
  const double kin = 0.5 * (gr * qm.de * (qm.vx * qm.vx + qm.vy * qm.vy + qm.vz * qm.vz) -
                            gi * qh.de * (qh.vx * qh.vx + qh.vy * qh.vy + qh.vz * qh.vz));
  ds[4] = kin + ((p.ir_type == 1 ? 0.5 : 1.0) * gr * qm.pr - gi * qh.pr) * p.igm1;
}

// Whether any of a cell's values is not finite (an all-ones exponent).
template <int N>
__device__ __forceinline__ bool not_finite(const double (&u)[N]) {
  int top = 0;
#pragma unroll
  for (int n = 0; n < N; ++n) top = max(top, __double2hiint(u[n]) & 0x7fffffff);
  return top >= 0x7ff00000;
}

// Ghost images of a cell whose NP FP64 values u are stored as hi (and, with PAIR, lo) planes:
// hi = (float)u, lo = (float)(u - hi), with the faces' sign flips.
template <int NDIM, int NP, bool PAIR>
__device__ __forceinline__ void write_ghosts(const KParams &p, int gi, int gj, float *hi, float *lo,
                                             const double (&u)[NP]) {
  const long long nc = p.nc;
  ghost_images<NDIM>(p, gi, gj, [&](long long t, unsigned flips) {
#pragma unroll
    for (int n = 0; n < NP; ++n) {
      const float h = (float)u[n];
      hi[t + n * nc] = flipped(h, flips, n);
      if (PAIR) lo[t + n * nc] = flipped((float)(u[n] - (double)h), flips, n);
    }
  });
}

// The same for a cell already stored in hi and lo.
template <int NDIM, int NP>
__device__ __forceinline__ void copy_ghosts(const KParams &p, int gi, int gj, float *hi, float *lo) {
  const long long nc = p.nc, q = (long long)gj * p.ix + gi;
  float h[NP], w[NP];
#pragma unroll
  for (int n = 0; n < NP; ++n) {
    h[n] = hi[q + n * nc];
    w[n] = lo[q + n * nc];
  }
  ghost_images<NDIM>(p, gi, gj, [&](long long t, unsigned flips) {
#pragma unroll
    for (int n = 0; n < NP; ++n) {
      hi[t + n * nc] = flipped(h[n], flips, n);
      lo[t + n * nc] = flipped(w[n], flips, n);
    }
  });
}

}  // namespace mixed
}  // namespace pip
