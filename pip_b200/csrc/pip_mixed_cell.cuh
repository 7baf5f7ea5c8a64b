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

// The source's results round to the FP32 stage state, and where one lands next to a rounding
// boundary a last bit moves the state by 1e-7 and the fluxes with it (in one of about fifteen
// 1024x1024 runs of 100 steps an exchange that differed by rounding did).  So its quotients are
// corrected ones, from one reciprocal a denominator: q = a y, then q + (a - x q) y (the last
// step of Markstein's division, IBM J. Res. Dev. 34, 1990), in three operations and without the
// division's scaling and branches.  His theorem asks for the correctly rounded reciprocal; with
// y = rcp_(x), right to an ulp, quotients very close to a rounding boundary are not covered.
// None of 2^30 sampled operand pairs differs from a / x (tests/div_check.cu).  For normal
// operands and quotients; y = rcp_(x) or 1/x.
__device__ __forceinline__ double div_rn(double a, double x, double y) {
  const double q = __dmul_rn(a, y);
  return fma(fma(-x, q, a), y, q);
}

// FP64 primitives of a conserved cell (cq2pv's expressions, without the rewrite), inv = 1/q.de.
template <int NVM>
__device__ __forceinline__ Prim<double> prim_mhd(const double (&u)[NVM], const KParams &p,
                                                 double &inv) {
  Prim<double> q;
  const double de = u[0];
  inv = 1.0 / de;
  q.vx = u[1] * inv;
  q.vy = u[2] * inv;
  q.vz = u[3] * inv;
  q.pr = fmax((p.gm - 1.0) * (u[4] - 0.5 * de * (q.vx * q.vx + q.vy * q.vy + q.vz * q.vz) -
                              0.5 * (u[5] * u[5] + u[6] * u[6] + u[7] * u[7])), p.pr_lim);
  q.de = fmax(de, p.ro_lim);
  inv = de > p.ro_lim ? inv : p.r_ro_lim;
  return q;
}
__device__ __forceinline__ Prim<double> prim_hd(const double (&u)[5], const KParams &p,
                                                double &inv) {
  Prim<double> q;
  const double de = u[0];
  inv = 1.0 / de;
  q.vx = u[1] * inv;
  q.vy = u[2] * inv;
  q.vz = u[3] * inv;
  q.pr = fmax((p.gm - 1.0) * (u[4] - 0.5 * de * (q.vx * q.vx + q.vy * q.vy + q.vz * q.vz)), p.pr_lim);
  q.de = fmax(de, p.ro_lim);
  inv = de > p.ro_lim ? inv : p.r_ro_lim;
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
  const double gm = p.gm;
  double pr = (gm - 1.0) * (u[4] - 0.5 * ((u[1] * u[1] + u[2] * u[2] + u[3] * u[3]) / u[0] +
                                          u[5] * u[5] + u[6] * u[6] + u[7] * u[7]));
  pr = fmax(pr, p.pr_lim);
  const double te = 0.5 * gm * (pr / u[0]);
  const double rs = 1.0 / sqrt(te);
  gr = p.ir_rec * rs;
  gi = p.ir_ion * rs * exp(-p.ir_chi / te);
}

// FP64 collisional dS (PIP_rot.f90:1333-1368) from FP64 primitives; im = 1/qm.de, ih = 1/qh.de.
// The exponential form takes four exp, and nine quotients from seven reciprocals: an ensemble
// of 256 tubes (three calls a step), 400 steps, 87 ms with divisions, 65 ms.
template <int NVM>
__device__ __forceinline__ void collision_ds(const double (&um)[NVM], const double (&uh)[5],
                                             const Prim<double> &qm, const Prim<double> &qh,
                                             double im, double ih, const KParams &p,
                                             double dt_coll, double (&ds)[5]) {
  const double gm = p.gm, ac = p.ac;
  ds[0] = 0.0;
  if (p.imp) {
    const double te = div_rn(qm.pr, qm.de, im) * gm * kMuP;
    const double nte = div_rn(qh.pr, qh.de, ih) * gm * kMuN;
    const double temp = dt_coll * (uh[0] + um[0]);
    const double e = (1.0 - exp(-ac * temp));
    const double it = rcp_(temp);
    ds[1] = div_rn((um[0] * uh[1] - uh[0] * um[1]) * e, temp, it);
    ds[2] = div_rn((um[0] * uh[2] - uh[0] * um[2]) * e, temp, it);
    ds[3] = div_rn((um[0] * uh[3] - uh[0] * um[3]) * e, temp, it);
    const double nde = qh.de, de = qm.de;
    const double lambda = ac * (nde + de);
    const double kap = 3.0 * (gm - 1.0) * ac * (kMuP * nde + kMuN * de);
    const double dvx = qh.vx - qm.vx, dvy = qh.vy - qm.vy, dvz = qh.vz - qm.vz;
    const double db = (nde + de) * (kap - lambda), dd = (de + nde) * (kap - 2.0 * lambda);
    const double B = -(div_rn(1.0 / 3.0 * gm * kap, db, rcp_(db)) *
                       (de * (dvx * qm.vx + dvy * qm.vy + dvz * qh.vz) +
                        nde * (dvx * qh.vx + dvy * qh.vy + dvz * qh.vz)));
    const double D = -(div_rn(p.gm_6 * kap * (de - nde), dd, rcp_(dd)) *
                       (dvx * dvx + dvy * dvy + dvz * dvz));
    ds[4] = -div_rn(div_rn(p.r3_gm * ac * de * nde, kap, rcp_(kap)) *
                    (+(exp(-kap * dt_coll) - 1.0) * (nte - te) - (B + D) * exp(-kap * dt_coll) +
                     B * exp(-lambda * dt_coll) + D * exp(-2.0 * lambda * dt_coll)),
                    dt_coll, rcp_(dt_coll));
  } else {
    ds[1] = ac * (um[0] * uh[1] - uh[0] * um[1]);
    ds[2] = ac * (um[0] * uh[2] - uh[0] * um[2]);
    ds[3] = ac * (um[0] * uh[3] - uh[0] * um[3]);
    // 3/gm/2 (nte - te) with te = 0.5 gm pr/de, nte = gm npr/nde: the gm cancels
    const double dte = 1.5 * (div_rn(qh.pr, qh.de, ih) - 0.5 * div_rn(qm.pr, qm.de, im));
    ds[4] = ac * qh.de * qm.de *
            (0.5 * ((qh.vx * qh.vx - qm.vx * qm.vx) + (qh.vy * qh.vy - qm.vy * qm.vy) +
                    (qh.vz * qh.vz - qm.vz * qm.vz)) +
             dte);
  }
}

__device__ __forceinline__ void ir_ds(const Prim<double> &qm, const Prim<double> &qh, double gr,
                                      double gi, const KParams &p, double (&ds)[5]) {
  const double gm = p.gm;
  ds[0] = gr * qm.de - gi * qh.de;
  ds[1] = gr * qm.de * qm.vx - gi * qh.de * qh.vx;
  ds[2] = gr * qm.de * qm.vy - gi * qh.de * qh.vy;
  ds[3] = gr * qm.de * qm.vz - gi * qh.de * qh.vz;
  const double kin = 0.5 * (gr * qm.de * (qm.vx * qm.vx + qm.vy * qm.vy + qm.vz * qm.vz) -
                            gi * qh.de * (qh.vx * qh.vx + qh.vy * qh.vy + qh.vz * qh.vz));
  if (p.ir_type == 1)
    ds[4] = kin - gi * qh.pr / (gm - 1.0) + 0.5 * gr * qm.pr / (gm - 1.0);
  else
    ds[4] = kin - gi * qh.pr / (gm - 1.0) + gr * qm.pr / (gm - 1.0);
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
