// pip_fp64_forms.cuh -- device forms of the FP64 solvers for the FMA-contracted build.
//
// The stage kernels of that build are bound by the instructions they issue (FP64 pipe 45 %,
// issue 57 % busy at 16 warps per SM, DRAM 15-22 %), so these forms reach the results of the literal ones
// (pip_physics.cuh) with fewer operations:
//   * minmod by selection instead of min/max/sign products (the same value bit for bit);
//   * HLLC and HLLD evaluate one side of the contact only (the one the face flux is taken
//     from) and use the jump relations F + S (U* - U) of that side in their solved form,
//     e.g. rho* sm for the mass flux; HLLD's other side is formed only in the double-star
//     region, whose flux is the single-star one plus s* (U** - U*);
//   * the region tests compare squares (sm - S)^2 rho* with bn^2, so the Alfven speeds'
//     square roots are taken only where the flux needs them;
//   * reciprocals and inverse square roots are hardware seeds refined by Newton-Raphson steps.
// Every sum that must cancel to +0 at a mirror wall is made of separately rounded products
// (mul_rn, see pip_physics.cuh).  Against the literal forms a flux differs by rounding.
//
// Measured on a B200, per step of two stage launches, the literal forms -> these, nothing else
// changed: Orszag-Tang 1024^2 0.551 -> 0.370 ms; 517x333 with walls and the exponential
// collisions 124 -> 85 us; 1024 cells in 1D 27.3 -> 20.5 us (a chain of dependent operations
// there).  With the other changes of the stage kernels 0.310 ms, 67 us and 8.2 us (that tube now runs
// the forms of pip_fp64_rcp.cu, 11.2 us).  Error of the
// state against 64-bit torch after 100 steps: 3.8e-15 -> 3.2e-15.
#pragma once

#include "pip_kernels.cuh"
#include "pip_physics.cuh"

namespace pip {

// Below this the roots' argument is taken as zero (their seed flushes subnormals).
constexpr double kTinyRoot = 1.0e-280;

// 1/sqrt(x) for x >= 0 (x below kTinyRoot as kTinyRoot, so that 0 * rsqrt_nr(0) is 0): the
// hardware's approximate inverse square root (PTX rsqrt.approx.ftz.f64) and two Newton-Raphson steps y <- y + y (1/2 - x/2 y^2).
__device__ __forceinline__ double rsqrt_nr(double x) {
  x = x > kTinyRoot ? x : kTinyRoot;
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  const double g = 0.5 * x;
  y = fma(y, fma(-(g * y), y, 0.5), y);
  return fma(y, fma(-(g * y), y, 0.5), y);
}

// sqrt(x) for x >= 0 (0 for x <= kTinyRoot): one Newton-Raphson step of the inverse square root, then
// Heron's step s <- s + (x - s^2)/(2 s) with 1/(2 s) taken from it.
__device__ __forceinline__ double sqrt_nr(double x) {
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  const double g = 0.5 * x;
  y = fma(y, fma(-(g * y), y, 0.5), y);
  const double s = x * y;
  const double r = fma(fma(-s, s, x), 0.5 * y, s);
  return x > kTinyRoot ? r : 0.0;
}

__device__ __forceinline__ double min_(double a, double b) { return a < b ? a : b; }
__device__ __forceinline__ double max_(double a, double b) { return a > b ? a : b; }

// The limited slope of minmod<double>(v0, v1, v2) as d (the smaller of the two differences)
// and the factor 1/2, or 0 where the differences' signs differ: h*d is 0.5*minmod bit for bit
// (h*d is exact, so fusing it into the caller's sum changes nothing).
__device__ __forceinline__ void half_minmod(double X, double Y, double &h, double &d) {
  d = fabs(X) < fabs(Y) ? X : Y;
  const int s = __double2hiint(X) ^ __double2hiint(Y);
  h = __hiloint2double(s < 0 ? 0 : 0x3fe00000, 0);
}

// Face states between cells 1 and 2 of four cells in a row (minmod MUSCL).
__device__ __forceinline__ void face_pair(double v0, double v1, double v2, double v3, double &l,
                                          double &r) {
  const double a = v1 - v0, b = v2 - v1, c = v3 - v2;
  double h, d;
  half_minmod(b, a, h, d);
  l = fma(h, d, v1);
  half_minmod(c, b, h, d);
  r = fma(-h, d, v2);
}

// hllc_flux (HLL_rot.f90:615-687).  The reference blends the two sides where a wave speed
// lies in (0, kHllcEpsi/2); those faces take the blended form.
__device__ __forceinline__ void hllc_flux_fast(const double (&l)[5], const double (&r)[5],
                                               double (&f)[5], double gm, double igm1) {
  const double gl = gm * l[4], gr = gm * r[4];
  const double cl = gl * rsqrt_nr(gl * l[0]), cr = gr * rsqrt_nr(gr * r[0]);
  const double sl = kHllcAcc * min_(l[1] - cl, r[1] - cr);
  const double sr = kHllcAcc * max_(l[1] + cl, r[1] + cr);
  const double tl = sl - l[1], tr = sr - r[1];
  const double ql = l[0] * tl, qr = r[0] * tr;
  const double sm = (mul_rn(r[0] * r[1], tr) - mul_rn(l[0] * l[1], tl) + l[4] - r[4]) * rcp_(qr - ql);
  constexpr double e = 0.5 * kHllcEpsi;
  if ((sl > 0.0 && sl < e) || (sm > 0.0 && sm < e) || (sr > 0.0 && sr < e)) {
    hllc_flux_rcp<double>(l, r, f, gm, igm1);
    return;
  }
  const bool left = sl > 0.0 || (sr > 0.0 && sm > 0.0);
  const double ro = left ? l[0] : r[0], vn = left ? l[1] : r[1], vy = left ? l[2] : r[2],
               vz = left ? l[3] : r[3], pr = left ? l[4] : r[4];
  const double E = fma(pr, igm1, 0.5 * ro * fma(vn, vn, fma(vy, vy, vz * vz)));
  const double S = left ? sl : sr, q = left ? ql : qr;
  double u = sm, m, p, en;   // normal velocity, mass flux, pressure and energy behind the wave
  if (sl > 0.0 || sr <= 0.0) {
    u = vn;
    m = ro * vn;
    p = pr;
    en = E;
  } else {
    const double i = rcp_(S - sm);
    m = q * i * sm;
    p = fma(q, sm - vn, pr);
    en = ((S - vn) * E - pr * vn + p * sm) * i;
  }
  f[0] = m;
  f[1] = fma(m, u, p);
  f[2] = m * vy;
  f[3] = m * vz;
  f[4] = (en + p) * u;
}

// hlld_flux (HLL_rot.f90:691-910) with the HLLC-G fallback and, for NVM == 9, the Dedner
// flux.  D = rho (S - vn) of a side; K is the side of the contact the flux is taken from.
template <int NVM>
__device__ __forceinline__ void hlld_flux_fast(const double (&l)[NVM], const double (&r)[NVM],
                                               double (&f)[NVM], double gm, double igm1,
                                               double cmax) {
  const double b2l = fma(l[5], l[5], fma(l[6], l[6], l[7] * l[7]));
  const double b2r = fma(r[5], r[5], fma(r[6], r[6], r[7] * r[7]));
  double sl, sr;
  {
    // the faster of the two fast speeds, sqrt((a + sqrt(a^2 - 4 gm p bn^2)) / (2 rho))
    const double gl = gm * l[4], gr = gm * r[4];
    const double al = gl + b2l, ar = gr + b2r;
    const double tl = al + sqrt_nr(fma(al, al, -4.0 * gl * (l[5] * l[5])));
    const double tr = ar + sqrt_nr(fma(ar, ar, -4.0 * gr * (r[5] * r[5])));
    const bool k = tl * r[0] > tr * l[0];
    const double t = k ? tl : tr, ro = k ? l[0] : r[0];
    const double c = t * rsqrt_nr(2.0 * ro * t);
    sl = min_(l[1], r[1]) - c;
    sr = max_(l[1], r[1]) + c;
  }
  const double tl = sl - l[1], tr = sr - r[1];
  const double Dl = l[0] * tl, Dr = r[0] * tr;
  const double pl = fma(0.5, b2l, l[4]), pr = fma(0.5, b2r, r[4]);
  const double iD = rcp_(Dr - Dl), iS = rcp_(sr - sl);
  const double sm = (mul_rn(r[1], Dr) - mul_rn(l[1], Dl) - fma(-r[5], r[5], pr) + fma(-l[5], l[5], pl)) * iD;
  const double bn = (mul_rn(sr, r[5]) - mul_rn(sl, l[5])) * iS, bn2 = bn * bn;
  const bool super = sl >= 0.0 || sr <= 0.0;
  const bool left = super ? sl >= 0.0 : sm >= 0.0;
  const double ro = left ? l[0] : r[0], vn = left ? l[1] : r[1], vy = left ? l[2] : r[2],
               vz = left ? l[3] : r[3], b5 = left ? l[5] : r[5], b6 = left ? l[6] : r[6],
               b7 = left ? l[7] : r[7];
  const double E = fma(left ? l[4] : r[4], igm1,
                       fma(0.5 * ro, fma(vn, vn, fma(vy, vy, vz * vz)), 0.5 * (left ? b2l : b2r)));
  const double pK = left ? pl : pr;
  const double vb = fma(vn, b5, fma(vy, b6, vz * b7));
  if (super) {
    const double m = ro * vn;
    f[0] = m;
    f[1] = fma(m, vn, fma(-b5, b5, pK));
    f[2] = fma(m, vy, -b5 * b6);
    f[3] = fma(m, vz, -b5 * b7);
    f[4] = fma(E + pK, vn, -vb * b5);
    f[5] = 0.0;
    f[6] = fma(vn, b6, -b5 * vy);
    f[7] = fma(vn, b7, -b5 * vz);
  } else {
    const double S = left ? sl : sr, tK = left ? tl : tr, D = left ? Dl : Dr;
    const double dm = S - sm;
    const double im = rcp_(dm);
    const double ro1 = D * im, m = ro1 * sm;
    const double pt = fma(Dl, sm - l[1], pl);          // the reference's, from the left state
    const double p1 = left ? pt : fma(Dr, sm - r[1], pr);
    double Y, Z, BY, BZ;                               // tangential star state
    double cy = 0.0, cz = 0.0, cb = 0.0, cc = 0.0, ce = 0.0;  // double-star corrections
    const double h = (kHllgFactor * kHllgFactor) * bn2;
    if (h >= Dl * (sl - sm) || h >= Dr * (sr - sm)) {
      // HLLC-G (HLL_rot.f90:776-807): the HLL averages
      Y = (mul_rn(Dr, r[2]) - mul_rn(Dl, l[2]) + (mul_rn(r[5], r[6]) - mul_rn(l[5], l[6]))) * iD;
      Z = (mul_rn(Dr, r[3]) - mul_rn(Dl, l[3]) + (mul_rn(r[5], r[7]) - mul_rn(l[5], l[7]))) * iD;
      BY = (mul_rn(r[6], tr) - mul_rn(l[6], tl) + (mul_rn(r[5], r[2]) - mul_rn(l[5], l[2]))) * iS;
      BZ = (mul_rn(r[7], tr) - mul_rn(l[7], tl) + (mul_rn(r[5], r[3]) - mul_rn(l[5], l[3]))) * iS;
    } else {
      // single star of side K (HLL_rot.f90:813-843)
      const double q = rcp_(fma(D, dm, -bn2));
      const double g = q * fma(D, tK, -bn2), w = q * bn * (sm - vn);
      BY = b6 * g;
      BZ = b7 * g;
      Y = fma(-w, b6, vy);
      Z = fma(-w, b7, vz);
      if (sm * sm * ro1 < bn2) {
        // double star (HLL_rot.f90:861-898): the other side O's star and the jump from U*
        const double So = left ? sr : sl, to = left ? tr : tl, Do = left ? Dr : Dl;
        const double vo = left ? r[1] : l[1], o6 = left ? r[6] : l[6], o7 = left ? r[7] : l[7];
        const double dmo = So - sm;
        const double qo = rcp_(fma(Do, dmo, -bn2));
        const double go = qo * fma(Do, to, -bn2), wo = qo * bn * (sm - vo);
        const double Yo = fma(-wo, o6, left ? r[2] : l[2]), Zo = fma(-wo, o7, left ? r[3] : l[3]);
        const double BYo = o6 * go, BZo = o7 * go;
        const double roo = Do * rcp_(dmo);
        const double ik = rsqrt_nr(ro1), io = rsqrt_nr(roo);
        const double rk = ro1 * ik, rO = roo * io;       // sqrt(rho*) of the two sides
        const double f1 = rcp_(rk + rO);
        const double sk = copysign(1.0, left ? bn : -bn);
        const double y2 = f1 * fma(rk, Y, fma(rO, Yo, (BYo - BY) * sk));
        const double z2 = f1 * fma(rk, Z, fma(rO, Zo, (BZo - BZ) * sk));
        const double b2 = f1 * fma(rk, BYo, fma(rO, BY, rk * rO * (Yo - Y) * sk));
        const double c2 = f1 * fma(rk, BZo, fma(rO, BZ, rk * rO * (Zo - Z) * sk));
        const double sal = fabs(bn) * ik;
        const double s1 = left ? sm - sal : sm + sal;
        cy = s1 * ro1 * (y2 - Y);
        cz = s1 * ro1 * (z2 - Z);
        cb = s1 * (b2 - BY);
        cc = s1 * (c2 - BZ);
        ce = -s1 * (rk * (fma(Y, BY, Z * BZ) - fma(y2, b2, z2 * c2)) * sk);
      }
    }
    const double W = fma(-sm, bn, vb) - fma(Y, BY, Z * BZ);
    const double e1 = (fma(tK, E, -pK * vn) + fma(pt, sm, bn * W)) * im;
    f[0] = m;
    f[1] = fma(m, sm, fma(-b5, b5, p1));
    f[2] = fma(m, Y, fma(D, Y - vy, fma(-b5, b6, cy)));
    f[3] = fma(m, Z, fma(D, Z - vz, fma(-b5, b7, cz)));
    f[4] = fma(e1 + pt, sm, fma(bn, W, fma(-vb, b5, ce)));
    f[5] = S * (bn - b5);
    f[6] = fma(S, BY, fma(-b6, tK, fma(-b5, vy, cb)));
    f[7] = fma(S, BZ, fma(-b7, tK, fma(-b5, vz, cc)));
  }
  if (NVM == 9) {
    f[5] = 0.5 * (l[NVM - 1] + r[NVM - 1] - cmax * (r[5] - l[5]));
    f[NVM - 1] = 0.5 * (cmax * cmax * (l[5] + r[5]) - cmax * (r[NVM - 1] - l[NVM - 1]));
  }
}

// Primitives of a conserved state with the velocity of the unfloored density and no floors
// applied (cq2pv's q before its floors), inv = 1/rho.
template <int NVM>
__device__ __forceinline__ Prim<double> prim_mhd(const double (&u)[NVM], double gm, double &inv) {
  Prim<double> q;
  inv = rcp_(u[0]);
  q.de = u[0];
  q.vx = u[1] * inv;
  q.vy = u[2] * inv;
  q.vz = u[3] * inv;
  const double k = fma(u[1], q.vx, fma(u[2], q.vy, u[3] * q.vz));
  const double b = fma(u[5], u[5], fma(u[6], u[6], u[7] * u[7]));
  q.pr = (gm - 1.0) * fma(-0.5, b, fma(-0.5, k, u[4]));
  return q;
}
__device__ __forceinline__ Prim<double> prim_hd(const double (&u)[5], double gm, double &inv) {
  Prim<double> q;
  inv = rcp_(u[0]);
  q.de = u[0];
  q.vx = u[1] * inv;
  q.vy = u[2] * inv;
  q.vz = u[3] * inv;
  const double k = fma(u[1], q.vx, fma(u[2], q.vy, u[3] * q.vz));
  q.pr = (gm - 1.0) * fma(-0.5, k, u[4]);
  return q;
}

// Whether cq2pv's floors leave the state alone (false for NaN): its rewrite is then the
// identity up to rounding.
__device__ __forceinline__ bool above_floors(const Prim<double> &q, double ro_lim, double pr_lim) {
  return q.de >= ro_lim && q.pr >= pr_lim;
}

// u2v_mhd / u2v_hd (HLL_rot.f90:1136-1186) with the Newton reciprocal.
template <int NVM>
__device__ __forceinline__ void u2v_mhd_fast(const double (&u)[NVM], double (&v)[NVM], double gm,
                                             double ro_lim, double pr_lim) {
  v[0] = max_(u[0], ro_lim);
  const double i = rcp_(v[0]);
  v[1] = u[1] * i;
  v[2] = u[2] * i;
  v[3] = u[3] * i;
  const double k = fma(u[1], v[1], fma(u[2], v[2], u[3] * v[3]));
  const double b = fma(u[5], u[5], fma(u[6], u[6], u[7] * u[7]));
  const double pr = (gm - 1.0) * fma(-0.5, b, fma(-0.5, k, u[4]));
  v[4] = pr < pr_lim ? pr_lim : pr;
  v[5] = u[5];
  v[6] = u[6];
  v[7] = u[7];
  if (NVM == 9) v[NVM - 1] = u[NVM - 1];
}
__device__ __forceinline__ void u2v_hd_fast(const double (&u)[5], double (&v)[5], double gm,
                                            double ro_lim, double pr_lim) {
  v[0] = max_(u[0], ro_lim);
  const double i = rcp_(v[0]);
  v[1] = u[1] * i;
  v[2] = u[2] * i;
  v[3] = u[3] * i;
  const double k = fma(u[1], v[1], fma(u[2], v[2], u[3] * v[3]));
  const double pr = (gm - 1.0) * fma(-0.5, k, u[4]);
  v[4] = pr < pr_lim ? pr_lim : pr;
}

// Collisional exchange dS of source_PIP (PIP_rot.f90:1333-1368) from the primitives alone:
// rho_i m_n - rho_n m_i = rho_i rho_n (v_n - v_i), and the exponential form's
// alpha (rho_n + rho_i) dt is the lambda dt of its energy term, so two exponentials serve it.
__device__ __forceinline__ void collision_prim(const Prim<double> &qm, const Prim<double> &qh,
                                               const KParams &p, double ac, double dt_coll,
                                               double (&ds)[5]) {
  const double gm = p.gm;
  const double dT = gm * fma(kMuN * qh.pr, rcp_(qh.de), -(kMuP * qm.pr) * rcp_(qm.de));  // nte - te
  const double dd = qm.de * qh.de;
  const double dvx = qh.vx - qm.vx, dvy = qh.vy - qm.vy, dvz = qh.vz - qm.vz;
  ds[0] = 0.0;
  if (p.imp) {
    const double nde = qh.de, de = qm.de, s = nde + de;
    const double lambda = ac * s;
    const double el = exp(-lambda * dt_coll);
    const double c = dd * (1.0 - el) * rcp_(s * dt_coll);
    ds[1] = c * dvx;
    ds[2] = c * dvy;
    ds[3] = c * dvz;
    const double kap = 3.0 * (gm - 1.0) * ac * (kMuP * nde + kMuN * de);
    const double ek = exp(-kap * dt_coll);
    // the ion term multiplies (nvz-vz) by nvz, as PIP_rot.f90:1348 does
    const double B = -(1.0 / 3.0 * gm * kap * rcp_(s * (kap - lambda)) *
                       (de * (dvx * qm.vx + dvy * qm.vy + dvz * qh.vz) +
                        nde * (dvx * qh.vx + dvy * qh.vy + dvz * qh.vz)));
    const double D = -(gm * (1.0 / 6.0) * kap * (de - nde) * rcp_(s * (kap - 2.0 * lambda)) *
                       (dvx * dvx + dvy * dvy + dvz * dvz));
    ds[4] = -((3.0 / gm) * ac * dd * rcp_(kap * dt_coll) *
              ((ek - 1.0) * dT - (B + D) * ek + B * el + D * (el * el)));
  } else {
    const double c = ac * dd;
    ds[1] = c * dvx;
    ds[2] = c * dvy;
    ds[3] = c * dvz;
    ds[4] = c * fma(p.c32g, dT,
                    0.5 * fma(dvx, qh.vx + qm.vx, fma(dvy, qh.vy + qm.vy, dvz * (qh.vz + qm.vz))));
  }
}

// min(cfl_mhd_cell, cfl_hd_cell) (Scheme_rot.f90:215-289): the candidate of the faster species.
__device__ __forceinline__ double cfl_cell_fast(const Prim<double> &m, const Prim<double> &h, double bx,
                                                double by, double bz, double gm, double sg) {
  const double b = fma(bx, bx, fma(by, by, bz * bz));
  const double cm = sqrt_nr(fma(m.vx, m.vx, fma(m.vy, m.vy, m.vz * m.vz))) +
                    sqrt_nr(fma(gm, m.pr, b) * rcp_(max_(m.de, kTiny)));
  const double ch = sqrt_nr(max_(fma(h.vx, h.vx, fma(h.vy, h.vy, h.vz * h.vz)), kTiny)) +
                    sqrt_nr(gm * h.pr * rcp_(h.de));
  return sg * rcp_(max_(ch, cm));
}

}  // namespace pip
