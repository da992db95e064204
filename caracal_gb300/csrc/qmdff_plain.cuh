// QMDFF terms of the plain form: FP64, and FP64 with a tangent (Dual) for the
// Hessian-vector products.
//
// What bounds them is the FP64 pipe, 64 cycles per warp instruction, so the
// roots, reciprocals, exponentials, powers, trigonometric functions and erf run
// on the integer pipe (fx64.cuh), what depends on a pair's parameters alone is
// folded into its table row, and the torsion's derivatives take the form of
// Blondel and Karplus (J. Comput. Chem. 17, 1132 (1996)), some 180 additions and
// multiplications instead of some 290.  Rounding errors over C20H42 geometries are
// no larger than the reference formulas' in FP64 (bead spreads 0.02 to 0.1 bohr, of
// the largest force: torsions 4e-16 against 5e-16).  Measured with the
// eight warps per bead: see kTeam.
#pragma once

#include "dual.cuh"
#include "fx64.cuh"

namespace cr {
namespace qmdff {

// ---- functions: value, and the textbook derivative rules for the tangent ----
__device__ inline double p_rcp(double x) { return fx::rcp(x); }
__device__ inline Dual p_rcp(Dual x) {
  const double v = fx::rcp(x.v);
  return Dual(v, -(v * v) * x.d);
}
__device__ inline double p_div(double a, double b) { return fx::div(a, b); }
__device__ inline Dual p_div(Dual a, Dual b) {
  const double r = fx::rcp(b.v), q = a.v * r;
  return Dual(q, (a.d - q * b.d) * r);
}
// sqrt(x) and 1 / sqrt(x); the derivative of sqrt at 0 is taken as 0
__device__ inline void p_root(double x, double& r, double& ir) { fx::sqrt_rsqrt(x, r, ir); }
__device__ inline void p_root(Dual x, Dual& r, Dual& ir) {
  fx::sqrt_rsqrt(x.v, r.v, ir.v);
  r.d = r.v > 0.0 ? 0.5 * x.d * ir.v : 0.0;
  ir.d = -(ir.v * ir.v) * r.d;
}
__device__ inline double p_exp(double x) { return fx::exp(x); }
__device__ inline Dual p_exp(Dual x) {
  const double e = fx::exp(x.v);
  return Dual(e, e * x.d);
}
__device__ inline double p_pow(double x, double p) { return fx::pow(x, p); }
__device__ inline Dual p_pow(Dual x, double p) {
  const double y = fx::pow(x.v, p);
  return Dual(y, x.v != 0.0 ? p * y * fx::rcp(x.v) * x.d : 0.0);
}
__device__ inline void p_sincos(double x, double& s, double& c) { fx::sincos(x, s, c); }
__device__ inline void p_sincos(Dual x, Dual& s, Dual& c) {
  fx::sincos(x.v, s.v, c.v);
  s.d = c.v * x.d;
  c.d = -s.v * x.d;
}
// the angle in [0, pi] of cosine c, and its sine sqrt((1 - c)(1 + c))
__device__ inline void p_angle(double c, double& phi, double& s) {
  phi = fx::acos(c);
  s = fx::sqrt((1.0 - c) * (1.0 + c));
}
__device__ inline void p_angle(Dual c, Dual& phi, Dual& s) {
  double is;
  fx::sqrt_rsqrt((1.0 - c.v) * (1.0 + c.v), s.v, is);
  phi.v = fx::acos(c.v);
  phi.d = s.v > 0.0 ? -c.d * is : 0.0;
  s.d = c.v * phi.d;
}
// the angle in [0, pi] of cosine c and sine s: of the sine near 0 and pi, where the
// cosine's rounding would be magnified by 1 / sin
__device__ inline double p_angle_of(double c, double s) {
  if (!(s < 0.5)) return fx::acos(c);
  const double a = fx::asin(s);
  return c < 0.0 ? 3.1415926535897932384626433832795029 - a : a;
}
__device__ inline Dual p_angle_of(Dual c, Dual s) { return Dual(p_angle_of(c.v, s.v), c.v * s.d - s.v * c.d); }
__device__ inline double p_asin(double x) { return fx::asin(x); }
__device__ inline Dual p_asin(Dual x) {
  double r, ir;
  fx::sqrt_rsqrt((1.0 - x.v) * (1.0 + x.v), r, ir);
  return Dual(fx::asin(x.v), r > 0.0 ? x.d * ir : 0.0);
}
// erf(x) and exp(-x^2) / sqrt(pi)
constexpr double kInvSqrtPi = 0.5641895835477562869;
__device__ inline void p_erf(double x, double& ef, double& ex) {
  ef = fx::erf(x);
  ex = fx::exp(-(x * x)) * kInvSqrtPi;
}
__device__ inline void p_erf(Dual x, Dual& ef, Dual& ex) {
  p_erf(x.v, ef.v, ex.v);
  ef.d = 2.0 * ex.v * x.d;
  ex.d = -x.v * ef.d;
}

// abdamp (src/abdamp.f90:36-51), irc = 1 / rcut
template <class F>
__device__ inline void abdamp_plain(double irc, F r2, F& damp, F& ddamp) {
  const F x = r2 * irc;
  damp = p_rcp(1.0 + x * x);
  ddamp = (-4.0 * irc) * (x * (damp * damp));
}

// Coulomb energy of a pair per charge product: 1 / r, or the Zahn form
__device__ inline double pair_coulomb(const Dev& D, double r, double oner) {
  return D.zahn ? (q_erfc<double>(D.zahn_a * r) * oner) - D.zahn_par * (r - D.coul_cut) : oner;
}

// Bond stretch, generalised Lennard-Jones (src/ff_eg.f90:87-163):
// e = k (1 + (r0/r)^a - 2 (r0/r)^(a/2)).
template <class F>
__device__ inline F bond_plain(const Dev& D, const Tables<double>& T, const BeadPos& x, int m, Contrib<F>& c,
                               F* vir = nullptr) {
  const unsigned at = __ldg(D.bond + m);
  const int i = lo16(at), j = hi16(at);
  F rb[3], r, ir;
  disp<F>(x, i, j, rb);
  p_root(dot3(rb, rb), r, ir);
  const double* v = T.bond + m;
  const double rij = __ldg(v), kij = __ldg(v + D.st[0]), aai = __ldg(v + 2 * D.st[0]);
  const F pa2 = p_pow(rij * ir, aai / 2), pa = pa2 * pa2;
  const F fac = (aai * kij) * (pa2 - pa) * (ir * ir);
  c.na = 2;
  c.a[0] = i;
  c.a[1] = j;
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    c.g[0][d] = fac * rb[d];
    c.g[1][d] = -c.g[0][d];
  }
  if (vir) *vir = dot3(rb, c.g[0]);
  return kij * (1. + pa - 2. * pa2);
}

// Angle bend with abdamp damping (src/ff_eg.f90:167-299).
template <class F>
__device__ inline F angle_plain(const Dev& D, const Tables<double>& T, const BeadPos& x, int m, Contrib<F>& c,
                                F* vir = nullptr) {
  const uint2 at = __ldg(D.angl + m);
  const int i = lo16(at.x), j = hi16(at.x), k = (int)at.y, st = D.st[1];
  const double* v = T.angl + m;
  const double c0 = __ldg(v), kijk = __ldg(v + st), cc0 = __ldg(v + 2 * st);
  F vab[3], vcb[3], vp[3], al, ial, bl, ibl;
  disp<F>(x, i, j, vab);
  disp<F>(x, k, j, vcb);
  const F rab2 = dot3(vab, vab), rcb2 = dot3(vcb, vcb);
  cross(vcb, vab, vp);
  const F vpl = dot3(vp, vp);
  F rp = F(0), irp;
  if (vpl > 0.0) p_root(vpl, rp, irp);
  irp = p_rcp(rp + 1e-14);
  p_root(rab2, al, ial);
  p_root(rcb2, bl, ibl);
  F cosa = (al > 0.0 && bl > 0.0) ? dot3(vab, vcb) * (ial * ibl) : F(0);
  cosa = fmin(F(1), fmax(F(-1), cosa));
  F dampij, damp2ij, dampjk, damp2jk;
  abdamp_plain<F>(__ldg(v + 4 * st), rab2, dampij, damp2ij);
  abdamp_plain<F>(__ldg(v + 5 * st), rcb2, dampjk, damp2jk);
  const F damp = dampij * dampjk;
  F ea, deddt, sth, is;
  if (__ldg(v + 3 * st) != 0.0) {  // linear reference angle: harmonic in theta
    F theta;
    p_angle(cosa, theta, sth);
    const F dt = theta - c0;
    ea = kijk * (dt * dt);
    deddt = (2.0 * kijk) * dt;
  } else {  // harmonic in cos(theta)
    p_root((1.0 - cosa) * (1.0 + cosa), sth, is);
    const F dd = cosa - cc0;
    ea = kijk * (dd * dd);
    deddt = (-2.0 * kijk) * (sth * dd);
  }
  F deda[3], dedc[3];
  cross(vab, vp, deda);
  cross(vcb, vp, dedc);
  const F w = deddt * irp * damp, wa = -w * (ial * ial), wc = w * (ibl * ibl);
  const F k1 = ea * damp2ij * dampjk, k2 = ea * damp2jk * dampij;
  c.na = 3;
  c.a[0] = i;
  c.a[1] = j;
  c.a[2] = k;
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    c.g[0][d] = deda[d] * wa + k1 * vab[d];
    c.g[2][d] = dedc[d] * wc + k2 * vcb[d];
    c.g[1][d] = -c.g[0][d] - c.g[2][d];
  }
  if (vir) *vir = dot3(vab, c.g[0]) + dot3(vcb, c.g[2]);
  return ea * damp;
}

// Torsions (erf-blended cosine series, src/ff_eg.f90:303-440, the angle of
// src/valijkl.f90 in [0, pi]) and inversions (tors type 2, src/ff_eg.f90:441-618).
template <class F>
__device__ inline F torsion_plain(const Dev& D, const Tables<double>& T, const BeadPos& x, int m, Contrib<F>& c,
                                  F* vir = nullptr) {
  const double pi = 3.1415926535897932384626433832795029;
  const double pi2 = 6.28318530717958623199592693708837;
  const uint4 at = __ldg(D.tors + m);
  const int i = lo16(at.x), j = hi16(at.x), k = lo16(at.y), l = hi16(at.y), nt = (int)(at.z & 255u), type = (int)(at.z >> 8);
  const int st = D.st[2];
  auto vt = [&](int c) { return __ldg(T.tors + c * st + m); };
  const double phi0 = vt(0);
  F vab[3], vcb[3], vdc[3];
  F et, dij, dampij, dampjk, dampX, d2ij, d2jk, d2X;
  c.na = 4;
  c.a[0] = i;
  c.a[1] = j;
  c.a[2] = k;
  c.a[3] = l;
  if (type != 2) {
    disp<F>(x, i, j, vab);
    disp<F>(x, j, k, vcb);
    disp<F>(x, k, l, vdc);
    const F rcb2 = dot3(vcb, vcb);
    abdamp_plain<F>(vt(14), dot3(vab, vab), dampij, d2ij);
    abdamp_plain<F>(vt(15), rcb2, dampjk, d2jk);
    abdamp_plain<F>(vt(16), dot3(vdc, vdc), dampX, d2X);
    F na[3], nb[3], nan_, ina, nbn, inb, L, iL, phi, sinphi;
    cross(vab, vcb, na);
    cross(vcb, vdc, nb);
    p_root(dot3(na, na), nan_, ina);
    p_root(dot3(nb, nb), nbn, inb);
    p_root(rcb2, L, iL);
    // the normals are normalised where longer than 1e-14 (valijkl); where one is not
    // (three atoms in line) the angle is the arc cosine of the product so formed, and its
    // derivative is left out
    const bool bent = nan_ > 1e-14 && nbn > 1e-14;
    const F ua = nan_ > 1e-14 ? ina : F(1), ub = nbn > 1e-14 ? inb : F(1);
    F s = dot3(na, nb) * ua * ub;
    // |na x nb| = |rb| |na . rc|; in line 1, with which p_angle_of takes the arc cosine
    const F tr = dot3(na, vdc);
    sinphi = bent ? (L * (ua * ub)) * fabs(tr) : F(1);
    if (bent && ::fabs(::fabs(ad::val(s)) - 1.0) < 1e-14) {
      s = ad::val(s) >= 0 ? F(1.0) : F(-1.0);
      sinphi = F(0);
    }
    phi = p_angle_of(s, sinphi);
    F ef, expo;
    p_erf(phi - pi, ef, expo);
    const F h1 = 0.5 - 0.5 * ef, h2 = 0.5 + 0.5 * ef;
    et = F(0);
    dij = F(0);
    for (int it = 0; it < nt; ++it) {
      const double rn = vt(2 + 3 * it), ph = vt(3 + 3 * it), vn = vt(4 + 3 * it);
      F s1, c1, s2, c2;
      p_sincos(rn * (phi - phi0) + ph, s1, c1);
      p_sincos(rn * (phi + (phi0 - pi2)) + ph, s2, c2);
      const F a = vn * h1, b = vn * h2;
      et = et + a * (1.0 + c1) + b * (1.0 + c2);
      dij = dij + expo * (vn * (c2 - c1)) - rn * (a * s1 + b * s2);
    }
    et = et * vt(1);
    const F damp = dampjk * dampij * dampX;
    dij = dij * (vt(1) * damp);
    // dphi/dr of the unsigned angle, s = sign(na . rc), rb = -vcb and so on:
    //   dphi/dr_i = -s |rb| na / |na|^2,  dphi/dr_l = s |rb| nb / |nb|^2,
    //   dphi/dr_j = -dphi/dr_i + s (u + v),  dphi/dr_k = -dphi/dr_l - s (u + v),
    //   u = (ra.rb) na / (|na|^2 |rb|),  v = (rc.rb) nb / (|nb|^2 |rb|);
    // none where the reference's denominator |na| |nb| sin(phi) is below 1e-14 (nor
    // where it is no number: the reciprocals are infinite then)
    F wa = F(0), wb = F(0), wu = F(0), wv = F(0);
    if (bent && nan_ * nbn * sinphi >= 1e-14) {
      const F ia2 = ua * ua, ib2 = ub * ub;
      const F w = tr < 0.0 ? dij : -dij;
      const F wl = w * L, wi = w * iL;
      wa = wl * ia2;
      wb = wl * ib2;
      wu = wi * ia2 * dot3(vab, vcb);
      wv = wi * ib2 * dot3(vdc, vcb);
    }
    const F k1 = et * d2ij * (dampjk * dampX), k2 = et * d2jk * (dampij * dampX), k3 = et * d2X * (dampij * dampjk);
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      const F uv = wu * na[d] + wv * nb[d], t2 = k2 * vcb[d];
      c.g[0][d] = k1 * vab[d] - wa * na[d];
      c.g[3][d] = wb * nb[d] - k3 * vdc[d];
      c.g[1][d] = uv - c.g[0][d] + t2;
      c.g[2][d] = -uv - c.g[3][d] - t2;
    }
    if (vir) *vir = tors_virial(vab, vcb, vdc, c);
    return et * damp;
  }
  // inversion: omega (src/omega.f90) and domegadr (src/domegadr.f90)
  F dda[3], ddb[3], ddc[3], ddd[3];
  disp<F>(x, j, i, vab);
  disp<F>(x, j, k, vcb);
  disp<F>(x, j, l, vdc);
  abdamp_plain<F>(vt(14), dot3(vab, vab), dampij, d2ij);
  abdamp_plain<F>(vt(15), dot3(vcb, vcb), dampjk, d2jk);
  abdamp_plain<F>(vt(16), dot3(vdc, vdc), dampX, d2X);
  const F re[3] = {-vab[0], -vab[1], -vab[2]};  // r_i - r_j
  const F rd[3] = {-vcb[0], -vcb[1], -vcb[2]};  // r_k - r_j
  F rv[3];
  disp<F>(x, l, i, rv);                          // r_l - r_i
  F rn[3], rnn, irn, rvn, irv, cosom, icos;
  cross(re, rd, rn);
  p_root(dot3(rn, rn), rnn, irn);
  p_root(dot3(rv, rv), rvn, irv);
  F sinom = dot3(rn, rv);
  if (rnn > 1e-14) sinom = sinom * irn;
  if (rvn > 1e-14) sinom = sinom * irv;
  const F om = p_asin(sinom);
  p_root((1.0 - sinom) * (1.0 + sinom), cosom, icos);
  const F rdme[3] = {rd[0] - re[0], rd[1] - re[1], rd[2] - re[2]};
  F rve[3], rne[3], rdv[3], rdn[3], rvdme[3], rndme[3];
  cross(rv, re, rve);
  cross(rn, re, rne);
  cross(rd, rv, rdv);
  cross(rd, rn, rdn);
  cross(rv, rdme, rvdme);
  cross(rn, rdme, rndme);
  const F nenner = rnn * rvn * cosom;
  if (above_1em14(nenner)) {
    const F on = p_rcp(nenner), f1 = sinom * (rvn * irn), f2 = sinom * (rnn * irv);
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      dda[d] = on * (rdv[d] - rn[d] - (f1 * rdn[d] - f2 * rv[d]));
      ddb[d] = on * (rvdme[d] - f1 * rndme[d]);
      ddc[d] = on * (rve[d] - f1 * rne[d]);
      ddd[d] = on * (rn[d] - f2 * rv[d]);
    }
  } else {
#pragma unroll
    for (int d = 0; d < 3; ++d) dda[d] = ddb[d] = ddc[d] = ddd[d] = F(0);
  }
  const F damp = dampjk * dampij * dampX;
  if (vt(2) > 1e-6) {
    F s1, c1;
    p_sincos((om - phi0) + pi, s1, c1);
    et = (1.0 + c1) * vt(1);
    dij = -s1 * (vt(1) * damp);
  } else {
    double s0, c0;
    p_sincos(phi0, s0, c0);
    const F dd = cosom - c0;
    et = vt(1) * (dd * dd);
    dij = (-2.0 * vt(1)) * (sinom * dd * damp);
  }
  const F k1 = et * d2ij * (dampjk * dampX), k2 = et * d2jk * (dampij * dampX), k3 = et * d2X * (dampij * dampjk);
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    const F t1 = k1 * vab[d], t2 = k2 * vcb[d], t3 = k3 * vdc[d];
    c.g[0][d] = dij * dda[d] - t1;
    c.g[1][d] = dij * ddb[d] + t1 + t2 + t3;
    c.g[2][d] = dij * ddc[d] - t2;
    c.g[3][d] = dij * ddd[d] - t3;
  }
  if (vir) *vir = tors_virial(vab, vcb, vdc, c);
  return et * damp;
}

// One NCI pair (src/ff_nonb.f90): BJ-damped C6/C8 dispersion and, for
// r < 25 bohr, exponential repulsion, both times eps2 (:79-193); Coulomb
// within coul_cut (:337-416), eps1 q_i q_j / r or the Zahn form.
__device__ inline double pair_plain(const Dev& D, const Tables<double>& T, const BeadPos& x, int kp, Contrib<double>& c,
                                    double* vir = nullptr) {
  const unsigned at = __ldg(D.pair + kp);
  const int i1 = lo16(at), i2 = hi16(at);
  double v[kVPair];
#pragma unroll
  for (int k = 0; k < kVPair; ++k) v[k] = __ldg(T.pair + k * D.st[3] + kp);
  double vab[3], r, oner;
  disp<double>(x, i1, i2, vab);
  const double r2 = dot3(vab, vab);
  p_root(r2, r, oner);
  const double r4 = r2 * r2, r6 = r4 * r2, ir2 = oner * oner;
  const double i6 = p_rcp(r6 + v[0]), i8 = p_rcp(r6 * r2 + v[1]);
  const double d6 = v[2] * i6, d8 = v[3] * i8;
  // periodic: dispersion and repulsion only within vdw_cut (src/ff_nonb.f90:107)
  const bool vdw = !x.pbc || !(r > D.vdw_cut);
  double e = vdw ? -(d6 + d8) : 0.0;
  double drij = vdw ? r4 * (6.0 * (d6 * i6) + 8.0 * (d8 * i8) * r2) : 0.0;
  if (vdw && r < 25.0) {
    const double ar = v[5] * r, t = v[4] * p_exp(-ar) * oner;
    e = e + t;
    drij = drij - t * ir2 * (ar + 1.0);
  }
  if (!(r > D.coul_cut)) {
    const double e0 = v[6] * pair_coulomb(D, r, oner);
    e = e + e0;
    drij = drij - e0 * ir2;
  }
  c.na = 2;
  c.a[0] = i1;
  c.a[1] = i2;
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    c.g[0][d] = vab[d] * drij;
    c.g[1][d] = -c.g[0][d];
  }
  if (vir) *vir = r2 * drij;
  return e;
}

// The same with the tangent w, by hand: the gradient is drij v, its tangent drij w +
// drij' (2 v.w) v with drij' = d drij / d r^2.  Some 60 FP64 additions and
// multiplications, where dual arithmetic takes over 100.
__device__ inline Dual pair_tangent(const Dev& D, const Tables<double>& T, const BeadPos& x, int kp, Contrib<Dual>& c) {
  const unsigned at = __ldg(D.pair + kp);
  const int i1 = lo16(at), i2 = hi16(at);
  double v[kVPair];
#pragma unroll
  for (int k = 0; k < kVPair; ++k) v[k] = __ldg(T.pair + k * D.st[3] + kp);
  double vab[3], w[3], r, oner;
  disp<double>(x, i1, i2, vab);
#pragma unroll
  for (int d = 0; d < 3; ++d) w[d] = x.w[3 * i1 + d] - x.w[3 * i2 + d];
  const double r2 = dot3(vab, vab), vw = dot3(vab, w);
  p_root(r2, r, oner);
  const double r4 = r2 * r2, r6 = r4 * r2, r8 = r6 * r2, ir2 = oner * oner;
  const double i6 = p_rcp(r6 + v[0]), i8 = p_rcp(r8 + v[1]);
  const double d6 = v[2] * i6, d8 = v[3] * i8;
  const bool vdw = !x.pbc || !(r > D.vdw_cut);
  double e = 0.0, drij = 0.0, dd = 0.0;  // dd: r^2 drij'
  if (vdw) {
    const double f6 = 6.0 * (d6 * i6) * r4, f8 = 8.0 * (d8 * i8) * r6;
    e = -(d6 + d8);
    drij = f6 + f8;
    dd = f6 * fma(-6.0 * r6, i6, 2.0) + f8 * fma(-8.0 * r8, i8, 3.0);
    if (r < 25.0) {
      const double ar = v[5] * r, t = v[4] * p_exp(-ar) * oner, u = t * ir2;
      e = e + t;
      drij = fma(-u, ar + 1.0, drij);
      dd = fma(0.5 * u, fma(ar, ar + 3.0, 3.0), dd);
    }
  }
  double de = drij * vw;
  if (!(r > D.coul_cut)) {
    // the reference's gradient of the Zahn form is that of e0 as if it were ~ 1/r
    const double e0 = v[6] * pair_coulomb(D, r, oner), f = e0 * ir2;
    double e1 = -0.5 * f;  // d e0 / d r^2
    if (D.zahn) {
      const double zr = D.zahn_a * r;
      e1 = -0.5 * oner * v[6] * (oner * (2.0 * D.zahn_a * kInvSqrtPi * p_exp(-zr * zr) + oner * q_erfc<double>(zr)) + D.zahn_par);
    }
    e = e + e0;
    de = fma(2.0 * e1, vw, de);
    drij = drij - f;
    dd = dd + f - e1;
  }
  const double s = 2.0 * vw * ir2 * dd;
  c.na = 2;
  c.a[0] = i1;
  c.a[1] = i2;
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    c.g[0][d] = Dual(vab[d] * drij, fma(s, vab[d], drij * w[d]));
    c.g[1][d] = -c.g[0][d];
  }
  return Dual(e, de);
}

}  // namespace qmdff
}  // namespace cr
