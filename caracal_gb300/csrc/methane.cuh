// The XH4 part shared by the CH4 + H, CH4 + OH and GeH4 + OH surfaces
// (src/egrad_ch4h.f, src/egrad_ch4oh.f, src/egrad_geh4oh.f): switching
// functions, reference angles, the LEPS stretches of X-H_i, X-B and B-H_i
// (B the attacking atom), out-of-plane and in-plane bends, energy and gradient
// of one bead by one thread.
//
// The gradient is taken in reverse: each term adds to the derivatives with
// respect to what it depends on (the bond lengths r(XH_i), r(BH_i), r(XB), the
// unit vectors u_i = (X - H_i)/r(XH_i), the five switching functions of each
// bond, the six reference angles, the plane normals), and the chain to the
// atoms runs once at the end.  The reference differentiates forward, every
// term to every coordinate (three nested loops in opforce and ipforce); the
// same derivatives in reverse take about 1500 additions and multiplications
// instead of some 10000, which is what bounds the FP64 form, and far fewer
// live values, which is what bounds the mixed one (255 registers and spills).
// FP64 exponentials, divisions, roots and arc cosines run on the integer pipe
// (fx64.cuh).  Measured against the forward form, whole runs: CH4 + H 1000 x
// 32 plain, 20 steps 12.9 -> 5.28 ms; 4096 x 32 mixed, 40 steps 19.3 -> 14.4 ms;
// CH4 + OH 512 x 64 mixed, 40 steps 7.68 -> 6.31 ms.  Mixed force error over
// 16 384 thermal beads (2-norm): CH4 + H 7.8e-8 -> 6.7e-8, CH4 + OH 5.3e-8 ->
// 4.9e-8, GeH4 + OH 4.3e-8 -> 4.3e-8.
//
// In FP64 1 - tanh(a) and its derivative come from one exponential:
// s = 2/(1 + e^2a), ds/da = -s (2 - s) = -1/cosh^2 a.
#pragma once
#include <cuda_runtime.h>

#include <type_traits>

#include "ff32.cuh"
#include "fx64.cuh"

namespace cr {
namespace methane {

template <class F> __device__ inline F m_exp(F x);
template <> __device__ inline double m_exp<double>(double x) { return fx::exp(x); }
template <> __device__ inline float m_exp<float>(float x) { return expf(x); }
template <class F> __device__ inline F m_rcp(F x);
template <> __device__ inline double m_rcp<double>(double x) { return fx::rcp(x); }
template <> __device__ inline float m_rcp<float>(float x) { return __frcp_rn(x); }
template <class F> __device__ inline F m_div(F a, F b);
template <> __device__ inline double m_div<double>(double a, double b) { return fx::div(a, b); }
template <> __device__ inline float m_div<float>(float a, float b) { return a * __frcp_rn(b); }
template <class F> __device__ inline F m_sqrt(F x);
template <> __device__ inline double m_sqrt<double>(double x) { return fx::sqrt(x); }
template <> __device__ inline float m_sqrt<float>(float x) { return sqrtf(x); }
template <class F> __device__ inline F m_rsqrt(F x);
template <> __device__ inline double m_rsqrt<double>(double x) { return fx::rsqrt(x); }
template <> __device__ inline float m_rsqrt<float>(float x) { return __frcp_rn(sqrtf(x)); }
template <class F> __device__ inline F m_acos(F x);
template <> __device__ inline double m_acos<double>(double x) { return fx::acos(x); }
template <> __device__ inline float m_acos<float>(float x) { return acosf(x); }
// sqrt and its reciprocal
__device__ inline void m_root(double x, double& r, double& ir) { fx::sqrt_rsqrt(x, r, ir); }
__device__ inline void m_root(float x, float& r, float& ir) {
  r = sqrtf(x);
  ir = __frcp_rn(r);
}

// methane H i (0..3, nnh order) -> atom index; X and the attacking atom B
__device__ constexpr int NH(int i) { return i == 0 ? 2 : i == 1 ? 3 : i == 2 ? 4 : 0; }
constexpr int NC = 1, NB = 5;

template <class F>
__device__ inline F dot3(const F* a, const F* b) { return a[0] * b[0] + a[1] * b[1] + a[2] * b[2]; }

// Bond vectors, lengths and the reverse-mode accumulators of one bead.
template <class F>
struct Bonds {
  F tcb[3], tbh[4][3];          // X - B, B - H_i
  F rcb, ircb, rch[4], irch[4], rbh[4], irbh[4];
  F u[4][3];                    // (X - H_i) / r(XH_i)
  F drcb, drch[4], drbh[4];     // dV/dr (the mixed form's stretches apart)
  F wu[4][3];                   // dV/du_i
  F gh[4][3];                   // dV/dH_i of the plane normals
};

// Float pairs of the mixed form: bond vectors, lengths and the stretches'
// dV/dr, which are small differences of large terms.
struct Pairs {
  ff tcb[3], tch[4][3], tbh[4][3], rch[4];
  ff drcb, drch[4], drbh[4];    // over r for cb and bh: dV/dr / r
};

// A switching function s = 1 - tanh(arg) as t = tanh(arg) and ds =
// -darg / cosh(arg)^2.  FP64: one exponential; FP32: t itself, whose rounding
// is relative (the products s_i s_j - 1 below are small differences).
__device__ inline void tanh_switch(double arg, double darg, double& t, double& ds) {
  const double s = 2.0 * fx::rcp(1.0 + fx::exp(2.0 * arg));
  t = 1.0 - s;
  ds = -darg * (s * (2.0 - s));
}
__device__ inline void tanh_switch(float arg, float darg, float& t, float& ds) {
  t = tanhf(arg);
  ds = -darg * ((1.f - t) * (1.f + t));
}
// s_i s_j - 1 of two switching functions
template <class F>
__device__ inline F product_m1(F ti, F tj) { return ti * tj - (ti + tj); }
// with Caracal's tanh(19) = 1 cutoff (switchf)
template <class F>
__device__ inline void switch_fn(F arg, F darg, F& t, F& ds) {
  if (arg < F(19.0)) {
    tanh_switch(arg, darg, t, ds);
  } else {
    t = F(1);
    ds = F(0);
  }
}

// index of the pair (i, j), i != j, of the six of four bonds
__device__ constexpr int pair_of(int i, int j) {
  const int a = i < j ? i : j, b = i < j ? j : i;
  return a == 0 ? b - 1 : a == 1 ? b + 1 : 5;
}

// Bond lengths and unit vectors from tcb, tch, tbh.
template <class F>
__device__ inline void lengths(const F (&tch)[4][3], Bonds<F>& G) {
  m_root(dot3(G.tcb, G.tcb), G.rcb, G.ircb);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    m_root(dot3(tch[i], tch[i]), G.rch[i], G.irch[i]);
    m_root(dot3(G.tbh[i], G.tbh[i]), G.rbh[i], G.irbh[i]);
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      G.u[i][d] = tch[i][d] * G.irch[i];
      G.wu[i][d] = F(0);
      G.gh[i][d] = F(0);
    }
    G.drch[i] = F(0);
    G.drbh[i] = F(0);
  }
  G.drcb = F(0);
}

// LEPS stretches, FP64 form: the energy, and dV/dr into G.
template <class K>
__device__ inline double stretch_plain(Bonds<double>& G) {
  constexpr double sqch = K::d1ch + K::d3ch, dfch = K::d1ch - K::d3ch;
  constexpr double sqhh = K::d1hh + K::d3hh, dfhh = K::d1hh - K::d3hh;
  constexpr double sqcb = K::d1cb + K::d3cb, dfcb = K::d1cb - K::d3cb;
  // 1/2 (d1 (e^2 - 2 e) +- d3 (e^2 + 2 e)) = 1/2 (sq e^2 - 2 df e), 1/2 (df e^2 - 2 sq e)
  const double rav = (G.rch[0] + G.rch[1] + G.rch[2] + G.rch[3]) * 0.25;
  const double arga = K::c1ch * (rav - K::r0ch);
  double ach = K::a1ch + K::b1ch, dach = 0.0;  // dach: d ach / d r(XH_j)
  if (arga < 19.0) {
    const double s = 2.0 * fx::rcp(1.0 + fx::exp(2.0 * arga));  // 1 - tanh
    ach = ach - K::b1ch * 0.5 * s;
    dach = (K::b1ch * K::c1ch * 0.125) * (s * (2.0 - s));
  }
  const double ecb1 = fx::exp(-K::acb * (G.rcb - K::r0cb)), ecb2 = ecb1 * ecb1;
  const double qcb = 0.5 * sqcb * ecb2 - dfcb * ecb1, jcb = 0.5 * dfcb * ecb2 - sqcb * ecb1;
  const double dqcb = -K::acb * (sqcb * ecb2 - dfcb * ecb1), djcb = -K::acb * (dfcb * ecb2 - sqcb * ecb1);
  double V = 4.0 * qcb, bach = 0.0, drcb = 4.0 * dqcb;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const double x = G.rch[i] - K::r0ch;
    const double c1 = fx::exp(-ach * x), c2 = c1 * c1;
    const double h1 = fx::exp(-K::ahh * (G.rbh[i] - K::r0hh)), h2 = h1 * h1;
    const double qch = 0.5 * sqch * c2 - dfch * c1, jch = 0.5 * dfch * c2 - sqch * c1;
    const double qbh = 0.5 * sqhh * h2 - dfhh * h1, jbh = 0.5 * dfhh * h2 - sqhh * h1;
    const double e12 = jch - jcb, e23 = jcb - jbh, e31 = jbh - jch;
    double root, iroot;
    m_root((e12 * e12 + e23 * e23 + e31 * e31) * 0.5, root, iroot);
    V += qch + qbh - root;
    const double fj = -0.5 * iroot;
    // dV/dz of z = ach (r - r0ch); dV/dr(XB), dV/dr(BH_i)
    const double dz = -((sqch * c2 - dfch * c1) + (e12 - e31) * fj * (dfch * c2 - sqch * c1));
    drcb += (e23 - e12) * fj * djcb;
    G.drbh[i] = -K::ahh * ((sqhh * h2 - dfhh * h1) + (e31 - e23) * fj * (dfhh * h2 - sqhh * h1));
    G.drch[i] = ach * dz;
    bach = fma(x, dz, bach);
  }
  G.drcb = drcb;
  const double b = bach * dach;
#pragma unroll
  for (int i = 0; i < 4; ++i) G.drch[i] += b;
  return V;
}

// The same in float pairs (mixed form): T_i, U, W_i are small differences of
// large Q and J derivatives near the bond minimum, so the scalars are formed
// in pairs; their dV/dr go into X.
template <class K>
__device__ inline float stretch_pairs(const Bonds<float>& G, Pairs& X) {
  constexpr ff Sqch = ff_const(K::d1ch + K::d3ch), Dfch = ff_const(K::d1ch - K::d3ch);
  constexpr ff Sqhh = ff_const(K::d1hh + K::d3hh), Dfhh = ff_const(K::d1hh - K::d3hh);
  constexpr ff Sqcb = ff_const(K::d1cb + K::d3cb), Dfcb = ff_const(K::d1cb - K::d3cb);
  constexpr ff R0ch = ff_const(K::r0ch), R0hh = ff_const(K::r0hh), R0cb = ff_const(K::r0cb);
  constexpr ff Acb = ff_const(K::acb), Ahh = ff_const(K::ahh);
  auto norm3 = [](const ff (&v)[3]) { return ff_sqrt(v[0] * v[0] + v[1] * v[1] + v[2] * v[2]); };
  // ach = a1 + b1 (tanh(arga) + 1) / 2 = a1 + b1 / (1 + exp(-2 arga)) as a
  // float pair: its rounding enters every exponent of the cancelling Q and J
  const float arga = float(K::c1ch) * ((G.rch[0] + G.rch[1] + G.rch[2] + G.rch[3]) * 0.25f - float(K::r0ch));
  ff ach = ff_const(K::a1ch + K::b1ch);
  float dach = 0.f;
  if (arga < 19.0f) {
    constexpr ff A1 = ff_const(K::a1ch), B1 = ff_const(K::b1ch), C1 = ff_const(K::c1ch);
    const ff ravx = (X.rch[0] + X.rch[1] + X.rch[2] + X.rch[3]) * 0.25f;
    const ff e2 = ff_exp(-(C1 * (ravx - R0ch)) * 2.f);
    ach = A1 + B1 / (ff_from(1.f) + e2);
    const float s = 2.f * e2.hi * __frcp_rn(1.f + e2.hi);  // 1 - tanh(arga)
    dach = float(K::b1ch * K::c1ch * 0.125) * (s * (2.f - s));
  }
  const ff rcb = norm3(X.tcb);
  const ff ecb1 = ff_exp(-(Acb * (rcb - R0cb))), ecb2 = ecb1 * ecb1;
  const ff sc2 = Sqcb * ecb2, sc1 = Sqcb * ecb1, fc2 = Dfcb * ecb2, fc1 = Dfcb * ecb1;
  const ff qcb = sc2 * 0.5f - fc1, jcb = fc2 * 0.5f - sc1;
  const ff dqcb = -(Acb * (sc2 - fc1)), djcb = -(Acb * (fc2 - sc1));
  ff V = qcb * 4.f, bach = ff_from(0.f), drcb = dqcb * 4.f;
#pragma unroll 1
  for (int i = 0; i < 4; ++i) {
    const ff rbh = norm3(X.tbh[i]), x = X.rch[i] - R0ch;
    const ff c1 = ff_exp(-(ach * x)), c2 = c1 * c1;
    const ff h1 = ff_exp(-(Ahh * (rbh - R0hh))), h2 = h1 * h1;
    const ff scc2 = Sqch * c2, scc1 = Sqch * c1, fcc2 = Dfch * c2, fcc1 = Dfch * c1;
    const ff shh2 = Sqhh * h2, shh1 = Sqhh * h1, fhh2 = Dfhh * h2, fhh1 = Dfhh * h1;
    const ff qch = scc2 * 0.5f - fcc1, jch = fcc2 * 0.5f - scc1;
    const ff qbh = shh2 * 0.5f - fhh1, jbh = fhh2 * 0.5f - shh1;
    const ff e12 = jch - jcb, e23 = jcb - jbh, e31 = jbh - jch;
    const ff root = ff_sqrt((e12 * e12 + e23 * e23 + e31 * e31) * 0.5f);
    V += qch + qbh - root;
    const ff fj = ff_recip(root) * -0.5f;
    const ff dz = -((scc2 - fcc1) + (e12 - e31) * fj * (fcc2 - scc1));
    drcb += (e23 - e12) * fj * djcb;
    X.drbh[i] = -(Ahh * ((shh2 - fhh1) + (e31 - e23) * fj * (fhh2 - shh1))) / rbh;
    X.drch[i] = ach * dz;
    bach += x * dz;
  }
  X.drcb = drcb / rcb;
  const ff b = bach * dach;
#pragma unroll
  for (int i = 0; i < 4; ++i) X.drch[i] += b;
  return ff_float(V);
}

// Switching functions, reference angles and both bends: the energy; dV/dr,
// dV/du and the plane normals' dV/dH into G.  th: H_k - H_j of the three
// hydrogens opposite bond i come from the bond vectors tch.
template <class F, class K>
__device__ inline F bends(const F (&tch)[4][3], const Pairs* X, Bonds<F>& G) {
  constexpr bool kPair = std::is_same<F, float>::value;
  const double tau = 1.9106332362490186;  // acos(-1/3)
  const double pi = 3.141592653589793;
  const F A = F(tau - K::tau_py), B = F(tau - 2.0 * pi / 3.0);
  // ---- switching functions (switchf)
  F t1[4], ds1[4], t2[4], ds2[4], t3[4], ds3[4], tp[4], dsp[4], tt[4], dst[4];  // tanh, d(1 - tanh)/dr
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const F r = G.rch[i], x = r - F(K::r0ch);
    const F y1 = r - F(K::b1s), y1_2 = y1 * y1, y1_4 = y1_2 * y1_2, y1_7 = F(K::a1s) * (y1_4 * y1_2 * y1);
    switch_fn<F>(x * (y1_7 * y1), y1_7 * (y1 + F(8) * x), t1[i], ds1[i]);
    const F y2 = r - F(K::b2s), y2_2 = y2 * y2, y2_5 = F(K::a2s) * (y2_2 * y2_2 * y2);
    switch_fn<F>(x * (y2_5 * y2), y2_5 * (y2 + F(6) * x), t2[i], ds2[i]);
    const F y3 = r - F(K::b3s), y3a = F(K::a3s) * y3;
    switch_fn<F>(x * (y3a * y3), y3a * (y3 + F(2) * x), t3[i], ds3[i]);
    tp[i] = F(1);
    dsp[i] = F(0);
    if (!K::sphi_cut || r < F(3.8)) {
      const F xc = r - F(K::cphi), xc2 = F(K::bphi) * (xc * xc);
      const F e = F(K::aphi) * m_exp<F>(xc2 * xc);
      const F arg = x * e;
      // FP32 only: past arg = 19, 1 - tanh is 0 in float and exp overflows
      // (GeH4 + OH, r > 17.9 A); FP64 follows the reference
      if (!kPair || arg < F(19.0)) tanh_switch(arg, e * (F(1) + F(3) * (x * xc2)), tp[i], dsp[i]);
    }
    tt[i] = F(1);
    dst[i] = F(0);
    if (r < F(3.8)) {
      const F xt = r - F(K::ctheta), xt2 = F(K::btheta) * (xt * xt);
      const F e = F(K::atheta) * m_exp<F>(xt2 * xt);
      tanh_switch(x * e, e * (F(1) + F(3) * (x * xt2)), tt[i], dst[i]);
    }
  }
  // ---- reference angles (refangles): theta0 - tau of the six bond pairs
  F th[6], bth[6];
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = i + 1; j < 4; ++j) {
      const int m = i != 0 && j != 0 ? 0 : i != 1 && j != 1 ? 1 : 2, n = 6 - i - j - m;
      th[pair_of(i, j)] = A * product_m1(tp[i], tp[j]) + B * product_m1(tt[m], tt[n]);
      bth[pair_of(i, j)] = F(0);
    }
  F V = F(0);
  // ---- out-of-plane bends (opbend, opforce, calcdelta)
  {
    F b3[4] = {F(0), F(0), F(0), F(0)};
    const F s3[4] = {F(1) - t3[0], F(1) - t3[1], F(1) - t3[2], F(1) - t3[3]};
    // tau as hi + lo: the difference of two ~1.9 rad angles keeps tau's rounding
    const F tau_lo = F(tau - (double)F(tau));
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int t[3] = {(i + 1) & 3, (i + 2) & 3, (i + 3) & 3};
      F a[3], b[3];  // H_k - H_j, H_l - H_j
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        a[d] = tch[t[0]][d] - tch[t[1]][d];
        b[d] = tch[t[0]][d] - tch[t[2]][d];
      }
      const F ab[3] = {a[1] * b[2] - a[2] * b[1], a[2] * b[0] - a[0] * b[2], a[0] * b[1] - a[1] * b[0]};
      const F in = m_rsqrt<F>(dot3(ab, ab));
      F c[3];  // (a x b) . u_m
#pragma unroll
      for (int k = 0; k < 3; ++k) c[k] = dot3(ab, G.u[t[k]]);
      // the reference swaps k and l for each negative one (src/egrad_ch4h.f
      // :757-764, cumulative): a x b changes sign with each swap
      const bool flip = (c[0] < F(0)) != (c[1] < F(0)) != (c[2] < F(0));
      const F sn = flip ? -in : in;
      const F nrm[3] = {ab[0] * sn, ab[1] * sn, ab[2] * sn};
      const F p01 = s3[t[0]] * s3[t[1]], p02 = s3[t[0]] * s3[t[2]], p12 = s3[t[1]] * s3[t[2]];
      const F q = t3[i], all = p01 * s3[t[2]], sw = q * all;
      F sum2 = F(0), sum4 = F(0), w[3] = {F(0), F(0), F(0)};
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        const int m = t[k];
        const F arg = -(c[k] * sn);
        const F dl = (m_acos<F>(arg) - F(tau)) - (th[pair_of(i, m)] + tau_lo);
        const F d2 = dl * dl;
        sum2 += d2;
        sum4 += d2 * d2;
        const F coef = (sw * dl) * (F(2.0 * K::fch3) + F(4.0 * K::hch3) * d2);
        bth[pair_of(i, m)] -= coef;
        const F ba = coef * m_rsqrt<F>(F(1) - arg * arg);  // -dV/d arg, arg = -n.u_m
#pragma unroll
        for (int d = 0; d < 3; ++d) {
          w[d] += ba * G.u[m][d];
          G.wu[m][d] += ba * nrm[d];
        }
      }
      const F E = F(K::fch3) * sum2 + F(K::hch3) * sum4;
      V += sw * E;
      b3[i] -= E * all;
      const F Eq = E * q;
      b3[t[0]] += Eq * p12;
      b3[t[1]] += Eq * p02;
      b3[t[2]] += Eq * p01;
      // dV/d(a x b) = sn (w - n (n.w)), then b x y on H_k and y x a on H_l
      const F nw = dot3(nrm, w);
      F y[3];
#pragma unroll
      for (int d = 0; d < 3; ++d) y[d] = sn * (w[d] - nrm[d] * nw);
      const F gk[3] = {b[1] * y[2] - b[2] * y[1], b[2] * y[0] - b[0] * y[2], b[0] * y[1] - b[1] * y[0]};
      const F gl[3] = {y[1] * a[2] - y[2] * a[1], y[2] * a[0] - y[0] * a[2], y[0] * a[1] - y[1] * a[0]};
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        G.gh[t[1]][d] += gk[d];
        G.gh[t[2]][d] += gl[d];
        G.gh[t[0]][d] -= gk[d] + gl[d];
      }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) G.drch[i] += b3[i] * ds3[i];
  }
  // ---- in-plane bends (ipbend, ipforce)
  {
    const F f0 = F(K::fkinf + K::ak), g0 = F((K::fkinf + K::ak) - K::fkinf);
    F f1[4], df1c[4], df1h[4], bf1[4], b1[4], b2[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const F rb = G.rbh[i], xh = rb - F(K::r0hh), x = G.rch[i] - F(K::r0ch), x2 = x * x;
      const F e1 = m_exp<F>(-F(K::aa1) * rb * rb), e2 = F(K::aa3) * m_exp<F>(-F(K::aa4) * xh * xh);
      const F a1 = F(1) - e1, a2 = F(K::aa2) + e2, eg = m_exp<F>(-a2 * x2);
      f1[i] = a1 * eg;
      df1c[i] = F(-2) * x * (f1[i] * a2);
      df1h[i] = F(2.0 * K::aa1) * rb * (e1 * eg) + F(2.0 * K::aa4) * xh * e2 * (x2 * f1[i]);
      bf1[i] = b1[i] = b2[i] = F(0);
    }
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
      for (int j = i + 1; j < 4; ++j) {
        const int m = i != 0 && j != 0 ? 0 : i != 1 && j != 1 ? 1 : 2, n = 6 - i - j - m;
        const F fk = f0 + (f0 * product_m1(t1[i], t1[j]) + g0 * product_m1(t2[m], t2[n]));
        F cs, dth;
        if constexpr (kPair) {
          // theta - tau as asin(sin(theta - tau)) from a float-pair cosine:
          // theta - th0 is a small difference of two ~1.9 rad angles, which
          // acosf of an FP32 cosine would leave with ~1e-7 rad of error
          const ff c = (X->tch[i][0] * X->tch[j][0] + X->tch[i][1] * X->tch[j][1] + X->tch[i][2] * X->tch[j][2]) /
                       (X->rch[i] * X->rch[j]);
          constexpr ff kCosTau = ff_const(-1.0 / 3.0), kSinTau = ff_const(0.94280904158206336587);
          const ff y = ff_sqrt(ff_from(1.f) - c * c) * kCosTau - c * kSinTau;
          cs = ff_float(c);
          const float dtau = fabsf(y.hi) < 0.9f ? asinf(y.hi) + y.lo * m_rsqrt<float>(1.f - y.hi * y.hi)
                                                : acosf(cs) - F(tau);
          dth = dtau - th[pair_of(i, j)];
        } else {
          cs = dot3(G.u[i], G.u[j]);
          dth = (m_acos<F>(cs) - F(tau)) - th[pair_of(i, j)];
        }
        const F h = F(0.5) * dth * dth, ff1 = f1[i] * f1[j], kf = fk * ff1, hk = h * fk, bk = h * ff1;
        V += h * kf;
        bf1[i] += hk * f1[j];
        bf1[j] += hk * f1[i];
        const F bk0 = bk * f0, bkg = bk * g0, kd = kf * dth;
        b1[i] += bk0 * (F(1) - t1[j]);
        b1[j] += bk0 * (F(1) - t1[i]);
        b2[m] += bkg * (F(1) - t2[n]);
        b2[n] += bkg * (F(1) - t2[m]);
        bth[pair_of(i, j)] -= kd;
        const F bc = kd * m_rsqrt<F>(F(1) - cs * cs);  // -dV/d cos
#pragma unroll
        for (int d = 0; d < 3; ++d) {
          G.wu[i][d] -= bc * G.u[j][d];
          G.wu[j][d] -= bc * G.u[i][d];
        }
      }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      G.drch[i] += bf1[i] * df1c[i] + b1[i] * ds1[i] + b2[i] * ds2[i];
      G.drbh[i] += bf1[i] * df1h[i];
    }
  }
  // ---- the reference angles' share
  F bp[4] = {F(0), F(0), F(0), F(0)}, bt[4] = {F(0), F(0), F(0), F(0)};
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = i + 1; j < 4; ++j) {
      const int m = i != 0 && j != 0 ? 0 : i != 1 && j != 1 ? 1 : 2, n = 6 - i - j - m;
      const F ba = bth[pair_of(i, j)] * A, bb = bth[pair_of(i, j)] * B;
      bp[i] += ba * (F(1) - tp[j]);
      bp[j] += ba * (F(1) - tp[i]);
      bt[m] += bb * (F(1) - tt[n]);
      bt[n] += bb * (F(1) - tt[m]);
    }
#pragma unroll
  for (int i = 0; i < 4; ++i) G.drch[i] += bp[i] * dsp[i] + bt[i] * dst[i];
  return V;
}

// dV/du_i to the part of dV/d(X - H_i) across the bond
template <class F>
__device__ inline void across(const Bonds<F>& G, int i, F (&g)[3]) {
  const F uw = dot3(G.u[i], G.wu[i]);
#pragma unroll
  for (int d = 0; d < 3; ++d) g[d] = (G.wu[i][d] - G.u[i][d] * uw) * G.irch[i];
}

// The chain to the atoms: adds the XH4 part to g (atoms of NH, NC, NB).
__device__ inline void chain(const Bonds<double>& G, double* g) {
  const double kc = G.drcb * G.ircb;
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    g[3 * NC + d] += G.tcb[d] * kc;
    g[3 * NB + d] -= G.tcb[d] * kc;
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    double a[3];
    across(G, i, a);
    const double kb = G.drbh[i] * G.irbh[i];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      const double t = fma(G.u[i][d], G.drch[i], a[d]), w = G.tbh[i][d] * kb;
      g[3 * NC + d] += t;
      g[3 * NB + d] += w;
      g[3 * NH(i) + d] += G.gh[i][d] - (t + w);
    }
  }
}

// Mixed form: the stretches' part in float pairs (their vectors cancel on
// each atom), the bends' radial derivatives joined to them.
__device__ inline void chain(const Bonds<float>& G, const Pairs& X, ff* g) {
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    const ff t = X.tcb[d] * X.drcb;
    g[3 * NC + d] += t;
    g[3 * NB + d] -= t;
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    float a[3];
    across(G, i, a);
    const ff kc = (X.drch[i] + G.drch[i]) / X.rch[i], kb = X.drbh[i] + G.drbh[i] * G.irbh[i];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      const ff t = X.tch[i][d] * kc + a[d], w = X.tbh[i][d] * kb;
      g[3 * NC + d] += t;
      g[3 * NB + d] += w;
      g[3 * NH(i) + d] += -(t + w) + G.gh[i][d];
    }
  }
}

// Positions in Angstrom as float pairs (bohr times 0.52918, POT_ch4h), from
// the FP64 bits: FP64 instructions would cost 64 cycles each.
template <int N3>
__device__ inline void scaled_pairs(const double (&q)[N3], ff (&x)[N3]) {
  constexpr ff kA = ff_const(0.52918);
#pragma unroll
  for (int k = 0; k < N3; ++k) x[k] = ff_split(q[k]) * kA;
}

// Bond vectors and lengths; the XH4 + B atoms come first in a bead.
template <int N3>
__device__ inline void bond_vectors(const double (&q)[N3], Bonds<double>& G, double (&tch)[4][3]) {
  double x[18];
#pragma unroll
  for (int k = 0; k < 18; ++k) x[k] = q[k] * 0.52918;
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    G.tcb[d] = x[3 * NC + d] - x[3 * NB + d];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      tch[i][d] = x[3 * NC + d] - x[3 * NH(i) + d];
      G.tbh[i][d] = x[3 * NB + d] - x[3 * NH(i) + d];
    }
  }
  lengths(tch, G);
}
template <int N3>
__device__ inline void bond_vectors(const ff (&x)[N3], Bonds<float>& G, Pairs& X, float (&tch)[4][3]) {
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    X.tcb[d] = x[3 * NC + d] - x[3 * NB + d];
    G.tcb[d] = ff_float(X.tcb[d]);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      X.tch[i][d] = x[3 * NC + d] - x[3 * NH(i) + d];
      X.tbh[i][d] = x[3 * NB + d] - x[3 * NH(i) + d];
      tch[i][d] = ff_float(X.tch[i][d]);
      G.tbh[i][d] = ff_float(X.tbh[i][d]);
    }
  }
#pragma unroll
  for (int i = 0; i < 4; ++i)
    X.rch[i] = ff_sqrt(X.tch[i][0] * X.tch[i][0] + X.tch[i][1] * X.tch[i][1] + X.tch[i][2] * X.tch[i][2]);
  lengths(tch, G);
}

}  // namespace methane
}  // namespace cr
