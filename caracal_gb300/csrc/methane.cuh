// The XH4 part shared by the CH4 + H, CH4 + OH and GeH4 + OH surfaces
// (src/egrad_ch4h.f, src/egrad_ch4oh.f, src/egrad_geh4oh.f): switching
// functions, reference angles, the LEPS stretches of X-H_i, X-B and B-H_i
// (B the attacking atom), out-of-plane and in-plane bends, energy and gradient
// of one bead by four lanes of a warp, one per X-H bond.
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
// Four lanes per bead: the four bonds' terms are the same instructions on
// other data, so one thread per bead spells them out four to six times, 13 000
// instructions in a row per step; fetching those, not executing them, took 42 %
// of the mixed step's cycles (ncu: 2.8 of 6.8 cycles per instruction without
// one).  A quad runs a quarter of the code, in half the registers; the lanes
// exchange what a term needs of the other bonds by shuffles (bond i ^ k is at
// lane i ^ k).  Per step, with the drift by fast transforms (ring_fast.cuh): CH4 + H
// 4096 x 32 mixed 122 -> 102 us, CH4 + OH 512 x 64 mixed 118 -> 80 us, plain 182 ->
// 165 us; whole runs CH4 + H 1000 x 32 mixed, with its children, 6.78 -> 5.77 ms.
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

constexpr unsigned kAll = 0xffffffffu;

template <class F> __device__ inline F m_exp(F x);
template <> __device__ inline double m_exp<double>(double x) { return fx::exp(x); }
template <> __device__ inline float m_exp<float>(float x) { return expf(x); }
template <class F> __device__ inline F m_rcp(F x);
template <> __device__ inline double m_rcp<double>(double x) { return fx::rcp(x); }
template <> __device__ inline float m_rcp<float>(float x) { return f_rcp(x); }
template <class F> __device__ inline F m_div(F a, F b);
template <> __device__ inline double m_div<double>(double a, double b) { return fx::div(a, b); }
template <> __device__ inline float m_div<float>(float a, float b) { return a * f_rcp(b); }
template <class F> __device__ inline F m_sqrt(F x);
template <> __device__ inline double m_sqrt<double>(double x) { return fx::sqrt(x); }
template <> __device__ inline float m_sqrt<float>(float x) {
  float r, ir;
  f_root(x, r, ir);
  return r;
}
template <class F> __device__ inline F m_rsqrt(F x);
template <> __device__ inline double m_rsqrt<double>(double x) { return fx::rsqrt(x); }
template <> __device__ inline float m_rsqrt<float>(float x) {
  float r, ir;
  f_root(x, r, ir);
  return ir;
}
template <class F> __device__ inline F m_acos(F x);
template <> __device__ inline double m_acos<double>(double x) { return fx::acos(x); }
template <> __device__ inline float m_acos<float>(float x) { return acosf(x); }
// sqrt and its reciprocal
__device__ inline void m_root(double x, double& r, double& ir) { fx::sqrt_rsqrt(x, r, ir); }
__device__ inline void m_root(float x, float& r, float& ir) {
  f_root(x, r, ir);
}

// methane H i (0..3, nnh order) -> atom index; X and the attacking atom B
__device__ inline int NH(int i) { return i == 3 ? 0 : i + 2; }
constexpr int NC = 1, NB = 5;

template <class F>
__device__ inline F dot3(const F* a, const F* b) { return a[0] * b[0] + a[1] * b[1] + a[2] * b[2]; }

// the value of bond i ^ k; of the lane src of the quad; the quad's sum
template <class F>
__device__ inline F of(F x, int k) { return __shfl_xor_sync(kAll, x, k); }
__device__ inline ff of(ff x, int k) { return ff{of(x.hi, k), of(x.lo, k)}; }
template <class F>
__device__ inline F from(F x, int src) { return __shfl_sync(kAll, x, src, 4); }
__device__ inline ff from(ff x, int src) { return ff{from(x.hi, src), from(x.lo, src)}; }
template <class F>
__device__ inline F quad_sum(F x) {
  x = x + of(x, 1);
  return x + of(x, 2);
}

// One lane's bond: vectors, lengths and reverse-mode accumulators.
template <class F>
struct Bond {
  F tcb[3], tch[3], tbh[3];     // X - B, X - H_i, B - H_i
  F rcb, ircb, rch, irch, rbh, irbh;
  F u[3];                       // (X - H_i) / r(XH_i)
  F drcb, drch, drbh;           // dV/dr (drcb of the bead, on every lane; the mixed form's stretches apart)
  F wu[3];                      // dV/du_i
  F gh[3];                      // dV/dH_i of the plane normals
};

// Float pairs of the mixed form: bond vectors, lengths and the stretches'
// dV/dr, which are small differences of large terms.
struct Pairs {
  ff tcb[3], tch[3], tbh[3], rch;
  ff drcb, drch, drbh;          // over r for cb and bh: dV/dr / r
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

// Bond lengths and the unit vector.
template <class F>
__device__ inline void lengths(Bond<F>& G) {
  m_root(dot3(G.tcb, G.tcb), G.rcb, G.ircb);
  m_root(dot3(G.tch, G.tch), G.rch, G.irch);
  m_root(dot3(G.tbh, G.tbh), G.rbh, G.irbh);
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    G.u[d] = G.tch[d] * G.irch;
    G.wu[d] = F(0);
    G.gh[d] = F(0);
  }
  G.drch = G.drbh = G.drcb = F(0);
}

// LEPS stretches, FP64 form: the energy (this lane's share), dV/dr into G.  The
// exponentials of X-B, of the mean X-H length and (CH4 + OH) of the further
// atom's stretch, whose argument is `more`, are one evaluation: lanes 0, 1, 2.
template <class K>
__device__ inline double stretch_plain(Bond<double>& G, int i, double more, double& more_exp) {
  constexpr double sqch = K::d1ch + K::d3ch, dfch = K::d1ch - K::d3ch;
  constexpr double sqhh = K::d1hh + K::d3hh, dfhh = K::d1hh - K::d3hh;
  constexpr double sqcb = K::d1cb + K::d3cb, dfcb = K::d1cb - K::d3cb;
  // 1/2 (d1 (e^2 - 2 e) +- d3 (e^2 + 2 e)) = 1/2 (sq e^2 - 2 df e), 1/2 (df e^2 - 2 sq e)
  const double arga = K::c1ch * (quad_sum(G.rch) * 0.25 - K::r0ch);
  const double ex = fx::exp(i == 0 ? -K::acb * (G.rcb - K::r0cb) : i == 1 ? 2.0 * arga : more);
  const double ecb1 = from(ex, 0), e2a = from(ex, 1);
  more_exp = from(ex, 2);
  double ach = K::a1ch + K::b1ch, dach = 0.0;  // dach: d ach / d r(XH_j)
  if (arga < 19.0) {
    const double s = 2.0 * fx::rcp(1.0 + e2a);  // 1 - tanh
    ach = ach - K::b1ch * 0.5 * s;
    dach = (K::b1ch * K::c1ch * 0.125) * (s * (2.0 - s));
  }
  const double ecb2 = ecb1 * ecb1;
  const double qcb = 0.5 * sqcb * ecb2 - dfcb * ecb1, jcb = 0.5 * dfcb * ecb2 - sqcb * ecb1;
  const double dqcb = -K::acb * (sqcb * ecb2 - dfcb * ecb1), djcb = -K::acb * (dfcb * ecb2 - sqcb * ecb1);
  const double x = G.rch - K::r0ch;
  const double c1 = fx::exp(-ach * x), c2 = c1 * c1;
  const double h1 = fx::exp(-K::ahh * (G.rbh - K::r0hh)), h2 = h1 * h1;
  const double qch = 0.5 * sqch * c2 - dfch * c1, jch = 0.5 * dfch * c2 - sqch * c1;
  const double qbh = 0.5 * sqhh * h2 - dfhh * h1, jbh = 0.5 * dfhh * h2 - sqhh * h1;
  const double e12 = jch - jcb, e23 = jcb - jbh, e31 = jbh - jch;
  double root, iroot;
  m_root((e12 * e12 + e23 * e23 + e31 * e31) * 0.5, root, iroot);
  const double fj = -0.5 * iroot;
  // dV/dz of z = ach (r - r0ch); dV/dr(XB), dV/dr(BH_i)
  const double dz = -((sqch * c2 - dfch * c1) + (e12 - e31) * fj * (dfch * c2 - sqch * c1));
  G.drcb = quad_sum(dqcb + (e23 - e12) * fj * djcb);
  G.drbh = -K::ahh * ((sqhh * h2 - dfhh * h1) + (e31 - e23) * fj * (dfhh * h2 - sqhh * h1));
  G.drch = fma(quad_sum(x * dz), dach, ach * dz);
  return qcb + qch + qbh - root;
}

// The same in float pairs (mixed form): T_i, U, W_i are small differences of
// large Q and J derivatives near the bond minimum, so the scalars are formed
// in pairs; their dV/dr go into X.
template <class K>
__device__ inline float stretch_pairs(const Bond<float>& G, Pairs& X, int i, ff more, ff& more_exp) {
  constexpr ff Sqch = ff_const(K::d1ch + K::d3ch), Dfch = ff_const(K::d1ch - K::d3ch);
  constexpr ff Sqhh = ff_const(K::d1hh + K::d3hh), Dfhh = ff_const(K::d1hh - K::d3hh);
  constexpr ff Sqcb = ff_const(K::d1cb + K::d3cb), Dfcb = ff_const(K::d1cb - K::d3cb);
  constexpr ff R0ch = ff_const(K::r0ch), R0hh = ff_const(K::r0hh), R0cb = ff_const(K::r0cb);
  constexpr ff Acb = ff_const(K::acb), Ahh = ff_const(K::ahh), C1 = ff_const(K::c1ch);
  auto norm3 = [](const ff (&v)[3]) { return ff_sqrt(v[0] * v[0] + v[1] * v[1] + v[2] * v[2]); };
  // ach = a1 + b1 (tanh(arga) + 1) / 2 = a1 + b1 / (1 + exp(-2 arga)) as a
  // float pair: its rounding enters every exponent of the cancelling Q and J
  const float arga = float(K::c1ch) * (quad_sum(G.rch) * 0.25f - float(K::r0ch));
  const ff rcb = norm3(X.tcb);
  const ff a_cb = -(Acb * (rcb - R0cb)), a_ch = -(C1 * (quad_sum(X.rch) * 0.25f - R0ch)) * 2.f;
  const ff ex = ff_exp(i == 0 ? a_cb : i == 1 ? a_ch : more);
  const ff ecb1 = from(ex, 0), e2 = from(ex, 1);
  more_exp = from(ex, 2);
  ff ach = ff_const(K::a1ch + K::b1ch);
  float dach = 0.f;
  if (arga < 19.0f) {
    constexpr ff A1 = ff_const(K::a1ch), B1 = ff_const(K::b1ch);
    ach = A1 + B1 / (ff_from(1.f) + e2);
    const float s = 2.f * e2.hi * f_rcp(1.f + e2.hi);  // 1 - tanh(arga)
    dach = float(K::b1ch * K::c1ch * 0.125) * (s * (2.f - s));
  }
  const ff ecb2 = ecb1 * ecb1;
  const ff sc2 = Sqcb * ecb2, sc1 = Sqcb * ecb1, fc2 = Dfcb * ecb2, fc1 = Dfcb * ecb1;
  const ff qcb = sc2 * 0.5f - fc1, jcb = fc2 * 0.5f - sc1;
  const ff dqcb = -(Acb * (sc2 - fc1)), djcb = -(Acb * (fc2 - sc1));
  const ff rbh = norm3(X.tbh), x = X.rch - R0ch;
  const ff c1 = ff_exp(-(ach * x)), c2 = c1 * c1;
  const ff h1 = ff_exp(-(Ahh * (rbh - R0hh))), h2 = h1 * h1;
  const ff scc2 = Sqch * c2, scc1 = Sqch * c1, fcc2 = Dfch * c2, fcc1 = Dfch * c1;
  const ff shh2 = Sqhh * h2, shh1 = Sqhh * h1, fhh2 = Dfhh * h2, fhh1 = Dfhh * h1;
  const ff qch = scc2 * 0.5f - fcc1, jch = fcc2 * 0.5f - scc1;
  const ff qbh = shh2 * 0.5f - fhh1, jbh = fhh2 * 0.5f - shh1;
  const ff e12 = jch - jcb, e23 = jcb - jbh, e31 = jbh - jch;
  const ff root = ff_sqrt((e12 * e12 + e23 * e23 + e31 * e31) * 0.5f);
  const ff fj = ff_recip(root) * -0.5f;
  const ff dz = -((scc2 - fcc1) + (e12 - e31) * fj * (fcc2 - scc1));
  X.drcb = quad_sum(dqcb + (e23 - e12) * fj * djcb) / rcb;
  X.drbh = -(Ahh * ((shh2 - fhh1) + (e31 - e23) * fj * (fhh2 - shh1))) / rbh;
  X.drch = ach * dz + quad_sum(x * dz) * dach;
  return ff_float(qcb + qch + qbh - root);
}

// Switching functions, reference angles and both bends: this lane's share of
// the energy; dV/dr, dV/du and the plane normals' dV/dH into G.  Partner k of
// bond i (k = 1, 2, 3) is bond i ^ k; the two bonds outside the pair (i, i ^ k)
// are the pair k of another lane.
template <class F, class K>
__device__ inline F bends(const Pairs* X, Bond<F>& G, int i) {
  constexpr bool kPair = std::is_same<F, float>::value;
  const double tau = 1.9106332362490186;  // acos(-1/3)
  const double pi = 3.141592653589793;
  const F A = F(tau - K::tau_py), B = F(tau - 2.0 * pi / 3.0);
  // ---- switching functions (switchf): tanh, d(1 - tanh)/dr
  F t1, ds1, t2, ds2, t3, ds3, tp = F(1), dsp = F(0), tt = F(1), dst = F(0);
  const F r = G.rch, x = r - F(K::r0ch);
  {
    const F y1 = r - F(K::b1s), y1_2 = y1 * y1, y1_4 = y1_2 * y1_2, y1_7 = F(K::a1s) * (y1_4 * y1_2 * y1);
    switch_fn<F>(x * (y1_7 * y1), y1_7 * (y1 + F(8) * x), t1, ds1);
    const F y2 = r - F(K::b2s), y2_2 = y2 * y2, y2_5 = F(K::a2s) * (y2_2 * y2_2 * y2);
    switch_fn<F>(x * (y2_5 * y2), y2_5 * (y2 + F(6) * x), t2, ds2);
    const F y3 = r - F(K::b3s), y3a = F(K::a3s) * y3;
    switch_fn<F>(x * (y3a * y3), y3a * (y3 + F(2) * x), t3, ds3);
    if (!K::sphi_cut || r < F(3.8)) {
      const F xc = r - F(K::cphi), xc2 = F(K::bphi) * (xc * xc);
      const F e = F(K::aphi) * m_exp<F>(xc2 * xc);
      const F arg = x * e;
      // FP32 only: past arg = 19, 1 - tanh is 0 in float and exp overflows
      // (GeH4 + OH, r > 17.9 A); FP64 follows the reference
      if (!kPair || arg < F(19.0)) tanh_switch(arg, e * (F(1) + F(3) * (x * xc2)), tp, dsp);
    }
    if (r < F(3.8)) {
      const F xt = r - F(K::ctheta), xt2 = F(K::btheta) * (xt * xt);
      const F e = F(K::atheta) * m_exp<F>(xt2 * xt);
      tanh_switch(x * e, e * (F(1) + F(3) * (x * xt2)), tt, dst);
    }
  }
  // ---- of the partners: unit vectors, 1 - tanh; theta0 - tau (refangles)
  F un[4][3], sp[4], st[4], s3[4], th[4], bth[4];
  {
    F tpn[4], ttn[4];
#pragma unroll
    for (int k = 1; k < 4; ++k) {
      tpn[k] = of(tp, k);
      ttn[k] = of(tt, k);
      sp[k] = F(1) - tpn[k];
      st[k] = F(1) - ttn[k];
      s3[k] = F(1) - of(t3, k);
#pragma unroll
      for (int d = 0; d < 3; ++d) un[k][d] = of(G.u[d], k);
    }
    th[1] = A * product_m1(tp, tpn[1]) + B * product_m1(ttn[2], ttn[3]);
    th[2] = A * product_m1(tp, tpn[2]) + B * product_m1(ttn[1], ttn[3]);
    th[3] = A * product_m1(tp, tpn[3]) + B * product_m1(ttn[1], ttn[2]);
  }
  F V;
  // ---- out-of-plane bends (opbend, opforce, calcdelta): the plane of the
  // three hydrogens opposite bond i
  {
    F a[3], b[3];  // H_{i^2} - H_{i^1}, H_{i^3} - H_{i^1}
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      const F h1 = of(G.tch[d], 1);
      a[d] = h1 - of(G.tch[d], 2);
      b[d] = h1 - of(G.tch[d], 3);
    }
    const F ab[3] = {a[1] * b[2] - a[2] * b[1], a[2] * b[0] - a[0] * b[2], a[0] * b[1] - a[1] * b[0]};
    const F in = m_rsqrt<F>(dot3(ab, ab));
    F c[4];  // (a x b) . u
#pragma unroll
    for (int k = 1; k < 4; ++k) c[k] = dot3(ab, un[k]);
    // the reference swaps two of the hydrogens for each negative one
    // (src/egrad_ch4h.f:757-764, cumulative): a x b changes sign with each swap,
    // and with the order of the three, of which the result is free
    const bool flip = (c[1] < F(0)) != (c[2] < F(0)) != (c[3] < F(0));
    const F sn = flip ? -in : in;
    const F nrm[3] = {ab[0] * sn, ab[1] * sn, ab[2] * sn};
    const F p12 = s3[1] * s3[2], p13 = s3[1] * s3[3], p23 = s3[2] * s3[3], all = p12 * s3[3], sw = t3 * all;
    // tau as hi + lo: the difference of two ~1.9 rad angles keeps tau's rounding
    const F tau_lo = F(tau - (double)F(tau));
    F sum2 = F(0), sum4 = F(0), w[3] = {F(0), F(0), F(0)};
#pragma unroll
    for (int k = 1; k < 4; ++k) {
      F arg = -(c[k] * sn), sin2 = F(1) - arg * arg;
      if constexpr (kPair) {
        // a bond along the normal: FP32 may round past +-1, and sin^2 to 0
        arg = fminf(1.f, fmaxf(-1.f, arg));
        sin2 = fmaxf((1.f - arg) * (1.f + arg), 1.2e-7f);
      }
      const F dl = (m_acos<F>(arg) - F(tau)) - (th[k] + tau_lo);
      const F d2 = dl * dl;
      sum2 += d2;
      sum4 += d2 * d2;
      const F coef = (sw * dl) * (F(2.0 * K::fch3) + F(4.0 * K::hch3) * d2);
      bth[k] = -(coef + of(coef, k));
      const F ba = coef * m_rsqrt<F>(sin2);  // -dV/d arg, arg = -n.u
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        w[d] += ba * un[k][d];
        G.wu[d] += of(ba * nrm[d], k);
      }
    }
    const F E = F(K::fch3) * sum2 + F(K::hch3) * sum4, Eq = E * t3;
    V = sw * E;
    const F b3 = of(Eq * p23, 1) + of(Eq * p13, 2) + of(Eq * p12, 3) - E * all;
    G.drch += b3 * ds3;
    // dV/d(a x b) = sn (w - n (n.w)), then b x y on H_{i^2} and y x a on H_{i^3}
    const F nw = dot3(nrm, w);
    F y[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) y[d] = sn * (w[d] - nrm[d] * nw);
    const F gk[3] = {b[1] * y[2] - b[2] * y[1], b[2] * y[0] - b[0] * y[2], b[0] * y[1] - b[1] * y[0]};
    const F gl[3] = {y[1] * a[2] - y[2] * a[1], y[2] * a[0] - y[0] * a[2], y[0] * a[1] - y[1] * a[0]};
#pragma unroll
    for (int d = 0; d < 3; ++d) G.gh[d] += of(gk[d], 2) + of(gl[d], 3) - of(gk[d] + gl[d], 1);
  }
  // ---- in-plane bends (ipbend, ipforce).  Six pairs in two rounds: lanes 0
  // and 3 take their pair 1, lanes 1 and 2 their pair 2, then all their pair 3
  // (twice each); each result goes to the pair's other lane.
  {
    const F f0 = F(K::fkinf + K::ak), g0 = F((K::fkinf + K::ak) - K::fkinf);
    const F rb = G.rbh, xh = rb - F(K::r0hh), x2 = x * x;
    const F e1 = m_exp<F>(-F(K::aa1) * rb * rb), e2 = F(K::aa3) * m_exp<F>(-F(K::aa4) * xh * xh);
    const F a1 = F(1) - e1, a2 = F(K::aa2) + e2, eg = m_exp<F>(-a2 * x2);
    const F f1 = a1 * eg;
    const F df1c = F(-2) * x * (f1 * a2);
    const F df1h = F(2.0 * K::aa1) * rb * (e1 * eg) + F(2.0 * K::aa4) * xh * e2 * (x2 * f1);
    const int first = i == 0 || i == 3 ? 1 : 2, other = 3 - first;
    // stiffness without the f1: f0 + f0 (s1 s1 - 1) + g0 (s2 s2 - 1) of pair k
    F t2n[4], f1n[4], s1n[4], fk[4], hk[4], bk[4];
#pragma unroll
    for (int k = 1; k < 4; ++k) {
      const F t1k = of(t1, k);
      s1n[k] = F(1) - t1k;
      t2n[k] = of(t2, k);
      f1n[k] = of(f1, k);
      fk[k] = f0 * product_m1(t1, t1k);
    }
    fk[1] = f0 + (fk[1] + g0 * product_m1(t2n[2], t2n[3]));
    fk[2] = f0 + (fk[2] + g0 * product_m1(t2n[1], t2n[3]));
    fk[3] = f0 + (fk[3] + g0 * product_m1(t2n[1], t2n[2]));
    F dth[4], is[4];  // theta - theta0, 1 / sin(theta)
#pragma unroll 1
    for (int round = 0; round < 2; ++round) {
      const int k = round == 0 ? first : 3, src = (int)(threadIdx.x & 3) ^ k;
      const F thk = k == 1 ? th[1] : k == 2 ? th[2] : th[3];
      F cs, dt, sin2;
      if constexpr (kPair) {
        // theta - tau as asin(sin(theta - tau)) from a float-pair cosine:
        // theta - th0 is a small difference of two ~1.9 rad angles, which
        // acosf of an FP32 cosine would leave with ~1e-7 rad of error
        const ff c = (X->tch[0] * from(X->tch[0], src) + X->tch[1] * from(X->tch[1], src) +
                      X->tch[2] * from(X->tch[2], src)) / (X->rch * from(X->rch, src));
        constexpr ff kCosTau = ff_const(-1.0 / 3.0), kSinTau = ff_const(0.94280904158206336587);
        const ff sq = ff_from(1.f) - c * c, y = ff_sqrt(sq) * kCosTau - c * kSinTau;
        cs = ff_float(c);
        // two bonds in line (one of them broken, its stiffness about 0): the FP32
        // 1 - cs^2 is 0 there, and 0 / 0 the force; the pair's has 2^-44
        sin2 = fmaxf(sq.hi, 1e-12f);
        const float dtau = fabsf(y.hi) < 0.9f ? asinf(y.hi) + y.lo * m_rsqrt<float>(1.f - y.hi * y.hi)
                                              : acosf(cs) - F(tau);
        dt = dtau - thk;
      } else {
        const F v[3] = {k == 1 ? un[1][0] : k == 2 ? un[2][0] : un[3][0], k == 1 ? un[1][1] : k == 2 ? un[2][1] : un[3][1],
                        k == 1 ? un[1][2] : k == 2 ? un[2][2] : un[3][2]};
        cs = dot3(G.u, v);
        dt = (m_acos<F>(cs) - F(tau)) - thk;
        sin2 = F(1) - cs * cs;
      }
      const F s = m_rsqrt<F>(sin2);
      if (round == 0) {
        const F dt2 = from(dt, (int)(threadIdx.x & 3) ^ other), s2 = from(s, (int)(threadIdx.x & 3) ^ other);
        dth[1] = first == 1 ? dt : dt2;
        dth[2] = first == 1 ? dt2 : dt;
        is[1] = first == 1 ? s : s2;
        is[2] = first == 1 ? s2 : s;
      } else {
        dth[3] = dt;
        is[3] = s;
      }
    }
    F bf1 = F(0), b1 = F(0);
#pragma unroll
    for (int k = 1; k < 4; ++k) {
      const F h = F(0.5) * dth[k] * dth[k], ff1 = f1 * f1n[k], kf = fk[k] * ff1;
      V += F(0.5) * h * kf;  // the pair's other lane has the other half
      hk[k] = h * fk[k];
      bk[k] = h * ff1;
      bf1 += hk[k] * f1n[k];
      b1 += (bk[k] * f0) * s1n[k];
      const F kd = kf * dth[k], bc = kd * is[k];  // -dV/d theta0, -dV/d cos
      bth[k] -= kd;
#pragma unroll
      for (int d = 0; d < 3; ++d) G.wu[d] -= bc * un[k][d];
    }
    const F b2 = g0 * (of(bk[1], 2) * (F(1) - t2n[1]) + of(bk[2], 1) * (F(1) - t2n[2]) + of(bk[3], 1) * (F(1) - t2n[3]));
    G.drch += bf1 * df1c + b1 * ds1 + b2 * ds2;
    G.drbh += bf1 * df1h;
  }
  // ---- the reference angles' share
  const F bp = A * (bth[1] * sp[1] + bth[2] * sp[2] + bth[3] * sp[3]);
  const F bt = B * (of(bth[1], 2) * st[1] + of(bth[2], 1) * st[2] + of(bth[3], 1) * st[3]);
  G.drch += bp * dsp + bt * dst;
  return V;
}

// The chain to the atoms: g[0..2] the gradient on H_i, g[3..5] on X, g[6..8] on
// B (both summed over the quad).
__device__ inline void chain(const Bond<double>& G, double (&g)[9]) {
  const double kc = G.drcb * G.ircb, kb = G.drbh * G.irbh, uw = dot3(G.u, G.wu);
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    const double t = fma(G.u[d], G.drch, (G.wu[d] - G.u[d] * uw) * G.irch), w = G.tbh[d] * kb;
    g[d] = G.gh[d] - (t + w);
    g[3 + d] = fma(G.tcb[d], kc, quad_sum(t));
    g[6 + d] = fma(-G.tcb[d], kc, quad_sum(w));
  }
}

// Mixed form: the stretches' part in float pairs (their vectors cancel on
// each atom), the bends' radial derivatives joined to them.
__device__ inline void chain(const Bond<float>& G, const Pairs& X, ff (&g)[9]) {
  const float uw = dot3(G.u, G.wu);
  const ff kc = (X.drch + G.drch) / X.rch, kb = X.drbh + G.drbh * G.irbh;
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    const ff t = X.tch[d] * kc + (G.wu[d] - G.u[d] * uw) * G.irch, w = X.tbh[d] * kb, b = X.tcb[d] * X.drcb;
    g[d] = -(t + w) + G.gh[d];
    g[3 + d] = quad_sum(t) + b;
    g[6 + d] = quad_sum(w) - b;
  }
}

// Bond vectors and lengths of lane i from the bead's coordinates x(c) (bohr),
// scaled to Angstrom (POT_ch4h: 0.52918).
template <class Get>
__device__ inline void bond_vectors(const Get& x, int i, Bond<double>& G) {
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    const double c = x(3 * NC + d) * 0.52918, b = x(3 * NB + d) * 0.52918, h = x(3 * NH(i) + d) * 0.52918;
    G.tcb[d] = c - b;
    G.tch[d] = c - h;
    G.tbh[d] = b - h;
  }
  lengths(G);
}
// a coordinate as a float pair in Angstrom, from the FP64 bits: FP64
// instructions would cost 64 cycles each
__device__ inline ff scaled_pair(double q) {
  constexpr ff kA = ff_const(0.52918);
  return ff_split(q) * kA;
}
template <class Get>
__device__ inline void bond_vectors(const Get& x, int i, Bond<float>& G, Pairs& X) {
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    const ff c = scaled_pair(x(3 * NC + d)), b = scaled_pair(x(3 * NB + d)), h = scaled_pair(x(3 * NH(i) + d));
    X.tcb[d] = c - b;
    X.tch[d] = c - h;
    X.tbh[d] = b - h;
    G.tcb[d] = ff_float(X.tcb[d]);
    G.tch[d] = ff_float(X.tch[d]);
    G.tbh[d] = ff_float(X.tbh[d]);
  }
  X.rch = ff_sqrt(X.tch[0] * X.tch[0] + X.tch[1] * X.tch[1] + X.tch[2] * X.tch[2]);
  lengths(G);
}

}  // namespace methane
}  // namespace cr
