// CH4 + OH potential (Espinosa-Garcia, Corchado, J. Chem. Phys. 112, 5731
// (2000)) as GB300 device code: a drop-in for Caracal's egrad_ch4oh
// (src/egrad_ch4oh.f:69-124) with its POTLIB wrapper in Caracal's settings
// (bohr/Hartree user units, no relabelling: the routines of
// src/util_ch4oh.f are identities).  The same code with the constants of
// src/egrad_geh4oh.f is the GeH4 + OH surface (egrad_geh4oh :33-67): its
// routines differ from CH4 + OH's only in the pyramid angle of refangles and
// the uncut sphi of switchf (ParCH4OH / ParGeH4OH below).
//
// Four lanes evaluate one bead.  Routines restated (src/egrad_ch4oh.f):
// POT_ch4oh :157, coorden :288, refangles :374, stretch :517, opbend :782,
// ipbend :938, calcdelta :1177, opforce :1435, ipforce :1549, switchf :1748;
// constants from BLOCK DATA PTPACM_ch4oh :2007 with PREPOT_ch4oh's unit
// factors (all REAL(8)).  Atoms: 0 H(methane, nnh(4)), 1 C (nnc), 2,3,4
// H(methane, nnh(1..3)), 5 O (nnb), 6 H of OH (nno); methane H i = 0..3 are
// atoms {2,3,4,0}.
//
// The surface is the CH4 + H one (methane.cuh: same functional forms, own
// constants and the original POTLIB switching constants) plus an O-H Morse
// stretch and four H(i)-O-H(O) harmonic bends with a tanh-switched force
// constant, which are here.  The switched C-B triplet depth d3cb(rav) of
// stretch_ch4oh has amplitude a3cb = 0, so d3cb = d3cbi and its derivative
// terms vanish; they are folded away at compile time.  The energy and gradient
// unit factors 0.03812 and 0.0201723 are the reference's.
//
// Mixed form (F = float): as for CH4 + H, positions enter as float pairs
// (ff32.cuh), the stretches and the bends' angle differences from their
// references are formed in float-pair arithmetic, and the stretch gradient is
// summed as float pairs; the rest is FP32.
#pragma once
#include <cuda_runtime.h>

#include "methane.cuh"

namespace cr {
namespace ch4oh {

// The constants of BLOCK DATA PTPACM_ch4oh (src/egrad_ch4oh.f:2064-2106) and
// PTPACM_geh4oh (src/egrad_geh4oh.f:2001-2045) after PREPOT's / initialize's
// conversions (src/egrad_ch4oh.f:1987-2003): d's * 0.041840, force constants
// * 6.022045, anh2oeq * 2 pi / 360.  The two surfaces share these:
constexpr double a3cb = 0.000000 * 0.041840;
struct ParXH4OH {
  static constexpr double r0hh = 0.97060;
  static constexpr double aphi = 0.5287900, bphi = 0.4006600;
  static constexpr double atheta = 0.9078700, btheta = 0.3548900, ctheta = 1.8915500;
  static constexpr double hch3 = 0.1915000 * 6.022045, ak = 0.1260000 * 6.022045;
  static constexpr double aa2 = 1.599960, aa4 = 11.569980;
  // switchf local constants (the original POTLIB values)
  static constexpr double a1s = 1.5313681e-7, b1s = -4.6696246, a2s = 1.0147402e-7, b2s = -12.363798;
};
constexpr double fkh2oeq = 0.7300000 * 6.022045, alph2o = 1.1080000;
constexpr double anh2oeq = 104.7132000 * (2.0 * 3.141592653589793 / 360.0);
static_assert(a3cb == 0.0, "the d3cb(rav) switch is folded away for a3cb = 0");

// The constants that differ.  tau_py is the pyramid angle of refangles'
// sphi term (pi/2: planar CH3; 0.678 pi: pyramidal GeH3,
// src/egrad_geh4oh.f:368-392); sphi_cut keeps switchf's rch < 3.8 condition
// on sphi (CH4 + OH; GeH4 + OH evaluates sphi at every distance,
// src/egrad_geh4oh.f:1792-1804).
struct ParCH4OH : ParXH4OH {
  static constexpr double r0ch = 1.09397, a1ch = 1.78000, b1ch = 0.15000, c1ch = 15.00000;
  static constexpr double ahh = 2.15000, r0cb = 1.49092, acb = 2.98688;
  static constexpr double d1ch = 112.17000 * 0.041840, d3ch = 32.65328 * 0.041840;
  static constexpr double d1hh = 125.44000 * 0.041840, d3hh = 20.41017 * 0.041840;
  static constexpr double d1cb = 91.47526 * 0.041840, d3cb = 112.69509 * 0.041840;
  static constexpr double a3s = 0.1419100, b3s = -0.3068400, cphi = 1.9209900;
  static constexpr double fch3 = 0.0740000 * 6.022045, fkinf = 0.4400000 * 6.022045;
  static constexpr double aa1 = 0.303746, aa3 = 3.216595;
  static constexpr double tau_py = 0.5 * 3.141592653589793;
  static constexpr bool sphi_cut = true;
};
struct ParGeH4OH : ParXH4OH {
  static constexpr double r0ch = 1.52500, a1ch = 1.43925, b1ch = 0.12330, c1ch = 2.00400;
  static constexpr double ahh = 2.18200, r0cb = 1.90035, acb = 0.67621;
  static constexpr double d1ch = 86.50000 * 0.041840, d3ch = 41.50000 * 0.041840;
  static constexpr double d1hh = 120.94800 * 0.041840, d3hh = 31.86417 * 0.041840;
  static constexpr double d1cb = 41.50283 * 0.041840, d3cb = 10.50589 * 0.041840;
  static constexpr double a3s = 0.2019100, b3s = -0.6068400, cphi = 11.8809900;
  static constexpr double fch3 = 0.0150000 * 6.022045, fkinf = 0.3060000 * 6.022045;
  static constexpr double aa1 = 0.173746, aa3 = 2.166595;
  static constexpr double tau_py = 0.678 * 3.141592653589793;
  static constexpr bool sphi_cut = false;
};

constexpr int NB = methane::NB, NO = 6;

// H(i)-O-H(O) bend of lane i (ipbend_ch4oh :1061-1172): the energy; dV/dr(BH_i)
// into G, the gradient across the bonds on H_i and H(O) into gh, go.
template <class F, class K>
__device__ inline F hoh_bend(const F (&tno)[3], F irno, const ff* xno, ff xrno, const methane::Pairs* X,
                             methane::Bond<F>& G, F (&gh)[3], F (&go)[3]) {
  constexpr bool kPair = std::is_same<F, float>::value;
  const F* tb = G.tbh;
  F cosine, dang;
  if constexpr (kPair) {
    // angle - anh2oeq as asin(sin(angle - anh2oeq)) from a float-pair
    // cosine: a small difference of two ~1.8 rad angles
    const ff* xb = X->tbh;
    const ff rbh = ff_sqrt(xb[0] * xb[0] + xb[1] * xb[1] + xb[2] * xb[2]);
    ff c = -((xno[0] * xb[0] + xno[1] * xb[1] + xno[2] * xb[2]) / (xrno * rbh));
    if (c.hi > 1.f) c = ff_from(1.f);
    if (c.hi < -1.f) c = ff_from(-1.f);
    constexpr ff kCosEq = ff_const(-0.25398078034139054), kSinEq = ff_const(0.9672092654731852);
    const ff y = ff_sqrt(ff_from(1.f) - c * c) * kCosEq - c * kSinEq;  // sin(angle - anh2oeq)
    cosine = ff_float(c);
    dang = fabsf(y.hi) < 0.9f ? asinf(y.hi) + y.lo * methane::m_rsqrt<float>(1.f - y.hi * y.hi)
                              : acosf(cosine) - F(anh2oeq);
  } else {
    cosine = -methane::dot3(tno, tb) * (irno * G.irbh);
    cosine = fmin(F(1), fmax(F(-1), cosine));
    dang = methane::m_acos<F>(cosine) - F(anh2oeq);
  }
  const F arga = F(alph2o) * (G.rbh - F(K::r0hh));
  F t, ds;  // tanh(arga), -alph2o / cosh(arga)^2 (also past the cutoff)
  methane::tanh_switch(arga, F(alph2o), t, ds);
  const F fk = (arga < F(19.0)) ? F(fkh2oeq) * (F(1) - t) : F(0);
  const F h = F(0.5) * dang * dang, dstda = fk * dang;
  G.drbh += F(fkh2oeq) * ds * h;
  const F xp = tno[1] * tb[2] - tno[2] * tb[1];
  const F yp = tno[2] * tb[0] - tno[0] * tb[2];
  const F zp = tno[0] * tb[1] - tno[1] * tb[0];
  F rp = methane::m_sqrt<F>(xp * xp + yp * yp + zp * zp);
  if (rp < F(1.0e-6)) rp = F(1.0e-6);
  const F k = methane::m_div<F>(dstda, rp);
  const F ta = k * (G.irbh * G.irbh), tc = k * (irno * irno);
  gh[0] = -ta * (tb[1] * zp - tb[2] * yp);
  gh[1] = -ta * (tb[2] * xp - tb[0] * zp);
  gh[2] = -ta * (tb[0] * yp - tb[1] * xp);
  go[0] = -tc * (tno[1] * zp - tno[2] * yp);
  go[1] = -tc * (tno[2] * xp - tno[0] * zp);
  go[2] = -tc * (tno[0] * yp - tno[1] * xp);
  return fk * h;
}

// Lane i of a quad, as in ch4h::egrad.  The O-H Morse stretch (stretch_ch4oh
// :602-605, :620-632, :711-716) is evaluated on every lane, its energy counted
// on lane 0; its 1 - exp(-a (r - r0)) near the minimum in float pairs too.
template <class F, class K, class Get, class Put>
__device__ inline void egrad(const Get& x, int i, double& V, const Put& put) {
  methane::Bond<F> G;
  F tno[3], gh[3], go[3], rno, irno;
  if constexpr (std::is_same<F, float>::value) {
    methane::Pairs X;
    ff g[9], xno[3], eoh;
    methane::bond_vectors(x, i, G, X);
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      xno[d] = methane::scaled_pair(x(3 * NO + d)) - methane::scaled_pair(x(3 * NB + d));
      tno[d] = ff_float(xno[d]);
    }
    const ff xrno = ff_sqrt(xno[0] * xno[0] + xno[1] * xno[1] + xno[2] * xno[2]);
    methane::m_root(methane::dot3(tno, tno), rno, irno);
    constexpr ff kA = ff_const(K::ahh), kR0 = ff_const(K::r0hh);
    float v = methane::stretch_pairs<K>(G, X, i, -(kA * (xrno - kR0)), eoh);
    const ff om = ff_from(1.f) - eoh, dno = (ff_const(2.0 * K::ahh * K::d1hh) * om * eoh) / xrno;
    if (i == 0) v += ff_float(ff_const(K::d1hh) * (om * om));
    v += methane::bends<float, K>(&X, G, i);
    v += hoh_bend<float, K>(tno, irno, xno, xrno, &X, G, gh, go);
    V = ff_to_double(methane::quad_sum(v)) * 0.03812;
    methane::chain(G, X, g);
    constexpr ff kUnit = ff_const(0.0201723);
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      const ff t = xno[d] * dno;
      const float so = methane::quad_sum(go[d]), sh = methane::quad_sum(gh[d]);
      put(3 * methane::NH(i) + d, ff_to_double(ff_float((g[d] + gh[d]) * kUnit)));
      const ff h = i == 0 ? g[3 + d] : i == 1 ? g[6 + d] - (t + (sh + so)) : t + so;
      if (i < 3) put(3 * (i == 0 ? methane::NC : i == 1 ? NB : NO) + d, ff_to_double(ff_float(h * kUnit)));
    }
  } else {
    double g[9], eoh;
    methane::bond_vectors(x, i, G);
#pragma unroll
    for (int d = 0; d < 3; ++d) tno[d] = x(3 * NO + d) * 0.52918 - x(3 * NB + d) * 0.52918;
    methane::m_root(methane::dot3(tno, tno), rno, irno);
    double v = methane::stretch_plain<K>(G, i, -K::ahh * (rno - K::r0hh), eoh);
    const double om = 1.0 - eoh, dno = (2.0 * K::ahh * K::d1hh) * om * eoh * irno;
    if (i == 0) v += K::d1hh * (om * om);
    v += methane::bends<double, K>(nullptr, G, i);
    v += hoh_bend<double, K>(tno, irno, nullptr, ff{0.f, 0.f}, nullptr, G, gh, go);
    V = methane::quad_sum(v) * 0.03812;
    methane::chain(G, g);
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      const double so = methane::quad_sum(go[d]), sh = methane::quad_sum(gh[d]), t = fma(tno[d], dno, so);
      put(3 * methane::NH(i) + d, (g[d] + gh[d]) * 0.0201723);
      const double h = i == 0 ? g[3 + d] : i == 1 ? g[6 + d] - (t + sh) : t;
      if (i < 3) put(3 * (i == 0 ? methane::NC : i == 1 ? NB : NO) + d, h * 0.0201723);
    }
  }
}

}  // namespace ch4oh

struct PesCH4OH {
  static constexpr int N = 7;
  static constexpr int kLanes = 4;  // per bead
  static constexpr bool kQuad = false;  // always four
  template <class F, class Get, class Put>
  __device__ static inline void egrad(const Get& x, int i, double& V, const Put& put) {
    ch4oh::egrad<F, ch4oh::ParCH4OH>(x, i, V, put);
  }
};

// GeH4 + OH (src/egrad_geh4oh.f, Espinosa-Garcia, Rangel, Corchado, Phys.
// Chem. Chem. Phys. 18, 16941 (2016)): the CH4 + OH functional forms and atom
// roles (Ge in C's place) with its own constants.
struct PesGeH4OH {
  static constexpr int N = 7;
  static constexpr int kLanes = 4;
  static constexpr bool kQuad = false;  // always four
  template <class F, class Get, class Put>
  __device__ static inline void egrad(const Get& x, int i, double& V, const Put& put) {
    ch4oh::egrad<F, ch4oh::ParGeH4OH>(x, i, V, put);
  }
};

}  // namespace cr
