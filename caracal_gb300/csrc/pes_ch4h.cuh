// CH4 + H potential (Corchado, Bravo, Espinosa-Garcia, J. Chem. Phys. 130,
// 184314 (2009)) as GB300 device code: a drop-in for Caracal's egrad_ch4h
// (src/egrad_ch4h.f:74-120) with its POTLIB wrapper in Caracal's settings
// (bohr/Hartree user units, no relabelling: src/util_ch4h.f CARTOU, CARTTOR,
// EUNITZERO, RTOCART, DEDCOU are identities).
//
// Four lanes evaluate one bead.  Routines restated: POT_ch4h :161,
// coorden :287, switchf :1545, refangles :367, stretch :506, opbend :713,
// calcdelta :986, opforce :1240, ipbend :865, ipforce :1350; constants from
// BLOCK DATA PTPACM_ch4h with PREPOT_ch4h's unit factors (all REAL(8)).
// Atoms: 0 H(methane, nnh(4)), 1 C (nnc), 2,3,4 H(methane, nnh(1..3)),
// 5 H_b (nnb, the abstracting H); the methane H are indexed i = 0..3 in the
// order of nnh, i.e. atoms {2,3,4,0}.
//
// The terms and their reverse-mode gradient are methane.cuh's; here are the
// constants, the geometry (displacements after Caracal's bohr -> Angstrom
// scaling, in FP64 or as float pairs) and the unit factors: the energy and
// gradient factors 0.03812 and 0.0201723 are the reference's (they differ
// from each other by 2.06e-6 relative; the gradient reproduces the reference,
// not the derivative of its energy).
#pragma once
#include <cuda_runtime.h>

#include "methane.cuh"

namespace cr {
namespace ch4h {

// BLOCK DATA PTPACM_ch4h (src/egrad_ch4h.f:1847-1887) after PREPOT_ch4h
// (src/egrad_ch4h.f:1724-1738): d's * 0.041840, force constants * 6.022045;
// switchf_ch4h's local constants (src/egrad_ch4h.f:1567-1570).
struct Par {
  static constexpr double r0ch = 1.08898, a1ch = 1.78374, b1ch = 0.14201, c1ch = 2.21773;
  static constexpr double r0hh = 0.74239, ahh = 1.9589, r0cb = 1.08898, acb = 1.4173200;
  static constexpr double d1ch = 111.266 * 0.041840, d3ch = 48.96226 * 0.041840;
  static constexpr double d1hh = 108.382 * 0.041840, d3hh = 38.42657 * 0.041840;
  static constexpr double d1cb = 56.505 * 0.041840, d3cb = 19.612 * 0.041840;
  static constexpr double a3s = 0.1475300, b3s = -2.9926300, aphi = 0.5307000, bphi = 0.4012200;
  static constexpr double cphi = 1.9235100, atheta = 0.9119800, btheta = 0.3537500, ctheta = 1.8970500;
  static constexpr double fch3 = 0.0693700 * 6.022045, hch3 = 0.1387400 * 6.022045;
  static constexpr double fkinf = 0.4291400 * 6.022045, ak = 0.1353000 * 6.022045;
  static constexpr double aa1 = 1.265960, aa2 = 0.000710, aa3 = 0.985920, aa4 = 2.785060;
  static constexpr double a1s = 1.5132681e-7, b1s = -4.3792246, a2s = 1.9202402e-7, b2s = -12.323018;
  static constexpr double tau_py = 0.5 * 3.141592653589793;  // planar CH3
  static constexpr bool sphi_cut = true;                     // switchf's rch < 3.8 condition on sphi
};

// Lane i of a quad (i = lane & 3; every lane of the warp takes part): the
// energy on all four, the gradient by put(coordinate, value), each coordinate
// from one lane.
template <class F, class Get, class Put>
__device__ inline void egrad(const Get& x, int i, double& V, const Put& put) {
  methane::Bond<F> G;
  if constexpr (std::is_same<F, float>::value) {
    methane::Pairs X;
    ff g[9], none;
    methane::bond_vectors(x, i, G, X);
    const float vs = methane::stretch_pairs<Par>(G, X, i, ff{0.f, 0.f}, none);
    const float vb = methane::bends<float, Par>(&X, G, i);
    V = ff_to_double(methane::quad_sum(vs + vb)) * 0.03812;
    methane::chain(G, X, g);
    constexpr ff kUnit = ff_const(0.0201723);
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      put(3 * methane::NH(i) + d, ff_to_double(ff_float(g[d] * kUnit)));
      const ff h = i == 0 ? g[3 + d] : g[6 + d];
      if (i < 2) put(3 * (i == 0 ? methane::NC : methane::NB) + d, ff_to_double(ff_float(h * kUnit)));
    }
  } else {
    double g[9], none;
    methane::bond_vectors(x, i, G);
    const double vs = methane::stretch_plain<Par>(G, i, 0.0, none);
    const double vb = methane::bends<double, Par>(nullptr, G, i);
    V = methane::quad_sum(vs + vb) * 0.03812;
    methane::chain(G, g);
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      put(3 * methane::NH(i) + d, g[d] * 0.0201723);
      if (i < 2) put(3 * (i == 0 ? methane::NC : methane::NB) + d, (i == 0 ? g[3 + d] : g[6 + d]) * 0.0201723);
    }
  }
}

}  // namespace ch4h

struct PesCH4H {
  static constexpr int N = 6;
  static constexpr int kLanes = 4;  // per bead
  static constexpr bool kQuad = false;  // always four
  template <class F, class Get, class Put>
  __device__ static inline void egrad(const Get& x, int i, double& V, const Put& put) {
    ch4h::egrad<F>(x, i, V, put);
  }
};

}  // namespace cr
