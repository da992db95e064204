// QMDFF force field on the GB300: one warp per bead in the mixed form, a block of eight
// (kTeam) in FP64, of one to eight for Hessian products.
//
// Drop-in for Caracal's per-bead QMDFF gradient (src/gradient.f90:342-358:
// ff_eg src/ff_eg.f90:41-629, ff_nonb src/ff_nonb.f90:34-889, E_zero shift),
// non-periodic, one molecule.  A bead's coordinates and gradient live in
// shared memory.  A lane evaluates a term and writes its gradient into a
// buffer in shared memory; once a segment of terms is done, every coordinate
// sums what the segment holds for it, along lists that the host prepared.  No
// atomics, fixed accumulation order: results are deterministic run to run.
//
// Precision: the plain form computes every term in FP64 with Caracal's
// formulas (divisions by a shared denominator taken as one reciprocal).  The
// mixed form splits each FP64 coordinate once per bead into an FP32 pair
// x = hi + lo; a displacement (hi_a - hi_b) + (lo_a - lo_b) is then within
// about one FP32 ulp of the exact difference without any FP64 work per term.
// Terms run in FP32 with cancellation-free rewrites where the FP64 formula
// subtracts nearly equal numbers (bond stretch from an FP64 r^2 - r0^2,
// dihedral angle from atan2 instead of acos); gradient and energy are
// accumulated with compensated (Neumaier) FP32 sums.
#pragma once
#include <cuda_runtime.h>

#include <type_traits>

#include "../../include/caracal_gb300.h"
#include "dual.cuh"

namespace cr {
namespace qmdff {

constexpr int kMaxAtoms = 1024;

// Values per term in the tables: bonds r0, k, a; angles theta0, k, cos(theta0),
// linear flag, 1 / rcut of its two bonds' damping (abdamp); torsions phi0, V, (rn,
// phase, Vn) x 4, 1 / rcut of its three; pairs R0^6, R0^8, eps2 C6, eps2 C6 sr42, eps2
// zab, alpha, qq (eps1 q_i q_j or q_i q_j).
constexpr int kVBond = 3, kVAngl = 6, kVTors = 17, kVPair = 7;
constexpr int kVClass = 8;  // mixed-form pair classes (Dev::pclass)

// Term tables in the arithmetic type of the form, value by value (value c of term m
// of kind k at [c st[k] + m]): the lanes of a warp, which take consecutive terms,
// read consecutive words.  With a term's values side by side the mixed
// force kernel waited for its tables a third of the time (1024 x 64 C20H42, 33
// distinct beads each: 1190 -> 940 us with the gather below).
template <class F>
struct Tables {
  const F* bond;
  const F* angl;
  const F* tors;
  const F* pair;  // (the mixed form's pairs: Dev::fpair)
};

constexpr int kKinds = 5;  // bonds, angles, torsions, NCI pairs, H/halogen bonds

// Schedule of the terms of one form.  A segment is as many terms of a kind as the
// gradient buffer holds; its gather works in rounds of 32 coordinates (the atoms
// with the most terms first, so that a round's lists are of like length), each
// lane summing its coordinate's list.  Written so, a term's gradient costs one
// store per component and one load and sum per component and atom; scattered
// colour by colour, as the terms of a batch share atoms, it cost a round of the
// warp per colour: a third of the mixed kernel's instructions and two thirds of the
// FP64 kernel's time.
struct Schedule {
  int seg0[kKinds], seg1[kKinds];  // segments of each kind
  const int4* seg;                 // first term, terms, first round, rounds
  const int2* round;               // first list entry (32 per step), steps
  const unsigned short* dst;       // [rounds][32]: coordinate, or kNoDst
  const unsigned short* ent;       // buffer offset, kNegate for the negative; the offset past the buffer holds 0
  int npair;                       // batches of 32 NCI pairs of the mixed form (Dev::fpair)
};
constexpr int kNoDst = 0xffff, kNegate = 0x8000;
constexpr unsigned kNoPair = 0xffffffffu;
__device__ __forceinline__ int lo16(unsigned x) { return (int)(x & 0xffffu); }
__device__ __forceinline__ int hi16(unsigned x) { return (int)(x >> 16); }

// Values per term in the buffer (a bond or pair: one atom's gradient, the mixed
// form's bonds as (hi, lo); the other atom's is its negative), and the terms of a
// segment.
__host__ __device__ constexpr int term_values(bool mixed, int kind) {
  return kind == 0 ? (mixed ? 6 : 3) : kind == 2 ? 12 : kind == 3 ? 3 : 9;
}
__host__ __device__ constexpr int segment_terms(bool mixed, int kind) {
  return mixed ? (kind == 0 ? 128 : 64) : (kind == 0 || kind == 3 ? 1024 : 256);
}
__host__ __device__ constexpr int buffer_values(bool mixed) { return mixed ? 768 : 3072; }

// A periodic box (src/box_image.f90): edges and halves in bohr, and for the
// mixed form the edges as (hi, lo) float pairs and the halves in FP32.
struct PBox {
  double len[3], half[3];
  float flen[3], flen_lo[3], fhalf[3], fhalf_lo[3];
  float fhalf_dn[3], fhalf_up[3];  // half -+ 4 ulps: outside, the hi part decides the image
};
__host__ __device__ inline PBox make_box(const double* len) {
  PBox b;
  for (int k = 0; k < 3; ++k) {
    b.len[k] = len[k];
    b.half[k] = len[k] * 0.5;
    b.flen[k] = (float)len[k];
    b.flen_lo[k] = (float)(len[k] - (double)b.flen[k]);
    b.fhalf[k] = (float)b.half[k];
    b.fhalf_lo[k] = (float)(b.half[k] - (double)b.fhalf[k]);
    b.fhalf_dn[k] = (float)(b.half[k] * (1.0 - 4.8e-7));
    b.fhalf_up[k] = (float)(b.half[k] * (1.0 + 4.8e-7));
  }
  return b;
}

struct Dev {
  int n;
  // [0] plain form, [1] mixed form
  Schedule sched[2];
  int st[kKinds];       // stride of the tables
  const unsigned* bond; // atoms (0-based) in 16 bits each: i, j
  const uint2* angl;    // i, centre; k
  const uint4* tors;    // i, j; k, l; nt + 256 type; number in the definition (the terms are ordered by type and nt)
  const unsigned* pair; // i, j
  const int* hb;     // 4 per H/halogen bond: A, B, H, type (1 hydrogen bond, 2 halogen bond)
  const double* vhb; // 2 per H/halogen bond: ca, cb
  Tables<double> d;
  Tables<float> f;
  double coul_cut, zahn_a, zahn_par, e_zero;
  float fcoul_cut, fzahn_a, fzahn_par;  // the same in FP32 (mixed form)
  int zahn;
  // periodic box (src/set_periodic.f90, src/box_image.f90) and the
  // dispersion/repulsion cutoff, bohr
  int periodic;
  PBox box;
  double vdw_cut;
  float fvdw_cut;
  // NpT, set per launch: the box of each trajectory (3 edges, bohr) for
  // beads [t tbox_beads, (t + 1) tbox_beads) in place of `box`, and the
  // virial trace of each bead out (src/ff_eg.f90, ff_nonb.f90, eabhag.f90,
  // eabxag.f90 `vir_ten`); NULL otherwise
  const double* tbox;
  int tbox_beads;
  double* vir;
  int nterm[kKinds];  // terms per kind
  // mixed form, bond stretch gradient as a double-FP32 polynomial (see
  // bond_mixed): per bond kBondSer (hi, lo) pairs: 1/r0^2, r0^2, (use flag,
  // 0), the kBondPoly coefficients, value by value as the tables
  const float2* bser;
  // mixed form, NCI pairs in batches of 32 in which no atom appears twice: atoms,
  // class (kNoPair: none), eps2 C6, qq; and per class R0^6, R0^8, sr42, eps2 zab, alpha
  // log2(e), alpha (which depend on the elements and the category alone)
  const uint4* fpair;
  const float4* pclass;
};

constexpr int kBondPoly = 24;             // polynomial of degree 23
constexpr int kBondSer = kBondPoly + 3;
constexpr double kBondSerMaxT = 0.45;     // used for |r^2/r0^2 - 1| <= this

// Double-FP32 ("float-float") numbers hi + lo, |lo| <= ulp(hi)/2: about 44
// bits of significand from FP32 operations (error-free sum of Knuth, product
// split by FMA).  Used where FP32 rounding would set the mixed form's error.
struct FF {
  float hi, lo;
};
__device__ inline FF ff_norm(float s, float e) {
  const float h = s + e;
  return FF{h, e - (h - s)};
}
__device__ inline FF ff_add(FF a, FF b) {
  const float s = a.hi + b.hi, bb = s - a.hi;
  const float e = (a.hi - (s - bb)) + (b.hi - bb);
  return ff_norm(s, e + (a.lo + b.lo));
}
__device__ inline FF ff_mul(FF a, FF b) {
  const float p = a.hi * b.hi;
  float e = fmaf(a.hi, b.hi, -p);
  e = fmaf(a.hi, b.lo, fmaf(a.lo, b.hi, e));
  return ff_norm(p, e);
}
__device__ inline FF ff_of(float2 v) { return FF{v.x, v.y}; }

template <class F> __device__ inline F q_sqrt(F x);
template <> __device__ inline double q_sqrt<double>(double x) { return sqrt(x); }
template <> __device__ inline float q_sqrt<float>(float x) { return sqrtf(x); }
template <class F> __device__ inline F q_erfc(F x);
template <> __device__ inline double q_erfc<double>(double x) { return erfc(x); }
template <> __device__ inline float q_erfc<float>(float x) { return erfcf(x); }

// |x| > 1e-14 as the reference tests its FP64 denominators; for FP32 the same set of
// values without a conversion (1e-14 is not a float: |x| > 1e-14 holds exactly for
// |x| > 1e-14f, the float below it).
template <class F> __device__ inline bool above_1em14(F x) { return fabs((double)ad::val(x)) > 1e-14; }
template <> __device__ inline bool above_1em14<float>(float x) { return fabsf(x) > 1e-14f; }

template <class F>
__device__ inline void cross(const F* a, const F* b, F* c) {
  c[0] = a[1] * b[2] - a[2] * b[1];
  c[1] = a[2] * b[0] - a[0] * b[2];
  c[2] = a[0] * b[1] - a[1] * b[0];
}
template <class F>
__device__ inline F dot3(const F* a, const F* b) { return a[0] * b[0] + a[1] * b[1] + a[2] * b[2]; }

// Gradient contribution of one term: up to four atoms.
template <class F>
struct Contrib {
  int na;
  int a[4];
  F g[4][3];
};

// A mixed-form pair's gradient onto its atoms: a plain FP32 sum (pair forces are
// ~1 % of the valence forces, so its rounding stays below the compensated sum's).
__device__ inline void scatter_pair(const Contrib<float>& c, float* pr) {
  float a[2][3];
#pragma unroll
  for (int m = 0; m < 2; ++m)
#pragma unroll
    for (int d = 0; d < 3; ++d) a[m][d] = pr[3 * c.a[m] + d];
#pragma unroll
  for (int m = 0; m < 2; ++m)
#pragma unroll
    for (int d = 0; d < 3; ++d) pr[3 * c.a[m] + d] = a[m][d] + c.g[m][d];
}

// abdamp (src/abdamp.f90:36-51), irc = 1 / rcut
__device__ inline void abdamp(float irc, float r2, float& damp, float& ddamp) {
  const float x = r2 * irc, rr = x * x;
  damp = __frcp_rn(1.0f + rr);  // = 1/(1 + rr), correctly rounded
  ddamp = -4.0f * irc * x * (damp * damp);
}

// A bead's coordinates: FP64 (mixed form: in global memory, for the H/halogen bonds),
// and (mixed form) the FP32 split x = hi + lo.
struct BeadPos {
  const double* x;
  const float2* hl;  // (hi, lo) per coordinate (mixed form only)
  const double* w;   // tangent direction (dual coordinates only)
  const PBox* pbc;   // the bead's box where periodic, else NULL
  int wrap;          // bit d: displacements along d may exceed half the edge (wrap_dims)
};

// box_image (src/box_image.f90:36-63): subtract the edge while a component
// exceeds half of it; bounded (a non-finite or absurd vector stops after
// kImageIters subtractions and the step's NaN check reports it).  In FP32
// the vector is a (hi, lo) pair and the edge is subtracted as one.
constexpr int kImageIters = 64;
__device__ inline double image1(double v, double len, double half) {
  for (int it = 0; it < kImageIters && fabs(v) > half; ++it) v = v - copysign(len, v);
  return v;
}
// FP32: the difference of two (hi, lo) coordinates as an exact float pair
// first (atoms a box edge apart are not close enough for the hi parts to
// subtract exactly), the edge subtracted as a pair, then rounded once.
// |d| > half, so that the choice of image agrees with FP64's except within
// ~1e-14 of half the edge: the hi part decides unless it lies within 4 ulps
// of half, where |d| - half is formed as a float pair.
static __device__ __noinline__ bool beyond_half_pair(FF d, float half, float half_lo) {
  const FF a = d.hi < 0.0f ? FF{-d.hi, -d.lo} : d;
  const FF t = ff_add(a, FF{-half, -half_lo});
  return t.hi > 0.0f || (t.hi == 0.0f && t.lo > 0.0f);
}
__device__ inline bool beyond_half(FF d, const PBox& b, int k) {
  const float ah = fabsf(d.hi);
  if (ah > b.fhalf_up[k]) return true;
  if (ah < b.fhalf_dn[k]) return false;
  return beyond_half_pair(d, b.fhalf[k], b.fhalf_lo[k]);  // out of line: rarely taken
}
__device__ inline float image1(FF d, const PBox& b, int k) {
  const float len = b.flen[k], len_lo = b.flen_lo[k];
  for (int it = 0; it < kImageIters && beyond_half(d, b, k); ++it) {
    const float s = copysignf(1.0f, d.hi);
    d = ff_add(d, FF{-s * len, -s * len_lo});
  }
  return d.hi + d.lo;
}

template <class F>
__device__ inline void disp(const BeadPos& X, int a, int b, F* v);
template <>
__device__ inline void disp<double>(const BeadPos& X, int a, int b, double* v) {
  v[0] = X.x[3 * a] - X.x[3 * b];
  v[1] = X.x[3 * a + 1] - X.x[3 * b + 1];
  v[2] = X.x[3 * a + 2] - X.x[3 * b + 2];
  if (X.pbc) {
#pragma unroll
    for (int d = 0; d < 3; ++d)
      if (X.wrap >> d & 1) v[d] = image1(v[d], X.pbc->len[d], X.pbc->half[d]);
  }
}
template <>
__device__ inline void disp<Dual>(const BeadPos& X, int a, int b, Dual* v) {
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    double x = X.x[3 * a + d] - X.x[3 * b + d];
    if (X.pbc) x = image1(x, X.pbc->len[d], X.pbc->half[d]);
    v[d] = Dual(x, X.w[3 * a + d] - X.w[3 * b + d]);
  }
}
template <>
__device__ inline void disp<float>(const BeadPos& X, int a, int b, float* v) {
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    const float2 u = X.hl[3 * a + d], w = X.hl[3 * b + d];
    if (X.pbc && (X.wrap >> d & 1))
      v[d] = image1(ff_add(FF{u.x, u.y}, FF{-w.x, -w.y}), *X.pbc, d);
    else v[d] = (u.x - w.x) + (u.y - w.y);
  }
}

// Bond stretch of the mixed form (src/ff_eg.f90:87-163): with u = (r0/r)^(a/2) = exp(-(a/2) log1p(x)), x = (r - r0)/r0
// taken from the FP64 r^2 - r0^2, e = k (1 - u)^2 and the gradient factor
// a k u (1 - u) / r^2 are free of the cancellation in 1 + u^2 - 2u.
// Bond stretches carry the largest forces of a molecule, so FP32 roundings
// of their gradient set the form's force error (~4e-7 of the largest force;
// angles, torsions and pairs stay below 7e-8).  The gradient is therefore
// taken in double-FP32 arithmetic without transcendentals: with
// t = r^2/r0^2 - 1,
// a k u (1 - u) / r^2 = (a k / r0^2) [(1+t)^-(a/4+1) - (1+t)^-(a/2+1)]
//                     = t H(t),
// H a degree-23 polynomial in t / kBondSerMaxT (Chebyshev interpolation of
// H on |t| <= kBondSerMaxT, fitted per bond on the host, relative error
// below 1e-10 for exponents a <= 16), summed by Horner; the displacement
// comes exactly from the (hi, lo) coordinates and the gradient is scattered
// as its (hi, lo) pair.  Beyond that range, and for the energy, the FP32
// formula above (the FP64 pipe would cost more than the whole FP32 term).
__device__ inline float bond_mixed(const Dev& D, const BeadPos& x, int m, Contrib<float>& c, float* vir) {
  const unsigned at = __ldg(D.bond + m);
  const int i = lo16(at), j = hi16(at), st = D.st[0];
  const float2* ser = D.bser + m;  // value c at [c st]
  const float* v = D.f.bond + m;
  // displacement as double-FP32 from the (hi, lo) coordinates
  FF dv[3];
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    const float2 a = x.hl[3 * i + d], b = x.hl[3 * j + d];
    dv[d] = ff_add(FF{a.x, a.y}, FF{-b.x, -b.y});
    if (x.pbc && (x.wrap >> d & 1)) {
      for (int it = 0; it < kImageIters && beyond_half(dv[d], *x.pbc, d); ++it) {
        const float sg = copysignf(1.0f, dv[d].hi);
        dv[d] = ff_add(dv[d], FF{-sg * x.pbc->flen[d], -sg * x.pbc->flen_lo[d]});
      }
    }
  }
  FF r2f = ff_mul(dv[0], dv[0]);
  r2f = ff_add(r2f, ff_mul(dv[1], dv[1]));
  r2f = ff_add(r2f, ff_mul(dv[2], dv[2]));
  const FF r0sq = ff_of(__ldg(ser + st));
  const float r2 = r2f.hi;
  const float r = sqrtf(r2);
  const float r0 = __ldg(v);
  const FF d2 = ff_add(r2f, FF{-r0sq.hi, -r0sq.lo});
  const float dr = (d2.hi + d2.lo) / (r + r0);  // r - r0
  const float kij = __ldg(v + st), aai = __ldg(v + 2 * st);
  const float lg = -0.5f * aai * log1pf(dr / r0);
  const float omu = -expm1f(lg);  // 1 - u
  const float u = 1.0f - omu;
  const float fac = aai * kij * u * omu / r2;  // a k (u - u^2) / r^2
  c.na = 2;
  c.a[0] = i;
  c.a[1] = j;
  const FF t = ff_add(ff_mul(r2f, ff_of(__ldg(ser))), FF{-1.0f, 0.0f});
  if (__ldg(ser + 2 * st).x != 0.0f && fabsf(t.hi) <= (float)kBondSerMaxT) {
    // 1 / kBondSerMaxT = 20/9 as a double-FP32 constant
    const FF xs = ff_mul(t, FF{2.22222232818603515625f, -1.0596381372e-07f});
    FF h = ff_of(__ldg(ser + (3 + kBondPoly - 1) * st));
#pragma unroll
    for (int k = kBondPoly - 2; k >= 0; --k) h = ff_add(ff_mul(h, xs), ff_of(__ldg(ser + (3 + k) * st)));
    const FF f = ff_mul(t, h);
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      const FF g = ff_mul(f, dv[d]);
      c.g[0][d] = g.hi;
      c.g[1][d] = -g.hi;
      c.g[2][d] = g.lo;
      c.g[3][d] = -g.lo;
    }
  } else {
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      const float rb = dv[d].hi;
      c.g[0][d] = fac * rb;
      c.g[1][d] = -fac * rb;
      c.g[2][d] = 0.0f;
      c.g[3][d] = 0.0f;
    }
  }
  if (vir) *vir = dv[0].hi * (c.g[0][0] + c.g[2][0]) + dv[1].hi * (c.g[0][1] + c.g[2][1]) + dv[2].hi * (c.g[0][2] + c.g[2][2]);
  return kij * omu * omu;
}

// Angle bend with abdamp damping (src/ff_eg.f90:167-299), mixed form.
__device__ inline float angle_mixed(const Dev& D, const BeadPos& x, int m, Contrib<float>& c, float* vir) {
  using F = float;
  const uint2 at = __ldg(D.angl + m);
  const int i = lo16(at.x), j = hi16(at.x), k = (int)at.y, st = D.st[1];
  const float* v = D.f.angl + m;
  const F c0 = __ldg(v), kijk = __ldg(v + st), cc0 = __ldg(v + 2 * st);
  const bool linear = __ldg(v + 3 * st) != 0.f;
  F vab[3], vcb[3], vp[3];
  disp<F>(x, i, j, vab);
  disp<F>(x, k, j, vcb);
  const F rab2 = dot3(vab, vab), rcb2 = dot3(vcb, vcb);
  cross(vcb, vab, vp);
  const F vpl = dot3(vp, vp);
  const F rp = (vpl > F(0) ? q_sqrt<F>(vpl) : F(0)) + F(1e-14);
  const F al = q_sqrt<F>(rab2), bl = q_sqrt<F>(rcb2);
  F cosa = (al > F(0) && bl > F(0)) ? dot3(vab, vcb) / (al * bl) : F(0);
  cosa = fmin(F(1), fmax(F(-1), cosa));
  // FP32: theta only for linear reference angles; sin(theta) of the
  // harmonic-cosine form as sqrt((1 - c)(1 + c)), free of cancellation away
  // from c = +-1 (where the linear form is used)
  F theta = F(0);
  if (linear) theta = acosf(cosa);
  F dampij, damp2ij, dampjk, damp2jk;
  abdamp(__ldg(v + 4 * st), rab2, dampij, damp2ij);
  abdamp(__ldg(v + 5 * st), rcb2, dampjk, damp2jk);
  const F damp = dampij * dampjk;
  F ea, deddt;
  if (linear) {  // linear reference angle: harmonic in theta
    const F dt = theta - c0;
    ea = kijk * (dt * dt);
    deddt = F(2) * kijk * dt;
  } else {
    const F dd = cosa - cc0;
    ea = kijk * (dd * dd);
    const F sth = sqrtf((1.0f - cosa) * (1.0f + cosa));
    deddt = F(2) * kijk * sth * (cc0 - cosa);
  }
  F deda[3], dedc[3];
  cross(vab, vp, deda);
  cross(vcb, vp, dedc);
  const F rmul1 = -deddt / (rab2 * rp), rmul2 = deddt / (rcb2 * rp);
  c.na = 3;
  c.a[0] = i;
  c.a[1] = j;
  c.a[2] = k;
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    const F da = deda[d] * rmul1, dc = dedc[d] * rmul2;
    const F t1 = ea * damp2ij * dampjk * vab[d];
    const F t2 = ea * damp2jk * dampij * vcb[d];
    c.g[0][d] = da * damp + t1;
    c.g[1][d] = -(da + dc) * damp - t1 - t2;
    c.g[2][d] = dc * damp + t2;
  }
  if (vir) *vir = dot3(vab, c.g[0]) + dot3(vcb, c.g[2]);
  return ea * damp;
}

// Torsion angle phi in [0, pi] of i-j-k-l (valijkl, src/valijkl.f90) with its
// cosine and sine, as atan2(|rb| |na . rc|, na . nb), accurate near 0 and pi.
__device__ inline float dihedral(const float* ra, const float* rb, const float* rc, float* na, float* nb, float& nan_,
                                 float& nbn, float& cosphi, float& sinphi) {
  cross(ra, rb, na);
  cross(rb, rc, nb);
  nan_ = sqrtf(dot3(na, na));
  nbn = sqrtf(dot3(nb, nb));
  const float cn = dot3(na, nb);
  const float sn = sqrtf(dot3(rb, rb)) * fabsf(dot3(na, rc));
  const float phi = atan2f(sn, cn);
  const float den = nan_ * nbn;
  const float id = den > 0.f ? __frcp_rn(den) : 0.f;
  cosphi = den > 0.f ? cn * id : 1.f;
  sinphi = den > 0.f ? sn * id : 0.f;
  return phi;
}

// vab.g_a + vcb.(g_c + g_d) + vdc.g_d with the term's own vectors: the
// torsions' and inversions' vir_ten (src/ff_eg.f90:420-440, 583-603).
template <class F>
__device__ inline F tors_virial(const F* vab, const F* vcb, const F* vdc, const Contrib<F>& c) {
  const F gcd[3] = {c.g[2][0] + c.g[3][0], c.g[2][1] + c.g[3][1], c.g[2][2] + c.g[3][2]};
  return dot3(vab, c.g[0]) + dot3(vcb, gcd) + dot3(vdc, c.g[3]);
}

// Torsions (erf-blended cosine series, src/ff_eg.f90:303-440) and
// inversions (tors type 2, src/ff_eg.f90:441-618), mixed form.
__device__ inline float torsion_mixed(const Dev& D, const BeadPos& x, int m, Contrib<float>& c, float* vir = nullptr) {
  using F = float;
  const F pi = (F)3.1415926535897932384626433832795029;
  const F pi2 = (F)6.28318530717958623199592693708837;
  const uint4 at = __ldg(D.tors + m);
  const int i = lo16(at.x), j = hi16(at.x), k = lo16(at.y), l = hi16(at.y), nt = (int)(at.z & 255u), type = (int)(at.z >> 8);
  const int st = D.st[2];
  auto vt = [&](int c) { return __ldg(D.f.tors + c * st + m); };
  const F phi0 = vt(0);
  F vab[3], vcb[3], vdc[3], dda[3], ddb[3], ddc[3], ddd[3];
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
    abdamp(vt(14), dot3(vab, vab), dampij, d2ij);
    abdamp(vt(15), dot3(vcb, vcb), dampjk, d2jk);
    abdamp(vt(16), dot3(vdc, vdc), dampX, d2X);
    // dphidr (src/dphidr.f90): ra = r_j - r_i, rb = r_k - r_j, rc = r_l - r_k
    const F ra[3] = {-vab[0], -vab[1], -vab[2]}, rb[3] = {-vcb[0], -vcb[1], -vcb[2]};
    const F rc[3] = {-vdc[0], -vdc[1], -vdc[2]};
    F na[3], nb[3], nan_, nbn, cosphi, sinphi;
    const F phi = dihedral(ra, rb, rc, na, nb, nan_, nbn, cosphi, sinphi);
    {
      // FP32: dphi/dr without the division by sin(phi) of dphidr.f90, whose
      // numerator cancels as phi -> 0 or pi (planar groups); the same
      // derivative, written with the plane normals (Blondel and Karplus,
      // J. Comput. Chem. 17, 1132 (1996)):
      //   dphi/dr_i = -s |rb| na / |na|^2,  dphi/dr_l = s |rb| nb / |nb|^2,
      //   dphi/dr_j = -dphi/dr_i + s (u + v),  dphi/dr_k = -dphi/dr_l - s (u + v),
      //   u = (ra.rb) na / (|na|^2 |rb|),  v = (rc.rb) nb / (|nb|^2 |rb|),
      // s = sign(na.rc) (phi is the unsigned angle)
      const float a2 = dot3(na, na), b2 = dot3(nb, nb), tr = dot3(na, rc);
      const float sg = (tr > 0.f) ? 1.f : ((tr < 0.f) ? -1.f : 0.f);
      if (!(a2 > 0.f) || !(b2 > 0.f)) {
#pragma unroll
        for (int d = 0; d < 3; ++d) dda[d] = ddb[d] = ddc[d] = ddd[d] = 0.f;
      } else {
        const float L = sqrtf(dot3(rb, rb)), ia2 = __frcp_rn(a2), ib2 = __frcp_rn(b2), iL = __frcp_rn(L);
        const float fa = sg * L * ia2, fb = sg * L * ib2;
        const float fu = sg * dot3(ra, rb) * ia2 * iL, fv = sg * dot3(rc, rb) * ib2 * iL;
#pragma unroll
        for (int d = 0; d < 3; ++d) {
          const float uv = fu * na[d] + fv * nb[d];
          dda[d] = -fa * na[d];
          ddd[d] = fb * nb[d];
          ddb[d] = fa * na[d] + uv;
          ddc[d] = -fb * nb[d] - uv;
        }
      }
    }
    et = F(0);
    dij = F(0);
    const F phipi = phi - pi;
    const F ef = erff(phipi);
    const F expo = expf(-(phipi * phipi)) * 0.564189583547756286948f;  // 1/sqrt(pi)
    for (int it = 0; it < nt; ++it) {
      const F rn = vt(2 + 3 * it), ph = vt(3 + 3 * it), vn = vt(4 + 3 * it);
      const F c1 = rn * (phi - phi0) + ph;
      const F c2 = rn * (phi + phi0 - pi2) + ph;
      F x1cos, x2cos, x1sin, x2sin;
      sincosf(c1, &x1sin, &x1cos);
      sincosf(c2, &x2sin, &x2cos);
      const F e1 = vn * (F(1) + x1cos), e2 = vn * (F(1) + x2cos);
      et = et + F(0.5) * (F(1) - ef) * e1 + (F(0.5) + F(0.5) * ef) * e2;
      dij = dij - expo * e1 - F(0.5) * (F(1) - ef) * vn * x1sin * rn + expo * e2 -
            (F(0.5) + F(0.5) * ef) * vn * x2sin * rn;
    }
    et = et * vt(1);
    const F damp = dampjk * dampij * dampX;
    dij = dij * vt(1) * damp;
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      const F t1 = et * d2ij * dampjk * dampX * vab[d];
      const F t2 = et * d2jk * dampij * dampX * vcb[d];
      const F t3 = et * d2X * dampij * dampjk * vdc[d];
      c.g[0][d] = dij * dda[d] + t1;
      c.g[1][d] = dij * ddb[d] - t1 + t2;
      c.g[2][d] = dij * ddc[d] + t3 - t2;
      c.g[3][d] = dij * ddd[d] - t3;
    }
    if (vir) *vir = tors_virial(vab, vcb, vdc, c);
    return et * damp;
  }
  // inversion: omega (src/omega.f90) and domegadr (src/domegadr.f90)
  disp<F>(x, j, i, vab);
  disp<F>(x, j, k, vcb);
  disp<F>(x, j, l, vdc);
  abdamp(vt(14), dot3(vab, vab), dampij, d2ij);
  abdamp(vt(15), dot3(vcb, vcb), dampjk, d2jk);
  abdamp(vt(16), dot3(vdc, vdc), dampX, d2X);
  const F re[3] = {-vab[0], -vab[1], -vab[2]};  // r_i - r_j
  const F rd[3] = {-vcb[0], -vcb[1], -vcb[2]};  // r_k - r_j
  F rv[3];
  disp<F>(x, l, i, rv);                          // r_l - r_i
  F rn[3];
  cross(re, rd, rn);
  const F rnn = q_sqrt<F>(dot3(rn, rn)), rvn = q_sqrt<F>(dot3(rv, rv));
  const F om = asinf(fmin(F(1), fmax(F(-1), dot3(rn, rv) / (rnn * rvn))));
  const F sinom = sinf(om), cosom = cosf(om);
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
    const F on = F(1) / nenner;
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      dda[d] = on * (rdv[d] - rn[d] - sinom * (rvn / rnn * rdn[d] - rnn / rvn * rv[d]));
      ddb[d] = on * (rvdme[d] - sinom * rvn / rnn * rndme[d]);
      ddc[d] = on * (rve[d] - sinom * rvn / rnn * rne[d]);
      ddd[d] = on * (rn[d] - sinom * rnn / rvn * rv[d]);
    }
  } else {
#pragma unroll
    for (int d = 0; d < 3; ++d) dda[d] = ddb[d] = ddc[d] = ddd[d] = F(0);
  }
  const F damp = dampjk * dampij * dampX;
  {
    // FP32: the differences of cosines as products of sines, cos a - cos b
    // = -2 sin((a+b)/2) sin((a-b)/2) and 1 - cos a = 2 sin^2(a/2): near
    // omega = phi0 the reference's forms cancel to a few bits in float,
    // which the large inversion barriers of planar centres (tens of Eh)
    // turn into force errors of 1e-6
    const float h = 0.5f * (om - phi0), sh = sinf(h);
    if (vt(2) > 1e-6f) {
      et = 2.f * sh * sh * vt(1);
      dij = sinf(om - phi0) * vt(1) * damp;
    } else {
      const float dd = -2.f * sinf(0.5f * (om + phi0)) * sh;  // cos(om) - cos(phi0)
      et = vt(1) * (dd * dd);
      dij = -2.f * vt(1) * sinf(om) * dd * damp;
    }
  }
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    const F t1 = et * d2ij * dampjk * dampX * vab[d];
    const F t2 = et * d2jk * dampij * dampX * vcb[d];
    const F t3 = et * d2X * dampij * dampjk * vdc[d];
    c.g[0][d] = dij * dda[d] - t1;
    c.g[1][d] = dij * ddb[d] + t1 + t2 + t3;
    c.g[2][d] = dij * ddc[d] - t2;
    c.g[3][d] = dij * ddd[d] - t3;
  }
  if (vir) *vir = tors_virial(vab, vcb, vdc, c);
  return et * damp;
}

}  // namespace qmdff
}  // namespace cr

#include "qmdff_plain.cuh"

namespace cr {
namespace qmdff {

// FP32 hardware approximations (PTX rsqrt / rcp / ex2 .approx.ftz, relative
// error about 2^-22): inputs here are normal numbers far from the limits.
__device__ inline float rsqrt_approx(float x) {
  float y;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ inline float rcp_approx(float x) {
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ inline float ex2_approx(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// One NCI pair in the mixed form: the formulas of pair_plain with the
// constants folded (R0^6 and R0^8 of the BJ damping, eps2 into the C6 and
// repulsion prefactors, alpha log2(e) for a base-2 exponential).  The pair forces are ~1 % of the valence
// forces, so hardware approximations stay far below the form's error budget.
__device__ inline float pair_mixed(const Dev& D, const BeadPos& x, uint4 pr, Contrib<float>& c, float* vir) {
  const int i1 = lo16(pr.x), i2 = hi16(pr.x);
  const float4 ca = __ldg(D.pclass + 2 * pr.y), cb = __ldg(D.pclass + 2 * pr.y + 1);
  const float c6 = __uint_as_float(pr.z), qq = __uint_as_float(pr.w);
  float vab[3];
  disp<float>(x, i1, i2, vab);
  const float r2 = dot3(vab, vab);
  const float oner = rsqrt_approx(r2), r = r2 * oner, ir2 = oner * oner;
  const float r4 = r2 * r2, r6 = r4 * r2;
  const float it6 = rcp_approx(r6 + ca.x), it8 = rcp_approx(r6 * r2 + ca.y);
  const float d6 = c6 * it6, d8 = c6 * ca.z * it8;
  const bool vdw = !x.pbc || !(r > D.fvdw_cut);
  float e = vdw ? -(d6 + d8) : 0.0f;
  float drij = vdw ? 6.0f * d6 * (r4 * it6) + 8.0f * d8 * (r6 * it8) : 0.0f;
  if (vdw && r < 25.0f) {
    const float t = ca.w * ex2_approx(-cb.x * r) * oner;
    e += t;
    drij = fmaf(-t * ir2, fmaf(cb.y, r, 1.0f), drij);
  }
  if (!(r > D.fcoul_cut)) {
    float e0;
    if (D.zahn) e0 = qq * ((q_erfc<float>(D.fzahn_a * r) * oner) - D.fzahn_par * (r - D.fcoul_cut));
    else e0 = qq * oner;
    e += e0;
    drij = fmaf(-e0, ir2, drij);
  }
  c.na = 2;
  c.a[0] = i1;
  c.a[1] = i2;
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    c.g[0][d] = vab[d] * drij;
    c.g[1][d] = -vab[d] * drij;
  }
  if (vir) *vir = r2 * drij;  // vab . g_i1 with g_i1 = vab drij (NpT)
  return e;
}

// x^5, x^6, x^12 by products (the reference's real-exponent ** operators)
template <class F>
__device__ inline F pow6(F x) {
  const F x2 = x * x;
  return x2 * x2 * x2;
}

// eabhag (src/eabhag.f90:35-220): hydrogen bond A...H-B; nothing if the
// energy is above -1e-8 (the reference returns before its gradient).
template <class F>
__device__ inline F hbond_term(const BeadPos& X, int A, int B, int H, F ca, F cb, Contrib<F>& c) {
  const F longcut = F(8.0), alp7 = F(12.0), alp3 = F(6.0);
  F drah[3], drbh[3], drab[3];
  disp<F>(X, A, H, drah);
  disp<F>(X, B, H, drbh);
  disp<F>(X, A, B, drab);
  c.a[0] = A;
  c.a[1] = B;
  c.a[2] = H;
  const F rab2 = dot3(drab, drab), rab = q_sqrt<F>(rab2);
  const F rah2 = dot3(drah, drah), rah = q_sqrt<F>(rah2);
  const F rbh2 = dot3(drbh, drbh), rbh = q_sqrt<F>(rbh2);
  const F q6 = pow6<F>(rab / longcut);
  const F ratio = q6 * q6;
  F rdampl = F(1) / (F(1) + ratio);
  rdampl = rdampl / rab2 / rab;
  const bool far_a = rah2 > rbh2;
  F cosabh, aprod;
  if (far_a) {
    aprod = F(1) / rbh / rab;
    cosabh = -dot3(drbh, drab) * aprod;
  } else {
    aprod = F(1) / rah / rab;
    cosabh = dot3(drah, drab) * aprod;
  }
  F aterm = F(0.5) * (cosabh + F(1));
  const F a2 = aterm * aterm;
  F apref = a2 * a2 * aterm;  // aterm**(alp3-1)
  aterm = aterm * apref;
  apref = alp3 * F(0.5) * apref;
  const F rah4 = rah2 * rah2, rbh4 = rbh2 * rbh2;
  const F denom = F(1) / (rah4 + rbh4);
  const F da = (ca * rah4 + cb * rbh4) * denom;
  const F eabh = -da * rdampl * aterm;
#pragma unroll
  for (int m = 0; m < 3; ++m)
#pragma unroll
    for (int d = 0; d < 3; ++d) c.g[m][d] = F(0);
  if (eabh > F(-1.0e-8)) return F(0);
  F ga[3], gb[3], gh[3];
  F gi = F(4) * (ca - cb) * rah2 * rbh4 * denom * denom;
  gi = -gi * rdampl * aterm;
  F gj = F(4) * (cb - ca) * rbh2 * rah4 * denom * denom;
  gj = -gj * rdampl * aterm;
  F gl = rdampl * rdampl * rab * (F(3) + (F(3) + alp7) * ratio);
  gl = gl * da * aterm;
  const F gn = -da * rdampl * apref;
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    ga[d] = gi * drah[d];
    gb[d] = gj * drbh[d];
    gh[d] = -ga[d] - gb[d];
    const F dl = gl * drab[d];
    ga[d] += dl;
    gb[d] -= dl;
    if (far_a) {
      const F dg = gn * (-aprod * drbh[d] - cosabh * drab[d] / rab2);
      const F dg2 = gn * (aprod * drab[d] + cosabh * drbh[d] / rbh2);
      ga[d] += dg;
      gh[d] += dg2;
      gb[d] = gb[d] - dg - dg2;
    } else {
      const F dg = gn * (-aprod * drah[d] + cosabh * drab[d] / rab2);
      const F dg2 = gn * (-aprod * drab[d] + cosabh * drah[d] / rah2);
      gb[d] += dg;
      gh[d] += dg2;
      ga[d] = ga[d] - dg - dg2;
    }
    c.g[0][d] = ga[d];
    c.g[1][d] = gb[d];
    c.g[2][d] = gh[d];
  }
  return eabh;
}

// eabx (src/eabx.f90:34-111) on the three atoms' coordinates xa, xb, xh.
__device__ inline double eabx(const double* xa, const double* xb, const double* xh, double ca) {
  double rb[3];
#pragma unroll
  for (int d = 0; d < 3; ++d) rb[d] = xa[d] - xb[d];
  const double rab2 = rb[0] * rb[0] + rb[1] * rb[1] + rb[2] * rb[2];
  const double dampl = 1.0 / (1.0 + pow6<double>(rab2 / 120.0));
#pragma unroll
  for (int d = 0; d < 3; ++d) rb[d] = xa[d] - xh[d];
  const double d2ik = rb[0] * rb[0] + rb[1] * rb[1] + rb[2] * rb[2];
#pragma unroll
  for (int d = 0; d < 3; ++d) rb[d] = xh[d] - xb[d];
  const double d2jk = rb[0] * rb[0] + rb[1] * rb[1] + rb[2] * rb[2];
  double term;
  if (d2ik > d2jk) term = 0.5 * (rab2 + d2jk - d2ik) / sqrt(rab2 * d2jk);
  else term = 0.5 * (rab2 + d2ik - d2jk) / sqrt(rab2 * d2ik);
  const double aterm = pow6<double>(0.5 * (term + 1.0));
  return -ca * dampl * aterm / d2jk;
}

// eabxag (src/eabxag.f90:35-156): halogen bond A...X-B, energy and Caracal's
// central-difference gradient (step 1e-6), FP64 in both forms.  As in the
// reference, each atom's three components all receive the z quotient.
template <class F>
__device__ inline F xbond_term(const BeadPos& X, int A, int B, int H, double ca, Contrib<F>& c) {
  double p[3][3];
  const int at[3] = {A, B, H};
#pragma unroll
  for (int m = 0; m < 3; ++m)
#pragma unroll
    for (int d = 0; d < 3; ++d) p[m][d] = X.x[3 * at[m] + d];
  const double e = eabx(p[0], p[1], p[2], ca);
  const double step = 1.0e-6, dum = 1.0 / (2.0 * step);
#pragma unroll
  for (int m = 0; m < 3; ++m) {
    double last = 0.0;
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      p[m][j] = p[m][j] + step;
      const double er = eabx(p[0], p[1], p[2], ca);
      p[m][j] = p[m][j] - step * 2.0;
      const double el = eabx(p[0], p[1], p[2], ca);
      p[m][j] = p[m][j] + step;
      last = (er - el) * dum;
    }
    c.a[m] = at[m];
#pragma unroll
    for (int d = 0; d < 3; ++d) c.g[m][d] = (F)last;
  }
  return (F)e;
}

// One entry of ff_hb (src/ff_hb.f90:55-79): skipped beyond 15 bohr A-B.
// Out of line (a handful of terms per molecule) to keep the register count
// of the frequent terms.
template <class F>
__device__ __noinline__ F hb_term(const Dev& D, const Tables<F>&, const BeadPos& X, int k, Contrib<F>& c) {
  const int4 t = __ldg(reinterpret_cast<const int4*>(D.hb) + k);
  double rb[3];
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    rb[d] = X.x[3 * t.x + d] - X.x[3 * t.y + d];
    if (X.pbc) rb[d] = image1(rb[d], X.pbc->len[d], X.pbc->half[d]);  // src/ff_hb.f90:64-66
  }
  const double r2 = rb[0] * rb[0] + rb[1] * rb[1] + rb[2] * rb[2];
  c.a[0] = t.x;
  c.a[1] = t.y;
  c.a[2] = t.z;
  if (sqrt(r2) > 15.0) {
#pragma unroll
    for (int m = 0; m < 3; ++m)
#pragma unroll
      for (int d = 0; d < 3; ++d) c.g[m][d] = F(0);
    return F(0);
  }
  if (t.w == 1) return hbond_term<F>(X, t.x, t.y, t.z, (F)D.vhb[2 * k], (F)D.vhb[2 * k + 1], c);
  return xbond_term<F>(X, t.x, t.y, t.z, D.vhb[2 * k], c);
}

// Energy of one term of kind KIND (0 bond, 1 angle, 2 torsion, 3 pair, 4 H/halogen
// bond); vir: its virial trace (but for H/halogen bonds: hb_virial), or NULL.
template <int KIND>
__device__ inline float term(const Dev& D, const BeadPos& x, int m, Contrib<float>& c, float* vir) {
  if constexpr (KIND == 0) return bond_mixed(D, x, m, c, vir);
  else if constexpr (KIND == 1) return angle_mixed(D, x, m, c, vir);
  else if constexpr (KIND == 2) return torsion_mixed(D, x, m, c, vir);
  else return hb_term<float>(D, D.f, x, m, c);
}
template <int KIND>
__device__ inline double term(const Dev& D, const BeadPos& x, int m, Contrib<double>& c, double* vir) {
  if constexpr (KIND == 0) return bond_plain<double>(D, D.d, x, m, c, vir);
  else if constexpr (KIND == 1) return angle_plain<double>(D, D.d, x, m, c, vir);
  else if constexpr (KIND == 2) return torsion_plain<double>(D, D.d, x, m, c, vir);
  else if constexpr (KIND == 3) return pair_plain(D, D.d, x, m, c, vir);
  else return hb_term<double>(D, D.d, x, m, c);
}

// The virial trace of one term as the reference accumulates `vir_ten` for
// NpT: bonds (src/ff_eg.f90:133-150) rbond.g_i, rbond = r_i - r_j; angles
// (:270-281) vab.g_i + vcb.g_k about the centre j; torsions (:317-320,
// 420-440) vab.g_i + vcb.(g_k + g_l) + vdc.g_l with vab = r_i - r_j,
// vcb = r_j - r_k, vdc = r_k - r_l, and inversions (:503-505, 583-603) the
// same formula with vab = r_j - r_i, vcb = r_j - r_k, vdc = r_j - r_l (for
// neither is it the sum of (r - r_j).g over the term's atoms); NCI pairs
// (src/ff_nonb.f90:180-190, 318-328, 405-415, 495-505) vab.g_i1, vab = r_i1 - r_i2; hydrogen bonds
// (src/eabhag.f90:54, 203-216) drah.g_A + drbh.g_B about H; halogen bonds
// (src/eabxag.f90:86-87, 140-153) (r_A - r_X).g_A + (r_B - r_X).g_X, the
// X atom's gradient with the B vector.  Vectors minimum-imaged as the
// terms' own.  Mixed-form bonds carry g_i as (hi, lo) in g[0] and g[2].
template <class F>
__device__ inline F hb_virial(const Dev& D, const BeadPos& X, int m, const Contrib<F>& c) {
  F u[3], v[3];
  disp<F>(X, c.a[0], c.a[2], u);
  disp<F>(X, c.a[1], c.a[2], v);
  const bool halogen = D.hb[4 * m + 3] != 1;
  return dot3(u, c.g[0]) + dot3(v, halogen ? c.g[2] : c.g[1]);
}

// Box modes of the force kernel, compile-time so the free molecule's kernel
// carries no imaging code: kFree (no box), kBox (the force field's periodic
// box), kNpt (each trajectory's box from Dev::tbox, and the virial).
constexpr int kFree = 0, kBox = 1, kNpt = 2;

// Buffer value of a list entry.
__device__ __forceinline__ double signed_value(const double* buf, unsigned e) {
  const double v = buf[e & (kNegate - 1)];
  return __hiloint2double(__double2hiint(v) ^ (int)((e & kNegate) << 16), __double2loint(v));
}

// Warps per bead of the FP64 forms.  An FP64 instruction holds its scheduler's
// pipe 64 cycles, so four warps could fill an SM's four pipes, and two per pipe hide
// the loads and the barriers; a bead is spread over eight: a small batch then takes an
// eighth of the time.  With the terms of qmdff_plain.cuh, against a warp per bead and
// their former terms, whole calls: the adjoint of 16 x 16 beads of C20H42 over 20 steps 47.4 ->
// 11.3 ms, C13H28 100 x 48, four steps 4.82 -> 1.82 ms; gradients of 65 536 beads of C2H6 4.96
// -> 3.38 ms, 16 384 of C4H10 1.56 -> 0.92, 1024 of C50H102 3.23 -> 1.70.
constexpr int kTeam = 8;

// The segment's values of one term at its slot i.
template <bool MIXED, int KIND, class G>
__device__ __forceinline__ void put_term(G* buf, int i, const Contrib<G>& c) {
  constexpr int C = segment_terms(MIXED, KIND), NA = KIND == 1 || KIND == 4 ? 3 : KIND == 2 ? 4 : 1;
#pragma unroll
  for (int a = 0; a < NA; ++a)
#pragma unroll
    for (int d = 0; d < 3; ++d) buf[(3 * a + d) * C + i] = c.g[a][d];
  if constexpr (MIXED && KIND == 0) {
#pragma unroll
    for (int d = 0; d < 3; ++d) buf[(3 + d) * C + i] = c.g[2][d];
  }
}

// Sums of a segment's gather, rounds r0, r0 + step, ...: list value x onto
// coordinate a by add(a, list).
template <class Sum>
__device__ __forceinline__ void gather(const Schedule& S, int4 sg, int r0, int step, int lane, Sum sum) {
  for (int r = sg.z + r0; r < sg.z + sg.w; r += step) {
    const int2 rd = __ldg(S.round + r);
    const int a = S.dst[32 * r + lane];
    if (a != kNoDst) sum(a, S.ent + rd.x + lane, rd.y);
  }
}

// All segments of one term kind, mixed form, by one warp: compensated sums.
template <int KIND, int MODE>
__device__ inline void kind_segments(const Dev& D, const BeadPos& X, float* buf, float2* sk, float& es, float& ec,
                                     float& wv, int lane) {
  const Schedule& S = D.sched[1];
  for (int sgi = S.seg0[KIND]; sgi < S.seg1[KIND]; ++sgi) {
    const int4 sg = __ldg(S.seg + sgi);
    for (int i = lane; i < sg.y; i += 32) {
      const int m = sg.x + i;
      Contrib<float> c;
      float w = 0.f;
      float v;
      v = term<KIND>(D, X, m, c, MODE == kNpt ? &w : nullptr);
      if constexpr (MODE == kNpt) {
        if constexpr (KIND == 4) w = hb_virial<float>(D, X, m, c);
        wv += w;
      }
      const float t = es + v;
      ec += (fabsf(es) >= fabsf(v)) ? ((es - t) + v) : ((v - t) + es);
      es = t;
      put_term<true, KIND>(buf, i, c);
    }
    __syncwarp();
    gather(S, sg, 0, 1, lane, [&](int a, const unsigned short* l, int n) {
      float2 k = sk[a];
#pragma unroll 4
      for (int j = 0; j < n; ++j) {
        const unsigned e = __ldg(l + 32 * j);
        const float v = __uint_as_float(__float_as_uint(buf[e & (kNegate - 1)]) ^ ((e & kNegate) << 16));
        const float t = k.x + v, z = t - k.x;
        k.y += (k.x - (t - z)) + (v - z);
        k.x = t;
      }
      sk[a] = k;
    });
    __syncwarp();
  }
}

// ... FP64 form, by a team of warps.
template <int KIND, int MODE>
__device__ inline void kind_segments(const Dev& D, const BeadPos& X, double* buf, double* g, double& es, double& wv) {
  const Schedule& S = D.sched[0];
  for (int sgi = S.seg0[KIND]; sgi < S.seg1[KIND]; ++sgi) {
    const int4 sg = __ldg(S.seg + sgi);
    for (int i = threadIdx.x; i < sg.y; i += kTeam * 32) {
      const int m = sg.x + i;
      Contrib<double> c;
      double w = 0.0;
      es += term<KIND>(D, X, m, c, MODE == kNpt ? &w : nullptr);
      if constexpr (MODE == kNpt) {
        if constexpr (KIND == 4) w = hb_virial<double>(D, X, m, c);
        wv += w;
      }
      put_term<false, KIND>(buf, i, c);
    }
    __syncthreads();
    gather(S, sg, threadIdx.x >> 5, kTeam, threadIdx.x & 31, [&](int a, const unsigned short* l, int n) {
      double v = g[a];
#pragma unroll 4
      for (int j = 0; j < n; ++j) v += signed_value(buf, __ldg(l + 32 * j));
      g[a] = v;
    });
    __syncthreads();
  }
}

// Mixed-form NCI pairs: every batch is one matching, so each lane adds its pair's
// gradient right after the term; the next batch's table row is loaded before
// the current batch's arithmetic, so its latency overlaps the work.
template <int MODE>
__device__ inline void pair_batches_mixed(const Dev& D, const BeadPos& X, float* pr, float& es, float& ec,
                                          float& wv, int lane) {
  const int nb = D.sched[1].npair;
  if (nb <= 0) return;
  uint4 next = __ldg(D.fpair + lane);
  for (int b = 0; b < nb; ++b) {
    const uint4 row = next;
    if (b + 1 < nb) next = __ldg(D.fpair + 32 * (b + 1) + lane);
    if (row.y != kNoPair) {
      Contrib<float> c;
      float w = 0.0f;
      const float e = pair_mixed(D, X, row, c, MODE == kNpt ? &w : nullptr);
      const float t = es + e;
      ec += (fabsf(es) >= fabsf(e)) ? ((es - t) + e) : ((e - t) + es);
      es = t;
      if constexpr (MODE == kNpt) wv += w;
      scatter_pair(c, pr);
    }
    __syncwarp();
  }
}

// Shared memory of a mixed-form warp (bytes): the coordinates' FP32 split (hi, lo)
// (3n float pairs), the gradient ((sum, compensation) float pairs and
// the 3n floats of the pair sum) and the buffer with its zero, in whole 16-byte
// units: the warps' regions follow one another.
__host__ __device__ inline size_t warp_smem_bytes(int n) {
  return ((size_t)3 * n * (4 + 4 + 8 + 4) + (buffer_values(true) + 1) * 4 + 15) / 16 * 16;
}
// ... of an FP64 team: coordinates, gradient, buffer and zero, the warps' energies and virials
__host__ __device__ inline size_t team_smem_bytes(int n) {
  return ((size_t)3 * n * 2 + buffer_values(false) + 1 + 2 * kTeam) * 8;
}

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o >= 1; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// The dimensions along which the bead is longer than half the edge (less a margin
// over the FP32 rounding here): along the others box_image subtracts nothing from
// any of its displacements, and skipping it spares the terms' largest part in
// periodic boxes (C20H42 256 x 64 in a 40 Angstrom
// box, per step with the berendsen kernel 559 -> 510 us).
__device__ inline int wrap_dims(const double* x, int n, const PBox& b, int lane) {
  int wrap = 0;
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    float lo = 3e38f, hi = -3e38f;
    bool fine = true;
    for (int a = lane; a < n; a += 32) {
      const float v = __double2float_rn(x[3 * a + d]);
      fine = fine && fabsf(v) < 1e30f;
      lo = fminf(lo, v);
      hi = fmaxf(hi, v);
    }
#pragma unroll
    for (int o = 16; o >= 1; o >>= 1) {
      lo = fminf(lo, __shfl_xor_sync(0xffffffffu, lo, o));
      hi = fmaxf(hi, __shfl_xor_sync(0xffffffffu, hi, o));
    }
    fine = __all_sync(0xffffffffu, fine);
    if (!fine || !(hi - lo < 0.999f * b.fhalf[d] - 4e-7f * (fabsf(hi) + fabsf(lo)))) wrap |= 1 << d;
  }
  return wrap;
}

// The box of a launch's mode as a local copy: taking the address of the kernel
// parameter D would move all of it from the constant bank to local memory.
template <int MODE>
__device__ inline const PBox* launch_box(const Dev& D, size_t bead, PBox& tb) {
  if constexpr (MODE == kNpt) {  // this trajectory's box
    tb = make_box(D.tbox + 3 * (size_t)(bead / (size_t)D.tbox_beads));
    return &tb;
  } else if constexpr (MODE == kBox) {
    tb = D.box;
    return &tb;
  }
  return nullptr;
}

// Energy (with E_zero) and gradient of one bead by one warp, mixed form.
// ws: the warp's shared memory; x: the bead's coordinates; gout, gout2: the gradient destinations (gout2 = gout: one).  Returns the energy on every lane.
// MODE (kFree, kBox, kNpt): with kNpt the bead's trajectory box from D.tbox
// and the virial trace into D.vir (rows bead and twin).
template <int MODE = kFree>
__device__ inline double warp_egrad(const Dev& D, void* ws, const double* x, double* gout, double* gout2, int lane,
                                    size_t bead, size_t twin) {
  const int n3 = 3 * D.n;
  float2* hl = (float2*)ws;
  PBox tb;
  const PBox* box = launch_box<MODE>(D, bead, tb);
  const BeadPos X{x, hl, nullptr, box, MODE == kFree ? 0 : wrap_dims(x, D.n, tb, lane)};
  float2* sk = hl + n3;
  float* pr = (float*)(sk + n3);
  float* buf = pr + n3;
  for (int a = lane; a < n3; a += 32) {
    const double v = x[a];
    const float h = __double2float_rn(v);
    hl[a] = make_float2(h, __double2float_rn(v - (double)h));
    sk[a] = make_float2(0.f, 0.f);
    pr[a] = 0.f;
  }
  if (lane == 0) buf[buffer_values(true)] = 0.f;
  __syncwarp();
  float es = 0.f, ec = 0.f;  // compensated lane sum of term energies
  float wv = 0.f;            // lane sum of the terms' virial traces (NpT)
  kind_segments<0, MODE>(D, X, buf, sk, es, ec, wv, lane);
  kind_segments<1, MODE>(D, X, buf, sk, es, ec, wv, lane);
  kind_segments<2, MODE>(D, X, buf, sk, es, ec, wv, lane);
  pair_batches_mixed<MODE>(D, X, pr, es, ec, wv, lane);
  kind_segments<4, MODE>(D, X, buf, sk, es, ec, wv, lane);
  for (int a = lane; a < n3; a += 32) {
    const double v = ((double)sk[a].x + (double)sk[a].y) + (double)pr[a];
    gout[a] = v;
    if (gout2 != gout) gout2[a] = v;
  }
  const double e = warp_sum((double)es + (double)ec);
  if constexpr (MODE == kNpt) {
    const double w = warp_sum((double)wv);
    if (lane == 0) {
      D.vir[bead] = w;
      if (twin != bead) D.vir[twin] = w;
    }
  }
  return e + D.e_zero;
}

// The same in FP64 by a block of kTeam warps.  ws: the block's shared memory with
// the coordinates in place (a barrier follows here).  The energy is thread 0's.
template <int MODE = kFree>
__device__ inline double team_egrad(const Dev& D, double* ws, double* gout, double* gout2, size_t bead, size_t twin) {
  const int n3 = 3 * D.n, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  PBox tb;
  const PBox* box = launch_box<MODE>(D, bead, tb);
  double* g = ws + n3;
  double* buf = g + n3;
  double* red = buf + buffer_values(false) + 1;
  for (int a = tid; a < n3; a += kTeam * 32) g[a] = 0.0;
  if (tid == 0) buf[buffer_values(false)] = 0.0;
  __syncthreads();
  const BeadPos X{ws, nullptr, nullptr, box, MODE == kFree ? 0 : wrap_dims(ws, D.n, tb, lane)};
  double es = 0.0, wv = 0.0;
  kind_segments<0, MODE>(D, X, buf, g, es, wv);
  kind_segments<1, MODE>(D, X, buf, g, es, wv);
  kind_segments<2, MODE>(D, X, buf, g, es, wv);
  kind_segments<3, MODE>(D, X, buf, g, es, wv);
  kind_segments<4, MODE>(D, X, buf, g, es, wv);
  es = warp_sum(es);
  if constexpr (MODE == kNpt) wv = warp_sum(wv);
  if (lane == 0) {
    red[warp] = es;
    red[kTeam + warp] = wv;
  }
  __syncthreads();
  for (int a = tid; a < n3; a += kTeam * 32) {
    gout[a] = g[a];
    if (gout2 != gout) gout2[a] = g[a];
  }
  double e = 0.0, w = 0.0;
#pragma unroll
  for (int k = 0; k < kTeam; ++k) e += red[k];
  if constexpr (MODE == kNpt) {
#pragma unroll
    for (int k = 0; k < kTeam; ++k) w += red[kTeam + k];
    if (tid == 0) {
      D.vir[bead] = w;
      if (twin != bead) D.vir[twin] = w;
    }
  }
  return e + D.e_zero;
}

// ---------------------------------------------------------------------------
// Derivatives for the adjoint (plain form only; bonds, angles, torsions and
// NCI pairs).
// ---------------------------------------------------------------------------

// All segments of one term kind with dual coordinates: values in buf, tangents behind.
template <int KIND>
__device__ inline void kind_segments_dual(const Dev& D, const BeadPos& X, double* buf, double* g, double* h, Dual& es) {
  constexpr int B = buffer_values(false) + 1, C = segment_terms(false, KIND), NA = KIND == 1 ? 3 : KIND == 2 ? 4 : 1;
  const Schedule& S = D.sched[0];
  for (int sgi = S.seg0[KIND]; sgi < S.seg1[KIND]; ++sgi) {
    const int4 sg = __ldg(S.seg + sgi);
    for (int i = threadIdx.x; i < sg.y; i += blockDim.x) {
      const int m = sg.x + i;
      Contrib<Dual> c;
      if constexpr (KIND == 0) es += bond_plain<Dual>(D, D.d, X, m, c);
      else if constexpr (KIND == 1) es += angle_plain<Dual>(D, D.d, X, m, c);
      else if constexpr (KIND == 2) es += torsion_plain<Dual>(D, D.d, X, m, c);
      else es += pair_tangent(D, D.d, X, m, c);
#pragma unroll
      for (int a = 0; a < NA; ++a)
#pragma unroll
        for (int d = 0; d < 3; ++d) {
          buf[(3 * a + d) * C + i] = c.g[a][d].v;
          buf[B + (3 * a + d) * C + i] = c.g[a][d].d;
        }
    }
    __syncthreads();
    gather(S, sg, threadIdx.x >> 5, blockDim.x >> 5, threadIdx.x & 31, [&](int a, const unsigned short* l, int n) {
      double v = g[a], t = h[a];
#pragma unroll 4
      for (int j = 0; j < n; ++j) {
        const unsigned e = __ldg(l + 32 * j);
        v += signed_value(buf, e);
        t += signed_value(buf + B, e);
      }
      g[a] = v;
      h[a] = t;
    });
    __syncthreads();
  }
}

// Shared memory of team_hvp: x, w, gradient, H w (3n doubles each), the buffer and
// zero for values and tangents, the warps' energies and derivatives.
__host__ __device__ inline size_t team_hvp_smem_bytes(int n) {
  return ((size_t)3 * n * 4 + 2 * (buffer_values(false) + 1) + 2 * kTeam) * 8;
}

// Energy (with E_zero), gradient and Hessian-vector product H w of one bead
// by a block of up to kTeam warps.  ws: the block's shared memory holding x (3n
// doubles) then w (3n doubles; a barrier follows here).  gout, gout2, hout, hout2: the
// destinations (equal: one).  dew receives the directional derivative w . grad E.
__device__ inline double team_hvp(const Dev& D, double* ws, double* gout, double* gout2, double* hout, double* hout2,
                                  double& dew) {
  const int n3 = 3 * D.n, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  double* w = ws + n3;
  double* g = w + n3;
  double* h = g + n3;
  double* buf = h + n3;
  double* red = buf + 2 * (buffer_values(false) + 1);
  for (int a = tid; a < 2 * n3; a += blockDim.x) g[a] = 0.0;
  if (tid < 2) buf[tid * (buffer_values(false) + 1) + buffer_values(false)] = 0.0;
  __syncthreads();
  PBox tb;
  if (D.periodic) tb = D.box;
  const BeadPos X{ws, nullptr, w, D.periodic ? &tb : nullptr, 7};
  Dual es(0.0);
  kind_segments_dual<0>(D, X, buf, g, h, es);
  kind_segments_dual<1>(D, X, buf, g, h, es);
  kind_segments_dual<2>(D, X, buf, g, h, es);
  kind_segments_dual<3>(D, X, buf, g, h, es);
  const double e1 = warp_sum(es.v), d1 = warp_sum(es.d);
  if (lane == 0) {
    red[warp] = e1;
    red[kTeam + warp] = d1;
  }
  __syncthreads();
  for (int a = tid; a < n3; a += blockDim.x) {
    if (gout) gout[a] = gout2[a] = g[a];
    hout[a] = hout2[a] = h[a];
  }
  double e = 0.0;
  dew = 0.0;
  for (int k = 0; k < (int)(blockDim.x >> 5); ++k) {
    e += red[k];
    dew += red[kTeam + k];
  }
  return e + D.e_zero;
}

// Linear parameters of the force field (the loss gradients of the adjoint are
// taken with respect to these): bond force constant k, angle force
// constant k, torsion barrier V and the NCI pair's
// Coulomb product qq ( eps1 q_i q_j, or q_i q_j in the Zahn form).
// Every term is linear in its parameter, so d/dtheta_t (v . grad E) is v .
// grad E_t evaluated with theta_t = 1; the tables U hold the parameters with
// those entries set to 1 (the pairs need none: their Coulomb term alone).
// Per term, out receives alpha * (v . grad E_t|unit) + beta * E_t|unit; the block's
// threads take the terms of each kind in turn.
template <int KIND>
__device__ inline void team_vjp_kind(const Dev& D, const Tables<double>& U, const BeadPos& X, const double* vs,
                                     double alpha, double beta, double* out) {
  constexpr int NA = KIND == 1 ? 3 : KIND == 2 ? 4 : 2;
  for (int m = threadIdx.x; m < D.nterm[KIND]; m += blockDim.x) {
    Contrib<double> c;
    double e;
    if constexpr (KIND == 0) e = bond_plain<double>(D, U, X, m, c);
    else if constexpr (KIND == 1) e = angle_plain<double>(D, U, X, m, c);
    else e = torsion_plain<double>(D, U, X, m, c);
    double s = 0.0;
#pragma unroll
    for (int a = 0; a < NA; ++a)
#pragma unroll
      for (int d = 0; d < 3; ++d) s = fma(vs[3 * c.a[a] + d], c.g[a][d], s);
    out[KIND == 2 ? (int)__ldg(D.tors + m).w : m] = alpha * s + beta * e;
  }
}
// ... of the pairs: the Coulomb energy alone depends on qq
__device__ inline void team_vjp_pairs(const Dev& D, const BeadPos& X, const double* vs, double alpha, double beta,
                                      double* out) {
  for (int m = threadIdx.x; m < D.nterm[3]; m += blockDim.x) {
    const unsigned at = __ldg(D.pair + m);
    const int i1 = lo16(at), i2 = hi16(at);
    double vab[3], r, oner, s = 0.0, e = 0.0;
    disp<double>(X, i1, i2, vab);
    p_root(dot3(vab, vab), r, oner);
    if (!(r > D.coul_cut)) {
      e = pair_coulomb(D, r, oner);
#pragma unroll
      for (int d = 0; d < 3; ++d) s = fma(vab[d], vs[3 * i1 + d] - vs[3 * i2 + d], s);
      s = s * (-e * (oner * oner));
    }
    out[m] = alpha * s + beta * e;
  }
}
__device__ inline void team_param_vjp(const Dev& D, const Tables<double>& U, const double* xs, const double* vs,
                                      double alpha, double beta, double* out) {
  PBox tb;
  if (D.periodic) tb = D.box;
  const BeadPos X{xs, nullptr, nullptr, D.periodic ? &tb : nullptr, 7};
  team_vjp_kind<0>(D, U, X, vs, alpha, beta, out);
  out += D.nterm[0];
  team_vjp_kind<1>(D, U, X, vs, alpha, beta, out);
  out += D.nterm[1];
  team_vjp_kind<2>(D, U, X, vs, alpha, beta, out);
  out += D.nterm[2];
  team_vjp_pairs(D, X, vs, alpha, beta, out);
}

}  // namespace qmdff
}  // namespace cr
