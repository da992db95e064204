// Persistent RPMD step kernel: many trajectories, all steps of a run in one
// launch, every bead's q, p, f held in shared memory across steps.
//
// Drop-in for the per-step work of Caracal's `verlet` (src/verlet.f90:65-1308)
// on the gas-phase path: 1/2 kick, free ring-polymer propagation in Caracal's
// cosine "normal modes", forces, 1/2 kick, Andersen or PILE thermostat,
// NaN check, `transrot`.
//
// Distinct beads.  Caracal's modes C = sqrt(1/P) cos(2 pi j k/P) (src/rfft.f90,
// src/irfft.f90), a per-mode 2x2 rotation (src/verlet.f90:405-454) and C again
// give a linear map p' = K1 p + m K2 q, q' = K3 p / m + K1 q with
// K[j][l] = K[-j][l] = K[j][-l]: its output is the same for beads j and P - j,
// and it reads only the sums x_l + x_{P-l}.  From the first drift on, positions,
// gradients and momenta of the two agree, so the kernel carries the U = P/2 + 1
// distinct beads (all P where nm_mode 1 uses orthonormal modes): the starting
// state enters as its symmetric part and sums over beads weigh the pairs twice.
// What a thermostat's draw adds to the antisymmetric part of p the next drift
// removes, but a state between steps has it: p = s +- a, rounded. Each draw
// therefore goes on with the symmetric part of that state, (fl(s + a) + fl(s - a)) / 2,
// whether the run ends there or not, so that a run in pieces, or from a state that was
// saved and set again, is the run in one, bit for bit.
//
// Thread layout: a block holds one or several trajectories.  The surface takes
// four lanes per bead, in passes over the block's beads (XH4; H3 in small batches),
// or one thread per bead (thread b: bead b mod U of trajectory b / U), and every
// other stage is a set of tasks (coordinate rows, row pairs, elements, sums) shared
// by all threads of the block through shared memory, where q, p and the gradient
// stay during the run.  The state out of the registers leaves them to the surface.
//
// The linear maps run on the integer pipe (fixed_map.cuh; 32 and 64 beads:
// ring_fast.cuh).  For even P
// (M = P/2), C[M-r][k] = (-1)^k C[r][k], so with K = Ke + Ko split by mode
// parity, K[r] = Ke[r] + Ko[r] and K[M-r] = Ke[r] - Ko[r]; Ke is even and Ko
// odd under l -> M-l: one pass over x_l + x_{M-l} and x_l - x_{M-l} gives rows
// r and M - r together.
//
// PILE (new; Caracal has Andersen and Nose-Hoover only) uses the orthonormal
// real normal modes; O^T diag(c) O is circulant, so each half step is two
// length-P circular convolutions: p' = a * p + sqrt(mP/beta) b * eta, folded
// onto the distinct beads.
#pragma once
#include <cuda_runtime.h>

#include <type_traits>

#include "bead_rows.cuh"
#include "cr_common.cuh"
#include "fixed_map.cuh"
#include "num.cuh"
#include "ring_fast.cuh"

namespace cr {

constexpr int kMaxBeads = 128;
constexpr int kMaxAtoms = 7;

// BIMOLEC reaction coordinate of Caracal's recrossing (calc_xi mode 2,
// src/calc_xi.f90:63-279): xi = xi_ideal*s1 + (1-xi_ideal)*s0 with
// s1 = (r_break - break_ref) - (r_form - form_ref), s0 = R_inf - |COM2 - COM1|.
struct XiDev {
  int nreac1, reac1[8], nreac2, reac2[8];  // 0-based atoms
  int form0, form1, brk0, brk1;
  double form_ref, break_ref, r_inf, xi_ideal;
  double mreac1, mreac2;
  double w1[8], w2[8];  // mass / mreac of each reactant atom (the step kernel's xi)
};

template <int N>
__host__ __device__ inline double xi_bimolec(const XiDev& x, const double* c, const double* mass,
                                             double* dxi) {
  double Rf[3], Rb[3];
  for (int d = 0; d < 3; ++d) {
    Rf[d] = c[3 * x.form0 + d] - c[3 * x.form1 + d];
    Rb[d] = c[3 * x.brk0 + d] - c[3 * x.brk1 + d];
  }
  const double rf = sqrt(Rf[0] * Rf[0] + Rf[1] * Rf[1] + Rf[2] * Rf[2]);
  const double rb = sqrt(Rb[0] * Rb[0] + Rb[1] * Rb[1] + Rb[2] * Rb[2]);
  const double s1 = (rb - x.break_ref) - (rf - x.form_ref);
  double c1[3] = {0, 0, 0}, c2[3] = {0, 0, 0};
  for (int k = 0; k < x.nreac1; ++k)
    for (int d = 0; d < 3; ++d) c1[d] += mass[x.reac1[k]] * c[3 * x.reac1[k] + d] / x.mreac1;
  for (int k = 0; k < x.nreac2; ++k)
    for (int d = 0; d < 3; ++d) c2[d] += mass[x.reac2[k]] * c[3 * x.reac2[k] + d] / x.mreac2;
  const double Red[3] = {c2[0] - c1[0], c2[1] - c1[1], c2[2] - c1[2]};
  const double reds = sqrt(Red[0] * Red[0] + Red[1] * Red[1] + Red[2] * Red[2]);
  const double s0 = x.r_inf - reds;
  if (dxi) {
    const double a = x.xi_ideal, b = 1.0 - x.xi_ideal;
    for (int i = 0; i < 3 * N; ++i) dxi[i] = 0.0;
    for (int d = 0; d < 3; ++d) {
      dxi[3 * x.form0 + d] -= a * Rf[d] / rf;
      dxi[3 * x.form1 + d] += a * Rf[d] / rf;
      dxi[3 * x.brk0 + d] += a * Rb[d] / rb;
      dxi[3 * x.brk1 + d] -= a * Rb[d] / rb;
    }
    for (int k = 0; k < x.nreac1; ++k)
      for (int d = 0; d < 3; ++d) dxi[3 * x.reac1[k] + d] += b * Red[d] / reds * mass[x.reac1[k]] / x.mreac1;
    for (int k = 0; k < x.nreac2; ++k)
      for (int d = 0; d < 3; ++d) dxi[3 * x.reac2[k] + d] -= b * Red[d] / reds * mass[x.reac2[k]] / x.mreac2;
  }
  return x.xi_ideal * s1 + (1.0 - x.xi_ideal) * s0;
}

// xi alone (no derivative) for the side bit of a recrossing child: the same
// formula as xi_bimolec with the reactant weights m / m_reac precomputed, so
// the COMs cost multiplications only (FP64 divisions take ~10 FP64-pipe
// instructions each on this GPU).
template <int N>
__device__ inline double xi_bimolec_value(const XiDev& x, const double* c) {
  double Rf[3], Rb[3], c1[3] = {0, 0, 0}, c2[3] = {0, 0, 0};
  for (int d = 0; d < 3; ++d) {
    Rf[d] = c[3 * x.form0 + d] - c[3 * x.form1 + d];
    Rb[d] = c[3 * x.brk0 + d] - c[3 * x.brk1 + d];
  }
  for (int k = 0; k < x.nreac1; ++k)
    for (int d = 0; d < 3; ++d) c1[d] = fma(x.w1[k], c[3 * x.reac1[k] + d], c1[d]);
  for (int k = 0; k < x.nreac2; ++k)
    for (int d = 0; d < 3; ++d) c2[d] = fma(x.w2[k], c[3 * x.reac2[k] + d], c2[d]);
  const double Red[3] = {c2[0] - c1[0], c2[1] - c1[1], c2[2] - c1[2]};
  const double rf = fx::sqrt(Rf[0] * Rf[0] + Rf[1] * Rf[1] + Rf[2] * Rf[2]);
  const double rb = fx::sqrt(Rb[0] * Rb[0] + Rb[1] * Rb[1] + Rb[2] * Rb[2]);
  const double reds = fx::sqrt(Red[0] * Red[0] + Red[1] * Red[1] + Red[2] * Red[2]);
  const double s1 = (rb - x.break_ref) - (rf - x.form_ref);
  return x.xi_ideal * s1 + (1.0 - x.xi_ideal) * (x.r_inf - reds);
}

// Shape of the parity-split propagator blocks for P beads.
struct PropDims {
  int M;      // P / 2
  int split;  // 1: even P, parity-split blocks; 0: odd P, unique rows only
  int nr;     // task rows
  int nu;     // length of u (even part)
  int nv;     // length of v (odd part)
  int su, sv; // padded (odd) shared-memory strides of u and v
};

__host__ __device__ inline PropDims prop_dims(int P) {
  PropDims d;
  d.M = P / 2;
  d.split = (P % 2 == 0) ? 1 : 0;
  if (d.split) {
    d.nr = d.M / 2 + 1;
    d.nu = d.M / 2 + 1;
    d.nv = d.M - d.M / 2;
  } else {
    d.nr = P / 2 + 1;
    d.nu = d.nr;
    d.nv = 0;
  }
  d.su = d.nu | 1;
  d.sv = d.nv > 0 ? (d.nv | 1) : 0;
  return d;
}

__device__ inline double sym_at(const double* x, int l, int P) {
  return (l == 0 || 2 * l == P) ? x[l] : x[l] + x[P - l];
}

// Nose-Hoover chain constants of one engine (src/nhc.f90:35-171 with the
// masses of src/mdinit.f90:128-147), precomputed on the host.
struct NhcParams {
  double ekt;     // nhc's kT: the REAL(4) quotient 1.380649E-23/4.3597447E-18 times kelvin
  double qnh[4];  // chain masses: 3N Q, Q, Q, Q with Q = k_B T nose_q^2
  double dtc;     // dt / nc
  double w[3];    // Suzuki-Yoshida weights
  int nfree;      // 3N
};

// One nhc call on a trajectory whose kinetic sum (centroid-normalised, as
// Caracal: sum p.p/(2m)/P/P) is eksum: advances the chain velocities vnh and
// returns the factor every momentum is scaled by.  Same operation order as
// the reference loop (nc = 5 passes of ns = 3 weights).  One thread's chain of 105
// exponentials and 120 divisions is most of a Nose-Hoover step of a small batch: on the
// integer pipe (fx64.cuh) H3 1000 x 32 mixed 450 -> 333 us per step.
__device__ inline double nhc_scale(const NhcParams& c, double eksum, double (&vnh)[4]) {
  double gnh[4];
  double scale = 1.0;
  for (int ic = 0; ic < 5; ++ic)
    for (int j = 0; j < 3; ++j) {
      const double dts = c.w[j] * c.dtc;
      const double dt2 = 0.5 * dts, dt4 = 0.25 * dts, dt8 = 0.125 * dts;
      double ex;
      gnh[3] = fx::div(c.qnh[2] * vnh[2] * vnh[2] - c.ekt, c.qnh[3]);
      vnh[3] = vnh[3] + gnh[3] * dt4;
      gnh[2] = fx::div(c.qnh[1] * vnh[1] * vnh[1] - c.ekt, c.qnh[2]);
      ex = fx::exp(-vnh[3] * dt8);
      vnh[2] = ex * (vnh[2] * ex + gnh[2] * dt4);
      gnh[1] = fx::div(c.qnh[0] * vnh[0] * vnh[0] - c.ekt, c.qnh[1]);
      ex = fx::exp(-vnh[2] * dt8);
      vnh[1] = ex * (vnh[1] * ex + gnh[1] * dt4);
      gnh[0] = fx::div(2.0 * eksum - (double)c.nfree * c.ekt, c.qnh[0]);
      ex = fx::exp(-vnh[1] * dt8);
      vnh[0] = ex * (vnh[0] * ex + gnh[0] * dt4);
      ex = fx::exp(-vnh[0] * dt2);
      scale = scale * ex;
      eksum = eksum * ex * ex;
      gnh[0] = fx::div(2.0 * eksum - (double)c.nfree * c.ekt, c.qnh[0]);
      ex = fx::exp(-vnh[1] * dt8);
      vnh[0] = ex * (vnh[0] * ex + gnh[0] * dt4);
      gnh[1] = fx::div(c.qnh[0] * vnh[0] * vnh[0] - c.ekt, c.qnh[1]);
      ex = fx::exp(-vnh[2] * dt8);
      vnh[1] = ex * (vnh[1] * ex + gnh[1] * dt4);
      gnh[2] = fx::div(c.qnh[1] * vnh[1] * vnh[1] - c.ekt, c.qnh[2]);
      ex = fx::exp(-vnh[3] * dt8);
      vnh[2] = ex * (vnh[2] * ex + gnh[2] * dt4);
      gnh[3] = fx::div(c.qnh[2] * vnh[2] * vnh[2] - c.ekt, c.qnh[3]);
      vnh[3] = vnh[3] + gnh[3] * dt4;
    }
  return scale;
}

// Umbrella windows (verlet with constrain = 0, src/umbrella.f90 mode 0).
struct UmbrellaDev {
  const double* center;  // [T] xi of each trajectory's window
  const double* kforce;  // [T] force constant (Eh)
  double beta;           // 1 / (k_B T) of the fs term
  double R[6];           // upper triangle (row by row) of R with R^T R = J M^-1 J^T of xi's three vectors
  const int* sampling;   // device flag: 1 while the statistics are collected
  double* xsum;          // [T] sum of xi over the sampled steps
  double* xsum2;         // [T] sum of xi^2
  int nbins;             // histogram of xi over [lo, hi) (0: none)
  double lo, hi;
  double* hist;          // [T][nbins]
};

struct StepParams {
  int T;           // trajectories in the launch
  int P;           // beads
  int U;           // beads carried: P/2 + 1 distinct ones, or all P (nm_mode 1)
  int pair;        // 1: bead j stands for j and P - j too
  int gpb;         // trajectories per block
  int subs;        // threads per carried bead
  int quad;        // the surface by four lanes per bead where it has that form (PES::kQuad)
  int thermostat;  // CR_THERMO_*
  int andersen_step;
  int transrot;
  uint32_t seed;
  uint32_t traj0;  // global index of trajectory 0 (noise key)
  double dt;
  double half_dt;
  double beta;
  double itm, kap; // transrot: 1/M and 2/M - W/M^2 of Caracal's total mass M = P^2 sum m and W = P sum m
  double mass[kMaxAtoms];
  double inv_mass[kMaxAtoms];
  double sigma[kMaxAtoms];    // sqrt(m P / beta): Andersen / PILE noise scale
  PropDims pd;
  const Limbs* ke;     // [3][nr][nu]: K1, K2, K3 (unit mass) on folded rows, even-mode part (odd P: all modes)
  const Limbs* ko;     // [3][nr][nv]: odd-mode part
  int ek[3];           // their exponents
  int guard;           // guard bits of the folded rows (fixed_map.cuh)
  int fast_M;          // P / 2 where the free ring polymer takes the fast transforms (ring_fast.cuh), else 0
  FastRing fast;
  const Limbs* pile;   // pairs: [2][U][U] friction and noise maps on the carried beads, [w][l][j], and [h][U] the noise map
                       // of the antisymmetric part on beads 1 .. h = (P - 1) / 2, [l - 1][j]; else the circulants [2][P]
  int ep[3];           // their exponents
  int pguard;
  NhcParams nhc;
  double* vnh;         // [T][4] Nose-Hoover chain velocities
  double* q;           // [T][P][N][3]
  double* p;
  double* f;
  double* anti;        // scratch [T][2][N][3][U]: limbs of the deviates' antisymmetric part, and its share of p (NULL: no draws
                       // or no pairs)
  int anti_smem;       // 1: the same in the block's shared memory
  double* epot;        // [T]
  int* status;         // [T]
  // recrossing children: after each step, side[t*side_stride + istep-side_step0-1]
  // records xi(centroid) > 0 (src/recross.f90:596-602)
  int xi_on;
  int side_step0;
  int side_stride;
  unsigned char* side;
  XiDev xi;
  // umbrella windows: bias towards the trajectory's window after the forces
  int umb_on;
  UmbrellaDev umb;
  // step counter on the device (a launch replayed from a CUDA graph reads its
  // first step index here); NULL: the launch argument
  const int* istep_dev;
  double inv_P;
  // nm_mode 1 (orthonormal normal modes): K1, K2, K3 are circulant, row j
  // holds circ[w][(j - l) mod P] (unit mass)
  int nm_mode;
  const Limbs* circ;  // [3][P], under the exponents ek
};

// Non-finite test on the exponent bits (integer pipe, no FP64 compare).
__device__ inline bool nonfinite_bits(double x) { return (__double2hiint(x) & 0x7ff00000) == 0x7ff00000; }

__device__ __forceinline__ Limbs ldg_limbs(const Limbs* p) {
  const int2 v = __ldg(reinterpret_cast<const int2*>(p));
  return Limbs{v.x, v.y};
}

// Umbrella bias at the centroid c (src/umbrella.f90:100-176, mode 0): the
// gradient of 1/2 k (xi - xi0)^2 - (1/beta) log fs with xi = s0 / (s0 - s1)
// (calc_xi mode 1, src/calc_xi.f90:63-279) and fs^2 = sum dxi^2/m / (2 pi beta),
// i.e. k (xi - xi0) dxi - H(dxi/m) / (beta sum dxi^2/m), into bias.  xi depends
// on c through three vectors J c only (forming bond, breaking bond, distance of
// the reactants) with unit vectors n: dxi = J^T b with b along n, its changes
// along dxi/m are u = J M^-1 J^T b = R^T R b and t = (u - n (n.u)) / r for n, and
// sum dxi^2/m = |R b|^2, so that atoms come in at the start and the end alone.
// Four lanes (lane = 0..3, all of an aligned quad) for a trajectory, three of them a
// component each: a chain of some 85 FP64 operations where one thread over the atoms
// had 250.  H3 1100 x 16 plain: 77.8 -> 72.9 us per step.
// Returns xi.
template <int N>
__device__ inline double umbrella_bias(const XiDev& x, const UmbrellaDev& w, const double* c, double center,
                                       double kforce, int lane, double* bias) {
  const int d = min(lane, 2);
  const unsigned mask = 0xfu << (threadIdx.x & 28);
  auto sum3 = [&](double y) {
    const double y0 = __shfl_sync(mask, y, 0, 4), y1 = __shfl_sync(mask, y, 1, 4), y2 = __shfl_sync(mask, y, 2, 4);
    return y0 + y1 + y2;
  };
  // n[0] forming bond, n[1] breaking bond, n[2] second reactant - first
  double n[3], r[3], ir[3];
  n[0] = c[3 * x.form0 + d] - c[3 * x.form1 + d];
  n[1] = c[3 * x.brk0 + d] - c[3 * x.brk1 + d];
  n[2] = 0.0;
  for (int i = 0; i < x.nreac2; ++i) n[2] = fma(x.w2[i], c[3 * x.reac2[i] + d], n[2]);
  for (int i = 0; i < x.nreac1; ++i) n[2] = fma(-x.w1[i], c[3 * x.reac1[i] + d], n[2]);
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    fx::sqrt_rsqrt(sum3(n[k] * n[k]), r[k], ir[k]);
    n[k] *= ir[k];
  }
  const double s1 = (r[1] - x.break_ref) - (r[0] - x.form_ref), s0 = x.r_inf - r[2];
  const double iD = fx::rcp(s0 - s1), iD2 = iD * iD;
  // dxi = s0/D^2 (n_b - n_f) + s1/D^2 n_e on the vectors' atoms
  const double a0 = s0 * iD2, a1 = s1 * iD2;
  const double b[3] = {-a0 * n[0], a0 * n[1], a1 * n[2]};
  const double y0 = fma(w.R[0], b[0], fma(w.R[1], b[1], w.R[2] * b[2])), y1 = fma(w.R[3], b[1], w.R[4] * b[2]),
               y2 = w.R[5] * b[2];
  const double fs = sum3(fma(y0, y0, fma(y1, y1, y2 * y2)));
  // along dxi / m: the vectors' changes, r' = n.u, n' = t
  const double u[3] = {w.R[0] * y0, fma(w.R[1], y0, w.R[3] * y1), fma(w.R[2], y0, fma(w.R[4], y1, w.R[5] * y2))};
  double rp[3], t[3];
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    rp[k] = sum3(n[k] * u[k]);
    t[k] = (u[k] - n[k] * rp[k]) * ir[k];
  }
  const double s1p = rp[1] - rp[0], s0p = -rp[2], Dp = s0p - s1p;
  const double coef = -fx::rcp(w.beta * fs);
  const double h0 = coef * iD2 * s0p, h1 = coef * iD2 * s0, e0 = coef * iD2 * s1p, e1 = coef * iD2 * s1;
  const double xi = s0 * iD, kd = kforce * (xi - center) - 2.0 * coef * Dp * iD;
  const double g0 = fma(kd, b[0], -(h0 * n[0] + h1 * t[0])), g1 = fma(kd, b[1], h0 * n[1] + h1 * t[1]),
               g2 = fma(kd, b[2], e0 * n[2] + e1 * t[2]);
  if (lane < 3) {
    for (int i = 0; i < N; ++i) bias[3 * i + d] = 0.0;
    for (int i = 0; i < x.nreac2; ++i) bias[3 * x.reac2[i] + d] = fma(x.w2[i], g2, bias[3 * x.reac2[i] + d]);
    for (int i = 0; i < x.nreac1; ++i) bias[3 * x.reac1[i] + d] = fma(-x.w1[i], g2, bias[3 * x.reac1[i] + d]);
    bias[3 * x.form0 + d] += g0;
    bias[3 * x.form1 + d] -= g0;
    bias[3 * x.brk0 + d] += g1;
    bias[3 * x.brk1 + d] -= g1;
  }
  return xi;
}

// Sampling statistics of one trajectory's xi.
__device__ inline void umbrella_sample(const UmbrellaDev& u, size_t t, double xi) {
  u.xsum[t] = u.xsum[t] + xi;
  u.xsum2[t] = u.xsum2[t] + xi * xi;
  if (u.nbins > 0) {
    const double y = (xi - u.lo) / (u.hi - u.lo) * u.nbins;
    if (y >= 0.0 && y < u.nbins) u.hist[t * u.nbins + (int)y] += 1.0;
  }
}

// The windows' bias in a step: centroids into cen, the bias behind them, added to
// every carried bead's gradient.  Out of line: code that few runs take stays out of
// the step's loop.
template <int N, class Sum>
__device__ __noinline__ void umbrella_step(const XiDev& x, const UmbrellaDev& w, Sum bead_sum, const double* sq, double* sf,
                                           double* cen, int t_first, int ng, int U, double inv_P) {
  constexpr int NC = 3 * N;
  const int tid = threadIdx.x, nth = blockDim.x, rows = ng * NC;
  double* bias = cen + rows;
  for (int y = tid; y < rows; y += nth) cen[y] = bead_sum(sq + y * U) * inv_P;
  __syncthreads();
#pragma unroll 1
  for (int y = tid; y < 4 * ng; y += nth) {
    const int g = y >> 2, t = t_first + g;
    const double xi = umbrella_bias<N>(x, w, cen + g * NC, w.center[t], w.kforce[t], y & 3, bias + g * NC);
    if ((y & 3) == 0 && *w.sampling) umbrella_sample(w, (size_t)t, xi);
  }
  __syncthreads();
  for (int y = tid; y < rows * U; y += nth) sf[y] += bias[y / U];
}

// The largest exponent field of a row.
__device__ __forceinline__ int row_exponent(const double* r, int U) {
  int e = 0;
#pragma unroll 4
  for (int l = 0; l < U; ++l) e = max(e, exponent_field(r[l]));
  return e;
}

// Bead sums of one atom's rows (row0 .. row0 + 2 of q and of p) in fixed point:
// v = 0..2 p, 3..5 q, 6..11 q_a p_b for (a, b) = (y z), (z y), (z x), (x z), (x y),
// (y x), 12..17 q_a q_b for xx, xy, xz, yy, yz, zz.  pair: interior beads count
// twice.
constexpr int kMoments = 18;
__device__ inline double atom_moment(const Limbs* q, const Limbs* p, const int* eq, const int* ep, int row0, int v, int U,
                                     int P, int pair, int guard) {
  const int ends = pair && U > 1 && (P & 1) == 0 ? U - 1 : 0;  // the last bead that counts once
  const int in = pair ? (P - 1) / 2 : U - 1;                     // beads 1 .. in, then `ends`
  int ex;
  int64_t s;
  bool bad;
  if (v < 6) {
    const int r = row0 + v % 3;
    const Limbs* x = (v < 3 ? p : q) + r * U;
    auto at = [&](int l) { return ((int64_t)x[l].hi << kLimbBits) + x[l].lo; };
    int64_t a = 0;
    for (int l = 1; l <= in; ++l) a += at(l);
    s = (pair ? 2 * a : a) + at(0) + (ends ? at(ends) : 0);
    const int e = (v < 3 ? ep : eq)[r];
    bad = e == kFixedNan;
    ex = e - 1078 + guard;
  } else {
    const int a = v < 12 ? (v == 6 || v == 11 ? 1 : v == 7 || v == 8 ? 2 : 0) : (v < 15 ? 0 : v < 17 ? 1 : 2);
    const int b = v < 12 ? (v == 6 || v == 9 ? 2 : v == 7 || v == 10 ? 1 : 0)
                         : (v == 12 ? 0 : v == 13 || v == 15 ? 1 : 2);
    const Limbs* x = q + (row0 + a) * U;
    const Limbs* y = (v < 12 ? p : q) + (row0 + b) * U;
    FixedSum m{0, 0}, o{0, 0};
#pragma unroll 4
    for (int l = 1; l <= in; ++l) m.add(x[l], y[l]);
    o.add(x[0], y[0]);
    if (ends) o.add(x[ends], y[ends]);
    s = (pair ? 2 * m.value() : m.value()) + o.value();
    const int ea = eq[row0 + a], eb = (v < 12 ? ep : eq)[row0 + b];
    bad = ea == kFixedNan || eb == kFixedNan;
    ex = ea + eb + 2 * (guard - 1078) + 2 * kLimbBits;
  }
  const double r = from_fixed(s, ex);
  return bad ? __longlong_as_double(0x7ff8000000000000ll) : r;
}

// transrot's move from the moment sums over beads and atoms (sum p; sum m x; x
// cross p; sum m x x^T as xx, xy, xz, yy, yz, zz), lanes 0, 1, 2 of a quad forming
// component d each: p <- p - m (b + va cross x).  With S = sum m x, M Caracal's
// total mass and W = sum m, the centre S/M gives the centred moments S_ab -
// kap S_a S_b, kap = 2/M - W/M^2, and the angular momentum L - S x (sum p) / M.  The inertia
// tensor is symmetric and positive, so pivots are taken on the diagonal (the
// reference inverts it with full pivoting): for a nearly linear molecule the last
// pivot is small, and what it divides turns the molecule about its own axis.
// tot(k): moment sum k; two_atoms: the reference's 1e-6 on the diagonal.  false:
// singular.
template <class Tot>
__device__ inline bool transrot_quad(Tot tot, int lane, double itm, double kap, bool two_atoms, double& bb, double& va) {
  const int d = lane < 3 ? lane : 0, e = d == 2 ? 0 : d + 1, f = d == 0 ? 2 : d - 1;
  const double Sd = tot(3 + d), Se = tot(3 + e), Sf = tot(3 + f);
  // centred second moments: dd and the product of the other two axes
  const int dd = d == 0 ? 9 : d == 1 ? 12 : 14, ef = d == 0 ? 13 : d == 1 ? 11 : 10;
  const double cdd = fma(-kap * Sd, Sd, tot(dd)), cef = fma(-kap * Se, Sf, tot(ef));
  const double L = fma(-itm, fma(Se, tot(f), -Sf * tot(e)), tot(6 + d));
  auto at = [](double x, int src) { return __shfl_sync(0xffffffffu, x, src, 4); };
  const double tdd = at(cdd, e) + at(cdd, f) + (two_atoms ? 0.000001 : 0.0);
  // first pivot: the largest of the diagonal (non-negative: the bits order them)
  auto bits = [](double x) { return __double_as_longlong(fabs(x)); };
  const double t0 = at(tdd, 0), t1 = at(tdd, 1), t2 = at(tdd, 2);
  const int p = bits(t0) >= bits(t1) ? (bits(t0) >= bits(t2) ? 0 : 2) : (bits(t1) >= bits(t2) ? 1 : 2);
  const int q = p == 2 ? 0 : p + 1, r = p == 0 ? 2 : p - 1;
  const double tpp = at(tdd, p), tqq = at(tdd, q), trr = at(tdd, r);
  const double tpq = -at(cef, r), tpr = -at(cef, q), tqr = -at(cef, p);
  const double Lp = at(L, p), Lq = at(L, q), Lr = at(L, r);
  const double ip = fx::rcp(tpp), a = tpq * ip, b = tpr * ip;
  const double sqq = fma(-a, tpq, tqq), srr = fma(-b, tpr, trr), sqr = fma(-a, tpr, tqr);
  const double yq = fma(-a, Lp, Lq), yr = fma(-b, Lp, Lr);
  const bool swap = bits(srr) > bits(sqq);
  const double s1 = swap ? srr : sqq, s2 = swap ? sqq : srr, y1 = swap ? yr : yq, y2 = swap ? yq : yr;
  const double i1 = fx::rcp(s1), c = sqr * i1;
  const double s3 = fma(-c, sqr, s2), v2 = fma(-c, y1, y2) * fx::rcp(s3), v1 = fma(-sqr, v2, y1) * i1;
  const double vq = swap ? v2 : v1, vr = swap ? v1 : v2;
  const double vp = fma(-tpr, vr, fma(-tpq, vq, Lp)) * ip;
  auto comp = [&](int x) { return x == p ? vp : x == q ? vq : vr; };
  va = comp(d);
  bb = fma(-comp(e), Sf, fma(comp(f), Se, tot(d))) * itm;
  return tpp != 0.0 && s1 != 0.0 && s3 != 0.0;
}

// The solve of transrot_quad by one thread, operation for operation: va = T^-1 L for the
// tensor with centred moments c (xx, yy, zz, yz, zx, xy).  false: singular.
__device__ inline bool transrot_solve(const double (&c)[6], const double (&L)[3], bool two_atoms, double (&va)[3]) {
  const double small = two_atoms ? 0.000001 : 0.0;
  const double t0 = c[1] + c[2] + small, t1 = c[2] + c[0] + small, t2 = c[0] + c[1] + small;
  auto bits = [](double x) { return __double_as_longlong(fabs(x)); };
  auto from = [](int k, double u, double v, double w) { return k == 0 ? u : k == 1 ? v : w; };
  const int p = bits(t0) >= bits(t1) ? (bits(t0) >= bits(t2) ? 0 : 2) : (bits(t1) >= bits(t2) ? 1 : 2);
  const int q = p == 2 ? 0 : p + 1, r = p == 0 ? 2 : p - 1;
  const double tpp = from(p, t0, t1, t2), tqq = from(q, t0, t1, t2), trr = from(r, t0, t1, t2);
  const double tqr = -from(p, c[3], c[4], c[5]), tpr = -from(q, c[3], c[4], c[5]), tpq = -from(r, c[3], c[4], c[5]);
  const double Lp = from(p, L[0], L[1], L[2]), Lq = from(q, L[0], L[1], L[2]), Lr = from(r, L[0], L[1], L[2]);
  const double ip = fx::rcp(tpp), a = tpq * ip, b = tpr * ip;
  const double sqq = fma(-a, tpq, tqq), srr = fma(-b, tpr, trr), sqr = fma(-a, tpr, tqr);
  const double yq = fma(-a, Lp, Lq), yr = fma(-b, Lp, Lr);
  const bool swap = bits(srr) > bits(sqq);
  const double s1 = swap ? srr : sqq, s2 = swap ? sqq : srr, y1 = swap ? yr : yq, y2 = swap ? yq : yr;
  const double i1 = fx::rcp(s1), m = sqr * i1, s3 = fma(-m, sqr, s2);
  const double v2 = fma(-m, y1, y2) * fx::rcp(s3), v1 = fma(-sqr, v2, y1) * i1;
  const double vq = swap ? v2 : v1, vr = swap ? v1 : v2, vp = fma(-tpr, vr, fma(-tpq, vq, Lp)) * ip;
  // axis 0 is p, r or q as p is 0, 1 or 2, and so on round
  va[0] = from(p, vp, vr, vq);
  va[1] = from(p, vq, vp, vr);
  va[2] = from(p, vr, vq, vp);
  return tpp != 0.0 && s1 != 0.0 && s3 != 0.0;
}

// transrot of ring polymers of one or two carried beads (rows q, p of NC x U in shared
// memory, bead 1 of three standing for two): the reference's sums over atoms and beads
// about its centre (src/transrot.f90:36-237) in FP64, by L = 4 lanes per trajectory, each
// with the atoms i = lane, lane + 4, or by one thread that goes through the four lanes'
// sums, with the same roundings (num.cuh). One thread per trajectory has the least
// operations, some 40 per atom and 80 for the solve; four are faster where a block
// has the threads to spare. The moments by limbs take 18 tasks of a hundred
// instructions per atom whatever the number of beads, and with one bead about the origin
// lose (R/r)^2 of the precision of a molecule at R. Per step, limbs and here: H3 100 000 x 1
// mixed 267 and 116 us, plain 387 and 239; CH4 + H 60 000 x 1 mixed 256 and 168; H3 1 x 1 11.9 and 12.8.
template <int N, int L>
__device__ __noinline__ void transrot_few(const StepParams& prm, const double* sq, double* sp, int ng, int* sstat) {
  using D = Num<double>;
  constexpr int NC = 3 * N;
  const int tid = threadIdx.x, nth = blockDim.x, U = prm.U, P = prm.P, lane = L == 4 ? tid & 3 : 0;
  const bool twins = prm.pair && P == 3;  // bead 1 stands for beads 1 and 2
  const D itm = prm.itm;
  // of the four lanes' values, in one order
  auto total = [&](auto part) {
    if constexpr (L == 4) {
      D x = part(lane);
      x = x + D(__shfl_xor_sync(0xffffffffu, x.v, 1));
      return x + D(__shfl_xor_sync(0xffffffffu, x.v, 2));
    } else {
      const D lo = N > 1 ? part(0) + part(1) : part(0);
      return N > 3 ? lo + (part(2) + part(3)) : N > 2 ? lo + part(2) : lo;
    }
  };
  for (int x0 = 0; x0 < ng; x0 += nth / L) {
    if (x0 + (tid & ~31) / L >= ng) break;  // a warp's shuffles want all of it
    const int gg = x0 + tid / L;
    const bool real = gg < ng;
    const double* q = sq + (real ? gg : x0) * NC * U;
    double* p = sp + (real ? gg : x0) * NC * U;
    struct First {
      D P[3], S[3], M[3];
    } first[L == 4 ? 1 : 4];
    auto sums = [&](int v, First& f) {
#pragma unroll
      for (int d = 0; d < 3; ++d) f.P[d] = f.S[d] = f.M[d] = D(0.0);
#pragma unroll
      for (int i = v; i < N; i += 4)
        for (int j = 0; j < U; ++j) {
          const D k = twins && j == 1 ? 2.0 : 1.0, w = k * D(prm.mass[i]);
          D x[3], y[3];
#pragma unroll
          for (int d = 0; d < 3; ++d) {
            x[d] = q[(3 * i + d) * U + j];
            y[d] = k * D(p[(3 * i + d) * U + j]);
            f.P[d] = f.P[d] + y[d];
            f.S[d] = w * x[d] + f.S[d];
          }
#pragma unroll
          for (int d = 0; d < 3; ++d) {
            const int e = d == 2 ? 0 : d + 1, g = d == 0 ? 2 : d - 1;
            f.M[d] = x[e] * y[g] + f.M[d];
            f.M[d] = f.M[d] - x[g] * y[e];
          }
        }
    };
    if constexpr (L == 4) {
      sums(lane, first[0]);
    } else {
#pragma unroll
      for (int v = 0; v < 4; ++v) sums(v, first[v]);
    }
    D Pt[3], xt[3], Lt[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      Pt[d] = total([&](int v) { return first[L == 4 ? 0 : v].P[d]; });
      xt[d] = total([&](int v) { return first[L == 4 ? 0 : v].S[d]; }) * itm;
      Lt[d] = total([&](int v) { return first[L == 4 ? 0 : v].M[d]; });
    }
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      const int e = d == 2 ? 0 : d + 1, g = d == 0 ? 2 : d - 1;
      Lt[d] = Lt[d] - xt[e] * Pt[g];
      Lt[d] = xt[g] * Pt[e] + Lt[d];
    }
    struct Second {
      D c[6];  // xx, yy, zz, yz, zx, xy
    } second[L == 4 ? 1 : 4];
    auto squares = [&](int v, Second& f) {
#pragma unroll
      for (int k = 0; k < 6; ++k) f.c[k] = D(0.0);
#pragma unroll
      for (int i = v; i < N; i += 4)
        for (int j = 0; j < U; ++j) {
          const D w = D(twins && j == 1 ? 2.0 : 1.0) * D(prm.mass[i]);
          D x[3], wx[3];
#pragma unroll
          for (int d = 0; d < 3; ++d) {
            x[d] = D(q[(3 * i + d) * U + j]) - xt[d];
            wx[d] = w * x[d];
            f.c[d] = wx[d] * x[d] + f.c[d];
          }
#pragma unroll
          for (int d = 0; d < 3; ++d) {
            const int e = d == 2 ? 0 : d + 1, g = d == 0 ? 2 : d - 1;
            f.c[3 + d] = wx[e] * x[g] + f.c[3 + d];
          }
        }
    };
    if constexpr (L == 4) {
      squares(lane, second[0]);
    } else {
#pragma unroll
      for (int v = 0; v < 4; ++v) squares(v, second[v]);
    }
    double c[6];
#pragma unroll
    for (int k = 0; k < 6; ++k) c[k] = total([&](int v) { return second[L == 4 ? 0 : v].c[k]; }).v;
    // the move vt + va x (x - xt)
    D vt[3], va[3];
    bool ok;
    if constexpr (L == 4) {
      // transrot_quad with the first moments taken out (kap = 0)
      auto tot = [&](int k) {
        double r = 0.0;
#pragma unroll
        for (int d = 0; d < 3; ++d) r = k == d ? Pt[d].v : k == 6 + d ? Lt[d].v : r;
        // xx, xy, xz, yy, yz, zz
        return k == 9 ? c[0] : k == 10 ? c[5] : k == 11 ? c[4] : k == 12 ? c[1] : k == 13 ? c[3] : k == 14 ? c[2] : r;
      };
      double b, w;
      ok = transrot_quad(tot, lane, itm.v, 0.0, N <= 2, b, w);
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        vt[d] = D(__shfl_sync(0xffffffffu, b, d, 4));
        va[d] = D(__shfl_sync(0xffffffffu, w, d, 4));
      }
    } else {
      const double Lv[3] = {Lt[0].v, Lt[1].v, Lt[2].v};
      double w[3];
      ok = transrot_solve(c, Lv, N <= 2, w);
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        vt[d] = Pt[d] * itm;
        va[d] = D(w[d]);
      }
    }
    if (!real) continue;
    if (!ok) {
      if (lane == 0) atomicOr(&sstat[gg], CR_TRAJ_SINGULAR_INERTIA);
      continue;
    }
    for (int v = lane; v < 4; v += L)
#pragma unroll
      for (int i = v; i < N; i += 4)
        for (int j = 0; j < U; ++j) {
          D x[3];
#pragma unroll
          for (int d = 0; d < 3; ++d) x[d] = D(q[(3 * i + d) * U + j]) - xt[d];
#pragma unroll
          for (int d = 0; d < 3; ++d) {
            const int e = d == 2 ? 0 : d + 1, g = d == 0 ? 2 : d - 1;
            const D u = va[e] * x[g] + (vt[d] - va[g] * x[e]);
            p[(3 * i + d) * U + j] = (double)(D(p[(3 * i + d) * U + j]) - D(prm.mass[i]) * u);
          }
        }
  }
}

// x[k] of an array in registers
__device__ __forceinline__ double pick(const double (&x)[16], int k) {
  double r = x[0];
#pragma unroll
  for (int j = 1; j < 16; ++j) r = k == j ? x[j] : r;
  return r;
}

// Dynamic shared memory: the propagator's limbs (3 nr (nu + nv)), then for the
// gpb trajectories of the block, each array over all of them:
//   q, p, f   [NC][U] doubles
//   area      [2 NC][U]: limbs of the folded rows, PILE limbs, partial sums; anti: two more [NC][U] (StepParams::anti)
//   energies  [U] doubles, transrot sums per atom [18 N] doubles, sums [16] doubles, move [8] doubles, chain velocities [4] doubles
//   exponent of each row [2 NC] int, status int
__host__ __device__ inline size_t step_group_bytes(int U, int NC, int anti) {
  return (size_t)((5 * NC + (anti ? 2 * NC : 0) + 1) * U + 6 * NC + 16 + 8 + 4) * 8 + ((size_t)(2 * NC + 1) * 4 + 7) / 8 * 8;
}
__host__ __device__ inline size_t step_smem_bytes(const PropDims& d, int U, int NC, int groups, int anti) {
  return (size_t)3 * d.nr * (d.nu + d.nv) * 8 + step_group_bytes(U, NC, anti) * groups;
}

// Most dynamic shared memory of a block (of the 227 KB that it may take).
constexpr int kStepSmemMax = 220 * 1024;

// The free ring polymer of the block's rows by fast transforms: lanes 2 y and
// 2 y + 1 take row y of q and of p.
template <int M, int NC>
__device__ __noinline__ void ring_rows(const StepParams& prm, double* sq, double* sp, int rows, int* sstat) {
  for (int x0 = threadIdx.x & ~31; x0 < 2 * rows; x0 += blockDim.x) {
    const int x = x0 + (threadIdx.x & 31), y = x >> 1;
    const bool active = x < 2 * rows, isp = x & 1;
    const int i = active ? (y % NC) / 3 : 0;
    double* r = (isp ? sp : sq) + (active ? y : x0 >> 1) * (M + 1);
    const bool fine = ring::row<M>(r, [=](int l, double v) { r[l] = v; }, isp, active, isp ? prm.mass[i] : prm.inv_mass[i],
                                   prm.fast);
    if (!fine) atomicOr(&sstat[y / NC], CR_TRAJ_NONFINITE);
  }
}

// The free ring polymer in orthonormal normal modes (nm_mode 1): circulants, on the
// rows as limbs. In FP64 the 4 P^2 products per coordinate held the pipe (H3 per step:
// 1 x 128 PILE mixed 684 -> 269 us with the noise's circulants in pile_half, 200 x 128
// without a thermostat plain 362 -> 181).
template <int NC>
__device__ __noinline__ void circulant_rows(const StepParams& prm, double* sq, double* sp, Limbs* limbs, int* sexp, int rows,
                                            int* sstat) {
  const int tid = threadIdx.x, nth = blockDim.x, U = prm.U, P = prm.P, flat = rows * U;
  for (int x = tid; x < 2 * rows; x += nth) sexp[x] = row_exponent(x < rows ? sq + x * U : sp + (x - rows) * U, U);
  __syncthreads();
  for (int x = tid; x < 2 * flat; x += nth)
    limbs[x] = to_limbs(to_fixed(x < flat ? sq[x] : sp[x - flat], sexp[x / U], prm.pguard));
  __syncthreads();
  for (int x = tid; x < flat; x += nth) {
    const int r = x / U, k = x - r * U, c = r % NC;
    const Limbs* lq = limbs + r * U;
    const Limbs* lp = lq + flat;
    FixedSum a1q{0, 0}, a1p{0, 0}, a2q{0, 0}, a3p{0, 0};
    int m = k;  // (k - l) mod P
#pragma unroll 4
    for (int l = 0; l < P; ++l) {
      const Limbs vq = lq[l], vp = lp[l], w1 = ldg_limbs(prm.circ + m);
      a1q.add(vq, w1);
      a1p.add(vp, w1);
      a2q.add(vq, ldg_limbs(prm.circ + P + m));
      a3p.add(vp, ldg_limbs(prm.circ + 2 * P + m));
      m = (m == 0) ? P - 1 : m - 1;
    }
    const int sq_e = sexp[r] - 1078 + prm.pguard, sp_e = sexp[rows + r] - 1078 + prm.pguard;
    const bool bad = sexp[r] == kFixedNan || sexp[rows + r] == kFixedNan;
    const double nan = __longlong_as_double(0x7ff8000000000000ll);
    const double pn = fma(prm.mass[c / 3], from_fixed(a2q.value(), prm.ek[1] + sq_e), from_fixed(a1p.value(), prm.ek[0] + sp_e));
    const double qn = fma(prm.inv_mass[c / 3], from_fixed(a3p.value(), prm.ek[2] + sp_e), from_fixed(a1q.value(), prm.ek[0] + sq_e));
    sp[x] = bad ? nan : pn;
    sq[x] = bad ? nan : qn;
    if (bad || nonfinite_bits(qn)) atomicOr(&sstat[r / NC], CR_TRAJ_NONFINITE);
  }
}

// The deviates of bead k of trajectory t and of its twin kt for coordinates 4 i .. 4 i + 3.
__device__ __forceinline__ void deviates(const StepParams& prm, int t, int k, int kt, int i, uint32_t step, uint32_t tag,
                                         double (&za)[4], double (&zb)[4]) {
  const uint32_t key = prm.traj0 + (uint32_t)t;
  const uint4 r = philox4x32_10(make_uint4((uint32_t)i, (uint32_t)k, step, tag), prm.seed, key);
  bm_pair(r.x, r.y, za[0], za[1]);
  bm_pair(r.z, r.w, za[2], za[3]);
  if (kt == k) {
    for (int d = 0; d < 4; ++d) zb[d] = za[d];
  } else {
    const uint4 w = philox4x32_10(make_uint4((uint32_t)i, (uint32_t)kt, step, tag), prm.seed, key);
    bm_pair(w.x, w.y, zb[0], zb[1]);
    bm_pair(w.z, w.w, zb[2], zb[3]);
  }
}

// Andersen's draw on the block's rows sp of p: the symmetric part, and the interior beads'
// antisymmetric part into santi.
template <int N>
__device__ __noinline__ void andersen_rows(const StepParams& prm, double* sp, double* santi, int t_first, int ng, uint32_t step) {
  constexpr int NC = 3 * N, NQ = (NC + 3) / 4;
  const int U = prm.U, P = prm.P, nb = ng * U;
  for (int x = threadIdx.x; x < nb * NQ; x += blockDim.x) {
    const int i = x / nb, y = x - i * nb, gg = y / U, k = y - gg * U, kt = prm.pair && k > 0 && 2 * k != P ? P - k : k;
    double za[4], zb[4];
    deviates(prm, t_first + gg, k, kt, i, step, TAG_ANDERSEN, za, zb);
#pragma unroll
    for (int d = 0; d < 4; ++d) {
      const int c = 4 * i + d, z = (gg * NC + c) * U + k;
      if (c >= NC) continue;
      const double s = prm.sigma[c / 3];
      sp[z] = kt == k ? za[d] * s : 0.5 * (za[d] + zb[d]) * s;
      if (kt != k) santi[z] = 0.5 * (za[d] - zb[d]) * s;
    }
  }
}

// PILE half step on the block's rows sp of p: by the limbs of the rows and of the
// deviates' symmetric part (|eta| < 8: one exponent for all), and with_anti of their
// antisymmetric part, whose share of p (b * half the difference of two beads'
// deviates, which the next drift removes) goes to the second half of anti. Out of line:
// both half steps fetch the same code (64 x 16 H3 mixed 18.6 -> 16.9 us per step).
template <int N>
__device__ __noinline__ void pile_half(const StepParams& prm, double* sp, Limbs* limbs, int* sexp, double* anti, int t_first,
                                       int ng, uint32_t step, uint32_t tag, bool with_anti) {
  constexpr int NC = 3 * N, NQ = (NC + 3) / 4, kEtaExp = 1025;
  const int tid = threadIdx.x, nth = blockDim.x, U = prm.U, P = prm.P, nb = ng * U, rows = ng * NC, flat = rows * U;
  const int pair = prm.pair, guard = prm.pguard;
  Limbs* le = limbs + flat;
  Limbs* la = reinterpret_cast<Limbs*>(anti);
  double* santi = anti + flat;
  // the rows by the last threads, while the first draw (64 x 16 H3, both half
  // steps: 15.1 -> 10.8 thousand cycles)
  for (int x = nth - 1 - tid; x < rows; x += nth) {
    const double* r = sp + x * U;
    const int e = row_exponent(r, U);
    sexp[x] = e;
#pragma unroll 3
    for (int k = 0; k < U; ++k) limbs[x * U + k] = to_limbs(to_fixed(r[k], e, guard + 1));
  }
  for (int x = tid; x < nb * NQ; x += nth) {
    const int i = x / nb, y = x - i * nb, gg = y / U, k = y - gg * U;
    double za[4], zb[4];
    deviates(prm, t_first + gg, k, pair && k > 0 && 2 * k != P ? P - k : k, i, step, tag, za, zb);
#pragma unroll
    for (int d = 0; d < 4; ++d)
      if (4 * i + d < NC) {
        const int64_t a = to_fixed(za[d], kEtaExp, guard + 1), b = to_fixed(zb[d], kEtaExp, guard + 1);
        const int z = (gg * NC + 4 * i + d) * U + k;
        le[z] = to_limbs(a + b);
        if (with_anti) la[z] = to_limbs(a - b);
      }
  }
  __syncthreads();
  // the carried beads' new momenta, then the interior beads' antisymmetric share
  const int h = with_anti ? (P - 1) / 2 : 0;
  for (int x = tid; x < flat + rows * h; x += nth) {
    if (x < flat) {
      const int r = x / U, k = x - r * U, c = r % NC;
      const Limbs* lp = limbs + r * U;
      const Limbs* ln = le + r * U;
      FixedSum a{0, 0}, e{0, 0};
      if (pair) {
        const Limbs* ka = prm.pile + k;
        const Limbs* kb = ka + U * U;
#pragma unroll 2
        for (int l = 0; l < U; ++l) {
          a.add(lp[l], ldg_limbs(ka + l * U));
          e.add(ln[l], ldg_limbs(kb + l * U));
        }
      } else {
        int m = k;  // (k - l) mod P
#pragma unroll 4
        for (int l = 0; l < U; ++l) {
          a.add(lp[l], ldg_limbs(prm.pile + m));
          e.add(ln[l], ldg_limbs(prm.pile + P + m));
          m = (m == 0) ? P - 1 : m - 1;
        }
      }
      double v = from_fixed(a.value(), prm.ep[0] + sexp[r] - 1077 + guard);
      if (sexp[r] == kFixedNan) v = __longlong_as_double(0x7ff8000000000000ll);
      // half the sum of the two deviates: one bit of the exponent
      sp[x] = fma(prm.sigma[c / 3], from_fixed(e.value(), prm.ep[1] + kEtaExp - 1078 + guard), v);
    } else {
      const int r = (x - flat) / h, k = x - flat - r * h + 1;
      const Limbs* ln = la + r * U;
      const Limbs* kc = prm.pile + 2 * U * U + k;
      FixedSum a{0, 0};
#pragma unroll 4
      for (int l = 1; l <= h; ++l) a.add(ln[l], ldg_limbs(kc + (l - 1) * U));
      santi[r * U + k] = prm.sigma[(r % NC) / 3] * from_fixed(a.value(), prm.ep[2] + kEtaExp - 1078 + guard);
    }
  }
  __syncthreads();
}

// Most threads of a block of the step kernel; MINB blocks stay resident per SM
// (the registers follow: 255 for 2, 168 for 3, 128 for 4).
constexpr int kStepThreads = 128;

// subs threads share a carried bead: the task stages spread over all threads of
// the block, a surface of one thread per bead is evaluated by the first gpb U.
// Worth it where the batch is too small to fill the GPU and the integrator weighs
// as much as the surface (H3, OH + H2).  The sums do not depend on the block's
// shape or on subs.
template <class PES, bool MIXED, int MINB>
__global__ void __launch_bounds__(kStepThreads, MINB) rpmd_run_kernel(const __grid_constant__ StepParams prm, int istep_arg, int nsteps) {
  const int istep0 = prm.istep_dev ? *prm.istep_dev : istep_arg;
  constexpr int N = PES::N;
  constexpr int NC = 3 * N;
  extern __shared__ double smem[];
  const int P = prm.P, U = prm.U, gpb = prm.gpb;
  const int tid = threadIdx.x, nth = blockDim.x;
  const int t_first = blockIdx.x * gpb;
  const int ng = min(gpb, prm.T - t_first);  // trajectories of this block
  const int nb = ng * U, rows = ng * NC, flat = rows * U;
  const PropDims pd = prm.pd;
  const int nke = 3 * pd.nr * pd.nu, nko = 3 * pd.nr * pd.nv;
  Limbs* s_ke = reinterpret_cast<Limbs*>(smem);
  Limbs* s_ko = s_ke + nke;
  double* sq = smem + nke + nko;
  double* sp = sq + gpb * NC * U;
  double* sf = sp + gpb * NC * U;
  double* area = sf + gpb * NC * U;
  Limbs* limbs = reinterpret_cast<Limbs*>(area);
  double* svb = area + (prm.anti_smem ? 4 : 2) * gpb * NC * U;  // bead energies
  double* smom = svb + gpb * U;
  double* ssum = smom + gpb * 6 * NC;
  double* smove = ssum + 16 * gpb;
  double* svnh = smove + 8 * gpb;
  int* sexp = reinterpret_cast<int*>(svnh + 4 * gpb);
  int* sstat = sexp + 2 * NC * gpb;
  // rows of the antisymmetric part: the deviates' limbs, and what they add to p
  double* anti = prm.anti_smem ? area + 2 * gpb * NC * U : prm.anti + (size_t)t_first * 2 * NC * U;
  double* santi = anti + flat;

  if (!prm.nm_mode) {
    for (int x = tid; x < nke; x += nth) s_ke[x] = prm.ke[x];
    for (int x = tid; x < nko; x += nth) s_ko[x] = prm.ko[x];
  }
  // the bead of this thread (threads below nb subs)
  const int sub = nb > 0 ? tid / nb : 0;
  const int b = tid - sub * nb, g = b / U, j = b - g * U;
  const bool bead = sub == 0;                    // evaluates the surface
  const int t = t_first + g;
  // does a carried bead stand for two
  auto twin_of = [&](int k) { return prm.pair && k > 0 && 2 * k != P ? P - k : k; };
  // sum over all P beads of a row of carried ones, in bead order
  auto bead_sum = [&](const double* x) {
    if (!prm.pair) {
      double r = x[0];
      for (int k = 1; k < U; ++k) r += x[k];
      return r;
    }
    double in = 0.0;
    for (int k = 1; k <= (P - 1) / 2; ++k) in += x[k];
    double r = fma(2.0, in, x[0]);
    if (U > 1 && (P & 1) == 0) r += x[U - 1];
    return r;
  };
  const size_t row_a = ((size_t)t * P + j) * NC, row_b = ((size_t)t * P + twin_of(j)) * NC;
  double ek_anti = 0.0;  // kinetic share of the antisymmetric starting momenta
  if (bead) {
    for (int c = 0; c < NC; ++c) {
      const int x = (g * NC + c) * U + j;
      double q = prm.q[row_a + c], p = prm.p[row_a + c], f = prm.f[row_a + c];
      if (row_b != row_a) {
        const double pb = prm.p[row_b + c], d = 0.5 * (p - pb);
        ek_anti = fma(d * d, prm.inv_mass[c / 3], ek_anti);
        q = 0.5 * (q + prm.q[row_b + c]);
        p = 0.5 * (p + pb);
        f = 0.5 * (f + prm.f[row_b + c]);
      }
      sq[x] = q;
      sp[x] = p;
      sf[x] = f;
    }
  }
  for (int x = tid; x < gpb; x += nth) sstat[x] = 0;
  const bool nhc = prm.thermostat == CR_THERMO_NHC, pile = prm.thermostat == CR_THERMO_PILE;
  if (nhc && tid < ng)
    for (int k = 0; k < 4; ++k) svnh[4 * tid + k] = prm.vnh[4 * (size_t)(t_first + tid) + k];
  bool drawn = false;  // the last step left an antisymmetric part of p (santi)
  __syncthreads();

  // nhc (src/nhc.f90): sum of p.p/(2m)/P/P, the chain, one scale
  auto nhc_half = [&](double extra) {
    if (bead) {
      double ek = extra;
      for (int c = 0; c < NC; ++c) {
        const double p = sp[(g * NC + c) * U + j];
        ek = fma(p * p, prm.inv_mass[c / 3], ek);
      }
      area[g * U + j] = ek;
    }
    __syncthreads();
    if (tid < ng) {
      double v[4];
      for (int k = 0; k < 4; ++k) v[k] = svnh[4 * tid + k];
      const double ek = bead_sum(area + tid * U) * (0.5 * prm.inv_P * prm.inv_P);
      smove[8 * tid] = nhc_scale(prm.nhc, ek, v);
      for (int k = 0; k < 4; ++k) svnh[4 * tid + k] = v[k];
    }
    __syncthreads();
    for (int x = tid; x < flat; x += nth) sp[x] = smove[8 * (x / (NC * U))] * sp[x];
    __syncthreads();
  };

  // the symmetric part of the state between two steps, of element x that carries p
  auto between = [&](int x, double p) {
    const int k = x % U;
    return twin_of(k) == k ? p : 0.5 * ((p + santi[x]) + (p - santi[x]));
  };

  for (int n = 1; n <= nsteps; ++n) {
    const int istep = istep0 + n;
    drawn = false;
    if (nhc) nhc_half(n == 1 ? ek_anti : 0.0);  // src/verlet.f90:186-208
    if (pile) pile_half<N>(prm, sp, limbs, sexp, anti, t_first, ng, (uint32_t)istep, TAG_PILE_A, false);

    // 1/2 kick (src/verlet.f90:216-218)
    for (int x = tid; x < flat; x += nth) sp[x] = fma(-prm.half_dt, sf[x], sp[x]);
    __syncthreads();

    // free ring polymer (src/verlet.f90:377-463): Caracal's cosine modes, or
    // orthonormal normal modes where nm_mode is set
    if (prm.nm_mode) {
      circulant_rows<NC>(prm, sq, sp, limbs, sexp, rows, sstat);
    } else if (prm.fast_M) {
      if (prm.fast_M == 16) ring_rows<16, NC>(prm, sq, sp, rows, sstat);
      else ring_rows<32, NC>(prm, sq, sp, rows, sstat);
    } else {
      // fold: rows of q, then of p, into limbs: x_l + x_{M-l}, x_l - x_{M-l}
      for (int x = tid; x < 2 * rows; x += nth) sexp[x] = row_exponent(x < rows ? sq + x * U : sp + (x - rows) * U, U);
      __syncthreads();
      const int nf = pd.split ? pd.nu : U;
      for (int x = tid; x < 2 * rows * nf; x += nth) {
        const int y = x / nf, l = x - y * nf, e = sexp[y];
        const double* r = y < rows ? sq + y * U : sp + (y - rows) * U;
        Limbs* o = limbs + y * U;
        const int64_t a = to_fixed(r[l], e, prm.guard);
        if (pd.split) {
          const int64_t c = 2 * l == pd.M ? 0 : to_fixed(r[pd.M - l], e, prm.guard);
          o[l] = to_limbs(a + c);
          if (l < pd.nv) o[pd.nu + l] = to_limbs(a - c);
        } else {
          o[l] = to_limbs(a);
        }
      }
      __syncthreads();
      // rows r and M - r of every coordinate
      for (int x = tid; x < rows * pd.nr; x += nth) {
        const int y = x / pd.nr, r = x - y * pd.nr, c = y % NC;
        const Limbs* uq = limbs + y * U;
        const Limbs* up = limbs + (rows + y) * U;
        const Limbs* k1 = s_ke + r * pd.nu;
        const Limbs* k2 = k1 + pd.nr * pd.nu;
        const Limbs* k3 = k2 + pd.nr * pd.nu;
        FixedSum a1q{0, 0}, a1p{0, 0}, a2q{0, 0}, a3p{0, 0};
#pragma unroll 4
        for (int l = 0; l < pd.nu; ++l) {
          const Limbs vq = uq[l], vp = up[l], w1 = k1[l];
          a1q.add(vq, w1);
          a1p.add(vp, w1);
          a2q.add(vq, k2[l]);
          a3p.add(vp, k3[l]);
        }
        const int64_t e1q = a1q.value(), e1p = a1p.value(), e2q = a2q.value(), e3p = a3p.value();
        int64_t o1q = 0, o1p = 0, o2q = 0, o3p = 0;
        if (pd.nv > 0) {
          a1q = a1p = a2q = a3p = FixedSum{0, 0};
          uq += pd.nu;
          up += pd.nu;
          k1 = s_ko + r * pd.nv;
          k2 = k1 + pd.nr * pd.nv;
          k3 = k2 + pd.nr * pd.nv;
#pragma unroll 4
          for (int l = 0; l < pd.nv; ++l) {
            const Limbs vq = uq[l], vp = up[l], w1 = k1[l];
            a1q.add(vq, w1);
            a1p.add(vp, w1);
            a2q.add(vq, k2[l]);
            a3p.add(vp, k3[l]);
          }
          o1q = a1q.value();
          o1p = a1p.value();
          o2q = a2q.value();
          o3p = a3p.value();
        }
        const double m = prm.mass[c / 3], im = prm.inv_mass[c / 3];
        const int sq_e = sexp[y] - 1078 + prm.guard, sp_e = sexp[rows + y] - 1078 + prm.guard;
        const bool bad = sexp[y] == kFixedNan || sexp[rows + y] == kFixedNan;
        const double nan = __longlong_as_double(0x7ff8000000000000ll);
#pragma unroll 1
        for (int h = 0; h < 2; ++h) {
          const int k = h == 0 ? r : pd.M - r;
          if (h == 1 && !(pd.split && 2 * r != pd.M)) break;
          const double pn = fma(m, from_fixed(e2q + o2q, prm.ek[1] + sq_e), from_fixed(e1p + o1p, prm.ek[0] + sp_e));
          const double qn = fma(im, from_fixed(e3p + o3p, prm.ek[2] + sp_e), from_fixed(e1q + o1q, prm.ek[0] + sq_e));
          sp[y * U + k] = bad ? nan : pn;
          sq[y * U + k] = bad ? nan : qn;
          // NaN / Inf check of the step (src/verlet.f90:1256-1275)
          if (bad || nonfinite_bits(qn)) atomicOr(&sstat[y / NC], CR_TRAJ_NONFINITE);
          o1q = -o1q;
          o1p = -o1p;
          o2q = -o2q;
          o3p = -o3p;
        }
      }
    }
    __syncthreads();

    // per-bead forces (src/verlet.f90:772-777)
    // by L lanes per bead, whole warps; a last partial pass repeats its first bead
    // without storing it
    auto by_lanes = [&](auto lanes, auto eval) {
      constexpr int L = decltype(lanes)::value;
      for (int b0 = 0; b0 < nb; b0 += nth / L) {
        const int y = b0 + tid / L;
        if (b0 + (tid & ~31) / L >= nb) break;  // none of the warp's
        const bool store = y < nb;
        const int yb = store ? y : b0, yg = yb / U, off = yg * NC * U + (yb - yg * U);
        double v;
        eval([&](int c) { return sq[off + c * U]; }, tid % L, v,
             [&](int c, double x) {
               if (store) sf[off + c * U] = x;
             });
        if (store && tid % L == 0) svb[yb] = v;
      }
    };
    using F = typename std::conditional<MIXED, float, double>::type;
    if constexpr (PES::kLanes > 1) {
      by_lanes(std::integral_constant<int, PES::kLanes>{},
               [](auto get, int lane, double& v, auto put) { PES::template egrad<F>(get, lane, v, put); });
    } else {
      bool quads = false;
      if constexpr (PES::kQuad) quads = prm.quad;
      if constexpr (PES::kQuad) {
        if (quads)
          by_lanes(std::integral_constant<int, 4>{},
                   [](auto get, int lane, double& v, auto put) { PES::template quad<F>(get, lane, v, put); });
      }
      if (!quads && bead) {
        double q[NC], gr[NC], v;
#pragma unroll
        for (int c = 0; c < NC; ++c) q[c] = sq[(g * NC + c) * U + j];
        PES::template egrad<F>(q, v, gr);
        svb[b] = v;
#pragma unroll
        for (int c = 0; c < NC; ++c) sf[(g * NC + c) * U + j] = gr[c];
      }
    }

    // reaction coordinate of the centroid (umbrella mode 1 of a child step,
    // src/verlet.f90:1049-1050 -> src/umbrella.f90:115-117): eight trajectories a
    // warp and the last warps first, which have the fewest passes over the beads
    // above, with no barrier between the two.  CH4 + H 4096 x 32, 40 steps: 4246 ->
    // 4004 us mixed; 1000 x 32, 20 steps: 2895 -> 2877 plain.  (Before the surface in
    // place of after it: 4074 and 2933.)
    if (prm.xi_on) {
      for (int x0 = (nth / 32 - 1 - tid / 32) * 8; x0 < ng; x0 += nth / 4) {
        const int end = min(x0 + 8, ng), gg = x0 + tid % 32;
        for (int y = x0 * NC + tid % 32; y < end * NC; y += 32) area[y] = bead_sum(sq + y * U) * prm.inv_P;
        __syncwarp();
        if (gg < end) {
          const double xi = xi_bimolec_value<N>(prm.xi, area + gg * NC);
          prm.side[(size_t)(t_first + gg) * prm.side_stride + (istep - prm.side_step0 - 1)] = xi > 0.0 ? 1 : 0;
        }
      }
    }

    // umbrella windows (src/verlet.f90:1043-1046): the bias at the centroid on
    // every bead's gradient
    if (prm.umb_on) umbrella_step<N>(prm.xi, prm.umb, bead_sum, sq, sf, area, t_first, ng, U, prm.inv_P);

    __syncthreads();

    // 1/2 kick (src/verlet.f90:1060-1062)
    for (int x = tid; x < flat; x += nth) sp[x] = fma(-prm.half_dt, sf[x], sp[x]);
    __syncthreads();

    if (nhc) nhc_half(0.0);  // src/verlet.f90:1085-1106

    // Andersen (src/verlet.f90:1159-1165): full resample every andersen_step
    if (prm.thermostat == CR_THERMO_ANDERSEN && (istep % prm.andersen_step) == 0) {
      andersen_rows<N>(prm, sp, santi, t_first, ng, (uint32_t)istep);
      drawn = prm.anti != nullptr;
      __syncthreads();
    }
    if (pile) {
      drawn = prm.anti != nullptr;
      pile_half<N>(prm, sp, limbs, sexp, anti, t_first, ng, (uint32_t)istep, TAG_PILE_B, drawn);
    }

    // transrot (src/transrot.f90:36-237): removed COM velocity and rotation
    // centre both carry Caracal's extra 1/P (total mass P^2 sum m)
    const bool few = PES::kLanes > 1 ? P == 1 : U <= 2;
    if (prm.transrot && few) {
      if (PES::kLanes > 1 || 4 * gpb <= nth) transrot_few<N, 4>(prm, sq, sp, ng, sstat);
      else if constexpr (PES::kLanes == 1) transrot_few<N, 1>(prm, sq, sp, ng, sstat);
      __syncthreads();
    } else if (prm.transrot) {
      // rows of q and p as limbs; per atom the bead sums of p, q, q_a p_b and
      // q_a q_b in fixed point (in FP64 some 20 instructions per bead and atom, and the
      // solve on one lane: per step H3 64 x 16 PILE mixed 32.2 -> 24.8 us, OH + H2 1000 x 24
      // plain 61 -> 51 us)
      for (int x = tid; x < 2 * rows; x += nth) sexp[x] = row_exponent(x < rows ? sq + x * U : sp + (x - rows) * U, U);
      __syncthreads();
      for (int x = tid; x < 2 * flat; x += nth)
        limbs[x] = to_limbs(to_fixed(x < flat ? sq[x] : sp[x - flat], sexp[x / U], prm.pguard));
      __syncthreads();
      for (int x = tid; x < ng * N * kMoments; x += nth) {
        const int y = x / kMoments, v = x - y * kMoments;  // y: trajectory and atom
        smom[x] = atom_moment(limbs, limbs + flat, sexp, sexp + rows, 3 * y, v, U, P, prm.pair, prm.pguard);
      }
      __syncthreads();
      // over the atoms: sum p, sum m q, q x p, sum m q q^T
      for (int x = tid; x < 15 * ng; x += nth) {
        const int gg = x / 15, v = x - 15 * gg;
        const double* mo = smom + gg * N * kMoments;
        double a = 0.0;
        if (v < 3) {
          for (int i = 0; i < N; ++i) a += mo[i * kMoments + v];
        } else if (v < 6) {
          for (int i = 0; i < N; ++i) a = fma(prm.mass[i], mo[i * kMoments + v], a);
        } else if (v < 9) {
          for (int i = 0; i < N; ++i) a += mo[i * kMoments + 2 * v - 6] - mo[i * kMoments + 2 * v - 5];
        } else {
          for (int i = 0; i < N; ++i) a = fma(prm.mass[i], mo[i * kMoments + v + 3], a);
        }
        ssum[16 * gg + v] = a;
      }
      __syncthreads();
      for (int x0 = 0; x0 < ng; x0 += nth / 4) {
        const int gg = x0 + tid / 4;
        if (x0 + (tid & ~31) / 4 >= ng) break;
        const bool real = gg < ng;
        double* mv = smove + 8 * (real ? gg : x0);
        double bb, va;
        const double* tot = ssum + 16 * (real ? gg : x0);
        const bool ok = transrot_quad([&](int k) { return tot[k]; }, tid & 3, prm.itm, prm.kap, N <= 2, bb, va);
        if (real && (tid & 3) < 3) {
          mv[tid & 3] = bb;
          mv[3 + (tid & 3)] = va;
          if ((tid & 3) == 0) {
            mv[6] = ok ? 0.0 : 1.0;
            if (!ok) atomicOr(&sstat[gg], CR_TRAJ_SINGULAR_INERTIA);
          }
        }
      }
      __syncthreads();
      for (int x = tid; x < flat; x += nth) {
        const int r = x / U, gg = r / NC, c = r - gg * NC, d = c % 3;
        const int e = d == 2 ? 0 : d + 1, f = d == 0 ? 2 : d - 1;
        const double* mv = smove + 8 * gg;
        const double qe = sq[x + (e - d) * U], qf = sq[x + (f - d) * U];
        const double u = fma(mv[3 + e], qf, fma(-mv[3 + f], qe, mv[d]));
        const double p = mv[6] != 0.0 ? sp[x] : fma(-prm.mass[c / 3], u, sp[x]);  // singular: left as it is
        sp[x] = drawn && n < nsteps ? between(x, p) : p;
      }
      __syncthreads();
    }

    if (drawn && n < nsteps && (!prm.transrot || few)) {
      for (int x = tid; x < flat; x += nth) sp[x] = between(x, sp[x]);
      __syncthreads();
    }
  }

  // the state of every bead, the potential energy of the last step
  if (bead) {
    for (int c = 0; c < NC; ++c) {
      const int x = (g * NC + c) * U + j;
      const double q = sq[x], p = sp[x], f = sf[x];
      prm.q[row_a + c] = q;
      prm.f[row_a + c] = f;
      if (row_b != row_a) {
        const double a = drawn ? santi[x] : 0.0;
        prm.p[row_a + c] = p + a;
        prm.p[row_b + c] = p - a;
        prm.q[row_b + c] = q;
        prm.f[row_b + c] = f;
      } else {
        prm.p[row_a + c] = p;
      }
    }
  }
  __syncthreads();
  if (tid < ng) {
    const int tt = t_first + tid;
    prm.epot[tt] = bead_sum(svb + tid * U);
    if (nhc)
      for (int k = 0; k < 4; ++k) prm.vnh[4 * (size_t)tt + k] = svnh[4 * tid + k];
    if (sstat[tid]) atomicOr(&prm.status[tt], sstat[tid]);
  }
}

// V and dV/dq, L threads per evaluated bead: PES::kLanes, or 4 where the surface has
// that form too (PES::kQuad).
template <class PES, bool MIXED, int L>
__global__ void egrad_kernel(int nbeads_total, BeadRows rows, const double* q, double* V, double* g) {
  constexpr int NC = 3 * PES::N;
  using F = typename std::conditional<MIXED, float, double>::type;
  const size_t n = (size_t)nbeads_total, e = evaluation_of(blockIdx.x, blockDim.x, threadIdx.x, L);
  const int lane = threadIdx.x % L;  // (blocks hold whole evaluations)
  if (L == 1 && e >= n) return;
  const bool store = e < n;  // a quad's shuffles need whole warps
  const size_t b = store ? e : n - 1;
  const size_t r = rows.row(b), r2 = rows.twin(b);
  double v;
  if constexpr (L > 1) {
    auto get = [&](int c) { return q[r * NC + c]; };
    auto put = [&](int c, double y) {
      if (!store) return;
      g[r * NC + c] = y;
      if (r2 != r) g[r2 * NC + c] = y;
    };
    if constexpr (PES::kLanes > 1) PES::template egrad<F>(get, lane, v, put);
    else PES::template quad<F>(get, lane, v, put);
  } else {
    double qq[NC], gg[NC];
#pragma unroll
    for (int c = 0; c < NC; ++c) qq[c] = q[r * NC + c];
    PES::template egrad<F>(qq, v, gg);
#pragma unroll
    for (int c = 0; c < NC; ++c) {
      g[r * NC + c] = gg[c];
      if (r2 != r) g[r2 * NC + c] = gg[c];
    }
  }
  if (store && lane == 0) {
    V[r] = v;
    if (r2 != r) V[r2] = v;
  }
}

}  // namespace cr
