// Step kernels of the RPMD engine for molecules too large to keep a bead's
// state in registers (QMDFF): the state stays in HBM, laid out
// q[traj][bead][atom][3], and one step is a short chain of kernels captured
// in a CUDA graph:
//   split_nhc_kernel     Nose-Hoover chain (NHC only)
//   split_drift_kernel   PILE half (if PILE), 1/2 kick, free ring polymer
//   (force kernel)       dV/dq and V of every bead
//   split_kick_kernel    1/2 kick, Andersen resample or PILE half
//   split_nhc_kernel     Nose-Hoover chain (NHC only)
//   split_berendsen_kernel  pressure and box scaling (NpT only)
//   split_moments_kernel, split_solve_kernel, split_apply_kernel
//                        NaN check, transrot, epot per trajectory
//   split_advance_kernel step counter + 1
// The order is Caracal's verlet (src/verlet.f90:216-218, 377-463, 772-777,
// 1060-1062, 1159-1165, 1256-1306).  The step index lives on the device so a
// captured step can be replayed.
//
// Free ring-polymer propagation.  Caracal's composite map K = C diag(poly) C
// (C = sqrt(1/P) cos(2 pi j k/P), src/rfft.f90 and src/irfft.f90 applied as
// the normal-mode transform) satisfies K[j][l] = K[-j][l] = K[j][-l], so the
// outputs of beads j and P-j coincide and only the P/2+1 symmetrised inputs
// s_l = x_l + x_{P-l} matter.  For even P, with M = P/2,
// C[M-r][k] = (-1)^k C[r][k]: splitting K = Ke + Ko by mode parity gives
// K[r] = Ke[r] + Ko[r] and K[M-r] = Ke[r] - Ko[r], with Ke even and Ko odd
// under l -> M-l.  One pass over u_l = s_l + s_{M-l} and v_l = s_l - s_{M-l}
// therefore yields rows r and M-r together: 4 (M/2+1)(M+1) FMAs per
// coordinate and trajectory for the four blocks, against 4 (M+1)^2 for the
// unique rows and 4 P (M+1) for one row per bead.
#pragma once
#include <cuda_runtime.h>

#include "cr_common.cuh"
#include "rpmd_kernel.cuh"

namespace cr {

struct SplitParams {
  int T, P, N, NC;
  int M;          // P / 2
  int split;      // 1: even P, parity-split blocks; 0: odd P, unique rows only
  int nr, nu, nv; // task rows, u length, v length
  int su, sv;     // padded smem row strides of u and v
  int thermostat, andersen_step, transrot;
  uint32_t seed, traj0;
  double half_dt;
  double itm, kap;         // transrot's masses (StepParams)
  const double* mass;      // [N]
  const int* wfix;         // [2 N] the masses, then twice the masses, as limbs under wexp (split_moments_kernel)
  int wexp;                // value 2^(wexp - 56)
  const double* inv_mass;  // [N]
  const double* sigma;     // [N] sqrt(m P / beta)
  const double* ke;        // [3][nr][nu]: K1, K2, K3 (unit mass), even-mode part (or full rows)
  const double* ko;        // [3][nr][nv]: odd-mode part
  const double* pile;      // [2][P] circulant a, b
  FastRing fast;           // split_drift_fast_kernel's mode tables
  int pair, U;             // 1: after a drift rows l and P - l of q are equal (nm_mode 0, P > 2); U rows to visit
  double* q;
  double* p;
  double* f;               // dV/dq
  double* V;               // [T][P] bead energies
  double* epot;            // [T]
  int* status;             // [T]
  int* istep;              // device step counter (last completed step)
  NhcParams nhc;
  double* vnh;             // [T][4] Nose-Hoover chain velocities
  // constrained parent (verlet with constrain = 1)
  int constrain;
  XiDev xi;
  double* dxi;             // [T][NC] dxi_act
  double* cq;              // [T][NC] centroid before SHAKE
  int* shake_fail;         // [T]
  int umbrella;            // 1: bias towards the trajectory's window after the forces
  UmbrellaDev umb;
  // nm_mode 1: orthonormal normal modes, K1, K2, K3 circulant: circ[w][(j - l) mod P]
  int nm_mode;
  const double* circ;      // [3][P]
  // transrot / energy scratch of split_moments_kernel and split_solve_kernel
  double* fsum;            // [T][S][16] partial sums per slice
  int* fstat;              // [T][S] status bits per slice
  double* fmove;           // [T][10] b, va, (3 unused), skip flag: kMoveDoubles
};

constexpr int kSplitBlock = 128;
constexpr int kFinishBlock = 256;

__host__ __device__ inline int split_chunk(int P) { return P <= 64 ? 32 : 16; }

// shared-memory doubles of split_drift_kernel / split_kick_kernel
__host__ __device__ inline size_t split_smem_doubles(const SplitParams& s, bool pile) {
  const int cw = split_chunk(s.P), sp = s.P + 1;
  size_t n = (size_t)3 * s.nr * (s.nu + s.nv);        // tables
  n += (size_t)2 * cw * sp;                            // xq, xp
  n += (size_t)2 * cw * (s.su + s.sv);                 // u, v (q and p)
  n += (size_t)cw;                                     // q shifts
  if (pile) n += (size_t)2 * cw * sp + 2 * (size_t)s.P;  // eta, tmp, circulants
  return n;
}

// Deterministic block sum of NV values per thread (fixed tree); red holds
// NV * blockDim.x doubles.  The result is returned on every thread.
template <int NV>
__device__ inline void block_sum(double (&v)[NV], double* red) {
  __syncthreads();
#pragma unroll
  for (int i = 0; i < NV; ++i) red[i * blockDim.x + threadIdx.x] = v[i];
  __syncthreads();
  for (int w = blockDim.x / 2; w >= 1; w >>= 1) {
    if ((int)threadIdx.x < w) {
#pragma unroll
      for (int i = 0; i < NV; ++i) red[i * blockDim.x + threadIdx.x] += red[i * blockDim.x + threadIdx.x + w];
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < NV; ++i) v[i] = red[i * blockDim.x];
}

// Normals of coordinates [c0, c0+cw) of every bead into eta[c][j] (row stride sp).
__device__ inline void chunk_normals(const SplitParams& s, uint32_t traj, uint32_t step, uint32_t tag, int c0,
                                     int cw, double* eta, int sp) {
  const int npair = (cw + 1) / 2;
  for (int idx = threadIdx.x; idx < s.P * npair; idx += blockDim.x) {
    const int j = idx / npair, ip = idx % npair;
    const int c = 2 * ip;
    double z0, z1;
    normal_pair(s.seed, traj, (uint32_t)((c0 + c) / 2), (uint32_t)j, step, tag, z0, z1);
    eta[c * sp + j] = z0;
    if (c + 1 < cw) eta[(c + 1) * sp + j] = z1;
  }
}

// PILE half step on xp (chunk of cw coordinates): p <- a * p + sigma b * eta.
__device__ inline void chunk_pile(const SplitParams& s, uint32_t traj, uint32_t step, uint32_t tag, int c0, int cw,
                                  double* xp, double* eta, double* tmp, const double* sa, const double* sb,
                                  int sp) {
  chunk_normals(s, traj, step, tag, c0, cw, eta, sp);
  __syncthreads();
  const int P = s.P;
  for (int idx = threadIdx.x; idx < P * cw; idx += blockDim.x) {
    const int c = idx % cw, j = idx / cw;
    const double* x = xp + c * sp;
    const double* e = eta + c * sp;
    double ap = 0.0, ae = 0.0;
    int m = j;  // (j - l) mod P
    for (int l = 0; l < P; ++l) {
      ap = fma(sa[m], x[l], ap);
      ae = fma(sb[m], e[l], ae);
      m = (m == 0) ? P - 1 : m - 1;
    }
    tmp[c * sp + j] = ap + s.sigma[(c0 + c) / 3] * ae;
  }
  __syncthreads();
  for (int idx = threadIdx.x; idx < P * cw; idx += blockDim.x) {
    const int c = idx % cw, j = idx / cw;
    xp[c * sp + j] = tmp[c * sp + j];
  }
  __syncthreads();
}

__global__ void __launch_bounds__(kSplitBlock) split_drift_kernel(SplitParams s) {
  extern __shared__ double sm[];
  const int P = s.P, NC = s.NC, cw_max = split_chunk(P), sp = P + 1;
  const int t = blockIdx.y, c0 = blockIdx.x * cw_max;
  const int cw = min(cw_max, NC - c0);
  const uint32_t istep = (uint32_t)(*s.istep + 1);
  const bool pile = s.thermostat == CR_THERMO_PILE;
  const int nke = 3 * s.nr * s.nu, nko = 3 * s.nr * s.nv;
  double* ske = sm;
  double* sko = ske + nke;
  double* xq = sko + nko;
  double* xp = xq + cw_max * sp;
  double* uq = xp + cw_max * sp;
  double* up = uq + cw_max * s.su;
  double* vq = up + cw_max * s.su;
  double* vp = vq + cw_max * s.sv;
  double* shq = vp + cw_max * s.sv;  // per-coordinate q shift
  double* eta = shq + cw_max;
  double* tmp = eta + cw_max * sp;
  double* sa = tmp + cw_max * sp;
  double* sb = sa + P;
  if (s.nm_mode) {
    for (int x = threadIdx.x; x < 3 * P; x += blockDim.x) ske[x] = s.circ[x];  // 3 P <= nke
  } else {
    for (int x = threadIdx.x; x < nke; x += blockDim.x) ske[x] = s.ke[x];
    for (int x = threadIdx.x; x < nko; x += blockDim.x) sko[x] = s.ko[x];
  }
  if (pile)
    for (int x = threadIdx.x; x < 2 * P; x += blockDim.x) sa[x] = s.pile[x];
  const size_t tb = (size_t)t * P * NC + c0;
  for (int idx = threadIdx.x; idx < P * cw; idx += blockDim.x) {
    const int c = idx % cw, j = idx / cw;
    const size_t g = tb + (size_t)j * NC + c;
    xq[c * sp + j] = s.q[g];
    xp[c * sp + j] = pile ? s.p[g] : s.p[g] - s.half_dt * s.f[g];
  }
  __syncthreads();
  if (pile) {
    chunk_pile(s, s.traj0 + (uint32_t)t, istep, TAG_PILE_A, c0, cw, xp, eta, tmp, sa, sb, sp);
    for (int idx = threadIdx.x; idx < P * cw; idx += blockDim.x) {
      const int c = idx % cw, j = idx / cw;
      xp[c * sp + j] = xp[c * sp + j] - s.half_dt * s.f[tb + (size_t)j * NC + c];
    }
    __syncthreads();
  }
  // q relative to its bead-0 value (the constant vector is the centroid
  // mode: K1 keeps it, K2 drops it; the products then round on bead spreads)
  for (int c = threadIdx.x; c < cw; c += blockDim.x) shq[c] = xq[c * sp];
  __syncthreads();
  for (int idx = threadIdx.x; idx < P * cw; idx += blockDim.x) {
    const int c = idx % cw, j = idx / cw;
    xq[c * sp + j] -= shq[c];
  }
  __syncthreads();
  if (s.nm_mode) {
    // orthonormal normal modes: row j of the circulant K1, K2, K3 (the
    // constant vector is an eigenvector of all three, so the q shift holds)
    for (int idx = threadIdx.x; idx < P * cw; idx += blockDim.x) {
      const int c = idx % cw, j = idx / cw;
      const double* xqc = xq + c * sp;
      const double* xpc = xp + c * sp;
      double a1p = 0.0, a1q = 0.0, a2q = 0.0, a3p = 0.0;
      int m = j;  // (j - l) mod P
      for (int l = 0; l < P; ++l) {
        const double c1 = ske[m], c2 = ske[P + m], c3 = ske[2 * P + m];
        a1p = fma(c1, xpc[l], a1p);
        a1q = fma(c1, xqc[l], a1q);
        a2q = fma(c2, xqc[l], a2q);
        a3p = fma(c3, xpc[l], a3p);
        m = (m == 0) ? P - 1 : m - 1;
      }
      const int atom = (c0 + c) / 3;
      const size_t g = tb + (size_t)j * NC + c;
      s.q[g] = fma(s.inv_mass[atom], a3p, a1q) + shq[c];
      s.p[g] = fma(s.mass[atom], a2q, a1p);
    }
    return;
  }
  // fold into u (and v)
  const int M = s.M;
  for (int idx = threadIdx.x; idx < cw * s.nu; idx += blockDim.x) {
    const int c = idx % cw, l = idx / cw;
    const double* a = xq + c * sp;
    const double* b = xp + c * sp;
    const double aq = sym_at(a, l, P), ap = sym_at(b, l, P);
    if (s.split && 2 * l != M) {
      const double bq = sym_at(a, M - l, P), bp = sym_at(b, M - l, P);
      uq[c * s.su + l] = aq + bq;
      up[c * s.su + l] = ap + bp;
      if (l < s.nv) {
        vq[c * s.sv + l] = aq - bq;
        vp[c * s.sv + l] = ap - bp;
      }
    } else {
      uq[c * s.su + l] = aq;
      up[c * s.su + l] = ap;
    }
  }
  __syncthreads();
  // rows r (and M - r): q' = K1 q + K3 p / m, p' = K1 p + m K2 q
  const int nr = s.nr, nu = s.nu, nv = s.nv;
  for (int idx = threadIdx.x; idx < cw * nr; idx += blockDim.x) {
    const int c = idx % cw, r = idx / cw;
    const double* k1e = ske + (0 * nr + r) * nu;
    const double* k2e = ske + (1 * nr + r) * nu;
    const double* k3e = ske + (2 * nr + r) * nu;
    const double* uqc = uq + c * s.su;
    const double* upc = up + c * s.su;
    double e1q = 0.0, e1p = 0.0, e2q = 0.0, e3p = 0.0;
    for (int l = 0; l < nu; ++l) {
      const double a1 = k1e[l], a2 = k2e[l], a3 = k3e[l];
      const double xq_ = uqc[l], xp_ = upc[l];
      e1q = fma(a1, xq_, e1q);
      e1p = fma(a1, xp_, e1p);
      e2q = fma(a2, xq_, e2q);
      e3p = fma(a3, xp_, e3p);
    }
    double o1q = 0.0, o1p = 0.0, o2q = 0.0, o3p = 0.0;
    if (nv > 0) {
      const double* k1o = sko + (0 * nr + r) * nv;
      const double* k2o = sko + (1 * nr + r) * nv;
      const double* k3o = sko + (2 * nr + r) * nv;
      const double* vqc = vq + c * s.sv;
      const double* vpc = vp + c * s.sv;
      for (int l = 0; l < nv; ++l) {
        const double a1 = k1o[l], a2 = k2o[l], a3 = k3o[l];
        const double xq_ = vqc[l], xp_ = vpc[l];
        o1q = fma(a1, xq_, o1q);
        o1p = fma(a1, xp_, o1p);
        o2q = fma(a2, xq_, o2q);
        o3p = fma(a3, xp_, o3p);
      }
    }
    const int atom = (c0 + c) / 3;
    const double m = s.mass[atom], im = s.inv_mass[atom];
    const double qa = fma(im, e3p + o3p, e1q + o1q) + shq[c];
    const double pa = fma(m, e2q + o2q, e1p + o1p);
    int rows[2] = {r, -1};
    double qv[2] = {qa, 0.0}, pv[2] = {pa, 0.0};
    if (s.split && 2 * r != M) {
      rows[1] = M - r;
      qv[1] = fma(im, e3p - o3p, e1q - o1q) + shq[c];
      pv[1] = fma(m, e2q - o2q, e1p - o1p);
    }
    for (int k = 0; k < 2; ++k) {
      const int row = rows[k];
      if (row < 0) continue;
      const size_t g = tb + (size_t)row * NC + c;
      s.q[g] = qv[k];
      s.p[g] = pv[k];
      if (row != 0 && 2 * row != P) {
        const size_t g2 = tb + (size_t)(P - row) * NC + c;
        s.q[g2] = qv[k];
        s.p[g2] = pv[k];
      }
    }
  }
}

// Row that equals row l after a drift (l itself: none).
__device__ __forceinline__ int twin_row(const SplitParams& s, int l) {
  return s.pair && l > 0 && 2 * l != s.P ? s.P - l : l;
}
__device__ __forceinline__ bool same_bits(double a, double b) {
  return __double_as_longlong(a) == __double_as_longlong(b);
}

// Free ring-polymer step of P = 2 M = 8, 16, 32, 64 beads with the 1/2 kick before
// it (no PILE) by fast transforms in fixed point (ring_fast.cuh): lanes 2 y and
// 2 y + 1 of a warp take coordinate y of q and of p - dt/2 dV/dq, on the mean of
// rows l and P - l (which mostly are equal: then nothing is added).  Block: 4 warps =
// 64 coordinates; grid (ceil(NC / 64), T).  In FP64 the transforms were bound by
// the FP64 pipe, some 900 instructions of 64 cycles per coordinate: 1024 x 64
// C20H42 526 -> 203 us, where reading q, p, f and writing q, p takes 70.
constexpr int kDriftThreads = 128;
template <int M>
__global__ void __launch_bounds__(kDriftThreads) split_drift_fast_kernel(const __grid_constant__ SplitParams s) {
  constexpr int P = 2 * M;
  __shared__ double rows[kDriftThreads * (M + 1)];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int NC = s.NC, t = blockIdx.y;
  const int c0 = (blockIdx.x * 4 + warp) * 16, c = c0 + (lane >> 1);
  if (c0 >= NC) return;
  const bool isp = lane & 1, active = c < NC;
  const size_t tb = (size_t)t * P * NC + (active ? c : c0);
  double* x = (isp ? s.p : s.q) + tb;
  const double* f = s.f + tb;
  const double hdt = isp ? s.half_dt : 0.0;
  double* buf = rows + threadIdx.x * (M + 1);
  // kLoad rows at a time, so that their loads are in flight together
  constexpr int kLoad = M < 8 ? 5 : 11;
#pragma unroll 1
  for (int l0 = 0; l0 <= M; l0 += kLoad) {
    double xa[kLoad], xb[kLoad], fa[kLoad], fb[kLoad];
#pragma unroll
    for (int k = 0; k < kLoad; ++k) {
      const int l = min(l0 + k, M);
      const size_t a = (size_t)l * NC, b = (size_t)(l == 0 || l == M ? l : P - l) * NC;
      xa[k] = x[a];
      xb[k] = x[b];
      fa[k] = isp ? f[a] : 0.0;
      fb[k] = isp ? f[b] : 0.0;
    }
#pragma unroll
    for (int k = 0; k < kLoad; ++k) {
      const int l = l0 + k;
      double v = fma(-hdt, fa[k], xa[k]);
      if (!(same_bits(xa[k], xb[k]) && same_bits(fa[k], fb[k]))) v = 0.5 * (v + fma(-hdt, fb[k], xb[k]));
      if (l <= M) buf[l] = v;
    }
  }
  auto put = [&](int l, double y) {
    x[(size_t)l * NC] = y;
    if (l > 0 && l < M) x[(size_t)(P - l) * NC] = y;
  };
  const int atom = active ? c / 3 : 0;
  ring::row<M>(buf, put, isp, active, isp ? s.mass[atom] : s.inv_mass[atom], s.fast);
}

// mode 0: 1/2 kick and thermostat; 1: 1/2 kick only; 2: thermostat only (the
// constrained parent runs RATTLE between the two).
__global__ void __launch_bounds__(kSplitBlock) split_kick_kernel(SplitParams s, int mode) {
  extern __shared__ double sm[];
  const int P = s.P, NC = s.NC, cw_max = split_chunk(P), sp = P + 1;
  const int t = blockIdx.y, c0 = blockIdx.x * cw_max;
  const int cw = min(cw_max, NC - c0);
  const int istep = *s.istep + 1;
  const size_t tb = (size_t)t * P * NC + c0;
  const uint32_t traj = s.traj0 + (uint32_t)t;
  const double hdt = mode == 2 ? 0.0 : s.half_dt;
  // the kick alone: after the drift and the forces, rows l and P - l of p and f
  // are equal (1024 x 64 C20H42 32 us)
  auto kick = [&]() {
    const int c = threadIdx.x % cw_max;
    if (c >= cw) return;
    for (int l = threadIdx.x / cw_max; l < s.U; l += kSplitBlock / cw_max) {
      const size_t g = tb + (size_t)l * NC + c;
      const double p = fma(-s.half_dt, s.f[g], s.p[g]);
      s.p[g] = p;
      const int k = twin_row(s, l);
      if (k != l) s.p[tb + (size_t)k * NC + c] = p;
    }
  };
  if (mode == 1) {
    kick();
    return;
  }
  if (s.thermostat == CR_THERMO_PILE) {
    double* xp = sm;
    double* eta = xp + cw_max * sp;
    double* tmp = eta + cw_max * sp;
    double* sa = tmp + cw_max * sp;
    double* sb = sa + P;
    for (int x = threadIdx.x; x < 2 * P; x += blockDim.x) sa[x] = s.pile[x];
    for (int idx = threadIdx.x; idx < P * cw; idx += blockDim.x) {
      const int c = idx % cw, j = idx / cw;
      const size_t g = tb + (size_t)j * NC + c;
      xp[c * sp + j] = s.p[g] - hdt * s.f[g];
    }
    __syncthreads();
    chunk_pile(s, traj, (uint32_t)istep, TAG_PILE_B, c0, cw, xp, eta, tmp, sa, sb, sp);
    for (int idx = threadIdx.x; idx < P * cw; idx += blockDim.x) {
      const int c = idx % cw, j = idx / cw;
      s.p[tb + (size_t)j * NC + c] = xp[c * sp + j];
    }
    return;
  }
  if (s.thermostat == CR_THERMO_ANDERSEN && (istep % s.andersen_step) == 0) {
    // full resample (src/andersen.f90:37-71); the kick is overwritten
    const int npair = (cw + 1) / 2;
    for (int idx = threadIdx.x; idx < P * npair; idx += blockDim.x) {
      const int j = idx / npair, ip = idx % npair;
      const int c = 2 * ip;
      double z0, z1;
      normal_pair(s.seed, traj, (uint32_t)((c0 + c) / 2), (uint32_t)j, (uint32_t)istep, TAG_ANDERSEN, z0, z1);
      s.p[tb + (size_t)j * NC + c] = z0 * s.sigma[(c0 + c) / 3];
      if (c + 1 < cw) s.p[tb + (size_t)j * NC + c + 1] = z1 * s.sigma[(c0 + c + 1) / 3];
    }
    return;
  }
  if (mode != 2) kick();
}

// ---- constrained parent (src/constrain_q.f90, src/constrain_p.f90) ----------
// One block per trajectory.  SHAKE: the centroid c (kept for the next dxi),
// Newton iterations for the multiplier on thread 0 (at most 200; the
// tolerances 1.0E-8 and 1.0E-10 are REAL(4) literals), then every bead moves:
// q by the coefficient of the last iteration's start, p by the updated
// multiplier.  A failed SHAKE leaves q, p unchanged and is flagged.
template <int N>
__global__ void split_shake_kernel(SplitParams s) {
  constexpr int NC = 3 * N;
  __shared__ double cq[NC], dxa[NC], res[3];
  const int t = blockIdx.x, P = s.P;
  const size_t tb = (size_t)t * P * NC;
  for (int c = threadIdx.x; c < NC; c += blockDim.x) {
    double acc = 0.0;
    for (int k = 0; k < P; ++k) acc = acc + s.q[tb + (size_t)k * NC + c];
    cq[c] = acc / P;
    dxa[c] = s.dxi[(size_t)t * NC + c];
    s.cq[(size_t)t * NC + c] = cq[c];
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    const double dt = 2.0 * s.half_dt;
    double mult = 0.0, coeff = 0.0, qt[NC], dxn[NC];
    int ok = 0;
    for (int iter = 1; iter <= 200; ++iter) {
      coeff = mult * dt * dt / P;
      for (int c = 0; c < NC; ++c) qt[c] = cq[c] + coeff * dxa[c] / s.mass[c / 3];
      const double sigma = xi_bimolec<N>(s.xi, qt, s.mass, dxn);
      double dsigma = 0.0;
      for (int c = 0; c < NC; ++c) dsigma = dsigma + dxn[c] * dt * dt * dxa[c] / (s.mass[c / 3] * P);
      const double dx = sigma / dsigma;
      mult = mult - dx;
      if (fabs(dx) < (double)1.0E-8f || fabs(sigma) < (double)1.0E-10f) {
        ok = 1;
        break;
      }
    }
    res[0] = coeff;
    res[1] = mult;
    res[2] = ok;
    s.shake_fail[t] = ok ? 0 : 1;
  }
  __syncthreads();
  if (res[2] == 0.0) return;
  const double coeff = res[0], mult = res[1], dt = 2.0 * s.half_dt;
  for (int idx = threadIdx.x; idx < P * NC; idx += blockDim.x) {
    const int c = idx % NC;
    const double m = s.mass[c / 3];
    s.q[tb + idx] = s.q[tb + idx] + coeff / m * dxa[c];
    s.p[tb + idx] = s.p[tb + idx] + mult * dt / P * dxa[c];
  }
}

// dxi_act <- dxi at the pre-SHAKE centroid (umbrella mode 1, src/verlet.f90:
// 1047-1049), then RATTLE: p -= (sum dxi.p/m) / (sum dxi^2/m) / P * dxi.
template <int N>
__global__ void split_rattle_kernel(SplitParams s) {
  constexpr int NC = 3 * N;
  __shared__ double dxa[NC], red[kFinishBlock];
  const int t = blockIdx.x, P = s.P;
  const size_t tb = (size_t)t * P * NC;
  if (threadIdx.x == 0) {
    double cq[NC], d[NC];
    for (int c = 0; c < NC; ++c) cq[c] = s.cq[(size_t)t * NC + c];
    xi_bimolec<N>(s.xi, cq, s.mass, d);
    for (int c = 0; c < NC; ++c) {
      dxa[c] = d[c];
      s.dxi[(size_t)t * NC + c] = d[c];
    }
  }
  __syncthreads();
  double c1[1] = {0.0};
  for (int idx = threadIdx.x; idx < P * NC; idx += blockDim.x) {
    const int c = idx % NC;
    c1[0] = c1[0] + dxa[c] * s.p[tb + idx] / s.mass[c / 3];
  }
  block_sum<1>(c1, red);
  double c2 = 0.0;
  for (int c = 0; c < NC; ++c) c2 = c2 + dxa[c] * dxa[c] / s.mass[c / 3];
  const double lambdas = -c1[0] / c2 / P;
  for (int idx = threadIdx.x; idx < P * NC; idx += blockDim.x) s.p[tb + idx] = s.p[tb + idx] + lambdas * dxa[idx % NC];
}

// initial dxi_act of each parent at its current centroid
template <int N>
__global__ void split_parent_init_kernel(SplitParams s) {
  constexpr int NC = 3 * N;
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= s.T) return;
  double cq[NC], d[NC];
  for (int c = 0; c < NC; ++c) {
    double acc = 0.0;
    for (int k = 0; k < s.P; ++k) acc = acc + s.q[((size_t)t * s.P + k) * NC + c];
    cq[c] = acc / s.P;
  }
  xi_bimolec<N>(s.xi, cq, s.mass, d);
  for (int c = 0; c < NC; ++c) s.dxi[(size_t)t * NC + c] = d[c];
  s.shake_fail[t] = 0;
}

// NaN check (src/verlet.f90:1256-1275), transrot (src/transrot.f90:36-237,
// COM velocity and rotation centre with Caracal's total mass P^2 sum m) and
// the potential energy summed over beads, as three kernels:
//   split_moments_kernel  grid (S, T): slice g of trajectory t's (bead, atom)
//                         items -> 15 moment sums (sum w v, sum w x,
//                         sum w x cross v, sum w x x^T), the bead energies
//                         (slice 0), the NaN bits; fixed-order block sums.  Rows l
//                         and P - l of q are equal after the drift, so an item
//                         covers both with the sum of their momenta
//   split_solve_kernel    four lanes per trajectory: the S partials summed in
//                         order, epot, status, and the 3x3 system for the
//                         angular velocity (transrot_quad)
//   split_apply_kernel    every item: p <- m (v - vt - va x (x - xt)),
//                         evaluated as p - m (b + va x x), b = vt - va x xt
// The second moments about Caracal's rotation centre xt come from the raw
// ones by the parallel-axis identity C = S - xt Sx^T - Sx xt^T + W xt xt^T,
// W = sum w.  Traffic: half of q and p read twice, p written once; 1024 x 64 C20H42
// 65, 6 and 64 us.
constexpr int kMomentThreads = 256;
constexpr int kApplyItems = 4 * kMomentThreads;  // items of one block of split_apply_kernel
constexpr int kFinishSums = 16;   // 15 moments + sum of bead energies
constexpr int kMoveDoubles = 10;  // b = vt - va x xt, va, (3 unused), skip flag per trajectory

// slices per trajectory of split_moments_kernel: about 4 items per thread
__host__ __device__ inline int finish_slices(int items) {
  const int s = (items + 4 * kMomentThreads - 1) / (4 * kMomentThreads);
  return s < 1 ? 1 : (s > 16 ? 16 : s);
}

// Warp sum of 16 values per lane as a reduce-scatter butterfly: at each of
// the first four levels a lane keeps half of its values and adds the
// partner's copy of that half (8 + 4 + 2 + 1 adds instead of 16 x 5),
// then one exchange finishes.  Lane l returns the warp sum of value l >> 1.
__device__ inline int64_t warp_sum16(int64_t (&v)[16], int lane) {
#pragma unroll
  for (int level = 0; level < 4; ++level) {
    const int half = 8 >> level;  // values kept per lane after this level
    const bool up = (lane >> (4 - level)) & 1;
#pragma unroll
    for (int j = 0; j < half; ++j) {
      const int64_t keep = up ? v[half + j] : v[j];
      const int64_t give = up ? v[j] : v[half + j];
      v[j] = keep + __shfl_xor_sync(0xffffffffu, give, 16 >> level);
    }
  }
  return v[0] + __shfl_xor_sync(0xffffffffu, v[0], 1);
}

// Moment sums.  In FP64 the 24 operations of an item held the FP64 pipe for 94 of
// 115 us (1024 x 64 C20H42; now 65 us); so a warp takes kWarpItems items per lane at
// a time, brings their q and p under one exponent each as 55-bit integers, and
// forms the products by limbs (fixed_map.cuh): rounded at 2^-55 of the largest
// product, 64 items at a time, and summed exactly before one conversion to FP64.
constexpr int kWarpItems = 2;
__global__ void __launch_bounds__(kMomentThreads, 3) split_moments_kernel(const __grid_constant__ SplitParams s) {
  constexpr int kWarps = kMomentThreads / 32, kGuard = 1;
  __shared__ double wpart[kWarps][kFinishSums];
  __shared__ int wstat[kWarps];
  const int S = gridDim.x, g = blockIdx.x, t = blockIdx.y, P = s.P, N = s.N;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const size_t tb = (size_t)t * P * s.NC;
  const int items = s.U * N;
  const int lo = (int)((long long)items * g / S), hi = (int)((long long)items * (g + 1) / S);
  double total = 0.0;  // of value lane >> 1
  bool bad = false;
  for (int i0 = lo + warp * 32 * kWarpItems; i0 < hi; i0 += kMomentThreads * kWarpItems) {
    double q[kWarpItems][3], p[kWarpItems][3], pt[kWarpItems][3];
    int atom[kWarpItems];  // [k]: + N where the item stands for two rows
    int eq = 0, ep = 0;
#pragma unroll
    for (int k = 0; k < kWarpItems; ++k) {
      const int i = i0 + 32 * k + lane;
      atom[k] = -1;
#pragma unroll
      for (int d = 0; d < 3; ++d) q[k][d] = p[k][d] = pt[k][d] = 0.0;
      if (i < hi) {
        const int l = i / N, a = i - l * N, kt = twin_row(s, l);
        atom[k] = a + (kt != l ? N : 0);
#pragma unroll
        for (int d = 0; d < 3; ++d) {
          q[k][d] = s.q[tb + 3 * (size_t)i + d];
          p[k][d] = s.p[tb + 3 * (size_t)i + d];
          if (kt != l) pt[k][d] = s.p[tb + 3 * (size_t)(kt * N + a) + d];
        }
      }
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        eq = max(eq, exponent_field(q[k][d]));
        ep = max(ep, max(exponent_field(p[k][d]), exponent_field(pt[k][d])));
      }
    }
    eq = __reduce_max_sync(0xffffffffu, eq);
    ep = __reduce_max_sync(0xffffffffu, ep);
    bad = bad || eq == kFixedNan;
    int64_t sp[3] = {0, 0, 0}, sq[3] = {0, 0, 0};
    FixedSum L[3], C[6];
#pragma unroll
    for (int d = 0; d < 3; ++d) L[d] = FixedSum{0, 0};
#pragma unroll
    for (int d = 0; d < 6; ++d) C[d] = FixedSum{0, 0};
#pragma unroll
    for (int k = 0; k < kWarpItems; ++k) {
      const int a = atom[k] < 0 ? 0 : atom[k];  // an empty item is zero in every value
      // the mass (twice it for two rows): mass * 2^-em below 1 as 56 bits
      const Limbs w{s.wfix[2 * a], s.wfix[2 * a + 1]};
      Limbs x[3], wx[3], y[3];
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        const int64_t fq = to_fixed(q[k][d], eq, kGuard);
        const int64_t fp = to_fixed(p[k][d], ep, kGuard + 1) + to_fixed(pt[k][d], ep, kGuard + 1);
        x[d] = to_limbs(fq);
        y[d] = to_limbs(fp);
        FixedSum m{0, 0};
        m.add(x[d], w);
        const int64_t fw = m.value();
        wx[d] = to_limbs(fw);
        sp[d] += fp;
        sq[d] += fw;
      }
      L[0].add(x[1], y[2]);
      L[0].sub(x[2], y[1]);
      L[1].add(x[2], y[0]);
      L[1].sub(x[0], y[2]);
      L[2].add(x[0], y[1]);
      L[2].sub(x[1], y[0]);
      C[0].add(wx[0], x[0]);
      C[1].add(wx[0], x[1]);
      C[2].add(wx[0], x[2]);
      C[3].add(wx[1], x[1]);
      C[4].add(wx[1], x[2]);
      C[5].add(wx[2], x[2]);
    }
    int64_t v[16] = {sp[0], sp[1], sp[2], sq[0], sq[1], sq[2], L[0].value(), L[1].value(), L[2].value(),
                     C[0].value(), C[1].value(), C[2].value(), C[3].value(), C[4].value(), C[5].value(), 0};
    const int64_t sum = warp_sum16(v, lane);
    // units: p 2^(ep - 1078 + guard + 1), q 2^(eq - 1078 + guard), m q the mass's exponent more
    const int up = ep - 1077 + kGuard, uq = eq - 1078 + kGuard, j = lane >> 1, two = 2 * kLimbBits;
    const int ex = j < 3 ? up : j < 6 ? uq + s.wexp : j < 9 ? uq + up + two : 2 * uq + s.wexp + two;
    double r = from_fixed(sum, ex);
    if (eq == kFixedNan || ep == kFixedNan) r = __longlong_as_double(0x7ff8000000000000ll);
    total += r;
  }
  if ((lane & 1) == 0) wpart[warp][lane >> 1] = total;
  if (lane == 0) wstat[warp] = bad ? CR_TRAJ_NONFINITE : 0;
  __syncthreads();
  const size_t slot = (size_t)t * S + g;
  if (threadIdx.x < kFinishSums - 1) {
    double v = 0.0;
    for (int w = 0; w < kWarps; ++w) v += wpart[w][threadIdx.x];
    s.fsum[slot * kFinishSums + threadIdx.x] = v;
  } else if (threadIdx.x == kFinishSums) {
    int st = 0;
    for (int w = 0; w < kWarps; ++w) st |= wstat[w];
    s.fstat[slot] = st;
  }
  // the bead energies, by slice 0's second warp, in order over 32 partial sums
  if (warp == 1) {
    double e = 0.0;
    if (g == 0)
      for (int j = lane; j < P; j += 32) e += s.V[(size_t)t * P + j];
#pragma unroll
    for (int o = 16; o >= 1; o >>= 1) e += __shfl_xor_sync(0xffffffffu, e, o);
    if (lane == 0) s.fsum[slot * kFinishSums + kFinishSums - 1] = e;
  }
}

__global__ void split_solve_kernel(const __grid_constant__ SplitParams s, int S) {
  const int x = blockIdx.x * 8 + threadIdx.x / 4, lane = threadIdx.x & 3;
  const bool real = x < s.T;
  const int t = real ? x : s.T - 1;  // a quad's shuffles need whole warps
  // the partial sums, a quarter per lane, then all of them on every lane
  double part[4] = {0.0, 0.0, 0.0, 0.0}, tot[kFinishSums];
  int status = 0;
  for (int g = 0; g < S; ++g) {
    const size_t slot = (size_t)t * S + g;
#pragma unroll
    for (int j = 0; j < 4; ++j) part[j] += s.fsum[slot * kFinishSums + 4 * lane + j];
    status |= s.fstat[slot];
  }
#pragma unroll
  for (int j = 0; j < kFinishSums; ++j) tot[j] = __shfl_sync(0xffffffffu, part[j & 3], j >> 2, 4);
  double* mv = s.fmove + (size_t)t * kMoveDoubles;
  if (s.transrot) {
    double bb, va;
    const bool ok = transrot_quad([&](int k) { return pick(tot, k); }, lane, s.itm, s.kap, s.N <= 2, bb, va);
    if (real && lane < 3) {
      mv[lane] = bb;
      mv[3 + lane] = va;
    }
    if (real && lane == 0) mv[9] = ok ? 0.0 : 1.0;
    if (!ok) status |= CR_TRAJ_SINGULAR_INERTIA;
  }
  if (!real || lane != 0) return;
  const bool shake_fail = s.constrain && s.shake_fail[t];
  if (shake_fail) status |= CR_TRAJ_SHAKE_FAILED;
  s.epot[t] = tot[15] + (shake_fail ? 100000.0 : 0.0);
  if (status) s.status[t] |= status;
}

__global__ void __launch_bounds__(kMomentThreads) split_apply_kernel(SplitParams s) {
  const int N = s.N, items = s.U * N, t = blockIdx.x;
  double mv[6];  // in registers: the stores to p below could be to fmove for all the compiler knows
#pragma unroll
  for (int k = 0; k < 6; ++k) mv[k] = s.fmove[(size_t)t * kMoveDoubles + k];
  if (s.fmove[(size_t)t * kMoveDoubles + 9] != 0.0) return;
  const double* q = s.q + (size_t)t * s.P * s.NC;
  double* p = s.p + (size_t)t * s.P * s.NC;
  const int lo = blockIdx.y * kApplyItems, hi = min(lo + kApplyItems, items);
  for (int i = lo + threadIdx.x; i < hi; i += kMomentThreads) {
    const int l = i / N, a = i - l * N, k = twin_row(s, l);
    const double* qq = q + 3 * (size_t)i;
    const double w = s.mass[a];
    const double u[3] = {fma(mv[4], qq[2], fma(-mv[5], qq[1], mv[0])), fma(mv[5], qq[0], fma(-mv[3], qq[2], mv[1])),
                         fma(mv[3], qq[1], fma(-mv[4], qq[0], mv[2]))};
    double* pa = p + 3 * (size_t)i;
    double* pb = p + 3 * (size_t)(k * N + a);
    double x[3], y[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      x[d] = pa[d];
      y[d] = pb[d];
    }
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      const double r = fma(-w, u[d], x[d]);
      pa[d] = r;
      if (k != l) pb[d] = same_bits(x[d], y[d]) ? r : fma(-w, u[d], y[d]);
    }
  }
}

// nhc (src/nhc.f90:35-171) on one trajectory per block: the kinetic sum
// p.p/(2m)/P/P over beads and atoms, the chain, one scale of every momentum.
__global__ void __launch_bounds__(kFinishBlock) split_nhc_kernel(SplitParams s) {
  __shared__ double red[kFinishBlock];
  __shared__ double ssc;
  const int t = blockIdx.x, P = s.P, N = s.N, NC = s.NC;
  const size_t tb = (size_t)t * P * NC;
  double ek[1] = {0.0};
  for (int idx = threadIdx.x; idx < P * N; idx += blockDim.x) {
    const double* pp = s.p + tb + 3 * (size_t)idx;
    ek[0] = fma(pp[0] * pp[0] + pp[1] * pp[1] + pp[2] * pp[2], s.inv_mass[idx % N], ek[0]);
  }
  ek[0] *= 0.5 / ((double)P * P);
  block_sum<1>(ek, red);
  if (threadIdx.x == 0) {
    double v[4];
    for (int k = 0; k < 4; ++k) v[k] = s.vnh[4 * (size_t)t + k];
    ssc = nhc_scale(s.nhc, ek[0], v);
    for (int k = 0; k < 4; ++k) s.vnh[4 * (size_t)t + k] = v[k];
  }
  __syncthreads();
  const double sc = ssc;
  for (int x = threadIdx.x; x < P * NC; x += blockDim.x) s.p[tb + x] = sc * s.p[tb + x];
}

// NpT with the Berendsen barostat (src/verlet.f90:1111-1151), one block per
// trajectory, after the second half kick: the pressure from the beads' virial
// traces (the reference's kinetic stress tensor stays zero, so
// p = (1/V)(0 - tr W)/3 with V the box at the start of the step), the scale
// (1 + rate (p - p0))^(1/3) with rate = dt compress / taupres, then the box
// and every bead's coordinates scaled.  A non-finite scale reaches the
// coordinates and the step's NaN check.
struct NptStep {
  double* box;        // [T][3] edges, bohr
  double* press;      // [T][2] the step's pressure and the running sum, a.u.
  const double* vir;  // [T][P] virial trace per bead
  double pressure;    // target, a.u.
  double rate;        // dt compress / taupres
};
__global__ void __launch_bounds__(kFinishBlock) split_berendsen_kernel(const __grid_constant__ SplitParams s, NptStep n) {
  const int t = blockIdx.x, P = s.P, NC = s.NC;
  __shared__ double scale;
  if (threadIdx.x < 32) {
    double w = 0.0;  // 32 partial sums, added as a tree
    for (int b = threadIdx.x; b < P; b += 32) w += n.vir[(size_t)t * P + b];
#pragma unroll
    for (int o = 16; o >= 1; o >>= 1) w += __shfl_xor_sync(0xffffffffu, w, o);
    if (threadIdx.x == 0) {
      double* L = n.box + 3 * (size_t)t;
      const double factor = 1.0 / (L[0] * L[1] * L[2]);
      const double pr = (factor * (0.0 - w)) / 3.0;
      const double sc = pow(1.0 + n.rate * (pr - n.pressure), 1.0 / 3.0);
      for (int k = 0; k < 3; ++k) L[k] = L[k] * sc;
      n.press[2 * (size_t)t] = pr;
      n.press[2 * (size_t)t + 1] += pr;  // press_avg (src/verlet.f90:1171-1173)
      scale = sc;
    }
  }
  __syncthreads();
  // rows l and P - l of q are equal after the drift
  const double sc = scale;
  double* q = s.q + (size_t)t * P * NC;
  const int nq = s.U * NC;
#pragma unroll 4
  for (int i = threadIdx.x; i < nq; i += kFinishBlock) {
    const int l = i / NC, k = twin_row(s, l);
    const double x = q[i] * sc;
    q[i] = x;
    if (k != l) q[i + (k - l) * NC] = x;
  }
}

__global__ void split_advance_kernel(int* istep) { *istep += 1; }
__global__ void advance_by_kernel(int* istep, int n) { *istep += n; }

// mdinit-style initial state for any atom count: per (trajectory, bead, pair).
__global__ void split_init_positions_kernel(int T, int P, int NC, uint32_t seed, uint32_t traj0, const double* q0,
                                            double sigma, double* q) {
  const int npair = (NC + 1) / 2;
  const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= (long long)T * P * npair) return;
  const int ip = (int)(idx % npair);
  const long long b = idx / npair;
  const int t = (int)(b / P), k = (int)(b % P);
  double z0, z1;
  normal_pair(seed, traj0 + (uint32_t)t, (uint32_t)ip, (uint32_t)k, 0u, TAG_BEAD_JITTER, z0, z1);
  const int c = 2 * ip;
  q[(size_t)b * NC + c] = q0[c] + sigma * z0;
  if (c + 1 < NC) q[(size_t)b * NC + c + 1] = q0[c + 1] + sigma * z1;
}

__global__ void split_init_momenta_kernel(int T, int P, int NC, uint32_t seed, uint32_t traj0, const double* sig,
                                          int zero, uint32_t draw, double* p) {
  const int npair = (NC + 1) / 2;
  const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= (long long)T * P * npair) return;
  const int ip = (int)(idx % npair);
  const long long b = idx / npair;
  const int t = (int)(b / P), k = (int)(b % P);
  const int c = 2 * ip;
  double z0 = 0.0, z1 = 0.0;
  if (!zero) normal_pair(seed, traj0 + (uint32_t)t, (uint32_t)ip, (uint32_t)k, draw, TAG_INIT_MOMENTA, z0, z1);
  p[(size_t)b * NC + c] = z0 * sig[c / 3];
  if (c + 1 < NC) p[(size_t)b * NC + c + 1] = z1 * sig[(c + 1) / 3];
}

// epot[t] = sum of the bead energies (after a force evaluation outside a step)
__global__ void split_sum_beads_kernel(int T, int P, const double* V, double* epot) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= T) return;
  double s = 0.0;
  for (int k = 0; k < P; ++k) s += V[(size_t)t * P + k];
  epot[t] = s;
}


// Umbrella bias outside a step (mdinit's forces, src/mdinit.f90:96-100): one
// block per trajectory.
template <int N>
__global__ void split_umbrella_kernel(SplitParams s) {
  constexpr int NC = 3 * N;
  __shared__ double cq[NC], bias[NC];
  const int t = blockIdx.x, P = s.P;
  const size_t tb = (size_t)t * P * NC;
  for (int c = threadIdx.x; c < NC; c += blockDim.x) {
    double acc = 0.0;
    for (int k = 0; k < P; ++k) acc = acc + s.q[tb + (size_t)k * NC + c];
    cq[c] = acc / P;
  }
  __syncthreads();
  if (threadIdx.x < 4) {
    const double xi = umbrella_bias<N>(s.xi, s.umb, cq, s.umb.center[t], s.umb.kforce[t], threadIdx.x, bias);
    if (threadIdx.x == 0 && *s.umb.sampling) umbrella_sample(s.umb, (size_t)t, xi);
  }
  __syncthreads();
  for (int idx = threadIdx.x; idx < P * NC; idx += blockDim.x) s.f[tb + idx] += bias[idx % NC];
}

}  // namespace cr
