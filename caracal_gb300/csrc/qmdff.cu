// QMDFF force field: host set-up (parameter tables, the warp term schedule)
// and the per-bead energy/gradient kernel behind cr_qmdff_* (C-ABI).
#include <algorithm>
#include <cmath>
#include <cstring>
#include <map>
#include <string>
#include <tuple>
#include <utility>
#include <vector>

#include "host_util.h"
#include "qmdff_host.h"

namespace {

using cr::qmdff::kVAngl;
using cr::qmdff::kVBond;
using cr::qmdff::kVPair;
using cr::qmdff::kVTors;

// Segments of one kind (qmdff.cuh, Schedule): the terms cut into segments, and for
// each coordinate the list of what a segment holds for it.
struct ScheduleHost {
  std::vector<int4> seg;
  std::vector<int2> round;
  std::vector<unsigned short> dst, ent;
};
void schedule_kind(bool mixed, int kind, int arity, const std::vector<int>& atoms, int natoms, ScheduleHost& h) {
  const int C = cr::qmdff::segment_terms(mixed, kind), zero = cr::qmdff::buffer_values(mixed);
  const int nterm = (int)atoms.size() / arity;
  for (int t0 = 0; t0 < nterm; t0 += C) {
    const int nt = std::min(nterm - t0, C);
    // per atom the entries of its x component (y, z: C and 2 C further)
    std::vector<std::vector<int>> list((size_t)natoms);
    for (int i = 0; i < nt; ++i)
      for (int a = 0; a < arity; ++a) {
        std::vector<int>& l = list[(size_t)atoms[(size_t)(t0 + i) * arity + a]];
        if (arity == 2) {  // the first atom's gradient (mixed-form bonds: hi, lo), the second's its negative
          const int sign = a == 1 ? cr::qmdff::kNegate : 0;
          l.push_back(i | sign);
          if (mixed && kind == 0) l.push_back((3 * C + i) | sign);
        } else {
          l.push_back(3 * a * C + i);
        }
      }
    std::vector<int> by((size_t)natoms);
    for (int a = 0; a < natoms; ++a) by[(size_t)a] = a;
    std::stable_sort(by.begin(), by.end(), [&](int x, int y) { return list[(size_t)x].size() > list[(size_t)y].size(); });
    int used = 0;  // coordinates with a list
    while (used < natoms && !list[(size_t)by[(size_t)used]].empty()) ++used;
    used *= 3;
    const int rounds = (used + 31) / 32;
    h.seg.push_back(make_int4(t0, nt, (int)h.round.size(), rounds));
    for (int r = 0; r < rounds; ++r) {
      const int steps = (int)list[(size_t)by[(size_t)(32 * r / 3)]].size();
      h.round.push_back(make_int2((int)h.ent.size(), steps));
      for (int x = 32 * r; x < 32 * r + 32; ++x)
        h.dst.push_back((unsigned short)(x < used ? 3 * by[(size_t)(x / 3)] + x % 3 : cr::qmdff::kNoDst));
      for (int k = 0; k < steps; ++k)
        for (int x = 32 * r; x < 32 * r + 32; ++x) {
          const std::vector<int>* l = x < used ? &list[(size_t)by[(size_t)(x / 3)]] : nullptr;
          h.ent.push_back((unsigned short)(l && k < (int)l->size() ? (*l)[(size_t)k] + (x % 3) * C : zero));
        }
    }
  }
}

// Pair terms: the circle method splits all atom pairs of n atoms (n even; a
// dummy atom for odd n) into n-1 perfect matchings; the pairs of one
// matching touch disjoint atoms, so each matching is one single-colour batch
// (split in 32-lane pieces when n > 64).
void schedule_pairs(int nterm, const std::vector<int>& atoms, int natoms, std::vector<int>& slot, int& nbatch) {
  const int m = natoms + (natoms & 1);  // players, even
  std::vector<std::vector<int>> rounds((size_t)(m > 1 ? m - 1 : 1));
  for (int t = 0; t < nterm; ++t) {
    int i = atoms[(size_t)2 * t], j = atoms[(size_t)2 * t + 1];
    if (i > j) std::swap(i, j);
    // round r holds (r, m-1) and the pairs (r + k, r - k) mod (m-1), i.e. the
    // pairs with i + j = 2r (mod m-1); m/2 is the inverse of 2 modulo m-1
    const int r = (j == m - 1) ? i : (int)(((long long)(i + j) * (m / 2)) % (m - 1));
    rounds[(size_t)r].push_back(t);
  }
  nbatch = 0;
  for (const auto& rd : rounds) {
    for (size_t k0 = 0; k0 < rd.size(); k0 += 32) {
      for (int l = 0; l < 32; ++l) {
        const size_t k = k0 + (size_t)l;
        slot.push_back(k < rd.size() ? rd[k] : -1);
      }
      ++nbatch;
    }
  }
}

// A force field's tables in one device allocation and one copy: a fit makes a
// force field per evaluation, and some thirty allocations, copies and frees took
// 1.0 of its 4.6 ms (2000 C20H42 geometries).
struct Arena {
  std::vector<unsigned char> bytes;
  std::vector<std::pair<const void**, size_t>> slots;
  template <class T>
  void add(const std::vector<T>& h, const T** d) {
    *d = nullptr;
    if (h.empty()) return;
    const size_t at = (bytes.size() + 255) / 256 * 256, n = h.size() * sizeof(T);
    bytes.resize(at + n);
    std::memcpy(bytes.data() + at, h.data(), n);
    slots.emplace_back(reinterpret_cast<const void**>(d), at);
  }
  int upload(cr_qmdff* ff) {
    if (bytes.empty()) return CR_OK;
    void* p = nullptr;
    CR_TRY_CUDA(cudaMalloc(&p, bytes.size()));
    ff->allocs.push_back(p);
    CR_TRY_CUDA(cudaMemcpy(p, bytes.data(), bytes.size(), cudaMemcpyHostToDevice));
    for (const auto& x : slots) *x.first = static_cast<unsigned char*>(p) + x.second;
    return CR_OK;
  }
};

template <class T>
std::vector<float> to_float(const std::vector<T>& v) {
  std::vector<float> o(v.size());
  for (size_t i = 0; i < v.size(); ++i) o[i] = (float)v[i];
  return o;
}

}  // namespace

namespace cr {

// MINB: blocks of kQmdffWarps warps kept resident per SM (the register cap
// follows: 65536 / (MINB * block) per thread).  The FP64 form trades spills for
// occupancy differently from the mixed form; the autotuner below picks.  Mixed: a
// warp per bead; FP64: a block per bead (kTeam).
constexpr int kQmdffThreads = kQmdffWarps * 32, kTeamThreads = qmdff::kTeam * 32;
template <bool MIXED, int MINB, int MODE = qmdff::kFree>
__global__ void __launch_bounds__(MIXED ? kQmdffThreads : kTeamThreads, MINB)
    qmdff_egrad_kernel(qmdff::Dev D, int nbeads, BeadRows rows, const double* q, double* e, double* g) {
  extern __shared__ double qsm[];
  const int n3 = 3 * D.n;
  if constexpr (MIXED) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    void* ws = qsm + (size_t)warp * (qmdff::warp_smem_bytes(D.n) / sizeof(double));
    for (int b = blockIdx.x * kQmdffWarps + warp; b < nbeads; b += gridDim.x * kQmdffWarps) {
      const size_t r = rows.row(b), r2 = rows.twin(b);
      const double v = qmdff::warp_egrad<MODE>(D, ws, q + r * n3, g + r * n3, g + r2 * n3, lane, r, r2);
      if (lane == 0) {
        e[r] = v;
        if (r2 != r) e[r2] = v;
      }
      __syncwarp();
    }
  } else {
    for (int b = blockIdx.x; b < nbeads; b += gridDim.x) {
      const size_t r = rows.row(b), r2 = rows.twin(b);
      const double* qb = q + r * n3;
      for (int a = threadIdx.x; a < n3; a += kTeamThreads) qsm[a] = qb[a];
      const double v = qmdff::team_egrad<MODE>(D, qsm, g + r * n3, g + r2 * n3, r, r2);
      if (threadIdx.x == 0) {
        e[r] = v;
        if (r2 != r) e[r2] = v;
      }
      __syncthreads();
    }
  }
}

// Energy, gradient and Hessian-vector product H w per bead (plain form, dual
// coordinates), a block per bead (hvp_threads); dew[b] = w . grad E.
__global__ void __launch_bounds__(kTeamThreads)
    qmdff_hvp_kernel(qmdff::Dev D, int nbeads, BeadRows rows, const double* q, const double* w, double* e, double* g,
                     double* hw, double* dew) {
  extern __shared__ double qsm[];
  const int n3 = 3 * D.n;
  for (int b = blockIdx.x; b < nbeads; b += gridDim.x) {
    const size_t r = rows.row(b), r2 = rows.twin(b);
    const double* qb = q + r * n3;
    const double* wb = w + r * n3;
    for (int a = threadIdx.x; a < n3; a += blockDim.x) {
      qsm[a] = qb[a];
      qsm[n3 + a] = wb[a];
    }
    double de = 0.0;
    const double v = qmdff::team_hvp(D, qsm, g ? g + r * n3 : nullptr, g ? g + r2 * n3 : nullptr, hw + r * n3, hw + r2 * n3, de);
    if (threadIdx.x == 0) {
      if (e) e[r] = e[r2] = v;
      if (dew) dew[r] = dew[r2] = de;
    }
    __syncthreads();
  }
}

// Per bead b and linear parameter t: out[b][t] = alpha_b (v_b . grad E_t|unit)
// + beta_b E_t|unit (alpha = 1, beta = 0 where the weights are NULL), a block per bead;
// out's row b: evaluation b0 + b, twice where it stands for two beads.
__global__ void __launch_bounds__(kTeamThreads)
    qmdff_vjp_kernel(qmdff::Dev D, qmdff::Tables<double> U, BeadRows rows, size_t b0, int nlin, const double* q,
                     const double* v, const double* alpha, const double* beta, double* out) {
  extern __shared__ double qsm[];
  const int n3 = 3 * D.n;
  const size_t b = rows.row(b0 + blockIdx.x);
  const double m = rows.twin(b0 + blockIdx.x) != b ? 2.0 : 1.0;
  for (int a = threadIdx.x; a < n3; a += kTeamThreads) {
    qsm[a] = q[b * n3 + a];
    qsm[n3 + a] = v[b * n3 + a];
  }
  __syncthreads();
  qmdff::team_param_vjp(D, U, qsm, qsm + n3, m * (alpha ? alpha[b] : 1.0), m * (beta ? beta[b] : 0.0),
                        out + (size_t)blockIdx.x * nlin);
}

// acc[t] += scale * sum_b in[b][t]: 32 columns per block, eight rows at a time in
// eight partial sums, added in order (deterministic).
constexpr int kSumCols = 32, kSumRows = 8;
__global__ void __launch_bounds__(kSumCols * kSumRows) sum_rows_kernel(int nrows, int ncols, const double* in, double scale, double* acc) {
  __shared__ double part[kSumRows][kSumCols];
  const int x = threadIdx.x, y = threadIdx.y, t = blockIdx.x * kSumCols + x;
  double s = 0.0;
  if (t < ncols) {
#pragma unroll 4
    for (int r = y; r < nrows; r += kSumRows) s += in[(size_t)r * ncols + t];
  }
  part[y][x] = s;
  __syncthreads();
  if (y == 0 && t < ncols) {
    s = 0.0;
    for (int k = 0; k < kSumRows; ++k) s += part[k][x];
    acc[t] += scale * s;
  }
}

}  // namespace cr

namespace {

// A kernel's limit on dynamic shared memory is the process's, whichever force field
// asks: always the most that a block may take, so that none lowers what another (in
// another thread) is about to launch.
template <class K>
int allow_smem(K kernel, size_t bytes) {
  constexpr int kMost = 227 * 1024;
  if (bytes > (size_t)kMost) return cr_set_error(CR_ERR_CUDA, cudaGetErrorString(cudaErrorInvalidValue));
  CR_TRY_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kMost));
  return CR_OK;
}

// Threads of a bead's block in the Hessian product: warps for the terms of the
// largest kind and for the coordinates, kTeam at most. With eight warps a molecule of a
// few atoms leaves all but one or two at the barriers, and registers let an SM hold
// one such block only: host calls, C2H6 65 536 beads 22.1 -> 7.4 ms, C4H10 8192
// beads 3.05 -> 1.19 ms, C6H14 (four warps) and larger unchanged.
int hvp_threads(const cr_qmdff* ff) {
  int most = 3 * ff->n;
  for (int k = 0; k < 4; ++k) most = std::max(most, ff->nterm[k]);
  return 32 * std::min((most + 31) / 32, cr::qmdff::kTeam);
}

}  // namespace

int qmdff_hvp_launch(const cr_qmdff* ff, const double* d_q, const double* d_w, int nbeads, double* d_e, double* d_g,
                     double* d_hw, double* d_dew, cudaStream_t s, cr::BeadRows rows) {
  if (ff->nterm[4] > 0) return cr_set_error(CR_ERR_UNSUPPORTED, "second derivatives of H/halogen-bond terms are not built");
  const size_t smem = cr::qmdff::team_hvp_smem_bytes(ff->n);
  if (const int rc = allow_smem(cr::qmdff_hvp_kernel, smem)) return rc;
  if (nbeads == 0) return CR_OK;
  const int grid = std::min(nbeads, 1 << 20);
  cr::qmdff_hvp_kernel<<<grid, hvp_threads(ff), smem, s>>>(ff->dev, nbeads, rows, d_q, d_w, d_e, d_g, d_hw, d_dew);
  CR_TRY_CUDA(cudaGetLastError());
  return CR_OK;
}

int qmdff_nlin(const cr_qmdff* ff) { return ff->nterm[0] + ff->nterm[1] + ff->nterm[2] + ff->nterm[3]; }

int qmdff_vjp_launch(const cr_qmdff* ff, const double* d_q, const double* d_v, int nbeads, const double* d_alpha,
                     const double* d_beta, double scale, double* d_scratch, int scratch_beads, double* d_acc,
                     cudaStream_t s, cr::BeadRows rows) {
  if (ff->nterm[4] > 0) return cr_set_error(CR_ERR_UNSUPPORTED, "parameter gradients of H/halogen-bond terms are not built");
  const int nlin = qmdff_nlin(ff);
  const size_t smem = (size_t)2 * 3 * ff->n * sizeof(double);
  if (const int rc = allow_smem(cr::qmdff_vjp_kernel, smem)) return rc;
  if (nlin == 0) return CR_OK;
  for (int b0 = 0; b0 < nbeads; b0 += scratch_beads) {
    const int nb = std::min(scratch_beads, nbeads - b0);
    cr::qmdff_vjp_kernel<<<nb, cr::kTeamThreads, smem, s>>>(ff->dev, ff->unit, rows, (size_t)b0, nlin, d_q, d_v, d_alpha,
                                                            d_beta, d_scratch);
    CR_TRY_CUDA(cudaGetLastError());
    cr::sum_rows_kernel<<<(nlin + cr::kSumCols - 1) / cr::kSumCols, dim3(cr::kSumCols, cr::kSumRows), 0, s>>>(nb, nlin, d_scratch, scale, d_acc);
    CR_TRY_CUDA(cudaGetLastError());
  }
  return CR_OK;
}

namespace {

using QmdffKernel = void (*)(cr::qmdff::Dev, int, cr::BeadRows, const double*, double*, double*);
constexpr int kVariants = 3;
// [precision][variant]: blocks per SM 1 / 2 / 3 (FP64), 5 / 7 / 8 (mixed:
// its stalls are on shared memory and L1, which warps hide better than registers:
// C20H42 1024 x 64, per step 1434 us with 6 blocks, 1282 with 7, 1256 with 8; molecules
// whose shared memory allows fewer are no slower for the cap: against the kernels before,
// 4 to 6 blocks, C100H202 512 beads 1.33 -> 0.87 ms, C200H402 256 beads 4.92 -> 2.91)
const QmdffKernel kKernels[2][kVariants] = {
    {cr::qmdff_egrad_kernel<false, 1>, cr::qmdff_egrad_kernel<false, 2>, cr::qmdff_egrad_kernel<false, 3>},
    {cr::qmdff_egrad_kernel<true, 5>, cr::qmdff_egrad_kernel<true, 7>, cr::qmdff_egrad_kernel<true, 8>}};
constexpr int kDefaultVariant = 1;
// the force field's periodic box, and NpT (per-trajectory boxes and the
// virial): one variant per form each
const QmdffKernel kBoxKernels[2] = {cr::qmdff_egrad_kernel<false, 2, cr::qmdff::kBox>,
                                    cr::qmdff_egrad_kernel<true, 7, cr::qmdff::kBox>};
const QmdffKernel kNptKernels[2] = {cr::qmdff_egrad_kernel<false, 2, cr::qmdff::kNpt>,
                                    cr::qmdff_egrad_kernel<true, 7, cr::qmdff::kNpt>};
constexpr int kTuneMinBeads = 2048;  // smaller batches keep the default

// Threads, blocks and dynamic shared memory of the force kernel's forms.
int egrad_threads(int prec) { return prec == 1 ? cr::kQmdffThreads : cr::kTeamThreads; }
int egrad_grid(int prec, int nbeads) {
  return std::min(prec == 1 ? (nbeads + kQmdffWarps - 1) / kQmdffWarps : nbeads, 1 << 20);
}
size_t egrad_smem(int prec, int n) {
  return prec == 1 ? (size_t)kQmdffWarps * cr::qmdff::warp_smem_bytes(n) : cr::qmdff::team_smem_bytes(n);
}

int allow_egrad_smem(int prec, size_t smem) {
  if (smem <= 48 * 1024) return CR_OK;
  int rc = allow_smem(kBoxKernels[prec], smem);
  for (int v = 0; v < kVariants && rc == CR_OK; ++v) rc = allow_smem(kKernels[prec][v], smem);
  return rc;
}

int launch_dev(const cr::qmdff::Dev& D, int prec, int v, cr::BeadRows rows, const double* d_q, int nbeads, double* d_e, double* d_g,
               cudaStream_t s) {
  const size_t smem = egrad_smem(prec, D.n);
  const int grid = egrad_grid(prec, nbeads);
  const QmdffKernel k = D.periodic ? kBoxKernels[prec] : kKernels[prec][v];
  k<<<grid, egrad_threads(prec), smem, s>>>(D, nbeads, rows, d_q, d_e, d_g);
  CR_TRY_CUDA(cudaGetLastError());
  return CR_OK;
}

int launch_variant(const cr_qmdff* ff, int prec, int v, cr::BeadRows rows, const double* d_q, int nbeads, double* d_e, double* d_g,
                   cudaStream_t s) {
  return launch_dev(ff->dev, prec, v, rows, d_q, nbeads, d_e, d_g, s);
}

// The NpT instantiation with the launch's boxes and virial array.
int launch_npt(const cr_qmdff* ff, int prec, const QmdffNpt& npt, cr::BeadRows rows, const double* d_q, int nbeads, double* d_e,
               double* d_g, cudaStream_t s) {
  cr::qmdff::Dev D = ff->dev;
  D.tbox = npt.tbox;
  D.tbox_beads = npt.beads_per_box;
  D.vir = npt.vir;
  const size_t smem = egrad_smem(prec, D.n);
  if (smem > 48 * 1024)
    if (const int rc = allow_smem(kNptKernels[prec], smem)) return rc;
  if (nbeads <= 0) return CR_OK;
  const int grid = egrad_grid(prec, nbeads);
  kNptKernels[prec]<<<grid, egrad_threads(prec), smem, s>>>(D, nbeads, rows, d_q, d_e, d_g);
  CR_TRY_CUDA(cudaGetLastError());
  return CR_OK;
}

// The force kernel over a subset of the term kinds (bit k of mask: kind k =
// bonds, angles, torsions, NCI pairs, H/halogen bonds), with or without
// E_zero: the pieces of Caracal's QMDFF call site (src/gradient.f90:341-358).
// The masked kinds' segments are left out of a copy of the schedule.
int qmdff_launch_kinds(const cr_qmdff* ff, unsigned mask, bool ezero, const double* d_q, int nbeads, double* d_e,
                       double* d_g, int precision, cudaStream_t s) {
  if (precision != CR_PREC_MIXED && precision != CR_PREC_FP64) return cr_set_error(CR_ERR_ARG, "unknown precision");
  const int prec = precision == CR_PREC_MIXED ? 1 : 0;
  const size_t smem = egrad_smem(prec, ff->n);
  if (const int rc = allow_egrad_smem(prec, smem)) return rc;
  if (nbeads <= 0) return CR_OK;
  cr::qmdff::Dev D = ff->dev;
  for (int p = 0; p < 2; ++p)
    for (int k = 0; k < cr::qmdff::kKinds; ++k)
      if (!((mask >> k) & 1u)) {
        D.sched[p].seg1[k] = D.sched[p].seg0[k];
        if (k == 3) D.sched[p].npair = 0;
      }
  if (!ezero) D.e_zero = 0.0;
  const int v = ff->variant[prec] >= 0 ? ff->variant[prec] : kDefaultVariant;
  return launch_dev(D, prec, v, cr::all_rows(), d_q, nbeads, d_e, d_g, s);
}

// Host-array call of a kind subset: e, g overwritten, or accumulated into.
int qmdff_host_kinds(cr_qmdff* ff, unsigned mask, bool ezero, bool accumulate, const double* xyz, int nbeads,
                     double* e, double* g, int precision) {
  if (!ff) return cr_set_error(CR_ERR_ARG, "NULL force field");
  if (nbeads < 0 || (nbeads > 0 && (!xyz || !e || !g))) return cr_set_error(CR_ERR_ARG, "bad egrad arguments");
  if (nbeads == 0) return CR_OK;
  const size_t nq = (size_t)3 * ff->n * nbeads;
  double *d_q = nullptr, *d_e = nullptr, *d_g = nullptr;
  CR_TRY_CUDA(cudaMalloc(&d_q, nq * sizeof(double)));
  cudaError_t e1 = cudaMalloc(&d_e, (size_t)nbeads * sizeof(double));
  cudaError_t e2 = cudaMalloc(&d_g, nq * sizeof(double));
  std::vector<double> pe, pg;
  int rc = CR_OK;
  if (e1 != cudaSuccess || e2 != cudaSuccess) {
    rc = cr_set_error(CR_ERR_CUDA, "cudaMalloc failed in the QMDFF term call");
  } else if (cudaMemcpy(d_q, xyz, nq * sizeof(double), cudaMemcpyHostToDevice) != cudaSuccess) {
    rc = cr_set_error(CR_ERR_CUDA, "copy of xyz failed");
  } else if ((rc = qmdff_launch_kinds(ff, mask, ezero, d_q, nbeads, d_e, d_g, precision, nullptr)) == CR_OK) {
    double* oe = e;
    double* og = g;
    if (accumulate) {
      pe.resize((size_t)nbeads);
      pg.resize(nq);
      oe = pe.data();
      og = pg.data();
    }
    if (cudaMemcpy(oe, d_e, (size_t)nbeads * sizeof(double), cudaMemcpyDeviceToHost) != cudaSuccess ||
        cudaMemcpy(og, d_g, nq * sizeof(double), cudaMemcpyDeviceToHost) != cudaSuccess) {
      rc = cr_set_error(CR_ERR_CUDA, "copy of results failed");
    } else if (accumulate) {
      for (int b = 0; b < nbeads; ++b) e[b] += pe[(size_t)b];
      for (size_t x = 0; x < nq; ++x) g[x] += pg[x];
    }
  }
  cudaFree(d_q);
  cudaFree(d_e);
  cudaFree(d_g);
  return rc;
}

}  // namespace

// Autotuner: the first launch with at least kTuneMinBeads beads outside a
// stream capture runs one untimed warm-up launch, then times every variant
// once on the caller's data (each writes the same outputs) and keeps the
// fastest for this force field and form.
int qmdff_launch(const cr_qmdff* ff_c, const double* d_q, int nbeads, double* d_e, double* d_g, int precision,
                 cudaStream_t s, const QmdffNpt* npt, cr::BeadRows rows) {
  cr_qmdff* ff = const_cast<cr_qmdff*>(ff_c);
  if (precision != CR_PREC_MIXED && precision != CR_PREC_FP64) return cr_set_error(CR_ERR_ARG, "unknown precision");
  const int prec = precision == CR_PREC_MIXED ? 1 : 0;
  if (npt) return launch_npt(ff, prec, *npt, rows, d_q, nbeads, d_e, d_g, s);
  const size_t smem = egrad_smem(prec, ff->n);
  // the attribute is set even for nbeads = 0, so a caller can prepare the
  // kernels before a stream capture
  if (const int rc = allow_egrad_smem(prec, smem)) return rc;
  if (nbeads <= 0) return CR_OK;
  int choice = ff->variant[prec];
  if (choice < 0) {
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    CR_TRY_CUDA(cudaStreamIsCapturing(s, &cap));
    if (nbeads >= kTuneMinBeads && cap == cudaStreamCaptureStatusNone) {
      cudaEvent_t a, b;
      CR_TRY_CUDA(cudaEventCreate(&a));
      CR_TRY_CUDA(cudaEventCreate(&b));
      float best = 0.f;
      // one untimed launch first: the first launch of a kernel pays for
      // module load and cold caches, which would count against variant 0
      int rc0 = launch_variant(ff, prec, 0, rows, d_q, nbeads, d_e, d_g, s);
      if (rc0) {
        cudaEventDestroy(a);
        cudaEventDestroy(b);
        return rc0;
      }
      for (int v = 0; v < kVariants; ++v) {
        cudaEventRecord(a, s);
        int rc = launch_variant(ff, prec, v, rows, d_q, nbeads, d_e, d_g, s);
        if (rc) {
          cudaEventDestroy(a);
          cudaEventDestroy(b);
          return rc;
        }
        cudaEventRecord(b, s);
        CR_TRY_CUDA(cudaEventSynchronize(b));
        float ms = 0.f;
        cudaEventElapsedTime(&ms, a, b);
        ff->tune_ms[prec][v] = ms;
        if (v == 0 || ms < best) {
          best = ms;
          choice = v;
        }
      }
      cudaEventDestroy(a);
      cudaEventDestroy(b);
      ff->variant[prec] = choice;
      return CR_OK;  // the last variant's outputs equal the chosen one's
    }
    choice = kDefaultVariant;
  }
  return launch_variant(ff, prec, choice, rows, d_q, nbeads, d_e, d_g, s);
}

extern "C" {

int cr_qmdff_destroy(cr_qmdff* ff) {
  if (!ff) return CR_OK;
  for (void* p : ff->allocs) cudaFree(p);
  delete ff;
  return CR_OK;
}

int cr_qmdff_create(const cr_qmdff_def* d, cr_qmdff** out) {
  if (!d || !out) return cr_set_error(CR_ERR_ARG, "NULL argument");
  *out = nullptr;
  const int n = d->natoms;
  if (n < 1 || n > cr::qmdff::kMaxAtoms) return cr_set_error(CR_ERR_ARG, "natoms must be 1..1024");
  if (d->nbond < 0 || d->nangl < 0 || d->ntors < 0 || d->nnci < 0)
    return cr_set_error(CR_ERR_ARG, "negative term count");
  if (!d->at || !d->q || !d->rad || (d->nbond && (!d->bond || !d->vbond)) || (d->nangl && (!d->angl || !d->vangl)) ||
      (d->ntors && (!d->tors || !d->vtors)) ||
      (d->nnci && (!d->nci || !d->r0ab || !d->zab || !d->r0094 || !d->sr42 || !d->c66ab)))
    return cr_set_error(CR_ERR_ARG, "missing force-field array");
  for (int i = 0; i < n; ++i)
    if (d->at[i] < 1 || d->at[i] > 94) return cr_set_error(CR_ERR_ARG, "element number out of 1..94");
  auto atom_ok = [&](int a) { return a >= 1 && a <= n; };
  for (int m = 0; m < 2 * d->nbond; ++m)
    if (!atom_ok(d->bond[m])) return cr_set_error(CR_ERR_ARG, "bond atom out of range");
  for (int m = 0; m < 3 * d->nangl; ++m)
    if (!atom_ok(d->angl[m])) return cr_set_error(CR_ERR_ARG, "angle atom out of range");
  for (int m = 0; m < d->ntors; ++m) {
    for (int a = 0; a < 4; ++a)
      if (!atom_ok(d->tors[6 * m + a])) return cr_set_error(CR_ERR_ARG, "torsion atom out of range");
    const int nt = d->tors[6 * m + 4];
    if (d->tors[6 * m + 5] != 2 && (nt < 0 || nt > 4)) return cr_set_error(CR_ERR_ARG, "torsion term count not 0..4");
  }
  for (int m = 0; m < d->nnci; ++m) {
    if (!atom_ok(d->nci[3 * m]) || !atom_ok(d->nci[3 * m + 1])) return cr_set_error(CR_ERR_ARG, "NCI atom out of range");
    if (d->nci[3 * m + 2] < 1 || d->nci[3 * m + 2] > 6) return cr_set_error(CR_ERR_ARG, "NCI category not 1..6");
  }
  if (d->nhb < 0 || (d->nhb > 0 && (!d->hb || !d->vhb))) return cr_set_error(CR_ERR_ARG, "missing H-bond arrays");
  for (int m = 0; m < 3 * d->nhb; ++m)
    if (!atom_ok(d->hb[m])) return cr_set_error(CR_ERR_ARG, "H-bond atom out of range");
  int ndev = 0;
  if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) return cr_set_error(CR_ERR_NO_DEVICE, "no CUDA device");

  const double pi = 3.1415926535897932384626433832795029;
  // the tables, value by value (qmdff.cuh, Tables); the torsions ordered by (type,
  // nt), so a warp runs one code path
  cr::qmdff::Dev devt{};
  const int count[cr::qmdff::kKinds] = {d->nbond, d->nangl, d->ntors, d->nnci, d->nhb};
  for (int k = 0; k < cr::qmdff::kKinds; ++k) devt.st[k] = (count[k] + 31) / 32 * 32;
  const int* st = devt.st;
  auto rad = [&](int atom) { return d->rad[d->at[atom] - 1]; };
  // 1 / rcut of abdamp (src/abdamp.f90:36-51); its prefactor is the REAL(4) product 3.0*3.5710642
  auto irc = [&](int a, int b) {
    const double r = rad(a) + rad(b);
    return 1.0 / ((double)(3.0f * 3.5710642f) * (r * r));
  };
  auto pack = [](int a, int b) { return (unsigned)a | (unsigned)b << 16; };
  std::vector<double> vbond((size_t)kVBond * st[0]), vangl((size_t)kVAngl * st[1]), vtors((size_t)kVTors * st[2]),
      vpair((size_t)kVPair * st[3]);
  std::vector<unsigned> bond((size_t)st[0]), pair((size_t)st[3]);
  std::vector<uint2> angl((size_t)st[1]);
  std::vector<uint4> tors((size_t)st[2]);
  std::vector<int> atoms[cr::qmdff::kKinds];  // per term in the order of its gradient
  for (int m = 0; m < d->nbond; ++m) {
    const int i = d->bond[2 * m] - 1, j = d->bond[2 * m + 1] - 1;
    bond[(size_t)m] = pack(i, j);
    for (int c = 0; c < 3; ++c) vbond[(size_t)c * st[0] + m] = d->vbond[3 * m + c];
    atoms[0].insert(atoms[0].end(), {i, j});
  }
  for (int m = 0; m < d->nangl; ++m) {
    const int j = d->angl[3 * m] - 1, i = d->angl[3 * m + 1] - 1, k = d->angl[3 * m + 2] - 1;
    angl[(size_t)m] = make_uint2(pack(i, j), (unsigned)k);
    const double th0 = d->vangl[2 * m];
    const double v[kVAngl] = {th0, d->vangl[2 * m + 1], std::cos(th0), (pi - th0 < 1e-6) ? 1.0 : 0.0, irc(i, j), irc(k, j)};
    for (int c = 0; c < kVAngl; ++c) vangl[(size_t)c * st[1] + m] = v[c];
    atoms[1].insert(atoms[1].end(), {i, j, k});
  }
  std::vector<int> order((size_t)d->ntors);
  for (int m = 0; m < d->ntors; ++m) order[(size_t)m] = m;
  std::stable_sort(order.begin(), order.end(), [&](int x, int y) {
    return d->tors[6 * x + 5] * 8 + d->tors[6 * x + 4] < d->tors[6 * y + 5] * 8 + d->tors[6 * y + 4];
  });
  for (int x = 0; x < d->ntors; ++x) {
    const int m = order[(size_t)x], *t = d->tors + 6 * m;
    const int i = t[0] - 1, j = t[1] - 1, k = t[2] - 1, l = t[3] - 1, type = t[5];
    // what the kernels tell apart: inversions (2) and torsions, which have 0..4 terms
    tors[(size_t)x] = make_uint4(pack(i, j), pack(k, l), (unsigned)(type == 2 ? 2 * 256 : t[4] + 256), (unsigned)m);
    for (int c = 0; c < 14; ++c) vtors[(size_t)c * st[2] + x] = d->vtors[14 * m + c];
    vtors[(size_t)14 * st[2] + x] = irc(i, j);
    vtors[(size_t)15 * st[2] + x] = irc(k, j);
    vtors[(size_t)16 * st[2] + x] = type != 2 ? irc(k, l) : irc(j, l);
    atoms[2].insert(atoms[2].end(), {i, j, k, l});
  }
  // a pair's class: what depends on its elements and its category alone
  struct PairClass {
    int z1, z2, nk;
    bool operator<(const PairClass& o) const { return std::tie(z1, z2, nk) < std::tie(o.z1, o.z2, o.nk); }
  };
  std::map<PairClass, int> classes;
  std::vector<float4> pclass;
  std::vector<int> class_of((size_t)d->nnci);
  for (int m = 0; m < d->nnci; ++m) {
    const int i1 = d->nci[3 * m] - 1, i2 = d->nci[3 * m + 1] - 1, nk = d->nci[3 * m + 2];
    pair[(size_t)m] = pack(i1, i2);
    atoms[3].insert(atoms[3].end(), {i1, i2});
    const int z1 = d->at[i1] - 1, z2 = d->at[i2] - 1;
    const size_t e12 = (size_t)z1 + 94 * (size_t)z2;  // (iz1, iz2) column-major
    const double R0 = d->r0094[e12], c6 = d->c66ab[(size_t)i2 + (size_t)n * i1], eps2 = d->eps2[nk - 1];  // c66ab(i2, i1)
    const double R02 = R0 * R0, R06 = R02 * R02 * R02, alpha = d->r0ab[e12];
    const double v[kVPair] = {R06, R06 * R02, eps2 * c6, eps2 * c6 * d->sr42[e12], eps2 * d->zab[e12], alpha,
                              d->zahn ? d->q[i1] * d->q[i2] : d->q[i1] * d->q[i2] * d->eps1[nk - 1]};
    for (int c = 0; c < kVPair; ++c) vpair[(size_t)c * st[3] + m] = v[c];
    const auto at = classes.emplace(PairClass{z1, z2, nk}, (int)classes.size());
    class_of[(size_t)m] = at.first->second;
    if (at.second) {
      pclass.push_back(make_float4((float)v[0], (float)v[1], (float)d->sr42[e12], (float)v[4]));
      pclass.push_back(make_float4((float)(alpha * 1.4426950408889634074), (float)alpha, 0.f, 0.f));  // log2(e)
    }
  }

  // H/halogen bonds: A, B, H (0-based) and the kind (src/ff_hb.f90:71-78)
  std::vector<int> hb((size_t)4 * d->nhb);
  std::vector<double> vhb(d->vhb, d->vhb + 2 * d->nhb);
  for (int m = 0; m < d->nhb; ++m) {
    for (int a = 0; a < 3; ++a) hb[(size_t)4 * m + a] = d->hb[3 * m + a] - 1;
    hb[(size_t)4 * m + 3] = d->at[d->hb[3 * m + 2] - 1] == 1 ? 1 : 2;
  }

  cr_qmdff* ff = new cr_qmdff();
  ff->n = n;
  ff->nterm[0] = d->nbond;
  ff->nterm[1] = d->nangl;
  ff->nterm[2] = d->ntors;
  ff->nterm[3] = d->nnci;
  ff->nterm[4] = d->nhb;

  for (int m = 0; m < d->nhb; ++m)
    for (int a = 0; a < 3; ++a) atoms[4].push_back(hb[(size_t)4 * m + a]);
  ScheduleHost sched[2];
  std::vector<int> mixed_pairs;
  cr::qmdff::Dev& D = ff->dev;
  D = devt;
  D.n = n;
  for (int form = 0; form < 2; ++form)
    for (int kind = 0; kind < cr::qmdff::kKinds; ++kind) {
      const int arity = kind == 0 || kind == 3 ? 2 : kind == 2 ? 4 : 3;
      cr::qmdff::Schedule& S = D.sched[form];
      S.seg0[kind] = (int)sched[form].seg.size();
      if (form == 1 && kind == 3) schedule_pairs(ff->nterm[kind], atoms[kind], n, mixed_pairs, S.npair);
      else schedule_kind(form == 1, kind, arity, atoms[kind], n, sched[form]);
      S.seg1[kind] = (int)sched[form].seg.size();
      if (form == 1) ff->batches[kind] = kind == 3 ? S.npair : (ff->nterm[kind] + 31) / 32;
    }

  Arena arena;
  auto up = [&](auto& h, auto** dp) { arena.add(h, dp); };
  for (int form = 0; form < 2; ++form) {
    up(sched[form].seg, &D.sched[form].seg);
    up(sched[form].round, &D.sched[form].round);
    up(sched[form].dst, &D.sched[form].dst);
    up(sched[form].ent, &D.sched[form].ent);
  }
  up(bond, &D.bond);
  up(angl, &D.angl);
  up(tors, &D.tors);
  up(pair, &D.pair);
  up(hb, &D.hb);
  up(vhb, &D.vhb);
  up(vbond, &D.d.bond);
  up(vangl, &D.d.angl);
  up(vtors, &D.d.tors);
  up(vpair, &D.d.pair);
  std::vector<float> fvbond = to_float(vbond), fvangl = to_float(vangl), fvtors = to_float(vtors);
  up(fvbond, &D.f.bond);
  up(fvangl, &D.f.angl);
  up(fvtors, &D.f.tors);
  std::vector<uint4> fpair;
  auto bits = [](double x) {
    const float f = (float)x;
    unsigned u;
    std::memcpy(&u, &f, 4);
    return u;
  };
  for (int m : mixed_pairs)
    fpair.push_back(m < 0 ? make_uint4(0, cr::qmdff::kNoPair, 0, 0)
                          : make_uint4(pair[(size_t)m], (unsigned)class_of[(size_t)m], bits(vpair[(size_t)2 * st[3] + m]),
                                       bits(vpair[(size_t)6 * st[3] + m])));
  up(fpair, &D.fpair);
  up(pclass, &D.pclass);
  D.coul_cut = d->coul_cut;
  D.zahn = d->zahn ? 1 : 0;
  D.zahn_a = d->zahn_a;
  D.zahn_par = d->zahn_par;
  D.fcoul_cut = (float)d->coul_cut;
  D.fzahn_a = (float)d->zahn_a;
  D.fzahn_par = (float)d->zahn_par;
  D.e_zero = d->e_zero;
  for (int k = 0; k < cr::qmdff::kKinds; ++k) D.nterm[k] = ff->nterm[k];
  // mixed form bond polynomial: a k u (1 - u) / r^2 = t H(t), t = r^2/r0^2 - 1,
  // H(t) = (a k / r0^2) [(1+t)^-(a/4+1) - (1+t)^-(a/2+1)] / t interpolated
  // at 48 Chebyshev nodes of |t| <= kBondSerMaxT, truncated to degree 23 and
  // written as a monomial in x = t / kBondSerMaxT; bonds with exponents
  // outside (0, 20] keep the FP32 formula
  {
    using cr::qmdff::kBondPoly;
    using cr::qmdff::kBondSer;
    const double T = cr::qmdff::kBondSerMaxT;
    const int nn = 48;
    std::vector<float2> bser((size_t)kBondSer * st[0], make_float2(0.f, 0.f));
    std::vector<double> node((size_t)nn), basis((size_t)kBondPoly * nn);
    for (int k = 0; k < nn; ++k) {
      node[(size_t)k] = std::cos(pi * (k + 0.5) / nn);
      for (int j = 0; j < kBondPoly; ++j) basis[(size_t)j * nn + k] = std::cos(pi * j * (k + 0.5) / nn);
    }
    std::map<double, std::vector<double>> of_exponent;  // the polynomial depends on the bond by its exponent alone
    auto split = [](double v) {
      const float hi = (float)v;
      return make_float2(hi, (float)(v - (double)hi));
    };
    for (int m = 0; m < d->nbond; ++m) {
      const double r0 = d->vbond[3 * m], kk = d->vbond[3 * m + 1], aa = d->vbond[3 * m + 2];
      auto row = [&](int c) -> float2& { return bser[(size_t)c * st[0] + m]; };
      row(0) = split(1.0 / (r0 * r0));
      row(1) = split(r0 * r0);
      if (!(aa > 0.0) || aa > 20.0 || !(r0 > 0.0)) continue;
      const double p1 = aa / 4.0 + 1.0, p2 = aa / 2.0 + 1.0, scale = aa * kk / (r0 * r0);
      std::vector<double>& mono = of_exponent[aa];
      if (mono.empty()) {
        std::vector<double> hv((size_t)nn), cheb((size_t)kBondPoly, 0.0);
        for (int k = 0; k < nn; ++k) {
          const double tk = T * node[(size_t)k];
          hv[(size_t)k] = (std::pow(1.0 + tk, -p1) - std::pow(1.0 + tk, -p2)) / tk;
        }
        for (int j = 0; j < kBondPoly; ++j) {
          double acc = 0.0;
          for (int k = 0; k < nn; ++k) acc += hv[(size_t)k] * basis[(size_t)j * nn + k];
          cheb[(size_t)j] = (j == 0 ? 1.0 : 2.0) * acc / nn;
        }
        // Chebyshev -> monomial in x: T_0 = 1, T_1 = x, T_{j+1} = 2x T_j - T_{j-1}
        std::vector<double> tm1((size_t)kBondPoly, 0.0), t0((size_t)kBondPoly, 0.0);
        mono.assign((size_t)kBondPoly, 0.0);
        tm1[0] = 1.0;
        if (kBondPoly > 1) t0[1] = 1.0;
        for (int j = 0; j < kBondPoly; ++j) {
          const std::vector<double>& tj = j == 0 ? tm1 : t0;
          for (int n = 0; n < kBondPoly; ++n) mono[(size_t)n] += cheb[(size_t)j] * tj[(size_t)n];
          if (j >= 1 && j + 1 < kBondPoly) {
            std::vector<double> tn((size_t)kBondPoly, 0.0);
            for (int n = 0; n + 1 < kBondPoly; ++n) tn[(size_t)n + 1] += 2.0 * t0[(size_t)n];
            for (int n = 0; n < kBondPoly; ++n) tn[(size_t)n] -= tm1[(size_t)n];
            tm1 = t0;
            t0 = tn;
          }
        }
      }
      row(2) = make_float2(1.0f, 0.0f);
      for (int n = 0; n < kBondPoly; ++n) row(3 + n) = split(scale * mono[(size_t)n]);
    }
    up(bser, &D.bser);
  }
  // unit tables of the linear parameters (parameter gradients)
  std::vector<double> ubond = vbond, uangl = vangl, utors = vtors;
  std::fill_n(ubond.begin() + st[0], st[0], 1.0);
  std::fill_n(uangl.begin() + st[1], st[1], 1.0);
  std::fill_n(utors.begin() + st[2], st[2], 1.0);
  up(ubond, &ff->unit.bond);
  up(uangl, &ff->unit.angl);
  up(utors, &ff->unit.tors);
  const int rc = arena.upload(ff);
  if (rc != CR_OK) {
    cr_qmdff_destroy(ff);
    return rc;
  }
  *out = ff;
  return CR_OK;
}

int cr_qmdff_set_periodic(cr_qmdff* ff, const double* box_ang, double coul_cut_ang, double vdw_cut_ang,
                          double* cuts) {
  if (!ff) return cr_set_error(CR_ERR_ARG, "NULL force field");
  cr::qmdff::Dev& D = ff->dev;
  if (!box_ang) {
    D.periodic = 0;
    return CR_OK;
  }
  for (int k = 0; k < 3; ++k)
    if (!(box_ang[k] > 0.0)) return cr_set_error(CR_ERR_ARG, "box edges must be positive (Angstrom)");
  if (!(coul_cut_ang > 0.0) || !(vdw_cut_ang > 0.0)) return cr_set_error(CR_ERR_ARG, "cutoffs must be positive");
  // set_periodic (src/set_periodic.f90:67-113)
  const double bohr = 0.52917721092;
  double len[3];
  for (int k = 0; k < 3; ++k) len[k] = box_ang[k] / bohr;
  D.box = cr::qmdff::make_box(len);
  const double hmin = std::min(D.box.half[0], std::min(D.box.half[1], D.box.half[2]));
  double coul = coul_cut_ang / bohr;
  if (coul < 5.0) coul = hmin - 0.1;
  if (D.zahn) {
    const double spi = std::sqrt(3.14159265358979323846);
    D.zahn_a = 0.2 * bohr;
    coul = 10.0 / bohr;
    const double acut = D.zahn_a * coul;
    D.zahn_par = std::erfc(acut) / (coul * coul) + 2 * D.zahn_a / spi * std::exp(-acut * acut) / coul;
  }
  if (coul > hmin) coul = hmin - 0.1;
  D.coul_cut = coul;
  D.vdw_cut = vdw_cut_ang / bohr;
  D.fcoul_cut = (float)D.coul_cut;
  D.fvdw_cut = (float)D.vdw_cut;
  D.fzahn_a = (float)D.zahn_a;
  D.fzahn_par = (float)D.zahn_par;
  D.periodic = 1;
  if (cuts) {
    cuts[0] = D.coul_cut;
    cuts[1] = D.vdw_cut;
    cuts[2] = D.zahn_a;
    cuts[3] = D.zahn_par;
  }
  return CR_OK;
}

int cr_qmdff_schedule_info(const cr_qmdff* ff, int* batches, int* colors) {
  if (!ff) return cr_set_error(CR_ERR_ARG, "NULL force field");
  int n = 0;
  for (int k = 0; k < cr::qmdff::kKinds; ++k) {
    if (batches) batches[k] = ff->batches[k];
    n += ff->batches[k];
  }
  if (colors) *colors = n;  // one pass each
  return CR_OK;
}

int cr_qmdff_tuning(const cr_qmdff* ff, int precision, int* variant, float* ms) {
  if (!ff) return cr_set_error(CR_ERR_ARG, "NULL force field");
  if (precision != CR_PREC_MIXED && precision != CR_PREC_FP64) return cr_set_error(CR_ERR_ARG, "unknown precision");
  const int prec = precision == CR_PREC_MIXED ? 1 : 0;
  if (variant) *variant = ff->variant[prec];
  if (ms)
    for (int v = 0; v < kVariants; ++v) ms[v] = ff->tune_ms[prec][v];
  return CR_OK;
}

int cr_qmdff_egrad_device(cr_qmdff* ff, const double* d_xyz, int nbeads, double* d_e, double* d_g, int precision,
                          void* stream) {
  if (!ff) return cr_set_error(CR_ERR_ARG, "NULL force field");
  if (nbeads < 0 || (nbeads > 0 && (!d_xyz || !d_e || !d_g))) return cr_set_error(CR_ERR_ARG, "bad egrad arguments");
  return qmdff_launch(ff, d_xyz, nbeads, d_e, d_g, precision, (cudaStream_t)stream);
}

int cr_qmdff_egrad(cr_qmdff* ff, const double* xyz, int nbeads, double* e, double* g, int precision) {
  if (!ff) return cr_set_error(CR_ERR_ARG, "NULL force field");
  if (nbeads < 0 || (nbeads > 0 && (!xyz || !e || !g))) return cr_set_error(CR_ERR_ARG, "bad egrad arguments");
  if (nbeads == 0) return CR_OK;
  const size_t nq = (size_t)3 * ff->n * nbeads;
  double* d_q = nullptr;  // q, gradient, energies
  CR_TRY_CUDA(cudaMalloc(&d_q, (2 * nq + (size_t)nbeads) * sizeof(double)));
  double *d_g = d_q + nq, *d_e = d_g + nq;
  int rc = CR_OK;
  if (cudaMemcpy(d_q, xyz, nq * sizeof(double), cudaMemcpyHostToDevice) != cudaSuccess) {
    rc = cr_set_error(CR_ERR_CUDA, "copy of xyz failed");
  } else if ((rc = qmdff_launch(ff, d_q, nbeads, d_e, d_g, precision, nullptr)) == CR_OK) {
    if (cudaMemcpy(e, d_e, (size_t)nbeads * sizeof(double), cudaMemcpyDeviceToHost) != cudaSuccess ||
        cudaMemcpy(g, d_g, nq * sizeof(double), cudaMemcpyDeviceToHost) != cudaSuccess)
      rc = cr_set_error(CR_ERR_CUDA, "copy of results failed");
  }
  cudaFree(d_q);
  return rc;
}

int cr_qmdff_egrad_virial(cr_qmdff* ff, const double* xyz, int nbeads, const double* box, double* e, double* g,
                          double* vir, int precision) {
  if (!ff) return cr_set_error(CR_ERR_ARG, "NULL force field");
  if (!ff->dev.periodic) return cr_set_error(CR_ERR_ARG, "the virial is formed for periodic force fields (NpT)");
  if (nbeads < 0 || (nbeads > 0 && (!xyz || !e || !g || !vir))) return cr_set_error(CR_ERR_ARG, "bad egrad arguments");
  if (precision != CR_PREC_MIXED && precision != CR_PREC_FP64) return cr_set_error(CR_ERR_ARG, "unknown precision");
  if (nbeads == 0) return CR_OK;
  const size_t nq = (size_t)3 * ff->n * nbeads, nb = (size_t)nbeads;
  std::vector<double> hb(3 * nb);
  for (size_t b = 0; b < nb; ++b)
    for (int k = 0; k < 3; ++k) hb[3 * b + k] = box ? box[3 * b + k] : ff->dev.box.len[k];
  double *d_q = nullptr, *d_e = nullptr, *d_g = nullptr, *d_b = nullptr, *d_w = nullptr;
  int rc = CR_OK;
  if (cudaMalloc(&d_q, nq * sizeof(double)) != cudaSuccess || cudaMalloc(&d_e, nb * sizeof(double)) != cudaSuccess ||
      cudaMalloc(&d_g, nq * sizeof(double)) != cudaSuccess || cudaMalloc(&d_b, 3 * nb * sizeof(double)) != cudaSuccess ||
      cudaMalloc(&d_w, nb * sizeof(double)) != cudaSuccess) {
    rc = cr_set_error(CR_ERR_CUDA, "cudaMalloc failed in cr_qmdff_egrad_virial");
  } else if (cudaMemcpy(d_q, xyz, nq * sizeof(double), cudaMemcpyHostToDevice) != cudaSuccess ||
             cudaMemcpy(d_b, hb.data(), 3 * nb * sizeof(double), cudaMemcpyHostToDevice) != cudaSuccess) {
    rc = cr_set_error(CR_ERR_CUDA, "copy of xyz failed");
  } else {
    const QmdffNpt np{d_b, 1, d_w};
    if ((rc = qmdff_launch(ff, d_q, nbeads, d_e, d_g, precision, nullptr, &np)) == CR_OK &&
        (cudaMemcpy(e, d_e, nb * sizeof(double), cudaMemcpyDeviceToHost) != cudaSuccess ||
         cudaMemcpy(g, d_g, nq * sizeof(double), cudaMemcpyDeviceToHost) != cudaSuccess ||
         cudaMemcpy(vir, d_w, nb * sizeof(double), cudaMemcpyDeviceToHost) != cudaSuccess))
      rc = cr_set_error(CR_ERR_CUDA, "copy of results failed");
  }
  cudaFree(d_q);
  cudaFree(d_e);
  cudaFree(d_g);
  cudaFree(d_b);
  cudaFree(d_w);
  return rc;
}

int cr_qmdff_eg(cr_qmdff* ff, const double* xyz, int nbeads, double* e, double* g, int precision) {
  return qmdff_host_kinds(ff, 0x7u, false, false, xyz, nbeads, e, g, precision);
}

int cr_qmdff_nonb(cr_qmdff* ff, const double* xyz, int nbeads, double* e, double* g, int precision) {
  return qmdff_host_kinds(ff, 0x8u, false, true, xyz, nbeads, e, g, precision);
}

int cr_qmdff_hb(cr_qmdff* ff, const double* xyz, int nbeads, double* e, double* g, int precision) {
  return qmdff_host_kinds(ff, 0x10u, false, true, xyz, nbeads, e, g, precision);
}

int cr_qmdff_nparams(const cr_qmdff* ff, int* nlin) {
  if (!ff || !nlin) return cr_set_error(CR_ERR_ARG, "NULL argument");
  *nlin = qmdff_nlin(ff);
  return CR_OK;
}

int cr_qmdff_hvp(cr_qmdff* ff, const double* xyz, const double* w, int nbeads, double* e, double* g, double* hw) {
  if (!ff) return cr_set_error(CR_ERR_ARG, "NULL force field");
  if (nbeads < 0 || (nbeads > 0 && (!xyz || !w || !hw))) return cr_set_error(CR_ERR_ARG, "bad hvp arguments");
  if (ff->nterm[4] > 0) return cr_set_error(CR_ERR_UNSUPPORTED, "second derivatives of H/halogen-bond terms are not built");
  if (nbeads == 0) return CR_OK;
  const size_t nq = (size_t)3 * ff->n * nbeads;
  double* d = nullptr;
  CR_TRY_CUDA(cudaMalloc(&d, (4 * nq + nbeads) * sizeof(double)));
  double *dq = d, *dw = dq + nq, *dg = dw + nq, *dh = dg + nq, *de = dh + nq;
  int rc = CR_OK;
  if (cudaMemcpy(dq, xyz, nq * 8, cudaMemcpyHostToDevice) != cudaSuccess ||
      cudaMemcpy(dw, w, nq * 8, cudaMemcpyHostToDevice) != cudaSuccess)
    rc = cr_set_error(CR_ERR_CUDA, "copy of the hvp inputs failed");
  else if ((rc = qmdff_hvp_launch(ff, dq, dw, nbeads, de, dg, dh, nullptr, nullptr)) == CR_OK &&
           (cudaMemcpy(hw, dh, nq * 8, cudaMemcpyDeviceToHost) != cudaSuccess ||
            (g && cudaMemcpy(g, dg, nq * 8, cudaMemcpyDeviceToHost) != cudaSuccess) ||
            (e && cudaMemcpy(e, de, (size_t)nbeads * 8, cudaMemcpyDeviceToHost) != cudaSuccess)))
    rc = cr_set_error(CR_ERR_CUDA, "copy of the hvp results failed");
  cudaFree(d);
  return rc;
}

int cr_qmdff_param_vjp(cr_qmdff* ff, const double* xyz, const double* v, int nbeads, double* grad) {
  if (!ff) return cr_set_error(CR_ERR_ARG, "NULL force field");
  if (nbeads < 0 || !grad || (nbeads > 0 && (!xyz || !v))) return cr_set_error(CR_ERR_ARG, "bad vjp arguments");
  if (ff->nterm[4] > 0) return cr_set_error(CR_ERR_UNSUPPORTED, "parameter gradients of H/halogen-bond terms are not built");
  const int nlin = qmdff_nlin(ff);
  for (int t = 0; t < nlin; ++t) grad[t] = 0.0;
  if (nbeads == 0 || nlin == 0) return CR_OK;
  const size_t nq = (size_t)3 * ff->n * nbeads;
  const int chunk = std::min(nbeads, 4096);
  double* d = nullptr;
  CR_TRY_CUDA(cudaMalloc(&d, (2 * nq + (size_t)chunk * nlin + nlin) * sizeof(double)));
  double *dq = d, *dv = dq + nq, *ds = dv + nq, *dacc = ds + (size_t)chunk * nlin;
  int rc = CR_OK;
  if (cudaMemcpy(dq, xyz, nq * 8, cudaMemcpyHostToDevice) != cudaSuccess ||
      cudaMemcpy(dv, v, nq * 8, cudaMemcpyHostToDevice) != cudaSuccess ||
      cudaMemset(dacc, 0, (size_t)nlin * 8) != cudaSuccess)
    rc = cr_set_error(CR_ERR_CUDA, "copy of the vjp inputs failed");
  else if ((rc = qmdff_vjp_launch(ff, dq, dv, nbeads, nullptr, nullptr, 1.0, ds, chunk, dacc, nullptr)) == CR_OK &&
           cudaMemcpy(grad, dacc, (size_t)nlin * 8, cudaMemcpyDeviceToHost) != cudaSuccess)
    rc = cr_set_error(CR_ERR_CUDA, "copy of the vjp result failed");
  cudaFree(d);
  return rc;
}

}  // extern "C"
