// Launch entry points of the analytic surfaces' kernels.  Each surface's
// persistent step kernel and one-thread-per-bead force kernel are compiled
// in their own translation unit (rpmd_h3.cu, rpmd_ch4h.cu, rpmd_ch4oh.cu,
// rpmd_oh3.cu, rpmd_geh4oh.cu, rpmd_brh2.cu), so the library builds them in parallel; the engine reaches
// them through this table.
#pragma once
#include <cstddef>

#include <cuda_runtime.h>

#include "bead_rows.cuh"

namespace cr {

struct StepParams;

// Most evaluated beads of a batch whose surface takes four lanes per bead where it has
// both forms: one warp of quads per scheduler (152 SMs).  H3 x 16 plain, per step:
// 300 trajectories (2700 beads) 27 us by quads, about 47 by single threads at any
// number up to 1100; 1000 trajectories (9000 beads) 53 to 62 by quads.
constexpr int kQuadBeads = 32 * 152;

struct PesRuns {
  int max_tpb;  // most threads per bead of the step kernel on the surface
  int lanes;    // threads that evaluate a bead together (PES::kLanes)
  bool quad;    // has the form by four lanes too (PES::kQuad)
  // rpmd_run_kernel<surface, mixed><<<grid, block, smem, st>>>(prm, istep, nsteps)
  cudaError_t (*run)(const StepParams& prm, bool mixed, int grid, int block, size_t smem, cudaStream_t st, int istep,
                     int nsteps);
  // raises that kernel's limit on dynamic shared memory (outside a stream capture)
  cudaError_t (*allow_smem)(bool mixed);
  // blocks of that many threads and bytes that an SM holds
  cudaError_t (*resident)(bool mixed, int block, size_t smem, int* blocks);
  // egrad_kernel<surface, mixed>: V and dV/dq of nbeads evaluations at the rows of `rows`
  cudaError_t (*egrad)(bool mixed, int nbeads, BeadRows rows, const double* q, double* V, double* g, cudaStream_t st);
};

// The table of CR_PES_H3 / CH4H / CH4OH / OH3 / GEH4OH / BRH2; NULL for any other surface.
const PesRuns* pes_runs(int pes);

extern const PesRuns kRunsH3, kRunsCH4H, kRunsCH4OH, kRunsOH3, kRunsGeH4OH, kRunsBrH2;

}  // namespace cr
