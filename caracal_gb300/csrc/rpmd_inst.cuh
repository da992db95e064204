// The PesRuns table of one analytic surface: instantiates its persistent
// step kernel and its force kernel (both precision forms); MAXTPB is the
// largest number of threads per bead that the surface's engines take.  Included
// once per surface, by rpmd_<surface>.cu.
#pragma once
#include "pes_runs.h"
#include "rpmd_kernel.cuh"

namespace cr {

// Blocks of the step kernel that stay resident per SM (its registers follow: 255; three
// or four blocks were measured and not kept).
constexpr int kStepBlocks = 2;

template <class PES, int MAXTPB>
struct RunsOf {
  static cudaError_t run(const StepParams& prm, bool mixed, int grid, int block, size_t smem, cudaStream_t st,
                         int istep, int nsteps) {
    if (mixed) rpmd_run_kernel<PES, true, kStepBlocks><<<grid, block, smem, st>>>(prm, istep, nsteps);
    else rpmd_run_kernel<PES, false, kStepBlocks><<<grid, block, smem, st>>>(prm, istep, nsteps);
    return cudaGetLastError();
  }
  // The limit belongs to the kernel, whichever engine asks, so it is always the most
  // that any launch shape takes: an engine's creation lowers no other's.
  static cudaError_t allow_smem(bool mixed) {
    return mixed ? cudaFuncSetAttribute(rpmd_run_kernel<PES, true, kStepBlocks>, cudaFuncAttributeMaxDynamicSharedMemorySize, kStepSmemMax)
                 : cudaFuncSetAttribute(rpmd_run_kernel<PES, false, kStepBlocks>, cudaFuncAttributeMaxDynamicSharedMemorySize, kStepSmemMax);
  }
  static cudaError_t resident(bool mixed, int block, size_t smem, int* blocks) {
    cudaError_t err = allow_smem(mixed);
    if (err != cudaSuccess) return err;
    return mixed ? cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks, rpmd_run_kernel<PES, true, kStepBlocks>, block, smem)
                 : cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks, rpmd_run_kernel<PES, false, kStepBlocks>, block, smem);
  }
  template <int L>
  static void egrad_lanes(bool mixed, int nbeads, BeadRows rows, const double* q, double* V, double* g, cudaStream_t st) {
    const int bs = 128 / L, nb = nbeads / bs + (nbeads % bs != 0);
    if (mixed) egrad_kernel<PES, true, L><<<nb, 128, 0, st>>>(nbeads, rows, q, V, g);
    else egrad_kernel<PES, false, L><<<nb, 128, 0, st>>>(nbeads, rows, q, V, g);
  }
  static cudaError_t egrad(bool mixed, int nbeads, BeadRows rows, const double* q, double* V, double* g, cudaStream_t st) {
    if (nbeads <= 0) return cudaSuccess;
    if constexpr (PES::kQuad) {
      if (nbeads <= kQuadBeads) {
        egrad_lanes<4>(mixed, nbeads, rows, q, V, g, st);
        return cudaGetLastError();
      }
    }
    egrad_lanes<PES::kLanes>(mixed, nbeads, rows, q, V, g, st);
    return cudaGetLastError();
  }
  static constexpr PesRuns table() { return PesRuns{MAXTPB, PES::kLanes, PES::kQuad, &run, &allow_smem, &resident, &egrad}; }
};

}  // namespace cr
