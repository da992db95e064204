// Device-side flexible SPC water box (the object behind cr_water) and its
// launch entry for the engine.
#pragma once
#include <cuda_runtime.h>

#include "../../include/caracal_gb300.h"
#include "bead_rows.cuh"
#include "water.cuh"

struct cr_water {
  cr::water::Dev dev{};
};

// e and g = dV/dq of nbeads evaluations at the rows of `rows` of d_q(3, n, beads).
int water_launch(const cr_water* w, const double* d_q, int nbeads, double* d_e, double* d_g, int precision,
                 cudaStream_t s, cr::BeadRows rows = cr::all_rows());
