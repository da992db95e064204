// Rows of the bead arrays that a force kernel evaluates.
//
// Caracal's free ring-polymer map (cosine transform, nm_mode 0) gives beads
// j and P - j the same position, bit for bit: the drift kernels write one
// value to both rows.  After a drift the surface is therefore evaluated once
// per distinct bead, j = 0 .. P/2, and its energy and gradient are written to
// both rows; what the other evaluation would return is that same value.
// Evaluations outside a step (arbitrary positions) take every row.
#pragma once
#include <cstddef>

namespace cr {

struct BeadRows {
  int U;  // evaluated beads per trajectory
  int P;  // rows per trajectory

  // row of evaluation b (b = 0 .. T U - 1)
  __host__ __device__ inline size_t row(size_t b) const {
    return U == P ? b : (b / (size_t)U) * (size_t)P + b % (size_t)U;
  }
  // the other row with the same position (row(b) itself where there is none)
  __host__ __device__ inline size_t twin(size_t b) const {
    if (U == P) return b;
    const size_t t = b / (size_t)U, j = b % (size_t)U;
    return t * (size_t)P + (j == 0 ? 0 : (size_t)P - j);
  }
};

// Evaluation that a thread belongs to where L threads take one together: the thread
// count passes 2^31 before an int count of evaluations does.
__host__ __device__ inline size_t evaluation_of(unsigned block, unsigned block_threads, unsigned thread, int L) {
  return ((size_t)block * block_threads + thread) / (size_t)L;
}

// Every row.
inline BeadRows all_rows() { return BeadRows{1, 1}; }
// The distinct beads of a trajectory of P beads after a drift in nm_mode 0.
inline BeadRows distinct_rows(int P) { return BeadRows{P / 2 + 1, P}; }

}  // namespace cr
