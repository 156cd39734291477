// Fraction-to-boundary bounds from the smallest eigenvalue (step_bound.cu).
#pragma once
#include "common.cuh"

namespace sdpx {

struct StepBoundDesc {
  const double* G;  // L⁻¹·dM·L⁻ᵀ, column-major k×k (symmetric up to rounding)
  int k;
};

// The largest order that the current device has a kernel for (448 on a whole B200; looked
// up once per device), orders from 3 on.
int step_bound_max_order();
// out[q] = min(1, −1/λ_min(G_q)) (1 when λ_min ≥ −1, 0 when G is not finite) for the
// n matrices of the device list; kmax: the largest order, at most that.
void step_bounds(const StepBoundDesc* d_list, int n, int kmax, double* out, cudaStream_t st);

}  // namespace sdpx
