// The wide tensor-memory solver, fast arithmetic (radm2_wide.cuh).
#define RADM2_WIDE_DIV 0
#include "radm2_wide.cuh"

namespace radm2 {
cudaError_t launch_solver_wide(const SolveArgs &a, int grid, cudaStream_t st) { return launch_wide<0>(a, grid, st); }
cudaError_t solver_info_wide(SolverInfo *out) { return info_wide<0>(out); }
}  // namespace radm2
