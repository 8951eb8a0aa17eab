// The wide tensor-memory solver in reference arithmetic (radm2_wide.cuh): pivot divisions
// kept, built without multiply-add contraction (Makefile).
#define RADM2_WIDE_DIV 1
#include "radm2_wide.cuh"

namespace radm2 {
cudaError_t launch_solver_widex(const SolveArgs &a, int grid, cudaStream_t st) { return launch_wide<1>(a, grid, st); }
cudaError_t solver_info_widex(SolverInfo *out) { return info_wide<1>(out); }
}  // namespace radm2
