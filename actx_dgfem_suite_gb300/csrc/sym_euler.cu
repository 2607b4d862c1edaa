// Symmetry-adapted FP64 RHS kernels of the euler equation (dg_sym.cuh).
#include "sym_instantiate.cuh"

namespace dg {
cudaError_t sym_shape_euler(int order, bool stage, LaunchShape* out) {
  return sym_shape_any<DG_EULER>(order, stage, out);
}
cudaError_t sym_launch_euler(int order, bool stage, const RhsArgs& a, int grid, cudaStream_t s) {
  return sym_launch_any<DG_EULER>(order, stage, a, grid, s);
}
}  // namespace dg
