// Mixed-precision RHS kernels of the wave equation on the CUDA cores
// (dg_mixed.cuh); the operator block of both equations.
#include <cstring>

#include "mixed_instantiate.cuh"

namespace dg {
cudaError_t mixed_shape_wave(int order, bool stage, LaunchShape* out) {
  return mixed_shape_any<DG_WAVE>(order, stage, out);
}
cudaError_t mixed_launch_wave(int order, bool stage, const RhsArgs& a, int grid,
                             cudaStream_t s) {
  return mixed_launch_any<DG_WAVE>(order, stage, a, grid, s);
}

namespace {
template <int N>
int pack(const double* diff, const double* lift, const int32_t* face_nodes,
         unsigned char* out, int out_bytes) {
  using O = mix::Ops<N>;
  if (!out) return O::SIZE;
  if (out_bytes < O::SIZE) return -1;
  std::memset(out, 0, O::SIZE);
  float* w = reinterpret_cast<float*>(out);
  int32_t* fn = reinterpret_cast<int32_t*>(out + O::FN);
  auto at = [](int column, int i) { return column * O::ROW + (i / O::R) * O::RP + i % O::R; };
  for (int r = 0; r < 3; ++r)
    for (int i = 0; i < O::NP; ++i)
      for (int j = 0; j < O::NP; ++j)
        w[at(r * O::NP + j, i)] = (float)diff[(r * O::NP + i) * O::NP + j];
  for (int i = 0; i < O::NP; ++i)
    for (int fj = 0; fj < O::NFPT; ++fj)
      w[O::L + at(fj, i)] = (float)lift[i * O::NFPT + fj];
  for (int k = 0; k < O::NFPT; ++k) fn[k] = face_nodes[k];
  return O::SIZE;
}
}  // namespace

int pack_mixed_ops(int order, const double* diff, const double* lift,
                   const int32_t* face_nodes, unsigned char* out, int out_bytes) {
  switch (order) {
    case 1: return pack<1>(diff, lift, face_nodes, out, out_bytes);
    case 2: return pack<2>(diff, lift, face_nodes, out, out_bytes);
    case 3: return pack<3>(diff, lift, face_nodes, out, out_bytes);
    case 4: return pack<4>(diff, lift, face_nodes, out, out_bytes);
    default: return -1;
  }
}
}  // namespace dg
