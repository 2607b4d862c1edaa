// Adjoint (transpose) kernels of the FP64 wave RHS, orders 1..4.
#include "dg_adjoint.cuh"
#include "dg_launch.h"
#include "dg_sym_adjoint.cuh"

namespace dg {
namespace {

template <int N>
cudaError_t adj_shape_n(LaunchShape* out) {
  using T = AdjTile<N>;
  int nb = 0;
  for (int stage = 0; stage < 2; ++stage) {  // both forms, the smaller occupancy
    auto* fn = stage ? dg_wave_adjoint_volume<N, true> : dg_wave_adjoint_volume<N, false>;
    cudaError_t err = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                           T::SMEM_BYTES);
    if (err != cudaSuccess) return err;
    int b = 0;
    err = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, fn, kBlock, T::SMEM_BYTES);
    if (err != cudaSuccess) return err;
    nb = stage == 0 || b < nb ? b : nb;
  }
  out->smem_bytes = T::SMEM_BYTES;
  out->blocks_per_sm = nb;
  out->elems_per_tile = T::E;
  out->ops_bytes = AdjOpsLayout<N>::SIZE;
  return cudaSuccess;
}

template <int N>
cudaError_t adj_sym_shape_n(LaunchShape* out) {
  using T = sym::AdjTile<N, DG_WAVE>;
  out->blocks_per_sm = 1 << 30;
  for (int stage = 0; stage < 2; ++stage) {  // both forms, the smaller occupancy
    auto* fn = stage ? sym::dg_wave_adjoint_sym_kernel<N, true>
                     : sym::dg_wave_adjoint_sym_kernel<N, false>;
    cudaError_t err =
        cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, T::SMEM);
    int b = 0;
    if (err == cudaSuccess)
      err = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, fn, T::BLOCK, T::SMEM);
    if (err != cudaSuccess) return err;
    if (b < out->blocks_per_sm) out->blocks_per_sm = b;
  }
  out->smem_bytes = T::SMEM;
  out->elems_per_tile = T::E;
  out->ops_bytes = T::O::SIZE;
  out->threads = T::BLOCK;
  return cudaSuccess;
}

template <int N, bool STAGE>
cudaError_t adj_launch_n(const AdjArgs& a, int grid, int nsm, cudaStream_t s) {
  using S = sym::AdjTile<N, DG_WAVE>;
  if (a.sym_ops)
    sym::dg_wave_adjoint_sym_kernel<N, STAGE><<<a.sym_grid, S::BLOCK, S::SMEM, s>>>(a);
  else
    dg_wave_adjoint_volume<N, STAGE><<<grid, kBlock, AdjTile<N>::SMEM_BYTES, s>>>(a);
  cudaError_t err = cudaGetLastError();
  if (err != cudaSuccess) return err;
  const int64_t nodes = a.nel * Shape<N>::NP;
  int64_t blocks = (nodes + kBlock - 1) / kBlock;
  const int64_t cap = (int64_t)nsm * 16;
  if (blocks > cap) blocks = cap;
  dg_wave_adjoint_surface<N, STAGE><<<(int)blocks, kBlock, 0, s>>>(a);
  return cudaGetLastError();
}

}  // namespace

cudaError_t adjoint_shape_wave(int order, LaunchShape* out) {
  switch (order) {
    case 1: return adj_shape_n<1>(out);
    case 2: return adj_shape_n<2>(out);
    case 3: return adj_shape_n<3>(out);
    case 4: return adj_shape_n<4>(out);
    default: return cudaErrorInvalidValue;
  }
}

cudaError_t adjoint_sym_shape_wave(int order, LaunchShape* out) {
  switch (order) {
    case 1: return adj_sym_shape_n<1>(out);
    case 2: return adj_sym_shape_n<2>(out);
    case 3: return adj_sym_shape_n<3>(out);
    case 4: return adj_sym_shape_n<4>(out);
    default: return cudaErrorInvalidValue;
  }
}

cudaError_t adjoint_launch_wave(int order, const AdjArgs& a, int grid, int nsm,
                                cudaStream_t s) {
  switch (order) {
    case 1: return adj_launch_n<1, false>(a, grid, nsm, s);
    case 2: return adj_launch_n<2, false>(a, grid, nsm, s);
    case 3: return adj_launch_n<3, false>(a, grid, nsm, s);
    case 4: return adj_launch_n<4, false>(a, grid, nsm, s);
    default: return cudaErrorInvalidValue;
  }
}

cudaError_t adjoint_stage_launch_wave(int order, const AdjArgs& a, int grid, int nsm,
                                      cudaStream_t s) {
  switch (order) {
    case 1: return adj_launch_n<1, true>(a, grid, nsm, s);
    case 2: return adj_launch_n<2, true>(a, grid, nsm, s);
    case 3: return adj_launch_n<3, true>(a, grid, nsm, s);
    case 4: return adj_launch_n<4, true>(a, grid, nsm, s);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace dg
