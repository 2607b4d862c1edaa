// Shape and launch entry points of dg_rhs_mixed_kernel for one equation, orders
// 1..4, plain RHS and Runge-Kutta stage.
#pragma once

#include "dg_launch.h"
#include "dg_mixed.cuh"

namespace dg {
namespace {

template <int N, int EQ, bool STAGE>
struct MixedKernel {
  using T = mix::Tile<N, EQ>;

  static cudaError_t shape(LaunchShape* out) {
    auto kern = mix::dg_rhs_mixed_kernel<N, EQ, STAGE>;
    cudaError_t err = cudaFuncSetAttribute(
        kern, cudaFuncAttributeMaxDynamicSharedMemorySize, T::SMEM);
    if (err != cudaSuccess) return err;
    int nb = 0;
    err = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, kern, T::BLOCK, T::SMEM);
    out->smem_bytes = T::SMEM;
    out->blocks_per_sm = nb;
    out->elems_per_tile = T::E;
    out->ops_bytes = mix::Ops<N>::SIZE;
    out->threads = T::BLOCK;
    return err;
  }

  static cudaError_t launch(const RhsArgs& a, int grid, cudaStream_t s) {
    mix::dg_rhs_mixed_kernel<N, EQ, STAGE><<<grid, T::BLOCK, T::SMEM, s>>>(a);
    return cudaGetLastError();
  }
};

// f(MixedKernel<...>{}) for the runtime order and stage
template <int EQ, class F>
cudaError_t mixed_pick(int order, bool stage, F f) {
  switch (order) {
    case 1: return stage ? f(MixedKernel<1, EQ, true>{}) : f(MixedKernel<1, EQ, false>{});
    case 2: return stage ? f(MixedKernel<2, EQ, true>{}) : f(MixedKernel<2, EQ, false>{});
    case 3: return stage ? f(MixedKernel<3, EQ, true>{}) : f(MixedKernel<3, EQ, false>{});
    case 4: return stage ? f(MixedKernel<4, EQ, true>{}) : f(MixedKernel<4, EQ, false>{});
    default: return cudaErrorInvalidValue;
  }
}

template <int EQ>
cudaError_t mixed_shape_any(int order, bool stage, LaunchShape* out) {
  return mixed_pick<EQ>(order, stage, [&](auto k) { return k.shape(out); });
}

template <int EQ>
cudaError_t mixed_launch_any(int order, bool stage, const RhsArgs& a, int grid,
                             cudaStream_t s) {
  return mixed_pick<EQ>(order, stage, [&](auto k) { return k.launch(a, grid, s); });
}

}  // namespace
}  // namespace dg
