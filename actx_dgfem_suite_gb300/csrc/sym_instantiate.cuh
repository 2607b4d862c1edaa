// Shape and launch entry points of dg_rhs_sym_kernel for one equation, orders
// 1..4, plain RHS and Runge-Kutta stage.  Included by exactly one .cu file per
// equation.
#pragma once

#include "dg_launch.h"
#include "dg_sym.cuh"

namespace dg {
namespace {

template <int N, int EQ, bool STAGE>
struct SymKernel {
  using T = sym::Tile<N, EQ>;

  static cudaError_t shape(LaunchShape* out) {
    auto kern = sym::dg_rhs_sym_kernel<N, EQ, STAGE>;
    cudaError_t err = cudaFuncSetAttribute(
        kern, cudaFuncAttributeMaxDynamicSharedMemorySize, T::SMEM);
    if (err != cudaSuccess) return err;
    int nb = 0;
    err = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, kern, T::BLOCK, T::SMEM);
    out->smem_bytes = T::SMEM;
    out->blocks_per_sm = nb;
    out->elems_per_tile = T::E;
    out->ops_bytes = T::O::SIZE;
    out->threads = T::BLOCK;
    return err;
  }

  static cudaError_t launch(const RhsArgs& a, int grid, cudaStream_t s) {
    sym::dg_rhs_sym_kernel<N, EQ, STAGE><<<grid, T::BLOCK, T::SMEM, s>>>(a);
    return cudaGetLastError();
  }
};

// f(SymKernel<...>{}) for the runtime order and stage
template <int EQ, class F>
cudaError_t sym_pick(int order, bool stage, F f) {
  switch (order) {
    case 1: return stage ? f(SymKernel<1, EQ, true>{}) : f(SymKernel<1, EQ, false>{});
    case 2: return stage ? f(SymKernel<2, EQ, true>{}) : f(SymKernel<2, EQ, false>{});
    case 3: return stage ? f(SymKernel<3, EQ, true>{}) : f(SymKernel<3, EQ, false>{});
    case 4: return stage ? f(SymKernel<4, EQ, true>{}) : f(SymKernel<4, EQ, false>{});
    default: return cudaErrorInvalidValue;
  }
}

template <int EQ>
cudaError_t sym_shape_any(int order, bool stage, LaunchShape* out) {
  return sym_pick<EQ>(order, stage, [&](auto k) { return k.shape(out); });
}

template <int EQ>
cudaError_t sym_launch_any(int order, bool stage, const RhsArgs& a, int grid, cudaStream_t s) {
  return sym_pick<EQ>(order, stage, [&](auto k) { return k.launch(a, grid, s); });
}

}  // namespace
}  // namespace dg
