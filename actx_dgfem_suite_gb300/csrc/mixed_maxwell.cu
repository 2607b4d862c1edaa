// Mixed-precision RHS kernels of Maxwell's equations on the tensor cores
// (dg_mixed_mma.cuh): shapes, launches and operator block.
#include <cstring>

#include "dg_launch.h"
#include "dg_mixed_mma.cuh"

namespace dg {
namespace {

template <int N, bool STAGE>
struct Kernel {
  using T = mma::Tile<N>;

  static cudaError_t shape(LaunchShape* out) {
    auto kern = mma::dg_maxwell_mma_kernel<N, STAGE>;
    cudaError_t err = cudaFuncSetAttribute(
        kern, cudaFuncAttributeMaxDynamicSharedMemorySize, T::SMEM);
    if (err != cudaSuccess) return err;
    int nb = 0;
    err = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, kern, T::BLOCK, T::SMEM);
    out->smem_bytes = T::SMEM;
    out->blocks_per_sm = nb;
    out->elems_per_tile = T::E * T::WARPS;
    out->ops_bytes = mma::Ops<N>::SIZE;
    out->threads = T::BLOCK;
    return err;
  }

  static cudaError_t launch(const RhsArgs& a, int grid, cudaStream_t s) {
    mma::dg_maxwell_mma_kernel<N, STAGE><<<grid, T::BLOCK, T::SMEM, s>>>(a);
    return cudaGetLastError();
  }
};

template <class F>
cudaError_t pick(int order, bool stage, F f) {
  switch (order) {
    case 2: return stage ? f(Kernel<2, true>{}) : f(Kernel<2, false>{});
    case 3: return stage ? f(Kernel<3, true>{}) : f(Kernel<3, false>{});
    default: return cudaErrorInvalidValue;
  }
}

// Nearest TF32 value, ties away from zero (cvt.rna.tf32.f32).
uint32_t tf32(float x) {
  uint32_t u;
  std::memcpy(&u, &x, 4);
  return (u + 0x1000u) & 0xffffe000u;
}

// One operand word pair: high part at w, low part 128 words on.
void put(uint32_t* w, float x) {
  w[0] = tf32(x);
  float hi;
  std::memcpy(&hi, w, 4);
  w[128] = tf32(x - hi);
}

template <int N>
int pack(const double* diff, const double* lift, const int32_t* face_nodes,
         unsigned char* out, int out_bytes) {
  using O = mma::Ops<N>;
  if (!out) return O::SIZE;
  if (out_bytes < O::SIZE) return -1;
  std::memset(out, 0, O::SIZE);
  uint32_t* w = reinterpret_cast<uint32_t*>(out);
  for (int lane = 0; lane < 32; ++lane)
    for (int c = 0; c < 4; ++c) {  // operand word c: row lane / 4 + 8 (c % 2), column
      const int row = lane / 4, half = c & 1, col = lane % 4 + 4 * (c >> 1);
      for (int mt = 0; mt < O::VM; ++mt)
        for (int kt = 0; kt < O::VK; ++kt) {
          const int s = 2 * mt + half, r = s % 3, i = 8 * (s / 3) + row, j = 8 * kt + col;
          if (s / 3 < O::NG && i < O::NP && j < O::NP)
            put(w + (mt * O::VK + kt) * 256 + lane * 4 + c,
                (float)diff[(r * O::NP + i) * O::NP + j]);
        }
      for (int mt = 0; mt < O::LM; ++mt)
        for (int kt = 0; kt < O::LK; ++kt) {
          const int i = 8 * (2 * mt + half) + row, fj = 8 * kt + col;
          if (i < O::NP && fj < O::NFPT)
            put(w + O::L + (mt * O::LK + kt) * 256 + lane * 4 + c,
                (float)lift[i * O::NFPT + fj]);
        }
    }
  int32_t* fn = reinterpret_cast<int32_t*>(out + O::FN);
  for (int k = 0; k < O::NFPT; ++k) fn[k] = face_nodes[k];
  return O::SIZE;
}

}  // namespace

cudaError_t mma_shape_maxwell(int order, bool stage, LaunchShape* out) {
  return pick(order, stage, [&](auto k) { return k.shape(out); });
}
cudaError_t mma_launch_maxwell(int order, bool stage, const RhsArgs& a, int grid,
                               cudaStream_t s) {
  return pick(order, stage, [&](auto k) { return k.launch(a, grid, s); });
}
int pack_mma_ops(int order, const double* diff, const double* lift, const int32_t* face_nodes,
                 unsigned char* out, int out_bytes) {
  switch (order) {
    case 2: return pack<2>(diff, lift, face_nodes, out, out_bytes);
    case 3: return pack<3>(diff, lift, face_nodes, out, out_bytes);
    default: return -1;
  }
}

}  // namespace dg
