// Symmetry-adapted RHS kernels on triangle meshes (dg_sym2d.cuh): wave, euler and
// maxwell (TM) at orders 1..4, plain RHS and fused RK stage; shape and launch entry
// points and the operator block.
#include <cmath>
#include <cstring>
#include <vector>

#include "dg_launch.h"
#include "dg_pair.h"
#include "dg_sym2d.cuh"

namespace dg {
namespace {

template <int N, int EQ, int MODE>
struct Kernel {
  using T = sym2::Tile<N, EQ>;

  static cudaError_t shape(LaunchShape* out) {
    auto kern = sym2::dg_rhs2d_sym_kernel<N, EQ, MODE>;
    cudaError_t err = cudaFuncSetAttribute(
        kern, cudaFuncAttributeMaxDynamicSharedMemorySize, T::SMEM);
    if (err != cudaSuccess) return err;
    int nb = 0;
    err = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, kern, T::BLOCK, T::SMEM);
    out->smem_bytes = T::SMEM;
    out->blocks_per_sm = nb;
    out->elems_per_tile = T::E;
    out->ops_bytes = sym2::Ops<N>::SIZE;
    out->threads = T::BLOCK;
    return err;
  }

  static cudaError_t launch(const RhsArgs& a, int grid, cudaStream_t s) {
    sym2::dg_rhs2d_sym_kernel<N, EQ, MODE><<<grid, T::BLOCK, T::SMEM, s>>>(a);
    return cudaGetLastError();
  }
};

template <int N, int EQ, class F>
cudaError_t pick_mode(int mode, F f) {
  return mode == MODE_RHS ? f(Kernel<N, EQ, MODE_RHS>{}) : f(Kernel<N, EQ, MODE_STAGE>{});
}

template <int EQ, class F>
cudaError_t pick_order(int order, int mode, F f) {
  switch (order) {
    case 1: return pick_mode<1, EQ>(mode, f);
    case 2: return pick_mode<2, EQ>(mode, f);
    case 3: return pick_mode<3, EQ>(mode, f);
    case 4: return pick_mode<4, EQ>(mode, f);
    default: return cudaErrorInvalidValue;
  }
}

template <class F>
cudaError_t pick(int eq, int order, int mode, F f) {
  if (mode != MODE_RHS && mode != MODE_STAGE) return cudaErrorInvalidValue;
  switch (eq) {
    case DG_WAVE: return pick_order<DG_WAVE>(order, mode, f);
    case DG_EULER: return pick_order<DG_EULER>(order, mode, f);
    case DG_MAXWELL: return pick_order<DG_MAXWELL>(order, mode, f);
    default: return cudaErrorInvalidValue;
  }
}

// as in sym_ops.cu: entries outside the pattern beyond this fraction of the largest
// one mean that the operators are not symmetric
constexpr double kAsymmetry = 5e-14;

struct Vec {  // a point on the mirror line, or the sum (difference) of a pair
  int n = 0;
  int idx[2] = {0, 0};
  int sign = 1;
};

template <int N>
int pack(const double* diff, const double* lift, const int32_t* edge_nodes, unsigned char* out,
         int out_bytes) {
  using B = sym2::Basis<N>;
  using O = sym2::Ops<N>;
  constexpr int NP = B::NP, NFP = B::NFP, NFPT = B::NFPT;
  if (!out) return O::SIZE;
  if (out_bytes < O::SIZE) return -1;
  // {{{ the swap of vertices 1 and 2 on nodes (multi-indices (i, j), i fastest) and
  // on edge points
  int index[N + 1][N + 1], mi[NP][2], perm[NP], fperm[NFPT];
  {
    int n = 0;
    for (int j = 0; j <= N; ++j)
      for (int i = 0; i <= N - j; ++i, ++n) {
        index[i][j] = n;
        mi[n][0] = i;
        mi[n][1] = j;
      }
    for (int k = 0; k < NP; ++k) perm[k] = index[mi[k][1]][mi[k][0]];
  }
  for (int f = 0; f < 3; ++f) {
    int target = -1;
    for (int f2 = 0; f2 < 3 && target < 0; ++f2) {
      bool all = true;
      for (int j = 0; j < NFP; ++j) {
        bool found = false;
        for (int j2 = 0; j2 < NFP; ++j2)
          found = found || edge_nodes[f2 * NFP + j2] == perm[edge_nodes[f * NFP + j]];
        all = all && found;
      }
      if (all) target = f2;
    }
    if (target < 0) return -1;
    for (int j = 0; j < NFP; ++j)
      for (int j2 = 0; j2 < NFP; ++j2)
        if (edge_nodes[target * NFP + j2] == perm[edge_nodes[f * NFP + j]])
          fperm[f * NFP + j] = target * NFP + j2;
  }
  // }}}

  // slots of `n` points under the swap p: pairs at (o, even + o), fixed points
  // after the pairs; false if their numbers are not the basis's
  auto slots = [](const int* p, int n, int npr, int nfx, Vec* by_slot, int* slot_of) {
    int pairs = 0, fixed = 0;
    const int even = npr + nfx;
    for (int k = 0; k < n; ++k) {
      if (p[k] < 0 || p[k] >= n || p[p[k]] != k) return false;
      if (p[k] < k) continue;
      if (p[k] == k) {
        if (fixed == nfx) return false;
        Vec& v = by_slot[npr + fixed];
        v.n = 1;
        v.idx[0] = k;
        slot_of[k] = npr + fixed++;
      } else {
        if (pairs == npr) return false;
        for (int odd = 0; odd < 2; ++odd) {
          Vec& v = by_slot[odd * even + pairs];
          v.n = 2;
          v.idx[0] = k;
          v.idx[1] = p[k];
          v.sign = odd ? -1 : 1;
        }
        slot_of[k] = pairs;
        slot_of[p[k]] = even + pairs++;
      }
    }
    return pairs == npr && fixed == nfx;
  };
  Vec node[NP], edge[NFPT];
  int node_slot[NP], edge_slot[NFPT];
  if (!slots(perm, NP, B::NPR, B::NFX, node, node_slot) ||
      !slots(fperm, NFPT, B::FPR, B::FFX, edge, edge_slot))
    return -1;

  // the operator in the basis of sums and differences, normalised for plain sums
  // on both sides; false unless the entries outside the pattern vanish
  std::vector<double> full;
  auto to_basis = [&](const Vec* in, int cols, int even, int flip, auto at) {
    full.assign((size_t)NP * cols, 0.0);
    double big = 0.0, off = 0.0;
    for (int i = 0; i < NP; ++i)
      for (int c = 0; c < cols; ++c) {
        Pair s;
        for (int a = 0; a < node[i].n; ++a)
          for (int b = 0; b < in[c].n; ++b)
            s.add((a ? node[i].sign : 1) * (b ? in[c].sign : 1),
                  at(node[i].idx[a], in[c].idx[b]));
        const double x = s.hi / (node[i].n * in[c].n);  // powers of two
        full[(size_t)i * cols + c] = x;
        if (!std::isfinite(x)) return false;
        const bool inside = ((i >= B::DE) ^ (c >= even)) == (flip != 0);
        double& m = inside ? big : off;
        if (std::fabs(x) > m) m = std::fabs(x);
      }
    return off <= kAsymmetry * big;
  };
  std::memset(out, 0, O::SIZE);
  double* ops = reinterpret_cast<double*>(out);
  for (int k = 0; k < 2; ++k) {
    // D' = (D_1 + D_2) / 2 and (D_1 - D_2) / 2
    if (!to_basis(node, NP, B::DE, k, [&](int i, int j) {
          Pair s;
          s.add(0.5, diff[(size_t)i * NP + j]);
          return s.add(k == 0 ? 0.5 : -0.5, diff[(size_t)(NP + i) * NP + j]);
        }))
      return -1;
    for (int r = 0; r < 2; ++r) {
      const int pitch = r == 0 ? O::PE : O::PO, d = r == 0 ? B::DE : B::DO, s = r ^ k;
      const int din = s == 0 ? B::DE : B::DO;
      const int skip = k == 0 ? 0 : (r == 0 ? B::DE : B::DO);  // rows of direction 0
      double* dst = ops + (r == 0 ? 0 : O::VOL1) + skip * pitch;
      for (int j = 0; j < din; ++j)
        for (int i = 0; i < d; ++i)
          dst[j * pitch + i] =
              full[(size_t)(r * B::DE + i) * NP + s * B::DE + j];
    }
  }
  if (!to_basis(edge, NFPT, B::FE, 0,
                [&](int i, int fj) { return Pair(lift[(size_t)i * NFPT + fj]); }))
    return -1;
  for (int r = 0; r < 2; ++r) {
    const int pitch = r == 0 ? O::PE : O::PO, d = r == 0 ? B::DE : B::DO;
    double* dst = ops + (r == 0 ? O::LIFT0 : O::LIFT1);
    for (int o = 0; o < (r == 0 ? B::FE : B::FO); ++o)
      for (int i = 0; i < d; ++i)
        dst[o * pitch + i] = full[(size_t)(r * B::DE + i) * NFPT + r * B::FE + o];
  }
  int32_t* ns = reinterpret_cast<int32_t*>(out + O::NODE_SLOT);
  int32_t* sn = reinterpret_cast<int32_t*>(out + O::SLOT_NODE);
  int32_t* es = reinterpret_cast<int32_t*>(out + O::EDGE_SLOT);
  int32_t* en = reinterpret_cast<int32_t*>(out + O::EDGE_NODE);
  for (int n = 0; n < NP; ++n) {
    ns[n] = node_slot[n];
    sn[node_slot[n]] = n;
  }
  for (int fj = 0; fj < NFPT; ++fj) {
    es[fj] = edge_slot[fj];
    en[fj] = edge_nodes[fj];
  }
  return O::SIZE;
}

}  // namespace

cudaError_t sym_shape_2d(int eq, int order, int mode, LaunchShape* out) {
  return pick(eq, order, mode, [&](auto k) { return k.shape(out); });
}

cudaError_t sym_launch_2d(int eq, int order, int mode, const RhsArgs& a, int grid,
                          cudaStream_t s) {
  return pick(eq, order, mode, [&](auto k) { return k.launch(a, grid, s); });
}

int pack_sym_ops_2d(int order, const double* diff, const double* lift,
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
