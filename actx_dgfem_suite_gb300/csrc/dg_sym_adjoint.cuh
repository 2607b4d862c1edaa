// Adjoint volume kernels in the symmetry-adapted basis of the tetrahedron
// (dg_sym.cuh): the transposed derivatives and the transposed LIFT split into
// the same four blocks, so the products cost a quarter of the dense ones on
// the FP64 pipe that bounds them.
//
//   dg_wave_adjoint_sym_kernel   replaces dg_wave_adjoint_volume: the volume
//     transpose into y and the lifted face adjoints a_u, a_v.  The dense kernel
//     lifts u and n_f.v (two fields, the normal inside); here u and the three
//     components of v are lifted (the parts mix faces, so the normal follows):
//     4 x 525 instead of 2 x 2100 multiply-adds at order 4.
//   dg_euler_vjp_sym_kernel      replaces dg_euler_vjp_volume: per direction k
//     T_k = D'_k^T x back at the nodes, then y += J(h_k)^T T_k with the flux
//     Jacobian in direction h_k (linear in the direction, so the metric needs no
//     combinations of its own: 3 Jacobian products of 36 operations per node,
//     where the dense kernel formed 45 combinations and 3 products of ~60);
//     and the lifted adjoints of the five fields.
//
// Measured (GB300, ncu launch times, dense -> here): see the kernels.
// Operators without the symmetry keep the dense kernels.
#pragma once

#include "dg_adjoint.cuh"
#include "dg_adjoint_euler.cuh"
#include "dg_sym.cuh"

namespace dg {
namespace sym {

// Shared memory: operator block, inputs x (NF arrays), a second area that holds
// one chunk of face adjoints at a time (Euler: or the transformed T_k), metric
// and (wave) face geometry and per-node products of the c-gradient.
template <int N, int EQ>
struct AdjTile {
  using B = Basis<N>;
  using O = AdjOps<N, EQ == DG_WAVE && N != 1 ? RED_OUT : RED_NONE>;
  static constexpr int NF = EqInfo<EQ>::NF;
  static constexpr int E = 32, PE = E + 1, BLOCK = 128;
  static constexpr int X = O::SIZE;
  static constexpr int X_BYTES = pad16(NF * B::NP * PE * 8);
  static constexpr int F_BYTES = pad16(NF * 4 * O::CH * PE * 8);
  static constexpr int F = X + X_BYTES;
  static constexpr int H =
      F + (EQ == DG_EULER && X_BYTES > F_BYTES ? X_BYTES : F_BYTES);
  static constexpr int FG = H + pad16(9 * PE * 8);
  static constexpr int PART = FG + (EQ == DG_WAVE ? pad16(16 * PE * 8) : 0);
  static constexpr int SMEM = PART + (EQ == DG_WAVE ? pad16(B::NP * PE * 8) : 0);
};

// Stage the operator block; false if the copy timed out.
__device__ __forceinline__ bool stage_ops(unsigned char* smem, const void* ops, uint32_t bytes,
                                          int* status) {
  __shared__ uint64_t bar;
  __shared__ int ok_s;
  if (threadIdx.x == 0) {
    mbar_init(&bar, 1);
    mbar_arrive_expect_tx(&bar, bytes);
    bulk_g2s(smem, ops, bytes, &bar);
    const bool ok = mbar_wait_bounded(&bar, 0);
    if (!ok) {
      raise_status(status, DG_ERR_TIMEOUT);
      mbar_wait_bounded(&bar, 0);  // give the copy one more bounded chance
    }
    ok_s = ok ? 1 : 0;
  }
  __syncthreads();
  return ok_s != 0;
}

// Direction metric of the tile's elements: h_1 = g_2 + g_3 (cyclic).
template <int PE, int E, int BLOCK>
__device__ __forceinline__ void load_metric(const double* mt, int ecount, double* sH) {
  for (int idx = threadIdx.x; idx < 9 * E; idx += BLOCK) {
    const int el = idx / 9, kx = idx - el * 9, k = kx / 3, x = kx - k * 3;
    double v = 0.0;
    if (el < ecount)
      v = __ldg(mt + el * 9 + (k == 0 ? 3 : 0) + x) + __ldg(mt + el * 9 + (k == 2 ? 3 : 6) + x);
    sH[kx * PE + el] = v;
  }
}

// The chunk's face adjoints of part rho (DIN inputs) into sF (transformed).
template <int N, class O, int NF, int DIN, int PE>
__device__ __forceinline__ void lift_transposed(const double* __restrict__ x,
                                                const double* __restrict__ row, int rho,
                                                double* __restrict__ f) {
  using B = Basis<N>;
  constexpr int XS = B::NP * PE, FS = 4 * O::CH * PE;
  double acc[NF][O::CH];
#pragma unroll
  for (int m = 0; m < NF; ++m)
#pragma unroll
    for (int o = 0; o < O::CH; ++o) acc[m][o] = 0.0;
#pragma unroll 1
  for (int j = 0; j < DIN; ++j, row += O::PC, x += PE) {
    double v[NF], t[O::PC];
#pragma unroll
    for (int m = 0; m < NF; ++m) v[m] = x[m * XS];
    load_row<O::PC>(row, t);
#pragma unroll
    for (int m = 0; m < NF; ++m)
#pragma unroll
      for (int o = 0; o < O::CH; ++o) acc[m][o] = fma(t[o], v[m], acc[m][o]);
  }
  f += rho * O::CH * PE;
#pragma unroll
  for (int m = 0; m < NF; ++m)
#pragma unroll
    for (int o = 0; o < O::CH; ++o) f[m * FS + o * PE] = acc[m][o];
}

// f(DIN, R, slot0): the part's size and its volume blocks' as compile-time constants
template <int N, class O, class F>
__device__ __forceinline__ void with_part(int rho, F f) {
  using B = Basis<N>;
  if ((B::DA != B::DB || O::F::RA != O::F::RB) && rho == 0)
    f(std::integral_constant<int, B::DA>{}, std::integral_constant<int, O::F::RA>{}, 0);
  else
    f(std::integral_constant<int, B::DB>{}, std::integral_constant<int, O::F::RB>{},
      rho == 0 ? 0 : B::DA + (rho - 1) * B::DB);
}

// Wave P3, 16,464 tets, reverse stage: 177 us dense, 127 us here (vjp at 82,944 tets,
// both launches, with the derivatives reduced as in dg_sym.cuh: 572 -> 557 us).
template <int N, bool STAGE>
__global__ void __launch_bounds__(AdjTile<N, DG_WAVE>::BLOCK)
    dg_wave_adjoint_sym_kernel(const AdjArgs a) {
  using T = AdjTile<N, DG_WAVE>;
  using O = typename T::O;
  using B = Basis<N>;
  constexpr int NP = B::NP, NFP = B::NFP, NFPT = B::NFPT, CH = O::CH;
  constexpr int E = T::E, PE = T::PE, BLOCK = T::BLOCK, XS = NP * PE, FS = 4 * CH * PE;
  extern __shared__ __align__(128) unsigned char smem[];
  const double* ops = reinterpret_cast<const double*>(smem);
  const int* node_slot = reinterpret_cast<const int*>(smem + O::NODE_SLOT);
  const int* face_point = reinterpret_cast<const int*>(smem + O::FACE_POINT);
  double* sX = reinterpret_cast<double*>(smem + T::X);
  double* sF = reinterpret_cast<double*>(smem + T::F);
  double* sH = reinterpret_cast<double*>(smem + T::H);
  double* sFG = reinterpret_cast<double*>(smem + T::FG);
  [[maybe_unused]] double* sPart = reinterpret_cast<double*>(smem + T::PART);
  if (!stage_ops(smem, a.sym_ops, a.sym_ops_bytes, a.status)) return;

  const int t = threadIdx.x, le = t & 31;
  const int64_t nel = a.nel, nelnp = nel * NP;
  const int64_t ntiles = (nel + E - 1) / E;
  for (int64_t tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
    const int64_t e0 = tile * E;
    const int ecount = (nel - e0) < (int64_t)E ? (int)(nel - e0) : E;
    // {{{ c s_e rbar -> slots; products for the c-gradient; geometry
    {
      const double* xk = a.x + e0 * NP;
      const double* lk = STAGE && a.lq ? a.lq + e0 * NP : nullptr;
      const double xs = STAGE ? a.xscale : 1.0;
      for (int rem = t; rem < E * NP; rem += BLOCK) {
        const int el = rem / NP, node = rem - el * NP;
        double* x = sX + node_slot[node] * PE + el;
        const bool in = rem < ecount * NP;
        const double sc = in && a.elem_scale ? __ldg(a.elem_scale + e0 + el) : 1.0;
        double part = 0.0;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          double v = 0.0;
          if (in) {
            const double rb = xs * __ldg(xk + k * nelnp + rem);
            if (STAGE && lk) part = fma(rb, __ldg(lk + k * nelnp + rem), part);
            v = a.c * rb;
            if (a.elem_scale) v *= sc;
          }
          x[k * XS] = v;
        }
        if (STAGE && lk) sPart[node * PE + el] = part;
      }
      load_metric<PE, E, BLOCK>(a.metric + e0 * 9, ecount, sH);
      const double* ft = a.face_geom + e0 * 16;
      for (int idx = t; idx < 16 * E; idx += BLOCK) {
        const int el = idx / 16;
        sFG[(idx - el * 16) * PE + el] = el < ecount ? __ldg(ft + idx) : 0.0;
      }
    }
    __syncthreads();
    if (STAGE && a.lq && a.cbar && t < ecount) {
      double g = 0.0;  // the element's <rbar_s, lq>, fixed order
      for (int j = 0; j < NP; ++j) g += sPart[j * PE + t];
      a.cbar[e0 + t] += a.dt * g;
    }
    transform<N, PE, E, BLOCK>(sX, 4);
    __syncthreads();
    // }}}

    const int rho = ((t >> 5) + (int)tile) & 3;  // parts rotate over the warps

    // {{{ lifted face adjoints, one chunk of orbits at a time
#pragma unroll 1
    for (int c = 0; c < O::NCH; ++c) {
      const double* lops = ops + O::LIFT + c * O::CHUNK;
      with_part<N, O>(rho, [&](auto dtag, auto, int slot0) {
        lift_transposed<N, O, 4, decltype(dtag)::value, PE>(sX + slot0 * PE + le,
                                                         lops + slot0 * O::PC, rho, sF + le);
      });
      __syncthreads();
      for (int idx = t; idx < ecount * CH; idx += BLOCK) {
        const int el = idx / CH, oc = idx - el * CH, o = c * CH + oc;
        if (NFP % CH != 0 && o >= NFP) continue;
        double z[4][4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
#pragma unroll
          for (int r = 0; r < 4; ++r) z[k][r] = sF[k * FS + (r * CH + oc) * PE + el];
          butterfly(z[k][0], z[k][1], z[k][2], z[k][3]);
        }
        double* sc = a.face_scratch + (e0 + el) * (2 * NFPT);
#pragma unroll
        for (int r = 0; r < 4; ++r) {  // the orbit's point on each face
          const int fj = face_point[r * NFP + o];
          const double* fg = sFG + (fj / NFP) * 4 * PE + el;
          const double s = fg[3 * PE];
          sc[fj] = s * z[0][r];
          sc[NFPT + fj] =
              s * fma(fg[0], z[1][r], fma(fg[PE], z[2][r], fg[2 * PE] * z[3][r]));
        }
      }
      __syncthreads();
    }
    // }}}

    // {{{ volume transpose: -sum_r W_r^T (G v)_r and -G^T W_r^T u
    with_part<N, O>(rho, [&](auto dtag, auto rtag, int slot0) {
      constexpr int D = decltype(dtag)::value, R = decltype(rtag)::value;
      double acc[4][D], c[4][R];
#pragma unroll
      for (int m = 0; m < 4; ++m)
#pragma unroll
        for (int i = 0; i < R; ++i) c[m][i] = 0.0;
      volume<N, DG_WAVE, R, (R + 1) & ~1, B::DA, B::DB, true>(
          sX + le, sH + le, ops + O::F::volume(rho), rho, 0, -1.0, c);
#pragma unroll
      for (int m = 0; m < 4; ++m)
#pragma unroll
        for (int i = 0; i < D; ++i) acc[m][i] = N == 1 ? c[m][i % R] : 0.0;
      if constexpr (N != 1)
        expand<4, R, D, (D + 1) & ~1>(ops + O::F::extra(rho), c, acc);
      cta_sync<BLOCK>();  // every warp has read its inputs
#pragma unroll
      for (int m = 0; m < 4; ++m)
#pragma unroll
        for (int i = 0; i < D; ++i) sX[m * XS + (slot0 + i) * PE + le] = acc[m][i];
    });
    __syncthreads();
    transform<N, PE, E, BLOCK>(sX, 4);
    __syncthreads();
    for (int rem = t; rem < ecount * NP; rem += BLOCK) {
      const int el = rem / NP;
      const double* y = sX + node_slot[rem - el * NP] * PE + el;
#pragma unroll
      for (int k = 0; k < 4; ++k) a.y[k * nelnp + e0 * NP + rem] = y[k * XS];
    }
    __syncthreads();
    // }}}
  }
}

// Euler P3, 82,944 tets: 1.93 ms dense, 1.07 ms here, 0.94 with the shorter flux adjoint
// (euler_flux_vjp).
template <int N>
__global__ void __launch_bounds__(AdjTile<N, DG_EULER>::BLOCK)
    dg_euler_vjp_sym_kernel(const VjpArgs a) {
  using T = AdjTile<N, DG_EULER>;
  using O = typename T::O;
  using B = Basis<N>;
  constexpr int NP = B::NP, NFP = B::NFP, NFPT = B::NFPT, CH = O::CH;
  constexpr int DA = B::DA, DB = B::DB, NO4 = B::NO4;
  constexpr int E = T::E, PE = T::PE, BLOCK = T::BLOCK, XS = NP * PE, FS = 4 * CH * PE;
  extern __shared__ __align__(128) unsigned char smem[];
  const double* ops = reinterpret_cast<const double*>(smem);
  const int* node_slot = reinterpret_cast<const int*>(smem + O::NODE_SLOT);
  const int* slot_node = reinterpret_cast<const int*>(smem + O::SLOT_NODE);
  const int* face_point = reinterpret_cast<const int*>(smem + O::FACE_POINT);
  double* sX = reinterpret_cast<double*>(smem + T::X);
  double* sF = reinterpret_cast<double*>(smem + T::F);  // face adjoints, or T_k
  double* sH = reinterpret_cast<double*>(smem + T::H);
  if (!stage_ops(smem, a.sym_ops, a.sym_ops_bytes, a.status)) return;

  const int t = threadIdx.x, le = t & 31;
  const int64_t nel = a.nel, nelnp = nel * NP, nfpt_all = nel * NFPT;
  const int64_t ntiles = (nel + E - 1) / E;
  for (int64_t tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
    const int64_t e0 = tile * E;
    const int ecount = (nel - e0) < (int64_t)E ? (int)(nel - e0) : E;
    // L = diag(s_e) L_1  =>  L^T x = L_1^T (s_e x)
    for (int rem = t; rem < E * NP; rem += BLOCK) {
      const int el = rem / NP;
      double* x = sX + node_slot[rem - el * NP] * PE + el;
      const bool in = rem < ecount * NP;
      const double sc = in && a.elem_scale ? __ldg(a.elem_scale + e0 + el) : 1.0;
#pragma unroll
      for (int k = 0; k < 5; ++k) {
        double v = in ? __ldg(a.x + k * nelnp + e0 * NP + rem) : 0.0;
        if (a.elem_scale) v *= sc;
        x[k * XS] = v;
      }
    }
    load_metric<PE, E, BLOCK>(a.metric + e0 * 9, ecount, sH);
    __syncthreads();
    transform<N, PE, E, BLOCK>(sX, 5);
    __syncthreads();
    const int rho = ((t >> 5) + (int)tile) & 3;  // parts rotate over the warps

    // {{{ lifted adjoints w_k(fj) = sum_i LIFT[i][fj] x_k(i) (unscaled)
#pragma unroll 1
    for (int c = 0; c < O::NCH; ++c) {
      const double* lops = ops + O::LIFT + c * O::CHUNK;
      with_part<N, O>(rho, [&](auto dtag, auto, int slot0) {
        lift_transposed<N, O, 5, decltype(dtag)::value, PE>(sX + slot0 * PE + le,
                                                         lops + slot0 * O::PC, rho, sF + le);
      });
      __syncthreads();
      for (int idx = t; idx < ecount * CH; idx += BLOCK) {
        const int el = idx / CH, oc = idx - el * CH, o = c * CH + oc;
        if (NFP % CH != 0 && o >= NFP) continue;
        double* sc = a.scratch + (e0 + el) * NFPT;
        int fj[4];
#pragma unroll
        for (int r = 0; r < 4; ++r) fj[r] = face_point[r * NFP + o];
#pragma unroll
        for (int k = 0; k < 5; ++k, sc += nfpt_all) {
          double z[4];
#pragma unroll
          for (int r = 0; r < 4; ++r) z[r] = sF[k * FS + (r * CH + oc) * PE + el];
          butterfly(z[0], z[1], z[2], z[3]);
#pragma unroll
          for (int r = 0; r < 4; ++r) sc[fj[r]] = z[r];
        }
      }
      __syncthreads();
    }
    // }}}

    // {{{ volume: per direction, T_k at the nodes, then y += J(h_k)^T T_k
#pragma unroll 1
    for (int k = 0; k < 3; ++k) {
      with_part<N, O>(rho, [&](auto dtag, auto, int slot0) {
        constexpr int D = decltype(dtag)::value, P = (D + 1) & ~1;
        double acc[5][D];
#pragma unroll
        for (int m = 0; m < 5; ++m)
#pragma unroll
          for (int i = 0; i < D; ++i) acc[m][i] = 0.0;
        const int sig = rho ^ (k + 1);
        const double* row = ops + O::F::volume(rho);
        for (int k2 = 0; k2 < k; ++k2) row += ((rho ^ (k2 + 1)) == 0 ? DA : DB) * P;
        if (N != 1 || rho == 0)  // order 1: transposed weak derivatives reach part A
          block_product<5, D, P, PE, XS>(sX + (sig == 0 ? 0 : DA + (sig - 1) * DB) * PE + le,
                                         row, sig == 0 ? DA : DB, acc);
#pragma unroll
        for (int m = 0; m < 5; ++m)
#pragma unroll
          for (int i = 0; i < D; ++i) sF[m * XS + (slot0 + i) * PE + le] = acc[m][i];
      });
      __syncthreads();
      // the orbit of CNT nodes at the given slots: the same thread adds to the
      // same nodes of y for every direction
      auto orbit = [&](auto tag, int el, int s0, int s1, int s2, int s3) {
        constexpr int CNT = decltype(tag)::value;
        if (el >= ecount) return;
        const int slot[4] = {s0, s1, s2, s3};
        double z[5][CNT];
        const double* x = sF + el;
#pragma unroll
        for (int m = 0; m < 5; ++m, x += XS) {
#pragma unroll
          for (int n = 0; n < CNT; ++n) z[m][n] = x[slot[n] * PE];
          if constexpr (CNT == 4) {
            butterfly(z[m][0], z[m][1], z[m][2], z[m][3]);
          } else if constexpr (CNT == 2) {
            const double s = z[m][0] + z[m][1], d = z[m][0] - z[m][1];
            z[m][0] = s;
            z[m][1] = d;
          }
        }
        const double* h = sH + k * 3 * PE + el;
        const double h0 = h[0], h1 = h[PE], h2 = h[2 * PE];
#pragma unroll
        for (int n = 0; n < CNT; ++n) {
          const int64_t g = (e0 + el) * NP + slot_node[slot[n]];
          double q[5], w[5], y[5];
#pragma unroll
          for (int m = 0; m < 5; ++m) {
            q[m] = __ldg(a.q + m * nelnp + g);
            w[m] = z[m][n];
            y[m] = k == 0 ? 0.0 : a.y[m * nelnp + g];
          }
          euler_flux_vjp(q, __ldg(a.aux + nelnp + g), __ldg(a.aux + g), h0, h1, h2, w, a.gamma,
                         y);
#pragma unroll
          for (int m = 0; m < 5; ++m) a.y[m * nelnp + g] = y[m];
        }
      };
      for (int idx = t; idx < E * NO4; idx += BLOCK) {
        const int el = idx / NO4, o = idx - el * NO4;
        orbit(std::integral_constant<int, 4>{}, el, o, DA + o, DA + DB + o, DA + 2 * DB + o);
      }
      if constexpr (B::NPR > 0)
        for (int idx = BLOCK - 1 - t; idx < E * 3; idx += BLOCK) {
          const int el = idx / 3, d = idx - el * 3;
          orbit(std::integral_constant<int, 2>{}, el, NO4 + d, DA + d * DB + NO4, 0, 0);
        }
      if constexpr (B::NSG > 0)
        for (int el = t; el < E; el += BLOCK)
          orbit(std::integral_constant<int, 1>{}, el, DA - 1, 0, 0, 0);
      __syncthreads();
    }
    // }}}
  }
}

}  // namespace sym
}  // namespace dg
