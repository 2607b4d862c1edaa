// DG-FEM RHS kernel for affine triangles in the basis adapted to the triangle's
// mirror symmetry (sm_103a, FP64), one launch per RHS or RK stage.
//
// Like the dense kernel (dg_rhs2d.cuh) it is bound by the FP64 pipe (two
// multiply-adds per SM and clock), so it spends fewer FP64 operations:
//
//   * the swap of vertices 1 and 2 maps node set and operators to themselves; sums
//     and differences over the node pairs split a field into an even and an odd
//     part.  The derivative along e_1 + e_2 keeps the parts, the one along
//     e_1 - e_2 exchanges them, LIFT keeps them (edge 0-1 and 0-2 swap, edge 1-2
//     reverses): half the multiply-adds of the dense products (order 3, per field:
//     104 instead of 200 for both derivatives, 60 instead of 120 for LIFT);
//   * an edge whose two sides both lie in the tile has its flux evaluated once,
//     and only exterior traces from outside the tile recompute pressure, 1/rho and
//     wave speed (Euler); a row of squares puts two thirds of a tile's edge sides
//     inside it.  Which sides glue is read off the gather index, point by point
//     and in both directions, and off the normals (opposite to 1e-12), for every tile;
//     sides that do not match are evaluated on their own.  Sides with outside traces
//     come first in the work list, because an FP64 instruction takes the pipe for
//     a whole warp however few lanes need it.
//
// Measured (GB300, whole RHS on 80,000 triangles, dense -> here, us): wave P1-P4
// 50 / 95 / 184 / 306 -> 47 / 81 / 134 / 202, Euler 150 / 257 / 460 / 712 -> 103 / 185 /
// 290 / 465, Maxwell 56 / 109 / 216 / 374 -> 52 / 86 / 144 / 213.  ncu (Euler P3,
// 180,000 triangles): FP64 pipe 88 % busy.
//
// One lane per element, 32 elements per tile, two warps per part (each for a part of
// the fields); operator entries are warp-uniform broadcasts.  The metric of the two directions is g_1 + g_2 and
// g_1 - g_2 with D' = D_d / 2.  Operators without the symmetry (checked when the
// plan is made, pack_sym_ops_2d) and meshes too small for it (dg_plan_create_2d)
// keep the dense kernel.
#pragma once

#include "dg_rhs2d.cuh"
#include "dg_sym.cuh"  // cta_sync

namespace dg {
namespace sym2 {

// NFX nodes on the mirror line, NPR mirrored pairs; the same for edge points.
template <int N>
struct Basis {
  static constexpr int NP = Shape2<N>::NP, NFP = Shape2<N>::NFP, NFPT = 3 * NFP;
  static constexpr int NFX = N / 2 + 1, NPR = (NP - NFX) / 2;
  static constexpr int DE = NPR + NFX, DO = NPR;
  static constexpr int FFX = N % 2 == 0 ? 1 : 0, FPR = (NFPT - FFX) / 2;
  static constexpr int FE = FPR + FFX, FO = FPR;
  static_assert(DE + DO == NP && FE + FO == NFPT, "the parts cover all points");
};

// Operator block: rows of one input padded to 16 bytes.  Even part: direction 0
// (even inputs), direction 1 (odd inputs); odd part: direction 0 (odd inputs),
// direction 1 (even inputs); LIFT of the even, then the odd part; tables node ->
// slot, slot -> node, edge point -> slot, edge point -> node.  Slots: even part (pairs, then
// fixed points), then the odd part.
template <int N>
struct Ops {
  using B = Basis<N>;
  static constexpr int PE = (B::DE + 1) & ~1, PO = (B::DO + 1) & ~1;
  static constexpr int VOL1 = (B::DE + B::DO) * PE;          // the odd part's blocks
  static constexpr int LIFT0 = VOL1 + (B::DE + B::DO) * PO;
  static constexpr int LIFT1 = LIFT0 + B::FE * PE;
  static constexpr int ENTRIES = LIFT1 + B::FO * PO;
  static constexpr int NODE_SLOT = ENTRIES * 8;              // bytes from here
  static constexpr int SLOT_NODE = NODE_SLOT + pad16(B::NP * 4);
  static constexpr int EDGE_SLOT = SLOT_NODE + pad16(B::NP * 4);
  static constexpr int EDGE_NODE = EDGE_SLOT + pad16(B::NFPT * 4);
  static constexpr int SIZE = EDGE_NODE + pad16(B::NFPT * 4);
};

template <int N, int EQ>
struct Tile {
  using B = Basis<N>;
  static constexpr int NF = Eq2<EQ>::NF, E = 32, PE = E + 1, BLOCK = 128;
  static constexpr int NQ = NF + Eq2<EQ>::NNODE;  // state; Euler: p, 1/rho, |u| + c
  static constexpr int NSIDE = 3 * E;
  static constexpr int Q = Ops<N>::SIZE;
  static constexpr int X = Q + pad16(NQ * B::NP * PE * 8);     // inputs, then result
  static constexpr int F = X + pad16(NF * B::NP * PE * 8);     // edge values
  static constexpr int H = F + pad16(NF * B::NFPT * PE * 8);
  static constexpr int FG = H + pad16(4 * PE * 8);
  static constexpr int GAT = FG + pad16(9 * PE * 8);
  static constexpr int MATE = GAT + pad16(B::NFPT * PE * 4);
  static constexpr int LIST = MATE + pad16(NSIDE * 4);
  static constexpr int SMEM = LIST + pad16((NSIDE + 1) * 4);
};

// acc += block * fields for `rows` inputs
template <int NA, int D, int P, int PE, int FS>
__device__ __forceinline__ void block_product(const double* __restrict__ x,
                                              const double* __restrict__ row, int rows,
                                              double (&acc)[NA][D]) {
#pragma unroll 1
  for (int j = 0; j < rows; ++j, row += P, x += PE) {
    double v[NA], t[P];
#pragma unroll
    for (int m = 0; m < NA; ++m) v[m] = x[m * FS];
#pragma unroll
    for (int k = 0; k < P; k += 2) {
      const double2 w = *reinterpret_cast<const double2*>(row + k);
      t[k] = w.x;
      t[k + 1] = w.y;
    }
#pragma unroll
    for (int m = 0; m < NA; ++m)
#pragma unroll
      for (int i = 0; i < D; ++i) acc[m][i] = fma(t[i], v[m], acc[m][i]);
  }
}

// Sums and differences over the pairs of `narrays` arrays (pairs npr, odd part at
// slot `odd`), in place.
template <int PE, int BLOCK>
__device__ __forceinline__ void mirror(double* x, int narrays, int stride, int npr, int odd) {
  const int le = threadIdx.x & 31;
  for (int job = threadIdx.x >> 5; job < narrays * npr; job += BLOCK / 32) {
    const int f = job / npr, o = job - f * npr;
    double* p = x + f * stride + le;
    double& u = p[o * PE];
    double& v = p[(odd + o) * PE];
    const double s = u + v, d = u - v;
    u = s;
    v = d;
  }
}

// Euler: p, 1/rho and |u| + c = sqrt(|m|^2) / |rho| + sqrt(gamma p / rho) of a state.
__device__ __forceinline__ void euler_node(const double* q, double gamma, double* s) {
  const double mm = fma(q[2], q[2], q[3] * q[3]);
  const double rinv = 1.0 / q[0];
  const double p = (gamma - 1.0) * fma(-0.5 * mm, rinv, q[1]);
  s[0] = p;
  s[1] = rinv;
  s[2] = fma(sqrt(mm), fabs(rinv), sqrt(gamma * (p * rinv)));
}

// Flux of one edge point with interior and exterior trace (and Euler's per-node
// values si, se): own side's and the glued side's lifted-flux inputs, before each
// side's sJ/J.
template <int EQ>
__device__ __forceinline__ void edge_flux(const RhsArgs& a, const double* qi, const double* qe,
                                          const double* si, const double* se, double nx,
                                          double ny, double* own, double* glued) {
  if constexpr (EQ == DG_WAVE) {
    // c/2 ((v- + v+).n + u+ - u-), c/2 (u- + u+ + (v+ - v-).n) n
    const double hc = 0.5 * a.p0;
    const double du = qe[0] - qi[0];
    const double dv = fma(qe[1] - qi[1], nx, (qe[2] - qi[2]) * ny);
    const double vn = fma(qi[1], nx, qi[2] * ny);
    const double gv = hc * (fma(2.0, qi[0], du) + dv);
    own[0] = hc * (du + fma(2.0, vn, dv));
    own[1] = gv * nx;
    own[2] = gv * ny;
#pragma unroll
    for (int k = 0; k < 3; ++k) glued[k] = -own[k];
  } else if constexpr (EQ == DG_EULER) {
    const double mi = fma(qi[2], nx, qi[3] * ny), me = fma(qe[2], nx, qe[3] * ny);
    const double ui = mi * si[1], ue = me * se[1], ps = si[0] + se[0];
    const double lnn = fmax(si[2], se[2]) * fma(nx, nx, ny * ny);
    const double sum[4] = {mi + me, fma(ue, qe[1] + se[0], ui * (qi[1] + si[0])),
                           fma(qe[2], ue, fma(qi[2], ui, ps * nx)),
                           fma(qe[3], ue, fma(qi[3], ui, ps * ny))};
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      glued[k] = 0.5 * fma(-lnn, qe[k] - qi[k], sum[k]);
      own[k] = -glued[k];
    }
  } else {  // DG_MAXWELL, TM: central part kept, penalty part negated by the swap
    const double alpha = a.p0, z = a.k[0], y = a.k[1], ce = -a.k[2], ch = -a.k[3];
    const double jez = qe[0] - qi[0], jhx = qe[1] - qi[1], jhy = qe[2] - qi[2];
    const double nh = fma(nx, jhy, -ny * jhx);        // (n x j_H)_z
    const double ca = ce * z * nh, cb = ce * alpha * fma(nx, nx, ny * ny) * jez;
    const double ha = ch * y * jez, hb = ch * alpha * nh;
    own[0] = ca + cb;
    glued[0] = ca - cb;
    own[1] = ny * (ha + hb);
    own[2] = -nx * (ha + hb);
    glued[1] = ny * (ha - hb);
    glued[2] = -nx * (ha - hb);
  }
}

template <int N, int EQ, int MODE>
__global__ void __launch_bounds__(Tile<N, EQ>::BLOCK) dg_rhs2d_sym_kernel(const RhsArgs a) {
  using T = Tile<N, EQ>;
  using O = Ops<N>;
  using B = Basis<N>;
  constexpr bool STAGE = (MODE & MODE_STAGE) != 0;
  constexpr int NP = B::NP, NFP = B::NFP, NFPT = B::NFPT, NF = T::NF;
  constexpr int E = T::E, PE = T::PE, BLOCK = T::BLOCK, XS = NP * PE, FS = NFPT * PE;
  extern __shared__ __align__(128) unsigned char smem[];
  __shared__ uint64_t bar;
  __shared__ int ops_ok;
  const double* ops = reinterpret_cast<const double*>(smem);
  const int* node_slot = reinterpret_cast<const int*>(smem + O::NODE_SLOT);
  [[maybe_unused]] const int* slot_node = reinterpret_cast<const int*>(smem + O::SLOT_NODE);
  const int* edge_slot = reinterpret_cast<const int*>(smem + O::EDGE_SLOT);
  const int* edge_node = reinterpret_cast<const int*>(smem + O::EDGE_NODE);
  double* sQ = reinterpret_cast<double*>(smem + T::Q);
  double* sX = reinterpret_cast<double*>(smem + T::X);
  double* sF = reinterpret_cast<double*>(smem + T::F);
  double* sH = reinterpret_cast<double*>(smem + T::H);
  double* sFG = reinterpret_cast<double*>(smem + T::FG);
  uint32_t* sGat = reinterpret_cast<uint32_t*>(smem + T::GAT);
  int* sMate = reinterpret_cast<int*>(smem + T::MATE);
  int* sList = reinterpret_cast<int*>(smem + T::LIST);  // [0]: length
  const int t = threadIdx.x, le = t & 31;
  if (t == 0) {
    mbar_init(&bar, 1);
    mbar_arrive_expect_tx(&bar, a.ops_bytes);
    bulk_g2s(smem, a.ops, a.ops_bytes, &bar);
    const bool ok = mbar_wait_bounded(&bar, 0);
    if (!ok) {
      raise_status(a.status, DG_ERR_TIMEOUT);
      mbar_wait_bounded(&bar, 0);  // give the copy one more bounded chance
    }
    ops_ok = ok ? 1 : 0;
  }
  __syncthreads();
  if (!ops_ok) return;

  const int64_t nel = a.nel, nelnp = nel * NP;
  const int64_t ntiles = (nel + E - 1) / E;
  for (int64_t tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
    const int64_t e0 = tile * E;
    const int ecount = (nel - e0) < (int64_t)E ? (int)(nel - e0) : E;
    const uint32_t node0 = (uint32_t)(e0 * NP);

    // {{{ state, metric, edge geometry, gather index; Euler: per-node values
    for (int rem = t; rem < E * NP; rem += BLOCK) {
      const int el = rem / NP;
      double* x = sQ + (rem - el * NP) * PE + el;
      double q[NF];
#pragma unroll
      for (int k = 0; k < NF; ++k) {
        q[k] = rem < ecount * NP ? __ldg(a.q + k * nelnp + e0 * NP + rem) : 0.0;
        x[k * XS] = q[k];
      }
      if constexpr (EQ == DG_EULER) {
        double s[3];
        euler_node(q, a.p0, s);
#pragma unroll
        for (int k = 0; k < 3; ++k) x[(NF + k) * XS] = s[k];
      } else {
        double* y = sX + node_slot[rem - el * NP] * PE + el;
#pragma unroll
        for (int k = 0; k < NF; ++k) y[k * XS] = q[k];
      }
    }
    for (int idx = t; idx < 4 * E; idx += BLOCK) {  // (g_1 + g_2, g_1 - g_2)
      const int el = idx >> 2, kx = idx & 3, x = kx & 1;
      double v = 0.0;
      if (el < ecount) {
        const double* mt = a.metric + (e0 + el) * 4;
        const double g1 = __ldg(mt + x), g2 = __ldg(mt + 2 + x);
        v = kx < 2 ? g1 + g2 : g1 - g2;
      }
      sH[kx * PE + el] = v;
    }
    for (int idx = t; idx < 12 * E; idx += BLOCK) {
      const int el = idx / 12, c = idx - el * 12;
      if ((c & 3) != 3)
        sFG[((c >> 2) * 3 + (c & 3)) * PE + el] =
            el < ecount ? __ldg(a.face_geom + (e0 + el) * 12 + c) : 0.0;
    }
    for (int idx = t; idx < E * NFPT; idx += BLOCK) {
      const int el = idx / NFPT, fj = idx - el * NFPT;
      uint32_t g = 0x80000000u;
      if (el < ecount) {
        g = __ldg(a.gather + e0 * NFPT + idx);
        if ((g & 0x7fffffffu) >= (uint32_t)nelnp) {  // never read out of bounds
          raise_status(a.status, DG_ERR_INDEX);
          g = (g & 0x80000000u) | (node0 + (uint32_t)(el * NP + edge_node[fj]));
        }
      }
      sGat[fj * PE + el] = g;
    }
    __syncthreads();
    // }}}

    // {{{ glued sides inside the tile: mate of side e + 32 f, or -1
    for (int s = t; s < T::NSIDE; s += BLOCK) {
      const int e = s & 31, f = s >> 5;
      int mate = -1;
      const uint32_t g0 = sGat[f * NFP * PE + e];
      const uint32_t off = (g0 & 0x7fffffffu) - node0;
      if (e < ecount && (g0 >> 31) == 0u && off < (uint32_t)(ecount * NP)) {
        const int e2 = (int)off / NP;
        for (int f2 = 0; f2 < 3 && mate < 0 && e2 != e; ++f2) {
          bool all = true;
          for (int j = 0; j < NFP && all; ++j) {
            const uint32_t g = sGat[(f * NFP + j) * PE + e];
            const uint32_t mine = node0 + (uint32_t)(e * NP + edge_node[f * NFP + j]);
            bool hit = false;
            for (int j2 = 0; j2 < NFP; ++j2)
              hit = hit || (g == node0 + (uint32_t)(e2 * NP + edge_node[f2 * NFP + j2]) &&
                            sGat[(f2 * NFP + j2) * PE + e2] == mine);
            all = hit;
          }
          const double dx = sFG[f * 3 * PE + e] + sFG[f2 * 3 * PE + e2];
          const double dy = sFG[(f * 3 + 1) * PE + e] + sFG[(f2 * 3 + 1) * PE + e2];
          if (all && fabs(dx) + fabs(dy) <= 1e-12) mate = e2 + 32 * f2;
        }
      }
      sMate[s] = mate;
    }
    if constexpr (EQ != DG_EULER) mirror<PE, BLOCK>(sX, NF, XS, B::NPR, B::DE);
    __syncthreads();
    // work list: sides that read outside the tile, then the others; of a glued
    // pair (mates of each other) the lower-numbered side
    if (t < 32) {
      int kind[3], mate[3], na = 0, nb = 0;
#pragma unroll
      for (int f = 0; f < 3; ++f) {
        const int s = le + 32 * f;
        mate[f] = sMate[s];
        if (mate[f] >= 0 && sMate[mate[f]] != s) mate[f] = -1;
        bool outside = false;
        for (int j = 0; j < NFP; ++j) {
          const uint32_t g = sGat[(f * NFP + j) * PE + le];
          outside = outside || ((g >> 31) == 0u && g - node0 >= (uint32_t)(ecount * NP));
        }
        kind[f] = le >= ecount || (mate[f] >= 0 && mate[f] < s) ? 0 : (outside ? 1 : 2);
        na += __popc(__ballot_sync(0xffffffffu, kind[f] == 1));
        nb += __popc(__ballot_sync(0xffffffffu, kind[f] == 2));
      }
      int pa = 1, pb = 1 + na;
      const uint32_t below = (1u << le) - 1u;
#pragma unroll
      for (int f = 0; f < 3; ++f) {
        const uint32_t ba = __ballot_sync(0xffffffffu, kind[f] == 1);
        const uint32_t bb = __ballot_sync(0xffffffffu, kind[f] == 2);
        const int entry = (le + 32 * f) | ((mate[f] + 1) << 8);
        if (kind[f] == 1) sList[pa + __popc(ba & below)] = entry;
        if (kind[f] == 2) sList[pb + __popc(bb & below)] = entry;
        pa += __popc(ba);
        pb += __popc(bb);
      }
      if (le == 0) sList[0] = na + nb;
    }
    __syncthreads();
    // }}}

    // {{{ edge fluxes
    const int npts = sList[0] * NFP;
    for (int idx = t; idx < npts; idx += BLOCK) {
      const int li = idx / NFP, j = idx - li * NFP;
      const int entry = sList[1 + li], s = entry & 0xff, mate = (entry >> 8) - 1;
      const int e = s & 31, f = s >> 5, fj = f * NFP + j;
      const double* qn = sQ + edge_node[fj] * PE + e;
      const uint32_t g = sGat[fj * PE + e];
      const bool bdry = (g >> 31) != 0u;
      const uint32_t gi = g & 0x7fffffffu, off = gi - node0;
      const double* fg = sFG + f * 3 * PE + e;
      const double nx = fg[0], ny = fg[PE], scale = fg[2 * PE];
      double qi[NF], qe[NF];
      [[maybe_unused]] double si[3], se[3];
#pragma unroll
      for (int k = 0; k < NF; ++k) qi[k] = qn[k * XS];
      if constexpr (EQ == DG_EULER) {
#pragma unroll
        for (int k = 0; k < 3; ++k) si[k] = se[k] = qn[(NF + k) * XS];
      }
      int m = 0;  // exterior node inside the tile
      if (bdry) {
        if constexpr (EQ == DG_WAVE) {  // Dirichlet mirror: (-u, v)
          qe[0] = -qi[0];
          qe[1] = qi[1];
          qe[2] = qi[2];
        } else if constexpr (EQ == DG_EULER) {  // wall: mirrored normal momentum
          const double mn = fma(qi[2], nx, qi[3] * ny);
          qe[0] = qi[0];
          qe[1] = qi[1];
          qe[2] = fma(-2.0 * nx, mn, qi[2]);
          qe[3] = fma(-2.0 * ny, mn, qi[3]);
        } else {  // PEC: (-E, H)
          qe[0] = -qi[0];
          qe[1] = qi[1];
          qe[2] = qi[2];
        }
      } else if (off < (uint32_t)(ecount * NP)) {
        const int e2 = (int)off / NP;
        m = (int)off - e2 * NP;
        const double* qx = sQ + m * PE + e2;
#pragma unroll
        for (int k = 0; k < NF; ++k) qe[k] = qx[k * XS];
        if constexpr (EQ == DG_EULER) {
#pragma unroll
          for (int k = 0; k < 3; ++k) se[k] = qx[(NF + k) * XS];
        }
      } else {
#pragma unroll
        for (int k = 0; k < NF; ++k) qe[k] = __ldg(a.q + k * nelnp + gi);
        if constexpr (EQ == DG_EULER) euler_node(qe, a.p0, se);
      }
      double own[NF], glued[NF];
      edge_flux<EQ>(a, qi, qe, si, se, nx, ny, own, glued);
      double* out = sF + edge_slot[fj] * PE + e;
#pragma unroll
      for (int k = 0; k < NF; ++k) out[k * FS] = scale * own[k];
      if (mate >= 0) {
        const int e2 = mate & 31, f2 = mate >> 5;
        int j2 = 0;
        while (j2 < NFP - 1 && edge_node[f2 * NFP + j2] != m) ++j2;
        const double scale2 = sFG[(f2 * 3 + 2) * PE + e2];
        double* out2 = sF + edge_slot[f2 * NFP + j2] * PE + e2;
#pragma unroll
        for (int k = 0; k < NF; ++k) out2[k * FS] = scale2 * glued[k];
      }
    }
    __syncthreads();
    mirror<PE, BLOCK>(sF, NF, FS, B::FPR, B::FE);
    // }}}

    // {{{ volume and LIFT blocks, one part per warp (rotating with the tile: the
    // even part is larger)
    const int rho = ((t >> 5) + (int)tile) & 1;
    // Euler: the four fluxes along direction k (metric row h), transformed
    auto euler_inputs = [&](int k) {
      const double h0 = sH[k * 2 * PE + le], h1 = sH[(k * 2 + 1) * PE + le];
      for (int o = t >> 5; o < B::DE; o += BLOCK / 32) {
        double w[2][4];
        const int cnt = o < B::NPR ? 2 : 1;
#pragma unroll
        for (int n = 0; n < 2; ++n) {
          if (n >= cnt) break;
          const double* x = sQ + slot_node[n == 0 ? o : B::DE + o] * PE + le;
          const double m0 = x[2 * XS], m1 = x[3 * XS], p = x[NF * XS];
          const double hm = fma(h0, m0, h1 * m1), u = hm * x[(NF + 1) * XS];
          w[n][0] = hm;
          w[n][1] = (x[XS] + p) * u;
          w[n][2] = fma(m0, u, p * h0);
          w[n][3] = fma(m1, u, p * h1);
        }
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          double* y = sX + c * XS + le;
          if (cnt == 2) {
            y[o * PE] = w[0][c] + w[1][c];
            y[(B::DE + o) * PE] = w[0][c] - w[1][c];
          } else {
            y[o * PE] = w[0][c];
          }
        }
      }
    };
    // the fields of this warp: Euler 0, 1 / 2, 3; wave and Maxwell 0 / 1, 2 (which
    // share the derivatives of field 0)
    const int half = t >> 6;
    auto part = [&](auto dtag, auto ptag, auto htag, int slot0, const double* vops,
                    const double* lops, int fslot0, int frows) {
      constexpr int D = decltype(dtag)::value, P = decltype(ptag)::value;
      constexpr int HALF = decltype(htag)::value;
      constexpr int F0 = EQ == DG_EULER ? 2 * HALF : HALF;
      constexpr int NA = EQ == DG_EULER ? 2 : 1 + HALF;
      double acc[NA][D];
#pragma unroll
      for (int m = 0; m < NA; ++m)
#pragma unroll
        for (int i = 0; i < D; ++i) acc[m][i] = 0.0;
#pragma unroll 1
      for (int k = 0; k < 2; ++k) {
        const int sig = rho ^ k, din = sig == 0 ? B::DE : B::DO;
        const double* xs = sX + (sig == 0 ? 0 : B::DE * PE) + le;
        if constexpr (EQ == DG_EULER) {
          euler_inputs(k);
          sym::cta_sync<BLOCK>();
          block_product<NA, D, P, PE, XS>(xs + F0 * XS, vops, din, acc);
          sym::cta_sync<BLOCK>();  // the inputs' slots are free
        } else {
          // wave: u from h.v, v from u (factor -c); maxwell: E_z from
          // h_x H_y - h_y H_x, (H_x, H_y) from (-h_y, h_x) E_z
          const double c = EQ == DG_WAVE ? -a.p0 : 1.0;
          const double h0 = c * sH[k * 2 * PE + le], h1 = c * sH[(k * 2 + 1) * PE + le];
          double g[D];  // this part's derivative (half 0: accumulated in place)
#pragma unroll
          for (int i = 0; i < D; ++i) g[i] = HALF == 0 ? acc[0][i] : 0.0;
          const double* row = vops;
#pragma unroll 1
          for (int j = 0; j < din; ++j, row += P, xs += PE) {
            double w;
            if constexpr (HALF == 1) w = xs[0];
            else if constexpr (EQ == DG_WAVE) w = fma(h0, xs[XS], h1 * xs[2 * XS]);
            else w = fma(h0, xs[2 * XS], -h1 * xs[XS]);
            double tr[P];
#pragma unroll
            for (int i = 0; i < P; i += 2) {
              const double2 w2 = *reinterpret_cast<const double2*>(row + i);
              tr[i] = w2.x;
              tr[i + 1] = w2.y;
            }
#pragma unroll
            for (int i = 0; i < D; ++i) g[i] = fma(tr[i], w, g[i]);
          }
          const double g0 = EQ == DG_WAVE ? h0 : -h1, g1 = EQ == DG_WAVE ? h1 : h0;
#pragma unroll
          for (int i = 0; i < D; ++i) {
            if constexpr (HALF == 0) {
              acc[0][i] = g[i];
            } else {
              acc[0][i] = fma(g0, g[i], acc[0][i]);
              acc[1][i] = fma(g1, g[i], acc[1][i]);
            }
          }
        }
        vops += din * P;
      }
      sym::cta_sync<BLOCK>();      // edge values transformed, inputs read
      block_product<NA, D, P, PE, FS>(sF + F0 * FS + fslot0 * PE + le, lops, frows, acc);
#pragma unroll
      for (int m = 0; m < NA; ++m)
#pragma unroll
        for (int i = 0; i < D; ++i)
          sX[(F0 + m) * XS + (slot0 + i) * PE + le] =
              EQ == DG_MAXWELL ? acc[m][i] * (F0 + m == 0 ? a.k[4] : a.k[5]) : acc[m][i];
    };
    using std::integral_constant;
    auto both = [&](auto htag) {
      if (rho == 0)
        part(integral_constant<int, B::DE>{}, integral_constant<int, O::PE>{}, htag, 0, ops,
             ops + O::LIFT0, 0, B::FE);
      else
        part(integral_constant<int, B::DO>{}, integral_constant<int, O::PO>{}, htag, B::DE,
             ops + O::VOL1, ops + O::LIFT1, B::FE, B::FO);
    };
    if (half == 0) both(integral_constant<int, 0>{});
    else both(integral_constant<int, 1>{});
    __syncthreads();
    // }}}

    // {{{ back to nodes, then store or fold into the RK stage
    mirror<PE, BLOCK>(sX, NF, XS, B::NPR, B::DE);
    __syncthreads();
    for (int rem = t; rem < ecount * NP; rem += BLOCK) {
      const int el = rem / NP, node = rem - el * NP;
      const double* y = sX + node_slot[node] * PE + el;
      const int64_t gidx = e0 * NP + rem;
      [[maybe_unused]] double res[NF];
      if constexpr (STAGE) {
#pragma unroll
        for (int k = 0; k < NF; ++k) res[k] = a.rk_a != 0.0 ? a.res[gidx + k * nelnp] : 0.0;
      }
#pragma unroll
      for (int k = 0; k < NF; ++k) {
        double val = y[k * XS];
        if constexpr (STAGE)
          if (a.rhs_unscaled) a.rhs_unscaled[gidx + k * nelnp] = val;
        if (a.elem_scale) val *= __ldg(a.elem_scale + e0 + el);
        if constexpr (!STAGE) {
          a.rhs[gidx + k * nelnp] = val;
        } else {
          const double r = (a.rk_a != 0.0 ? a.rk_a * res[k] : 0.0) + a.rk_dt * val;
          a.res[gidx + k * nelnp] = r;
          a.q_out[gidx + k * nelnp] = sQ[k * XS + node * PE + el] + a.rk_b * r;
        }
      }
    }
    __syncthreads();
    // }}}
  }
}

}  // namespace sym2
}  // namespace dg
