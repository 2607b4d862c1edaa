// Face-shared numerical fluxes for the FP64 RHS on sm_103a.
//
// The fused RHS kernel (dg_rhs.cuh) evaluates the numerical flux at every
// element face point: twice per glued pair of face points, once from each
// side, and for Euler it recovers pressure and wave speed of both traces at
// every one of them.  GB300's FP64 pipe issues a small fraction of its FP32
// rate, so on the low orders that repeated FP64 work is a large share of the
// RHS.  The face-shared path splits one RHS into
//
//   (a) Euler only, dg_euler_aux_kernel: pressure, 1/rho and the local wave
//       speed |u| + c of every volume node, once per node;
//   (b) dg_face_flux_kernel: one thread per face point of an OWNED face (a
//       boundary face, or the lower-numbered face of a glued pair) evaluates
//       the flux once and writes the lifted-flux input of BOTH glued face
//       points; the neighbour's value follows from how each flux transforms
//       when the two sides swap (n -> -n, jumps change sign);
//   (c) the volume term and the LIFT of the stored face values:
//       dg_rhs_sym_kernel (dg_sym.cuh) for operators with the tetrahedron's
//       symmetry, dg_rhs_kernel with MODE_SPLIT for any others.
//
// What bounds it: the FP64 pipe (79-85 % busy), so each flux is written for the
// fewest FP64 operations that keep jumps as differences of traces: wave 26 per
// pair of points, Euler 50, Maxwell 62.  Measured (GB300, ncu, against 30 / 55 /
// 68 before): wave P1 at 5.14 M tets 1.91 -> 1.75 ms, Euler P2 at 413,526 tets 617
// -> 569 us, Maxwell P4 at 584,016 tets 2.09 ms either way.
//
// Face values live in HBM as (nfields, Nel, 4 Nfp) doubles, face point
// (e, f, j) at e * 4 Nfp + f Nfp + j -- the fused kernel's shared-memory
// flux layout -- already multiplied by sJ/J and signed as that kernel's.
// The flux formulas are the fused kernel's (which follow
// actx_dgfem_suite/equations/wave.py:80-114 and grudge's Euler LF and
// Maxwell alpha fluxes as configured at equations/euler.py:168-174 and
// equations/maxwell.py:55-59).
#pragma once

#include "dg_rhs.cuh"

namespace dg {

constexpr int kFaceBlock = 256;

struct FaceArgs {
  const double* q;            // (NF, Nel, Np) state
  const double* aux;          // euler: (3, Nel, Np) p, 1/rho, |u| + c
  const double* face_geom;    // (Nel, 4, 4) n_x, n_y, n_z, sJ/J
  const uint32_t* gather;     // (Nel, 4, Nfp) exterior node, bit 31 = boundary
  const int32_t* partner;     // (Nel, 4, Nfp) glued face point, -1 on boundary
  const int32_t* owned;       // owned faces e * 4 + f, ascending
  const int32_t* face_nodes;  // (4, Nfp) volume node of each face node
  double* flux;               // (NF, Nel, 4 Nfp) lifted-flux input
  int64_t nel;
  int64_t nowned;
  int* status;
  double p0, p1, p2;          // equation parameters
  // flux constants, folded on the host (every FP64 multiply counts here): wave c/2;
  // maxwell, with z the impedance, ce = -1/(2z), ch = z/2: -ce z, ce alpha, -ch / z,
  // -ch alpha
  double c[4];
};

// Pressure, 1/rho and |u| + c of every node (the per-trace quantities of the
// Lax-Friedrichs flux), evaluated once per node instead of once per face
// point and side.
template <int EQ>
__global__ void __launch_bounds__(kFaceBlock)
    dg_euler_aux_kernel(const double* __restrict__ q, double* __restrict__ aux,
                        uint32_t nelnp, double gamma) {
  const uint32_t stride = gridDim.x * blockDim.x;
  for (uint32_t idx = blockIdx.x * blockDim.x + threadIdx.x; idx < nelnp;
       idx += stride) {
    const double* qn = q + idx;
    const double rho = __ldg(qn);
    const double en = __ldg(qn + nelnp);
    const double m0 = __ldg(qn + 2 * (size_t)nelnp);
    const double m1 = __ldg(qn + 3 * (size_t)nelnp);
    const double m2 = __ldg(qn + 4 * (size_t)nelnp);
    const double rinv = 1.0 / rho;
    const double mm = fma(m0, m0, fma(m1, m1, m2 * m2));
    const double p = (gamma - 1.0) * fma(-0.5 * mm, rinv, en);
    // |u| + c = sqrt(|m|^2) / rho + sqrt(gamma p / rho)
    const double lam = fma(sqrt(mm), rinv, sqrt(gamma * (p * rinv)));
    double* an = aux + idx;
    an[0] = p;
    an[nelnp] = rinv;
    an[2 * (size_t)nelnp] = lam;
  }
}

template <int N, int EQ>
__global__ void __launch_bounds__(kFaceBlock) dg_face_flux_kernel(const FaceArgs a) {
  constexpr int NP = Shape<N>::NP, NFP = Shape<N>::NFP, NFPT = Shape<N>::NFPT;
  constexpr int NF = EqInfo<EQ>::NF;
  __shared__ int sFN[NFPT];
  for (int t = threadIdx.x; t < NFPT; t += blockDim.x) sFN[t] = __ldg(a.face_nodes + t);
  __syncthreads();

  // 32-bit indices throughout (Nel * 4 Nfp < 2^31 is checked at plan creation)
  const uint32_t nelnp = (uint32_t)(a.nel * NP);
  const uint32_t nfp_all = (uint32_t)(a.nel * NFPT);
  const uint32_t total = (uint32_t)(a.nowned * NFP);
  const uint32_t stride = gridDim.x * blockDim.x;
  for (uint32_t idx = blockIdx.x * blockDim.x + threadIdx.x; idx < total;
       idx += stride) {
    const uint32_t of = idx / NFP;
    const uint32_t j = idx - of * NFP;
    const uint32_t face = (uint32_t)__ldg(a.owned + of);
    const uint32_t e = face >> 2, f = face & 3u;
    const uint32_t fp = face * NFP + j;
    const uint32_t ii = e * NP + (uint32_t)sFN[f * NFP + j];
    const uint32_t g = __ldg(a.gather + fp);
    const bool bdry = (g >> 31) != 0u;
    uint32_t gi = g & 0x7fffffffu;
    if (gi >= nelnp) {  // never read out of bounds
      raise_status(a.status, DG_ERR_INDEX);
      gi = ii;
    }
    int32_t pp = -1;
    if (!bdry) {
      pp = __ldg(a.partner + fp);
      if (pp < 0 || (uint32_t)pp >= nfp_all) {  // never write out of bounds
        raise_status(a.status, DG_ERR_INDEX);
        pp = -1;
      }
    }
    // n_x, n_y, n_z, sJ/J of the face: two 16-byte loads (rows of 32 bytes)
    const double2* fg = reinterpret_cast<const double2*>(a.face_geom) + face * 2u;
    const double2 g01 = __ldg(fg), g23 = __ldg(fg + 1);
    const double nx = g01.x, ny = g01.y, nz = g23.x;
    const double scale_o = g23.y;
    const double scale_p =
        pp >= 0 ? __ldg(a.face_geom + ((uint32_t)pp / NFP) * 4u + 3) : 0.0;

    double qi[NF], qe[NF];
    {
      const double* qk = a.q + ii;
      const double* qx = a.q + gi;
#pragma unroll
      for (int k = 0; k < NF; ++k, qk += nelnp, qx += nelnp) {
        qi[k] = __ldg(qk);
        qe[k] = bdry ? 0.0 : __ldg(qx);
      }
    }
    // own[k]: value for this face point; part[k]: for the glued face point, each
    // with its side's sJ/J
    double own[NF], part[NF];

    if constexpr (EQ == DG_WAVE) {
      if (bdry) {  // Dirichlet mirror: exterior (-u, v)
        qe[0] = -qi[0];
        qe[1] = qi[1];
        qe[2] = qi[2];
        qe[3] = qi[3];
      }
      // F_u = c (avg(v).n + (u+ - u-)/2) = c/2 ((v- + v+).n + u+ - u-),
      // F_v = c (avg(u) + (v+ - v-).n/2) n = c/2 (u- + u+ + (v+ - v-).n) n, the
      // sums as 2 x interior + jump; c/2 goes into the side scales
      const double du = qe[0] - qi[0];
      const double dv = fma(qe[1] - qi[1], nx, fma(qe[2] - qi[2], ny, (qe[3] - qi[3]) * nz));
      const double vn = fma(qi[1], nx, fma(qi[2], ny, qi[3] * nz));
      const double su = du + fma(2.0, vn, dv), gv = fma(2.0, qi[0], du) + dv;
      const double so = a.c[0] * scale_o, sp = -a.c[0] * scale_p;
      const double go = so * gv, gp = sp * gv;
      own[0] = so * su;
      own[1] = go * nx;
      own[2] = go * ny;
      own[3] = go * nz;
      part[0] = sp * su;
      part[1] = gp * nx;
      part[2] = gp * ny;
      part[3] = gp * nz;
    } else if constexpr (EQ == DG_EULER) {
      const double* an = a.aux;
      const double pi = __ldg(an + ii), ri = __ldg(an + nelnp + ii),
                   li = __ldg(an + 2 * (size_t)nelnp + ii);
      double pe, re, le;
      if (bdry) {  // InviscidWallBC: mirror the normal momentum; rho, E, |m| kept
        const double mn = qi[2] * nx + qi[3] * ny + qi[4] * nz;
        qe[0] = qi[0];
        qe[1] = qi[1];
        qe[2] = qi[2] - 2.0 * nx * mn;
        qe[3] = qi[3] - 2.0 * ny * mn;
        qe[4] = qi[4] - 2.0 * nz * mn;
        pe = pi;
        re = ri;
        le = li;
      } else {
        pe = __ldg(an + gi);
        re = __ldg(an + nelnp + gi);
        le = __ldg(an + 2 * (size_t)nelnp + gi);
      }
      // (F- + F+).n through m.n and u.n = (m.n) / rho of both sides
      const double mi = fma(qi[2], nx, fma(qi[3], ny, qi[4] * nz));
      const double me = fma(qe[2], nx, fma(qe[3], ny, qe[4] * nz));
      const double ui = mi * ri, ue = me * re, ps = pi + pe;
      const double lnn = fmax(li, le) * fma(nx, nx, fma(ny, ny, nz * nz));
      const double sum[5] = {mi + me, fma(ue, qe[1] + pe, ui * (qi[1] + pi)),
                             fma(qe[2], ue, fma(qi[2], ui, ps * nx)),
                             fma(qe[3], ue, fma(qi[3], ui, ps * ny)),
                             fma(qe[4], ue, fma(qi[4], ui, ps * nz))};
      // f_k = 1/2 (F- + F+).n - 1/2 lam (q+ - q-) n.n = 1/2 t_k; the glued side
      // sees -f_k
      const double so = -0.5 * scale_o, sp = 0.5 * scale_p;
#pragma unroll
      for (int k = 0; k < 5; ++k) {
        const double tk = fma(-lnn, qe[k] - qi[k], sum[k]);
        own[k] = so * tk;
        part[k] = sp * tk;
      }
    } else {  // DG_MAXWELL
      if (bdry) {  // PEC: exterior (-E, H)
        qe[0] = -qi[0];
        qe[1] = -qi[1];
        qe[2] = -qi[2];
        qe[3] = qi[3];
        qe[4] = qi[4];
        qe[5] = qi[5];
      }
      const double je[3] = {qe[0] - qi[0], qe[1] - qi[1], qe[2] - qi[2]};
      const double jh[3] = {qe[3] - qi[3], qe[4] - qi[4], qe[5] - qi[5]};
      const double n[3] = {nx, ny, nz};
      auto cross = [](const double* a_, const double* b_, double* c_) {
        c_[0] = a_[1] * b_[2] - a_[2] * b_[1];
        c_[1] = a_[2] * b_[0] - a_[0] * b_[2];
        c_[2] = a_[0] * b_[1] - a_[1] * b_[0];
      };
      // fe = n x (z jh - alpha n x je) = Ae + Be, fh = n x (y je + alpha n x jh)
      // = Ah + Bh; swapping the sides keeps Ae, Ah and negates Be, Bh.  With
      // the constants folded: -ce fe = c0 (n x jh) + c1 (n x n x je),
      // -ch fh = c2 (n x je) + c3 (n x n x jh).  (The side's scale folded into the
      // constants saves six more multiplies per point but measured 5 % slower: 60
      // registers, four CTAs per SM instead of five.)
      double nxe[3], nxh[3], nnxe[3], nnxh[3];
      cross(n, je, nxe);
      cross(n, jh, nxh);
      cross(n, nxe, nnxe);
      cross(n, nxh, nnxh);
#pragma unroll
      for (int x = 0; x < 3; ++x) {
        const double ae = a.c[0] * nxh[x], be = a.c[1] * nnxe[x];
        const double ah = a.c[2] * nxe[x], bh = a.c[3] * nnxh[x];
        own[x] = scale_o * (ae + be);
        own[3 + x] = scale_o * (ah + bh);
        part[x] = scale_p * (ae - be);
        part[3 + x] = scale_p * (ah - bh);
      }
    }

    double* out = a.flux + fp;
#pragma unroll
    for (int k = 0; k < NF; ++k, out += nfp_all) out[0] = own[k];
    if (pp >= 0) {
      double* outp = a.flux + (uint32_t)pp;
#pragma unroll
      for (int k = 0; k < NF; ++k, outp += nfp_all) outp[0] = part[k];
    }
  }
}

}  // namespace dg
