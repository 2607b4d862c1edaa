// Mixed-precision RHS of the wave and Euler equations on the CUDA cores
// (sm_103a): FP32 derivative, flux and LIFT arithmetic on an FP64 state,
// variants 0 (persistent) and 2 (one CTA per tile) of meshes that fill its tiles
// (dg_plan_create; dg_rhs_kernel serves smaller ones).
//
// One lane per element and R = 5 rows of the operators per warp (P2-P4; 2 at P1),
// so that operator entries are warp-uniform broadcasts shared by all fields of a
// thread and every data word is read once per R rows (7 shared-memory words per
// 25 multiply-adds at Euler P3, where one thread per (element, node) read two for
// every four in LIFT).  Data lies in shared memory as [array][node][element] with
// an odd element pitch.
//
// Euler: a launch before it (dg_nodes_f32_kernel, in place of the pressure
// table's) writes one 32-byte FP32 record per node: the state, the pressure
// recovered in FP64, 1/rho and |u| + c.  A gathered trace is then one memory
// sector instead of six, and every value is converted, and every reciprocal and
// square root taken, once per node instead of once per face point and side.  The
// wave plans hold no per-call buffers (their calls may run concurrently on several
// streams), so wave converts its traces in the kernel.
//
// The arithmetic is that of dg_rhs_kernel in FP32, operation for operation: the
// sums run over four columns at a time from the last to the first, derivatives
// along t before s before r, LIFT continues the volume sum, so results are bit
// for bit the same and the choice between the kernels is one of speed alone.
//
// What bounds it: instruction issue (55 % of the slots at Euler P3) and the
// gathers' latency; hence loads issued ahead for R nodes and two face points at a
// time, and 16 warps per SM.  Measured (GB300, whole RHS, one thread per
// (element, node) -> here): wave P1-P4 at n = 48 / 40 / 32 / 24 cells per axis
// 153 / 301 / 363 / 325 -> 150 / 201 / 192 / 191 us, Euler 279 / 616 / 584 / 545 ->
// 205 / 292 / 301 / 318 us; Euler P3 LSRK step (196,608 tets) 3.57 -> 2.13 ms.
// Maxwell stays on dg_rhs_kernel.
#pragma once

#include "dg_rhs.cuh"

namespace dg {
namespace mix {

// Rows of a warp, warps, and the operator block: W[r][j][warp][RP] and
// LIFT[fj][warp][RP] in FP32 (RP = R padded to 16 bytes; entry (i, j) at row
// i = warp R + k), then the int32 face node table.
template <int N>
struct Ops {
  static constexpr int NP = Shape<N>::NP, NFPT = Shape<N>::NFPT;
  static constexpr int R = N == 1 ? 2 : 5, RP = (R + 3) & ~3, NW = NP / R;
  static_assert(NW * R == NP, "whole rows per warp");
  static constexpr int ROW = NW * RP;                        // entries per column
  static constexpr int L = 3 * NP * ROW;                     // LIFT, in entries
  static constexpr int FN = (L + NFPT * ROW) * 4;            // bytes from here
  static constexpr int SIZE = FN + pad16(NFPT * 4);
};

// Shared memory of a CTA: operators, (wave) the state in FP32, one area for the
// volume inputs (wave: three directions of G v; Euler: three directions of five
// fluxes), the face values and the result in turn, metric, face geometry.
template <int N, int EQ>
struct Tile {
  static constexpr int NP = Shape<N>::NP, NFPT = Shape<N>::NFPT;
  static constexpr int NF = EqInfo<EQ>::NF, E = 32, PE = E + 1;
  static constexpr int BLOCK = 32 * Ops<N>::NW;
  static constexpr int NAUX = EQ == DG_EULER ? 15 : 3;
  static constexpr int X = Ops<N>::SIZE;
  static constexpr int A = X + (EQ == DG_WAVE ? pad16(NF * NP * PE * 4) : 0);
  static constexpr int AREA = NAUX * NP > NF * NFPT ? NAUX * NP : NF * NFPT;
  static constexpr int G = A + pad16(AREA * PE * 4);
  static constexpr int FG = G + pad16(9 * PE * 4);
  static constexpr int SMEM = FG + pad16(16 * PE * 4);
  // 16 warps per SM at least (128 registers per thread); at order 1, whose short
  // tiles need more of them in flight, 32 for wave (663,552 tets: 180 us with 16, 148
  // with 32) and 20 for Euler, whose stage spills at 32 (RK stage at 162,000 / 235,824 /
  // 663,552 tets with 32, 28, 24, 20: 94 / 127 / 290, 87 / 118 / 280, 82 / 123 / 289, 80
  // / 105 / 267 us, dg_rhs_kernel 90 / 122 / 324; RHS 66 / 91 / 211 with 32, 59 / 79 /
  // 205 with 20)
  static constexpr int WARPS = N == 1 ? (EQ == DG_EULER ? 20 : 32) : 16;
  static constexpr int MIN_CTAS = WARPS / Ops<N>::NW;
};

struct Trace {
  float p, rinv, lam;
};

// A node's record: (rho, E, m_x, m_y), (m_z, p, 1/rho, |u| + c).
__device__ __forceinline__ void load_node(const float4* __restrict__ rec, int64_t n, float* q,
                                          Trace& s) {
  const float4 a = __ldg(rec + 2 * n), b = __ldg(rec + 2 * n + 1);
  q[0] = a.x;
  q[1] = a.y;
  q[2] = a.z;
  q[3] = a.w;
  q[4] = b.x;
  s.p = b.y;
  s.rinv = b.z;
  s.lam = b.w;
}

// a x + b y + c z in the order in which dg_rhs_kernel's sums of products contract;
// written out because the compiler's own choice depends on the surrounding code.
__device__ __forceinline__ float dot3(float a, float b, float c, float x, float y, float z) {
  return fmaf(c, z, fmaf(a, x, __fmul_rn(b, y)));
}

// Euler trace: pressure (recovered in FP64 once per node), 1/rho and |u| + c.
__device__ __forceinline__ Trace euler_trace(const float* q, float p, float gamma) {
  Trace s;
  s.p = p;
  s.rinv = 1.0f / q[0];
  const float ux = q[2] * s.rinv, uy = q[3] * s.rinv, uz = q[4] * s.rinv;
  s.lam = __fadd_rn(sqrtf(dot3(ux, uy, uz, ux, uy, uz)), sqrtf(gamma * (p * s.rinv)));
  return s;
}

// Lifted-flux input of one face point as in dg_rhs_kernel, with both sides' Euler
// traces given: interior trace qi, exterior trace qe (set here to the mirror state
// where `bdry`), unit normal, sJ/J; field k goes to out[k stride].
template <int EQ>
__device__ __forceinline__ void face_flux(const RhsArgs& a, const float* qi, float* qe,
                                          const Trace& si, Trace se, bool bdry, float nx,
                                          float ny, float nz, float scale, float* out,
                                          int stride) {
  if constexpr (EQ == DG_WAVE) {
    if (bdry) {  // Dirichlet mirror: exterior (-u, v)
      qe[0] = -qi[0];
      qe[1] = qi[1];
      qe[2] = qi[2];
      qe[3] = qi[3];
    }
    const float c = a.c32[0];
    const float vavg_n = dot3(0.5f * (qi[1] + qe[1]), 0.5f * (qi[2] + qe[2]),
                              0.5f * (qi[3] + qe[3]), nx, ny, nz);
    const float uavg = 0.5f * (qi[0] + qe[0]);
    const float vjump = dot3(qe[1] - qi[1], qe[2] - qi[2], qe[3] - qi[3], nx, ny, nz);
    const float fu = c * fmaf(0.5f, qe[0] - qi[0], vavg_n);
    const float fv = c * fmaf(0.5f, vjump, uavg);
    out[0] = scale * fu;
    out[stride] = scale * (fv * nx);
    out[2 * stride] = scale * (fv * ny);
    out[3 * stride] = scale * (fv * nz);
  } else {
    if (bdry) {  // InviscidWallBC: mirror the normal momentum; |u| from the mirror
      const float mn = dot3(qi[2], qi[3], qi[4], nx, ny, nz);
      qe[0] = qi[0];
      qe[1] = qi[1];
      qe[2] = fmaf(-2.0f * nx, mn, qi[2]);
      qe[3] = fmaf(-2.0f * ny, mn, qi[3]);
      qe[4] = fmaf(-2.0f * nz, mn, qi[4]);
      se = euler_trace(qe, si.p, a.c32[0]);
    }
    const float uni = dot3(qi[2] * si.rinv, qi[3] * si.rinv, qi[4] * si.rinv, nx, ny, nz);
    const float une = dot3(qe[2] * se.rinv, qe[3] * se.rinv, qe[4] * se.rinv, nx, ny, nz);
    const float hlam = 0.5f * fmaxf(si.lam, se.lam);
    const float nn = dot3(nx, ny, nz, nx, ny, nz);
    float sum[5];  // F_i.n + F_e.n
    sum[0] = __fadd_rn(dot3(qi[2], qi[3], qi[4], nx, ny, nz),
                       dot3(qe[2], qe[3], qe[4], nx, ny, nz));
    sum[1] = fmaf(uni, __fadd_rn(qi[1], si.p), __fmul_rn(une, __fadd_rn(qe[1], se.p)));
    const float n[3] = {nx, ny, nz};
#pragma unroll
    for (int c = 0; c < 3; ++c)
      sum[2 + c] = __fadd_rn(fmaf(si.p, n[c], __fmul_rn(qi[2 + c], uni)),
                             fmaf(se.p, n[c], __fmul_rn(qe[2 + c], une)));
#pragma unroll
    for (int k = 0; k < 5; ++k) {
      const float jump = __fmul_rn(__fmul_rn(hlam, __fsub_rn(qe[k], qi[k])), nn);
      out[k * stride] = __fmul_rn(-scale, fmaf(0.5f, sum[k], -jump));
    }
  }
}

template <int R>
__device__ __forceinline__ void load_rows(const float* p, float (&w)[R]) {
  if constexpr (R == 2) {
    const float2 v = *reinterpret_cast<const float2*>(p);
    w[0] = v.x;
    w[1] = v.y;
  } else {
    static_assert(R == 5, "rows of a warp");
    const float4 v = *reinterpret_cast<const float4*>(p);
    w[0] = v.x;
    w[1] = v.y;
    w[2] = v.z;
    w[3] = v.w;
    w[4] = p[4];
  }
}

template <int N, int EQ, bool STAGE>
__global__ void __launch_bounds__(Tile<N, EQ>::BLOCK, Tile<N, EQ>::MIN_CTAS)
    dg_rhs_mixed_kernel(const RhsArgs a) {
  using T = Tile<N, EQ>;
  using O = Ops<N>;
  constexpr int NP = T::NP, NFP = Shape<N>::NFP, NFPT = T::NFPT, NF = T::NF;
  constexpr int E = T::E, PE = T::PE, BLOCK = T::BLOCK, R = O::R, ROW = O::ROW;
  constexpr int XS = NP * PE, FS = NFPT * PE;  // array strides
  extern __shared__ __align__(128) unsigned char smem[];
  __shared__ uint64_t bar;
  __shared__ int ops_ok;
  const int t = threadIdx.x, le = t & 31, wid = t >> 5;
  const float* sW = reinterpret_cast<const float*>(smem) + wid * O::RP;
  const float* sL = sW + O::L;
  const int* sFN = reinterpret_cast<const int*>(smem + O::FN);
  [[maybe_unused]] float* sX = reinterpret_cast<float*>(smem + T::X);  // wave: state
  float* sA = reinterpret_cast<float*>(smem + T::A);
  float* sG = reinterpret_cast<float*>(smem + T::G);
  float* sFG = reinterpret_cast<float*>(smem + T::FG);
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
  const float p0 = a.c32[0];
  for (int64_t tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
    const int64_t e0 = tile * E;
    const int ecount = (nel - e0) < (int64_t)E ? (int)(nel - e0) : E;

    // {{{ state (R nodes per thread, all loads in flight at once) and geometry,
    // then the volume inputs of every node
    double v[EQ == DG_WAVE ? R : 1][NF];
    float q[R][NF];
    [[maybe_unused]] Trace tr[R];
#pragma unroll
    for (int n = 0; n < R; ++n) {  // E NP = R BLOCK
      const int rem = t + n * BLOCK;
      const bool in = rem < ecount * NP;
      if constexpr (EQ == DG_WAVE) {
#pragma unroll
        for (int k = 0; k < NF; ++k) v[n][k] = in ? __ldg(a.q + k * nelnp + e0 * NP + rem) : 0.0;
      } else {
        load_node(a.nodes, e0 * NP + (in ? rem : 0), q[n], tr[n]);
      }
    }
    {
      const double* mt = a.metric + e0 * 9;
      for (int idx = t; idx < 9 * E; idx += BLOCK) {
        const int el = idx / 9;
        sG[(idx - el * 9) * PE + el] = d2f_alu(el < ecount ? __ldg(mt + idx) : 0.0);
      }
      const double* ft = a.face_geom + e0 * 16;
      for (int idx = t; idx < 16 * E; idx += BLOCK) {
        const int el = idx / 16;
        sFG[(idx - el * 16) * PE + el] = d2f_alu(el < ecount ? __ldg(ft + idx) : 0.0);
      }
    }
    __syncthreads();
#pragma unroll
    for (int n = 0; n < R; ++n) {
      const int rem = t + n * BLOCK, el = rem / NP;
      float* out = sA + (rem - el * NP) * PE + el;
      const float* Gs = sG + el;
      if constexpr (EQ == DG_WAVE) {
        float* x = sX + (rem - el * NP) * PE + el;
#pragma unroll
        for (int k = 0; k < NF; ++k) x[k * XS] = q[n][k] = d2f_alu(v[n][k]);
      }
#pragma unroll
      for (int r = 0; r < 3; ++r) {
        const float g0 = Gs[r * 3 * PE], g1 = Gs[(r * 3 + 1) * PE], g2 = Gs[(r * 3 + 2) * PE];
        if constexpr (EQ == DG_WAVE) {
          out[r * XS] = fmaf(g0, q[n][1], fmaf(g1, q[n][2], g2 * q[n][3]));
        } else {
          // U_r = (G u)_r; fluxes (G m)_r, (E + p) U_r, m_c U_r + p G[r][c] in
          // array 3 k + r
          const float p = tr[n].p, ep = q[n][1] + p, rinv = tr[n].rinv;
          const float u0 = q[n][2] * rinv, u1 = q[n][3] * rinv, u2 = q[n][4] * rinv;
          const float ur = fmaf(g0, u0, fmaf(g1, u1, g2 * u2));
          out[r * XS] = fmaf(g0, q[n][2], fmaf(g1, q[n][3], g2 * q[n][4]));
          out[(3 + r) * XS] = ep * ur;
          out[(6 + r) * XS] = fmaf(q[n][2], ur, p * g0);
          out[(9 + r) * XS] = fmaf(q[n][3], ur, p * g1);
          out[(12 + r) * XS] = fmaf(q[n][4], ur, p * g2);
        }
      }
    }
    // this thread's face points: their gather indices, read ahead of the fluxes
    constexpr int NPT = (E * NFPT + BLOCK - 1) / BLOCK;
    uint32_t gidx_f[NPT];
#pragma unroll
    for (int n = 0; n < NPT; ++n) {
      const int pidx = t + n * BLOCK;
      gidx_f[n] = pidx < ecount * NFPT ? __ldg(a.gather + e0 * NFPT + pidx) : 0u;
    }
    __syncthreads();
    // }}}

    // {{{ volume term: four columns at a time, last to first
    float acc[NF][R];
#pragma unroll
    for (int k = 0; k < NF; ++k)
#pragma unroll
      for (int i = 0; i < R; ++i) acc[k][i] = 0.0f;
    if constexpr (EQ == DG_WAVE) {
      float ur[3][R];
#pragma unroll
      for (int r = 0; r < 3; ++r)
#pragma unroll
        for (int i = 0; i < R; ++i) ur[r][i] = 0.0f;
#pragma unroll 1
      for (int j0 = 0; j0 < NP; j0 += 4) {
#pragma unroll
        for (int r = 2; r >= 0; --r)
#pragma unroll
          for (int d = 3; d >= 0; --d) {
            const int j = j0 + d;
            if (NP % 4 != 0 && j >= NP) continue;
            float w[R];
            load_rows<R>(sW + (r * NP + j) * ROW, w);
            const float av = sA[r * XS + j * PE + le], u = sX[j * PE + le];
#pragma unroll
            for (int i = 0; i < R; ++i) {
              acc[0][i] = fmaf(w[i], av, acc[0][i]);
              ur[r][i] = fmaf(w[i], u, ur[r][i]);
            }
          }
      }
      const float c = p0;
      float G[9];
#pragma unroll
      for (int k = 0; k < 9; ++k) G[k] = sG[k * PE + le];
#pragma unroll
      for (int i = 0; i < R; ++i) {
        acc[0][i] = -c * acc[0][i];
#pragma unroll
        for (int x = 0; x < 3; ++x)
          acc[1 + x][i] =
              -c * fmaf(G[x], ur[0][i], fmaf(G[3 + x], ur[1][i], G[6 + x] * ur[2][i]));
      }
    } else {
#pragma unroll 1
      for (int j0 = 0; j0 < NP; j0 += 4) {
#pragma unroll
        for (int r = 2; r >= 0; --r)
#pragma unroll
          for (int d = 3; d >= 0; --d) {
            const int j = j0 + d;
            if (NP % 4 != 0 && j >= NP) continue;
            float w[R], v[5];
            load_rows<R>(sW + (r * NP + j) * ROW, w);
            const float* in = sA + r * XS + j * PE + le;
#pragma unroll
            for (int k = 0; k < 5; ++k) v[k] = in[3 * k * XS];
#pragma unroll
            for (int k = 0; k < 5; ++k)
#pragma unroll
              for (int i = 0; i < R; ++i) acc[k][i] = fmaf(w[i], v[k], acc[k][i]);
          }
      }
    }
    __syncthreads();
    // }}}

    // {{{ face gather + numerical flux, over the volume inputs
    // two points per thread at a time, so that both points' loads are in flight
    const uint32_t tile_node0 = (uint32_t)(e0 * NP);
    constexpr int PPT = 2;
#pragma unroll
    for (int n0 = 0; n0 < NPT; n0 += PPT) {
      [[maybe_unused]] double ve[PPT][NF];
      float qi[PPT][NF], qe[PPT][NF];
      [[maybe_unused]] Trace si[PPT], se[PPT];
#pragma unroll
      for (int n = 0; n < PPT; ++n) {
        const int pidx = t + (n0 + n) * BLOCK;
        if (n0 + n >= NPT || pidx >= ecount * NFPT) continue;
        const int el = pidx / NFPT, node = sFN[pidx - el * NFPT];
        uint32_t gi = gidx_f[n0 + n < NPT ? n0 + n : 0] & 0x7fffffffu;
        if (gi >= (uint32_t)nelnp) {  // never read out of bounds
          raise_status(a.status, DG_ERR_INDEX);
          gi = tile_node0 + (uint32_t)(el * NP + node);
        }
        if constexpr (EQ == DG_WAVE) {
#pragma unroll
          for (int k = 0; k < NF; ++k) ve[n][k] = __ldg(a.q + k * nelnp + gi);
        } else {
          load_node(a.nodes, (int64_t)tile_node0 + el * NP + node, qi[n], si[n]);
          load_node(a.nodes, gi, qe[n], se[n]);  // boundary: its own node
        }
      }
#pragma unroll
      for (int n = 0; n < PPT; ++n) {
        const int pidx = t + (n0 + n) * BLOCK;
        if (n0 + n >= NPT || pidx >= ecount * NFPT) continue;
        const int el = pidx / NFPT, fj = pidx - el * NFPT;
        const bool bdry = (gidx_f[n0 + n < NPT ? n0 + n : 0] >> 31) != 0u;
        if constexpr (EQ == DG_WAVE) {
          const int node = sFN[fj];
#pragma unroll
          for (int k = 0; k < NF; ++k) {
            qi[n][k] = sX[k * XS + node * PE + el];
            qe[n][k] = d2f_alu(ve[n][k]);
          }
        }
        const float* fg = sFG + (fj / NFP) * 4 * PE + el;
        face_flux<EQ>(a, qi[n], qe[n], si[n], se[n], bdry, fg[0], fg[PE], fg[2 * PE],
                      fg[3 * PE], sA + fj * PE + el, FS);
      }
    }
    __syncthreads();
    // }}}

    // {{{ LIFT, in the same order
#pragma unroll 1
    for (int j0 = 0; j0 < NFPT; j0 += 4) {  // 4 Nfp is a multiple of 4
#pragma unroll
      for (int d = 3; d >= 0; --d) {
        const int fj = j0 + d;
        float w[R], v[NF];
        load_rows<R>(sL + fj * ROW, w);
#pragma unroll
        for (int k = 0; k < NF; ++k) v[k] = sA[k * FS + fj * PE + le];
#pragma unroll
        for (int k = 0; k < NF; ++k)
#pragma unroll
          for (int i = 0; i < R; ++i) acc[k][i] = fmaf(w[i], v[k], acc[k][i]);
      }
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < NF; ++k)
#pragma unroll
      for (int i = 0; i < R; ++i) sA[k * XS + (wid * R + i) * PE + le] = acc[k][i];
    __syncthreads();
    // }}}

    // {{{ store or fold into the RK stage (all loads of a node before its stores)
    for (int rem = t; rem < ecount * NP; rem += BLOCK) {
      const int el = rem / NP;
      const float* y = sA + (rem - el * NP) * PE + el;
      const int64_t gidx = e0 * NP + rem;
      [[maybe_unused]] double res[NF], qn[NF];
      if constexpr (STAGE) {
#pragma unroll
        for (int k = 0; k < NF; ++k) {
          res[k] = a.rk_a != 0.0 ? a.res[gidx + k * nelnp] : 0.0;
          qn[k] = __ldg(a.q + gidx + k * nelnp);
        }
      }
      const double scale = a.elem_scale ? __ldg(a.elem_scale + e0 + el) : 1.0;
#pragma unroll
      for (int k = 0; k < NF; ++k) {
        double val = f2d_alu(y[k * XS]);
        if constexpr (STAGE)
          if (a.rhs_unscaled) a.rhs_unscaled[gidx + k * nelnp] = val;
        if (a.elem_scale) val *= scale;
        if constexpr (!STAGE) {
          a.rhs[gidx + k * nelnp] = val;
        } else {
          const double r = fma(a.rk_dt, val, a.rk_a != 0.0 ? __dmul_rn(a.rk_a, res[k]) : 0.0);
          a.res[gidx + k * nelnp] = r;
          a.q_out[gidx + k * nelnp] = fma(a.rk_b, r, qn[k]);
        }
      }
    }
    __syncthreads();
    // }}}
  }
}

}  // namespace mix
}  // namespace dg
