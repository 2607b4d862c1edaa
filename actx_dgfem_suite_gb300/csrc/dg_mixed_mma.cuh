// Mixed-precision RHS of Maxwell's equations with the products on the tensor cores
// (mma.sync, 3xTF32), orders 2 and 3: variants 1 (persistent) and 3 (one CTA per 128
// elements) of meshes that fill its tiles (dg_plan_create).
//
// What bounded dg_rhs_kernel there: instruction issue.  It split both operands of
// every product into their TF32 parts at each use, moved the products' results
// through shared memory and synchronised the CTA after every phase.  Here one warp
// evaluates 8 elements from the state to the result without a CTA barrier:
//   - columns of a product are the 8 elements of one field, rows eight nodes each of
//     d/dr, d/ds, d/dt, so a thread holds all three derivatives of its nodes and
//     elements and forms the curl in registers; LIFT's results meet it there;
//   - operators are split once, on the host, and lie in the order of the mma
//     operands (two 16-byte loads per 16 x 8 block); data is split once per product
//     and field group;
//   - a thread's gathered traces are loaded for two face points at a time, the
//     indices of the next two meanwhile.
// Measured (GB300, whole RHS, the fastest variant of dg_rhs_kernel -> here): P2 at
// 511,104 tets 557 -> 371 us, P3 at 279,936 tets 651 -> 407 us; RK stage P3 at 82,944
// tets 237 -> 188 us (the stage's FP64 operations, 180 FP64-pipe cycles per element,
// come on top).  ncu (P3, 82,944 tets, 16 warps): issue slots 49 % busy while the SMs
// are, tensor pipe 26 %, 7.9 cycles per issued instruction of a warp (waits for fixed
// latencies 1.9, loads 1.4, shared memory 1.0, math pipes 0.8).
// The m16n8k8 products run over the same columns k in the same order as there, and
// the flux in the same operations, so results are bit for bit the same.
#pragma once

#include "dg_rhs.cuh"

namespace dg {
namespace mma {

// Eight-node groups; slot s = 3 q + r of the volume product holds derivative r of
// group q in rows 8 (s % 2) .. of m-tile s / 2, slot q of LIFT group q.  Operator
// block: per m-tile and k-step 32 lanes x (4 high, 4 low) words, volume then LIFT;
// then the int32 face node table.
template <int N>
struct Ops {
  static constexpr int NP = Shape<N>::NP, NFPT = Shape<N>::NFPT;
  static constexpr int NG = (NP + 7) / 8;
  static constexpr int VM = (3 * NG + 1) / 2, VK = (NP + 7) / 8;
  static constexpr int LM = (NG + 1) / 2, LK = (NFPT + 7) / 8;
  static constexpr int L = VM * VK * 256;                   // LIFT, in words
  static constexpr int FN = (L + LM * LK * 256) * 4;        // bytes from here
  static constexpr int SIZE = FN + pad16(NFPT * 4);
};

// Shared memory: operators, then per warp the state and the face values in FP32
// ([field][node][8 elements]), metric and face geometry.  One CTA per SM: 16 warps of
// 128 registers at order 2; at order 3, whose products need more, 12 of 168 (279,936
// tets: RHS 419 -> 407 us, RK stage 609 -> 558; at order 2 12 warps took 462 us, 16 371).
template <int N>
struct Tile {
  static constexpr int NP = Shape<N>::NP, NFPT = Shape<N>::NFPT;
  static constexpr int E = 8, WARPS = N == 3 ? 12 : 16, BLOCK = 32 * WARPS;
  static constexpr int X = 0, F = X + 6 * NP * E, G = F + 6 * NFPT * E, FG = G + 9 * E;
  static constexpr int WORDS = FG + 16 * E;                 // of a warp
  static constexpr int SMEM = Ops<N>::SIZE + WARPS * WORDS * 4;
};

// Word of (row, element) in an array [row][8 elements]: the element is permuted by
// the row so that both the accesses along elements with four consecutive rows
// (products) and those along 32 rows of one element (fluxes) touch 32 banks.
__device__ __forceinline__ int at(int row, int el) { return row * 8 + (el ^ ((row >> 2) & 7)); }

__device__ __forceinline__ void load_operand(const uint32_t* p, uint32_t (&hi)[4],
                                             uint32_t (&lo)[4]) {
  const uint4 h = *reinterpret_cast<const uint4*>(p);
  const uint4 l = *reinterpret_cast<const uint4*>(p + 128);
  hi[0] = h.x, hi[1] = h.y, hi[2] = h.z, hi[3] = h.w;
  lo[0] = l.x, lo[1] = l.y, lo[2] = l.z, lo[3] = l.w;
}

// acc[m][f] += operator x (rows of field f) for NFLD fields, FS words apart.  K rows,
// KT k-steps, MT m-tiles.
template <int MT, int KT, int K, int NFLD, int FS>
__device__ __forceinline__ void product(const uint32_t* __restrict__ ops,
                                        const float* __restrict__ x, float (&acc)[MT][NFLD][4]) {
  const int lane = threadIdx.x & 31, g = lane >> 2, tq = lane & 3;
  __syncwarp();
#pragma unroll 1
  for (int kt = 0; kt < KT; ++kt) {
    uint32_t bh[NFLD][2], bl[NFLD][2];
#pragma unroll
    for (int f = 0; f < NFLD; ++f)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int k0 = kt * 8 + 4 * h;                      // rows k0 + tq
        float v = 0.0f;
        if (k0 + 3 < K || (k0 < K && k0 + tq < K)) v = x[f * FS + at(k0 + tq, g)];
        tf32_split(v, bh[f][h], bl[f][h]);
      }
#pragma unroll
    for (int mt = 0; mt < MT; ++mt) {
      uint32_t ah[4], al[4];
      load_operand(ops + (mt * KT + kt) * 256 + lane * 4, ah, al);
#pragma unroll
      for (int f = 0; f < NFLD; ++f) mma_tf32(acc[mt][f], al, bh[f][0], bh[f][1]);
#pragma unroll
      for (int f = 0; f < NFLD; ++f) mma_tf32(acc[mt][f], ah, bl[f][0], bl[f][1]);
#pragma unroll
      for (int f = 0; f < NFLD; ++f) mma_tf32(acc[mt][f], ah, bh[f][0], bh[f][1]);
    }
  }
}

// a b - c d, contracted as in dg_rhs_kernel (written out: the compiler's choice
// depends on the surrounding code)
__device__ __forceinline__ float det2(float a, float b, float c, float d) {
  return fmaf(a, b, -__fmul_rn(c, d));
}

__device__ __forceinline__ void cross(const float* a, const float* b, float* c) {
  c[0] = det2(a[1], b[2], a[2], b[1]);
  c[1] = det2(a[2], b[0], a[0], b[2]);
  c[2] = det2(a[0], b[1], a[1], b[0]);
}

template <int N, bool STAGE>
__global__ void __launch_bounds__(Tile<N>::BLOCK) dg_maxwell_mma_kernel(const RhsArgs a) {
  using T = Tile<N>;
  using O = Ops<N>;
  constexpr int NP = T::NP, NFP = Shape<N>::NFP, NFPT = T::NFPT, E = T::E, NG = O::NG;
  extern __shared__ __align__(128) unsigned char smem[];
  __shared__ uint64_t bar;
  __shared__ int ops_ok;
  const uint32_t* sV = reinterpret_cast<const uint32_t*>(smem);
  const uint32_t* sL = sV + O::L;
  const int* sFN = reinterpret_cast<const int*>(smem + O::FN);
  const int t = threadIdx.x, lane = t & 31, wid = t >> 5;
  float* sX = reinterpret_cast<float*>(smem + O::SIZE) + wid * T::WORDS;
  float* sF = sX + T::F;
  float* sG = sX + T::G;
  float* sFG = sX + T::FG;
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
  const int el = lane & 7, l4 = lane >> 3;   // loads: element, node
  const int g = lane >> 2, tq = lane & 3;    // products: row group, columns 2 tq, + 1
  for (int64_t tile = (int64_t)blockIdx.x * T::WARPS + wid; tile < ntiles;
       tile += (int64_t)gridDim.x * T::WARPS) {
    const int64_t e0 = tile * E;
    const int ecount = (nel - e0) < (int64_t)E ? (int)(nel - e0) : E;
    const bool live = el < ecount;

    // {{{ state and geometry
#pragma unroll
    for (int k = 0; k < 6; ++k) {
      double v[(NP + 3) / 4];
#pragma unroll
      for (int n = 0; n < (NP + 3) / 4; ++n) {
        const int node = l4 + 4 * n;
        v[n] = live && node < NP ? __ldg(a.q + k * nelnp + (e0 + el) * NP + node) : 0.0;
      }
#pragma unroll
      for (int n = 0; n < (NP + 3) / 4; ++n) {
        const int node = l4 + 4 * n;
        if (NP % 4 == 0 || node < NP) sX[k * NP * E + at(node, el)] = d2f_alu(v[n]);
      }
    }
    for (int idx = l4; idx < 9; idx += 4)
      sG[idx * E + el] = d2f_alu(live ? __ldg(a.metric + (e0 + el) * 9 + idx) : 0.0);
#pragma unroll
    for (int n = 0; n < 4; ++n)
      sFG[(l4 + 4 * n) * E + el] =
          d2f_alu(live ? __ldg(a.face_geom + (e0 + el) * 16 + l4 + 4 * n) : 0.0);
    __syncwarp();
    // }}}

    // {{{ volume term: E_t = curl H, then H_t = -curl E, in registers
    float vol[6][NG][2];  // field, node group, column
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      float acc[O::VM][3][4];
#pragma unroll
      for (int m = 0; m < O::VM; ++m)
#pragma unroll
        for (int f = 0; f < 3; ++f)
#pragma unroll
          for (int c = 0; c < 4; ++c) acc[m][f][c] = 0.0f;
      product<O::VM, O::VK, NP, 3, NP * E>(sV, sX + (3 - 3 * half) * NP * E, acc);
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        float G[9];
#pragma unroll
        for (int k = 0; k < 9; ++k) G[k] = sG[k * E + 2 * tq + c];
#pragma unroll
        for (int q = 0; q < NG; ++q) {
          auto d = [&](int f, int r) { return acc[(3 * q + r) / 2][f][((3 * q + r) & 1) * 2 + c]; };
          auto dx = [&](int f, int x) {
            return fmaf(G[x], d(f, 0), fmaf(G[3 + x], d(f, 1), __fmul_rn(G[6 + x], d(f, 2))));
          };
          const float w0 = dx(2, 1) - dx(1, 2), w1 = dx(0, 2) - dx(2, 0),
                      w2 = dx(1, 0) - dx(0, 1);
          vol[3 * half + 0][q][c] = half == 0 ? w0 : -w0;
          vol[3 * half + 1][q][c] = half == 0 ? w1 : -w1;
          vol[3 * half + 2][q][c] = half == 0 ? w2 : -w2;
        }
      }
    }
    // }}}

    // {{{ face gather + numerical flux: 8 NFPT points, consecutive ones of an element
    // on consecutive lanes (a face's traces share memory sectors)
    const float alpha = a.c32[0], z = a.c32[1], y = a.c32[2];
    const float ce = a.c32[3], ch = a.c32[4];
    constexpr int PPT = 2;  // points whose loads are in flight together
    static_assert(E * NFPT % (32 * PPT) == 0, "whole rounds of face points");
    const uint32_t* gt = a.gather + e0 * NFPT + lane;
    uint32_t gnext[PPT];
#pragma unroll
    for (int n = 0; n < PPT; ++n)
      gnext[n] = lane + 32 * n < ecount * NFPT ? __ldg(gt + 32 * n) : 0x80000000u;
#pragma unroll 1
    for (int p0 = lane; p0 < E * NFPT; p0 += 32 * PPT) {
      uint32_t gi[PPT];
      double ve[PPT][6];
#pragma unroll
      for (int n = 0; n < PPT; ++n) {
        gi[n] = gnext[n];
        uint32_t gn = gi[n] & 0x7fffffffu;
        if (gn >= (uint32_t)nelnp) {  // never read out of bounds
          raise_status(a.status, DG_ERR_INDEX);
          const int ep = (p0 + 32 * n) / NFPT;
          gn = (uint32_t)((e0 + ep) * NP + sFN[p0 + 32 * n - ep * NFPT]);
        }
        if (!(gi[n] >> 31))
#pragma unroll
          for (int k = 0; k < 6; ++k) ve[n][k] = __ldg(a.q + k * nelnp + gn);
      }
#pragma unroll
      for (int n = 0; n < PPT; ++n) {  // the next round's indices
        const int pn = p0 + 32 * (PPT + n);
        gnext[n] = pn < ecount * NFPT ? __ldg(gt + (pn - lane)) : 0x80000000u;
      }
#pragma unroll
      for (int n = 0; n < PPT; ++n) {
        const int ep = (p0 + 32 * n) / NFPT, fj = p0 + 32 * n - ep * NFPT, node = sFN[fj];
        const bool bdry = (gi[n] >> 31) != 0u;
        float qi[6], qe[6];
#pragma unroll
        for (int k = 0; k < 6; ++k) {
          qi[k] = sX[k * NP * E + at(node, ep)];
          // PEC: exterior (-E, H)
          qe[k] = bdry ? (k < 3 ? -qi[k] : qi[k]) : d2f_alu(ve[n][k]);
        }
        const float* fg = sFG + (fj / NFP) * 4 * E + ep;
        const float nv[3] = {fg[0], fg[E], fg[2 * E]}, scale = fg[3 * E];
        const float je[3] = {qe[0] - qi[0], qe[1] - qi[1], qe[2] - qi[2]};
        const float jh[3] = {qe[3] - qi[3], qe[4] - qi[4], qe[5] - qi[5]};
        float nxe[3], nxh[3], te[3], th[3], fe[3], fh[3];
        cross(nv, je, nxe);
        cross(nv, jh, nxh);
#pragma unroll
        for (int x = 0; x < 3; ++x) {
          te[x] = det2(z, jh[x], alpha, nxe[x]);
          th[x] = fmaf(y, je[x], __fmul_rn(alpha, nxh[x]));
        }
        cross(nv, te, fe);
        cross(nv, th, fh);
        float* out = sF + at(fj, ep);
#pragma unroll
        for (int x = 0; x < 3; ++x) {
          out[x * NFPT * E] = __fmul_rn(-scale, __fmul_rn(ce, fe[x]));
          out[(3 + x) * NFPT * E] = __fmul_rn(-scale, __fmul_rn(ch, fh[x]));
        }
      }
    }
    __syncwarp();
    // }}}

    // {{{ LIFT; the sums go over the state's arrays, so that the loads and stores of
    // the epilogue are coalesced and independent
    const float inv_eps = a.c32[5], inv_mu = a.c32[6];
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      float acc[O::LM][3][4];
#pragma unroll
      for (int m = 0; m < O::LM; ++m)
#pragma unroll
        for (int f = 0; f < 3; ++f)
#pragma unroll
          for (int c = 0; c < 4; ++c) acc[m][f][c] = 0.0f;
      product<O::LM, O::LK, NFPT, 3, NFPT * E>(sL, sF + 3 * half * NFPT * E, acc);
#pragma unroll
      for (int q = 0; q < NG; ++q)
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          const int node = 8 * q + g;
          if (NP % 8 != 0 && node >= NP) continue;
#pragma unroll
          for (int f = 0; f < 3; ++f)
            sX[(3 * half + f) * NP * E + at(node, 2 * tq + c)] =
                (vol[3 * half + f][q][c] + acc[q / 2][f][(q & 1) * 2 + c]) *
                (half == 0 ? inv_eps : inv_mu);
        }
    }
    __syncwarp();
    // }}}

    // {{{ store or fold into the RK stage (the loads of a group before its stores)
    if (live) {
      constexpr int NQ = (NP + 3) / 4, KG = STAGE ? 2 : 6;  // nodes of a thread, fields
      const double scale = a.elem_scale ? __ldg(a.elem_scale + e0 + el) : 1.0;
      const int64_t base = (e0 + el) * NP + l4;
#pragma unroll 1
      for (int k0 = 0; k0 < 6; k0 += KG) {
        [[maybe_unused]] double res[KG][NQ], qn[KG][NQ];
        if constexpr (STAGE) {
#pragma unroll
          for (int k = 0; k < KG; ++k)
#pragma unroll
            for (int n = 0; n < NQ; ++n) {
              const int64_t gidx = base + 4 * n + (k0 + k) * nelnp;
              const bool in = NP % 4 == 0 || l4 + 4 * n < NP;
              res[k][n] = in && a.rk_a != 0.0 ? a.res[gidx] : 0.0;
              qn[k][n] = in ? __ldg(a.q + gidx) : 0.0;
            }
        }
#pragma unroll
        for (int k = 0; k < KG; ++k)
#pragma unroll
          for (int n = 0; n < NQ; ++n) {
            if (NP % 4 != 0 && l4 + 4 * n >= NP) continue;
            const int64_t gidx = base + 4 * n + (k0 + k) * nelnp;
            double val = f2d_alu(sX[(k0 + k) * NP * E + at(l4 + 4 * n, el)]);
            if constexpr (STAGE)
              if (a.rhs_unscaled) a.rhs_unscaled[gidx] = val;
            if (a.elem_scale) val *= scale;
            if constexpr (!STAGE) {
              a.rhs[gidx] = val;
            } else {
              const double r =
                  fma(a.rk_dt, val, a.rk_a != 0.0 ? __dmul_rn(a.rk_a, res[k][n]) : 0.0);
              a.res[gidx] = r;
              a.q_out[gidx] = fma(a.rk_b, r, qn[k][n]);
            }
          }
      }
    }
    __syncwarp();
    // }}}
  }
}

}  // namespace mma
}  // namespace dg
