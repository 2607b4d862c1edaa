// FP64 volume/LIFT kernel in the symmetry-adapted basis of the tetrahedron
// (sm_103a), the main kernel of the face-shared path (dg_face.cuh).
//
// What bounds it: the FP64 pipe.  GB300 issues two FP64 multiply-adds per SM
// and clock (measured 1.25 TFLOP/s), so the dense products of dg_rhs_kernel
// held that pipe at 94-97 % for orders 2-4 and the only way down is fewer
// FP64 operations.  The reference tetrahedron gives them: its node set and
// operators are invariant under permutations of its vertices, and the
// four-group V = {id, g1 = (01)(23), g2 = (02)(13), g3 = (03)(12)} is enough
// to split every operator into blocks.  With one butterfly (sum and difference
// transform) per orbit of nodes a field splits into four parts, A (even under
// every g) and B1, B2, B3 (B_k even under g_k, odd under the other two).
// Along the directions that join the midpoints of opposite edges,
// d_k = v0 + v_k - (the other two), every g maps d_k to plus or minus itself,
// so the derivative along d_k takes part sigma to the single part
// rho = sigma xor k (parts numbered 0 for A and k for B_k), and LIFT takes each
// part of the face values (V permutes the faces without fixed points: Nfp
// orbits of four points) to the same part of the nodes.  The dense Np x Np
// derivatives and the Np x 4 Nfp LIFT become four blocks each: a quarter of
// the multiply-adds for two additions per node or face point and field.
//
//   multiply-adds per field   derivative (one direction)      LIFT
//   order 1 / 2 / 3 / 4       16 / 100 / 400 / 1225 dense     48 / 240 / 800 / 2100
//                              1 /  24 / 100 /  304 here      12 /  60 / 200 /  525
//
// (wave and Maxwell fewer still: see Ops).
//
// The direction metric follows from the element's dr/dx:
// sum_r g_r D_r = sum_k h_k D'_k with h_1 = g_2 + g_3 (cyclic) and
// D'_k = -1/2 D_{d_k}; the host folds all constants and the butterflies'
// normalisation into the blocks, and takes this path only for operators whose
// blocks outside the pattern vanish to rounding (pack_sym_ops, sym_ops.cu);
// others keep dg_rhs_kernel.
//
// Measured (GB300, CUDA events, whole RHS with its face kernel, dense kernel
// before -> now): Maxwell P4 584,016 tets 38.9 -> 13.1 ms, Euler P4 118,098 tets
// 7.08 -> 2.88 ms, wave P3 215,622 tets 2.69 -> 1.17 ms, Euler P2 LSRK step
// 413,526 tets 16.7 -> 10.8 ms, wave P1 5.14 M tets 5.77 -> 4.17 ms.  ncu: FP64
// pipe 83 % (wave P1) to 92 % (Maxwell P4) busy.
//
// Work split: a tile of E elements with one lane per element and one warp per
// part rho, so that every operator entry is the same for a whole warp and is
// read once, by a broadcast, for all fields of the thread; accumulators stay
// in registers.  Data sits in shared memory as [array][slot][element] with an
// odd element pitch (no bank conflicts along elements or slots).  Per tile:
// state -> slots; transform; volume blocks; face values (transformed on the
// way in, over the state's shared memory); LIFT blocks; inverse transform;
// store or Runge-Kutta stage.
#pragma once

#include "dg_rhs.cuh"

namespace dg {
namespace sym {

// Orbits of the node set under V: NO4 orbits of four nodes, NPR pairs (edge
// midpoints) per direction, NSG fixed points (the centroid); DA and DB nodes
// in parts A and B_k.
template <int N>
struct Basis {
  static constexpr int NP = Shape<N>::NP, NFP = Shape<N>::NFP, NFPT = 4 * NFP;
  static constexpr int NPR = N % 2 == 0 ? 1 : 0, NSG = N == 4 ? 1 : 0;
  static constexpr int NO4 = (NP - 6 * NPR - NSG) / 4;
  static constexpr int DB = NO4 + NPR, DA = NO4 + 3 * NPR + NSG;
  static_assert(DA + 3 * DB == NP, "the parts cover the node set");
};

// Operator block: doubles in rows of one input each, padded to 16 bytes.
// Volume blocks of part 0, then 1, 2, 3, each for k = 1, 2, 3 (inputs of part
// rho xor k); LIFT blocks the same way (NFP inputs).  Then three int32 tables:
// node -> slot, slot -> node, and the face point of every face slot (part r of
// orbit o at r NFP + o).  AdjOps: the transposed derivatives' blocks in the same
// place and the transposed LIFT blocks, in chunks of CH orbits: the chunk's
// rows of part 0 (DA inputs), then of parts 1, 2, 3, each CH entries padded.
template <int N>
constexpr int chunk_orbits() {  // orbits of face values held at a time
  return N == 1 ? Basis<N>::NFP : (Basis<N>::NFP + 1) / 2;
}

// A derivative lowers the degree by one.  Strong derivatives (RED = 1) therefore map
// into the polynomials of degree N - 1, RA and RB of them in parts A and B_k: the
// blocks go to coefficients in an orthonormal basis of that space and one more block
// per part takes the summed coefficients to the nodes.  Weak derivatives (RED = 2)
// see of their input only its projection onto that space: one block per part takes
// the nodes to coefficients, which the volume blocks read.  A field's product along
// one direction costs 10 / 50 / 175 multiply-adds at orders 2 / 3 / 4 (24 / 100 / 304
// without), the extra block as much once per field: less where fields share a
// product's result (Maxwell P4, 584,016 tets, whole RHS: 14.3 -> 13.1 ms) or a field
// enters several (wave P3, 215,622 tets: 1.24 -> 1.17 ms).  Order 1 has one non-zero
// block per direction as it is, and Euler's 15 products have 15 different inputs.
enum { RED_NONE = 0, RED_OUT = 1, RED_IN = 2 };

template <int N, int EQ>
constexpr int reduction() {
  return N == 1 || EQ == DG_EULER ? RED_NONE : (EQ == DG_MAXWELL ? RED_OUT : RED_IN);
}

template <int N, int RED = RED_NONE>
struct Ops {
  using B = Basis<N>;
  static constexpr int RA = RED ? Basis<N - (RED != 0)>::DA : B::DA;
  static constexpr int RB = RED ? Basis<N - (RED != 0)>::DB : B::DB;
  // inputs and outputs of the volume blocks in part A and in the others
  static constexpr int INA = RED == RED_IN ? RA : B::DA, INB = RED == RED_IN ? RB : B::DB;
  static constexpr int OUTA = RED == RED_OUT ? RA : B::DA, OUTB = RED == RED_OUT ? RB : B::DB;
  static constexpr int PA = (B::DA + 1) & ~1, PB = (B::DB + 1) & ~1;
  static constexpr int PRA = (RA + 1) & ~1, PRB = (RB + 1) & ~1;
  static constexpr int POA = (OUTA + 1) & ~1, POB = (OUTB + 1) & ~1;
  static constexpr int VOL0 = 3 * INB * POA;                // entries of part 0
  static constexpr int VOLB = (INA + 2 * INB) * POB;        // of each part B_k
  // coefficients -> nodes (RA rows of pitch PA) or nodes -> coefficients (DA of PRA)
  static constexpr int EXTRA = VOL0 + 3 * VOLB;
  static constexpr int EXA = RED == RED_NONE ? 0 : (RED == RED_OUT ? RA * PA : B::DA * PRA);
  static constexpr int EXB = RED == RED_NONE ? 0 : (RED == RED_OUT ? RB * PB : B::DB * PRB);
  static constexpr int LIFT = EXTRA + EXA + 3 * EXB;
  static constexpr int LIFTB = LIFT + B::NFP * PA;
  static constexpr int ENTRIES = LIFTB + 3 * B::NFP * PB;
  static constexpr int NODE_SLOT = ENTRIES * 8;             // bytes from here
  static constexpr int SLOT_NODE = NODE_SLOT + pad16(B::NP * 4);
  static constexpr int FACE_POINT = SLOT_NODE + pad16(B::NP * 4);
  static constexpr int SIZE = FACE_POINT + pad16(B::NFPT * 4);
  static __host__ __device__ constexpr int volume(int rho) {
    return rho == 0 ? 0 : VOL0 + (rho - 1) * VOLB;
  }
  static __host__ __device__ constexpr int extra(int rho) {
    return EXTRA + (rho == 0 ? 0 : EXA + (rho - 1) * EXB);
  }
};

// RED: RED_OUT for the transposed weak derivatives (wave), RED_NONE
template <int N, int RED = RED_NONE>
struct AdjOps {
  using B = Basis<N>;
  using F = Ops<N, RED>;
  static constexpr int CH = chunk_orbits<N>(), NCH = (B::NFP + CH - 1) / CH;
  static constexpr int PC = (CH + 1) & ~1;
  static constexpr int LIFT = F::LIFT;                      // entries before LIFT^T
  static constexpr int CHUNK = B::NP * PC;                  // entries of a chunk
  static constexpr int NODE_SLOT = (LIFT + NCH * CHUNK) * 8;
  static constexpr int SLOT_NODE = NODE_SLOT + pad16(B::NP * 4);
  static constexpr int FACE_POINT = SLOT_NODE + pad16(B::NP * 4);
  static constexpr int SIZE = FACE_POINT + pad16(B::NFPT * 4);
};

// Tile shape.  Maxwell's E and H equations have the same form, so the two
// halves of a warp take one each, on 16 elements per tile; wave and Euler keep
// all fields in a thread and 32 elements per tile.  Face values and result
// reuse the state's arrays; from order 2 on the face values come in two chunks
// of orbits, so that a tile's shared memory is little more than its state and
// three to four CTAs share an SM at order 4: their phases (loads, transforms,
// products) must overlap to keep the FP64 pipe busy.
template <int N, int EQ>
struct Tile {
  using B = Basis<N>;
  using O = Ops<N, reduction<N, EQ>()>;
  static constexpr int NF = EqInfo<EQ>::NF;
  static constexpr int GROUPS = EQ == DG_MAXWELL ? 2 : 1;
  static constexpr int NA = NF / GROUPS;                    // fields of a thread
  static constexpr int E = 32 / GROUPS, PE = E + 1;
  static constexpr int BLOCK = 128;
  // CTAs per SM the registers must allow (order-4 Euler: 168 instead of 186; order-1
  // Euler: 64 instead of 92)
  static constexpr int MIN_CTAS = N == 4 ? 3 : (N == 1 && EQ == DG_EULER ? 8 : 4);
  static constexpr int CH = chunk_orbits<N>();
  static constexpr int X = O::SIZE;
  static constexpr int X_BYTES = pad16(NF * B::NP * PE * 8);
  static constexpr int F_BYTES = pad16(NF * 4 * CH * PE * 8);
  static constexpr int H = X + (X_BYTES > F_BYTES ? X_BYTES : F_BYTES);
  static constexpr int SMEM = H + pad16(9 * PE * 8);
};

// (x0, x1, x2, x3) at (n, g1 n, g2 n, g3 n) <-> parts A, B1, B2, B3 (its own
// inverse up to the factor 4 that the operator blocks hold)
__device__ __forceinline__ void butterfly(double& a, double& b, double& c, double& d) {
  const double s = a + b, t = a - b, u = c + d, v = c - d;
  a = s + u;
  b = s - u;
  c = t + v;
  d = t - v;
}

// Barrier of the whole CTA for warps that arrive from different branches (the
// parts' code differs where their sizes do); the branch is uniform per warp.
template <int BLOCK>
__device__ __forceinline__ void cta_sync() {
  asm volatile("bar.sync 1, %0;" ::"n"(BLOCK) : "memory");
}

// One row of operator entries, the same for the whole warp.
template <int P>
__device__ __forceinline__ void load_row(const double* p, double (&r)[P]) {
#pragma unroll
  for (int k = 0; k < P; k += 2) {
    const double2 v = *reinterpret_cast<const double2*>(p + k);
    r[k] = v.x;
    r[k + 1] = v.y;
  }
}

// Volume term of part rho (D outputs, row pitch P; IA and IB inputs of parts A and
// B_k), wave and Maxwell.  x: the thread's element in shared memory; h: metric of the three directions (pitch
// PE per entry); f0: first input field (Maxwell); sgn: Maxwell's curl sign,
// wave's -c.  At order 1 one block per direction is not zero: into part A for
// strong (and transposed weak) derivatives, from part A for weak ones.
template <int N, int EQ, int D, int P, int IA, int IB, bool INTO_A = EQ == DG_MAXWELL>
__device__ __forceinline__ void volume(const double* __restrict__ x,
                                       const double* __restrict__ h,
                                       const double* __restrict__ row, int rho, int f0,
                                       double sgn, double (&acc)[Tile<N, EQ>::NA][D]) {
  using B = Basis<N>;
  constexpr int PE = Tile<N, EQ>::PE, FS = B::NP * PE;  // array stride
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const int sig = rho ^ (k + 1);
    const int din = sig == 0 ? IA : IB;
    const double* xs = x + (sig == 0 ? 0 : B::DA + (sig - 1) * B::DB) * PE;
    if (N == 1 && (INTO_A ? rho : sig) != 0) {
      row += din * P;
      continue;
    }
    const double h0 = sgn * h[(k * 3 + 0) * PE], h1 = sgn * h[(k * 3 + 1) * PE],
                 h2 = sgn * h[(k * 3 + 2) * PE];
    if constexpr (EQ == DG_WAVE) {
      double g[D];
#pragma unroll
      for (int i = 0; i < D; ++i) g[i] = 0.0;
#pragma unroll 1
      for (int j = 0; j < din; ++j, row += P, xs += PE) {
        const double u = xs[0];
        const double w = fma(h0, xs[FS], fma(h1, xs[2 * FS], h2 * xs[3 * FS]));
        double t[P];
        load_row<P>(row, t);
#pragma unroll
        for (int i = 0; i < D; ++i) {
          acc[0][i] = fma(t[i], w, acc[0][i]);
          g[i] = fma(t[i], u, g[i]);
        }
      }
#pragma unroll
      for (int i = 0; i < D; ++i) {
        acc[1][i] = fma(h0, g[i], acc[1][i]);
        acc[2][i] = fma(h1, g[i], acc[2][i]);
        acc[3][i] = fma(h2, g[i], acc[3][i]);
      }
    } else {
      const double* xf = xs + f0 * FS;
#pragma unroll 1
      for (int j = 0; j < din; ++j, row += P, xf += PE) {
        const double v0 = xf[0], v1 = xf[FS], v2 = xf[2 * FS];
        double t[P];
        load_row<P>(row, t);
        const double w0 = fma(h1, v2, -h2 * v1);
        const double w1 = fma(h2, v0, -h0 * v2);
        const double w2 = fma(h0, v1, -h1 * v0);
#pragma unroll
        for (int i = 0; i < D; ++i) {
          acc[0][i] = fma(t[i], w0, acc[0][i]);
          acc[1][i] = fma(t[i], w1, acc[1][i]);
          acc[2][i] = fma(t[i], w2, acc[2][i]);
        }
      }
    }
  }
}

// acc += block * fields for `rows` inputs: x is the thread's element at the
// first input of the first field, FS the field stride.
template <int NA, int D, int P, int PE, int FS>
__device__ __forceinline__ void block_product(const double* __restrict__ x,
                                              const double* __restrict__ row, int rows,
                                              double (&acc)[NA][D]) {
#pragma unroll 1
  for (int j = 0; j < rows; ++j, row += P, x += PE) {
    double v[NA], t[P];
#pragma unroll
    for (int m = 0; m < NA; ++m) v[m] = x[m * FS];
    load_row<P>(row, t);
#pragma unroll
    for (int m = 0; m < NA; ++m)
#pragma unroll
      for (int i = 0; i < D; ++i) acc[m][i] = fma(t[i], v[m], acc[m][i]);
  }
}

// acc += expansion of the coefficients c (part's R rows of pitch P).
template <int NA, int R, int D, int P>
__device__ __forceinline__ void expand(const double* __restrict__ row,
                                       const double (&c)[NA][R], double (&acc)[NA][D]) {
#pragma unroll
  for (int j = 0; j < R; ++j) {
    double t[P];
    load_row<P>(row + j * P, t);
#pragma unroll
    for (int m = 0; m < NA; ++m)
#pragma unroll
      for (int i = 0; i < D; ++i) acc[m][i] = fma(t[i], c[m][j], acc[m][i]);
  }
}

// In-place (inverse) transform of `narrays` node arrays of a tile.  A_ONLY (order 1,
// weak derivatives): the volume term reads part A alone, 3 of the butterfly's 8
// additions (with the same for Euler below; wave P1, 5.14 M tets: 4.36 -> 4.17 ms).
template <int N, int PE, int E, int BLOCK, bool A_ONLY = false>
__device__ __forceinline__ void transform(double* x, int narrays) {
  using B = Basis<N>;
  constexpr int NO = B::NO4 + 3 * B::NPR;
  const int le = threadIdx.x % E;
  for (int job = threadIdx.x / E; job < narrays * NO; job += BLOCK / E) {
    const int f = job / NO, o = job - f * NO;
    double* p = x + f * (B::NP * PE) + le;
    if (o < B::NO4) {
      double* b = p + (B::DA + o) * PE;
      if constexpr (A_ONLY)
        p[o * PE] = (p[o * PE] + b[0]) + (b[B::DB * PE] + b[2 * B::DB * PE]);
      else
        butterfly(p[o * PE], b[0], b[B::DB * PE], b[2 * B::DB * PE]);
    } else {  // the pair of direction o - NO4 + 1
      double& u = p[o * PE];
      double& v = p[(B::DA + (o - B::NO4) * B::DB + B::NO4) * PE];
      const double s = u + v, d = u - v;
      u = s;
      v = d;
    }
  }
}

// Euler: the five fluxes along direction k (metric row h_k), transformed.  With
// U = h.m / rho: h.m, (E + p) U and m_c U + p h_c, 12 operations per node.  The
// state is read from memory once per direction (twice from L2): with the
// twelve flux components in shared memory instead (82 operations per node with
// the metric combinations, here 66) one CTA fitted on an SM at order 4 and the
// FP64 pipe was 74 % busy (kernel at P4, 118,098 tets: 2.89 ms, now 2.24; RK
// stage at P2, 413,526 tets: 1.47 ms, now 1.37).
// Orbits of the same length go to the same warps (an FP64 instruction costs the
// pipe a whole warp's time however many of its lanes are active).
template <int N>
__device__ __forceinline__ void euler_inputs(const RhsArgs& a, int64_t e0, int ecount, int k,
                                             const int* __restrict__ slot_node,
                                             const double* __restrict__ sH, double* sX) {
  using B = Basis<N>;
  using T = Tile<N, DG_EULER>;
  constexpr int PE = T::PE, XS = B::NP * PE, DA = B::DA, DB = B::DB, NO4 = B::NO4;
  const int64_t nelnp = a.nel * B::NP;
  // the orbit of CNT nodes at the given slots, element el of the tile
  auto orbit = [&](auto tag, int el, int s0, int s1, int s2, int s3) {
    constexpr int CNT = decltype(tag)::value;
    const int slot[4] = {s0, s1, s2, s3};
    const double* h = sH + k * 3 * PE + el;
    const double h0 = h[0], h1 = h[PE], h2 = h[2 * PE];
    double f[5][CNT];
#pragma unroll
    for (int n = 0; n < CNT; ++n) {
      double en = 0.0, m0 = 0.0, m1 = 0.0, m2 = 0.0, p = 0.0, rinv = 0.0;
      if (el < ecount) {
        const int64_t g = (e0 + el) * B::NP + slot_node[slot[n]];
        const double* q = a.q + nelnp + g;
        en = __ldg(q);
        m0 = __ldg(q + nelnp);
        m1 = __ldg(q + 2 * nelnp);
        m2 = __ldg(q + 3 * nelnp);
        p = __ldg(a.aux + g);
        rinv = __ldg(a.aux + nelnp + g);
      }
      const double hm = fma(h0, m0, fma(h1, m1, h2 * m2));
      const double u = hm * rinv;
      f[0][n] = hm;
      f[1][n] = (en + p) * u;
      f[2][n] = fma(m0, u, p * h0);
      f[3][n] = fma(m1, u, p * h1);
      f[4][n] = fma(m2, u, p * h2);
    }
    double* x = sX + el;
#pragma unroll
    for (int m = 0; m < 5; ++m, x += XS) {
      if constexpr (N == 1) {  // order 1 reads part A alone
        x[slot[0] * PE] = (f[m][0] + f[m][1]) + (f[m][2] + f[m][3]);
        continue;
      } else if constexpr (CNT == 4) {
        butterfly(f[m][0], f[m][1], f[m][2], f[m][3]);
      } else if constexpr (CNT == 2) {
        const double s = f[m][0] + f[m][1], d = f[m][0] - f[m][1];
        f[m][0] = s;
        f[m][1] = d;
      }
#pragma unroll
      for (int n = 0; n < CNT; ++n) x[slot[n] * PE] = f[m][n];
    }
  };
  for (int idx = threadIdx.x; idx < T::E * NO4; idx += T::BLOCK) {
    const int el = idx / NO4, o = idx - el * NO4;
    orbit(std::integral_constant<int, 4>{}, el, o, DA + o, DA + DB + o, DA + 2 * DB + o);
  }
  if constexpr (B::NPR > 0)  // backwards, so that other warps take these
    for (int idx = T::BLOCK - 1 - threadIdx.x; idx < T::E * 3; idx += T::BLOCK) {
      const int el = idx / 3, d = idx - el * 3;
      orbit(std::integral_constant<int, 2>{}, el, NO4 + d, DA + d * DB + NO4, 0, 0);
    }
  if constexpr (B::NSG > 0)
    for (int el = threadIdx.x; el < T::E; el += T::BLOCK)
      orbit(std::integral_constant<int, 1>{}, el, DA - 1, 0, 0, 0);
}

template <int N, int EQ, bool STAGE>
__global__ void __launch_bounds__(Tile<N, EQ>::BLOCK, Tile<N, EQ>::MIN_CTAS)
    dg_rhs_sym_kernel(const RhsArgs a) {
  using T = Tile<N, EQ>;
  using O = typename T::O;
  using B = Basis<N>;
  constexpr int NP = B::NP, NFP = B::NFP, NFPT = B::NFPT, NF = T::NF, NA = T::NA;
  constexpr int E = T::E, PE = T::PE, BLOCK = T::BLOCK;
  constexpr int XS = NP * PE, CH = T::CH, FS = 4 * CH * PE;  // array strides
  constexpr int RED = reduction<N, EQ>();
  extern __shared__ __align__(128) unsigned char smem[];
  __shared__ uint64_t bar;
  __shared__ int ops_ok;
  const double* ops = reinterpret_cast<const double*>(smem);
  const int* node_slot = reinterpret_cast<const int*>(smem + O::NODE_SLOT);
  [[maybe_unused]] const int* slot_node = reinterpret_cast<const int*>(smem + O::SLOT_NODE);
  const int* face_point = reinterpret_cast<const int*>(smem + O::FACE_POINT);
  double* sX = reinterpret_cast<double*>(smem + T::X);
  double* sH = reinterpret_cast<double*>(smem + T::H);

  const int t = threadIdx.x;
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

  const int lane = t & 31;
  const int le = lane % E;              // element of the tile
  const int grp = lane / E;             // Maxwell: 0 the E fields, 1 the H fields
  const int64_t nel = a.nel;
  const int64_t nelnp = nel * NP;
  const int64_t ntiles = (nel + E - 1) / E;

  for (int64_t tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
    const int64_t e0 = tile * E;
    const int ecount = (nel - e0) < (int64_t)E ? (int)(nel - e0) : E;

    // {{{ metric and (wave, Maxwell) state -> shared memory, transformed
    {
      if constexpr (EQ != DG_EULER) {
        const double* qk = a.q + e0 * NP;
        for (int rem = t; rem < E * NP; rem += BLOCK) {
          const int el = rem / NP;
          double* x = sX + node_slot[rem - el * NP] * PE + el;
          const bool in = rem < ecount * NP;
          double v[NF];
#pragma unroll
          for (int k = 0; k < NF; ++k) v[k] = in ? __ldg(qk + k * nelnp + rem) : 0.0;
#pragma unroll
          for (int k = 0; k < NF; ++k) x[k * XS] = v[k];
        }
      }
      const double* mt = a.metric + e0 * 9;
      for (int idx = t; idx < 9 * E; idx += BLOCK) {
        const int el = idx / 9, kx = idx - el * 9, k = kx / 3, x = kx - k * 3;
        double v = 0.0;
        if (el < ecount)
          v = __ldg(mt + el * 9 + (k == 0 ? 3 : 0) + x) + __ldg(mt + el * 9 + (k == 2 ? 3 : 6) + x);
        sH[kx * PE + el] = v;
      }
    }
    __syncthreads();
    if constexpr (EQ != DG_EULER) {
      transform<N, PE, E, BLOCK, N == 1 && EQ == DG_WAVE>(sX, NF);
      __syncthreads();
    }
    // }}}

    // {{{ volume and LIFT blocks, one part per warp.  The parts differ in size
    // at orders 2 and 4, so they rotate over the warps (and with them over
    // the SM's four quadrants) from tile to tile.
    const int rho = ((t >> 5) + (int)tile) & 3;
    const int f_in = EQ == DG_MAXWELL ? 3 - 3 * grp : 0;
    const int f_out = EQ == DG_MAXWELL ? 3 * grp : 0;
    const double sgn = EQ == DG_MAXWELL ? (grp == 0 ? 1.0 : -1.0)
                                        : (EQ == DG_WAVE ? -a.p0 : 1.0);

    // orbits o0 .. o0 + CH - 1 of the tile's face values, transformed
    auto load_faces = [&](int o0) {
      const int64_t nfpt_all = nel * NFPT;
      const double* fk = a.flux_in + e0 * NFPT;
      for (int idx = t; idx < E * CH; idx += BLOCK) {
        const int el = idx / CH, oc = idx - el * CH, o = o0 + oc;
        if (NFP % CH != 0 && o >= NFP) continue;
        // the orbit's four points, one per face
        const int p0 = face_point[o], p1 = face_point[NFP + o],
                  p2 = face_point[2 * NFP + o], p3 = face_point[3 * NFP + o];
        const double* fe = fk + el * NFPT;
        const bool in = el < ecount;
        double v[NF][4];
#pragma unroll
        for (int k = 0; k < NF; ++k, fe += nfpt_all) {
          v[k][0] = in ? __ldg(fe + p0) : 0.0;
          v[k][1] = in ? __ldg(fe + p1) : 0.0;
          v[k][2] = in ? __ldg(fe + p2) : 0.0;
          v[k][3] = in ? __ldg(fe + p3) : 0.0;
        }
#pragma unroll
        for (int k = 0; k < NF; ++k) {
          butterfly(v[k][0], v[k][1], v[k][2], v[k][3]);
#pragma unroll
          for (int r = 0; r < 4; ++r) sX[k * FS + (r * CH + oc) * PE + el] = v[k][r];
        }
      }
    };

    auto part = [&](auto dtag, auto rtag, int slot0, const double* lops) {
      constexpr int D = decltype(dtag)::value, P = (D + 1) & ~1;
      constexpr int R = decltype(rtag)::value, PR = (R + 1) & ~1;
      const double* vops = ops + O::volume(rho);
      [[maybe_unused]] const double* xops = ops + O::extra(rho);
      double acc[NA][D];
#pragma unroll
      for (int m = 0; m < NA; ++m)
#pragma unroll
        for (int i = 0; i < D; ++i) acc[m][i] = 0.0;
      if constexpr (EQ == DG_EULER) {
#pragma unroll 1
        for (int k = 0; k < 3; ++k) {
          euler_inputs<N>(a, e0, ecount, k, slot_node, sH, sX);
          cta_sync<BLOCK>();
          const int sig = rho ^ (k + 1), din = sig == 0 ? B::DA : B::DB;
          if (N != 1 || sig == 0)  // order 1: weak derivatives leave part A only
            block_product<NA, D, P, PE, XS>(
                sX + (sig == 0 ? 0 : B::DA + (sig - 1) * B::DB) * PE + le, vops, din, acc);
          vops += din * P;
          cta_sync<BLOCK>();       // the inputs' slots are free
        }
      } else if constexpr (RED == RED_OUT) {
        double c[NA][R];
#pragma unroll
        for (int m = 0; m < NA; ++m)
#pragma unroll
          for (int i = 0; i < R; ++i) c[m][i] = 0.0;
        volume<N, EQ, R, PR, O::INA, O::INB>(sX + le, sH + le, vops, rho, f_in, sgn, c);
        expand<NA, R, D, P>(xops, c, acc);
        cta_sync<BLOCK>();         // the state's slots are free
      } else {
        if constexpr (RED == RED_IN) {  // the part's coefficients, in its first slots
          double c[NF][R];
#pragma unroll
          for (int m = 0; m < NF; ++m)
#pragma unroll
            for (int i = 0; i < R; ++i) c[m][i] = 0.0;
          double* x = sX + slot0 * PE + le;
          block_product<NF, R, PR, PE, XS>(x, xops, D, c);
#pragma unroll
          for (int m = 0; m < NF; ++m)
#pragma unroll
            for (int i = 0; i < R; ++i) x[m * XS + i * PE] = c[m][i];
          cta_sync<BLOCK>();
        }
        volume<N, EQ, D, P, O::INA, O::INB>(sX + le, sH + le, vops, rho, f_in, sgn, acc);
        cta_sync<BLOCK>();         // the state's slots are free
      }
#pragma unroll 1
      for (int o0 = 0; o0 < NFP; o0 += CH) {
        load_faces(o0);
        cta_sync<BLOCK>();
        block_product<NA, D, P, PE, FS>(sX + f_out * FS + rho * CH * PE + le, lops + o0 * P,
                                        NFP - o0 < CH ? NFP - o0 : CH, acc);
        cta_sync<BLOCK>();         // every warp has read its inputs
      }
      [[maybe_unused]] const double post = grp == 0 ? a.k[4] : a.k[5];  // 1/eps, 1/mu
#pragma unroll
      for (int m = 0; m < NA; ++m)
#pragma unroll
        for (int i = 0; i < D; ++i)
          sX[(f_out + m) * XS + (slot0 + i) * PE + le] =
              EQ == DG_MAXWELL ? acc[m][i] * post : acc[m][i];
    };
    using IA = std::integral_constant<int, B::DA>;
    using IB = std::integral_constant<int, B::DB>;
    using RA = std::integral_constant<int, O::RA>;
    using RB = std::integral_constant<int, O::RB>;
    if ((B::DA != B::DB || O::RA != O::RB) && rho == 0)
      part(IA{}, RA{}, 0, ops + O::LIFT);
    else
      part(IB{}, RB{}, rho == 0 ? 0 : B::DA + (rho - 1) * B::DB,
           ops + (rho == 0 ? O::LIFT : O::LIFTB + (rho - 1) * (NFP * O::PB)));
    __syncthreads();
    // }}}

    // {{{ back to nodes, then store or fold into the RK stage (all loads of a node
    // before its stores, which the compiler must assume to alias them)
    transform<N, PE, E, BLOCK>(sX, NF);
    __syncthreads();
    for (int rem = t; rem < ecount * NP; rem += BLOCK) {
      const int el = rem / NP;
      const double* y = sX + node_slot[rem - el * NP] * PE + el;
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
        double val = y[k * XS];
        if constexpr (STAGE)
          if (a.rhs_unscaled) a.rhs_unscaled[gidx + k * nelnp] = val;
        if (a.elem_scale) val *= scale;
        if constexpr (!STAGE) {
          a.rhs[gidx + k * nelnp] = val;
        } else {
          const double r = (a.rk_a != 0.0 ? a.rk_a * res[k] : 0.0) + a.rk_dt * val;
          a.res[gidx + k * nelnp] = r;
          a.q_out[gidx + k * nelnp] = qn[k] + a.rk_b * r;
        }
      }
    }
    __syncthreads();
    // }}}
  }
}

}  // namespace sym
}  // namespace dg
