// Operator blocks of the symmetry-adapted kernels (layout: sym::Ops in
// dg_sym.cuh), derived on the host from the caller's derivative matrices and
// LIFT.
#include <cmath>
#include <cstring>
#include <type_traits>
#include <vector>

#include "dg_launch.h"
#include "dg_pair.h"
#include "dg_sym.cuh"

namespace dg {
namespace {

// vertex permutations id, (01)(23), (02)(13), (03)(12)
constexpr int kGroup[4][4] = {{0, 1, 2, 3}, {1, 0, 3, 2}, {2, 3, 0, 1}, {3, 2, 1, 0}};
// value of part r's functions under group element g
constexpr int kChar[4][4] = {{1, 1, 1, 1}, {1, 1, -1, -1}, {1, -1, 1, -1}, {1, -1, -1, 1}};
// Operators whose entries outside the block pattern exceed this fraction of
// the largest entry are not symmetric and keep the general kernels.  FP64
// operators assembled in FP64 stay below 4e-15 at orders 1-4.
constexpr double kAsymmetry = 5e-14;

struct Vec {  // one symmetric combination of nodes or face points
  int n = 0;
  int idx[4];
  int sign[4];
};

Vec combo(const int* orbit, int n, int part) {
  Vec v;
  v.n = n;
  for (int k = 0; k < n; ++k) {
    v.idx[k] = orbit[k];
    v.sign[k] = n == 4 ? kChar[part][k] : (k == 0 || part == 0 ? 1 : -1);
  }
  return v;
}

double dot(const double* a, const double* b, int n) {  // rounded once
  Pair s;
  for (int k = 0; k < n; ++k) {
    const double p = a[k] * b[k];
    s.add(1.0, p).add(1.0, std::fma(a[k], b[k], -p));
  }
  return s.hi;
}

// Orthonormal basis q (rank x n) of the range of the columns x (cols x n):
// Gram-Schmidt with the largest remaining column next, each orthogonalised twice.
// False unless the columns have that rank to rounding.
bool range_basis(std::vector<double> x, int cols, int n, int rank, double* q) {
  auto inner = [n](const double* a, const double* b) {
    double s = 0.0;
    for (int k = 0; k < n; ++k) s = std::fma(a[k], b[k], s);
    return s;
  };
  auto norm = [&](int c) { return std::sqrt(inner(&x[c * n], &x[c * n])); };
  double big = 0.0;
  for (int c = 0; c < cols; ++c) big = std::fmax(big, norm(c));
  for (int r = 0; r <= rank; ++r) {
    int best = 0;
    double len = -1.0;
    for (int c = 0; c < cols; ++c) {
      const double l = norm(c);
      if (l > len) {
        len = l;
        best = c;
      }
    }
    if (r == rank) return len <= 1e-13 * big;
    if (!(len > 1e-6 * big)) return false;
    double* v = q + r * n;
    std::memcpy(v, &x[best * n], n * sizeof(double));
    for (int pass = 0; pass < 2; ++pass) {
      for (int p = 0; p < r; ++p) {
        const double h = inner(q + p * n, v);
        for (int k = 0; k < n; ++k) v[k] = std::fma(-h, q[p * n + k], v[k]);
      }
      const double l = std::sqrt(inner(v, v));
      for (int k = 0; k < n; ++k) v[k] /= l;
    }
    for (int c = 0; c < cols; ++c)
      for (int pass = 0; pass < 2; ++pass) {
        const double h = inner(v, &x[c * n]);
        for (int k = 0; k < n; ++k) x[c * n + k] = std::fma(-h, v[k], x[c * n + k]);
      }
  }
  return false;
}

// ADJ: the blocks of the transposed operators (sym::AdjOps); RED: derivatives
// through coefficients of degree N - 1 (sym::Ops); `into_a`: which order-1 blocks
// may be non-zero (those into part A, else those from it).
template <int N, bool ADJ, int RED>
int pack(const double* diff, const double* lift, const int32_t* face_nodes, bool into_a,
         unsigned char* out, int out_bytes) {
  using B = sym::Basis<N>;
  using F = sym::Ops<N, RED>;
  using O = std::conditional_t<ADJ, sym::AdjOps<N, RED>, F>;
  constexpr int NP = B::NP, NFP = B::NFP, NFPT = B::NFPT;
  if (!out) return O::SIZE;
  if (out_bytes < O::SIZE) return -1;

  // {{{ action of the group on nodes (barycentric multi-indices, first index
  // fastest) and on face points
  int alpha[NP][4], perm[4][NP];
  {
    int n = 0;
    for (int k = 0; k <= N; ++k)
      for (int j = 0; j <= N - k; ++j)
        for (int i = 0; i <= N - k - j; ++i, ++n) {
          alpha[n][0] = N - i - j - k;
          alpha[n][1] = i;
          alpha[n][2] = j;
          alpha[n][3] = k;
        }
  }
  for (int g = 0; g < 4; ++g)
    for (int n = 0; n < NP; ++n)
      for (int m = 0; m < NP; ++m) {
        bool same = true;
        for (int v = 0; v < 4; ++v) same = same && alpha[m][v] == alpha[n][kGroup[g][v]];
        if (same) perm[g][n] = m;
      }
  int fperm[4][NFPT];
  for (int g = 0; g < 4; ++g)
    for (int f = 0; f < 4; ++f) {
      int target = -1;
      for (int f2 = 0; f2 < 4 && target < 0; ++f2) {
        bool all = true;
        for (int j = 0; j < NFP; ++j) {
          bool found = false;
          for (int j2 = 0; j2 < NFP; ++j2)
            found = found || face_nodes[f2 * NFP + j2] == perm[g][face_nodes[f * NFP + j]];
          all = all && found;
        }
        if (all) target = f2;
      }
      if (target < 0 || (g > 0 && target == f)) return -1;  // not the faces of a tetrahedron
      for (int j = 0; j < NFP; ++j) {
        int hit = -1;
        for (int j2 = 0; j2 < NFP; ++j2)
          if (face_nodes[target * NFP + j2] == perm[g][face_nodes[f * NFP + j]]) hit = j2;
        fperm[g][f * NFP + j] = target * NFP + hit;
      }
    }
  // a face that lists a node twice has no such permutation: its points would be left
  // without a slot
  for (int g = 0; g < 4; ++g) {
    bool seen[NFPT] = {};
    for (int k = 0; k < NFPT; ++k) {
      if (seen[fperm[g][k]]) return -1;
      seen[fperm[g][k]] = true;
    }
  }
  // }}}

  // {{{ orbits, slots and the symmetric combinations
  Vec node[NP];                     // by slot
  int part_of[NP], node_slot[NP];
  {
    bool seen[NP] = {};
    int nfull = 0, npair[4] = {}, nsingle = 0;
    for (int n = 0; n < NP; ++n) {
      if (seen[n]) continue;
      int orbit[4];
      for (int g = 0; g < 4; ++g) orbit[g] = perm[g][n];
      for (int g = 0; g < 4; ++g) seen[orbit[g]] = true;
      int fix = 0, nfix = 0;
      for (int g = 1; g < 4; ++g)
        if (orbit[g] == n) fix = g, ++nfix;
      if (nfix == 0) {
        for (int r = 0; r < 4; ++r) {
          const int slot = r == 0 ? nfull : B::DA + (r - 1) * B::DB + nfull;
          node[slot] = combo(orbit, 4, r);
          part_of[slot] = r;
          node_slot[orbit[r]] = slot;
        }
        ++nfull;
      } else if (nfix == 1) {
        const int pair[2] = {n, orbit[fix == 1 ? 2 : 1]};
        const int sa = B::NO4 + fix - 1, sb = B::DA + (fix - 1) * B::DB + B::NO4;
        node[sa] = combo(pair, 2, 0);
        node[sb] = combo(pair, 2, 1);
        part_of[sa] = 0;
        part_of[sb] = fix;
        node_slot[pair[0]] = sa;
        node_slot[pair[1]] = sb;
        ++npair[fix];
      } else {
        node[B::DA - 1] = combo(orbit, 1, 0);
        part_of[B::DA - 1] = 0;
        node_slot[n] = B::DA - 1;
        ++nsingle;
      }
    }
    if (nfull != B::NO4 || npair[1] != B::NPR || npair[2] != B::NPR || npair[3] != B::NPR ||
        nsingle != B::NSG)
      return -1;
  }
  // the combinations that each node enters, and with which sign
  int nslots[NP] = {}, slots[NP][4], signs[NP][4];
  for (int i = 0; i < NP; ++i)
    for (int a = 0; a < node[i].n; ++a) {
      const int n = node[i].idx[a];
      slots[n][nslots[n]] = i;
      signs[n][nslots[n]++] = node[i].sign[a];
    }
  Vec face[NFPT];
  int face_slot[NFPT];
  for (int o = 0; o < NFP; ++o) {   // orbit o starts at point o of face 0
    int orbit[4];
    for (int g = 0; g < 4; ++g) orbit[g] = fperm[g][o];
    for (int r = 0; r < 4; ++r) {
      face[r * NFP + o] = combo(orbit, 4, r);
      face_slot[orbit[r]] = r * NFP + o;
    }
  }
  // }}}

  // an operator of `cols` columns in the combinations' basis (outputs by node
  // slot, inputs by slot of `in`), normalised for plain sums on both sides
  std::vector<Pair> half;
  std::vector<double> full;
  auto to_basis = [&](const Vec* in, int cols, auto at) {
    half.assign((size_t)NP * cols, Pair());
    full.assign((size_t)NP * cols, 0.0);
    for (int n = 0; n < NP; ++n)
      for (int c = 0; c < cols; ++c) {
        const Pair x = at(n, c);
        for (int k = 0; k < nslots[n]; ++k)
          half[(size_t)slots[n][k] * cols + c].add(signs[n][k], x);
      }
    for (int i = 0; i < NP; ++i)
      for (int c = 0; c < cols; ++c) {
        Pair s;
        for (int b = 0; b < in[c].n; ++b)
          s.add(in[c].sign[b], half[(size_t)i * cols + in[c].idx[b]]);
        full[(size_t)i * cols + c] = s.hi / (node[i].n * in[c].n);  // powers of two
      }
  };
  // whether the entries outside the pattern vanish to rounding
  auto symmetric = [&](int cols, auto inside) {
    double big = 0.0, off = 0.0;
    for (int i = 0; i < NP; ++i)
      for (int c = 0; c < cols; ++c) {
        const double x = std::fabs(full[(size_t)i * cols + c]);
        if (!std::isfinite(x)) return false;
        double& m = inside(i, c) ? big : off;
        if (x > m) m = x;
      }
    return off <= kAsymmetry * big;
  };
  auto slot0 = [](int r) { return r == 0 ? 0 : B::DA + (r - 1) * B::DB; };
  auto dim = [](int r) { return r == 0 ? B::DA : B::DB; };

  std::memset(out, 0, O::SIZE);
  double* ops = reinterpret_cast<double*>(out);
  std::vector<double> block[4][3];  // of part r and direction k + 1, by columns
  for (int k = 1; k < 4; ++k) {
    // D'_k = -1/2 (D_k - D_other - D_other')
    to_basis(node, NP, [&](int i, int j) {
      Pair s;
      for (int r = 0; r < 3; ++r)
        s.add(r == k - 1 ? -0.5 : 0.5,
              diff[(size_t)(r * NP + (ADJ ? j : i)) * NP + (ADJ ? i : j)]);
      return s;
    });
    if (!symmetric(NP, [&](int i, int j) {
          const int ri = part_of[i], rj = part_of[j];
          return (ri ^ rj) == k && (N != 1 || (into_a ? ri : rj) == 0);
        }))
      return -1;
    for (int r = 0; r < 4; ++r)
      for (int j = 0; j < dim(r ^ k); ++j)
        for (int i = 0; i < dim(r); ++i)
          block[r][k - 1].push_back(full[(size_t)(slot0(r) + i) * NP + slot0(r ^ k) + j]);
  }
  auto rank = [](int r) { return r == 0 ? F::RA : F::RB; };
  std::vector<double> q[4];  // basis of the space of degree N - 1, per part
  for (int r = 0; RED && r < 4; ++r) {
    const int d = dim(r);
    q[r].resize((size_t)rank(r) * d);
    std::vector<double> all;  // columns of the blocks into r, or rows of those from r
    for (int k = 0; k < 3; ++k) {
      const int s = r ^ (k + 1), ds = dim(s);
      if (RED == sym::RED_OUT)
        all.insert(all.end(), block[r][k].begin(), block[r][k].end());
      else
        for (int i = 0; i < ds; ++i)
          for (int j = 0; j < d; ++j) all.push_back(block[s][k][(size_t)j * ds + i]);
    }
    if (!range_basis(all, (int)all.size() / d, d, rank(r), q[r].data())) return -1;
    double* dst = ops + F::extra(r);
    for (int j = 0; j < rank(r); ++j)
      for (int i = 0; i < d; ++i)
        dst[RED == sym::RED_OUT ? j * (r == 0 ? F::PA : F::PB) + i
                                : i * (r == 0 ? F::PRA : F::PRB) + j] = q[r][(size_t)j * d + i];
  }
  for (int r = 0; r < 4; ++r) {
    double* dst = ops + F::volume(r);
    for (int k = 0; k < 3; ++k) {
      const int s = r ^ (k + 1), d = dim(r), ds = dim(s);
      const std::vector<double>& b = block[r][k];
      for (int j = 0; j < (s == 0 ? F::INA : F::INB); ++j, dst += r == 0 ? F::POA : F::POB)
        for (int i = 0; i < (r == 0 ? F::OUTA : F::OUTB); ++i) {
          if (RED == sym::RED_OUT) {
            dst[i] = dot(&q[r][(size_t)i * d], &b[(size_t)j * d], d);
          } else if (RED == sym::RED_IN) {
            double row[B::DA];
            for (int c = 0; c < ds; ++c) row[c] = b[(size_t)c * d + i];
            dst[i] = dot(&q[s][(size_t)j * ds], row, ds);
          } else {
            dst[i] = b[(size_t)j * d + i];
          }
        }
    }
  }
  to_basis(face, NFPT,
           [&](int i, int fj) { return Pair(lift[(size_t)i * NFPT + fj]); });
  if (!symmetric(NFPT, [&](int i, int c) { return part_of[i] == c / NFP; })) return -1;
  for (int r = 0; r < 4; ++r)
    for (int o = 0; o < NFP; ++o)
      for (int i = 0; i < dim(r); ++i) {
        const double x = full[(size_t)(slot0(r) + i) * NFPT + r * NFP + o];
        if constexpr (ADJ)
          ops[O::LIFT + (o / O::CH) * O::CHUNK + (slot0(r) + i) * O::PC + o % O::CH] = x;
        else
          ops[(r == 0 ? F::LIFT : F::LIFTB + (r - 1) * NFP * F::PB) +
              o * (r == 0 ? F::PA : F::PB) + i] = x;
      }
  int32_t* ns = reinterpret_cast<int32_t*>(out + O::NODE_SLOT);
  int32_t* fp = reinterpret_cast<int32_t*>(out + O::FACE_POINT);
  int32_t* sn = reinterpret_cast<int32_t*>(out + O::SLOT_NODE);
  for (int n = 0; n < NP; ++n) ns[n] = node_slot[n];
  for (int n = 0; n < NP; ++n) sn[node_slot[n]] = n;
  for (int fj = 0; fj < NFPT; ++fj) fp[face_slot[fj]] = fj;
  return O::SIZE;
}

}  // namespace

// RED_OUT for strong and transposed weak derivatives, RED_IN for weak ones
template <bool ADJ, bool INTO_A>
static int pack_order(int order, bool reduce, const double* diff, const double* lift,
                      const int32_t* face_nodes, unsigned char* out, int out_bytes) {
  constexpr int RED = INTO_A ? sym::RED_OUT : sym::RED_IN;
  switch (reduce ? -order : order) {
    case 1:
    case -1: return pack<1, ADJ, 0>(diff, lift, face_nodes, INTO_A, out, out_bytes);
    case 2: return pack<2, ADJ, 0>(diff, lift, face_nodes, INTO_A, out, out_bytes);
    case 3: return pack<3, ADJ, 0>(diff, lift, face_nodes, INTO_A, out, out_bytes);
    case 4: return pack<4, ADJ, 0>(diff, lift, face_nodes, INTO_A, out, out_bytes);
    case -2: return pack<2, ADJ, RED>(diff, lift, face_nodes, INTO_A, out, out_bytes);
    case -3: return pack<3, ADJ, RED>(diff, lift, face_nodes, INTO_A, out, out_bytes);
    case -4: return pack<4, ADJ, RED>(diff, lift, face_nodes, INTO_A, out, out_bytes);
    default: return -1;
  }
}

int pack_sym_ops(int order, const double* diff, const double* lift, const int32_t* face_nodes,
                 bool strong, bool reduce, unsigned char* out, int out_bytes) {
  return (strong ? pack_order<false, true> : pack_order<false, false>)(
      order, reduce, diff, lift, face_nodes, out, out_bytes);
}

int pack_sym_adj_ops(int order, const double* weak, const double* lift,
                     const int32_t* face_nodes, bool reduce, unsigned char* out, int out_bytes) {
  return pack_order<true, true>(order, reduce, weak, lift, face_nodes, out, out_bytes);
}

}  // namespace dg
