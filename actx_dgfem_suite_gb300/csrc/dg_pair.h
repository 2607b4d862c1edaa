// Sums of doubles kept as an unevaluated pair (Knuth's two-sum, with the errors
// accumulated beside the sum), for host code that derives operators: results are
// rounded once, at the speed of double arithmetic (long double is software on Arm).
#pragma once

namespace dg {

struct Pair {
  double hi = 0.0, lo = 0.0;

  Pair() = default;
  Pair(double x) : hi(x) {}  // NOLINT: a double is a pair
  Pair& add(double sign, const Pair& b) {
    const double x = sign * b.hi;      // sign: 1, -1 or a power of two
    const double s = hi + x, t = s - hi;
    const double err = (hi - (s - t)) + (x - t);
    const double low = lo + sign * b.lo + err;
    hi = s + low;
    lo = low - (hi - s);
    return *this;
  }
};

}  // namespace dg
