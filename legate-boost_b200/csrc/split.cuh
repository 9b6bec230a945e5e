// Split candidates, their total order and the gain of a bin (reference behaviour: see split.cu).
#pragma once
#include "device_utils.cuh"
#include "division.cuh"

namespace lbk {

struct Cand {
  double gain;
  int bin;
  int feature;
};
__device__ inline bool Better(const Cand& a, const Cand& b)
{
  if (a.gain > b.gain) return true;
  if (a.gain < b.gain) return false;
  if (a.bin < 0 || b.bin < 0) return b.bin < 0 && a.bin >= 0;
  const int ta = a.bin & 511, tb = b.bin & 511;
  if (ta != tb) return ta > tb;
  return a.bin < b.bin;
}

// The largest of a warp's values (all not negative), in every lane: their bit patterns are ordered as the values.
__device__ inline double WarpMax(double v)
{
  const unsigned hi = __reduce_max_sync(0xffffffffu, static_cast<unsigned>(__double2hiint(v)));
  const unsigned lo = __reduce_max_sync(0xffffffffu, static_cast<unsigned>(__double2hiint(v)) == hi ? static_cast<unsigned>(__double2loint(v)) : 0u);
  return __hiloint2double(static_cast<int>(hi), static_cast<int>(lo));
}

// The bin of the warp's best candidate (a bin and a gain per lane, gain 0 = none), or -1.
__device__ inline int WarpBest(double gain, int bin)
{
  const double top = WarpMax(gain);
  if (top == 0.0) return -1;
  const unsigned holders = __ballot_sync(0xffffffffu, gain == top);
  Cand best{top, __shfl_sync(0xffffffffu, bin, __ffs(holders) - 1), 0};
  for (unsigned rest = holders & (holders - 1u); rest != 0u; rest &= rest - 1u) {  // equal gains: the order of the bins decides
    const Cand o{top, __shfl_sync(0xffffffffu, bin, __ffs(rest) - 1), 0};
    if (Better(o, best)) best = o;
  }
  return best.bin;
}

// What the gains of one output need of a node: its sums as whole numbers in float64 and its own gain.
struct NodeTerms {
  double g, h, gain;
};

// (double)v for |v| < 2^51, exact: adding 1.5 * 2^52 to the bit pattern of the integer makes a float64 whose
// value is that constant plus v.  Two instructions of full rate instead of a conversion of a sixteenth of it.
__device__ inline double WholeToDouble(long long v)
{
  return __longlong_as_double(v + 0x4338000000000000ll) - 6755399441055744.0;
}

__device__ inline NodeTerms TermsOf(GPairI64 sum, const QuantParams& qp, double l1, double reg)
{
  NodeTerms t;
  t.g    = WholeToDouble(sum.grad);
  t.h    = WholeToDouble(sum.hess);
  t.gain = LeafGain(GPairF64{t.g * qp.inv_g, t.h * qp.inv_h}, l1, reg);
  return t;
}

// LeafGain's numerator
__device__ inline double LeafNumerator(double g, double l1)
{
  const double z = g > l1 ? g - l1 : g < -l1 ? g + l1 : 0.0;
  return z * z;
}

// Without an l1 term, and with scales and a regulariser of moderate size, the numerator is a square and every division of a gain
// is plain whatever the bin (DivisionIsPlain; sums are whole numbers below 2^52, so a square is zero or at least inv_g^2, a
// divisor at least reg), but for a divisor whose mantissa is all ones, of which the low word is looked at.  Of the 408
// instructions a warp took for 32 bins of an output of two nodes the tests of the general form were a fifth.
__device__ inline bool GainsArePlain(const QuantParams& qp, double l1, double reg)
{
  return l1 == 0.0 && qp.inv_g >= 0x1p-250 && qp.inv_g < 0x1p198 && qp.inv_h >= 0.0 && qp.inv_h < 0x1p340 && reg >= 0x1p-400 && reg < 0x1p400;
}
__device__ inline bool LowWordOnes(double d) { return __double2loint(d) == -1; }

// The gain of one output at a lane's bin, added to `gain` where `ok`; returns whether both sides have a positive hessian
// too (sums are below 2^51, so their differences are exact in float64).  All lanes of a warp call it.  plain: GainsArePlain.
__device__ inline unsigned AddGain(const GPairI64& left, unsigned ok, const NodeTerms& n, const QuantParams& qp, double l1,
                                   double reg, double msg, bool plain, double& gain)
{
  const double lg = WholeToDouble(left.grad), lh = WholeToDouble(left.hess);
  const double rg = n.g - lg, rh = n.h - lh;
  if (lh <= 0.0 || rh <= 0.0) ok = 0u;
  double a = lg * qp.inv_g, b = rg * qp.inv_g;
  const double da = lh * qp.inv_h + reg, db = rh * qp.inv_h + reg;
  bool all_plain;
  if (plain) {
    a         = a * a;
    b         = b * b;
    all_plain = !__any_sync(0xffffffffu, LowWordOnes(da) || LowWordOnes(db));
  } else {
    a         = LeafNumerator(a, l1);
    b         = LeafNumerator(b, l1);
    all_plain = __all_sync(0xffffffffu, ok == 0u || (DivisionIsPlain(a, da) && DivisionIsPlain(b, db)));
  }
  if (all_plain) {
    a = DividePlain(a, da);
    b = DividePlain(b, db);
  } else if (ok != 0u) {
    a = a / da;
    b = b / db;
  }
  gain += (0.5 * (a + b - n.gain)) - msg;
  return ok;
}

// The same for a node and its sibling: the four divisions of a lane are under way together (one after the other's vote they
// take twice as long, and a lone chain is what small levels wait for).
__device__ inline void AddGains(const GPairI64& left_a, unsigned& ok_a, const NodeTerms& a, double& gain_a, const GPairI64& left_b, unsigned& ok_b,
                                const NodeTerms& b, double& gain_b, const QuantParams& qp, double l1, double reg, double msg, bool plain)
{
  const double alg = WholeToDouble(left_a.grad), alh = WholeToDouble(left_a.hess), arg = a.g - alg, arh = a.h - alh;
  const double blg = WholeToDouble(left_b.grad), blh = WholeToDouble(left_b.hess), brg = b.g - blg, brh = b.h - blh;
  if (alh <= 0.0 || arh <= 0.0) ok_a = 0u;
  if (blh <= 0.0 || brh <= 0.0) ok_b = 0u;
  double n0 = alg * qp.inv_g, n1 = arg * qp.inv_g, n2 = blg * qp.inv_g, n3 = brg * qp.inv_g;
  const double d0 = alh * qp.inv_h + reg, d1 = arh * qp.inv_h + reg, d2 = blh * qp.inv_h + reg, d3 = brh * qp.inv_h + reg;
  bool all_plain;
  if (plain) {
    n0        = n0 * n0;
    n1        = n1 * n1;
    n2        = n2 * n2;
    n3        = n3 * n3;
    all_plain = !__any_sync(0xffffffffu, LowWordOnes(d0) || LowWordOnes(d1) || LowWordOnes(d2) || LowWordOnes(d3));
  } else {
    n0        = LeafNumerator(n0, l1);
    n1        = LeafNumerator(n1, l1);
    n2        = LeafNumerator(n2, l1);
    n3        = LeafNumerator(n3, l1);
    all_plain = __all_sync(0xffffffffu, (ok_a == 0u || (DivisionIsPlain(n0, d0) && DivisionIsPlain(n1, d1))) &&
                                          (ok_b == 0u || (DivisionIsPlain(n2, d2) && DivisionIsPlain(n3, d3))));
  }
  if (all_plain) {
    n0 = DividePlain(n0, d0);
    n1 = DividePlain(n1, d1);
    n2 = DividePlain(n2, d2);
    n3 = DividePlain(n3, d3);
  } else {
    if (ok_a != 0u) {
      n0 = n0 / d0;
      n1 = n1 / d1;
    }
    if (ok_b != 0u) {
      n2 = n2 / d2;
      n3 = n3 / d3;
    }
  }
  gain_a += (0.5 * (n0 + n1 - a.gain)) - msg;
  gain_b += (0.5 * (n2 + n3 - b.gain)) - msg;
}

// Leaf value and hessian of entry i = node * K + output, from the node's quantised sums; the leaf value of a node whose
// parent did not split is 0.
__device__ inline double2 FinishedNode(const TreeArrays& tree, const QuantParams& qp, int K, int64_t i, double l1, double l2)
{
  const int node   = static_cast<int>(i / K);
  const GPairF64 s = Dequantise(tree.node_sums[i], qp);
  const bool here  = node == 0 || tree.feature[(node - 1) / 2] >= 0;
  return make_double2(here ? CalculateLeafValue(s.grad, s.hess, l1, l2) : 0.0, s.hess);
}

}  // namespace lbk
