// Device-side arithmetic shared by the kernels: the reference's random-number and hash
// functions restated with plain integer arithmetic, and its gain / leaf-value formulas.
// Translation units that include this file are compiled with -fmad=false so that no product
// is fused into a following add (the results are compared bit-for-bit with a CPU restatement
// compiled with -ffp-contract=off).
#pragma once
#include <cstdint>

#include "internal.h"

namespace lbk {

// First statement of a kernel that LaunchChained (internal.h) launches; nothing to wait for where it was launched otherwise.
__device__ inline void AfterTheKernelBefore() { asm volatile("griddepcontrol.wait;\n" ::: "memory"); }

// Stores a fault code into the context's status word (mapped host memory).
__device__ inline void ReportFault(int* status, int code)
{
  *reinterpret_cast<volatile int*>(status) = code;
  __threadfence_system();
}

// x mod (2^31 - 1) for x < 2^62: the two 31-bit halves add up to the same residue (2^31 is 1 modulo the
// Mersenne prime), twice, and one subtraction is left.
__host__ __device__ inline uint32_t ModMersenne31(unsigned long long x)
{
  x = (x & 2147483647ull) + (x >> 31);
  uint32_t r = static_cast<uint32_t>(x & 2147483647ull) + static_cast<uint32_t>(x >> 31);
  return r >= 2147483647u ? r - 2147483647u : r;
}

// thrust::default_random_engine (minstd_rand): x <- 48271 x mod (2^31-1); a seed congruent to 0
// becomes 1; the seed argument is first converted to the engine's 32-bit unsigned state type.
struct MinStd {
  uint32_t x;
  __host__ __device__ explicit MinStd(uint32_t s)
  {
    uint32_t r = (s & 2147483647u) + (s >> 31);
    if (r >= 2147483647u) r -= 2147483647u;
    x = r == 0 ? 1u : r;
  }
  // (the product is below 2^47: one fold and one subtraction are enough)
  __host__ __device__ uint32_t next()
  {
    const unsigned long long p = 48271ull * x;
    x = static_cast<uint32_t>(p & 2147483647ull) + static_cast<uint32_t>(p >> 31);
    if (x >= 2147483647u) x -= 2147483647u;
    return x;
  }
  __host__ __device__ void discard(unsigned long long z)
  {
    unsigned long long mult = 48271ull, mult_z = 1ull;
    while (z > 0) {
      if (z & 1ull) mult_z = ModMersenne31(mult_z * mult);
      z >>= 1;
      mult = ModMersenne31(mult * mult);
    }
    x = ModMersenne31(mult_z * x);
  }
  // thrust::uniform_real_distribution<double>(a,b)
  __host__ __device__ double uniform_real(double a, double b)
  {
    double r = static_cast<double>(next() - 1u);
    r /= 2147483646.0;
    return (r * (b - a)) + a;
  }
  // uniform_real(0, 1) < r, for 0 <= r < 1.  The quotient is only formed when the product with the rounded
  // reciprocal (off by less than 4e-16) is too close to r to tell.  The draw becomes a float64 as the low bits of 2^52.
  __device__ bool uniform_below(double r)
  {
    const double n = __hiloint2double(0x43300000, static_cast<int>(next() - 1u)) - 4503599627370496.0;
    const double d = __fma_rn(n, 1.0 / 2147483646.0, -r);
    if (fabs(d) > 1e-14) return d < 0.0;
    return n / 2147483646.0 < r;
  }
  // thrust::uniform_int_distribution<int64_t>(a,b): truncated real draw from [a, b+1)
  __host__ __device__ long long uniform_int(long long a, long long b)
  {
    return static_cast<long long>(uniform_real(static_cast<double>(a), static_cast<double>(b) + 1.0));
  }
};

// MurmurHash3 fmix64 on a signed value and boost-style hash_combine (reference:
// build_tree.cu:143-165).  Right shifts are arithmetic, multiplications and additions wrap.
__host__ __device__ inline long long Hash64(long long k)
{
  k ^= k >> 33;
  k = static_cast<long long>(static_cast<unsigned long long>(k) * 0xff51afd7ed558ccdULL);
  k ^= k >> 33;
  k = static_cast<long long>(static_cast<unsigned long long>(k) * 0xc4ceb9fe1a85ec53ULL);
  k ^= k >> 33;
  return k;
}
__host__ __device__ inline long long HashCombine1(long long seed, long long v)
{
  unsigned long long add = static_cast<unsigned long long>(Hash64(v)) + 0x9e3779b9ULL +
                           (static_cast<unsigned long long>(seed) << 6) +
                           static_cast<unsigned long long>(seed >> 2);
  return seed ^ static_cast<long long>(add);
}
__host__ __device__ inline long long HashCombine(long long seed, long long a, long long b)
{
  return HashCombine1(HashCombine1(seed, a), b);
}

// Stochastic rounding of one (g,h) pair (reference: QuantiseStochasticRounding,
// build_tree.cu:112-129): first uniform draw for the gradient, second for the hessian.
__device__ inline int2 QuantisePair(double g, double h, const QuantParams& qp, long long seed)
{
  MinStd eng(static_cast<uint32_t>(static_cast<unsigned long long>(seed)));
  const double sg = g * qp.scale_g;
  const double sh = h * qp.scale_h;
  // floor(v) for |v| < 2^51: v + 1.5 * 2^52 rounded down, whose low word is the whole number itself.  Additions of full
  // rate instead of conversions of a quarter of it (100M rows: 804 -> 615 us).
  constexpr double kWhole = 6755399441055744.0;
  const double wg = __dadd_rd(sg, kWhole), wh = __dadd_rd(sh, kWhole);
  const bool plain = fabs(sg) < 2251799813685248.0 && fabs(sh) < 2251799813685248.0;  // (else a scale or a value is not finite)
  const double fg  = plain ? wg - kWhole : floor(sg);
  const double fh  = plain ? wh - kWhole : floor(sh);
  const double rg  = sg - fg;
  const double rh  = sh - fh;
  const bool up_g  = eng.uniform_below(rg);
  const bool up_h  = eng.uniform_below(rh);
  if (plain) return make_int2(__double2loint(wg) + (up_g ? 1 : 0), __double2loint(wh) + (up_h ? 1 : 0));
  const long long qg = static_cast<long long>(fg + static_cast<double>(up_g));
  const long long qh = static_cast<long long>(fh + static_cast<double>(up_h));
  return make_int2(static_cast<int>(qg), static_cast<int>(qh));
}

__device__ inline GPairF64 Dequantise(GPairI64 v, const QuantParams& qp)
{
  GPairF64 r;
  r.grad = static_cast<double>(v.grad) * qp.inv_g;
  r.hess = static_cast<double>(v.hess) * qp.inv_h;
  return r;
}

// reference: build_tree.h:106-152
__device__ inline double LeafGain(GPairF64 s, double l1, double reg)
{
  double z = 0.0;
  if (s.grad > l1) {
    z = s.grad - l1;
  } else if (s.grad < -l1) {
    z = s.grad + l1;
  }
  return (z * z) / (s.hess + reg);
}
__device__ inline double CalculateGain(GPairF64 l, GPairF64 r, GPairF64 p, double l1, double l2, double msg)
{
  const double reg = fmax(1e-5, l2);
  return (0.5 * (LeafGain(l, l1, reg) + LeafGain(r, l1, reg) - LeafGain(p, l1, reg))) - msg;
}
__device__ inline double CalculateLeafValue(double G, double H, double l1, double l2)
{
  double z = 0.0;
  if (G > l1) {
    z = G - l1;
  } else if (G < -l1) {
    z = G + l1;
  }
  return -z / (H + l2);
}

__device__ inline GPairI64 LoadPair(const GPairI64* p)
{
  const longlong2 v = *reinterpret_cast<const longlong2*>(p);
  return GPairI64{v.x, v.y};
}
__device__ inline void StorePair(GPairI64* p, GPairI64 v)
{
  *reinterpret_cast<longlong2*>(p) = make_longlong2(v.grad, v.hess);
}
__device__ inline void StorePair(GPairF64* p, GPairF64 v)
{
  *reinterpret_cast<double2*>(p) = make_double2(v.grad, v.hess);
}
// 16-byte loads that go to L2 / the owning GPU every time (no L1 copy): for memory that another
// GPU or an earlier level wrote
__device__ inline GPairI64 LoadPairStreaming(const GPairI64* p)
{
  const longlong2 v = __ldcg(reinterpret_cast<const longlong2*>(p));
  return GPairI64{v.x, v.y};
}
__device__ inline GPairF64 LoadPairStreaming(const GPairF64* p)
{
  const double2 v = __ldcg(reinterpret_cast<const double2*>(p));
  return GPairF64{v.x, v.y};
}

// Which child of a split node is built, the other one being derived from the parent: the one with the
// smaller quantised hessian of output 0, ties to the right (reference: build_tree.h:80-104).
__device__ inline bool SmallerChildIsLeft(const GPairI64* node_sums, int K, int left_child)
{
  return node_sums[static_cast<int64_t>(left_child) * K].hess < node_sums[static_cast<int64_t>(left_child + 1) * K].hess;
}

}  // namespace lbk
