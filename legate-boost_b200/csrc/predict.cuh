// What the kernels of the ensemble predict share: packed trees, bulk copies and bounded waits, the end of a row.
#pragma once
#include "device_utils.cuh"
#include "internal.h"

namespace lbk {
namespace {

using TreePtrs = lbk_tree_ref;  // node_off: offset of the tree's first node in the packed arrays

// Bulk asynchronous copy global -> shared (the copy engine moves whole lines; nothing passes
// through the load/store pipe), completion counted in bytes on an mbarrier; a plain copy into this block only.
__device__ inline void MbarInit(unsigned bar, unsigned count)
{
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(bar), "r"(count) : "memory");
}
__device__ inline void MbarInval(unsigned bar)
{
  asm volatile("mbarrier.inval.shared::cta.b64 [%0];\n" ::"r"(bar) : "memory");
}
__device__ inline void MbarExpectTx(unsigned bar, unsigned bytes)
{
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ inline void BulkCopy(unsigned smem_dst, const void* gsrc, unsigned bytes, unsigned bar)
{
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n" ::"r"(smem_dst),
               "l"(gsrc), "r"(bytes), "r"(bar)
               : "memory");
}
__device__ inline bool MbarTryWait(unsigned bar, unsigned parity)
{
  unsigned ok;
  asm volatile(
    "{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\nselp.u32 %0, 1, 0, p;\n}\n"
    : "=r"(ok)
    : "r"(bar), "r"(parity)
    : "memory");
  return ok != 0;
}
// Bounded wait: gives up after about a second, reports through the context's status word and lets the block finish instead
// of spinning for ever.  A call with a table of trees has returned by then, so the producer warp makes the
// block's predictions NaN: they are not taken for those of the trees that it did see.
constexpr int kFaultPredictStaging = 21;
__device__ inline bool MbarWait(unsigned bar, unsigned parity, int* status, int* failed)
{
  for (unsigned spin = 0; spin < (1u << 22); ++spin) {
    if (MbarTryWait(bar, parity)) return true;
    if (spin > 64) __nanosleep(256);
  }
  ReportFault(status, kFaultPredictStaging);
  *failed = 1;
  return false;
}

__device__ inline void MbarArrive(unsigned bar)
{
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(bar) : "memory");
}
__device__ inline unsigned LdsU32(unsigned addr)
{
  unsigned v;
  asm volatile("ld.shared.b32 %0, [%1];\n" : "=r"(v) : "r"(addr));
  return v;
}
__device__ inline float LdsX(unsigned addr, float)
{
  float v;
  asm volatile("ld.shared.f32 %0, [%1];\n" : "=f"(v) : "r"(addr));
  return v;
}
__device__ inline double LdsX(unsigned addr, double)
{
  double v;
  asm volatile("ld.shared.f64 %0, [%1];\n" : "=d"(v) : "r"(addr));
  return v;
}
__device__ inline double LdsF64(unsigned addr)
{
  double v;
  asm volatile("ld.shared.f64 %0, [%1];\n" : "=d"(v) : "r"(addr));
  return v;
}

// (on a 16-byte boundary)
__device__ inline double2 LdsF64x2(unsigned addr)
{
  double2 v;
  asm volatile("ld.shared.v2.f64 {%0, %1}, [%2];\n" : "=d"(v.x), "=d"(v.y) : "r"(addr));
  return v;
}

__device__ inline void MakeSplit(float& s, double split) { s = __double2float_rd(split); }
__device__ inline void MakeSplit(double& s, double split) { s = split; }

// What is added to the sums and what becomes of them: initial prediction, then probabilities.
struct PredictOut {
  double* pred;
  int64_t ldp;
  const double* init;  // [K] or null
  int transform;       // LBK_RAW, LBK_LOGISTIC (two columns: 1 - p, p) or LBK_SOFTMAX
};

// The K raw predictions of one row -> its row of the output.  `raw` and the row may be the same.
__device__ inline void FinishRow(const double* raw, int stride, int K, double* out, int transform)
{
  if (transform == LBK_RAW) {
    for (int k = 0; k < K; ++k) out[k] = raw[k * stride];
  } else if (transform == LBK_LOGISTIC) {
    const double p = 1.0 / (1.0 + exp(-raw[0]));
    out[0] = 1.0 - p;
    out[1] = p;
  } else {
    double top = raw[0];
    for (int k = 1; k < K; ++k) top = fmax(top, raw[k * stride]);
    double sum = 0.0;
    for (int k = 0; k < K; ++k) {
      const double e = exp(raw[k * stride] - top);
      out[k]         = e;
      sum += e;
    }
    for (int k = 0; k < K; ++k) out[k] = out[k] / sum;
  }
}

}  // namespace
}  // namespace lbk
