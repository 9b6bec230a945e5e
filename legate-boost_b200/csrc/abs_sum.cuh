// The sums of |g| and |h| that the quantiser's scale comes from, in a fixed order (the reference leaves it
// to thrust::reduce): blocks of 4096 elements; thread t of 256 adds elements t, t+256, ... in order; groups
// of 32 threads fold with offsets 16,8,4,2,1; the 8 group sums are added left to right; block sums are
// reduced the same way until one value is left.  The CPU oracle uses the same order.
#pragma once
#include "device_utils.cuh"
#include "objective.cuh"

namespace lbk {

constexpr int kSumThreads = 256;
constexpr int kSumItems   = 16;
constexpr int kSumBlock   = kSumThreads * kSumItems;  // 4096

// The second half of a block's sum: groups of 32 threads fold into s_sum (16 values per 256 threads), and,
// after a barrier, one thread adds the 8 group sums left to right.
__device__ inline void FoldAbsSums(double sg, double sh, int tid, double* s_sum)
{
#pragma unroll
  for (int off = 16; off >= 1; off >>= 1) {
    sg += __shfl_down_sync(0xffffffffu, sg, off);
    sh += __shfl_down_sync(0xffffffffu, sh, off);
  }
  if ((tid & 31) == 0) {
    s_sum[tid >> 5]                      = sg;
    s_sum[kSumThreads / 32 + (tid >> 5)] = sh;
  }
}
__device__ inline void JoinAbsSums(const double* s_sum, double& tg, double& th)
{
  tg = s_sum[0];
  th = s_sum[kSumThreads / 32];
#pragma unroll
  for (int w = 1; w < kSumThreads / 32; ++w) {
    tg += s_sum[w];
    th += s_sum[kSumThreads / 32 + w];
  }
}

// Sums of block `block`, returned to thread 0 of the 256 (`tid` = 0..255 within the group; all threads of the
// CTA call it, several groups may do so at once).  kFirst: |g|, |h| of the strided [n / K, K] inputs, else the
// partial sums themselves.  s_sum: shared, 16 values per group.
template <bool kFirst>
__device__ inline void AbsSumPartial(const double* g, const double* h, int64_t ldg, const GradientForm& form, int K, int64_t n,
                                     int64_t block, int tid, double* s_sum, double& tg, double& th)
{
  const int64_t base = block * kSumBlock;
  double sg = 0.0, sh = 0.0;
#pragma unroll
  for (int j = 0; j < kSumItems; ++j) {
    const int64_t idx = base + static_cast<int64_t>(j) * kSumThreads + tid;
    double vg = 0.0, vh = 0.0;
    if (idx < n) {
      if (kFirst) {
        const int64_t row = K == 1 ? idx : idx / K;
        const int k       = static_cast<int>(idx - row * K);
        const double2 v   = GradientAt(g, h, row * ldg + k, form);
        vg                = fabs(v.x);
        vh                = fabs(v.y);
      } else {
        vg = g[idx];
        vh = h[idx];
      }
    }
    sg += vg;
    sh += vh;
  }
  FoldAbsSums(sg, sh, tid, s_sum);
  __syncthreads();
  tg = th = 0.0;
  if (tid == 0) JoinAbsSums(s_sum, tg, th);
}

template <bool kFirst>
__device__ inline void AbsSumBlock(const double* g, const double* h, int64_t ldg, const GradientForm& form, int K, int64_t n,
                                   int64_t block, int tid, double* s_sum, double* out_g, double* out_h)
{
  double tg, th;
  AbsSumPartial<kFirst>(g, h, ldg, form, K, n, block, tid, s_sum, tg, th);
  if (tid == 0) {
    *out_g = tg;
    *out_h = th;
  }
}

// scale = INT32_MAX / (max over ranks of the local sum), 1 if that sum is 0 (reference: build_tree.cu:69-104)
__device__ inline QuantParams MakeScale(double sum_g, double sum_h)
{
  const double max_int = 2147483647.0;
  QuantParams p;
  p.scale_g = sum_g == 0 ? 1.0 : max_int / sum_g;
  p.scale_h = sum_h == 0 ? 1.0 : max_int / sum_h;
  p.inv_g   = 1.0 / p.scale_g;
  p.inv_h   = 1.0 / p.scale_h;
  return p;
}

}  // namespace lbk
