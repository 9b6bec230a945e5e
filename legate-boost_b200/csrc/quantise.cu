// Gradient quantiser: scale from the local |g|,|h| sums, one stochastic-rounded int32 pair per
// (row, output), and the root node sums.
//
// Reference behaviour restated here:
//   GradientQuantiser ctor   src/models/tree/build_tree.cu:69-104  - scale = INT32_MAX / max over
//     ranks of the local sum of |g| (resp. |h|), 1 if that sum is 0.
//   QuantiseStochasticRounding  :112-129, hash_combine :143-165.
//   reduce_base_sums            :168-204 - node_sums[0,k] = sum of the quantised pairs.
// The reference recomputes the quantised pair of a row for every feature group on every level;
// its value depends only on (seed, global row, output), so it is computed once here.
//
// (The sums of |g| and |h|: abs_sum.cuh, made in the prologue of the tree.)
#include "device_utils.cuh"
#include "internal.h"
#include "objective.cuh"

namespace lbk {
namespace {

// Per-output block sums go to node_sums[0,k] with one 64-bit atomic pair per block and output;
// blocks walk the elements with a grid stride so that the number of atomics stays small.
// Element (row, k) = flat index row * K + k; a thread keeps one k (the grid's stride is a multiple
// of K), so the loads and stores of a warp are contiguous whatever K is.
// Bound by its instructions (the hash's multiplications, twelve float64 operations of half rate): 100M rows 615 us, of which
// HBM asks for 370; with conversions between float64 and integers 804.
__global__ void __launch_bounds__(256)
  k_quantise(const double* __restrict__ g, const double* __restrict__ h, int64_t ldg, const GradientForm form,
             int64_t row_offset, int64_t n_local, int K, long long seed, const QuantParams* __restrict__ qp_ptr,
             int2* __restrict__ gpair, GPairI64* __restrict__ root_sums, int* __restrict__ max_abs,
             int* __restrict__ hess_below_one)
{
  AfterTheKernelBefore();
  extern __shared__ unsigned long long s_sum[];  // [K][2]
  __shared__ int s_max[2];
  const QuantParams qp = *qp_ptr;
  const int tid        = threadIdx.x;
  for (int i = tid; i < 2 * K; i += blockDim.x) s_sum[i] = 0ull;
  if (tid < 2) s_max[tid] = 0;
  __syncthreads();
  const int64_t threads = static_cast<int64_t>(gridDim.x) * blockDim.x;
  const int64_t rows_per_turn = threads / K;  // >= 1: the launcher gives at least K threads
  const int64_t t = blockIdx.x * static_cast<int64_t>(blockDim.x) + tid;
  int mg = 0, mh = 0, lowest = INT32_MAX;
  if (t < rows_per_turn * K) {
    const int k = static_cast<int>(t % K);
    long long sg = 0, sh = 0;
#pragma unroll 4
    for (int64_t row = t / K; row < n_local; row += rows_per_turn) {
      const double2 v = GradientAt(g, h, row * ldg + k, form);
      const int2 q    = QuantisePair(v.x, v.y, qp, HashCombine(seed, row_offset + row, k));
      gpair[row * K + k] = q;
      sg += q.x;
      sh += q.y;
      mg = max(mg, q.x == INT32_MIN ? INT32_MAX : abs(q.x));
      mh = max(mh, q.y == INT32_MIN ? INT32_MAX : abs(q.y));
      lowest = min(lowest, q.y);
    }
    if (K == 1) {
      // every lane holds the same output: one pair of shared-memory atomics per warp
      for (int off = 16; off >= 1; off >>= 1) {
        sg += __shfl_down_sync(0xffffffffu, sg, off);
        sh += __shfl_down_sync(0xffffffffu, sh, off);
      }
      if ((tid & 31) == 0) {
        atomicAdd(&s_sum[0], static_cast<unsigned long long>(sg));
        atomicAdd(&s_sum[1], static_cast<unsigned long long>(sh));
      }
    } else {
      atomicAdd(&s_sum[2 * k], static_cast<unsigned long long>(sg));
      atomicAdd(&s_sum[2 * k + 1], static_cast<unsigned long long>(sh));
    }
  }
  if (__syncthreads_or(lowest < 1) != 0 && tid == 0 && hess_below_one != nullptr) *hess_below_one = 1;
  for (int i = tid; i < 2 * K; i += blockDim.x) {
    unsigned long long* dst = reinterpret_cast<unsigned long long*>(root_sums) + i;  // grad, hess of k = i / 2
    if (s_sum[i] != 0ull) atomicAdd(dst, s_sum[i]);
  }
  for (int off = 16; off >= 1; off >>= 1) {
    mg = max(mg, __shfl_down_sync(0xffffffffu, mg, off));
    mh = max(mh, __shfl_down_sync(0xffffffffu, mh, off));
  }
  // one pair per block: all blocks meet at these two words, which take about one atomic per clock (200k rows: 11.3 ->
  // 4.8 us)
  if ((tid & 31) == 0) {
    atomicMax(s_max, mg);
    atomicMax(s_max + 1, mh);
  }
  __syncthreads();
  if (tid < 2) atomicMax(max_abs + tid, s_max[tid]);
}

}  // namespace

void Quantise(lbk_context* ctx, const double* g, const double* h, int64_t ldg, const GradientForm& form, int64_t row_offset,
              int64_t n_local, int K, int seed, int2* gpair, GPairI64* root_sums, const QuantParams* params, int* max_abs, int* hess_below_one,
              cudaStream_t stream)
{
  if (n_local > 0) {
    int64_t blocks = (n_local * K + 511) / 512;  // (two elements per thread: fewer blocks at the common words)
    const int64_t cap = static_cast<int64_t>(ctx->sm_count) * 4;  // (as many as are resident)
    if (blocks > cap) blocks = cap;
    if (blocks * 256 < K) blocks = (K + 255) / 256;  // a thread keeps one output: at least K threads
    const size_t smem = sizeof(unsigned long long) * 2 * K;
    LBK_EXPECT(smem <= 48 * 1024, "too many outputs for the quantiser's block sums");
    if (smem > 40 * 1024) AllowSharedMemory(ctx, k_quantise, 1024);  // (the limit without it counts the static part too)
    LaunchChained(k_quantise, static_cast<unsigned>(blocks), 256, smem, stream, g, h, ldg, form, row_offset, n_local, K,
                                                                  static_cast<long long>(seed), params, gpair, root_sums, max_abs,
                                                                  hess_below_one);
    LBK_LAUNCH_CHECK();
  }
  AllReduce(ctx, root_sums, static_cast<size_t>(2) * K, LBK_I64, LBK_SUM, stream);
}

}  // namespace lbk
