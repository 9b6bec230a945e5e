// Prefix scan with sibling subtraction and split evaluation of a level, in one pass over its histograms.
//
// Reference behaviour restated here (src/models/tree/):
//   SelectHistogramNode / ComputeHistogramBin  build_tree.h:80-104 - only the child with the
//     smaller quantised hessian of output 0 is built (ties: the right child) when the parent's
//     histogram is available (SmallerChildIsLeft, device_utils.cuh);
//   scan_kernel        build_tree.cu:597-668 - inclusive prefix over the bins of each feature; the
//     prefix replaces the bin value only if prefix.grad > 0 or prefix.hess > 0; then
//     sibling = parent - node;
//   perform_best_split build_tree.cu:682-782 - gain of every bin summed over outputs in float64 on
//     dequantised sums, zero if any output has a non-positive hessian on either side, accept if
//     the best gain exceeds 1e-5.  Ties: the reference keeps, per thread t = bin mod 512, the
//     first strict maximum and reduces with op(a,b) = a.gain > b.gain ? a : b where a always
//     comes from lower thread ids, so equal gains resolve to the largest (bin mod 512) and then
//     the smallest bin.  That total order is applied here, independent of the reduction shape.
// Compiled with -fmad=false.
#include "device_utils.cuh"
#include "internal.h"

namespace lbk {
namespace {

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

constexpr int kSplitWarps = 8;  // most warps of a block

// What a rank knows about its best split of a node when the features are divided among the ranks:
// the candidate and the sums left of it; K pairs follow the header.
struct SplitRecordHeader {
  double gain;
  int bin;
  int pad;
};
__host__ __device__ inline size_t SplitRecordBytes(int K) { return sizeof(SplitRecordHeader) + sizeof(GPairI64) * K; }

// The winner of a node becomes the tree: feature, split value, gain and the sums of the two children.
// left_of(k) = the sums left of the winning bin, output k (called by one thread per k).
template <typename T, typename LeftOf>
__device__ inline void ApplyWinner(const Cand& nb, int node, int K, const int32_t* __restrict__ row_ptr,
                                   const T* __restrict__ cuts, int64_t cut_stride, const TreeArrays& tree, LeftOf left_of,
                                   int tid, int n_threads)
{
  if (!(nb.gain > 1e-5)) return;
  GPairI64* node_sums = tree.node_sums;
  const int l = 2 * node + 1, r = 2 * node + 2;
  for (int k = tid; k < K; k += n_threads) {
    const GPairI64 ns = LoadPair(node_sums + static_cast<int64_t>(node) * K + k);
    const GPairI64 ls = left_of(k);
    StorePair(node_sums + static_cast<int64_t>(l) * K + k, ls);
    StorePair(node_sums + static_cast<int64_t>(r) * K + k, GPairI64{ns.grad - ls.grad, ns.hess - ls.hess});
    if (k == 0) {
      const int b            = nb.bin - row_ptr[nb.feature];
      tree.feature[node]     = nb.feature;
      tree.split_value[node] = static_cast<double>(cuts[nb.feature * cut_stride + b]);
      tree.gain[node]        = nb.gain;
      tree.split_bin[node]   = b;
    }
  }
}

template <typename T>
struct ScanSplitParams {
  ScanSplitLevel lv;
  const int32_t* row_ptr;
  const T* cuts;
  int64_t cut_stride;
  const QuantParams* qp;
  SplitParams sp;
  TreeArrays tree;
  struct SliceBest* slice_best;  // [units][slices][2]
  unsigned int* arrived;
  unsigned char* records;
};

// The best candidate of one slice of a unit; with one output also the sums left of it.
struct SliceBest {
  Cand c;
  GPairI64 left;
};

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

// The gain of one output at one bin, added to `gain`; false if a side has no positive hessian (sums are
// below 2^51, so their differences are exact in float64).
__device__ inline bool AddGain(GPairI64 left, const NodeTerms& n, const QuantParams& qp, double l1, double reg, double msg,
                               double& gain)
{
  const double lg = WholeToDouble(left.grad), lh = WholeToDouble(left.hess);
  const double rg = n.g - lg, rh = n.h - lh;
  if (lh <= 0.0 || rh <= 0.0) return false;
  const double gl = LeafGain(GPairF64{lg * qp.inv_g, lh * qp.inv_h}, l1, reg);
  const double gr = LeafGain(GPairF64{rg * qp.inv_g, rh * qp.inv_h}, l1, reg);
  gain += (0.5 * (gl + gr - n.gain)) - msg;
  return true;
}

// grid = (units, slices).  A unit is a pair of siblings of which one was built (derive) or a single
// built node; a warp takes one feature at a time: it scans the built histogram, derives the sibling's
// from the parent's, writes both for the level below (not on the last level: nobody reads them there)
// and evaluates both nodes' gains while the sums are in registers, so that a level's histograms cross
// the memory once.  The buffer of the nodes built on the next level is zeroed on the way.  With several
// slices every block leaves its best candidates in `slice_best`, and the block of the unit that arrives
// last (a counter per node, zeroed once per tree) picks the winners and writes the tree.  Better() is a
// total order, so the winners do not depend on how the features were cut.
//
// What bounds it: on wide levels the issue slots (two float64 divisions per bin, output and node, and a
// 64-bit scan), on the upper levels the latency of one chain load - scan - division - reduction - claim.
// kRun bins per lane and turn: four with one output (few warps, long chains), two with several, where
// the registers that this saves keep three blocks on an SM.
template <typename T, bool kManyOutputs, bool kDerive, int kRun>
__global__ void __launch_bounds__(kSplitWarps * 32, kManyOutputs ? 3 : 2)
  k_scan_split(const __grid_constant__ ScanSplitParams<T> p)
{
  extern __shared__ __align__(16) unsigned char smem_raw[];  // several outputs: terms [2][K], then [warps][K] carries
  __shared__ SliceBest s_c[2][kSplitWarps];
  __shared__ SliceBest s_best[2];
  __shared__ bool s_last;
  const ScanSplitLevel& lv = p.lv;
  const int K = lv.K, unit = blockIdx.x, slices = gridDim.y;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, n_warps = blockDim.x >> 5;
  const int node0 = lv.node_begin + (kDerive ? 2 * unit : unit);
  GPairI64* node_sums = p.tree.node_sums;
  // everything the block needs first, asked for at once
  const int parent_feature = node0 > 0 ? p.tree.feature[(node0 - 1) / 2] : 0;
  const GPairI64 sum_0 = LoadPair(node_sums + static_cast<int64_t>(node0) * K);
  const GPairI64 sum_1 = kDerive ? LoadPair(node_sums + static_cast<int64_t>(node0 + 1) * K) : GPairI64{0, 0};
  const QuantParams qp = *p.qp;
  int f  = lv.f_begin + blockIdx.y * n_warps + warp;
  int fb = f < lv.f_end ? p.row_ptr[f] : 0, fe = f < lv.f_end ? p.row_ptr[f + 1] : 0;
  if (parent_feature < 0) return;  // the parent did not split: no such node
  // _a: the built node, _b: its sibling (SmallerChildIsLeft)
  const bool left_built = !kDerive || sum_0.hess < sum_1.hess;
  const int node_a = left_built ? node0 : node0 + 1, node_b = left_built ? node0 + 1 : node0;
  const int ja = node_a - lv.node_begin, jb = node_b - lv.node_begin;
  const GPairI64 sum_a = left_built ? sum_0 : sum_1, sum_b = left_built ? sum_1 : sum_0;
  const bool eval_a = sum_a.hess > 0, eval_b = kDerive && sum_b.hess > 0;
  const double l1 = p.sp.l1, reg = fmax(1e-5, p.sp.l2), msg = p.sp.min_split_gain;
  const int64_t Bs    = lv.bin_stride;
  const GPairI64* src = lv.built + static_cast<int64_t>(unit) * K * Bs;
  GPairI64* dst_a     = lv.level_hist + static_cast<int64_t>(ja) * K * Bs;
  GPairI64* dst_b     = lv.level_hist + static_cast<int64_t>(jb) * K * Bs;
  GPairI64* next_a    = lv.next_built + static_cast<int64_t>(ja) * K * Bs;
  GPairI64* next_b    = lv.next_built + static_cast<int64_t>(jb) * K * Bs;
  const GPairI64* par = lv.parent_hist + static_cast<int64_t>((node0 - 1) / 2 - lv.parent_begin) * K * Bs;
  NodeTerms* s_terms  = reinterpret_cast<NodeTerms*>(smem_raw);
  GPairI64* s_carry   = reinterpret_cast<GPairI64*>(smem_raw + sizeof(NodeTerms) * 2 * ((K + 1) / 2 * 2)) + warp * K;
  NodeTerms ta{}, tb{};
  if (kManyOutputs) {
    for (int i = tid; i < 2 * K; i += blockDim.x) {
      const int k = i >> 1, node = (i & 1) ? node_b : node_a;
      if (kDerive || !(i & 1)) s_terms[i] = TermsOf(LoadPair(node_sums + static_cast<int64_t>(node) * K + k), qp, l1, reg);
    }
    __syncthreads();
  } else {
    ta = TermsOf(sum_a, qp, l1, reg);
    if (kDerive) tb = TermsOf(sum_b, qp, l1, reg);
  }

  Cand best_a{0.0, -1, -1}, best_b{0.0, -1, -1};
  GPairI64 left_a{0, 0}, left_b{0, 0};
  while (f < lv.f_end) {
    const bool search = p.sp.feature_set == nullptr || p.sp.feature_set[f] != 0;
    GPairI64 carry{0, 0};
    if (kManyOutputs) {
      __syncwarp();
      for (int k = lane; k < K; k += 32) s_carry[k] = GPairI64{0, 0};
      __syncwarp();
    }
    for (int base = fb; base < fe; base += 32 * kRun) {
      double gain_a[kRun], gain_b[kRun];
      GPairI64 va[kRun], vb[kRun];
      unsigned in = 0;
#pragma unroll
      for (int i = 0; i < kRun; ++i) {
        gain_a[i] = gain_b[i] = 0.0;
        if (base + i * 32 + lane < fe) in |= 1u << i;
      }
      unsigned ok_a = eval_a && search ? in : 0u, ok_b = eval_b && search ? in : 0u;
      for (int k = 0; k < (kManyOutputs ? K : 1); ++k) {
        const int64_t ko = (kManyOutputs ? static_cast<int64_t>(k) * Bs : 0) + base + lane;
        if (kManyOutputs) {
          ta = s_terms[2 * k];
          if (kDerive) tb = s_terms[2 * k + 1];
        }
        const bool scanned = ta.h > 0.0;  // else the raw values stay and no sibling is derived
        long long sg[kRun], sh[kRun];
#pragma unroll
        for (int i = 0; i < kRun; ++i) {
          va[i] = in & (1u << i) ? LoadPair(src + ko + i * 32) : GPairI64{0, 0};
          if (kDerive) vb[i] = (in & (1u << i)) && scanned ? LoadPair(par + ko + i * 32) : GPairI64{0, 0};
          sg[i] = va[i].grad;
          sh[i] = va[i].hess;
        }
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
#pragma unroll
          for (int i = 0; i < kRun; ++i) {
            const long long ng = __shfl_up_sync(0xffffffffu, sg[i], off);
            const long long nh = __shfl_up_sync(0xffffffffu, sh[i], off);
            if (lane >= off) {
              sg[i] += ng;
              sh[i] += nh;
            }
          }
        }
        GPairI64 run = kManyOutputs ? s_carry[k] : carry;
#pragma unroll
        for (int i = 0; i < kRun; ++i) {
          const long long tg = __shfl_sync(0xffffffffu, sg[i], 31), th = __shfl_sync(0xffffffffu, sh[i], 31);
          sg[i] += run.grad;
          sh[i] += run.hess;
          run.grad += tg;
          run.hess += th;
        }
        if (kManyOutputs) {
          __syncwarp();
          if (lane == 0) s_carry[k] = run;
        } else {
          carry = run;
        }
#pragma unroll
        for (int i = 0; i < kRun; ++i) {
          if (!(in & (1u << i))) continue;
          if (scanned && (sg[i] > 0 || sh[i] > 0)) va[i] = GPairI64{sg[i], sh[i]};
          if (kDerive) vb[i] = scanned ? GPairI64{vb[i].grad - va[i].grad, vb[i].hess - va[i].hess} : GPairI64{0, 0};
          if (lv.write_hist) {
            StorePair(dst_a + ko + i * 32, va[i]);
            if (kDerive) StorePair(dst_b + ko + i * 32, vb[i]);
          }
          if (lv.next_built != nullptr) {
            StorePair(next_a + ko + i * 32, GPairI64{0, 0});
            if (kDerive) StorePair(next_b + ko + i * 32, GPairI64{0, 0});
          }
          if (ok_a & (1u << i))
            if (!AddGain(va[i], ta, qp, l1, reg, msg, gain_a[i])) ok_a &= ~(1u << i);
          if (kDerive && (ok_b & (1u << i)))
            if (!AddGain(vb[i], tb, qp, l1, reg, msg, gain_b[i])) ok_b &= ~(1u << i);
        }
      }
#pragma unroll
      for (int i = 0; i < kRun; ++i) {
        const int b = base + i * 32 + lane;
        if ((ok_a & (1u << i)) && gain_a[i] > 0) {
          const Cand c{gain_a[i], b, f};
          if (Better(c, best_a)) {
            best_a = c;
            if (!kManyOutputs) left_a = va[i];
          }
        }
        if (kDerive && (ok_b & (1u << i)) && gain_b[i] > 0) {
          const Cand c{gain_b[i], b, f};
          if (Better(c, best_b)) {
            best_b = c;
            if (!kManyOutputs) left_b = vb[i];
          }
        }
      }
    }
    f += slices * n_warps;
    if (f < lv.f_end) {
      fb = p.row_ptr[f];
      fe = p.row_ptr[f + 1];
    }
  }
  // the warp's best: the lane that holds it writes it down
  auto warp_best = [&](const Cand& mine, const GPairI64& left, SliceBest* out) {
    Cand best = mine;
#pragma unroll
    for (int off = 16; off >= 1; off >>= 1) {
      Cand o;
      o.gain    = __shfl_xor_sync(0xffffffffu, best.gain, off);
      o.bin     = __shfl_xor_sync(0xffffffffu, best.bin, off);
      o.feature = __shfl_xor_sync(0xffffffffu, best.feature, off);
      if (Better(o, best)) best = o;
    }
    if (best.bin < 0 ? lane == 0 : mine.bin == best.bin) *out = SliceBest{best, left};
  };
  auto block_best = [&]() {
    warp_best(best_a, left_a, &s_c[0][warp]);
    if (kDerive) warp_best(best_b, left_b, &s_c[1][warp]);
    __syncthreads();
    if (tid < (kDerive ? 2 : 1)) {
      int at = 0;
      for (int w = 1; w < n_warps; ++w)
        if (Better(s_c[tid][w].c, s_c[tid][at].c)) at = w;
      s_best[tid] = s_c[tid][at];
    }
    __syncthreads();
  };
  block_best();
  if (slices > 1) {
    SliceBest* mine = p.slice_best + static_cast<int64_t>(unit) * slices * 2;
    if (tid == 0) {
      mine[blockIdx.y * 2] = s_best[0];
      if (kDerive) mine[blockIdx.y * 2 + 1] = s_best[1];
      __threadfence();
      s_last = atomicAdd(p.arrived + node0, 1u) == static_cast<unsigned>(slices - 1);
    }
    // (what the other threads wrote to the level's histogram is ordered before thread 0's fence by the
    // barrier inside block_best)
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    best_a = best_b = Cand{0.0, -1, -1};
    for (int i = tid; i < slices; i += blockDim.x) {
      const volatile SliceBest* a = mine + i * 2;
      const Cand ca{a[0].c.gain, a[0].c.bin, a[0].c.feature};
      if (Better(ca, best_a)) {
        best_a = ca;
        left_a = GPairI64{a[0].left.grad, a[0].left.hess};
      }
      if (kDerive) {
        const Cand cb{a[1].c.gain, a[1].c.bin, a[1].c.feature};
        if (Better(cb, best_b)) {
          best_b = cb;
          left_b = GPairI64{a[1].left.grad, a[1].left.hess};
        }
      }
    }
    block_best();
  }

  // The sums left of the winning bin: with one output they came along; else from the level's histogram
  // where it was written, else scanned again from the raw sums (one feature), a warp per output.
  for (int side = 0; side < (kDerive ? 2 : 1); ++side) {
    if (!(side == 0 ? eval_a : eval_b)) continue;
    const int node = side == 0 ? node_a : node_b;
    const Cand nb  = s_best[side].c;
    unsigned char* rec = p.records ? p.records + static_cast<size_t>(node - lv.node_begin) * SplitRecordBytes(K) : nullptr;
    if (rec != nullptr && tid == 0) *reinterpret_cast<SplitRecordHeader*>(rec) = SplitRecordHeader{nb.gain, nb.bin, 0};
    GPairI64* rec_sums = reinterpret_cast<GPairI64*>(rec + sizeof(SplitRecordHeader));
    if (nb.bin < 0) {
      if (rec != nullptr)
        for (int k = tid; k < K; k += blockDim.x) StorePair(rec_sums + k, GPairI64{0, 0});
      continue;
    }
    for (int k = warp; k < K; k += n_warps) {
      const int64_t ko = static_cast<int64_t>(k) * Bs;
      GPairI64 ls;
      if (!kManyOutputs) {
        ls = s_best[side].left;
      } else if (lv.write_hist) {
        ls = LoadPairStreaming((side == 0 ? dst_a : dst_b) + ko + nb.bin);
      } else {
        const bool scanned = s_terms[2 * k].h > 0.0;
        const GPairI64 raw = LoadPair(src + ko + nb.bin);
        GPairI64 pre{0, 0};
        for (int b = p.row_ptr[nb.feature] + lane; b <= nb.bin; b += 32) {
          const GPairI64 v = LoadPair(src + ko + b);
          pre.grad += v.grad;
          pre.hess += v.hess;
        }
        for (int off = 16; off >= 1; off >>= 1) {
          pre.grad += __shfl_xor_sync(0xffffffffu, pre.grad, off);
          pre.hess += __shfl_xor_sync(0xffffffffu, pre.hess, off);
        }
        ls = scanned && (pre.grad > 0 || pre.hess > 0) ? pre : raw;
        if (side == 1) {
          const GPairI64 pv = LoadPair(par + ko + nb.bin);
          ls = scanned ? GPairI64{pv.grad - ls.grad, pv.hess - ls.hess} : GPairI64{0, 0};
        }
      }
      if (rec != nullptr) {
        if (lane == 0) StorePair(rec_sums + k, ls);
      } else if (lane == 0) {
        ApplyWinner<T>(nb, node, K, p.row_ptr, p.cuts, p.cut_stride, p.tree, [&](int) { return ls; }, k, K);
      }
    }
  }
}

// One block per node: the best of the ranks' candidates (the same total order as inside a rank, so
// the winner is the one a single rank would have found over all features) becomes the tree.
template <typename T>
__global__ void __launch_bounds__(64)
  k_apply_records(const unsigned char* __restrict__ all_records, int n_ranks, int n_nodes, int node_begin, int K, int F,
                  const int32_t* __restrict__ row_ptr, const T* __restrict__ cuts, int64_t cut_stride, TreeArrays tree)
{
  const int j    = blockIdx.x;
  const int node = node_begin + j;
  if (LoadPair(tree.node_sums + static_cast<int64_t>(node) * K).hess <= 0) return;
  const size_t rb = SplitRecordBytes(K);
  Cand best{0.0, -1, -1};
  int best_rank = -1;
  for (int r = 0; r < n_ranks; ++r) {
    const SplitRecordHeader* h =
      reinterpret_cast<const SplitRecordHeader*>(all_records + (static_cast<size_t>(r) * n_nodes + j) * rb);
    const Cand c{h->gain, h->bin, -1};
    if (c.gain > 0 && c.bin >= 0 && Better(c, best)) {
      best      = c;
      best_rank = r;
    }
  }
  if (best_rank < 0) return;
  int lo = 0, hi = F;  // the feature of the bin: the last one with row_ptr <= bin
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (row_ptr[mid] <= best.bin) lo = mid; else hi = mid;
  }
  best.feature = lo;
  const GPairI64* ls = reinterpret_cast<const GPairI64*>(
    all_records + (static_cast<size_t>(best_rank) * n_nodes + j) * rb + sizeof(SplitRecordHeader));
  ApplyWinner<T>(best, node, K, row_ptr, cuts, cut_stride, tree, [&](int k) { return LoadPair(ls + k); }, threadIdx.x, blockDim.x);
}

// hessian and leaf value of every node from its quantised sums; a node whose parent did not split keeps 0
__global__ void __launch_bounds__(256)
  k_finish_tree(TreeArrays tree, const QuantParams* __restrict__ qp_ptr, int K, int64_t n, double l1, double l2,
                double* __restrict__ hessian)
{
  const int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
  if (i >= n) return;
  const int node   = static_cast<int>(i / K);
  const GPairF64 s = Dequantise(tree.node_sums[i], *qp_ptr);
  hessian[i]       = s.hess;
  const bool here  = node == 0 || tree.feature[(node - 1) / 2] >= 0;
  tree.leaf_value[i] = here ? CalculateLeafValue(s.grad, s.hess, l1, l2) : 0.0;
}

}  // namespace

template <typename T>
void ScanSplit(lbk_context* ctx, Scratch& s, const ScanSplitLevel& lv, int F, const int32_t* row_ptr, const T* cuts,
               int64_t cut_stride, const QuantParams* qp, const SplitParams& sp, const TreeArrays& tree,
               unsigned int* arrived, bool exchange_records, cudaStream_t stream)
{
  const int n_features = lv.f_end - lv.f_begin;
  const int units      = lv.derive ? lv.n_nodes / 2 : lv.n_nodes;
  if (units <= 0) return;
  // with several outputs a block keeps K terms of two nodes and every warp K running prefixes in shared
  // memory: fewer warps for very many outputs
  int warps = kSplitWarps;
  auto need = [&](int w) {
    return lv.K > 1 ? sizeof(NodeTerms) * 2 * ((lv.K + 1) / 2 * 2) + static_cast<size_t>(w) * lv.K * sizeof(GPairI64) : 0;
  };
  while (warps > 1 && need(warps) > 40 * 1024) warps /= 2;
  const size_t smem = need(warps);
  // one feature per warp until there are about eight blocks per SM, then several
  int slices     = (n_features + warps - 1) / warps;
  const int most = (8 * ctx->sm_count + units - 1) / units;
  if (slices > most) slices = most;
  if (slices < 1) slices = 1;
  ScanSplitParams<T> p;
  p.lv         = lv;
  p.row_ptr    = row_ptr;
  p.cuts       = cuts;
  p.cut_stride = cut_stride;
  p.qp         = qp;
  p.sp         = sp;
  p.tree       = tree;
  p.slice_best = slices > 1 ? s.alloc<SliceBest>(static_cast<size_t>(units) * slices * 2) : nullptr;
  p.arrived    = arrived;
  p.records    = nullptr;
  unsigned char *mine = nullptr, *all = nullptr;
  const size_t rb = SplitRecordBytes(lv.K);
  if (exchange_records) {
    mine = s.alloc<unsigned char>(rb * lv.n_nodes);
    all  = s.alloc<unsigned char>(rb * lv.n_nodes * ctx->n_ranks);
    LBK_CUDA(cudaMemsetAsync(mine, 0, rb * lv.n_nodes, stream));
    p.records = mine;
  }
  auto fn = lv.K > 1 ? (lv.derive ? k_scan_split<T, true, true, 2> : k_scan_split<T, true, false, 2>)
                     : (lv.derive ? k_scan_split<T, false, true, 4> : k_scan_split<T, false, false, 4>);
  if (smem > 48 * 1024)
    LBK_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)));
  fn<<<dim3(units, slices), warps * 32, smem, stream>>>(p);
  LBK_LAUNCH_CHECK();
  if (exchange_records) {
    // every rank has searched its own features: the candidates of all ranks meet on every rank
    if (!AllGatherBytes(ctx, mine, all, rb * lv.n_nodes, stream))
      throw Error(LBK_ERR_COMM, "the split records need an NCCL communicator");
    k_apply_records<T><<<lv.n_nodes, 64, 0, stream>>>(all, ctx->n_ranks, lv.n_nodes, lv.node_begin, lv.K, F, row_ptr, cuts,
                                                      cut_stride, tree);
    LBK_LAUNCH_CHECK();
    s.free_one(mine);
    s.free_one(all);
  }
  if (p.slice_best) s.free_one(p.slice_best);
}

void FinishTree(const TreeArrays& tree, const QuantParams* qp, int K, double l1, double l2, double* hessian,
                cudaStream_t stream)
{
  const int64_t n = static_cast<int64_t>(tree.max_nodes) * K;
  k_finish_tree<<<static_cast<unsigned>((n + 255) / 256), 256, 0, stream>>>(tree, qp, K, n, l1, l2, hessian);
  LBK_LAUNCH_CHECK();
}

template void ScanSplit<float>(lbk_context*, Scratch&, const ScanSplitLevel&, int, const int32_t*, const float*, int64_t,
                               const QuantParams*, const SplitParams&, const TreeArrays&, unsigned int*, bool, cudaStream_t);
template void ScanSplit<double>(lbk_context*, Scratch&, const ScanSplitLevel&, int, const int32_t*, const double*, int64_t,
                                const QuantParams*, const SplitParams&, const TreeArrays&, unsigned int*, bool, cudaStream_t);

}  // namespace lbk
