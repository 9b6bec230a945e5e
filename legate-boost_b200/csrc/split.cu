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
#include "internal.h"
#include "split.cuh"

namespace lbk {
namespace {

constexpr int kSplitThreads = 256;
constexpr int kSplitWarps   = kSplitThreads / 32;

// A warp takes a feature (kWide) where there are so many units x features that no warp is alone on its scheduler: no
// barrier, and no totals of eight warps to add up, per output and 256 bins.  Microseconds with a block per feature and with
// a warp: one output, 400 features, 8 units 36 and 27, 128 units 272 and 259; 64 features, 32 units 29 and 24, 16 units 17.7 and 20; 20
// features, 128 units 36.7 and 27.7, 32 units 15.7 and 20.4; three outputs, 100 features, 32 units 79 and 66, 16 units 46 and
// 48; ten outputs, 64 units 296 and 287, 32 units 167 and 177.  A warp's chain is as long as its feature has bins: with more than 256
// (several outputs: 700) of them on average the line moves up with their number.  One output, 34 features, 256 units of 1000
// bins 44 and 62, 150 features, 32 and 64 units of 1024 bins 126 and 152, 160 and 150, of 512 bins 69 and 55, 90 and 86.
//
// Units of a level need not exist: nodes of few or of pure rows do not split.  For matrices of which a level takes no more than tens of
// microseconds anyway (kCountedCells) the kernel counts those that do, 1 to 2 us, and takes the other form if they are too
// few.  5921 x 206, three classes, 16 units, most of them gone: 33 us with a block per feature, 64 with a warp, 40 with a block and
// the count; five rounds 1915, 2098 and 1951.
constexpr int kWideOutputs = 64;  // (what a block has room for)
__host__ inline int64_t WideUnits(int n_features, int K, int64_t bins_per_feature)  // so many and the level is wide
{
  const int64_t least = K <= 1 ? 1500 : K < 6 ? 1000 * K : 6000, usual = K <= 1 ? 256 : 700;
  const int64_t bins  = bins_per_feature > usual ? bins_per_feature : usual, one = usual * (n_features > 0 ? n_features : 1);
  return K <= kWideOutputs ? (least * bins + one - 1) / one : INT64_MAX;
}
constexpr int kCountedUnits     = 4096;  // (more units are taken as they are)
constexpr int64_t kCountedCells = int64_t{1} << 25;  // rows x features x outputs

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
  int wide_units;  // (kWide) with fewer units that exist a block takes a feature; 0: they are not counted
};

// The best candidate of one slice of a unit; with one output also the sums left of it.
struct SliceBest {
  Cand c;
  GPairI64 left;
};

// grid = (units, slices).  A unit is a pair of siblings of which one was built (derive) or a single
// built node; a block takes one feature at a time, a thread one bin: it scans the built histogram, derives
// the sibling's from the parent's, writes both for the level below (not on the last level: nobody reads
// them there) and evaluates both nodes' gains while the sums are in registers, so that a level's histograms
// cross the memory once.  The buffer of the nodes built on the next level is zeroed on the way.  With
// several slices every block leaves its best candidates in `slice_best`, and the block of the unit that
// arrives last (a counter per node, zeroed once per tree) picks the winners and writes the tree.  Better()
// is a total order, so the winners do not depend on how the features were cut.
//
// What bounds it: on wide levels the issue slots (two float64 divisions per bin, output and node, and a
// 64-bit scan), on the upper levels the latency of one chain load - scan - division - reduction - claim, whose loads are
// asked for before anything is made of the nodes' sums and whose two winners are written by a warp each (200k x 50: 8.7
// -> 8.2 us a level).  There a thread takes a bin and not a warp a feature: a warp alone on its scheduler gets one
// instruction in about five clocks, and a feature's instructions were 9 us longer whatever the level held.  On wide levels
// (WideUnits) a warp takes a feature, 32 bins at a time.  Without the tests that GainsArePlain makes needless: 1M x 100, ten outputs,
// levels 1 to 7 422 -> 396 us and 294 -> 250 for the last one; 1M x 64, depth 9 192 -> 178; 200k x 50, six levels 67 -> 64.  Four blocks an SM and not three: 64 features, 8 and 16 units 11.2 and 16.9
// us instead of 12.8 and 18.4, for spills that cost the upper levels 0.3.
template <typename T, bool kManyOutputs, bool kDerive, bool kWide>
__global__ void __launch_bounds__(kSplitThreads, kManyOutputs || kWide ? 3 : 4)
  k_scan_split(const __grid_constant__ ScanSplitParams<T> p)
{
  extern __shared__ __align__(16) unsigned char smem_raw[];  // several outputs: terms [2][K]; then carries [K]
  __shared__ GPairI64 s_tot[2][kSplitWarps];
  __shared__ SliceBest s_c[2][kSplitWarps];
  __shared__ SliceBest s_best[2];
  __shared__ bool s_last;
  __shared__ int s_live[kWide ? kSplitWarps : 1];
  AfterTheKernelBefore();
  const ScanSplitLevel& lv = p.lv;
  if (lv.build_all != nullptr && (*lv.build_all != 0) == kDerive) return;
  const int K = lv.K, unit = blockIdx.x;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int node0 = lv.node_begin + (kDerive ? 2 * unit : unit);
  GPairI64* node_sums = p.tree.node_sums;
  // everything the block needs first, asked for at once
  const int parent_feature = node0 > 0 ? p.tree.feature[(node0 - 1) / 2] : 0;
  const GPairI64 sum_0 = LoadPair(node_sums + static_cast<int64_t>(node0) * K);
  const GPairI64 sum_1 = kDerive ? LoadPair(node_sums + static_cast<int64_t>(node0 + 1) * K) : GPairI64{0, 0};
  const QuantParams qp = *p.qp;
  bool wide  = kWide;
  int slices = gridDim.y;
  if constexpr (kWide) {
    const int units = gridDim.x;
    if (p.wide_units > 0) {
      int live = 0;
      for (int i = tid; i < units; i += kSplitThreads) live += p.tree.feature[(lv.node_begin + (kDerive ? 2 * i : i) - 1) / 2] >= 0 ? 1 : 0;
      live = __reduce_add_sync(0xffffffffu, live);
      if (lane == 0) s_live[warp] = live;
      __syncthreads();
      live = 0;
#pragma unroll
      for (int w = 0; w < kSplitWarps; ++w) live += s_live[w];
      wide = live >= p.wide_units;
    }
    if (wide) slices = min(slices, max((lv.f_end - lv.f_begin + kSplitWarps - 1) / kSplitWarps, 1));
    if (static_cast<int>(blockIdx.y) >= slices) return;
  }
  const int f_step = wide ? kSplitWarps * slices : slices;
  int f  = lv.f_begin + (wide ? kSplitWarps * blockIdx.y + warp : blockIdx.y);
  int fb = f < lv.f_end ? p.row_ptr[f] : 0, fe = f < lv.f_end ? p.row_ptr[f + 1] : 0;
  if (parent_feature < 0) return;  // the parent did not split: no such node
  // _a: the built node, _b: its sibling (SmallerChildIsLeft)
  const bool left_built = !kDerive || sum_0.hess < sum_1.hess;
  const int node_a = left_built ? node0 : node0 + 1, node_b = left_built ? node0 + 1 : node0;
  const int ja = node_a - lv.node_begin, jb = node_b - lv.node_begin;
  const GPairI64 sum_a = left_built ? sum_0 : sum_1, sum_b = left_built ? sum_1 : sum_0;
  const bool eval_a = sum_a.hess > 0, eval_b = kDerive && sum_b.hess > 0;
  const double l1 = p.sp.l1, reg = fmax(1e-5, p.sp.l2), msg = p.sp.min_split_gain;
  const bool plain    = GainsArePlain(qp, l1, reg);
  const int64_t Bs    = lv.bin_stride;
  const GPairI64* src = lv.built + static_cast<int64_t>(unit) * K * Bs;
  GPairI64* dst_a     = lv.level_hist + static_cast<int64_t>(ja) * K * Bs;
  GPairI64* dst_b     = lv.level_hist + static_cast<int64_t>(jb) * K * Bs;
  GPairI64* next_a    = lv.next_built + static_cast<int64_t>(ja) * K * Bs;
  GPairI64* next_b    = lv.next_built + static_cast<int64_t>(jb) * K * Bs;
  const GPairI64* par = lv.parent_hist + static_cast<int64_t>((node0 - 1) / 2 - lv.parent_begin) * K * Bs;
  NodeTerms* s_terms  = reinterpret_cast<NodeTerms*>(smem_raw);
  GPairI64* s_carry   = reinterpret_cast<GPairI64*>(smem_raw + (kManyOutputs ? sizeof(NodeTerms) * 2 * ((K + 1) / 2 * 2) : 0));
  // one output: the first bins are on their way before the nodes' terms are made
  GPairI64 first_a{0, 0}, first_b{0, 0};
  if (!kManyOutputs && !kWide && fb + tid < fe) {
    first_a = LoadPair(src + fb + tid);
    if (kDerive) first_b = LoadPair(par + fb + tid);
  }
  bool first = !kManyOutputs && !kWide;
  NodeTerms ta{}, tb{};
  if (kManyOutputs) {
    for (int i = tid; i < 2 * K; i += kSplitThreads) {
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
  int turn = 0;
  auto keep_best = [&](unsigned ok, double gain, int bin, const GPairI64& v, Cand& best, GPairI64& left) {
    if (ok && gain > 0) {
      const Cand c{gain, bin, f};
      if (Better(c, best)) {
        best = c;
        if (!kManyOutputs) left = v;
      }
    }
  };
  while (wide && f < lv.f_end) {
    const bool search = p.sp.feature_set == nullptr || p.sp.feature_set[f] != 0;
    GPairI64* carry = s_carry + (kManyOutputs ? warp * K : 0);  // (several outputs: sums of the bins before)
    GPairI64 before{0, 0};
    for (int base = fb; base < fe; base += 32) {
      const bool in = base + lane < fe;
      double gain_a = 0.0, gain_b = 0.0;
      GPairI64 va, vb{0, 0};
      unsigned ok_a = eval_a && search && in ? 1u : 0u, ok_b = eval_b && search && in ? 1u : 0u;
      GPairI64 ahead_a{0, 0}, ahead_b{0, 0};
      if (in) {
        ahead_a = LoadPair(src + base + lane);
        if (kDerive) ahead_b = LoadPair(par + base + lane);
      }
      if (kManyOutputs) __syncwarp();
      for (int k = 0; k < (kManyOutputs ? K : 1); ++k) {
        const int64_t at = (kManyOutputs ? static_cast<int64_t>(k) * Bs : 0) + base + lane;
        if (kManyOutputs) {
          ta = s_terms[2 * k];
          if (kDerive) tb = s_terms[2 * k + 1];
          before = base > fb ? carry[k] : GPairI64{0, 0};
        }
        const bool scanned = ta.h > 0.0;
        va = ahead_a;
        if (kDerive) vb = ahead_b;
        if (kManyOutputs && in && k + 1 < K) {
          ahead_a = LoadPair(src + at + Bs);
          if (kDerive) ahead_b = LoadPair(par + at + Bs);
        }
        long long sg = va.grad, sh = va.hess;
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
          const long long ng = __shfl_up_sync(0xffffffffu, sg, off);
          const long long nh = __shfl_up_sync(0xffffffffu, sh, off);
          if (lane >= off) {
            sg += ng;
            sh += nh;
          }
        }
        sg += before.grad;
        sh += before.hess;
        if (kManyOutputs) {
          __syncwarp();
          if (lane == 31) carry[k] = GPairI64{sg, sh};
        } else {
          before = GPairI64{__shfl_sync(0xffffffffu, sg, 31), __shfl_sync(0xffffffffu, sh, 31)};
        }
        if (in) {
          if (scanned && (sg > 0 || sh > 0)) va = GPairI64{sg, sh};
          if (kDerive) vb = scanned ? GPairI64{vb.grad - va.grad, vb.hess - va.hess} : GPairI64{0, 0};
          if (lv.write_hist) {
            StorePair(dst_a + at, va);
            if (kDerive) StorePair(dst_b + at, vb);
          }
          if (lv.next_built != nullptr) {
            StorePair(next_a + at, GPairI64{0, 0});
            if (kDerive) StorePair(next_b + at, GPairI64{0, 0});
          }
        }
        if (kDerive) {
          if (__any_sync(0xffffffffu, ok_a | ok_b)) AddGains(va, ok_a, ta, gain_a, vb, ok_b, tb, gain_b, qp, l1, reg, msg, plain);
        } else if (__any_sync(0xffffffffu, ok_a)) {
          ok_a = AddGain(va, ok_a, ta, qp, l1, reg, msg, plain, gain_a);
        }
      }
      keep_best(ok_a, gain_a, base + lane, va, best_a, left_a);
      if (kDerive) keep_best(ok_b, gain_b, base + lane, vb, best_b, left_b);
    }
    f += f_step;
    if (f >= lv.f_end) break;
    fb = p.row_ptr[f];
    fe = p.row_ptr[f + 1];
  }
  while (!wide && f < lv.f_end) {
    const bool search = p.sp.feature_set == nullptr || p.sp.feature_set[f] != 0;
    for (int base = fb; base < fe; base += kSplitThreads) {
      const bool in = base + tid < fe;
      double gain_a = 0.0, gain_b = 0.0;
      GPairI64 va, vb{0, 0};
      unsigned ok_a = eval_a && search && in ? 1u : 0u, ok_b = eval_b && search && in ? 1u : 0u;
      // (several outputs: the next output's sums are on their way while this one's are scanned, for which 24 warps
      // an SM instead of 32 are the price: 1M x 100, 10 outputs, 128 nodes: 416 -> 386 us)
      GPairI64 ahead_a{0, 0}, ahead_b{0, 0};
      if (kManyOutputs && in) {
        ahead_a = LoadPair(src + base + tid);
        if (kDerive) ahead_b = LoadPair(par + base + tid);
      }
      for (int k = 0; k < (kManyOutputs ? K : 1); ++k) {
        const int64_t at = (kManyOutputs ? static_cast<int64_t>(k) * Bs : 0) + base + tid;
        if (kManyOutputs) {
          ta = s_terms[2 * k];
          if (kDerive) tb = s_terms[2 * k + 1];
        }
        const bool scanned = ta.h > 0.0;  // else the raw values stay and no sibling is derived
        if (kManyOutputs) {
          va = ahead_a;
          if (kDerive) vb = ahead_b;
          if (in && k + 1 < K) {
            ahead_a = LoadPair(src + at + Bs);
            if (kDerive) ahead_b = LoadPair(par + at + Bs);
          }
        } else {
          va = first ? first_a : in ? LoadPair(src + at) : GPairI64{0, 0};
          if (kDerive) vb = first ? first_b : in && scanned ? LoadPair(par + at) : GPairI64{0, 0};
          first = false;
        }
        long long sg = va.grad, sh = va.hess;
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
          const long long ng = __shfl_up_sync(0xffffffffu, sg, off);
          const long long nh = __shfl_up_sync(0xffffffffu, sh, off);
          if (lane >= off) {
            sg += ng;
            sh += nh;
          }
        }
        // the warps before this one (two buffers: one barrier per turn is enough)
        const int buf = turn++ & 1;
        if (lane == 31) s_tot[buf][warp] = GPairI64{sg, sh};
        __syncthreads();
        GPairI64 before{0, 0};
        if (base > fb) before = s_carry[kManyOutputs ? k : 0];
#pragma unroll
        for (int w = 0; w < kSplitWarps - 1; ++w) {
          if (w < warp) {
            const GPairI64 t = s_tot[buf][w];
            before.grad += t.grad;
            before.hess += t.hess;
          }
        }
        sg += before.grad;
        sh += before.hess;
        if (fe - base > kSplitThreads) {  // more bins than threads: the next turn starts from this one's total
          __syncthreads();
          if (tid == kSplitThreads - 1) s_carry[kManyOutputs ? k : 0] = GPairI64{sg, sh};
        }
        if (in) {
          if (scanned && (sg > 0 || sh > 0)) va = GPairI64{sg, sh};
          if (kDerive) vb = scanned ? GPairI64{vb.grad - va.grad, vb.hess - va.hess} : GPairI64{0, 0};
          if (lv.write_hist) {
            StorePair(dst_a + at, va);
            if (kDerive) StorePair(dst_b + at, vb);
          }
          if (lv.next_built != nullptr) {
            StorePair(next_a + at, GPairI64{0, 0});
            if (kDerive) StorePair(next_b + at, GPairI64{0, 0});
          }
        }
        if (kDerive) {
          if (__any_sync(0xffffffffu, ok_a | ok_b)) AddGains(va, ok_a, ta, gain_a, vb, ok_b, tb, gain_b, qp, l1, reg, msg, plain);
        } else if (__any_sync(0xffffffffu, ok_a)) {
          ok_a = AddGain(va, ok_a, ta, qp, l1, reg, msg, plain, gain_a);
        }
      }
      keep_best(ok_a, gain_a, base + tid, va, best_a, left_a);
      if (kDerive) keep_best(ok_b, gain_b, base + tid, vb, best_b, left_b);
    }
    f += f_step;
    if (f >= lv.f_end) break;
    fb = p.row_ptr[f];
    fe = p.row_ptr[f + 1];
  }
  // the warp's best: the lane that holds it writes it down
  auto warp_best = [&](const Cand& mine, const GPairI64& left, SliceBest* out) {
    const int bin = WarpBest(mine.bin >= 0 ? mine.gain : 0.0, mine.bin);
    if (bin < 0 ? lane == 0 : mine.bin == bin) *out = SliceBest{bin < 0 ? Cand{0.0, -1, -1} : mine, left};
  };
  auto block_best = [&]() {
    warp_best(best_a, left_a, &s_c[0][warp]);
    if (kDerive) warp_best(best_b, left_b, &s_c[1][warp]);
    __syncthreads();
    if (tid < (kDerive ? 2 : 1)) {
      int at = 0;
      for (int w = 1; w < kSplitWarps; ++w)
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
    for (int i = tid; i < slices; i += kSplitThreads) {
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
        for (int k = tid; k < K; k += kSplitThreads) StorePair(rec_sums + k, GPairI64{0, 0});
      continue;
    }
    // (one output: a warp per node, so that the loads of either node's winner are on their way together)
    for (int k = kManyOutputs ? warp : warp == side ? 0 : K; k < K; k += kSplitWarps) {
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

// hessian and leaf value of every node from its quantised sums
__global__ void __launch_bounds__(256)
  k_finish_tree(TreeArrays tree, const QuantParams* __restrict__ qp_ptr, int K, int64_t n, double l1, double l2,
                double* __restrict__ hessian)
{
  AfterTheKernelBefore();
  const int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
  if (i >= n) return;
  const double2 v    = FinishedNode(tree, *qp_ptr, K, i, l1, l2);
  tree.leaf_value[i] = v.x;
  hessian[i]         = v.y;
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
  const int64_t wide_units = WideUnits(n_features, lv.K, lv.bin_stride / F);
  const bool wide          = units >= wide_units;
  // with several outputs a block keeps K terms of two nodes and K running prefixes (of every warp) in shared memory
  const size_t smem = (lv.K > 1 ? sizeof(NodeTerms) * 2 * ((lv.K + 1) / 2 * 2) : 0) + lv.K * sizeof(GPairI64) * (wide ? kSplitWarps : 1);
  // one feature per block until there are about sixteen blocks per SM, then several
  int slices     = n_features > 0 ? n_features : 1;
  const int most = (16 * ctx->sm_count + units - 1) / units;
  if (slices > most) slices = most;
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
  p.wide_units = wide && lv.cells <= kCountedCells && units <= kCountedUnits && lv.node_begin > 0 ? static_cast<int>(wide_units) : 0;
  unsigned char *mine = nullptr, *all = nullptr;
  const size_t rb = SplitRecordBytes(lv.K);
  if (exchange_records) {
    mine = s.alloc<unsigned char>(rb * lv.n_nodes);
    all  = s.alloc<unsigned char>(rb * lv.n_nodes * ctx->n_ranks);
    LBK_CUDA(cudaMemsetAsync(mine, 0, rb * lv.n_nodes, stream));
    p.records = mine;
  }
  auto fn = lv.K > 1 ? (lv.derive ? (wide ? k_scan_split<T, true, true, true> : k_scan_split<T, true, true, false>)
                                  : (wide ? k_scan_split<T, true, false, true> : k_scan_split<T, true, false, false>))
                     : (lv.derive ? (wide ? k_scan_split<T, false, true, true> : k_scan_split<T, false, true, false>)
                                  : (wide ? k_scan_split<T, false, false, true> : k_scan_split<T, false, false, false>));
  if (smem > 40 * 1024) AllowSharedMemory(ctx, fn, 2048);  // (the limit without it counts the static part too)
  LaunchChained(fn, dim3(units, slices), kSplitThreads, smem, stream, p);
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
  LaunchChained(k_finish_tree, static_cast<unsigned>((n + 255) / 256), 256, 0, stream, tree, qp, K, n, l1, l2, hessian);
  LBK_LAUNCH_CHECK();
}

template void ScanSplit<float>(lbk_context*, Scratch&, const ScanSplitLevel&, int, const int32_t*, const float*, int64_t,
                               const QuantParams*, const SplitParams&, const TreeArrays&, unsigned int*, bool, cudaStream_t);
template void ScanSplit<double>(lbk_context*, Scratch&, const ScanSplitLevel&, int, const int32_t*, const double*, int64_t,
                                const QuantParams*, const SplitParams&, const TreeArrays&, unsigned int*, bool, cudaStream_t);

}  // namespace lbk
