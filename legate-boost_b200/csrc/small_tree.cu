// A whole tree on a small matrix in one cooperative launch.
//
// With a few thousand rows every kernel of the general path (build_tree.cu) takes its fixed cost - launch,
// dependent loads, a last block that everybody waits for - and a tree has more than a dozen of them.  Here the
// features are divided among the blocks and the blocks meet at one grid barrier per level:
//   * block (feature, part) draws, sorts and prunes the feature's proposals, bins its column and quantises a
//     slice of the rows; the |g|, |h| sums (canonical order, abs_sum.cuh) are made by every block for itself;
//   * every block keeps the node of every row in shared memory.  On a level it sums its feature's
//     histograms of the built nodes in shared memory, scans them, derives the siblings from the parents'
//     (kept in global memory, one region per feature) and leaves its best candidate of every node;
//   * after the barrier every block picks the winners of the level by itself (same candidates, same total
//     order, so all blocks agree) and moves the rows down, reading the winning features' bin ids.
// No repartition, no list of rows, no merge of partial histograms.
//
// What one block writes and another reads is ordered by the barriers alone.  Written once, before the first of them:
// cuts, counts, bins_t, pairs, root_part, the cleared tree and outputs.  Written on every level:
//   * cand, cand_left: before the barrier of level d, read after it; two regions by the parity of the level
//     (small_layout.h), so that level d is overwritten on level d + 2, behind the barrier of level d + 1, which no
//     block reaches before it has read level d;
//   * hist: before the barrier of level d, read on level d + 1 before its barrier; two buffers, overwritten on level
//     d + 2, behind that barrier;
//   * the nodes of the tree: by block 0 only, each once; read by all behind the last barrier.
//
// 32-bit shared-memory sums are exact here without a bound on the magnitudes: a quantised value is added as
// its high and its low 16 bits, whose sums over at most 65536 rows fit 32 bits.
//
// What bounds it: the chain of latencies of a level - pass over the rows 1.2 us, scan, float64 divisions and candidates 2.5,
// barrier 1 to 2, winners and move 1.5 - and about 8 us for everything before the root.  Where a block has one or two pairs of
// nodes a thread takes a bin; with a warp per node (four bins per lane) a level of 500 x 10 took 9 us longer, because a lone
// warp gets an instruction in about five clocks.  Deeper levels have a warp per pair: the chain, most of it waiting, came
// once for every two pairs before.  500 x 10, depth 4: 39 us per tree (260 us of kernels in 70 launches before
// there was this form).  Five rounds, a thread per bin on all levels, proposals sorted by a bitonic network (3.3 us), the four
// divisions of a pair of nodes one after the other, and this: 500 x 10, depth 4: 482 -> 433 us; 2000 x 30, depth 8 1122 -> 851;
// 4000 x 64, depth 10 4211 -> 2392; 15000 x 100, depth 8 2872 -> 1965.

#include "abs_sum.cuh"
#include "count_sort.cuh"
#include "internal.h"
#include "objective.cuh"
#include "small_layout.h"
#include "split.cuh"

namespace lbk {
namespace {

constexpr int kSmallThreads     = 512;
constexpr int kSmallWarps       = kSmallThreads / 32;
constexpr int kSmallBins        = 256;
constexpr int kFaultGridBarrier = 51;  // status word: a block did not reach the barrier

struct alignas(16) SmallCand {
  double gain;
  int bin;  // of the feature
  int pad;
  GPairI64 left;  // the sums left of it (one output)
};

template <typename T>
struct SmallParams {
  const T* X;
  int64_t ldx;
  int N, F, K, D, S, seed;
  int parts, part_shift;  // blocks per feature: a power of two
  int64_t row_offset, dataset_rows;
  // gradients: given (objective < 0), or made from the current prediction
  const double* g;
  const double* h;
  int64_t ldg;
  int objective;
  const double* y;
  double* pred;  // objective >= 0: [N][K], the tree's leaf values are added at the end
  double lr;
  double l1, l2, msg;
  const uint8_t* feature_set;
  TreeArrays tree;
  double* hessian;
  int32_t* leaf;  // may be null
  // scratch
  T* cuts;             // [F][S]
  int32_t* counts;     // [F]
  uint8_t* bins_t;     // [F][pitch]
  int pitch;
  int2* pairs;         // [N][K]
  GPairI64* root_part; // [blocks][K]
  GPairI64* hist[2];   // levels alternate: [F][nodes of the level][K][256]
  SmallCand* cand;     // levels alternate (SmallCandBegin): [nodes of the level][F]
  GPairI64* cand_left; // several outputs: likewise, [nodes of the level][F][K]
  int max_slots;       // histograms in shared memory at a time
  unsigned int* barrier;  // zero at the start
  int* status;
  int32_t* info_host;     // mapped host word for the number of bins, or null
};

// All blocks of the (cooperative) grid; bounded: after about a second it gives up, reports and returns false
// in every thread of the block.
__device__ inline bool GridBarrier(unsigned int* word, unsigned int target, int* status, int* s_ok)
{
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    atomicAdd(word, 1u);
    int ok = 0;
    for (unsigned spin = 0; spin < (1u << 21); ++spin) {
      unsigned int v;
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];\n" : "=r"(v) : "l"(word) : "memory");
      if (static_cast<int>(v - target) >= 0) {
        ok = 1;
        break;
      }
    }
    if (!ok) ReportFault(status, kFaultGridBarrier);
    *s_ok = ok;
  }
  __syncthreads();
  return *s_ok != 0;
}

// What a tree is grown on, as far as it is one output: less code, which every launch of this kernel fetches anew.
enum SmallForm { kGiven, kSquaredError, kAnyForm };

template <SmallForm kForm, typename T>
__device__ inline double2 SmallGradient(const SmallParams<T>& p, int row, int k)
{
  if (kForm == kSquaredError) return GradientSquaredError(p.pred[row], p.y[row], p.lr);
  if (kForm == kGiven || p.objective < 0) return make_double2(p.g[row * p.ldg + k], p.h[row * p.ldg + k]);
  const double raw = p.pred[static_cast<int64_t>(row) * p.K + k], y = p.y[static_cast<int64_t>(row) * p.K + k];
  return p.objective == LBK_SQUARED_ERROR ? GradientSquaredError(raw, y, p.lr) : GradientLogistic(raw, y, p.lr);
}

template <typename T, bool kMany, SmallForm kForm>
__global__ void __launch_bounds__(kSmallThreads, 1)
  k_tree_small(const SmallParams<T> p)
{
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ int s_ok, s_cnt[kSmallWarps + 1];
  __shared__ double s_sum[2][2 * kSumThreads / 32];
  __shared__ QuantParams s_qp;
  __shared__ GPairI64 s_tot[2][kSmallWarps / 2];
  __shared__ SmallCand s_best[2][2][kSmallWarps / 2];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int N = p.N, F = p.F, K = kMany ? p.K : 1, D = p.D, S = p.S;
  const int n_blocks = gridDim.x, block = blockIdx.x;
  const int part     = block % p.parts;            // of the feature's rows (binning) and node pairs (levels)
  const int f_first = block / p.parts, f_step = n_blocks / p.parts;
  const int n_sums  = max(1, (1 << max(D - 1, 0)) * K);  // node sums of a level
  // shared memory: histograms | candidate gains (several outputs) | node sums of two levels, terms | row_ptr | winners |
  // node of every row
  int* s_hist         = reinterpret_cast<int*>(smem_raw);  // [slot][4][256]: g high, g low, h high, h low
  double* s_gain      = reinterpret_cast<double*>(s_hist + p.max_slots * 4 * kSmallBins);
  GPairI64* s_nodes   = reinterpret_cast<GPairI64*>(s_gain + (K > 1 ? p.max_slots * 2 * kSmallBins : 0));
  GPairI64* s_next    = s_nodes + n_sums;
  NodeTerms* s_terms  = reinterpret_cast<NodeTerms*>(s_next + n_sums);  // of the level's nodes
  int* s_rp           = reinterpret_cast<int*>(s_terms + n_sums);       // [F + 1]
  int* s_wfeat        = s_rp + F + 1;                             // [nodes of a level], -1: no split / no node
  int* s_wbin         = s_wfeat + (1 << max(D - 1, 0));
  T* s_cuts           = reinterpret_cast<T*>(s_hist);  // (before the levels) [256]
  int* s_wnew         = s_wbin + (1 << max(D - 1, 0));            // (the next s_wfeat while it is made)
  uint16_t* s_pos     = reinterpret_cast<uint16_t*>(s_wnew + (1 << max(D - 1, 0)));
  unsigned int target = 0;

  // ---- proposals and bins of the block's features
  for (int f = f_first; f < F; f += f_step) {
    T v = static_cast<T>(INFINITY);
    if (tid < S) {
      MinStd eng(static_cast<uint32_t>(p.seed));
      eng.discard(static_cast<unsigned long long>(tid));
      const long long row = eng.uniform_int(0, p.dataset_rows - 1) - p.row_offset;
      v = row >= 0 && row < N ? p.X[row * p.ldx + f] : T(0);
      v = v == v ? v + T(0) : static_cast<T>(INFINITY);  // (-0 becomes +0, or timing would say which of them is kept)
    }
    // sorted by counting, two threads per value
    __syncthreads();
    T* s_sorted = s_cuts + kSmallBins;                              // [256]
    int* s_mark = reinterpret_cast<int*>(s_sorted + kSmallBins);    // [256]
    if (tid < kSmallBins) {
      s_cuts[tid] = v;
      s_mark[tid] = 0;
    }
    __syncthreads();
    {
      const T mine     = s_cuts[tid >> 1];
      constexpr int kPer = 16 / sizeof(T);
      const int n_vec  = (S + 2 * kPer - 1) / (2 * kPer);  // 16-byte words of a half
      int below        = CountBelow(s_cuts + (tid & 1) * n_vec * kPer, n_vec, mine);
      below += __shfl_xor_sync(0xffffffffu, below, 1);
      if ((tid & 1) == 0 && (tid >> 1) < S) {
        s_sorted[below] = mine;
        s_mark[below]   = 1;
      }
    }
    __syncthreads();
    const bool keep  = tid < S && s_mark[tid] != 0;
    const unsigned m = __ballot_sync(0xffffffffu, keep);
    if (lane == 0) s_cnt[warp] = __popc(m);
    if (keep) v = s_sorted[tid];
    __syncthreads();
    int pos = __popc(m & ((1u << lane) - 1u)), count = 0;
    for (int w = 0; w < kSmallWarps; ++w) {
      if (w < warp) pos += s_cnt[w];
      count += s_cnt[w];
    }
    if (keep) s_cuts[pos] = pos == count - 1 ? static_cast<T>(INFINITY) : v;
    __syncthreads();
    if (part == 0) {
      for (int i = tid; i < count; i += kSmallThreads) p.cuts[static_cast<int64_t>(f) * S + i] = s_cuts[i];
      if (tid == 0) p.counts[f] = count;
    }
    // bin = first proposal >= x; the part's share of the rows
    for (int row0 = part * kSmallThreads + tid; row0 < N; row0 += 4 * p.parts * kSmallThreads) {
      T x[4];
      int b[4] = {0, 0, 0, 0};
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int row = row0 + e * p.parts * kSmallThreads;
        x[e]          = row < N ? p.X[row * p.ldx + f] : T(0);
      }
      for (int len = count; len > 1;) {
        const int half = len >> 1;
#pragma unroll
        for (int e = 0; e < 4; ++e)
          if (s_cuts[b[e] + half - 1] < x[e]) b[e] += half;
        len -= half;
      }
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int row = row0 + e * p.parts * kSmallThreads;
        if (row < N) p.bins_t[static_cast<int64_t>(f) * p.pitch + row] = static_cast<uint8_t>(b[e] + (s_cuts[b[e]] < x[e] ? 1 : 0));
      }
    }
    __syncthreads();
  }

  // ---- the quantiser's scale: |g| and |h| sums of all rows
  {
    const int64_t n = static_cast<int64_t>(N) * K;
    const int n_chunks = static_cast<int>((n + kSumBlock - 1) / kSumBlock);
    const int grp = tid / kSumThreads, t = tid % kSumThreads;
    double* s_part = reinterpret_cast<double*>(s_hist);  // [2][n_chunks]
    for (int c0 = 0; c0 < n_chunks; c0 += 2) {
      double sg = 0.0, sh = 0.0;
#pragma unroll 4
      for (int j = 0; j < kSumItems; ++j) {
        const int64_t idx = static_cast<int64_t>(c0 + grp) * kSumBlock + j * kSumThreads + t;
        double vg = 0.0, vh = 0.0;
        if (idx < n) {
          const int row    = static_cast<int>(K == 1 ? idx : idx / K);
          const double2 gh = SmallGradient<kForm>(p, row, static_cast<int>(idx - static_cast<int64_t>(row) * K));
          vg               = fabs(gh.x);
          vh               = fabs(gh.y);
        }
        sg += vg;
        sh += vh;
      }
      FoldAbsSums(sg, sh, t, s_sum[grp]);
      __syncthreads();
      if (t == 0 && c0 + grp < n_chunks) {
        double tg, th;
        JoinAbsSums(s_sum[grp], tg, th);
        s_part[c0 + grp]            = tg;
        s_part[n_chunks + c0 + grp] = th;
      }
      __syncthreads();
    }
    // at most 4096 partial sums are left: one more step of the same order (none if there is one)
    double tg = n_chunks > 0 ? s_part[0] : 0.0, th = n_chunks > 0 ? s_part[n_chunks] : 0.0;
    if (n_chunks > 1) {
      double sg = 0.0, sh = 0.0;
      if (grp == 0) {
        for (int j = 0; j < kSumItems; ++j) {
          const int i = j * kSumThreads + t;
          sg += i < n_chunks ? s_part[i] : 0.0;
          sh += i < n_chunks ? s_part[n_chunks + i] : 0.0;
        }
      }
      FoldAbsSums(sg, sh, t, s_sum[grp]);
      __syncthreads();
      if (tid == 0) JoinAbsSums(s_sum[0], tg, th);
    }
    if (tid == 0) s_qp = MakeScale(tg, th);
    __syncthreads();
  }
  const QuantParams qp = s_qp;

  // ---- quantised pairs of a slice of the rows, and the slice's sums
  {
    const int per = (N + n_blocks - 1) / n_blocks;
    const int r0 = min(N, block * per), r1 = min(N, r0 + per);
    long long* s_root = reinterpret_cast<long long*>(s_hist);  // [K][2]
    for (int i = tid; i < 2 * K; i += kSmallThreads) s_root[i] = 0;
    __syncthreads();
    for (int i0 = r0 * K + warp * 32; i0 < r1 * K; i0 += kSmallThreads) {
      const int i   = i0 + lane;
      const int row = i / K, k = i - row * K;
      long long qg = 0, qh = 0;
      if (i < r1 * K) {
        const double2 gh = SmallGradient<kForm>(p, row, k);
        const int2 q     = QuantisePair(gh.x, gh.y, qp, HashCombine(static_cast<long long>(p.seed), p.row_offset + row, k));
        p.pairs[i]       = q;
        qg               = q.x;
        qh               = q.y;
      }
      if (K == 1) {  // (one address for all lanes: one pair of atomics per warp)
        for (int off = 16; off >= 1; off >>= 1) {
          qg += __shfl_down_sync(0xffffffffu, qg, off);
          qh += __shfl_down_sync(0xffffffffu, qh, off);
        }
      }
      if (K == 1 ? lane == 0 : i < r1 * K) {
        atomicAdd(reinterpret_cast<unsigned long long*>(s_root + 2 * k), static_cast<unsigned long long>(qg));
        atomicAdd(reinterpret_cast<unsigned long long*>(s_root + 2 * k + 1), static_cast<unsigned long long>(qh));
      }
    }
    __syncthreads();
    for (int k = tid; k < K; k += kSmallThreads)
      p.root_part[static_cast<int64_t>(block) * K + k] = GPairI64{s_root[2 * k], s_root[2 * k + 1]};
  }
  // cleared outputs; the nodes that split are written over below, after the barrier.  The values and the rows' nodes
  // too: if a barrier gives up, the kernels that are queued behind this one still find nodes of the tree, with value 0.
  for (int i = block * kSmallThreads + tid; i < p.tree.max_nodes; i += n_blocks * kSmallThreads) {
    p.tree.feature[i]     = -1;
    p.tree.split_value[i] = 0.0;
    p.tree.gain[i]        = 0.0;
    for (int k = 0; k < K; ++k) {
      p.tree.node_sums[static_cast<int64_t>(i) * K + k]  = GPairI64{0, 0};
      p.tree.leaf_value[static_cast<int64_t>(i) * K + k] = p.hessian[static_cast<int64_t>(i) * K + k] = 0.0;
    }
  }
  if (p.leaf != nullptr)
    for (int row = block * kSmallThreads + tid; row < N; row += n_blocks * kSmallThreads) p.leaf[row] = 0;
  target += n_blocks;
  if (!GridBarrier(p.barrier, target, p.status, &s_ok)) return;

  // ---- root: sums, positions; where each feature's bins begin in the order of all bins
  for (int k = warp; k < K; k += kSmallWarps) {
    GPairI64 s{0, 0};
    for (int b = lane; b < n_blocks; b += 32) {
      const GPairI64 v = LoadPairStreaming(p.root_part + static_cast<int64_t>(b) * K + k);
      s.grad += v.grad;
      s.hess += v.hess;
    }
    for (int off = 16; off >= 1; off >>= 1) {
      s.grad += __shfl_xor_sync(0xffffffffu, s.grad, off);
      s.hess += __shfl_xor_sync(0xffffffffu, s.hess, off);
    }
    if (lane == 0) {
      s_nodes[k] = s;
      if (block == 0) p.tree.node_sums[k] = s;
    }
  }
  for (int row = tid; row < N; row += kSmallThreads) s_pos[row] = 0;
  {
    // one warp scans the counts
    if (warp == kSmallWarps - 1) {
      int carry = 0;
      for (int base = 0; base < F; base += 32) {
        const int f = base + lane;
        int incl    = f < F ? __ldcg(p.counts + f) : 0;
        for (int off = 1; off < 32; off <<= 1) {
          const int v = __shfl_up_sync(0xffffffffu, incl, off);
          if (lane >= off) incl += v;
        }
        if (f < F) s_rp[f + 1] = carry + incl;
        carry += __shfl_sync(0xffffffffu, incl, 31);
      }
      if (lane == 0) s_rp[0] = 0;
      if (lane == 0 && block == 0 && p.info_host != nullptr) *static_cast<volatile int32_t*>(p.info_host) = carry;
    }
    if (tid == 0) s_wfeat[0] = 0;
  }
  __syncthreads();

  const double l1 = p.l1, reg = fmax(1e-5, p.l2), msg = p.msg;
  const bool plain = GainsArePlain(qp, l1, reg);
  for (int depth = 0; depth < D; ++depth) {
    const int begin = (1 << depth) - 1, nodes = 1 << depth;
    const bool derive = depth > 0, write_hist = depth < D - 1;
    const int units = derive ? nodes / 2 : 1;
    SmallCand* cand     = p.cand + static_cast<int64_t>(SmallCandBegin(depth, D)) * F;
    GPairI64* cand_left = p.cand_left + static_cast<int64_t>(SmallCandBegin(depth, D)) * F * K;
    // (read behind the next barrier of the block)
    for (int i = tid; i < nodes * K; i += kSmallThreads) s_terms[i] = TermsOf(s_nodes[i], qp, l1, reg);
    // (s_wfeat still holds the winners of the level above: unit u exists if node u there was split)
    for (int f = f_first; f < F; f += f_step) {
      const bool search = p.feature_set == nullptr || p.feature_set[f] != 0;
      const int nb      = s_rp[f + 1] - s_rp[f];
      const uint8_t* bins = p.bins_t + static_cast<int64_t>(f) * p.pitch;
      GPairI64* hist_f      = p.hist[depth & 1] + static_cast<int64_t>(f) * nodes * K * kSmallBins;
      const GPairI64* par_f = p.hist[(depth & 1) ^ 1] + static_cast<int64_t>(f) * (nodes / 2) * K * kSmallBins;
      // the part's units, max_slots at a time: unit = part + (c0 + slot) * parts
      const int my_units = units > part ? (units - part + p.parts - 1) / p.parts : 0;
      for (int c0 = 0; c0 < my_units; c0 += p.max_slots) {
        const int slots = min(p.max_slots, my_units - c0);
        for (int k = 0; k < K; ++k) {
          for (int i = tid; i < slots * kSmallBins; i += kSmallThreads) reinterpret_cast<int4*>(s_hist)[i] = make_int4(0, 0, 0, 0);
          if (k == 0 && K > 1)
            for (int i = tid; i < slots * 2 * kSmallBins; i += kSmallThreads) s_gain[i] = 0.0;
          __syncthreads();
          // rows of the built nodes, four per thread at a time so that their loads overlap
          for (int row0 = tid; row0 < N; row0 += 4 * kSmallThreads) {
            int slot[4];
            int2 q[4];
            int bin[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              const int row = row0 + e * kSmallThreads;
              const int j   = row < N ? static_cast<int>(s_pos[row]) - begin : -1;
              const int u   = derive ? j >> 1 : 0;
              slot[e]       = (u >> p.part_shift) - c0;
              if (j < 0 || (u & (p.parts - 1)) != part || slot[e] < 0 || slot[e] >= slots) slot[e] = -1;
              if (slot[e] >= 0 && derive) {
                const bool left = s_nodes[static_cast<int64_t>(2 * u) * K].hess < s_nodes[static_cast<int64_t>(2 * u + 1) * K].hess;
                if (left != ((j & 1) == 0)) slot[e] = -1;
              }
              if (slot[e] >= 0) {
                q[e]   = p.pairs[static_cast<int64_t>(row) * K + k];
                bin[e] = bins[row];
              }
            }
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              if (slot[e] < 0) continue;
              int* dst = s_hist + slot[e] * 4 * kSmallBins + bin[e];
              atomicAdd(dst, q[e].x >> 16);
              atomicAdd(dst + kSmallBins, q[e].x & 0xffff);
              atomicAdd(dst + 2 * kSmallBins, q[e].y >> 16);
              atomicAdd(dst + 3 * kSmallBins, q[e].y & 0xffff);
            }
          }
          __syncthreads();
          // What a unit's scan needs of it.  _a: the built node, _b: its sibling.
          struct Unit {
            bool here, scanned, eval_a, eval_b;
            int ja, jb, u;
          };
          auto unit_of = [&](int i) {
            Unit n;
            n.u             = part + (c0 + i) * p.parts;
            n.here          = i < slots && (!derive || s_wfeat[n.u] >= 0);  // node u of the level above was split
            const bool left = n.here && derive && s_nodes[static_cast<int64_t>(2 * n.u) * K].hess < s_nodes[static_cast<int64_t>(2 * n.u + 1) * K].hess;
            n.ja            = n.here && derive ? 2 * n.u + (left ? 0 : 1) : 0;
            n.jb            = n.here && derive ? 2 * n.u + (left ? 1 : 0) : 0;
            n.eval_a        = n.here && search && s_nodes[static_cast<int64_t>(n.ja) * K].hess > 0;
            n.eval_b        = n.here && search && derive && s_nodes[static_cast<int64_t>(n.jb) * K].hess > 0;
            n.scanned       = s_nodes[static_cast<int64_t>(n.ja) * K + k].hess > 0;
            return n;
          };
          // The candidate of node j, by the lanes of a warp: `best` is the same in all of them.
          auto write_cand = [&](int j, const SmallCand& best) {
            const int64_t at = static_cast<int64_t>(j) * F + f;
            if (lane == 0) cand[at] = best;
            if (K > 1 && best.bin >= 0)  // (written by threads of this block, before the barrier)
              for (int kk = lane; kk < K; kk += 32)
                StorePair(cand_left + at * K + kk, LoadPairStreaming(hist_f + (static_cast<int64_t>(j) * K + kk) * kSmallBins + best.bin));
          };
          if (slots <= 2) {
            // a thread per bin, both units at a time
            const int grp = tid / kSmallBins, b = tid % kSmallBins, gw = warp % (kSmallWarps / 2);
            const int i   = grp;
            const Unit n  = unit_of(i);
            const bool in = n.here && b < nb;
            const int64_t at_a = (static_cast<int64_t>(n.ja) * K + k) * kSmallBins + b, at_b = (static_cast<int64_t>(n.jb) * K + k) * kSmallBins + b;
            const int* hs      = s_hist + i * 4 * kSmallBins;
            double* gains      = s_gain + i * 2 * kSmallBins;
            GPairI64 va{0, 0}, vb{0, 0};
            double ga = 0.0, gb = 0.0;
            if (in) {
              if (derive && n.scanned) vb = LoadPairStreaming(par_f + (static_cast<int64_t>(n.u) * K + k) * kSmallBins + b);
              va.grad = static_cast<long long>(hs[b]) * 65536 + static_cast<unsigned>(hs[kSmallBins + b]);
              va.hess = static_cast<long long>(hs[2 * kSmallBins + b]) * 65536 + static_cast<unsigned>(hs[3 * kSmallBins + b]);
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
            if (lane == 31) s_tot[grp][gw] = GPairI64{sg, sh};
            __syncthreads();
#pragma unroll
            for (int w = 0; w < kSmallWarps / 2 - 1; ++w) {
              if (w < gw) {
                const GPairI64 t = s_tot[grp][w];
                sg += t.grad;
                sh += t.hess;
              }
            }
            if (in) {
              if (n.scanned && (sg > 0 || sh > 0)) va = GPairI64{sg, sh};
              vb = n.scanned && derive ? GPairI64{vb.grad - va.grad, vb.hess - va.hess} : GPairI64{0, 0};
              if (write_hist || K > 1) {
                StorePair(hist_f + at_a, va);
                if (derive) StorePair(hist_f + at_b, vb);
              }
            }
            unsigned ok_a = n.eval_a && in ? 1u : 0u, ok_b = n.eval_b && in ? 1u : 0u;
            if (K > 1 && in) {  // the gains so far are in shared memory, -1e300 = a side without hessian
              ga = gains[b];
              gb = gains[kSmallBins + b];
              if (ga < -1e299) ok_a = 0u;
              if (gb < -1e299) ok_b = 0u;
            }
            if (__any_sync(0xffffffffu, ok_a | ok_b))
              AddGains(va, ok_a, s_terms[static_cast<int64_t>(n.ja) * K + k], ga, vb, ok_b, s_terms[static_cast<int64_t>(n.jb) * K + k], gb, qp, l1, reg, msg, plain);
            if (k < K - 1) {
              if (in) {
                gains[b]              = ok_a ? ga : -1e300;
                gains[kSmallBins + b] = ok_b ? gb : -1e300;
              }
            } else {
              // the best bin of either node: of the warp, then of the unit's eight warps
              const double gain_a = ok_a && ga > 0 ? ga : 0.0, gain_b = ok_b && gb > 0 ? gb : 0.0;
              const int bin_a = WarpBest(gain_a, s_rp[f] + b), bin_b = derive ? WarpBest(gain_b, s_rp[f] + b) : -1;
              if (bin_a < 0 ? lane == 0 : bin_a == s_rp[f] + b) s_best[grp][0][gw] = SmallCand{gain_a, bin_a < 0 ? -1 : b, 0, va};
              if (bin_b < 0 ? lane == 0 : bin_b == s_rp[f] + b) s_best[grp][1][gw] = SmallCand{gain_b, bin_b < 0 ? -1 : b, 0, vb};
              __syncthreads();
              if (n.here && gw < (derive ? 2 : 1)) {  // a warp per node
                const SmallCand mine = s_best[grp][gw][lane % (kSmallWarps / 2)];
                const int best       = WarpBest(lane < kSmallWarps / 2 && mine.bin >= 0 ? mine.gain : 0.0, s_rp[f] + mine.bin);
                const int from       = best < 0 ? 0 : (best - s_rp[f]) / 32;  // the warp that has the bin
                write_cand(gw == 0 ? n.ja : n.jb, s_best[grp][gw][from]);
              }
            }
          } else {
            // A warp per unit.  The four words of the bins become their prefix sums where they lie (at most sums of all rows, which
            // fit 32 bits): a lane adds up eight neighbouring bins; then the lanes take the bins 32 at a time.
            for (int i = warp; i < slots; i += kSmallWarps) {
              const Unit n = unit_of(i);
              if (!n.here) continue;
              int* hs = s_hist + i * 4 * kSmallBins;
#pragma unroll
              for (int word = 0; word < 4; ++word) {
                int4* at = reinterpret_cast<int4*>(hs + word * kSmallBins) + 2 * lane;
                int4 x = at[0], y = at[1];
                x.y += x.x;
                x.z += x.y;
                x.w += x.z;
                y.x += x.w;
                y.y += y.x;
                y.z += y.y;
                y.w += y.z;
                int incl = y.w;
#pragma unroll
                for (int off = 1; off < 32; off <<= 1) {
                  const int v = __shfl_up_sync(0xffffffffu, incl, off);
                  if (lane >= off) incl += v;
                }
                const int before = incl - y.w;
                at[0]     = make_int4(x.x + before, x.y + before, x.z + before, x.w + before);
                at[1]     = make_int4(y.x + before, y.y + before, y.z + before, y.w + before);
              }
              __syncwarp();
              const NodeTerms ta = s_terms[static_cast<int64_t>(n.ja) * K + k], tb = s_terms[static_cast<int64_t>(n.jb) * K + k];
              double* gains      = s_gain + i * 2 * kSmallBins;
              auto prefix        = [&](int b) {
                return GPairI64{static_cast<long long>(hs[b]) * 65536 + static_cast<unsigned>(hs[kSmallBins + b]),
                                static_cast<long long>(hs[2 * kSmallBins + b]) * 65536 + static_cast<unsigned>(hs[3 * kSmallBins + b])};
              };
              SmallCand best_a{0.0, -1, 0, GPairI64{0, 0}}, best_b = best_a;
              auto parent_of = [&](int b) {
                return derive && n.scanned && b < nb ? LoadPairStreaming(par_f + (static_cast<int64_t>(n.u) * K + k) * kSmallBins + b) : GPairI64{0, 0};
              };
              GPairI64 ahead = parent_of(lane);
              for (int b0 = 0; b0 < nb; b0 += 32) {
                const int b   = b0 + lane;
                const bool in = b < nb;
                GPairI64 va = prefix(b), vb = ahead;
                ahead = parent_of(b + 32);
                if (!(n.scanned && (va.grad > 0 || va.hess > 0)) && b > 0) {  // the bin itself
                  const GPairI64 before = prefix(b - 1);
                  va = GPairI64{va.grad - before.grad, va.hess - before.hess};
                }
                vb = n.scanned && derive ? GPairI64{vb.grad - va.grad, vb.hess - va.hess} : GPairI64{0, 0};
                if (in && (write_hist || K > 1)) {
                  StorePair(hist_f + (static_cast<int64_t>(n.ja) * K + k) * kSmallBins + b, va);
                  if (derive) StorePair(hist_f + (static_cast<int64_t>(n.jb) * K + k) * kSmallBins + b, vb);
                }
                unsigned ok_a = n.eval_a && in ? 1u : 0u, ok_b = n.eval_b && in ? 1u : 0u;
                double ga = 0.0, gb = 0.0;
                if (K > 1) {
                  ga = gains[b];
                  gb = gains[kSmallBins + b];
                  if (ga < -1e299) ok_a = 0u;
                  if (gb < -1e299) ok_b = 0u;
                }
                if (__any_sync(0xffffffffu, ok_a | ok_b)) AddGains(va, ok_a, ta, ga, vb, ok_b, tb, gb, qp, l1, reg, msg, plain);
                if (k < K - 1) {
                  if (in) {
                    gains[b]              = ok_a ? ga : -1e300;
                    gains[kSmallBins + b] = ok_b ? gb : -1e300;
                  }
                  continue;
                }
                auto better = [&](double gain, const SmallCand& best) {
                  return gain > 0 && Better(Cand{gain, s_rp[f] + b, f}, Cand{best.gain, best.bin < 0 ? -1 : s_rp[f] + best.bin, f});
                };
                if (ok_a && better(ga, best_a)) best_a = SmallCand{ga, b, 0, va};
                if (ok_b && better(gb, best_b)) best_b = SmallCand{gb, b, 0, vb};
              }
              if (k < K - 1) continue;
              __syncwarp();  // (the level's histogram is read again with several outputs)
#pragma unroll
              for (int side = 0; side < 2; ++side) {
                if (side == 1 && !derive) continue;
                SmallCand best  = side == 0 ? best_a : best_b;
                const int bin   = WarpBest(best.bin >= 0 ? best.gain : 0.0, s_rp[f] + best.bin);
                const unsigned holder = __ballot_sync(0xffffffffu, bin >= 0 && best.bin >= 0 && s_rp[f] + best.bin == bin);
                const int from        = holder != 0u ? __ffs(holder) - 1 : 0;
                best.gain      = bin < 0 ? 0.0 : __shfl_sync(0xffffffffu, best.gain, from);
                best.left.grad = __shfl_sync(0xffffffffu, best.left.grad, from);
                best.left.hess = __shfl_sync(0xffffffffu, best.left.hess, from);
                best.bin       = bin < 0 ? -1 : bin - s_rp[f];
                write_cand(side == 0 ? n.ja : n.jb, best);
              }
            }
          }
          __syncthreads();
        }
      }
    }
    target += n_blocks;
    if (!GridBarrier(p.barrier, target, p.status, &s_ok)) return;

    // ---- winners of the level: a warp per node picks, the next node's candidates already on their way
    const int words = derive ? nodes : 1;
    auto exists = [&](int j) { return j < words && (!derive || s_wfeat[j >> 1] >= 0) && s_nodes[static_cast<int64_t>(j) * K].hess > 0; };
    auto cand_of = [&](int j, int f) {
      SmallCand c{0.0, -1, 0, GPairI64{0, 0}};
      if (exists(j) && f < F) {
        const int4* at = reinterpret_cast<const int4*>(cand + static_cast<int64_t>(j) * F + f);
        const int4 raw = __ldcg(at);
        if (K == 1) c.left = LoadPairStreaming(reinterpret_cast<const GPairI64*>(at + 1));
        c.gain = __hiloint2double(raw.y, raw.x);
        c.bin  = raw.z;
      }
      return c;
    };
    // the sums of the children of node j
    auto set_children = [&](int j, int k, bool split, const GPairI64& left) {
      GPairI64 ls{0, 0}, rs{0, 0};
      if (split) {
        const GPairI64 ns = s_nodes[static_cast<int64_t>(j) * K + k];
        ls                = left;
        rs                = GPairI64{ns.grad - ls.grad, ns.hess - ls.hess};
        if (block == 0) {
          const int node = begin + j;
          StorePair(p.tree.node_sums + static_cast<int64_t>(2 * node + 1) * K + k, ls);
          StorePair(p.tree.node_sums + static_cast<int64_t>(2 * node + 2) * K + k, rs);
        }
      }
      if (depth < D - 1) {
        s_next[static_cast<int64_t>(2 * j) * K + k]     = ls;
        s_next[static_cast<int64_t>(2 * j + 1) * K + k] = rs;
      }
    };
    SmallCand ahead = cand_of(warp, lane);
    for (int j = warp; j < words; j += kSmallWarps) {
      SmallCand mine = ahead;
      int feature    = lane;
      ahead          = cand_of(j + kSmallWarps, lane);
      for (int f = lane + 32; f < F; f += 32) {
        const SmallCand c = cand_of(j, f);
        if (c.bin >= 0 && (mine.bin < 0 || Better(Cand{c.gain, s_rp[f] + c.bin, f}, Cand{mine.gain, s_rp[feature] + mine.bin, feature}))) {
          mine    = c;
          feature = f;
        }
      }
      const int own = mine.bin >= 0 ? s_rp[feature] + mine.bin : -1;
      const int bin = WarpBest(mine.bin >= 0 ? mine.gain : 0.0, own);
      const unsigned holder = __ballot_sync(0xffffffffu, bin >= 0 && own == bin);
      const int from        = holder != 0u ? __ffs(holder) - 1 : 0;
      const bool split      = bin >= 0 && __shfl_sync(0xffffffffu, mine.gain, from) > 1e-5;
      if (lane == from) {
        s_wbin[j] = split ? mine.bin : -1;
        s_wnew[j] = split ? feature : -1;
        if (K == 1) set_children(j, 0, split, mine.left);
        if (split && block == 0) {
          p.tree.feature[begin + j]     = feature;
          p.tree.split_value[begin + j] = static_cast<double>(p.cuts[static_cast<int64_t>(feature) * S + mine.bin]);
          p.tree.gain[begin + j]        = mine.gain;
        }
      }
    }
    __syncthreads();
    if (K > 1) {
      for (int i = tid; i < words * K; i += kSmallThreads) {
        const int j = i / K, k = i - j * K, wf = s_wnew[j];
        set_children(j, k, wf >= 0, wf >= 0 ? LoadPairStreaming(cand_left + (static_cast<int64_t>(j) * F + wf) * K + k) : GPairI64{0, 0});
      }
    }
    for (int j = tid; j < words; j += kSmallThreads) s_wfeat[j] = s_wnew[j];
    __syncthreads();
    // ---- rows move down; a row whose node did not split stays where it is
    for (int row0 = tid; row0 < N; row0 += 4 * kSmallThreads) {
      int bin[4], j[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int row = row0 + e * kSmallThreads;
        j[e]          = row < N ? static_cast<int>(s_pos[row]) - begin : -1;
        const int wf  = j[e] >= 0 ? s_wfeat[j[e]] : -1;
        if (wf < 0) j[e] = -1;
        else bin[e] = p.bins_t[static_cast<int64_t>(wf) * p.pitch + row];
      }
#pragma unroll
      for (int e = 0; e < 4; ++e)
        if (j[e] >= 0)
          s_pos[row0 + e * kSmallThreads] = static_cast<uint16_t>(2 * (begin + j[e]) + 1 + (bin[e] > s_wbin[j[e]] ? 1 : 0));
    }
    GPairI64* t = s_nodes;
    s_nodes     = s_next;
    s_next      = t;
    __syncthreads();
  }

  // ---- leaf values and hessians, the node of every row, the prediction
  target += n_blocks;
  if (!GridBarrier(p.barrier, target, p.status, &s_ok)) return;
  for (int i = block * kSmallThreads + tid; i < p.tree.max_nodes * K; i += n_blocks * kSmallThreads) {
    const int node   = i / K;
    const GPairF64 s = Dequantise(LoadPairStreaming(p.tree.node_sums + i), qp);
    p.hessian[i]     = s.hess;
    const bool here  = node == 0 || __ldcg(p.tree.feature + (node - 1) / 2) >= 0;
    p.tree.leaf_value[i] = here ? CalculateLeafValue(s.grad, s.hess, l1, p.l2) : 0.0;
  }
  const int per = (N + n_blocks - 1) / n_blocks;
  const int r0 = min(N, block * per), r1 = min(N, r0 + per);
  if (p.leaf != nullptr)
    for (int row = r0 + tid; row < r1; row += kSmallThreads) p.leaf[row] = s_pos[row];
  if (kForm != kGiven && p.objective >= 0) {
    for (int i = r0 * K + tid; i < r1 * K; i += kSmallThreads) {
      const int row = i / K, k = i - row * K;
      const GPairF64 s = Dequantise(LoadPairStreaming(p.tree.node_sums + static_cast<int64_t>(s_pos[row]) * K + k), qp);
      p.pred[i] += CalculateLeafValue(s.grad, s.hess, l1, p.l2);
    }
  }
}

}  // namespace

// The shapes this form takes, and how it is cut: nothing is launched.
struct SmallPlan {
  int blocks, parts, max_slots;
  size_t smem;
};

// Is this form faster than the general path?  A block passes over all rows for every feature, output and chunk of pairs of
// nodes that it has, and takes the pairs in turns; the general path pays for launches, whatever they do, and a little for
// bins and rows.  Fitted to 318 shapes of both (microseconds for three rounds; what the histograms' memory costs is the same
// on either side), before the general path's launches were chained (LaunchChained), which took a third of what a level costs
// whatever it holds: with that third less, 31 shapes on either side of the line are told right or are within 2 %.  General and small,
// microseconds for five rounds: 20k rows x 30, depth 6 1013 and 1035, 10k x 30 992 and 770; 16k x 100, depth 8 1584 and 1775, 6k x 100 1605 and
// 1435; 8k x 200, depth 6 1157 and 1235, 2k x 200 1195 and 978; three classes, 3k x 50, depth 6 1377 and 1205; ten classes, 1500 x 40,
// depth 6 1650 and 2075.
static bool SmallPays(const SmallPlan& plan, int64_t N, int F, int K, int D)
{
  int64_t passes = 0, turns = 0;
  auto turns_of  = [](int64_t slots) { return slots > 2 ? (slots + kSmallWarps - 1) / kSmallWarps : int64_t{1}; };
  for (int d = 0; d < D; ++d) {
    const int64_t units = d == 0 ? 1 : int64_t{1} << (d - 1), mine = (units + plan.parts - 1) / plan.parts;
    const int64_t whole = mine / plan.max_slots, rest = mine - whole * plan.max_slots;
    passes += whole + (rest > 0 ? 1 : 0);
    turns += whole * turns_of(plan.max_slots) + (rest > 0 ? turns_of(rest) : 0);
  }
  const int abreast  = plan.blocks / plan.parts;  // features that are worked on at a time
  const double each  = static_cast<double>((F + abreast - 1) / abreast) * K;
  const double small = each * (2.4e-3 * static_cast<double>(passes * N) + 20.0 * static_cast<double>(turns) - 9.0 * D);
  const double general = D * (49.0 + 5.0 * K + (K > 1 ? 7.0 : 0.0) + 3.4e-6 * static_cast<double>(N) * F * K);
  return small <= general;
}

static bool PlanSmall(lbk_context* ctx, int64_t N, int F, int K, int D, int S, SmallPlan& plan)
{
  // One-byte bins; 16-bit node ids; the canonical sum's second step in one piece; the range that SmallPays was measured over.
  if (S > kSmallBins || D < 1 || D > 12 || N < 1 || N > kSmallMaxRows || N * K > 2 * kSmallMaxRows || F > 4 * ctx->sm_count) return false;
  const int64_t level = int64_t{1} << (D - 1);
  if (level * K > 1536) return false;
  const int64_t hist_bytes = (K > 1 ? level * 3 / 2 + 1 : level) * F * K * kSmallBins * 16;
  if (hist_bytes > (int64_t{256} << 20)) return false;
  // several blocks per feature: they share its node pairs on the deeper levels and its rows for the binning
  plan.parts  = static_cast<int>(std::min<int64_t>(std::max(1, ctx->sm_count / F), std::max<int64_t>({level / 2, N / 2048, 1})));
  while (plan.parts & (plan.parts - 1)) plan.parts &= plan.parts - 1;  // a power of two
  plan.blocks = F <= ctx->sm_count ? F * plan.parts : ctx->sm_count;
  const size_t fixed = (2 * sizeof(GPairI64) + sizeof(NodeTerms)) * std::max<int64_t>(1, level * K) + sizeof(int) * (F + 1 + 3 * level) + 2 * N + 64;
  const size_t slot  = 4 * kSmallBins * sizeof(int) + (K > 1 ? 2 * kSmallBins * sizeof(double) : 0);
  const size_t room  = static_cast<size_t>(ctx->max_smem_optin) - 4096;
  if (fixed + slot > room) return false;
  const int64_t units = std::max<int64_t>(1, level / 2);
  plan.max_slots      = static_cast<int>(std::min<int64_t>((units + plan.parts - 1) / plan.parts, (room - fixed) / slot));
  plan.max_slots      = std::max(plan.max_slots, 1);
  if (plan.max_slots > kSmallWarps) plan.max_slots = plan.max_slots / kSmallWarps * kSmallWarps;  // (a warp per unit: whole turns)
  // (the proposals, three arrays of kSmallBins, begin where the histograms do and may reach beyond them)
  plan.smem = std::max(fixed + plan.max_slots * slot, kSmallBins * size_t{2 * 8 + 4});
  // (the partial sums, the proposals and the root sums share the histograms' place)
  const size_t early = std::max({size_t{2} * ((N * K + kSumBlock - 1) / kSumBlock) * 8, kSmallBins * size_t{8}, size_t{16} * K});
  if (early > plan.max_slots * slot) return false;
  return SmallPays(plan, N, F, K, D);
}

bool SmallTreeFits(lbk_context* ctx, int64_t N, int F, int K, int D, int S)
{
  SmallPlan plan;
  return PlanSmall(ctx, N, F, K, D, S, plan);
}

template <typename T>
void SmallTree(lbk_context* ctx, Scratch& s, const SmallTreeArgs<T>& a, cudaStream_t stream)
{
  SmallPlan plan;
  LBK_EXPECT(PlanSmall(ctx, a.N, a.F, a.K, a.D, a.S, plan), "shape outside the small form");
  const int N = static_cast<int>(a.N), F = a.F, K = a.K, D = a.D;
  const int64_t level = int64_t{1} << (D - 1);
  SmallParams<T> p{};
  p.X = a.X;
  p.ldx = a.ldx;
  p.N = N;
  p.F = F;
  p.K = K;
  p.D = D;
  p.S = a.S;
  p.seed = a.seed;
  p.parts = plan.parts;
  while ((2 << p.part_shift) <= p.parts) ++p.part_shift;
  p.row_offset = a.row_offset;
  p.dataset_rows = a.dataset_rows;
  p.g = a.g;
  p.h = a.h;
  p.ldg = a.ldg;
  p.objective = a.objective;
  p.y = a.y;
  p.pred = a.pred;
  p.lr = a.lr;
  p.l1 = a.sp.l1;
  p.l2 = a.sp.l2;
  p.msg = a.sp.min_split_gain;
  p.feature_set = a.sp.feature_set;
  p.tree = a.tree;
  p.hessian = a.hessian;
  p.leaf = a.leaf;
  p.cuts = s.alloc<T>(static_cast<size_t>(F) * a.S);
  p.counts = s.alloc<int32_t>(F);
  p.pitch = (N + 31) / 32 * 32;
  p.bins_t = s.alloc<uint8_t>(static_cast<size_t>(F) * p.pitch);
  p.pairs = s.alloc<int2>(static_cast<size_t>(N) * K);
  p.root_part = s.alloc<GPairI64>(static_cast<size_t>(plan.blocks) * K);
  // level d's histograms are written for d < D - 1 (every level with several outputs: the left sums are read
  // back from them)
  const int64_t top = K > 1 ? level : std::max<int64_t>(level / 2, 1), below = std::max<int64_t>(top / 2, 1);
  const int last    = K > 1 ? D - 1 : D - 2;  // the last level written
  p.hist[last & 1]       = s.alloc<GPairI64>(static_cast<size_t>(F) * top * K * kSmallBins);
  p.hist[(last & 1) ^ 1] = s.alloc<GPairI64>(static_cast<size_t>(F) * below * K * kSmallBins);
  p.cand      = s.alloc<SmallCand>(static_cast<size_t>(SmallCandNodes(D)) * F);
  p.cand_left = K > 1 ? s.alloc<GPairI64>(static_cast<size_t>(SmallCandNodes(D)) * F * K) : nullptr;
  p.max_slots = plan.max_slots;
  p.status    = ctx->d_status;
  p.info_host = a.info_host;
  p.barrier   = a.barrier;
  auto fn = K > 1                                ? k_tree_small<T, true, kAnyForm>
            : a.objective < 0                     ? k_tree_small<T, false, kGiven>
            : a.objective == LBK_SQUARED_ERROR    ? k_tree_small<T, false, kSquaredError>
                                                  : k_tree_small<T, false, kAnyForm>;
  AllowSharedMemory(ctx, fn, 2048);
  void* args[] = {&p};
  LBK_CUDA(cudaLaunchCooperativeKernel(reinterpret_cast<const void*>(fn), dim3(plan.blocks), dim3(kSmallThreads), args,
                                       plan.smem, stream));
}

template void SmallTree<float>(lbk_context*, Scratch&, const SmallTreeArgs<float>&, cudaStream_t);
template void SmallTree<double>(lbk_context*, Scratch&, const SmallTreeArgs<double>&, cudaStream_t);

}  // namespace lbk
