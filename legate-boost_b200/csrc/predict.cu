// Ensemble predict: pred[row, :] = sum over trees of leaf_value[leaf reached by row, :].
//
// Reference behaviour restated here: predict_fn, src/models/tree/predict.cu:26-84 - one kernel
// launch per tree, each re-reading and re-writing pred; rows walk from node 0 while
// feature[pos] != -1 (at most 100 steps), going left iff (double)x <= split_value[pos].
//
// Three ways, all of one result: a few rows walk the trees where they lie (k_predict_rows); large ensembles of one output are
// walked on ranks of X (predict_ranked.cu: a pass over X that finds them, and the walks); everything else, and what
// the device declines to rank, is tiled:
//
// Design for B200: one launch for the whole ensemble (after one that packs the trees), everything a step of the walk touches
// lives in shared memory.  The load/store data pipe of the SM is what bounds it (one pass per clock; a 4-byte load of
// a warp is one pass, an 8-byte load two, plus one per bank conflict), so the layouts save passes:
//   * A block owns a tile of rows (one thread per row); every thread stages its own row,
//     feature-major with a pitch of one element per thread, so thread t only ever touches bank
//     t mod 32 whatever feature a tree asks for: the x lookups of a walk never conflict.  Every row
//     of X is read from HBM once (16-byte loads, the rest of a sector comes from L1).
//   * The trees are first packed into records: the splits of the heap, then the feature ids of a node and its
//     two children in one word (10 bits each), then (one output) the bottom level of leaf values.  Two
//     levels of a walk are two split loads, one feature load and two x loads: 5 passes for float32, where
//     {split, feature} nodes of 8 bytes took 6 and conflicted twice as often (24 passes per walk of depth 8
//     against 34).  A walk keeps the shared-memory address of its node: a step is one addition for the
//     left child and one more for the right one, whatever the level (with the position in the level and offsets per
//     level a walk was 120 instructions, and those bound it).
//   * For float32 X a split is a float - "x <= split" with x a float is the same test as "x <= the largest
//     float not above split", so the split is rounded down once at packing time.
//   * At packing time every tree is completed to the depth S of the deepest one: below a leaf
//     the nodes become pass-through nodes (split = +inf) and the leaf's value is copied to the
//     bottom level.  A walk is then exactly S steps with no leaf test, and only the bottom level of leaf
//     values is kept.
//   * Trees are brought into shared memory in groups of up to eight by a producer warp (bulk async copies, two
//     buffers, full and empty mbarriers): no warp waits for another one's walks.  A thread walks the trees
//     of a group as independent chains, which hides the latency that one dependent chain exposes.
//   * With several outputs the leaf values stay in global memory and a warp reads them together: its 32 x K
//     sums are spread over the lanes, output innermost, so that a load covers the K values of three or more
//     rows' leaves as whole pieces of lines.  (A lane reading its own row's K values cost 32 passes per value.)
//   * Predictions are accumulated in float64 in tree order (bit-identical to the reference's
//     tree-by-tree accumulation), transformed and written once.
// A fallback kernel with the nodes in global memory covers shapes whose tile or trees do not fit.
#include <algorithm>

#include "predict.cuh"
#include "predict_sums.h"

namespace lbk {
namespace {

// Nodes of the fallback; `foff` = feature index, or -1 for a leaf
struct Node8 {
  float split;
  int foff;
};
struct Node16 {
  double split;
  int foff;
  int pad;
};
template <typename T>
struct NodeOf {
  using type = Node16;
};
template <>
struct NodeOf<float> {
  using type = Node8;
};

__device__ inline void MakeNode(Node8& n, double split, int foff)
{
  n.split = __double2float_rd(split);  // x <= split  <=>  x <= round-down(split) for float x
  n.foff  = foff;
}
__device__ inline void MakeNode(Node16& n, double split, int foff)
{
  n.split = split;
  n.foff  = foff;
  n.pad   = 0;
}

// Kernels that are queued behind the walk on ranks run where it was declined (PredictRanked); null: always.
__device__ inline bool SkipFor(const int* gate) { return gate != nullptr && *gate == 0; }

// A split node whose children would fall outside the arrays is treated as a leaf, so a walk can
// never leave the tree whatever the input arrays hold.
template <typename NodeT>
__global__ void k_pack_trees(const int* __restrict__ gate, const TreePtrs* __restrict__ trees, int K, int F, NodeT* __restrict__ nodes,
                             double* __restrict__ leaves)
{
  AfterTheKernelBefore();
  if (SkipFor(gate)) return;
  const TreePtrs t = trees[blockIdx.x];
  for (int i = threadIdx.x; i < t.max_nodes; i += blockDim.x) {
    int f = t.feature[i];
    if (2 * i + 2 >= t.max_nodes || f < 0 || f >= F) f = -1;
    NodeT n;
    MakeNode(n, t.split[i], f);
    nodes[t.node_off + i] = n;
  }
  for (int64_t i = threadIdx.x; i < static_cast<int64_t>(t.max_nodes) * K; i += blockDim.x)
    leaves[static_cast<int64_t>(t.node_off) * K + i] = t.leaf[i];
}

// A completed tree of depth S as the tiled kernel reads it.  Nodes are counted from 1: those of level l are
// [2^l, 2^(l + 1)), the children of i are 2 i and 2 i + 1.  Splits [2^S] of T; words with the feature ids of a
// node and its children (used for the nodes of even levels); leaf values [2^S] (one output only).  The parts
// are whole multiples of 16 bytes.
struct TreeRecord {
  int S;
  int split_bytes, word_bytes, leaf_bytes, bytes;
};
constexpr int kIdBits     = 10;  // feature ids in a word: three of them
constexpr int kMaxFeature = 1 << kIdBits;
static TreeRecord RecordOf(int S, size_t elem, int leaf_values /* of a leaf; 0: they are elsewhere */)
{
  auto up16 = [](int v) { return (v + 15) / 16 * 16; };
  TreeRecord r;
  r.S           = S;
  r.split_bytes = up16((1 << S) * static_cast<int>(elem));
  r.word_bytes  = up16((S > 0 ? 2 << ((S - 1) / 2 * 2) : 0) * 4);
  r.leaf_bytes  = up16((1 << S) * 8 * leaf_values);
  r.bytes       = r.split_bytes + r.word_bytes + r.leaf_bytes;
  return r;
}

// One block packs one tree.  A node whose children would fall outside the input arrays, or whose feature
// id is outside [0, F), counts as a leaf, so a walk can never leave the arrays.
template <typename T>
__global__ void k_pack_complete(const int* __restrict__ gate, const TreePtrs* __restrict__ trees, int K, int F, TreeRecord rec,
                                unsigned char* __restrict__ records, double* __restrict__ leaves_c)
{
  AfterTheKernelBefore();
  if (SkipFor(gate)) return;
  const TreePtrs t   = trees[blockIdx.x];
  const int M = t.max_nodes, S = rec.S;
  unsigned char* out = records + static_cast<int64_t>(blockIdx.x) * rec.bytes;
  T* splits          = reinterpret_cast<T*>(out);
  unsigned* words    = reinterpret_cast<unsigned*>(out + rec.split_bytes);
  double* leaves     = rec.leaf_bytes > 0 ? reinterpret_cast<double*>(out + rec.split_bytes + rec.word_bytes)
                                          : leaves_c + (static_cast<int64_t>(blockIdx.x) << S) * K;
  // the features of the nodes above the bottom level, kNoSplit: none; then the paths are followed in shared memory (through the
  // arrays, a load behind the other: 50 trees of depth 8, ten outputs 9.9 us, now 9.4, of which most are the values; a thread per value 12.2)
  extern __shared__ uint16_t s_feature[];
  constexpr int kNoSplit = 0xffff;
  for (int a = threadIdx.x; a < (1 << S) - 1; a += blockDim.x) {
    const int f  = 2 * a + 2 < M ? t.feature[a] : -1;
    s_feature[a] = static_cast<uint16_t>(f >= 0 && f < F ? f : kNoSplit);
  }
  __syncthreads();
  auto splits_here = [&](int a) { return s_feature[a] != kNoSplit; };
  // first leaf on the path root -> i (of level L), or -1
  auto cover_of = [&](int i, int L) {
    for (int l = 0; l <= L; ++l) {
      const int a = ((i + 1) >> (L - l)) - 1;
      if (l == S || !splits_here(a)) return a;
    }
    return -1;
  };
  const int total = (2 << S) - 1;  // nodes of the complete tree
  for (int i = threadIdx.x; i < total; i += blockDim.x) {
    const int L = 31 - __clz(i + 1), cover = cover_of(i, L);
    if (L < S) {
      // (a pass-through node sends a NaN to the right: the same leaf value is there)
      MakeSplit(splits[i + 1], cover >= 0 ? static_cast<double>(INFINITY) : t.split[i]);
      if ((L & 1) == 0) {
        unsigned w = cover >= 0 ? 0u : static_cast<unsigned>(s_feature[i]);
        if (cover < 0 && L + 1 < S) {
          if (splits_here(2 * i + 1)) w |= static_cast<unsigned>(s_feature[2 * i + 1]) << kIdBits;
          if (splits_here(2 * i + 2)) w |= static_cast<unsigned>(s_feature[2 * i + 2]) << (2 * kIdBits);
        }
        words[i + 1] = w;
      }
    } else {
      const int j = i - ((1 << S) - 1);
      for (int k = 0; k < K; ++k) leaves[static_cast<int64_t>(j) * K + k] = t.leaf[static_cast<int64_t>(cover) * K + k];
    }
  }
}

// ---- few rows ---------------------------------------------------------------------------------
// One launch that walks the trees where they lie: a block takes `rows_per_block` rows, its threads take
// (row, tree) pairs, trees in neighbouring lanes, and leave what each walk adds in shared memory; the
// sums are then made in tree order, one thread per (row, output).  Bound by the latency of one walk
// (two dependent loads per level from L2) plus the ordered sum, as long as there are few rows; nothing
// is packed or staged, which for 16 rows and 100 trees of depth 6 takes longer than the walks.
constexpr int kRowsThreads = 256;

template <typename T>
__global__ void __launch_bounds__(kRowsThreads)
  k_predict_rows(const T* __restrict__ X, int64_t ldx, int64_t n_rows, int F, int K, int n_trees, int rows_per_block,
                 const TreePtrs* __restrict__ trees, PredictOut o)
{
  AfterTheKernelBefore();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  // [rows][trees] values (K == 1) or addresses of the leaves' values | [rows][K] sums | [rows][F] X
  double* vals        = reinterpret_cast<double*>(smem_raw);
  const double** adrs = reinterpret_cast<const double**>(smem_raw);
  double* sums        = vals + static_cast<size_t>(rows_per_block) * n_trees;
  T* xs               = reinterpret_cast<T*>(sums + static_cast<size_t>(rows_per_block) * K);
  const int tid       = threadIdx.x;
  const int64_t row0  = static_cast<int64_t>(blockIdx.x) * rows_per_block;
  const int rows      = static_cast<int>(n_rows - row0 < rows_per_block ? n_rows - row0 : rows_per_block);
  for (int i = tid; i < rows * F; i += kRowsThreads) {
    const int r = i / F;
    xs[i]       = X[(row0 + r) * ldx + (i - r * F)];
  }
  __syncthreads();
  for (int i = tid; i < rows * n_trees; i += kRowsThreads) {
    const int r      = i / n_trees, t = i - r * n_trees;
    const TreePtrs p = trees[t];
    const T* xr      = xs + r * F;
    int pos          = 0;
    for (int depth = 0; depth < 100; ++depth) {
      const int f        = __ldg(p.feature + pos);
      const double split = __ldg(p.split + pos);
      if (f < 0 || f >= F || 2 * pos + 2 >= p.max_nodes) break;
      pos = 2 * pos + 1 + (static_cast<double>(xr[f]) <= split ? 0 : 1);
    }
    if (K == 1) vals[i] = __ldg(p.leaf + pos);
    else adrs[i] = p.leaf + static_cast<int64_t>(pos) * K;
  }
  __syncthreads();
  for (int i = tid; i < rows * K; i += kRowsThreads) {
    const int r = i / K, k = i - r * K;
    double acc  = 0.0;
    if (K == 1) {
      const double* v = vals + static_cast<size_t>(r) * n_trees;
#pragma unroll 8
      for (int t = 0; t < n_trees; ++t) acc += v[t];
    } else {
      const double* const* v = adrs + static_cast<size_t>(r) * n_trees;
#pragma unroll 8
      for (int t = 0; t < n_trees; ++t) acc += __ldg(v[t] + k);
    }
    sums[i] = o.init ? o.init[k] + acc : acc;
  }
  __syncthreads();
  for (int r = tid; r < rows; r += kRowsThreads) FinishRow(sums + r * K, 1, K, o.pred + (row0 + r) * o.ldp, o.transform);
}

constexpr int kTileThreads = 512;  // of all blocks of an SM, producer warps included: 128 registers each

template <typename T>
struct TiledArgs {
  const T* X;
  int64_t ldx, n_rows;
  int F, K, n_trees;
  int rb;            // rows per block, a multiple of 32
  int nbuf;          // group buffers: 2, or 1 if all trees are one group
  unsigned x_bytes;  // of the X tile (and of what takes its place at the end)
  const unsigned char* records;
  TreeRecord rec;
  const double* leaves_c;  // [tree][2^S][K] (several outputs)
  PredictOut o;
  int* status;
};

// Tiled kernel.  Shared memory: X tile [F][rb] | sums [K][rb] (KR < 0) | nbuf x TG records.
// KR: outputs whose sums a warp holds in registers (at most KR of them); 0: one output, leaf values in the
// records; -1: any number of outputs, sums in shared memory.
// Measured against {split, feature} nodes, a block barrier per group, 256 rows per block and every lane reading
// its own row's values: 100003 x 100, 10 outputs, 50 trees: 224 -> 131 us (now 107: kStaged); and, since then walked on ranks,
// 10M x 100 float32, 500 trees of depth 8: 23.2 -> 19.5 ms, 1M x 64 float64, 100 trees: 1117 -> 803 us.
// kStaged (KR > 0): the leaf values of several outputs are in the records too; 2: of an even number, and a lane has the sums of two
// neighbouring outputs, whose values are one 16-byte load.  Per tree and 32 rows of ten outputs that is 30 passes instead of 55
// (as 8-byte loads, 12 values for 10), of about 80 with the walks: 100 features, ten outputs, 50 trees of depth 8, 1M rows 1141 -> 946 us,
// 100003 rows 97 -> 92 (what is left is the latency of the walks in flight, eleven warps with two trees each: ncu has the load/store pipe
// at 56 %, the issue slots at 25 and L2 at 15, and an instruction of a warp every eleven cycles); 300k x 20, 100 trees of depth 6 303 -> 256; sixteen
// outputs, 200003 x 30 170 -> 160.  Three outputs with three sums instead of four: 2M x 50, 100 trees of depth 7 1229 -> 1153 (which numbers: predict_sums.h).
// kGated: the launch stands in for the walk on ranks and does nothing where that was not declined.  A resident block then takes tile
// after tile: a launch that finds nothing to do ends in 2.5 us, where a block per tile would come and go.
template <typename T, int TG, int KR, int kStaged, bool kGated = false>
__global__ void __launch_bounds__(kTileThreads, 1) k_predict_tiled(const TiledArgs<T> a, const int* __restrict__ gate)
{
  AfterTheKernelBefore();
  __shared__ __align__(8) unsigned long long s_bar[4];  // full[2], empty[2]
  __shared__ int s_failed;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int rb = a.rb, F = a.F, K = a.K, S = a.rec.S;
  T* xs        = reinterpret_cast<T*>(smem_raw);
  double* accs = reinterpret_cast<double*>(smem_raw + a.x_bytes);
  const unsigned rec_bytes = a.rec.bytes, buf_bytes = TG * rec_bytes;
  const unsigned tree0 = static_cast<unsigned>(__cvta_generic_to_shared(smem_raw)) + a.x_bytes + (KR < 0 ? 8u * K * rb : 0u);
  const unsigned full0 = static_cast<unsigned>(__cvta_generic_to_shared(&s_bar[0])), empty0 = full0 + 16;

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (kGated && *gate == 0) return;
  int64_t tile   = blockIdx.x;
  auto next_tile = [&]() {
    __syncthreads();  // (barriers and tile are made anew)
    tile += gridDim.x;
    return s_failed == 0 && tile * rb < a.n_rows;
  };
  for (;;) {
    const int64_t row0 = tile * rb;
    const int n_groups = (a.n_trees + TG - 1) / TG;
    if (tid == 0) {
      s_failed = 0;
      for (int b = 0; b < 2; ++b) {
        if (kGated && tile != blockIdx.x) {
          MbarInval(full0 + 8 * b);
          MbarInval(empty0 + 8 * b);
        }
        MbarInit(full0 + 8 * b, 1);
        MbarInit(empty0 + 8 * b, rb / 32);
      }
      asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    __syncthreads();

    if (warp == rb / 32) {  // the producer: brings group after group into the buffer that every warp is done with
      if (lane == 0) {
        int g   = 0;
        bool ok = true;
        for (; g < n_groups && ok; ++g) {
          const int b = a.nbuf == 2 ? g & 1 : 0;
          if (g >= 2) ok = MbarWait(empty0 + 8 * b, ((g >> 1) - 1) & 1, a.status, &s_failed);
          if (!ok) break;
          const unsigned bytes = min(TG, a.n_trees - g * TG) * rec_bytes;
          MbarExpectTx(full0 + 8 * b, bytes);
          BulkCopy(tree0 + b * buf_bytes, a.records + static_cast<int64_t>(g) * buf_bytes, bytes, full0 + 8 * b);
        }
        // nothing is in flight when the block ends, whatever the other warps waited for
        for (int h = max(g - 2, 0); h < g; ++h) MbarWait(full0 + 8 * (a.nbuf == 2 ? h & 1 : 0), (h >> 1) & 1, a.status, &s_failed);
      }
      __syncthreads();
      if (s_failed != 0) {  // (the other warps have written what they have)
        const int columns = a.o.transform == LBK_LOGISTIC ? 2 : K;
        for (int64_t at = row0; at < a.n_rows; at += static_cast<int64_t>(gridDim.x) * rb) {  // (gated: the block takes no more tiles)
          for (int64_t row = at + lane; row < at + rb && row < a.n_rows; row += 32)
            for (int k = 0; k < columns; ++k) a.o.pred[row * a.o.ldp + k] = NAN;
          if (!kGated) break;
        }
      }
      if (!kGated || !next_tile()) return;
      continue;
    }

    // Every thread copies its own row into its own column of the tile and reads nothing else of it, with 16-byte loads; the
    // sectors of a row are reused from L1 by the following loads of the same thread.  Rows that are not all on 16-byte
    // boundaries: from the row's first whole vector on, value by value before and behind (all value by value, a pass per row
    // and load: 1M x 75 float32, 100 trees of depth 8: 884 us, now 543; 1M x 127, 50 trees of depth 6: 712 and 406).  In a
    // function of its own that path takes 687 and 676; inlined, it costs the float64 kernel 0.6 %.
    if (row0 + tid < a.n_rows) {
      const T* xr     = a.X + (row0 + tid) * a.ldx;
      constexpr int V = 16 / sizeof(T);
      if ((reinterpret_cast<uintptr_t>(a.X) & 15) == 0 && a.ldx % V == 0) {
        int f = 0;
#pragma unroll 8
        for (; f + V <= F; f += V) {
          const int4 v = *reinterpret_cast<const int4*>(xr + f);
#pragma unroll
          for (int i = 0; i < V; ++i) xs[(f + i) * rb + tid] = reinterpret_cast<const T*>(&v)[i];
        }
        for (; f < F; ++f) xs[f * rb + tid] = xr[f];
      } else {
        const int head  = min(F, (V - static_cast<int>(reinterpret_cast<uintptr_t>(xr) / sizeof(T) % V)) % V);
        const int whole = (F - head) / V;
#pragma unroll
        for (int f = 0; f < V - 1; ++f)
          if (f < head) xs[f * rb + tid] = xr[f];
        const int4* xv = reinterpret_cast<const int4*>(xr + head);
        T* column      = xs + head * rb + tid;
#pragma unroll 8
        for (int v = 0; v < whole; ++v) {
          const int4 x = xv[v];
#pragma unroll
          for (int i = 0; i < V; ++i) column[(v * V + i) * rb] = reinterpret_cast<const T*>(&x)[i];
        }
#pragma unroll
        for (int i = 0; i < V - 1; ++i) {
          const int f = head + whole * V + i;
          if (f < F) xs[f * rb + tid] = xr[f];
        }
      }
    } else {
      // the walks of the missing rows are made too (any value leads to some leaf) and not written
      for (int f = 0; f < F; ++f) xs[f * rb + tid] = T(0);
    }
    if (KR < 0)
      for (int k = 0; k < K; ++k) accs[k * rb + tid] = 0.0;

    // KR > 0: the warp's sums (kStaged 2: pairs of them) are numbered output innermost, lane l holds l, l + 32, ...
    constexpr int kWide  = kStaged == 2 ? 2 : 1;
    constexpr int kSums  = KR > 0 ? KR : 1, kSlots = kSums / kWide;
    const int slots      = K / kWide;  // of the warp's, per row
    double acc[kSums];
    int which[kSlots];  // of each slot: lane (row of the warp) + 32 x output (pair)
#pragma unroll
    for (int i = 0; i < kSums; ++i) acc[i] = 0.0;
#pragma unroll
    for (int i = 0; i < kSlots; ++i) {
      const int r = KR > 0 ? (lane + 32 * i) / slots : 0;
      which[i]    = KR > 0 && i < slots ? r + 32 * (lane + 32 * i - r * slots) : 0;  // (what is beyond is dropped)
    }

    // The walk works on 32-bit shared addresses; at[j] is that of the split of tree j's current node.
    constexpr unsigned kT    = sizeof(T);
    const unsigned xcol_s    = static_cast<unsigned>(__cvta_generic_to_shared(xs + tid));
    const unsigned pitch     = static_cast<unsigned>(rb * sizeof(T));
    const unsigned word_off  = a.rec.split_bytes;
    const unsigned leaf_off  = a.rec.split_bytes + a.rec.word_bytes - (8u << S);
    constexpr unsigned kMask = kMaxFeature - 1;
    for (int g = 0; g < n_groups; ++g) {
      const int b = a.nbuf == 2 ? g & 1 : 0;
      if (!__all_sync(0xffffffffu, MbarWait(full0 + 8 * b, (g >> 1) & 1, a.status, &s_failed) ? 1 : 0)) break;
      const int nt = min(TG, a.n_trees - g * TG);
      unsigned at[TG], base[TG];
#pragma unroll
      for (int j = 0; j < TG; ++j) {
        base[j] = tree0 + b * buf_bytes + j * rec_bytes;
        at[j]   = base[j] + kT;
      }
      // Two levels of all walks at a time: first every split and word, then every x, then the compares, so that
      // the loads of the independent walks are in flight together (the loads are volatile and keep
      // their order).  `here(j)` is always true but in the last group.
      auto walk = [&](auto here) {
        T split[TG], x[TG];
        unsigned w[TG];
        auto first_loads = [&]() {
#pragma unroll
          for (int j = 0; j < TG; ++j)
            if (here(j)) {
              w[j]     = LdsU32(kT == 4 ? at[j] + word_off : base[j] + word_off + ((at[j] - base[j]) >> 1));
              split[j] = LdsX(at[j], T());
            }
        };
        auto x_loads = [&]() {
#pragma unroll
          for (int j = 0; j < TG; ++j)
            if (here(j)) x[j] = LdsX(xcol_s + (w[j] & kMask) * pitch, T());
        };
        auto descend = [&](int j) {
          const bool left = x[j] <= split[j];
          at[j]           = at[j] + at[j] - base[j];
          if (!left) at[j] += kT;
          return left;
        };
        int l = 0;
#pragma unroll 1
        for (; l + 1 < S; l += 2) {
          first_loads();
          x_loads();
#pragma unroll
          for (int j = 0; j < TG; ++j)
            if (here(j)) {
              w[j] >>= descend(j) ? kIdBits : 2 * kIdBits;
              split[j] = LdsX(at[j], T());
            }
          x_loads();
#pragma unroll
          for (int j = 0; j < TG; ++j)
            if (here(j)) descend(j);
        }
        if (l < S) {
          first_loads();
          x_loads();
#pragma unroll
          for (int j = 0; j < TG; ++j)
            if (here(j)) descend(j);
        }
        if (KR == 0) {
          double v[TG];
#pragma unroll
          for (int j = 0; j < TG; ++j)
            if (here(j)) v[j] = LdsF64(base[j] + leaf_off + (at[j] - base[j]) * (8u / kT));
#pragma unroll
          for (int j = 0; j < TG; ++j)
            if (here(j)) acc[0] += v[j];
        }
      };
      if (nt == TG) walk([](int) { return true; });
      else walk([&](int j) { return j < nt; });
      __syncwarp();
      if (kStaged == 0 && lane == 0) MbarArrive(empty0 + 8 * b);  // this warp is done with the buffer
      if constexpr (kStaged != 0) {
        const unsigned values = a.rec.split_bytes + a.rec.word_bytes;
        auto add = [&](auto here) {
#pragma unroll
          for (int j = 0; j < TG; ++j) {
            if (!here(j)) continue;
            const unsigned v = base[j] + values + ((at[j] - base[j]) / kT - (1u << S)) * (8u * K);  // where the row's values are
            if constexpr (kStaged == 2) {
              double2 x[kSlots];
#pragma unroll
              for (int i = 0; i < kSlots; ++i) x[i] = LdsF64x2(__shfl_sync(0xffffffffu, v, which[i] & 31) + 16u * (which[i] >> 5));
#pragma unroll
              for (int i = 0; i < kSlots; ++i) {
                acc[2 * i] += x[i].x;
                acc[2 * i + 1] += x[i].y;
              }
            } else {
#pragma unroll
              for (int i = 0; i < kSlots; ++i) acc[i] += LdsF64(__shfl_sync(0xffffffffu, v, which[i] & 31) + 8u * (which[i] >> 5));
            }
          }
        };
        if (nt == TG) add([](int) { return true; });
        else add([&](int j) { return j < nt; });
        __syncwarp();
        if (lane == 0) MbarArrive(empty0 + 8 * b);
      } else if (KR != 0) {
        const int64_t tree_values = static_cast<int64_t>(K) << S;
        const double* lf          = a.leaves_c + g * TG * tree_values;
        auto add = [&](auto here) {
#pragma unroll
          for (int j = 0; j < TG; ++j) {
            if (!here(j)) continue;
            const int v = (static_cast<int>((at[j] - base[j]) / kT) - (1 << S)) * K;  // the row's first value
            if (KR > 0) {
#pragma unroll
              for (int i = 0; i < kSums; ++i) acc[i] += __ldg(lf + __shfl_sync(0xffffffffu, v, which[i] & 31) + (which[i] >> 5));
            } else {
              for (int k = 0; k < K; ++k) accs[k * rb + tid] += lf[v + k];
            }
            lf += tree_values;
          }
        };
        if (nt == TG) add([](int) { return true; });
        else add([&](int j) { return j < nt; });
      }
    }

    const PredictOut& o = a.o;
    const int64_t row   = row0 + tid;
    if (KR == 0) {
      const double raw = o.init ? o.init[0] + acc[0] : acc[0];
      if (row < a.n_rows) FinishRow(&raw, 1, 1, o.pred + row * o.ldp, o.transform);
    } else if (KR < 0) {
      if (o.init)
        for (int k = 0; k < K; ++k) accs[k * rb + tid] = o.init[k] + accs[k * rb + tid];
      if (row < a.n_rows) FinishRow(accs + tid, rb, K, o.pred + row * o.ldp, o.transform);
    } else {
      double* rows = reinterpret_cast<double*>(smem_raw) + static_cast<int64_t>(warp) * 32 * K;  // of the warp, [32][K]
      if (o.transform != LBK_RAW) {
        asm volatile("bar.sync 1, %0;\n" ::"r"(rb) : "memory");  // the walks are done: the rows take the place of X
#pragma unroll
        for (int i = 0; i < kSlots; ++i)
          if (i < slots) {
#pragma unroll
            for (int e = 0; e < kWide; ++e) {
              const double sum                  = acc[kWide * i + e];
              rows[kWide * (lane + 32 * i) + e] = o.init ? o.init[kWide * (which[i] >> 5) + e] + sum : sum;
            }
          }
        __syncwarp();
        FinishRow(rows + lane * K, 1, K, rows + lane * K, o.transform);
        __syncwarp();
      }
#pragma unroll
      for (int i = 0; i < kSlots; ++i) {
        const int64_t r = row0 + warp * 32 + (which[i] & 31);
        if (i < slots && r < a.n_rows) {
#pragma unroll
          for (int e = 0; e < kWide; ++e) {
            const int k = kWide * (which[i] >> 5) + e;
            const double sum = acc[kWide * i + e];
            o.pred[r * o.ldp + k] = o.transform != LBK_RAW ? rows[kWide * (lane + 32 * i) + e] : o.init ? o.init[k] + sum : sum;
          }
        }
      }
    }
    __syncthreads();  // (the producer's copies)
    if (!kGated || !next_tile()) return;
  }
}

// The raw sums of an ensemble without trees; nothing of X is read.
__global__ void __launch_bounds__(256) k_predict_nothing(int64_t n_rows, int K, PredictOut o)
{
  AfterTheKernelBefore();
  const int64_t row = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (row >= n_rows) return;
  for (int k = 0; k < K; ++k) o.pred[row * o.ldp + k] = o.init ? o.init[k] : 0.0;
}

// What is left to do after a kernel that wrote the raw sums.
__global__ void __launch_bounds__(256) k_finish_rows(const int* __restrict__ gate, int64_t n_rows, int K, PredictOut o)
{
  AfterTheKernelBefore();
  if (SkipFor(gate)) return;
  const int64_t row = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (row >= n_rows) return;
  double* p = o.pred + row * o.ldp;
  FinishRow(p, 1, K, p, o.transform);
}

// Fallback: original (uncompleted) trees, nodes and leaves in global memory, X read directly.
template <typename T>
__global__ void __launch_bounds__(128)
  k_predict_global(const int* __restrict__ gate, const T* __restrict__ X, int64_t ldx, int64_t n_rows, int K, int n_trees,
                   const TreePtrs* __restrict__ trees, const typename NodeOf<T>::type* __restrict__ nodes,
                   const double* __restrict__ leaves, PredictOut o)
{
  AfterTheKernelBefore();
  using NodeT       = typename NodeOf<T>::type;
  if (SkipFor(gate)) return;
  const int64_t row = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (row >= n_rows) return;
  const T* xr = X + row * ldx;
  double* pred = o.pred + row * o.ldp;
  for (int k = 0; k < K; ++k) pred[k] = 0.0;
  for (int t = 0; t < n_trees; ++t) {
    const int off = trees[t].node_off;
    int pos       = 0;
    for (int depth = 0; depth < 100; ++depth) {
      const NodeT n = nodes[off + pos];
      if (n.foff < 0) break;
      pos = 2 * pos + 1 + (xr[n.foff] <= n.split ? 0 : 1);
    }
    const double* lf = leaves + static_cast<int64_t>(off + pos) * K;
    for (int k = 0; k < K; ++k) pred[k] += lf[k];
  }
  if (o.init)
    for (int k = 0; k < K; ++k) pred[k] = o.init[k] + pred[k];
}

// How the tiled kernel is cut.  rb == 0: the shape does not fit, or fewer than kTileMinRows rows do on an SM (one output:
// if they are of more than kTileOneWarpBytes).
//
// A single warp per SM does not hide the walks' latency; nodes and rows are then read through the caches
// (k_predict_global), which is fast where the trees ask for few of the features and slow where they ask for all of
// them, while the tile's time does not depend on that.  Microseconds, tile and caches, 200k rows, 100 fitted trees of
// depth 6: two warps, float32, 700 features, splits on five of them 662 and 422, on all of them 664 and 2278 (30k rows:
// 144 and 270, 147 and 345); 850 features 1112 and 432, 1112 and 2367; three classes, 700 features 672 and 348, 673
// and 1227; float64, 350 features 660 and 457, 660 and 2294; 20 outputs, 50 trees on random features, 100k rows 1060
// and 2123.  One warp: float32, 1000 features 1492 and 439, 1493 and 2418; three classes 1542 and 353, 1540 and 1285.  Shorter rows come to one warp
// beside deep trees: float64, 300 features, ten classes, 15 trees of depth 9 1354 and 840; with one output they stay
// (float32, 600 features, 30 trees of depth 9, splits on all of them 906 and 1010).
constexpr int kTileMinRows         = 64;
constexpr size_t kTileOneWarpBytes = 2560;
struct TilePlan {
  int rb = 0, tg = 0, nbuf = 0, resident = 1;
  int sm_rows = 0;  // rows that an SM has at a time
  unsigned x_bytes = 0;
  size_t smem      = 0;
  int64_t waves    = 0;
  TreeRecord rec{};
};
constexpr int kStagedOutputs   = 6;    // from which leaf values may come with the records (PlanTile), ...
constexpr int kStagedTrees     = 16;   // ... and trees: of fewer the rows are most of the work, which more blocks an SM overlap
constexpr int kTileStaticBytes = 256;  // (a bound of what the kernel declares)

// The pipe is kept busy by the walks in flight: warps x trees per group.  That product is made as large as shared
// memory allows, over groups of 8, 4, 2 or 1 trees and 1 to 4 blocks per SM, up to kTileThreads; equal products go to
// more blocks, of which one stages its rows while another walks.  The rows are then spread evenly over the
// waves that this takes, so that the last one is not nearly empty.
//
// With six to kRegisterSums outputs the leaf values come with the records where a block reads them often enough: a
// block of rb rows would gather rb x K of a tree's values from L2, sectors of 32 bytes for pieces of 8 K, and brings 2^S x K in
// one piece instead.  100003 x 100, ten outputs, 50 trees of depth 8: the gathers' 500 MB were most of 124 us, now 107; depth 6,
// 20000 rows 52 -> 31, 600000 rows of float64 818 -> 631; sixteen outputs, 100003 x 300 float64 658 -> 362.  Small tables stay
// in L1 where rows come in many waves: depth 4, 600000 rows 401 and 460.
template <typename T>
TilePlan PlanTile(lbk_context* ctx, int64_t n_rows, int F, int K, int n_trees, int S, int transform)
{
  const size_t row_bytes = sizeof(T) * static_cast<size_t>(F) + (K > kRegisterSums ? 8 * static_cast<size_t>(K) : 0);
  // (the finished rows of a few outputs take the place of X)
  const size_t x_row = K > 1 && K <= kRegisterSums && transform != LBK_RAW ? std::max<size_t>(sizeof(T) * F, 8 * static_cast<size_t>(K)) : sizeof(T) * static_cast<size_t>(F);
  const size_t per_row = std::max(row_bytes, x_row);
  auto plan = [&](int leaf_values) {
    TilePlan best;
    int best_score = 0, best_res = 1;
    for (int tg = 8; tg >= 1; tg /= 2) {
      if (tg > n_trees && tg > 1) continue;  // no wider than the ensemble
      const TreeRecord rec = RecordOf(S, sizeof(T), leaf_values);
      const int nbuf       = n_trees > tg ? 2 : 1;
      const size_t trees   = static_cast<size_t>(nbuf) * tg * rec.bytes;
      for (int res = 1; res <= 4; ++res) {
        const size_t room = res == 1 ? static_cast<size_t>(ctx->max_smem_optin) - kTileStaticBytes
                                      : (static_cast<size_t>(ctx->max_smem_optin) + 1024) / res - 1024 - kTileStaticBytes;
        if (trees + 32 * per_row > room) continue;
        const int rb    = static_cast<int>(std::min<size_t>((room - trees) / per_row, kTileThreads / res - 32) / 32 * 32);
        const int score = res * rb / 32 * tg;
        // (with a table of leaf values per tree, more trees at a time are fewer rows: not for one more wave of them)
        const int64_t waves = (n_rows + static_cast<int64_t>(rb) * res * ctx->sm_count - 1) / (static_cast<int64_t>(rb) * res * ctx->sm_count);
        if (leaf_values > 1 && best_score > 0 && waves != best.waves ? waves > best.waves : score < best_score || (score == best_score && tg < best.tg)) continue;
        best_score   = score;
        best.sm_rows = res * rb;
        best.waves   = waves;
        best_res     = res;
        best.rb      = rb;
        best.tg      = tg;
        best.nbuf    = nbuf;
        best.rec     = rec;
      }
    }
    if (best.rb == 0 || (best_res * best.rb < kTileMinRows && (K > 1 || sizeof(T) * F > kTileOneWarpBytes))) return TilePlan{};
    const int64_t slots = static_cast<int64_t>(ctx->sm_count) * best_res;
    const int64_t waves = (n_rows + best.rb * slots - 1) / (best.rb * slots);
    best.rb             = static_cast<int>(((n_rows + waves * slots - 1) / (waves * slots) + 31) / 32 * 32);
    best.x_bytes        = static_cast<unsigned>((x_row * best.rb + 15) / 16 * 16);
    best.smem = best.x_bytes + (K > kRegisterSums ? 8 * static_cast<size_t>(K) * best.rb : 0) + static_cast<size_t>(best.nbuf) * best.tg * best.rec.bytes;
    best.waves    = waves;
    best.resident = best_res;
    return best;
  };
  if (K == 1) return plan(1);
  const TilePlan apart = plan(0);
  if (K < kStagedOutputs || K > kRegisterSums || n_trees < kStagedTrees || apart.rb == 0) return apart;
  const TilePlan with = plan(K);
  return with.rb >= (1 << S) && with.waves <= apart.waves && (S >= 5 || with.waves <= 4) ? with : apart;
}

template <typename T, int TG, int KR>
void LaunchTiledAs(lbk_context* ctx, const int* gate, const TiledArgs<T>& a, const TilePlan& plan, cudaStream_t stream)
{
  auto fn = k_predict_tiled<T, TG, KR, 0>;
  if constexpr (KR >= kStagedOutputs)
    if (a.leaves_c == nullptr) fn = k_predict_tiled<T, TG, KR, 2>;
  if constexpr (KR > kStagedOutputs)
    if (a.leaves_c == nullptr && a.K % 2 != 0) fn = k_predict_tiled<T, TG, KR, 1>;
  int64_t grid = (a.n_rows + a.rb - 1) / a.rb;
  if constexpr (KR == 0)
    if (gate != nullptr) {
      fn   = k_predict_tiled<T, TG, 0, 0, true>;
      grid = std::min<int64_t>(grid, static_cast<int64_t>(ctx->sm_count) * plan.resident);
    }
  // (whatever the size: the limit without it is for the static and the dynamic part together)
  AllowSharedMemory(ctx, fn, kTileStaticBytes);
  LaunchChained(fn, static_cast<unsigned>(grid), a.rb + 32, plan.smem, stream, a, gate);
  LBK_LAUNCH_CHECK();
}

template <typename T, int TG>
void LaunchTiled(lbk_context* ctx, const int* gate, const TiledArgs<T>& a, const TilePlan& plan, cudaStream_t stream)
{
  switch (SumsOf(a.K)) {
    case 0: LaunchTiledAs<T, TG, 0>(ctx, gate, a, plan, stream); break;
    case 2: LaunchTiledAs<T, TG, 2>(ctx, gate, a, plan, stream); break;
    case 3: LaunchTiledAs<T, TG, 3>(ctx, gate, a, plan, stream); break;
    case 4: LaunchTiledAs<T, TG, 4>(ctx, gate, a, plan, stream); break;
    case 6: LaunchTiledAs<T, TG, 6>(ctx, gate, a, plan, stream); break;
    case 8: LaunchTiledAs<T, TG, 8>(ctx, gate, a, plan, stream); break;
    case 10: LaunchTiledAs<T, TG, 10>(ctx, gate, a, plan, stream); break;
    case 12: LaunchTiledAs<T, TG, 12>(ctx, gate, a, plan, stream); break;
    case 14: LaunchTiledAs<T, TG, 14>(ctx, gate, a, plan, stream); break;
    case 16: LaunchTiledAs<T, TG, 16>(ctx, gate, a, plan, stream); break;
    default: LaunchTiledAs<T, TG, -1>(ctx, gate, a, plan, stream); break;
  }
}

}  // namespace

template <typename T>
void PredictLaunch(lbk_context* ctx, Scratch& s, const T* X, int64_t ldx, int64_t n_rows, int F, int K, int n_trees,
                   const lbk_tree_ref* d_trees, int m_max, int64_t total_nodes, const double* init, int transform,
                   double* pred, int64_t ldp, cudaStream_t stream)
{
  using NodeT = typename NodeOf<T>::type;
  if (n_rows < 1) return;  // an empty shard returns at once (reference: predict.cu:35)
  const PredictOut o{pred, ldp, init, transform};
  auto finish = [&](const int* gate) {
    if (transform == LBK_RAW) return;
    LaunchChained(k_finish_rows, static_cast<unsigned>((n_rows + 255) / 256), 256, 0, stream, gate, n_rows, K, o);
    LBK_LAUNCH_CHECK();
  };
  if (n_trees == 0) {
    LaunchChained(k_predict_nothing, static_cast<unsigned>((n_rows + 255) / 256), 256, 0, stream, n_rows, K, o);
    LBK_LAUNCH_CHECK();
    finish(nullptr);
    return;
  }
  // Few rows: walk the trees in place.  The tiled kernel brings every tree into shared memory per block (of up to
  // 480 rows), so that it needs tens of thousands of rows to fill the chip.
  {
    constexpr int64_t kRowsMax = 8192;
    int r = static_cast<int>((n_rows + 4 * ctx->sm_count - 1) / (4 * ctx->sm_count));
    r     = r < 1 ? 1 : r > 8 ? 8 : r;
    auto need = [&](int rows) { return static_cast<size_t>(rows) * ((n_trees + K) * sizeof(double) + F * sizeof(T)); };
    while (r > 1 && need(r) > 48 * 1024) r /= 2;
    if (n_rows <= kRowsMax && need(r) <= 48 * 1024) {
      const unsigned grid = static_cast<unsigned>((n_rows + r - 1) / r);
      LaunchChained(k_predict_rows<T>, grid, kRowsThreads, need(r), stream, X, ldx, n_rows, F, K, n_trees, r, d_trees, o);
      LBK_LAUNCH_CHECK();
      return;
    }
  }
  // a walk through M heap-ordered nodes takes at most S = floor(log2(M)) steps
  int S = 0;
  while ((2 << S) <= m_max) ++S;
  const TilePlan plan     = S <= 14 && F <= kMaxFeature ? PlanTile<T>(ctx, n_rows, F, K, n_trees, S, transform) : TilePlan{};
  const RankedPlan ranked = K == 1 ? PlanRanked<T>(ctx, n_rows, F, n_trees, S, total_nodes, RankTile{plan.sm_rows, plan.tg, plan.rec.bytes}) : RankedPlan{};
  auto by_ranks = [&]() {
    return PredictRanked<T>(ctx, s, ranked, X, ldx, n_rows, F, n_trees, d_trees, S, total_nodes, init, transform, pred, ldp, stream);
  };
  if (ranked.threads > 0 && ranked.sure && by_ranks() != nullptr) return;
  // (what the rows are walked with where the ranks are declined comes first: without room for it the call fails, with or without ranks)
  NodeT* nodes = nullptr;
  double *leaves = nullptr, *leaves_c = nullptr;
  unsigned char* records = nullptr;
  if (plan.rb == 0) {
    nodes  = s.alloc<NodeT>(total_nodes);
    leaves = s.alloc<double>(total_nodes * K);
  } else {
    records = static_cast<unsigned char*>(s.alloc_bytes(static_cast<size_t>(n_trees) * plan.rec.bytes));
    if (plan.rec.leaf_bytes == 0) leaves_c = s.alloc<double>((static_cast<size_t>(n_trees) << S) * K);
  }
  const int* gate = nullptr;
  if (ranked.threads > 0 && !ranked.sure) gate = by_ranks();
  if (plan.rb == 0) {
    LaunchChained(k_pack_trees<NodeT>, n_trees, 256, 0, stream, gate, d_trees, K, F, nodes, leaves);
    LBK_LAUNCH_CHECK();
    const unsigned grid = static_cast<unsigned>((n_rows + 127) / 128);
    LaunchChained(k_predict_global<T>, grid, 128, 0, stream, gate, X, ldx, n_rows, K, n_trees, d_trees, nodes, leaves, o);
    LBK_LAUNCH_CHECK();
    finish(gate);
    return;
  }
  LaunchChained(k_pack_complete<T>, n_trees, 256, sizeof(uint16_t) << S, stream, gate, d_trees, K, F, plan.rec, records, leaves_c);
  LBK_LAUNCH_CHECK();
  const TiledArgs<T> a{X, ldx, n_rows, F, K, n_trees, plan.rb, plan.nbuf, plan.x_bytes, records, plan.rec, leaves_c, o, ctx->d_status};
  switch (plan.tg) {
    case 8: LaunchTiled<T, 8>(ctx, gate, a, plan, stream); break;
    case 4: LaunchTiled<T, 4>(ctx, gate, a, plan, stream); break;
    case 2: LaunchTiled<T, 2>(ctx, gate, a, plan, stream); break;
    default: LaunchTiled<T, 1>(ctx, gate, a, plan, stream); break;
  }
}

// How a call would be made: see lbk.h.
template <typename T>
static void PlanOfPredict(lbk_context* ctx, int64_t n_rows, int F, int K, int n_trees, int m_max, int64_t total_nodes, int transform, int64_t* out)
{
  int S = 0;
  while ((2 << S) <= m_max) ++S;
  const TilePlan tile     = S <= 14 && F <= kMaxFeature ? PlanTile<T>(ctx, n_rows, F, K, n_trees, S, transform) : TilePlan{};
  const RankedPlan ranked = K == 1 ? PlanRanked<T>(ctx, n_rows, F, n_trees, S, total_nodes, RankTile{tile.sm_rows, tile.tg, tile.rec.bytes}) : RankedPlan{};
  const int64_t words[8]  = {ranked.threads, ranked.tg, ranked.piece, static_cast<int64_t>(ranked.bytes), static_cast<int64_t>(ranked.o_words),
                             tile.rb, tile.tg, tile.rec.leaf_bytes > 0};
  std::copy(words, words + 8, out);
}

template void PredictLaunch<float>(lbk_context*, Scratch&, const float*, int64_t, int64_t, int, int, int, const lbk_tree_ref*,
                                   int, int64_t, const double*, int, double*, int64_t, cudaStream_t);
template void PredictLaunch<double>(lbk_context*, Scratch&, const double*, int64_t, int64_t, int, int, int,
                                    const lbk_tree_ref*, int, int64_t, const double*, int, double*, int64_t, cudaStream_t);

}  // namespace lbk

extern "C" int lbk_selftest_predict_plan(lbk_context* ctx, int64_t n_rows, int n_features, int n_outputs, int n_trees, int max_nodes,
                                         int64_t total_nodes, int x_dtype, int transform, int64_t* out)
{
  return lbk::Guard(ctx, [&] {
    LBK_EXPECT(ctx != nullptr && out != nullptr, "null argument");
    LBK_EXPECT(x_dtype == LBK_F32 || x_dtype == LBK_F64, "X must be float32 or float64");
    LBK_EXPECT(n_rows >= 1 && n_features >= 1 && n_outputs >= 1 && n_trees >= 1 && max_nodes >= 1 && total_nodes >= 1, "bad shape");
    (x_dtype == LBK_F32 ? lbk::PlanOfPredict<float> : lbk::PlanOfPredict<double>)(ctx, n_rows, n_features, n_outputs, n_trees, max_nodes, total_nodes,
                                                                                 transform, out);
  });
}
