// lbk_build_tree and the stage-level entry points: host-side orchestration of one tree.
//
// Reference behaviour restated here: build_tree_fn / TreeBuilder, src/models/tree/build_tree.cu:
//   :1274-1359 task body (argument checks, level loop), :1000-1017 histogram cache rule,
//   :1191-1258 batching of a level when its histograms exceed the cache, :1154-1187 root,
//   :826-845 outputs.
// Differences in how, not in what: bins and quantised pairs are computed once per tree; rows are
// kept grouped by node with a two-way partition instead of a radix sort; only the nodes that are
// built are held in the reduction buffer that crosses ranks; a level is three launches (histograms, scan
// and split search, repartition), enqueued without host synchronisation (where the number of bins decides
// the layout the call waits once, for that number).
#include <algorithm>
#include <cstring>

#include "internal.h"
#include "split.cuh"

namespace lbk {
namespace {

// The node each row ends in, read off the binned matrix: "x <= split value" is "bin <= split bin"
// because a split value is one of the feature's proposals (the repartition relies on the same
// fact), so this is the walk the predict kernel does on X, on a quarter of the bytes (float32 X).
//
// Tiled form (rows of at most kLeafMaxPitch bytes, at most kLeafMaxNodes nodes): the load/store
// pipe spends one pass per distinct 128-byte line of a load, so a thread per row reading its own
// line costs 32 passes per level.  Instead a warp copies its 32 consecutive rows - one contiguous
// piece of the matrix - into shared memory with 16-byte loads (the shared rows are one word longer,
// which spreads equal features of the 32 rows over the banks), and the tree's nodes sit in shared
// memory too, feature + 1 and split bin packed into one word.
//
// In a boosting round the same kernel makes the tree's leaf values and hessians (every block its own table, where there
// are few enough; the first one writes them out) and adds the leaf values to the prediction (up to kLeafOutputs outputs),
// which took two launches more and the leaf record's way through memory: per round 200k x 50, depth 6: 9.2 -> 5.9 us; 10M x 64,
// depth 8: 182 -> 149.
constexpr int kLeafMaxPitch = 256;
constexpr int kLeafMaxNodes = 8192;
constexpr int kLeafWarps    = 8;
constexpr int kLeafTable    = 1024;  // leaf values (nodes x outputs) that every block makes for itself
constexpr int kLeafOutputs  = 24;    // up to so many a round adds where it finds the leaves
constexpr int kLeafAhead    = 4;     // of several outputs: values of a lane on their way

struct LeafRound {
  double* pred;      // [n_rows][K]
  int K;
  TreeArrays tree;   // node_sums != null: leaf_value and hessian are made here
  const QuantParams* qp;
  double l1, l2;
  double* hessian;
};

// kForm: 0 no round, 1 a round of one output, 2 of several
template <typename BinT, int kForm>
__global__ void __launch_bounds__(kLeafWarps * 32, kForm == 0 ? 6 : 5)
  k_leaf_of_row_tiled(const BinT* __restrict__ bins, int pitch_bytes, int64_t n_rows, const int32_t* __restrict__ feature,
                      const int32_t* __restrict__ split_bin, int max_depth, int n_nodes, int32_t* __restrict__ leaf,
                      const __grid_constant__ LeafRound rnd)
{
  AfterTheKernelBefore();
  constexpr bool kRound = kForm != 0;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  unsigned* s_node = reinterpret_cast<unsigned*>(smem_raw);
  __shared__ double s_value[kRound ? kLeafTable : 1];
  const double* value = rnd.tree.leaf_value;
  if (kRound && rnd.tree.node_sums != nullptr) {
    const QuantParams qp = *rnd.qp;
    for (int i = threadIdx.x; i < n_nodes * rnd.K; i += blockDim.x) {
      const double2 v = FinishedNode(rnd.tree, qp, rnd.K, i, rnd.l1, rnd.l2);
      s_value[i]      = v.x;
      if (blockIdx.x == 0) {
        rnd.tree.leaf_value[i] = v.x;
        rnd.hessian[i]         = v.y;
      }
    }
    value = s_value;
  }
  for (int i = threadIdx.x; i < n_nodes; i += blockDim.x) {
    const int f = feature[i];
    s_node[i]   = f < 0 ? 0u : (static_cast<unsigned>(f + 1) << 16) | static_cast<unsigned>(split_bin[i] & 0xffff);
  }
  __syncthreads();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int spitch = pitch_bytes + 4;  // bytes of a row in shared memory
  unsigned char* tile = smem_raw + (static_cast<size_t>(n_nodes) * 4 + 15) / 16 * 16 + static_cast<size_t>(warp) * 32 * spitch;
  const int vec_per_row  = pitch_bytes / 16;
  const int64_t n_chunks = (n_rows + 31) / 32;
  for (int64_t chunk = blockIdx.x * static_cast<int64_t>(kLeafWarps) + warp; chunk < n_chunks;
       chunk += static_cast<int64_t>(gridDim.x) * kLeafWarps) {
    const int64_t row0 = chunk * 32;
    const int rows     = static_cast<int>(n_rows - row0 < 32 ? n_rows - row0 : 32);
    const uint4* src   = reinterpret_cast<const uint4*>(reinterpret_cast<const unsigned char*>(bins) + row0 * pitch_bytes);
    const int n_vec    = rows * vec_per_row;
    double before = 0.0;  // (one output: on its way while the row is copied and walked)
    if (kForm == 1 && lane < rows) before = rnd.pred[row0 + lane];
    __syncwarp();  // the previous chunk's walks are done with the tile
    for (int v = lane; v < n_vec; v += 32) {
      const uint4 w = __ldcs(src + v);
      const int r = v / vec_per_row, c = v - r * vec_per_row;
      unsigned* dst = reinterpret_cast<unsigned*>(tile + r * spitch + c * 16);
      dst[0] = w.x;
      dst[1] = w.y;
      dst[2] = w.z;
      dst[3] = w.w;
    }
    __syncwarp();
    int node = 0;
    if (lane < rows) {
      const BinT* b = reinterpret_cast<const BinT*>(tile + lane * spitch);
      for (int d = 0; d < max_depth; ++d) {
        // a node without children in the arrays is a leaf (its feature is -1 by construction)
        const unsigned nd = node < n_nodes ? s_node[node] : 0u;
        if (nd == 0u) break;
        node = 2 * node + 1 + (static_cast<unsigned>(b[(nd >> 16) - 1]) > (nd & 0xffffu) ? 1 : 0);
      }
      if (leaf != nullptr) leaf[row0 + lane] = node;
      if (kForm == 1) rnd.pred[row0 + lane] = before + value[node];
    }
    if (kForm == 2) {
      // the lanes over the warp's rows x outputs, kLeafAhead of a lane's at a time: the loads of one after the other's
      // store would wait for memory each (depth 7, 16 outputs: 20k x 20 17.7 us, now 11.2, 200k x 30 31.0 and 17.6; ten outputs,
      // 1M x 100 65.5 and 55.6)
      double* p   = rnd.pred + row0 * rnd.K;
      const int n = rows * rnd.K;
      for (int e0 = lane; e0 - lane < n; e0 += 32 * kLeafAhead) {
        double sum[kLeafAhead], add[kLeafAhead];
#pragma unroll
        for (int u = 0; u < kLeafAhead; ++u)
          if (e0 + 32 * u < n) sum[u] = p[e0 + 32 * u];
#pragma unroll
        for (int u = 0; u < kLeafAhead; ++u) {
          const int e = e0 + 32 * u, r = e / rnd.K;
          const int nd = __shfl_sync(0xffffffffu, node, min(r, 31));
          if (e < n) add[u] = value[static_cast<int64_t>(nd) * rnd.K + (e - r * rnd.K)];
        }
#pragma unroll
        for (int u = 0; u < kLeafAhead; ++u)
          if (e0 + 32 * u < n) p[e0 + 32 * u] = sum[u] + add[u];
      }
    }
  }
}

// One thread per row, everything from global memory: wide rows and very deep trees.
template <typename BinT>
__global__ void __launch_bounds__(256)
  k_leaf_of_row(const BinT* __restrict__ bins, int64_t pitch, int64_t n_rows, const int32_t* __restrict__ feature,
                const int32_t* __restrict__ split_bin, int max_depth, int32_t* __restrict__ leaf)
{
  AfterTheKernelBefore();
  const int64_t row = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
  if (row >= n_rows) return;
  const BinT* b = bins + row * pitch;
  int node      = 0;
  for (int d = 0; d < max_depth; ++d) {
    const int f = __ldg(feature + node);
    if (f < 0) break;
    node = 2 * node + 1 + (static_cast<int>(b[f]) > __ldg(split_bin + node) ? 1 : 0);
  }
  leaf[row] = node;
}

bool LeafTiled(const void* bins, int64_t pitch_bytes, int F, int M)
{
  return pitch_bytes <= kLeafMaxPitch && M <= kLeafMaxNodes && F < 65535 && Aligned16(bins);
}

// `rnd`: a boosting round (LeafTiled only); leaf may then be null.
template <typename BinT>
void LeafOfRow(lbk_context* ctx, const void* bins, int64_t pitch, int64_t N, int F, const int32_t* feature,
               const int32_t* split_bin, int D, int M, int32_t* leaf, const LeafRound* rnd, cudaStream_t stream)
{
  const int64_t pitch_bytes = pitch * static_cast<int64_t>(sizeof(BinT));
  if (LeafTiled(bins, pitch_bytes, F, M)) {
    const size_t smem = (static_cast<size_t>(M) * 4 + 15) / 16 * 16 + static_cast<size_t>(kLeafWarps) * 32 * (pitch_bytes + 4);
    auto fn           = rnd == nullptr ? k_leaf_of_row_tiled<BinT, 0> : rnd->K == 1 ? k_leaf_of_row_tiled<BinT, 1> : k_leaf_of_row_tiled<BinT, 2>;
    if (smem > 36 * 1024) AllowSharedMemory(ctx, fn, 12 * 1024);  // (the limit without it counts the static part too)
    int per_sm = 0;
    LBK_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, kLeafWarps * 32, smem));
    const int64_t chunks = (N + 31) / 32;
    int64_t blocks       = static_cast<int64_t>(ctx->sm_count) * (per_sm > 0 ? per_sm : 1);
    blocks               = std::min<int64_t>(blocks, (chunks + kLeafWarps - 1) / kLeafWarps);
    LaunchChained(fn, static_cast<unsigned>(std::max<int64_t>(blocks, 1)), kLeafWarps * 32, smem, stream,
      static_cast<const BinT*>(bins), static_cast<int>(pitch_bytes), N, feature, split_bin, D, M, leaf,
      rnd != nullptr ? *rnd : LeafRound{});
  } else {
    const unsigned blocks = static_cast<unsigned>((N + 255) / 256);
    LaunchChained(k_leaf_of_row<BinT>, blocks, 256, 0, stream, static_cast<const BinT*>(bins), pitch, N, feature, split_bin, D, leaf);
  }
  LBK_LAUNCH_CHECK();
}

// out[i, :] = table[index[i], :]: the leaf values of the nodes a set of rows ended in.
__global__ void __launch_bounds__(256)
  k_gather_rows(const double* __restrict__ table, const int32_t* __restrict__ index, int64_t n, int K,
                double* __restrict__ out)
{
  AfterTheKernelBefore();
  const int64_t e = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
  if (e >= n * K) return;
  const int64_t i = e / K;
  const int k     = static_cast<int>(e - i * K);
  out[e]          = __ldg(table + static_cast<int64_t>(__ldg(index + i)) * K + k);
}

// The caller's sketch buffer: a header, then the split proposals, their row pointers, the binned
// matrix and its feature-major copy, each on a 512-byte boundary and sized for the widest case
// (two-byte bins when a feature can have more than 256 proposals).
constexpr int32_t kSketchMagic = 0x4c424b53;
struct SketchHeader {
  int32_t magic, total_bins, max_bins_per_feature, n_features, split_samples, elem_bytes, has_feature_major, pad;
  int64_t n_rows;
};
struct SketchLayout {
  size_t proposals, row_ptr, bins, bins_t, bytes;
};
SketchLayout SketchLayoutOf(int64_t N, int F, int S, size_t elem_bytes)
{
  auto up = [](size_t v) { return (v + 511) / 512 * 512; };
  const int bin_bytes   = S <= 256 ? 1 : 2;
  const int64_t pitch_t = (N + 31) / 32 * 32;
  SketchLayout l;
  l.proposals = up(sizeof(SketchHeader));
  l.row_ptr   = l.proposals + up(static_cast<size_t>(F) * S * elem_bytes);
  l.bins      = l.row_ptr + up(sizeof(int32_t) * (static_cast<size_t>(F) + 1));
  l.bins_t    = l.bins + up(lbk_bin_matrix_bytes(N, F, bin_bytes));
  l.bytes     = l.bins_t + up(static_cast<size_t>(F) * pitch_t * bin_bytes + 16);
  return l;
}

// pred[i] += table[leaf[i]]: the leaf values of a round's tree onto the current prediction
__global__ void __launch_bounds__(256)
  k_add_leaf_values(const double* __restrict__ table, const int32_t* __restrict__ leaf, int64_t n, int K,
                    double* __restrict__ pred)
{
  AfterTheKernelBefore();
  const int64_t e = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
  if (e >= n * K) return;
  const int64_t i = K == 1 ? e : e / K;
  const int k     = static_cast<int>(e - i * K);
  pred[e] += __ldg(table + static_cast<int64_t>(__ldg(leaf + i)) * K + k);
}

// Rows x features x outputs up to which a tree of more than 256 samples has the memory of two-byte ids, 32 MB for either
// matrix, before it knows whether one byte will do (BuildTreeImpl); above, nothing is laid out before the bins are counted.
constexpr int64_t kWidthLaterCells = int64_t{1} << 24;
constexpr int64_t kHistogramCacheBytes = 1000000000;  // (reference: build_tree.cu:1000-1017)

// Histograms of whole levels kept so that the level below need not build all its nodes, beyond the reference's cache (whose
// rule the results follow, see BuildTreeImpl).
constexpr int64_t kHeldHistogramBytes = 2000000000;

// Clears the slots of a batch's nodes where *gate is not 0: those of nodes that exist (parent_feature [n_nodes / 2]: their parents'
// splits) and are not clear already, which the first `clear` slots are - all of them, or (by_search) those of pairs that exist.
constexpr int kZeroPiece = 512;  // pairs that a warp clears at a time
__global__ void __launch_bounds__(256)
  k_zero_if(const int* __restrict__ gate, int4* __restrict__ at, int64_t slot, int n_nodes, const int32_t* __restrict__ parent_feature, int clear,
            bool by_search)
{
  AfterTheKernelBefore();
  if (*gate == 0) return;
  const int lane = threadIdx.x & 31;
  const int64_t pieces = (slot + kZeroPiece - 1) / kZeroPiece, items = pieces * n_nodes;
  for (int64_t item = (blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x) / 32; item < items; item += static_cast<int64_t>(gridDim.x) * blockDim.x / 32) {
    const int j = static_cast<int>(item / pieces);
    if (parent_feature[j >> 1] < 0 || (j < clear && (!by_search || parent_feature[j] >= 0))) continue;
    const int64_t from = (item - j * pieces) * kZeroPiece, to = from + kZeroPiece < slot ? from + kZeroPiece : slot;
    int4* dst = at + j * slot;
    for (int64_t i = from + lane; i < to; i += 32) dst[i] = make_int4(0, 0, 0, 0);
  }
}

// `round`: a boosting round instead of a tree on given gradients (they are those of round->pred, which gets
// the leaf values added); the call is then asynchronous.  held: levels may be held beyond the reference's cache; set while they are and
// the call, if it fails, may be made again.
template <typename T>
void BuildTreeImpl(lbk_context* ctx, const lbk_build_tree_args& a, cudaStream_t stream, const lbk_boost_round_args* round, bool* held)
{
  const int F = a.n_features, K = a.n_outputs, D = a.max_depth;
  const int64_t N = a.n_local_rows;
  const int M     = a.max_nodes;
  Scratch s(ctx, stream);
  HostWords words(ctx);

  const T* X      = static_cast<const T*>(a.X);
  const double* g = a.g;
  const double* h = a.h;
  const uint8_t* fset = a.feature_set;
  int64_t ldx = a.ldx, ldg = a.ldg;
  double *leaf_value = a.leaf_value, *split_value = a.split_value, *gain = a.gain, *hessian = a.hessian;
  int32_t* feature = a.feature;
  if (a.host_buffers) {
    // stage host inputs; outputs are produced on the device and copied back at the end
    T* dX = s.alloc<T>(static_cast<size_t>(N) * F);
    LBK_CUDA(cudaMemcpy2DAsync(dX, sizeof(T) * F, X, sizeof(T) * ldx, sizeof(T) * F, N > 0 ? N : 0, cudaMemcpyHostToDevice, stream));
    double* dg = s.alloc<double>(static_cast<size_t>(N) * K);
    double* dh = s.alloc<double>(static_cast<size_t>(N) * K);
    LBK_CUDA(cudaMemcpy2DAsync(dg, sizeof(double) * K, g, sizeof(double) * ldg, sizeof(double) * K, N > 0 ? N : 0, cudaMemcpyHostToDevice, stream));
    LBK_CUDA(cudaMemcpy2DAsync(dh, sizeof(double) * K, h, sizeof(double) * ldg, sizeof(double) * K, N > 0 ? N : 0, cudaMemcpyHostToDevice, stream));
    X   = dX;
    g   = dg;
    h   = dh;
    ldx = F;
    ldg = K;
    if (fset) {
      uint8_t* df = s.alloc<uint8_t>(F);
      LBK_CUDA(cudaMemcpyAsync(df, fset, F, cudaMemcpyHostToDevice, stream));
      fset = df;
    }
    leaf_value  = s.alloc<double>(static_cast<size_t>(M) * K);
    hessian     = s.alloc<double>(static_cast<size_t>(M) * K);
    split_value = s.alloc<double>(M);
    gain        = s.alloc<double>(M);
    feature     = s.alloc<int32_t>(M);
  }
  auto copy_tree_back = [&]() {
    LBK_CUDA(cudaMemcpyAsync(a.leaf_value, leaf_value, sizeof(double) * M * K, cudaMemcpyDeviceToHost, stream));
    LBK_CUDA(cudaMemcpyAsync(a.feature, feature, sizeof(int32_t) * M, cudaMemcpyDeviceToHost, stream));
    LBK_CUDA(cudaMemcpyAsync(a.split_value, split_value, sizeof(double) * M, cudaMemcpyDeviceToHost, stream));
    LBK_CUDA(cudaMemcpyAsync(a.gain, gain, sizeof(double) * M, cudaMemcpyDeviceToHost, stream));
    LBK_CUDA(cudaMemcpyAsync(a.hessian, hessian, sizeof(double) * M * K, cudaMemcpyDeviceToHost, stream));
  };

  // The kernels work on node sums in the caller's own array where they can: device memory that their 16-byte accesses may
  // go to.  Else the sums are copied there at the end.
  const bool keep_sums = a.trace_node_sums != nullptr && !a.host_buffers && Aligned16(a.trace_node_sums);

  // Tree (reference: struct Tree, build_tree.cu:785-809)
  if (ctx->n_ranks <= 1 && a.sketch_mode == LBK_SKETCH_OFF && a.trace_hist == nullptr &&
      SmallTreeFits(ctx, N, F, K, D, a.split_samples)) {
    SmallTreeArgs<T> t{};
    t.X            = X;
    t.ldx          = ldx;
    t.N            = N;
    t.F            = F;
    t.K            = K;
    t.D            = D;
    t.S            = a.split_samples;
    t.seed         = a.seed;
    t.row_offset   = a.row_offset;
    t.dataset_rows = a.dataset_rows;
    t.g            = g;
    t.h            = h;
    t.ldg          = ldg;
    t.objective    = -1;
    const bool fused = round != nullptr && (round->objective == LBK_SQUARED_ERROR || K == 1);
    if (fused) {
      t.objective = round->objective;
      t.y         = round->y;
      t.pred      = round->pred;
      t.lr        = round->learning_rate;
    } else if (round != nullptr) {
      double* rg = s.alloc<double>(static_cast<size_t>(N) * K);
      double* rh = s.alloc<double>(static_cast<size_t>(N) * K);
      Gradient(round->objective, round->pred, round->y, N, K, round->learning_rate, rg, rh, stream);
      t.g   = rg;
      t.h   = rh;
      t.ldg = K;
    }
    t.sp          = SplitParams{a.l1_regularization, a.l2_regularization, a.min_split_gain, fset};
    t.tree        = TreeArrays{leaf_value, feature, split_value, gain,
                        keep_sums ? reinterpret_cast<GPairI64*>(a.trace_node_sums) : s.alloc<GPairI64>(static_cast<size_t>(M) * K),
                        nullptr, M};
    t.hessian     = hessian;
    int32_t* leaf = a.out_leaf != nullptr && !a.host_buffers ? a.out_leaf
                    : a.out_leaf != nullptr || (round != nullptr && !fused) ? s.alloc<int32_t>(static_cast<size_t>(N)) : nullptr;
    t.leaf        = leaf;
    t.barrier     = round != nullptr ? static_cast<unsigned int*>(round->zeroed) : nullptr;
    if (t.barrier == nullptr) {
      t.barrier = s.alloc<unsigned int>(1);
      LBK_CUDA(cudaMemsetAsync(t.barrier, 0, sizeof(unsigned int), stream));
    }
    t.info_host = a.out_total_bins != nullptr ? words.get() : nullptr;
    SmallTree<T>(ctx, s, t, stream);
    if (round != nullptr && !fused) {
      LaunchChained(k_add_leaf_values, static_cast<unsigned>((N * K + 255) / 256), 256, 0, stream, leaf_value, leaf, N, K, round->pred);
      LBK_LAUNCH_CHECK();
    }
    if (a.trace_node_sums && !keep_sums)
      LBK_CUDA(cudaMemcpyAsync(a.trace_node_sums, t.tree.node_sums, sizeof(GPairI64) * M * K, cudaMemcpyDefault, stream));
    if (a.host_buffers) {
      if (a.out_leaf) LBK_CUDA(cudaMemcpyAsync(a.out_leaf, leaf, sizeof(int32_t) * N, cudaMemcpyDeviceToHost, stream));
      copy_tree_back();
    }
    if (round != nullptr) return;
    CheckDeviceStatus(ctx, stream);
    words.settled();
    if (a.out_total_bins) *a.out_total_bins = words.get()[0];
    return;
  }
  GradientForm form;
  if (round != nullptr && round->objective == LBK_SQUARED_ERROR) {
    form = GradientForm{true, round->learning_rate};
    g    = round->pred;
    h    = round->y;
    ldg  = K;
  } else if (round != nullptr) {
    double* rg = s.alloc<double>(static_cast<size_t>(N) * K);
    double* rh = s.alloc<double>(static_cast<size_t>(N) * K);
    Gradient(round->objective, round->pred, round->y, N, K, round->learning_rate, rg, rh, stream);
    g   = rg;
    h   = rh;
    ldg = K;
  }
  TreeArrays tree;
  tree.leaf_value  = leaf_value;
  tree.feature     = feature;
  tree.split_value = split_value;
  tree.gain        = gain;
  tree.split_bin   = s.alloc<int32_t>(M);
  tree.max_nodes   = M;

  const bool sketch_save = a.sketch_mode == LBK_SKETCH_SAVE, sketch_reuse = a.sketch_mode == LBK_SKETCH_REUSE;
  const int S            = a.split_samples;
  const SketchLayout sk  = SketchLayoutOf(N, F, S, sizeof(T));
  unsigned char* skb     = static_cast<unsigned char*>(a.sketch);
  const bool in_sketch   = sketch_save || sketch_reuse;
  T* cuts          = in_sketch ? reinterpret_cast<T*>(skb + sk.proposals) : s.alloc<T>(static_cast<size_t>(F) * S);
  int32_t* row_ptr = in_sketch ? reinterpret_cast<int32_t*>(skb + sk.row_ptr) : s.alloc<int32_t>(F + 1);

  // Does the host have to know how many bins there are before anything is laid out?  They decide the batches of a level
  // whose histograms are larger than the cache (the reference's rule, below), the layout that a trace, a sketch or other
  // ranks see and, above 256 samples, the memory for the ids of a large matrix or for a root of more than the cache.
  // Otherwise everything is laid out for the upper bound F x S, and up to 256 samples nothing waits for the device before
  // the end of the tree.  Above them the width of the ids is still open: the host polls for the largest feature's number of
  // bins, which the device has before it has summed |g| and quantised the pairs, so that it does not run dry (to wait
  // for the stream and then lay out and queue everything costs 15 us per tree of 300k x 37 float64, this nothing).
  // Three rounds of depth 6, two-byte ids whatever the columns hold and the width they ask for: columns of 50 values,
  // 300k x 37 float64, 512 samples 1068 and 964 us, 2048 samples 1500 and 1123; 100k x 64 1155 and 1039 (2048), 921 and 879
  // (300); 8k x 500 1265 and 1190 (300); 10^6 values, 300k x 37 1242 and 1244, 100k x 64 1043 and 1042, 5k x 20 884 and 882.
  // (Trees of few rows are bound by the host: two rounds of 1.4k x 48, 512 samples, all values distinct 667 and 677.)
  auto cache_depth = [&](int64_t bins, size_t& max_histogram_nodes) {
    // histogram cache rule (reference: build_tree.cu:1000-1017); identical on every rank
    max_histogram_nodes = std::max<size_t>(1, static_cast<size_t>(kHistogramCacheBytes) / (static_cast<size_t>(K) * bins * sizeof(GPairI64)));
    int d = 0;
    while (static_cast<size_t>(LevelEnd(d + 1)) <= max_histogram_nodes && d <= D) d++;
    return d;
  };
  const int64_t bins_bound   = static_cast<int64_t>(F) * S;
  size_t max_histogram_nodes = 0;
  const bool wait_for_bins   = in_sketch || a.trace_hist != nullptr || ctx->n_ranks > 1 ||
                             (S > 256 && (N * F * K > kWidthLaterCells ||
                                          bins_bound * K > kHistogramCacheBytes / static_cast<int64_t>(sizeof(GPairI64)))) ||
                             cache_depth(bins_bound, max_histogram_nodes) < D - 1;
  const bool wait_for_width  = S > 256 && !wait_for_bins;

  // words that have to be zero before the first level: node sums, arrival counters and partition cursors of
  // the nodes, tickets and merge counters of the histogram launches
  constexpr int kTickets = 256;
  HistScratch hist_scratch;
  HistScratchNeeds(ctx, F, K, S <= 256 ? 1 : 2, S, N, hist_scratch);
  size_t zero_bytes = 0;
  auto reserve = [&](size_t bytes) {
    const size_t at = zero_bytes;
    zero_bytes += (bytes + 15) / 16 * 16;
    return at;
  };
  const size_t o_sums    = reserve(keep_sums ? 0 : sizeof(GPairI64) * M * K);
  const size_t o_arrived = reserve(sizeof(unsigned int) * M);
  const size_t o_cursor  = reserve(sizeof(unsigned long long) * M);
  const size_t o_ticket  = reserve(sizeof(unsigned int) * kTickets);
  const size_t o_arrive  = reserve(sizeof(unsigned int) * hist_scratch.n_arrive);
  const size_t o_abs     = reserve(3 * sizeof(int));
  unsigned char* zeroed  = static_cast<unsigned char*>(s.alloc_bytes(zero_bytes));
  tree.node_sums = keep_sums ? reinterpret_cast<GPairI64*>(a.trace_node_sums) : reinterpret_cast<GPairI64*>(zeroed + o_sums);
  unsigned int* split_arrived  = reinterpret_cast<unsigned int*>(zeroed + o_arrived);
  unsigned long long* cursor   = reinterpret_cast<unsigned long long*>(zeroed + o_cursor);
  int* max_abs                 = reinterpret_cast<int*>(zeroed + o_abs);
  int* hess_below_one          = max_abs + 2;
  hist_scratch.tickets         = reinterpret_cast<unsigned int*>(zeroed + o_ticket);
  hist_scratch.n_tickets       = kTickets;
  hist_scratch.arrive          = reinterpret_cast<unsigned int*>(zeroed + o_arrive);

  // segments of a level's nodes: begins, then ends
  const size_t max_level_nodes = D > 0 ? (size_t{1} << (D - 1)) : 1;
  int32_t* seg_a  = s.alloc<int32_t>(2 * max_level_nodes);
  int32_t* seg_b  = s.alloc<int32_t>(2 * max_level_nodes);
  QuantParams* qp = s.alloc<QuantParams>(1);
  double* sums    = s.alloc<double>(2);
  int32_t* info   = s.alloc<int32_t>(2);
  SketchHeader head{};
  if (sketch_reuse) {
    LBK_CUDA(cudaMemcpyAsync(&head, skb, sizeof(head), cudaMemcpyDeviceToHost, stream));
    LBK_CUDA(cudaStreamSynchronize(stream));
    LBK_EXPECT(head.magic == kSketchMagic, "the sketch buffer holds no saved sketch");
    LBK_EXPECT(head.n_rows == N && head.n_features == F && head.split_samples == S &&
                 head.elem_bytes == static_cast<int32_t>(sizeof(T)),
               "the sketch was saved for a matrix of another shape or type");
    LBK_EXPECT(D <= 1 || head.has_feature_major, "the sketch was saved without the feature-major copy");
  }
  // the root's histogram, where its size is known already
  const bool root_zeroed = !wait_for_bins && D > 0;
  GPairI64* cache        = nullptr;
  if (root_zeroed)
    cache = s.alloc<GPairI64>(static_cast<size_t>(LevelEnd(std::max(D - 2, 0))) * K * bins_bound);
  {
    PrologueArgs<T> pa{};
    pa.X            = X;
    pa.ldx          = ldx;
    pa.row_offset   = a.row_offset;
    pa.n_local      = N;
    pa.F            = F;
    pa.S            = S;
    pa.seed         = a.seed;
    pa.dataset_rows = a.dataset_rows;
    pa.cuts         = cuts;
    pa.counts       = sketch_reuse ? nullptr : s.alloc<int32_t>(F);
    pa.g            = g;
    pa.h            = h;
    pa.ldg          = ldg;
    pa.form         = form;
    pa.K            = K;
    pa.n_elements   = N * K;
    pa.tree         = tree;
    pa.root_begin   = seg_a;
    pa.root_end     = seg_a + max_level_nodes;
    pa.zero[0]      = zeroed;
    pa.zero_n16[0]  = static_cast<int64_t>(zero_bytes / 16);
    pa.zero[1]      = tree.node_sums;
    pa.zero_n16[1]  = keep_sums ? static_cast<int64_t>(M) * K : 0;
    pa.zero[2]      = cache;
    pa.zero_n16[2]  = root_zeroed ? static_cast<int64_t>(K) * bins_bound : 0;
    // (a sketch that is reused knows its bins: no kernel counts any and no words are borrowed for them)
    int32_t* info_host = !sketch_reuse && (wait_for_bins || wait_for_width || a.out_total_bins) ? words.get() : nullptr;
    if (wait_for_width) words.expect();
    Prologue<T>(ctx, s, pa, row_ptr, info, info_host, sums, qp, stream);
  }
  ProposalInfo pi{static_cast<int>(std::min<int64_t>(bins_bound, INT32_MAX)), S};
  if (sketch_reuse) {
    pi.total_bins           = head.total_bins;
    pi.max_bins_per_feature = head.max_bins_per_feature;
  } else if (wait_for_bins) {
    LBK_CUDA(cudaStreamSynchronize(stream));
    pi.total_bins           = words.get()[0];
    pi.max_bins_per_feature = words.get()[1];
    words.settled();
    LBK_EXPECT(pi.total_bins >= F, "every feature must have at least one proposal");
  }
  const int B = pi.total_bins;  // (an upper bound unless wait_for_bins)
  const int* max_bins_ptr = wait_for_bins || wait_for_width ? nullptr : info + 1;

  // binned matrix, once per tree
  const int bin_bytes_bound = pi.max_bins_per_feature <= 256 ? 1 : 2;
  void* bins = in_sketch ? static_cast<void*>(skb + sk.bins) : s.alloc_bytes(lbk_bin_matrix_bytes(N, F, bin_bytes_bound));
  // feature-major copy for the repartition (no copy for a stump: nothing is repartitioned; a saved
  // sketch always has it, later trees may be deeper)
  const int64_t pitch_t = (N + 31) / 32 * 32;
  void* bins_t          = in_sketch ? static_cast<void*>(skb + sk.bins_t)
                          : D > 1   ? s.alloc_bytes(static_cast<size_t>(F) * pitch_t * bin_bytes_bound + 16)
                                    : nullptr;

  // quantised pairs and root sums
  int2* gpair   = s.alloc<int2>(static_cast<size_t>(N) * K);
  auto quantise = [&]() {
    Quantise(ctx, g, h, ldg, form, a.row_offset, N, K, a.seed, gpair, tree.node_sums, qp, max_abs, hess_below_one, stream);
  };
  if (wait_for_width) {
    quantise();
    words.await(stream);
    pi.max_bins_per_feature = words.get()[1];
    LBK_EXPECT(words.get()[0] >= F, "every feature must have at least one proposal");
  }
  const int bin_bytes = pi.max_bins_per_feature <= 256 ? 1 : 2;
  if (!sketch_reuse)
    BinMatrix<T>(X, ldx, N, F, cuts, S, row_ptr, bins, bins_t, pitch_t, bin_bytes, pi.max_bins_per_feature, ctx->d_status, stream);
  if (sketch_save) {
    head.magic                = kSketchMagic;
    head.total_bins           = pi.total_bins;
    head.max_bins_per_feature = pi.max_bins_per_feature;
    head.n_features           = F;
    head.split_samples        = S;
    head.elem_bytes           = static_cast<int32_t>(sizeof(T));
    head.has_feature_major    = 1;
    head.n_rows               = N;
    LBK_CUDA(cudaMemcpyAsync(skb, &head, sizeof(head), cudaMemcpyHostToDevice, stream));
    LBK_CUDA(cudaStreamSynchronize(stream));  // `head` is on this frame
  }

  if (!wait_for_width) quantise();

  const int cdepth = cache_depth(B, max_histogram_nodes);
  // levels >= D are never evaluated; no need to hold them.  The last level's histograms are evaluated as
  // they are scanned and not written, unless they are built in place or a trace wants them.
  int cache_levels = std::min(cdepth, std::max(D - 1, 0));
  const int64_t max_batch = static_cast<int>(max_histogram_nodes);
  // The reference builds all nodes of a level outside its cache.  A node that is built and one that is derived differ only where
  // a prefix has no hessian but a gradient (the scan then leaves the raw bin): never, if every quantised hessian is at
  // least one, since such a prefix has no rows, and a split's children have a positive hessian.  The quantiser
  // finds out; where it is so, such a level is derived too, from the level above, which is kept up to kHeldHistogramBytes: half
  // of the rows are summed and half of the histograms read.  Level 7 of 1M x 100, ten classes: 808 -> 324 us for the
  // histograms and 391 -> 302 for scan and search; the launch that finds the other answer 4 us.
  bool hold = held != nullptr && ctx->n_ranks <= 1 && a.trace_hist == nullptr && max_batch > 1 && cdepth < D - 1;
  const int reference_levels = cache_levels;
  while (hold && cache_levels < D - 1 && LevelEnd(cache_levels + 1) * static_cast<int64_t>(K) * B * static_cast<int64_t>(sizeof(GPairI64)) <= kHeldHistogramBytes)
    ++cache_levels;
  const int cache_end_ref = LevelEnd(cdepth);  // extent of the reference's cached histogram
  const size_t node_elems = static_cast<size_t>(K) * B;

  // What a tree needs whatever its levels are derived from comes first.
  // rows grouped by node, ping-pong; the root's rows are in order and need no list
  int32_t* rows_a = nullptr;
  int32_t* rows_b = D > 1 ? s.alloc<int32_t>(N) : nullptr;
  int32_t* rows_c = D > 2 ? s.alloc<int32_t>(N) : nullptr;
  // With few outputs the quantised pairs are kept in row_index order: at the root that is the order
  // they are in already, and every repartition moves them together with the row ids (8 K bytes read
  // and written per row and level, as streams), so that the histogram kernel reads the pairs of a
  // node as a stream instead of gathering 8 bytes per row from all over the array.
  constexpr int kMaxStreamedOutputs = 4;
  const bool stream_pairs = K <= kMaxStreamedOutputs && D > 0;
  int2* pairs_a = gpair;
  int2* pairs_b = stream_pairs && D > 1 ? s.alloc<int2>(static_cast<size_t>(N) * K) : nullptr;
  if (hist_scratch.partial_bytes > 0 && N > 0) hist_scratch.partial = s.alloc_bytes(hist_scratch.partial_bytes);
  // leaves of the rows, where something wants them: by the kernel that finds them.  A warp adds the outputs of 32 rows: of many outputs
  // and few rows too little is in flight.  Depth 7, this and the three kernels: 5k x 60, 16 outputs 11.7 and 12.5 us, 40 outputs 17.2
  // and 12.6, 100 outputs 62 and 14 (with one value of a lane on its way); 200k x 30, 16 outputs 17.6 and 25.4, 40 outputs 27.8 and 43.5.
  const int64_t pitch  = static_cast<int64_t>((F + kGroup - 1) / kGroup) * kGroup;
  const bool add_here  = round != nullptr && N > 0 && K <= kLeafOutputs && LeafTiled(bins, pitch * bin_bytes, F, M);
  const bool make_here = add_here && static_cast<int64_t>(M) * K <= kLeafTable;
  int32_t* d_leaf      = nullptr;
  if ((a.out_leaf != nullptr || round != nullptr) && N > 0)
    d_leaf = a.out_leaf != nullptr && !a.host_buffers ? a.out_leaf
             : a.out_leaf != nullptr || !add_here     ? s.alloc<int32_t>(static_cast<size_t>(N)) : nullptr;

  // raw sums of the built nodes of a level, alternating so that a level can zero the next one's
  GPairI64* built[2]    = {nullptr, nullptr};
  size_t built_nodes[2] = {0, 0};
  auto built_buffer = [&](int which, size_t nodes) {
    if (built_nodes[which] < nodes) {
      if (built[which]) s.free_one(built[which]);
      built[which]       = nullptr;
      built_nodes[which] = 0;
      built[which]       = s.alloc<GPairI64>(nodes * node_elems);
      built_nodes[which] = nodes;
    }
    return built[which];
  };
  GPairI64* fresh    = nullptr;  // histogram of a batch that lies outside the cache
  size_t fresh_nodes = 0;
  auto fresh_buffer = [&](size_t nodes) {
    if (fresh_nodes < nodes) {
      if (fresh) s.free_one(fresh);
      fresh       = nullptr;
      fresh_nodes = 0;
      fresh       = s.alloc<GPairI64>(nodes * node_elems);
      fresh_nodes = nodes;
    }
    return fresh;
  };
  auto allocate_cache = [&]() {
    const bool last_held = a.trace_hist != nullptr || cache_levels < D - 1 || D <= 1;
    cache = s.alloc<GPairI64>(static_cast<size_t>(last_held ? LevelEnd(cache_levels) : LevelEnd(D - 2)) * node_elems);
  };
  // Levels that are derived beyond the reference's cache take more memory than if they were built: the levels held, and a
  // buffer for all nodes of each of them.  All of that is asked for here; if there is no room, nothing is held.
  if (hold) {
    size_t nodes[3] = {0, 0, 0};  // of either built buffer, of a batch
    for (int depth = 1; depth < D; ++depth) {
      const int64_t level = int64_t{1} << depth, batch = std::min(level, max_batch & ~int64_t{1});
      size_t& most        = nodes[depth <= cdepth || LevelBegin(depth) <= LevelEnd(cache_levels) ? depth & 1 : 2];
      most                = std::max<size_t>(most, depth <= cdepth ? level / 2 : batch);
    }
    try {
      allocate_cache();
      for (int which : {0, 1}) built_buffer(which, nodes[which]);
      fresh_buffer(nodes[2]);
    } catch (const Error& e) {
      if (e.code != LBK_ERR_ALLOC) throw;
      for (GPairI64* p : {built[0], built[1], fresh, cache})
        if (p != nullptr) s.free_one(p);
      built[0] = built[1] = fresh = cache = nullptr;
      built_nodes[0] = built_nodes[1] = fresh_nodes = 0;
      hold         = false;
      cache_levels = reference_levels;
    }
    if (held != nullptr) *held = hold;
  }
  if (cache == nullptr) allocate_cache();
  const int cache_nodes = LevelEnd(cache_levels);

  SplitParams sp{a.l1_regularization, a.l2_regularization, a.min_split_gain, fset};

  bool built_zeroed = root_zeroed;
  // the most recently replaced "cache" of the reference, to decide parent availability
  int ref_hist_begin = 0, ref_hist_end = cache_end_ref;

  // the exchange buffers of a multi-rank call, sized once for the largest batch of the tree (the
  // receive form needs up to twice a batch: see BuildHistogramSummed)
  const size_t exchange_bytes =
    2 * sizeof(GPairI64) * node_elems * static_cast<size_t>(std::min<int64_t>(max_batch, static_cast<int64_t>(max_level_nodes))) +
    (size_t{1} << 20);

  for (int depth = 0; depth < D; ++depth) {
    const int level_begin = LevelBegin(depth), level_end = LevelEnd(depth);
    const int level_nodes = level_end - level_begin;
    // batches (reference: PrepareBatches, :1207-1258)
    std::vector<std::pair<int, int>> batches;
    if (level_nodes <= max_batch) {
      batches.push_back({level_begin, level_end});
    } else {
      // (Siblings stay in one batch where a batch has room for two.  The nodes of these levels are built one by one in the
      // reference, so that the boundaries carry no meaning.)
      const int64_t size = hold ? max_batch & ~int64_t{1} : max_batch;
      for (int64_t bb = level_begin; bb < level_end; bb += size)
        batches.push_back({static_cast<int>(bb), static_cast<int>(std::min<int64_t>(bb + size, level_end))});
    }
    for (auto [nb, ne] : batches) {
      const int n_nodes = ne - nb;
      // GetHistogram (:1191-1205): a batch outside the current histogram replaces it
      const bool in_ref_hist = nb >= ref_hist_begin && ne <= ref_hist_end;
      if (!in_ref_hist) {
        ref_hist_begin = nb;
        ref_hist_end   = ne;
      }
      // a parent's histogram is there only for the whole levels of the cache
      const bool derive = nb > 0 && ((nb - 1) / 2) >= ref_hist_begin && ((nb - 1) / 2) < ref_hist_end;
      const bool in_cache = ne <= cache_nodes;
      // derived all the same, unless the quantiser says no: the device decides (hess_below_one)
      const bool may_derive = hold && !derive && depth > 0 && level_begin <= cache_nodes && n_nodes % 2 == 0;
      // is this batch's histogram written out?  The level below reads it if it derives from it.
      const bool write_hist = (depth < D - 1 && (in_cache || !may_derive)) || a.trace_hist != nullptr;
      // where this batch's histograms live
      GPairI64* level_hist = nullptr;
      if (in_cache) {
        if (write_hist || !(derive || may_derive)) level_hist = cache + static_cast<size_t>(nb) * node_elems;
      } else if (!may_derive) {
        level_hist = fresh_buffer(n_nodes);
      }
      const int n_slots = derive || may_derive ? n_nodes / 2 : n_nodes;  // (all n_nodes of the buffer where may_derive comes to no)
      // With several ranks the level is built into a buffer the other ranks' GPUs can read, and
      // every rank sums, scans and searches only the features it owns (see exchange.cu); where the
      // peers cannot be mapped the whole buffer is all-reduced and every rank does everything.
      const bool owned = ctx->n_ranks > 1 && EnsureExchange(ctx, exchange_bytes, stream);
      const int f_begin = owned ? OwnedBegin(ctx->rank, ctx->n_ranks, F) : 0;
      const int f_end   = owned ? OwnedBegin(ctx->rank + 1, ctx->n_ranks, F) : F;
      // built buffer: when nothing is derived the level histogram itself is the target
      GPairI64* target = derive ? built_buffer(depth & 1, n_slots) : may_derive ? built_buffer(depth & 1, n_nodes) : level_hist;
      if (may_derive) {
        LaunchChained(k_zero_if, ctx->sm_count * 8, 256, 0, stream, hess_below_one, reinterpret_cast<int4*>(target), static_cast<int64_t>(node_elems), n_nodes,
                                                         tree.feature + (nb - 1) / 2, n_slots, built_zeroed);
        LBK_LAUNCH_CHECK();
      }
      if (a.trace_hist != nullptr && derive)  // (nodes that do not exist read as zeros in a trace)
        LBK_CUDA(cudaMemsetAsync(level_hist, 0, sizeof(GPairI64) * n_nodes * node_elems, stream));

      HistLevel lv;
      lv.bins                 = bins;
      lv.bin_bytes            = bin_bytes;
      lv.n_rows               = N;
      lv.F                    = F;
      lv.K                    = K;
      lv.B                    = B;
      lv.max_bins_per_feature = pi.max_bins_per_feature;
      lv.max_bins_ptr         = max_bins_ptr;
      lv.row_ptr              = row_ptr;
      lv.gpair                = stream_pairs ? pairs_a : gpair;
      lv.pairs_by_position    = stream_pairs;
      lv.gpair_f              = nullptr;
      lv.max_abs              = max_abs;
      lv.row_index            = rows_a;
      lv.seg_begin            = seg_a + (nb - level_begin);
      lv.seg_end              = seg_a + max_level_nodes + (nb - level_begin);
      lv.n_nodes              = n_nodes;
      lv.node_sums            = derive || may_derive ? tree.node_sums : nullptr;
      lv.build_all            = may_derive ? hess_below_one : nullptr;
      lv.node_begin           = nb;
      lv.out                  = target;
      lv.float_mode           = false;
      lv.scratch              = &hist_scratch;
      // build + sum over ranks (reference: :1107-1113 reduces the whole batch; only built nodes here)
      const GPairI64* summed = static_cast<const GPairI64*>(
        BuildHistogramSummed(ctx, s, lv, n_slots, HistSum::kSumOwned, false, !built_zeroed, stream));

      ScanSplitLevel sl;
      sl.built        = summed;
      sl.level_hist   = level_hist;
      sl.parent_begin = derive || may_derive ? LevelBegin(depth - 1) : 0;
      sl.parent_hist  = derive || may_derive ? cache + static_cast<size_t>(sl.parent_begin) * node_elems : nullptr;
      // does the next level derive?  (the same rule as above, one level ahead)
      const int next_begin = LevelBegin(depth + 1), next_end = LevelEnd(depth + 1);
      const bool next_derives = depth + 1 < D && level_nodes * int64_t{2} <= max_batch && next_begin >= ref_hist_begin &&
                                next_end <= ref_hist_end && (next_begin - 1) / 2 >= ref_hist_begin;
      const bool next_may = hold && depth + 1 < D && !next_derives && level_nodes * int64_t{2} <= max_batch && next_begin <= cache_nodes;
      built_zeroed    = (next_derives || next_may) && batches.size() == 1 && ctx->n_ranks <= 1;
      sl.next_built   = built_zeroed ? built_buffer((depth + 1) & 1, next_may ? 2 * n_nodes : n_nodes) : nullptr;
      sl.bin_stride   = B;
      sl.node_begin   = nb;
      sl.n_nodes      = n_nodes;
      sl.K            = K;
      sl.f_begin      = f_begin;
      sl.f_end        = f_end;
      sl.derive       = derive || may_derive;
      sl.write_hist   = write_hist;
      sl.cells        = N * F * K;
      sl.build_all    = lv.build_all;
      ScanSplit<T>(ctx, s, sl, F, row_ptr, cuts, S, qp, sp, tree, split_arrived, owned, stream);
      if (may_derive) {  // the other answer: one of the two launches does nothing
        sl.derive = false;
        ScanSplit<T>(ctx, s, sl, F, row_ptr, cuts, S, qp, sp, tree, split_arrived, owned, stream);
      }
      if (a.trace_hist && nb < a.trace_nodes) {
        const int cnt = std::min(ne, a.trace_nodes) - nb;
        LBK_CUDA(cudaMemcpyAsync(a.trace_hist + static_cast<size_t>(nb) * node_elems * 2, level_hist,
                                 sizeof(GPairI64) * cnt * node_elems, cudaMemcpyDeviceToDevice, stream));
      }
    }
    if (depth < D - 1) {
      PartitionLevel pl;
      pl.bins          = bins_t;
      pl.bin_bytes     = bin_bytes;
      pl.bin_pitch     = pitch_t;
      pl.n_features    = F;
      pl.n_rows        = N;
      pl.row_index_in  = rows_a;
      pl.seg_begin     = seg_a;
      pl.seg_end       = seg_a + max_level_nodes;
      pl.row_index_out = rows_b;
      pl.seg_begin_out = seg_b;
      pl.seg_end_out   = seg_b + max_level_nodes;
      pl.cursor        = cursor;
      pl.node_begin    = level_begin;
      pl.n_nodes       = level_nodes;
      pl.feature       = tree.feature;
      pl.split_bin     = tree.split_bin;
      if (stream_pairs) {
        pl.pairs_in  = pairs_a;
        pl.pairs_out = pairs_b;
        pl.K         = K;
      }
      PartitionRows(ctx, s, pl, stream);
      // the lists alternate; the root had none
      int32_t* spare = depth == 0 ? rows_c : rows_a;
      rows_a         = rows_b;
      rows_b         = spare;
      std::swap(seg_a, seg_b);
      std::swap(pairs_a, pairs_b);
    }
  }

  if (held != nullptr) *held = false;
  if (!make_here) FinishTree(tree, qp, K, a.l1_regularization, a.l2_regularization, hessian, stream);
  if ((a.out_leaf != nullptr || round != nullptr) && N > 0) {
    LeafRound rnd{};
    if (add_here) {
      rnd = LeafRound{round->pred, K, tree, qp, a.l1_regularization, a.l2_regularization, hessian};
      if (!make_here) rnd.tree.node_sums = nullptr;
    }
    const LeafRound* r = add_here ? &rnd : nullptr;
    if (bin_bytes == 1) LeafOfRow<uint8_t>(ctx, bins, pitch, N, F, tree.feature, tree.split_bin, D, M, d_leaf, r, stream);
    else LeafOfRow<uint16_t>(ctx, bins, pitch, N, F, tree.feature, tree.split_bin, D, M, d_leaf, r, stream);
    if (a.host_buffers && a.out_leaf)
      LBK_CUDA(cudaMemcpyAsync(a.out_leaf, d_leaf, sizeof(int32_t) * N, cudaMemcpyDeviceToHost, stream));
    if (round != nullptr && !add_here) {
      LaunchChained(k_add_leaf_values, static_cast<unsigned>((N * K + 255) / 256), 256, 0, stream, leaf_value, d_leaf, N, K, round->pred);
      LBK_LAUNCH_CHECK();
    }
  }
  if (a.trace_node_sums && !keep_sums)
    LBK_CUDA(cudaMemcpyAsync(a.trace_node_sums, tree.node_sums, sizeof(GPairI64) * M * K, cudaMemcpyDefault, stream));
  if (a.host_buffers) copy_tree_back();
  if (round != nullptr) return;
  CheckDeviceStatus(ctx, stream);  // synchronises, as the reference's task does (:1356)
  words.settled();
  if (a.out_total_bins) *a.out_total_bins = sketch_reuse ? head.total_bins : words.get()[0];
}

// Where what a level allocates for itself finds no room beside the levels that are held, the tree is made again without them: all that it
// is made from is as it was, and its outputs are written anew.
template <typename T>
void BuildTree(lbk_context* ctx, const lbk_build_tree_args& a, cudaStream_t stream, const lbk_boost_round_args* round)
{
  bool held = false;
  try {
    BuildTreeImpl<T>(ctx, a, stream, round, &held);
  } catch (const Error& e) {
    if (e.code != LBK_ERR_ALLOC || !held) throw;
    BuildTreeImpl<T>(ctx, a, stream, round, nullptr);
  }
}

void CheckTreeArgs(const lbk_build_tree_args& a)
{
  LBK_EXPECT(a.x_dtype == LBK_F32 || a.x_dtype == LBK_F64, "X must be float32 or float64");
  LBK_EXPECT(a.n_features >= 1 && a.n_outputs >= 1, "need at least one feature and one output");
  LBK_EXPECT(a.n_local_rows >= 0 && a.n_local_rows < (int64_t{1} << 31), "rows per rank must fit 31 bits");
  LBK_EXPECT(a.dataset_rows >= 1, "dataset_rows must be positive");
  LBK_EXPECT(a.max_depth >= 0 && a.max_depth <= 29, "max_depth out of range");
  LBK_EXPECT(a.max_nodes == (1 << (a.max_depth + 1)) - 1, "max_nodes must be 2^(max_depth+1)-1");
  LBK_EXPECT(a.split_samples >= 1 && a.split_samples <= 2048, "split_samples must be in [1, 2048]");
  LBK_EXPECT(a.sketch_mode == LBK_SKETCH_OFF || a.sketch_mode == LBK_SKETCH_SAVE || a.sketch_mode == LBK_SKETCH_REUSE,
             "unknown sketch mode");
  LBK_EXPECT(a.sketch_mode == LBK_SKETCH_OFF || a.sketch != nullptr, "sketch mode without a sketch buffer");
  LBK_EXPECT(a.n_local_rows == 0 || (a.X || a.sketch_mode == LBK_SKETCH_REUSE), "null input");
  LBK_EXPECT(a.n_local_rows == 0 || a.ldx >= a.n_features, "Expected a dense row major store");
  LBK_EXPECT(a.leaf_value && a.feature && a.split_value && a.gain && a.hessian, "null output");
  LBK_EXPECT(a.row_offset >= 0 && a.row_offset + a.n_local_rows <= a.dataset_rows, "row range outside the data set");
}

}  // namespace
}  // namespace lbk

extern "C" {

size_t lbk_sketch_bytes(int64_t n_local_rows, int n_features, int split_samples, int x_dtype)
{
  if (n_local_rows < 0 || n_features < 1 || split_samples < 1) return 0;
  return lbk::SketchLayoutOf(n_local_rows, n_features, split_samples, x_dtype == LBK_F64 ? 8 : 4).bytes;
}

size_t lbk_bin_matrix_bytes(int64_t n_rows, int n_features, int bin_bytes)
{
  const int64_t G = (n_features + lbk::kGroup - 1) / lbk::kGroup;
  return static_cast<size_t>(G) * static_cast<size_t>(n_rows > 0 ? n_rows : 0) * lbk::kGroup * bin_bytes + 16;
}

int lbk_build_tree(lbk_context* ctx, const lbk_build_tree_args* a)
{
  return lbk::Guard(ctx, [&] {
    LBK_EXPECT(ctx && a, "null argument");
    LBK_CUDA(cudaSetDevice(ctx->device));
    lbk::CheckTreeArgs(*a);
    LBK_EXPECT(a->n_local_rows == 0 || (a->g && a->h), "null input");
    LBK_EXPECT(a->n_local_rows == 0 || a->ldg >= a->n_outputs, "Expected a dense row major store");
    cudaStream_t stream = static_cast<cudaStream_t>(a->stream);
    if (a->x_dtype == LBK_F32)
      lbk::BuildTree<float>(ctx, *a, stream, nullptr);
    else
      lbk::BuildTree<double>(ctx, *a, stream, nullptr);
  });
}

int lbk_boost_round(lbk_context* ctx, const lbk_boost_round_args* r)
{
  return lbk::Guard(ctx, [&] {
    LBK_EXPECT(ctx && r, "null argument");
    LBK_CUDA(cudaSetDevice(ctx->device));
    const lbk_build_tree_args& a = r->tree;
    lbk::CheckTreeArgs(a);
    LBK_EXPECT(r->objective == LBK_SQUARED_ERROR || r->objective == LBK_LOG_LOSS, "unknown objective");
    LBK_EXPECT(!a.host_buffers && a.trace_hist == nullptr && a.out_total_bins == nullptr, "a round takes device buffers and no trace");
    LBK_EXPECT(a.n_local_rows == 0 || (r->y && r->pred), "null input");
    lbk::ThrowReportedFault(ctx);
    cudaStream_t stream = static_cast<cudaStream_t>(a.stream);
    if (a.x_dtype == LBK_F32)
      lbk::BuildTree<float>(ctx, a, stream, r);
    else
      lbk::BuildTree<double>(ctx, a, stream, r);
  });
}

int lbk_synchronize(lbk_context* ctx, void* stream)
{
  return lbk::Guard(ctx, [&] {
    LBK_EXPECT(ctx != nullptr, "context is null");
    LBK_CUDA(cudaSetDevice(ctx->device));
    lbk::CheckDeviceStatus(ctx, static_cast<cudaStream_t>(stream));
  });
}

int lbk_predict(lbk_context* ctx, const lbk_predict_args* a)
{
  return lbk::Guard(ctx, [&] {
    LBK_EXPECT(ctx && a, "null argument");
    LBK_CUDA(cudaSetDevice(ctx->device));
    LBK_EXPECT(a->x_dtype == LBK_F32 || a->x_dtype == LBK_F64, "X must be float32 or float64");
    if (a->n_rows < 1) return;
    LBK_EXPECT(a->X && a->pred, "null argument");
    LBK_EXPECT(a->n_features >= 1 && a->n_outputs >= 1 && a->n_trees >= 0, "bad shape");
    LBK_EXPECT(a->n_trees == 0 || a->table || (a->leaf_value && a->feature && a->split_value && a->max_nodes), "null tree arrays");
    LBK_EXPECT(!a->table || (!a->host_buffers && a->table_max_nodes >= 1), "a table of trees is for device buffers");
    LBK_EXPECT(a->transform == LBK_RAW || a->transform == LBK_SOFTMAX || (a->transform == LBK_LOGISTIC && a->n_outputs == 1),
               "unknown transform");
    const int columns = a->transform == LBK_LOGISTIC ? 2 : a->n_outputs;
    LBK_EXPECT(a->ldx >= a->n_features && a->ldp >= columns, "Expected a dense row major store");
    cudaStream_t stream = static_cast<cudaStream_t>(a->stream);
    lbk::Scratch s(ctx, stream);
    const int F = a->n_features, K = a->n_outputs, T = a->n_trees;
    const int64_t N = a->n_rows;
    const void* X   = a->X;
    double* pred    = a->pred;
    int64_t ldx = a->ldx, ldp = a->ldp;
    const lbk_tree_ref* table = a->table;
    int m_max                 = a->table_max_nodes;
    int64_t total             = a->table_total_nodes;
    std::vector<lbk_tree_ref> h;
    if (table) {
      lbk::ThrowReportedFault(ctx);
    } else {
      h.resize(T > 0 ? T : 1);
      m_max = 1;
      total = 0;
      for (int t = 0; t < T; ++t) {
        LBK_EXPECT(a->leaf_value[t] && a->feature[t] && a->split_value[t] && a->max_nodes[t] >= 1, "bad tree arrays");
        LBK_EXPECT(total + a->max_nodes[t] < (int64_t{1} << 31), "ensemble too large");
        h[t] = lbk_tree_ref{a->leaf_value[t], a->feature[t], a->split_value[t], a->max_nodes[t], static_cast<int32_t>(total)};
        total += a->max_nodes[t];
        m_max = std::max(m_max, a->max_nodes[t]);
      }
    }
    const size_t esz = a->x_dtype == LBK_F32 ? 4 : 8;
    if (a->host_buffers) {
      void* dX = s.alloc_bytes(esz * N * F);
      LBK_CUDA(cudaMemcpy2DAsync(dX, esz * F, X, esz * ldx, esz * F, N, cudaMemcpyHostToDevice, stream));
      X   = dX;
      ldx = F;
      pred = s.alloc<double>(static_cast<size_t>(N) * columns);
      ldp  = columns;
      for (int t = 0; t < T; ++t) {
        const int m = h[t].max_nodes;
        double* dl  = s.alloc<double>(static_cast<size_t>(m) * K);
        double* ds  = s.alloc<double>(m);
        int32_t* df = s.alloc<int32_t>(m);
        LBK_CUDA(cudaMemcpyAsync(dl, h[t].leaf, sizeof(double) * m * K, cudaMemcpyHostToDevice, stream));
        LBK_CUDA(cudaMemcpyAsync(ds, h[t].split, sizeof(double) * m, cudaMemcpyHostToDevice, stream));
        LBK_CUDA(cudaMemcpyAsync(df, h[t].feature, sizeof(int32_t) * m, cudaMemcpyHostToDevice, stream));
        h[t].leaf    = dl;
        h[t].split   = ds;
        h[t].feature = df;
      }
    }
    if (!table) {
      lbk_tree_ref* d = s.alloc<lbk_tree_ref>(h.size());
      if (T > 0) LBK_CUDA(cudaMemcpyAsync(d, h.data(), sizeof(lbk_tree_ref) * T, cudaMemcpyHostToDevice, stream));
      table = d;  // (h is read before the call returns: it synchronises below)
    }
    if (a->x_dtype == LBK_F32)
      lbk::PredictLaunch<float>(ctx, s, static_cast<const float*>(X), ldx, N, F, K, T, table, m_max, total, a->init,
                                a->transform, pred, ldp, stream);
    else
      lbk::PredictLaunch<double>(ctx, s, static_cast<const double*>(X), ldx, N, F, K, T, table, m_max, total, a->init,
                                 a->transform, pred, ldp, stream);
    if (a->host_buffers)
      LBK_CUDA(cudaMemcpy2DAsync(a->pred, sizeof(double) * a->ldp, pred, sizeof(double) * columns, sizeof(double) * columns, N,
                                 cudaMemcpyDeviceToHost, stream));
    if (!a->table) lbk::CheckDeviceStatus(ctx, stream);
  });
}

int lbk_split_proposals(lbk_context* ctx, const void* X, int x_dtype, int64_t ldx, int64_t row_offset,
                        int64_t n_local_rows, int n_features, int split_samples, int seed, int64_t dataset_rows,
                        void* proposals, int32_t* row_ptr, int32_t* total_bins, void* stream_)
{
  return lbk::Guard(ctx, [&] {
    LBK_EXPECT(ctx && proposals && row_ptr, "null argument");
    LBK_CUDA(cudaSetDevice(ctx->device));
    LBK_EXPECT(x_dtype == LBK_F32 || x_dtype == LBK_F64, "X must be float32 or float64");
    LBK_EXPECT(split_samples >= 1 && split_samples <= 2048, "split_samples must be in [1, 2048]");
    cudaStream_t stream = static_cast<cudaStream_t>(stream_);
    lbk::Scratch s(ctx, stream);
    lbk::ProposalInfo pi;
    if (x_dtype == LBK_F32)
      pi = lbk::SplitProposals<float>(ctx, s, static_cast<const float*>(X), ldx, row_offset, n_local_rows, n_features,
                                      split_samples, seed, dataset_rows, static_cast<float*>(proposals), row_ptr, stream);
    else
      pi = lbk::SplitProposals<double>(ctx, s, static_cast<const double*>(X), ldx, row_offset, n_local_rows, n_features,
                                       split_samples, seed, dataset_rows, static_cast<double*>(proposals), row_ptr, stream);
    if (total_bins) *total_bins = pi.total_bins;
  });
}

int lbk_bin_matrix(lbk_context* ctx, const void* X, int x_dtype, int64_t ldx, int64_t n_rows, int n_features,
                   const void* proposals, const int32_t* row_ptr, void* bins, int bin_bytes, void* stream_)
{
  return lbk::Guard(ctx, [&] {
    LBK_EXPECT(ctx && X && proposals && row_ptr && bins, "null argument");
    LBK_CUDA(cudaSetDevice(ctx->device));
    LBK_EXPECT(bin_bytes == 1 || bin_bytes == 2, "bin_bytes must be 1 or 2");
    cudaStream_t stream = static_cast<cudaStream_t>(stream_);
    // the largest feature decides whether the proposals of a feature group fit shared memory
    std::vector<int32_t> rp(n_features + 1);
    LBK_CUDA(cudaMemcpyAsync(rp.data(), row_ptr, sizeof(int32_t) * (n_features + 1), cudaMemcpyDeviceToHost, stream));
    LBK_CUDA(cudaStreamSynchronize(stream));
    int mb = 1;
    for (int f = 0; f < n_features; ++f) mb = std::max(mb, rp[f + 1] - rp[f]);
    LBK_EXPECT(bin_bytes == 2 || mb <= 256, "one-byte bins need <= 256 proposals per feature");
    if (x_dtype == LBK_F32)
      lbk::BinMatrix<float>(static_cast<const float*>(X), ldx, n_rows, n_features, static_cast<const float*>(proposals), 0,
                            row_ptr, bins, nullptr, 0, bin_bytes, mb, ctx->d_status, stream);
    else
      lbk::BinMatrix<double>(static_cast<const double*>(X), ldx, n_rows, n_features,
                             static_cast<const double*>(proposals), 0, row_ptr, bins, nullptr, 0, bin_bytes, mb,
                             ctx->d_status, stream);
  });
}

int lbk_quantise(lbk_context* ctx, const double* g, const double* h, int64_t ldg, int64_t row_offset,
                 int64_t n_local_rows, int n_outputs, int seed, int32_t* gpair, int64_t* root_sums, double* scale,
                 int32_t* max_abs, void* stream_)
{
  return lbk::Guard(ctx, [&] {
    LBK_EXPECT(ctx && gpair && root_sums && scale, "null argument");
    LBK_CUDA(cudaSetDevice(ctx->device));
    cudaStream_t stream = static_cast<cudaStream_t>(stream_);
    lbk::Scratch s(ctx, stream);
    int* abs = max_abs ? max_abs : s.alloc<int>(2);
    LBK_CUDA(cudaMemsetAsync(root_sums, 0, sizeof(lbk::GPairI64) * n_outputs, stream));
    LBK_CUDA(cudaMemsetAsync(abs, 0, 2 * sizeof(int), stream));
    lbk::PrologueArgs<float> pa{};
    pa.g          = g;
    pa.h          = h;
    pa.ldg        = ldg;
    pa.K          = n_outputs;
    pa.n_elements = n_local_rows * n_outputs;
    pa.S          = 1;
    lbk::QuantParams* qp = reinterpret_cast<lbk::QuantParams*>(scale);
    lbk::Prologue<float>(ctx, s, pa, nullptr, nullptr, nullptr, s.alloc<double>(2), qp, stream);
    lbk::Quantise(ctx, g, h, ldg, lbk::GradientForm{}, row_offset, n_local_rows, n_outputs, seed, reinterpret_cast<int2*>(gpair),
                  reinterpret_cast<lbk::GPairI64*>(root_sums), qp, abs, nullptr, stream);
  });
}

static int StageHistogram(lbk_context* ctx, const lbk_histogram_args* a, bool merge_tree)
{
  return lbk::Guard(ctx, [&] {
    LBK_EXPECT(ctx && a, "null argument");
    LBK_CUDA(cudaSetDevice(ctx->device));
    LBK_EXPECT(a->bins && a->row_ptr && a->row_index && a->seg && a->hist, "null argument");
    LBK_EXPECT(a->mode == 0 || a->mode == 1, "mode must be 0 or 1");
    LBK_EXPECT(a->mode == 0 ? a->gpair != nullptr : a->gpair_f32 != nullptr, "missing gradient pairs");
    LBK_EXPECT(a->bin_bytes == 1 || a->bin_bytes == 2, "bin_bytes must be 1 or 2");
    LBK_EXPECT(a->n_nodes >= 1 && a->n_features >= 1 && a->n_outputs >= 1 && a->total_bins >= a->n_features, "bad shape");
    LBK_EXPECT(a->all_reduce >= 0 && a->all_reduce <= 2, "all_reduce must be 0, 1 or 2");
    LBK_EXPECT(!a->pairs_by_position || !a->host_buffers, "pairs stored by position are for device buffers");
    LBK_EXPECT(!a->pairs_by_position || a->mode == 1 || a->max_abs != nullptr,
               "pairs stored by position need max_abs (the library cannot know how many entries the array has)");
    cudaStream_t stream = static_cast<cudaStream_t>(a->stream);
    lbk::Scratch s(ctx, stream);
    const int F = a->n_features, K = a->n_outputs, B = a->total_bins;
    const int64_t N = a->n_rows;
    const void* bins         = a->bins;
    const int32_t* row_ptr   = a->row_ptr;
    const void* gp           = a->mode == 0 ? static_cast<const void*>(a->gpair) : static_cast<const void*>(a->gpair_f32);
    const int32_t* row_index = a->row_index;
    const int32_t* seg       = a->seg;
    void* hist               = a->hist;
    const size_t hist_bytes  = sizeof(lbk::GPairI64) * a->n_nodes * K * B;
    std::vector<int32_t> rp(F + 1);
    if (a->host_buffers) {
      std::memcpy(rp.data(), a->row_ptr, sizeof(int32_t) * (F + 1));
      const int32_t n_idx = a->seg[a->n_nodes];
      const size_t bb     = lbk_bin_matrix_bytes(N, F, a->bin_bytes) - 16;
      void* d_bins        = s.alloc_bytes(bb + 16);
      int32_t* d_rp       = s.alloc<int32_t>(F + 1);
      void* d_gp          = s.alloc_bytes(sizeof(int2) * N * K);
      int32_t* d_idx      = s.alloc<int32_t>(n_idx);
      int32_t* d_seg      = s.alloc<int32_t>(a->n_nodes + 1);
      void* d_hist        = s.alloc_bytes(hist_bytes);
      LBK_CUDA(cudaMemcpyAsync(d_bins, bins, bb, cudaMemcpyHostToDevice, stream));
      LBK_CUDA(cudaMemcpyAsync(d_rp, row_ptr, sizeof(int32_t) * (F + 1), cudaMemcpyHostToDevice, stream));
      LBK_CUDA(cudaMemcpyAsync(d_gp, gp, sizeof(int2) * N * K, cudaMemcpyHostToDevice, stream));
      LBK_CUDA(cudaMemcpyAsync(d_idx, row_index, sizeof(int32_t) * n_idx, cudaMemcpyHostToDevice, stream));
      LBK_CUDA(cudaMemcpyAsync(d_seg, seg, sizeof(int32_t) * (a->n_nodes + 1), cudaMemcpyHostToDevice, stream));
      bins = d_bins; row_ptr = d_rp; gp = d_gp; row_index = d_idx; seg = d_seg; hist = d_hist;
    } else if (a->max_bins <= 0) {
      LBK_CUDA(cudaMemcpyAsync(rp.data(), row_ptr, sizeof(int32_t) * (F + 1), cudaMemcpyDeviceToHost, stream));
      LBK_CUDA(cudaStreamSynchronize(stream));
    }
    int mb = 1;
    if (!a->host_buffers && a->max_bins > 0) {
      mb = a->max_bins;  // the caller vouches for it: row_ptr stays on the device, no wait before the launch
    } else {
      LBK_EXPECT(rp[F] == B, "total_bins does not match row_ptr");
      for (int f = 0; f < F; ++f) mb = std::max(mb, rp[f + 1] - rp[f]);
    }
    LBK_EXPECT(a->bin_bytes == 2 || mb <= 256, "one-byte bins need <= 256 proposals per feature");
    // (the summed forms zero what they need themselves; the staging copy of a host buffer is fresh
    // scratch and must not return what it held before)
    if (a->all_reduce == 0 || a->host_buffers) LBK_CUDA(cudaMemsetAsync(hist, 0, hist_bytes, stream));
    lbk::HistLevel lv;
    lv.bins                 = bins;
    lv.bin_bytes            = a->bin_bytes;
    lv.n_rows               = N;
    lv.F                    = F;
    lv.K                    = K;
    lv.B                    = B;
    lv.max_bins_per_feature = mb;
    lv.row_ptr              = row_ptr;
    lv.gpair                = a->mode == 0 ? static_cast<const int2*>(gp) : nullptr;
    lv.gpair_f              = a->mode == 1 ? static_cast<const float2*>(gp) : nullptr;
    lv.max_abs              = a->host_buffers ? nullptr : reinterpret_cast<const int*>(a->max_abs);
    lv.pairs_by_position    = a->pairs_by_position != 0;
    lv.row_index            = row_index;
    lv.seg_begin            = seg;
    lv.seg_end              = seg + 1;
    lv.n_nodes              = a->n_nodes;
    lv.out                  = hist;
    lv.float_mode           = a->mode == 1;
    lv.merge_tree           = merge_tree;
    if (a->all_reduce == 1) lbk::BuildHistogramSummed(ctx, s, lv, a->n_nodes, lbk::HistSum::kSumEverywhere, true, true, stream);
    else if (a->all_reduce == 2) lbk::BuildHistogramSummed(ctx, s, lv, a->n_nodes, lbk::HistSum::kSumOwned, true, true, stream);
    else lbk::BuildHistogram(ctx, s, lv, stream);
    // host buffers: the histogram has to be back before the call returns; device buffers: the call
    // is one more piece of work on the caller's stream
    if (a->host_buffers) {
      LBK_CUDA(cudaMemcpyAsync(a->hist, hist, hist_bytes, cudaMemcpyDeviceToHost, stream));
      lbk::CheckDeviceStatus(ctx, stream);
    }
  });
}

int lbk_histogram(lbk_context* ctx, const lbk_histogram_args* a) { return StageHistogram(ctx, a, false); }
int lbk_selftest_histogram(lbk_context* ctx, const lbk_histogram_args* a) { return StageHistogram(ctx, a, true); }

int lbk_group_rows(lbk_context* ctx, const int32_t* node_of_row, int64_t n_rows, int node_begin, int n_nodes,
                   int32_t* row_index, int32_t* seg, void* stream_)
{
  return lbk::Guard(ctx, [&] {
    LBK_EXPECT(ctx && node_of_row && row_index && seg, "null argument");
    LBK_CUDA(cudaSetDevice(ctx->device));
    cudaStream_t stream = static_cast<cudaStream_t>(stream_);
    lbk::Scratch s(ctx, stream);
    lbk::GroupRows(ctx, s, node_of_row, n_rows, node_begin, n_nodes, row_index, seg, stream);
    LBK_CUDA(cudaStreamSynchronize(stream));
  });
}

int lbk_leaf_values(lbk_context* ctx, const double* leaf_value, const int32_t* leaf, int64_t n_rows, int n_outputs,
                    double* out, void* stream_)
{
  return lbk::Guard(ctx, [&] {
    LBK_EXPECT(ctx != nullptr, "context is null");
    LBK_EXPECT(n_rows >= 0 && n_outputs >= 1, "bad shape");
    if (n_rows == 0) return;
    LBK_EXPECT(leaf_value && leaf && out, "null argument");
    LBK_CUDA(cudaSetDevice(ctx->device));
    cudaStream_t stream  = static_cast<cudaStream_t>(stream_);
    const int64_t total  = n_rows * n_outputs;
    const int64_t blocks = (total + 255) / 256;
    LBK_EXPECT(blocks <= 2147483647ll, "too many elements for one launch");
    lbk::LaunchChained(lbk::k_gather_rows, static_cast<unsigned>(blocks), 256, 0, stream, leaf_value, leaf, n_rows, n_outputs, out);
    LBK_LAUNCH_CHECK();
  });
}

}  // extern "C"
