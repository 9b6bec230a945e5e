// Internal declarations shared by the translation units of liblbk.so.
#pragma once
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <functional>
#include <mutex>
#include <stdexcept>
#include <string>
#include <utility>
#include <vector>

#include "lbk.h"

namespace lbk {

struct Error : public std::runtime_error {
  int code;
  Error(int c, const std::string& m) : std::runtime_error(m), code(c) {}
};

#define LBK_CUDA(call)                                                                        \
  do {                                                                                        \
    cudaError_t e_ = (call);                                                                  \
    if (e_ != cudaSuccess) {                                                                  \
      throw ::lbk::Error(LBK_ERR_CUDA, std::string(__FILE__) + ":" + std::to_string(__LINE__) + \
                                         ": " #call ": " + cudaGetErrorString(e_));           \
    }                                                                                         \
  } while (0)

#define LBK_EXPECT(cond, msg)                                                                 \
  do {                                                                                        \
    if (!(cond)) {                                                                            \
      throw ::lbk::Error(LBK_ERR_ARGUMENT, std::string(__FILE__) + ":" + std::to_string(__LINE__) + \
                                             ": " + (msg));                                   \
    }                                                                                         \
  } while (0)

#define LBK_LAUNCH_CHECK() LBK_CUDA(cudaGetLastError())

// A launch that the GPU prepares while the kernel before it on the stream still runs: its blocks may begin as soon as those of
// the other are all done, before its end has been made known to the host and to other streams.  Such a kernel begins, in
// every block and before any return, with AfterTheKernelBefore() (device_utils.cuh), which waits for the end of that kernel and for
// what it has written.  No kernel says earlier than with its end that the next one may begin: blocks that come while others
// work take room from these (200k x 50, ten rounds 2.25 -> 2.39 ms with that behind every wait; what was computed stayed the same, though
// kernels then began long before the ones they wait for had ended).  The gap between two kernels of a chain was 2 us, of which
// some 0.5 are left: 200k x 50, depth 6, ten rounds 2.70 -> 2.25 ms, 60k x 100, depth 8, five rounds 2.06 -> 1.74, 300003 x 37 float64 1.68 -> 1.50,
// 10M x 64, depth 8, three rounds 7.92 -> 7.73; predictions of 100003 x 100, ten outputs 92 -> 86 us, 1M x 64 float64 513 -> 495.
template <typename... P, typename... A>
void LaunchChained(void (*fn)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, A&&... args)
{
  cudaLaunchAttribute attr[1];
  attr[0].id                                         = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim          = grid;
  cfg.blockDim         = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream           = stream;
  cfg.attrs            = attr;
  cfg.numAttrs         = 1;
  const cudaError_t launched = cudaLaunchKernelEx(&cfg, fn, static_cast<P>(args)...);
  if (launched != cudaSuccess) cudaGetLastError();  // (left with the runtime, it would be the answer to the next launch, whoever's)
  LBK_CUDA(launched);
}

// 16-byte (grad, hess) pairs
struct GPairI64 {
  long long grad, hess;
};
struct GPairF64 {
  double grad, hess;
};

// Quantiser parameters, device resident (reference: GradientQuantiser, build_tree.cu:51-104)
struct QuantParams {
  double scale_g, scale_h, inv_g, inv_h;
};

inline int LevelBegin(int level) { return (1 << level) - 1; }
inline int LevelEnd(int level) { return (1 << (level + 1)) - 1; }

constexpr int kGroup = 32;  // features per feature group (one lane per feature)

inline bool Aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

}  // namespace lbk

namespace lbk {
struct PeerExchange;
}

// The context is an opaque C struct for callers.
struct lbk_context {
  int device        = 0;
  int sm_count      = 0;
  int max_smem_optin = 0;
  cudaMemPool_t pool = nullptr;
  // the caller's allocator for scratch (both set or both null)
  lbk_alloc_fn alloc_cb     = nullptr;
  lbk_release_fn release_cb = nullptr;
  void* alloc_user          = nullptr;
  mutable std::mutex err_mutex;
  std::string err;  // of the last call that failed, whatever its thread
  // status word in mapped host memory: 0 = ok, otherwise a kernel stored a fault code
  int* d_status = nullptr;
  // pairs of words in mapped host memory that a call borrows for what its kernels tell the host (HostWords)
  std::mutex words_mutex;
  std::vector<void*> words_pages;
  std::vector<int32_t*> words_free;
  int words_lent = 0;
  // communicator
  int rank = 0, n_ranks = 1;
  void* nccl_comm     = nullptr;
  bool owns_nccl      = false;
  lbk_allreduce_fn cb = nullptr;
  void* cb_user       = nullptr;
  // buffers that the other ranks' GPUs can read (see exchange.cu); made on first use
  lbk::PeerExchange* xchg = nullptr;
  // optional timing of the histogram kernel alone (events on the caller's stream)
  bool profile            = false;
  std::vector<std::pair<cudaEvent_t, cudaEvent_t>> prof_events;  // one pair per timed launch since the last total
  size_t prof_used        = 0;
};

namespace lbk {

// Stream-ordered scratch allocation from the context's pool (replaces legate::create_buffer).
class Scratch {
 public:
  Scratch(lbk_context* ctx, cudaStream_t stream) : ctx_(ctx), stream_(stream) {}
  ~Scratch();
  Scratch(const Scratch&)            = delete;
  Scratch& operator=(const Scratch&) = delete;
  void* alloc_bytes(size_t bytes);
  template <typename T>
  T* alloc(size_t n)
  {
    return static_cast<T*>(alloc_bytes(sizeof(T) * (n > 0 ? n : 1)));
  }
  void free_one(void* p);  // (a small buffer stays until the end)

 private:
  void* AllocBlock(size_t bytes);
  lbk_context* ctx_;
  cudaStream_t stream_;
  std::vector<void*> ptrs_;
  char* slab_       = nullptr;
  size_t slab_used_ = 0;
};

// Two words of mapped host memory for one call: number of bins, bins of the largest feature.  Calls in progress
// on several streams or threads must not see each other's; a pair goes back only once the call has waited for its
// kernels (`settled`) - after an error a kernel may still write it, and it stays out of use.
class HostWords {
 public:
  explicit HostWords(lbk_context* ctx) : ctx_(ctx) {}
  ~HostWords();
  HostWords(const HostWords&)            = delete;
  HostWords& operator=(const HostWords&) = delete;
  int32_t* get();  // borrowed on first use
  void settled() { settled_ = true; }
  // Before the kernel that writes the words (both with one store) is queued; and, afterwards, the wait for that store,
  // which does not wait for what the kernel does besides.
  void expect();
  void await(cudaStream_t stream);

 private:
  lbk_context* ctx_;
  int32_t* words_ = nullptr;
  bool settled_   = false;
};

// In-place all-reduce over the context's communicator; no-op for a single rank.
void AllReduce(lbk_context* ctx, void* buf, size_t count, lbk_dtype dtype, lbk_redop op, cudaStream_t stream);
// Every rank contributes `bytes` bytes at `send` and receives all contributions, in rank order, at
// `recv` (device pointers; NCCL communicators only: returns false where the communicator is a
// callback or missing).
bool AllGatherBytes(lbk_context* ctx, const void* send, void* recv, size_t bytes, cudaStream_t stream);

// ---- peer exchange (exchange.cu) ------------------------------------------------------------
// Two buffers per rank that every other rank's GPU can read directly over NVLink (CUDA IPC between
// processes, plain peer access inside one process), used to sum the histograms of a level: every
// rank builds into its own buffer, a barrier, then rank r reads the bins of the features it owns
// from all ranks and adds them up (a reduce-scatter made of peer loads).  The two buffers
// alternate so that one barrier per level is enough.
//
// Collective: every rank calls with the same `bytes`.  Returns false (on every rank alike) where the
// peers cannot be mapped or the communicator is not NCCL; callers then fall back to AllReduce.
bool EnsureExchange(lbk_context* ctx, size_t bytes, cudaStream_t stream);
void DestroyExchange(lbk_context* ctx);
// The buffer the next build goes into (alternates on every call), its first `bytes` bytes zeroed.
void* NextExchangeBuffer(lbk_context* ctx, size_t bytes, cudaStream_t stream);
// Features [OwnedBegin(r), OwnedBegin(r + 1)) belong to rank r.
__host__ __device__ inline int OwnedBegin(int rank, int n_ranks, int F) { return static_cast<int>(static_cast<long long>(rank) * F / n_ranks); }
// After every rank has built [n_seg][B] pairs into `buf` (the buffer NextExchangeBuffer returned):
// dst[seg][b] = sum over ranks of their buf[seg][b] for the bins b of this rank's features; dst may
// be `buf` itself (in place).  Includes the barrier.
void ExchangeReduceOwned(lbk_context* ctx, void* buf, void* dst, int n_seg, int B, int F, const int32_t* row_ptr,
                         bool float_mode, cudaStream_t stream);
// The push form.  NextPushBuffers: the device array of every rank's receive buffer for the next
// build (alternating, all zero when handed out).  ExchangeReducePushed, after every rank has built
// with them: a barrier, then dst[seg][b] = sum over source ranks of this rank's receive slots, for the
// bins b of its features (dst is local memory, [n_seg][B] pairs); the slots are zeroed as they are
// read, so the buffer is clean when its turn comes again.
void* const* NextPushBuffers(lbk_context* ctx, cudaStream_t stream);
void ExchangeReducePushed(lbk_context* ctx, void* dst, int n_seg, int push_len, int B, int F, const int32_t* row_ptr,
                          bool float_mode, cudaStream_t stream);
// After ExchangeReduceOwned in place on every rank: dst[seg][b] = the owner's sum, for all bins.
// Includes a barrier.
void ExchangeGatherAll(lbk_context* ctx, void* buf, void* dst, int n_seg, int B, int F, const int32_t* row_ptr,
                       cudaStream_t stream);
// The event pair that brackets the next timed histogram launch (profile mode): the first that is
// free, made on demand; when kMaxProfiledLaunches are in use the last one is used again.
std::pair<cudaEvent_t, cudaEvent_t> NextProfileEvents(lbk_context* ctx);
// Synchronises the stream, then throws LBK_ERR_DEVICE if a kernel stored a fault code.
void CheckDeviceStatus(lbk_context* ctx, cudaStream_t stream);
// The same without the synchronisation: what earlier, asynchronous calls have reported so far.
void ThrowReportedFault(lbk_context* ctx);

// Runs f, turning exceptions into a status code and an error text (the ABI boundary).
int Guard(lbk_context* ctx, const std::function<void()>& f);

// Lets launches of `fn` ask for up to the device's limit of dynamic shared memory, less `static_bytes`, a bound of what the
// kernel declares itself.  The limit belongs to the function and not to a launch: one constant per function,
// or a call on another thread could lower it between this call's setting and its launch.
template <typename Fn>
inline void AllowSharedMemory(const lbk_context* ctx, Fn fn, int static_bytes)
{
  LBK_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, ctx->max_smem_optin - static_bytes));
}

// ---- stage launchers (defined in the .cu files named in the comments) ------------------------
struct TreeArrays {
  double* leaf_value;
  int32_t* feature;
  double* split_value;
  double* gain;
  GPairI64* node_sums;
  int32_t* split_bin;  // feature-relative bin of the chosen split, per node
  int max_nodes;
};
// proposals.cu
struct ProposalInfo {
  int total_bins;            // B
  int max_bins_per_feature;  // largest feature
};
// The first two launches of a tree: split proposals, |g| and |h| sums, cleared arrays (k_prologue), then
// what follows from all features or all sums (k_prologue_finish).
constexpr int kZeroRanges = 3;
// What a tree's (g, h) arrays hold: gradients, or (squared_error) raw predictions and labels, of which a round makes the
// gradients as it reads them: for 10M rows the kernel that writes them took 52 us and the reads are the same.
struct GradientForm {
  bool squared_error   = false;
  double learning_rate = 0.0;
};
template <typename T>
struct PrologueArgs {
  const T* X;
  int64_t ldx, row_offset, n_local;
  int F, S, S_pad, seed;
  int64_t dataset_rows;
  const T* draft;    // set by Prologue: the sampled values where they were summed over ranks first
  T* cuts;           // out [F][S]: sorted distinct samples, the last one +inf
  int32_t* counts;   // out [F]; null: no proposals are drawn
  const double* g;
  const double* h;
  int64_t ldg;
  GradientForm form;
  int K;
  int64_t n_elements;      // rows x K
  double *part_g, *part_h; // set by Prologue
  TreeArrays tree;         // feature, split_value and gain are cleared (max_nodes may be 0)
  int32_t *root_begin, *root_end;  // the root's segment: all local rows (may be null)
  void* zero[kZeroRanges];        // 16-byte aligned ranges to zero ...
  int64_t zero_n16[kZeroRanges];  // ... in units of 16 bytes
  int64_t sort_blocks, sum_blocks;
  int fill_blocks;
};
// info: device [2] = bins, bins of the largest feature; info_host: the same in mapped host memory (may be
// null).  sums (may be null: none are made): device [2]; params: the scale from the sums, maximum over ranks.
template <typename T>
void Prologue(lbk_context* ctx, Scratch& s, PrologueArgs<T> p, int32_t* row_ptr, int32_t* info, int32_t* info_host,
              double* sums, QuantParams* params, cudaStream_t stream);
template <typename T>
ProposalInfo SplitProposals(lbk_context* ctx, Scratch& s, const T* X, int64_t ldx, int64_t row_offset,
                            int64_t n_local, int F, int S, int seed, int64_t dataset_rows, T* proposals,
                            int32_t* row_ptr, cudaStream_t stream);  // synchronises the stream
template <typename T>
// bins_t (optional): feature-major copy, bins_t[f * pitch_t + row], pitch_t a multiple of 32 >= n_rows
// cut_stride > 0: the proposals of feature f begin at f * cut_stride (0: at row_ptr[f])
void BinMatrix(const T* X, int64_t ldx, int64_t n_rows, int F, const T* proposals, int64_t cut_stride, const int32_t* row_ptr,
               void* bins, void* bins_t, int64_t pitch_t, int bin_bytes, int max_bins_per_feature, int* status,
               cudaStream_t stream);
// quantise.cu.  root_sums, max_abs and hess_below_one (may be null; 1 if some quantised hessian is below one) are zero before
// the call.
void Quantise(lbk_context* ctx, const double* g, const double* h, int64_t ldg, const GradientForm& form, int64_t row_offset,
              int64_t n_local, int K, int seed, int2* gpair, GPairI64* root_sums, const QuantParams* params, int* max_abs /* device [2] */,
              int* hess_below_one, cudaStream_t stream);
// histogram.cu
struct HistScratch {
  unsigned int* arrive   = nullptr;  // [n_arrive], zero
  int n_arrive           = 0;
  unsigned int* tickets  = nullptr;  // one per launch, zero
  int next_ticket        = 0;
  int n_tickets          = 0;
  void* partial          = nullptr;
  size_t partial_bytes   = 0;
};
// What a tree with these shapes needs of it (n_arrive, partial_bytes).
void HistScratchNeeds(lbk_context* ctx, int F, int K, int bin_bytes, int max_bins_per_feature, int64_t n_rows, HistScratch& need);
struct HistLevel {
  const void* bins;
  int bin_bytes;
  int64_t n_rows;      // rows of the bin matrix (local rows)
  int F, K, B;
  int max_bins_per_feature;          // an upper bound ...
  const int* max_bins_ptr = nullptr; // ... and where the device knows the number itself (may be null)
  const int32_t* row_ptr;
  const int2* gpair;       // int path
  const float2* gpair_f;   // float path
  bool pairs_by_position = false;  // gpair / gpair_f are stored in row_index order: entry i belongs to row_index[i]
  const int* max_abs;      // device [2]: largest |grad|, |hess| of gpair (null: computed by the call)
  const int32_t* row_index;  // null: row i is at position i (the root)
  const int32_t* seg_begin;  // rows of node j of the batch: row_index[seg_begin[j] .. seg_end[j])
  const int32_t* seg_end;
  int n_nodes;             // nodes in this batch
  // node_sums null: every node is built, node j into slot j of `out`.  Else the batch is made of pairs of
  // siblings and only the smaller one is built (SmallerChildIsLeft), into slot j / 2.
  const GPairI64* node_sums = nullptr;
  int node_begin            = 0;
  const int* build_all      = nullptr;  // device word: where it is not 0 every node is built although node_sums is given
  void* out;               // [n_slots, K, B] pairs (int64 or double), already zeroed
  bool float_mode;
  // scratch that a tree keeps for all its levels (null: the call makes its own): words that are zero
  // before the call and again after it, a zero ticket of this level, slots for partial sums
  HistScratch* scratch      = nullptr;
  // set by BuildHistogramSummed only: the histograms go into the owners' receive buffers (see
  // HistParams in histogram.cu)
  void* const* push_recv     = nullptr;
  long long push_slot_pairs = 0;
  int push_len              = 0;
  bool merge_tree           = false;  // pieces of a node meet in a merge tree although the histograms are local (lbk_selftest_histogram)
};
void BuildHistogram(lbk_context* ctx, Scratch& s, const HistLevel& lv, cudaStream_t stream);
// BuildHistogram followed by the sum over ranks of the n_slots histograms.
//   kSumEverywhere: lv.out holds the sums of all bins on every rank when the call returns.
//   kSumOwned:      only the bins of the features this rank owns are summed (OwnedBegin); the
//                   result is where the returned pointer says: lv.out, or the exchange buffer the
//                   level was built in (which stays valid until the build after the next).
// Through the peer exchange where it is available, else one all-reduce of the whole buffer (then
// every bin is summed on every rank, whatever the mode).  The sequence of collectives depends only
// on values that are equal on every rank; a rank without rows skips the kernel, nothing else.
// zero_out: lv.out has not been zeroed; the call zeroes it where the build goes into it (through the
// exchange it does not: what is not written there stays as it was).
enum class HistSum { kSumEverywhere, kSumOwned };
void* BuildHistogramSummed(lbk_context* ctx, Scratch& s, const HistLevel& lv, int n_slots, HistSum mode,
                           bool result_in_out, bool zero_out, cudaStream_t stream);
void GroupRows(lbk_context* ctx, Scratch& s, const int32_t* node_of_row, int64_t n_rows, int node_begin,
               int n_nodes, int32_t* row_index, int32_t* seg, cudaStream_t stream);
// split.cu
struct SplitParams {
  double l1, l2, min_split_gain;
  const uint8_t* feature_set;
};
// One level (or batch of one) after its histograms have been built.
struct ScanSplitLevel {
  const GPairI64* built;        // raw sums, [unit][K][bin_stride]; may be level_hist itself when nothing is derived
  GPairI64* level_hist;         // [n_nodes][K][bin_stride]; only touched if write_hist
  const GPairI64* parent_hist;  // histograms of the level above, its first node is parent_begin (derive only)
  int parent_begin;
  GPairI64* next_built;         // [n_nodes][K][bin_stride]: zeroed for the level below; may be null
  int64_t bin_stride;
  int node_begin, n_nodes, K;
  int f_begin, f_end;           // the features scanned and searched (the owned ones with several ranks)
  bool derive;                  // pairs of siblings, one of them built
  bool write_hist;
  int64_t cells;                // of the matrix: rows x features x outputs
  const int* build_all = nullptr;  // device word (HistLevel): the call does nothing where it says the other of `derive`
};
// cuts: the split proposals, feature f's from f * cut_stride on.  arrived: one counter per tree node, zero
// before the first call of a tree.  With exchange_records every rank's best candidate of every node
// (and the sums left of it) is gathered on all ranks and the best of them becomes the tree - the same
// total order as within a rank, so the tree is the one a single rank would grow.
template <typename T>
void ScanSplit(lbk_context* ctx, Scratch& s, const ScanSplitLevel& lv, int F, const int32_t* row_ptr, const T* cuts,
               int64_t cut_stride, const QuantParams* qp, const SplitParams& sp, const TreeArrays& tree,
               unsigned int* arrived, bool exchange_records, cudaStream_t stream);
// hessians and leaf values of all nodes from their sums
void FinishTree(const TreeArrays& tree, const QuantParams* qp, int K, double l1, double l2, double* hessian,
                cudaStream_t stream);
// partition.cu
struct PartitionLevel {
  const void* bins;   // feature-major copy of the bin ids: bins[f * bin_pitch + row]
  int bin_bytes;
  int64_t bin_pitch;  // elements per feature
  int n_features;
  int64_t n_rows;
  const int32_t* row_index_in;  // null: row i is at position i (the root)
  const int32_t* seg_begin;     // [n_nodes]
  const int32_t* seg_end;
  int32_t* row_index_out;
  int32_t* seg_begin_out;       // [2 * n_nodes], for the next level
  int32_t* seg_end_out;
  unsigned long long* cursor;   // one per tree node, zero before the first call of a tree
  int node_begin, n_nodes;
  const int32_t* feature;
  const int32_t* split_bin;
  // optional: the quantised pairs in row_index order, moved together with the row ids
  const int2* pairs_in = nullptr;  // [rows of the level][K]
  int2* pairs_out      = nullptr;
  int K                = 0;
};
void PartitionRows(lbk_context* ctx, Scratch& s, const PartitionLevel& pl, cudaStream_t stream);
// objective.cu
void Gradient(int objective, const double* raw_pred, const double* y, int64_t n_rows, int n_outputs, double learning_rate,
              double* g, double* h, cudaStream_t stream);
// small_tree.cu: a whole tree in one launch, for matrices of at most kSmallMaxRows rows
constexpr int64_t kSmallMaxRows = 32768;
template <typename T>
struct SmallTreeArgs {
  const T* X;
  int64_t ldx, N;
  int F, K, D, S, seed;
  int64_t row_offset, dataset_rows;
  const double* g;
  const double* h;
  int64_t ldg;
  // objective >= 0: the gradients are those of `pred` (squared error, or log loss with one output), and the
  // tree's leaf values are added to it; g and h are not read
  int objective;
  const double* y;
  double* pred;
  double lr;
  SplitParams sp;
  TreeArrays tree;   // node_sums [max_nodes][K]; split_bin is not used
  double* hessian;
  int32_t* leaf;     // may be null
  unsigned int* barrier;  // device word, zero; this tree's alone
  int32_t* info_host;     // mapped host word for the number of bins, or null
};
bool SmallTreeFits(lbk_context* ctx, int64_t N, int F, int K, int D, int S);
template <typename T>
void SmallTree(lbk_context* ctx, Scratch& s, const SmallTreeArgs<T>& a, cudaStream_t stream);
// predict.cu
template <typename T>
void PredictLaunch(lbk_context* ctx, Scratch& s, const T* X, int64_t ldx, int64_t n_rows, int F, int K, int n_trees,
                   const lbk_tree_ref* d_trees /* device */, int m_max /* nodes of the largest tree */, int64_t total_nodes,
                   const double* init, int transform, double* pred, int64_t ldp, cudaStream_t stream);
// predict_ranked.cu: one output, more rows and trees than k_predict_tiled is better for.
struct RankTile {  // of k_predict_tiled: rows that an SM has at a time (0: not tiled), trees that a thread walks together
  int rows = 0, trees = 0, tree_bytes = 0;
};
struct RankedPlan {  // threads == 0: the shape does not fit, or is not worth it
  int threads = 0, tg = 0, nbuf = 0;  // of the walk, and trees per group: what is in flight is threads x trees x 2 walks
  size_t smem   = 0;
  int64_t piece = 0;  // rows whose ranks are held at a time
  double budget = 0;  // microseconds that finding the ranks may take
  bool sure     = false;  // whatever the splits are, they take no more: the device does not decline
  int max_items = 0;  // pieces of the features' lists of splits
  size_t bytes = 0, o_words = 0, o_off = 0, o_items = 0, o_lists = 0, o_cuts = 0, o_lut = 0, o_tables = 0, o_records = 0, o_ranks = 0;  // scratch
};
template <typename T>
RankedPlan PlanRanked(const lbk_context* ctx, int64_t n_rows, int F, int n_trees, int S, int64_t total_nodes,
                      const RankTile& tiled);
// Null: there is no room for it, nothing was done.  Else a device word: where it is not 0 when the stream comes to it, the
// kernels queued here have done nothing, because the ensemble's splits lie so that the ranks would cost more than they give.
template <typename T>
const int* PredictRanked(lbk_context* ctx, Scratch& s, const RankedPlan& plan, const T* X, int64_t ldx, int64_t n_rows, int F, int n_trees,
                         const lbk_tree_ref* d_trees, int S, int64_t total_nodes, const double* init, int transform, double* pred, int64_t ldp,
                         cudaStream_t stream);

}  // namespace lbk
