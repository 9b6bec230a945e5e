// Histogram construction: hist[node][output][bin] += (grad, hess) for the rows of the nodes that
// have to be built on this level.
//
// Reference behaviour restated here: fill_histogram_shared / HistogramAgent,
// src/models/tree/build_tree.cu:213-577 (shared-memory int32 pairs per block flushed with 64-bit
// global atomics, impure tiles straight to global atomics).
//
// Design for B200:
//   * rows arrive grouped by node (an index array plus per-node offsets), so a thread block only
//     ever accumulates one node at a time and its private histogram lives in shared memory;
//   * bins are one byte per element, row-major with rows padded to whole 32-feature groups (see
//     proposals.cu): the pieces of a row that different tickets need share DRAM bursts and L2 lines;
//   * the kernel is bound by the load/store data pipe of the SM, not by HBM: the two shared-memory
//     reductions a warp issues per 32 updates are unavoidable (64-bit shared atomics are
//     compare-and-swap loops on this part), and a gather costs the pipe one pass per distinct
//     128-byte line.  So a ticket covers two feature groups (one pass per row for 64 bin bytes),
//     the rows of a batch go straight from global memory into registers with one 16-byte load per
//     lane, and the lanes of a row walk their bytes in an xor-skewed order that keeps the 32
//     reductions of a warp on 32 different banks whatever the bins are (k_hist_smem);
//   * every warp runs its own pipeline over batches of rows (no block barrier in the main loop, no
//     staging in shared memory): the rows of the next two batches and the row ids of the two after
//     are in flight in registers;
//   * accumulation is in int32 like the reference, but guarded: with m = the largest |q| of the
//     call, at most floor((2^31-1)/m) rows are accumulated between flushes, so no partial sum can
//     wrap whatever the bins are;
//   * the rows of the level are handed to the resident blocks in equal static ranges (a block walks
//     through the nodes its range touches) or, for small levels, as tickets drawn from a counter;
//     every block works the plan out for itself (levels of many nodes: k_hist_plan);
//   * matrices of moderate size, and bins of two bytes, are built by k_hist_tile: many small blocks with
//     the histograms of eight features each;
//   * a node built in one piece owns its output region and flushes with plain stores, turned in
//     shared memory so that four bins of a feature leave as 64 contiguous bytes; the pieces of a
//     node that reaches over a range boundary add to it with 64-bit atomics on whole sectors or, where the
//     histograms go to other ranks' memory, meet in a merge tree of arrival counters in which nobody
//     waits (k_hist_smem); chunks of <= 128 rows skip shared memory.
#include <mutex>
#include <string>
#include <type_traits>

#include "device_utils.cuh"
#include "hist_units.h"
#include "internal.h"

namespace lbk {
namespace {

constexpr int kHistThreads = 512;
constexpr int kTileRows    = 32;    // chunk sizes are multiples of this
constexpr int kDirectRows  = 128;   // chunks up to this size go straight to global atomics
constexpr int kMinChunk    = 2048;
constexpr int kSmemBins    = 256;   // bins per feature held by the private histogram
constexpr int kHistBase    = 4096;  // shared-memory address of k_hist_smem's histograms
constexpr int kFlushBins   = 4;     // bins of a tile of the flush
constexpr int kFaultHistLayout = 31;  // status word: shared memory did not start where the kernel needs it
constexpr int kTreeFanIn   = 4;     // partial sums that meet in one step of the merge tree
constexpr int kPlanNodes   = 1024;  // levels of up to this many nodes are planned inside the kernels

// Dynamic shared memory of k_hist_smem for W feature groups: (up to) kHistBase bytes before the histograms,
// the two histograms, a staging tile per warp, the plan.  The sum decides how much of the SM's 256 KB is left as
// L1, which the row gathers land in: 152 KB leave 64 KB, 193 KB 32 KB, 198 KB nothing (10M x 128, 128
// nodes: 495 / 523 / 584 us).
__host__ __device__ constexpr unsigned HistSmemBytes(int W)
{
  return kHistBase + 2u * kSmemBins * kGroup * W * 4 + (kHistThreads * W / 32) * kFlushBins * 32 * 4 + (kPlanNodes + 1 + 32) * 4;
}

struct HistParams {
  const void* bins;
  int64_t n_rows;
  int F, K, B, G, mb;
  const int* mb_ptr;           // the bins of the largest feature where the host only knows the bound mb; may be null
  const int32_t* row_ptr;
  const void* gpair;
  const int32_t* row_index;    // null: row i is at position i
  const int32_t* seg_begin;
  const int32_t* seg_end;
  const GPairI64* node_sums;   // null: every node is built; else the smaller child of every pair
  int node_begin;
  int n_nodes;
  const int* build_all;        // not null and not 0 there: every node is built although node_sums is given
  const int* max_abs;          // largest |grad|, |hess| of the pairs (null for float pairs)
  // the plan, where it was made by k_hist_plan (plan == null: the kernel plans for itself)
  const int32_t* chunk_off;  // [n_nodes+1] chunks before each node (tickets drawn from a counter)
  const int32_t* wpre;       // [n_nodes+1] built rows before each node (static ranges); may be null
  const int32_t* plan;       // [0] rows per chunk, [1] total chunks, [3] rows between flushes, [4] rows per
                             // range (0 = tickets from the counter), [7] ranges
  int tile_items;            // k_hist_tile: units of work a level is cut into if its nodes alone are fewer
  bool ranges;               // static ranges may be used
  long long slot_capacity;   // slots and counters of the merge trees
  int n_arrive;
  unsigned int* ticket;
  unsigned int* arrive;      // counters of the merge trees (zero before the kernel and after it); null: no merge trees
  void* partial;             // partial-sum slots of the merge trees: [slot][2][mb * 32 W] of the
                             // accumulator type; may be null
  int pairs_by_position;     // 1: gpair is stored in row_index order (pair i belongs to row_index[i]): a stream
  int* status;               // the context's status word; may be null
  void* out;
  // Several ranks, features divided among them: the histogram of a feature goes straight into the
  // memory of the rank that owns the feature (a peer store over NVLink), into that rank's receive
  // slot for this rank: recv[owner][this rank][slot * K + k][bins of the owner's features].
  void* const* push_recv;    // [push_ranks] receive buffers as this device addresses them; null = `out`
  int push_rank, push_ranks;
  long long push_slot_pairs; // pairs per (source rank) block of a receive buffer: segments x push_len
  int push_len;              // pairs per segment in a receive buffer (bound of the owned bins)
};

__device__ inline bool OneOfTwo(const HistParams& p) { return p.node_sums != nullptr && (p.build_all == nullptr || *p.build_all == 0); }

// Rows of node j of the batch that have to be summed: 0 for the sibling that is derived.
__device__ inline int BuiltRows(const HistParams& p, int j)
{
  const int rows = p.seg_end[j] - p.seg_begin[j];
  if (rows <= 0) return 0;
  if (!OneOfTwo(p)) return rows;
  const bool left = SmallerChildIsLeft(p.node_sums, p.K, p.node_begin + (j & ~1));
  return left == ((j & 1) == 0) ? rows : 0;
}
__device__ inline int SlotOf(const HistParams& p, int j) { return OneOfTwo(p) ? j >> 1 : j; }
__device__ inline int RowsSafe(const int* max_abs)
{
  return max_abs ? 2147483647 / max(1, max(max_abs[0], max_abs[1])) : 2147483647;
}

// Where the bins of feature `f` of segment (slot * K + k) go: the base to which the bin is added.
template <typename out_t>
__device__ inline out_t* FeatureBase(const HistParams& p, int f, int seg)
{
  if (p.push_recv == nullptr) return static_cast<out_t*>(p.out) + static_cast<int64_t>(seg) * p.B + p.row_ptr[f];
  // owner of f: the largest r with r * F / R <= f
  int o = static_cast<int>((static_cast<long long>(f + 1) * p.push_ranks - 1) / p.F);
  if (o > p.push_ranks - 1) o = p.push_ranks - 1;
  const int lo = p.row_ptr[OwnedBegin(o, p.push_ranks, p.F)];
  return static_cast<out_t*>(p.push_recv[o]) + static_cast<long long>(p.push_rank) * p.push_slot_pairs +
         static_cast<long long>(seg) * p.push_len + (p.row_ptr[f] - lo);
}

__device__ inline unsigned SmemAddr(const void* p) { return static_cast<unsigned>(__cvta_generic_to_shared(p)); }

// largest |grad| and |hess| of a set of quantised pairs (for the stage-level entry point; the
// tree builder gets them from the quantiser)
__global__ void k_max_abs(const int2* __restrict__ gpair, int64_t n, int* __restrict__ max_abs)
{
  AfterTheKernelBefore();
  int mg = 0, mh = 0;
  for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < n;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int2 v = gpair[i];
    // |INT32_MIN| does not fit: saturate
    mg = max(mg, v.x == INT32_MIN ? INT32_MAX : abs(v.x));
    mh = max(mh, v.y == INT32_MIN ? INT32_MAX : abs(v.y));
  }
  for (int off = 16; off >= 1; off >>= 1) {
    mg = max(mg, __shfl_down_sync(0xffffffffu, mg, off));
    mh = max(mh, __shfl_down_sync(0xffffffffu, mh, off));
  }
  if ((threadIdx.x & 31) == 0) {
    atomicMax(max_abs, mg);
    atomicMax(max_abs + 1, mh);
  }
}

// Rows per static range, and the number of ranges; 0 rows where ranges are not used.
__device__ inline void RangesOf(const HistParams& p, long long total, int GK, int resident, int& range_rows, int& ranges)
{
  range_rows = ranges = 0;
  if (!p.ranges || GK > resident) return;
  // (divisions of 32 bits: those of 64 are calls of a hundred instructions, in every block's plan)
  int n      = resident / GK;
  unsigned q = (static_cast<unsigned>(total) + n - 1) / n;
  q          = (q + kTileRows - 1) / kTileRows * kTileRows;
  if (q < 2 * kMinChunk) return;
  n = static_cast<int>((static_cast<unsigned>(total) + q - 1) / q);
  if (p.partial != nullptr) {
    const long long slots = static_cast<long long>(kTreeFanIn) * (n - 1) * GK;
    if (slots > p.slot_capacity || slots > p.n_arrive) return;
  }
  range_rows = static_cast<int>(q);
  ranges     = n;
}

// Rows per ticket.
__device__ inline int ChunkRowsOf(long long total, int nonempty_nodes, int GK, int resident, int min_chunk)
{
  long long ch = (total * GK + resident - 1) / resident;
  if (static_cast<long long>(nonempty_nodes) * GK >= resident) ch = 1ll << 30;
  if (ch < min_chunk) ch = min_chunk;
  ch = (ch + kTileRows - 1) / kTileRows * kTileRows;
  return static_cast<int>(ch < (1ll << 30) ? ch : (1ll << 30));
}

// The same for k_hist_tile with copies, whose pieces should fill the SMs once (or a whole number of times: 154 pieces
// on 148 SMs take as long as 296): pieces of ch rows are fewer than total / ch + nodes, so that w x SMs pieces are
// kept by ch = total / (w x SMs / GK - nodes); of the turns w the one whose rows (and fixed cost, about as much as
// kTileFixedRows rows) come to the least.  Nodes no longer than ch stay whole.  (A piece takes 0.7 us per 1000 rows, and 3.5 to
// be cleared, begun, turned and added: with 1500 rows for that, 100k x 50, 8 nodes were cut in two turns: 13.3 us, now 11.0;
// 300k x 64, 4 nodes 22.6 and 20.7.)
constexpr int kTileFixedRows = 5000;
__device__ inline int TileChunkRows(long long total, int nodes, int largest, int GK, int sms, int min_chunk)
{
  unsigned best = 1u << 30;
  long long best_cost = 1ll << 60;
  for (int w = 1; w <= 4; ++w) {
    const int pieces = w * sms / GK;
    if (pieces < nodes) continue;
    unsigned ch = pieces > nodes ? (static_cast<unsigned>(total) + pieces - nodes - 1) / static_cast<unsigned>(pieces - nodes) : largest;
    ch          = min(max(ch, static_cast<unsigned>(min_chunk)), static_cast<unsigned>(max(largest, min_chunk)));
    const long long cost = static_cast<long long>(w) * (ch + kTileFixedRows);
    if (cost < best_cost) {
      best_cost = cost;
      best      = ch;
    }
  }
  return static_cast<int>(best);
}

// Single block: how the rows of the built nodes are handed to the resident blocks on this level.
//
// A unit of work is (rows, group set, output), GK = group sets x outputs per row.
//
// Static ranges (needs `wpre`): the built rows of the level, laid
// end to end in node order, are cut into resident / GK equal ranges; block b takes range b / GK
// for (group set, output) b % GK and walks through the nodes its range touches.  Every block gets the
// same number of rows whatever the node sizes are (256 equal tickets on 148 blocks would otherwise
// take two rounds, the second one partly empty).  A node that reaches over a range boundary is
// built in pieces (see k_hist_smem).  Chosen when every
// range gets at least 2 * kMinChunk rows.
//
// Tickets (everything else): one chunk per node when there are at least as many non-empty nodes as
// resident blocks, else equal chunks of about total / resident rows whose sums are added to the
// histogram with 64-bit atomics; blocks draw (chunk, group set, output) tickets from a counter.
__global__ void __launch_bounds__(1024)
  k_hist_plan(const __grid_constant__ HistParams p, int GK, int resident, int min_chunk, bool whole_turns, int32_t* __restrict__ chunk_off,
              int32_t* __restrict__ wpre, int32_t* __restrict__ plan)
{
  AfterTheKernelBefore();
  __shared__ long long red[32];
  __shared__ long long wsum[32];
  __shared__ long long carry;
  __shared__ long long total_s;
  __shared__ int ch_s, nodes_s, largest_s;
  const int n_nodes = p.n_nodes;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, n_warps = blockDim.x >> 5;
  auto rows_of = [&](int j) -> int { return BuiltRows(p, j); };
  for (int i = tid; i < p.n_arrive; i += blockDim.x) p.arrive[i] = 0u;
  long long rows = 0, nonempty = 0;
  int largest = 0;
  if (tid == 0) largest_s = 0;
  for (int j = tid; j < n_nodes; j += blockDim.x) {
    const int r = rows_of(j);
    rows += r;
    nonempty += r > 0;
    largest = max(largest, r);
  }
  rows += nonempty << 40;
  for (int off = 16; off >= 1; off >>= 1) rows += __shfl_down_sync(0xffffffffu, rows, off);
  if (lane == 0) red[warp] = rows;
  __syncthreads();
  largest = __reduce_max_sync(0xffffffffu, largest);
  if (lane == 0) atomicMax(&largest_s, largest);
  if (tid == 0) {
    long long total = 0;
    for (int w = 0; w < n_warps; ++w) total += red[w];
    nodes_s = static_cast<int>(total >> 40);
    total_s = total & ((1ll << 40) - 1);
    plan[3] = RowsSafe(p.max_abs);
  }
  __syncthreads();
  const long long total = total_s;

  // exclusive scan over the nodes: store(j, sum of value(0..j)); 1024 nodes per step
  auto scan_nodes = [&](auto value, auto store) {
    __syncthreads();
    if (tid == 0) carry = 0;
    __syncthreads();
    for (int base = 0; base < n_nodes; base += blockDim.x) {
      const int j       = base + tid;
      const long long c = j < n_nodes ? value(j) : 0;
      long long incl    = c;
      for (int off = 1; off < 32; off <<= 1) {
        const long long n = __shfl_up_sync(0xffffffffu, incl, off);
        if (lane >= off) incl += n;
      }
      if (lane == 31) wsum[warp] = incl;
      __syncthreads();
      if (warp == 0) {
        const long long w = lane < n_warps ? wsum[lane] : 0;
        long long wi      = w;
        for (int off = 1; off < 32; off <<= 1) {
          const long long n = __shfl_up_sync(0xffffffffu, wi, off);
          if (lane >= off) wi += n;
        }
        wsum[lane] = wi - w;
      }
      __syncthreads();
      const long long before = carry + wsum[warp];
      if (j < n_nodes) store(j, before + incl);
      __syncthreads();
      if (tid == blockDim.x - 1) carry = before + incl;
      __syncthreads();
    }
  };

  // static ranges
  int range_rows = 0, ranges = 0;
  if (wpre != nullptr && total < (1ll << 31)) RangesOf(p, total, GK, resident, range_rows, ranges);
  if (wpre != nullptr) {
    scan_nodes([&](int j) -> long long { return rows_of(j); },
               [&](int j, long long incl) { wpre[j + 1] = static_cast<int>(incl); });
    if (tid == 0) wpre[0] = 0;
  }

  // tickets
  if (tid == 0) {
    ch_s = whole_turns ? TileChunkRows(total, nodes_s, largest_s, GK, resident, min_chunk) : ChunkRowsOf(total, nodes_s, GK, resident, min_chunk);
  }
  __syncthreads();
  const int ch = ch_s;
  scan_nodes(
    [&](int j) -> long long {
      const int r = rows_of(j);
      return r > 0 ? (r - 1) / ch + 1 : 0;
    },
    [&](int j, long long incl) { chunk_off[j + 1] = static_cast<int>(incl); });
  if (tid == 0) {
    chunk_off[0] = 0;
    plan[0]      = ch;
    plan[1]      = static_cast<int>(carry);
    plan[4]      = range_rows;
    plan[7]      = range_rows > 0 ? ranges : 0;
    *p.ticket    = 0;
  }
}

// The same plan, made by every block of a histogram kernel for itself: a level of at most kPlanNodes
// nodes costs one pass over their sizes (about a microsecond, all blocks at once) instead of a
// single-block launch that everybody waits for.
struct PlanView {
  const int32_t* off;  // [n_nodes + 1]: built rows before each node (ranges) or chunks before each node (tickets)
  int rows_safe, range_rows, ranges, total_chunks;
};
template <int kThreads, bool kWholeTurns = false>
__device__ inline PlanView PlanInside(const HistParams& p, int GK, int resident, int min_chunk, bool ranges_too,
                                      int32_t* s_off /* [kPlanNodes + 1] */, int* s_tmp /* [kThreads / 32] */)
{
  constexpr int kPer = kPlanNodes / kThreads;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, n = p.n_nodes;
  int c[kPer];
#pragma unroll
  for (int i = 0; i < kPer; ++i) {
    const int j = tid * kPer + i;
    c[i]        = j < n ? BuiltRows(p, j) : 0;
  }
  int nonempty = 0;
#pragma unroll
  for (int i = 0; i < kPer; ++i) nonempty += __syncthreads_count(c[i] > 0);
  auto scan = [&]() {
    int sum = 0;
#pragma unroll
    for (int i = 0; i < kPer; ++i) sum += c[i];
    int incl = sum;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, incl, off);
      if (lane >= off) incl += v;
    }
    __syncthreads();
    if (lane == 31) s_tmp[warp] = incl;
    __syncthreads();
    if (warp == 0) {
      const int w = lane < kThreads / 32 ? s_tmp[lane] : 0;
      int wi      = w;
#pragma unroll
      for (int off = 1; off < 32; off <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, wi, off);
        if (lane >= off) wi += v;
      }
      if (lane < kThreads / 32) s_tmp[lane] = wi - w;
    }
    __syncthreads();
    int before = s_tmp[warp] + incl - sum;
#pragma unroll
    for (int i = 0; i < kPer; ++i) {
      const int j = tid * kPer + i;
      if (j < n) s_off[j] = before;
      before += c[i];
      if (j == n - 1) s_off[n] = before;
    }
    __syncthreads();
  };
  scan();
  const int total = s_off[n];
  PlanView v;
  v.off       = s_off;
  v.rows_safe = RowsSafe(p.max_abs);
  v.range_rows = v.ranges = 0;
  if (ranges_too) RangesOf(p, total, GK, resident, v.range_rows, v.ranges);
  v.total_chunks = 0;
  if (v.range_rows == 0) {
    int ch;
    if (kWholeTurns) {
      int largest = 0;
#pragma unroll
      for (int i = 0; i < kPer; ++i) largest = max(largest, c[i]);
      largest = __reduce_max_sync(0xffffffffu, largest);
      if (lane == 0) s_tmp[warp] = largest;
      __syncthreads();
      for (int w = 0; w < kThreads / 32; ++w) largest = max(largest, s_tmp[w]);
      __syncthreads();
      ch = TileChunkRows(total, nonempty, largest, GK, resident, min_chunk);
    } else {
      ch = ChunkRowsOf(total, nonempty, GK, resident, min_chunk);
    }
#pragma unroll
    for (int i = 0; i < kPer; ++i) c[i] = c[i] > 0 ? (c[i] - 1) / ch + 1 : 0;
    scan();
    v.total_chunks = s_off[n];
  }
  return v;
}

template <bool kFloat>
struct Acc;
template <>
struct Acc<false> {
  using smem_t = int;
  using in_t   = int2;
  using out_t  = GPairI64;
  __device__ static void add_global(out_t* dst, int g, int h)
  {
    atomicAdd(reinterpret_cast<unsigned long long*>(&dst->grad), static_cast<unsigned long long>(static_cast<long long>(g)));
    atomicAdd(reinterpret_cast<unsigned long long*>(&dst->hess), static_cast<unsigned long long>(static_cast<long long>(h)));
  }
  __device__ static void add_word(out_t* dst, int word, int v)
  {
    atomicAdd(reinterpret_cast<unsigned long long*>(dst) + word, static_cast<unsigned long long>(static_cast<long long>(v)));
  }
  __device__ static void store_global(out_t* dst, int g, int h)
  {
    *reinterpret_cast<longlong2*>(dst) = make_longlong2(g, h);
  }
  __device__ static bool nonzero(int g, int h) { return (g | h) != 0; }
  __device__ static int4 add4(int4 a, int4 b) { return make_int4(a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w); }
  __device__ static void red_shared(unsigned addr, int bits)
  {
    asm volatile("red.shared.add.s32 [%0], %1;\n" ::"r"(addr), "r"(bits) : "memory");
  }
  template <int kOffset>
  __device__ static void red_shared_at(unsigned addr, int bits)
  {
    asm volatile("red.shared.add.s32 [%0+%2], %1;\n" ::"r"(addr), "r"(bits), "n"(kOffset) : "memory");
  }
};
template <>
struct Acc<true> {
  using smem_t = float;
  using in_t   = float2;
  using out_t  = GPairF64;
  __device__ static void add_global(out_t* dst, float g, float h)
  {
    atomicAdd(&dst->grad, static_cast<double>(g));
    atomicAdd(&dst->hess, static_cast<double>(h));
  }
  __device__ static void add_word(out_t* dst, int word, float v) { atomicAdd(reinterpret_cast<double*>(dst) + word, static_cast<double>(v)); }
  __device__ static void store_global(out_t* dst, float g, float h)
  {
    *reinterpret_cast<double2*>(dst) = make_double2(g, h);
  }
  __device__ static bool nonzero(float g, float h) { return g != 0.f || h != 0.f; }
  __device__ static int4 add4(int4 a, int4 b)
  {
    return make_int4(__float_as_int(__int_as_float(a.x) + __int_as_float(b.x)),
                     __float_as_int(__int_as_float(a.y) + __int_as_float(b.y)),
                     __float_as_int(__int_as_float(a.z) + __int_as_float(b.z)),
                     __float_as_int(__int_as_float(a.w) + __int_as_float(b.w)));
  }
  __device__ static void red_shared(unsigned addr, int bits)
  {
    asm volatile("red.shared.add.f32 [%0], %1;\n" ::"r"(addr), "f"(__int_as_float(bits)) : "memory");
  }
  template <int kOffset>
  __device__ static void red_shared_at(unsigned addr, int bits)
  {
    asm volatile("red.shared.add.f32 [%0+%2], %1;\n" ::"r"(addr), "f"(__int_as_float(bits)), "n"(kOffset) : "memory");
  }
};

// One piece of work of a block: rows [rb, re) of row_index, all of one node.
struct Piece {
  int j;          // node of the batch
  int slot;       // the node's histogram in `out`
  int rb, re;
  int index;      // which piece of its node this is, 0 .. pieces-1
  int pieces;     // pieces the node is built in
  int tree_base;  // first slot / counter of the node's merge tree (pieces > 1, static ranges)
  int node_rows;  // rows of the whole node
};

__device__ inline Piece DecodeChunk(const HistParams& p, const int32_t* __restrict__ chunk_off, int c)
{
  // node that owns chunk c: last j with chunk_off[j] <= c
  int lo = 0, hi = p.n_nodes;
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (chunk_off[mid] <= c) lo = mid; else hi = mid;
  }
  Piece pc;
  pc.j         = lo;
  pc.pieces    = chunk_off[lo + 1] - chunk_off[lo];
  pc.slot      = SlotOf(p, lo);
  pc.index     = c - chunk_off[lo];
  pc.tree_base = -1;
  // the chunks of a node are equal in size (a multiple of 32 rows, the last one takes the rest)
  const int nrows = p.seg_end[lo] - p.seg_begin[lo];
  pc.node_rows    = nrows;
  const int size  = pc.pieces > 1 ? ((nrows + pc.pieces - 1) / pc.pieces + kTileRows - 1) / kTileRows * kTileRows : nrows;
  pc.rb = min(p.seg_end[lo], p.seg_begin[lo] + pc.index * size);
  pc.re = min(p.seg_end[lo], pc.rb + size);
  return pc;
}

// Rows [b, e) of one node, features [f0, f0 + 32 * groups): one lane per feature, the warps of the
// block stride over the rows, every update is a pair of 64-bit global atomics.
template <typename BinT, typename A>
__device__ inline void DirectRows(const HistParams& p, int b, int e, int f0, int groups, int k,
                                  int seg, int warp, int n_warps, int lane)
{
  using in_t          = typename A::in_t;
  const BinT* bins    = static_cast<const BinT*>(p.bins);
  const in_t* gpair   = static_cast<const in_t*>(p.gpair);
  const int64_t pitch = static_cast<int64_t>(p.G) * kGroup;
  for (int u = 0; u < groups; ++u) {
    const int feat = f0 + u * kGroup + lane;
    if (feat >= p.F) continue;
    typename A::out_t* obase = FeatureBase<typename A::out_t>(p, feat, seg);
    for (int r = b + warp; r < e; r += n_warps) {
      const int ridx = p.row_index != nullptr ? p.row_index[r] : r;
      const in_t v   = gpair[static_cast<int64_t>(p.pairs_by_position ? r : ridx) * p.K + k];
      const int bin  = bins[static_cast<int64_t>(ridx) * pitch + feat];
      A::add_global(obase + bin, v.x, v.y);
    }
  }
}

// Bins of two bytes, or more than 256 bins in a feature: every ticket goes straight to global atomics.
template <typename BinT, bool kFloat>
__global__ void __launch_bounds__(kHistThreads)
  k_hist_direct(const HistParams p)
{
  AfterTheKernelBefore();
  using A = Acc<kFloat>;
  __shared__ unsigned int s_ticket;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const long long total = static_cast<long long>(p.plan[1]) * p.G * p.K;  // (always planned by k_hist_plan)
  while (true) {
    __syncthreads();
    if (tid == 0) s_ticket = atomicAdd(p.ticket, 1u);
    __syncthreads();
    const long long t = s_ticket;
    if (t >= total) break;
    const int k    = static_cast<int>(t % p.K);
    const int g    = static_cast<int>((t / p.K) % p.G);
    const Piece pc = DecodeChunk(p, p.chunk_off, static_cast<int>(t / (static_cast<long long>(p.K) * p.G)));
    DirectRows<BinT, A>(p, pc.rb, pc.re, g * kGroup, 1, k, pc.slot * p.K + k, warp, kHistThreads / 32, lane);
  }
}

// One update step of a lane: byte J of its bin bytes (already permuted so that step J reads
// the static byte J; at most 16, with places for eight main and eight extra ones), both words of the pair.  `lane_word` is the shared-memory address of the
// lane's word in bin row 0 of the gradient histogram.
template <typename A, int W, int J, bool kMask>
__device__ inline void HistStep(const unsigned (&x)[4], unsigned lane_word, const int2& v, unsigned steps)
{
  if (kMask && (steps >> J & 1u) == 0u) return;
  constexpr int kHistBytes = kSmemBins * kGroup * W * 4;
  if (W == 2) {
    // a bin row is 256 bytes: the offset is (bin << 8) | (lane_word ^ skew), one byte permute and one
    // three-input logic op; where the histograms begin is an immediate of the instruction
    constexpr unsigned cj = ((J & 7u) << 2) | ((J >> 3) << 7);
    const unsigned b8     = __byte_perm(x[J >> 2], 0u, 0x4404u | ((J & 3) << 4));
    unsigned addr;
    asm("lop3.b32 %0, %1, %2, %3, 0xF6;\n" : "=r"(addr) : "r"(b8), "r"(lane_word), "n"(cj));
    A::template red_shared_at<kHistBase>(addr, v.x);
    A::template red_shared_at<kHistBase + kHistBytes>(addr, v.y);
  } else {
    constexpr unsigned cj = 4u * J;
    const unsigned bin    = __byte_perm(x[J >> 2], 0u, 0x4440u | (J & 3));
    const unsigned addr   = (bin * (kGroup * 4) + lane_word) ^ cj;
    A::template red_shared_at<kHistBase>(addr, v.x);
    A::template red_shared_at<kHistBase + kHistBytes>(addr, v.y);
  }
}

template <typename A, int W, int kFrom, int kTo, bool kMask>
__device__ inline void HistSteps(const unsigned (&x)[4], unsigned lane_word, const int2& v, unsigned steps)
{
  if constexpr (kFrom < kTo) {
    HistStep<A, W, kFrom, kMask>(x, lane_word, v, steps);
    HistSteps<A, W, kFrom + 1, kTo, kMask>(x, lane_word, v, steps);
  }
}

// The rows [sb, se) of row_index, all of one node, added to the block's private histograms: the
// main loop of k_hist_smem for one warp.  The warps of the block take the batches of 32 / (2 W)
// rows in turn.  Every load of the loop is unconditional: batch numbers beyond the warp's last one
// are clamped to it (the rows are fetched again and dropped), and the last, partial batch of the range is
// handled after the loop.  In flight per warp: the rows of the next two batches and the row ids of
// the two after; the loop is unrolled three times so that the three row buffers rotate by name.
// The row's bin bytes come with a plain load that bypasses L1 and, where a row is longer than a unit's 64 bytes (kLine),
// asks L2 for the whole 128-byte line (the other half of the row is wanted soon by the block that builds the neighbouring
// groups).  A row of 64 bytes has its neighbour in the other half: asking for 128 brought 132 bytes a row from DRAM where a node
// has one row in 64, now 79 (100M x 64, depth 10: 26.2 -> 25.2 ms).  kOrder: kPairsByPosition - the pairs are stored in row_index order and read as a stream;
// kPairsByRow - they are gathered by row id; kRowsInOrder - there is no row_index, row i is at position i.
//
// kMain, kExtra: the form of the unit (UnitForm).  Of 33 to 48 features (kExtra 1, 2, 4) the 16-byte loads are not as the steps
// want them: lane 3 takes the upper half of lane 0's piece, and a word or two go from lane 1 (and 2) to the others by shuffle,
// cheaper than a second load, which would touch the row's line again.
enum RowOrder { kPairsByRow, kPairsByPosition, kRowsInOrder };
template <typename A, int W, RowOrder kOrder, int kMain, int kExtra, bool kLine, bool kMask>
__device__ __forceinline__ void HistRows(const HistParams& p, int sb, int se, int g0, int k, int warp, int lane, unsigned lane_word)
{
  using in_t = typename A::in_t;
  constexpr int kWarps        = kHistThreads * W / 32;
  constexpr int kLanesPerRow  = 2 * W;
  constexpr int kRowsPerBatch = 32 / kLanesPerRow;
  constexpr UnitForm kForm{kMain, kExtra};
  constexpr int kLoad         = LaneBytes(kForm);  // bytes of a lane's load
  constexpr bool kShared      = kExtra == 1 || kExtra == 2 || kExtra == 4;
  const unsigned rslot = lane / kLanesPerRow, q = lane % kLanesPerRow;
  const unsigned wsel = rslot >> 2, bsel = rslot & 3;
  const unsigned perm = bsel == 0 ? 0x3210u : bsel == 1 ? 0x2301u : bsel == 2 ? 0x1032u : 0x0123u;
  const unsigned sel0 = perm + ((wsel & 1) ? 0x4444u : 0u), sel1 = perm + ((wsel & 1) ? 0u : 0x4444u);
  const unsigned sel2 = (rslot & 1) ? 0x4401u : 0x4410u;  // two bytes
  const int from      = PieceOfLane(W, kForm, kLine ? min(W, p.G - g0) : W, static_cast<int>(q));  // the lane's piece of the row
  const int64_t pitch = static_cast<int64_t>(p.G) * kGroup;
  const unsigned char* gb = static_cast<const unsigned char*>(p.bins) + g0 * kGroup + from * kLoad;
  unsigned steps = 0u;  // kMask: those in which the lane has a feature
  if (kMask) {
#pragma unroll 1
    for (int j = 0; j < 16; ++j) {
      const int n = W == 1 || j < 8 ? kMain : kExtra, col = (static_cast<int>(rslot) ^ j) & (n - 1);
      const int w = W == 1 ? 16 * static_cast<int>(q) + col : 32 * (j >> 3) + 8 * static_cast<int>(q) + col;
      if (n > 0 && g0 * kGroup + FeatureOfWord(W, kForm, w) < p.F) steps |= 1u << j;
    }
  }
  const in_t* gpair    = static_cast<const in_t*>(p.gpair);
  const int pos0       = sb + static_cast<int>(rslot);  // the lane's row of batch 0, as a position in row_index
  const int32_t* rp    = p.row_index + pos0;            // + batch * kRowsPerBatch

  // rid: the row; pos: its position in row_index (only used for pairs stored by position)
  auto load = [&](int rid, int pos, int4& w, int2& v) {
    const unsigned char* ap = gb + static_cast<int64_t>(rid) * pitch;
    if (kLoad == 16 && kLine) {
      asm volatile("ld.global.nc.L1::no_allocate.L2::128B.v4.s32 {%0,%1,%2,%3}, [%4];" : "=r"(w.x), "=r"(w.y), "=r"(w.z), "=r"(w.w) : "l"(ap));
    } else if (kLoad == 16) {
      asm volatile("ld.global.nc.L1::no_allocate.L2::64B.v4.s32 {%0,%1,%2,%3}, [%4];" : "=r"(w.x), "=r"(w.y), "=r"(w.z), "=r"(w.w) : "l"(ap));
    } else if (kLoad == 8) {
      asm volatile("ld.global.nc.L1::no_allocate.L2::64B.v2.s32 {%0,%1}, [%2];" : "=r"(w.x), "=r"(w.y) : "l"(ap));
    } else if (kLoad == 4) {
      asm volatile("ld.global.nc.L1::no_allocate.L2::64B.s32 %0, [%1];" : "=r"(w.x) : "l"(ap));
    } else {
      asm volatile("{.reg .u16 t; ld.global.nc.L1::no_allocate.L2::64B.u16 t, [%1]; cvt.u32.u16 %0, t;}" : "=r"(w.x) : "l"(ap));
    }
    if (kOrder != kPairsByRow) v = __ldcs(reinterpret_cast<const int2*>(gpair + static_cast<int64_t>(pos) * p.K + k));
    else v = __ldcg(reinterpret_cast<const int2*>(gpair + static_cast<int64_t>(rid) * p.K + k));
  };
  auto consume = [&](const int4& w, const int2& v) {
    unsigned x[4] = {};
    if (kShared) {
      const int l1 = lane - static_cast<int>(q) + 1;  // the row's lane 1
      int m0 = q == 3 ? w.z : w.x, m1 = q == 3 ? w.w : w.y;
      if (kExtra == 4) {
        const int other = __shfl_sync(0xffffffffu, w.w, q == 3 ? l1 + 1 : l1);
        x[2]            = __byte_perm(q == 1 || q == 2 ? w.z : other, 0, perm);
      } else {
        const int s6 = __shfl_sync(0xffffffffu, w.z, l1), s7 = __shfl_sync(0xffffffffu, w.w, l1);
        if (kExtra == 1) {
          x[2] = __byte_perm(s7, 0, 0x4440u | q);
          if (q == 2) m1 = s6;
        } else {
          x[2] = __byte_perm(s6, s7, (sel2 & 0xffu) + 0x22u * q);
        }
      }
      x[0] = __byte_perm(m0, m1, sel0);
      x[1] = __byte_perm(m0, m1, sel1);
    } else if (kMain == 2) {
      x[0] = __byte_perm(w.x, 0, sel2);
    } else if (kMain == 4) {
      x[0] = __byte_perm(w.x, 0, perm);
    } else if (kMain == 8) {
      x[0] = __byte_perm(w.x, w.y, sel0);
      x[1] = __byte_perm(w.x, w.y, sel1);
      if (kExtra == 8) {
        x[2] = __byte_perm(w.z, w.w, sel0);
        x[3] = __byte_perm(w.z, w.w, sel1);
      }
    } else {
      const unsigned a0 = (wsel & 2) ? w.z : w.x, a1 = (wsel & 2) ? w.w : w.y;
      const unsigned b0 = (wsel & 2) ? w.x : w.z, b1 = (wsel & 2) ? w.y : w.w;
      x[0] = __byte_perm(a0, a1, sel0);
      x[1] = __byte_perm(a0, a1, sel1);
      x[2] = __byte_perm(b0, b1, sel0);
      x[3] = __byte_perm(b0, b1, sel1);
    }
    HistSteps<A, W, 0, kMain, kMask>(x, lane_word, v, steps);
    HistSteps<A, W, 8, 8 + kExtra, kMask>(x, lane_word, v, steps);
  };

  const int n_here  = se - sb;
  const int nb_full = n_here / kRowsPerBatch;
  int cnt           = nb_full > warp ? (nb_full - warp + kWarps - 1) / kWarps : 0;  // this warp's whole batches
  if (cnt > 0) {
    const int bl = warp + (cnt - 1) * kWarps;  // the warp's last batch
    auto rid_at  = [&](int bb) -> int {
      return kOrder == kRowsInOrder ? pos0 + bb * kRowsPerBatch : __ldcg(rp + bb * kRowsPerBatch);
    };
    int b = warp;
    int4 wa, wb, wc;
    int2 va, vb, vc;
    {
      const int b1 = min(b + kWarps, bl);
      load(rid_at(b), pos0 + b * kRowsPerBatch, wa, va);
      load(rid_at(b1), pos0 + b1 * kRowsPerBatch, wb, vb);
    }
    int ba = min(b + 2 * kWarps, bl), bb = min(b + 3 * kWarps, bl);
    int ra = rid_at(ba), rb = rid_at(bb);
#pragma unroll 1
    while (cnt >= 3) {
      load(ra, pos0 + ba * kRowsPerBatch, wc, vc);
      ba = min(b + 4 * kWarps, bl);
      ra = rid_at(ba);
      consume(wa, va);
      load(rb, pos0 + bb * kRowsPerBatch, wa, va);
      bb = min(b + 5 * kWarps, bl);
      rb = rid_at(bb);
      consume(wb, vb);
      load(ra, pos0 + ba * kRowsPerBatch, wb, vb);
      ba = min(b + 6 * kWarps, bl);
      ra = rid_at(ba);
      consume(wc, vc);
      // now the buffers hold batches b + 3, b + 4 (in units of kWarps) and the ids b + 5 (rb), b + 6 (ra)
      int t = ra; ra = rb; rb = t;
      t = ba; ba = bb; bb = t;
      b += 3 * kWarps;
      cnt -= 3;
    }
    if (cnt >= 1) consume(wa, va);
    if (cnt >= 2) consume(wb, vb);
  }
  // the partial batch at the end of the range
  const int tail = n_here - nb_full * kRowsPerBatch;
  if (tail > 0 && warp == nb_full % kWarps) {
    const bool valid = static_cast<int>(rslot) < tail;
    // lanes without a row read the first row of the range (it exists) and add nothing
    const int pos    = valid ? pos0 + nb_full * kRowsPerBatch : sb;
    const int rid    = kOrder == kRowsInOrder ? pos : __ldcg(p.row_index + pos);
    int4 w;
    int2 v;
    load(rid, pos, w, v);
    if (!valid) v = make_int2(0, 0);
    consume(w, v);
  }
}

// One-byte bins, at most 256 per feature: private histograms in shared memory.
//
// W = 1: a unit covers one 32-feature group, 512 threads, two blocks per SM.
// W = 2: a unit covers two neighbouring groups (64 features), 1024 threads, one block per SM.
// The wide form exists because the load/store pipe of the SM spends one pass per distinct
// 128-byte line a gather touches, however few bytes it takes from it: with 64 bin bytes per row
// the row gather costs half as many passes per update, and the row ids and gradient pairs are
// fetched once for two groups.
//
// Shared memory: the gradient histogram [256 bins][32 W words] sits at the fixed address kHistBase, the
// hessian histogram behind it, so that an update needs no base register; then the staging area of the
// flush and the plan.  Every warp runs its own pipeline over batches of 32 / (2 W) rows (no block barrier
// inside).  2 W lanes own one row of the batch and load its bin bytes straight from global memory
// into registers.  Units of all their features, and those of several units of whole numbers, take 16 bytes per lane: in step j of 16
// the lanes of row slot r handle byte (j xor r) of their 16, and the histogram words of a bin are laid out so that the 32 lanes of a
// warp always update 32 different banks, whatever the bins:
//   W = 1 (r < 16, quarter q < 2):  word = 16 q + byte                   (bank = word)
//   W = 2 (r < 8,  quarter q < 4):  word = 32 (byte / 8) + 8 q + byte % 8 (bank = 8 q + byte % 8)
// Other units load fewer bytes per lane and take fewer steps, and words that no feature needs are copies of other ones, so that the
// banks stay different (UnitForm, FeatureOfWord and PieceOfLane, hist_units.h).
// The bytes are permuted once per batch (a word swap and one byte permute per word) so that step
// j reads the static byte j.  Per 32 updates that leaves the two reductions on the pipe.
//
// Flush: a warp takes a tile of 4 bins x 32 words, turns it in its staging area (a skewed 4 x 32
// array, conflict free both ways) and writes, per word, the 4 bins of a feature as 64 contiguous
// bytes of the output.  Copies of a word are added up on the way into the staging area, by shuffle, and the words without a feature are left out;
// an image that goes into a slot of a merge tree (below) is the words as they are, copies apart.
//
// The pieces of a node that reaches over range boundaries add their sums to its histogram with 64-bit atomics. An
// instruction of the warp covers 16 whole (grad, hess) pairs, so that every sector is touched once: 148 blocks adding 256 KB
// each, all to the same region, take 10 us, as long as plain stores to regions of their own (15 with the two words
// of a pair in two instructions).  The merge tree took 28 us for the 148 pieces of one node, mostly on few SMs, and
// scratch for the pieces.  One node, 10M x 64: 240 -> 214 us; 8 nodes 270 -> 241, 128 nodes 277 -> 252; 10M x 128, 128 nodes
// 470 -> 462; 1.25M x 64, one node 68 -> 46.
//
// Merge tree (static ranges, histograms of other ranks' features, where the atomics would cross NVLink): the P pieces of a
// node that reaches over range boundaries are summed without waits.  A piece writes its 32-bit partial sums to its slot and
// adds one to the counter of its group of four; the last one to arrive adds the others' slots to its own sums and goes on
// as one member of the next level, until one block holds the node's total and writes the histogram.  Nobody waits for
// anybody: whoever arrives first leaves.  (lbk_selftest_histogram takes it with local histograms.)
template <bool kFloat, int W, RowOrder kOrder, bool kLine>
__global__ void __launch_bounds__(kHistThreads * W, W == 1 ? 2 : 1)
  k_hist_smem(const HistParams p)
{
  using A      = Acc<kFloat>;
  using smem_t = typename A::smem_t;
  using in_t   = typename A::in_t;
  using out_t  = typename A::out_t;
  constexpr int kThreads      = kHistThreads * W;
  constexpr int kWarps        = kThreads / 32;
  constexpr int kCols         = kGroup * W;   // histogram words per bin
  constexpr int kHistBytes    = kSmemBins * kCols * 4;
  constexpr int kLanesPerRow  = 2 * W;
  constexpr int kRowsPerBatch = 32 / kLanesPerRow;
  constexpr int kStageWords   = kFlushBins * 32;  // per warp
  AfterTheKernelBefore();
  extern __shared__ __align__(128) unsigned char smem_raw[];
  __shared__ unsigned int s_ticket;
  __shared__ int s_nb[kCols];  // bins of the feature of each word (0: no feature, or a copy of another word)
  __shared__ typename Acc<kFloat>::out_t* s_base[kCols];  // where its bin 0 goes, for the piece at hand

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const unsigned base = SmemAddr(smem_raw);
  unsigned dyn_bytes;
  asm("mov.u32 %0, %%dynamic_smem_size;" : "=r"(dyn_bytes));
  // the histograms begin at kHistBase: behind what comes before the dynamic shared memory, and everything
  // inside what was asked for
  if (base > kHistBase || HistSmemBytes(W) > base + dyn_bytes) {
    if (tid == 0 && p.status != nullptr) ReportFault(p.status, kFaultHistLayout);
    return;
  }
  smem_t* hg        = reinterpret_cast<smem_t*>(smem_raw + (kHistBase - base));
  smem_t* hh        = hg + kSmemBins * kCols;
  smem_t* stage_all = hh + kSmemBins * kCols;
  int32_t* s_off    = reinterpret_cast<int32_t*>(stage_all + kWarps * kStageWords);  // [kPlanNodes + 1]
  int* s_tmp        = s_off + kPlanNodes + 1;                                        // [32]

  const int GP = (p.G + W - 1) / W;  // group sets per row
  // (the plan stays in shared memory: the main loop needs the registers)
  __shared__ PlanView pv;
  {
    PlanView v{};
    if (p.plan == nullptr) {
      v = PlanInside<kThreads>(p, GP * p.K, gridDim.x, kMinChunk, true, s_off, s_tmp);
    } else {
      v.rows_safe    = p.plan[3];
      v.range_rows   = p.wpre != nullptr ? p.plan[4] : 0;
      v.ranges       = p.plan[7];
      v.total_chunks = p.plan[1];
      v.off          = v.range_rows > 0 ? p.wpre : p.chunk_off;
    }
    if (tid == 0) pv = v;
    __syncthreads();
  }
  const int rows_safe   = pv.rows_safe;
  const int range_rows  = pv.range_rows;
  const int mb          = p.mb_ptr != nullptr ? min(p.mb, *p.mb_ptr) : p.mb;
  const in_t* gpair     = static_cast<const in_t*>(p.gpair);
  const int hist_words  = mb * kCols;
  const int64_t pitch   = static_cast<int64_t>(p.G) * kGroup;  // bins are row-major, rows padded to whole groups
  // chunks that merge through slots never flush in the middle: they stay below the safe count
  const int cap_rows    = rows_safe >= (1 << 30) ? (1 << 30) : (rows_safe & ~(kTileRows - 1));

  const unsigned rslot    = lane / kLanesPerRow, q = lane % kLanesPerRow;
  const unsigned wsel     = rslot >> 2, bsel = rslot & 3;
  const unsigned perm     = bsel == 0 ? 0x3210u : bsel == 1 ? 0x2301u : bsel == 2 ? 0x1032u : 0x0123u;
  const unsigned lane_word = (W == 1 ? 16 * q + rslot : 8 * q + rslot) * 4;

  auto zero = [&]() {
    int4* g4 = reinterpret_cast<int4*>(hg);
    int4* h4 = reinterpret_cast<int4*>(hh);
    for (int e = tid; e < (hist_words >> 2); e += kThreads) {
      g4[e] = make_int4(0, 0, 0, 0);
      h4[e] = make_int4(0, 0, 0, 0);
    }
  };

  // One piece: accumulate its rows, then flush / merge.
  auto process = [&](const Piece& pc, int gp, int k) {
    const int g0     = gp * W;
    const int groups = min(W, p.G - g0);
    const int seg    = pc.slot * p.K + k;
    // the merge tree adds 32-bit images: a piece (at most range_rows rows) has to stay below the safe
    // count, and the tree is climbed only as far as the merged images do (see below)
    const bool tree  = pc.pieces > 1 && pc.tree_base >= 0 && p.partial != nullptr && range_rows <= cap_rows &&
                      rows_safe >= kTileRows;
    if (rows_safe < kTileRows || (pc.re - pc.rb <= kDirectRows && !tree)) {
      DirectRows<uint8_t, A>(p, pc.rb, pc.re, g0 * kGroup, groups, k, seg, warp, kWarps, lane);
      return;
    }
    __syncthreads();  // whoever still reads the histogram or s_nb of the piece before
    const UnitForm form = kLine && !kFloat ? UnitForm{8, 8} : FormOf(kFloat, W, kLine, min(kCols, p.F - g0 * kGroup));
    for (int i = tid; i < kCols; i += kThreads) {
      const int r = FeatureOfWord(W, form, i), f = g0 * kGroup + r;
      const bool is = r >= 0 && f < p.F;
      s_nb[i]       = is ? p.row_ptr[f + 1] - p.row_ptr[f] : 0;
      s_base[i]     = is ? FeatureBase<out_t>(p, f, seg) : nullptr;
    }
    zero();
    __syncthreads();

    // the flush: tiles of kFlushBins bins x 32 words, turned in the warp's staging area
    auto flush = [&](bool atomics) {
      constexpr int kWordsPer = 32 / kFlushBins;  // words of a tile that leave with one store of the warp
      smem_t* stage      = stage_all + warp * kStageWords;
      const int n_btiles = (mb + kFlushBins - 1) / kFlushBins;
      const int a = lane / kFlushBins, b = lane % kFlushBins;
      const int halves   = W == 2 && (!kFloat || form.extra != 0) ? 2 : 1;
      for (int t = warp; t < n_btiles * halves; t += kWarps) {
        const int half = t / n_btiles, bin0 = (t - half * n_btiles) * kFlushBins;
        const int own  = half == 0 ? form.main : form.extra;  // columns that are not copies
        smem_t gv[kFlushBins];
#pragma unroll
        for (int pass = 0; pass < 2; ++pass) {
          const smem_t* src = (pass == 0 ? hg : hh) + half * 32 + lane;
#pragma unroll
          for (int bb = 0; bb < kFlushBins; ++bb) {
            const int bin = bin0 + bb;
            smem_t v      = bin < mb ? src[bin * kCols] : smem_t(0);
            if (!kLine || kFloat)
              for (int d = own; d < (W == 1 ? 16 : 8); d <<= 1) v += __shfl_xor_sync(0xffffffffu, v, d);
            stage[bb * 32 + ((lane + kWordsPer * bb) & 31)] = v;
          }
          __syncwarp();
          if (pass == 0) {
#pragma unroll
            for (int i = 0; i < kFlushBins; ++i) gv[i] = stage[b * 32 + ((kWordsPer * i + a + kWordsPer * b) & 31)];
          } else {
#pragma unroll
            for (int i = 0; i < kFlushBins; ++i) {
              const smem_t hv = stage[b * 32 + ((kWordsPer * i + a + kWordsPer * b) & 31)];
              if (atomics) {
                // the lanes of an instruction add to whole sectors: lane l the word l % 2 of the pair that lane
                // l / 2 (or 16 + l / 2) holds
#pragma unroll
                for (int part = 0; part < 2; ++part) {
                  const int from  = part * 16 + (lane >> 1);
                  const smem_t vg = __shfl_sync(0xffffffffu, gv[i], from), vh = __shfl_sync(0xffffffffu, hv, from);
                  const int f     = half * 32 + kWordsPer * i + from / kFlushBins;
                  const int bin   = bin0 + from % kFlushBins;
                  const smem_t v  = (lane & 1) ? vh : vg;
                  if (bin < s_nb[f] && v != smem_t(0)) A::add_word(s_base[f] + bin, lane & 1, v);
                }
                continue;
              }
              const int f   = half * 32 + kWordsPer * i + a;
              const int bin = bin0 + b;
              if (bin < s_nb[f] && A::nonzero(gv[i], hv)) A::store_global(s_base[f] + bin, gv[i], hv);
            }
          }
          __syncwarp();
        }
      }
    };

    bool use_atomics   = pc.pieces > 1 && !tree;
    const int seg_rows = rows_safe >= (1 << 30) ? (1 << 30) : (rows_safe & ~31);
    for (int sb = pc.rb; sb < pc.re; sb += seg_rows) {
      const int se = min(pc.re, sb + seg_rows);
      if (sb > pc.rb) {
        __syncthreads();
        flush(true);
        use_atomics = true;
        __syncthreads();
        zero();
        __syncthreads();
      }
      auto rows = [&](auto main, auto extra, auto mask) {
        HistRows<A, W, kOrder, decltype(main)::value, decltype(extra)::value, kLine, decltype(mask)::value>(p, sb, se, g0, k, warp, lane, lane_word);
      };
      using std::false_type;
      using std::integral_constant;
      using mask           = integral_constant<bool, kFloat>;
      const int form_steps = form.main + form.extra;
      const bool no_mask   = !kFloat || p.F - g0 * kGroup >= kCols;  // (of 16 steps)
      if constexpr (W == 1) {
        if (form_steps == 16 && no_mask) rows(integral_constant<int, 16>{}, integral_constant<int, 0>{}, false_type{});
        else if (kFloat && form_steps == 16) rows(integral_constant<int, 16>{}, integral_constant<int, 0>{}, mask{});
        else if (form_steps == 8) rows(integral_constant<int, 8>{}, integral_constant<int, 0>{}, mask{});
        else rows(integral_constant<int, 4>{}, integral_constant<int, 0>{}, mask{});
      } else {
        if ((kLine && !kFloat) || (form_steps == 16 && no_mask)) rows(integral_constant<int, 8>{}, integral_constant<int, 8>{}, false_type{});
        else if (kFloat && form_steps == 16) rows(integral_constant<int, 8>{}, integral_constant<int, 8>{}, mask{});
        else if (!kFloat || form_steps == 12) rows(integral_constant<int, 8>{}, integral_constant<int, 4>{}, mask{});
        else if (form_steps == 10) rows(integral_constant<int, 8>{}, integral_constant<int, 2>{}, mask{});
        else if (form_steps == 9) rows(integral_constant<int, 8>{}, integral_constant<int, 1>{}, mask{});
        else if (form_steps == 8) rows(integral_constant<int, 8>{}, integral_constant<int, 0>{}, mask{});
        else if (form_steps == 4) rows(integral_constant<int, 4>{}, integral_constant<int, 0>{}, mask{});
        else rows(integral_constant<int, 2>{}, integral_constant<int, 0>{}, mask{});
      }
    }
    __syncthreads();
    if (!tree) {
      flush(use_atomics);
      return;
    }
    // merge tree
    const int GK          = GP * p.K;
    const int gk          = gp * p.K + k;
    const size_t stride   = static_cast<size_t>(hist_words) * 2;  // words per slot
    smem_t* slots         = static_cast<smem_t*>(p.partial);
    const int n4          = hist_words >> 2;
    int idx = pc.index, members = pc.pieces, soff = 0, coff = 0;
    long long image_rows = range_rows;  // rows an image of this tree level holds at most
    while (true) {
      const int n_groups = (members + kTreeFanIn - 1) / kTreeFanIn;
      const int grp      = idx / kTreeFanIn;
      const int gsize    = min(kTreeFanIn, members - grp * kTreeFanIn);
      // A node with more rows than 32-bit sums are safe for: its images are merged as far as they
      // stay below that count, and what is left (a handful instead of one per piece) is added into
      // the output with 64-bit atomics.  Every holder of an image of this level decides alike.
      if (min(static_cast<long long>(pc.node_rows), image_rows * kTreeFanIn) > cap_rows) {
        flush(true);
        return;
      }
      if (gsize > 1) {
        // leave my sums where the last one of the group finds them, then count myself in
        smem_t* mine = slots + (static_cast<size_t>(pc.tree_base + soff + idx) * GK + gk) * stride;
        for (int e4 = tid; e4 < n4; e4 += kThreads) {
          __stcg(reinterpret_cast<int4*>(mine) + e4, reinterpret_cast<const int4*>(hg)[e4]);
          __stcg(reinterpret_cast<int4*>(mine + hist_words) + e4, reinterpret_cast<const int4*>(hh)[e4]);
        }
        __threadfence();
        __syncthreads();
        if (tid == 0) {
          unsigned int* counter = p.arrive + static_cast<size_t>(pc.tree_base + coff + grp) * GK + gk;
          s_ticket              = atomicAdd(counter, 1u);
          if (s_ticket == static_cast<unsigned>(gsize - 1)) *counter = 0u;  // everybody has been: zero for the next launch
        }
        __syncthreads();
        const int arrived = static_cast<int>(s_ticket);
        if (arrived != gsize - 1) return;  // somebody else carries the group on
        __threadfence();
        for (int m = grp * kTreeFanIn; m < grp * kTreeFanIn + gsize; ++m) {
          if (m == idx) continue;
          const smem_t* other = slots + (static_cast<size_t>(pc.tree_base + soff + m) * GK + gk) * stride;
          for (int e4 = tid; e4 < n4; e4 += kThreads) {
            int4* mg = reinterpret_cast<int4*>(hg) + e4;
            int4* mh = reinterpret_cast<int4*>(hh) + e4;
            *mg = A::add4(*mg, __ldcg(reinterpret_cast<const int4*>(other) + e4));
            *mh = A::add4(*mh, __ldcg(reinterpret_cast<const int4*>(other + hist_words) + e4));
          }
        }
        __syncthreads();
      }
      if (n_groups == 1) break;  // this block holds the node's total
      soff += members;
      coff += n_groups;
      idx     = grp;
      members = n_groups;
      image_rows *= kTreeFanIn;
    }
    flush(false);
  };

  // The pieces of this block: the nodes its static range touches, or the chunks it draws as
  // tickets; one loop so that the piece code exists once.
  const int GK = GP * p.K;
  int gp = 0, k = 0, bj = 0;
  long long lo = 0, hi = 0;
  if (range_rows > 0) {
    // static ranges: block b = (range, group set, output)
    const int c = static_cast<int>(blockIdx.x) / GK;
    if (c >= pv.ranges) return;
    const int gk = static_cast<int>(blockIdx.x) - c * GK;
    gp = gk / p.K;
    k  = gk - gp * p.K;
    const long long all = pv.off[p.n_nodes];
    lo = static_cast<long long>(c) * range_rows;
    hi = lo + range_rows < all ? lo + range_rows : all;
    int a = 0, b = p.n_nodes;  // last node whose rows begin at or before lo
    while (b - a > 1) {
      const int m = (a + b) >> 1;
      if (pv.off[m] <= lo) a = m; else b = m;
    }
    bj = a;
  }
  const long long total = static_cast<long long>(pv.total_chunks) * GK;
  while (true) {
    Piece pc;
    if (range_rows > 0) {
      if (lo >= hi) break;
      const int c = static_cast<int>(blockIdx.x) / GK;
      while (pv.off[bj + 1] <= lo) ++bj;  // nodes without built rows
      const long long ws = pv.off[bj], we = pv.off[bj + 1];
      const long long pe = we < hi ? we : hi;
      const int first_c  = static_cast<int>(static_cast<unsigned>(ws) / range_rows);      // range that holds the node's first row
      const int last_c   = static_cast<int>(static_cast<unsigned>(we - 1) / range_rows);  // ... and its last one
      pc.j         = bj;
      pc.slot      = SlotOf(p, bj);
      pc.pieces    = last_c - first_c + 1;
      pc.index     = c - first_c;
      pc.tree_base = kTreeFanIn * first_c;  // the node owns the boundaries first_c+1 .. last_c
      pc.node_rows = static_cast<int>(we - ws);
      pc.rb        = p.seg_begin[bj] + static_cast<int>(lo - ws);
      pc.re        = p.seg_begin[bj] + static_cast<int>(pe - ws);
      lo           = pe;
    } else {
      __syncthreads();
      if (tid == 0) s_ticket = atomicAdd(p.ticket, 1u);
      __syncthreads();
      const long long t = s_ticket;
      if (t >= total) break;
      k  = static_cast<int>(t % p.K);
      gp = static_cast<int>((t / p.K) % GP);
      pc = DecodeChunk(p, pv.off, static_cast<int>(t / GK));
    }
    process(pc, gp, k);
  }
}

// Bins of one or two bytes, eight features per unit of work, many small blocks: the form for matrices of
// moderate size and for more than 256 bins per feature.
//
// k_hist_smem keeps 128 KB of histograms per block: clearing, turning and merging them costs 10 - 15 us per
// launch however few rows there are, and cutting a level into the pieces that fill the chip multiplies
// the 64-bit atomics of the merge.  Here a unit is (piece of a node, eight features, output) with
// kBins x 8 x 8 bytes of histograms (16 KB for 256 bins), once or four times; a level is cut into fewer pieces of
// rows because the feature groups fill the chip too (with four copies one piece per SM, TileChunkRows; two cost more
// atomics than they give, 200k x 50: 111 -> 132 us per tree).  A lane owns a row: one 8-byte (16-byte for
// two-byte bins) load brings its eight bin ids, in step j of eight it handles feature (j xor lane % 8).
// Piece sums go out with plain stores if the node is one piece, else with 64-bit atomics; the histogram
// is zeroed as it is read.
//
// Measured (B200, kernel time per level): 200k x 50, 256 bins: 23.3 us with one copy and 256 threads, 16.3 with four
// copies, pieces that fill the SMs once and 512 threads (256 threads: 25.3, 1024: 16.9); 300k x 37, 512 bins, 1024
// threads: 29 -> 22.7 us (64-bit global atomics at first: 267).  The sums of a piece added by whole sectors, and a plan
// without 64-bit divisions: 16.2 -> 14.6 us and 21.5 -> 18.1.
constexpr int kTileFeatures = 8;
constexpr int kTileMinRows  = 1024;
constexpr int kTileItemsPerSm = 1;

// kCopies: 1, or 4 copies of the histograms, one per eight lanes of a warp: the 32 lanes then update 32 different
// banks, where with one copy four lanes share eight banks and a reduction is three passes on average; but all copies
// are read and cleared for every piece.
template <typename BinT, int kBins, int kThreads, int kCopies>
__global__ void __launch_bounds__(kThreads, kThreads == 256 ? 6 : 1)
  k_hist_tile(const HistParams p)
{
  AfterTheKernelBefore();
  using A = Acc<false>;
  constexpr int kRow = kTileFeatures * kCopies;  // words of a bin
  extern __shared__ __align__(128) int s_hist[];  // [2][kBins][copies][8]
  __shared__ int32_t s_off[kPlanNodes + 1];
  __shared__ int s_tmp[32];
  __shared__ GPairI64* s_base[kTileFeatures];
  __shared__ int s_nb[kTileFeatures];
  constexpr int kWarps = kThreads / 32;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int FG  = (p.F + kTileFeatures - 1) / kTileFeatures, Q = FG * p.K;
  PlanView pv;
  if (p.plan == nullptr) {
    pv = PlanInside<kThreads, kCopies != 1>(p, Q, p.tile_items, kTileMinRows, false, s_off, s_tmp);
  } else {
    pv.rows_safe    = p.plan[3];
    pv.total_chunks = p.plan[1];
    pv.off          = p.chunk_off;
  }
  const int mb        = p.mb_ptr != nullptr ? min(p.mb, *p.mb_ptr) : p.mb;
  const int words     = mb * kTileFeatures;  // of a histogram, copies added up
  const int64_t pitch = static_cast<int64_t>(p.G) * kGroup;
  const int2* gpair   = static_cast<const int2*>(p.gpair);
  const bool by_pos   = p.pairs_by_position != 0 || p.row_index == nullptr;
  for (int i = tid; i < mb * kRow / 4; i += kThreads)
    reinterpret_cast<int4*>(s_hist)[i] = reinterpret_cast<int4*>(s_hist + kBins * kRow)[i] = make_int4(0, 0, 0, 0);
  const unsigned lane_word = SmemAddr(s_hist) + (lane & (kRow - 1)) * 4;
  const unsigned swap = lane & 7, bsel = swap & 3;
  // one-byte ids: step j reads byte j of the pair of words permuted by `swap`; two-byte ids likewise
  const unsigned perm = bsel == 0 ? 0x3210u : bsel == 1 ? 0x2301u : bsel == 2 ? 0x1032u : 0x0123u;
  const unsigned sel0 = perm + ((swap & 4) ? 0x4444u : 0u), sel1 = perm + ((swap & 4) ? 0u : 0x4444u);

  const long long total = static_cast<long long>(pv.total_chunks) * Q;
  for (long long t = blockIdx.x; t < total; t += gridDim.x) {
    const int chunk = total < (1ll << 31) ? static_cast<int>(static_cast<unsigned>(t) / static_cast<unsigned>(Q)) : static_cast<int>(t / Q);
    const int qk    = static_cast<int>(t - static_cast<long long>(chunk) * Q);
    const int fg    = p.K == 1 ? qk : qk / p.K, k = qk - fg * p.K;
    const Piece pc  = DecodeChunk(p, pv.off, chunk);
    const int f0    = fg * kTileFeatures;
    const int seg  = pc.slot * p.K + k;
    if (pv.rows_safe < 64) {
      // (magnitudes so uneven that 32-bit sums of 64 rows may overflow: straight to 64-bit atomics)
      const int f = f0 + (lane & 7);
      if (f < p.F) {
        GPairI64* obase = FeatureBase<GPairI64>(p, f, seg);
        for (int r = pc.rb + warp * 4 + (lane >> 3); r < pc.re; r += kWarps * 4) {
          const int rid = p.row_index != nullptr ? p.row_index[r] : r;
          const int2 v  = gpair[static_cast<int64_t>(by_pos ? r : rid) * p.K + k];
          A::add_global(obase + static_cast<const BinT*>(p.bins)[rid * pitch + f], v.x, v.y);
        }
      }
      continue;
    }
    __syncthreads();  // the histogram is zero again, s_base is free
    if (tid < kTileFeatures) {
      const int f = f0 + tid;
      s_nb[tid]   = f < p.F ? p.row_ptr[f + 1] - p.row_ptr[f] : 0;
      s_base[tid] = f < p.F ? FeatureBase<GPairI64>(p, f, seg) : nullptr;
    }
    const BinT* col = static_cast<const BinT*>(p.bins) + f0;
    struct Row {
      uint4 w;
      int2 v;
    };
    auto rid_at = [&](int r) -> int { return p.row_index != nullptr ? __ldcg(p.row_index + r) : r; };
    auto load   = [&](int rid, int r) -> Row {
      Row x;
      const BinT* a = col + rid * pitch;
      if (sizeof(BinT) == 1) {
        const uint2 u = __ldg(reinterpret_cast<const uint2*>(a));
        x.w           = make_uint4(u.x, u.y, 0u, 0u);
      } else {
        x.w = __ldg(reinterpret_cast<const uint4*>(a));
      }
      x.v = __ldcg(gpair + static_cast<int64_t>(by_pos ? r : rid) * p.K + k);
      return x;
    };
    auto consume = [&](const Row& x) {
      unsigned bin[8];
      if (sizeof(BinT) == 1) {
        const unsigned a = __byte_perm(x.w.x, x.w.y, sel0), b = __byte_perm(x.w.x, x.w.y, sel1);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          bin[j]     = __byte_perm(a, 0u, 0x4440u | j);
          bin[4 + j] = __byte_perm(b, 0u, 0x4440u | j);
        }
      } else {
        // halves (bit 0 of swap) inside a word, then words (bits 1 and 2)
        const unsigned hs = (swap & 1) ? 0x1032u : 0x3210u;
        unsigned w0 = __byte_perm(x.w.x, 0u, hs), w1 = __byte_perm(x.w.y, 0u, hs);
        unsigned w2 = __byte_perm(x.w.z, 0u, hs), w3 = __byte_perm(x.w.w, 0u, hs);
        const unsigned a0 = (swap & 2) ? w1 : w0, a1 = (swap & 2) ? w0 : w1;
        const unsigned a2 = (swap & 2) ? w3 : w2, a3 = (swap & 2) ? w2 : w3;
        w0 = (swap & 4) ? a2 : a0;
        w1 = (swap & 4) ? a3 : a1;
        w2 = (swap & 4) ? a0 : a2;
        w3 = (swap & 4) ? a1 : a3;
        const unsigned w[4] = {w0, w1, w2, w3};
#pragma unroll
        for (int j = 0; j < 8; ++j)  // (an id beyond the caller's bound must not leave the array)
          bin[j] = min((j & 1) ? w[j >> 1] >> 16 : w[j >> 1] & 0xffffu, static_cast<unsigned>(kBins - 1));
      }
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const unsigned addr = (lane_word ^ (4u * j)) + bin[j] * (kRow * 4);
        A::red_shared(addr, x.v.x);
        A::template red_shared_at<kBins * kRow * 4>(addr, x.v.y);
      }
    };
    bool atomics = pc.pieces > 1;
    for (int sb = pc.rb; sb < pc.re; sb += pv.rows_safe) {
      const int se = pc.re - sb > pv.rows_safe ? sb + pv.rows_safe : pc.re;
      if (se < pc.re) atomics = true;
      __syncthreads();
      // the rows of the warp: two batches in flight, row ids one batch further ahead
      const int step = kThreads, last = se - 1;
      int r = sb + tid;
      Row x{}, y{};
      int rn = 0;
      if (sb + warp * 32 < se) {
        x  = load(rid_at(min(r, last)), min(r, last));
        rn = rid_at(min(r + step, last));
      }
      for (int b = sb + warp * 32; b < se; b += step) {
        const int nr = min(r + step, last);
        y  = load(rn, nr);
        rn = rid_at(min(r + 2 * step, last));
        if (r >= se) x.v = make_int2(0, 0);
        consume(x);
        x = y;
        r += step;
      }
      __syncthreads();
      for (int i0 = warp * 32; i0 < words; i0 += kThreads) {
        const int i = i0 + lane, f = i & 7, bin = i >> 3;
        int g = 0, h = 0;
        if (i < words) {
#pragma unroll
          for (int c = 0; c < kCopies; ++c) {  // (neighbouring bins begin with different copies: other banks)
            int* at = s_hist + bin * kRow + ((c + bin) & (kCopies - 1)) * kTileFeatures + f;
            g += at[0];
            h += at[kBins * kRow];
            at[0] = at[kBins * kRow] = 0;
          }
        }
        if (!atomics) {
          if ((g | h) != 0 && bin < s_nb[f]) A::store_global(s_base[f] + bin, g, h);
          continue;
        }
        // whole sectors, as in k_hist_smem: an instruction adds the pairs of four bins of four features
#pragma unroll
        for (int part = 0; part < 2; ++part) {
          const int from = (((lane >> 1) & 3) << 3) | (part * 4 + (lane >> 3));
          const int vg = __shfl_sync(0xffffffffu, g, from), vh = __shfl_sync(0xffffffffu, h, from);
          const int v = (lane & 1) ? vh : vg, ff = from & 7, b = (i0 >> 3) + (from >> 3);
          if (v != 0 && b < s_nb[ff]) A::add_word(s_base[ff] + b, lane & 1, v);
        }
      }
      if (pc.re - sb <= pv.rows_safe) break;  // (sb + rows_safe may not fit 32 bits)
    }
  }
}

// ---- row grouping (utility for the stage-level API) -------------------------------------------
constexpr int kGroupTile = 4096;

// Kernel, dynamic shared memory and persistent grid (resident blocks of the whole device, from the
// occupancy calculator) for one combination of bin width, pair type and path.
struct HistLaunch {
  void (*fn)(HistParams);
  size_t smem;
  int threads;
  int grid;
  int width;  // feature groups per unit of work
  bool smem_path;  // k_hist_smem
  bool tile;       // k_hist_tile
  int copies = 1;  // of its histograms
};

// Which one-byte matrices take the tile form: its fixed cost is smaller, and its gathers take more passes per update
// (eight bin bytes per line instead of 64).  Up to kTileMaxCellsFew cells (rows x features x outputs), and with one
// output, one rank (the atomics of a node's pieces would cross NVLink) and few units of (node, eight features) up
// to kTileMaxCells.  Kernel time per tree of depth 7, tile form and k_hist_smem: 300k x 64: 136 and 235 us, 600k x 64:
// 211 and 315, 400k x 128: 296 and 380, 2M x 20: 290 and 296, 1.2M x 64: 424 and 408; ten outputs, 60k x 50: 274 and
// 264, 100k x 100: 608 and 479.  A unit's histograms are read and cleared whatever they hold: 200k x 200, 256
// nodes: 281 us and 197, 32 nodes: 76 and 65; hence also not many units with rows in them: 60k x 256, 8 nodes: 51 and
// 43, 64 nodes: 70 and 54 (but 15k x 256, 64 nodes, 234 rows each: 47 and 47; 30k x 200, 256 nodes: 127 and 251).
// These points are all there is: the lines between them follow the points, not a model of the two kernels' costs, and a
// shape far from all of them may lie on the wrong side.
//
// Its wide accesses need the bins and the histograms on 16-byte boundaries (`aligned`); arrays that are not go to the
// kernels that take them as they are.
//
// Four copies pay where a level is cut into about one piece per SM (no more units than SMs) and has something to
// add: 200k x 40, one node: 33 -> 24 us; 30k x 40, 32 nodes (160 units) would be 19 -> 23 us, 30k x 200, 256 nodes 127
// -> 215, 5k x 40, one node 17.2 -> 18.7.
constexpr int64_t kCopiesMinCells = 1 << 20;
constexpr int64_t kTileMaxCells = 3 << 24, kTileMaxCellsFew = 1 << 24, kTileMaxCellsMany = 1 << 23;

RowOrder OrderOf(const HistParams& p)
{
  return p.row_index == nullptr ? kRowsInOrder : p.pairs_by_position != 0 ? kPairsByPosition : kPairsByRow;
}

template <bool kFloat, int W, bool kLine>
void (*SmemKernel(RowOrder order))(HistParams)
{
  return order == kPairsByRow         ? k_hist_smem<kFloat, W, kPairsByRow, kLine>
         : order == kPairsByPosition ? k_hist_smem<kFloat, W, kPairsByPosition, kLine>
                                     : k_hist_smem<kFloat, W, kRowsInOrder, kLine>;
}
template <bool kFloat>
void (*SmemKernel(int n_groups, RowOrder order))(HistParams)
{
  return n_groups > 2 ? SmemKernel<kFloat, 2, true>(order) : n_groups == 2 ? SmemKernel<kFloat, 2, false>(order) : SmemKernel<kFloat, 1, false>(order);
}

HistLaunch PickHistKernel(int bin_bytes, int mb, bool float_mode, RowOrder order, int F, int K, int64_t n_rows, int n_nodes, bool derive, int sm_count, int ranks, bool aligned)
{
  const int n_groups = (F + kGroup - 1) / kGroup;
  const int n_slots   = derive ? n_nodes / 2 : n_nodes;
  const int64_t cells = n_rows * F * K, units = static_cast<int64_t>(n_slots) * ((F + kTileFeatures - 1) / kTileFeatures) * K;
  const bool many     = units > sm_count && (derive ? cells / 2 : cells) >= kTileMaxCellsMany && n_rows >= int64_t{512} * n_nodes;
  HistLaunch h;
  h.smem_path = bin_bytes == 1 && mb <= kSmemBins;
  h.tile      = !float_mode && aligned && mb <= 2048 && (bin_bytes == 2 || (h.smem_path && ((cells <= kTileMaxCellsFew && !many) ||
                                                   (K == 1 && ranks <= 1 && cells <= kTileMaxCells && units <= 2 * sm_count))));
  h.width     = h.smem_path && n_groups >= 2 ? 2 : 1;
  h.threads   = kHistThreads * h.width;
  h.smem      = 0;
  if (h.tile) {
    h.smem_path    = false;
    h.width        = 1;
    const int bins = mb <= 256 ? 256 : mb <= 512 ? 512 : mb <= 1024 ? 1024 : 2048;
    h.copies  = bins <= 512 && cells >= kCopiesMinCells && (units <= sm_count || (bin_bytes == 1 && cells > kTileMaxCellsFew)) ? 4 : 1;
    h.threads = bins > 256 ? 1024 : h.copies == 4 ? 512 : 256;
    h.smem    = static_cast<size_t>(bins) * kTileFeatures * h.copies * 8;
    if (bin_bytes == 1) h.fn = h.copies == 4 ? k_hist_tile<uint8_t, 256, 512, 4> : k_hist_tile<uint8_t, 256, 256, 1>;
    else if (bins == 256) h.fn = h.copies == 4 ? k_hist_tile<uint16_t, 256, 512, 4> : k_hist_tile<uint16_t, 256, 256, 1>;
    else if (bins == 512) h.fn = h.copies == 4 ? k_hist_tile<uint16_t, 512, 1024, 4> : k_hist_tile<uint16_t, 512, 1024, 1>;
    else if (bins == 1024) h.fn = k_hist_tile<uint16_t, 1024, 1024, 1>;
    else h.fn = k_hist_tile<uint16_t, 2048, 1024, 1>;
  } else if (h.smem_path) {
    h.smem = HistSmemBytes(h.width);
    h.fn   = float_mode ? SmemKernel<true>(n_groups, order) : SmemKernel<false>(n_groups, order);
  } else if (bin_bytes == 1) {
    h.fn = float_mode ? k_hist_direct<uint8_t, true> : k_hist_direct<uint8_t, false>;
  } else {
    h.fn = float_mode ? k_hist_direct<uint16_t, true> : k_hist_direct<uint16_t, false>;
  }
  if (h.smem > 32 * 1024)
    LBK_CUDA(cudaFuncSetAttribute(h.fn, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(h.smem)));
  int per_sm = 0;
  LBK_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, h.fn, h.threads, h.smem));
  if (per_sm < 1) per_sm = 1;
  if (!h.smem_path && !h.tile && per_sm > 4) per_sm = 4;
  h.grid = sm_count * per_sm;
  return h;
}

__global__ void k_group_count(const int32_t* __restrict__ node_of_row, int64_t n_rows, int node_begin, int n_nodes,
                              int32_t* __restrict__ counts /* [blocks][n_nodes] */)
{
  extern __shared__ int cnt[];
  for (int i = threadIdx.x; i < n_nodes; i += blockDim.x) cnt[i] = 0;
  __syncthreads();
  const int64_t base = static_cast<int64_t>(blockIdx.x) * kGroupTile;
  for (int i = threadIdx.x; i < kGroupTile; i += blockDim.x) {
    const int64_t r = base + i;
    if (r < n_rows) {
      const int nd = node_of_row[r] - node_begin;
      if (nd >= 0 && nd < n_nodes) atomicAdd(&cnt[nd], 1);
    }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < n_nodes; i += blockDim.x)
    counts[static_cast<int64_t>(blockIdx.x) * n_nodes + i] = cnt[i];
}

// counts[b][nd] -> exclusive offset of (nd, b) in node-major order; seg[nd] = start of node nd
__global__ void k_group_scan(int32_t* __restrict__ counts, int n_blocks, int n_nodes, int32_t* __restrict__ seg)
{
  // one thread per node sums its column, then a serial scan over nodes by thread 0
  extern __shared__ int tot[];
  for (int nd = threadIdx.x; nd < n_nodes; nd += blockDim.x) {
    int s = 0;
    for (int b = 0; b < n_blocks; ++b) s += counts[static_cast<int64_t>(b) * n_nodes + nd];
    tot[nd] = s;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    int run = 0;
    for (int nd = 0; nd < n_nodes; ++nd) {
      seg[nd] = run;
      run += tot[nd];
    }
    seg[n_nodes] = run;
  }
  __syncthreads();
  for (int nd = threadIdx.x; nd < n_nodes; nd += blockDim.x) {
    int run = seg[nd];
    for (int b = 0; b < n_blocks; ++b) {
      const int c = counts[static_cast<int64_t>(b) * n_nodes + nd];
      counts[static_cast<int64_t>(b) * n_nodes + nd] = run;
      run += c;
    }
  }
}

// one warp per tile walks its rows in order so that rows keep their relative order inside a node
__global__ void k_group_scatter(const int32_t* __restrict__ node_of_row, int64_t n_rows, int node_begin, int n_nodes,
                                const int32_t* __restrict__ offsets, int32_t* __restrict__ row_index)
{
  extern __shared__ int cur[];
  const int lane = threadIdx.x;
  for (int i = lane; i < n_nodes; i += 32) cur[i] = offsets[static_cast<int64_t>(blockIdx.x) * n_nodes + i];
  __syncwarp();
  const int64_t base = static_cast<int64_t>(blockIdx.x) * kGroupTile;
  for (int i = 0; i < kGroupTile; i += 32) {
    const int64_t r = base + i + lane;
    int nd          = -1;
    if (r < n_rows) {
      nd = node_of_row[r] - node_begin;
      if (nd < 0 || nd >= n_nodes) nd = -1;
    }
    const unsigned peers = __match_any_sync(0xffffffffu, nd);
    const int rank       = __popc(peers & ((1u << lane) - 1u));
    int start            = 0;
    if (nd >= 0) start = cur[nd];
    __syncwarp();
    if (nd >= 0) {
      row_index[start + rank] = static_cast<int32_t>(r);
      if (rank == __popc(peers) - 1) cur[nd] = start + rank + 1;
    }
    __syncwarp();
  }
}

}  // namespace

void HistScratchNeeds(lbk_context* ctx, int F, int K, int bin_bytes, int mb, int64_t n_rows, HistScratch& need)
{
  // what k_hist_smem needs, where some level may take it
  if (ctx->n_ranks <= 1 || bin_bytes != 1 || mb > kSmemBins || n_rows * F * K < kTileMaxCellsMany) return;
  constexpr int64_t kManyRows = int64_t{1} << 36;  // (beyond every bound of the tile form)
  const HistLaunch hl = PickHistKernel(bin_bytes, mb, false, kPairsByPosition, F, K, kManyRows, 1, false, ctx->sm_count, ctx->n_ranks, true);
  need.n_arrive       = kTreeFanIn * hl.grid;
  need.partial_bytes  = static_cast<size_t>(need.n_arrive) * mb * kGroup * hl.width * 8;
}

void BuildHistogram(lbk_context* ctx, Scratch& s, const HistLevel& lv, cudaStream_t stream)
{
  if (lv.n_nodes <= 0) return;
  HistParams p;
  p.bins         = lv.bins;
  p.n_rows       = lv.n_rows;
  p.F            = lv.F;
  p.K            = lv.K;
  p.B            = lv.B;
  p.G            = (lv.F + kGroup - 1) / kGroup;
  p.row_ptr      = lv.row_ptr;
  p.gpair        = lv.float_mode ? static_cast<const void*>(lv.gpair_f) : static_cast<const void*>(lv.gpair);
  p.row_index    = lv.row_index;
  p.seg_begin    = lv.seg_begin;
  p.seg_end      = lv.seg_end;
  p.node_sums    = lv.node_sums;
  p.node_begin   = lv.node_begin;
  p.build_all    = lv.build_all;
  p.n_nodes      = lv.n_nodes;
  p.status       = ctx->d_status;
  p.pairs_by_position = lv.pairs_by_position ? 1 : 0;
  p.out              = lv.out;
  p.push_recv        = lv.push_recv;
  p.push_rank        = ctx->rank;
  p.push_ranks       = ctx->n_ranks;
  p.push_slot_pairs  = lv.push_slot_pairs;
  p.push_len         = lv.push_len;
  p.mb               = lv.max_bins_per_feature;
  p.mb_ptr           = lv.max_bins_ptr;
  const HistLaunch hl = PickHistKernel(lv.bin_bytes, p.mb, lv.float_mode, OrderOf(p), p.F, p.K, lv.n_rows, p.n_nodes, p.node_sums != nullptr, ctx->sm_count, ctx->n_ranks,
                                       Aligned16(p.bins) && Aligned16(p.out));

  const int* max_abs = lv.max_abs;
  if (!lv.float_mode && max_abs == nullptr) {
    // the caller gave quantised pairs without their largest magnitude: find it
    int* m = s.alloc<int>(2);
    LBK_CUDA(cudaMemsetAsync(m, 0, 2 * sizeof(int), stream));
    const int64_t n = lv.n_rows * lv.K;
    if (n > 0) {
      LaunchChained(k_max_abs, ctx->sm_count * 8, 256, 0, stream, lv.gpair, n, m);
      LBK_LAUNCH_CHECK();
    }
    max_abs = m;
  }
  p.max_abs = lv.float_mode ? nullptr : max_abs;
  p.tile_items = ctx->sm_count * kTileItemsPerSm;
  // histograms that go to other ranks' memory: slots and counters for the merge trees of the nodes that reach over a
  // range boundary, kTreeFanIn per resident block covers every cut
  HistScratch own;
  HistScratch* hs = lv.scratch;
  const int need_arrive  = hl.smem_path && (p.push_recv != nullptr || lv.merge_tree) ? kTreeFanIn * hl.grid : 0;
  const size_t need_bytes = static_cast<size_t>(need_arrive) * p.mb * kGroup * hl.width * 8;
  const bool kept = hs != nullptr && hs->next_ticket < hs->n_tickets && hs->n_arrive >= need_arrive && hs->partial_bytes >= need_bytes;
  if (!kept) hs = &own;
  p.arrive = nullptr;
  p.partial = nullptr;
  p.slot_capacity = 0;
  p.n_arrive = 0;
  p.ranges   = hl.smem_path;
  if (need_arrive > 0) {
    p.n_arrive      = need_arrive;
    p.slot_capacity = need_arrive;
    if (!kept) {
      own.arrive  = s.alloc<unsigned int>(static_cast<size_t>(need_arrive));
      own.partial = s.alloc<unsigned char>(need_bytes);
    }
    p.arrive  = hs->arrive;
    p.partial = hs->partial;
  }
  p.plan      = nullptr;
  p.chunk_off = nullptr;
  p.wpre      = nullptr;
  // a plan of its own launch: levels of many nodes, the kernels that do not plan, and calls whose counters
  // have to be zeroed
  if (!kept || lv.n_nodes > kPlanNodes || !(hl.smem_path || hl.tile)) {
    const int units = (hl.tile ? (p.F + kTileFeatures - 1) / kTileFeatures : (p.G + hl.width - 1) / hl.width) * p.K;
    int32_t* chunk_off = s.alloc<int32_t>(static_cast<size_t>(lv.n_nodes) + 1);
    int32_t* wpre      = hl.smem_path ? s.alloc<int32_t>(static_cast<size_t>(lv.n_nodes) + 1) : nullptr;
    int32_t* plan      = s.alloc<int32_t>(8);
    p.ticket           = reinterpret_cast<unsigned int*>(plan + 2);
    LaunchChained(k_hist_plan, 1, 1024, 0, stream, p, units, hl.tile ? p.tile_items : hl.grid, hl.tile ? kTileMinRows : kMinChunk, hl.copies != 1, chunk_off, wpre, plan);
    LBK_LAUNCH_CHECK();
    p.chunk_off = chunk_off;
    p.wpre      = wpre;
    p.plan      = plan;
  } else {
    p.ticket = hs->tickets + hs->next_ticket++;
  }
  std::pair<cudaEvent_t, cudaEvent_t> ev{nullptr, nullptr};
  if (ctx->profile) {
    ev = NextProfileEvents(ctx);
    LBK_CUDA(cudaEventRecord(ev.first, stream));
  }
  LaunchChained(hl.fn, hl.grid, hl.threads, hl.smem, stream, p);
  if (ctx->profile) LBK_CUDA(cudaEventRecord(ev.second, stream));
  // stream ordered: the slots go back to the pool once the kernel has run
  if (own.partial) s.free_one(own.partial);
}

void* BuildHistogramSummed(lbk_context* ctx, Scratch& s, const HistLevel& lv, int n_slots, HistSum mode,
                           bool result_in_out, bool zero_out, cudaStream_t stream)
{
  const size_t slot_words = static_cast<size_t>(lv.K) * lv.B * 2;  // 64-bit words per slot
  const size_t bytes      = static_cast<size_t>(n_slots) * slot_words * 8;
  if (ctx->n_ranks <= 1) {
    if (zero_out) LBK_CUDA(cudaMemsetAsync(lv.out, 0, bytes, stream));
    if (lv.n_rows > 0) BuildHistogram(ctx, s, lv, stream);
    return lv.out;
  }
  // every decision below depends only on what is equal on every rank (the shapes, the kind of
  // communicator, the collective answer of EnsureExchange): all ranks issue the same collectives
  // The owned sums by push: every rank's kernel stores the histogram of a feature straight into
  // the owner's receive slot while it runs, a barrier, then the owner adds up its slots locally.
  // The receive buffers hold ranks x segments x (a bound of the owned bins): where the features'
  // bin counts are so uneven that the bound is far above the real size, the pull form below is used.
  if (mode == HistSum::kSumOwned) {
    const int R          = ctx->n_ranks;
    const long long fo   = (lv.F + R - 1) / R;  // features of the largest owner
    long long push_len   = fo * (lv.max_bins_per_feature > 0 ? lv.max_bins_per_feature : lv.B);
    if (push_len > lv.B) push_len = lv.B;
    const int n_seg      = n_slots * lv.K;
    const size_t push_bytes = static_cast<size_t>(R) * n_seg * static_cast<size_t>(push_len) * 16;
    if (push_bytes <= 2 * bytes + (size_t{1} << 20) && EnsureExchange(ctx, push_bytes, stream)) {
      void* dst = lv.out;  // every owned bin is written below; the others are not touched
      HistLevel sub       = lv;
      sub.push_recv       = NextPushBuffers(ctx, stream);
      sub.push_slot_pairs = static_cast<long long>(n_seg) * push_len;
      sub.push_len        = static_cast<int>(push_len);
      if (lv.n_rows > 0) BuildHistogram(ctx, s, sub, stream);
      ExchangeReducePushed(ctx, dst, n_seg, static_cast<int>(push_len), lv.B, lv.F, lv.row_ptr, lv.float_mode, stream);
      return dst;
    }
  }
  if (EnsureExchange(ctx, bytes, stream)) {
    void* buf = NextExchangeBuffer(ctx, bytes, stream);
    HistLevel sub = lv;
    sub.out       = buf;
    if (lv.n_rows > 0) BuildHistogram(ctx, s, sub, stream);
    const int n_seg = n_slots * lv.K;
    if (mode == HistSum::kSumOwned) {
      void* dst = result_in_out ? lv.out : buf;
      ExchangeReduceOwned(ctx, buf, dst, n_seg, lv.B, lv.F, lv.row_ptr, lv.float_mode, stream);
      return dst;
    }
    ExchangeReduceOwned(ctx, buf, buf, n_seg, lv.B, lv.F, lv.row_ptr, lv.float_mode, stream);
    ExchangeGatherAll(ctx, buf, lv.out, n_seg, lv.B, lv.F, lv.row_ptr, stream);
    return lv.out;
  }
  if (zero_out) LBK_CUDA(cudaMemsetAsync(lv.out, 0, bytes, stream));
  if (lv.n_rows > 0) BuildHistogram(ctx, s, lv, stream);
  AllReduce(ctx, lv.out, static_cast<size_t>(n_slots) * slot_words, lv.float_mode ? LBK_F64 : LBK_I64, LBK_SUM, stream);
  return lv.out;
}

void GroupRows(lbk_context* ctx, Scratch& s, const int32_t* node_of_row, int64_t n_rows, int node_begin,
               int n_nodes, int32_t* row_index, int32_t* seg, cudaStream_t stream)
{
  LBK_EXPECT(n_nodes >= 1 && n_nodes <= 8192, "group_rows supports 1..8192 nodes");
  const int64_t n_blocks = (n_rows + kGroupTile - 1) / kGroupTile;
  if (n_blocks == 0) {
    LBK_CUDA(cudaMemsetAsync(seg, 0, sizeof(int32_t) * (n_nodes + 1), stream));
    return;
  }
  int32_t* counts   = s.alloc<int32_t>(static_cast<size_t>(n_blocks) * n_nodes);
  const size_t smem = sizeof(int) * n_nodes;
  k_group_count<<<static_cast<unsigned>(n_blocks), 256, smem, stream>>>(node_of_row, n_rows, node_begin, n_nodes, counts);
  LBK_LAUNCH_CHECK();
  k_group_scan<<<1, 1024, smem, stream>>>(counts, static_cast<int>(n_blocks), n_nodes, seg);
  LBK_LAUNCH_CHECK();
  k_group_scatter<<<static_cast<unsigned>(n_blocks), 32, smem, stream>>>(node_of_row, n_rows, node_begin, n_nodes, counts,
                                                                         row_index);
  LBK_LAUNCH_CHECK();
  (void)ctx;
}

}  // namespace lbk

// ---------------------------------------------------------------------------------------------
// lbk_histogram_noalloc: the histogram build for callers that must not allocate device memory.
//
// Who needs it: code that runs under a memory budget that a runtime has already handed out
// completely (a task variant registered without the right to allocate: any cudaMalloc there fails or
// takes memory the runtime believes it owns), or a process that wants its device footprint fixed
// after start-up so that no later call can fail for lack of memory.  lbk_histogram takes its
// per-call scratch (chunk offsets, the level plan, the largest magnitudes) from the context's
// pool; this entry point keeps that scratch in a fixed array inside the library image instead
// and needs no context at all.
//
// Limits and rules
//   * at most LBK_NOALLOC_MAX_NODES nodes and LBK_NOALLOC_MAX_FEATURES features per call,
//     device pointers only (host_buffers must be 0), one rank (all_reduce must be 0: there is no
//     context and so no communicator); larger or other calls are rejected with LBK_ERR_ARGUMENT
//     before anything is launched;
//   * the array (about 16 KB) exists once per GPU that loads the library, until the process ends;
//   * the first call on a device looks the array's device address up (the array's name is only a
//     host-side handle; kernels get the address found here).  Make that first call before any
//     stream capture begins;
//   * the call blocks: it reads row_ptr back and synchronises `stream` before it returns (so it is
//     not something to issue from a host callback of a stream); it makes `device` current for the
//     duration of the call and restores the caller's device before it returns;
//   * all calls on a device share the array: what has to start at zero is cleared by each call, and
//     two calls whose kernels overlap on the GPU (different streams, different threads) race -
//     serialise them on one stream.
namespace lbk {
namespace {

constexpr int kNoAllocMaxNodes    = LBK_NOALLOC_MAX_NODES;
constexpr int kNoAllocMaxFeatures = LBK_NOALLOC_MAX_FEATURES;
constexpr int kNoAllocPlanOffset  = kNoAllocMaxNodes + 4;   // chunk offsets first, then plan[8], max_abs[2]
constexpr int kNoAllocInts        = kNoAllocPlanOffset + 12;

static __device__ __align__(256) int32_t g_hist_scratch[kNoAllocInts];

constexpr int kMaxDevices = 64;
std::mutex g_scratch_mutex;
int32_t* g_scratch_addr[kMaxDevices] = {};

// Device address of the scratch array on `device`, which must be the current device.
int32_t* HistScratchAddress(int device)
{
  std::lock_guard<std::mutex> lock(g_scratch_mutex);
  if (g_scratch_addr[device] == nullptr) {
    void* ptr = nullptr;
    LBK_CUDA(cudaGetSymbolAddress(&ptr, g_hist_scratch));
    g_scratch_addr[device] = static_cast<int32_t*>(ptr);
  }
  return g_scratch_addr[device];
}

}  // namespace
}  // namespace lbk

extern "C" int lbk_histogram_noalloc(int device, const lbk_histogram_args* a)
{
  using namespace lbk;
  return Guard(nullptr, [&] {
    LBK_EXPECT(a != nullptr, "null argument");
    LBK_EXPECT(device >= 0 && device < kMaxDevices, "device index out of range");
    LBK_EXPECT(a->host_buffers == 0, "lbk_histogram_noalloc takes device pointers only");
    LBK_EXPECT(a->all_reduce == 0, "lbk_histogram_noalloc has no communicator: all_reduce must be 0");
    LBK_EXPECT(!a->pairs_by_position || a->mode == 1 || a->max_abs != nullptr,
               "pairs stored by position need max_abs (the library cannot know how many entries the array has)");
    LBK_EXPECT(a->bins && a->row_ptr && a->row_index && a->seg && a->hist, "null argument");
    LBK_EXPECT(a->mode == 0 || a->mode == 1, "mode must be 0 or 1");
    LBK_EXPECT(a->mode == 0 ? a->gpair != nullptr : a->gpair_f32 != nullptr, "missing gradient pairs");
    LBK_EXPECT(a->bin_bytes == 1 || a->bin_bytes == 2, "bin_bytes must be 1 or 2");
    LBK_EXPECT(a->n_features >= 1 && a->n_outputs >= 1 && a->total_bins >= a->n_features, "bad shape");
    LBK_EXPECT(a->n_nodes >= 1 && a->n_nodes <= kNoAllocMaxNodes,
               "lbk_histogram_noalloc handles at most " + std::to_string(kNoAllocMaxNodes) + " nodes per call");
    LBK_EXPECT(a->n_features <= kNoAllocMaxFeatures,
               "lbk_histogram_noalloc handles at most " + std::to_string(kNoAllocMaxFeatures) + " features per call");
    int caller_device = -1;
    LBK_CUDA(cudaGetDevice(&caller_device));
    struct RestoreDevice {
      int d;
      ~RestoreDevice() { cudaSetDevice(d); }
    } restore{caller_device};
    LBK_CUDA(cudaSetDevice(device));
    cudaStream_t stream = static_cast<cudaStream_t>(a->stream);
    int32_t* scratch    = HistScratchAddress(device);
    int32_t* chunk_off  = scratch;
    int32_t* plan       = scratch + kNoAllocPlanOffset;
    int* max_abs        = reinterpret_cast<int*>(plan + 8);

    const int F = a->n_features, K = a->n_outputs, B = a->total_bins;
    int32_t rp[kNoAllocMaxFeatures + 1];
    LBK_CUDA(cudaMemcpyAsync(rp, a->row_ptr, sizeof(int32_t) * (F + 1), cudaMemcpyDeviceToHost, stream));
    LBK_CUDA(cudaStreamSynchronize(stream));
    LBK_EXPECT(rp[F] == B, "total_bins does not match row_ptr");
    int mb = 1;  // (max_bins is not needed here: row_ptr has been read back anyway)
    for (int f = 0; f < F; ++f) mb = rp[f + 1] - rp[f] > mb ? rp[f + 1] - rp[f] : mb;
    LBK_EXPECT(a->bin_bytes == 2 || mb <= 256, "one-byte bins need <= 256 proposals per feature");

    int sm_count = 0;
    LBK_CUDA(cudaDeviceGetAttribute(&sm_count, cudaDevAttrMultiProcessorCount, device));

    const bool float_mode = a->mode == 1;
    HistParams p;
    p.bins         = a->bins;
    p.n_rows       = a->n_rows;
    p.F            = F;
    p.K            = K;
    p.B            = B;
    p.G            = (F + kGroup - 1) / kGroup;
    p.row_ptr      = a->row_ptr;
    p.gpair        = float_mode ? static_cast<const void*>(a->gpair_f32) : static_cast<const void*>(a->gpair);
    p.row_index    = a->row_index;
    p.seg_begin    = a->seg;
    p.seg_end      = a->seg + 1;
    p.node_sums    = nullptr;
    p.node_begin   = 0;
    p.build_all    = nullptr;
    p.n_nodes      = a->n_nodes;
    p.chunk_off    = chunk_off;
    p.plan         = plan;
    p.ticket       = reinterpret_cast<unsigned int*>(plan + 2);
    p.out          = a->hist;
    p.mb                 = mb;
    p.mb_ptr             = nullptr;
    p.pairs_by_position  = a->pairs_by_position != 0 ? 1 : 0;
    const HistLaunch hl  = PickHistKernel(a->bin_bytes, mb, float_mode, OrderOf(p), F, K, a->n_rows, a->n_nodes, false, sm_count, 1,
                                          Aligned16(p.bins) && Aligned16(p.out));

    // the array keeps what the previous call left: clear the words that accumulate
    LBK_CUDA(cudaMemsetAsync(plan, 0, sizeof(int32_t) * 12, stream));
    LBK_CUDA(cudaMemsetAsync(a->hist, 0, sizeof(GPairI64) * a->n_nodes * K * B, stream));
    if (!float_mode && a->max_abs != nullptr) {
      max_abs = const_cast<int*>(reinterpret_cast<const int*>(a->max_abs));
    } else if (!float_mode) {
      const int64_t n = a->n_rows * K;
      if (n > 0) {
        LaunchChained(k_max_abs, sm_count * 8, 256, 0, stream, static_cast<const int2*>(p.gpair), n, max_abs);
        LBK_LAUNCH_CHECK();
      }
    }
    // no merge-tree slots here (they would have to be allocated): nodes cut into chunks flush with atomics
    p.wpre      = nullptr;
    p.ranges    = false;
    p.arrive    = nullptr;
    p.partial   = nullptr;
    p.status    = nullptr;
    p.push_recv = nullptr;
    p.push_rank = 0;
    p.push_ranks = 1;
    p.push_slot_pairs = 0;
    p.push_len  = 0;
    p.max_abs           = float_mode ? nullptr : max_abs;
    p.slot_capacity     = 0;
    p.n_arrive          = 0;
    p.tile_items        = sm_count * kTileItemsPerSm;
    const int units     = (hl.tile ? (F + kTileFeatures - 1) / kTileFeatures : (p.G + hl.width - 1) / hl.width) * K;
    LaunchChained(k_hist_plan, 1, 1024, 0, stream, p, units, hl.tile ? p.tile_items : hl.grid, hl.tile ? kTileMinRows : kMinChunk, hl.copies != 1, chunk_off, nullptr, plan);
    LBK_LAUNCH_CHECK();
    LaunchChained(hl.fn, hl.grid, hl.threads, hl.smem, stream, p);
    LBK_LAUNCH_CHECK();
    LBK_CUDA(cudaStreamSynchronize(stream));
  });
}
