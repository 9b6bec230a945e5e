// Row-to-node repartition: after a level's splits are chosen, the rows of every split node are divided
// between its two children; rows of nodes that stay leaves drop out.
//
// Reference behaviour restated here: UpdatePositions, src/models/tree/build_tree.cu:1026-1080 -
// position := -1 for rows in leaves, else left child iff (double)x <= split_value, followed by a
// full radix sort of all (node,row) pairs by node.  Because a split value is one of the feature's
// proposals, "x <= split_value" is the same as "bin(x) <= bin(split)", so the decision needs one
// byte of the binned matrix instead of the raw feature value, and because the rows are already
// grouped by parent the sort reduces to a two-way partition inside each segment.
//
// The order of the rows inside a node carries no meaning (the histograms are sums of whole numbers),
// so one pass does: the left child fills the node's segment from its start, the right child from
// its end, and a block claims room for the rows of a chunk with one 64-bit addition to the node's
// cursor (lefts in the low half, rights in the high half).  Chunks are handed out in order and keep the
// order of their rows, so rows that are neighbours in a node stay (nearly) neighbours in the matrix.
// The claim that completes the node writes the segments of its children.
#include "device_utils.cuh"
#include "internal.h"

namespace lbk {
namespace {

constexpr int kPartThreads   = 256;
constexpr int kPartWarps     = kPartThreads / 32;
constexpr int kPartItems     = 8;
constexpr int kPartTile      = kPartThreads * kPartItems;  // rows per chunk
constexpr int kPartBlocks    = 4;    // per SM: as many as are resident
// Bands of a level (see k_partition): as many as bring the columns of a band's rows to kPartBandBytes of L2, but with
// kPartBandTurns chunks for every block, because a band is planned anew.  Levels 1 to 8 of 100M x 64: 4.83 ms with one turn,
// 4.66 with two, 4.67 with four; 10M x 64, six levels: 339, 329 and 322 us.  So a level has bands where its bins are more than
// 24 MB and its rows at least eight chunks for every block (9.7 million rows on 148 SMs), whatever the number of features.
constexpr int64_t kPartBandBytes = 24 << 20;
constexpr int kPartBandTurns     = 4;
constexpr int kPartMaxLogBands   = 7;
constexpr int kPartPlanNodes = 1024;  // levels of up to this many nodes are planned inside the kernel

__device__ inline int ChunksOf(const PartitionLevel& p, int j)
{
  const int rows = p.seg_end[j] - p.seg_begin[j];
  return p.feature[p.node_begin + j] != -1 && rows > 0 ? (rows + kPartTile - 1) / kPartTile : 0;
}

// chunks before each node of a level with more nodes than a block can hold
__global__ void __launch_bounds__(1024)
  k_part_plan(const __grid_constant__ PartitionLevel p, int32_t* __restrict__ chunk_off)
{
  AfterTheKernelBefore();
  __shared__ int carry, wsum[32];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (tid == 0) {
    carry        = 0;
    chunk_off[0] = 0;
  }
  __syncthreads();
  for (int base = 0; base < p.n_nodes; base += blockDim.x) {
    const int i = base + tid;
    int incl    = i < p.n_nodes ? ChunksOf(p, i) : 0;
    for (int off = 1; off < 32; off <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, incl, off);
      if (lane >= off) incl += v;
    }
    if (lane == 31) wsum[warp] = incl;
    __syncthreads();
    if (warp == 0) {
      const int w = wsum[lane];
      int wi      = w;
      for (int off = 1; off < 32; off <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, wi, off);
        if (lane >= off) wi += v;
      }
      wsum[lane] = wi - w;
    }
    __syncthreads();
    incl += carry + wsum[warp];
    if (i < p.n_nodes) chunk_off[i + 1] = incl;
    __syncthreads();
    if (tid == blockDim.x - 1) carry = incl;
    __syncthreads();
  }
}

// Persistent blocks, a chunk at a time.  Bound by HBM: per row and level the row id, its pair and the
// byte of its bin in, row id and pair out.  Four blocks of 64 registers a thread are resident on an SM, and no
// more are launched (six: the two that come later do their third of the chunks on a half-empty SM).  512 threads with four rows
// each: 1.60 -> 1.70 ms at 40M x 64, depth 8; five blocks of 48 registers: 2.06 ms.  kPlanInside: every block finds the chunks before
// each node by itself (a scan of at most kPartPlanNodes counts once per block and band, about a microsecond,
// instead of a launch of its own).
//
// A chunk is a chain of waits (row ids, bins, the claim), and the L1 holds what is on its way: shared memory taken from it costs more
// than the loads it could hold (row ids and pairs staged there, six blocks, 28 KB of L1: level 8 of 100M x 64 1.26 -> 2.27 ms;
// three stages of chunks of 1024 rows in a pipeline: 1.44).  So everything stays in registers, and the pairs are asked
// for after the bins have come, while the room is claimed: level 0 435 -> 400 us, level 1 520 -> 488.
//
// Bands.  The rows of a node lie thin in the matrix at depth, so that a 64-byte piece of a column is fetched for one byte.  But
// many nodes of a level split on the same few features, and their rows use other bytes of the same piece.  The chunks of
// a level are therefore handed out in bands: band b of n has from every node the b-th n-th of its chunks, in the order
// of the matrix, so that all nodes pass through the same rows at about the same time and a piece that one of them has
// fetched is in L2 for the others.  A left child's rows lie in the order of the matrix, a right child's (filled from the end)
// in the opposite one: its chunks are taken from its end, on every level.  (Upper levels gain nothing from their bands, but
// keep the rows in order for the ones below: levels 5 to 8 778, 868, 952, 1125 us without, 592, 638, 669, 743 with them.)
// 100M x 64, nine levels: 6.71 -> 5.07 ms, the last one 1.25 -> 0.74; 30M x 64, seven levels: 1.18 -> 1.08; 20M x 300: 1.08 -> 0.99.
__device__ inline int BandBegin(int chunks, int band, int log_bands) { return static_cast<int>((static_cast<long long>(chunks) * band) >> log_bands); }

// The whole block: off[j] = the sum of count(0 .. j - 1), off[n] = all of them.
template <typename Count>
__device__ inline void PlanInside(int n, Count count, int32_t* off /* [kPartPlanNodes + 1] */, int* wsum /* [kPartWarps] */)
{
  constexpr int kPer = kPartPlanNodes / kPartThreads;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  int c[kPer], sum = 0;
#pragma unroll
  for (int i = 0; i < kPer; ++i) {
    const int j = tid * kPer + i;
    c[i]        = j < n ? count(j) : 0;
    sum += c[i];
  }
  int incl = sum;
  for (int d = 1; d < 32; d <<= 1) {
    const int v = __shfl_up_sync(0xffffffffu, incl, d);
    if (lane >= d) incl += v;
  }
  if (lane == 31) wsum[warp] = incl;
  __syncthreads();  // (and whoever still looks for a node of the band before)
  int before = incl - sum;
  for (int w = 0; w < warp; ++w) before += wsum[w];
#pragma unroll
  for (int i = 0; i < kPer; ++i) {
    const int j = tid * kPer + i;
    if (j < n) off[j] = before;
    before += c[i];
    if (j == n - 1) off[n] = before;
  }
  __syncthreads();
}

__device__ inline int LoadOnce(const int32_t* a)
{
  int v;
  asm volatile("ld.global.cs.s32 %0, [%1];\n" : "=r"(v) : "l"(a));
  return v;
}
__device__ inline int2 LoadOnce(const int2* a)
{
  int2 v;
  asm volatile("ld.global.cs.v2.s32 {%0, %1}, [%2];\n" : "=r"(v.x), "=r"(v.y) : "l"(a));
  return v;
}
template <bool kL2Only>
__device__ inline int LoadBin(const uint8_t* a)
{
  unsigned short v;
  if (kL2Only) asm volatile("ld.global.cg.u8 %0, [%1];\n" : "=h"(v) : "l"(a));
  else asm volatile("ld.global.u8 %0, [%1];\n" : "=h"(v) : "l"(a));
  return v;
}
template <bool kL2Only>
__device__ inline int LoadBin(const uint16_t* a)
{
  unsigned short v;
  if (kL2Only) asm volatile("ld.global.cg.u16 %0, [%1];\n" : "=h"(v) : "l"(a));
  else asm volatile("ld.global.u16 %0, [%1];\n" : "=h"(v) : "l"(a));
  return v;
}

template <typename BinT, bool kPlanInside, bool kBands>
__global__ void __launch_bounds__(kPartThreads, kPartBlocks)
  k_partition(const __grid_constant__ PartitionLevel p, const int32_t* __restrict__ chunk_off_global, int log_bands)
{
  AfterTheKernelBefore();
  __shared__ int32_t s_off[kPlanInside ? kPartPlanNodes + 1 : 1];
  __shared__ int32_t s_count[kBands ? kPartPlanNodes : 1];
  __shared__ int32_t s_band[kBands ? (1 << kPartMaxLogBands) + 1 : 1];  // chunks before each band
  __shared__ int s_cnt[kPartItems * kPartWarps];  // per (item, warp): lefts | rows << 16, then prefixes
  __shared__ int s_wsum[kPartWarps];
  __shared__ int s_base[2];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int n   = p.n_nodes;
  const int32_t* chunk_off = kPlanInside ? s_off : chunk_off_global;
  int band = -1, total;
  if (kBands) {
    // where every band begins: the nodes are divided among the threads of a band
    const int bands = 1 << log_bands, parts = kPartThreads >> log_bands;
    for (int j = tid; j < n; j += kPartThreads) s_count[j] = ChunksOf(p, j);
    for (int i = tid; i <= bands; i += kPartThreads) s_band[i] = 0;
    __syncthreads();
    int sum = 0;
    for (int j = tid >> log_bands; j < n; j += parts) sum += BandBegin(s_count[j], (tid & (bands - 1)) + 1, log_bands);
    atomicAdd(&s_band[(tid & (bands - 1)) + 1], sum);
    __syncthreads();
    total = s_band[bands];
  } else {
    if (kPlanInside) PlanInside(n, [&](int j) { return ChunksOf(p, j); }, s_off, s_wsum);
    total = chunk_off[n];
  }
  // nodes that were not split, or have no rows here, leave two empty segments
  for (int j = blockIdx.x * kPartThreads + tid; j < n; j += gridDim.x * kPartThreads) {
    if ((kBands ? s_count[j] : chunk_off[j + 1] - chunk_off[j]) == 0) {
      p.seg_begin_out[2 * j] = p.seg_end_out[2 * j] = 0;
      p.seg_begin_out[2 * j + 1] = p.seg_end_out[2 * j + 1] = 0;
    }
  }
  // The c-th chunk of the level (the whole block asks, in ascending order).
  struct Chunk {
    int j, begin, rows;
  };
  auto chunk_at = [&](int c) -> Chunk {
    if (c >= total) return Chunk{0, 0, 0};
    if (kBands) {
      int b = max(band, 0);
      while (c >= s_band[b + 1]) ++b;
      if (b != band) {
        band = b;
        PlanInside(n, [&](int j) { return BandBegin(s_count[j], b + 1, log_bands) - BandBegin(s_count[j], b, log_bands); }, s_off, s_wsum);
      }
      c -= s_band[band];
    }
    int lo = 0, hi = n;  // last node with chunk_off <= c
    while (hi - lo > 1) {
      const int mid = (lo + hi) >> 1;
      if (chunk_off[mid] <= c) lo = mid; else hi = mid;
    }
    int i = c - chunk_off[lo];
    if (kBands) {
      i += BandBegin(s_count[lo], band, log_bands);
      if (lo & 1) i = s_count[lo] - 1 - i;
    }
    const int begin = p.seg_begin[lo] + i * kPartTile;
    return Chunk{lo, begin, min(p.seg_end[lo] - begin, kPartTile)};
  };
  const bool move_pairs = p.pairs_in != nullptr && p.K == 1;  // (of several outputs: read where they are written)
  for (int c = blockIdx.x;; c += gridDim.x) {
    const Chunk a = chunk_at(c);
    if (a.rows == 0) break;
    const int node  = p.node_begin + a.j;
    const int sb    = p.split_bin[node];
    const BinT* col = static_cast<const BinT*>(p.bins) + static_cast<int64_t>(p.feature[node]) * p.bin_pitch;
    // The loads in this order (as volatile statements, so that all of a kind are on their way before one is waited for).
    int rid[kPartItems], bin[kPartItems];
    int2 pair[kPartItems];
    const bool whole = a.rows == kPartTile;
    auto at = [&](int i) -> int {  // position of the thread's i-th row in the chunk (of the chunk's last row, if it has none)
      const int e = i * kPartThreads + tid;
      return whole ? e : min(e, a.rows - 1);
    };
    if (p.row_index_in != nullptr) {
      const int32_t* from = p.row_index_in + a.begin;
#pragma unroll
      for (int i = 0; i < kPartItems; ++i) rid[i] = LoadOnce(from + at(i));
    } else {
#pragma unroll
      for (int i = 0; i < kPartItems; ++i) rid[i] = a.begin + at(i);
    }
    auto load_pairs = [&]() {
      const int2* from = p.pairs_in + a.begin;
#pragma unroll
      for (int i = 0; i < kPartItems; ++i) pair[i] = LoadOnce(from + at(i));
    };
#pragma unroll
    for (int i = 0; i < kPartItems; ++i) bin[i] = LoadBin<kBands>(col + rid[i]);
    unsigned ml[kPartItems];
    // lanes of item i that hold a row
    auto valid = [&](int i) -> unsigned {
      const int left = a.rows - i * kPartThreads - warp * 32;
      return left >= 32 ? 0xffffffffu : left <= 0 ? 0u : (1u << left) - 1u;
    };
#pragma unroll
    for (int i = 0; i < kPartItems; ++i) {
      const unsigned mv = valid(i);
      ml[i]             = __ballot_sync(0xffffffffu, bin[i] <= sb) & mv;
      if (lane == 0) s_cnt[i * kPartWarps + warp] = __popc(ml[i]) | (__popc(mv) << 16);
    }
    if (move_pairs) load_pairs();
    __syncthreads();
    if (warp == 0) {
      // 64 counts, two per lane, in (item, warp) order = row order
      static_assert(kPartItems * kPartWarps == 64, "two counts per lane");
      const int x = s_cnt[2 * lane], y = s_cnt[2 * lane + 1];
      int incl = x + y;
      for (int off = 1; off < 32; off <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, incl, off);
        if (lane >= off) incl += v;
      }
      const int excl      = incl - x - y;
      s_cnt[2 * lane]     = excl;
      s_cnt[2 * lane + 1] = excl + x;
      if (lane == 31) {
        const int nb = p.seg_begin[a.j], ne = p.seg_end[a.j];
        const int lefts = incl & 0xffff, rights = (incl >> 16) - lefts;
        const unsigned long long old =
          atomicAdd(p.cursor + node, static_cast<unsigned long long>(lefts) | (static_cast<unsigned long long>(rights) << 32));
        const int l0 = static_cast<int>(old & 0xffffffffull), r0 = static_cast<int>(old >> 32);
        s_base[0] = nb + l0;
        s_base[1] = ne - r0 - rights;
        if (l0 + lefts + r0 + rights == ne - nb) {
          p.seg_begin_out[2 * a.j]     = nb;
          p.seg_end_out[2 * a.j]       = nb + l0 + lefts;
          p.seg_begin_out[2 * a.j + 1] = nb + l0 + lefts;
          p.seg_end_out[2 * a.j + 1]   = ne;
        }
      }
    }
    __syncthreads();
    const unsigned below = (1u << lane) - 1u;
#pragma unroll
    for (int i = 0; i < kPartItems; ++i) {
      const int e = i * kPartThreads + tid;
      if (e < a.rows) {
        const int before = s_cnt[i * kPartWarps + warp];
        const int lefts = before & 0xffff, rights = (before >> 16) - lefts;
        const int pos = (ml[i] >> lane) & 1u ? s_base[0] + lefts + __popc(ml[i] & below)
                                             : s_base[1] + rights + __popc(~ml[i] & below);
        p.row_index_out[pos] = rid[i];
        if (move_pairs) {
          p.pairs_out[pos] = pair[i];
        } else if (p.pairs_in != nullptr) {
          for (int k = 0; k < p.K; ++k)
            p.pairs_out[static_cast<int64_t>(pos) * p.K + k] = p.pairs_in[static_cast<int64_t>(a.begin + e) * p.K + k];
        }
      }
    }
    __syncthreads();  // s_cnt, s_base are written again
  }
}

template <typename BinT>
auto PartitionKernel(bool inside, bool bands)
{
  return bands ? k_partition<BinT, true, true> : inside ? k_partition<BinT, true, false> : k_partition<BinT, false, false>;
}

}  // namespace

void PartitionRows(lbk_context* ctx, Scratch& s, const PartitionLevel& pl, cudaStream_t stream)
{
  if (pl.n_rows <= 0) {
    LBK_CUDA(cudaMemsetAsync(pl.seg_begin_out, 0, sizeof(int32_t) * 2 * pl.n_nodes, stream));
    LBK_CUDA(cudaMemsetAsync(pl.seg_end_out, 0, sizeof(int32_t) * 2 * pl.n_nodes, stream));
    return;
  }
  // an upper bound of the number of chunks; no more blocks than are resident at once
  const int64_t max_chunks = pl.n_rows / kPartTile + std::min<int64_t>(pl.n_nodes, pl.n_rows) + 1;
  const unsigned grid      = static_cast<unsigned>(std::min<int64_t>(max_chunks, static_cast<int64_t>(ctx->sm_count) * kPartBlocks));
  const bool inside        = pl.n_nodes <= kPartPlanNodes;
  int32_t* chunk_off       = nullptr;
  if (!inside) {
    chunk_off = s.alloc<int32_t>(static_cast<size_t>(pl.n_nodes) + 1);
    LaunchChained(k_part_plan, 1, 1024, 0, stream, pl, chunk_off);
    LBK_LAUNCH_CHECK();
  }
  int log_bands = 0;
  if (inside && pl.n_nodes > 1)
    while (log_bands < kPartMaxLogBands && (pl.n_rows * pl.n_features * pl.bin_bytes) >> log_bands > kPartBandBytes &&
           (pl.n_rows / kPartTile) >> (log_bands + 1) >= kPartBandTurns * grid)
      ++log_bands;
  auto fn = pl.bin_bytes == 1 ? PartitionKernel<uint8_t>(inside, log_bands > 0) : PartitionKernel<uint16_t>(inside, log_bands > 0);
  LaunchChained(fn, grid, kPartThreads, 0, stream, pl, chunk_off, log_bands);
}

}  // namespace lbk
