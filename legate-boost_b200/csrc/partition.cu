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
constexpr int kPartItems     = 8;
constexpr int kPartTile      = kPartThreads * kPartItems;  // rows per chunk
constexpr int kPartBlocks    = 4;    // per SM: as many as are resident
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
// 32-byte sector of its bin in, row id and pair out.  Four blocks of 64 registers a thread are resident on an SM, and no
// more are launched (six: the two that come later do their third of the chunks on a half-empty SM): 40M x 64, depth 8,
// seven levels: 1.91 -> 1.60 ms, 10M: 454 -> 414 us; the second level 26 bytes per row at 5.0 TB/s.  512 threads with four rows
// each: 1.70 ms; five blocks of 48 registers: 2.06 ms; the rows put in order in shared memory and written as
// whole lines while the next chunk's are on their way: 1.77 ms.  kPlanInside: every block finds the chunks before
// each node by itself (a scan of at most kPartPlanNodes counts once per block, about a microsecond,
// instead of a launch of its own).
template <typename BinT, bool kPlanInside>
__global__ void __launch_bounds__(kPartThreads, kPartBlocks)
  k_partition(const __grid_constant__ PartitionLevel p, const int32_t* __restrict__ chunk_off_global)
{
  __shared__ int32_t s_off[kPlanInside ? kPartPlanNodes + 1 : 1];
  __shared__ int s_cnt[kPartItems * kPartThreads / 32];  // per (item, warp): lefts | rows << 16, then prefixes
  __shared__ int s_wsum[kPartThreads / 32];
  __shared__ int s_base[2];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int n   = p.n_nodes;
  const int32_t* chunk_off = chunk_off_global;
  if (kPlanInside) {
    constexpr int kPer = kPartPlanNodes / kPartThreads;
    int c[kPer], sum = 0;
#pragma unroll
    for (int i = 0; i < kPer; ++i) {
      const int j = tid * kPer + i;
      c[i]        = j < n ? ChunksOf(p, j) : 0;
      sum += c[i];
    }
    int incl = sum;
    for (int off = 1; off < 32; off <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, incl, off);
      if (lane >= off) incl += v;
    }
    if (lane == 31) s_wsum[warp] = incl;
    __syncthreads();
    int before = incl - sum;
    for (int w = 0; w < warp; ++w) before += s_wsum[w];
#pragma unroll
    for (int i = 0; i < kPer; ++i) {
      const int j = tid * kPer + i;
      if (j < n) s_off[j] = before;
      before += c[i];
      if (j == n - 1) s_off[n] = before;
    }
    __syncthreads();
    chunk_off = s_off;
  }
  // nodes that were not split, or have no rows here, leave two empty segments
  for (int j = blockIdx.x * kPartThreads + tid; j < n; j += gridDim.x * kPartThreads) {
    if (chunk_off[j + 1] == chunk_off[j]) {
      p.seg_begin_out[2 * j] = p.seg_end_out[2 * j] = 0;
      p.seg_begin_out[2 * j + 1] = p.seg_end_out[2 * j + 1] = 0;
    }
  }
  const int total = chunk_off[n];
  for (int c = blockIdx.x; c < total; c += gridDim.x) {
    int lo = 0, hi = n;  // last node with chunk_off <= c
    while (hi - lo > 1) {
      const int mid = (lo + hi) >> 1;
      if (chunk_off[mid] <= c) lo = mid; else hi = mid;
    }
    const int j    = lo;
    const int node = p.node_begin + j;
    const int sb   = p.split_bin[node];
    const int nb = p.seg_begin[j], ne = p.seg_end[j];
    const int rb = nb + (c - chunk_off[j]) * kPartTile;
    const int re = min(ne, rb + kPartTile);
    const BinT* col = static_cast<const BinT*>(p.bins) + static_cast<int64_t>(p.feature[node]) * p.bin_pitch;
    int rid[kPartItems];
    int2 pair[kPartItems];
    unsigned ml[kPartItems], mv[kPartItems];
#pragma unroll
    for (int i = 0; i < kPartItems; ++i) {
      const int r = rb + i * kPartThreads + tid;
      rid[i]      = r < re ? (p.row_index_in != nullptr ? __ldcs(p.row_index_in + r) : r) : 0;
    }
    if (p.pairs_in != nullptr && p.K == 1) {
#pragma unroll
      for (int i = 0; i < kPartItems; ++i) {
        const int r = rb + i * kPartThreads + tid;
        if (r < re) pair[i] = __ldcs(p.pairs_in + r);
      }
    }
    int bin[kPartItems];
#pragma unroll
    for (int i = 0; i < kPartItems; ++i) bin[i] = rb + i * kPartThreads + tid < re ? static_cast<int>(col[rid[i]]) : 0;
#pragma unroll
    for (int i = 0; i < kPartItems; ++i) {
      const bool in = rb + i * kPartThreads + tid < re;
      mv[i]         = __ballot_sync(0xffffffffu, in);
      ml[i]         = __ballot_sync(0xffffffffu, in && bin[i] <= sb);
      if (lane == 0) s_cnt[i * (kPartThreads / 32) + warp] = __popc(ml[i]) | (__popc(mv[i]) << 16);
    }
    __syncthreads();
    if (warp == 0) {
      // 64 counts, two per lane, in (item, warp) order = row order
      const int a = s_cnt[2 * lane], b = s_cnt[2 * lane + 1];
      int incl = a + b;
      for (int off = 1; off < 32; off <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, incl, off);
        if (lane >= off) incl += v;
      }
      const int excl      = incl - a - b;
      s_cnt[2 * lane]     = excl;
      s_cnt[2 * lane + 1] = excl + a;
      if (lane == 31) {
        const int lefts = incl & 0xffff, rights = (incl >> 16) - lefts;
        const unsigned long long old =
          atomicAdd(p.cursor + node, static_cast<unsigned long long>(lefts) | (static_cast<unsigned long long>(rights) << 32));
        const int l0 = static_cast<int>(old & 0xffffffffull), r0 = static_cast<int>(old >> 32);
        s_base[0] = nb + l0;
        s_base[1] = ne - r0 - rights;
        if (l0 + lefts + r0 + rights == ne - nb) {
          p.seg_begin_out[2 * j]     = nb;
          p.seg_end_out[2 * j]       = nb + l0 + lefts;
          p.seg_begin_out[2 * j + 1] = nb + l0 + lefts;
          p.seg_end_out[2 * j + 1]   = ne;
        }
      }
    }
    __syncthreads();
    const unsigned below = (1u << lane) - 1u;
#pragma unroll
    for (int i = 0; i < kPartItems; ++i) {
      const int r = rb + i * kPartThreads + tid;
      if (r < re) {
        const int before = s_cnt[i * (kPartThreads / 32) + warp];
        const int lefts = before & 0xffff, rights = (before >> 16) - lefts;
        const int pos = (ml[i] >> lane) & 1u ? s_base[0] + lefts + __popc(ml[i] & below)
                                             : s_base[1] + rights + __popc(mv[i] & ~ml[i] & below);
        p.row_index_out[pos] = rid[i];
        if (p.pairs_in != nullptr) {
          if (p.K == 1) {
            p.pairs_out[pos] = pair[i];
          } else {
            for (int k = 0; k < p.K; ++k)
              p.pairs_out[static_cast<int64_t>(pos) * p.K + k] = p.pairs_in[static_cast<int64_t>(r) * p.K + k];
          }
        }
      }
    }
    __syncthreads();  // s_cnt, s_base are written again
  }
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
    k_part_plan<<<1, 1024, 0, stream>>>(pl, chunk_off);
    LBK_LAUNCH_CHECK();
  }
  auto fn = pl.bin_bytes == 1 ? (inside ? k_partition<uint8_t, true> : k_partition<uint8_t, false>)
                              : (inside ? k_partition<uint16_t, true> : k_partition<uint16_t, false>);
  fn<<<grid, kPartThreads, 0, stream>>>(pl, chunk_off);
  LBK_LAUNCH_CHECK();
}

}  // namespace lbk
