// Ensemble predict on ranks: x <= split as a comparison of whole numbers.
//
// A walk only compares x[f] with the splits on feature f.  With the ensemble's splits on every feature sorted, x[f] may be
// replaced by its rank among them (how many are smaller), and a split by its own: x <= split if and only if rank(x) <=
// rank(split).  Ranks fit 16 bits, so that a node - rank and feature - is one 4-byte word for float32 and float64 alike, and
// the values of two rows share a word of shared memory.  That is worth a pass over X which finds the ranks as soon as the
// ensemble is large enough (RankedPays): the walks are bound by the load/store data pipe of the SM, and a level is two
// passes (node, rank) plus bank conflicts, where k_predict_tiled takes two and a half (float32: split, value, half a
// word of ids) or five (float64).  Measured against that kernel: 10M x 100 float32, 500 trees of depth 8: 19.3 -> 13.5 ms (2.4
// of it for the ranks); 1M x 64 float64, 100 trees: 807 -> 531 us (170 for the ranks, 30 for the tables).
//
// Launches:
//   k_rank_count, k_rank_scatter   the ensemble's splits, feature by feature
//   k_rank_tables                  sorted, and an index by value into them (a block per feature)
//   k_rank_pack                    the trees' records, completed to one depth as for k_predict_tiled
// then for pieces of the rows that bound the memory of their ranks:
//   k_rank_rows                    X -> ranks, in the order of the walking blocks' tiles
//   k_predict_ranked               the walks
//
// One output.  Sums are made in tree order in float64, as everywhere.
#include "predict.cuh"

namespace lbk {
namespace {

constexpr int kMaxRank      = 32764;  // entries of a feature's table: ranks 1 .. 32765, one more for a NaN, below 2^15
constexpr int kSortChunk    = 16384;  // values sorted in shared memory at a time
constexpr int kMaxChunks    = 16;
constexpr int kRankThreads  = 512;    // of k_rank_rows
constexpr int kRankAhead    = 8;      // rows of a lane whose values are on their way together
constexpr int kRankTileRows = 32;     // rows of a warp per turn: as many of either half of a tile
constexpr int kWalkThreads  = 512;    // of k_predict_ranked at most, without the producer

// A feature's table.  Values are sorted; bucket b of nb holds those that RankBucket sends there.
struct RankTable {
  float lo, scale;
  int off;    // first entry in `cuts`, `lut`
  int m, nb;
};

// Monotone in x, for any lo and scale >= 0 (a NaN on the way is bucket 0: scale is then 0 or infinite and x not above lo), so
// the values of lower buckets are below x and those of higher ones above it.
__device__ inline int RankBucket(float x, float lo, float scale, int nb)
{
  const int b = __float2int_rz((x - lo) * scale);
  return b < 0 ? 0 : b < nb ? b : nb - 1;
}

// The value that x is compared with at node i, or false if no split is made there (or none that anything passes: a NaN).
template <typename T>
__device__ inline bool SplitAt(const TreePtrs& t, int i, int F, int& f, T& cut)
{
  if (i >= t.max_nodes || 2 * i + 2 >= t.max_nodes) return false;
  f = t.feature[i];
  if (f < 0 || f >= F) return false;
  MakeSplit(cut, t.split[i]);
  return true;
}

template <typename T>
__global__ void __launch_bounds__(256) k_rank_count(const TreePtrs* __restrict__ trees, int F, int* __restrict__ counts)
{
  const TreePtrs t = trees[blockIdx.x];
  for (int i = threadIdx.x; i < t.max_nodes; i += blockDim.x) {
    int f;
    T cut;
    if (SplitAt(t, i, F, f, cut) && cut == cut) atomicAdd(counts + f, 1);
  }
}

// off [F + 1]: where each feature's values begin in `lists`
template <typename T>
__global__ void __launch_bounds__(256)
  k_rank_scatter(const TreePtrs* __restrict__ trees, int F, const int* __restrict__ counts, int* __restrict__ cursor, int* __restrict__ off,
                 T* __restrict__ lists)
{
  constexpr int kPer = 4;  // (F <= 1024)
  __shared__ int s_off[256 * kPer], s_wsum[8];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  int c[kPer], sum = 0;
#pragma unroll
  for (int i = 0; i < kPer; ++i) {
    const int f = tid * kPer + i;
    c[i]        = f < F ? counts[f] : 0;
    sum += c[i];
  }
  int incl = sum;
  for (int o = 1; o < 32; o <<= 1) {
    const int v = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += v;
  }
  if (lane == 31) s_wsum[warp] = incl;
  __syncthreads();
  int before = incl - sum;
  for (int w = 0; w < warp; ++w) before += s_wsum[w];
#pragma unroll
  for (int i = 0; i < kPer; ++i) {
    const int f = tid * kPer + i;
    s_off[f]    = before;
    if (blockIdx.x == 0 && f < F) off[f] = before;
    before += c[i];
    if (blockIdx.x == 0 && f == F - 1) off[F] = before;
  }
  __syncthreads();
  const TreePtrs t = trees[blockIdx.x];
  for (int i = tid; i < t.max_nodes; i += blockDim.x) {
    int f;
    T cut;
    if (SplitAt(t, i, F, f, cut) && cut == cut) lists[s_off[f] + atomicAdd(cursor + f, 1)] = cut;
  }
}

// The first index of n sorted values that is not below v (kUpper: that is above v).
template <bool kUpper, typename T>
__device__ inline int BoundOf(const T* a, int n, T v)
{
  int lo = 0;
  while (n > 0) {
    const int half = n >> 1;
    if (kUpper ? !(v < a[lo + half]) : a[lo + half] < v) {
      lo += half + 1;
      n -= half + 1;
    } else {
      n = half;
    }
  }
  return lo;
}

// A block per feature: its values sorted, equal ones once, and the index.  More values than shared memory holds
// are sorted in chunks (equal values of different chunks stay, which changes no comparison of ranks) and placed by their
// ranks in the other chunks.  A feature with more values than ranks sets *too_many.
template <typename T>
__global__ void __launch_bounds__(1024)
  k_rank_tables(const int* __restrict__ off, T* __restrict__ lists, T* __restrict__ cuts, unsigned* __restrict__ lut,
                RankTable* __restrict__ tables, int* __restrict__ too_many)
{
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T* s = reinterpret_cast<T*>(smem_raw);
  __shared__ int s_wsum[32], s_len[kMaxChunks];
  const int f = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int begin = off[f], n = off[f + 1] - begin;
  T* list = lists + begin;
  T* out  = cuts + begin;
  const int chunks = (n + kSortChunk - 1) / kSortChunk;
  int m            = 0;
  bool fits        = chunks <= kMaxChunks;
  for (int c = 0; c < chunks && fits; ++c) {
    const int c0 = c * kSortChunk, len = min(kSortChunk, n - c0);
    int P = 1;
    while (P < len) P <<= 1;
    __syncthreads();
    for (int i = tid; i < P; i += 1024) s[i] = i < len ? list[c0 + i] : static_cast<T>(INFINITY);
    for (int k = 2; k <= P; k <<= 1) {
      for (int j = k >> 1; j > 0; j >>= 1) {
        // (up to 32 apart, values that meet are of one warp)
        if (j >= 64 || j == k >> 1) __syncthreads();
        else if (j == 32) __syncthreads();
        else __syncwarp();
        for (int e = tid; e < P / 2; e += 1024) {
          const int i = 2 * e - (e & (j - 1));  // the e-th index without bit j
          const T a = s[i], b = s[i + j];
          if ((i & k) == 0 ? b < a : a < b) {
            s[i]     = b;
            s[i + j] = a;
          }
        }
      }
    }
    __syncthreads();
    // equal values once: to the front of the chunk, or straight to the table
    T* dst   = chunks == 1 ? out : list + c0;
    int kept = 0;
    for (int i0 = 0; i0 < len; i0 += 1024) {
      const int i      = i0 + tid;
      const bool keep  = i < len && (i == 0 || s[i] != s[i - 1]);
      const unsigned b = __ballot_sync(0xffffffffu, keep);
      if (lane == 0) s_wsum[warp] = __popc(b);
      __syncthreads();
      int at = kept + __popc(b & ((1u << lane) - 1u)), all = 0;
      for (int w = 0; w < 32; ++w) {
        if (w < warp) at += s_wsum[w];
        all += s_wsum[w];
      }
      if (keep) dst[at] = s[i];
      kept += all;
      __syncthreads();
    }
    if (tid == 0) s_len[c] = kept;
    m += kept;
  }
  fits = fits && m <= kMaxRank;
  if (!fits) {
    if (tid == 0) {
      *too_many = 1;
      tables[f] = RankTable{0.f, 0.f, begin, 0, 1};
    }
    return;
  }
  __syncthreads();
  if (chunks > 1) {
    for (int c = 0; c < chunks; ++c) {
      for (int i = tid; i < s_len[c]; i += 1024) {
        const T v = list[c * kSortChunk + i];
        int at    = i;
        for (int o = 0; o < chunks; ++o)
          if (o != c)
            at += o < c ? BoundOf<true>(list + o * kSortChunk, s_len[o], v) : BoundOf<false>(list + o * kSortChunk, s_len[o], v);
        out[at] = v;
      }
    }
    __syncthreads();
  }
  // the index: buckets of equal width between the first and the last finite value
  constexpr float kMax = 3.402823466e38f;
  RankTable t{0.f, 0.f, begin, m, max(m, 1)};
  if (m > 0) {
    t.lo           = fmaxf(static_cast<float>(out[0]), -kMax);
    const float hi = fminf(static_cast<float>(out[m - 1]), kMax);
    t.scale        = hi > t.lo ? static_cast<float>(t.nb) / (hi - t.lo) : 0.f;
  }
  int* start = reinterpret_cast<int*>(list);  // first value of every bucket (the values are in `out`)
  for (int i = tid; i < m; i += 1024) {
    const int b      = RankBucket(static_cast<float>(out[i]), t.lo, t.scale, t.nb);
    const int before = i > 0 ? RankBucket(static_cast<float>(out[i - 1]), t.lo, t.scale, t.nb) : -1;
    for (int q = before + 1; q <= b; ++q) start[q] = i;
    if (i == m - 1)
      for (int q = b + 1; q < t.nb; ++q) start[q] = m;
  }
  __syncthreads();
  for (int b = tid; b < m; b += 1024) {
    const int first = start[b], next = b + 1 < m ? start[b + 1] : m;
    lut[begin + b]  = static_cast<unsigned>(first) | (static_cast<unsigned>(next - first) << 16);
  }
  if (tid == 0) tables[f] = t;
}

// A completed tree of depth S: words [2^S], nodes counted from 1 (the children of i are 2 i and 2 i + 1), then leaf values
// [2^S].  A word holds the split's rank in its high half (0: nothing passes, a NaN) and, in its low half, where the
// feature's ranks begin in a walking block's tile, in units of 128 bytes.
__host__ __device__ inline int RankRecordBytes(int S) { return 12 << S; }

template <typename T>
__global__ void __launch_bounds__(256)
  k_rank_pack(const TreePtrs* __restrict__ trees, int F, int S, int lines, const RankTable* __restrict__ tables,
              const T* __restrict__ cuts, const unsigned* __restrict__ lut, const int* __restrict__ too_many, unsigned char* __restrict__ records)
{
  if (*too_many != 0) return;  // (a feature has no table)
  const TreePtrs t   = trees[blockIdx.x];
  unsigned char* out = records + static_cast<int64_t>(blockIdx.x) * RankRecordBytes(S);
  unsigned* words    = reinterpret_cast<unsigned*>(out);
  double* leaves     = reinterpret_cast<double*>(out + (4 << S));
  if (threadIdx.x == 0) words[0] = 0u;
  for (int i = threadIdx.x; i < (2 << S) - 1; i += blockDim.x) {
    const int L = 31 - __clz(i + 1);
    int cover = -1, f = 0;  // the first leaf on the path root -> i
    T cut{};
    for (int l = 0; l <= L && cover < 0; ++l) {
      const int a = ((i + 1) >> (L - l)) - 1;
      if (!SplitAt(t, a, F, f, cut)) cover = a;
    }
    if (L == S) {
      leaves[i - ((1 << S) - 1)] = t.leaf[cover];
    } else {
      // (below a leaf either way leads to its value)
      unsigned w = 0u;
      if (cover < 0) {
        const RankTable r = tables[f];
        int rank          = 0;
        if (cut == cut) {  // (it is in the table)
          const unsigned e = lut[r.off + RankBucket(static_cast<float>(cut), r.lo, r.scale, r.nb)];
          const int first  = static_cast<int>(e & 0xffffu);
          rank             = 1 + first + BoundOf<false>(cuts + r.off + first, static_cast<int>(e >> 16), cut);
        }
        w                 = (static_cast<unsigned>(rank) << 16) | static_cast<unsigned>(f * lines);
      }
      words[i + 1] = w;
    }
  }
}

template <typename T>
struct RankRowsArgs {
  const T* X;  // the piece's first row
  int64_t ldx;
  int64_t n_rows;
  int F, threads;  // of a walking block: a tile is 2 x threads rows
  int64_t n_tiles;
  const RankTable* tables;
  const T* cuts;
  const unsigned* lut;
  const int* too_many;
  unsigned* out;  // [tile][F][threads]
  int tail_blocks;  // blocks for the last group of features
};

// c = *at where n >= h, else as it was: a load without a branch.
__device__ inline void LoadSharedIf(float& c, int n, int h, unsigned at)
{
  asm volatile("{\n.reg .pred p;\nsetp.ge.s32 p, %1, %2;\n@p ld.shared.f32 %0, [%3];\n}\n" : "+f"(c) : "r"(n), "r"(h), "r"(at));
}
__device__ inline void LoadSharedIf(double& c, int n, int h, unsigned at)
{
  asm volatile("{\n.reg .pred p;\nsetp.ge.s32 p, %1, %2;\n@p ld.shared.f64 %0, [%3];\n}\n" : "+d"(c) : "r"(n), "r"(h), "r"(at));
}

// The rows of a block of k_rank_rows.  lut, cuts: the lane's feature's table, in shared memory (kInside) or in global.
template <typename T, bool kInside>
__device__ __forceinline__ void RankRows(const RankRowsArgs<T>& a, const RankTable& t, unsigned* turn, const unsigned* lut, const T* cuts, int f0,
                                         int width, int fl, int sub, int subs, int part, int parts)
{
  constexpr int kPitch     = kRankTileRows + 1;
  constexpr unsigned kSize = sizeof(T);
  const unsigned lut_at = kInside ? static_cast<unsigned>(__cvta_generic_to_shared(lut)) : 0u;
  const unsigned cuts_at = kInside ? static_cast<unsigned>(__cvta_generic_to_shared(cuts)) : 0u;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int per_tile = a.threads / kRankTileRows;
  const int n_work = static_cast<int>(a.n_tiles) * per_tile, stride = parts * (kRankThreads / 32);
  const T* column     = a.X + f0 + min(fl, width - 1);
  const int step_rows = kRankAhead * subs, steps = max(1, kRankTileRows / step_rows);  // of half a turn
  const int64_t lane_step = a.ldx * subs;
  struct Item {
    int tile, t0;
  };
  auto item_of = [&](int w) {
    Item i;
    i.tile = w / per_tile;
    i.t0   = (w - i.tile * per_tile) * kRankTileRows;
    return i;
  };
  // the rows of a step of an item; those behind the last one are the last one again
  auto load = [&](const Item& i, int st, T (&x)[kRankAhead]) {
    const int half = st >= steps ? 1 : 0;
    const int64_t row = static_cast<int64_t>(2 * i.tile + half) * a.threads + i.t0 + (st - half * steps) * step_rows;
    if (row + step_rows <= a.n_rows) {
      const T* p = column + (row + sub) * a.ldx;
#pragma unroll
      for (int u = 0; u < kRankAhead; ++u) {
        if (u * subs < kRankTileRows) x[u] = __ldg(p);  // (the others are dropped)
        p += lane_step;
      }
    } else {
#pragma unroll
      for (int u = 0; u < kRankAhead; ++u) x[u] = __ldg(column + min(row + sub + u * subs, a.n_rows - 1) * a.ldx);
    }
  };
  T ahead[kRankAhead] = {};
  int w     = part * (kRankThreads / 32) + warp;
  Item here = item_of(min(w, n_work - 1));
  load(here, 0, ahead);
  for (; w < n_work; w += stride) {
    const Item next = item_of(min(w + stride, n_work - 1));
    for (int st = 0; st < 2 * steps; ++st) {
      T x[kRankAhead];
#pragma unroll
      for (int u = 0; u < kRankAhead; ++u) x[u] = ahead[u];
      const bool more = st + 1 < 2 * steps;
      load(more ? here : next, more ? st + 1 : 0, ahead);
      // at: where the value is that x is compared with next, an address or an index
      unsigned at[kRankAhead];
      int n[kRankAhead];
      int most = 0;
#pragma unroll
      for (int u = 0; u < kRankAhead; ++u) {
        const int b      = RankBucket(static_cast<float>(x[u]), t.lo, t.scale, t.nb);
        const unsigned e = kInside ? LdsU32(lut_at + 4u * b) : __ldg(lut + b);
        at[u]            = kInside ? cuts_at + (e & 0xffffu) * kSize : e & 0xffffu;
        n[u]             = static_cast<int>(e >> 16);
        most             = max(most, n[u]);
      }
      most = __reduce_max_sync(0xffffffffu, most);
      // how many of the bucket's values are below x, in steps of falling powers of two: all rows' values are asked for before
      // the first is compared
      auto descend = [&](int h) {
        T cut[kRankAhead];
#pragma unroll
        for (int u = 0; u < kRankAhead; ++u) {
          cut[u] = static_cast<T>(INFINITY);
          if (kInside) LoadSharedIf(cut[u], n[u], h, at[u] + (h - 1) * kSize);
          else if (n[u] >= h) cut[u] = __ldg(cuts + at[u] + (h - 1));
        }
#pragma unroll
        for (int u = 0; u < kRankAhead; ++u)
          if (cut[u] < x[u]) {
            at[u] += kInside ? h * kSize : h;
            n[u] -= h;
          }
      };
      for (int h = most >= 8 ? 1 << (31 - __clz(most)) : 0; h >= 8; h >>= 1) descend(h);
      if (most >= 4) descend(4);
      if (most >= 2) descend(2);
      if (most >= 1) descend(1);
      if (fl < width) {
        const int half = st >= steps ? 1 : 0, r0 = (st - half * steps) * step_rows + sub;
        uint16_t* mine = reinterpret_cast<uint16_t*>(turn) + 2 * (fl * kPitch + r0) + half;
#pragma unroll
        for (int u = 0; u < kRankAhead; ++u)
          if (step_rows <= kRankTileRows || r0 + u * subs < kRankTileRows)
            mine[2 * u * subs] = static_cast<uint16_t>(x[u] == x[u] ? 1 + (kInside ? (at[u] - cuts_at) / kSize : at[u]) : t.m + 2);
      }
    }
    __syncwarp();
    unsigned* out = a.out + (static_cast<int64_t>(here.tile) * a.F + f0) * a.threads + here.t0 + lane;
#pragma unroll 8
    for (int f = 0; f < width; ++f) out[static_cast<int64_t>(f) * a.threads] = turn[f * kPitch + lane];
    __syncwarp();
    here = next;
  }
}

// X -> ranks.  A block serves one group of 32 features and keeps their tables in shared memory; lane = feature, a warp takes
// kRankTileRows rows of either half of a tile, turns their ranks in shared memory and writes them as words of two rows.  A
// last group of fewer features puts several rows side by side in a warp.
//
// Bound by the load/store pipe and the latency of its lookups: per 32 values a load of X, the bucket and about three steps of
// a search, each with the conflicts of 32 lanes on random banks, and the turn: twelve to sixteen passes and about 65
// instructions; 1.2M x 96 float32 238 us, x 64 float64 224.  (The values of a step asked for under branches, one row after
// the other: 700 us.)  Where the tables of a
// group do not fit (20 thousand values of float32) its features are taken in several turns over the rows; a feature
// that has no room alone is searched where its table lies.
template <typename T>
__global__ void __launch_bounds__(kRankThreads, 1) k_rank_rows(const RankRowsArgs<T> a)
{
  constexpr int kWarps = kRankThreads / 32, kPitch = kRankTileRows + 1;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  if (*a.too_many != 0) return;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  // the block's group of features and its share of the rows
  const int groups = (a.F + 31) / 32, last = groups - 1, blocks = gridDim.x;
  const int b = blockIdx.x, others = blocks - a.tail_blocks;
  const bool is_last = b >= others;
  const int g = is_last ? last : b % last, part = is_last ? b - others : b / last;
  const int parts = is_last ? a.tail_blocks : (others - g + last - 1) / last;
  const int f0 = 32 * g, width = min(32, a.F - f0);
  unsigned* turn    = reinterpret_cast<unsigned*>(smem_raw) + warp * 32 * kPitch;  // [feature][rows]: low half, high half
  unsigned* s_table = reinterpret_cast<unsigned*>(smem_raw) + kWarps * 32 * kPitch;
  __shared__ int s_begin[33], s_from[32];  // entries before the tables of the group's features, and where these lie in `cuts`
  if (warp == 0) {
    const RankTable r = a.tables[f0 + min(lane, width - 1)];
    const int m       = lane < width ? max(r.m, 1) : 0;
    int incl          = m;
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += v;
    }
    s_begin[lane + 1] = incl;
    s_from[lane]      = r.m > 0 ? r.off : -1;
    if (lane == 0) s_begin[0] = 0;
  }
  unsigned dyn_bytes;
  asm("mov.u32 %0, %%dynamic_smem_size;" : "=r"(dyn_bytes));
  const unsigned room = dyn_bytes - kWarps * 32 * kPitch * 4;
  auto fits = [&](int entries) { return static_cast<unsigned>((entries + 1) / 2 * 2) * 4u + static_cast<unsigned>(entries) * sizeof(T) <= room; };
  for (int w0 = 0, w1; w0 < width; w0 = w1) {
    __syncthreads();  // (the tables before have been read)
    // features [w0, w1): as many as have room for their tables; a power of two of them but at the end
    w1 = w0 + 1;
    while (w1 < width && fits(s_begin[w1 + 1] - s_begin[w0])) ++w1;
    if (w1 < width) w1 = w0 + (1 << (31 - __clz(w1 - w0)));
    const int n = w1 - w0, entries = s_begin[w1] - s_begin[w0];
    int per_row = 1;  // lanes that a row takes
    while (per_row < n) per_row <<= 1;
    const int sub = lane / per_row, subs = 32 / per_row, fl = lane % per_row, f = w0 + min(fl, n - 1);
    const RankTable t = a.tables[f0 + f];
    if (fits(entries)) {
      unsigned* s_lut = s_table;
      T* s_cuts       = reinterpret_cast<T*>(s_lut + (entries + 1) / 2 * 2);
      for (int e = w0 + warp; e < w1; e += kWarps) {
        const int from = s_from[e], at = s_begin[e] - s_begin[w0], m = s_begin[e + 1] - s_begin[e];
#pragma unroll 4
        for (int i = lane; i < m; i += 32) {
          s_lut[at + i]  = from >= 0 ? a.lut[from + i] : 0u;
          s_cuts[at + i] = from >= 0 ? a.cuts[from + i] : T(0);
        }
      }
      __syncthreads();
      const int at = s_begin[f] - s_begin[w0];
      RankRows<T, true>(a, t, turn, s_lut + at, s_cuts + at, f0 + w0, n, fl, sub, subs, part, parts);
    } else {
      // (a feature without values: the zero word says that its only bucket is empty)
      RankRows<T, false>(a, t, turn, t.m > 0 ? a.lut + t.off : reinterpret_cast<const unsigned*>(a.too_many), a.cuts + t.off, f0 + w0, n, fl, sub, subs, part, parts);
    }
  }
}

template <typename T>
struct RankedArgs {
  const T* X;  // the piece's first row; only read where the tables hold too many values
  int64_t ldx, n_rows;
  int F, n_trees, S;
  int nbuf;
  const unsigned* ranks;
  const unsigned char* records;
  const TreePtrs* trees;
  const int* too_many;
  PredictOut o;  // (of the piece's first row)
  int* status;
};

// The walks of a tile of 2 x threads rows: a thread has row t and row threads + t, whose ranks share a word, so that thread t
// only ever touches bank t mod 32.  The tile and the trees (groups of TG, two buffers) come by bulk copies of a producer
// warp, as in k_predict_tiled.  The top three nodes of a tree are one 16-byte load for both rows; below, a level of a
// walk is a load of its node, a load of a rank and four operations: the rank subtracted (the sign says where to go), the
// sign shifted into the node's number, two addresses (the rank's by a dot product of halves: with a mask and a
// multiplication 75 instructions per walk of depth 8 instead of 61, 307 us instead of 285 for 3.1M walks of a warp).
//
// Bound by the load/store pipe: 18 to 22 passes per walk of depth 8 (fitted trees; all nodes split), of which five are the
// 8-byte leaf value, at 20 to 25 clocks; 84 to 93 % of one pass per clock.
template <typename T, int TG>
__global__ void __launch_bounds__(kWalkThreads + 32, 1) k_predict_ranked(const RankedArgs<T> a)
{
  __shared__ __align__(8) unsigned long long s_bar[5];  // full[2], empty[2], the tile
  __shared__ int s_failed;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  const int F = a.F, S = a.S, threads = blockDim.x - 32;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int64_t row0 = static_cast<int64_t>(blockIdx.x) * 2 * threads;
  if (*a.too_many != 0) {
    // (a feature with more distinct splits than ranks: the walks read X and the trees where they lie)
    for (int64_t row = row0 + tid; row < row0 + 2 * threads && row < a.n_rows; row += blockDim.x) {
      const T* x = a.X + row * a.ldx;
      double sum = 0.0;
      for (int j = 0; j < a.n_trees; ++j) {
        const TreePtrs t = a.trees[j];
        int pos = 0, f;
        T cut;
        while (SplitAt(t, pos, F, f, cut)) pos = 2 * pos + 1 + (x[f] <= cut ? 0 : 1);
        sum += t.leaf[pos];
      }
      const double raw = a.o.init ? a.o.init[0] + sum : sum;
      FinishRow(&raw, 1, 1, a.o.pred + row * a.o.ldp, a.o.transform);
    }
    return;
  }
  const unsigned tile_bytes = static_cast<unsigned>(F) * threads * 4;
  const unsigned rec_bytes = RankRecordBytes(S), buf_bytes = TG * rec_bytes;
  const unsigned tile0 = static_cast<unsigned>(__cvta_generic_to_shared(smem_raw)), tree0 = tile0 + tile_bytes;
  const unsigned full0 = static_cast<unsigned>(__cvta_generic_to_shared(&s_bar[0])), empty0 = full0 + 16, tile_bar = full0 + 32;
  const int n_groups   = (a.n_trees + TG - 1) / TG;
  if (tid == 0) {
    s_failed = 0;
    for (int b = 0; b < 2; ++b) {
      MbarInit(full0 + 8 * b, 1);
      MbarInit(empty0 + 8 * b, threads / 32);
    }
    MbarInit(tile_bar, 1);
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  __syncthreads();

  if (warp == threads / 32) {  // the producer
    if (lane == 0) {
      MbarExpectTx(tile_bar, tile_bytes);
      const unsigned char* src = reinterpret_cast<const unsigned char*>(a.ranks) + static_cast<int64_t>(blockIdx.x) * tile_bytes;
      for (unsigned at = 0; at < tile_bytes; at += 32768u) BulkCopy(tile0 + at, src + at, min(32768u, tile_bytes - at), tile_bar);
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
      MbarWait(tile_bar, 0, a.status, &s_failed);
      for (int h = max(g - 2, 0); h < g; ++h) MbarWait(full0 + 8 * (a.nbuf == 2 ? h & 1 : 0), (h >> 1) & 1, a.status, &s_failed);
    }
    __syncthreads();
    if (s_failed != 0) {  // (the other warps have written what they have)
      const int columns = a.o.transform == LBK_LOGISTIC ? 2 : 1;
      for (int64_t row = row0 + lane; row < row0 + 2 * threads && row < a.n_rows; row += 32)
        for (int k = 0; k < columns; ++k) a.o.pred[row * a.o.ldp + k] = NAN;
    }
    return;
  }

  const unsigned column = tile0 + tid * 4;  // of the thread's first row; the second row's ranks are two bytes on
  double acc[2] = {0.0, 0.0};
  bool ok = __all_sync(0xffffffffu, MbarWait(tile_bar, 0, a.status, &s_failed) ? 1 : 0) != 0;
  auto rank_of = [&](unsigned word, int r) {
    unsigned v;
    const unsigned at = __dp2a_lo(word, 128u, column);  // column + 128 x the low half
    if (r == 0) asm volatile("{\n.reg .u16 h;\nld.shared.u16 h, [%1];\ncvt.u32.u16 %0, h;\n}\n" : "=r"(v) : "r"(at));
    else asm volatile("{\n.reg .u16 h;\nld.shared.u16 h, [%1+2];\ncvt.u32.u16 %0, h;\n}\n" : "=r"(v) : "r"(at));
    return v;
  };
  // the node's number one level down: negative if the rank is above the split's
  auto down = [](unsigned node, unsigned word, unsigned rank) { return __funnelshift_l(word - (rank << 16), node, 1); };
  for (int g = 0; g < n_groups && ok; ++g) {
    const int b = a.nbuf == 2 ? g & 1 : 0;
    if (!__all_sync(0xffffffffu, MbarWait(full0 + 8 * b, (g >> 1) & 1, a.status, &s_failed) ? 1 : 0)) break;
    const int nt        = min(TG, a.n_trees - g * TG);
    const unsigned base = tree0 + b * buf_bytes;
    auto walk = [&](auto here) {
      unsigned node[TG][2], w[TG][2], x[TG][2];
      {
        uint4 top[TG];
#pragma unroll
        for (int j = 0; j < TG; ++j)
          if (here(j))
            asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];\n" : "=r"(top[j].x), "=r"(top[j].y), "=r"(top[j].z), "=r"(top[j].w) : "r"(base + j * rec_bytes));
#pragma unroll
        for (int j = 0; j < TG; ++j)
          if (here(j)) x[j][0] = LdsU32(column + (top[j].y & 0xffffu) * 128u);
#pragma unroll
        for (int j = 0; j < TG; ++j)
          if (here(j)) {
#pragma unroll
            for (int r = 0; r < 2; ++r) {
              node[j][r] = down(1u, top[j].y, r == 0 ? x[j][0] & 0xffffu : x[j][0] >> 16);
              w[j][r]    = (node[j][r] & 1u) ? top[j].w : top[j].z;
            }
          }
      }
      auto ranks = [&]() {
#pragma unroll
        for (int j = 0; j < TG; ++j)
          if (here(j)) {
            x[j][0] = rank_of(w[j][0], 0);
            x[j][1] = rank_of(w[j][1], 1);
          }
      };
      auto descend = [&]() {
#pragma unroll
        for (int j = 0; j < TG; ++j)
          if (here(j)) {
            node[j][0] = down(node[j][0], w[j][0], x[j][0]);
            node[j][1] = down(node[j][1], w[j][1], x[j][1]);
          }
      };
      ranks();
      descend();
#pragma unroll 1
      for (int l = 2; l < S; ++l) {
#pragma unroll
        for (int j = 0; j < TG; ++j)
          if (here(j)) {
            w[j][0] = LdsU32(base + j * rec_bytes + 4u * node[j][0]);
            w[j][1] = LdsU32(base + j * rec_bytes + 4u * node[j][1]);
          }
        ranks();
        descend();
      }
      // leaf i of the bottom level is node 2^S + i: its value lies at 4 * 2^S + 8 i
      double v[TG][2];
#pragma unroll
      for (int j = 0; j < TG; ++j)
        if (here(j)) {
          v[j][0] = LdsF64(base + j * rec_bytes - (4u << S) + 8u * node[j][0]);
          v[j][1] = LdsF64(base + j * rec_bytes - (4u << S) + 8u * node[j][1]);
        }
#pragma unroll
      for (int j = 0; j < TG; ++j)
        if (here(j)) {
          acc[0] += v[j][0];
          acc[1] += v[j][1];
        }
    };
    if (nt == TG) walk([](int) { return true; });
    else walk([&](int j) { return j < nt; });
    __syncwarp();
    if (lane == 0) MbarArrive(empty0 + 8 * b);  // this warp is done with the buffer
  }
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    const int64_t row = row0 + r * threads + tid;
    const double raw  = a.o.init ? a.o.init[0] + acc[r] : acc[r];
    if (row < a.n_rows) FinishRow(&raw, 1, 1, a.o.pred + row * a.o.ldp, a.o.transform);
  }
  __syncthreads();  // (the producer's copies)
}

constexpr int kRankedStatic = 256;  // a bound of what k_predict_ranked declares itself

// Threads and trees per group: what is in flight is threads x trees x 2 walks.
struct RankedPlan {
  int threads = 0, tg = 0, nbuf = 0;
  size_t smem = 0;
};
RankedPlan PlanRanked(const lbk_context* ctx, int F, int n_trees, int S)
{
  RankedPlan best;
  int best_score = 0;
  const size_t room = static_cast<size_t>(ctx->max_smem_optin) - kRankedStatic;
  for (int tg = 4; tg >= 1; tg /= 2) {
    if (tg > n_trees && tg > 1) continue;
    const int nbuf     = n_trees > tg ? 2 : 1;
    const size_t trees = static_cast<size_t>(nbuf) * tg * RankRecordBytes(S);
    if (trees + static_cast<size_t>(F) * 128 > room) continue;
    const int threads = static_cast<int>(std::min<size_t>((room - trees) / (static_cast<size_t>(F) * 4), kWalkThreads) / 32 * 32);
    const int score   = threads * tg;
    if (score <= best_score) continue;
    best_score = score;
    best       = RankedPlan{threads, tg, nbuf, static_cast<size_t>(F) * threads * 4 + trees};
  }
  return best;
}

}  // namespace

constexpr size_t kRankBytes = size_t{256} << 20;  // of a piece of the rows

template <typename T>
bool PredictRanked(lbk_context* ctx, Scratch& s, const T* X, int64_t ldx, int64_t n_rows, int F, int n_trees, const lbk_tree_ref* d_trees, int S,
                   int64_t total_nodes, const double* init, int transform, double* pred, int64_t ldp, cudaStream_t stream)
{
  if (S < 3 || S > 12 || F > 1024 || total_nodes > (int64_t{1} << 28)) return false;
  const RankedPlan plan = PlanRanked(ctx, F, n_trees, S);
  if (plan.threads < 128) return false;
  // rows are walked in whole waves of tiles
  const int64_t tile    = 2 * plan.threads;
  const int64_t wave    = tile * ctx->sm_count;
  const int64_t waves   = std::max<int64_t>(1, static_cast<int64_t>(kRankBytes / (static_cast<size_t>(wave) * F * 2)));
  const int64_t piece   = std::min(waves * wave, (n_rows + tile - 1) / tile * tile);
  // one piece of scratch, so that a call which has no room for it is left as it was: it takes the other path
  size_t bytes = 0;
  auto reserve = [&](size_t n) {
    const size_t at = bytes;
    bytes += (n + 255) / 256 * 256;
    return at;
  };
  const size_t nodes = static_cast<size_t>(total_nodes), words_bytes = sizeof(int) * (2 * static_cast<size_t>(F) + 1);
  const size_t o_words = reserve(words_bytes), o_off = reserve(sizeof(int) * (static_cast<size_t>(F) + 1));
  const size_t o_lists = reserve(nodes * sizeof(T)), o_cuts = reserve(nodes * sizeof(T)), o_lut = reserve(nodes * sizeof(unsigned));
  const size_t o_tables = reserve(sizeof(RankTable) * F), o_records = reserve(static_cast<size_t>(n_trees) * RankRecordBytes(S));
  const size_t o_ranks  = reserve(static_cast<size_t>(piece / 2) * F * sizeof(unsigned));
  unsigned char* room   = nullptr;
  try {
    room = static_cast<unsigned char*>(s.alloc_bytes(bytes));
  } catch (const Error& e) {
    if (e.code != LBK_ERR_ALLOC) throw;
    return false;
  }
  int* words             = reinterpret_cast<int*>(room + o_words);  // counts, cursors, too many
  int* too_many          = words + 2 * F;
  int* off               = reinterpret_cast<int*>(room + o_off);
  T* lists               = reinterpret_cast<T*>(room + o_lists);
  T* cuts                = reinterpret_cast<T*>(room + o_cuts);
  unsigned* lut          = reinterpret_cast<unsigned*>(room + o_lut);
  RankTable* tables      = reinterpret_cast<RankTable*>(room + o_tables);
  unsigned char* records = room + o_records;
  unsigned* ranks        = reinterpret_cast<unsigned*>(room + o_ranks);
  LBK_CUDA(cudaMemsetAsync(words, 0, words_bytes, stream));
  k_rank_count<T><<<n_trees, 256, 0, stream>>>(d_trees, F, words);
  LBK_LAUNCH_CHECK();
  k_rank_scatter<T><<<n_trees, 256, 0, stream>>>(d_trees, F, words, words + F, off, lists);
  LBK_LAUNCH_CHECK();
  AllowSharedMemory(ctx, k_rank_tables<T>, 1024);
  k_rank_tables<T><<<F, 1024, kSortChunk * sizeof(T), stream>>>(off, lists, cuts, lut, tables, too_many);
  LBK_LAUNCH_CHECK();
  k_rank_pack<T><<<n_trees, 256, 0, stream>>>(d_trees, F, S, plan.threads / 32, tables, cuts, lut, too_many, records);
  LBK_LAUNCH_CHECK();
  AllowSharedMemory(ctx, k_rank_rows<T>, 1024);
  const int groups = (F + 31) / 32;
  int lanes        = 16;  // (no less: rows of few features are bound by the sectors an SM can have on their way)
  while (lanes < F - 32 * (groups - 1)) lanes *= 2;
  const int blocks      = std::max(ctx->sm_count, groups);
  const int tail_blocks = groups == 1 ? blocks
                                      : std::min(blocks - (groups - 1), std::max(1, (blocks * lanes + 16 * (groups - 1) + lanes / 2) / (32 * (groups - 1) + lanes)));
  auto walk = plan.tg == 4 ? k_predict_ranked<T, 4> : plan.tg == 2 ? k_predict_ranked<T, 2> : k_predict_ranked<T, 1>;
  AllowSharedMemory(ctx, walk, kRankedStatic);
  const size_t rank_smem = static_cast<size_t>(ctx->max_smem_optin) - 1024;
  for (int64_t r0 = 0; r0 < n_rows; r0 += piece) {
    const int64_t rows = std::min(piece, n_rows - r0), tiles = (rows + tile - 1) / tile;
    RankRowsArgs<T> ra{X + r0 * ldx, ldx, rows, F, plan.threads, tiles, tables, cuts, lut, too_many, ranks, tail_blocks};
    k_rank_rows<T><<<blocks, kRankThreads, rank_smem, stream>>>(ra);
    LBK_LAUNCH_CHECK();
    RankedArgs<T> wa{X + r0 * ldx, ldx, rows, F, n_trees, S, plan.nbuf, ranks, records, d_trees, too_many, PredictOut{pred + r0 * ldp, ldp, init, transform}, ctx->d_status};
    walk<<<static_cast<unsigned>(tiles), plan.threads + 32, plan.smem, stream>>>(wa);
    LBK_LAUNCH_CHECK();
  }
  return true;
}

template bool PredictRanked<float>(lbk_context*, Scratch&, const float*, int64_t, int64_t, int, int, const lbk_tree_ref*, int, int64_t,
                                   const double*, int, double*, int64_t, cudaStream_t);
template bool PredictRanked<double>(lbk_context*, Scratch&, const double*, int64_t, int64_t, int, int, const lbk_tree_ref*, int, int64_t,
                                    const double*, int, double*, int64_t, cudaStream_t);

}  // namespace lbk
