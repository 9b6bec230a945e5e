// Ensemble predict on ranks: x <= split as a comparison of whole numbers.
//
// A walk only compares x[f] with the splits on feature f.  With the ensemble's splits on every feature sorted, x[f] may be
// replaced by its rank among them (how many are smaller), and a split by its own: x <= split if and only if rank(x) <=
// rank(split).  Ranks fit 16 bits, so that a node - rank and feature - is one 4-byte word for float32 and float64 alike, and
// the values of two rows share a word of shared memory.  That is worth a pass over X which finds the ranks as soon as the
// ensemble is large enough (RanksPay): the walks are bound by the load/store data pipe of the SM, and a level is two
// passes (node, rank) plus bank conflicts, where k_predict_tiled takes two and a half (float32: split, value, half a
// word of ids) or five (float64).  Measured against that kernel: 10M x 100 float32, 500 trees of depth 8: 19.3 -> 13.4 ms (2.4
// of it for the ranks); 1M x 64 float64, 100 trees: 807 -> 525 us (170 for the ranks, 65 for the tables and records).
//
// Launches:
//   k_rank_count, k_rank_scatter   the ensemble's splits, feature by feature
//   k_rank_sort                    sorted, up to kSortChunk of a feature by a block; an index by value into them
//   k_rank_merge                   features of more than that: the chunks as one table with its index
//   k_rank_pack                    is it worth it, with the tables as they are?  The trees' records, completed to one depth as for
//                                  k_predict_tiled
// then for pieces of the rows that bound the memory of their ranks:
//   k_rank_rows                    X -> ranks, in the order of the walking blocks' tiles
//   k_predict_ranked               the walks
//
// Boosted ensembles put most splits on a few features, which the host does not see.  A feature with more values than ranks, or
// tables so uneven that they are searched in many turns over the rows, is known when the tables are made: a device word
// (`declined`) then turns the kernels that follow into nothing, and the path for every other call, queued behind the same
// word, runs instead.  1M x 100 float32, 500 trees of depth 8 with 25 % of the splits on one feature: 35.4 ms when every block
// walked X and the trees where they lie, 2.22 now, 2.13 by k_predict_tiled alone (4M rows: 142, 8.22, 8.06).
//
// One output.  Sums are made in tree order in float64, as everywhere.
#include "predict.cuh"

namespace lbk {
namespace {

constexpr int kMaxRank      = 32764;  // entries of a feature's table: ranks 1 .. 32765, one more for a NaN, below 2^15
constexpr int kSortChunk    = 4096;   // values that a block sorts
constexpr int kSortThreads  = 1024;
constexpr int kMaxChunks    = 32;     // of a feature; with more the ranks are declined unseen
constexpr int kMaxFeatures  = 1024;
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

// Splits of a tree by feature, in shared memory [kMaxFeatures] (global atomics of every node took 28 us for 500 trees of depth 8).
template <typename T>
__device__ inline void CountSplits(const TreePtrs& t, int F, int* s_n)
{
  for (int f = threadIdx.x; f < F; f += blockDim.x) s_n[f] = 0;
  __syncthreads();
  for (int i = threadIdx.x; i < t.max_nodes; i += blockDim.x) {
    int f;
    T cut;
    if (SplitAt(t, i, F, f, cut) && cut == cut) atomicAdd(s_n + f, 1);
  }
  __syncthreads();
}

template <typename T>
__global__ void __launch_bounds__(256) k_rank_count(const TreePtrs* __restrict__ trees, int F, int* __restrict__ counts)
{
  AfterTheKernelBefore();
  __shared__ int s_n[kMaxFeatures];
  CountSplits<T>(trees[blockIdx.x], F, s_n);
  for (int f = threadIdx.x; f < F; f += blockDim.x)
    if (s_n[f] != 0) atomicAdd(counts + f, s_n[f]);
}

// Exclusive prefix sums of four values per thread of a block of 256; returns what is before the thread's first one.
__device__ inline int BlockPrefix4(const int (&c)[4], int* s_wsum /* [8] */)
{
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int sum = c[0] + c[1] + c[2] + c[3];
  int incl = sum;
  for (int o = 1; o < 32; o <<= 1) {
    const int v = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += v;
  }
  __syncthreads();
  if (lane == 31) s_wsum[warp] = incl;
  __syncthreads();
  int before = incl - sum;
  for (int w = 0; w < warp; ++w) before += s_wsum[w];
  return before;
}

__host__ __device__ inline int ChunksOf(int n) { return n > kSortChunk ? (n + kSortChunk - 1) / kSortChunk : 1; }

// off [F + 1]: where each feature's values begin in `lists`; items [*n_items]: (feature, chunk), the chunks of a feature one after
// the other, at most kMaxChunks of them (more values: *declined).
template <typename T>
__global__ void __launch_bounds__(256)
  k_rank_scatter(const TreePtrs* __restrict__ trees, int F, const int* __restrict__ counts, int* __restrict__ cursor, int* __restrict__ off,
                 int2* __restrict__ items, int* __restrict__ n_items, int* __restrict__ declined, T* __restrict__ lists)
{
  AfterTheKernelBefore();
  constexpr int kPer = kMaxFeatures / 256;
  __shared__ int s_n[kMaxFeatures], s_at[kMaxFeatures], s_wsum[8];
  const int tid = threadIdx.x;
  int c[kPer], chunks[kPer];
#pragma unroll
  for (int i = 0; i < kPer; ++i) {
    const int f = tid * kPer + i;
    c[i]        = f < F ? counts[f] : 0;
    chunks[i]   = f < F ? ChunksOf(c[i]) : 0;
  }
  int before = BlockPrefix4(c, s_wsum);
#pragma unroll
  for (int i = 0; i < kPer; ++i) {
    const int f = tid * kPer + i;
    s_at[f]     = before;
    if (blockIdx.x == 0 && f < F) off[f] = before;
    before += c[i];
    if (blockIdx.x == 0 && f == F - 1) off[F] = before;
  }
  if (blockIdx.x == 0) {
#pragma unroll
    for (int i = 0; i < kPer; ++i)
      if (chunks[i] > kMaxChunks) {
        *declined = 1;
        chunks[i] = 1;
      }
    int at = BlockPrefix4(chunks, s_wsum);
#pragma unroll
    for (int i = 0; i < kPer; ++i) {
      for (int q = 0; q < chunks[i]; ++q) items[at++] = make_int2(tid * kPer + i, q);
      if (tid * kPer + i == F - 1) *n_items = at;
    }
  }
  const TreePtrs t = trees[blockIdx.x];
  CountSplits<T>(t, F, s_n);
  for (int f = tid; f < F; f += blockDim.x)
    if (s_n[f] != 0) s_at[f] += atomicAdd(cursor + f, s_n[f]);
  __syncthreads();
  for (int i = tid; i < t.max_nodes; i += blockDim.x) {
    int f;
    T cut;
    if (SplitAt(t, i, F, f, cut) && cut == cut) lists[atomicAdd(s_at + f, 1)] = cut;
  }
}

// The first index of n sorted values that is not below v.
template <typename T>
__device__ inline int LowerBound(const T* a, int n, T v)
{
  int lo = 0;
  while (n > 0) {
    const int half = n >> 1;
    if (a[lo + half] < v) {
      lo += half + 1;
      n -= half + 1;
    } else {
      n = half;
    }
  }
  return lo;
}

// How many of each of kAbreast chunks come before v: those below it and, in the chunks before number `upto`, those equal to it.  In steps of
// falling powers of two; the chunks' loads are on their way together (a lone search is twelve of them, one after the other).
constexpr int kAbreast = 8;
template <typename T>
__device__ inline void CountBefore(const T* lists, const int* len, int first, int chunks, int upto, T v, int (&pos)[kAbreast])
{
#pragma unroll
  for (int u = 0; u < kAbreast; ++u) pos[u] = 0;
#pragma unroll 1
  for (int h = kSortChunk; h > 0; h >>= 1) {
    T x[kAbreast];
#pragma unroll
    for (int u = 0; u < kAbreast; ++u) {
      const int n = first + u < chunks ? len[first + u] : 0;
      x[u]        = pos[u] + h <= n ? lists[(first + u) * kSortChunk + pos[u] + h - 1] : static_cast<T>(NAN);
    }
#pragma unroll
    for (int u = 0; u < kAbreast; ++u)
      if (x[u] < v || (first + u < upto && x[u] == v)) pos[u] += h;
  }
}

// What the tables are made from and of.
template <typename T>
struct RankTables {
  const int* off;
  const int2* items;
  const int* n_items;
  int* len;           // [items] distinct values of a chunk
  int* arrived;       // [F] blocks of k_rank_merge that are done with a feature
  T* lists;           // [values] as scattered; then the sorted chunks
  T* cuts;            // [values] the tables
  unsigned* lut;      // [values] of a bucket: its first value, and in the high half how many it has
  RankTable* tables;  // [F]
  int* declined;
};

// Buckets of equal width between the first and the last finite value.
template <typename T>
__device__ inline RankTable IndexOf(T first, T last, int off, int m)
{
  constexpr float kMax = 3.402823466e38f;
  RankTable t{0.f, 0.f, off, m, max(m, 1)};
  if (m > 0) {
    t.lo           = fmaxf(static_cast<float>(first), -kMax);
    const float hi = fminf(static_cast<float>(last), kMax);
    t.scale        = hi > t.lo ? static_cast<float>(t.nb) / (hi - t.lo) : 0.f;
  }
  return t;
}
// (memory of the block, or what other blocks may have written)
__device__ inline float ValueAt(const float* p) { return __isShared(p) ? *p : __ldcg(p); }
__device__ inline double ValueAt(const double* p) { return __isShared(p) ? *p : __ldcg(p); }

// The index of a table whose values lie in `out`, by a block.  start [m]: scratch, first value of every bucket.
template <typename T, typename Start>
__device__ inline void MakeIndex(const RankTable& t, const T* out, Start* start, unsigned* lut)
{
#pragma unroll 4
  for (int i = threadIdx.x; i < t.m; i += kSortThreads) {
    const int b = RankBucket(static_cast<float>(ValueAt(out + i)), t.lo, t.scale, t.nb);
    const int a = i > 0 ? RankBucket(static_cast<float>(ValueAt(out + i - 1)), t.lo, t.scale, t.nb) : -1;
    for (int q = a + 1; q <= b; ++q) start[q] = static_cast<Start>(i);
    if (i == t.m - 1)
      for (int q = b + 1; q < t.nb; ++q) start[q] = static_cast<Start>(t.m);
  }
  __syncthreads();
#pragma unroll 4
  for (int b = threadIdx.x; b < t.m; b += kSortThreads) {
    const int first = static_cast<int>(start[b]), next = b + 1 < t.m ? static_cast<int>(start[b + 1]) : t.m;
    lut[b]          = static_cast<unsigned>(first) | (static_cast<unsigned>(next - first) << 16);
  }
}

// The threads' values that are to be kept, in order, to dst + kept; returns kept and how many there are.
template <typename T>
__device__ inline int KeepInOrder(bool keep, T v, T* dst, int kept, int* s_wsum /* [kSortThreads / 32] */)
{
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const unsigned b = __ballot_sync(0xffffffffu, keep);
  if (lane == 0) s_wsum[warp] = __popc(b);
  __syncthreads();
  const int n = s_wsum[lane];  // (as many warps as lanes)
  int incl    = n;
  for (int o = 1; o < 32; o <<= 1) {
    const int x = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += x;
  }
  const int before = __shfl_sync(0xffffffffu, incl - n, warp);
  if (keep) dst[kept + before + __popc(b & ((1u << lane) - 1u))] = v;
  kept += __shfl_sync(0xffffffffu, incl, 31);
  __syncthreads();
  return kept;
}
static_assert(kSortThreads == 1024, "KeepInOrder: as many warps as lanes");

template <typename T>
__device__ inline void ExchangeLanes(T& v, int j, bool up)
{
  const T o = __shfl_xor_sync(0xffffffffu, v, j);
  if (((threadIdx.x & j) == 0) == up ? o < v : v < o) v = o;
}
template <typename T>
__device__ inline void ExchangePair(T& a, T& b, bool up)
{
  if (up ? b < a : a < b) {
    const T t = a;
    a         = b;
    b         = t;
  }
}

// P values in shared memory (a power of two, 64 or more), by a bitonic network.  A warp takes 64 neighbours and makes the steps that
// stay among them in registers: of 2048 values 15 steps of 66 go through shared memory (all of them: 22 us, float64).
template <typename T>
__device__ inline void SortShared(T* s, int P)
{
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  __syncthreads();
  for (int q = warp; 64 * q < P; q += kSortThreads / 32) {
    T a = s[64 * q + lane], b = s[64 * q + 32 + lane];
#pragma unroll
    for (int k = 2; k <= 32; k <<= 1)
#pragma unroll
      for (int j = k >> 1; j > 0; j >>= 1) {
        ExchangeLanes(a, j, k == 32 || (lane & k) == 0);
        ExchangeLanes(b, j, k != 32 && (lane & k) == 0);
      }
    const bool up = (q & 1) == 0;
    ExchangePair(a, b, up);
#pragma unroll
    for (int j = 16; j > 0; j >>= 1) {
      ExchangeLanes(a, j, up);
      ExchangeLanes(b, j, up);
    }
    s[64 * q + lane]      = a;
    s[64 * q + 32 + lane] = b;
  }
  for (int k = 128; k <= P; k <<= 1) {
    for (int j = k >> 1; j >= 64; j >>= 1) {
      __syncthreads();
      for (int e = tid; e < P / 2; e += kSortThreads) {
        const int i = 2 * e - (e & (j - 1));  // the e-th index without bit j
        T a = s[i], b = s[i + j];
        ExchangePair(a, b, (i & k) == 0);
        s[i]     = a;
        s[i + j] = b;
      }
    }
    __syncthreads();
    for (int q = warp; 64 * q < P; q += kSortThreads / 32) {
      T a = s[64 * q + lane], b = s[64 * q + 32 + lane];
      const bool up = (64 * q & k) == 0;
      ExchangePair(a, b, up);
#pragma unroll
      for (int j = 16; j > 0; j >>= 1) {
        ExchangeLanes(a, j, up);
        ExchangeLanes(b, j, up);
      }
      s[64 * q + lane]      = a;
      s[64 * q + 32 + lane] = b;
    }
  }
  __syncthreads();
}

// The values of a chunk in order, by as many buckets of equal width: counted, scattered, and put where they belong in their bucket, each
// by the number of its values that come before it.  False, with the values in another order, where more than kSortBucket share a
// bucket and are not all equal (columns of few values have splits that are).  start: scratch.  k_rank_sort of 64 features of 170 to
// 2000 float64 values: 29 us by the network, 12; of 100 features, float32, 27 and 12.  (A bucket put in order by one thread is a chain
// of 100 dependent steps where it is full, and full ones are neighbours: 64 features of 400 lognormal values 36 us, by the network 11, now 12.)
constexpr int kSortBucket = 24;
template <typename T>
__device__ inline bool SortByBuckets(T* s, unsigned* start /* [kSortChunk / 2]: two of 16 bits */, int* s_wsum, float2* s_range /* [32] */, int len)
{
  constexpr int kPer = kSortChunk / kSortThreads;
  static_assert(kPer == 4, "two words of counts a thread");
  constexpr float kMax = 3.402823466e38f;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  T v[kPer];
  float lo = kMax, hi = -kMax;
  reinterpret_cast<uint2*>(start)[tid] = make_uint2(0u, 0u);
#pragma unroll
  for (int u = 0; u < kPer; ++u) {
    const int i = tid + u * kSortThreads;
    v[u]        = i < len ? s[i] : T(0);
    if (i < len) {
      const float x = fminf(fmaxf(static_cast<float>(v[u]), -kMax), kMax);
      lo            = fminf(lo, x);
      hi            = fmaxf(hi, x);
    }
  }
  auto range_of_warp = [&]() {
    for (int o = 16; o > 0; o >>= 1) {
      lo = fminf(lo, __shfl_xor_sync(0xffffffffu, lo, o));
      hi = fmaxf(hi, __shfl_xor_sync(0xffffffffu, hi, o));
    }
  };
  range_of_warp();
  if (lane == 0) s_range[warp] = make_float2(lo, hi);
  __syncthreads();
  lo = s_range[lane].x;
  hi = s_range[lane].y;
  range_of_warp();
  const float scale = hi > lo ? static_cast<float>(len) / (hi - lo) : 0.f;
  int bucket[kPer], before[kPer], count[kPer];  // of each value: its bucket (then that one's first place), who came before, how many are in it
#pragma unroll
  for (int u = 0; u < kPer; ++u) {
    bucket[u] = RankBucket(static_cast<float>(v[u]), lo, scale, len);
    before[u] = count[u] = 0;
    if (tid + u * kSortThreads < len) {
      const int shift = 16 * (bucket[u] & 1);
      before[u]       = static_cast<int>(atomicAdd(start + (bucket[u] >> 1), 1u << shift) >> shift & 0xffffu);
    }
  }
  __syncthreads();
  // counts become first places
  const uint2 c  = reinterpret_cast<uint2*>(start)[tid];
  const int n[4] = {static_cast<int>(c.x & 0xffffu), static_cast<int>(c.x >> 16), static_cast<int>(c.y & 0xffffu), static_cast<int>(c.y >> 16)};
  int incl       = n[0] + n[1] + n[2] + n[3];
  const int own  = incl;
  for (int o = 1; o < 32; o <<= 1) {
    const int x = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += x;
  }
  if (lane == 31) s_wsum[warp] = incl;
  __syncthreads();
  int sums = s_wsum[lane];
  for (int o = 1; o < 32; o <<= 1) {
    const int x = __shfl_up_sync(0xffffffffu, sums, o);
    if (lane >= o) sums += x;
  }
  const int below_warp = __shfl_sync(0xffffffffu, sums, max(warp - 1, 0));
  int at[4];
  at[0] = incl - own + (warp > 0 ? below_warp : 0);
#pragma unroll
  for (int k = 1; k < 4; ++k) at[k] = at[k - 1] + n[k - 1];
  reinterpret_cast<uint2*>(start)[tid] = make_uint2(at[0] | at[1] << 16, at[2] | at[3] << 16);
  __syncthreads();
  auto first_of = [&](int b) { return static_cast<int>(start[b >> 1] >> (16 * (b & 1)) & 0xffffu); };
#pragma unroll
  for (int u = 0; u < kPer; ++u)
    if (tid + u * kSortThreads < len) {
      const int b = bucket[u], next = b + 1 < kSortChunk ? first_of(b + 1) : len;
      bucket[u]   = first_of(b);
      count[u]    = next - bucket[u];
      s[bucket[u] + before[u]] = v[u];
    }
  __syncthreads();
  bool crowded = false;
#pragma unroll
  for (int u = 0; u < kPer; ++u)
    if (count[u] > kSortBucket) crowded = crowded || s[bucket[u]] != v[u];
  if (__syncthreads_or(crowded)) return false;
#pragma unroll
  for (int u = 0; u < kPer; ++u) {
    const int own = before[u];
    if (count[u] > 1 && count[u] <= kSortBucket) {
      before[u] = 0;
#pragma unroll 4
      for (int i = 0; i < count[u]; ++i) {
        const T x = s[bucket[u] + i];
        before[u] += x < v[u] || (x == v[u] && i < own) ? 1 : 0;
      }
    }
  }
  __syncthreads();
#pragma unroll
  for (int u = 0; u < kPer; ++u)
    if (count[u] > 1) s[bucket[u] + before[u]] = v[u];
  __syncthreads();
  return true;
}

// A block per chunk: its values sorted, equal ones once.  A feature of one chunk has its table then.
template <typename T>
__global__ void __launch_bounds__(kSortThreads) k_rank_sort(const RankTables<T> a)
{
  AfterTheKernelBefore();
  __shared__ T s[kSortChunk];
  __shared__ __align__(8) unsigned s_start[kSortChunk / 2];
  __shared__ int s_wsum[kSortThreads / 32];
  __shared__ float2 s_range[kSortThreads / 32];
  if (*a.declined != 0 || static_cast<int>(blockIdx.x) >= *a.n_items) return;
  const int2 item = a.items[blockIdx.x];
  const int f = item.x, tid = threadIdx.x;
  const int begin = a.off[f], n = a.off[f + 1] - begin, c0 = item.y * kSortChunk, len = min(kSortChunk, n - c0);
  T* list = a.lists + begin + c0;
  int P   = 64;
  while (P < len) P <<= 1;
  for (int i = tid; i < P; i += kSortThreads) s[i] = i < len ? list[i] : static_cast<T>(INFINITY);
  __syncthreads();
  if (!SortByBuckets(s, s_start, s_wsum, s_range, len)) SortShared(s, P);
  // (kept values move to the front, never beyond what has been read)
  int m = 0;
  for (int i0 = 0; i0 < len; i0 += kSortThreads) {
    const int i     = i0 + tid;
    const bool keep = i < len && (i == 0 || s[i] != s[i - 1]);
    m               = KeepInOrder(keep, keep ? s[i] : T(0), s, m, s_wsum);
  }
  const bool alone = ChunksOf(n) == 1;
  T* dst           = alone ? a.cuts + begin : list;
  for (int i = tid; i < m; i += kSortThreads) dst[i] = s[i];
  if (tid == 0) a.len[blockIdx.x] = m;
  if (!alone) return;
  const RankTable t = IndexOf(m > 0 ? s[0] : T(0), m > 0 ? s[m - 1] : T(0), begin, m);
  MakeIndex(t, s, reinterpret_cast<uint16_t*>(s_start), a.lut + begin);
  if (tid == 0) a.tables[f] = t;
}

// Features of several chunks.  Every value goes to its place among all of them: its own in its chunk, and how many of each other
// chunk come before it (equal values in the order of the chunks).  The last block that is done with a feature then drops equal values
// and makes the index.  A feature with more distinct values than ranks sets *declined.
template <typename T>
__global__ void __launch_bounds__(kSortThreads) k_rank_merge(const RankTables<T> a)
{
  AfterTheKernelBefore();
  __shared__ int s_len[kMaxChunks], s_wsum[kSortThreads / 32];
  __shared__ bool s_last;
  if (__syncthreads_or(*reinterpret_cast<volatile int*>(a.declined)) || static_cast<int>(blockIdx.x) >= *a.n_items) return;  // (all threads or none)
  const int2 item = a.items[blockIdx.x];
  const int f = item.x, tid = threadIdx.x;
  const int begin = a.off[f], chunks = ChunksOf(a.off[f + 1] - begin), first = blockIdx.x - item.y;
  if (chunks == 1) return;
  const T* src = a.lists + begin;
  T* out       = a.cuts + begin;
  for (int o = tid; o < chunks; o += kSortThreads) s_len[o] = a.len[first + o];
  __syncthreads();
  int all = 0;
  for (int o = 0; o < chunks; ++o) all += s_len[o];
  // More than there are ranks, and so few of them twice in a chunk (one in 32: values drawn from 65 thousand) that they will not be
  // few enough once those of several chunks are dropped: declined now, before 50 us of placing and dropping.
  if (all > kMaxRank && (a.off[f + 1] - begin - all) * 32 < a.off[f + 1] - begin) {
    if (tid == 0) *a.declined = 1;
    return;
  }
  const int own = blockIdx.y * kSortThreads + tid;  // (a value per thread)
  if (own < s_len[item.y]) {
    const T v = src[item.y * kSortChunk + own];
    int at    = own;
    for (int o0 = 0; o0 < chunks; o0 += kAbreast) {
      int pos[kAbreast];
      CountBefore(src, s_len, o0, chunks, item.y, v, pos);
#pragma unroll
      for (int u = 0; u < kAbreast; ++u)
        if (o0 + u != item.y) at += pos[u];
    }
    out[at] = v;
  }
  __threadfence();
  __syncthreads();
  if (tid == 0) s_last = atomicAdd(a.arrived + f, 1) == chunks * static_cast<int>(gridDim.y) - 1;
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  // (kept values move to the front, never beyond what has been read; the next ones are on their way)
  int m   = 0;
  T ahead = __ldcg(out + min(tid, all - 1)), ahead_before = __ldcg(out + max(min(tid, all - 1) - 1, 0));
  for (int i0 = 0; i0 < all; i0 += kSortThreads) {
    const int i     = i0 + tid, next = min(i + kSortThreads, all - 1);
    const T v       = ahead;
    const bool keep = i < all && (i == 0 || v != ahead_before);
    ahead           = __ldcg(out + next);
    ahead_before    = __ldcg(out + next - 1);
    m               = KeepInOrder(keep, v, out, m, s_wsum);
  }
  if (m > kMaxRank) {
    if (tid == 0) *a.declined = 1;
    return;
  }
  const RankTable t = IndexOf(__ldcg(out), __ldcg(out + m - 1), begin, m);
  MakeIndex(t, out, reinterpret_cast<int*>(a.lists + begin), a.lut + begin);
  if (tid == 0) a.tables[f] = t;
}

// ---- turns of k_rank_rows, and what they cost ---------------------------------------------------
// Bytes of shared memory of the tables of `entries` values.
template <typename T>
__host__ __device__ inline unsigned TableBytes(int entries)
{
  return static_cast<unsigned>((entries + 1) / 2 * 2) * 4u + static_cast<unsigned>(entries) * sizeof(T);
}
// The features of a group that a turn from w0 on takes, those up to the result: as many as have room for their tables; a power
// of two of them but at the end.  begin [width + 1]: entries before each feature.
template <typename T>
__host__ __device__ inline int TurnEnd(const int* begin, int w0, int width, unsigned room)
{
  int w1 = w0 + 1;
  while (w1 < width && TableBytes<T>(begin[w1 + 1] - begin[w0]) <= room) ++w1;
  if (w1 < width) {
    int n = 1;
    while (2 * n <= w1 - w0) n *= 2;
    w1 = w0 + n;
  }
  return w1;
}
// Shares of k_rank_rows' blocks: those of a last group of fewer than 32 features stand for this many lanes.  (No less than 16: rows of
// few features are bound by the sectors that an SM can have on their way.)
__host__ __device__ inline int TailLanes(int F)
{
  int lanes = 16;
  while (lanes < F - 32 * ((F + 31) / 32 - 1)) lanes *= 2;
  return lanes;
}

// Microseconds that k_rank_rows takes for group g of F features, as its tables are.  Per million rows and with all SMs: kLane of a
// turn per lane that a row takes (of less than eight the loads of a step are not all used), kGlobal for a table that is
// searched where it lies, kAgain for every turn but the first where rows have more than one group (what they share of a
// line is gone by then).  kFill per entry brought to shared memory.  Fitted to 154 (float32) and 145 (float64) ensembles of 4 to
// 511 trees of depth 3 to 10 on 6 to 236 features, up to all splits on one of them, and 80 thousand to 6 million rows: 9 and 13 %
// off (rms).
template <typename T>
struct RowsCost {
  static constexpr float kLane = sizeof(T) == 4 ? 2.2f : 2.77f, kGlobal = sizeof(T) == 4 ? 15.f : 22.f, kAgain = sizeof(T) == 4 ? 15.6f : 12.f;
  static constexpr float kFill = sizeof(T) == 4 ? 0.5e-3f : 0.6e-3f, kLaunch = 8.5f;
  __host__ __device__ static float Group(const int* begin, int g, int F, unsigned room, float millions)
  {
    const int last = (F + 31) / 32 - 1, width = g < last ? 32 : F - 32 * last, tail = TailLanes(F);
    float per_million = 0.f, filled = 0.f;
    for (int w0 = 0, w1; w0 < width; w0 = w1) {
      w1 = TurnEnd<T>(begin, w0, width, room);
      int lanes = 8;
      while (lanes < w1 - w0) lanes *= 2;
      per_million += kLane * static_cast<float>(lanes) + (w0 > 0 && last > 0 ? kAgain : 0.f);
      const int entries = begin[w1] - begin[w0];
      if (TableBytes<T>(entries) <= room) filled += static_cast<float>(entries);
      else per_million += kGlobal;
    }
    const float sms = last == 0 ? 1.f : static_cast<float>(32 * last + tail) / static_cast<float>(g == last ? tail : 32);
    return millions * sms * per_million + kFill * filled + kLaunch;
  }
};

// A completed tree of depth S: words [2^S], nodes counted from 1 (the children of i are 2 i and 2 i + 1), then leaf values
// [2^S].  A word holds the split's rank in its high half (0: nothing passes, a NaN) and, in its low half, where the
// feature's ranks begin in a walking block's tile, in units of 128 bytes.
__host__ __device__ inline int RankRecordBytes(int S) { return 12 << S; }

// Every block finds out for itself, from all tables, whether finding the ranks of `millions` of rows stays within `budget` microseconds
// (millions 0: it does).
template <typename T>
__global__ void __launch_bounds__(256)
  k_rank_pack(const TreePtrs* __restrict__ trees, int F, int S, int lines, float millions, float budget, unsigned room, const RankTable* __restrict__ tables,
              const T* __restrict__ cuts, const unsigned* __restrict__ lut, int* __restrict__ declined, unsigned char* __restrict__ records)
{
  AfterTheKernelBefore();
  // (a feature has no table; or another block has found the same as this one would: all threads or none)
  if (__syncthreads_or(*reinterpret_cast<volatile int*>(declined))) return;
  __shared__ int s_begin[8][33];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  float most = 0.f;
  for (int g = warp; millions > 0.f && 32 * g < F; g += 8) {
    const int width = min(32, F - 32 * g);
    int incl        = lane < width ? tables[32 * g + lane].nb : 0;
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += v;
    }
    __syncwarp();
    s_begin[warp][lane + 1] = incl;
    if (lane == 0) s_begin[warp][0] = 0;
    __syncwarp();
    most = fmaxf(most, RowsCost<T>::Group(s_begin[warp], g, F, room, millions));
  }
  if (__syncthreads_or(most > budget)) {
    if (blockIdx.x == 0 && threadIdx.x == 0) *declined = 1;
    return;
  }
  const TreePtrs t   = trees[blockIdx.x];
  unsigned char* out = records + static_cast<int64_t>(blockIdx.x) * RankRecordBytes(S);
  unsigned* words    = reinterpret_cast<unsigned*>(out);
  double* leaves     = reinterpret_cast<double*>(out + (4 << S));
  if (threadIdx.x == 0) words[0] = 0u;
  // (the paths are followed in shared memory, as in k_pack_complete: 100 trees of depth 8 15 us, now 10; 500 trees 18 and 12)
  extern __shared__ uint16_t s_feature[];  // of the nodes above the bottom level
  constexpr int kNoSplit = 0xffff;
  for (int a = threadIdx.x; a < (1 << S) - 1; a += blockDim.x) {
    const int f  = 2 * a + 2 < t.max_nodes ? t.feature[a] : -1;
    s_feature[a] = static_cast<uint16_t>(f >= 0 && f < F ? f : kNoSplit);
  }
  __syncthreads();
  for (int i = threadIdx.x; i < (2 << S) - 1; i += blockDim.x) {
    const int L = 31 - __clz(i + 1);
    int cover = -1, f = 0;  // the first leaf on the path root -> i
    for (int l = 0; l <= L && cover < 0; ++l) {
      const int a = ((i + 1) >> (L - l)) - 1;
      if (l == S || (f = s_feature[a]) == kNoSplit) cover = a;
    }
    if (L == S) {
      leaves[i - ((1 << S) - 1)] = t.leaf[cover];
    } else {
      // (below a leaf either way leads to its value)
      unsigned w = 0u;
      if (cover < 0) {
        const RankTable r = tables[f];
        int rank          = 0;
        T cut;
        MakeSplit(cut, t.split[i]);
        if (cut == cut) {  // (it is in the table)
          const unsigned e = lut[r.off + RankBucket(static_cast<float>(cut), r.lo, r.scale, r.nb)];
          const int first  = static_cast<int>(e & 0xffffu);
          rank             = 1 + first + LowerBound(cuts + r.off + first, static_cast<int>(e >> 16), cut);
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
  const int* declined;
  unsigned* out;  // [tile][F][threads]
  int tail_blocks;  // blocks for the last group of features
};

constexpr int kMaxSteps = 4, kPad = 1 << (kMaxSteps - 2);

// c = *at where n >= h, else as it was: a load without a branch.
__device__ inline void LoadSharedIf(float& c, int n, int h, unsigned at)
{
  asm volatile("{\n.reg .pred p;\nsetp.ge.s32 p, %1, %2;\n@p ld.shared.f32 %0, [%3];\n}\n" : "+f"(c) : "r"(n), "r"(h), "r"(at));
}
__device__ inline void LoadSharedIf(double& c, int n, int h, unsigned at)
{
  asm volatile("{\n.reg .pred p;\nsetp.ge.s32 p, %1, %2;\n@p ld.shared.f64 %0, [%3];\n}\n" : "+d"(c) : "r"(n), "r"(h), "r"(at));
}

// The rows of a block of k_rank_rows.  lut, cuts: the lane's feature's table, in shared memory (kInside) or in global.  kSteps: no bucket
// has 2^kSteps values or more, and kPad infinities follow the table; 0: any.
template <typename T, bool kInside, int kSteps>
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
  const unsigned below_first = cuts_at - kSize;
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
#pragma unroll
      for (int u = 0; u < kRankAhead; ++u) {
        const int b      = RankBucket(static_cast<float>(x[u]), t.lo, t.scale, t.nb);
        const unsigned e = kInside ? LdsU32(lut_at + 4u * b) : __ldg(lut + b);
        at[u]            = kInside ? (e & 0xffffu) * kSize : e & 0xffffu;
        n[u]             = static_cast<int>(e >> 16);
      }
      // how many of the bucket's values are below x, in steps of falling powers of two: all rows' values are asked for before
      // the first is compared
      auto descend = [&](int h) {
        T cut[kRankAhead];
#pragma unroll
        for (int u = 0; u < kRankAhead; ++u) {
          cut[u] = kSteps > 0 ? x[u] : static_cast<T>(INFINITY);
          if (kInside) LoadSharedIf(cut[u], n[u], h, at[u] + (h - 1) * kSize);
          else if (n[u] >= h) cut[u] = __ldg(cuts + at[u] + (h - 1));
        }
#pragma unroll
        for (int u = 0; u < kRankAhead; ++u)
          if (cut[u] < x[u]) {
            at[u] += kInside ? h * kSize : h;
            if (kSteps == 0) n[u] -= h;
          }
      };
      if (kSteps > 0) {
        // (what a step looks at beyond the bucket is not below x: a value of another one or an infinity)
        if (kSteps > 3) descend(8);
        descend(4);
        descend(2);
        descend(1);
      } else {
        int most = 0;
#pragma unroll
        for (int u = 0; u < kRankAhead; ++u) most = max(most, n[u]);
        most = __reduce_max_sync(0xffffffffu, most);
        for (int h = most >= 8 ? 1 << (31 - __clz(most)) : 0; h >= 8; h >>= 1) descend(h);
        if (most >= 4) descend(4);
        if (most >= 2) descend(2);
        if (most >= 1) descend(1);
      }
      if (fl < width) {
        const int half = st >= steps ? 1 : 0, r0 = (st - half * steps) * step_rows + sub;
        uint16_t* mine = reinterpret_cast<uint16_t*>(turn) + 2 * (fl * kPitch + r0) + half;
#pragma unroll
        for (int u = 0; u < kRankAhead; ++u)
          if (step_rows <= kRankTileRows || r0 + u * subs < kRankTileRows)
            mine[2 * u * subs] = static_cast<uint16_t>(x[u] == x[u] ? (kInside ? (at[u] - below_first) / kSize : 1 + at[u]) : t.m + 2);
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

// The tables of features [w0, w1) of a group to shared memory, by a block; four entries of a thread at a time: places, then loads, then
// stores.  (A warp per feature, 32 entries at a time: 50 us for one feature of 20 thousand.  Inlined, or with the two arrays as
// arguments, the float32 loop over the rows comes out 3 % slower: 10M x 100, 500 trees 300 and 310 us a piece.)  A word of a table:
// the address of the bucket's first value in units of values, and in the high half how many there are.  `pad` infinities
// follow the values of a feature.  Returns the values of the fullest bucket of the thread's.
template <typename T>
__device__ __noinline__ unsigned FillTables(const RankRowsArgs<T>& a, const int* s_begin, const int* s_from, int w0, int w1, int pad, unsigned* s_lut, T* s_cuts)
{
  constexpr int kFill = 4;
  const int base = s_begin[w0], entries = s_begin[w1] - base;
  const unsigned cuts_at = static_cast<unsigned>(__cvta_generic_to_shared(s_cuts)) / sizeof(T);
  unsigned fullest = 0;
  for (int i = threadIdx.x; i < (w1 - w0) * pad; i += kRankThreads) {
    const int e = i / pad;
    s_cuts[s_begin[w0 + e + 1] - base + e * pad + i - e * pad] = static_cast<T>(INFINITY);
  }
  for (int i0 = threadIdx.x; i0 < entries; i0 += kFill * kRankThreads) {
    int from[kFill];  // where the entry lies, -1: of a feature without values, whose only bucket is empty
    int first[kFill], to[kFill];  // in s_cuts: the feature's first value, and the entry's
    unsigned word[kFill];
    T cut[kFill];
#pragma unroll
    for (int u = 0; u < kFill; ++u) {
      const int i = base + min(i0 + u * kRankThreads, entries - 1);
      int e       = w0;  // the feature: the last one that begins at or before the entry
#pragma unroll
      for (int h = 16; h > 0; h >>= 1)
        if (e + h < w1 && s_begin[e + h] <= i) e += h;
      from[u]  = s_from[e] >= 0 ? s_from[e] + i - s_begin[e] : -1;
      first[u] = s_begin[e] - base + (e - w0) * pad;
      to[u]    = first[u] + i - s_begin[e];
    }
#pragma unroll
    for (int u = 0; u < kFill; ++u) {
      word[u] = from[u] >= 0 ? __ldg(a.lut + from[u]) : 0u;
      cut[u]  = from[u] >= 0 ? __ldg(a.cuts + from[u]) : T(0);
    }
#pragma unroll
    for (int u = 0; u < kFill; ++u) {
      const int i = i0 + u * kRankThreads;
      if (i < entries) {
        const unsigned n = word[u] >> 16;
        s_lut[i]         = word[u] + cuts_at + first[u];
        s_cuts[to[u]]    = cut[u];
        fullest          = max(fullest, n);
      }
    }
  }
  return fullest;
}

// X -> ranks.  A block serves one group of 32 features and keeps their tables in shared memory; lane = feature, a warp takes
// kRankTileRows rows of either half of a tile, turns their ranks in shared memory and writes them as words of two rows.  A
// last group of fewer features puts several rows side by side in a warp.
//
// Bound by the load/store pipe and the latency of its lookups: per 32 values a load of X, the bucket and about three steps of
// a search, each with the conflicts of 32 lanes on random banks, and the turn: twelve to sixteen passes and about 65
// instructions; 1.2M x 96 float32 238 us, x 64 float64 224.  (The values of a step asked for under branches, one row after
// the other: 700 us.)  Where no bucket of a turn has 16 values (8) the search takes four (three) steps without counting
// what is left of the bucket; only tables whose values crowd together take as many as their fullest bucket wants.  300003 x 130
// float32, 300 trees of depth 7 384 -> 366 us, 1M x 64 float64, 100 trees 533 -> 524.  Where the tables of a
// group do not fit (20 thousand values of float32) its features are taken in several turns over the rows; a feature
// that has no room alone is searched where its table lies.
template <typename T>
__global__ void __launch_bounds__(kRankThreads, 1) k_rank_rows(const RankRowsArgs<T> a)
{
  AfterTheKernelBefore();
  constexpr int kWarps = kRankThreads / 32, kPitch = kRankTileRows + 1;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  if (*a.declined != 0) return;
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
  __shared__ int s_begin[33], s_from[32];  // entries before the tables of the group's features, and where these lie
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
  for (int w0 = 0, w1; w0 < width; w0 = w1) {
    __syncthreads();  // (the tables before have been read)
    w1 = TurnEnd<T>(s_begin, w0, width, room);
    const int n = w1 - w0, entries = s_begin[w1] - s_begin[w0];
    int per_row = 1;  // lanes that a row takes
    while (per_row < n) per_row <<= 1;
    const int sub = lane / per_row, subs = 32 / per_row, fl = lane % per_row, f = w0 + min(fl, n - 1);
    const RankTable t = a.tables[f0 + f];
    if (TableBytes<T>(entries) <= room) {
      unsigned* s_lut = s_table;
      T* s_cuts       = reinterpret_cast<T*>(s_lut + (entries + 1) / 2 * 2);
      const int pad   = TableBytes<T>(entries) + n * kPad * static_cast<unsigned>(sizeof(T)) <= room ? kPad : 0;
      const unsigned fullest = FillTables(a, s_begin, s_from, w0, w1, pad, s_lut, s_cuts);
      const int beyond = __syncthreads_or(fullest >= 16) != 0 || pad == 0 ? 2 : __syncthreads_or(fullest >= 8) != 0 ? 1 : 0;
      const int at = s_begin[f] - s_begin[w0], cut = at + (f - w0) * pad;
      if (beyond == 0) RankRows<T, true, 3>(a, t, turn, s_lut + at, s_cuts + cut, f0 + w0, n, fl, sub, subs, part, parts);
      else if (beyond == 1) RankRows<T, true, 4>(a, t, turn, s_lut + at, s_cuts + cut, f0 + w0, n, fl, sub, subs, part, parts);
      else RankRows<T, true, 0>(a, t, turn, s_lut + at, s_cuts + cut, f0 + w0, n, fl, sub, subs, part, parts);
    } else {
      // (a feature without values has room: no index would say here that its only bucket is empty)
      RankRows<T, false, 0>(a, t, turn, a.lut + t.off, a.cuts + t.off, f0 + w0, n, fl, sub, subs, part, parts);
    }
  }
}

struct RankedArgs {
  int64_t n_rows;
  int F, n_trees, S;
  int nbuf;
  const unsigned* ranks;
  const unsigned char* records;
  const int* declined;
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
template <int TG>
__global__ void __launch_bounds__(kWalkThreads + 32, 1) k_predict_ranked(const RankedArgs a)
{
  AfterTheKernelBefore();
  __shared__ __align__(8) unsigned long long s_bar[5];  // full[2], empty[2], the tile
  __shared__ int s_failed;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  if (*a.declined != 0) return;
  const int F = a.F, S = a.S, threads = blockDim.x - 32;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int64_t row0 = static_cast<int64_t>(blockIdx.x) * 2 * threads;
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

constexpr size_t kRankBytes = size_t{256} << 20;  // of a piece of the rows
constexpr int kRankStatic   = 1024;               // of k_rank_rows
__host__ inline size_t RowsSmem(const lbk_context* ctx) { return static_cast<size_t>(ctx->max_smem_optin) - kRankStatic; }
__host__ inline unsigned TableRoom(const lbk_context* ctx)
{
  return static_cast<unsigned>(RowsSmem(ctx) - kRankThreads / 32 * 32 * (kRankTileRows + 1) * 4);
}

}  // namespace

// Is it worth it, as far as the host can tell?  In microseconds: what k_predict_tiled takes, what the walk on ranks takes (whole waves
// of tiles), and of the difference, less what the tables take, how much there is for finding the ranks.  The device decides with the tables
// as they are; here the ensemble's splits are spread evenly over the features.  Not for less than 4 % of the tiled kernel's time,
// and not where a feature is likely to have more splits than there are ranks.
//
// Both are fitted to RowsCost's ensembles (12 and 10 % off).  As it is decided here and on the device, 310 of them take 0.94 of
// k_predict_tiled's time on average, 0.54 at best and 1.17 at worst (their kernels; with a line of two factors per type, which knew
// neither the tables nor the tiles, 1.3 without one uneven feature and 19 with).  Microseconds by k_predict_tiled and as it is
// decided, a million rows, depth 8, none, 25, 40, 80 % of the splits on one feature: float32, 100 features, 500 trees 2136 and 1790 (on ranks),
// 2121 and 2232, 2108 and 2218, 2060 and 2168 (declined); float64, 64 features, 100 trees 806 and 514, 807 and 562, 800 and 621, 779 and 774
// (on ranks).  What declining costs is the tables: 300k x 20 float64, 300 trees, 40 % 522 and 588.
template <typename T>
static bool RanksPay(const lbk_context* ctx, int64_t n_rows, int F, int n_trees, int S, const RankTile& tile, RankedPlan& plan)
{
  const double splits = static_cast<double>(n_trees) * ((1 << S) - 1), millions = static_cast<double>(n_rows) * 1e-6;
  if ((splits > kMaxRank && splits > 16384.0 * F) || n_trees * S < 32) return false;
  const auto waves    = [&](int64_t rows) { return static_cast<double>((n_rows + rows * ctx->sm_count - 1) / (rows * ctx->sm_count)); };
  const double walked = waves(2 * plan.threads) * 2 * plan.threads * ctx->sm_count * 1e-6;
  const bool whole    = F * sizeof(T) % 16 == 0;  // (rows of whole vectors)
  // a tile's rows are staged and its trees brought, then its warps walk: the pipe's passes, and the latency of a step once per wave
  // and group of trees
  const double steps = static_cast<double>(n_trees) * S;
  double tiled       = 3.5 * millions * steps;  // (through the caches, at best)
  if (tile.rows > 0) {
    const double n = waves(tile.rows), chain = n * steps / tile.trees, brought = n * n_trees * tile.tree_bytes / 1024.0;
    tiled = sizeof(T) == 4 ? millions * ((whole ? 0.88 : 1.04) * F + 0.376 * steps) + 0.016 * chain + 0.027 * n * F + 0.005 * brought + 1.3 * n + 9.0
                           : millions * ((whole ? 2.14 : 2.28) * F + 0.55 * steps) + 0.035 * chain + 0.034 * n * F + 0.003 * brought + 1.3 * n + 7.0;
  }
  const double walk = walked * (0.312 * steps + n_trees * (0.55 * kWalkThreads / plan.threads - 0.56)) + millions * 0.31 * F + 6.0;
  plan.budget       = 0.98 * tiled - walk;
  int begin[33];
  for (int i = 0; i <= 32; ++i) begin[i] = i * std::max(1, static_cast<int>(splits / F));
  float even = 0.f;
  for (int g : {0, (F + 31) / 32 - 1}) even = std::max(even, RowsCost<T>::Group(begin, g, F, TableRoom(ctx), static_cast<float>(millions)));
  const double tables = 18.0 + 4.8 * S;
  plan.sure           = splits <= kMaxRank && TableBytes<T>(static_cast<int>(splits) + 32) <= TableRoom(ctx);  // (one turn per group)
  return plan.budget > even + tables + 0.02 * tiled;
}

template <typename T>
RankedPlan PlanRanked(const lbk_context* ctx, int64_t n_rows, int F, int n_trees, int S, int64_t total_nodes, const RankTile& tiled)
{
  RankedPlan best;
  if (S < 3 || S > 12 || F > kMaxFeatures || total_nodes > (int64_t{1} << 28)) return best;
  int best_score = 0;
  const size_t smem = static_cast<size_t>(ctx->max_smem_optin) - kRankedStatic;
  for (int tg = 4; tg >= 1; tg /= 2) {
    if (tg > n_trees && tg > 1) continue;
    const int nbuf     = n_trees > tg ? 2 : 1;
    const size_t trees = static_cast<size_t>(nbuf) * tg * RankRecordBytes(S);
    if (trees + static_cast<size_t>(F) * 128 > smem) continue;
    const int threads = static_cast<int>(std::min<size_t>((smem - trees) / (static_cast<size_t>(F) * 4), kWalkThreads) / 32 * 32);
    const int score   = threads * tg;
    if (score <= best_score) continue;
    best_score   = score;
    best.threads = threads;
    best.tg      = tg;
    best.nbuf    = nbuf;
    best.smem    = static_cast<size_t>(F) * threads * 4 + trees;
  }
  if (best.threads < 128 || !RanksPay<T>(ctx, n_rows, F, n_trees, S, tiled, best)) return RankedPlan{};
  // rows are walked in whole waves of tiles
  const int64_t tile  = 2 * best.threads;
  const int64_t wave  = tile * ctx->sm_count;
  const int64_t waves = std::max<int64_t>(1, static_cast<int64_t>(kRankBytes / (static_cast<size_t>(wave) * F * 2)));
  best.piece          = std::min(waves * wave, (n_rows + tile - 1) / tile * tile);
  best.max_items      = static_cast<int>(F + total_nodes / 2 / kSortChunk);
  auto reserve = [&](size_t n) {
    const size_t at = best.bytes;
    best.bytes += (n + 255) / 256 * 256;
    return at;
  };
  const size_t nodes = static_cast<size_t>(total_nodes), items = static_cast<size_t>(best.max_items);
  best.o_words   = reserve(sizeof(int) * (3 * static_cast<size_t>(F) + 2));  // declined, items, counts, cursors, blocks that are done
  best.o_off     = reserve(sizeof(int) * (static_cast<size_t>(F) + 1));
  best.o_items   = reserve((sizeof(int2) + sizeof(int)) * items);
  best.o_lists   = reserve(nodes * sizeof(T));
  best.o_cuts    = reserve(nodes * sizeof(T));
  best.o_lut     = reserve(nodes * sizeof(unsigned));
  best.o_tables  = reserve(sizeof(RankTable) * F);
  best.o_records = reserve(static_cast<size_t>(n_trees) * RankRecordBytes(S));
  best.o_ranks   = reserve(static_cast<size_t>(best.piece / 2) * F * sizeof(unsigned));
  return best;
}

template <typename T>
const int* PredictRanked(lbk_context* ctx, Scratch& s, const RankedPlan& plan, const T* X, int64_t ldx, int64_t n_rows, int F, int n_trees,
                         const lbk_tree_ref* d_trees, int S, int64_t total_nodes, const double* init, int transform, double* pred, int64_t ldp, cudaStream_t stream)
{
  unsigned char* room = nullptr;
  try {  // (one piece, so that a call which has no room for it is left as it was)
    room = static_cast<unsigned char*>(s.alloc_bytes(plan.bytes));
  } catch (const Error& e) {
    if (e.code != LBK_ERR_ALLOC) throw;
    return nullptr;
  }
  int* words    = reinterpret_cast<int*>(room + plan.o_words);
  int* declined = words;
  int* counts   = words + 2;
  T* cuts       = reinterpret_cast<T*>(room + plan.o_cuts);
  RankTables<T> t;
  t.off      = reinterpret_cast<int*>(room + plan.o_off);
  t.items    = reinterpret_cast<int2*>(room + plan.o_items);
  t.n_items  = words + 1;
  t.len      = reinterpret_cast<int*>(room + plan.o_items + sizeof(int2) * plan.max_items);
  t.arrived  = counts + 2 * F;
  t.lists    = reinterpret_cast<T*>(room + plan.o_lists);
  t.cuts     = cuts;
  t.lut      = reinterpret_cast<unsigned*>(room + plan.o_lut);
  t.tables   = reinterpret_cast<RankTable*>(room + plan.o_tables);
  t.declined = declined;
  unsigned char* records = room + plan.o_records;
  unsigned* ranks        = reinterpret_cast<unsigned*>(room + plan.o_ranks);
  const unsigned items   = static_cast<unsigned>(plan.max_items);
  LBK_CUDA(cudaMemsetAsync(words, 0, sizeof(int) * (3 * static_cast<size_t>(F) + 2), stream));
  LaunchChained(k_rank_count<T>, n_trees, 256, 0, stream, d_trees, F, counts);
  LBK_LAUNCH_CHECK();
  LaunchChained(k_rank_scatter<T>, n_trees, 256, 0, stream, d_trees, F, counts, counts + F, const_cast<int*>(t.off), const_cast<int2*>(t.items), words + 1, declined, t.lists);
  LBK_LAUNCH_CHECK();
  LaunchChained(k_rank_sort<T>, items, kSortThreads, 0, stream, t);
  LBK_LAUNCH_CHECK();
  if (total_nodes / 2 > kSortChunk) {
    LaunchChained(k_rank_merge<T>, dim3(items, kSortChunk / kSortThreads), kSortThreads, 0, stream, t);
    LBK_LAUNCH_CHECK();
  }
  LaunchChained(k_rank_pack<T>, n_trees, 256, sizeof(uint16_t) << S, stream, d_trees, F, S, plan.threads / 32, plan.sure ? 0.f : static_cast<float>(n_rows) * 1e-6f, static_cast<float>(plan.budget), TableRoom(ctx), t.tables, cuts, t.lut, declined, records);
  LBK_LAUNCH_CHECK();
  AllowSharedMemory(ctx, k_rank_rows<T>, kRankStatic);
  const int64_t tile    = 2 * plan.threads;
  const int groups      = (F + 31) / 32;
  const int lanes       = TailLanes(F);
  const int blocks      = std::max(ctx->sm_count, groups);
  const int tail_blocks = groups == 1 ? blocks
                                      : std::min(blocks - (groups - 1), std::max(1, (blocks * lanes + 16 * (groups - 1) + lanes / 2) / (32 * (groups - 1) + lanes)));
  auto walk = plan.tg == 4 ? k_predict_ranked<4> : plan.tg == 2 ? k_predict_ranked<2> : k_predict_ranked<1>;
  AllowSharedMemory(ctx, walk, kRankedStatic);
  for (int64_t r0 = 0; r0 < n_rows; r0 += plan.piece) {
    const int64_t rows = std::min(plan.piece, n_rows - r0), tiles = (rows + tile - 1) / tile;
    RankRowsArgs<T> ra{X + r0 * ldx, ldx, rows, F, plan.threads, tiles, t.tables, cuts, t.lut, declined, ranks, tail_blocks};
    LaunchChained(k_rank_rows<T>, blocks, kRankThreads, RowsSmem(ctx), stream, ra);
    LBK_LAUNCH_CHECK();
    RankedArgs wa{rows, F, n_trees, S, plan.nbuf, ranks, records, declined, PredictOut{pred + r0 * ldp, ldp, init, transform}, ctx->d_status};
    LaunchChained(walk, static_cast<unsigned>(tiles), plan.threads + 32, plan.smem, stream, wa);
    LBK_LAUNCH_CHECK();
  }
  return declined;
}

#define LBK_PREDICT_RANKED(T)                                                                                                                  \
  template RankedPlan PlanRanked<T>(const lbk_context*, int64_t, int, int, int, int64_t, const RankTile&);                                                    \
  template const int* PredictRanked<T>(lbk_context*, Scratch&, const RankedPlan&, const T*, int64_t, int64_t, int, int, const lbk_tree_ref*,    \
                                       int, int64_t, const double*, int, double*, int64_t, cudaStream_t);
LBK_PREDICT_RANKED(float)
LBK_PREDICT_RANKED(double)

}  // namespace lbk
