// Split proposals and the binned matrix.
//
// Reference behaviour restated here:
//   SelectSplitSamples  src/models/tree/build_tree.cu:867-964 - draw split_samples row ids from
//     the seed, gather those rows (zeros where another rank owns the row), sum over ranks, keep
//     the sorted unique values per feature as a CSR, overwrite each feature's largest value
//     with +inf.
//   FindBin             src/models/tree/build_tree.h:178-185 - bin = first proposal >= x.
// The reference re-runs the search for every element on every tree level; here it runs once per
// tree and the result is kept as one byte (or two) per element, grouped 32 features at a time
// so that a warp reads one 32-byte sector per row with one lane per feature.
#include <cfloat>
#include <cmath>
#include <limits>

#include "device_utils.cuh"
#include <type_traits>

#include "abs_sum.cuh"
#include "count_sort.cuh"
#include "bin_grid.h"
#include "internal.h"

namespace lbk {
namespace {

constexpr int kSortThreads = 256;

// The value of feature f in the i-th sampled row of the data set; 0 if another rank holds the row.
template <typename T>
__device__ inline T SampledValue(const PrologueArgs<T>& p, int i, int f)
{
  MinStd eng(static_cast<uint32_t>(p.seed));
  eng.discard(static_cast<unsigned long long>(i));
  const long long row = eng.uniform_int(0, p.dataset_rows - 1);
  const bool has      = row >= p.row_offset && row < p.row_offset + p.n_local;
  return has ? p.X[(row - p.row_offset) * p.ldx + f] : T(0);
}

// [F][S] sampled values, for the sum over ranks that comes before the sort
template <typename T>
__global__ void k_gather_samples(const __grid_constant__ PrologueArgs<T> p, T* __restrict__ draft)
{
  const int64_t idx = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
  if (idx >= static_cast<int64_t>(p.F) * p.S) return;
  const int i = static_cast<int>(idx / p.F);
  const int f = static_cast<int>(idx % p.F);
  draft[static_cast<int64_t>(f) * p.S + i] = SampledValue(p, i, f);
}

// Samples of a feature that are sorted by counting, beyond them by a bitonic network; and the shared memory of either.
constexpr int kCountMax = 512;
template <typename T>
__host__ __device__ constexpr size_t SortSmem(int S_pad)
{
  return S_pad <= kCountMax ? (sizeof(T) + 1) * (S_pad < 4 ? 4 : S_pad) : sizeof(T) * S_pad;
}

// One block: the S samples of feature f sorted, the distinct ones kept in cuts[f * S ..], the last of them replaced by +inf.
template <typename T>
__device__ inline void SortUniqueBlock(const PrologueArgs<T>& p, int f, T* vals /* shared, SortSmem */, int* s_cnt /* shared [9] */)
{
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int S = p.S, S_pad = p.S_pad;
  auto sample = [&](int i) -> T {
    if (i >= S) return static_cast<T>(INFINITY);
    const T v = p.draft != nullptr ? p.draft[static_cast<int64_t>(f) * S + i] : SampledValue(p, i, f);
    // (-0 becomes +0: they are equal, and which of them was kept would be up to the threads' timing.  A NaN counts as +inf.)
    return v == v ? v + T(0) : static_cast<T>(INFINITY);
  };
  const int P     = S_pad < 4 ? 4 : S_pad;  // (whole 16-byte words)
  const uint8_t* mark = nullptr;  // counted: where there is a value
  if (S_pad <= kCountMax) {
    constexpr int kPer = kCountMax / kSortThreads;
    uint8_t* here = reinterpret_cast<uint8_t*>(vals + P);
    mark          = here;
    T mine[kPer];
#pragma unroll
    for (int u = 0; u < kPer; ++u) {
      const int i = tid + u * kSortThreads;
      mine[u]     = sample(i);
      if (i < P) {
        vals[i] = mine[u];
        here[i] = 0;
      }
    }
    __syncthreads();
    int below[kPer];
#pragma unroll
    for (int u = 0; u < kPer; ++u)
      below[u] = u == 0 || P > kSortThreads ? CountBelow(vals, P / static_cast<int>(16 / sizeof(T)), mine[u]) : 0;
    __syncthreads();  // (the places are those of the same array: the sum blocks of the launch want the rest of the SM as L1)
#pragma unroll
    for (int u = 0; u < kPer; ++u)
      if (tid + u * kSortThreads < S) {
        vals[below[u]] = mine[u];
        here[below[u]] = 1;
      }
    __syncthreads();
  } else {
    for (int i = tid; i < S_pad; i += kSortThreads) vals[i] = sample(i);
    __syncthreads();
    for (int k = 2; k <= S_pad; k <<= 1) {
      for (int j = k >> 1; j > 0; j >>= 1) {
        for (int i = tid; i < S_pad; i += kSortThreads) {
          const int ixj = i ^ j;
          if (ixj > i) {
            const T a = vals[i], b = vals[ixj];
            const bool up = (i & k) == 0;
            if (up ? (b < a) : (a < b)) {
              vals[i]   = b;
              vals[ixj] = a;
            }
          }
        }
        __syncthreads();
      }
    }
  }
  // unique over the first S sorted entries, 256 at a time
  T* out     = p.cuts + static_cast<int64_t>(f) * S;
  int before = 0;
  for (int base = 0; base < S; base += kSortThreads) {
    const int i      = base + tid;
    const bool keep  = i < S && (mark != nullptr ? mark[i] != 0 : i == 0 || vals[i] != vals[i - 1]);
    const unsigned m = __ballot_sync(0xffffffffu, keep);
    if (lane == 0) s_cnt[warp] = __popc(m);
    __syncthreads();
    int pos = before;
    for (int w = 0; w < warp; ++w) pos += s_cnt[w];
    int total = before;
    for (int w = 0; w < kSortThreads / 32; ++w) total += s_cnt[w];
    pos += __popc(m & ((1u << lane) - 1u));
    if (keep) out[pos] = vals[i];
    before = total;
    __syncthreads();
  }
  if (tid == 0) {
    out[before - 1] = static_cast<T>(INFINITY);
    p.counts[f]     = before;
  }
}

// Everything a tree needs that depends on no other step, one launch with three kinds of blocks: a block
// per feature draws, sorts and prunes the split proposals; a block per 4096 elements sums |g| and |h|
// (the canonical order of quantise.cu); the rest clear the tree's arrays and counters.
template <typename T>
__global__ void __launch_bounds__(kSortThreads)
  k_prologue(const __grid_constant__ PrologueArgs<T> p)
{
  AfterTheKernelBefore();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ int s_cnt[kSortThreads / 32 + 1];
  __shared__ double s_sum[2 * kSumThreads / 32];
  int b = blockIdx.x;
  if (b < p.sort_blocks) {
    SortUniqueBlock(p, b, reinterpret_cast<T*>(smem_raw), s_cnt);
    return;
  }
  b -= p.sort_blocks;
  if (b < p.sum_blocks) {
    AbsSumBlock<true>(p.g, p.h, p.ldg, p.form, p.K, p.n_elements, b, threadIdx.x, s_sum, p.part_g + b, p.part_h + b);
    return;
  }
  b -= p.sum_blocks;
  const int64_t t = static_cast<int64_t>(b) * kSortThreads + threadIdx.x, n = static_cast<int64_t>(p.fill_blocks) * kSortThreads;
  for (int z = 0; z < kZeroRanges; ++z)
    for (int64_t i = t; i < p.zero_n16[z]; i += n) static_cast<uint4*>(p.zero[z])[i] = make_uint4(0u, 0u, 0u, 0u);
  if (t == 0 && p.root_begin != nullptr) {
    *p.root_begin = 0;
    *p.root_end   = static_cast<int32_t>(p.n_local);
  }
  for (int64_t i = t; i < p.tree.max_nodes; i += n) {
    p.tree.feature[i]     = -1;
    p.tree.split_value[i] = 0.0;
    p.tree.gain[i]        = 0.0;
  }
}

// Single block: row_ptr = exclusive scan of the counts, the number of bins and the largest feature (to the
// device and, if info_host is given, to mapped host memory), the rest of the |g|, |h| sums and, if
// `params` is given, the quantiser's scale from them.
__global__ void __launch_bounds__(1024)
  k_prologue_finish(const int32_t* __restrict__ counts, int F, int32_t* __restrict__ row_ptr, int32_t* __restrict__ info,
                    int32_t* info_host, double* part_g, double* part_h, int64_t n_parts, double* sums,
                    QuantParams* params)
{
  AfterTheKernelBefore();
  __shared__ int warp_sums[32];
  __shared__ int carry_s;
  __shared__ int max_s;
  __shared__ double s_sum[4 * 2 * kSumThreads / 32];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (counts != nullptr) {
    if (tid == 0) {
      carry_s    = 0;
      max_s      = 0;
      row_ptr[0] = 0;
    }
    __syncthreads();
    for (int base = 0; base < F; base += blockDim.x) {
      const int i = base + tid;
      const int c = i < F ? counts[i] : 0;
      int incl    = c;
      for (int off = 1; off < 32; off <<= 1) {
        int n = __shfl_up_sync(0xffffffffu, incl, off);
        if (lane >= off) incl += n;
      }
      if (lane == 31) warp_sums[warp] = incl;
      const int top = __reduce_max_sync(0xffffffffu, c);
      if (lane == 0) atomicMax(&max_s, top);
      __syncthreads();
      if (warp == 0) {
        int w  = warp_sums[lane];
        int wi = w;
        for (int off = 1; off < 32; off <<= 1) {
          int n = __shfl_up_sync(0xffffffffu, wi, off);
          if (lane >= off) wi += n;
        }
        warp_sums[lane] = wi - w;  // exclusive
      }
      __syncthreads();
      const int total_before = carry_s + warp_sums[warp];
      if (i < F) row_ptr[i + 1] = total_before + incl;
      __syncthreads();
      if (tid == blockDim.x - 1) carry_s = total_before + incl;
      __syncthreads();
    }
    if (tid == 0) {
      info[0] = carry_s;
      info[1] = max_s;
      // (one store of 8 bytes: a host that polls sees both or neither)
      if (info_host != nullptr)
        *reinterpret_cast<volatile unsigned long long*>(info_host) = static_cast<unsigned>(carry_s) | static_cast<unsigned long long>(max_s) << 32;
    }
  }
  if (sums == nullptr) return;
  // four groups of 256 threads, each sums 4096 values at a time in the canonical order; a level's results
  // overwrite its inputs block by block (block b of four per turn writes entry b, all inputs up to then
  // have been read)
  int64_t n = n_parts;
  while (n > 1) {
    const int64_t blocks = (n + kSumBlock - 1) / kSumBlock;
    for (int64_t b0 = 0; b0 < blocks; b0 += 4) {
      const int q     = tid / kSumThreads;
      const int64_t b = b0 + q;
      double tg, th;
      AbsSumPartial<false>(part_g, part_h, 0, GradientForm{}, 1, n, b, tid % kSumThreads, s_sum + q * 2 * kSumThreads / 32, tg, th);
      __syncthreads();
      if (tid % kSumThreads == 0 && b < blocks) {
        part_g[b] = tg;
        part_h[b] = th;
      }
      __syncthreads();
    }
    n = blocks;
  }
  if (tid == 0) {
    sums[0] = n_parts > 0 ? part_g[0] : 0.0;
    sums[1] = n_parts > 0 ? part_h[0] : 0.0;
    if (params != nullptr) *params = MakeScale(sums[0], sums[1]);
  }
}

__global__ void k_make_scale(const double* __restrict__ sums /* g,h */, QuantParams* __restrict__ qp)
{
  *qp = MakeScale(sums[0], sums[1]);
}

template <typename T>
__global__ void k_write_proposals(const T* __restrict__ cuts, int S, const int32_t* __restrict__ row_ptr,
                                  T* __restrict__ proposals)
{
  AfterTheKernelBefore();
  const int f     = blockIdx.x;
  const int begin = row_ptr[f], end = row_ptr[f + 1];
  for (int j = threadIdx.x; j < end - begin; j += blockDim.x) proposals[begin + j] = cuts[static_cast<int64_t>(f) * S + j];
}

// Streaming global loads as volatile asm: they stay where they are written, ahead of the search
// of the previous rows (the compiler otherwise sinks them to their first use).
__device__ inline float LdgStream(const float* p)
{
  float v;
  asm volatile("ld.global.cs.f32 %0, [%1];\n" : "=f"(v) : "l"(p));
  return v;
}
__device__ inline double LdgStream(const double* p)
{
  double v;
  asm volatile("ld.global.cs.f64 %0, [%1];\n" : "=d"(v) : "l"(p));
  return v;
}

template <int kOffset>
__device__ inline float LdsT(unsigned addr, float)
{
  float v;
  asm volatile("ld.shared.f32 %0, [%1+%2];\n" : "=f"(v) : "r"(addr), "n"(kOffset));
  return v;
}
template <int kOffset>
__device__ inline double LdsT(unsigned addr, double)
{
  double v;
  asm volatile("ld.shared.f64 %0, [%1+%2];\n" : "=d"(v) : "r"(addr), "n"(kOffset));
  return v;
}

// One lower_bound step for U rows at once: "advance by 2^kLevel proposals if the proposal just
// before that point is below x".  The probe offset is an immediate of the load; what remains per
// row and step is one shared-memory load, one compare and one predicated add.
template <typename T, int U, int kLevel, unsigned kPitch>
struct SearchLevels {
  __device__ static void run(unsigned (&pos)[U], const T (&x)[U])
  {
    constexpr int step = 1 << kLevel;
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (LdsT<(step - 1) * static_cast<int>(kPitch)>(pos[u], T()) < x[u]) pos[u] += step * kPitch;
    SearchLevels<T, U, kLevel - 1, kPitch>::run(pos, x);
  }
};
template <typename T, int U, unsigned kPitch>
struct SearchLevels<T, U, -1, kPitch> {
  __device__ static void run(unsigned (&)[U], const T (&)[U]) {}
};

// Where the search for x begins, as in k_bin_lut: x falls into one of P buckets by a map that never decreases, and a table says
// how many proposals lie in the buckets below.  The map goes through float32 whatever T is (rounding does not decrease either), is
// spread from the fifth proposal to the fifth from the end, and sends a NaN on the way to bucket 0.
struct StartMap {
  float lo, scale;
};
template <int P>
__device__ inline int StartBucket(float x, const StartMap& m)
{
  const int b = __float2int_rz((x - m.lo) * m.scale);
  return b < 0 ? 0 : b < P ? b : P - 1;
}
constexpr int kStartSpare = 16;  // rows of the table behind the proposals, +inf: the last steps may look beyond the last one

// Fills the table of a block, sp[P + kStartSpare][kFeatures], with the proposals of the features from f0 on.
template <typename T, int kFeatures, int kRows>
__device__ inline void FillProposals(T* sp, int* s_begin, int* s_n, const T* proposals, int64_t cut_stride, const int32_t* row_ptr, int f0, int F)
{
  if (threadIdx.x < kFeatures) {
    const int f = f0 + static_cast<int>(threadIdx.x), b = f < F ? row_ptr[f] : 0;
    s_begin[threadIdx.x] = cut_stride > 0 ? 0 : b;
    s_n[threadIdx.x]     = f < F ? row_ptr[f + 1] - b : 0;
  }
  __syncthreads();
#pragma unroll 8
  for (int idx = threadIdx.x; idx < kRows * kFeatures; idx += blockDim.x) {
    const int j = idx / kFeatures, fl = idx % kFeatures;
    sp[idx]     = j < s_n[fl] ? proposals[(cut_stride > 0 ? (f0 + fl) * cut_stride : s_begin[fl]) + j] : static_cast<T>(INFINITY);
  }
  __syncthreads();
}

// starts [P][kFeatures] and the maps, by kThreads threads; returns how many steps of a search from there are enough for every
// feature of the block: 3 (no more than 7 proposals share a bucket), 4 (15), or 0: the whole search, without the table
// (they crowd together more, or are not in order with +inf at the end).
template <typename T, int kFeatures, int P, int kThreads>
__device__ inline int MakeStarts(const T* sp, uint16_t* starts, const int* s_n, StartMap* s_map)
{
  if (threadIdx.x < kFeatures) {
    const int fl = threadIdx.x, n = s_n[fl], end = n >= 32 ? 4 : 0;
    StartMap m{0.0f, 0.0f};
    if (n >= 3) {  // (the last proposal is +inf)
      m.lo    = static_cast<float>(sp[end * kFeatures + fl]);
      m.scale = static_cast<float>(P) / (static_cast<float>(sp[(n - 2 - end) * kFeatures + fl]) - m.lo);
      if (!(m.scale > 0.0f) || !(m.scale < INFINITY) || !(fabsf(m.lo) < INFINITY)) m.lo = m.scale = 0.0f;  // all in one bucket
    }
    s_map[fl] = m;
  }
  __syncthreads();
  // a thread has kOwn neighbouring proposals (and then buckets) of one feature
  constexpr int kOwn = P * kFeatures / kThreads;
  const int fl = threadIdx.x % kFeatures, n = s_n[fl], j0 = threadIdx.x / kFeatures * kOwn;
  const StartMap m = s_map[fl];
  auto at_of  = [&](int i) { return StartBucket<P>(static_cast<float>(sp[i * kFeatures + fl]), m); };
  int crowd   = 0;
  int before  = j0 > 0 && j0 < n ? at_of(j0 - 1) : -1;
#pragma unroll 4
  for (int i = 0; i < kOwn; ++i) {
    const int j = j0 + i;
    if (j < n) {
      const int at = at_of(j);
      const T v = sp[j * kFeatures + fl], next = sp[(j + 1) * kFeatures + fl];
      for (int k = before + 1; k <= at; ++k) starts[k * kFeatures + fl] = static_cast<uint16_t>(j);
      if (j == n - 1 ? v != static_cast<T>(INFINITY) : !(v < next)) crowd = 2;
      if (j == n - 1)  // (+inf is in the last bucket, unless all are in the first)
        for (int k = at + 1; k < P; ++k) starts[k * kFeatures + fl] = static_cast<uint16_t>(n);
      before = at;
    }
  }
  if (n == 0)
    for (int i = 0; i < kOwn; ++i) starts[(j0 + i) * kFeatures + fl] = 0;
  if (__syncthreads_or(crowd)) return 0;
#pragma unroll 4
  for (int i = 0; i < kOwn; ++i) {
    const int b = j0 + i, first = starts[b * kFeatures + fl], next = b + 1 < P ? starts[(b + 1) * kFeatures + fl] : n;
    crowd = max(crowd, next - first);
  }
  if (!__syncthreads_or(crowd > 7)) return 3;
  return !__syncthreads_or(crowd > 15) ? 4 : 0;
}

// One warp per row, one lane per feature of the group.
//
// Shared-memory variant: the proposals of the group are kept transposed and padded, sp[j][lane] =
// proposal j of the lane's feature (+inf beyond the feature's last one and for the lanes beyond
// the last feature, P = 2^kLog2P rows), so that every probe of lane l goes to bank l: the probes
// of a lower_bound are conflict-free passes whatever the values.  The search is the branchless
// form "pos += step while sp[pos+step-1] < x" on the shared-memory address of the lane's column,
// fully unrolled; it returns the number of proposals below x, i.e. the index of the first
// proposal >= x.  The pivots of the first two levels are kept in registers.
//
// A warp takes kTileRows consecutive rows per turn, eight at a time.  What bounds the kernel is
// the load/store pipe (one pass per distinct 128-byte line of an instruction) and the issue slots,
// so: the turns that lie wholly inside the matrix run without row checks; and the feature-major
// copy of one-byte ids goes through a per-warp tile in shared memory, [32 features][kTileRows
// bytes], from which the warp writes kTileRows contiguous bytes per feature (two features per
// store instruction) instead of one 16-byte piece per lane and line.
constexpr int kBinTileRows  = 64;
constexpr int kBinTilePitch = kBinTileRows + 8;  // bytes; 18 words: 8-byte stores of 16 lanes fall on distinct banks

template <typename T, typename BinT, int kLog2P, bool kCopyT>
__global__ void __launch_bounds__(256, sizeof(T) == 4 ? 4 : 2)
  k_bin_smem(const T* __restrict__ X, int64_t ldx, int64_t n_rows, int F, const T* __restrict__ proposals,
             int64_t cut_stride, const int32_t* __restrict__ row_ptr, BinT* __restrict__ bins, BinT* __restrict__ bins_t, int64_t pitch_t)
{
  AfterTheKernelBefore();
  constexpr int P = 1 << kLog2P;
  constexpr bool kTile = kCopyT && sizeof(BinT) == 1;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T* sp          = reinterpret_cast<T*>(smem_raw);
  const int g    = blockIdx.y;
  const int f0   = g * kGroup;
  const int lane = threadIdx.x & 31;
  for (int idx = threadIdx.x; idx < P * kGroup; idx += blockDim.x) {
    const int j = idx >> 5, f = f0 + (idx & 31);
    T v = static_cast<T>(INFINITY);
    if (f < F) {
      const int b = row_ptr[f];
      if (j < row_ptr[f + 1] - b) v = proposals[(cut_stride > 0 ? f * cut_stride : b) + j];
    }
    sp[idx] = v;
  }
  __syncthreads();
  // Lanes beyond the last feature read the last feature's values (in bounds); their column of the
  // table is all +inf, so their ids are 0.
  const bool active = f0 + lane < F;
  constexpr unsigned kPitch = kGroup * sizeof(T);  // bytes from one proposal of a feature to the next
  const unsigned col_s      = static_cast<unsigned>(__cvta_generic_to_shared(sp + lane));
  unsigned char* tile = smem_raw + sizeof(T) * P * kGroup + (threadIdx.x >> 5) * (kGroup * kBinTilePitch);
  const unsigned tile_s = static_cast<unsigned>(__cvta_generic_to_shared(tile));
  // rows are counted in 32 bits (row indices are 32-bit everywhere in this library)
  const int pitch   = static_cast<int>(gridDim.y) * kGroup;  // bins are row-major, rows padded to groups
  constexpr int U   = 8;  // rows per warp in flight
  const int n       = static_cast<int>(n_rows);
  const int ld      = static_cast<int>(ldx);
  constexpr int kSubs = kBinTileRows / U;
  constexpr int kTurn = kBinTileRows;
  const int hop     = static_cast<int>(gridDim.x) * (blockDim.x >> 5) * kTurn;  // rows from one turn of a warp to the next
  int turn          = (blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * kTurn;
  const T* xcol     = X + (active ? f0 + lane : F - 1);
  BinT* ocol        = bins + f0 + lane;
  BinT* tcol        = kCopyT ? bins_t + static_cast<int64_t>(active ? f0 + lane : F - 1) * pitch_t : nullptr;
  // pivots of the first two levels
  T piv_h = T(), piv_q1 = T(), piv_q3 = T();
  if (kLog2P >= 2) {
    piv_h  = sp[(P / 2 - 1) * kGroup + lane];
    piv_q1 = sp[(P / 4 - 1) * kGroup + lane];
    piv_q3 = sp[(3 * P / 4 - 1) * kGroup + lane];
  }
  // the values of the warp's next eight rows are loaded while the current eight are searched
  auto load_rows = [&](int first, T (&x)[U]) {
    const T* src = xcol + static_cast<int64_t>(first) * ld;
#pragma unroll
    for (int u = 0; u < U; ++u) x[u] = LdgStream(src + u * ld);
  };
  auto load_rows_checked = [&](int first, T (&x)[U]) {
    const T* src = xcol + static_cast<int64_t>(first) * ld;
#pragma unroll
    for (int u = 0; u < U; ++u) x[u] = first + u < n ? LdgStream(src + u * ld) : static_cast<T>(-INFINITY);
  };
  T xn[U];
  if (turn < n) load_rows_checked(turn, xn);
  // one turn; kChecked: the turn may reach beyond the last row
  auto do_turn = [&](auto checked) {
    constexpr bool kChecked = decltype(checked)::value;
#pragma unroll 2
    for (int sub = 0; sub < kSubs; ++sub) {
      const int base = turn + sub * U;
      T x[U];
      unsigned pos[U];
#pragma unroll
      for (int u = 0; u < U; ++u) x[u] = xn[u];
      {
        const int nb = sub + 1 < kSubs ? base + U : turn + hop;
        if (sub + 1 < kSubs && !kChecked) load_rows(nb, xn);
        else if (nb < n) load_rows_checked(nb, xn);
      }
      if (kLog2P >= 2) {
#pragma unroll
        for (int u = 0; u < U; ++u) {
          const bool c1 = piv_h < x[u];
          pos[u]        = c1 ? col_s + (P / 2) * kPitch : col_s;
          const T piv   = c1 ? piv_q3 : piv_q1;
          if (piv < x[u]) pos[u] += (P / 4) * kPitch;
        }
        SearchLevels<T, U, kLog2P - 3, kPitch>::run(pos, x);
      } else {
#pragma unroll
        for (int u = 0; u < U; ++u) pos[u] = col_s;
        SearchLevels<T, U, kLog2P - 1, kPitch>::run(pos, x);
      }
      unsigned id[U];
#pragma unroll
      for (int u = 0; u < U; ++u) id[u] = (pos[u] - col_s) / kPitch;
      BinT* orow = ocol + static_cast<int64_t>(base) * pitch;
#pragma unroll
      for (int u = 0; u < U; ++u)
        if (!kChecked || base + u < n) orow[u * pitch] = static_cast<BinT>(id[u]);
      if (kCopyT) {
        if (kTile) {
          const unsigned lo = id[0] | (id[1] << 8) | (id[2] << 16) | (id[3] << 24);
          const unsigned hi = id[4] | (id[5] << 8) | (id[6] << 16) | (id[7] << 24);
          asm volatile("st.shared.v2.b32 [%0], {%1, %2};\n" ::"r"(tile_s + lane * kBinTilePitch + sub * U), "r"(lo), "r"(hi)
                       : "memory");
        } else if (active && base < n) {
          uint4 pk;
          pk.x = id[0] | (id[1] << 16);
          pk.y = id[2] | (id[3] << 16);
          pk.z = id[4] | (id[5] << 16);
          pk.w = id[6] | (id[7] << 16);
          *reinterpret_cast<uint4*>(tcol + base) = pk;
        }
      }
    }
    if (kTile) {
      // the tile leaves feature by feature: lanes 0-15 write the 64 bytes of one feature, lanes
      // 16-31 those of the next (rows up to the padded end of a feature's row of the copy; the ids
      // of rows beyond the last one are 0)
      __syncwarp();
      const int w    = lane & 15;
      const bool in  = turn + 4 * w < pitch_t;
#pragma unroll 4
      for (int i = 0; i < kGroup / 2; ++i) {
        const int fl = 2 * i + (lane >> 4);
        unsigned v;
        asm volatile("ld.shared.b32 %0, [%1];\n" : "=r"(v) : "r"(tile_s + fl * kBinTilePitch + 4 * w));
        if (in && f0 + fl < F)
          *reinterpret_cast<unsigned*>(bins_t + static_cast<int64_t>(f0 + fl) * pitch_t + turn + 4 * w) = v;
      }
      __syncwarp();
    }
  };
  for (; turn + kTurn <= n; turn += hop) do_turn(std::false_type());
  if (turn < n) do_turn(std::true_type());
}

// One-byte ids of float32 values, up to 256 proposals per feature: the search starts from a table lookup.
//
// k_bin_smem is bound by its issue slots and the load/store pipe (72 % each): five instructions for the two
// levels in registers and three more and a pass for each of the other six.  Here a value is first mapped to one of
// 512 buckets, of which a table says where the search begins: at the number of proposals in the buckets below.  Since
// the map never decreases, those are below x and the proposals of the buckets above are not, and what is left to
// search are the proposals of x's own bucket.  The map spreads the buckets evenly from the fifth proposal to the
// fifth from the end (beyond them lie four proposals and any outliers): t = x s + b, saturated to [0, 1], then
// t 511 + 2^23 rounds to the bucket.  A block looks how many proposals share a bucket in its features at worst and
// takes three steps of the search (up to 7: uniform and normal columns), four (up to 15) or, where the values crowd
// together more, the whole search without the table.  A NaN ends in bucket 0 and fails every comparison: id 0, as
// in the other kernels.
//
// Shared memory: rows of 256 bytes from the address 32768 on, row j = proposal j of the 32 features | what the
// bucket j of each feature begins with, as the address of that proposal.  So a lookup and a probe are one pass
// (bank = lane), the search goes on with what was looked up, and the id is byte 1 of the address it ends at, less 128.
// A block of 32 warps has one such table; the warps' tiles for the feature-major copy lie before and behind it.  The
// row-major ids leave as words of four features, turned among four lanes.
//
// The feature-major copy is 32 streams per block that lie n_rows bytes apart.  Four warps with neighbouring rows write
// their tiles together, 128 bytes of a feature at a time: with 32 bytes per warp the 100M rows took 9430 us (and 5960
// without the copy, of which that is 1 ms at the copy rate of HBM), with eight or sixteen warps 6940 and 8120 (they wait for
// each other; 10M: 712 and 818).  Of 1M x 100, whose copy stays in L2, a warp by itself takes 158 instead of 175.
//
// Bound by the issue slots and the load/store pipe (262 instructions and about 62 passes per 256 ids), close to HBM.
// Measured with the copy, before (a table of bytes, whose lookups are three passes, a store per row, eight values ahead, a
// table filled by reads 1 KB apart) and now: 100M x 64: 8430 -> 6960 us (the copy rate of HBM gives 5870), 10M x 64: 840 -> 696, 1M x 100: 221 -> 175,
// 200k x 50: 42 -> 25.  Eight values ahead instead of sixteen, in this layout: 10M x 64 827 us.
constexpr int kFaultBinLayout  = 32;  // status word: shared memory is not laid out as the kernel's addresses need it
constexpr int kBuckets         = 512;
constexpr int kLutThreads      = 1024;
constexpr int kLutWarps        = kLutThreads / 32;
constexpr int kLutRows         = 256 + 16;  // of the table: the last steps may look beyond the last proposal
constexpr unsigned kLutRow     = 2 * kGroup * sizeof(float);
constexpr unsigned kLutAt      = 32768;     // an id is byte 1 of the address of its row, less 128
constexpr int kLutTurn         = 32;        // rows of a warp's tile
constexpr int kLutTeam         = 4;         // warps that write the feature-major copy of their rows together
constexpr unsigned kLutTile    = kGroup * kLutTurn + 32;  // (the tiles of a team begin in different banks)
constexpr int kLutTilesBefore  = 29;        // (1 KB is reserved, the kernel declares less than another)
constexpr unsigned kLutTilesAt = kLutAt - kLutTilesBefore * kLutTile;
constexpr unsigned kLutEnd     = kLutAt + kBuckets * kLutRow + (kLutWarps - kLutTilesBefore / kLutTeam * kLutTeam) * kLutTile;
constexpr unsigned kLutStageAt = kLutAt + kLutRows * kLutRow;  // (the proposals are turned there before the buckets are made)
static_assert(kLutTilesAt >= 2048 && kLutStageAt + kLutRows * (kGroup + 1) * 4 <= kLutEnd, "room around the table");

template <bool kCopyT>
__global__ void __launch_bounds__(kLutThreads, 1)
  k_bin_lut(const float* __restrict__ X, int64_t ldx, int64_t n_rows, int F, const float* __restrict__ proposals,
            int64_t cut_stride, const int32_t* __restrict__ row_ptr, uint8_t* __restrict__ bins, uint8_t* __restrict__ bins_t, int64_t pitch_t,
            int* __restrict__ status)
{
  AfterTheKernelBefore();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ int s_n[kGroup];
  __shared__ float2 s_map[kGroup];
  // (addresses of the shared window as offsets from where the dynamic part begins)
  const unsigned dynamic_at = static_cast<unsigned>(__cvta_generic_to_shared(smem_raw));
  unsigned dynamic_bytes;
  asm("mov.u32 %0, %%dynamic_smem_size;" : "=r"(dynamic_bytes));
  if (dynamic_at > kLutTilesAt || kLutEnd > dynamic_at + dynamic_bytes) {  // (not what the constants above were made for)
    if (threadIdx.x == 0 && status != nullptr) ReportFault(status, kFaultBinLayout);
    return;
  }
  unsigned char* window = smem_raw - dynamic_at;
  auto row_of     = [&](int j) { return reinterpret_cast<float*>(window + kLutAt + j * kLutRow); };
  const int f0    = blockIdx.y * kGroup;
  const int lane  = threadIdx.x & 31, warp = threadIdx.x >> 5;
  {
    // a warp reads the proposals of one feature
    float* stage = reinterpret_cast<float*>(window + kLutStageAt);
    const int f  = f0 + warp;
    int begin = 0, n = 0;
    if (f < F) {
      begin = row_ptr[f];
      n     = row_ptr[f + 1] - begin;
    }
    const float* src = proposals + (cut_stride > 0 ? f * cut_stride : begin);
    for (int j = lane; j < kLutRows; j += 32) stage[j * (kGroup + 1) + warp] = j < n ? src[j] : INFINITY;
    if (lane == 0) s_n[warp] = n;
    __syncthreads();
    for (int j = warp; j < kLutRows; j += kLutWarps) row_of(j)[lane] = stage[j * (kGroup + 1) + lane];
  }
  __syncthreads();
  if (threadIdx.x < kGroup) {
    const int n = s_n[threadIdx.x], end = n >= 32 ? 4 : 0;
    float s = 0.0f, b = 0.0f;
    if (n >= 3) {  // (the last proposal is +inf)
      const float lo = row_of(end)[threadIdx.x], hi = row_of(n - 2 - end)[threadIdx.x];
      s = (kBuckets - 3) / (hi - lo) / (kBuckets - 1);
      b = 1.0f / (kBuckets - 1) - lo * s;
      if (!(s > 0.0f) || !(s < INFINITY) || !(fabsf(b) < INFINITY)) s = b = 0.0f;  // all in one bucket
    }
    s_map[threadIdx.x] = make_float2(s, b);
  }
  __syncthreads();
  const float2 map = s_map[lane];
  // the bucket of x plus the bits of 2^23
  auto bucket_bits = [&](float x) {
    float t;
    asm("fma.rn.sat.f32 %0, %1, %2, %3;\n" : "=f"(t) : "f"(x), "f"(map.x), "f"(map.y));  // (NaN: 0)
    return __float_as_uint(__fmaf_rn(t, static_cast<float>(kBuckets - 1), 8388608.0f));
  };
  const unsigned col_s = kLutAt + lane * 4;
  int crowd = 0;  // 1: more than 7 of a feature's proposals share a bucket, 2: more than 15, or they are not in order
  {
    auto at_of  = [&](int j) { return static_cast<int>(bucket_bits(row_of(j)[lane]) & (kBuckets - 1)); };
    auto begins = [&](int k, int j) { reinterpret_cast<unsigned*>(row_of(k))[kGroup + lane] = col_s + j * kLutRow; };
    const int n = s_n[lane];
    for (int j = warp; j < n; j += kLutWarps) {
      const int at = at_of(j);
      for (int k = j > 0 ? at_of(j - 1) + 1 : 0; k <= at; ++k) begins(k, j);
      if (j == n - 1)  // (+inf is in the last bucket, unless all are in the first)
        for (int k = at + 1; k < kBuckets; ++k) begins(k, 0);
      // the table is only right for proposals in order that end in +inf (a NaN among the samples is neither)
      const float v = row_of(j)[lane];
      if (j == n - 1 ? v != INFINITY : !(v < row_of(j + 1)[lane])) crowd |= 2;
      if (j >= 7 && at_of(j - 7) == at) crowd |= 1;
      if (j >= 15 && at_of(j - 15) == at) crowd |= 2;
    }
    if (n == 0)
      for (int k = warp; k < kBuckets; k += kLutWarps) begins(k, 0);
  }
  const int most = __syncthreads_or(crowd & 2) ? 2 : __syncthreads_or(crowd & 1) ? 1 : 0;
  // Lanes beyond the last feature read the last feature's values (in bounds); their column of the
  // table is all +inf, so their ids are 0.
  const bool active     = f0 + lane < F;
  const unsigned lut_s  = col_s + kGroup * 4 - 0x4b000000u * kLutRow;  // (the bits of 2^23)
  // (a team's tiles lie together: the teams that do not fit before the table come after it)
  constexpr int kTeamsBefore = kLutTilesBefore / kLutTeam;
  const unsigned tiles_s = warp / kLutTeam < kTeamsBefore ? kLutTilesAt + warp / kLutTeam * kLutTeam * kLutTile
                                                         : kLutAt + kBuckets * kLutRow + (warp / kLutTeam - kTeamsBefore) * kLutTeam * kLutTile;
  const unsigned tile_s = tiles_s + warp % kLutTeam * kLutTile, team_s = tiles_s + (lane >> 3) * kLutTile;
  const int pitch   = static_cast<int>(gridDim.y) * kGroup;
  constexpr int U   = 8;  // rows per warp in flight
  const int n       = static_cast<int>(n_rows);
  const int ld      = static_cast<int>(ldx);
  constexpr int kTurn = kLutTurn;
  static_assert(kTurn == 4 * U, "four times eight rows");
  const int hop     = static_cast<int>(gridDim.x) * kLutWarps * kTurn;  // rows from one turn of a warp to the next
  const int team    = warp / kLutTeam, mate = warp - team * kLutTeam;
  // the rows of a team follow each other (and a small matrix is spread over the blocks)
  int turn          = ((team * gridDim.x + blockIdx.x) * kLutTeam + mate) * kTurn;
  const float* xcol = X + (active ? f0 + lane : F - 1);
  // the lane's word of the row-major ids: row lane % 4 of four, features lane / 4 * 4 and the next three
  uint8_t* ocol     = bins + static_cast<int64_t>(lane & 3) * pitch + f0 + (lane & ~3);
  const unsigned sel1 = (lane & 1) ? 0x3715u : 0x6240u, sel2 = (lane & 2) ? 0x3276u : 0x5410u;
  // four ids of the lane's feature (one per row) -> the ids of four features in the lane's row
  auto turned = [&](unsigned w) {
    w = __byte_perm(w, __shfl_xor_sync(0xffffffffu, w, 1), sel1);
    return __byte_perm(w, __shfl_xor_sync(0xffffffffu, w, 2), sel2);
  };
  // Sixteen rows of the warp are on their way or searched: the values of eight are asked for as soon as the eight rows
  // sixteen before them have been.
  auto load_rows = [&](int first, float (&x)[U]) {
    const float* src = xcol + static_cast<int64_t>(first) * ld;
#pragma unroll
    for (int u = 0; u < U; ++u, src += ld) x[u] = LdgStream(src);  // (a sum per row: eight offsets would take registers)
  };
  auto load_rows_checked = [&](int first, float (&x)[U]) {
    const float* src = xcol + static_cast<int64_t>(first) * ld;
#pragma unroll
    for (int u = 0; u < U; ++u, src += ld) x[u] = first + u < n ? LdgStream(src) : -INFINITY;
  };
  float xa[U], xb[U];
  load_rows_checked(turn, xa);
  load_rows_checked(turn + U, xb);
  const unsigned swap = lane >> 2;  // the words of a feature's 32 bytes are swapped so that the lanes' stores fall on distinct banks
  // one turn; checked: the turn may reach beyond the last row; levels: steps of the search, 8 = without the buckets
  auto do_turn = [&](auto checked, auto levels) {
    constexpr bool kChecked = decltype(checked)::value;
    constexpr int kLevels   = decltype(levels)::value;
    auto eight_rows = [&](int sub, float (&x)[U]) {
      const int base = turn + sub * U;
      unsigned pos[U];
      if (kLevels == 8) {
#pragma unroll
        for (int u = 0; u < U; ++u) pos[u] = col_s;
      } else {
#pragma unroll
        for (int u = 0; u < U; ++u)
          asm volatile("ld.shared.b32 %0, [%1];\n" : "=r"(pos[u]) : "r"(lut_s + bucket_bits(x[u]) * kLutRow));
      }
      SearchLevels<float, U, kLevels - 1, kLutRow>::run(pos, x);
      if (sub < 2 && !kChecked) load_rows(base + 2 * U, x);
      else if (sub < 2 || turn + hop < n) load_rows_checked(base + 2 * U + (sub < 2 ? 0 : hop - kTurn), x);
      // byte 1 of each, less 128
      const unsigned lo = __byte_perm(__byte_perm(pos[0], pos[1], 0x0051), __byte_perm(pos[2], pos[3], 0x0051), 0x5410) ^ 0x80808080u;
      const unsigned hi = __byte_perm(__byte_perm(pos[4], pos[5], 0x0051), __byte_perm(pos[6], pos[7], 0x0051), 0x5410) ^ 0x80808080u;
      uint8_t* orow = ocol + static_cast<int64_t>(base) * pitch;
      const unsigned first4 = turned(lo), last4 = turned(hi);
      if (!kChecked || base + (lane & 3) < n) *reinterpret_cast<unsigned*>(orow) = first4;
      if (!kChecked || base + 4 + (lane & 3) < n) *reinterpret_cast<unsigned*>(orow + 4 * pitch) = last4;
      if (kCopyT) {
        asm volatile("st.shared.b32 [%0], %1;\n" ::"r"(tile_s + lane * kTurn + ((2 * sub) ^ swap) * 4), "r"(lo) : "memory");
        asm volatile("st.shared.b32 [%0], %1;\n" ::"r"(tile_s + lane * kTurn + ((2 * sub + 1) ^ swap) * 4), "r"(hi) : "memory");
      }
    };
#pragma unroll 1
    for (int sub = 0; sub < 4; sub += 2) {
      eight_rows(sub, xa);
      eight_rows(sub + 1, xb);
    }
    if (kCopyT) {
      // The tiles of the team leave feature by feature, 128 bytes per store (the rows of a warp up to the padded end of a
      // feature's row of the copy; the ids of rows beyond the last one are 0).
      auto meet = [&]() { asm volatile("bar.sync %0, %1;\n" ::"r"(1 + team), "n"(kLutTeam * 32) : "memory"); };
      meet();
      const int row0 = turn - mate * kTurn + 4 * lane;
      uint8_t* dst   = bins_t + static_cast<int64_t>(f0 + mate) * pitch_t + row0;
#pragma unroll 4
      for (int fl = mate; fl < kGroup; fl += kLutTeam) {
#pragma unroll
        for (int piece = 0; piece < kLutTeam / 4; ++piece) {
          unsigned v;
          asm volatile("ld.shared.b32 %0, [%1];\n" : "=r"(v) : "r"(team_s + piece * 4 * kLutTile + fl * kTurn + ((lane & 7) ^ (fl >> 2)) * 4));
          if (f0 + fl < F && (!kChecked || row0 + piece * 128 < pitch_t)) *reinterpret_cast<unsigned*>(dst + piece * 128) = v;
        }
        dst += kLutTeam * pitch_t;
      }
      meet();
    }
  };
  // (every warp of a team takes the same turns; the last ones may have no rows for some of its warps)
  auto all_turns = [&](auto levels) {
    for (; turn + (kLutTeam - mate) * kTurn <= n; turn += hop) do_turn(std::false_type(), levels);
    if (turn - mate * kTurn < n) do_turn(std::true_type(), levels);
  };
  if (most == 0) all_turns(std::integral_constant<int, 3>());
  else if (most == 1) all_turns(std::integral_constant<int, 4>());
  else all_turns(std::integral_constant<int, 8>());
}

// Two-byte ids, more proposals than k_bin_smem's table of 32 features holds: a table of as many features
// (16, 8 or 4) as fill 64 KB, three blocks per SM.  A lane has one feature and eight consecutive rows, which leave as
// one 16-byte store of the feature-major copy; the 32 / kFeatures row groups of a warp may meet in a bank
// (a probe is 1 to 2.5 passes), which costs less than the probes going to L2: 300003 x 37 float64,
// 512 proposals: 70 us with the copy against 425 of k_bin_global.  Small float32 matrices stay with k_bin_global.
//
// With enough rows the search begins from a table of starts and takes three or four steps instead of nine to eleven.  (Two
// blocks and their tables stay within 196 KB: the next larger share of the SM leaves an L1 of 28 KB, which is less than
// the rows on their way: 2M x 64 float32, 2048 proposals: 540 and 660 us.)  Before (three blocks of 256 threads, the whole
// search, a table filled by one load after the other) and now: 300003 x 37 float64, 512 proposals 57.6 -> 51 us (exponential
// columns, which crowd together: 57.3 -> 62), 2048 proposals 152 -> 97; 2M x 64, 512 proposals 342 -> 259; float32, 1024 proposals
// 366 -> 306, 2048 704 -> 540; 10000 x 37 float64 14.2 -> 11.8.
constexpr int kWideTableBytes = 64 * 1024;
constexpr int kWideThreads    = 512;
constexpr int kStartMinRows   = 2500;  // of a block, from which the table of starts (4 us) pays
template <typename T, int kLog2P>
struct WideTable {
  static constexpr int P         = 1 << kLog2P;
  static constexpr int kFeatures = kWideTableBytes / (P * static_cast<int>(sizeof(T)));
  static constexpr size_t kSmem  = (P + kStartSpare) * kFeatures * sizeof(T) + P * kFeatures * sizeof(uint16_t);
};

template <typename T, int kLog2P, bool kCopyT>
__global__ void __launch_bounds__(kWideThreads, 2)
  k_bin_wide(const T* __restrict__ X, int64_t ldx, int64_t n_rows, int F, const T* __restrict__ proposals, int64_t cut_stride,
             const int32_t* __restrict__ row_ptr, int pitch, uint16_t* __restrict__ bins, uint16_t* __restrict__ bins_t, int64_t pitch_t)
{
  AfterTheKernelBefore();
  using Table             = WideTable<T, kLog2P>;
  constexpr int P         = Table::P;
  constexpr int kFeatures = Table::kFeatures;
  constexpr int U         = 8;
  constexpr int kTurn     = 32 / kFeatures * U;  // rows of a warp
  constexpr unsigned kPitch = kFeatures * sizeof(T);
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ int s_begin[kFeatures], s_n[kFeatures];
  __shared__ StartMap s_map[kFeatures];
  T* sp            = reinterpret_cast<T*>(smem_raw);
  uint16_t* starts = reinterpret_cast<uint16_t*>(sp + (P + kStartSpare) * kFeatures);
  const int f0     = blockIdx.y * kFeatures;
  if (f0 >= F) {  // padding columns
    const int64_t all = n_rows * kFeatures;
    for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < all; i += static_cast<int64_t>(gridDim.x) * blockDim.x)
      bins[i / kFeatures * pitch + f0 + i % kFeatures] = 0;
    return;
  }
  FillProposals<T, kFeatures, P + kStartSpare>(sp, s_begin, s_n, proposals, cut_stride, row_ptr, f0, F);
  const int steps = n_rows >= static_cast<int64_t>(gridDim.x) * kStartMinRows ? MakeStarts<T, kFeatures, P, kWideThreads>(sp, starts, s_n, s_map) : 0;
  const int lane = threadIdx.x & 31, fl = lane % kFeatures, f = f0 + fl;
  // lanes beyond the last feature read the last feature's values; their column is all +inf, their ids are 0
  const bool active    = f < F;
  const unsigned col_s = static_cast<unsigned>(__cvta_generic_to_shared(sp + fl));
  const StartMap map   = steps != 0 ? s_map[fl] : StartMap{};
  const T* xcol        = X + (active ? f : F - 1);
  const int n          = static_cast<int>(n_rows);
  const int hop        = static_cast<int>(gridDim.x) * (blockDim.x >> 5) * kTurn;
  auto all_rows = [&](auto levels) {
    constexpr int kLevels = decltype(levels)::value;  // 0: the whole search
    int base = (blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * kTurn + lane / kFeatures * U;
    T xn[U];
    auto load_rows = [&](int first) {
      const T* src = xcol + static_cast<int64_t>(first) * ldx;
#pragma unroll
      for (int u = 0; u < U; ++u, src += ldx) xn[u] = first + u < n ? LdgStream(src) : static_cast<T>(-INFINITY);
    };
    load_rows(base);
    for (; base < n; base += hop) {
      T x[U];
      unsigned pos[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        x[u]   = xn[u];
        pos[u] = col_s;
        if (kLevels != 0) pos[u] += starts[StartBucket<P>(static_cast<float>(x[u]), map) * kFeatures + fl] * kPitch;
      }
      if (base + hop < n) load_rows(base + hop);
      SearchLevels<T, U, (kLevels != 0 ? kLevels : kLog2P) - 1, kPitch>::run(pos, x);
      unsigned id[U];
#pragma unroll
      for (int u = 0; u < U; ++u) id[u] = (pos[u] - col_s) / kPitch;
      uint16_t* out = bins + static_cast<int64_t>(base) * pitch + f;
#pragma unroll
      for (int u = 0; u < U; ++u)
        if (base + u < n) out[static_cast<int64_t>(u) * pitch] = static_cast<uint16_t>(id[u]);
      if (kCopyT && active)  // (the copy's rows are padded to 32; ids beyond the last row are 0)
        *reinterpret_cast<uint4*>(bins_t + static_cast<int64_t>(f) * pitch_t + base) =
          make_uint4(id[0] | (id[1] << 16), id[2] | (id[3] << 16), id[4] | (id[5] << 16), id[6] | (id[7] << 16));
    }
  };
  if (steps == 3) all_rows(std::integral_constant<int, 3>());
  else if (steps == 4) all_rows(std::integral_constant<int, 4>());
  else all_rows(std::integral_constant<int, 0>());
}

// Global-memory variant: more proposals than any table here holds, or too few rows to pay for filling one.
template <typename T, typename BinT>
__global__ void __launch_bounds__(256)
  k_bin_global(const T* __restrict__ X, int64_t ldx, int64_t n_rows, int F, const T* __restrict__ proposals,
               int64_t cut_stride, const int32_t* __restrict__ row_ptr, BinT* __restrict__ bins, BinT* __restrict__ bins_t, int64_t pitch_t)
{
  AfterTheKernelBefore();
  const int g    = blockIdx.y;
  const int f0   = g * kGroup;
  const int lane = threadIdx.x & 31;
  const int f    = f0 + lane;
  const bool active = f < F;
  int begin = 0, n = 0;
  if (active) {
    begin = row_ptr[f];
    n     = row_ptr[f + 1] - begin;
  }
  const T* p = proposals + (cut_stride > 0 && active ? f * cut_stride : begin);
  const int64_t pitch = static_cast<int64_t>(gridDim.y) * kGroup;
  BinT* out  = bins + f0;
  const int64_t warps_total = static_cast<int64_t>(gridDim.x) * (blockDim.x >> 5);
  for (int64_t row = blockIdx.x * static_cast<int64_t>(blockDim.x >> 5) + (threadIdx.x >> 5); row < n_rows;
       row += warps_total) {
    int bin = 0;
    if (active) {
      const T x = X[row * ldx + f];
      int len = n, base = 0;
      while (len > 1) {
        const int half = len >> 1;
        base           = (p[base + half] < x) ? base + half : base;
        len -= half;
      }
      bin = base + ((p[base] < x) ? 1 : 0);
    }
    out[row * pitch + lane] = static_cast<BinT>(bin);
    if (bins_t != nullptr && active) bins_t[static_cast<int64_t>(f) * pitch_t + row] = static_cast<BinT>(bin);
  }
}

// k_bin_wide pays for filling its table from this many cells on
template <typename T>
constexpr int64_t kWideMinCells = sizeof(T) == 8 ? 0 : int64_t{1} << 20;

int NextPow2(int v)
{
  int p = 1;
  while (p < v) p <<= 1;
  return p;
}

}  // namespace

template <typename T>
void Prologue(lbk_context* ctx, Scratch& s, PrologueArgs<T> p, int32_t* row_ptr, int32_t* info, int32_t* info_host,
              double* sums, QuantParams* params, cudaStream_t stream)
{
  p.S_pad       = NextPow2(p.S);
  p.sort_blocks = p.F;
  if (p.counts == nullptr) p.sort_blocks = 0;
  p.sum_blocks = sums != nullptr ? (p.n_elements + kSumBlock - 1) / kSumBlock : 0;
  p.part_g     = s.alloc<double>(static_cast<size_t>(p.sum_blocks) + 1);
  p.part_h     = s.alloc<double>(static_cast<size_t>(p.sum_blocks) + 1);
  if (ctx->n_ranks > 1 && p.sort_blocks > 0) {
    // every rank fills in the sampled rows it holds; the sum over the ranks makes them complete
    const int64_t FS = static_cast<int64_t>(p.F) * p.S;
    T* draft         = s.alloc<T>(FS);
    k_gather_samples<T><<<static_cast<unsigned>((FS + 255) / 256), 256, 0, stream>>>(p, draft);
    LBK_LAUNCH_CHECK();
    AllReduce(ctx, draft, static_cast<size_t>(FS), sizeof(T) == 4 ? LBK_F32 : LBK_F64, LBK_SUM, stream);
    p.draft = draft;
  }
  int64_t fill = p.tree.max_nodes;
  for (int z = 0; z < kZeroRanges; ++z) fill += p.zero_n16[z];
  p.fill_blocks = static_cast<int>(std::min<int64_t>((fill + 4 * kSortThreads - 1) / (4 * kSortThreads), ctx->sm_count * 4));
  const int64_t blocks = p.sort_blocks + p.sum_blocks + p.fill_blocks;
  if (blocks > 0) {
    LaunchChained(k_prologue<T>, static_cast<unsigned>(blocks), kSortThreads, SortSmem<T>(p.S_pad), stream, p);
    LBK_LAUNCH_CHECK();
  }
  const bool one_rank = ctx->n_ranks <= 1;
  LaunchChained(k_prologue_finish, 1, 1024, 0, stream, p.counts, p.F, row_ptr, info, info_host, p.part_g, p.part_h, p.sum_blocks, sums,
                                            one_rank ? params : nullptr);
  LBK_LAUNCH_CHECK();
  if (!one_rank && sums != nullptr) {
    AllReduce(ctx, sums, 2, LBK_F64, LBK_MAX, stream);
    k_make_scale<<<1, 1, 0, stream>>>(sums, params);
    LBK_LAUNCH_CHECK();
  }
}

template <typename T>
ProposalInfo SplitProposals(lbk_context* ctx, Scratch& s, const T* X, int64_t ldx, int64_t row_offset, int64_t n_local,
                   int F, int S, int seed, int64_t dataset_rows, T* proposals, int32_t* row_ptr,
                   cudaStream_t stream)
{
  PrologueArgs<T> p{};
  p.X            = X;
  p.ldx          = ldx;
  p.row_offset   = row_offset;
  p.n_local      = n_local;
  p.F            = F;
  p.S            = S;
  p.seed         = seed;
  p.dataset_rows = dataset_rows;
  p.cuts         = s.alloc<T>(static_cast<size_t>(F) * S);
  p.counts       = s.alloc<int32_t>(F);
  int32_t* info  = s.alloc<int32_t>(2);
  Prologue<T>(ctx, s, p, row_ptr, info, nullptr, nullptr, nullptr, stream);
  LaunchChained(k_write_proposals<T>, F, 128, 0, stream, p.cuts, S, row_ptr, proposals);
  LBK_LAUNCH_CHECK();
  int32_t h[2] = {0, 0};
  LBK_CUDA(cudaMemcpyAsync(h, info, sizeof(h), cudaMemcpyDeviceToHost, stream));
  LBK_CUDA(cudaStreamSynchronize(stream));
  return ProposalInfo{h[0], h[1]};
}

// Rows that take a block as long as filling its table: about 10 us.
constexpr int64_t kLutFillRows = 2048, kSmemFillRows = 512;

template <typename T>
void BinMatrix(const T* X, int64_t ldx, int64_t n_rows, int F, const T* proposals, int64_t cut_stride, const int32_t* row_ptr,
               void* bins, void* bins_t, int64_t pitch_t, int bin_bytes, int max_bins_per_feature, int* status,
               cudaStream_t stream)
{
  if (n_rows <= 0) return;
  LBK_EXPECT(n_rows <= 2000000000ll && ldx <= (1 << 27), "bin_matrix: at most 2e9 rows per rank and a row pitch of 2^27 elements");
  const int G           = (F + kGroup - 1) / kGroup;
  // the shared-memory table is padded to one of a few sizes (each is its own fully unrolled kernel)
  const int need   = NextPow2(max_bins_per_feature);
  const int log2p  = need <= 16 ? 4 : need <= 64 ? 6 : need <= 256 ? 8 : 9;
  // the table, and one tile per warp for the feature-major copy of one-byte ids
  const size_t table    = sizeof(T) * static_cast<size_t>(kGroup) * (size_t{1} << log2p);
  const size_t smem     = table + (bins_t != nullptr && bin_bytes == 1 ? size_t{8} * kGroup * kBinTilePitch : 0);
  const bool use_smem   = need <= 512 && table <= 96 * 1024;
  // a block fills its table once and then walks the rows with a grid stride: whole waves of what is resident at once
  // (from the occupancy calculator), spread over the tables (bin_grid.h)
  auto blocks_of = [&](int64_t tables, int blocks_per_sm, int64_t fill_rows) {
    int sms = 148;
    int dev = 0;
    if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    return static_cast<unsigned>(BinGridBlocks(n_rows, tables, static_cast<int64_t>(sms) * (blocks_per_sm > 0 ? blocks_per_sm : 1), fill_rows));
  };
  auto make_grid = [&](int blocks_per_sm, int64_t fill_rows) { return dim3(blocks_of(G, blocks_per_sm, fill_rows), G); };
#define LBK_BIN_SMEM2(BinT, L, CT)                                                                        \
  do {                                                                                                    \
    auto fn_ = k_bin_smem<T, BinT, L, CT>;                                                                \
    if (smem > 48 * 1024)                                                                                 \
      LBK_CUDA(cudaFuncSetAttribute(fn_, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem))); \
    int per_sm_ = 0;                                                                                      \
    LBK_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm_, fn_, 256, smem));                    \
    LaunchChained(fn_, make_grid(per_sm_, kSmemFillRows), 256, smem, stream, X, ldx, n_rows, F, proposals, cut_stride, row_ptr,                 \
                                                   static_cast<BinT*>(bins), static_cast<BinT*>(bins_t), pitch_t); \
  } while (0)
#define LBK_BIN_SMEM(BinT, L)                                                                             \
  do {                                                                                                    \
    if (bins_t != nullptr) LBK_BIN_SMEM2(BinT, L, true); else LBK_BIN_SMEM2(BinT, L, false);              \
  } while (0)
#define LBK_BIN_LAUNCH(BinT)                                                                              \
  do {                                                                                                    \
    if (use_smem) {                                                                                       \
      if (log2p == 4) LBK_BIN_SMEM(BinT, 4);                                                              \
      else if (log2p == 6) LBK_BIN_SMEM(BinT, 6);                                                         \
      else if (log2p == 8) LBK_BIN_SMEM(BinT, 8);                                                         \
      else LBK_BIN_SMEM(BinT, 9);                                                                         \
    } else {                                                                                              \
      LaunchChained(k_bin_global<T, BinT>, make_grid(8, 0), 256, 0, stream, X, ldx, n_rows, F, proposals, cut_stride, row_ptr,     \
                                                       static_cast<BinT*>(bins), static_cast<BinT*>(bins_t), \
                                                       pitch_t);                                          \
    }                                                                                                     \
  } while (0)
  if constexpr (sizeof(T) == 4) {
    // (words of four row-major ids: an array on an odd boundary is left to k_bin_smem)
    if (bin_bytes == 1 && log2p == 8 && (reinterpret_cast<uintptr_t>(bins) & 3) == 0) {
      auto fn = bins_t != nullptr ? k_bin_lut<true> : k_bin_lut<false>;
      LBK_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kLutEnd)));
      LaunchChained(fn, make_grid(1, kLutFillRows), kLutThreads, kLutEnd, stream, X, ldx, n_rows, F, proposals, cut_stride, row_ptr, static_cast<uint8_t*>(bins),
                                                  static_cast<uint8_t*>(bins_t), pitch_t, status);
      LBK_LAUNCH_CHECK();
      return;
    }
  }
  if (bin_bytes == 2 && !use_smem && need <= 2048 && n_rows * F >= kWideMinCells<T> && Aligned16(bins_t)) {
    auto wide = [&](auto log2p_, auto copy_) {
      constexpr int L    = decltype(log2p_)::value;
      constexpr bool CT  = decltype(copy_)::value;
      using Table = WideTable<T, L>;
      constexpr int kFeatures = Table::kFeatures;
      auto fn = k_bin_wide<T, L, CT>;
      LBK_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(Table::kSmem)));
      // (two blocks per SM, spread over the tables that hold features)
      const dim3 grid(blocks_of((F + kFeatures - 1) / kFeatures, 2, kSmemFillRows), G * kGroup / kFeatures);
      LaunchChained(fn, grid, kWideThreads, Table::kSmem, stream, X, ldx, n_rows, F, proposals, cut_stride, row_ptr, G * kGroup,
                                                 static_cast<uint16_t*>(bins), static_cast<uint16_t*>(bins_t), pitch_t);
    };
    auto by_copy = [&](auto log2p_) {
      if (bins_t != nullptr) wide(log2p_, std::true_type());
      else wide(log2p_, std::false_type());
    };
    if (need <= 512 && sizeof(T) == 8) by_copy(std::integral_constant<int, sizeof(T) == 8 ? 9 : 10>());
    else if (need <= 1024) by_copy(std::integral_constant<int, 10>());
    else by_copy(std::integral_constant<int, 11>());
  } else if (bin_bytes == 1) {
    LBK_BIN_LAUNCH(uint8_t);
  } else {
    LBK_BIN_LAUNCH(uint16_t);
  }
#undef LBK_BIN_SMEM
#undef LBK_BIN_SMEM2
#undef LBK_BIN_LAUNCH
  LBK_LAUNCH_CHECK();
}

template ProposalInfo SplitProposals<float>(lbk_context*, Scratch&, const float*, int64_t, int64_t, int64_t, int, int, int,
                                   int64_t, float*, int32_t*, cudaStream_t);
template ProposalInfo SplitProposals<double>(lbk_context*, Scratch&, const double*, int64_t, int64_t, int64_t, int, int, int,
                                    int64_t, double*, int32_t*, cudaStream_t);
template void Prologue<float>(lbk_context*, Scratch&, PrologueArgs<float>, int32_t*, int32_t*, int32_t*, double*, QuantParams*,
                              cudaStream_t);
template void Prologue<double>(lbk_context*, Scratch&, PrologueArgs<double>, int32_t*, int32_t*, int32_t*, double*,
                               QuantParams*, cudaStream_t);
template void BinMatrix<float>(const float*, int64_t, int64_t, int, const float*, int64_t, const int32_t*, void*, void*, int64_t,
                               int, int, int*, cudaStream_t);
template void BinMatrix<double>(const double*, int64_t, int64_t, int, const double*, int64_t, const int32_t*, void*, void*,
                                int64_t, int, int, int*, cudaStream_t);

}  // namespace lbk
