// How a block of k_hist_smem (histogram.cu) shares the features of its unit of work among the lanes of a row: which bytes of the row a
// lane loads, which it adds to which word of a bin.
#pragma once

#ifdef __CUDACC__
#define LBK_HOST_DEVICE __host__ __device__
#else
#define LBK_HOST_DEVICE
#endif

namespace lbk {

// How the lanes of k_hist_smem share the nt features of a unit: `main` neighbouring bytes a lane and `extra` ones.  Each of the
// two takes a power of two of features and eight (W = 1: the main ones sixteen) columns of words for each lane of a row, so that
// fewer features have several copies of their words and a step still updates 32 banks; 2 (main + extra) reductions are issued per
// batch of rows instead of 32.  Whole numbers use it where a row is one unit: 8M x 40, 4 nodes 200 -> 185 us, 10M x 40, depth 8
// 2.65 -> 2.62 ms.  Of several units the last one keeps its 16 steps, so that the units' blocks go through the rows at one
// pace and share the 128-byte lines of a row in L2: with the steps it needs (and blocks dealt by what a unit costs) 8M x 72
// took 427 -> 528 us and 10M x 200, depth 8, 8.7 -> 9.6 ms, without the dealing 1M x 72, ten outputs, 6.93 -> 7.15 ms.
// Floating-point reductions are loops where another one of the same word is on its way, and the columns that pad a row all fall
// into their bin 0: there every unit has the steps it needs, and lanes without a feature leave a step out (HistRows, kMask).
// 3M x 100 1222 -> 429 us, 3M x 20 341 -> 151, 3M x 64 256 -> 242.
struct UnitForm {
  int main, extra;
};
LBK_HOST_DEVICE constexpr UnitForm FormOf(bool is_float, int W, bool several_units, int nt)
{
  if (W == 1) return {nt > 16 ? 16 : nt > 8 ? 8 : 4, 0};
  if (nt > 48 || (!is_float && several_units)) return {8, 8};
  if (!is_float) return {8, 4};
  if (nt > 32) return {8, nt > 40 ? 4 : nt > 36 ? 2 : 1};
  return {nt > 16 ? 8 : nt > 8 ? 4 : 2, 0};
}
// Feature (relative to the unit's first) of histogram word w of a bin, -1 where the word is a copy of another one.
LBK_HOST_DEVICE constexpr int FeatureOfWord(int W, UnitForm fm, int w)
{
  if (W == 1) {
    const int q = w >> 4, col = w & 15;
    return col < fm.main ? fm.main * q + col : -1;
  }
  const int half = w >> 5, q = (w >> 3) & 3, col = w & 7;
  if (col >= (half == 0 ? fm.main : fm.extra)) return -1;
  if (fm.extra == 8) return 16 * q + 8 * half + col;
  if (fm.extra == 0) return fm.main * q + col;
  // 33 to 48 features: lanes 0 and 3 share the first 16 bytes, lanes 1 and 2 have the next 32
  if (half == 0) {
    if (fm.extra == 1 && q == 2 && col >= 4) return 24 + (col - 4);
    return (q == 0 ? 0 : q == 3 ? 8 : 16 * q) + col;
  }
  if (fm.extra == 1) return 28 + q;
  if (fm.extra == 2) return 24 + 2 * q + col;
  return (q == 0 ? 28 : q == 1 ? 24 : q == 2 ? 40 : 44) + col;
}

// The 2 W lanes of a row load LaneBytes neighbouring bytes each, lane q (0, 1 ...) the PieceOfLane-th of the unit's `groups` x 32.  A matrix
// may end with its last row, so that no lane reads beyond these: where a unit of 16 steps has one group only (the last of an odd
// number), lanes 2 and 3 load the pieces of lanes 0 and 1 once more, and what they add goes to words without a feature, which
// the flush leaves out.  One level of 64 nodes, 10M x 72: 591 us, 10M x 96: 592 (10M x 64, one unit: 357).
LBK_HOST_DEVICE constexpr int LaneBytes(UnitForm fm) { return fm.extra != 0 ? 16 : fm.main; }
LBK_HOST_DEVICE constexpr int PieceOfLane(int W, UnitForm fm, int groups, int q)
{
  if ((fm.extra == 1 || fm.extra == 2 || fm.extra == 4) && q == 3) return 0;
  if (fm.extra == 8 && groups == 1) return q & 1;
  return q;
}

}  // namespace lbk
