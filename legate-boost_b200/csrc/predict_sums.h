// How many sums a row has in the registers of k_predict_tiled (predict.cu).
#pragma once

namespace lbk {

constexpr int kRegisterSums = 16;  // outputs whose sums a warp keeps in registers

// KR of the kernel for K outputs.  0: one output, whose leaf values are in the records; -1: sums in shared memory.  Two to four outputs
// have as many sums; more have the next even number, since sums beyond K are loaded, added and dropped, and a kernel for every
// number would be half as many again for one sum of six at most.  Five and six outputs with eight sums, and thirteen
// and fourteen with sixteen, 300k x 20, 100 trees of depth 6: 257, 206, 350, 318 us; with six and fourteen 232, 194, 344, 300.
constexpr int SumsOf(int K) { return K == 1 ? 0 : K > kRegisterSums ? -1 : K <= 4 ? K : (K + 1) / 2 * 2; }

}  // namespace lbk
