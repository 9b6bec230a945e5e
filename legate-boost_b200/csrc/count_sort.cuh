// The place of a value among a few hundred in shared memory: how many are smaller.  Equal values have the same place, which
// is what proposals want (each once), and all places are found at once, without the 36 dependent steps of a bitonic
// network for 256 values.
#pragma once
#include <cuda_runtime.h>

namespace lbk {

// Smaller ones among vals[0 .. 16 / sizeof(T) * n_vec), which begins on a 16-byte boundary; the lanes of a warp read the same
// words.
template <typename T>
__device__ inline int CountBelow(const T* vals, int n_vec, T mine)
{
  constexpr int kPer = 16 / sizeof(T);
  const float4* at   = reinterpret_cast<const float4*>(vals);
  int below          = 0;
#pragma unroll 8
  for (int i = 0; i < n_vec; ++i) {
    const float4 w = at[i];
#pragma unroll
    for (int e = 0; e < kPer; ++e) below += reinterpret_cast<const T*>(&w)[e] < mine ? 1 : 0;
  }
  return below;
}

}  // namespace lbk
