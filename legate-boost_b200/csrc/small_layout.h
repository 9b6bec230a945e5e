// Where a level of the one-launch tree (small_tree.cu) leaves its split candidates.
//
// Blocks meet at one barrier per level: they write the level's candidates before it and read them after it, while
// blocks that are done with that already write the next level's.  Neighbouring levels therefore lie in two different
// regions, taken in turn: a block that writes level d + 2 over level d has passed the barrier of level d + 1, which
// no block reaches before it has read level d.
#pragma once

#ifdef __CUDACC__
#define LBK_HOST_DEVICE __host__ __device__
#else
#define LBK_HOST_DEVICE
#endif

namespace lbk {

// Nodes of the region that the last level (depth D - 1) takes; the other one is half of it.
LBK_HOST_DEVICE inline int SmallCandTop(int D) { return D > 1 ? 1 << (D - 1) : 1; }
// First node of level `depth` of a tree of depth D, and the nodes of both regions.
LBK_HOST_DEVICE inline int SmallCandBegin(int depth, int D) { return ((D - 1 - depth) & 1) != 0 ? SmallCandTop(D) : 0; }
LBK_HOST_DEVICE inline int SmallCandNodes(int D) { return SmallCandTop(D) + (SmallCandTop(D) + 1) / 2; }

}  // namespace lbk
