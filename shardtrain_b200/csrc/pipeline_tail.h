// Which barrier phases a CTA has to see ended before it may give up its shared memory.
//
// TMA copies and tcgen05.commit arrivals are asynchronous: they land in a CTA's shared memory on
// their own time, and nothing orders one commit's arrival behind another's.  A CTA that leaves while
// one is still on its way lets it land in memory that may belong to the next CTA by then.  The index
// arithmetic sits here, apart from the kernels, so that it can be run against a model on the host.
#pragma once

#ifdef __CUDACC__
#define STB_HD __host__ __device__ __forceinline__
#else
#define STB_HD inline
#endif

namespace stb {

// A ring of `stages` barriers of which use k ends a phase of barrier k % stages: how many phases of
// barrier `s` the first `count` uses end.  (Waiting for the last of them is enough: a barrier's next use
// waits for the one before.)
STB_HD int ring_uses(int count, int stages, int s) { return count > s ? (count - s - 1) / stages + 1 : 0; }

// The copies of a CTA pair.  Both CTAs load half of each k-block into a stage of their own and both
// halves complete on rank 0's barrier, whose phase expects the two together.  When a pair gives up, its
// ranks may have issued different numbers of k-blocks (never more than `stages` apart: a stage is
// filled again only after both halves were used).  Rank 0 makes its barriers expect what was really
// issued, then waits for it.
struct PairStage {
  int uses;       // phases of rank 0's barrier to wait for
  bool expect;    // rank 1 has loaded a block that rank 0 has not: stand in for rank 0's arrival
  bool forgive;   // rank 0 has loaded a block that rank 1 has not: take rank 1's half back
};
STB_HD PairStage pair_stage(int mine, int theirs, int stages, int s) {
  const int a = ring_uses(mine, stages, s), b = ring_uses(theirs, stages, s);
  return PairStage{a > b ? a : b, b > a, a > b};
}

}  // namespace stb
