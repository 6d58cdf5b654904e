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

// A ring of `stages` barriers of which use k ends phase k / stages of barrier k % stages: after
// `count` uses, wait(barrier, parity) is called for the last use of every barrier that had one.
// (The uses before those have ended: a barrier's next use waits for its last one.)
template <typename Wait>
STB_HD void ring_tail(int count, int stages, Wait wait) {
  for (int k = count > stages ? count - stages : 0; k < count; ++k) wait(k % stages, (k / stages) & 1);
}

// The copies of a CTA pair.  Both CTAs load half of each k-block into a stage of their own and both
// halves complete on rank 0's barrier, whose phase expects the two together.  When a pair gives up, its
// ranks may have issued different numbers of k-blocks (never more than `stages` apart: a stage is
// filled again only after both halves were used).  Rank 0 makes its barriers expect what was really
// issued, then waits for it: expect(barrier) stands in for its own share of a block that only rank 1
// loads, forgive(barrier) takes back rank 1's half of a block that only rank 0 loads.
template <typename Expect, typename Forgive, typename Wait>
STB_HD void pair_copies_tail(int mine, int theirs, int stages, Expect expect, Forgive forgive, Wait wait) {
  const int most = mine > theirs ? mine : theirs;
  for (int k = most > stages ? most - stages : 0; k < most; ++k) {
    if (k >= mine)
      expect(k % stages);
    else if (k >= theirs)
      forgive(k % stages);
    wait(k % stages, (k / stages) & 1);
  }
}

}  // namespace stb
