"""What a CTA waits for before it gives up its shared memory, run on the host against a model in which
asynchronous arrivals land in any order (csrc/pipeline_tail.h is compiled by g++ here)."""

import subprocess
from pathlib import Path

CSRC = Path(__file__).resolve().parents[1] / "shardtrain_b200" / "csrc"

MODEL = r"""
#include <cstdio>
#include <deque>
#include <random>
#include <vector>
#include "pipeline_tail.h"

// A ring of one-arrival barriers: phase[s] phases of barrier s have ended.
struct Ring {
  std::vector<int> phase;
  std::deque<int> pending;      // commits on their way, by barrier
  explicit Ring(int stages) : phase(stages, 0) {}
  void land(size_t i) { ++phase[pending[i]]; pending.erase(pending.begin() + i); }
  bool ended(int s, int parity) const { return (phase[s] & 1) != parity; }   // mbarrier.try_wait.parity
};

// `count` k-blocks: the copies of block k wait until its stage was freed by block k - stages, then a
// commit frees it again.  Commits land at random, out of order.  Returns the arrivals still on
// their way when the CTA leaves, with or without the waits of the tail.
int leave(int count, int stages, bool tail, std::mt19937& rng) {
  Ring ring(stages);
  auto wait = [&](int s, int parity) {
    while (!ring.ended(s, parity)) {
      if (ring.pending.empty()) return false;          // would wait for good
      ring.land(rng() % ring.pending.size());
    }
    return true;
  };
  for (int k = 0; k < count; ++k) {
    if (!wait(k % stages, ((k / stages) & 1) ^ 1)) return -1;
    ring.pending.push_back(k % stages);
    if (rng() % 2 && !ring.pending.empty()) ring.land(rng() % ring.pending.size());
  }
  bool ok = true;
  for (int s = 0; tail && s < stages; ++s) {
    const int uses = stb::ring_uses(count, stages, s);
    if (uses > 0) ok = ok && wait(s, (uses - 1) & 1);
  }
  return ok ? static_cast<int>(ring.pending.size()) : -1;
}

int main() {
  std::mt19937 rng(7);
  int left_without = 0;
  for (int stages : {1, 2, 3, 6, 8})
    for (int count = 0; count <= 3 * stages + 2; ++count)
      for (int trial = 0; trial < 200; ++trial) {
        const int left = leave(count, stages, true, rng);
        if (left != 0) return std::printf("stages %d count %d: %d\n", stages, count, left), 1;
        left_without += leave(count, stages, false, rng) > 0;
      }
  if (left_without == 0) return std::printf("the model never leaves early\n"), 1;
  return 0;
}
"""


def run_model(tmp_path, source):
    (tmp_path / "model.cpp").write_text(source)
    binary = tmp_path / "model"
    subprocess.run(["g++", "-std=c++17", "-O1", f"-I{CSRC}", str(tmp_path / "model.cpp"), "-o", str(binary)],
                   check=True)
    done = subprocess.run([str(binary)], capture_output=True, text=True, timeout=120)
    assert done.returncode == 0, done.stdout


def test_a_pipeline_leaves_no_arrival_behind(tmp_path):
    run_model(tmp_path, MODEL)


PAIR_MODEL = r"""
#include <cstdio>
#include <random>
#include <vector>
#include "pipeline_tail.h"

// One arrival per phase; a phase ends once it has arrived and the announced bytes have come (which may
// happen before they are announced).
struct Barrier {
  int phase = 0, arrivals = 0;
  long tx = 0;
  void settle() { if (arrivals == 1 && tx == 0) { ++phase; arrivals = 0; } }
  void expect(long bytes) { tx += bytes; ++arrivals; settle(); }
  void complete(long bytes) { tx -= bytes; settle(); }
  bool ended(int parity) const { return (phase & 1) != parity; }
};
struct Copy { int block, rank; };
constexpr long kHalf = 3;

int give_up(int stages, int consumed, int mine, int theirs, bool fix, std::mt19937& rng) {
  std::vector<Barrier> full(stages);
  std::vector<Copy> flying;
  auto land = [&](size_t i) {
    full[flying[i].block % stages].complete(kHalf);
    flying.erase(flying.begin() + i);
  };
  for (int k = 0; k < (mine > theirs ? mine : theirs); ++k) {
    for (int rank = 0; rank < 2; ++rank)
      if (k < (rank ? theirs : mine)) flying.push_back({k, rank});
    if (k < mine) full[k % stages].expect(2 * kHalf);
    if (k < consumed)                               // the MMAs took block k before its stage was reused
      while (!flying.empty() && flying.front().block <= k) land(0);
  }
  while (!flying.empty() && rng() % 4) land(rng() % flying.size());
  bool ok = true;
  auto wait = [&](int s, int parity) {
    while (ok && !full[s].ended(parity)) {
      if (flying.empty()) ok = false; else land(rng() % flying.size());
    }
  };
  for (int s = 0; s < stages; ++s) {
    stb::PairStage stage = stb::pair_stage(mine, theirs, stages, s);
    if (!fix) stage = {stb::ring_uses(mine, stages, s), false, false};
    if (stage.expect) full[s].expect(kHalf);
    if (stage.forgive) full[s].complete(kHalf);
    if (stage.uses > 0) wait(s, (stage.uses - 1) & 1);
  }
  return ok ? static_cast<int>(flying.size()) : -1;
}

int main() {
  std::mt19937 rng(11);
  int wrong_without = 0;
  for (int stages : {1, 2, 3, 6, 8})
    for (int consumed = 0; consumed <= 2 * stages + 1; ++consumed)
      for (int mine = consumed; mine <= consumed + stages; ++mine)
        for (int theirs = consumed; theirs <= consumed + stages; ++theirs)
          for (int trial = 0; trial < 40; ++trial) {
            const int left = give_up(stages, consumed, mine, theirs, true, rng);
            if (left != 0)
              return std::printf("stages %d consumed %d loads %d %d: %d\n", stages, consumed, mine, theirs, left), 1;
            wrong_without += give_up(stages, consumed, mine, theirs, false, rng) != 0;
          }
  if (wrong_without == 0) return std::printf("the model never leaves early\n"), 1;
  return 0;
}
"""


def test_a_pair_that_gives_up_waits_for_what_each_rank_issued(tmp_path):
    run_model(tmp_path, PAIR_MODEL)
