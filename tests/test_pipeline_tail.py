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
  if (tail) stb::ring_tail(count, stages, [&](int s, int parity) { ok = ok && wait(s, parity); });
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
