"""Branches of a captured launch sequence (csrc/branch.h), run on the host against a stand-in for the CUDA
runtime: whatever fails on the way to a second stream, the launches go in line and nothing stays locked; and a
sequence branches only where the capture that it is part of gave it a second stream."""
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "shardtrain_b200" / "csrc"

MODEL = r"""
#include <cstdio>
#include <cstring>
#include <string>
#include <vector>
#include "branch.h"

struct Fake {
  using Stream = int;                 // 0: none
  using Event = int;
  static inline std::string fails;    // which call fails
  static inline std::vector<std::string> log;
  static inline int made = 10, events = 0, cleared = 0;
  static int device() { return 0; }
  static bool make_event(Event* e) { return fails != "event" && (*e = ++made, ++events, true); }
  static void drop_event(Event) { --events; }
  static bool make_stream(Stream* s) { return fails != "stream" && (*s = 7, true); }
  static bool record(Event, Stream s) { return log.push_back("record " + std::to_string(s)), fails != "record"; }
  static bool wait(Stream s, Event) { return log.push_back("wait " + std::to_string(s)), fails != "wait"; }
  static void clear_error() { ++cleared; }
  static void chain_break() { log.push_back("break"); }
};
using Branch = stb::Branch<Fake>;
using Side = stb::SideStream<Fake>;

int main(int argc, char** argv) {
  Fake::fails = argv[1];
  {                                   // somebody else's capture, or none: in line, nothing is touched
    Branch none(1, nullptr);
    if (none.stream() != 1) return std::printf("forked\n"), 1;
    none.join();
    if (!Fake::log.empty()) return std::printf("touched\n"), 1;
  }
  stb::SideStreams<Fake> sides;
  int captures = 0;
  const int want = Fake::fails == "nothing" ? 7 : 1;
  for (int i = 0; i < 3; ++i) {       // three in one scope, as a layer's backward has them
    Side* side = sides.get();
    captures += side == nullptr;
    Branch a(1, side);
    if (a.stream() != want) return std::printf("stream %d\n", a.stream()), 1;
    a.join();
    if (a.stream() != 1) return std::printf("after join\n"), 1;
    Branch b(1, side);
    if (b.stream() != want) return std::printf("second stream %d\n", b.stream()), 1;
    b.join();
  }
  if (Fake::events != (captures != 0 ? 0 : 2)) return std::printf("%d events left\n", Fake::events), 1;
  if (want == 7) {
    const std::vector<std::string> one = {"record 1", "wait 7", "break", "record 7", "wait 1", "break"};
    for (size_t i = 0; i < Fake::log.size(); ++i)
      if (Fake::log[i] != one[i % one.size()]) return std::printf("call %zu: %s\n", i, Fake::log[i].c_str()), 1;
    return Fake::log.size() != 6 * one.size();
  }
  // what failed leaves no error behind for the next launch to report
  return Fake::cleared != (captures != 0 ? captures : 6);
}
"""


@pytest.fixture(scope="module")
def model(tmp_path_factory):
    folder = tmp_path_factory.mktemp("branch")
    (folder / "model.cpp").write_text(MODEL)
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", f"-I{CSRC}", str(folder / "model.cpp"), "-o",
                    str(folder / "model")], check=True)
    return folder / "model"


@pytest.mark.parametrize("fails", ["nothing", "event", "stream", "record", "wait"])
def test_launches_go_in_line_where_there_is_no_branch(model, fails):
    done = subprocess.run([str(model), fails], capture_output=True, text=True, timeout=20)
    assert done.returncode == 0, done.stdout
