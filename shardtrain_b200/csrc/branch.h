// Work of a launch sequence that nothing after it in the sequence reads (or only much later): a branch of
// its graph while the sequence is being captured, the same launches in line otherwise -- also where the
// second stream cannot be made or the fork fails.  `stream()` is where the branch's kernels go; `join()`
// makes the sequence wait for them.
//
// A stream that forked from a capture belongs to it until that capture ENDS, not until the join: nobody
// else may use it in between.  So whoever captures owns the second stream (SideStreams, under the lock of
// the replay cache) and hands it to the sequence.  A sequence that was given none runs in line, also
// when it finds its stream in a capture that somebody else began.
//
// `Api` is the CUDA runtime (or a stand-in on the host): Stream, Event, device, make_stream, make_event,
// drop_event, record, wait, clear_error, chain_break; those that can fail say whether they succeeded.
#pragma once

#include <map>
#include <stdexcept>

namespace stb {

template <class Api>
struct SideStream {
  typename Api::Stream stream{};
  typename Api::Event fork{}, join{};
};

// The second streams of one owner, per device (a process drives one; a second one gets its own).  Whoever
// uses them holds the owner's lock from the begin of a capture to its end.
template <class Api>
class SideStreams {
 public:
  // null where it cannot be made; tried again the next time
  SideStream<Api>* get() {
    SideStream<Api>& s = table_[Api::device()];
    if (s.stream != typename Api::Stream{}) return &s;
    SideStream<Api> made{};
    const bool fork = Api::make_event(&made.fork), join = fork && Api::make_event(&made.join);
    if (join && Api::make_stream(&made.stream)) {
      s = made;
      return &s;
    }
    if (join) Api::drop_event(made.join);
    if (fork) Api::drop_event(made.fork);
    Api::clear_error();
    return nullptr;
  }

 private:
  std::map<int, SideStream<Api>> table_;
};

template <class Api>
class Branch {
 public:
  using Stream = typename Api::Stream;
  // `side`: of the capture that `main` is in; null outside one
  Branch(Stream main, SideStream<Api>* side) : main_(main) {
    if (side == nullptr) return;
    if (Api::record(side->fork, main) && Api::wait(side->stream, side->fork)) {
      side_ = side;
      Api::chain_break();
    } else {
      Api::clear_error();
    }
  }
  Stream stream() const { return side_ != nullptr ? side_->stream : main_; }
  void join() {
    if (side_ == nullptr) return;
    if (!Api::record(side_->join, side_->stream) || !Api::wait(main_, side_->join))
      throw std::runtime_error("shardtrain_b200: a branch of a launch sequence could not be joined");
    Api::chain_break();
    side_ = nullptr;
  }

 private:
  Stream main_;
  SideStream<Api>* side_ = nullptr;
};

}  // namespace stb
