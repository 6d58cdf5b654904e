// Work of a launch sequence that nothing after it in the sequence reads (or only much later): a branch of
// its graph while the sequence is being captured, the same launches in line otherwise -- also where the
// second stream cannot be made or the fork fails.  `stream()` is where the branch's kernels go; `join()`
// makes the sequence wait for them.
//
// `Api` is the CUDA runtime (or a stand-in on the host): Stream, Event, capturing, device, make_stream,
// make_event, record, wait, clear_error, chain_break; record and wait say whether they succeeded.
#pragma once

#include <map>
#include <mutex>
#include <stdexcept>

namespace stb {

// One second stream and two events per device serve all captures: a branch holds their lock from its
// fork to its join, and none when it runs in line.
template <class Api>
class Branch {
 public:
  using Stream = typename Api::Stream;
  using Event = typename Api::Event;
  explicit Branch(Stream main) : main_(main) {
    if (!Api::capturing(main)) return;
    lock_ = std::unique_lock<std::mutex>(mutex());
    Shared& shared = streams();
    if (shared.side != Stream{} && Api::record(shared.fork, main) && Api::wait(shared.side, shared.fork)) {
      side_ = shared.side;
      Api::chain_break();
    } else {
      Api::clear_error();
      lock_.unlock();
    }
  }
  Stream stream() const { return side_ != Stream{} ? side_ : main_; }
  void join() {
    if (side_ == Stream{}) return;
    Shared& shared = streams();
    if (!Api::record(shared.join, side_) || !Api::wait(main_, shared.join))
      throw std::runtime_error("shardtrain_b200: a branch of a launch sequence could not be joined");
    Api::chain_break();
    side_ = Stream{};
    lock_.unlock();
  }

 private:
  struct Shared {
    Stream side{};
    Event fork{}, join{};
  };
  static std::mutex& mutex() {
    static std::mutex m;
    return m;
  }
  // per device (a process drives one; a second one gets its own)
  static Shared& streams() {
    static std::map<int, Shared> table;
    Shared& s = table[Api::device()];
    if (s.side == Stream{} && !(Api::make_event(&s.fork) && Api::make_event(&s.join) && Api::make_stream(&s.side)))
      s = Shared{};
    return s;
  }
  Stream main_, side_{};
  std::unique_lock<std::mutex> lock_;
};

}  // namespace stb
