// Whether the counters at the head of the split's scratch are zero, which a small sort relies on and leaves behind it when it runs to
// its end. They are not in new scratch, nor after a sort that was enqueued only in part or failed. Host logic only.
#pragma once
#include <cstddef>

namespace gqs {

// Which scratch the device had no room for. A sort that needs as much goes without the split, like one that cannot use it, and does
// not ask again; smaller ones, and all of them after forget(), may.
class SplitRoom {
  size_t refused_ = ~(size_t)0;

 public:
  bool may_hold(size_t bytes) const { return bytes < refused_; }
  void refuse(size_t bytes) {
    if (bytes < refused_) refused_ = bytes;
  }
  void forget() { refused_ = ~(size_t)0; }
};

class SplitCounters {
  bool unclear_ = false;

 public:
  void spoil() { unclear_ = true; }
  bool unclear() const { return unclear_; }
  void cleared() { unclear_ = false; }

  // Enqueues one sort with launch(), behind clear() if the counters may not be zero; both return a status, S{} for success. In a
  // stream that is being captured (captured(), asked only after a clearing) neither has run when this returns: the graph clears
  // them for itself.
  template <class S, class Captured, class Clear, class Launch>
  S enqueue(Captured&& captured, Clear&& clear, Launch&& launch) {
    const bool was = unclear_;
    if (was) {
      const S e = clear();
      if (e != S{}) return e;
    }
    unclear_ = true;
    const S e = launch();
    if (e == S{}) unclear_ = was && captured();
    return e;
  }
};

}  // namespace gqs
