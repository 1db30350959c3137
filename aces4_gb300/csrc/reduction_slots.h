// Which scratch of the deterministic reductions a launch uses.
//
// A reduction's CTAs leave partial sums and a counter for the last of them to
// read, so two launches that can be on the GPU at once need different slots.
// Launches on one stream follow each other: a stream has a slot of its own,
// found by the stream's id (ids are never reused, handles are).  A launch
// captured into a graph runs wherever and whenever the graph is replayed, and
// follows only what was captured on the same stream of the same capture: that
// pair has a slot of its own for as long as the graph or an instance of it
// lives.
//
// Streams beyond kMaxStreams get none (-1): their launches take stream-ordered
// memory of their own (runtime.cpp).
#pragma once

#include <map>
#include <utility>
#include <vector>

namespace a4g {

class SlotTable {
 public:
  static constexpr int kMaxStreams = 256;
  static constexpr int kMaxSlots = 16384;

  // The slot of stream `stream` outside capture (capture 0) or inside capture
  // `capture`; -1 where there is none.
  int slot(unsigned long long capture, unsigned long long stream) {
    const auto it = at_.find({capture, stream});
    if (it != at_.end()) return it->second;
    if (!capture && streams_ == kMaxStreams) return -1;
    int q = -1;
    if (!free_.empty()) q = free_.back(), free_.pop_back();
    else if (used_ < kMaxSlots) q = used_++;
    else return -1;
    at_.emplace(std::make_pair(capture, stream), q);
    if (!capture) ++streams_;
    return q;
  }
  bool has_capture(unsigned long long capture) const {
    const auto it = at_.lower_bound({capture, 0ull});
    return it != at_.end() && it->first.first == capture;
  }
  // The graph of `capture` and its instances are gone.
  void release(unsigned long long capture) {
    auto it = at_.lower_bound({capture, 0ull});
    while (it != at_.end() && it->first.first == capture) free_.push_back(it->second), it = at_.erase(it);
  }
  int slots() const { return used_; }  // slots ever handed out: 0 .. slots() - 1

 private:
  std::map<std::pair<unsigned long long, unsigned long long>, int> at_;
  std::vector<int> free_;
  int used_ = 0, streams_ = 0;
};

}  // namespace a4g
