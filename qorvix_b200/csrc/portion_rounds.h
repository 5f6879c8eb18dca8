// Which chunks of a step's segments go through a recurrence's launches together, where every chunk takes a slot of a workspace.
// Only segments that take these launches get slots, each as many as it has chunks; what does not fit follows in further rounds, every
// segment from where its last one ended.  Host code without CUDA.
#pragma once
#include <algorithm>
#include <vector>

struct PortionItem {
  int seg, place;        // the segment, counted over all and over those that take part
  int first, count;      // its chunks first .. first + count - 1
  int slot;              // in the workspace from this slot on
};
template <int N> struct PortionRound {
  int items, slots;      // slots in use: 0 .. slots - 1
  PortionItem item[N];
};

class PortionRounds {
 public:
  // lens [S]: tokens; chunk: tokens a chunk; from: shorter segments take no part; room: slots there is room for (one at least); few: chunks of
  // a segment that are worth a round of launches, where it has as many.
  PortionRounds(const int* lens, int S, int chunk, int from, size_t room, int few) : room_(std::max<size_t>(room, 1)), few_(few) {
    for (int s = 0; s < S; ++s)
      if (lens[s] > 0 && lens[s] >= from) {
        left_.push_back({s, (int)left_.size(), 0, (lens[s] + chunk - 1) / chunk, 0});
        chunks_ += left_.back().count;
      }
    places_ = (int)left_.size();
  }
  int places() const { return places_; }               // segments that take part
  size_t slots() const { return std::min(chunks_, room_); }

  // The next round, false when there is none.  Segments advance side by side, as long as each gets `few` chunks or all it has left.
  template <int N> bool next(PortionRound<N>& r) {
    if (left_.empty()) return false;
    size_t active = 0, least = 0;
    for (const PortionItem& i : left_) {
      const size_t wants = (size_t)std::min(i.count, few_);
      if (active && (active == (size_t)N || least + wants > room_)) break;
      least += wants;
      ++active;
    }
    // the room shared out: whoever needs less than an equal share leaves the rest to the others
    size_t budget = room_, sharers = active;
    std::vector<int> give(active, 0);
    for (bool settled = false; !settled && sharers;) {
      settled = true;
      const size_t share = std::max<size_t>(budget / sharers, 1);
      for (size_t i = 0; i < active; ++i)
        if (!give[i] && (size_t)left_[i].count <= share) {
          give[i] = left_[i].count;
          budget -= give[i];
          --sharers;
          settled = false;
        }
    }
    for (size_t i = 0; i < active; ++i)
      if (!give[i]) give[i] = (int)std::max<size_t>(budget / sharers, 1);
    r.items = r.slots = 0;
    std::vector<PortionItem> rest;
    for (size_t i = 0; i < left_.size(); ++i) {
      PortionItem p = left_[i];
      if (i < active) {
        r.item[r.items] = {p.seg, p.place, p.first, give[i], r.slots};
        ++r.items;
        r.slots += give[i];
        p.first += give[i];
        p.count -= give[i];
      }
      if (p.count) rest.push_back(p);
    }
    left_.swap(rest);
    return true;
  }

 private:
  std::vector<PortionItem> left_;      // count: chunks that are left
  size_t room_, chunks_ = 0;
  int few_, places_ = 0;
};
