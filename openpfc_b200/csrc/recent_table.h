// recent_table.h -- a fixed number of values by key, the longest unused making room.
#pragma once
#include <algorithm>
#include <vector>

namespace opfc {

// Pointers stay valid until N - 1 other keys have been found or kept since: the
// table never grows past the N entries it reserves.
template <typename Key, typename Value, int N> class RecentTable {
 public:
  RecentTable() { entries_.reserve(N); }

  // the value kept under `key`, or null
  const Value *find(const Key &key) {
    for (auto &e : entries_)
      if (e.key == key) {
        e.used = ++clock_;
        return &e.value;
      }
    return nullptr;
  }

  const Value *keep(const Key &key, const Value &value) {
    const Entry e{key, value, ++clock_};
    if (entries_.size() < N) {
      entries_.push_back(e);
      return &entries_.back().value;
    }
    auto oldest = std::min_element(entries_.begin(), entries_.end(),
                                   [](const Entry &a, const Entry &b) { return a.used < b.used; });
    *oldest = e;
    return &oldest->value;
  }

 private:
  struct Entry {
    Key key;
    Value value;
    unsigned long long used;  // clock_ of the last use
  };
  std::vector<Entry> entries_;
  unsigned long long clock_ = 0;
};

}  // namespace opfc
