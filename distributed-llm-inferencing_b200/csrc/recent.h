// The last few results of a function, found again by their key: plain C++, no device code.
#pragma once

namespace dli {

// Fully associative, first in first out: whatever the keys are, the last N distinct ones are kept (a hashed table loses
// two keys that share a slot on every turn).  Key needs operator==.  Not synchronised: one per thread.
template <typename Key, typename Value, int N>
class RecentResults {
 public:
  const Value* find(const Key& key) const {
    for (int i = 0; i < used_; ++i)
      if (keys_[i] == key) return &values_[i];
    return nullptr;
  }
  void put(const Key& key, const Value& value) {
    keys_[next_] = key;
    values_[next_] = value;
    next_ = next_ + 1 == N ? 0 : next_ + 1;
    if (used_ < N) ++used_;
  }

 private:
  Key keys_[N] = {};
  Value values_[N] = {};
  int used_ = 0, next_ = 0;
};

}  // namespace dli
