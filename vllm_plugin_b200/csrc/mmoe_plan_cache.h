// Launch parameters kept from one call to the next (host code).
#pragma once

#include <stdint.h>

#include <memory>
#include <mutex>
#include <vector>

namespace mmoe {

// At most kCapacity values by key; the least recently used one gives way.  A value is handed out with shared ownership: it stays
// valid for the call that has it while another thread's call replaces the entry.  Key: operator== and same_workspace(), which
// says that the other key's value may serve as the beginning of this one's.
template <typename Key, typename Value, int kCapacity>
class PlanCache {
 public:
  // The value of `key`, made by `build(sibling)` on first use.  `sibling`: the value of a key with the same workspace, or null.
  // build() returns null when it fails, and then nothing is kept.
  template <typename Build>
  std::shared_ptr<const Value> get(const Key& key, Build&& build) {
    std::lock_guard<std::mutex> lock(mutex_);
    // Mostly the key of the last call, or, as the layers of a model come round, the one behind it.
    const size_t n = entries_.size();
    for (size_t i = 0; i < n; ++i) {
      const size_t at = last_ + i < n ? last_ + i : last_ + i - n;
      if (entries_[at].key == key) return touch(at);
    }
    const Value* sibling = nullptr;
    size_t victim = 0;
    for (size_t i = 0; i < n; ++i) {
      if (entries_[i].stamp < entries_[victim].stamp) victim = i;
      if (entries_[i].key.same_workspace(key)) sibling = entries_[i].value.get();
    }
    std::shared_ptr<const Value> value = build(sibling);
    if (value == nullptr) return value;
    if (n < kCapacity) {
      victim = n;
      entries_.emplace_back();
    }
    entries_[victim].key = key;
    entries_[victim].value = std::move(value);
    return touch(victim);
  }

 private:
  struct Entry {
    Key key;
    std::shared_ptr<const Value> value;
    uint64_t stamp = 0;
  };
  std::shared_ptr<const Value> touch(size_t at) {
    entries_[at].stamp = ++clock_;
    last_ = at;
    return entries_[at].value;
  }
  std::mutex mutex_;
  std::vector<Entry> entries_;
  size_t last_ = 0;
  uint64_t clock_ = 0;
};

}  // namespace mmoe
