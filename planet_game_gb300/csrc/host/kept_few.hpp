// Values kept by key, the most recently used few of them.
#pragma once

#include <cstddef>
#include <list>
#include <utility>

namespace psgb {

// At most `Most` values: one more drops the least recently used. A value's reference holds until
// `Most` other keys have been asked for.
template <typename Key, typename Value, std::size_t Most>
class KeptFew {
  public:
    // The key's value, made by `make()` where it is not kept.
    template <typename Make>
    Value& of(const Key& key, Make&& make) {
        for (auto it = kept_.begin(); it != kept_.end(); ++it) {
            if (it->first != key) continue;
            kept_.splice(kept_.begin(), kept_, it);
            return kept_.front().second;
        }
        if (kept_.size() >= Most) kept_.pop_back();   // given back before the next is made
        kept_.emplace_front(key, std::forward<Make>(make)());
        return kept_.front().second;
    }
    void clear() { kept_.clear(); }
    std::size_t size() const { return kept_.size(); }

  private:
    std::list<std::pair<Key, Value>> kept_;   // the last used first
};

}  // namespace psgb
