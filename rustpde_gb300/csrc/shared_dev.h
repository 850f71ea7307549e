// shared_dev.h -- read-only device tables that depend on a size alone and are
// shared by every object of that size (digit operators, unsplit transform
// tables).
//
// An object's arena holds what the object uses (Arena::keep); a table goes with
// its last owner.  The most recently used ones are held a little longer, up to
// kSharedRecentBytes in all, because making one costs milliseconds of host
// arithmetic and programs make objects of one size again and again; they are
// given up when an allocation fails (shared_recent_drop).
#pragma once
#include <map>
#include <memory>
#include <mutex>
#include <utility>

#include "prims.h"

namespace rbc {

constexpr size_t kSharedRecentBytes = 64u << 20;

struct DevBlock {
  void* p = nullptr;
  size_t bytes = 0;
  ~DevBlock();  // cudaFree
};
// Allocate a block on the current device (throws std::runtime_error).
std::shared_ptr<DevBlock> make_dev_block(size_t bytes);
// Hold a block among the recently used ones (the oldest beyond the limit go).
void shared_recent_touch(const std::shared_ptr<const DevBlock>& b);

// Tables T by key; make(T&) fills one in and returns its memory.  Keys name the
// device.  The lock is held while a table is made, so that it is made once.
template <class Key, class T>
class SharedDev {
 public:
  template <class Make>
  T get(const Key& key, Arena& owner, Make make) {
    std::shared_ptr<const DevBlock> b;
    T t{};
    {
      std::lock_guard<std::mutex> lk(mu_);
      auto& e = map_[key];
      b = e.first.lock();
      if (b == nullptr) {
        b = make(e.second);
        e.first = b;
      }
      t = e.second;
    }
    // (a table that its owner has had before is not new use: set-up calls of a
    // case that exists allocate and free nothing)
    if (owner.keep(b)) shared_recent_touch(b);
    return t;
  }

 private:
  std::mutex mu_;
  std::map<Key, std::pair<std::weak_ptr<const DevBlock>, T>> map_;
};

}  // namespace rbc
