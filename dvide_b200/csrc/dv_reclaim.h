// dv_reclaim.h -- memory that objects of this process hold for a later use, and
// give back when an allocation fails anywhere in it.
//
// A holder registers itself, and touches what it holds under the registry's
// lock: reclaim_all may come from any thread.  The lock is recursive, since a
// holder that is given back may own another.
#pragma once

#include <stddef.h>

#include <algorithm>
#include <mutex>
#include <vector>

namespace dv {

class Holder {
 public:
  // Gives back what is held on `device`; returns the bytes.  Under the lock.
  virtual size_t reclaim(int device) = 0;

 protected:
  ~Holder() = default;
};

class Holders {
 public:
  static std::recursive_mutex& lock() { return the().m_; }
  static void add(Holder* h) {
    std::lock_guard<std::recursive_mutex> g(lock());
    the().all_.push_back(h);
  }
  static void remove(Holder* h) {
    std::lock_guard<std::recursive_mutex> g(lock());
    auto& v = the().all_;
    v.erase(std::remove(v.begin(), v.end(), h), v.end());
  }
  static size_t reclaim_all(int device) {
    std::lock_guard<std::recursive_mutex> g(lock());
    size_t bytes = 0;
    const std::vector<Holder*> now = the().all_;
    for (Holder* h : now) {
      const auto& v = the().all_;  // one that is given back may take others with it
      if (std::find(v.begin(), v.end(), h) != v.end()) bytes += h->reclaim(device);
    }
    return bytes;
  }

 private:
  static Holders& the() {
    static Holders* h = new Holders();  // outlives every static object that may still hold
    return *h;
  }
  std::recursive_mutex m_;
  std::vector<Holder*> all_;
};

}  // namespace dv
