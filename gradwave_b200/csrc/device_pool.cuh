// Device memory of the operator handles. Free of CUDA calls of its own: Api has
// bool alloc(void**, size_t) and void free(void*).
#pragma once

#include <cstddef>
#include <initializer_list>
#include <map>
#include <mutex>
#include <utility>

namespace gwb {

// Every allocation of a handle goes through a pool. The band-chunk scratch of a
// destroyed handle waits there for the next handle on the device (mapping half a
// GB takes milliseconds, as long as many an apply): at most one buffer per
// device, kept only while a handle lives there and given back when an
// allocation of any handle fails. (Allocations outside the library cannot ask
// for it.)
template <class Api> class DevicePool {
 public:
  // n handles more (or fewer) on the device; the last one takes the kept buffer along.
  void handles(int dev, int n) {
    void* drop = nullptr;
    {
      std::lock_guard<std::mutex> lk(mu_);
      Slot& s = slots_[dev];
      s.handles += n;
      if (s.handles == 0) drop = s.release();
    }
    if (drop) Api::free(drop);
  }

  // A kept buffer of at least need bytes, or null.
  void* take(int dev, size_t need, size_t* bytes) {
    std::lock_guard<std::mutex> lk(mu_);
    Slot& s = slots_[dev];
    if (!s.p || s.bytes < need) return nullptr;
    *bytes = s.bytes;
    return s.release();
  }

  // p is idle. The larger of it and the kept buffer stays.
  void give(int dev, void* p, size_t bytes) {
    {
      std::lock_guard<std::mutex> lk(mu_);
      Slot& s = slots_[dev];
      if (s.handles > 0 && bytes > s.bytes) {
        std::swap(p, s.p);
        s.bytes = bytes;
      }
    }
    if (p) Api::free(p);
  }

  // *p = bytes of device memory (null where there is none, the kept buffer given back first).
  bool alloc(int dev, void** p, size_t bytes) {
    if (Api::alloc(p, bytes)) return true;
    size_t n = 0;
    void* kept = take(dev, 0, &n);
    if (kept) {
      Api::free(kept);
      if (Api::alloc(p, bytes)) return true;
    }
    *p = nullptr;
    return false;
  }

  // All of the (pointer, bytes) buffers, or none: those made before a failure are freed, all pointers null.
  bool alloc_all(int dev, std::initializer_list<std::pair<void**, size_t>> bufs) {
    for (const auto& b : bufs) *b.first = nullptr;
    for (const auto& b : bufs)
      if (!alloc(dev, b.first, b.second)) {
        for (const auto& c : bufs) {
          if (*c.first) Api::free(*c.first);
          *c.first = nullptr;
        }
        return false;
      }
    return true;
  }

  // *p of at least need bytes; what it held is lost when it has to grow.
  bool ensure(int dev, void** p, size_t* have, size_t need) {
    if (*have >= need) return true;
    if (*p) Api::free(*p);
    *have = 0;
    if (!alloc(dev, p, need)) return false;
    *have = need;
    return true;
  }

 private:
  struct Slot {
    int handles = 0;
    void* p = nullptr;
    size_t bytes = 0;
    void* release() {
      void* q = p;
      p = nullptr;
      bytes = 0;
      return q;
    }
  };
  std::mutex mu_;
  std::map<int, Slot> slots_;
};

}  // namespace gwb
