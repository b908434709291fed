// Device memory of the operator handles. Free of CUDA calls of its own: Api has
// bool alloc(void**, size_t) and void free(void*).
#pragma once

#include <algorithm>
#include <cstddef>
#include <cstdint>
#include <initializer_list>
#include <map>
#include <mutex>
#include <utility>

namespace gwb {

// Scratch of a chunk of bands.
struct ChunkScratch {
  void* p = nullptr;
  size_t bytes = 0;
  size_t denied = SIZE_MAX;  // the least size that could not be had
};

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

  // Bands per chunk, with scratch for one in w: as few chunks as the budget
  // allows, all of (nearly) equal size; where the device has no room for that,
  // chunks of the low budget or of what w held. 0: no room at all. A size that
  // was refused is not asked for again: every call would give up its scratch and
  // map it anew (and could not be captured).
  int chunk(int dev, ChunkScratch& w, int nb, size_t per_band, size_t budget, size_t low) {
    const size_t had = w.bytes;
    auto bands = [&](size_t bytes) {
      const size_t most = std::min<size_t>(32768, std::max<size_t>(1, bytes / per_band));  // bands are a grid axis
      const size_t nchunks = ((size_t)nb + most - 1) / most;
      return (int)(((size_t)nb + nchunks - 1) / nchunks);
    };
    auto fits = [&](size_t need) {
      if (w.bytes >= need) return true;
      size_t n = 0;
      if (void* p = take(dev, need, &n)) {
        if (w.p) Api::free(w.p);
        w.p = p;
        w.bytes = n;
        return true;
      }
      return ensure(dev, &w.p, &w.bytes, need);
    };
    int n = bands(budget);
    const size_t want = per_band * n;
    if (want <= w.bytes || (want < w.denied && fits(want))) return n;
    n = std::min(n, bands(std::max(low, had)));
    if (!fits(per_band * n)) return 0;     // nothing can be had (under a capture, say): asked for again
    if (want > w.bytes) w.denied = std::min(w.denied, want);
    return n;
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
