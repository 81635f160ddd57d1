// The workspaces that the contexts of a device keep for their products'
// scratch: who holds how much, who may grow, and what can be taken back.
//
// A product takes its scratch from its context's workspace and asks an
// allocator for what does not fit; the next product finds a workspace grown to
// that need, so from the second product of a size on no allocator call is left.
// The workspaces of a device stay within a limit together: one that may not
// grow stays as it is, so that a product over the limit costs the smaller ones
// around it nothing.  A workspace that no product runs in can be taken back
// from any thread, which an allocation that finds no memory does.
//
// Plain C++ (the memory itself comes from the caller's functions), so that it
// is tested without a device.
#pragma once
#include <algorithm>
#include <cstddef>
#include <cstdint>
#include <mutex>
#include <vector>

namespace cas {

struct Workspace {
  char* mem = nullptr;  // cap bytes
  size_t cap = 0;
  size_t used = 0;      // taken by the current product
  size_t need = 0;      // what the current product has asked for, then what the last one did
  bool busy = false;    // a product runs in it: the context's thread alone looks at it

  // `bytes` for the current product, or null where they do not fit.
  char* take(size_t bytes) {
    bytes = (std::max<size_t>(bytes, 16) + 255) & ~size_t(255);
    need += bytes;
    if (!mem || used + bytes > cap) return nullptr;
    used += bytes;
    return mem + used - bytes;
  }
};

class WorkspaceBook {
 public:
  void join(Workspace& w) {
    std::lock_guard<std::mutex> lock(mu_);
    all_.push_back(&w);
  }

  template <typename Release>
  void leave(Workspace& w, Release&& release) {
    drop(w, release);
    std::lock_guard<std::mutex> lock(mu_);
    all_.erase(std::remove(all_.begin(), all_.end(), &w), all_.end());
  }

  // Before a product: w is busy, and has grown to what the last product asked
  // for where all workspaces then stay within `limit`.
  template <typename Alloc, typename Release>
  void begin(Workspace& w, size_t limit, Alloc&& alloc, Release&& release) {
    size_t want = 0;
    char* old = nullptr;
    {
      std::lock_guard<std::mutex> lock(mu_);
      w.busy = true;
      want = (w.need + (size_t(2) << 20) - 1) & ~((size_t(2) << 20) - 1);
      w.used = w.need = 0;
      if (want <= w.cap || held_ - w.cap + want > limit) return;
      held_ += want - w.cap;
      old = w.mem;
      w.mem = nullptr;
      w.cap = want;
    }
    if (old) release(old);
    w.mem = alloc(want);
    if (w.mem) return;
    std::lock_guard<std::mutex> lock(mu_);
    held_ -= w.cap;
    w.cap = 0;
  }

  // After a product, once nothing on the device uses the workspace any more.
  void end(Workspace& w) {
    std::lock_guard<std::mutex> lock(mu_);
    w.used = 0;
    w.busy = false;
  }

  // The context's own workspace given up, by the context's thread.
  template <typename Release>
  void drop(Workspace& w, Release&& release) {
    std::lock_guard<std::mutex> lock(mu_);
    give_up(w, release);
  }

  // Every workspace that no product runs in, given up.
  template <typename Release>
  void reclaim(Release&& release) {
    std::lock_guard<std::mutex> lock(mu_);
    for (Workspace* w : all_)
      if (!w->busy) give_up(*w, release);
  }

  size_t held() {
    std::lock_guard<std::mutex> lock(mu_);
    return held_;
  }

 private:
  template <typename Release>
  void give_up(Workspace& w, Release&& release) {
    if (w.mem) release(w.mem);
    held_ -= w.cap;
    w.mem = nullptr;
    w.cap = w.used = 0;
  }

  std::mutex mu_;
  std::vector<Workspace*> all_;
  size_t held_ = 0;
};

// Heavy-row bitmaps kept from the symbolic phase for the numeric one: every
// slice of each row when that fits a quarter of the free device memory, at most
// 24 GiB and at least 8, else the rows of one slice.  The free memory is asked
// for only where it decides: cudaMemGetInfo waits for the driver's lock, which
// other processes hold for 1 to 90 ms now and then (every product with heavy
// rows asked, one in five to thirty of a 7.6 ms batch's passes took 10 to 90).
struct SavedBitmaps {
  int slices;  // of a row, at most
  bool any;
};
template <typename Free>
SavedBitmaps saved_bitmaps(int64_t rows, int64_t max_slices, size_t slice_bytes, double share, Free&& free_bytes) {
  const double gib = (double)(size_t(1) << 30), whole = (double)rows * (double)max_slices * (double)slice_bytes;
  double cap = share * 8.0 * gib;
  if (whole > cap) cap = share * std::max(8.0 * gib, std::min(24.0 * gib, 0.25 * free_bytes()));
  const int slices = whole <= cap ? (int)max_slices : 1;
  return {slices, (double)rows * slices * (double)slice_bytes <= cap};
}

}  // namespace cas
