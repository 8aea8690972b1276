// Device memory that is kept for the next caller, and allocation that gives it
// back first when the device is out of memory.  Host logic alone: the callers
// allocate and free.
#ifndef HISV_KEPT_BLOCKS_H_
#define HISV_KEPT_BLOCKS_H_

#include <stddef.h>
#include <stdint.h>

#include <deque>
#include <mutex>
#include <vector>

namespace hisv {

// Idle blocks of one device, at most `Most` bytes of them: a block that has no
// room takes that of the oldest ones, so the sizes a program uses now replace
// those it used once.  They belong to one context (by its id, 0 = none known).
// A device that is reset takes its context and their memory with it; the first
// block of a later context takes their place, and they are forgotten, not freed
// (their addresses may be in use again).
template <size_t Most>
class KeptBlocks {
 public:
  // a kept block of exactly `bytes`, or null
  void* take(uint64_t ctx, size_t bytes) {
    std::lock_guard<std::mutex> lk(mu_);
    if (ctx != ctx_) return nullptr;
    for (size_t i = blocks_.size(); i-- > 0;)  // the newest first
      if (blocks_[i].bytes == bytes) {
        void* const p = blocks_[i].p;
        blocks_.erase(blocks_.begin() + long(i));
        held_ -= bytes;
        return p;
      }
    return nullptr;
  }
  // keeps an idle block of context `ctx`; returns the blocks to be freed instead
  // (`p` itself where it cannot be kept)
  std::vector<void*> put(uint64_t ctx, void* p, size_t bytes) {
    std::lock_guard<std::mutex> lk(mu_);
    std::vector<void*> out;
    if (bytes > Most || ctx < ctx_ || ctx == 0) {
      out.push_back(p);
      return out;
    }
    if (ctx != ctx_) {
      blocks_.clear();
      held_ = 0;
      ctx_ = ctx;
    }
    while (held_ + bytes > Most) {
      out.push_back(blocks_.front().p);
      held_ -= blocks_.front().bytes;
      blocks_.pop_front();
    }
    blocks_.push_back({p, bytes});
    held_ += bytes;
    return out;
  }
  // every block of context `ctx`, to be freed
  std::vector<void*> drain(uint64_t ctx) {
    std::lock_guard<std::mutex> lk(mu_);
    std::vector<void*> out;
    if (ctx != ctx_) return out;
    for (const Block& b : blocks_) out.push_back(b.p);
    blocks_.clear();
    held_ = 0;
    return out;
  }

 private:
  struct Block {
    void* p;
    size_t bytes;
  };
  std::mutex mu_;
  std::deque<Block> blocks_;  // oldest first
  size_t held_ = 0;
  uint64_t ctx_ = 0;
};

// alloc(); where that fails with `oom` and release() (free what is kept) freed
// something, once more
template <class Error, class Alloc, class Release>
Error alloc_releasing(Error oom, Alloc alloc, Release release) {
  const Error e = alloc();
  return e == oom && release() ? alloc() : e;
}

}  // namespace hisv

#endif  // HISV_KEPT_BLOCKS_H_
