// Host memory that a topology is laid out in before it is copied to the
// device: one block of an engine, kept and grown, freed with it.  Pinned, so
// that the copies need no staging; where pinned memory is refused the block is
// pageable (the copies are waited for before it is reused either way).  It
// grows to at least twice its size: pinning a block takes 1 to 4 ms and
// unpinning it 0.4 ms (up to 1 MB), which a series of growing molecules would
// otherwise pay at every call.
#pragma once

#include <algorithm>
#include <cstddef>
#include <cstdlib>

namespace xtb {

// Pinned: static void* allocate(size_t) (nullptr when refused) and
// static void release(void*).
template <class Pinned>
class HostArena {
 public:
  HostArena() = default;
  HostArena(const HostArena&) = delete;
  HostArena& operator=(const HostArena&) = delete;
  ~HostArena() { free_block(); }

  // Room for `bytes`, empty; false when there is no memory of either kind.
  bool reset(size_t bytes) {
    used_ = 0;
    if (bytes <= cap_) return true;
    const size_t want = std::max(bytes, 2 * cap_);
    free_block();
    for (const size_t size : {want, bytes}) {
      if ((base_ = static_cast<char*>(Pinned::allocate(size))) != nullptr) {
        pinned_ = true;
        cap_ = size;
        return true;
      }
    }
    if ((base_ = static_cast<char*>(std::malloc(bytes))) != nullptr) cap_ = bytes;
    return base_ != nullptr;
  }
  static size_t padded(size_t bytes) { return (bytes + 63) / 64 * 64; }
  template <class T>
  T* take(size_t count) {   // within the reset size, by its computation
    T* p = reinterpret_cast<T*>(base_ + used_);
    used_ += padded(count * sizeof(T));
    return p;
  }
  size_t capacity() const { return cap_; }
  bool pinned() const { return pinned_; }

 private:
  void free_block() {
    if (base_ != nullptr) {
      if (pinned_) Pinned::release(base_);
      else std::free(base_);
    }
    base_ = nullptr;
    cap_ = 0;
    pinned_ = false;
  }
  char* base_ = nullptr;
  size_t cap_ = 0, used_ = 0;
  bool pinned_ = false;
};

}  // namespace xtb
