// Blocks of device memory kept between cubes: the list alone, without CUDA
// calls (birp_host.h says what it is for), checked on the host by
// tests/cpp/block_cache_test.cpp.
//
// A block that is given back is kept for the next request of nearly its size
// when it is large enough, belongs to the device the list is open for and the
// giver says that nothing on the device uses it any more; else it is freed. At
// most kKeepMax bytes are kept: the oldest blocks go first. Any thread; frees
// run outside the lock. Nothing here allocates host memory.
#pragma once
#include <cstddef>
#include <mutex>

namespace birp {

class BlockCache {
 public:
  static constexpr size_t kKeepMin = (size_t)8 << 20, kKeepMax = (size_t)1 << 30;

  explicit BlockCache(void (*release)(void*)) : release_(release) {}

  // Blocks of `device` are kept from here on.
  void open(int device) {
    std::lock_guard<std::mutex> lk(mu_);
    device_ = device;
  }
  // No block is kept any more; the kept ones are freed.
  void close() { drop_all(true); }
  // Frees the kept blocks.
  void release_all() { drop_all(false); }

  // A kept block of at least *bytes and at most an eighth more (the smallest
  // such), or nullptr; *bytes becomes its size.
  void* take(int device, size_t* bytes) {
    if (*bytes < kKeepMin) return nullptr;
    std::lock_guard<std::mutex> lk(mu_);
    if (device != device_) return nullptr;
    int best = -1;
    for (int i = 0; i < n_; ++i)
      if (list_[i].bytes >= *bytes && list_[i].bytes <= *bytes + *bytes / 8 &&
          (best < 0 || list_[i].bytes < list_[best].bytes))
        best = i;
    if (best < 0) return nullptr;
    void* p = list_[best].p;
    *bytes = list_[best].bytes;
    remove(best);
    return p;
  }

  // Keeps p or frees it. idle: nothing on the device uses it any more.
  void give(void* p, size_t bytes, int device, bool idle) {
    if (!p) return;
    void* out[kBlocks + 1];
    int n_out = 0;
    {
      std::lock_guard<std::mutex> lk(mu_);
      if (!idle || bytes < kKeepMin || bytes > kKeepMax || device < 0 || device != device_) {
        out[n_out++] = p;
      } else {
        while (held_ + bytes > kKeepMax) {
          out[n_out++] = list_[0].p;
          remove(0);
        }
        list_[n_++] = {p, bytes};
        held_ += bytes;
      }
    }
    for (int i = 0; i < n_out; ++i) release_(out[i]);
  }

  size_t held() {
    std::lock_guard<std::mutex> lk(mu_);
    return held_;
  }

 private:
  struct Block {
    void* p;
    size_t bytes;
  };
  static constexpr int kBlocks = (int)(kKeepMax / kKeepMin);  // as many of the smallest as the bound holds

  void remove(int i) {
    held_ -= list_[i].bytes;
    for (int j = i + 1; j < n_; ++j) list_[j - 1] = list_[j];
    --n_;
  }
  void drop_all(bool closing) {
    void* out[kBlocks];
    int n_out = 0;
    {
      std::lock_guard<std::mutex> lk(mu_);
      if (closing) device_ = -1;
      for (; n_out < n_; ++n_out) out[n_out] = list_[n_out].p;
      n_ = 0;
      held_ = 0;
    }
    for (int i = 0; i < n_out; ++i) release_(out[i]);
  }

  void (*release_)(void*);
  std::mutex mu_;
  int device_ = -1;
  int n_ = 0;
  size_t held_ = 0;
  Block list_[kBlocks];  // oldest first
};

}  // namespace birp
