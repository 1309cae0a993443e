// Memory that copies are faster with and can do without.
#pragma once
#include <cstddef>
#include <cstdint>

namespace kvx {

// A size that could not be had is not asked for again: on a GPU that a cache fills, every layer would try and fail.
class StagingBuffer {
 public:
  // `bytes` are at hand.  alloc(bytes): memory or nullptr; release(p): gives the smaller buffer back, once nothing uses it.
  template <typename ALLOC, typename RELEASE>
  bool reserve(size_t bytes, ALLOC&& alloc, RELEASE&& release) {
    if (bytes <= cap_) return true;
    if (bytes >= refused_) return false;
    char* p = static_cast<char*>(alloc(bytes));
    if (p == nullptr) {
      refused_ = bytes;
      return false;
    }
    if (data_ != nullptr) release(data_);
    data_ = p;
    cap_ = bytes;
    return true;
  }
  char* data() const { return data_; }

 private:
  char* data_{nullptr};
  size_t cap_{0};
  size_t refused_{SIZE_MAX};
};

}  // namespace kvx
