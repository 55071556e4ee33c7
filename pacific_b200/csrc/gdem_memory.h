// gdem_memory.h -- bookkeeping of one system's device memory.
#pragma once
#include <algorithm>
#include <cstddef>
#include <vector>

namespace gdem {

// Two kinds of arrays.  Those of their own (own) can be given back one by one
// (giveBack).  Those that live as long as the system (shared) come out of
// common blocks, and a block goes back with the system only: it holds other
// arrays beside the one at its start, so giveBack does not know the blocks'
// addresses at all, and an array out of a block that is given back simply
// stays where it is.  take returns null when there is no memory.
class DeviceMemory {
 public:
  using Take = void* (*)(std::size_t);
  using Give = void (*)(void*);
  DeviceMemory(Take take, Give give) : take_(take), give_(give) {}
  DeviceMemory(DeviceMemory const&) = delete;
  DeviceMemory& operator=(DeviceMemory const&) = delete;
  ~DeviceMemory() { release(); }

  void* own(std::size_t bytes) {
    void* p = take_(std::max<std::size_t>(bytes, 1));
    if (p) own_.push_back(p);
    return p;
  }
  // block: bytes of a block opened for it (a longer array has a block to
  // itself).  An array for which no block can be had gets an allocation of its
  // own.
  void* shared(std::size_t bytes, std::size_t block) {
    bytes = (std::max<std::size_t>(bytes, 1) + 255) & ~std::size_t(255);
    if (left_ < bytes) {
      void* p = take_(std::max(bytes, block));
      if (!p) return own(bytes);
      blocks_.push_back(p);
      total_ += std::max(bytes, block);
      if (bytes >= block) return p;
      at_ = static_cast<char*>(p);
      left_ = block;
    }
    void* r = at_;
    at_ += bytes;
    left_ -= bytes;
    return r;
  }
  void giveBack(void* p) {
    for (auto& a : own_)
      if (a == p) {
        give_(p);
        a = own_.back();
        own_.pop_back();
        return;
      }
  }
  // Bytes of the blocks opened so far.
  std::size_t sharedTotal() const { return total_; }
  void release() {
    for (void* p : own_) give_(p);
    for (void* p : blocks_) give_(p);
    own_.clear();
    blocks_.clear();
    at_ = nullptr;
    left_ = total_ = 0;
  }

 private:
  Take take_;
  Give give_;
  std::vector<void*> own_, blocks_;
  char* at_ = nullptr;       // rest of the last block
  std::size_t left_ = 0, total_ = 0;
};

}  // namespace gdem
