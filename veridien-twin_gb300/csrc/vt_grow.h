// Growth of a device buffer that several entry points share (the wavefront's path state).
#pragma once

#include <cstddef>
#include <cstdint>

namespace vtapi {

// Dev: void* alloc(size_t) (null: refused), void free(void*), void sync() (work on the buffer has ended), size_t room()
struct GrowBuffer {
  void* p = nullptr;
  size_t cap = 0;
  size_t refused = SIZE_MAX;   // the smallest size that try_grow was refused

  template <typename Dev>
  void put(Dev& dev, void* q, size_t bytes) {
    if (p) { dev.sync(); dev.free(p); }
    p = q;
    cap = q ? bytes : 0;
  }
  // at least `bytes`, which the caller cannot do without: beside the old buffer, or in its place where both do not fit
  template <typename Dev>
  bool grow(Dev& dev, size_t bytes) {
    if (cap >= bytes) return true;
    void* q = dev.alloc(bytes);
    if (!q && p) {
      put(dev, nullptr, 0);
      q = dev.alloc(bytes);
    }
    if (!q) return false;
    put(dev, q, bytes);
    return true;
  }
  // `bytes` where they are to be had beside the old buffer, which stays as it is otherwise: another entry point may count on
  // its size. A refusal is remembered until the device has that much room.
  template <typename Dev>
  bool try_grow(Dev& dev, size_t bytes) {
    if (cap >= bytes) return true;
    if (bytes >= refused && dev.room() < bytes) return false;
    void* q = dev.alloc(bytes);
    if (!q) {
      refused = bytes;
      return false;
    }
    put(dev, q, bytes);
    refused = SIZE_MAX;
    return true;
  }
};

}  // namespace vtapi
