// Where a host buffer lies as kernels see it. Plain C++ without CUDA headers: the walk is tested with a host compiler.
#pragma once

#include <cstddef>
#include <cstdint>

namespace fb {

// What the driver knows about one byte of page-locked host memory.
struct PinnedByte {
  uintptr_t device;  // its address on the device, 0: none
  uintptr_t start;   // the allocation or registration that holds it: first byte ...
  size_t bytes;      // ... and size
};

// Device address of [host, host + bytes), or 0 unless every byte is page-locked and the device addresses follow each other
// as the host's do. `query(p, out)` asks about the byte at p (false: not page-locked). One question per allocation: a
// kernel that goes by the first byte alone faults where a registration ends inside the buffer.
template <class Query>
uintptr_t pinned_range(uintptr_t host, size_t bytes, Query query) {
  uintptr_t first = 0;
  for (uintptr_t p = host, end = host + bytes; p < end;) {
    PinnedByte b{};
    if (!query(p, b) || !b.device || p < b.start || p - b.start >= b.bytes) return 0;
    if (p == host) first = b.device;
    else if (b.device - first != p - host) return 0;
    p = b.start + b.bytes;
  }
  return first;
}

}  // namespace fb
