// fftoc — whether a whole host buffer lies in memory that the device can reach.
#pragma once
#include <cstddef>
#include <cstdint>

namespace fftoc {

// One allocation or registration of host memory.  `start` and `size` are host
// addresses; `shift` is the distance from them to the device's.
struct HostRange {
  bool mapped;  // pinned, mapped into the device's address space, not managed
  uintptr_t start;
  size_t size;
  ptrdiff_t shift;
};

// The device address of the `bytes` bytes at p if every one of them lies in a
// mapped range and all ranges are equally far from the device's addresses, else
// null.  find(address) is the range that holds an address.  A buffer may span
// several registrations; the check ends at the first gap between them.
template <class Find>
void* mapped_range(const void* p, size_t bytes, Find find) {
  const uintptr_t a = (uintptr_t)p, end = a + bytes;
  ptrdiff_t shift = 0;
  for (uintptr_t at = a; at < end;) {
    const HostRange r = find(at);
    if (!r.mapped || at < r.start || at - r.start >= r.size) return nullptr;
    if (at == a) shift = r.shift;
    if (r.shift != shift) return nullptr;
    at = r.start + r.size;
  }
  return bytes > 0 ? (void*)(a + (uintptr_t)shift) : nullptr;
}

}  // namespace fftoc
