// Host check of mapped_range (fft_onchip_gb300/csrc/host_range.h) on made-up
// registrations: a buffer is taken only when every byte of it lies in mapped
// ranges at one distance from the device's addresses.  Prints "ok" or the
// failing case.
#include <cstdio>
#include <vector>

#include "host_range.h"

using fftoc::HostRange;

int main() {
  constexpr uintptr_t A = 0x100000;
  constexpr ptrdiff_t D = 0x7000;
  struct Case {
    const char* name;
    std::vector<HostRange> ranges;
    uintptr_t p;
    size_t bytes;
    bool taken;
  };
  const std::vector<Case> cases = {
      {"whole range", {{true, A, 4096, D}}, A, 4096, true},
      {"inside a range", {{true, A, 4096, D}}, A + 16, 4064, true},
      {"one point", {{true, A, 16, D}}, A, 16, true},
      {"past the end", {{true, A, 4096, D}}, A + 16, 4096, false},
      {"before the start", {{true, A, 4096, D}}, A - 16, 4096, false},
      {"not registered", {}, A, 4096, false},
      {"not mapped", {{false, A, 4096, D}}, A, 4096, false},
      {"ends registered, gap between", {{true, A, 4096, 0}, {true, A + 8192, 4096, 0}}, A, 12288, false},
      {"ends registered, middle not mapped", {{true, A, 4096, 0}, {false, A + 4096, 4096, 0}, {true, A + 8192, 4096, 0}}, A,
       12288, false},
      {"adjacent registrations", {{true, A, 4096, D}, {true, A + 4096, 4096, D}, {true, A + 8192, 4096, D}}, A + 32, 12000,
       true},
      {"adjacent at other distances", {{true, A, 4096, D}, {true, A + 4096, 4096, D + 4096}}, A, 8192, false},
      {"empty", {{true, A, 4096, D}}, A, 0, false},
  };
  for (const Case& c : cases) {
    auto find = [&](uintptr_t at) {
      for (const HostRange& r : c.ranges)
        if (at >= r.start && at - r.start < r.size) return r;
      return HostRange{false, 0, 0, 0};
    };
    void* want = c.taken ? (void*)(c.p + D * (c.ranges[0].shift != 0)) : nullptr;
    if (fftoc::mapped_range((const void*)c.p, c.bytes, find) != want) {
      std::printf("failed: %s\n", c.name);
      return 1;
    }
  }
  std::puts("ok");
  return 0;
}
