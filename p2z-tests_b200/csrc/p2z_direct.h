// p2z_direct.h -- the host arrays that p2z_run may hand to a kernel.
//
// A copy takes any byte address, reports a range that is not page-locked as
// an error, and has every input on the device before an output lands.  A kernel
// that reads and writes the caller's arrays itself does none of this: an address
// off a word's boundary or past the page-locked part faults, and the kernels
// load tracks and hits as data that nobody writes meanwhile.  So each array has
// to start on a 4-byte boundary and be page-locked to its last byte, at device
// addresses without a gap, and the output may share no byte with an input.
// Host code only (the page-locked ranges come from a function), tested on the CPU.
#pragma once

#include <cstddef>
#include <cstdint>

namespace p2z {

// Page-locked host memory [begin, end) and the device's address of `begin`.
struct HostRange {
  uintptr_t begin, end, device;
};
// An array of more pieces (cudaHostRegister called part by part) is copied instead.
constexpr int kMaxHostRanges = 64;

// The device's address of [p, p + bytes), 0 where a kernel cannot take it.
// range_of(address, HostRange *): the page-locked range that holds an address, false if none does.
template <class RangeOf>
uintptr_t mapped_array(const void *p, size_t bytes, RangeOf &&range_of) {
  const uintptr_t a = (uintptr_t)p, end = a + bytes;
  if (a % 4 != 0 || end <= a) return 0;
  uintptr_t device = 0, at = a;
  for (int i = 0; at < end; ++i) {
    HostRange r = {0, 0, 0};
    if (i == kMaxHostRanges || !range_of(at, &r) || r.begin > at || r.end <= at || r.device == 0) return 0;
    const uintptr_t d = r.device + (at - r.begin);
    if (at == a) device = d;
    else if (d - device != at - a) return 0;
    at = r.end;
  }
  return device % 4 == 0 ? device : 0;
}

inline bool overlap(const void *a, size_t na, const void *b, size_t nb) {
  const uintptr_t x = (uintptr_t)a, y = (uintptr_t)b;
  return x < y + nb && y < x + na;
}

}  // namespace p2z
