// The rule on the host arrays that p2z_run hands to a kernel (csrc/p2z_direct.h),
// on page-locked ranges that exist only here: prints one line a case.
#include <cstdio>
#include <vector>

#include "p2z_direct.h"

using p2z::HostRange;

static uintptr_t ask(const std::vector<HostRange> &locked, uintptr_t p, size_t bytes) {
  return p2z::mapped_array((const void *)p, bytes, [&](uintptr_t at, HostRange *r) {
    for (const HostRange &h : locked)
      if (h.begin <= at && at < h.end) {
        *r = h;
        return true;
      }
    return false;
  });
}

int main() {
  auto say = [](const char *name, uintptr_t got) { std::printf("%s %#llx\n", name, (unsigned long long)got); };
  const std::vector<HostRange> one = {{0x10000, 0x20000, 0x910000}};
  say("whole", ask(one, 0x10000, 0x10000));
  say("inside", ask(one, 0x10404, 0x100));
  say("last_byte_past", ask(one, 0x10000, 0x10001));
  say("first_byte_before", ask(one, 0xfffc, 0x100));
  say("pageable", ask(one, 0x40000, 0x100));
  for (int odd = 1; odd < 4; ++odd) say("off_a_word", ask(one, 0x10000 + odd, 0x100));
  say("empty", ask(one, 0x10000, 0));
  say("wraps", ask({{0, UINTPTR_MAX, 0x1000}}, UINTPTR_MAX - 3, 8));
  say("not_mapped", ask({{0x10000, 0x20000, 0}}, 0x10000, 4));
  const HostRange first = {0x10000, 0x18000, 0x910000};
  say("two_pieces", ask({first, {0x18000, 0x20000, 0x918000}}, 0x10004, 0xfffc));
  say("hole_between", ask({first, {0x18004, 0x20000, 0x918004}}, 0x10004, 0xfffc));
  say("device_gap", ask({first, {0x18000, 0x20000, 0xa18000}}, 0x10004, 0xfffc));
  std::vector<HostRange> many;
  for (uintptr_t i = 0; i < 65; ++i) many.push_back({0x10000 + i * 0x100, 0x10100 + i * 0x100, 0x910000 + i * 0x100});
  say("most_pieces", ask(many, 0x10000, 64 * 0x100));
  say("too_many_pieces", ask(many, 0x10000, 64 * 0x100 + 4));
  char a[64];
  auto both = [&](const char *name, int x, int nx, int y, int ny) {
    say(name, 2 * p2z::overlap(a + x, nx, a + y, ny) + p2z::overlap(a + y, ny, a + x, nx));
  };
  both("same", 0, 8, 0, 8);
  both("apart", 0, 8, 8, 8);
  both("by_one", 0, 9, 8, 8);
  both("within", 0, 64, 8, 8);
  return 0;
}
