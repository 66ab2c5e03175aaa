// The launch shape of a run (csrc/p2z_shape.h): prints block, schedule, threads per
// track and sorting for runs of each mask kind, with and without measurements.
#include <cstdio>

#include "p2z_shape.h"

using namespace p2z;

static const int kSms = 148;
static const int64_t kLarge = kSms * kSortMinSlotsPerSm;

static RunKind kind(MaskKind mask) { return {P2Z_UPDATE_V2, 0, 32, false, mask}; }

static void say(const char *name, const std::vector<Tuned> &tuned, MaskKind mask, Shape ask, int64_t nslots) {
  const Shape s = choose_shape(tuned, kind(mask), ask, nslots, kSms);
  std::printf("%s: block %d schedule %d tpt %d sort %d\n", name, s.block, s.schedule, s.tpt, (int)s.sort);
}

int main() {
  const Shape open = {0, P2Z_SCHED_AUTO, 0, false};
  std::vector<Tuned> none, pad, own;
  say("none", none, MASK_NONE, open, kLarge);
  say("padding", none, MASK_PADDING, open, kLarge);
  say("caller, large", none, MASK_CALLER, open, kLarge);
  say("caller, small", none, MASK_CALLER, open, kLarge - 1);
  say("caller, flat asked", none, MASK_CALLER, {0, P2Z_SCHED_FLAT, 0, false}, kLarge);
  say("caller, sorting asked", none, MASK_CALLER, {64, P2Z_SCHED_PERSISTENT, 2, true}, 1);
  // measured on uneven events without a mask: nothing for runs with one
  record_shape(pad, kind(MASK_PADDING), {64, P2Z_SCHED_FLAT, 2, false});
  say("padding, measured", pad, MASK_PADDING, open, kLarge);
  say("caller after padding", pad, MASK_CALLER, open, kLarge);
  say("none after padding", pad, MASK_NONE, open, kLarge);
  // and the other way round
  record_shape(own, kind(MASK_CALLER), {256, P2Z_SCHED_FLAT, 1, true});
  say("caller, measured", own, MASK_CALLER, open, 1);
  say("padding after caller", own, MASK_PADDING, open, kLarge);
  say("none after caller", own, MASK_NONE, open, kLarge);
  // a second measurement replaces the first; what the caller sets stays
  record_shape(own, kind(MASK_CALLER), {32, P2Z_SCHED_PERSISTENT, 2, false});
  say("caller, again", own, MASK_CALLER, open, kLarge);
  say("caller, staged", own, MASK_CALLER, {0, P2Z_SCHED_STAGED, 0, false}, kLarge);
  say("caller, all set", own, MASK_CALLER, {128, P2Z_SCHED_FLAT, 1, true}, kLarge);
  return 0;
}
