// The launch shape of a run (csrc/p2z_shape.h): prints block, schedule, threads per
// track and sorting for runs of each mask kind, with and without measurements.
#include <cstdio>

#include "p2z_shape.h"

using namespace p2z;

static const int kSms = 148;
static const int64_t kNo = kNeverSort;

static RunKind kind(MaskKind mask, int upd = P2Z_UPDATE_V2, int B = 32, bool soa = false) {
  return {upd, 0, B, soa, mask};
}

static void say(const char *name, const std::vector<Tuned> &tuned, const RunKind &k, Shape ask) {
  const Shape s = choose_shape(tuned, k, ask, kSms);
  std::printf("%s: block %d schedule %d tpt %d sort ", name, s.block, s.schedule, s.tpt);
  if (s.sort_from == kNeverSort) std::printf("never\n");
  else std::printf("from %lld\n", (long long)s.sort_from);
}

int main() {
  const Shape open = {0, P2Z_SCHED_AUTO, 0, kNo};
  const RunKind none = kind(MASK_NONE), padding = kind(MASK_PADDING), caller = kind(MASK_CALLER);
  std::vector<Tuned> nothing, pad, own;
  say("none", nothing, none, open);
  say("padding", nothing, padding, open);
  say("caller", nothing, caller, open);
  say("caller, flat asked", nothing, caller, {0, P2Z_SCHED_FLAT, 0, kNo});
  say("caller, sorting asked", nothing, caller, {64, P2Z_SCHED_PERSISTENT, 2, 0});
  say("caller, auto and sorting asked", nothing, caller, {0, P2Z_SCHED_AUTO, 0, 0});
  // batches of 8: the 2-D update alone keeps the stored order
  say("8", nothing, kind(MASK_CALLER, P2Z_UPDATE_V2, 8), open);
  say("8, sorting asked", nothing, kind(MASK_CALLER, P2Z_UPDATE_V2, 8), {0, P2Z_SCHED_AUTO, 0, 0});
  say("8, 3-D", nothing, kind(MASK_CALLER, P2Z_UPDATE_3X3_F64, 8), open);
  say("16", nothing, kind(MASK_CALLER, P2Z_UPDATE_V2, 16), open);
  say("SoA of 8", nothing, kind(MASK_CALLER, P2Z_UPDATE_V2, 8, true), open);
  // measured on uneven events without a mask: nothing for runs with one
  record_shape(pad, padding, {64, P2Z_SCHED_FLAT, 2, kNo});
  say("padding, measured", pad, padding, open);
  say("caller after padding", pad, caller, open);
  say("none after padding", pad, none, open);
  // and the other way round
  record_shape(own, caller, {256, P2Z_SCHED_FLAT, 1, 0});
  say("caller, measured", own, caller, open);
  say("padding after caller", own, padding, open);
  say("none after caller", own, none, open);
  // a second measurement replaces the first; what the caller sets stays
  record_shape(own, caller, {32, P2Z_SCHED_PERSISTENT, 2, kNo});
  say("caller, again", own, caller, open);
  say("caller, staged", own, caller, {0, P2Z_SCHED_STAGED, 0, kNo});
  say("caller, all set", own, caller, {128, P2Z_SCHED_FLAT, 1, 0});
  return 0;
}
