// p2z_shape.h -- the launch shape of a run: what the caller's config leaves open is
// taken from the context's p2z_autotune measurements of the same kind of run,
// else from the rules here.  Host code only, tested on the CPU.
#pragma once

#include <cstdint>
#include <vector>

#include "p2z.h"

namespace p2z {

// What a run's hit mask holds: there is none; uneven events given without one
// (their padding, every layer of the real tracks present); the caller's.
// The last two are different work: sorting windows by hit count gains only
// where the counts differ, so neither's measured shape says anything of the other's.
enum MaskKind { MASK_NONE = 0, MASK_PADDING, MASK_CALLER };

// The kind of run that a measured shape applies to.
struct RunKind {
  int upd, sc, B;
  bool soa;
  MaskKind mask;
  bool operator==(const RunKind &o) const {
    return upd == o.upd && sc == o.sc && B == o.B && soa == o.soa && mask == o.mask;
  }
};

struct Shape {
  int block;     // threads per CTA, 0: the schedule's default
  int schedule;  // p2z_schedule
  int tpt;       // threads per track, 0: one
  bool sort;     // P2Z_FLAG_SORT_WINDOWS
};

// p2z_autotune's fastest shape of one kind of run.
struct Tuned {
  RunKind kind;
  Shape shape;
};

inline void record_shape(std::vector<Tuned> &tuned, const RunKind &kind, const Shape &shape) {
  for (Tuned &t : tuned)
    if (t.kind == kind) {
      t.shape = shape;
      return;
    }
  tuned.push_back({kind, shape});
}

// Runs that leave the schedule open sort from this many slots an SM on: a launch
// whose warps are all resident at once lasts as long as its longest track anyway.
// One B200, 2-D update, us per pass, stored order / sorted: 51,000 tracks 18.6 /
// 20.8, 102,000 30.7 / 30.8, 152,000 41.0 / 39.2, 406,000 88.1 / 81.6.
constexpr int64_t kSortMinSlotsPerSm = 768;

// Fills what `s`, the caller's wishes, leaves open (block 0, schedule AUTO -- with
// the window sorting measured with it --, tpt 0).  A tuned shape whose schedule
// the caller overrides with STAGED keeps one thread per track.
inline Shape choose_shape(const std::vector<Tuned> &tuned, const RunKind &kind, Shape s, int64_t nslots, int num_sms) {
  for (const Tuned &t : tuned) {
    if (!(t.kind == kind)) continue;
    if (s.block == 0) s.block = t.shape.block;
    if (s.schedule == P2Z_SCHED_AUTO) {
      s.schedule = t.shape.schedule;
      s.sort = s.sort || t.shape.sort;
    }
    if (s.tpt == 0 && s.schedule != P2Z_SCHED_STAGED) s.tpt = t.shape.tpt;
    break;
  }
  if (s.schedule == P2Z_SCHED_AUTO) {
    s.schedule = P2Z_SCHED_FLAT;
    s.sort = s.sort || (kind.mask == MASK_CALLER && nslots >= num_sms * kSortMinSlotsPerSm);
  }
  if (s.tpt == 0) s.tpt = 1;
  return s;
}

}  // namespace p2z
