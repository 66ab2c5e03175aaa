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

// Shape::sort_from of runs that never sort.  (P2Z_FLAG_SORT_WINDOWS: 0.)
constexpr int64_t kNeverSort = INT64_MAX;

struct Shape {
  int block;          // threads per CTA, 0: the schedule's default
  int schedule;       // p2z_schedule
  int tpt;            // threads per track, 0: one
  int64_t sort_from;  // a masked launch of this many slots or more sorts its windows
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

// Launches of runs that leave the schedule open sort from this many slots an SM on:
// one whose warps are all resident at once lasts as long as its longest track anyway.
// A launch, not a run: p2z_run cuts a run into chunks, the last ones small.
// One B200, 32 slots a batch, 2-D update, us per pass, stored order / sorted: 64,000
// slots 18.1 / 19.4, 113,000 27.5 / 26.2, 154,000 38.3 / 36.8, 306,000 68.9 / 61.9,
// 1,006,000 201.6 / 172.8; the other updates gain more (reference rounding 549.9 /
// 408.2, 3-D with FP64 421.4 / 319.9), 64 slots a batch and SoA as much, 16 slots less
// (203.6 / 181.7).  In batches of 8 a sorted warp's loads reach 16 batches, a sector each:
// the 2-D update loses (113,000 28.9 / 31.0, 306,000 71.1 / 73.8, 1,004,000 207.3 /
// 208.7) and keeps the stored order, the others still gain (235.2 / 215.2 the least).
constexpr int64_t kSortMinSlotsPerSm = 768;

// Fills what `s`, the caller's wishes, leaves open (block 0, schedule AUTO -- with
// the window sorting measured with it --, tpt 0).  A tuned shape whose schedule
// the caller overrides with STAGED keeps one thread per track.
inline Shape choose_shape(const std::vector<Tuned> &tuned, const RunKind &kind, Shape s, int num_sms) {
  for (const Tuned &t : tuned) {
    if (!(t.kind == kind)) continue;
    if (s.block == 0) s.block = t.shape.block;
    if (s.schedule == P2Z_SCHED_AUTO) {
      s.schedule = t.shape.schedule;
      if (t.shape.sort_from < s.sort_from) s.sort_from = t.shape.sort_from;
    }
    if (s.tpt == 0 && s.schedule != P2Z_SCHED_STAGED) s.tpt = t.shape.tpt;
    break;
  }
  if (s.schedule == P2Z_SCHED_AUTO) {
    s.schedule = P2Z_SCHED_FLAT;
    const bool scattered = kind.upd == P2Z_UPDATE_V2 && kind.B == 8 && !kind.soa;
    if (kind.mask == MASK_CALLER && !scattered && s.sort_from == kNeverSort) s.sort_from = num_sms * kSortMinSlotsPerSm;
  }
  if (s.tpt == 0) s.tpt = 1;
  return s;
}

}  // namespace p2z
