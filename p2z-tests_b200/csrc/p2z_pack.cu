// p2z_pack.cu -- packing an uneven sample in order of hit count on the device.
//
// A warp's 32 tracks take as many steps as the one with the most hits, so
// tracks with missing layers run fastest when each batch holds tracks of
// similar hit counts.  p2z_pack_by_hits_device writes a copy of the arrays in
// which every event's tracks are in order of decreasing hit count (equal
// counts keep their order; each event keeps its slots, padding last), plus the
// permutation; p2z_unpack_tracks_device puts a packed output back in the
// caller's order.  No counterpart in the reference, whose events hold every
// layer of every track (src/propagate-toz-test_OMP.cpp:731-748).
//
// Both directions move windows of kWindow slots through shared memory: the side
// whose slots are neighbours (the caller's order) is read or written in
// 16-byte pieces, and the other side in the order of the packed slots, where a
// window's slots of one event and hit count are neighbours (512 slots of events
// with 16 hit counts: runs of 30).  A copy that takes each slot's words where they
// are moves a 32-byte sector through L2 for every 4-byte word.  The order itself
// is a counting sort (a radix sort of 64-bit keys before).  One B200, 3.2M slots, 20
// layers, before / now: pack 1885 / 1238 us (5.6 GB of DRAM traffic, 4.5 TB/s; with
// registers capped for 3 or 4 CTAs an SM instead of 2, 1383 and 1468), unpack
// 240 / 156 us.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdio>
#include <vector>

#include "p2z.h"
#include "p2z_kernels.cuh"

namespace p2z {
void set_context_free_error(const char *msg);
int context_device(const p2z_context *ctx);
int context_sms(const p2z_context *ctx);
cudaStream_t context_stream(const p2z_context *ctx);
p2z_status context_fail(p2z_context *ctx, p2z_status st, const char *msg);
void *context_scratch(p2z_context *ctx, size_t bytes);
}  // namespace p2z

using namespace p2z;

namespace {

#define PACK_CUDA(ctx, call)                                                                    \
  do {                                                                                          \
    cudaError_t e_ = (call);                                                                    \
    if (e_ != cudaSuccess) {                                                                    \
      char m_[300];                                                                             \
      std::snprintf(m_, sizeof m_, "%s: %s (%s:%d)", #call, cudaGetErrorString(e_), __FILE__, \
                    __LINE__);                                                                  \
      return context_fail((ctx), e_ == cudaErrorMemoryAllocation ? P2Z_OOM : P2Z_CUDA_ERROR, m_); \
    }                                                                                           \
  } while (0)

size_t up256(size_t n) { return (n + 255) / 256 * 256; }

constexpr int kWindow = 512;   // slots, one a thread
constexpr int kClasses = 34;   // 32 - hit count of a real track (0: all of 32 layers), 33 padding
constexpr int kMaxParts = 64;  // events a window can meet (bsize 8)
constexpr int kFillPerSm = 4;    // CTAs an SM that fill the GPU
constexpr int kUnpackPerSm = 6;  // windows an SM from which unpacking goes through shared memory

// The events' tables on the device: slots from beg[e] on, count[e] real tracks.
struct Events {
  const int64_t *beg;    // n + 1
  const int64_t *count;  // n
  int n;
};
__device__ __forceinline__ int event_of(const Events &ev, int64_t s) {  // the last e with beg[e] <= s
  int lo = 0, hi = ev.n - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (ev.beg[mid] <= s) lo = mid;
    else hi = mid - 1;
  }
  return lo;
}

// A slot's part of its window w (the event's first slot there, in eighths of a
// batch: 0..63) and hit-count class.
__device__ __forceinline__ int part_class(const Events &ev, const uint32_t *mask, uint32_t all, int64_t s, int64_t w0,
                                          int *event, int *part) {
  const int e = event_of(ev, s);
  *event = e;
  *part = (int)(max(ev.beg[e], w0) - w0) / 8;
  const uint32_t m = mask ? (__ldg(mask + s) & all) : all;
  return s - ev.beg[e] < ev.count[e] ? 32 - __popc(m) : 33;
}

// Per window and event in it: the slots of each class.  The row of event e and
// window w is e + w: rows in the order of the slots, no two the same.
__global__ void __launch_bounds__(kWindow) k_pack_count(Events ev, const uint32_t *__restrict__ mask, uint32_t all,
                                                        int64_t nslots, uint32_t *__restrict__ rows) {
  __shared__ uint32_t count[kMaxParts][kClasses];
  for (int i = threadIdx.x; i < kMaxParts * kClasses; i += kWindow) (&count[0][0])[i] = 0u;
  __syncthreads();
  const int64_t w0 = (int64_t)blockIdx.x * kWindow, s = w0 + threadIdx.x;
  int e = 0, part = 0;
  if (s < nslots) {
    const int cls = part_class(ev, mask, all, s, w0, &e, &part);
    atomicAdd(&count[part][cls], 1u);
  }
  __syncthreads();
  if (s < nslots && max(ev.beg[e], w0) == s)
    for (int c = 0; c < kClasses; ++c) rows[((int64_t)e + blockIdx.x) * kClasses + c] = count[part][c];
}

// An event's rows' counts become the offsets, from the event's first slot on, of
// the row's first slot of each class.  Lane l of a warp takes class l, lanes 0 and
// 1 classes 32 and 33 as well.  The sums over rows [r0, r1):
struct ClassSums {
  uint32_t a, b;
};
constexpr int kRowsAhead = 8;  // loads in flight; the walk is otherwise a load's latency a row
__device__ __forceinline__ ClassSums sum_rows(const uint32_t *rows, int64_t r0, int64_t r1) {
  const int lane = threadIdx.x & 31;
  const bool two = lane < kClasses - 32;
  ClassSums s = {0u, 0u};
#pragma unroll 8
  for (int64_t r = r0; r < r1; ++r) {
    s.a += rows[r * kClasses + lane];
    if (two) s.b += rows[r * kClasses + 32 + lane];
  }
  return s;
}
// The first offset of each class in an event with these sums.
__device__ __forceinline__ ClassSums first_offsets(ClassSums s) {
  const int lane = threadIdx.x & 31;
  uint32_t at = s.a;
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t u = __shfl_up_sync(0xffffffffu, at, o);
    if (lane >= o) at += u;
  }
  const uint32_t real32 = __shfl_sync(0xffffffffu, at, 31), b0 = __shfl_sync(0xffffffffu, s.b, 0);
  return {at - s.a, real32 + (lane ? b0 : 0u)};
}
// Rows [r0, r1) from counts to offsets, the first row's from `at` on.
__device__ __forceinline__ void place_rows(uint32_t *rows, int64_t r0, int64_t r1, ClassSums at) {
  const int lane = threadIdx.x & 31;
  const bool two = lane < kClasses - 32;
  for (int64_t r = r0; r < r1; r += kRowsAhead) {
    uint32_t a[kRowsAhead], b[kRowsAhead];
#pragma unroll
    for (int j = 0; j < kRowsAhead; ++j) {
      a[j] = r + j < r1 ? rows[(r + j) * kClasses + lane] : 0u;
      b[j] = r + j < r1 && two ? rows[(r + j) * kClasses + 32 + lane] : 0u;
    }
#pragma unroll
    for (int j = 0; j < kRowsAhead; ++j) {
      if (r + j < r1) {
        rows[(r + j) * kClasses + lane] = at.a;
        if (two) rows[(r + j) * kClasses + 32 + lane] = at.b;
      }
      at.a += a[j];
      at.b += b[j];
    }
  }
}
__device__ __forceinline__ void event_rows(const Events &ev, int64_t e, int64_t *r0, int64_t *r1) {
  *r0 = e + ev.beg[e] / kWindow;
  *r1 = ev.beg[e + 1] == ev.beg[e] ? *r0 : e + (ev.beg[e + 1] - 1) / kWindow + 1;
}

// Events of at most kWarpRows rows: one warp each.  The others: one CTA each, whose
// warps share the rows.  (With one warp for every event, one event of a million
// tracks and one layer took 444 us to pack, now 132, and of 10 million 4211, now 922; with 20
// layers, a million, 711 and 398.)
constexpr int64_t kWarpRows = 32;
__global__ void __launch_bounds__(128) k_pack_offsets(Events ev, uint32_t *__restrict__ rows) {
  const int64_t e = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (e >= ev.n) return;
  int64_t r0, r1;
  event_rows(ev, e, &r0, &r1);
  if (r1 - r0 > kWarpRows) return;
  place_rows(rows, r0, r1, first_offsets(sum_rows(rows, r0, r1)));
}
__global__ void __launch_bounds__(1024) k_pack_offsets_wide(Events ev, const int64_t *__restrict__ events,
                                                            uint32_t *__restrict__ rows) {
  __shared__ ClassSums sums[32][32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int64_t r0, r1;
  event_rows(ev, events[blockIdx.x], &r0, &r1);
  const int64_t per = (r1 - r0 + 31) / 32, w0 = min(r1, r0 + warp * per), w1 = min(r1, w0 + per);
  sums[warp][lane] = sum_rows(rows, w0, w1);
  __syncthreads();
  ClassSums all = {0u, 0u}, before = {0u, 0u};
  for (int w = 0; w < 32; ++w) {
    const ClassSums s = sums[w][lane];
    all.a += s.a;
    all.b += s.b;
    if (w < warp) {
      before.a += s.a;
      before.b += s.b;
    }
  }
  const ClassSums first = first_offsets(all);
  place_rows(rows, w0, w1, {first.a + before.a, first.b + before.b});
}

// Sorts kWindow keys, ascending, a key a thread (bitonic: partners in the same
// warp exchange by shuffle, the others through sh); returns the thread's key and
// leaves all of them in sh.
template <typename K>
__device__ __forceinline__ K sort_window(K key, K *sh) {
  const int i = threadIdx.x;
  for (int k = 2; k <= kWindow; k <<= 1)
    for (int j = k >> 1; j > 0; j >>= 1) {
      K other;
      if (j < 32) {
        other = __shfl_xor_sync(0xffffffffu, key, j);
      } else {
        __syncthreads();
        sh[i] = key;
        __syncthreads();
        other = sh[i ^ j];
      }
      const bool low = ((i & j) == 0) == ((i & k) == 0);  // keep the smaller
      key = (key < other) == low ? key : other;
    }
  __syncthreads();
  sh[i] = key;
  __syncthreads();
  return key;
}

// One slot's words in an AOSOA array whose batches are `bw` words long (28 B
// for tracks; nlayer * 9 * B for hits, whose layers of a batch are
// contiguous): word r of slot s is at (s / B) * bw + s % B + r * B.
template <int B>
__device__ __forceinline__ int64_t slot_base(int64_t s, int64_t bw) {
  return (s / B) * bw + s % B;
}

// R rows of a window's slots (n of them, a multiple of B) between `flat`, the
// window's first batch at those rows, and shared memory, where batch b's R rows
// of B words lie from b R B on.  quads: the array is 16-byte aligned.
template <int B, int R>
__device__ __forceinline__ void fetch_window(const uint32_t *flat, int64_t bw, int n, uint32_t *sh, bool quads) {
  constexpr int kPer = R * B / 4;  // 16-byte pieces a batch
  const uint32_t dst = (uint32_t)__cvta_generic_to_shared(sh);
  if (quads) {
    for (int p = threadIdx.x; p < n / B * kPer; p += kWindow)
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + p * 16),
                   "l"(flat + (int64_t)(p / kPer) * bw + p % kPer * 4)
                   : "memory");
  } else {
    for (int p = threadIdx.x; p < n * R; p += kWindow)
      asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst + p * 4),
                   "l"(flat + (int64_t)(p / (R * B)) * bw + p % (R * B))
                   : "memory");
  }
}
template <int B, int R>
__device__ __forceinline__ void write_window(uint32_t *flat, int64_t bw, int n, const uint32_t *sh, bool quads) {
  constexpr int kPer = R * B / 4;
  if (quads) {
    for (int p = threadIdx.x; p < n / B * kPer; p += kWindow)
      __stcs(reinterpret_cast<uint4 *>(flat + (int64_t)(p / kPer) * bw) + p % kPer,
             reinterpret_cast<const uint4 *>(sh)[p]);
  } else {
    for (int p = threadIdx.x; p < n * R; p += kWindow) flat[(int64_t)(p / (R * B)) * bw + p % (R * B)] = sh[p];
  }
}

// The packed copy of the window blockIdx.x: blockIdx.y's share of the hit layers
// and, for blockIdx.y == 0, the tracks, the masks and the permutation.
template <int B>
__global__ void __launch_bounds__(kWindow) k_pack_move(Events ev, const uint32_t *__restrict__ mask, uint32_t all,
                                                       int64_t nslots, const uint32_t *__restrict__ rows, int nlayer,
                                                       int per, const uint32_t *trk, const uint32_t *hits,
                                                       uint32_t *trk_out, uint32_t *hits_out, uint32_t *mask_out,
                                                       int64_t *perm, bool quads) {
  __shared__ uint32_t key[kWindow];                  // part, class and slot, sorted
  __shared__ __align__(16) uint32_t sh[2][9 * kWindow];
  const int i = threadIdx.x;
  const int64_t w0 = (int64_t)blockIdx.x * kWindow, b0 = w0 / B;
  const int n = (int)min((int64_t)kWindow, nslots - w0);
  // this CTA's rows: its layers, 9 a turn, then (blockIdx.y == 0) the tracks, 7 a turn
  const int64_t bw = (int64_t)nlayer * 9 * B;
  const int l0 = blockIdx.y * per, layers = min(nlayer - l0, per), turns = layers + (blockIdx.y == 0 ? 4 : 0);
  auto fetch = [&](int t) {
    if (t < layers)
      fetch_window<B, 9>(hits + b0 * bw + (int64_t)(l0 + t) * 9 * B, bw, n, sh[t & 1], quads);
    else if (t < turns)
      fetch_window<B, 7>(trk + b0 * (TRK_WORDS * B) + (t - layers) * 7 * B, (int64_t)TRK_WORDS * B, n, sh[t & 1], quads);
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  fetch(0);
  uint32_t own = 0xffffffffu;
  if (i < n) {
    int e, part;
    const int cls = part_class(ev, mask, all, w0 + i, w0, &e, &part);
    own = ((uint32_t)part << 15) | ((uint32_t)cls << 9) | (uint32_t)i;
  }
  const uint32_t k = sort_window(own, key);
  // thread i: the window's i-th slot in that order, its place among those of its
  // part and class, and so its packed slot
  int from = 0;
  int64_t to = 0;
  if (i < n) {
    from = (int)(k & (kWindow - 1));
    int lo = 0, hi = i;  // the first of the same part and class
    while (lo < hi) {
      const int mid = (lo + hi) >> 1;
      if (key[mid] >> 9 == k >> 9) hi = mid;
      else lo = mid + 1;
    }
    const int ev_i = event_of(ev, w0 + from);
    to = ev.beg[ev_i] + rows[((int64_t)ev_i + blockIdx.x) * kClasses + ((k >> 9) & 63u)] + (i - lo);
  }
  uint32_t *hit_to = hits_out + slot_base<B>(to, bw) + (int64_t)l0 * 9 * B;
  uint32_t *trk_to = trk_out + slot_base<B>(to, (int64_t)TRK_WORDS * B);
  const int hit_at = from / B * (9 * B) + from % B, trk_at = from / B * (7 * B) + from % B;
  for (int t = 0; t < turns; ++t) {
    fetch(t + 1);
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    __syncthreads();
    if (i < n) {
      if (t < layers) {
#pragma unroll
        for (int r = 0; r < 9; ++r) __stcs(hit_to + (int64_t)(t * 9 + r) * B, sh[t & 1][hit_at + r * B]);
      } else {
#pragma unroll
        for (int r = 0; r < 7; ++r) __stcs(trk_to + ((t - layers) * 7 + r) * B, sh[t & 1][trk_at + r * B]);
      }
    }
    __syncthreads();
  }
  if (blockIdx.y != 0) return;
  int64_t *inv = reinterpret_cast<int64_t *>(&sh[0][0]);
  if (i < n) {
    perm[to] = w0 + from;
    if (mask) mask_out[to] = __ldg(mask + w0 + from);
    inv[from] = to;
  }
  __syncthreads();
  if (i < n) perm[nslots + w0 + i] = inv[i];
}

// The tracks of the window blockIdx.x of the caller's slots from their packed
// ones: inv[s] is the packed slot of slot s.
template <int B>
__global__ void __launch_bounds__(kWindow) k_unpack(const int64_t *__restrict__ inv, int64_t nslots,
                                                    const uint32_t *__restrict__ packed, uint32_t *out, bool quads) {
  __shared__ uint64_t key[kWindow];
  __shared__ __align__(16) uint32_t sh[2][7 * kWindow];
  const int i = threadIdx.x;
  const int64_t w0 = (int64_t)blockIdx.x * kWindow;
  const int n = (int)min((int64_t)kWindow, nslots - w0);
  // (packed slots below 2^54)
  const uint64_t k = sort_window<uint64_t>(i < n ? ((uint64_t)inv[w0 + i] << 9) | (uint64_t)i : ~(uint64_t)0, key);
  const int to = (int)(k & (kWindow - 1));
  const uint32_t *in = packed + (i < n ? slot_base<B>((int64_t)(k >> 9), (int64_t)TRK_WORDS * B) : 0);
  uint32_t v[7];
  auto read = [&](int q) {
#pragma unroll
    for (int r = 0; r < 7; ++r) v[r] = __ldg(in + (q * 7 + r) * B);
  };
  if (i < n) read(0);
  for (int q = 0; q < 4; ++q) {
    uint32_t *s = sh[q & 1];
    if (i < n) {
#pragma unroll
      for (int r = 0; r < 7; ++r) s[to / B * (7 * B) + r * B + to % B] = v[r];
      if (q < 3) read(q + 1);
    }
    __syncthreads();
    write_window<B, 7>(out + w0 / B * (TRK_WORDS * B) + q * 7 * B, (int64_t)TRK_WORDS * B, n, s, quads);
  }
}

// Small unpacks: thread = slot, its words read where they are.
__global__ void __launch_bounds__(256) k_unpack_direct(const int64_t *__restrict__ inv, int64_t nslots, int B,
                                                       const uint32_t *__restrict__ packed, uint32_t *out) {
  const int64_t s = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= nslots) return;
  const int64_t p = inv[s];
  const uint32_t *in = packed + p / B * (TRK_WORDS * B) + p % B;
  uint32_t *to = out + s / B * (TRK_WORDS * B) + s % B;
#pragma unroll 4
  for (int r = 0; r < TRK_WORDS; ++r) to[r * B] = in[r * B];
}

bool aligned16(const void *a, const void *b) { return (((uintptr_t)a | (uintptr_t)b) & 15u) == 0; }

// Event tables of a config: per-event real tracks and first slots (nevts + 1), and the
// events of more than kWarpRows rows.
void event_tables(const p2z_config *c, std::vector<int64_t> &counts, std::vector<int64_t> &beg,
                  std::vector<int64_t> &wide) {
  const int64_t ne = c->nevts;
  counts.assign((size_t)ne, 0);
  beg.assign((size_t)ne + 1, 0);
  for (int64_t e = 0; e < ne; ++e) {
    counts[e] = c->event_ntrks ? c->event_ntrks[e] : c->ntrks;
    beg[e + 1] = beg[e] + (counts[e] + c->bsize - 1) / c->bsize * c->bsize;
    if (counts[e] > (kWarpRows - 1) * kWindow && (beg[e + 1] - 1) / kWindow - beg[e] / kWindow >= kWarpRows)
      wide.push_back(e);
  }
}

p2z_status check_config(p2z_context *ctx, const p2z_config *cfg, int64_t *nslots) {
  if (!cfg) return context_fail(ctx, P2Z_BAD_ARG, "config is NULL");
  const int64_t nb = p2z_num_batches(cfg);
  if (nb < 0) return context_fail(ctx, P2Z_BAD_ARG, p2z_last_error(nullptr));
  if (cfg->layout != P2Z_LAYOUT_AOSOA) return context_fail(ctx, P2Z_UNSUPPORTED, "packing needs the AOSOA layout");
  if (cfg->nevts >= (1LL << 30)) return context_fail(ctx, P2Z_BAD_ARG, "too many events");
  *nslots = nb * cfg->bsize;
  return P2Z_OK;
}

}  // namespace

extern "C" {

p2z_status p2z_pack_by_hits_device(p2z_context *ctx, const p2z_config *cfg, const void *d_trk_in,
                                   const void *d_hits_in, const uint32_t *d_mask_in, void *d_trk_out,
                                   void *d_hits_out, uint32_t *d_mask_out, int64_t *d_perm, void *stream) {
  if (!ctx) {
    set_context_free_error("context is NULL");
    return P2Z_BAD_ARG;
  }
  int64_t ns = 0;
  p2z_status r = check_config(ctx, cfg, &ns);
  if (r != P2Z_OK) return r;
  if ((d_mask_in == nullptr) != (d_mask_out == nullptr))
    return context_fail(ctx, P2Z_BAD_ARG, "pass both masks or neither");
  if (ns == 0) return P2Z_OK;
  if (!d_trk_in || !d_hits_in || !d_trk_out || !d_hits_out || !d_perm)
    return context_fail(ctx, P2Z_BAD_ARG, "NULL device buffer");
  if (d_trk_in == d_trk_out || d_hits_in == d_hits_out || (d_mask_in && d_mask_in == d_mask_out))
    return context_fail(ctx, P2Z_BAD_ARG, "the packed copy must not alias the input");
  PACK_CUDA(ctx, cudaSetDevice(context_device(ctx)));
  cudaStream_t st = stream ? (cudaStream_t)stream : context_stream(ctx);
  std::vector<int64_t> counts, beg, wide;
  event_tables(cfg, counts, beg, wide);
  const int ne = (int)cfg->nevts;
  const int64_t nwin = (ns + kWindow - 1) / kWindow;
  if (nwin > 0x7fffffff) return context_fail(ctx, P2Z_BAD_ARG, "too many slots");
  // scratch, from the context's reusable device buffer (parts 256-byte aligned): event tables and
  // the rows of counts (one per event and window)
  const size_t nwide = wide.size();
  const size_t b_tab = up256(sizeof(int64_t) * (2 * (size_t)ne + 1 + nwide));
  char *scr = static_cast<char *>(
      context_scratch(ctx, b_tab + up256(sizeof(uint32_t) * kClasses * ((size_t)ne + (size_t)nwin))));
  if (!scr) return context_fail(ctx, P2Z_OOM, "no device memory for the packing scratch");
  int64_t *d_counts = (int64_t *)scr, *d_beg = d_counts + ne, *d_wide = d_beg + ne + 1;
  uint32_t *rows = (uint32_t *)(scr + b_tab);
  PACK_CUDA(ctx, cudaMemcpyAsync(d_counts, counts.data(), sizeof(int64_t) * ne, cudaMemcpyHostToDevice, st));
  PACK_CUDA(ctx, cudaMemcpyAsync(d_beg, beg.data(), sizeof(int64_t) * (ne + 1), cudaMemcpyHostToDevice, st));
  if (nwide)
    PACK_CUDA(ctx, cudaMemcpyAsync(d_wide, wide.data(), sizeof(int64_t) * nwide, cudaMemcpyHostToDevice, st));
  const Events ev{d_beg, d_counts, ne};
  const int nl = cfg->nlayer;
  const uint32_t all = nl >= 32 ? 0xffffffffu : ((1u << nl) - 1u);
  k_pack_count<<<(unsigned)nwin, kWindow, 0, st>>>(ev, d_mask_in, all, ns, rows);
  PACK_CUDA(ctx, cudaGetLastError());
  k_pack_offsets<<<(unsigned)(((int64_t)ne * 32 + 127) / 128), 128, 0, st>>>(ev, rows);
  PACK_CUDA(ctx, cudaGetLastError());
  if (nwide) {
    k_pack_offsets_wide<<<(unsigned)nwide, 1024, 0, st>>>(ev, d_wide, rows);
    PACK_CUDA(ctx, cudaGetLastError());
  }
  // small samples: a window's layers are shared out until the GPU is full
  const int shares = (int)std::max<int64_t>(1, std::min<int64_t>(nl, (int64_t)kFillPerSm * context_sms(ctx) / nwin));
  const int per = (nl + shares - 1) / shares;
  auto *f = cfg->bsize == 8 ? k_pack_move<8> : cfg->bsize == 16 ? k_pack_move<16> : cfg->bsize == 32 ? k_pack_move<32>
                                                                                                     : k_pack_move<64>;
  f<<<dim3((unsigned)nwin, (unsigned)((nl + per - 1) / per)), kWindow, 0, st>>>(
      ev, d_mask_in, all, ns, rows, nl, per, (const uint32_t *)d_trk_in, (const uint32_t *)d_hits_in,
      (uint32_t *)d_trk_out, (uint32_t *)d_hits_out, d_mask_out, d_perm, aligned16(d_trk_in, d_hits_in));
  PACK_CUDA(ctx, cudaGetLastError());
  PACK_CUDA(ctx, cudaStreamSynchronize(st));
  return P2Z_OK;
}

p2z_status p2z_unpack_tracks_device(p2z_context *ctx, const p2z_config *cfg, const int64_t *d_perm,
                                    const void *d_trk_packed, void *d_trk_out, void *stream) {
  if (!ctx) {
    set_context_free_error("context is NULL");
    return P2Z_BAD_ARG;
  }
  int64_t ns = 0;
  p2z_status r = check_config(ctx, cfg, &ns);
  if (r != P2Z_OK) return r;
  if (ns == 0) return P2Z_OK;
  if (!d_perm || !d_trk_packed || !d_trk_out) return context_fail(ctx, P2Z_BAD_ARG, "NULL device buffer");
  if (d_trk_packed == d_trk_out) return context_fail(ctx, P2Z_BAD_ARG, "d_trk_out must not alias d_trk_packed");
  PACK_CUDA(ctx, cudaSetDevice(context_device(ctx)));
  cudaStream_t st = stream ? (cudaStream_t)stream : context_stream(ctx);
  const int64_t nwin = (ns + kWindow - 1) / kWindow;
  if (nwin > 0x7fffffff) return context_fail(ctx, P2Z_BAD_ARG, "too many slots");
  auto *f = cfg->bsize == 8 ? k_unpack<8> : cfg->bsize == 16 ? k_unpack<16> : cfg->bsize == 32 ? k_unpack<32>
                                                                                               : k_unpack<64>;
  // through the inverse permutation (d_perm's second half); below kUnpackPerSm windows an SM the
  // window's sort costs more than the scattered reads (one B200, us: 92,000 slots 10.7 with it, 8.8
  // without, 520,000 39.0 and 41.8, 3.2M 156 and 240)
  if (nwin < (int64_t)kUnpackPerSm * context_sms(ctx))
    k_unpack_direct<<<(unsigned)((ns + 255) / 256), 256, 0, st>>>(d_perm + ns, ns, cfg->bsize,
                                                                  (const uint32_t *)d_trk_packed, (uint32_t *)d_trk_out);
  else
    f<<<(unsigned)nwin, kWindow, 0, st>>>(d_perm + ns, ns, (const uint32_t *)d_trk_packed, (uint32_t *)d_trk_out,
                                        aligned16(d_trk_out, nullptr));
  PACK_CUDA(ctx, cudaGetLastError());
  return P2Z_OK;
}

}  // extern "C"
