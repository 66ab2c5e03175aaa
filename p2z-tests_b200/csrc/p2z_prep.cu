// p2z_prep.cu -- p2z_prepare_device: the reference's input preparation
// (srand(1), prepareTracks, prepareHits: src/propagate-toz-test_OMP.cpp:
// 127-145, :243-293) generated on the GPU into device buffers, word for word
// the output of p2z_prepare.
//
// The reference draws every smearing factor from one sequential stream: the C
// library's rand(), turned into N(0,1) variates by the polar method, two per
// accepted attempt.  That stream parallelises:
//  * rand() is an additive lagged Fibonacci generator (r[k] = r[k-31] +
//    r[k-3] mod 2^32, output r[k] >> 1; p2z_refrng.h), linear over Z/2^32 with
//    the characteristic polynomial x^31 - x^28 - 1: the word n draws ahead is
//    sum c_i r[k+i] with x^n mod that polynomial = sum c_i x^i.  A CTA takes
//    kCtaDraws draws, its warp 0's lanes kLaneDraws each; the polynomials of the
//    lanes' and of the CTAs' jumps (by powers of two) are compile-time tables.
//  * attempt j of the polar method always consumes draws 2j and 2j+1, and
//    whether it is accepted depends on those two draws only.  A first kernel
//    counts each CTA's accepted attempts; their prefix sum gives each
//    CTA's first accepted-attempt index, and accepted attempt a yields
//    variates 2a and 2a+1 (randn returns the second variate of a pair on the
//    next call).
//  * variate v is the smearing factor of one output word: the first
//    nevts*ntrks*27 are prepareTracks' (track order, then element), the rest
//    prepareHits' (layer, event, batch, lane, element).
// A second kernel generates each CTA's draws again, gathers the accepted
// attempts, turns them into variates -- all in shared memory, in the stream's
// order -- and writes the words they smear in the arrays' order, so that a warp
// writes neighbouring words.
// Bound by the instructions of the attempts and variates (k_emit issues on 69% of
// its cycles; the 80 MB of words take 12 us to write).  One B200, 10 x 9600 tracks
// x 20 layers (19.9M variates): 202 us a call, of which k_count 47, k_scan 5 and
// k_emit 136; with a thread per chunk of 1984 attempts, the chunk states and the
// prefix sum on the host and 64-bit divisions per word it took 4570.
// The arithmetic is the host's (p2z_host.cpp, p2z_refrng.h) with one
// exception: the variate's log is (float)log((double)W), correctly rounded,
// where the host calls the C library's logf, which differs by one unit in
// the last place for about 0.3% of the variates; on 200M variates that
// changed no output word (the smearing factor 1 + smear*r rounds the same),
// and the GPU tests compare the two outputs word for word.  This translation
// unit is compiled without FMA contraction, as the host side is.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>

#include "p2z.h"
#include "p2z_refrng.h"

namespace p2z {
int context_device(const p2z_context *ctx);
cudaStream_t context_stream(const p2z_context *ctx);
p2z_status context_fail(p2z_context *ctx, p2z_status st, const char *msg);
void *context_scratch(p2z_context *ctx, size_t bytes);
}  // namespace p2z

namespace {

constexpr int kLag = 31;
constexpr int kLaneDraws = 496;               // a multiple of 2
constexpr int kCtaDraws = 32 * kLaneDraws;
constexpr int kCtaAttempts = kCtaDraws / 2;   // 31 tiles of kThreads
constexpr int kThreads = 256;
constexpr int kWarps = kThreads / 32;
static_assert(kCtaAttempts % kThreads == 0, "whole tiles of attempts");
// A lane's draws in shared memory: a stride of 2 modulo 16, so that a pair of
// draws is one 8-byte access without bank conflicts and the generating warp's
// stores meet in twos.
constexpr int kLaneStride = kLaneDraws + 2;
constexpr int kBufWords = 32 * kLaneStride;

// The 31 words before draw k0: slot j holds s[j] = r[k0 - 31 + j], and
// s[n + 31] = s[n + 28] + s[n].
struct State {
  uint32_t w[kLag];
};

// x^n mod x^31 - x^28 - 1 over Z/2^32.
struct Poly {
  uint32_t c[kLag];
};
constexpr Poly poly_mul(const Poly &a, const Poly &b) {
  uint32_t t[2 * kLag - 1] = {};
  for (int i = 0; i < kLag; ++i)
    for (int j = 0; j < kLag; ++j) t[i + j] += a.c[i] * b.c[j];
  for (int d = 2 * kLag - 2; d >= kLag; --d) {  // x^d = x^(d-3) + x^(d-31)
    t[d - 3] += t[d];
    t[d - kLag] += t[d];
  }
  Poly r{};
  for (int i = 0; i < kLag; ++i) r.c[i] = t[i];
  return r;
}
constexpr int kLevels = 31;
struct Jumps {
  uint32_t lane[kLag][32];       // [i][l]: coefficient i of the jump by l * kLaneDraws
  uint32_t level[kLevels][32];   // [b][i]: of the jump by kCtaDraws * 2^b
};
constexpr Jumps make_jumps() {
  Jumps t{};
  Poly x{}, lane{}, p{};
  x.c[1] = 1u;
  p.c[0] = 1u;
  for (int n = kLaneDraws; n; n >>= 1) {
    if (n & 1) p = poly_mul(p, x);
    x = poly_mul(x, x);
  }
  lane.c[0] = 1u;
  for (int l = 0; l < 32; ++l) {
    for (int i = 0; i < kLag; ++i) t.lane[i][l] = lane.c[i];
    lane = poly_mul(lane, p);
  }
  for (int b = 0; b < kLevels; ++b) {
    for (int i = 0; i < kLag; ++i) t.level[b][i] = lane.c[i];
    lane = poly_mul(lane, lane);
  }
  return t;
}
__device__ const Jumps d_jumps = make_jumps();

struct Seeds {
  float par[6];
  float cov[21];
  int32_t q;
  float hpos[32][3];
  float hcov[32][6];
};

struct Geometry {
  int B;
  int nlayer;
  int64_t nb;           // batches per event
  int64_t ntracks;      // nevts * ntrks
  int64_t nvar_trk;     // ntracks * 27
  int64_t nvar;         // + nlayer * ntracks * 9
  double smear, cov_scale;
};

__device__ __forceinline__ bool accepted(int32_t d1, int32_t d2, float *u1, float *u2) {
  const float w = p2z_refrng::attempt(d1, d2, u1, u2);
  return !(w >= 1 || w == 0);
}

// log of a normal float in (0, 1) in double, to about 1e-16 relative (the caller
// rounds it to float): w = 2^e m with m in [1/sqrt 2, sqrt 2), and log m = 2 atanh s
// = 2 s (1 + s^2/3 + s^4/5 + ...) with s = (m - 1)/(m + 1), |s| <= 0.1716 (the
// next term, s^22/23, is below 1e-18).  The quotient by Newton's iteration: one step
// on the hardware's approximate reciprocal, then the quotient corrected by its residual.
// (With CUDA's log(double), which covers every double, k_emit took 150 us where it
// takes 136.)  Its float agrees with the rounded logarithm on 3e7 values of the range.
__device__ __forceinline__ double log01(float w) {
  uint32_t bits = __float_as_uint(w);
  const uint32_t up = (bits & 0x7fffffu) > 0x3504f3u ? 1u : 0u;  // mantissa past sqrt 2
  const int e = (int)(bits >> 23) - 127 + (int)up;
  const float m = __uint_as_float((bits & 0x7fffffu) | ((127u - up) << 23));
  const double f = (double)m - 1.0, g = (double)m + 1.0;
  float rf;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(rf) : "f"(m + 1.f));
  double r = (double)rf;
  r = fma(r, fma(-g, r, 1.0), r);
  double s = f * r;
  s = fma(r, fma(-g, s, f), s);
  const double z = s * s;
  double p = 2.0 / 21.0;
  p = fma(p, z, 2.0 / 19.0);
  p = fma(p, z, 2.0 / 17.0);
  p = fma(p, z, 2.0 / 15.0);
  p = fma(p, z, 2.0 / 13.0);
  p = fma(p, z, 2.0 / 11.0);
  p = fma(p, z, 2.0 / 9.0);
  p = fma(p, z, 2.0 / 7.0);
  p = fma(p, z, 2.0 / 5.0);
  p = fma(p, z, 2.0 / 3.0);
  return fma((double)e, 0.6931471805599453, fma(s * z, p, 2.0 * s));
}

// A word of the sequence is needed 31 to 61 places on: s[31..60] from s[0..30]
// (one warp; three new words are independent of one another).
__device__ __forceinline__ void extend(uint32_t *s) {
  const int lane = threadIdx.x & 31;
  __syncwarp();
  for (int m = 0; m < 30; m += 3) {
    if (lane < 3) s[kLag + m + lane] = s[kLag - 3 + m + lane] + s[m + lane];
    __syncwarp();
  }
}

// The CTA's kCtaDraws draws into buf (lane l's from l * kLaneStride on), from
// the state before its first one.
__device__ __forceinline__ void generate(const State *base, uint32_t *buf) {
  __shared__ uint32_t seq[64];
  __shared__ uint32_t start[kLag][32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (warp == 0) {
    if (lane < kLag) seq[lane] = base->w[lane];
    extend(seq);
  }
  __syncthreads();
  // word j of lane l's state: all warps, j = warp, warp + 8, ...
  uint32_t acc[4] = {0u, 0u, 0u, 0u};
  for (int i = 0; i < kLag; ++i) {
    const uint32_t c = d_jumps.lane[i][lane];
#pragma unroll
    for (int q = 0; q < 4; ++q) acc[q] += c * seq[min(i + warp + kWarps * q, 60)];
  }
#pragma unroll
  for (int q = 0; q < 4; ++q)
    if (warp + kWarps * q < kLag) start[warp + kWarps * q][lane] = acc[q];
  __syncthreads();
  if (warp == 0) {
    uint32_t s[kLag];
#pragma unroll
    for (int j = 0; j < kLag; ++j) s[j] = start[j][lane];
    uint32_t *out = buf + lane * kLaneStride;
    for (int blk = 0; blk < kLaneDraws / kLag; ++blk) {
#pragma unroll
      for (int j = 0; j < kLag; ++j) {
        s[j] += s[(j + 28) % kLag];
        out[blk * kLag + j] = s[j] >> 1;
      }
    }
  }
  __syncthreads();
}
static_assert(kLaneDraws % kLag == 0, "whole blocks of 31 draws");

constexpr int kLaneAttempts = kLaneDraws / 2;

// Per CTA: its state (kept for k_emit) and its accepted attempts.
__global__ void __launch_bounds__(kThreads) k_count(State first, State *states, uint32_t *counts) {
  extern __shared__ __align__(16) uint32_t buf[];
  __shared__ uint32_t seq[64];
  __shared__ uint32_t sums[kWarps];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (warp == 0) {
    if (lane < kLag) seq[lane] = first.w[lane];
    __syncwarp();
    for (unsigned c = blockIdx.x, b = 0; c; c >>= 1, ++b) {
      if (!(c & 1u)) continue;
      extend(seq);
      uint32_t acc = 0u;
      if (lane < kLag)
        for (int i = 0; i < kLag; ++i) acc += d_jumps.level[b][i] * seq[i + lane];
      __syncwarp();
      if (lane < kLag) seq[lane] = acc;
      __syncwarp();
    }
    if (lane < kLag) states[blockIdx.x].w[lane] = seq[lane];
  }
  __syncthreads();  // (a block sees its own global writes after the barrier)
  generate(states + blockIdx.x, buf);
  uint32_t n = 0;
  for (int a = warp; a < kLaneAttempts; a += kWarps) {  // (in any order)
    const uint2 d = *reinterpret_cast<const uint2 *>(buf + lane * kLaneStride + 2 * a);
    float u1, u2;
    n += accepted((int32_t)d.x, (int32_t)d.y, &u1, &u2) ? 1u : 0u;
  }
  n = __reduce_add_sync(0xffffffffu, n);
  if (lane == 0) sums[warp] = n;
  __syncthreads();
  if (threadIdx.x == 0) {
    uint32_t t = 0;
    for (int w = 0; w < kWarps; ++w) t += sums[w];
    counts[blockIdx.x] = t;
  }
}

// Exclusive prefix sum of n counts, and their total in first[n]: one block, a
// run of counts a thread.
__global__ void __launch_bounds__(1024) k_scan(const uint32_t *counts, int n, uint64_t *first) {
  __shared__ uint64_t sums[32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int per = (n + 1023) / 1024, c0 = min(n, (int)threadIdx.x * per), c1 = min(n, c0 + per);
  uint64_t t = 0;
  for (int c = c0; c < c1; ++c) t += counts[c];
  uint64_t sum = t;
  for (int o = 1; o < 32; o <<= 1) {
    const uint64_t u = __shfl_up_sync(0xffffffffu, sum, o);
    if (lane >= o) sum += u;
  }
  if (lane == 31) sums[warp] = sum;
  __syncthreads();
  uint64_t at = sum - t;
  for (int w = 0; w < warp; ++w) at += sums[w];
  for (int c = c0; c < c1; ++c) {
    first[c] = at;
    at += counts[c];
  }
  if (threadIdx.x == 1023) first[n] = at;
}

// Writes the words of the variates r[0, n): element ip of track t0 + i is
// smeared by r[27 i + ip + off] (9 for hits), where that lies in [0, n); `out` is
// the first batch's array, batches of B tracks `bw` words apart.  A warp takes an
// element and an eighth of the tracks: neighbouring lanes write neighbouring
// words and read r at an odd stride, and all but the element's seed is 32-bit
// arithmetic.  q: the charge word of every track whose first element is here.
template <int E, class Seed, class Scale>
__device__ __forceinline__ void write_rows(const float *r, int off, int n, float *out, int64_t bw, int B, int64_t t0,
                                              double smear, Seed seed, Scale scale, const int32_t *q) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, shift = __ffs(B) - 1;
  const int span = (n - off + E - 1) / E, part = (span + 7) / 8;
  float *base = out + (t0 >> shift) * bw;
  const int lane0 = (int)(t0 & (B - 1));
  for (int u = warp; u < 8 * E; u += kWarps) {
    const int ip = u % E, i0 = u / E * part, i1 = min(span, i0 + part);
    const double x = seed(ip), c = scale(ip);
    for (int i = i0 + lane; i < i1; i += 32) {
      const int at = E * i + ip + off;
      if (at < 0 || at >= n) continue;
      const double sf = fma(smear, (double)r[at], 1.0);  // the reference's (1 + smear*randn), one rounding
      const int t = lane0 + i;
      float *w = base + (int64_t)(t >> shift) * bw + (t & (B - 1));
      w[ip * B] = (float)(sf * x * c);
      if (q && ip == 0) reinterpret_cast<int32_t *>(w)[27 * B] = *q;
    }
  }
}

__global__ void __launch_bounds__(kThreads) k_emit(const State *states, const uint64_t *first, Geometry g,
                                                   const __grid_constant__ Seeds sd, float *trk, float *hits) {
  extern __shared__ __align__(16) uint32_t buf[];
  __shared__ uint32_t votes[2][kWarps];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t v0 = 2 * (int64_t)first[blockIdx.x];
  if (v0 >= g.nvar) return;
  generate(states + blockIdx.x, buf);
  // the accepted attempts' (u1, u2) to the front of buf, in order: attempt a's
  // draws lie at 2a or later, so a tile's pairs never reach the next tile's draws
  int n = 0;
  int in_lane = threadIdx.x, at = 2 * threadIdx.x;  // of attempt threadIdx.x + kThreads * tile
  if (in_lane >= kLaneAttempts) {
    in_lane -= kLaneAttempts;
    at += kLaneStride - kLaneDraws;
  }
  for (int k = 0, tile = 0; k < kCtaAttempts / kThreads; ++k, tile ^= 1) {
    const uint2 d = *reinterpret_cast<const uint2 *>(buf + at);
    in_lane += kThreads - kLaneAttempts;
    at += 2 * kThreads + kLaneStride - kLaneDraws;
    if (in_lane >= kLaneAttempts) {
      in_lane -= kLaneAttempts;
      at += kLaneStride - kLaneDraws;
    }
    float u1, u2;
    const bool ok = accepted((int32_t)d.x, (int32_t)d.y, &u1, &u2);
    const unsigned vote = __ballot_sync(0xffffffffu, ok);
    if (lane == 0) votes[tile][warp] = __popc(vote);
    __syncthreads();
    int below = 0, all = 0;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) {
      const int c = (int)votes[tile][w];
      below += w < warp ? c : 0;
      all += c;
    }
    if (ok) {
      const int to = n + below + __popc(vote & ((1u << lane) - 1u));
      reinterpret_cast<float2 *>(buf)[to] = make_float2(u1, u2);
    }
    n += all;
  }
  __syncthreads();
  // their variates, in place
  float *r = reinterpret_cast<float *>(buf);
  for (int a = threadIdx.x; a < n; a += kThreads) {
    const float2 u = reinterpret_cast<const float2 *>(r)[a];
    const float w = (float)((double)u.x * (double)u.x + (double)u.y * (double)u.y);
    const float lg = (float)log01(w);
    const float mult = sqrtf((-2 * lg) / w);
    reinterpret_cast<float2 *>(r)[a] = make_float2(0.f + 1.f * (u.x * mult), 0.f + 1.f * (u.y * mult));
  }
  __syncthreads();
  // the words they smear
  const int64_t v1 = min(v0 + 2 * (int64_t)n, g.nvar);
  const int B = g.B;
  if (v0 < g.nvar_trk) {
    const int64_t t0 = v0 / 27;
    write_rows<27>(r, (int)(t0 * 27 - v0), (int)(min(v1, g.nvar_trk) - v0), trk, (int64_t)28 * B, B, t0, g.smear,
                   [&](int ip) { return ip < 6 ? (double)sd.par[ip] : (double)sd.cov[ip - 6]; },
                   [&](int ip) { return ip < 6 ? 1.0 : g.cov_scale; }, &sd.q);
  }
  // (hits: one layer's tracks after the other's; few ranges meet more than one)
  for (int64_t v = max(v0, g.nvar_trk); v < v1;) {
    const int64_t h0 = (v - g.nvar_trk) / 9;
    const int lay = (int)(h0 / g.ntracks);
    const int64_t end = min(v1, g.nvar_trk + (int64_t)(lay + 1) * g.ntracks * 9);  // of this layer's variates
    write_rows<9>(r + (v - v0), (int)(h0 * 9 + g.nvar_trk - v), (int)(end - v), hits + (int64_t)lay * 9 * B,
                  (int64_t)g.nlayer * 9 * B, B, h0 - (int64_t)lay * g.ntracks, g.smear,
                  [&](int ip) { return ip < 3 ? (double)sd.hpos[lay][ip] : (double)sd.hcov[lay][ip - 3]; },
                  [&](int) { return 1.0; }, nullptr);
    v = end;
  }
}

#define PP_CUDA(call)                                                            \
  do {                                                                           \
    cudaError_t e_ = (call);                                                     \
    if (e_ != cudaSuccess) {                                                     \
      char m_[256];                                                              \
      std::snprintf(m_, sizeof m_, "%s: %s", #call, cudaGetErrorString(e_));     \
      return p2z::context_fail(ctx, P2Z_CUDA_ERROR, m_);                         \
    }                                                                            \
  } while (0)

}  // namespace

extern "C" p2z_status p2z_prepare_device(p2z_context *ctx, const p2z_atrk *seed, const p2z_ahit *hit_seeds,
                                         int nseeds, int bsize, int64_t nevts, int64_t ntrks, int nlayer,
                                         double smear, double cov_scale, void *d_trk_out, void *d_hits_out,
                                         void *stream) {
  if (!ctx) return P2Z_BAD_ARG;
  if (!seed || !hit_seeds) return p2z::context_fail(ctx, P2Z_BAD_ARG, "NULL seed");
  if (!(bsize == 8 || bsize == 16 || bsize == 32 || bsize == 64))
    return p2z::context_fail(ctx, P2Z_UNSUPPORTED, "bsize not in {8,16,32,64}");
  if (nevts < 0 || ntrks < 0 || ntrks % bsize || nlayer < 1 || nlayer > 32)
    return p2z::context_fail(ctx, P2Z_BAD_ARG, "bad sizes");
  if (nseeds < nlayer) return p2z::context_fail(ctx, P2Z_BAD_ARG, "fewer hit seeds than layers");
  Geometry g;
  g.B = bsize;
  g.nlayer = nlayer;
  g.nb = ntrks / bsize;
  g.ntracks = nevts * ntrks;
  g.nvar_trk = g.ntracks * 27;
  g.nvar = g.nvar_trk + (int64_t)nlayer * g.ntracks * 9;
  g.smear = smear;
  g.cov_scale = cov_scale;
  if (g.ntracks == 0) return P2Z_OK;
  if (!d_trk_out || !d_hits_out) return p2z::context_fail(ctx, P2Z_BAD_ARG, "NULL device buffer");
  PP_CUDA(cudaSetDevice(p2z::context_device(ctx)));
  cudaStream_t st = stream ? (cudaStream_t)stream : p2z::context_stream(ctx);

  Seeds sd;
  std::memcpy(sd.par, seed->par, sizeof sd.par);
  std::memcpy(sd.cov, seed->cov, sizeof sd.cov);
  sd.q = seed->q;
  for (int l = 0; l < nlayer; ++l) {
    std::memcpy(sd.hpos[l], hit_seeds[l].pos, sizeof sd.hpos[l]);
    std::memcpy(sd.hcov[l], hit_seeds[l].cov, sizeof sd.hcov[l]);
  }
  // Accepted attempts needed: nvar/2 rounded up; attempts are accepted with
  // probability pi/4.  CTAs for that many attempts plus 6 standard
  // deviations; more are added if the count falls short.
  const uint64_t need = (uint64_t)((g.nvar + 1) / 2);
  const double att = (double)need / 0.7853981633974483;
  int64_t nctas = (int64_t)std::ceil((att + 6.0 * std::sqrt(att) + 1.0) / kCtaAttempts);
  State s0;
  {
    p2z_ref_rng r;
    p2z_refrng::seed(&r, 1u);  // srand(1): the reference's initial state
    for (int j = 0; j < kLag; ++j) s0.w[j] = r.ring[(r.next - kLag + j) % kLag];
  }
  constexpr int kSmem = kBufWords * 4;
  PP_CUDA(cudaFuncSetAttribute(k_count, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem));
  PP_CUDA(cudaFuncSetAttribute(k_emit, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem));
  for (int pass = 0; pass < 4; ++pass) {
    if (nctas > 0x7fffffff) return p2z::context_fail(ctx, P2Z_BAD_ARG, "too many tracks and layers for one call");
    // scratch: the CTAs' states, counts and first indices, each part starting on
    // a 256-byte boundary (sizeof(State) is 124, so the parts' sizes are rounded up)
    auto up256 = [](size_t n) { return (n + 255) / 256 * 256; };
    const size_t sbytes = up256(sizeof(State) * (size_t)nctas), cbytes = up256(sizeof(uint32_t) * (size_t)nctas);
    char *scr = static_cast<char *>(
        p2z::context_scratch(ctx, sbytes + cbytes + up256(sizeof(uint64_t) * ((size_t)nctas + 1))));
    if (!scr) return P2Z_OOM;
    State *d_states = reinterpret_cast<State *>(scr);
    uint32_t *d_counts = reinterpret_cast<uint32_t *>(scr + sbytes);
    uint64_t *d_first = reinterpret_cast<uint64_t *>(scr + sbytes + cbytes);
    k_count<<<(unsigned)nctas, kThreads, kSmem, st>>>(s0, d_states, d_counts);
    PP_CUDA(cudaGetLastError());
    k_scan<<<1, 1024, 0, st>>>(d_counts, (int)nctas, d_first);
    PP_CUDA(cudaGetLastError());
    k_emit<<<(unsigned)nctas, kThreads, kSmem, st>>>(d_states, d_first, g, sd, (float *)d_trk_out,
                                                     (float *)d_hits_out);
    PP_CUDA(cudaGetLastError());
    uint64_t total = 0;
    PP_CUDA(cudaMemcpyAsync(&total, d_first + nctas, sizeof total, cudaMemcpyDeviceToHost, st));
    PP_CUDA(cudaStreamSynchronize(st));
    if (total >= need) return P2Z_OK;
    nctas += nctas / 16 + 1;  // rare: the words past the stream's end are missing; take more of it
  }
  return p2z::context_fail(ctx, P2Z_CUDA_ERROR, "the random stream fell short of the variates needed");
}
