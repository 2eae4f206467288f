// Kernel 3 of the chain: search_by_triplet, one warp per event, or a block of four for the
// largest of a batch (persistent, queues), events handed out largest first
// (order_events_kernel, velo_order.cuh).
//
// The module loop, forwarding and weak-track rules are those of the reference
// (ProcessModules.cu:8-163, TrackForwarding.cu:41-181, TrackSeeding.cu:7-200,
// WeakTracksAdder.cu:88-115). What changes is the mapping onto the warp:
//   * seeding: the phi windows of every h1 come precomputed from fill_candidates (in the
//     pruned mode the scorer has cleared the windows of pruned seeds, and forwarding skips
//     candidates without the extension-keep bit when that pruning is on);
//     the h1 candidates of a step are compacted into a shared list and searched in three
//     passes (seed_flush below): their (h1, h0) pairs flattened over the lanes, which keeps the
//     pairs inside the slope cut; a lane per kept pair, which marks the h2 of its window near the
//     straight line; and the marked triplets over the lanes, which get the reference's test.
//     Each h1 keeps its best triplet in a shared 64-bit key (scatter bits, h0 offset, h2
//     offset): the winner is the minimal scatter, first in (h0, h2) order, and exact ties
//     (which the reference resolves by thread scheduling) are flagged;
//   * hit_used is a bitmask in shared memory; appends to the ring buffers go in lane order
//     through ballots, so the result does not depend on scheduling.
#pragma once
#include "velo_kernels.cuh"

namespace velo {

// h1 candidates per seeding pass (multiple of 32). The per-warp shared state is small so
// that L1, which shares the SM's 256 KB with shared memory, keeps more of the events' hit
// records: 64 measured faster than 128 (4.46 vs 4.60 ms per 16,384 events).
constexpr uint32_t kSeedChunk = 64;

__device__ __forceinline__ bool test_used(const uint32_t* used, uint32_t h) { return (used[h >> 5] >> (h & 31)) & 1u; }
__device__ __forceinline__ void set_used(uint32_t* used, uint32_t h) { atomicOr(used + (h >> 5), 1u << (h & 31)); }

__device__ __forceinline__ uint32_t ballot_rank(bool pred, uint32_t& total)
{
  const uint32_t b = __ballot_sync(0xFFFFFFFFu, pred);
  total = __popc(b);
  return __popc(b & ((1u << lane_id()) - 1u));
}

// Slope cut of the doublet (h0, h1) (TrackSeeding.cu:137-152).
__device__ __forceinline__ bool seed_slope(const float4 h0, const float4 h1)
{
  const float dmax = kMaxSlope * (h0.z - h1.z);
  return fabsf(h1.x - h0.x) < dmax && fabsf(h1.y - h0.y) < dmax;
}

// Scatter of the triplet (h0, h1, h2) and whether it passes the seeding cuts beyond the
// doublet's slope (TrackSeeding.cu:137-152).
__device__ __forceinline__ bool seed_triplet(const float4 h0, const float4 h1, const float4 h2, float& scatter)
{
  const float scatterDenom2 = 1.f / ((h2.z - h1.z) * (h2.z - h1.z));
  const float z2_tz = (h2.z - h0.z) / (h1.z - h0.z);
  const float x = h0.x + (h1.x - h0.x) * z2_tz;
  const float y = h0.y + (h1.y - h0.y) * z2_tz;
  const float dx = x - h2.x;
  const float dy = y - h2.y;
  const float scatterNum = (dx * dx) + (dy * dy);
  scatter = scatterNum * scatterDenom2;
  return fabsf(dx) < kTolerance && fabsf(dy) < kTolerance && scatter < kMaxScatterSeeding;
}

// Forwarding fit of one candidate (TrackForwarding.cu:12-35).
__device__ __forceinline__ float forward_fit(float h0x, float h0y, float h2x, float h2y, float predx, float predy,
                                             float scatterDenom2)
{
  const float x_prediction = h0x + predx;
  const float dx = fabsf(x_prediction - h2x);
  const bool tolx_condition = dx < kTolerance;
  const float y_prediction = h0y + predy;
  const float dy = fabsf(y_prediction - h2y);
  const bool toly_condition = dy < kTolerance;
  const float scatterNum = (dx * dx) + (dy * dy);
  const float scatter = scatterNum * scatterDenom2;
  const bool scatter_condition = scatter < kMaxScatterForwarding;
  const bool condition = tolx_condition && toly_condition && scatter_condition;
  return condition * scatter + !condition * 3.402823466e+38f;
}

// phi window of a forwarded track in one module (TrackForwarding.cuh:28-59).
__device__ __forceinline__ void forward_window(const float4* H, uint32_t mstart, uint32_t mnum, float mz, float tx,
                                               float ty, float h0x, float h0y, float h0z, bool odd, int& first,
                                               int& last, uint32_t& flags)
{
  const float dz = mz - h0z;
  const float predx = tx * dz;
  const float predy = ty * dz;
  const float x_prediction = h0x + predx;
  const float y_prediction = h0y + predy;
  const float phi = odd ? phi_odd_side(x_prediction, y_prediction) : phi_even_side(x_prediction, y_prediction);
  first = -1;
  last = -1;
  if (mnum == 0) {
    // The reference binary-searches an empty range here and reads the element at the
    // module start, outside the module; this implementation takes no candidates.
    flags |= kStatusEmptyModuleRead;
    return;
  }
  phi_window4(H, mstart, mnum, phi, kForwardPhiTolerance, first, last);
}

// 3-hit straight-line chi2 of weak_tracks_adder (WeakTracksAdder.cu:9-86).
__device__ __forceinline__ float weak_chi2(const float4* H, const uint16_t* h)
{
  float s0, sx, sz, sxz, sz2;
  float u0, uy, uz, uyz, uz2;
  s0 = sx = sz = sxz = sz2 = 0.0f;
  u0 = uy = uz = uyz = uz2 = 0.0f;
  float4 p[3];
  for (int k = 0; k < 3; ++k) {
    p[k] = H[h[k]];
    const float x = p[k].x, y = p[k].y, z = p[k].z;
    const float wx = kParamW;
    const float wx_t_x = wx * x;
    const float wx_t_z = wx * z;
    s0 += wx;
    sx += wx_t_x;
    sz += wx_t_z;
    sxz += wx_t_x * z;
    sz2 += wx_t_z * z;
    const float wy = kParamW;
    const float wy_t_y = wy * y;
    const float wy_t_z = wy * z;
    u0 += wy;
    uy += wy_t_y;
    uz += wy_t_z;
    uyz += wy_t_y * z;
    uz2 += wy_t_z * z;
  }
  float tx, x0, ty, y0;
  {
    const float dens = 1.0f / (sz2 * s0 - sz * sz);
    tx = (sxz * s0 - sx * sz) * dens;
    x0 = (sx * sz2 - sxz * sz) * dens;
    const float denu = 1.0f / (uz2 * u0 - uz * uz);
    ty = (uyz * u0 - uy * uz) * denu;
    y0 = (uy * uz2 - uyz * uz) * denu;
  }
  float ch = 0.0f;
  int nDoF = -4;
  for (int k = 0; k < 3; ++k) {
    const float z = p[k].z;
    const float x = x0 + tx * z;
    const float y = y0 + ty * z;
    const float dx = x - p[k].x;
    const float dy = y - p[k].y;
    ch += dx * dx * kParamW + dy * dy * kParamW;
    nDoF += 2;
  }
  return ch / nDoF;
}

constexpr uint32_t kPairQueue = 64;  // doublets waiting for a full round of 32

struct SeedSlots {
  uint16_t h1[kSeedChunk];
  uint16_t f0[kSeedChunk];
  uint16_t f2[kSeedChunk];
  uint16_t n2[kSeedChunk];
  uint32_t pair_start[kSeedChunk];    // number of h0 of each candidate, then its exclusive scan
  unsigned long long best[kSeedChunk];  // scatter bits << 32 | h0 offset << 16 | h2 offset
  uint32_t tie[kSeedChunk];           // smallest scatter that two triplets share
  uint32_t pair[kPairQueue];          // candidate << 16 | h0 offset in its window
  uint32_t triplet[32];               // lane of its pair << 16 | h2 offset
};

// Exclusive scan of v[0 .. n) in place by one warp; returns the total.
__device__ __forceinline__ uint32_t warp_scan_in_place(uint32_t* v, uint32_t n)
{
  const uint32_t lane = lane_id();
  uint32_t total = 0;
  for (uint32_t k0 = 0; k0 < n; k0 += 32) {
    const uint32_t k = k0 + lane;
    const uint32_t x = k < n ? v[k] : 0;
    uint32_t incl = x;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t t = __shfl_up_sync(0xFFFFFFFFu, incl, o);
      if (lane >= static_cast<uint32_t>(o)) incl += t;
    }
    if (k < n) v[k] = total + incl - x;
    total += __shfl_sync(0xFFFFFFFFu, incl, 31);
  }
  __syncwarp();
  return total;
}

// Segment of position p0 + lane, for p0 = 0, 32, 64, ... in turn: start[0 .. n) are the
// segments' first positions (no segment is empty), `lo` the segment of position p0 - 1 (0 at
// first; advanced here). The segments starting inside the 32 positions are lo + 1 .. lo + 32,
// so one shared load, an OR across the warp and a popcount replace a binary search.
__device__ __forceinline__ uint32_t warp_segment(const uint32_t* start, uint32_t n, uint32_t p0, uint32_t& lo)
{
  const uint32_t lane = lane_id();
  uint32_t head = 0;
  if (lo + 1 + lane < n) {
    const uint32_t s = start[lo + 1 + lane] - p0;
    if (s < 32u) head = 1u << s;
  }
  const uint32_t heads = __reduce_or_sync(0xFFFFFFFFu, head);
  const uint32_t k = lo + __popc(heads & (0xFFFFFFFFu >> (31 - lane)));
  lo = __shfl_sync(0xFFFFFFFFu, k, 31);
  return k;
}

// The triplets of the first n (<= 32) queued pairs, by one warp: a lane per pair marks the h2
// of its window near the straight line through h0 and h1, and the marked ones, packed over the
// lanes, get the reference's test (TrackSeeding.cu:137-175) and compete for their candidate's
// key.
//
// The marking is a superset of the reference's cut: its prediction and the reference's differ
// by the rounding of a quotient, a product and a sum, at most 7.2e-7 (|x| + |x0|); the box is
// widened by 1e-5 of both and by 1e-4 mm (a NaN marks). So the loop over a window, whose length
// the longest window of the 32 pairs sets, holds no division and no branch.
__device__ __forceinline__ void seed_round(SeedSlots& sl, uint32_t n, const float4* H, const uint32_t* used)
{
  const uint32_t lane = lane_id();
  uint32_t n2 = 0, f2 = 0;
  float x0 = 0.f, y0 = 0.f, z0 = 0.f, tx = 0.f, ty = 0.f, tol0 = 0.f;
  if (lane < n) {
    const uint32_t pk = sl.pair[lane], k = pk >> 16;
    const float4 h0 = H[sl.f0[k] + (pk & 0xFFFFu)];
    const float4 h1 = H[sl.h1[k]];
    f2 = sl.f2[k];
    n2 = sl.n2[k];
    x0 = h0.x;
    y0 = h0.y;
    z0 = h0.z;
    const float inv = __fdividef(1.f, h1.z - h0.z);
    tx = (h1.x - h0.x) * inv;
    ty = (h1.y - h0.y) * inv;
    tol0 = kTolerance + 1e-4f + 1e-5f * fmaxf(fabsf(x0), fabsf(y0));
  }
  const uint32_t longest = __reduce_max_sync(0xFFFFFFFFu, n2);
  for (uint32_t c0 = 0; c0 < longest; c0 += 32) {
    uint32_t marks = 0;
    const uint32_t m = n2 > c0 ? min(n2 - c0, 32u) : 0u;
    const float4* W = H + f2 + c0;
#pragma unroll 2
    for (uint32_t j = 0; j < m; ++j) {
      const float4 h2 = W[j];
      const float dz = h2.z - z0;
      const float x = x0 + tx * dz;
      const float y = y0 + ty * dz;
      const float d = fmaxf(fabsf(x - h2.x), fabsf(y - h2.y));
      const float tol = tol0 + 1e-5f * fmaxf(fabsf(x), fabsf(y));
      if (!(d >= tol)) marks |= 1u << j;
    }
    const uint32_t cnt = __popc(marks);
    uint32_t incl = cnt;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t t = __shfl_up_sync(0xFFFFFFFFu, incl, o);
      if (lane >= static_cast<uint32_t>(o)) incl += t;
    }
    const uint32_t total = __shfl_sync(0xFFFFFFFFu, incl, 31);
    uint32_t pos = incl - cnt;
    for (uint32_t w0 = 0; w0 < total; w0 += 32) {
      while (marks && pos < w0 + 32) {
        sl.triplet[pos - w0] = (lane << 16) | (c0 + __ffs(marks) - 1);
        marks &= marks - 1;
        ++pos;
      }
      __syncwarp();
      if (w0 + lane < total) {
        const uint32_t t = sl.triplet[lane], pk = sl.pair[t >> 16], k = pk >> 16;
        const uint32_t h2rel = t & 0xFFFFu, h2i = sl.f2[k] + h2rel;
        if (!test_used(used, h2i)) {
          float scatter;
          if (seed_triplet(H[sl.f0[k] + (pk & 0xFFFFu)], H[sl.h1[k]], H[h2i], scatter)) {
            const uint32_t sb = __float_as_uint(scatter);
            const unsigned long long key = (static_cast<unsigned long long>(sb) << 32) | (pk << 16) | h2rel;
            // once the smallest scatter has come, every equal one meets it here
            const unsigned long long old = atomicMin(&sl.best[k], key);
            if (static_cast<uint32_t>(old >> 32) == sb) atomicMin(&sl.tie[k], sb);
          }
        }
      }
      __syncwarp();
    }
  }
}

// Seeding of the nc candidates queued in `sl` by one warp (TrackSeeding.cu:90-183): leaves
// each candidate's best triplet in sl.best.
//
// Bound by instruction issue and by the latency of the hit records. A lane per (h1, h0) pair
// that tested every h2 of its window kept 17.8 lanes busy (the longest window of 32 pairs sets
// the loop) at about 35 instructions a step; here the pairs outside the slope cut (42% of the
// triplets) leave first and the step of the window loop is 15 instructions. Search of 65,536
// events at nu ~ U(2,20) 15.16 -> 13.80 ms (1.41 -> 1.23 G warp instructions per 8,192 events),
// of 3,000 events at nu = 15 with noise 8.31 -> 6.04 ms. Flattening the triplets too kept 24
// lanes busy and was slower (15.5 and 9.2 ms): locating a triplet costs more than its test.
__device__ __forceinline__ void seed_flush(SeedSlots& sl, uint32_t nc, const float4* H, const uint32_t* used)
{
  const uint32_t lane = lane_id();
  __syncwarp();
  const uint32_t total_pairs = warp_scan_in_place(sl.pair_start, nc);
  uint32_t n_queued = 0;
  uint32_t k_lo = 0;  // candidate of the last pair seen
  for (uint32_t p0 = 0; p0 < total_pairs; p0 += 32) {
    const uint32_t p = p0 + lane;
    const uint32_t k = warp_segment(sl.pair_start, nc, p0, k_lo);
    bool pair = false;
    uint32_t h0rel = 0;
    if (p < total_pairs) {
      h0rel = p - sl.pair_start[k];
      const uint32_t h0i = sl.f0[k] + h0rel;
      if (!test_used(used, h0i)) pair = seed_slope(H[h0i], H[sl.h1[k]]);
    }
    uint32_t n_new;
    const uint32_t rank = ballot_rank(pair, n_new);
    if (pair) sl.pair[n_queued + rank] = (k << 16) | h0rel;
    n_queued += n_new;
    const bool last = p0 + 32 >= total_pairs;
    while (n_queued >= 32 || (last && n_queued > 0)) {
      __syncwarp();
      const uint32_t n = min(n_queued, 32u);
      seed_round(sl, n, H, used);
      // the pairs beyond the round move to the front
      n_queued -= n;
      uint32_t v = 0;
      if (lane < n_queued) v = sl.pair[32 + lane];
      __syncwarp();
      if (lane < n_queued) sl.pair[lane] = v;
    }
  }
  __syncwarp();
}

// Eight warps an event are for a batch too small to fill the device (kSmallBatch): the steps are
// chains of dependent loads with most warps waiting at the barriers, so what a step will read is
// fetched during the one before. In a full device the extra loads (the windows of used h1, the
// copies' instructions) cost more than they hide: four warps an event with it took 1.90 ms for
// 3,000 noisy events, 1.73 without.
template<int G>
constexpr bool kFetchAhead = G >= 8;

// The phi of the two modules that forwarding searches, one after the other in shared memory: in
// a staging area that reuses the seeding slots (the two phases never overlap), so that L1 keeps
// its share of the SM, or in one of its own where it is filled during the seeding.
template<int G, bool kAhead = kFetchAhead<G>>
union SeedArea {
  static constexpr uint32_t kFwdStage = G * sizeof(SeedSlots) / sizeof(float);
  SeedSlots seed[G];  // one per warp
  float fphi[kFwdStage];
};
template<int G>
union SeedArea<G, true> {
  static constexpr uint32_t kFwdStage = 2048;
  struct {
    SeedSlots seed[G];
    float fphi[kFwdStage];
  };
};

// Shared state of one event of at most kHits hits searched by G warps.
template<int G, uint32_t kHits = kEventHitCap>
struct SearchShared {
  static constexpr int kWarps = G;
  static constexpr uint32_t kFwdStage = SeedArea<G>::kFwdStage;
  SeedArea<G> u;
  uint32_t used[kHits / 32];
  uint16_t mstart[kModules];
  uint16_t mnum[kModules];
  uint32_t count[2][G];  // counts of the warps (group_rank), two in turn
  uint32_t sum;          // OR of the flags and sum of the track hits at the end
  uint32_t flags;
};

// The G warps that search one event: one warp, or the G warps of a block.
template<int G>
__device__ __forceinline__ uint32_t group_thread()
{
  return G == 1 ? lane_id() : threadIdx.x;
}
// Asynchronous copy of one float from global to shared memory; a thread's copies are complete
// after async_wait.
__device__ __forceinline__ void async_copy4(float* dst, const float* src)
{
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(static_cast<uint32_t>(__cvta_generic_to_shared(dst))),
               "l"(src)
               : "memory");
}
__device__ __forceinline__ void async_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

template<int G>
__device__ __forceinline__ void group_sync()
{
  if (G == 1) __syncwarp();
  else __syncthreads();
}

// Exclusive rank of each thread over the group for three predicates (each count <= 32 G fits 10
// bits), and the totals. `turn` alternates between two count buffers, so one barrier a call
// suffices: a buffer is written again only after the barrier of the call between.
template<class Shared>
__device__ __forceinline__ void group_rank(Shared& sh, uint32_t& turn, bool p0, bool p1, bool p2,
                                           uint32_t (&rank)[3], uint32_t (&total)[3])
{
  constexpr int G = Shared::kWarps;
  const uint32_t lt = (1u << lane_id()) - 1u;
  const uint32_t b0 = __ballot_sync(0xFFFFFFFFu, p0), b1 = __ballot_sync(0xFFFFFFFFu, p1),
                 b2 = __ballot_sync(0xFFFFFFFFu, p2);
  uint32_t before = 0, all = __popc(b0) | (__popc(b1) << 10) | (__popc(b2) << 20);
  if constexpr (G > 1) {
    static_assert(32 * G < 1024, "counts of 10 bits");
    const uint32_t warp = threadIdx.x >> 5;
    if (lane_id() == 0) sh.count[turn][warp] = all;
    __syncthreads();
    all = 0;
#pragma unroll
    for (uint32_t w = 0; w < G; ++w) {
      const uint32_t v = sh.count[turn][w];
      before += w < warp ? v : 0u;
      all += v;
    }
    turn ^= 1u;
  }
  rank[0] = (before & 0x3FFu) + __popc(b0 & lt);
  rank[1] = ((before >> 10) & 0x3FFu) + __popc(b1 & lt);
  rank[2] = (before >> 20) + __popc(b2 & lt);
  total[0] = all & 0x3FFu;
  total[1] = (all >> 10) & 0x3FFu;
  total[2] = all >> 20;
}

// phi window of a forwarded track in one module (TrackForwarding.cuh:28-59), with the
// module's phi staged in shared memory (`sphi`, null when the module did not fit): the
// same probes on the same values as phi_window4 over the cluster records.
__device__ __forceinline__ void forward_window_staged(const float4* H, const float* sphi, uint32_t mstart,
                                                      uint32_t mnum, float mz, float tx, float ty, float h0x,
                                                      float h0y, float h0z, bool odd, int& first, int& last,
                                                      uint32_t& flags)
{
  if (!sphi) {
    forward_window(H, mstart, mnum, mz, tx, ty, h0x, h0y, h0z, odd, first, last, flags);
    return;
  }
  const float dz = mz - h0z;
  const float predx = tx * dz;
  const float predy = ty * dz;
  const float x_prediction = h0x + predx;
  const float y_prediction = h0y + predy;
  const float phi = odd ? phi_odd_side(x_prediction, y_prediction) : phi_even_side(x_prediction, y_prediction);
  first = -1;
  last = -1;
  if (mnum == 0) {
    flags |= kStatusEmptyModuleRead;
    return;
  }
  phi_window_flat(sphi, mnum, phi, kForwardPhiTolerance, first, last);
  if (first != -1) {
    first += static_cast<int>(mstart);
    last += static_cast<int>(mstart);
  }
}

// Best forwarding fit of one track (direction tx, ty of its last hits h0 -> h1) over the n
// candidates of its two windows, first in order on equal fits (TrackForwarding.cu:41-110):
// candidate j is hit odd + j below n_odd and even + j from there on. FLT_MAX: none fits.
//
// Two passes over up to 32 candidates: a loop without a division or a branch marks the ones
// near the prediction - a superset of the reference's box, widened by more than the rounding of
// its sum (a NaN marks) - and the marked ones, one in eight, get the reference's fit. The first
// loop's length is set by the longest windows among the warp's tracks (42% of its lanes are
// busy), so its step decides: 15 instructions against 40 with the fit inside. With the
// branch-free window searches, search of 65,536 events at nu ~ U(2,20) 13.80 -> 13.35 ms.
__device__ __forceinline__ float forward_best(const float4* H, const uint8_t* KE, const float4 h0, const float4 h1,
                                              float tx, float ty, int odd, int n_odd, int even, int n,
                                              uint16_t& best_h2)
{
  float best_fit = 3.402823466e+38f;
  const float tol0 = kTolerance + 1e-4f + 1e-5f * fmaxf(fabsf(h0.x), fabsf(h0.y));
  for (int c0 = 0; c0 < n; c0 += 32) {
    const int m = min(n - c0, 32);
    uint32_t marks = 0;
#pragma unroll 2
    for (int j = 0; j < m; ++j) {
      const float4 h2 = H[c0 + j + (c0 + j < n_odd ? odd : even)];
      const float dz = h2.z - h0.z;
      const float x = h0.x + tx * dz;
      const float y = h0.y + ty * dz;
      const float d = fmaxf(fabsf(x - h2.x), fabsf(y - h2.y));
      const float tol = tol0 + 1e-5f * fmaxf(fabsf(x), fabsf(y));
      if (!(d >= tol)) marks |= 1u << j;
    }
    while (marks) {
      const int j = c0 + __ffs(marks) - 1;
      marks &= marks - 1;
      const int h2i = j + (j < n_odd ? odd : even);
      if (KE && !(KE[h2i] & 2u)) continue;
      const float4 h2 = H[h2i];
      const float dz = h2.z - h0.z;
      const float predx = tx * dz;
      const float predy = ty * dz;
      const float scatterDenom2 = 1.f / ((h2.z - h1.z) * (h2.z - h1.z));
      const float fit = forward_fit(h0.x, h0.y, h2.x, h2.y, predx, predy, scatterDenom2);
      if (fit < best_fit) {
        best_fit = fit;
        best_h2 = static_cast<uint16_t>(h2i);
      }
    }
  }
  return best_fit;
}

// Per-event scratch of the search: the reference's Velo::TrackHits slots and the rings
// of tracklets, of tracks to follow and of weak tracklets (SearchByTripletVisitor.cu:11-18).
struct EventScratch {
  uint16_t* track_n;     // [kMaxTracks]
  uint16_t* track_hits;  // [kMaxTracks * kMaxTrackSize]
  uint16_t* tracklets;   // [kTrackletRing * 3]
  uint2* ttf;            // [kTtfModulo] {track and state bits, last hit << 16 | the hit before}
  uint16_t* weak;        // [kWeakCap * 3]
};

// Seeding windows read from the fill_candidates output: {h0 first | last << 16, h2 first |
// last << 16} per hit, event-relative (0xFFFF: no window). Each is read once per event, so
// it is loaded evict-first: the cache keeps the cluster records, which the search rereads.
struct StoredWindows {
  const uint2* w;
  __device__ __forceinline__ uint2 operator()(uint32_t h1, uint32_t) const { return __ldcs(w + h1); }
};

// Seeding windows computed where they are needed, with the searches of fill_candidates
// (FillCandidates.cu:31-68): h0 window in module m + 2, h2 window in module m - 2.
struct ComputedWindows {
  const float4* H;
  const uint16_t* mstart;
  const uint16_t* mnum;
  __device__ __forceinline__ uint2 operator()(uint32_t h1, uint32_t m) const
  {
    const float p = H[h1].w;
    int f0 = -1, l0 = -1, f2 = -1, l2 = -1;
    if (mnum[m + 2] > 0) phi_window4(H, mstart[m + 2], mnum[m + 2], p, kPhiExtrapolation, f0, l0);
    if (mnum[m - 2] > 0) phi_window4(H, mstart[m - 2], mnum[m - 2], p, kPhiExtrapolation, f2, l2);
    return make_uint2((static_cast<uint32_t>(f0) & 0xFFFFu) | (static_cast<uint32_t>(l0) << 16),
                      (static_cast<uint32_t>(f2) & 0xFFFFu) | (static_cast<uint32_t>(l2) << 16));
  }
};

// Loads the module table of one event into the group's shared state and clears its used-hit
// bitmask. module_start holds absolute hit indices; base is the event's first hit.
template<class Shared>
__device__ __forceinline__ void search_event_setup(Shared& sh, const uint32_t* module_start,
                                                   const uint32_t* module_num, uint32_t base, uint32_t nhits)
{
  constexpr int G = Shared::kWarps;
  const uint32_t tid = group_thread<G>();
  for (uint32_t i = tid; i < (nhits + 31) / 32; i += 32 * G) sh.used[i] = 0u;
  for (uint32_t m = tid; m < kModules; m += 32 * G) {
    sh.mstart[m] = static_cast<uint16_t>(module_start[m] - base);
    sh.mnum[m] = static_cast<uint16_t>(module_num[m]);
  }
  if (tid == 0) {
    sh.sum = 0;
    sh.flags = 0;
  }
  group_sync<G>();
}

// search_by_triplet and weak_tracks_adder of one event by G warps (ProcessModules.cu:37-162,
// TrackSeeding.cu:7-200, TrackForwarding.cu:41-181, WeakTracksAdder.cu:88-115), after
// search_event_setup. H: the event's phi-sorted cluster records; windows(h1, module): the
// seeding windows of h1; KE: extension-keep bits per hit (bit 1), or null. Returns the
// number of tracks written to sc.track_n / sc.track_hits; status bits go to `flags` (per
// thread: OR-reduce them over the group). Every append is ranked in the order of one warp
// taking the work from the front, so the result does not depend on G.
template<class Shared, class Windows>
__device__ __forceinline__ uint32_t search_event(Shared& sh, const float4* H, const Windows& windows,
                                                 const uint8_t* KE, const EventScratch& sc, uint32_t& flags)
{
  constexpr int G = Shared::kWarps;
  const uint32_t lane = lane_id(), tid = group_thread<G>();
  const uint32_t warp = G == 1 ? 0u : threadIdx.x >> 5;
  uint32_t* used = sh.used;
  const uint16_t* mstart = sh.mstart;
  const uint16_t* mnum = sh.mnum;
  SeedSlots& sl = sh.u.seed[warp];
  uint16_t* track_n = sc.track_n;
  uint16_t* track_hits = sc.track_hits;
  uint16_t* tracklets = sc.tracklets;
  uint2* ttf = sc.ttf;
  uint16_t* weak = sc.weak;
  uint32_t n_tracks = 0, tracklet_ptr = 0, ttf_ptr = 0, weak_ptr = 0;
  uint32_t last_seeded = 0;
  uint32_t turn = 0;
  // An event with more tracks to follow than the ring holds overwrites entries before they are
  // read, and may follow a track twice: what becomes of it depends on how many entries are read
  // ahead of the writes. From the first step that can come to that (kStatusTtfOverflow follows
  // if it does), one warp takes 32 entries in turn, as G = 1 does.
  bool in_turn = false;

  // Ahead of their step: the phi of the forwarding's modules (stage) and the windows of the
  // seeding's first run (fetch).
  auto stage = [&](uint32_t first) {
    const uint32_t mo = first - 4, me = first - 5, mon = mnum[mo], men = mnum[me];
    if (mon + men > Shared::kFwdStage) return;
    const float4 *Ho = H + mstart[mo], *He = H + mstart[me];
    for (uint32_t i = tid; i < mon; i += 32 * G) async_copy4(&sh.u.fphi[i], &Ho[i].w);
    for (uint32_t i = tid; i < men; i += 32 * G) async_copy4(&sh.u.fphi[mon + i], &He[i].w);
  };
  uint2 fetched[kSeedChunk / 32];
  auto fetch = [&](uint32_t first) {
    const uint32_t ma = first - 2, mb = first - 3, na = mnum[ma], n_list = na + mnum[mb];
    const uint32_t run = (min(n_list, G * kSeedChunk) + G - 1) / G;
    const uint32_t lo = min(n_list, warp * run), hi = min(n_list, lo + run);
#pragma unroll
    for (uint32_t j = 0; j < kSeedChunk / 32; ++j) {
      const uint32_t r = lo + 32 * j + lane;
      fetched[j] = make_uint2(0xFFFFu, 0xFFFFu);
      if (r < hi) fetched[j] = r < na ? windows(mstart[ma] + r, ma) : windows(mstart[mb] + r - na, mb);
    }
  };

  // ---- seeding: h1 in modules first-2 / first-3, h0 in h1+2, h2 in h1-2 ----
  // The two modules' seeds are independent (seeding marks no hit used). One warp takes the
  // modules' h1 in turn (first - 2, then first - 3), queueing unused ones with windows until
  // kSeedChunk wait: a module's last few hits share a pass with the next module's first ones.
  // G warps take G equal runs of both modules' h1, at most kSeedChunk each, at a time, and
  // append their winners run after run.
  auto seeding = [&](uint32_t first) {
    uint32_t n_h1 = 0;
    const uint32_t tracklets_before = tracklet_ptr;
    uint32_t nc = 0;  // candidates queued by this warp
    uint2 wv[kSeedChunk / 32];
    bool hv[kSeedChunk / 32];
    // the next (up to) kSeedChunk h1, hit_of(r) for r in [r0, r_end): unused, with both phi
    // windows (FillCandidates.cu:31-68, TrackSeeding.cu:24-49); the windows of their 32-hit
    // groups are loaded together so that their latencies overlap
    auto gather = [&](uint32_t r0, uint32_t r_end, auto hit_of, auto module_of, bool have_windows) {
      uint32_t n_new = 0;
#pragma unroll
      for (uint32_t j = 0; j < kSeedChunk / 32; ++j) {
        const uint32_t r = r0 + 32 * j + lane;
        wv[j] = make_uint2(0xFFFFu, 0xFFFFu);
        if (r < r_end && !test_used(used, hit_of(r))) {
          if constexpr (kFetchAhead<G>) wv[j] = have_windows ? fetched[j] : windows(hit_of(r), module_of(r));
          else wv[j] = windows(hit_of(r), module_of(r));
        }
      }
#pragma unroll
      for (uint32_t j = 0; j < kSeedChunk / 32; ++j) {
        const uint32_t r = r0 + 32 * j + lane;
        hv[j] = r < r_end && (wv[j].x & 0xFFFFu) != 0xFFFFu && (wv[j].y & 0xFFFFu) != 0xFFFFu;
        n_new += __popc(__ballot_sync(0xFFFFFFFFu, hv[j]));
      }
      return n_new;
    };
    auto queue = [&](uint32_t r0, auto hit_of) {
#pragma unroll
      for (uint32_t j = 0; j < kSeedChunk / 32; ++j) {
        uint32_t cnt;
        const uint32_t rank = ballot_rank(hv[j], cnt);
        if (hv[j]) {
          const uint32_t k = nc + rank;
          const uint32_t f0 = wv[j].x & 0xFFFFu, l0 = wv[j].x >> 16, f2 = wv[j].y & 0xFFFFu, l2 = wv[j].y >> 16;
          sl.h1[k] = static_cast<uint16_t>(hit_of(r0 + 32 * j + lane));
          sl.f0[k] = static_cast<uint16_t>(f0);
          sl.f2[k] = static_cast<uint16_t>(f2);
          sl.n2[k] = static_cast<uint16_t>(l2 - f2);
          sl.pair_start[k] = l0 - f0;
          sl.best[k] = ~0ull;
          sl.tie[k] = 0xFFFFFFFFu;
        }
        nc += cnt;
      }
    };
    // winners of this warp's queue, appended in candidate order from position `at` on
    // (TrackSeeding.cu:185-195)
    auto append = [&](uint32_t at) {
      for (uint32_t k0 = 0; k0 < nc; k0 += 32) {
        const uint32_t k = k0 + lane;
        const bool win = k < nc && sl.best[k] != ~0ull;
        uint32_t nwin;
        const uint32_t rank = at + ballot_rank(win, nwin);
        if (win) {
          const unsigned long long key = sl.best[k];
          if (static_cast<uint32_t>(key >> 32) == sl.tie[k]) flags |= kStatusSeedTie;
          const uint32_t tp = (tracklet_ptr + rank) % kTrackletRing;
          const uint32_t h1 = sl.h1[k], h2 = sl.f2[k] + (static_cast<uint32_t>(key) & 0xFFFFu);
          tracklets[3 * tp] = static_cast<uint16_t>(sl.f0[k] + (static_cast<uint32_t>(key) >> 16));
          tracklets[3 * tp + 1] = static_cast<uint16_t>(h1);
          tracklets[3 * tp + 2] = static_cast<uint16_t>(h2);
          ttf[(ttf_ptr + rank) % kTtfModulo] = make_uint2(0x80000000u | tp, (h2 << 16) | h1);
        }
        at += nwin;
      }
      __syncwarp();
      nc = 0;
      return at;
    };
    if constexpr (G == 1) {
      int side = 2;
      uint32_t r0 = 0;
      for (;;) {
        while (side <= 3 && r0 >= mnum[first - side]) {
          ++side;
          r0 = 0;
        }
        const bool have = side <= 3;
        const uint32_t m = first - (have ? side : 3);
        const uint32_t start = mstart[m];
        auto hit_of = [&](uint32_t r) { return start + r; };
        const uint32_t n_new = gather(r0, have ? min(mnum[m], r0 + kSeedChunk) : 0u, hit_of, [&](uint32_t) { return m; }, false);
        if (nc > 0 && (!have || nc + n_new > kSeedChunk)) {
          seed_flush(sl, nc, H, used);
          const uint32_t n = append(0);
          tracklet_ptr += n;
          ttf_ptr += n;
        }
        if (!have) break;
        queue(r0, hit_of);
        n_h1 += n_new;
        r0 += kSeedChunk;
      }
    } else {
      const uint32_t ma = first - 2, mb = first - 3;
      const uint32_t na = mnum[ma], n_list = na + mnum[mb], sa = mstart[ma], sb = mstart[mb] - na;
      auto hit_of = [&](uint32_t r) { return (r < na ? sa : sb) + r; };
      for (uint32_t r0 = 0; r0 < n_list; r0 += G * kSeedChunk) {
        const uint32_t run = (min(n_list - r0, G * kSeedChunk) + G - 1) / G;
        const uint32_t lo = min(n_list, r0 + warp * run), hi = min(n_list, lo + run);
        const uint32_t n_new = gather(lo, hi, hit_of, [&](uint32_t r) { return r < na ? ma : mb; },
                                      kFetchAhead<G> && r0 == 0);
        queue(lo, hit_of);
        if (nc > 0) seed_flush(sl, nc, H, used);
        uint32_t nwin = 0;
        for (uint32_t k0 = 0; k0 < nc; k0 += 32)
          nwin += __popc(__ballot_sync(0xFFFFFFFFu, k0 + lane < nc && sl.best[k0 + lane] != ~0ull));
        if (lane == 0) sh.count[turn][warp] = nwin | (n_new << 16);
        __syncthreads();
        uint32_t before = 0, all = 0;
#pragma unroll
        for (uint32_t w = 0; w < G; ++w) {
          const uint32_t v = sh.count[turn][w];
          before += w < warp ? v : 0u;
          all += v;
        }
        turn ^= 1u;
        append(before & 0xFFFFu);
        tracklet_ptr += all & 0xFFFFu;
        ttf_ptr += all & 0xFFFFu;
        n_h1 += all >> 16;
      }
      __syncthreads();  // the appended seeds, and the slots before they are staged over
    }
    if (n_h1 > kMaxHitsPerModule) flags |= kStatusH1Overflow;
    const uint32_t seeded = tracklet_ptr - tracklets_before;
    if (seeded + last_seeded > kTrackletRing) flags |= kStatusTtfOverflow;
    last_seeded = seeded;
  };

  // ---- forwarding of the tracks to follow into modules first-4 (odd) / first-5 (even) ----
  auto forwarding = [&](uint32_t first, uint32_t prev_ttf, uint32_t diff) {
    const uint32_t mo = first - 4, me = first - 5;
    const uint32_t mos = mstart[mo], mon = mnum[mo], mes = mstart[me], men = mnum[me];
    const float moz = c_module_z[mo], mez = c_module_z[me];
    // the phi of both target modules in shared memory, where their searches stay; a pair of
    // modules above the staging size is searched in global memory
    const bool fits = mon + men <= Shared::kFwdStage;
    const float* sphi_o = fits ? sh.u.fphi : nullptr;
    const float* sphi_e = fits ? sh.u.fphi + mon : nullptr;
    if constexpr (kFetchAhead<G>) {
      async_wait();  // staged during the seeding before
    } else if (diff > 0 && fits) {
      for (uint32_t i = tid; i < mon; i += 32 * G) sh.u.fphi[i] = H[mos + i].w;
      for (uint32_t i = tid; i < men; i += 32 * G) sh.u.fphi[mon + i] = H[mes + i].w;
    }
    group_sync<G>();
    // the writes come nearest to the reads at the start: an entry read writes at most one
    in_turn |= diff + 32 * G > kTtfModulo;
    const uint32_t step = in_turn ? 32 : 32 * G;
    for (uint32_t i0 = 0; i0 < diff; i0 += step) {
      const uint32_t i = tid < step ? i0 + tid : diff;
      int action = 0;  // 1 extend, 2 keep with a skipped module, 3 demote to weak
      uint32_t full = 0, last_two = 0, trackno = 0, nhit = 0;
      uint16_t t0 = 0, best_h2 = 0;
      if (i < diff) {
        // the entry brings the hits the prediction needs, two dependent loads fewer than through
        // the track (search of 65,536 events 13.18 -> 12.81 ms, of 1,000 0.271 -> 0.255); what
        // only an extension needs follows
        const uint2 entry = ttf[(prev_ttf + i) % kTtfModulo];
        full = entry.x;
        last_two = entry.y;
        const float4 h0 = H[last_two & 0xFFFFu];
        const float4 h1 = H[last_two >> 16];
        const uint32_t skipped = (full & 0x70000000u) >> 28;
        trackno = full & 0x0FFFFFFFu;
        if (full & 0x80000000u) {
          t0 = tracklets[3 * trackno];
          nhit = 3;
        } else {
          nhit = track_n[trackno];
        }
        const float td = 1.0f / (h1.z - h0.z);
        const float txn = (h1.x - h0.x);
        const float tyn = (h1.y - h0.y);
        const float tx = txn * td;
        const float ty = tyn * td;
        int of, ol, ef, el;
        forward_window_staged(H, sphi_o, mos, mon, moz, tx, ty, h0.x, h0.y, h0.z, true, of, ol, flags);
        forward_window_staged(H, sphi_e, mes, men, mez, tx, ty, h0.x, h0.y, h0.z, false, ef, el, flags);
        const int n_odd = ol - of, n_even = el - ef;
        const float best_fit = forward_best(H, KE, h0, h1, tx, ty, of, n_odd, ef - n_odd, n_odd + n_even, best_h2);
        // a track holds at most one hit per module pair: 26 hits (VeloDefinitions.cuh:26)
        if (best_fit != 3.402823466e+38f && nhit < kMaxTrackSize) action = 1;
        else if (skipped < kMaxSkippedModules) action = 2;
        else if (nhit == 3) action = 3;
      }
      if (action == 1) {
        set_used(used, best_h2);
        if (nhit == 3) {
          set_used(used, t0);
          set_used(used, last_two & 0xFFFFu);
          set_used(used, last_two >> 16);
        }
      }
      const bool is_new = action == 1 && nhit == 3;
      uint32_t rank[3], total[3];  // new tracks, tracks followed on, weak tracklets
      group_rank(sh, turn, is_new, action == 1 || action == 2, action == 3, rank, total);
      // new tracks beyond the last slot are dropped, and not followed
      const uint32_t slot = n_tracks + rank[0];
      const uint32_t dropped = slot > kMaxTracks ? slot - kMaxTracks : 0u;  // before this thread's
      const uint32_t all_tracks = n_tracks + total[0];
      const uint32_t all_dropped = all_tracks > kMaxTracks ? all_tracks - kMaxTracks : 0u;
      bool stored = action == 1;
      if (is_new) {
        if (slot < kMaxTracks) {
          uint16_t* th = track_hits + slot * kMaxTrackSize;
          th[0] = t0;
          th[1] = static_cast<uint16_t>(last_two);
          th[2] = static_cast<uint16_t>(last_two >> 16);
          th[3] = best_h2;
          track_n[slot] = 4;
          trackno = slot;
        } else {
          stored = false;
        }
      } else if (action == 1) {
        track_hits[trackno * kMaxTrackSize + nhit] = best_h2;
        track_n[trackno] = static_cast<uint16_t>(nhit + 1);
      }
      if (all_dropped) flags |= kStatusTrackOverflow;
      n_tracks = all_tracks - all_dropped;
      if (stored || action == 2) {
        ttf[(ttf_ptr + rank[1] - dropped) % kTtfModulo] =
          action == 2 ? make_uint2(((((full & 0x70000000u) >> 28) + 1) << 28) | (full & 0x8FFFFFFFu), last_two)
                      : make_uint2(trackno, (last_two >> 16) | (static_cast<uint32_t>(best_h2) << 16));
      }
      ttf_ptr += total[1] - all_dropped;
      if (action == 3 && weak_ptr + rank[2] < kWeakCap) {
        uint16_t* w = weak + 3 * (weak_ptr + rank[2]);
        w[0] = t0;
        w[1] = static_cast<uint16_t>(last_two);
        w[2] = static_cast<uint16_t>(last_two >> 16);
      }
      weak_ptr += total[2];
      if (step == 32) group_sync<G>();
    }
    group_sync<G>();
  };

  // ---- module loop (ProcessModules.cu:37-162) ----
  uint32_t first = kModules - 1;
  if constexpr (kFetchAhead<G>) {
    fetch(first);
    stage(first - 2);
  }
  seeding(first);
  uint32_t last_ttf = 0;
  first -= 2;
  while (first >= 4) {
    const uint32_t prev = last_ttf;
    last_ttf = ttf_ptr;
    if (last_ttf - prev > kTtfModulo) flags |= kStatusTtfOverflow;
    if constexpr (kFetchAhead<G>) fetch(first);
    forwarding(first, prev, last_ttf - prev);
    if (ttf_ptr - prev > kTtfModulo) flags |= kStatusTtfOverflow;
    if constexpr (kFetchAhead<G>)
      if (first >= 6) stage(first - 2);
    seeding(first);
    first -= 2;
  }
  {
    // tracklets still waiting become weak (ProcessModules.cu:146-162)
    const uint32_t prev = last_ttf;
    const uint32_t diff = ttf_ptr - prev;
    for (uint32_t i0 = 0; i0 < diff; i0 += 32 * G) {
      const uint32_t i = i0 + tid;
      uint32_t full = 0;
      if (i < diff) full = ttf[(prev + i) % kTtfModulo].x;
      const bool is_weak = i < diff && (full & 0x80000000u);
      uint32_t rank[3], total[3];
      group_rank(sh, turn, is_weak, false, false, rank, total);
      if (is_weak && weak_ptr + rank[0] < kWeakCap) {
        const uint32_t tp = full & 0x0FFFFFFFu;
        uint16_t* w = weak + 3 * (weak_ptr + rank[0]);
        w[0] = tracklets[3 * tp];
        w[1] = tracklets[3 * tp + 1];
        w[2] = tracklets[3 * tp + 2];
      }
      weak_ptr += total[0];
    }
  }
  if (weak_ptr > kMaxWeakTracks) flags |= kStatusWeakOverflow;
  group_sync<G>();
  // ---- weak_tracks_adder (WeakTracksAdder.cu:88-115) ----
  const uint32_t n_weak = min(weak_ptr, kWeakCap);
  for (uint32_t i0 = 0; i0 < n_weak; i0 += 32 * G) {
    const uint32_t i = i0 + tid;
    bool accept = false;
    uint16_t h[3] = {0, 0, 0};
    if (i < n_weak) {
      h[0] = weak[3 * i];
      h[1] = weak[3 * i + 1];
      h[2] = weak[3 * i + 2];
      const bool any_used = test_used(used, h[0]) || test_used(used, h[1]) || test_used(used, h[2]);
      const float chi2 = weak_chi2(H, h);
      accept = !any_used && chi2 < kMaxChi2;
    }
    uint32_t rank[3], total[3];
    group_rank(sh, turn, accept, false, false, rank, total);
    if (accept) {
      const uint32_t slot = n_tracks + rank[0];
      if (slot < kMaxTracks) {
        uint16_t* th = track_hits + slot * kMaxTrackSize;
        th[0] = h[0];
        th[1] = h[1];
        th[2] = h[2];
        track_n[slot] = 3;
      }
    }
    if (n_tracks + total[0] > kMaxTracks) flags |= kStatusTrackOverflow;
    n_tracks = min(n_tracks + total[0], kMaxTracks);
  }
  group_sync<G>();
  return n_tracks;
}

// One event of the chain by G warps: its tracks, their count and hit count and its status.
template<class Shared>
__device__ __forceinline__ void search_chain_event(Shared& sh, const ChainPointers& P, uint32_t e)
{
  constexpr int G = Shared::kWarps;
  const uint32_t lane = lane_id(), tid = group_thread<G>();
  const uint32_t nhits = P.event_hits[e];
  const uint32_t status = P.status[e];
  const uint32_t base = P.event_hit_base[e];
  uint32_t flags = 0;  // per thread, OR-reduced at the end
  uint32_t n_tracks = 0, track_hits = 0;
  const bool runnable = !(status & (kStatusBadRawEvent | kStatusHitOverflow)) && nhits <= kEventHitCap && nhits > 0;
  if (nhits > kEventHitCap) flags |= kStatusHitOverflow;
  if (runnable) {
    search_event_setup(sh, P.module_start + e * kModules, P.module_num + e * kModules, base, nhits);
    const EventScratch sc{P.scratch.track_n + static_cast<size_t>(e) * kMaxTracks,
                          P.scratch.track_hits + static_cast<size_t>(e) * kMaxTracks * kMaxTrackSize,
                          P.scratch.tracklets + static_cast<size_t>(e) * kTrackletRing * 3,
                          P.scratch.ttf + static_cast<size_t>(e) * kTtfModulo,
                          P.scratch.weak + static_cast<size_t>(e) * kWeakCap * 3};
    const uint8_t* KE = (P.keep && P.mlp.use_ext) ? P.keep + base : nullptr;  // extension pruning
    n_tracks = search_event(sh, P.hits.xyzp + base, StoredWindows{P.windows + base}, KE, sc, flags);
    for (uint32_t t = tid; t < n_tracks; t += 32 * G) track_hits += sc.track_n[t];
  }
  flags = __reduce_or_sync(0xFFFFFFFFu, flags);
  track_hits = __reduce_add_sync(0xFFFFFFFFu, track_hits);
  if (G > 1 && runnable) {
    if (lane == 0) {
      atomicOr(&sh.flags, flags);
      atomicAdd(&sh.sum, track_hits);
    }
    __syncthreads();
    flags = sh.flags;
    track_hits = sh.sum;
  }
  if (tid == 0) {
    P.event_tracks[e] = n_tracks;
    P.event_track_hits[e] = track_hits;
    P.status[e] = status | flags;
  }
  group_sync<G>();
}

// Persistent; the events largest first (order_events_kernel). The first queue[5] of them take
// a whole block, four warps an event, the others a warp each: a warp's events follow one
// another, so an event that alone takes longer than a warp's share of the batch would set the
// kernel's length. Four warps search an event in less than half of a warp's time (the module
// steps' barriers and part-filled rounds take the rest), so a batch that fills the device with
// events keeps to one warp each. Against one warp per event throughout: search of 1,000 events
// at nu = 7.6 0.64 -> 0.28 ms, of 3,000 at nu = 15 with noise 5.95 -> 1.79 ms, of 8,191 at
// nu ~ U(2,20) with every candidate scored 2.50 -> 1.32 ms; of 65,536, where no event takes a
// block, 13.35 -> 13.17 ms.
//
// 8 blocks of 4 warps per SM at 64 registers: more resident events (10 or 12 blocks at 48 or
// 40 registers) measured slower, their hit records competing for L1.
constexpr int kSearchWarps = 4;

// A batch of at most kSmallBatch events per SM takes eight warps an event, all of them resident
// at once: search of 10 / 148 / 300 / 590 events at nu ~ U(2,15) 0.251 / 0.273 / 0.325 / 0.398 ms
// with four, 0.183 / 0.185 / 0.221 / 0.287 with eight. Beyond one wave the uneven batches still
// gain (1,000 events 0.44 -> 0.39), the even ones lose (1,000 at nu = 7.6 0.26 -> 0.32).
constexpr int kSmallBatchWarps = 8;
constexpr uint32_t kSmallBatch = 4;

template<int W>
__global__ void __launch_bounds__(W * 32, 32 / W) search_kernel(ChainPointers P)
{
  __shared__ union {
    SearchShared<W> block;
    SearchShared<1, kWarpHitCap> warp[W];
  } s;
  __shared__ uint32_t s_next;
  const uint32_t lane = lane_id();
  const uint32_t n_events = P.run->n_events, n_block = P.queue[5];

  for (;;) {
    if (threadIdx.x == 0) s_next = atomicAdd(P.queue + 2, 1u);
    __syncthreads();
    const uint32_t q = s_next;
    __syncthreads();
    if (q >= n_block) break;
    search_chain_event(s.block, P, P.event_order[q]);
  }
  for (;;) {
    uint32_t q = 0;
    if (lane == 0) q = n_block + atomicAdd(P.queue + 1, 1u);
    q = __shfl_sync(0xFFFFFFFFu, q, 0);
    if (q >= n_events) break;
    search_chain_event(s.warp[threadIdx.x >> 5], P, P.event_order[q]);
  }
}

}  // namespace velo
