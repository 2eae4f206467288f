// Kernels 3 and 4 of the chain: exclusive scans over the events, then consolidation of
// the tracks into the reference's output layout with the beamline least-squares state and
// the simplified Kalman state.
#pragma once
#include "velo_kernels.cuh"

namespace velo {

// The run's totals, where velo_sync reads them: pinned host memory, written by the kernel that
// knows them, so no copy follows the run.
__device__ __forceinline__ void store_totals(const ChainPointers& P, uint32_t tracks, uint32_t hits)
{
  P.totals[0] = tracks;
  P.totals[1] = hits;
  P.totals[2] = P.queue[6];
}

// Exclusive scans of tracks and track hits per event by one block of 1024 threads, in the
// layout of copy_and_prefix_sum_single_block + the track-hit prefix sum
// (PrefixSumSingleBlock.cu:130-168). Sum holds the tracks and track hits of the whole batch.
//
// An event beyond the consolidated output capacity keeps no tracks and is flagged: each thread
// drops those of its run of events that do not fit behind the sum of all events before the run.
// So one run, where the sums pass the capacity, may keep some of its events, the runs before it
// keep all and those behind it none. The offsets and the totals count the kept events only:
// what is kept lies packed inside the buffers, and all of it is written.
template<class Sum>
__device__ __forceinline__ void scan_events_one_block(const ChainPointers& P)
{
  __shared__ Sum s_warp_t[32], s_warp_h[32];
  __shared__ uint32_t s_kept_t, s_kept_h;  // of a batch beyond the capacity
  const uint32_t N = P.run->n_events;
  const uint32_t per = (N + blockDim.x - 1) / blockDim.x;
  const uint32_t a = min(N, threadIdx.x * per), b = min(N, a + per);
  Sum t = 0, h = 0;
  for (uint32_t e = a; e < b; ++e) {
    t += P.event_tracks[e];
    h += P.event_track_hits[e];
  }
  const uint32_t lane = lane_id(), warp = threadIdx.x >> 5;
  Sum it = t, ih = h;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const Sum vt = __shfl_up_sync(0xFFFFFFFFu, it, o), vh = __shfl_up_sync(0xFFFFFFFFu, ih, o);
    if (lane >= static_cast<uint32_t>(o)) {
      it += vt;
      ih += vh;
    }
  }
  if (lane == 31) {
    s_warp_t[warp] = it;
    s_warp_h[warp] = ih;
  }
  __syncthreads();
  if (warp == 0) {
    Sum wt = lane < (blockDim.x >> 5) ? s_warp_t[lane] : 0, wh = lane < (blockDim.x >> 5) ? s_warp_h[lane] : 0;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const Sum vt = __shfl_up_sync(0xFFFFFFFFu, wt, o), vh = __shfl_up_sync(0xFFFFFFFFu, wh, o);
      if (lane >= static_cast<uint32_t>(o)) {
        wt += vt;
        wh += vh;
      }
    }
    s_warp_t[lane] = wt;
    s_warp_h[lane] = wh;
  }
  __syncthreads();
  const Sum first_t = it - t + (warp ? s_warp_t[warp - 1] : 0), first_h = ih - h + (warp ? s_warp_h[warp - 1] : 0);
  const bool behind = first_t > P.max_tracks_total || first_h > P.max_track_hits_total;
  const bool over = first_t + t > P.max_tracks_total || first_h + h > P.max_track_hits_total;
  uint32_t ot = static_cast<uint32_t>(first_t), oh = static_cast<uint32_t>(first_h);
  auto put = [&](uint32_t e, uint32_t nt) {
    P.atomics[e] = nt;
    P.atomics[N + e] = ot;
    P.event_hit_offset[e] = oh;
  };
  auto drop = [&](uint32_t e) {
    P.status[e] |= kStatusTrackOverflow;
    P.event_tracks[e] = 0;
    P.event_track_hits[e] = 0;
    put(e, 0);
  };
  if (!behind) {
    for (uint32_t e = a; e < b; ++e) {
      const uint32_t nt = P.event_tracks[e], nh = P.event_track_hits[e];
      if (over && (static_cast<Sum>(ot) + nt > P.max_tracks_total || static_cast<Sum>(oh) + nh > P.max_track_hits_total)) {
        drop(e);
        continue;
      }
      put(e, nt);
      ot += nt;
      oh += nh;
    }
    if (over) {  // one thread: every later run starts behind the capacity
      s_kept_t = ot;
      s_kept_h = oh;
    }
  }
  if (__syncthreads_or(behind) && behind) {
    ot = s_kept_t;
    oh = s_kept_h;
    for (uint32_t e = a; e < b; ++e) drop(e);
  }
  // the last thread that owns events (or thread 0 when N == 0) writes the totals
  if (b == N && (a < b || (N == 0 && threadIdx.x == 0))) {
    P.atomics[2 * N] = ot;
    P.event_hit_offset[N] = oh;
    P.track_hit_number[ot] = oh;
    store_totals(P, ot, oh);
  }
}

// (one block takes at most kScanOneBlock events: their sums fit 32 bits)
__global__ void __launch_bounds__(1024) event_scan_kernel(ChainPointers P)
{
  scan_events_one_block<uint32_t>(P);
}

// The same scans for batches of more than kScanOneBlock events, kScanBlock events a block in two
// launches: one block walks a thread's run of events one after the other, at uncoalesced
// addresses, and takes 4.8 us per 1,000 events (65,536: 0.315 ms, so 0.014). A batch that exceeds
// the output capacity goes through the one block, whose rule for what is dropped holds then.
constexpr uint32_t kScanBlock = 1024;
constexpr uint32_t kScanOneBlock = 4096;
static_assert(static_cast<uint64_t>(kScanOneBlock) * kMaxTracks * kMaxTrackSize < (1ull << 32), "32-bit sums");

// Sum over the block of x and y; s_sum: 32 entries.
__device__ __forceinline__ ulonglong2 scan_block_sum(unsigned long long x, unsigned long long y, ulonglong2* s_sum)
{
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    x += __shfl_xor_sync(0xFFFFFFFFu, x, o);
    y += __shfl_xor_sync(0xFFFFFFFFu, y, o);
  }
  __syncthreads();
  if (lane_id() == 0) s_sum[threadIdx.x >> 5] = make_ulonglong2(x, y);
  __syncthreads();
  ulonglong2 t = s_sum[lane_id()];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    t.x += __shfl_xor_sync(0xFFFFFFFFu, t.x, o);
    t.y += __shfl_xor_sync(0xFFFFFFFFu, t.y, o);
  }
  return t;
}

__global__ void __launch_bounds__(kScanBlock) event_sum_kernel(ChainPointers P)
{
  __shared__ ulonglong2 s_sum[32];
  const uint32_t e = blockIdx.x * kScanBlock + threadIdx.x;
  const bool in = e < P.run->n_events;
  const ulonglong2 t = scan_block_sum(in ? P.event_tracks[e] : 0u, in ? P.event_track_hits[e] : 0u, s_sum);
  if (threadIdx.x == 0) P.scan_sums[blockIdx.x] = t;
}

__global__ void __launch_bounds__(kScanBlock) event_scan_blocks_kernel(ChainPointers P)
{
  __shared__ ulonglong2 s_sum[32];
  __shared__ uint2 s_warp[32];
  const uint32_t N = P.run->n_events, lane = lane_id(), warp = threadIdx.x >> 5;
  // sums of the blocks before this one, and of all
  unsigned long long bt = 0, bh = 0, at = 0, ah = 0;
  for (uint32_t b = threadIdx.x; b < gridDim.x; b += kScanBlock) {
    const ulonglong2 v = P.scan_sums[b];
    at += v.x;
    ah += v.y;
    if (b < blockIdx.x) {
      bt += v.x;
      bh += v.y;
    }
  }
  const ulonglong2 all = scan_block_sum(at, ah, s_sum), before = scan_block_sum(bt, bh, s_sum);
  if (all.x > P.max_tracks_total || all.y > P.max_track_hits_total) {
    if (blockIdx.x == 0) scan_events_one_block<unsigned long long>(P);
    return;
  }
  const uint32_t e = blockIdx.x * kScanBlock + threadIdx.x;
  const uint32_t t = e < N ? P.event_tracks[e] : 0u, h = e < N ? P.event_track_hits[e] : 0u;
  uint32_t it = t, ih = h;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t vt = __shfl_up_sync(0xFFFFFFFFu, it, o), vh = __shfl_up_sync(0xFFFFFFFFu, ih, o);
    if (lane >= static_cast<uint32_t>(o)) {
      it += vt;
      ih += vh;
    }
  }
  if (lane == 31) s_warp[warp] = make_uint2(it, ih);
  __syncthreads();
  uint32_t wt = static_cast<uint32_t>(before.x), wh = static_cast<uint32_t>(before.y);
  for (uint32_t w = 0; w < warp; ++w) {
    wt += s_warp[w].x;
    wh += s_warp[w].y;
  }
  if (e < N) {
    P.atomics[e] = t;
    P.atomics[N + e] = wt + it - t;
    P.event_hit_offset[e] = wh + ih - h;
    if (e == N - 1) {
      P.atomics[2 * N] = wt + it;
      P.event_hit_offset[N] = wh + ih;
      P.track_hit_number[wt + it] = wh + ih;
      store_totals(P, wt + it, wh + ih);
    }
  }
}

struct FitState {
  float x, y, tx, ty, c00, c20, c22, c11, c31, c33, chi2, z;
  bool backward;
};

// means_square_fit (ConsolidateVelo.cu:6-114)
__device__ __forceinline__ FitState beamline_fit(const float* hx, const float* hy, const float* hz, uint32_t n)
{
  FitState state;
  float s0, sx, sz, sxz, sz2;
  float u0, uy, uz, uyz, uz2;
  s0 = sx = sz = sxz = sz2 = 0.0f;
  u0 = uy = uz = uyz = uz2 = 0.0f;
  for (uint32_t h = 0; h < n; ++h) {
    const float x = hx[h];
    const float y = hy[h];
    const float z = hz[h];
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
  {
    const float dens = 1.0f / (sz2 * s0 - sz * sz);
    state.tx = (sxz * s0 - sx * sz) * dens;
    state.x = (sx * sz2 - sxz * sz) * dens;
    const float denu = 1.0f / (uz2 * u0 - uz * uz);
    state.ty = (uyz * u0 - uy * uz) * denu;
    state.y = (uy * uz2 - uyz * uz) * denu;
    state.z = -(state.x * state.tx + state.y * state.ty) / (state.tx * state.tx + state.ty * state.ty);
    state.backward = state.z > hz[0];
  }
  {
    const float m00 = s0;
    const float m11 = u0;
    const float m20 = sz - state.z * s0;
    const float m31 = uz - state.z * u0;
    const float m22 = sz2 - 2 * state.z * sz + state.z * state.z * s0;
    const float m33 = uz2 - 2 * state.z * uz + state.z * state.z * u0;
    const float den20 = 1.0f / (m22 * m00 - m20 * m20);
    const float den31 = 1.0f / (m33 * m11 - m31 * m31);
    state.c00 = m22 * den20;
    state.c20 = -m20 * den20;
    state.c22 = m00 * den20;
    state.c11 = m33 * den31;
    state.c31 = -m31 * den31;
    state.c33 = m11 * den31;
  }
  {
    float ch = 0.0f;
    int nDoF = -4;
    for (uint32_t h = 0; h < n; ++h) {
      const float z = hz[h];
      const float x = state.x + state.tx * z;
      const float y = state.y + state.ty * z;
      const float dx = x - hx[h];
      const float dy = y - hy[h];
      ch += dx * dx * kParamW + dy * dy * kParamW;
      nDoF += 2;
    }
    state.chi2 = ch / nDoF;
  }
  state.x = state.x + state.tx * state.z;
  state.y = state.y + state.ty * state.z;
  return state;
}

// velo_kalman_filter_step (VeloKalmanFilter.cu:6-41)
__device__ __forceinline__ float kalman_step(const float z, const float zhit, const float xhit, const float whit,
                                             float& x, float& tx, float& covXX, float& covXTx, float& covTxTx)
{
  const float dz = zhit - z;
  const float predx = x + dz * tx;
  const float dz_t_covTxTx = dz * covTxTx;
  const float predcovXTx = covXTx + dz_t_covTxTx;
  const float dx_t_covXTx = dz * covXTx;
  const float predcovXX = covXX + 2 * dx_t_covXTx + dz * dz_t_covTxTx;
  const float predcovTxTx = covTxTx;
  const float R = 1.0f / ((1.0f / whit) + predcovXX);
  const float Kx = predcovXX * R;
  const float KTx = predcovXTx * R;
  const float r = xhit - predx;
  x = predx + Kx * r;
  tx = tx + KTx * r;
  covXX = (1 - Kx) * predcovXX;
  covXTx = (1 - Kx) * predcovXTx;
  covTxTx = predcovTxTx - KTx * predcovXTx;
  return r * r * R;
}

// simplified_fit<true> (VeloKalmanFilter.cuh:27-93)
__device__ __forceinline__ FitState kalman_fit(const float* hx, const float* hy, const float* hz, uint32_t nhits,
                                               const FitState& beam)
{
  const bool backward = beam.z > hz[0];
  const int direction = (backward ? 1 : -1) * 1;
  const float noise2PerLayer = 1e-8 + 7e-6 * (beam.tx * beam.tx + beam.ty * beam.ty);
  int firsthit = 0;
  int lasthit = nhits - 1;
  int dhit = 1;
  if ((hz[lasthit] - hz[firsthit]) * direction < 0) {
    const int temp = firsthit;
    firsthit = lasthit;
    lasthit = temp;
    dhit = -1;
  }
  FitState state;
  state.x = hx[firsthit];
  state.y = hy[firsthit];
  state.z = hz[firsthit];
  state.tx = beam.tx;
  state.ty = beam.ty;
  state.c00 = kParamWInverted;
  state.c11 = kParamWInverted;
  state.c20 = 0.f;
  state.c31 = 0.f;
  state.c22 = 1.f;
  state.c33 = 1.f;
  state.chi2 = 0.0f;
  for (uint32_t i = firsthit + dhit; i != static_cast<uint32_t>(lasthit + dhit); i += dhit) {
    const int hitindex = i;
    const float hit_x = hx[hitindex];
    const float hit_y = hy[hitindex];
    const float hit_z = hz[hitindex];
    state.c22 += noise2PerLayer;
    state.c33 += noise2PerLayer;
    state.chi2 += kalman_step(state.z, hit_z, hit_x, kParamW, state.x, state.tx, state.c00, state.c20, state.c22);
    state.chi2 += kalman_step(state.z, hit_z, hit_y, kParamW, state.y, state.ty, state.c11, state.c31, state.c33);
    state.z = hit_z;
  }
  state.c22 += noise2PerLayer;
  state.c33 += noise2PerLayer;
  state.backward = backward;  // not set by the reference's fit
  return state;
}

__device__ __forceinline__ void store_state(char* base, uint32_t T, uint32_t i, const FitState& s)
{
  float* f = reinterpret_cast<float*>(base);
  f[i] = s.x;
  f[T + i] = s.y;
  f[2 * T + i] = s.tx;
  f[3 * T + i] = s.ty;
  f[4 * T + i] = s.c00;
  f[5 * T + i] = s.c20;
  f[6 * T + i] = s.c22;
  f[7 * T + i] = s.c11;
  f[8 * T + i] = s.c31;
  f[9 * T + i] = s.c33;
  f[10 * T + i] = s.chi2;
  f[11 * T + i] = s.z;
  reinterpret_cast<bool*>(base + sizeof(float) * 12 * T)[i] = s.backward;
}

// Consolidation, beamline state and Kalman state, one event per block of W warps, largest
// events first. The block scans the hit counts of the event's tracks; its warps then take 32
// tracks at a time, one per lane. The hits of 32 tracks form one contiguous range of the
// Velo::Consolidated::Hits SoA, which the warp writes in order (coalesced), finding the track
// of an output position from the starts. The same loop keeps x, y, z of the range in shared
// memory (up to kConsolidateStage hits), from where the fits run per lane on their track's
// slice; a larger range (32 tracks averaging more than 16 hits) fits from per-lane copies
// instead.
//
// Bound by the latency of its chain of gathers (hit index, then record and id): a warp per
// event ran the chain once per 32 tracks, five times over for an average event, and a block
// waited for the largest of its four events. Four warps an event, of 65,536 at nu ~ U(2,20):
// 3.75 -> 1.96 ms (two warps: 3.52).
constexpr uint32_t kConsolidateStage = 512;
constexpr int kConsolidateWarps = 4;

template<int W>
__global__ void __launch_bounds__(W * 32) consolidate_fit_kernel(ChainPointers P)
{
  static_assert(kMaxTracks * kMaxTrackSize < 65536, "hit offsets of an event in 16 bits");
  __shared__ uint16_t s_off[kMaxTracks + 1];  // first hit of each track in the event
  __shared__ uint32_t s_warp[W];
  __shared__ float s_hit[W][3][kConsolidateStage];
  const uint32_t lane = lane_id(), warp = threadIdx.x >> 5;
  const uint32_t N = P.run->n_events;
  if (blockIdx.x >= N) return;
  const uint32_t e = P.event_order[blockIdx.x];
  const uint32_t T = P.atomics[2 * N];
  const uint32_t Htot = P.event_hit_offset[N];
  const uint32_t nt = P.atomics[e];
  if (nt == 0) return;
  const uint32_t t0 = P.atomics[N + e];
  const float4* H = P.hits.xyzp + P.event_hit_base[e];
  const uint32_t* ids = P.hits.id + P.event_hit_base[e];
  float* ox = reinterpret_cast<float*>(P.track_hits_out);
  float* oy = ox + Htot;
  float* oz = ox + 2 * static_cast<size_t>(Htot);
  uint32_t* oid = reinterpret_cast<uint32_t*>(ox + 3 * static_cast<size_t>(Htot));
  const uint16_t* track_n = P.scratch.track_n + static_cast<size_t>(e) * kMaxTracks;
  const uint16_t* track_hits = P.scratch.track_hits + static_cast<size_t>(e) * kMaxTracks * kMaxTrackSize;
  const uint32_t first_hit = P.event_hit_offset[e];
  // ---- exclusive scan of the hit counts ----
  uint32_t before = 0;
  for (uint32_t i0 = 0; i0 < nt; i0 += 32 * W) {
    const uint32_t i = i0 + threadIdx.x;
    const uint32_t n = i < nt ? track_n[i] : 0;
    uint32_t incl = n;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t v = __shfl_up_sync(0xFFFFFFFFu, incl, o);
      if (lane >= static_cast<uint32_t>(o)) incl += v;
    }
    if (lane == 31) s_warp[warp] = incl;
    __syncthreads();
    uint32_t lower = 0, all = 0;
#pragma unroll
    for (uint32_t w = 0; w < W; ++w) {
      const uint32_t v = s_warp[w];
      lower += w < warp ? v : 0u;
      all += v;
    }
    if (i < nt) s_off[i] = static_cast<uint16_t>(before + lower + incl - n);
    before += all;
    __syncthreads();
  }
  if (threadIdx.x == 0) s_off[nt] = static_cast<uint16_t>(before);
  __syncthreads();
  // ---- 32 tracks at a time ----
  for (uint32_t i0 = 32 * warp; i0 < nt; i0 += 32 * W) {
    const uint32_t i = i0 + lane;
    const uint32_t n_chunk = min(32u, nt - i0);  // tracks of this chunk
    const uint32_t chunk0 = s_off[i0], chunk_hits = s_off[i0 + n_chunk] - chunk0;
    const uint32_t carry = first_hit + chunk0;
    // coalesced write of the chunk's hit range [carry, carry + chunk_hits)
    const bool staged = chunk_hits <= kConsolidateStage;
    // eight output positions per lane at a time, as many as 32 average tracks have: their dependent
    // gathers (hit index, then record and id) are in flight together (65,536 events 1.98 ms with
    // four, 1.78 with eight at 96 registers, 1.87 with nine at 111; four at 64 registers, which one
    // more block an SM would need, 3.24). The track of a position: every track has hits,
    // so the tracks starting inside 32 consecutive positions are marked by one bit each (an
    // OR across the warp of the lanes' own starts) and counted with a popcount.
    const uint32_t my_start = lane < n_chunk ? s_off[i] - chunk0 : 0xFFFFFFFFu;
    uint32_t started = 0;  // tracks starting before the current group of 32 positions
    for (uint32_t base = 0; base < chunk_hits; base += 8 * 32) {  // warp-uniform
      const uint32_t j0 = base + lane;
      uint32_t hh[8];
#pragma unroll
      for (uint32_t u = 0; u < 8; ++u) {
        const uint32_t p0 = base + 32 * u;  // first position of this group
        const uint32_t heads =
          __reduce_or_sync(0xFFFFFFFFu, my_start - p0 < 32u ? 1u << (my_start - p0) : 0u);
        const uint32_t j = p0 + lane;
        const uint32_t t = started + __popc(heads & (0xFFFFFFFFu >> (31 - lane))) - 1;  // track of j
        started += __popc(heads);
        hh[u] = j < chunk_hits ? track_hits[(i0 + t) * kMaxTrackSize + (chunk0 + j - s_off[i0 + t])] : 0u;
      }
      float4 p[8];
      uint32_t id[8];
#pragma unroll
      for (uint32_t u = 0; u < 8; ++u) {
        if (j0 + 32 * u < chunk_hits) {
          p[u] = H[hh[u]];
          id[u] = ids[hh[u]];
        }
      }
#pragma unroll
      for (uint32_t u = 0; u < 8; ++u) {
        const uint32_t j = j0 + 32 * u;
        if (j < chunk_hits) {
          ox[carry + j] = p[u].x;
          oy[carry + j] = p[u].y;
          oz[carry + j] = p[u].z;
          oid[carry + j] = id[u];
          if (staged) {
            s_hit[warp][0][j] = p[u].x;
            s_hit[warp][1][j] = p[u].y;
            s_hit[warp][2][j] = p[u].z;
          }
        }
      }
    }
    __syncwarp();
    if (i < nt) {
      const uint32_t o = s_off[i] - chunk0, n = s_off[i + 1] - s_off[i];
      P.track_hit_number[t0 + i] = carry + o;
      FitState beam, kal;
      if (staged) {
        beam = beamline_fit(&s_hit[warp][0][o], &s_hit[warp][1][o], &s_hit[warp][2][o], n);
        kal = kalman_fit(&s_hit[warp][0][o], &s_hit[warp][1][o], &s_hit[warp][2][o], n, beam);
      } else {
        float hx[kMaxTrackSize], hy[kMaxTrackSize], hz[kMaxTrackSize];
        for (uint32_t k = 0; k < n; ++k) {
          const float4 p = H[track_hits[i * kMaxTrackSize + k]];
          hx[k] = p.x;
          hy[k] = p.y;
          hz[k] = p.z;
        }
        beam = beamline_fit(hx, hy, hz, n);
        kal = kalman_fit(hx, hy, hz, n, beam);
      }
      store_state(P.states, T, t0 + i, beam);
      store_state(P.kalman_states, T, t0 + i, kal);
    }
    __syncwarp();
  }
}

}  // namespace velo
