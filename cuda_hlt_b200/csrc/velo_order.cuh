// Launched between fill_candidates and search_by_triplet: the queue order of the warp search.
#pragma once
#include "velo_kernels.cuh"

namespace velo {

// Longest-processing-time-first order of the search's events. The search hands events out
// through an atomic queue, a few per warp in a batch, and its time per event spreads about
// tenfold with the occupancy, so large events that come last set the kernel's length. Taken
// largest first (counting sort on the cluster count in buckets of 16, one CTA), the small
// events fill the tail. The order within a bucket is free: every event's result is independent
// of when it runs.
//
// It also says how many of the first events take a block instead of a warp (queue[5]): those
// above the caller's cluster count or what a warp's search holds, and those whose search on one warp would last longer than
// kBlockShare of a warp's share of the batch, by an estimate of a search's time, n (n + 2000)
// for n clusters. Search in ms at shares 0.5 / 0.75 / 1 / 1.4: 4,001 events at nu ~ U(2,15)
// 0.92 / 0.94 / 0.91 / 1.03, 8,191 at U(2,20) 1.47 / 1.41 / 1.32 / 1.29, 16,384 3.47 / 3.30 /
// 3.19 / 3.19, 3,000 noisy ones 1.79 / 1.81 / 1.79 / 1.86.
constexpr uint32_t kOrderThreads = 1024;
constexpr uint32_t kOrderBuckets = kOrderThreads;
constexpr uint32_t kOrderShift = 4;
constexpr float kBlockShare = 1.0f;

// Sum of x over the block's threads (whole numbers below 2^24 exactly).
__device__ __forceinline__ float order_sum(float x, float* s_sum)
{
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xFFFFFFFFu, x, o);
  __syncthreads();
  if (lane_id() == 0) s_sum[threadIdx.x >> 5] = x;
  __syncthreads();
  float t = s_sum[lane_id()];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xFFFFFFFFu, t, o);
  return t;
}

__global__ void __launch_bounds__(kOrderThreads) order_events_kernel(ChainPointers P)
{
  __shared__ uint32_t s_off[kOrderBuckets];
  __shared__ uint32_t s_warp[kOrderThreads / 32];
  __shared__ float s_sum[kOrderThreads / 32];
  const uint32_t n = P.run->n_events;
  const uint32_t t = threadIdx.x, lane = t & 31u;
  auto bucket = [&](uint32_t e) {
    return kOrderBuckets - 1u - min(P.event_hits[e] >> kOrderShift, kOrderBuckets - 1u);
  };
  s_off[t] = 0;
  __syncthreads();
#pragma unroll 4
  for (uint32_t e = t; e < n; e += kOrderThreads) atomicAdd(&s_off[bucket(e)], 1u);
  __syncthreads();
  // exclusive scan of the bucket counts
  const uint32_t v = s_off[t];
  uint32_t incl = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, incl, o);
    if (lane >= static_cast<uint32_t>(o)) incl += y;
  }
  if (lane == 31) s_warp[t >> 5] = incl;
  __syncthreads();
  if (t < 32) {
    const uint32_t w = s_warp[t];
    uint32_t wi = w;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, wi, o);
      if (lane >= static_cast<uint32_t>(o)) wi += y;
    }
    s_warp[t] = wi - w;
  }
  __syncthreads();
  s_off[t] = s_warp[t >> 5] + incl - v;
  // events that take a block: this thread's bucket, and all before it
  const uint32_t clusters = (kOrderBuckets - 1u - t) << kOrderShift;  // the bucket's lower edge
  const float mid = static_cast<float>(clusters) + 0.5f * (1u << kOrderShift);
  const float cost = mid * (mid + 2000.f);
  const float all = order_sum(v * cost, s_sum);
  const bool block = clusters + (1u << kOrderShift) - 1u > min(P.block_threshold, kWarpHitCap) ||
                     cost * static_cast<float>(P.search_warps) > kBlockShare * all;
  const float n_block = order_sum(block ? static_cast<float>(v) : 0.f, s_sum);
  if (t == 0) P.queue[5] = static_cast<uint32_t>(n_block);
  __syncthreads();
#pragma unroll 4
  for (uint32_t e = t; e < n; e += kOrderThreads) P.event_order[atomicAdd(&s_off[bucket(e)], 1u)] = e;
}

}  // namespace velo
