// Kernel 1 of the chain: SuperPixel decode, masked clustering, phi and per-module sort.
//
// One block per event (persistent; events are pulled from a device queue), one pass over
// the event's SP words:
//   * isolated SPs give their one or two clusters from the pattern table at once;
//   * a non-isolated SP finds its neighbours by binary search in its bank (banks are
//     address-sorted in LHCb raw data; unsorted banks fall back to the reference's linear
//     scan, with the same result) and pushes its candidate pixels to a shared list, which
//     the block then flood-fills with every thread busy;
//   * clusters go to their module's slice of a staging area sized by the module's SP count
//     (at most two clusters per SP), one shared atomic per cluster;
//   * one warp per module sorts the slice on (phi, LHCb id) - up to 256 clusters in registers
//     on 32-bit keys with warp shuffles, up to 512 (and where short keys agree) in shared memory
//     on the full keys - and writes it to the compact phi-sorted layout.
// The result equals the reference's estimate -> prefix sum -> masked clustering ->
// calculate_phi_and_sort sequence, whose order within a module depends on the order of its
// atomics only for exactly equal phi.
#pragma once
#include "velo_kernels.cuh"

namespace velo {

constexpr uint32_t kSortCap = 512;  // clusters per module sorted in shared memory

// SPs around one SP: the non-isolated ones of the 4x3-SP flood window
// (MaskedVeloClustering.cu:221-272) and, over every SP of the bank, the five neighbours the
// candidate search reads (EstimateInputSize.cu:124-153).
struct SpWindow {
  uint32_t px[3];
  uint32_t top, top_right, right, right_bottom, bottom;
};

__device__ __forceinline__ void window_add(SpWindow& w, uint32_t o, int32_t r, int32_t c)
{
  const int32_t orow = sp_row(o), ocol = sp_col(o);
  const uint32_t osp = sp_mask(o);
  if (!sp_isolated(o) && orow >= r - 2 && orow <= r + 1 && ocol >= c - 1 && ocol <= c + 1) {
    const int32_t rr = orow - (r - 2), rc = ocol - (c - 1);
    const uint32_t v = (osp & 0x0Fu) << (4 * rr) | (osp & 0xF0u) << (12 + 4 * rr);
    // constant register indices: a runtime index would put the window in local memory
    w.px[0] |= rc == 0 ? v : 0u;
    w.px[1] |= rc == 1 ? v : 0u;
    w.px[2] |= rc == 2 ? v : 0u;
  }
  if (ocol == c) {
    if (orow == r + 1) w.top |= osp;
    if (orow == r - 1) w.bottom |= osp;
  } else if (ocol == c + 1) {
    if (orow == r + 1) w.top_right |= osp;
    if (orow == r) w.right |= osp;
    if (orow == r - 1) w.right_bottom |= osp;
  }
}

__device__ __forceinline__ uint32_t bank_lower_bound(const uint32_t* bank, uint32_t count, uint32_t addr)
{
  uint32_t lo = 0, hi = count;
  while (lo < hi) {
    const uint32_t mid = (lo + hi) >> 1;
    if (sp_addr(__ldg(bank + mid)) < addr) lo = mid + 1; else hi = mid;
  }
  return lo;
}

__device__ __forceinline__ SpWindow gather_window(const uint32_t* bank, uint32_t count, bool sorted, int32_t r,
                                                  int32_t c)
{
  SpWindow w{{0u, 0u, 0u}, 0u, 0u, 0u, 0u, 0u};
  if (sorted) {
    // the three columns are adjacent in address order (column << 6 | row): one search and
    // one scan over [(c - 1, r - 2), (c + 1, r + 1)]; the rows outside [r - 2, r + 1] that
    // the scan also meets are rejected by window_add
    const uint32_t a_lo = (static_cast<uint32_t>(max(c - 1, 0)) << 6) | static_cast<uint32_t>(max(r - 2, 0));
    const uint32_t a_hi = (static_cast<uint32_t>(min(c + 1, 511)) << 6) | static_cast<uint32_t>(min(r + 1, 63));
    for (uint32_t i = bank_lower_bound(bank, count, a_lo); i < count; ++i) {
      const uint32_t o = __ldg(bank + i);
      if (sp_addr(o) > a_hi) break;
      window_add(w, o, r, c);
    }
  } else {
    for (uint32_t i = 0; i < count; ++i) window_add(w, __ldg(bank + i), r, c);
  }
  return w;
}

// Candidate-pixel code of a non-isolated SP from its neighbours (EstimateInputSize.cu:118-183).
__device__ __forceinline__ uint32_t window_candidate_code(uint32_t sp, const SpWindow& w)
{
  uint32_t pixels = (sp & 0x0Fu) | ((sp & 0xF0u) << 2);
  pixels |= ((w.top & 0x01u) | ((w.top & 0x10u) << 2)) << 4;
  pixels |= (w.top_right & 0x01u) << 16;
  pixels |= (w.right & 0x0Fu) << 12;
  pixels |= (w.right_bottom & 0x08u) << 8;
  pixels |= (w.bottom & 0x80u) >> 2;
  const uint32_t inside = pixels & 0x3CFu;
  const uint32_t mask = (inside << 1) | (inside << 5) | (inside << 6) | (inside << 7);
  const uint32_t open = mask & (~pixels);
  const uint32_t cand = (open >> 1) & (open >> 5) & (open >> 6) & (open >> 7) & pixels;
  return (cand & 0x03u) | ((cand & 0xC0u) >> 4) | ((cand & 0x0Cu) << 2) | ((cand & 0x0300u) >> 2);
}

// Flood fill seeded by pixel k of the SP at (sp_r, sp_c) over the window pixels
// (MaskedVeloClustering.cu:274-398). True when the cluster is stored.
__device__ __forceinline__ bool flood_window(uint32_t px0, uint32_t px1, uint32_t px2, int32_t sp_r, int32_t sp_c,
                                             uint32_t k, int32_t& xs, int32_t& ys, int32_t& n)
{
  const int32_t row_lower_limit = (sp_r - 2) * 4, col_lower_limit = (sp_c - 1) * 2;
  const uint32_t row = sp_r * 4 + (k % 4);
  const uint32_t col = sp_c * 2 + (k >= 4);
  const uint32_t seed = (0x01u << (row - row_lower_limit)) << (16 * (col % 2));
  uint32_t cl0 = 0, cl1 = seed, cl2 = 0;
  uint32_t w0 = 0, w1 = seed, w2 = 0;
  px1 &= ~cl1;
#pragma unroll 1
  for (uint32_t it = 0; it < kMaxClusteringIterations; ++it) {
    const uint32_t m0 = flood_mask(w0) | flood_right_to_left(w1);
    const uint32_t m1 = flood_mask(w1) | flood_right_to_left(w2) | flood_left_to_right(w0);
    const uint32_t m2 = flood_mask(w2) | flood_left_to_right(w1);
    w0 = px0 & m0;
    w1 = px1 & m1;
    w2 = px2 & m2;
    if ((w0 | w1 | w2) == 0u) break;
    cl0 |= w0;
    cl1 |= w1;
    cl2 |= w2;
    px0 &= ~cl0;
    px1 &= ~cl1;
    px2 &= ~cl2;
  }
  if (cl2) return false;  // a pixel in the SP column to the right owns this cluster
  n = __popc(cl0) + __popc(cl1);
  if (n >= 3) {
    const uint32_t c0 = found_cluster_mask(cl0) & ~cl0;
    const uint32_t c1 = (found_cluster_mask(cl1) | flood_left_to_right(cl0)) & ~cl1;
    const uint32_t c2 = flood_left_to_right(cl1);
    const uint32_t cand0 = precedence_candidates(c0, c1) & cl0;
    const uint32_t cand1 = (precedence_candidates(c1, c2) & cl1) ^ seed;
    if (cand0 | cand1) {
      const int32_t neg = ~(-static_cast<int32_t>(seed));
      const bool under = seed < 4096u;
      uint32_t smaller_row = under * (0xFFF & neg) | (!under) * (0xFFF & (neg >> 16));
      smaller_row |= smaller_row << 16;
      const uint32_t current = smaller_row | under * 0xFFFF0000u;
      if (((cand0 & smaller_row) | (cand1 & current)) != 0u) return false;
    }
  }
  xs = __popc(cl0 & 0x0000FFFFu) * col_lower_limit + __popc(cl0 & 0xFFFF0000u) * (col_lower_limit + 1) +
       __popc(cl1 & 0x0000FFFFu) * (col_lower_limit + 2) + __popc(cl1 & 0xFFFF0000u) * (col_lower_limit + 3);
  const uint32_t t0 = (cl0 & 0x000F000Fu) | ((cl1 & 0x000F000Fu) << 4);
  const uint32_t t1 = ((cl0 & 0x00F000F0u) >> 4) | (cl1 & 0x00F000F0u);
  const uint32_t t2 = ((cl0 & 0x0F000F00u) >> 8) | ((cl1 & 0x0F000F00u) >> 4);
  const uint32_t t3 = ((cl0 & 0xF000F000u) >> 12) | ((cl1 & 0xF000F000u) >> 8);
  int32_t y = 0;
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    const uint32_t m = 0x11111111u << r;
    y += __popc(t0 & m) * (row_lower_limit + r) + __popc(t1 & m) * (row_lower_limit + 4 + r) +
         __popc(t2 & m) * (row_lower_limit + 8 + r) + __popc(t3 & m) * (row_lower_limit + 12 + r);
  }
  ys = y;
  return true;
}

constexpr uint32_t kCandCap = 4096;    // candidate pixels listed per event (more: flooded inline)
constexpr uint32_t kNoCandidate = 0xFFFFFFFFu;  // (bank 255 does not exist)
constexpr uint32_t kNonIsoCap = 2048;   // non-isolated SPs listed per event (more: full rescan)
constexpr uint32_t kRegSortMax = 256;  // modules up to this size are sorted in registers

struct DecodeShared {
  uint32_t bank_start[kSensors];  // word index (from the event start) of the first SP word
  uint32_t bank_count[kSensors];
  uint32_t bank_sensor[kSensors];
  uint32_t sp_prefix[kSensors + 1];  // exclusive scan of bank_count
  uint32_t unsorted[(kSensors + 31) / 32];
  uint32_t mod_count[kModules];  // clusters per module
  uint32_t mod_start[kModules];  // exclusive scan of mod_count: compact layout
  uint32_t mod_phi[kModules];    // exclusive scan over the modules of the same parity
  uint32_t event;
  uint32_t n_events;             // events of the run
  uint32_t skipped;              // 1: position left empty (beyond the selection); 2: bad list entry
  uint64_t ev_off, ev_bytes;     // the event's raw bytes: offset in the batch and size
  uint32_t flags;
  uint32_t n_candidates;
  uint32_t n_list;
  uint32_t n_noniso;  // non-isolated SPs met by the first pass
};

__device__ __forceinline__ uint32_t bank_of(const DecodeShared& sh, uint32_t f)
{
  uint32_t lo = 0, hi = kSensors;  // last b with sp_prefix[b] <= f
  while (hi - lo > 1) {
    const uint32_t mid = (lo + hi) >> 1;
    if (sh.sp_prefix[mid] <= f) lo = mid; else hi = mid;
  }
  return lo;
}

struct DecodeEvent {
  const uint32_t* ev;       // raw event words
  uint32_t stage_base;      // first staging slot of the event
  float4* stage;
  uint32_t* stage_id;
};

// Bits 26-27 of an LHCb VP id are always zero (sensor < 208 ends at bit 25): the staging
// record carries the cluster's pixel count there, at most 3.
constexpr uint32_t kSizeShift = 26;
constexpr uint32_t kSizeMask = 3u << kSizeShift;

// Appends one cluster of `pixels` pixels to module m's staging slice: slots
// [2 * SPs before m, ...).
__device__ __forceinline__ void stage_cluster(DecodeShared& sh, const DecodeEvent& d, uint32_t m,
                                              const ClusterPoint& p, uint32_t pixels)
{
  const uint32_t slot = atomicAdd(&sh.mod_count[m], 1u);
  const uint32_t o = d.stage_base + 2 * sh.sp_prefix[4 * m] + slot;
  const float phi = (m & 1) ? phi_odd_side(p.x, p.y) : phi_even_side(p.x, p.y);
  d.stage[o] = make_float4(p.x, p.y, p.z, phi);
  d.stage_id[o] = p.id | (min(pixels, 3u) << kSizeShift);
}

// Flood fill of candidate pixel k of flat SP f, of bank b, and staging of the cluster
// (MaskedVeloClustering.cu:175-461).
__device__ __forceinline__ void flood_candidate(DecodeShared& sh, const DecodeEvent& d, const DeviceConstants& g,
                                                uint32_t f, uint32_t b, uint32_t k)
{
  const uint32_t s = f - sh.sp_prefix[b];
  const uint32_t* bank = d.ev + sh.bank_start[b];
  const uint32_t count = sh.bank_count[b];
  const bool sorted = !((sh.unsorted[b >> 5] >> (b & 31)) & 1u);
  // The reference packs the SP index into a u8 when it decodes candidates
  // (MaskedVeloClustering.cu:179), so above 255 SPs the flood runs on SP s & 0xFF.
  const uint32_t word2 = __ldg(bank + (s & 0xFFu));
  const int32_t r2 = sp_row(word2), c2 = sp_col(word2);
  const SpWindow w = gather_window(bank, count, sorted, r2, c2);
  int32_t xs, ys, np;
  if (!flood_window(w.px[0], w.px[1], w.px[2], r2, c2, k, xs, ys, np)) return;
  const uint32_t cx = xs / np;
  const uint32_t cy = ys / np;
  const float fx = xs / static_cast<float>(np) - cx;
  const float fy = ys / static_cast<float>(np) - cy;
  stage_cluster(sh, d, b >> 2, place_cluster(g, sh.bank_sensor[b], cx, cy, fx, fy, cx / kChipColumns),
                static_cast<uint32_t>(np));
}

// Sort key of a staged cluster: phi (orderable bits), LHCb id within the module (20 bits:
// sensor in module, chip, column, row), staging slot (12 bits).
__device__ __forceinline__ unsigned long long cluster_key(const float4* src, const uint32_t* src_id, uint32_t i)
{
  return (static_cast<unsigned long long>(orderable(src[i].w)) << 32) |
         (static_cast<unsigned long long>(src_id[i] & 0xFFFFFu) << 12) | i;
}

// Short sort key: phi to 24..26 bits above the staging slot (5 + log2 PER bits). phi + 4 is
// between 0.85 and 10.3, so the float's bit pattern less that of 0.5 orders it in 26 bits;
// anything else (a NaN) is cut to a value below the padding key.
template<uint32_t PER>
__device__ __forceinline__ uint32_t short_key(float phi, uint32_t slot)
{
  constexpr uint32_t kSlotBits = PER == 8 ? 8 : PER == 4 ? 7 : PER == 2 ? 6 : 5;
  constexpr uint32_t kDrop = kSlotBits > 6 ? kSlotBits - 6 : 0;
  const uint32_t q = min(__float_as_uint(phi + 4.0f) - 0x3F000000u, 0x3FFFFF0u);
  return ((q >> kDrop) << kSlotBits) | slot;
}

// Bitonic sort of 32 * PER 32-bit keys held PER per lane, element lane * PER + j in key[j]
// (the input may sit in any slots: only the sorted order is read back this way). The
// exchanges between elements less than PER apart stay inside a lane, the others take one
// shuffle per key; loops unrolled, so every register index is a compile-time constant. Blocks
// that sort downwards hold their keys complemented, so every exchange is a plain min and max.
template<uint32_t PER>
__device__ __forceinline__ void warp_register_sort(uint32_t (&key)[PER])
{
  const uint32_t lane = lane_id();
  uint32_t held = 0;  // complement of this lane's keys
#pragma unroll
  for (uint32_t k = 2; k <= 32 * PER; k <<= 1) {
    if (k >= PER) {
      const uint32_t want = (lane * PER) & k ? 0xFFFFFFFFu : 0u;  // none in the last merge
      const uint32_t flip = (k < 32 * PER ? want : 0u) ^ held;
      held ^= flip;
#pragma unroll
      for (uint32_t j = 0; j < PER; ++j) key[j] ^= flip;
    }
#pragma unroll
    for (uint32_t d = k >> 1; d > 0; d >>= 1) {
      if (d >= PER) {
        const uint32_t ld = d / PER;  // partner lane distance
        const bool lower = (lane & ld) == 0;
#pragma unroll
        for (uint32_t j = 0; j < PER; ++j) {
          const uint32_t p = __shfl_xor_sync(0xFFFFFFFFu, key[j], ld);
          key[j] = (p < key[j]) == lower ? p : key[j];
        }
      } else {
#pragma unroll
        for (uint32_t j = 0; j < PER; ++j) {
          if (j & d) continue;
          const bool down = k < PER && (j & k);  // a block inside the lane
          const uint32_t lo = min(key[j], key[j + d]), hi = max(key[j], key[j + d]);
          key[j] = down ? hi : lo;
          key[j + d] = down ? lo : hi;
        }
      }
    }
  }
}

// Sorts a module's n (<= 32 * PER) staged clusters on (phi, LHCb id) into the compact layout
// by their short keys. Short keys that agree leave their clusters in slot order: the full keys
// of neighbours are compared on the way out, and false is returned when one pair stands the
// wrong way round (about one module in 400): the caller sorts that module on the full keys.
//
// Bound by the integer pipe: 32-bit keys take 3 instructions a key and exchange (shuffle,
// compare, select) where the full 64-bit keys took 9, and 256 of them fit the registers that
// held 128. Decode of 65,536 events at nu ~ U(2,20) 13.51 -> 11.24 ms.
template<uint32_t PER>
__device__ __forceinline__ bool sort_module_short(const float4* src, const uint32_t* src_id, uint32_t n, float4* dst,
                                                  uint32_t* dst_id, uint8_t* dst_size)
{
  const uint32_t lane = lane_id();
  uint32_t key[PER];
#pragma unroll
  for (uint32_t j = 0; j < PER; ++j) {  // coalesced loads
    const uint32_t i = j * 32 + lane;
    key[j] = i < n ? short_key<PER>(src[i].w, i) : 0xFFFFFFFFu;
  }
  warp_register_sort<PER>(key);
  bool wrong = false;
  unsigned long long first = 0, prev = 0;  // full keys without the slot
#pragma unroll
  for (uint32_t j = 0; j < PER; ++j) {
    const uint32_t i = lane * PER + j;  // rank of key[j]
    unsigned long long full = ~0ull;
    if (i < n) {
      const uint32_t from = key[j] & (32 * PER - 1);
      const uint32_t id = src_id[from];
      const float4 c = src[from];
      dst[i] = c;
      dst_id[i] = id & ~kSizeMask;
      dst_size[i] = static_cast<uint8_t>(id >> kSizeShift) & 3u;
      full = (static_cast<unsigned long long>(orderable(c.w)) << 32) | (id & 0xFFFFFu);
    }
    if (j == 0) first = full;
    else wrong |= full < prev;
    prev = full;
  }
  const unsigned long long next = __shfl_down_sync(0xFFFFFFFFu, first, 1);
  wrong |= lane < 31 && next < prev;
  return !__any_sync(0xFFFFFFFFu, wrong);
}

// Bitonic sort of `size` keys (power of two) in shared memory by one warp.
__device__ __forceinline__ void warp_smem_sort(unsigned long long* key, uint32_t size)
{
  const uint32_t lane = lane_id();
  for (uint32_t k = 2; k <= size; k <<= 1) {
    for (uint32_t j = k >> 1; j > 0; j >>= 1) {
      for (uint32_t i = lane; i < size; i += 32) {
        const uint32_t ixj = i ^ j;
        if (ixj > i) {
          const unsigned long long a = key[i], b = key[ixj];
          if ((a > b) == ((i & k) == 0)) {
            key[i] = b;
            key[ixj] = a;
          }
        }
      }
      __syncwarp();
    }
  }
}

// Phi windows of the h1 of one module, after the event's modules are sorted
// (fill_candidates, FillCandidates.cu:8-70, VeloTools.cuh:6-42): for each hit h1 of module m
// (2..49) the hits within kPhiExtrapolation of phi(h1) in module m + 2 (h0) and m - 2 (h2),
// as event-relative u16 pairs {first | last << 16} (0xFFFF: none). `sphi` holds the modules'
// phi, module m's from mphi[m] on (null: read the cluster records). In the pruned mode also the scorer's
// inputs: keep bits (3: seeding candidate, verdict to come; 2: no seed) and, for each
// candidate the gates admit, an 8-byte record (event hit base, h1 | m << 16) appended to the
// candidate list (queue slot 7). One warp per module; every lane takes part in each 32-hit
// round (ballots). Bound by the integer pipe: the branch-free searches took decode of 65,536
// events at nu ~ U(2,20) from 11.24 to 10.80 ms.
template<bool kPruned>
__device__ __forceinline__ void module_windows(const ChainPointers& P, const float* sphi, const uint32_t* mphi,
                                               const float4* H, uint2* Wn,
                                               uint8_t* K, uint32_t base, uint32_t m, const uint32_t* mstart,
                                               const uint32_t* mcount, bool score)
{
  const uint32_t lane = lane_id();
  const uint32_t s1 = mstart[m], n1 = mcount[m];
  const uint32_t s0 = mstart[m + 2], n0 = mcount[m + 2], s2 = mstart[m - 2], n2 = mcount[m - 2];
  for (uint32_t r0 = 0; r0 < n1; r0 += 32) {
    const uint32_t r = r0 + lane;
    const bool valid = r < n1;
    const uint32_t h = s1 + r;
    int f0 = -1, l0 = -1, f2 = -1, l2 = -1;
    if (valid) {
      if (sphi) {
        const float p = sphi[mphi[m] + r];
        if (n0 > 0) phi_window_flat(sphi + mphi[m + 2], n0, p, kPhiExtrapolation, f0, l0);
        if (n2 > 0) phi_window_flat(sphi + mphi[m - 2], n2, p, kPhiExtrapolation, f2, l2);
        if (f0 != -1) {
          f0 += s0;
          l0 += s0;
        }
        if (f2 != -1) {
          f2 += s2;
          l2 += s2;
        }
      } else {
        const float p = H[h].w;
        if (n0 > 0) phi_window4(H, s0, n0, p, kPhiExtrapolation, f0, l0);
        if (n2 > 0) phi_window4(H, s2, n2, p, kPhiExtrapolation, f2, l2);
      }
      Wn[h] = make_uint2((static_cast<uint32_t>(f0) & 0xFFFFu) | (static_cast<uint32_t>(l0) << 16),
                         (static_cast<uint32_t>(f2) & 0xFFFFu) | (static_cast<uint32_t>(l2) << 16));
    }
    if (kPruned) {
      const bool cand = valid && f0 != -1 && f2 != -1;
      if (valid) K[h] = cand ? 3u : 2u;  // candidates: verdict from score_candidates
      // seeds whose pair loop is cheaper than their scoring stay kept, unscored
      const bool append = cand && score && static_cast<uint32_t>((l0 - f0) * (l2 - f2)) >= P.mlp.min_pairs;
      const uint32_t bal = __ballot_sync(0xFFFFFFFFu, append);
      uint32_t row0 = 0;
      if (lane == 0 && bal) row0 = atomicAdd(P.queue + 7, static_cast<uint32_t>(__popc(bal)));
      row0 = __shfl_sync(0xFFFFFFFFu, row0, 0);
      if (append) P.cand_rec[row0 + __popc(bal & ((1u << lane) - 1u))] = make_uint2(base, h | (m << 16));
    }
  }
}

// The block's lists, then its sort buffers (one a warp), then the event's phi: never live
// together. Dynamic shared memory: 16 warps need 64 KB.
template<int W>
union DecodeLists {
  struct {
    uint32_t cand[kCandCap];      // flat SP index << 12 | bank << 4 | pixel
    uint32_t noniso[kNonIsoCap];  // non-isolated SPs: bank << 16 | flat SP index
  } lists;
  unsigned long long key[W][kSortCap];
};

// 40 warps per SM (5 blocks of 8): 48 registers, no spills (6 blocks at 40 registers: 10.5
// instead of 10.0 ms for 65,536 events). Bound by the integer pipe and issue; a batch of at most
// kDecodeWide events per SM, which leaves the device idle, takes 16 warps an event (10 events at
// nu ~ U(2,15) 92 -> 60 us, 148 100 -> 66, 290 133 -> 90; two such blocks fill an SM). kPruned:
// the windows pass also prepares the learned scorer's candidate list.
constexpr uint32_t kDecodeWide = 2;

template<int W, bool kPruned>
__global__ void __launch_bounds__(W * 32, 40 / W) decode_cluster_sort_kernel(ChainPointers P)
{
  __shared__ DecodeShared sh;
  extern __shared__ __align__(16) uint8_t s_dyn[];
  DecodeLists<W>& su = *reinterpret_cast<DecodeLists<W>*>(s_dyn);
  const uint32_t warp = threadIdx.x >> 5, lane = lane_id();

  for (;;) {
    if (threadIdx.x == 0) {
      // the event of this pass and its raw bytes, for the whole block
      const uint32_t e = atomicAdd(P.queue + 0, 1u);
      const RunParams& R = *P.run;
      sh.event = e;
      sh.n_events = R.n_events;
      if (e < R.n_events) {
        uint32_t src = e;  // raw event of this position
        uint32_t skipped = 0;
        if (P.event_list) {  // the global event cut of this chain
          if (e < *P.n_selected) src = P.event_list[e];
          else skipped = 1;
        } else if (R.event_list) {  // a selection made by the caller
          src = R.event_list[e];
          if (src >= R.n_raw) skipped = 2;
        }
        sh.skipped = skipped;
        sh.ev_off = skipped ? 0 : raw_offset(R, src);
        sh.ev_bytes = skipped ? 0 : raw_offset(R, src + 1) - sh.ev_off;
      }
      sh.flags = 0;
      sh.n_candidates = 0;
      sh.n_list = 0;
      sh.n_noniso = 0;
    }
    if (threadIdx.x < (kSensors + 31) / 32) sh.unsorted[threadIdx.x] = 0;
    if (threadIdx.x < kModules) sh.mod_count[threadIdx.x] = 0;
    __syncthreads();
    const uint32_t e = sh.event;
    if (e >= sh.n_events) break;
    const uint32_t skipped = sh.skipped;
    const uint64_t off = sh.ev_off;
    const uint64_t bytes = sh.ev_bytes;
    const uint32_t* ev = reinterpret_cast<const uint32_t*>(P.run->raw + off);
    const uint64_t words = bytes / 4;
    const uint32_t header = 2 + kSensors;  // number_of_raw_banks + raw_bank_offset[209]
    // ---- validate the raw event and index its banks ----
    // a batch may start anywhere in the caller's buffer: check the address itself
    const bool bad_header = (reinterpret_cast<uintptr_t>(ev) & 3) || words < header + 1 ||
                            off / 4 + words > P.hit_capacity || __ldg(ev) != kSensors;
    if (!bad_header) {
      const uint64_t payload_bytes = (words - header) * 4;
      for (uint32_t b = threadIdx.x; b < kSensors; b += blockDim.x) {
        const uint32_t o = __ldg(ev + 1 + b), o1 = __ldg(ev + 2 + b);
        bool ok = !(o & 3) && o1 >= o + 8 && o1 <= payload_bytes;
        uint32_t sensor = 0, count = 0;
        if (ok) {
          sensor = __ldg(ev + header + o / 4);
          count = __ldg(ev + header + o / 4 + 1);
          ok = sensor == b && 8ull + 4ull * count <= static_cast<uint64_t>(o1 - o);
        }
        if (!ok) {
          atomicOr(&sh.flags, kStatusBadRawEvent);
          count = 0;
        }
        sh.bank_start[b] = header + o / 4 + 2;
        sh.bank_count[b] = count;
        sh.bank_sensor[b] = sensor;
        if (count > 256) atomicOr(&sh.flags, kStatusBigSpIndex);
      }
    } else if (threadIdx.x == 0) {
      atomicOr(&sh.flags, skipped == 1 ? kStatusNotSelected : kStatusBadRawEvent);
    }
    __syncthreads();
    const bool event_ok = !(sh.flags & (kStatusBadRawEvent | kStatusNotSelected));
    if (!event_ok)
      for (uint32_t b = threadIdx.x; b <= kSensors; b += blockDim.x) sh.sp_prefix[b] = 0;
    // ---- bank prefix (warp 0) ----
    if (event_ok) {
      if (warp == 0) {
        uint32_t carry = 0;
        for (uint32_t b0 = 0; b0 < kSensors; b0 += 32) {
          const uint32_t b = b0 + lane;
          const uint32_t v = b < kSensors ? sh.bank_count[b] : 0;
          uint32_t incl = v;
#pragma unroll
          for (int o = 1; o < 32; o <<= 1) {
            const uint32_t t = __shfl_up_sync(0xFFFFFFFFu, incl, o);
            if (lane >= static_cast<uint32_t>(o)) incl += t;
          }
          if (b < kSensors) sh.sp_prefix[b] = carry + incl - v;
          carry += __shfl_sync(0xFFFFFFFFu, incl, 31);
        }
        if (lane == 0) sh.sp_prefix[kSensors] = carry;
      }
    }
    __syncthreads();
    const uint32_t total_sp = sh.sp_prefix[kSensors];
    const uint32_t base = static_cast<uint32_t>(off / 4);
    const DecodeEvent d{ev, 2 * base, P.stage.xyzp, P.stage.id};
    // ---- pass 1, one pass over the flat SP index: the sortedness of each bank, and the clusters of the isolated SPs from the pattern table (they need neither);
    // the non-isolated SPs are listed for pass 2. Every thread's loads are independent, so
    // the first touches of the raw event overlap instead of queueing bank by bank ----
    const bool can_list = total_sp <= 0x10000u;  // list entries are 16-bit
    if (event_ok) {
      // each warp takes one run of the index, so that a lane finds its bank from the one before
      // instead of by a search over the 208 (decode of 65,536 events 10.80 -> 10.58 ms)
      const uint32_t run = (total_sp + 32 * W - 1) / (32 * W) * 32;
      const uint32_t f_end = min(total_sp, (warp + 1) * run);
      uint32_t b = warp * run < f_end ? bank_of(sh, warp * run) : 0u;
      for (uint32_t f = warp * run + lane; f < f_end; f += 32) {
        while (sh.sp_prefix[b + 1] <= f) ++b;
        const uint32_t s = f - sh.sp_prefix[b];
        const uint32_t* bank = ev + sh.bank_start[b];
        const uint32_t word = __ldg(bank + s);
        if (s > 0 && sp_addr(word) < sp_addr(__ldg(bank + s - 1))) atomicOr(&sh.unsorted[b >> 5], 1u << (b & 31));
        if (sp_isolated(word)) {
          // pattern table (MaskedVeloClustering.cu:105-167)
          const uint32_t sp = sp_mask(word);
          const int32_t sp_r = sp_row(word), sp_c = sp_col(word);
          const uint32_t chip = sp_c / (kChipColumns / 2);
          const uint32_t sensor = sh.bank_sensor[b];
          for (int c = 0; c < 2; ++c) {
            const uint4 v = __ldg(reinterpret_cast<const uint4*>(P.k.sp + 2 * sp + c));
            const uint32_t cx = sp_c * 2 + ((v.z >> 2) & 1u);
            const uint32_t cy = sp_r * 4 + (v.z & 3u);
            stage_cluster(sh, d, b >> 2,
                          place_cluster(P.k, sensor, cx, cy, __uint_as_float(v.x), __uint_as_float(v.y), chip),
                          (v.z >> 4) & 0xFu);
            if (!(v.z & 8u)) break;
          }
        } else if (can_list) {
          const uint32_t q = atomicAdd(&sh.n_noniso, 1u);
          if (q < kNonIsoCap) su.lists.noniso[q] = (b << 16) | f;
        }
      }
    }
    __syncthreads();
    // ---- pass 2: candidate search of the non-isolated SPs (from the list, or every SP when
    // the list overflowed) ----
    uint32_t my_cands = 0;
    const bool listed = can_list && sh.n_noniso <= kNonIsoCap;
    const uint32_t n_scan = listed ? sh.n_noniso : total_sp;
    for (uint32_t i = threadIdx.x; i < n_scan; i += blockDim.x) {
      const uint32_t f = listed ? su.lists.noniso[i] & 0xFFFFu : i;
      const uint32_t b = listed ? su.lists.noniso[i] >> 16 : bank_of(sh, f);
      const uint32_t s = f - sh.sp_prefix[b];
      const uint32_t* bank = ev + sh.bank_start[b];
      const uint32_t word = __ldg(bank + s);
      if (sp_isolated(word)) continue;  // emitted in pass 1
      const uint32_t sp = sp_mask(word);
      const int32_t sp_r = sp_row(word), sp_c = sp_col(word);
      const bool sorted = !((sh.unsorted[b >> 5] >> (b & 31)) & 1u);
      const uint32_t code = window_candidate_code(sp, gather_window(bank, sh.bank_count[b], sorted, sp_r, sp_c));
      for (int half = 0; half < 2; ++half) {
        const uint32_t nib = half ? code >> 4 : code & 0xFu;
        if (!nib) continue;
        ++my_cands;
        const uint32_t k = candidate_k(nib) + 2 * half;
        const uint32_t slot = atomicAdd(&sh.n_list, 1u);
        if (slot < kCandCap && f < (1u << 20)) su.lists.cand[slot] = (f << 12) | (b << 4) | k;
        else {
          if (slot < kCandCap) su.lists.cand[slot] = kNoCandidate;
          flood_candidate(sh, d, P.k, f, b, k);
        }
      }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) my_cands += __shfl_xor_sync(0xFFFFFFFFu, my_cands, o);
    if (lane == 0 && my_cands) atomicAdd(&sh.n_candidates, my_cands);
    __syncthreads();
    // ---- pass 3: flood fill of the listed candidates ----
    const uint32_t n_list = min(sh.n_list, kCandCap);
    for (uint32_t i = threadIdx.x; i < n_list; i += blockDim.x) {
      const uint32_t c = su.lists.cand[i];
      if (c != kNoCandidate) flood_candidate(sh, d, P.k, c >> 12, (c >> 4) & 0xFFu, c & 0xFu);
    }
    __syncthreads();
    // ---- compact layout: exclusive scan of the module counts ----
    if (warp == 0) {
      const uint32_t a = lane < kModules ? sh.mod_count[lane] : 0;
      const uint32_t a2 = lane + 32 < kModules ? sh.mod_count[lane + 32] : 0;
      uint32_t ia = a, ib = a2;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t va = __shfl_up_sync(0xFFFFFFFFu, ia, o), vb = __shfl_up_sync(0xFFFFFFFFu, ib, o);
        if (lane >= static_cast<uint32_t>(o)) {
          ia += va;
          ib += vb;
        }
      }
      const uint32_t first_half = __shfl_sync(0xFFFFFFFFu, ia, 31);
      if (lane < kModules) sh.mod_start[lane] = ia - a;
      if (lane + 32 < kModules) sh.mod_start[lane + 32] = first_half + ib - a2;
      const uint32_t total = first_half + __shfl_sync(0xFFFFFFFFu, ib, 31);
      if (lane == 0) {
        uint32_t fl = 0;
        // the event's hit region is its raw word range: one hit per raw word
        if (total > words) fl |= kStatusHitOverflow;
        if (sh.n_candidates > kMaxCandidatesEvent) fl |= kStatusCandidateOverflow;
        if (fl) atomicOr(&sh.flags, fl);
      }
    }
    __syncthreads();
    const bool write = event_ok && !(sh.flags & kStatusHitOverflow);
    // ---- per-module sort on (phi, LHCb id) into the compact layout ----
    for (uint32_t m = warp; m < kModules; m += W) {
      const uint32_t n = write ? sh.mod_count[m] : 0;
      const uint32_t p0 = base + sh.mod_start[m];
      const float4* src = d.stage + d.stage_base + 2 * sh.sp_prefix[4 * m];
      const uint32_t* src_id = d.stage_id + d.stage_base + 2 * sh.sp_prefix[4 * m];
      float4* dst = P.hits.xyzp + p0;
      uint32_t* dst_id = P.hits.id + p0;
      uint8_t* dst_size = P.hit_size + p0;
      if (n > kMaxHitsPerModule && lane == 0) atomicOr(&sh.flags, kStatusModuleOverflow);
      bool sorted = n == 0;
      if (n > 128 && n <= kRegSortMax) sorted = sort_module_short<8>(src, src_id, n, dst, dst_id, dst_size);
      else if (n > 64 && n <= 128) sorted = sort_module_short<4>(src, src_id, n, dst, dst_id, dst_size);
      else if (n > 32 && n <= 64) sorted = sort_module_short<2>(src, src_id, n, dst, dst_id, dst_size);
      else if (n > 0 && n <= 32) sorted = sort_module_short<1>(src, src_id, n, dst, dst_id, dst_size);
      if (sorted) {
        // in registers
      } else if (n <= kSortCap) {
        unsigned long long* key = su.key[warp];
        uint32_t size = 32;
        while (size < n) size <<= 1;
        __syncwarp();  // the short keys' order, if any, has been written
        for (uint32_t i = lane; i < size; i += 32) key[i] = i < n ? cluster_key(src, src_id, i) : ~0ull;
        __syncwarp();
        warp_smem_sort(key, size);
        for (uint32_t i = lane; i < n; i += 32) {
          const uint32_t from = static_cast<uint32_t>(key[i] & 0xFFFu);
          const uint32_t id = src_id[from];
          dst[i] = src[from];
          dst_id[i] = id & ~kSizeMask;
          dst_size[i] = static_cast<uint8_t>(id >> kSizeShift) & 3u;
        }
        __syncwarp();
      } else {
        // beyond the reference's 500-cluster module buffer (flagged above): kept unsorted
        for (uint32_t i = lane; i < n; i += 32) {
          dst[i] = src[i];
          dst_id[i] = src_id[i] & ~kSizeMask;
          dst_size[i] = static_cast<uint8_t>(src_id[i] >> kSizeShift) & 3u;
        }
      }
      if (lane == 0) {
        P.module_start[e * kModules + m] = p0;
        P.module_num[e * kModules + m] = n;
      }
    }
    __syncthreads();
    // ---- phi windows of every h1 (fill_candidates), while the event is in L2: the sorted phi
    // are read back into the shared memory the lists and sort buffers no longer need ----
    {
      const uint32_t nh = write ? sh.mod_start[kModules - 1] + sh.mod_count[kModules - 1] : 0;
      if (nh > 0 && nh <= kEventHitCap) {  // the events the search runs
        const float4* H = P.hits.xyzp + base;
        // A window joins modules of one parity, so an event whose phi do not fit the shared
        // memory takes the even modules first, then the odd ones; what does not fit then either
        // searches the cluster records.
        constexpr uint32_t kPhiCap = sizeof(DecodeLists<W>) / sizeof(float);
        const bool whole = nh <= kPhiCap;
        if (!whole && threadIdx.x < 2) {
          uint32_t n = 0;
          for (uint32_t m = threadIdx.x; m < kModules; m += 2) {
            sh.mod_phi[m] = n;
            n += sh.mod_count[m];
          }
        }
        bool score = false;
        uint8_t* K = nullptr;
        if (kPruned) {
          K = P.keep + base;
          const bool fallback = nh > P.mlp.max_hits;  // above the trained occupancy: plain search
          if (fallback && threadIdx.x == 0) sh.flags |= kStatusMlpFallback;
          score = !fallback && nh >= P.mlp.min_hits;
          if (score) {
            // modules 0, 1, 50, 51 hold no h1: extension candidates only
            for (uint32_t h = threadIdx.x; h < sh.mod_start[2]; h += blockDim.x) K[h] = 2;
            for (uint32_t h = sh.mod_start[50] + threadIdx.x; h < nh; h += blockDim.x) K[h] = 2;
          } else {
            // an event the scorer does not score: every seed kept, its windows as in the
            // plain mode (the branch is uniform over the block)
            for (uint32_t h = threadIdx.x; h < nh; h += blockDim.x) K[h] = 3;
          }
        }
        for (uint32_t half = 0; half < (whole ? 1u : 2u); ++half) {
          float* sphi = reinterpret_cast<float*>(&su);
          const uint32_t* mphi = whole ? sh.mod_start : sh.mod_phi;
          __syncthreads();  // mod_phi written; the half before searched
          if (whole) {
            for (uint32_t i = threadIdx.x; i < nh; i += blockDim.x) sphi[i] = H[i].w;
          } else if (mphi[kModules - 2 + half] + sh.mod_count[kModules - 2 + half] <= kPhiCap) {
            for (uint32_t m = half + 2 * warp; m < kModules; m += 2 * W)
              for (uint32_t i = lane; i < sh.mod_count[m]; i += 32) sphi[mphi[m] + i] = H[sh.mod_start[m] + i].w;
          } else {
            sphi = nullptr;
          }
          __syncthreads();
          const uint32_t first = 2 + (whole ? warp : half + 2 * warp), step = whole ? W : 2 * W;
          bool scored = false;
          if constexpr (kPruned) {
            if (score) {
              for (uint32_t m = first; m < 50; m += step)
                module_windows<true>(P, sphi, mphi, H, P.windows + base, K, base, m, sh.mod_start, sh.mod_count, true);
              scored = true;
            }
          }
          if (!scored)
            for (uint32_t m = first; m < 50; m += step)
              module_windows<false>(P, sphi, mphi, H, P.windows + base, K, base, m, sh.mod_start, sh.mod_count, false);
        }
      }
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      const uint32_t nhits = write ? sh.mod_start[kModules - 1] + sh.mod_count[kModules - 1] : 0;
      P.event_hit_base[e] = base;
      P.event_hits[e] = nhits;
      P.status[e] = sh.flags;
    }
    __syncthreads();
  }
}

}  // namespace velo
