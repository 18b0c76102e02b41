// cluster_select.cuh -- exact k-th smallest of up to 8192 kPer values held in
// the registers of a cluster of eight 1024-thread CTAs.
//
// Radix selection on order-preserving keys in three passes (11, 11, 10 bits),
// equivalent to std::nth_element. A CTA re-reading its values from memory in
// four 8-bit passes was bound by those loads and by its one SM (437 us for the
// two selections among an NTSC field's 182,000 noise samples, 58 us among
// 26,000 envelope samples); here a value is read once, each CTA counts its own
// share, and the counts are added over the cluster through distributed shared
// memory.
#pragma once

#include <cooperative_groups.h>

#include "hvdg_common.cuh"

namespace hvdg {

constexpr int kSelCtas = 8;
constexpr int kSelThreads = 1024;
constexpr int kSelBins = 2048;

struct SelScratch {
  unsigned hist[kSelBins];  // this CTA's counts (read by the whole cluster)
  unsigned tot[kSelBins];   // the cluster's
  unsigned wsum[kSelThreads / 32];
  unsigned bin, rank;
};

// Thread t of a CTA holds key[q] of its elements t + 1024 q < count. All
// threads of the cluster call with the same k (0-based rank over the cluster).
template <int kPer>
__device__ __forceinline__ float cluster_select(const uint32_t (&key)[kPer], int count, unsigned k,
                                                SelScratch& s) {
  namespace cg = cooperative_groups;
  cg::cluster_group cl = cg::this_cluster();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const unsigned me = cl.block_rank();
  uint32_t prefix = 0, mask = 0;
#pragma unroll 1
  for (int shift = 21; shift >= 0; shift = shift == 21 ? 10 : shift == 10 ? 0 : -1) {
    const unsigned digit = shift == 0 ? 1023u : 2047u;
    s.hist[tid] = 0;
    s.hist[tid + kSelThreads] = 0;
    __syncthreads();
#pragma unroll
    for (int q = 0; q < kPer; ++q)
      if (tid + q * kSelThreads < count && (key[q] & mask) == prefix)
        atomicAdd(&s.hist[(key[q] >> shift) & digit], 1u);
    cl.sync();
    // CTA r adds the counts of bins 256 r .. 256 r + 255 and tells all
    if (tid < kSelBins / kSelCtas) {
      const int b = (int)me * (kSelBins / kSelCtas) + tid;
      unsigned t = 0;
#pragma unroll
      for (int r = 0; r < kSelCtas; ++r) t += *cl.map_shared_rank(&s.hist[b], r);
#pragma unroll
      for (int r = 0; r < kSelCtas; ++r) *cl.map_shared_rank(&s.tot[b], r) = t;
    }
    cl.sync();
    // the bin holding rank k: thread t owns bins 2 t, 2 t + 1
    const unsigned c0 = s.tot[2 * tid], pair = c0 + s.tot[2 * tid + 1];
    unsigned incl = pair;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned v = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += v;
    }
    if (lane == 31) s.wsum[warp] = incl;
    __syncthreads();
    unsigned base = lane < warp ? s.wsum[lane] : 0u;
    base = __reduce_add_sync(0xffffffffu, base);
    const unsigned excl = base + incl - pair;
    if (excl <= k && k < excl + pair) {
      const bool hi = k >= excl + c0;
      s.bin = 2 * tid + hi;
      s.rank = k - excl - (hi ? c0 : 0u);
    }
    __syncthreads();
    prefix |= s.bin << shift;
    mask |= digit << shift;
    k = s.rank;
  }
  return key_float(prefix);
}

}  // namespace hvdg
