// csort.cuh — stable radix sort by one cluster of CTAs (device parts).
//
// Up to CS_MAX CTAs of 1,024 threads sort in one launch: a pass counts the
// digits of the CTA's chunk a warp, exchanges the chunk totals through
// distributed shared memory and scatters; the cluster's barrier stands where
// launches stood.  A chunk's warps own contiguous runs and walk them 32 keys
// at a time, ranks inside a step come from __match_any_sync, so equal keys
// keep their order.  Every key is read by two passes of the chip's caches;
// what bounds a pass is latency: two cluster barriers, the exchange and the
// step loop.
#pragma once
#include <cooperative_groups.h>

#include "common.cuh"

#ifdef __CUDACC__
namespace rtr {

constexpr int CS_THREADS = 1024;
constexpr int CS_WARPS = CS_THREADS / 32;
constexpr int CS_RADIX = 256;
constexpr int CS_MAX = 16;  // CTAs (more than 8: where the device has room for such a cluster)

struct CsShared {
  uint32_t wcnt[CS_WARPS][CS_RADIX];  // a warp's count of each digit, then its next output slot in the chunk
  uint32_t hist[CS_RADIX];            // the chunk's count of each digit (read by the other CTAs)
  uint32_t boff[CS_RADIX];            // output offset of the chunk's first key of each digit
  uint32_t ws[CS_RADIX / 32];
};

struct CsChunk {
  int n, steps, beg;  // items; steps of 32 a warp; this warp's first item
  __device__ CsChunk(int n_, int rank, int ctas) {
    n = n_;
    steps = ((n + ctas - 1) / ctas + CS_THREADS - 1) / CS_THREADS;
    beg = (rank * CS_WARPS + (int)(threadIdx.x >> 5)) * steps * 32;
  }
};

// Digit counts of this CTA's chunk; key(i) gives item i's key.
template <class Key>
__device__ __forceinline__ void cs_count(CsShared& s, const CsChunk& c, int shift, Key key) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int i = threadIdx.x; i < CS_WARPS * CS_RADIX; i += CS_THREADS) (&s.wcnt[0][0])[i] = 0u;
  __syncthreads();
#pragma unroll 4
  for (int j = 0; j < c.steps; ++j) {
    const int i = c.beg + j * 32 + lane;
    if (i < c.n) atomicAdd(&s.wcnt[warp][(key(i) >> shift) & (CS_RADIX - 1)], 1u);
  }
  __syncthreads();
}

// From the counts to output slots: s.boff and, per warp, s.wcnt.  Holds one
// cluster barrier.
__device__ __forceinline__ void cs_offsets(CsShared& s, cooperative_groups::cluster_group cl) {
  const int d = threadIdx.x, lane = d & 31, warp = d >> 5;
  if (d < CS_RADIX) {
    uint32_t run = 0;
#pragma unroll
    for (int w = 0; w < CS_WARPS; ++w) {
      const uint32_t t = s.wcnt[w][d];
      s.wcnt[w][d] = run;
      run += t;
    }
    s.hist[d] = run;
  }
  cl.sync();
  uint32_t tot = 0, pre = 0, inc = 0;
  if (d < CS_RADIX) {
    const unsigned ctas = cl.num_blocks(), rank = cl.block_rank();
#pragma unroll
    for (unsigned r = 0; r < CS_MAX; ++r) {
      const uint32_t h = r < ctas ? cl.map_shared_rank(s.hist, r)[d] : 0u;
      tot += h;
      pre += r < rank ? h : 0u;
    }
    inc = tot;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t v = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= o) inc += v;
    }
    if (lane == 31) s.ws[warp] = inc;
  }
  __syncthreads();
  if (d < CS_RADIX) {
    uint32_t wpre = 0;
#pragma unroll
    for (int w = 0; w < CS_RADIX / 32; ++w) wpre += w < warp ? s.ws[w] : 0u;
    s.boff[d] = wpre + inc - tot + pre;
  }
  __syncthreads();
}

// Scatter of this CTA's chunk; vin NULL: the item's index.  Ends with a
// cluster barrier (the output is complete, the counts may be reused).
__device__ __forceinline__ void cs_scatter(CsShared& s, const CsChunk& c, int shift, const uint32_t* kin,
                                           const uint32_t* vin, uint32_t* kout, uint32_t* vout,
                                           cooperative_groups::cluster_group cl) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const unsigned lt = lanemask_lt();
  for (int j0 = 0; j0 < c.steps; j0 += 4) {
    uint32_t k[4], v[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int i = c.beg + (j0 + j) * 32 + lane;
      const bool in = j0 + j < c.steps && i < c.n;
      k[j] = in ? __ldcg(kin + i) : 0u;  // (written by other SMs of the cluster: not through L1)
      v[j] = in && vin ? __ldcg(vin + i) : (uint32_t)i;
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      if (j0 + j >= c.steps) break;
      const int i = c.beg + (j0 + j) * 32 + lane;
      const bool in = i < c.n;
      const uint32_t d = in ? (k[j] >> shift) & (CS_RADIX - 1) : CS_RADIX;
      const unsigned peers = __match_any_sync(0xffffffffu, d);
      const uint32_t at = in ? s.wcnt[warp][d] : 0u;
      __syncwarp();
      if (in && (peers & lt) == 0u) s.wcnt[warp][d] = at + __popc(peers);
      __syncwarp();
      if (in) {
        const uint32_t pos = s.boff[d] + at + __popc(peers & lt);
        kout[pos] = k[j];
        vout[pos] = v[j];
      }
    }
  }
  cl.sync();
}

}  // namespace rtr
#endif
