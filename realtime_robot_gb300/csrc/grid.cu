// grid.cu — stable LSD radix sort and the uniform-grid build (counted into place).
#include <math.h>

#include "csort.cuh"
#include "grid.cuh"

namespace rtr {

constexpr int RS_BLOCK = 256;
constexpr int RS_WARPS = RS_BLOCK / 32;
constexpr int RS_ITEMS = 16;
constexpr int RS_TILE = RS_BLOCK * RS_ITEMS;  // 4096 keys per block
constexpr int RS_RADIX = 256;
constexpr int RS_CLUSTER_MAX = 131072;  // items that one cluster sorts in a launch (more: a grid, two launches a pass)
constexpr int RS_CLUSTER_ITEMS = 1024;   // items a CTA before the cluster grows

__device__ __forceinline__ int count_of(int n_host, const int* d_n) { return d_n ? *d_n : n_host; }

// Sorts of at most this many tiles skip the scan kernel: each scatter block
// sums the tile-major histogram itself (nb rows of 1 KB from L2).
constexpr int RS_FUSE_TILES = 128;

// Per-tile digit histogram, written digit-major, hist[d * nb + tile], or
// tile-major, hist[tile * 256 + d] (TILE_MAJOR, read by k_rs_scatter_own).
template <bool TILE_MAJOR>
__global__ void __launch_bounds__(RS_BLOCK) k_rs_hist(const uint32_t* __restrict__ keys, int n_host,
                                                      const int* d_n, int shift,
                                                      uint32_t* __restrict__ hist, int nb) {
  __shared__ uint32_t cnt[RS_RADIX];
  const int n = count_of(n_host, d_n);
  for (int i = threadIdx.x; i < RS_RADIX; i += RS_BLOCK) cnt[i] = 0;
  __syncthreads();
  const int base = blockIdx.x * RS_TILE;
  uint32_t k[RS_ITEMS];  // all loads in flight before the first count (300k keys: 6.6 -> 3.1 us a pass)
#pragma unroll
  for (int j = 0; j < RS_ITEMS; ++j) {
    const int i = base + j * RS_BLOCK + threadIdx.x;
    k[j] = i < n ? keys[i] : 0u;
  }
#pragma unroll
  for (int j = 0; j < RS_ITEMS; ++j)
    if (base + j * RS_BLOCK + (int)threadIdx.x < n) atomicAdd(&cnt[(k[j] >> shift) & (RS_RADIX - 1)], 1u);
  __syncthreads();
  for (int d = threadIdx.x; d < RS_RADIX; d += RS_BLOCK)
    hist[TILE_MAJOR ? blockIdx.x * RS_RADIX + d : d * nb + blockIdx.x] = cnt[d];
}

// In-place exclusive scan of `total` entries by one block of 1024 threads,
// in chunks of 8192 entries staged through shared memory with coalesced
// loads and stores (eight per thread), a carry between chunks.
__global__ void __launch_bounds__(1024) k_rs_scan(uint32_t* __restrict__ h, int total) {
  constexpr int PER = 8, CH = 1024 * PER;
  __shared__ uint32_t sh[CH];
  __shared__ uint32_t wsum[32];
  __shared__ uint32_t s_carry;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (threadIdx.x == 0) s_carry = 0;
  for (int c0 = 0; c0 < total; c0 += CH) {
    const int cn = min(CH, total - c0);
#pragma unroll
    for (int k = 0; k < PER; ++k) {
      const int i = k * 1024 + threadIdx.x;
      sh[i] = i < cn ? h[c0 + i] : 0u;
    }
    __syncthreads();
    // thread t owns sh[t*PER .. t*PER+PER)
    uint32_t v[PER], s = 0;
#pragma unroll
    for (int k = 0; k < PER; ++k) {
      v[k] = sh[threadIdx.x * PER + k];
      s += v[k];
    }
    uint32_t incl = s;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t t = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += t;
    }
    if (lane == 31) wsum[warp] = incl;
    __syncthreads();
    if (warp == 0) {
      const uint32_t w = wsum[lane];
      uint32_t wi = w;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t t = __shfl_up_sync(0xffffffffu, wi, o);
        if (lane >= o) wi += t;
      }
      wsum[lane] = wi - w;
    }
    __syncthreads();
    uint32_t run = s_carry + wsum[warp] + incl - s;
#pragma unroll
    for (int k = 0; k < PER; ++k) {
      sh[threadIdx.x * PER + k] = run;
      run += v[k];
    }
    __syncthreads();
    if (threadIdx.x == 1023) s_carry = run;  // the last thread ends with the chunk's total
#pragma unroll
    for (int k = 0; k < PER; ++k) {
      const int i = k * 1024 + threadIdx.x;
      if (i < cn) h[c0 + i] = sh[i];
    }
    __syncthreads();
  }
}

// This block's output offset of each digit from the tile-major histogram:
// the keys of smaller digits in every tile plus those of the same digit in
// earlier tiles (thread d owns digit d; a block-wide exclusive scan of the
// digit totals).
__device__ __forceinline__ void rs_own_offsets(const uint32_t* __restrict__ hist, int nb, uint32_t* boff,
                                               uint32_t* wsum) {
  static_assert(RS_BLOCK == RS_RADIX, "one thread per digit");
  const int d = threadIdx.x, lane = d & 31, warp = d >> 5;
  const int b = blockIdx.x;
  uint32_t tot = 0, pre = 0;
  for (int t0 = 0; t0 < nb; t0 += 32) {  // 32 loads in flight (four at a time: 12.1 us a pass, now 11.4)
    uint32_t h[32];
#pragma unroll
    for (int k = 0; k < 32; ++k) h[k] = t0 + k < nb ? hist[(t0 + k) * RS_RADIX + d] : 0u;
#pragma unroll
    for (int k = 0; k < 32; ++k) {
      tot += h[k];
      pre += t0 + k < b ? h[k] : 0u;
    }
  }
  uint32_t inc = tot;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t v = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= o) inc += v;
  }
  if (lane == 31) wsum[warp] = inc;
  __syncthreads();
  uint32_t wpre = 0;
#pragma unroll
  for (int w = 0; w < RS_WARPS; ++w) wpre += w < warp ? wsum[w] : 0u;
  boff[d] = wpre + inc - tot + pre;
}

// Stable scatter.  Warp w of a block owns a contiguous run of RS_ITEMS*32 keys
// and walks it 32 at a time, so (warp, step, lane) is the input order; ranks
// inside a step come from __match_any_sync, so equal digits keep their order.
// OWN: the block computes its offsets from the tile-major histogram
// (rs_own_offsets); otherwise it reads them from the scanned digit-major one.
template <bool OWN>
__global__ void __launch_bounds__(RS_BLOCK) k_rs_scatter(const uint32_t* __restrict__ kin,
                                                         const uint32_t* __restrict__ vin,
                                                         uint32_t* __restrict__ kout,
                                                         uint32_t* __restrict__ vout, int n_host,
                                                         const int* d_n, int shift,
                                                         const uint32_t* __restrict__ hist, int nb) {
  __shared__ uint32_t wcnt[RS_WARPS][RS_RADIX];
  __shared__ uint32_t boff[RS_RADIX];
  __shared__ uint32_t wsum[RS_WARPS];
  const int n = count_of(n_host, d_n);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int i = threadIdx.x; i < RS_WARPS * RS_RADIX; i += RS_BLOCK) (&wcnt[0][0])[i] = 0;
  if (OWN) {
    if (blockIdx.x * RS_TILE >= n) return;  // whole tile empty (uniform per block)
    rs_own_offsets(hist, nb, boff, wsum);
  } else {
    for (int d = threadIdx.x; d < RS_RADIX; d += RS_BLOCK) boff[d] = hist[d * nb + blockIdx.x];
  }
  __syncthreads();
  const int base = blockIdx.x * RS_TILE + warp * (RS_ITEMS * 32);
  if (blockIdx.x * RS_TILE >= n) return;  // whole tile empty (uniform per block)
  const unsigned lt = lanemask_lt();
  uint32_t key[RS_ITEMS];
  uint32_t loc[RS_ITEMS];
#pragma unroll
  for (int j = 0; j < RS_ITEMS; ++j) {
    const int i = base + j * 32 + lane;
    key[j] = i < n ? kin[i] : 0u;
  }
#pragma unroll
  for (int j = 0; j < RS_ITEMS; ++j) {
    const int i = base + j * 32 + lane;
    const bool valid = i < n;
    const uint32_t k = key[j];
    const uint32_t d = valid ? ((k >> shift) & (RS_RADIX - 1)) : RS_RADIX;
    const unsigned peers = __match_any_sync(0xffffffffu, d);
    uint32_t before = valid ? wcnt[warp][d] : 0u;
    __syncwarp();
    if (valid && (peers & lt) == 0) wcnt[warp][d] = before + __popc(peers);
    __syncwarp();
    loc[j] = before + __popc(peers & lt);
  }
  __syncthreads();
  for (int d = threadIdx.x; d < RS_RADIX; d += RS_BLOCK) {
    uint32_t run = 0;
#pragma unroll
    for (int w = 0; w < RS_WARPS; ++w) {
      uint32_t t = wcnt[w][d];
      wcnt[w][d] = run;
      run += t;
    }
  }
  __syncthreads();
#pragma unroll
  for (int j = 0; j < RS_ITEMS; ++j) {
    const int i = base + j * 32 + lane;
    if (i < n) {
      const uint32_t d = (key[j] >> shift) & (RS_RADIX - 1);
      const uint32_t pos = boff[d] + wcnt[warp][d] + loc[j];
      kout[pos] = key[j];
      vout[pos] = vin ? vin[i] : (uint32_t)i;
    }
  }
}

// All passes by one cluster (csort.cuh).
__global__ void __launch_bounds__(CS_THREADS) k_rs_cluster(uint32_t* __restrict__ k0, uint32_t* __restrict__ v0,
                                                           uint32_t* __restrict__ k1, uint32_t* __restrict__ v1,
                                                           int n_host, const int* d_n, int passes, int iota) {
  __shared__ CsShared s;
  cooperative_groups::cluster_group cl = cooperative_groups::this_cluster();
  const CsChunk c(count_of(n_host, d_n), (int)cl.block_rank(), (int)cl.num_blocks());
  for (int p = 0; p < passes; ++p) {
    uint32_t* ki = p & 1 ? k1 : k0;
    uint32_t* vi = p & 1 ? v1 : v0;
    cs_count(s, c, 8 * p, [&](int i) { return __ldcg(ki + i); });
    cs_offsets(s, cl);
    cs_scatter(s, c, 8 * p, ki, p == 0 && iota ? nullptr : vi, p & 1 ? k0 : k1, p & 1 ? v0 : v1, cl);
  }
}

// Whether the current device schedules clusters of CS_MAX CTAs of this kernel
// (more than 8 is up to the device).
static bool cluster_max_ok(const void* kern, ClusterFit& fit) {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return false;
  int k = fit.known[dev].load(std::memory_order_relaxed);
  if (k == 0) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(CS_MAX);
    cfg.blockDim = dim3(CS_THREADS);
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = CS_MAX;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    int n = 0;
    const bool ok =
        cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess &&
        cudaOccupancyMaxActiveClusters(&n, kern, &cfg) == cudaSuccess && n > 0;
    if (!ok) cudaGetLastError();
    k = ok ? 2 : 1;
    fit.known[dev].store(k, std::memory_order_relaxed);
  }
  return k == 2;
}

// One cluster sorts up to RS_CLUSTER_MAX items in a launch (13 us for two
// passes of 2k items, 26 for four of 12k; a grid takes two launches a pass,
// 6.6 us each there).  Voxels and keypoints of a 123k-point scan: 767 us with
// the line at 32k items, 667 at 131k; the 300k-point room's recognition 3,210
// us with it there, 3,243 with the line beyond its points.  Clusters of at
// most 8 CTAs: the scan 727 us.
int cluster_sort_ctas(const rtr_context* ctx, int n_cap, const void* kern, ClusterFit& fit) {
  if (n_cap > RS_CLUSTER_MAX || (ctx && ctx->grid_sorts)) return 0;
  const int want = (n_cap + RS_CLUSTER_ITEMS - 1) / RS_CLUSTER_ITEMS;
  int c = 1;
  while (c < want && c < (c < 8 || cluster_max_ok(kern, fit) ? CS_MAX : 8)) c *= 2;
  return c;
}

int radix_hist_entries(int n_cap) {
  int nb = (n_cap + RS_TILE - 1) / RS_TILE;
  if (nb < 1) nb = 1;
  return nb * RS_RADIX;
}

rtr_status radix_sort_pairs(const rtr_context* ctx, uint32_t* k0, uint32_t* v0, uint32_t* k1, uint32_t* v1, uint32_t* hist,
                      int n_cap, int n_host, const int* d_n, int bits, bool vals_iota,
                      cudaStream_t st, uint32_t** k_out, uint32_t** v_out) {
  int nb = (n_cap + RS_TILE - 1) / RS_TILE;
  if (nb < 1) nb = 1;
  int passes = (bits + 7) / 8;
  if (passes < 1) passes = 1;
  static ClusterFit fit;
  const int ctas = cluster_sort_ctas(ctx, n_cap, reinterpret_cast<const void*>(k_rs_cluster), fit);
  if (ctas > 0) RTR_TRY(launch_cluster(k_rs_cluster, ctas, st, k0, v0, k1, v1, n_host, d_n, passes, (int)vals_iota));
  for (int p = 0; p < passes && ctas == 0; ++p) {
    const int shift = 8 * p;
    const bool even = (p & 1) == 0;
    uint32_t* ki = even ? k0 : k1;
    uint32_t* vi = even ? ((p == 0 && vals_iota) ? nullptr : v0) : v1;
    uint32_t* ko = even ? k1 : k0;
    uint32_t* vo = even ? v1 : v0;
    if (nb <= RS_FUSE_TILES) {
      k_rs_hist<true><<<nb, RS_BLOCK, 0, st>>>(ki, n_host, d_n, shift, hist, nb);
      k_rs_scatter<true><<<nb, RS_BLOCK, 0, st>>>(ki, vi, ko, vo, n_host, d_n, shift, hist, nb);
    } else {
      k_rs_hist<false><<<nb, RS_BLOCK, 0, st>>>(ki, n_host, d_n, shift, hist, nb);
      k_rs_scan<<<1, 1024, 0, st>>>(hist, nb * RS_RADIX);
      k_rs_scatter<false><<<nb, RS_BLOCK, 0, st>>>(ki, vi, ko, vo, n_host, d_n, shift, hist, nb);
    }
  }
  RTR_LAUNCHED(ctas > 0 ? 1 : (nb <= RS_FUSE_TILES ? 2 : 3) * passes);
  const bool odd = (passes & 1) != 0;
  *k_out = odd ? k1 : k0;
  *v_out = odd ? v1 : v0;
  RTR_CUDA(cudaGetLastError());
  return RTR_OK;
}

// ---------------------------------------------------------------------------
// grid build
// ---------------------------------------------------------------------------

// Origin, cell edge and dimensions from the bounding box (one thread).
__device__ void grid_setup(GridMeta* m, float h_req, unsigned cell_cap, int n) {
  float lo[3], hi[3];
  for (int a = 0; a < 3; ++a) {
    if (n > 0) {
      lo[a] = ordered_to_float(~__ldcg(&m->nmin[a]));
      hi[a] = ordered_to_float(__ldcg(&m->bmax[a]));
    } else {
      lo[a] = hi[a] = 0.f;
    }
    // non-finite coordinates (NaN / inf points) must not size the grid: such
    // points land in a clamped border cell and never match (d^2 is NaN/inf)
    if (!isfinite(lo[a]) || !isfinite(hi[a]) || !(hi[a] >= lo[a])) {
      lo[a] = isfinite(lo[a]) ? lo[a] : (isfinite(hi[a]) ? hi[a] : 0.f);
      hi[a] = isfinite(hi[a]) && hi[a] >= lo[a] ? hi[a] : lo[a];
    }
  }
  float h = h_req;
  if (!(h > 0.f)) {
    // automatic edge: twice the mean spacing of n points spread over the box
    double vol = 1.0;
    for (int a = 0; a < 3; ++a) vol *= fmax((double)(hi[a] - lo[a]), 1e-3);
    h = (float)(2.0 * cbrt(vol / (double)(n > 0 ? n : 1)));
  }
  int dims[3];
  for (int tries = 0; tries < 64; ++tries) {
    double cells = 1.0;
    for (int a = 0; a < 3; ++a) {
      double e = floor((double)(hi[a] - lo[a]) / (double)h) + 1.0;
      if (e > 2.0e9) e = 2.0e9;
      dims[a] = (int)e;
      cells *= e;
    }
    if (cells <= (double)cell_cap) break;
    h = (float)(h * cbrt(cells / (double)cell_cap) * 1.001);
  }
  m->ox = lo[0];
  m->oy = lo[1];
  m->oz = lo[2];
  m->h = h;
  m->inv_h = 1.0f / h;
  m->nx = dims[0];
  m->ny = dims[1];
  m->nz = dims[2];
  m->n = n;
  m->ncells = (unsigned)dims[0] * (unsigned)dims[1] * (unsigned)dims[2];
}

// Bounding box of the points into *m, which starts zeroed.  Launched with 256
// threads and at most bbox_blocks(n) blocks.  SETUP: the last block to finish
// also lays out the grid, which saves a launch.
template <bool SETUP>
__global__ void __launch_bounds__(256) k_bbox(const float4* __restrict__ pts, int n_host,
                                              const int* d_n, GridMeta* m, float h_req, unsigned cell_cap) {
  const int n = count_of(n_host, d_n);
  unsigned mn[3] = {0u, 0u, 0u}, mx[3] = {0u, 0u, 0u};  // largest complement, largest
#pragma unroll 4
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    float4 p = pts[i];
    // a point with a non-finite coordinate does not size the grid: it sits in
    // a clamped border cell and never matches (its d^2 is NaN or inf)
    if (!(isfinite(p.x) && isfinite(p.y) && isfinite(p.z))) continue;
    unsigned u[3] = {float_to_ordered(p.x), float_to_ordered(p.y), float_to_ordered(p.z)};
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      mn[a] = max(mn[a], ~u[a]);
      mx[a] = max(mx[a], u[a]);
    }
  }
#pragma unroll
  for (int a = 0; a < 3; ++a) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      mn[a] = max(mn[a], __shfl_xor_sync(0xffffffffu, mn[a], o));
      mx[a] = max(mx[a], __shfl_xor_sync(0xffffffffu, mx[a], o));
    }
  }
  // the block's extremes, then six atomics per block (atomics from every
  // warp on the same six words serialise: 39 us for 1216 blocks)
  __shared__ unsigned s_mn[3][8], s_mx[3][8];
  const int warp = threadIdx.x >> 5;
  if ((threadIdx.x & 31) == 0) {
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      s_mn[a][warp] = mn[a];
      s_mx[a][warp] = mx[a];
    }
  }
  __syncthreads();
  if (threadIdx.x < 3) {
    const int a = threadIdx.x;
    unsigned lo = s_mn[a][0], hi = s_mx[a][0];
    for (int w = 1; w < (int)(blockDim.x >> 5); ++w) {
      lo = max(lo, s_mn[a][w]);
      hi = max(hi, s_mx[a][w]);
    }
    atomicMax(&m->nmin[a], lo);
    atomicMax(&m->bmax[a], hi);
  }
  if (SETUP) {
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0 && atomicAdd(&m->ticket, 1u) == gridDim.x - 1) {
      __threadfence();
      grid_setup(m, h_req, cell_cap, n);
    }
  }
}

__device__ __forceinline__ int clampi(int v, int lo, int hi) { return v < lo ? lo : (v > hi ? hi : v); }

__device__ __forceinline__ int cell_of(float v, float o, float inv_h) {
  float f = __fmul_rn(__fsub_rn(v, o), inv_h);
  f = fminf(fmaxf(f, -1.0e8f), 1.0e8f);
  return (int)floorf(f);
}

// Cell of every point, counted into the table (which starts zeroed), and the
// point's rank in its cell in the order the counts were taken.  Lanes with
// the same cell are counted by one atomic: points that come in voxel order
// share cells, and a cell holding the whole cloud would otherwise serialise
// an atomic per point.  COUNT false: the cells alone (the ordered form counts
// them once they are sorted).
template <bool COUNT>
__global__ void __launch_bounds__(256) k_grid_count(const float4* __restrict__ pts, int n_host, const int* d_n,
                                                    const GridMeta* __restrict__ m, uint32_t* __restrict__ keys,
                                                    uint32_t* __restrict__ rank, uint32_t* __restrict__ counts) {
  const int n = count_of(n_host, d_n);
  const float ox = m->ox, oy = m->oy, oz = m->oz, ih = m->inv_h;
  const int nx = m->nx, ny = m->ny, nz = m->nz;
  const int lane = threadIdx.x & 31;
  const unsigned lt = lanemask_lt();
  for (int i0 = blockIdx.x * blockDim.x + (threadIdx.x & ~31); i0 < n; i0 += gridDim.x * blockDim.x) {
    const int i = i0 + lane;
    uint32_t key = 0xffffffffu;  // no cell: ncells stays below it
    if (i < n) {
      const float4 p = pts[i];
      const int cx = clampi(cell_of(p.x, ox, ih), 0, nx - 1);
      const int cy = clampi(cell_of(p.y, oy, ih), 0, ny - 1);
      const int cz = clampi(cell_of(p.z, oz, ih), 0, nz - 1);
      key = ((uint32_t)cz * (uint32_t)ny + (uint32_t)cy) * (uint32_t)nx + (uint32_t)cx;
    }
    if (!COUNT) {
      if (i < n) keys[i] = key;
      continue;
    }
    const unsigned peers = __match_any_sync(0xffffffffu, key);
    const int leader = __ffs(peers) - 1;
    uint32_t base = 0;
    if (i < n && lane == leader) base = atomicAdd(&counts[key], (uint32_t)__popc(peers));
    base = __shfl_sync(0xffffffffu, base, leader);
    if (i < n) {
      keys[i] = key;
      rank[i] = base + __popc(peers & lt);
    }
  }
}

// The table's exclusive scan in place, two launches: sums of its tiles, then
// each block adds up the tiles before its own and scans its tile.
constexpr int CT_BLOCK = 256, CT_ITEMS = 16, CT_TILE = CT_BLOCK * CT_ITEMS;
__global__ void __launch_bounds__(CT_BLOCK) k_cells_sums(const uint32_t* __restrict__ counts,
                                                         const GridMeta* __restrict__ m,
                                                         uint32_t* __restrict__ tiles) {
  const unsigned nc = m->ncells, base = blockIdx.x * (unsigned)CT_TILE;
  if (base >= nc) return;
  uint32_t s = 0;
#pragma unroll
  for (int j = 0; j < CT_ITEMS; ++j) {
    const unsigned c = base + j * CT_BLOCK + threadIdx.x;
    s += c < nc ? counts[c] : 0u;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  __shared__ uint32_t ws[CT_BLOCK / 32];
  if ((threadIdx.x & 31) == 0) ws[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    uint32_t t = 0;
#pragma unroll
    for (int w = 0; w < CT_BLOCK / 32; ++w) t += ws[w];
    tiles[blockIdx.x] = t;
  }
}

__global__ void __launch_bounds__(CT_BLOCK) k_cells_scan(uint32_t* __restrict__ counts,
                                                         const GridMeta* __restrict__ m,
                                                         const uint32_t* __restrict__ tiles) {
  const unsigned nc = m->ncells, base = blockIdx.x * (unsigned)CT_TILE;
  if (base >= nc) return;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t before = 0;
  for (unsigned t = threadIdx.x; t < blockIdx.x; t += CT_BLOCK) before += tiles[t];
  // whole lines in and out, a thread's entries side by side in between (2.4M
  // cells: 12.6 us with each thread walking its own 64 bytes, 4.9 so)
  __shared__ uint32_t tile[CT_TILE + CT_TILE / 32];  // (one word of padding a row of 32)
  uint32_t v[CT_ITEMS], s = 0;
#pragma unroll
  for (int j = 0; j < CT_ITEMS; ++j) {
    const unsigned i = (unsigned)j * CT_BLOCK + threadIdx.x;
    v[j] = base + i < nc ? counts[base + i] : 0u;
  }
#pragma unroll
  for (int j = 0; j < CT_ITEMS; ++j) {
    const unsigned i = (unsigned)j * CT_BLOCK + threadIdx.x;
    tile[i + (i >> 5)] = v[j];
  }
  __syncthreads();
#pragma unroll
  for (int j = 0; j < CT_ITEMS; ++j) {
    const unsigned i = threadIdx.x * CT_ITEMS + (unsigned)j;
    v[j] = tile[i + (i >> 5)];
    s += v[j];
  }
  uint32_t inc = s;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t t = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= o) inc += t;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) before += __shfl_xor_sync(0xffffffffu, before, o);
  __shared__ uint32_t ws[CT_BLOCK / 32], wb[CT_BLOCK / 32];
  if (lane == 31) ws[warp] = inc;
  if (lane == 0) wb[warp] = before;
  __syncthreads();
  uint32_t run = inc - s;
#pragma unroll
  for (int w = 0; w < CT_BLOCK / 32; ++w) run += wb[w] + (w < warp ? ws[w] : 0u);
#pragma unroll
  for (int j = 0; j < CT_ITEMS; ++j) {
    const unsigned i = threadIdx.x * CT_ITEMS + (unsigned)j;
    tile[i + (i >> 5)] = run;
    run += v[j];
    if (base + i + 1 == nc) counts[nc] = run;  // the end of the last cell
  }
  __syncthreads();
#pragma unroll
  for (int j = 0; j < CT_ITEMS; ++j) {
    const unsigned i = (unsigned)j * CT_BLOCK + threadIdx.x;
    if (base + i < nc) counts[base + i] = tile[i + (i >> 5)];
  }
}

__global__ void __launch_bounds__(256) k_grid_scatter(const float4* __restrict__ pts,
                                                      const uint32_t* __restrict__ keys,
                                                      const uint32_t* __restrict__ rank,
                                                      const uint32_t* __restrict__ starts, int n_host,
                                                      const int* d_n, float4* __restrict__ out) {
  const int n = count_of(n_host, d_n);
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    float4 p = pts[i];
    p.w = __int_as_float(i);  // original index travels with the point
    out[starts[keys[i]] + rank[i]] = p;
  }
}

// Points in sorted order, and the sorted cells counted into the table (which
// starts zeroed): neighbours share a cell, so there is about an atomic a cell
// and warp, where counting the points as they come takes an atomic per point
// of a cloud in random order, many on one word when cells are large (300k
// points at random in 2,400 cells, grid and 500 queries: 328 -> 310 us).
__global__ void __launch_bounds__(256) k_grid_gather(const float4* __restrict__ pts,
                                                     const uint32_t* __restrict__ keys,
                                                     const uint32_t* __restrict__ order, int n_host,
                                                     const int* d_n, uint32_t* __restrict__ counts,
                                                     float4* __restrict__ out) {
  const int n = count_of(n_host, d_n), lane = threadIdx.x & 31;
  for (int i0 = blockIdx.x * blockDim.x + (threadIdx.x & ~31); i0 < n; i0 += gridDim.x * blockDim.x) {
    const int i = i0 + lane;
    const uint32_t key = i < n ? keys[i] : 0xffffffffu;
    const unsigned peers = __match_any_sync(0xffffffffu, key);
    if (i < n) {
      if (lane == __ffs(peers) - 1) atomicAdd(&counts[key], (uint32_t)__popc(peers));
      const uint32_t o = order[i];
      float4 p = pts[o];
      p.w = __int_as_float((int)o);
      out[i] = p;
    }
  }
}

// The header and the table are one allocation, cleared together.
static size_t table_bytes(unsigned cell_cap) { return 256 + ((size_t)cell_cap + 1) * sizeof(uint32_t); }
static_assert(sizeof(GridMeta) <= 256, "the table follows the header");
static unsigned table_tiles(unsigned cell_cap) { return (cell_cap + CT_TILE - 1) / CT_TILE; }

void grid_plan(ScratchPlan& plan, int n_cap, unsigned cell_cap, bool ordered) {
  int n = n_cap > 0 ? n_cap : 1;
  plan.add<char>(table_bytes(cell_cap));
  plan.add<uint32_t>(table_tiles(cell_cap));
  plan.add<float4>(n);
  for (int i = 0; i < (ordered ? 4 : 2); ++i) plan.add<uint32_t>(n);
  if (ordered) plan.add<uint32_t>(radix_hist_entries(n));
}

bool grid_take(Scratch& s, int n_cap, unsigned cell_cap, GridBufs* b, bool ordered) {
  int n = n_cap > 0 ? n_cap : 1;
  char* t = s.take<char>(table_bytes(cell_cap));
  b->meta = reinterpret_cast<GridMeta*>(t);
  b->starts = t ? reinterpret_cast<uint32_t*>(t + 256) : nullptr;
  b->tiles = s.take<uint32_t>(table_tiles(cell_cap));
  b->pts = s.take<float4>(n);
  b->k0 = s.take<uint32_t>(n);
  b->v0 = s.take<uint32_t>(n);
  b->k1 = ordered ? s.take<uint32_t>(n) : nullptr;
  b->v1 = ordered ? s.take<uint32_t>(n) : nullptr;
  b->hist = ordered ? s.take<uint32_t>(radix_hist_entries(n)) : nullptr;
  b->n_cap = n_cap;
  b->cell_cap = cell_cap;
  return b->meta && b->tiles && b->pts && b->k0 && b->v0 && (!ordered || (b->k1 && b->v1 && b->hist));
}

static int grid_blocks(int n) {
  int b = (n + 255) / 256;
  if (b < 1) b = 1;
  if (b > 152 * 8) b = 152 * 8;
  return b;
}
// Blocks of a reduction to a few words: two per SM at most.
static int bbox_blocks(int n) {
  int b = (n + 255) / 256;
  if (b < 1) b = 1;
  if (b > 152 * 2) b = 152 * 2;
  return b;
}

rtr_status bbox_build(GridMeta* m, const float4* pts, int n, cudaStream_t st) {
  return bbox_build(m, pts, n, nullptr, st);
}

rtr_status bbox_build(GridMeta* m, const float4* pts, int n_cap, const int* d_n, cudaStream_t st) {
  RTR_CUDA(cudaMemsetAsync(m, 0, sizeof(GridMeta), st));
  k_bbox<false><<<bbox_blocks(n_cap), 256, 0, st>>>(pts, n_cap, d_n, m, 0.f, 0u);
  RTR_LAUNCHED(1);
  return RTR_OK;
}

// One memset and five launches: box and layout, count, two for the scan of
// the table, scatter.  Sorting the points by cell instead (radix passes,
// gather, table clear and bounds: 12 to 14 launches) took 99 us on the room's
// 213k voxels at 4 cm; this takes 45 us.  The ordered form keeps that
// sort, for the searches whose output order follows the points of a cell.
rtr_status grid_build(const GridBufs& b, const float4* pts, int n_host, const int* d_n, float h_req, cudaStream_t st,
                      bool ordered) {
  const int nb = grid_blocks(b.n_cap);
  const unsigned nt = table_tiles(b.cell_cap);
  RTR_CUDA(cudaMemsetAsync(b.meta, 0, table_bytes(b.cell_cap), st));
  k_bbox<true><<<bbox_blocks(b.n_cap), 256, 0, st>>>(pts, n_host, d_n, b.meta, h_req, b.cell_cap);
  if (ordered) {
    k_grid_count<false><<<nb, 256, 0, st>>>(pts, n_host, d_n, b.meta, b.k0, nullptr, nullptr);
    int bits = 1;
    while (bits < 32 && (1ull << bits) < (unsigned long long)b.cell_cap) ++bits;
    uint32_t *ks, *vs;
    RTR_TRY(radix_sort_pairs(nullptr, b.k0, b.v0, b.k1, b.v1, b.hist, b.n_cap, n_host, d_n, bits, true, st, &ks, &vs));
    k_grid_gather<<<nb, 256, 0, st>>>(pts, ks, vs, n_host, d_n, b.starts, b.pts);
  } else {
    k_grid_count<true><<<nb, 256, 0, st>>>(pts, n_host, d_n, b.meta, b.k0, b.v0, b.starts);
  }
  k_cells_sums<<<nt, CT_BLOCK, 0, st>>>(b.starts, b.meta, b.tiles);
  k_cells_scan<<<nt, CT_BLOCK, 0, st>>>(b.starts, b.meta, b.tiles);
  if (!ordered) k_grid_scatter<<<nb, 256, 0, st>>>(pts, b.k0, b.v0, b.starts, n_host, d_n, b.pts);
  RTR_LAUNCHED(5);
  RTR_CUDA(cudaGetLastError());
  return RTR_OK;
}

}  // namespace rtr
